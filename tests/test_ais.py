"""Annealed importance sampling (deepnet/ais.py:131-208) on the matrix API: the CPU restatement
against exact enumeration, and the device run against both."""
import numpy as np
import pytest

from deepnet_b200 import ais


def small_rbm(V=12, H=10, scale=0.5, seed=3):
    rng = np.random.default_rng(seed)
    return ((rng.standard_normal((V, H)) * scale).astype(np.float32),
            (rng.standard_normal(H) * 0.3).astype(np.float32), (rng.standard_normal(V) * 0.3).astype(np.float32))


def brute_force_log_z(w, a, b):
    V, H = w.shape
    x = ((np.arange(1 << V)[None, :] >> np.arange(V)[:, None]) & 1).astype(np.float64)
    act = w.astype(np.float64).T @ x + a.astype(np.float64)[:, None]
    lp = np.logaddexp(0, act).sum(axis=0) + b.astype(np.float64) @ x
    return lp.max() + np.log(np.exp(lp - lp.max()).sum())


def test_exact_enumeration_matches_numpy(oracle):
    w, a, b = small_rbm()
    assert abs(ais.exact_log_z(oracle, w, a, b) - brute_force_log_z(w, a, b)) < 1e-4


def test_ais_on_the_cpu_restatement_agrees_with_enumeration(oracle):
    w, a, b = small_rbm()
    schedule = np.linspace(0.0, 1.0, 400)
    log_z, logw = ais.ais_binary_rbm(oracle, w, a, b, 512, schedule, seed=5, fused=False)
    assert logw.shape == (512,)
    assert abs(log_z - brute_force_log_z(w, a, b)) < 0.15


def test_zero_rbm_has_log_z_of_the_uniform_model(oracle):
    V, H = 8, 6
    log_z, logw = ais.ais_binary_rbm(oracle, np.zeros((V, H)), np.zeros(H), np.zeros(V), 16, np.linspace(0, 1, 5),
                                     fused=False)
    assert np.allclose(logw, 0.0) and abs(log_z - (V + H) * np.log(2)) < 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("fused", [False, True])
def test_ais_on_the_device_matches_the_cpu_restatement(cm, oracle, fused):
    w, a, b = small_rbm(V=16, H=24)
    schedule = np.linspace(0.0, 1.0, 300)
    want, logw_o = ais.ais_binary_rbm(oracle, w, a, b, 256, schedule, seed=7, fused=False)
    got, logw_g = ais.ais_binary_rbm(cm, w, a, b, 256, schedule, seed=7, fused=fused)
    # same random stream: the chains coincide unless a probability lands within rounding of its uniform
    close = np.abs(logw_g - logw_o) < 1e-3 * np.maximum(1.0, np.abs(logw_o))
    assert close.mean() > 0.95
    assert abs(got - want) < 0.05
    assert abs(got - brute_force_log_z(w, a, b)) < 0.25
    assert abs(ais.exact_log_z(cm, w, a, b) - brute_force_log_z(w, a, b)) < 1e-3


@pytest.mark.gpu
def test_ais_at_layer_sizes_of_the_reference_models(cm):
    # 784 x 500 RBM, small weights: against the second-order cumulant expansion of
    # log E[exp(v'Wh)] under the uniform distribution (E[v_i h_j] = 1/4, Var = 3/16, covariance
    # 1/16 between entries that share a unit); the next cumulant is below 0.1 at this scale
    rng = np.random.default_rng(11)
    V, H = 784, 500
    w = (rng.standard_normal((V, H)) * 0.01).astype(np.float32)
    log_z, logw = ais.ais_binary_rbm(cm, w, np.zeros(H), np.zeros(V), 128, np.linspace(0, 1, 200), seed=1)
    assert np.isfinite(log_z) and logw.std() < 1.0
    w64 = w.astype(np.float64)
    sq = (w64 ** 2).sum()
    var = 3.0 / 16 * sq + 1.0 / 16 * ((w64.sum(axis=1) ** 2).sum() - sq + (w64.sum(axis=0) ** 2).sum() - sq)
    want = (V + H) * np.log(2) + w64.sum() / 4 + var / 2
    assert abs(log_z - want) < 0.5


ONE_LAUNCH, PRODUCTS = 1, 2


@pytest.fixture
def ais_form(cm):
    yield cm._lib.b200_test_ais_form
    cm._lib.b200_test_ais_form(0)


@pytest.mark.gpu
@pytest.mark.parametrize("form", [ONE_LAUNCH, PRODUCTS])
@pytest.mark.parametrize("col0", [0, 3])
@pytest.mark.parametrize("V,H,B", [(301, 517, 5), (17, 33, 203), (260, 255, 1), (260, 132, 137)])
def test_annealing_steps_match_the_call_by_call_form(cm, ais_form, form, col0, V, H, B):
    """The steps issued from C, in either form, against the reference's calls on the device, chain by chain: layers of more than
    one pass of a block and odd ones, products of both kernels, nonzero biases, a shard whose first column is not a multiple of
    four.  Both consume one random stream; a draw may differ where two correct probabilities straddle its uniform, about one
    in 10^7."""
    w, a, b = small_rbm(V=V, H=H, scale=0.1, seed=V)
    schedule = np.linspace(0.0, 1.0, 8)
    assert ais_form(form) == 0
    cm.set_rng_column_offset(col0)
    try:
        got, want = (ais.ais_binary_rbm(cm, w, a, b, B, schedule, seed=9, fused=fused) for fused in (True, False))
    finally:
        cm.set_rng_column_offset(0)
    # bound: fp32 sums of V + H terms a step, whose sizes are those of the log weights' own parts
    np.testing.assert_allclose(got[1], want[1], rtol=0, atol=1e-4 * np.abs(want[1]).max() + 1e-3)
    assert cm.CUDAMatrix.rnd_state.calls == 1 + 2 * (len(schedule) - 1)


@pytest.mark.gpu
@pytest.mark.parametrize("V,H,B,steps", [(784, 500, 100, 20), (64, 9, 1, 4), (97, 128, 33, 300), (1024, 129, 37, 5), (5, 3, 2, 3),
                                         (1023, 600, 20, 4), (1999, 70, 17, 3), (2001, 9, 3, 2), (1024, 1024, 120, 3)])
def test_annealing_in_one_launch_matches_the_products(cm, ais_form, V, H, B, steps):
    """All steps in one launch against three launches a step (the products on CUDA cores), chain by chain, with the states both
    leave: columns left in global memory (some of them, all, of whole and of ragged quads of rows), fewer hidden units than
    blocks, more temperatures than travel with a launch, 1 to 16 chains a cluster.  The draws are the same ones: a chain may go
    elsewhere where two correct probabilities straddle a uniform (one draw in 10^7; only the longest run has that many)."""
    w, a, b = small_rbm(V=V, H=H, scale=0.05, seed=V)
    schedule = np.linspace(0.0, 1.0, steps + 1)
    rng = np.random.default_rng(V)
    start, host = (rng.random((V, B)) < 0.5).astype(np.float32), {}
    for form, path in ((ONE_LAUNCH, 0), (PRODUCTS, 2)):
        m = dict(v_state=cm.CUDAMatrix(np.full((V, B), 0.5, np.float32)), v_sample=cm.CUDAMatrix(start), h_pre=cm.empty((H, B)),
                 h_sample=cm.empty((H, B)), weights=cm.empty((1, B)))
        W = cm.CUDAMatrix(w)
        cm.CUDAMatrix.init_random(9)
        assert ais_form(form) == 0
        cm.set_gemm_path(path)
        try:
            cm.ais_binary_steps(W, W.split_bf16(cm.empty_aux((V, H))), cm.CUDAMatrix(a.reshape(H, 1)), cm.CUDAMatrix(b.reshape(V, 1)),
                                schedule=schedule, **m)
        finally:
            cm.set_gemm_path(0)
        assert cm.CUDAMatrix.rnd_state.calls == 2 * steps
        host[form] = {k: np.array(x.asarray()) for k, x in m.items()}
    got, want = host[ONE_LAUNCH], host[PRODUCTS]
    assert all(np.isfinite(x).all() for x in got.values())
    # bound: the log weights of the other form are fp32 sums over `steps` of fp32 sums of V + H terms
    same = np.abs(got["weights"] - want["weights"])[0] <= 1e-4 * np.abs(want["weights"]).max() + 1e-3
    assert (~same).sum() <= (1 if steps * (V + H) * B > 10 ** 6 else 0)
    for k in ("v_sample", "h_sample"):
        np.testing.assert_array_equal(got[k][:, same], want[k][:, same])
    np.testing.assert_allclose(got["v_state"][:, same], want["v_state"][:, same], rtol=0, atol=1e-5)
    np.testing.assert_allclose(got["h_pre"][:, same], want["h_pre"][:, same], rtol=0, atol=1e-5 * np.abs(want["h_pre"]).max())
    assert cm.read_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("V,H,B", [(300, 200, 40), (97, 33, 5), (1023, 301, 9)])
def test_annealing_starts_from_states_of_any_value(cm, ais_form, V, H, B):
    """Means and counts, not only 0 and 1: the first pre-activations of the form in one launch, against float64.  Bound: 2^-24 a
    sum of doubles rounded once, and the bias added."""
    w, a, b = small_rbm(V=V, H=H, scale=0.1, seed=V)
    rng = np.random.default_rng(B)
    v = rng.random((V, B)).astype(np.float32)
    v[:, 0] = rng.integers(0, 1000, V)
    h_pre, W = cm.empty((H, B)), cm.CUDAMatrix(w)
    cm.CUDAMatrix.init_random(2)
    assert ais_form(ONE_LAUNCH) == 0
    cm.ais_binary_steps(W, W.split_bf16(cm.empty_aux((V, H))), cm.CUDAMatrix(a.reshape(H, 1)), cm.CUDAMatrix(b.reshape(V, 1)),
                        cm.CUDAMatrix(v), cm.CUDAMatrix(v), h_pre, cm.empty((H, B)), cm.empty((1, B)), [0.0, 0.5])
    want = w.T.astype(np.float64) @ v + a[:, None]
    assert (np.abs(np.array(h_pre.asarray()) - want).max(axis=0) <= 2e-7 * np.abs(want).max(axis=0)).all()


@pytest.mark.gpu
def test_annealing_takes_one_launch_only_where_that_is_faster(cm):
    """Measured, us a step, one launch / products: 784 x 500 with 100 chains 10.5 / 25, with 500 43 / 39, with 2048 137 / 60; 2000 x
    500 with 250 chains 72 / 42."""
    takes = lambda V, H, B, steps: cm._lib.b200_test_ais_in_one_launch(V, H, B, steps + 1)
    assert takes(784, 500, 100, 100) and takes(784, 500, 250, 100) and takes(64, 64, 250, 10)
    assert not takes(784, 500, 500, 100) and not takes(784, 500, 1000, 100) and not takes(784, 500, 2048, 100)
    assert not takes(2000, 500, 250, 100) and not takes(784, 500, 100, 1)


@pytest.mark.gpu
def test_annealing_of_layers_far_beyond_shared_memory_takes_the_products(cm):
    """Sizes that wrap around 2^31 when a block's shared memory is added up."""
    for units in (460174946, 460175205, 2 ** 31 - 100):
        assert not cm._lib.b200_test_ais_in_one_launch(units, 1, 1, 101)
        assert not cm._lib.b200_test_ais_in_one_launch(1, units, 1, 101)


@pytest.mark.gpu
def test_annealing_steps_refuse_shapes_that_do_not_fit(cm):
    cm.CUDAMatrix.init_random(1)
    V, H, B = 12, 8, 5
    good = dict(w=(V, H), a=(H, 1), b=(V, 1), v_state=(V, B), v_sample=(V, B), h_pre=(H, B), h_sample=(H, B), weights=(1, B))

    def call(**shapes):
        m = {k: cm.empty(s) for k, s in dict(good, **shapes).items()}
        cm.ais_binary_steps(m["w"], m["w"].split_bf16(cm.empty_aux(m["w"].shape)), m["a"], m["b"], m["v_state"], m["v_sample"],
                            m["h_pre"], m["h_sample"], m["weights"], [0.0, 0.5, 1.0])

    call()
    for name, shape in (("w", (V, H + 1)), ("a", (H + 1, 1)), ("b", (V + 1, 1)), ("v_state", (V + 1, B)), ("v_sample", (V, B + 1)),
                        ("h_pre", (H, B + 1)), ("h_sample", (H + 1, B)), ("weights", (1, B - 1))):
        with pytest.raises(cm.CUDAMatException):
            call(**{name: shape})


def small_rs_rbm(V=30, H=8, seed=4):
    rng = np.random.default_rng(seed)
    return ((rng.standard_normal((V, H)) * 0.3).astype(np.float32), (rng.standard_normal(H) * 0.1).astype(np.float32),
            (rng.standard_normal(V) * 0.5).astype(np.float32))


def test_replicated_softmax_enumeration_against_brute_force():
    # tiny model: every document of D words over V words, every hidden configuration
    import itertools
    rng = np.random.default_rng(0)
    V, H, D = 3, 2, 3
    w, a, b = rng.standard_normal((V, H)), rng.standard_normal(H), rng.standard_normal(V)
    total = []
    for h in itertools.product((0, 1), repeat=H):
        h = np.array(h, float)
        for doc in itertools.product(range(V), repeat=D):      # word sequences, as the base-rate term D logsumexp counts them
            v = np.bincount(doc, minlength=V).astype(float)
            total.append(v @ w @ h + b @ v + D * (a @ h))
    want = ais.log_sum_exp(np.array(total))
    assert abs(ais.exact_log_z_replicated_softmax(w, a, b, D) - want) < 1e-9


def test_replicated_softmax_ais_on_the_cpu_restatement_agrees_with_enumeration(oracle):
    w, a, b = small_rs_rbm()
    D = 6
    schedule = np.linspace(0.0, 1.0, 300)
    log_z, logw = ais.ais_replicated_softmax(oracle, w, a, b, D, 256, schedule=schedule, seed=3, fused=False)
    assert logw.shape == (256,)
    assert abs(log_z - ais.exact_log_z_replicated_softmax(w, a, b, D)) < 0.15
    # a model without weights or hidden biases equals its base-rate model at f = 1
    z0, lw0 = ais.ais_replicated_softmax(oracle, np.zeros((5, 3)), np.zeros(3), b[:5], 4, 8, schedule=np.linspace(0, 1, 4),
                                         fused=False, base_rate_fraction=1.0)
    assert np.allclose(lw0, 0) and abs(z0 - (4 * ais.log_sum_exp(b[:5].astype(np.float64)) + 3 * np.log(2))) < 1e-6
    sched = ais.replicated_softmax_schedule()                   # deepnet/ais.py:62-68: 700 + 2000 + 5000 steps (+1 by rounding)
    assert len(sched) in (7700, 7701) and sched[0] == 0 and 0.9999 < sched[-1] < 1


@pytest.mark.gpu
@pytest.mark.parametrize("fused", [False, True])
def test_replicated_softmax_ais_on_the_device_matches_the_cpu_restatement(cm, oracle, fused):
    w, a, b = small_rs_rbm(V=60, H=10)
    D = 12
    schedule = np.linspace(0.0, 1.0, 200)
    want, logw_o = ais.ais_replicated_softmax(oracle, w, a, b, D, 128, schedule=schedule, seed=7, fused=False)
    got, logw_g = ais.ais_replicated_softmax(cm, w, a, b, D, 128, schedule=schedule, seed=7, fused=fused)
    assert cm.CUDAMatrix.rnd_state.calls == oracle._Rng.calls          # D calls per softmax draw, one per hidden draw
    # same random stream: chains coincide unless a value lands within rounding of a tie or a uniform
    close = np.abs(logw_g - logw_o) < 1e-3 * np.maximum(1.0, np.abs(logw_o))
    assert close.mean() > 0.9
    assert abs(got - want) < 0.1
    assert abs(got - ais.exact_log_z_replicated_softmax(w, a, b, D)) < 0.3
    assert cm.read_status() == 0


@pytest.mark.gpu
def test_fused_gumbel_draws_equal_the_call_by_call_loop(cm, oracle):
    rng = np.random.default_rng(8)
    V, B, D = 500, 37, 9
    e = (rng.standard_normal((V, B)) * 2).astype(np.float32)
    counts = {}
    for backend in (cm, oracle):
        backend.CUDAMatrix.init_random(6)
        en, smp, tmp = backend.CUDAMatrix(e), backend.empty((V, B)), backend.empty((V, B))
        ais.sample_energy_softmax(backend, en, smp, tmp, D, fused=False)
        counts[backend] = np.array(smp.asarray(), copy=True)
    cm.CUDAMatrix.init_random(6)
    fused = cm.empty((V, B))
    cm.CUDAMatrix(e).sample_energy_softmax(fused, D)
    got = np.array(fused.asarray())
    np.testing.assert_array_equal(got, counts[cm])                    # same GPU arithmetic: identical counts
    assert np.abs(got - counts[oracle]).sum() <= 4                    # libm vs GPU logf may move a rare near-tie
    np.testing.assert_array_equal(got.sum(axis=0), np.full(B, D))
    assert cm.CUDAMatrix.rnd_state.calls == D
