"""GPU parity of the whole contrastive-divergence step: the per-call driver and the
fused engine on b200mat against the oracle-generated golden traces and against the
oracle run side by side; then size-independent properties at the full 8192 x 8192,
batch 4096 configuration.

Bounds: mean-field activations and gradients within 1e-5 relative (to the largest
magnitude), reconstruction-error curves within 2 %."""
import os

import numpy as np
import pytest

from deepnet_b200 import configs, dbm
from deepnet_b200.fused_rbm import FusedRBM

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
TOL = 1e-5


def get(m):
    return np.array(m.asarray(), copy=True)


def relerr(got, want):
    return np.abs(got - want).max() / max(np.abs(want).max(), 1e-30)


def assert_same_draws(got, want, p_got, p_want, full_size=False):
    """Bernoulli bits must be identical.  At a configuration's full size (millions of draws) a
    draw may differ where the two sides' probabilities, both inside the 1e-5 bound, fall on
    opposite sides of the shared uniform: allowed for at most two entries of the LAST draw (an
    earlier one would have sent the chains apart and failed every other check), and only where
    the probabilities do differ and by less than 2e-6."""
    bad = np.argwhere(got != want)
    if not full_size:
        assert len(bad) == 0, bad[:5]
        return
    assert len(bad) <= 2, len(bad)
    for r, c in bad:
        assert 0 < abs(float(p_got[r, c]) - float(p_want[r, c])) < 2e-6, (r, c, p_got[r, c], p_want[r, c])


def run_driver(backend, cfg, cases, steps):
    B = cfg["batchsize"]
    m = dbm.DBM(backend, cfg["layers"], cfg["edges"], cfg["hyperparams"], B, cfg["optimizer"], seed=cfg["seed"])
    data = backend.CUDAMatrix(cfg["data"])
    losses = []
    for step in range(steps):
        s = (step % (cases // B)) * B
        m.SetBatch([data.slice(s, s + B)])
        losses.append(m.TrainOneBatch(step)[0])
    return m, losses


@pytest.mark.parametrize("name,config,scale,cases,steps", [
    ("cd1_c0.npz", 0, 0.25, 300, 3), ("cd1_c1.npz", 1, 0.0625, 768, 3), ("pcd_c3.npz", 3, 0.1, 200, 2)])
def test_per_call_driver_matches_golden_trace(cm, name, config, scale, cases, steps):
    g = np.load(os.path.join(GOLDEN, name))
    cfg = configs.build(config, cases=cases, dims_scale=scale)
    m, losses = run_driver(cm, cfg, cases, steps)
    np.testing.assert_allclose(losses, g["losses"], rtol=1e-5)
    for i, e in enumerate(m.edge):
        assert relerr(get(e.params["weight"]), g["W%d" % i]) < TOL
        assert relerr(get(e.gradient_history), g["dW%d" % i]) < 2 * TOL
    for l in m.layer:
        assert relerr(get(l.state), g["state_" + l.name]) < TOL, l.name
        assert np.abs(get(l.params["bias"]) - g["b_" + l.name]).max() < 1e-6
    assert cm.read_status() == 0


@pytest.mark.parametrize("scale", [0.02, 1.0])
def test_replicated_softmax_step_matches_oracle(cm, oracle, scale):
    # config 2 at 1/50 size and at full size: multinomial sampling of the visible layer (sample_input on)
    cfg = configs.build(2, cases=200, dims_scale=scale)
    mg, lg = run_driver(cm, cfg, 200, 2)
    mo, lo = run_driver(oracle, cfg, 200, 2)
    np.testing.assert_allclose(lg, lo, rtol=1e-4)
    vg, vo = mg.GetLayerByName("v"), mo.GetLayerByName("v")
    np.testing.assert_array_equal(get(vg.sample), get(vo.sample))        # word counts: integers
    assert get(vg.sample).sum(axis=0) == pytest.approx(get(vg.NN).ravel(), abs=1e-3)
    assert relerr(get(mg.edge[0].params["weight"]), get(mo.edge[0].params["weight"])) < TOL


@pytest.mark.parametrize("config,scale,cases,form,gibbs", [
    (0, 0.25, 300, "derived", 1), (1, 0.0625, 768, "derived", 1), (0, 1.0, 200, "derived", 1),
    (0, 0.25, 300, "bf16 aux", 1), (0, 0.25, 300, "f16", 1), (0, 1.0, 200, "f16", 1),
    # 804 visible units: the 16-bit planes of a column are padded to 808 rows
    (0, 1.024, 300, "f16", 1), (0, 1.024, 300, "bf16 aux", 1),
    # configuration 1 at its full size (1024 x 4096, batch 256)
    (1, 1.0, 512, "derived", 1), (1, 1.0, 512, "bf16 aux", 1),
    # CD-k with k > 1: the intermediate Gibbs steps store only what the next product reads
    (0, 0.25, 300, "derived", 3), (4, 0.03125, 384, "f16", 10), (4, 0.03125, 384, "bf16 aux", 10),
    (4, 0.0625, 512, "f16", 10)])
def test_fused_engine_matches_oracle(cm, oracle, config, scale, cases, form, gibbs, monkeypatch):
    # the three forms the products' operands take: parts derived in the kernel (small models),
    # bfloat16 parts from aux matrices, scaled half precision (what the big binary model runs on)
    monkeypatch.setenv("B200_RBM_STATE_AUX", "0" if form == "derived" else "1")
    monkeypatch.setenv("B200_RBM_F16", "1" if form == "f16" else "0")
    cfg = configs.build(config, cases=cases, dims_scale=scale)
    if config == 4:
        # the benchmarked model (8192 x 8192, CD-10, batch 4096) shrunk until the CPU restatement
        # runs it in seconds: 256 units a side at batch 128 (one CTA per tile) and 512 at batch 256
        # (paired CTAs on 256 x 256 tiles, as at full size), the same ten Gibbs steps
        cfg["batchsize"] = 128 if scale < 0.05 else 256
    cfg["hyperparams"].gibbs_steps = gibbs
    B, steps = cfg["batchsize"], (3 if gibbs <= 3 else 2)
    mo, lo = run_driver(oracle, cfg, cases, steps)
    V, H = cfg["layers"][0]["numdims"], cfg["layers"][1]["numdims"]
    eng = FusedRBM(cm, V, H, B, cfg["edges"][0]["weight"], cfg["hyperparams"],
                   edge_hyperparams=cfg["edges"][0].get("hyperparams"), visible=cfg["layers"][0]["activation"],
                   binary_data=(config != 1), seed=cfg["seed"])
    assert eng.f16 == (form == "f16") and eng.state_aux == (form != "derived")
    data = cm.CUDAMatrix(cfg["data"])
    lg = []
    for step in range(steps):
        s = (step % (cases // B)) * B
        eng.TrainOneBatch(step, data.slice(s, s + B))
        lg.append(eng.read_loss())
    np.testing.assert_allclose(lg, lo, rtol=1e-5)
    assert relerr(get(eng.W), get(mo.edge[0].params["weight"])) < TOL
    assert relerr(get(eng.dW), get(mo.edge[0].gradient_history)) < 2 * TOL
    assert relerr(get(eng.h_neg), get(mo.GetLayerByName("h").state)) < TOL       # mean-field activations
    assert relerr(get(eng.v_neg), get(mo.GetLayerByName("v").state)) < TOL
    assert_same_draws(get(eng.h_samp), get(mo.GetLayerByName("h").sample), get(eng.h_neg),
                      get(mo.GetLayerByName("h").state), full_size=(config == 1 and scale == 1.0))   # Bernoulli bits
    assert np.abs(get(eng.bh) - get(mo.GetLayerByName("h").params["bias"])).max() < 1e-6
    assert cm.read_status() == 0


@pytest.mark.parametrize("form", ["derived", "bf16 aux", "f16"])
@pytest.mark.parametrize("branch", ["sample_input", "step_up_cd"])
def test_fused_engine_follows_the_step_schedules(cm, oracle, form, branch, monkeypatch):
    """deepnet/dbm.py:202-208 (a Gibbs step more every step_up_cd_after updates) and :217-222 (the
    visible layer feeds its Bernoulli draw upward): same random stream as the call-by-call driver."""
    monkeypatch.setenv("B200_RBM_STATE_AUX", "0" if form == "derived" else "1")
    monkeypatch.setenv("B200_RBM_F16", "1" if form == "f16" else "0")
    cases, steps = 300, 3
    cfg = configs.build(0, cases=cases, dims_scale=0.25)
    hyp = cfg["hyperparams"]
    if branch == "sample_input":
        hyp.sample_input, hyp.sample_input_after, hyp.gibbs_steps = True, 1, 2     # means at step 0, draws from step 1
    else:
        hyp.start_step_up_cd_after, hyp.step_up_cd_after = 1, 1                    # 1, 1, 3 Gibbs steps
    B = cfg["batchsize"]
    mo, lo = run_driver(oracle, cfg, cases, steps)
    V, H = cfg["layers"][0]["numdims"], cfg["layers"][1]["numdims"]
    eng = FusedRBM(cm, V, H, B, cfg["edges"][0]["weight"], hyp, edge_hyperparams=cfg["edges"][0].get("hyperparams"),
                   binary_data=True, seed=cfg["seed"])
    data = cm.CUDAMatrix(cfg["data"])
    lg = []
    for step in range(steps):
        eng.TrainOneBatch(step, data.slice(step * B, (step + 1) * B))
        lg.append(eng.read_loss())
    np.testing.assert_allclose(lg, lo, rtol=1e-5)
    assert cm.CUDAMatrix.rnd_state.calls == oracle._Rng.calls                      # same number of sampling calls
    assert relerr(get(eng.W), get(mo.edge[0].params["weight"])) < TOL
    assert relerr(get(eng.h_neg), get(mo.GetLayerByName("h").state)) < TOL
    assert relerr(get(eng.v_neg), get(mo.GetLayerByName("v").state)) < TOL
    np.testing.assert_array_equal(get(eng.h_samp), get(mo.GetLayerByName("h").sample))
    if branch == "sample_input" and form != "f16":                                 # (the f16 form keeps only the draw's 16-bit plane)
        np.testing.assert_array_equal(get(eng.v_samp), get(mo.GetLayerByName("v").sample))
    assert cm.read_status() == 0


@pytest.mark.parametrize("config,scale,cases", [(0, 0.25, 300), (2, 0.02, 200), (3, 0.1, 300)])
def test_recorded_step_equals_the_call_by_call_step(cm, config, scale, cases, monkeypatch):
    """The engines record their step once and replay it with one library call; issued operation by
    operation instead (B200_RBM_PROGRAM=0) the same kernels run in the same order: identical bits."""
    results = []
    for mode in ("1", "0"):
        monkeypatch.setenv("B200_RBM_PROGRAM", mode)
        cfg = configs.build(config, cases=cases, dims_scale=scale)
        B = cfg["batchsize"]
        if config == 3:
            from deepnet_b200.fused_dbm import FusedDBM
            eng = FusedDBM(cm, [l["numdims"] for l in cfg["layers"]], B, [e["weight"] for e in cfg["edges"]],
                           cfg["hyperparams"], seed=cfg["seed"])
        else:
            V, H = cfg["layers"][0]["numdims"], cfg["layers"][1]["numdims"]
            eng = FusedRBM(cm, V, H, B, cfg["edges"][0]["weight"], cfg["hyperparams"],
                           edge_hyperparams=cfg["edges"][0].get("hyperparams"), visible=cfg["layers"][0]["activation"],
                           binary_data=True, seed=cfg["seed"])
        assert eng.use_program == (mode == "1")
        data = cm.CUDAMatrix(cfg["data"])
        losses = []
        for step in range(3):
            s = (step % (cases // B)) * B
            eng.TrainOneBatch(step, data.slice(s, s + B))
            losses.append(eng.read_loss())
        W = eng.W if isinstance(eng.W, list) else [eng.W]
        results.append((losses, [get(w) for w in W], cm.CUDAMatrix.rnd_state.calls, eng.kernel_launches))
    assert results[0][0] == results[1][0]
    for a, b in zip(results[0][1], results[1][1]):
        np.testing.assert_array_equal(a, b)
    assert results[0][2] == results[1][2] and results[0][3] == results[1][3]
    assert cm.read_status() == 0


@pytest.mark.parametrize("config,scale,cases,form", [(0, 1.0, 400, None), (1, 0.25, 512, None), (2, 0.02, 200, None),
                                                     (3, 0.25, 300, None), (0, 0.5, 300, "f16")])
def test_dependent_launch_changes_no_bit(cm, config, scale, cases, form, monkeypatch):
    """With programmatic dependent launch every kernel of the step is scheduled while its predecessor
    drains and waits for it before touching memory: 20 updates give the bits of ordinary launches."""
    if form:
        monkeypatch.setenv("B200_RBM_STATE_AUX", "1")
        monkeypatch.setenv("B200_RBM_F16", "1")
    results = []
    try:
        for on in (True, False):
            cm.set_dependent_launch(on)
            cfg = configs.build(config, cases=cases, dims_scale=scale)
            B = cfg["batchsize"]
            if config == 3:
                from deepnet_b200.fused_dbm import FusedDBM
                eng = FusedDBM(cm, [l["numdims"] for l in cfg["layers"]], B, [e["weight"] for e in cfg["edges"]],
                               cfg["hyperparams"], seed=cfg["seed"])
            else:
                V, H = cfg["layers"][0]["numdims"], cfg["layers"][1]["numdims"]
                eng = FusedRBM(cm, V, H, B, cfg["edges"][0]["weight"], cfg["hyperparams"],
                               edge_hyperparams=cfg["edges"][0].get("hyperparams"),
                               visible=cfg["layers"][0]["activation"], binary_data=True, seed=cfg["seed"])
            data = cm.CUDAMatrix(cfg["data"])
            for step in range(20):
                s = (step % (cases // B)) * B
                eng.TrainOneBatch(step, data.slice(s, s + B))
            W = eng.W if isinstance(eng.W, list) else [eng.W]
            results.append((eng.read_loss(), [get(w) for w in W]))
    finally:
        cm.set_dependent_launch(True)
    assert results[0][0] == results[1][0]
    for a, b in zip(results[0][1], results[1][1]):
        np.testing.assert_array_equal(a, b)
    assert cm.read_status() == 0


def test_half_precision_engine_from_zero_weights(cm, oracle, monkeypatch):
    """W's exponent follows the weights from nothing to their first values (the update gathers the
    largest |W| and writes the half-precision form with the exponent that fits it)."""
    monkeypatch.setenv("B200_RBM_STATE_AUX", "1")
    monkeypatch.setenv("B200_RBM_F16", "1")
    cfg = configs.build(0, cases=300, dims_scale=0.25)
    cfg["edges"][0]["weight"] = np.zeros_like(cfg["edges"][0]["weight"])
    B, steps = cfg["batchsize"], 3
    mo, lo = run_driver(oracle, cfg, 300, steps)
    V, H = cfg["layers"][0]["numdims"], cfg["layers"][1]["numdims"]
    eng = FusedRBM(cm, V, H, B, cfg["edges"][0]["weight"], cfg["hyperparams"],
                   edge_hyperparams=cfg["edges"][0].get("hyperparams"), binary_data=True, seed=cfg["seed"])
    assert eng.f16
    data = cm.CUDAMatrix(cfg["data"])
    lg = []
    for step in range(steps):
        eng.TrainOneBatch(step, data.slice(step * B, (step + 1) * B))
        lg.append(eng.read_loss())
    np.testing.assert_allclose(lg, lo, rtol=1e-5)
    assert relerr(get(eng.W), get(mo.edge[0].params["weight"])) < TOL
    np.testing.assert_array_equal(get(eng.h_samp), get(mo.GetLayerByName("h").sample))
    assert cm.read_status() == 0


def test_fused_softmax_ops_match_the_call_sequence(cm, oracle):
    rng = np.random.default_rng(21)
    V, B = 400, 12
    pre = rng.standard_normal((V, B)).astype(np.float32) * 2
    lens = rng.integers(1, 60, (1, B)).astype(np.float32)
    lens[0, 3] = 1030                                   # more draws than the 1000-draw cap
    # activation: NN * softmax, against replicated_softmax_layer.py:12-21 issued call by call on the oracle
    st, tmp, nn = oracle.CUDAMatrix(pre), oracle.empty((1, B)), oracle.CUDAMatrix(lens)
    st.max(axis=0, target=tmp)
    st.add_row_mult(tmp, -1)
    oracle.exp(st)
    st.sum(axis=0, target=tmp)
    nn.divide(tmp, target=tmp)
    st.mult_by_row(tmp)
    g = cm.CUDAMatrix(pre).softmax_scaled(cm.CUDAMatrix(lens), target=cm.empty((V, B)))
    assert relerr(get(g), get(st)) < TOL
    # sampling: fused kernel vs the per-document loop of the call-by-call layer, same stream
    from deepnet_b200 import dbm
    counts = {}
    for backend in (cm, oracle):
        lay = dbm.ReplicatedSoftmaxLayer(backend, "v", V, dbm.Hyperparams(sample_input=True), is_input=True)
        lay.AllocateMemory(B)
        lay.state.assign(backend.CUDAMatrix(get(st)))
        lay.NN.assign(backend.CUDAMatrix(lens))
        backend.CUDAMatrix.init_random(5)
        lay.Sample()
        counts[backend] = get(lay.sample)
    cm.CUDAMatrix.init_random(5)
    fused = get(cm.CUDAMatrix(get(st)).sample_multinomial(cm.CUDAMatrix(lens), cm.empty((V, B))))
    np.testing.assert_array_equal(fused, counts[cm])          # same GPU arithmetic: identical counts
    assert np.abs(fused - counts[oracle]).sum() <= 4           # libm vs GPU logf may move a rare near-tie
    np.testing.assert_array_equal(fused.sum(axis=0), np.minimum(lens.ravel(), 1000))
    assert cm.CUDAMatrix.rnd_state.calls == B


@pytest.mark.parametrize("V", [512, 513, 4096, 4097, 9001])
def test_multinomial_draws_equal_the_call_sequence_at_any_vocabulary(cm, V):
    """Words that a bound rules out are passed over without their logarithm: the counts stay those of the per-document
    loop, word for word, also with words of probability zero, one dominant word, one usable word and none."""
    rng = np.random.default_rng(V)
    B = 5
    p = rng.random((V, B)).astype(np.float32) ** 8
    p[rng.random((V, B)) < 0.3] = 0.0
    p[V - 1, 1] = 50.0 * p[:, 1].sum()
    p[:, 2] = 0.0
    p[V // 2, 2] = 3.0
    p[:, 3] = 0.0
    lens = np.array([[40, 7, 9, 5, 1]], np.float32)
    cm.CUDAMatrix.init_random(8)
    lay = dbm.ReplicatedSoftmaxLayer(cm, "v", V, dbm.Hyperparams(sample_input=True), is_input=True)
    lay.AllocateMemory(B)
    lay.state.assign(cm.CUDAMatrix(p))
    lay.NN.assign(cm.CUDAMatrix(lens))
    cm.CUDAMatrix.init_random(8)
    lay.Sample()
    cm.CUDAMatrix.init_random(8)
    fused = get(cm.CUDAMatrix(p).sample_multinomial(cm.CUDAMatrix(lens), cm.empty((V, B))))
    np.testing.assert_array_equal(fused, get(lay.sample))
    np.testing.assert_array_equal(fused.sum(axis=0), lens.ravel())


@pytest.mark.parametrize("V", [10, 600, 5000])
def test_multinomial_draws_without_a_positive_word_equal_the_call_sequence(cm, V):
    """Values of either sign: where no word of the first is positive nothing bounds the race, and every word stays in it."""
    rng = np.random.default_rng(V)
    p = -rng.random((V, 2)).astype(np.float32) - 0.01
    p[V - 1, 1] = 0.5
    lens = np.array([[30, 9]], np.float32)
    lay = dbm.ReplicatedSoftmaxLayer(cm, "v", V, dbm.Hyperparams(sample_input=True), is_input=True)
    lay.AllocateMemory(2)
    lay.state.assign(cm.CUDAMatrix(p))
    lay.NN.assign(cm.CUDAMatrix(lens))
    cm.CUDAMatrix.init_random(8)
    lay.Sample()
    cm.CUDAMatrix.init_random(8)
    fused = get(cm.CUDAMatrix(p).sample_multinomial(cm.CUDAMatrix(lens), cm.empty((V, 2))))
    np.testing.assert_array_equal(fused, get(lay.sample))
    np.testing.assert_array_equal(fused[:, 1], 9.0 * (np.arange(V) == V - 1))


@pytest.mark.parametrize("scale", [0.02, 1.0])
def test_fused_engine_replicated_softmax_matches_oracle(cm, oracle, scale):
    # config 2 at 1/50 size and at its full size (10 000 words, 512 hidden units, documents of about
    # 100 words) through the fused engine against the call-by-call driver on the oracle
    cases = 200
    cfg = configs.build(2, cases=cases, dims_scale=scale)
    B, steps = cfg["batchsize"], 2
    mo, lo = run_driver(oracle, cfg, cases, steps)
    V, H = cfg["layers"][0]["numdims"], cfg["layers"][1]["numdims"]
    eng = FusedRBM(cm, V, H, B, cfg["edges"][0]["weight"], cfg["hyperparams"], visible=dbm.REPLICATED_SOFTMAX,
                   binary_data=True, seed=cfg["seed"])
    data = cm.CUDAMatrix(cfg["data"])
    lg = []
    for step in range(steps):
        eng.TrainOneBatch(step, data.slice(step * B, (step + 1) * B))
        lg.append(eng.read_loss())
    np.testing.assert_allclose(lg, lo, rtol=1e-4)
    np.testing.assert_array_equal(get(eng.v_samp), get(mo.GetLayerByName("v").sample))
    np.testing.assert_array_equal(get(eng.h_samp), get(mo.GetLayerByName("h").sample))
    assert relerr(get(eng.W), get(mo.edge[0].params["weight"])) < TOL
    assert relerr(get(eng.dW), get(mo.edge[0].gradient_history)) < 2 * TOL
    assert relerr(get(eng.v_neg), get(mo.GetLayerByName("v").state)) < TOL
    assert cm.read_status() == 0


def test_fused_dbm_matches_oracle(cm, oracle):
    # config 3 (784-500-1000 DBM, 10 mean-field + 5 Gibbs sweeps, PCD) at 1/10 and at full size
    from deepnet_b200.fused_dbm import FusedDBM
    for scale, cases, steps in ((0.1, 300, 3), (1.0, 200, 2)):
        cfg = configs.build(3, cases=cases, dims_scale=scale)
        B = cfg["batchsize"]
        mo, lo = run_driver(oracle, cfg, cases, steps)
        sizes = [l["numdims"] for l in cfg["layers"]]
        eng = FusedDBM(cm, sizes, B, [e["weight"] for e in cfg["edges"]], cfg["hyperparams"], seed=cfg["seed"])
        data = cm.CUDAMatrix(cfg["data"])
        lg = []
        for step in range(steps):
            s = (step % (cases // B)) * B
            eng.TrainOneBatch(step, data.slice(s, s + B))
            lg.append(eng.read_loss())
        np.testing.assert_allclose(lg, lo, rtol=1e-5)
        for i, e in enumerate(mo.edge):
            assert relerr(get(eng.W[i]), get(e.params["weight"])) < TOL
            assert relerr(get(eng.dW[i]), get(e.gradient_history)) < 2 * TOL
        for j, l in enumerate(mo.layer):
            assert relerr(get(eng.neg[j]), get(l.neg_state)) < TOL, l.name          # persistent particles
            assert relerr(get(eng.pos[j]), get(l.pos_state)) < TOL, l.name          # mean-field activations
            if j > 0:
                np.testing.assert_array_equal(get(eng.neg_sample[j]), get(l.neg_sample))
            assert np.abs(get(eng.b[j]) - get(l.params["bias"])).max() < 1e-6
    assert cm.read_status() == 0


@pytest.mark.parametrize("config,scale,cases", [(0, 0.25, 300), (1, 0.0625, 512), (2, 0.02, 200)])
def test_inference_path_matches_oracle(cm, oracle, config, scale, cases):
    # representation extraction: positive phase only, no sampling, no statistics (deepnet/dbm.py:340-398)
    cfg = configs.build(config, cases=cases, dims_scale=scale)
    B = cfg["batchsize"]
    mo = dbm.DBM(oracle, cfg["layers"], cfg["edges"], cfg["hyperparams"], B, cfg["optimizer"], seed=cfg["seed"])
    want = mo.Inference(oracle.CUDAMatrix(cfg["data"]), ["h"], input_recon=True)
    mg = dbm.DBM(cm, cfg["layers"], cfg["edges"], cfg["hyperparams"], B, cfg["optimizer"], seed=cfg["seed"])
    got = mg.Inference(cm.CUDAMatrix(cfg["data"]), ["h"], input_recon=True)
    assert relerr(got["h"], want["h"]) < TOL
    assert abs(got["error"] - want["error"]) < 1e-5 * want["error"]
    V, H = cfg["layers"][0]["numdims"], cfg["layers"][1]["numdims"]
    eng = FusedRBM(cm, V, H, B, cfg["edges"][0]["weight"], cfg["hyperparams"], visible=cfg["layers"][0]["activation"],
                   binary_data=(config != 1), seed=cfg["seed"])
    rep, err = eng.Inference(cm.CUDAMatrix(cfg["data"]), input_recon=True)
    assert rep.shape == want["h"].shape
    assert relerr(rep, want["h"]) < TOL
    assert abs(err - want["error"]) < 1e-5 * want["error"]


@pytest.mark.parametrize("form", ["derived", "f16"])
def test_reconstruction_error_curve_within_two_percent(cm, oracle, form, monkeypatch):
    monkeypatch.setenv("B200_RBM_STATE_AUX", "0" if form == "derived" else "1")
    monkeypatch.setenv("B200_RBM_F16", "1" if form == "f16" else "0")
    cases, steps = 1000, 60
    cfg = configs.build(0, cases=cases, dims_scale=0.25)
    B = cfg["batchsize"]
    _, lo = run_driver(oracle, cfg, cases, steps)
    V, H = cfg["layers"][0]["numdims"], cfg["layers"][1]["numdims"]
    eng = FusedRBM(cm, V, H, B, cfg["edges"][0]["weight"], cfg["hyperparams"],
                   edge_hyperparams=cfg["edges"][0].get("hyperparams"), binary_data=True, seed=cfg["seed"])
    data = cm.CUDAMatrix(cfg["data"])
    lg = []
    for step in range(steps):
        s = (step % (cases // B)) * B
        eng.TrainOneBatch(step, data.slice(s, s + B))
        lg.append(eng.read_loss())
    lo, lg = np.array(lo), np.array(lg)
    assert np.abs(lg - lo).max() / lo.max() < 0.02
    assert np.abs(lg / lo - 1).max() < 0.02
    assert lg[-1] < 0.6 * lg[0]


def _f16_planes(aux):
    """(lo, hi) planes of an aux matrix in scaled half-precision form, as float32."""
    raw = np.array(aux.asarray(), copy=True)
    words = np.ascontiguousarray(raw.T).view(np.uint16)
    lda = raw.shape[0]
    f = lambda w: np.ascontiguousarray(w).view(np.float16).astype(np.float32).T[:aux.rows]
    return f(words[:, :lda]), f(words[:, lda:])


def test_full_size_properties(cm):
    """Config 4 as benchmarked (V = H = 8192, batch 4096, CD-10): checks that do not need a CPU run
    of the step.  Every product kind of the update is pinned at inner dimension 8192 (4096 for
    the statistics) against float64 dot products of the operands it actually read."""
    V = H = 8192
    B = 4096
    rng = np.random.default_rng(44)
    W = (rng.standard_normal((V, H)) * 0.01).astype(np.float32)
    p = rng.beta(0.3, 2.0, size=(V, 1)).astype(np.float32)
    x = (rng.random((V, B), dtype=np.float32) < p).astype(np.float32)
    hyp = dbm.Hyperparams(base_epsilon=0.05, initial_momentum=0.9, final_momentum=0.9, gibbs_steps=10)
    eng = FusedRBM(cm, V, H, B, W, hyp, binary_data=True, seed=3004)
    assert eng.f16                       # at this size every product runs on scaled half-precision operands
    data = cm.CUDAMatrix(x)
    eng.TrainOneBatch(0, data)
    h_pos, h_samp, v_neg = get(eng.h_pos), get(eng.h_samp), get(eng.v_neg)
    sig = lambda t: 1 / (1 + np.exp(-t))
    # (1) the two-term up product on 0/1 data: sampled entries of the positive hidden
    # activations against float64 dot products
    idx = rng.integers(0, H, 200), rng.integers(0, B, 200)
    pre = np.einsum("ki,ki->i", W[:, idx[0]].astype(np.float64), x[:, idx[1]].astype(np.float64))
    assert np.abs(h_pos[idx] - sig(pre)).max() < TOL
    # (1b) the three-term up product on probabilities: the last hidden means against the last
    # visible means they were computed from (biases are still zero during the first update)
    h_neg = get(eng.h_neg)
    pre = np.einsum("ki,ki->i", W[:, idx[0]].astype(np.float64), v_neg[:, idx[1]].astype(np.float64))
    assert np.abs(h_neg[idx] - sig(pre)).max() < TOL
    # (1c) what the next product would read of those visible means: their half-precision planes
    lo, hi = _f16_planes(eng.v_neg_aux)
    cols = slice(0, 64)
    want_hi = (v_neg[:, cols] * np.float32(2.0 ** 14)).astype(np.float16).astype(np.float32)
    np.testing.assert_array_equal(hi[:, cols], want_hi)
    np.testing.assert_array_equal(lo[:, cols], (v_neg[:, cols] * np.float32(2.0 ** 14) - want_hi).astype(np.float16))
    # (2) Bernoulli draws are 0/1 and their mean tracks the mean probability (checksum of the draw);
    # h_samp holds the draw of the last negative-phase hidden state
    assert set(np.unique(h_samp)) <= {0.0, 1.0}
    assert abs(h_samp.mean() - h_neg.mean()) < 5 * 0.5 / np.sqrt(h_samp.size)
    np.testing.assert_array_equal(_f16_planes(eng.h_samp_aux)[1][:, cols], h_samp[:, cols] * 2.0 ** 14)
    # (3) statistics: row sums and the packed gradient against float64 on sampled entries
    sb = get(eng.suff_bh).ravel()
    np.testing.assert_allclose(sb, h_pos.astype(np.float64).sum(axis=1) - h_neg.astype(np.float64).sum(axis=1),
                               rtol=1e-5, atol=2e-3)
    ii, jj = rng.integers(0, V, 64), rng.integers(0, H, 64)
    want_s = (x[ii].astype(np.float64) * h_pos[jj]).sum(axis=1) - (v_neg[ii].astype(np.float64) * h_neg[jj]).sum(axis=1)
    suff = get(eng.suff_W)
    got_s = suff[ii, jj]
    assert np.abs(got_s - want_s).max() < TOL * np.abs(suff).max()     # gradients: 1e-5 of the largest
    # (4) the update applied what the statistics say: W1 = W0 - eps * (-(suff)/B) with zero history
    W1 = get(eng.W)
    want_w = W[ii, jj] - np.float32(0.05) * (-(got_s) / B)
    assert np.abs(W1[ii, jj] - want_w).max() < 1e-6
    # (5) the down product (W read along its rows, 0/1 hidden draws, inner dimension 8192) on the
    # updated parameters and their rewritten half-precision form
    out = cm.empty((V, B))
    cm.fused_gemm(cm.f16_passes(eng.W, eng.W_aux, eng.h_samp, eng.h_samp_aux, exact_b=True), out=out, bias=eng.bv,
                  activation=1, scale_exp=eng.W_exp, scale_exp_const=14)
    got_v, bv1 = get(out), get(eng.bv).ravel().astype(np.float64)
    vi, vb = rng.integers(0, V, 200), rng.integers(0, B, 200)
    pre = np.einsum("ik,ki->i", W1[vi, :].astype(np.float64), h_samp[:, vb].astype(np.float64)) + bv1[vi]
    assert np.abs(got_v[vi, vb] - sig(pre)).max() < TOL
    # (6) a zero learning rate leaves the parameters untouched (idempotence of the update path)
    eng.hyp.base_epsilon = 0.0
    eng.ehyp.base_epsilon = 0.0
    eng.TrainOneBatch(1, data)
    np.testing.assert_array_equal(get(eng.W), W1)
    assert cm.read_status() == 0


def joint_dbm_spec(seed=11, cases=120, B=40, sizes=(64, 48, 40, 32), labels=10):
    """A small DBM shaped like deepnet/examples/dbm/model.pbtxt: input - hidden1 - hidden2 - joint hidden,
    with a softmax label layer (a second input) attached to the joint layer (:57-81, :138-140)."""
    from deepnet_b200 import synthetic
    rng = np.random.default_rng(seed)
    V, H1, H2, J = sizes
    hyp = dbm.Hyperparams(base_epsilon=0.01, initial_momentum=0.5, final_momentum=0.9, momentum_change_steps=100,
                          apply_l2_decay=True, l2_decay=1e-4, mf_steps=5, gibbs_steps=5)
    layers = [dict(name="input_layer", activation=dbm.LOGISTIC, numdims=V, is_input=True),
              # an input layer feeds its means upward unless sample_input is set (deepnet/dbm.py:217-222)
              dict(name="label_layer", activation=dbm.SOFTMAX, numdims=labels, is_input=True,
                   hyperparams=hyp.copy(sample_input=True)),
              dict(name="hidden1", activation=dbm.LOGISTIC, numdims=H1),
              dict(name="hidden2", activation=dbm.LOGISTIC, numdims=H2),
              dict(name="joint_hidden", activation=dbm.LOGISTIC, numdims=J)]
    w = lambda r, c: (rng.standard_normal((r, c)) * 0.05).astype(np.float32)
    edges = [dict(node1="input_layer", node2="hidden1", weight=w(V, H1)),
             dict(node1="hidden1", node2="hidden2", weight=w(H1, H2)),
             dict(node1="hidden2", node2="joint_hidden", weight=w(H2, J)),
             dict(node1="label_layer", node2="joint_hidden", weight=w(labels, J))]
    data, _ = synthetic.binary_data(V, cases, seed)
    lab = rng.integers(0, labels, (1, cases)).astype(np.float32)
    return dict(layers=layers, edges=edges, hyp=hyp, B=B, data=data, labels=lab, seed=seed)


def run_joint_dbm(backend, spec, steps):
    m = dbm.DBM(backend, spec["layers"], spec["edges"], spec["hyp"], spec["B"], dbm.PCD, seed=spec["seed"])
    data, lab = backend.CUDAMatrix(spec["data"]), backend.CUDAMatrix(spec["labels"])
    B, losses = spec["B"], []
    for step in range(steps):
        m.SetBatch([data.slice(step * B, (step + 1) * B), lab.slice(step * B, (step + 1) * B)])
        losses.append(m.TrainOneBatch(step))
    return m, losses


def test_dbm_with_softmax_label_layer_matches_oracle(cm, oracle):
    """deepnet/softmax_layer.py on the path: the label layer is clamped to one-hot labels in the
    positive phase, reconstructed through a softmax, and drawn categorically in every Gibbs sweep."""
    spec = joint_dbm_spec()
    mg, lg = run_joint_dbm(cm, spec, 3)
    mo, lo = run_joint_dbm(oracle, spec, 3)
    np.testing.assert_allclose(lg, lo, rtol=1e-5)                     # both inputs' reconstruction errors
    assert cm.CUDAMatrix.rnd_state.calls == oracle._Rng.calls
    lab_g, lab_o = mg.GetLayerByName("label_layer"), mo.GetLayerByName("label_layer")
    np.testing.assert_array_equal(get(lab_g.neg_sample), get(lab_o.neg_sample))       # categorical draws
    assert np.array_equal(get(lab_g.neg_sample).sum(axis=0), np.ones(spec["B"]))      # one label per case
    assert relerr(get(lab_g.neg_state), get(lab_o.neg_state)) < TOL                   # softmax probabilities
    for eg, eo in zip(mg.edge, mo.edge):
        assert relerr(get(eg.params["weight"]), get(eo.params["weight"])) < TOL, eg.name
    for l_g, l_o in zip(mg.layer, mo.layer):
        assert relerr(get(l_g.pos_state), get(l_o.pos_state)) < TOL, l_g.name
        if l_g.name != "input_layer":
            np.testing.assert_array_equal(get(l_g.neg_sample), get(l_o.neg_sample))
    assert cm.read_status() == 0


@pytest.mark.parametrize("labels,B", [(10, 100), (1000, 37), (4, 5)])
def test_fused_softmax_and_categorical_draw_match_the_call_sequence(cm, oracle, labels, B):
    rng = np.random.default_rng(labels)
    pre = (rng.standard_normal((labels, B)) * 2).astype(np.float32)
    bias = rng.standard_normal((labels, 1)).astype(np.float32)
    # the reference's calls on the oracle: add_col_vec, apply_softmax, perturb_prob, choose_max
    oracle.EigenMatrix.init_random(9)
    st = oracle.EigenMatrix(pre)
    st.add_col_vec(oracle.EigenMatrix(bias))
    st.apply_softmax()
    smp = oracle.empty((labels, B))
    st.perturb_prob_for_softmax_sampling(target=smp)
    smp.choose_max(axis=0)
    cm.CUDAMatrix.init_random(9)
    g_state, g_smp = cm.empty((labels, B)), cm.empty((labels, B))
    cm.CUDAMatrix(pre).softmax_sample(g_state, g_smp, bias=cm.CUDAMatrix(bias))
    assert relerr(get(g_state), get(st)) < TOL
    np.testing.assert_array_equal(get(g_smp), get(smp))
    assert cm.CUDAMatrix.rnd_state.calls == 1
    # activation only: no sampling call consumed
    cm.CUDAMatrix(pre).softmax_sample(g_state, None)
    assert cm.CUDAMatrix.rnd_state.calls == 1


def test_loss_read_back_behind_the_updates(cm):
    """loss_begin / loss_end hand back every update's loss one update later, without a blocking read
    in between: the same numbers as read_loss after each update."""
    cfg = configs.build(0, cases=400, dims_scale=0.25)
    B = cfg["batchsize"]
    V, H = cfg["layers"][0]["numdims"], cfg["layers"][1]["numdims"]
    data_host = cfg["data"]
    want, got = [], []
    for mode in ("blocking", "behind"):
        eng = FusedRBM(cm, V, H, B, cfg["edges"][0]["weight"], cfg["hyperparams"],
                       edge_hyperparams=cfg["edges"][0].get("hyperparams"), binary_data=True, seed=cfg["seed"])
        data = cm.CUDAMatrix(data_host)
        for step in range(4):
            eng.TrainOneBatch(step, data.slice(step * B, (step + 1) * B))
            if mode == "blocking":
                want.append(eng.read_loss())
            else:
                eng.loss_begin(step & 1)
                if step > 0:
                    got.append(eng.loss_end((step - 1) & 1))
        if mode == "behind":
            got.append(eng.loss_end(3 & 1))
    assert got == want
    assert cm.read_status() == 0


@pytest.mark.parametrize("V", [1, 100, 4096, 4097, 10001, 16384, 16385])
def test_softmax_columns_match_their_definition(cm, V):
    """Whole columns in registers (4 or 16 values a thread) and, past 16384 rows, the calls one by one: state, its normalised form,
    the error and the document lengths against float64.  Bound: a sum of V positive fp32 terms and a handful of roundings."""
    rng = np.random.default_rng(V)
    B = 7
    pre = (3 * rng.standard_normal((V, B))).astype(np.float32)
    counts = rng.poisson(2.0, (V, B)).astype(np.float32)
    counts[0] += 1
    m = {n: cm.empty((V, B)) for n in ("state", "norm", "v0n")}
    nn, loss = cm.empty((1, B)), cm.empty((1, 1))
    X, data = cm.Immediate(), cm.CUDAMatrix(counts)
    X.document_lengths(data, nn, m["v0n"], 1e-10)
    X.softmax_reconstruction(cm.CUDAMatrix(pre), nn, m["state"], m["norm"], data, loss)
    lengths = counts.astype(np.float64).sum(axis=0)
    np.testing.assert_array_equal(get(nn)[0], lengths.astype(np.float32))        # sums of small integers are exact
    np.testing.assert_allclose(get(m["v0n"]), counts / lengths, rtol=1e-6)
    e = np.exp(pre.astype(np.float64) - pre.max(axis=0))
    p = e / e.sum(axis=0)
    np.testing.assert_allclose(get(m["norm"]), p, rtol=1e-5, atol=1e-12)
    np.testing.assert_allclose(get(m["state"]), p * lengths, rtol=1e-5, atol=1e-12)
    np.testing.assert_allclose(get(loss)[0, 0], ((p - counts) ** 2).sum(), rtol=1e-5)
    X.softmax_reconstruction(cm.CUDAMatrix(pre), nn, m["state"], m["norm"])
    np.testing.assert_allclose(get(m["norm"]), p, rtol=1e-5, atol=1e-12)
    again = get(cm.CUDAMatrix(pre).softmax_scaled(nn, target=cm.empty((V, B))))
    np.testing.assert_array_equal(again, get(m["state"]))


@pytest.mark.parametrize("sizes,B", [((784, 500), 100), ((33, 1, 64), 7), ((5, 31, 32, 129), 1024), ((40, 30), 1025)])
@pytest.mark.parametrize("rows", [64, 37])
def test_updates_in_one_launch_match_the_separate_calls(cm, sizes, B, rows):
    """Biases of two to four layers (whole and ragged blocks of rows, past the cases one launch takes) and a weight matrix of
    whole and odd columns: bit for bit what the separate calls give, whose sums over at most 1024 cases differ only in order:
    1e-5 of the largest sum."""
    rng = np.random.default_rng(B)
    f = lambda *s: rng.standard_normal(s).astype(np.float32)
    host = [(f(n, B), f(n, B), f(n, 1), f(n, 1)) for n in sizes]
    w, d, g = f(rows, 50), f(rows, 50), f(rows, 50)
    X = cm.Immediate()
    results = []
    for fused in (True, False):
        layers = [(cm.CUDAMatrix(p), cm.CUDAMatrix(n), cm.empty((p.shape[0], 1)), cm.CUDAMatrix(b), cm.CUDAMatrix(db))
                  for p, n, b, db in host]
        W, D, S, acc = cm.CUDAMatrix(w), cm.CUDAMatrix(d), cm.CUDAMatrix(g), cm.empty((1, 1))
        aux = W.split_bf16(cm.empty_aux((rows, 50)))
        if fused:
            X.update_all(layers, W, D, S, aux, 1.0 / B, 0.5, 0.1, 0.9, 0.2, l2=1e-3, l1=1e-4, sq_acc=acc)
        else:
            X.sq_diff(layers[0][0], layers[0][1], acc)
            for p, n, s, b, db in layers:
                X.row_sum_diff(p, n, s)
                X.momentum_update(b, db, None, s, 1.0 / B, 0.5, 0.1)
            X.momentum_update(W, D, None, S, 1.0 / B, 0.9, 0.2, l2=1e-3, l1=1e-4, w_aux=aux)
        results.append(([get(m) for m in (W, D, aux)], [get(m) for l in layers for m in l[2:]], float(get(acc)[0, 0])))
    for a, b in zip(results[0][0], results[1][0]):
        np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32))
    for a, b in zip(results[0][1], results[1][1]):
        assert np.abs(a - b).max() <= 1e-5 * max(1.0, np.abs(b).max())
    assert abs(results[0][2] - results[1][2]) <= 1e-6 * results[1][2]


@pytest.mark.parametrize("rows,n", [(64, 45), (37, 45), (1024, 516)])
@pytest.mark.parametrize("growth", [0.0, 1.0, 1000.0, -1.0])
def test_updates_in_one_launch_keep_the_exponent_of_the_planes(cm, rows, n, growth):
    """The scaled half-precision planes written by the launch that updates everything: bit for bit those of momentum_update,
    over two updates, where the exponent stays, where the weights outgrow it (every plane rewritten, by one block and by a launch
    of its own) and where they vanish."""
    rng = np.random.default_rng(rows)
    f = lambda *s: rng.standard_normal(s).astype(np.float32)
    B = 20
    layers_h = [(f(rows, B), f(rows, B), f(rows, 1), f(rows, 1)), (f(n, B), f(n, B), f(n, 1), f(n, 1))]
    w = f(rows, n)
    d = -w if growth < 0 else growth * f(rows, n)          # -1: the update takes the weights away
    g = np.zeros_like(w) if growth < 0 else f(rows, n)
    X, results = cm.Immediate(), []
    for fused in (True, False):
        layers = [(cm.CUDAMatrix(p), cm.CUDAMatrix(q), cm.empty((p.shape[0], 1)), cm.CUDAMatrix(b), cm.CUDAMatrix(db))
                  for p, q, b, db in layers_h]
        W, D, S = cm.CUDAMatrix(w), cm.CUDAMatrix(d), cm.CUDAMatrix(g)
        scale = cm.f16_scale_state(np.abs(w).max())
        aux = W.split_f16(cm.empty_aux((rows, n)), exp_dev=scale.slice(0, 1))
        for _ in range(2):
            if fused:
                X.update_all(layers, W, D, S, aux, 1.0 / B, 0.5, 0.1, 1.0, -1.0 if growth < 0 else 0.2, w_scale=scale)
            else:
                X.momentum_update(W, D, None, S, 1.0 / B, 1.0, -1.0 if growth < 0 else 0.2, w_aux=aux, w_scale=scale)
        results.append([get(W), get(D)] + list(_f16_planes(aux)) + [get(scale)[:, :3]])
    for a, b in zip(*results):
        np.testing.assert_array_equal(a, b)
    if growth > 1:
        assert results[0][4][0, 0] < cm.f16_scale_state(np.abs(w).max()).asarray()[0, 0]
    e = results[0][4][0, 0]
    np.testing.assert_array_equal(results[0][3], (results[0][0] * np.float32(2.0) ** e).astype(np.float16).astype(np.float32))


@pytest.mark.parametrize("V,H,B,gibbs,sample", [(301, 203, 78, 1, False), (130, 67, 1030, 2, False), (97, 515, 33, 3, True),
                                                      (130, 67, 1030, 2, True)])
def test_half_precision_engine_on_odd_models_matches_oracle(cm, oracle, V, H, B, gibbs, sample, monkeypatch):
    """Odd layers and batches on half-precision planes (the update in one launch, and past 1024 cases in its parts): draws bit
    for bit, parameters and states to 1e-5 of the largest."""
    monkeypatch.setenv("B200_RBM_STATE_AUX", "1")
    rng = np.random.default_rng(V)
    hyp = dbm.Hyperparams(base_epsilon=0.05, initial_momentum=0.5, final_momentum=0.9, momentum_change_steps=10, gibbs_steps=gibbs,
                          sample_input=sample)
    w = (0.05 * rng.standard_normal((V, H))).astype(np.float32)
    x = (rng.random((V, 2 * B)) < 0.3).astype(np.float32)
    edge = hyp.copy(apply_l2_decay=True, l2_decay=2e-4)
    layers = [dict(name="v", activation=dbm.LOGISTIC, numdims=V, is_input=True), dict(name="h", activation=dbm.LOGISTIC, numdims=H)]
    ref = dbm.DBM(oracle, layers, [dict(node1="v", node2="h", weight=w, hyperparams=edge)], hyp, B, dbm.CD, seed=9)
    eng = FusedRBM(cm, V, H, B, w, hyp, edge_hyperparams=edge, binary_data=True, seed=9)
    assert eng.f16
    xo, xg = oracle.CUDAMatrix(x), cm.CUDAMatrix(x)
    for step in range(3):
        s = (step % 2) * B
        ref.SetBatch([xo.slice(s, s + B)])
        want = ref.TrainOneBatch(step)[0]
        eng.TrainOneBatch(step, xg.slice(s, s + B))
        np.testing.assert_allclose(eng.read_loss(), want, rtol=1e-5)
    assert relerr(get(eng.W), get(ref.edge[0].params["weight"])) < TOL
    assert relerr(get(eng.dW), get(ref.edge[0].gradient_history)) < 2 * TOL
    assert relerr(get(eng.v_neg), get(ref.GetLayerByName("v").state)) < TOL
    assert relerr(get(eng.h_neg), get(ref.GetLayerByName("h").state)) < TOL
    np.testing.assert_array_equal(get(eng.h_samp), get(ref.GetLayerByName("h").sample))
    if sample:
        np.testing.assert_array_equal(get(eng.v_samp), get(ref.GetLayerByName("v").sample))
    for mine, theirs in ((eng.bv, "v"), (eng.bh, "h")):
        assert relerr(get(mine), get(ref.GetLayerByName(theirs).params["bias"])) < TOL
    assert cm.read_status() == 0


@pytest.mark.parametrize("V,H,B,gibbs,scale", [(64, 128, 40, 1, 1.0), (301, 203, 78, 3, 1.0), (130, 67, 1030, 2, 1e-3), (97, 515, 33, 1, 300.0),
                                               (60, 40, 16, 2, 0.0)])
def test_engine_on_real_data_with_parts_in_memory_matches_oracle(cm, oracle, V, H, B, gibbs, scale, monkeypatch):
    """Linear visible units on bfloat16 parts from memory: data of any magnitude, all zero among them, and one outlier of a thousand
    times the rest; draws bit for bit, parameters and states to 1e-5 of the largest."""
    monkeypatch.setenv("B200_RBM_STATE_AUX", "1")
    rng = np.random.default_rng(V)
    hyp = dbm.Hyperparams(base_epsilon=1e-3 / max(scale, 1.0) ** 2, initial_momentum=0.5, final_momentum=0.9, momentum_change_steps=10,
                          gibbs_steps=gibbs)
    w = (0.05 / max(scale, 1.0) * rng.standard_normal((V, H))).astype(np.float32)
    x = (scale * rng.standard_normal((V, 2 * B))).astype(np.float32)
    if scale == 1e-3:
        x[5, 7] = 1.0
    layers = [dict(name="v", activation=dbm.LINEAR, numdims=V, is_input=True), dict(name="h", activation=dbm.LOGISTIC, numdims=H)]
    ref = dbm.DBM(oracle, layers, [dict(node1="v", node2="h", weight=w, hyperparams=hyp)], hyp, B, dbm.CD, seed=9)
    eng = FusedRBM(cm, V, H, B, w, hyp, visible=dbm.LINEAR, seed=9)
    assert eng.state_aux and not eng.f16
    xo, xg = oracle.CUDAMatrix(x), cm.CUDAMatrix(x)
    for step in range(3):
        s = (step % 2) * B
        ref.SetBatch([xo.slice(s, s + B)])
        want = ref.TrainOneBatch(step)[0]
        eng.TrainOneBatch(step, xg.slice(s, s + B))
        np.testing.assert_allclose(eng.read_loss(), want, rtol=1e-5)
    assert relerr(get(eng.W), get(ref.edge[0].params["weight"])) < TOL
    assert relerr(get(eng.dW), get(ref.edge[0].gradient_history)) < 2 * TOL
    assert relerr(get(eng.v_neg), get(ref.GetLayerByName("v").state)) < TOL
    assert relerr(get(eng.h_neg), get(ref.GetLayerByName("h").state)) < TOL
    np.testing.assert_array_equal(get(eng.h_samp), get(ref.GetLayerByName("h").sample))
    assert cm.read_status() == 0


@pytest.mark.parametrize("V,H,B,n,visible,binary", [(61, 130, 90, 15, "LOGISTIC", True), (61, 130, 90, 12, "LOGISTIC", False),
                                                    (40, 33, 1, 7, "LINEAR", False), (61, 130, 600, 3, "LOGISTIC", True), (60, 44, 250, 5, "LINEAR", False),
                                                    (785, 301, 600, 3, "LOGISTIC", True), (501, 512, 250, 5, "LINEAR", False)])
@pytest.mark.parametrize("planes", ["0", "1"])
def test_representations_of_several_minibatches_a_product(cm, V, H, B, n, visible, binary, planes, monkeypatch):
    """Groups of minibatches, whole and a ragged last one, in every form of the engine: representation and reconstruction error
    against float64 (1e-5 of the largest, 1e-5 of the error), the engine's states those of the last minibatch."""
    monkeypatch.setenv("B200_RBM_STATE_AUX", planes)
    rng = np.random.default_rng(n)
    w, bv, bh = (0.1 * rng.standard_normal(s).astype(np.float32) for s in ((V, H), (V, 1), (H, 1)))
    w /= max(1.0, (V / 100) ** 0.5)
    x = (rng.random((V, n * B)) < 0.3 if binary else rng.standard_normal((V, n * B)) if visible == "LINEAR" else rng.random((V, n * B)))
    x = x.astype(np.float32)
    eng = FusedRBM(cm, V, H, B, w, dbm.Hyperparams(), visible=getattr(dbm, visible), binary_data=binary, bias_v=bv, bias_h=bh, seed=1)
    data = cm.CUDAMatrix(x)
    rep, err = eng.Inference(data, input_recon=True)
    sig = lambda z: 1 / (1 + np.exp(-z))
    h = sig(w.T.astype(np.float64) @ x + bh)
    v = w.astype(np.float64) @ h + bv
    v = v if visible == "LINEAR" else sig(v)
    assert np.abs(rep.T - h).max() < 1e-5
    np.testing.assert_allclose(err, ((v - x) ** 2).sum(), rtol=1e-5)
    np.testing.assert_array_equal(get(eng.h_pos).T, rep[(n - 1) * B:])
    assert np.abs(get(eng.v_neg) - v[:, (n - 1) * B:]).max() < 1e-5 * max(1.0, np.abs(v).max())
    np.testing.assert_array_equal(eng.Inference(data), rep)
    assert cm.read_status() == 0


@pytest.mark.parametrize("scale", [1e8, 1e-3])
def test_results_depend_on_no_data_of_earlier_calls(cm, scale):
    """Real-valued data of another magnitude first: representations, reconstruction error and an update afterwards are a fresh
    engine's, bit for bit."""
    rng = np.random.default_rng(11)
    V, H, B = 256, 512, 512
    w = (0.05 * rng.standard_normal((V, H))).astype(np.float32)
    x, other = (rng.standard_normal((V, 4 * B)).astype(np.float32) for _ in range(2))
    data, first = cm.CUDAMatrix(x), cm.CUDAMatrix(other * np.float32(scale))
    mk = lambda: FusedRBM(cm, V, H, B, w, dbm.Hyperparams(base_epsilon=1e-3), visible=dbm.LINEAR, seed=2)
    used, fresh = mk(), mk()
    used.Inference(first, input_recon=True)
    for a, b in zip(used.Inference(data, input_recon=True), fresh.Inference(data, input_recon=True)):
        np.testing.assert_array_equal(a, b)
    weights = []
    for used in (True, False):
        eng = mk()                       # (the random stream starts over)
        if used:
            eng.Inference(first)
        eng.TrainOneBatch(0, data.slice(0, B))
        weights.append(get(eng.W))
    np.testing.assert_array_equal(*weights)
    assert cm.read_status() == 0


@pytest.mark.parametrize("outlier", [0.0, 1e3, 1e6, 1e8, 1e12])
def test_one_case_of_large_values_leaves_the_others_exact(cm, outlier):
    """One entry of any size in one case of real-valued data: every other case's representation, and the statistics of every other
    visible unit, against float64 (1e-5 of the largest)."""
    rng = np.random.default_rng(12)
    V, H, B = 512, 516, 512
    w = (0.05 * rng.standard_normal((V, H))).astype(np.float32)
    x = rng.standard_normal((V, 2 * B)).astype(np.float32)
    x[3, 7] += np.float32(outlier)
    eng = FusedRBM(cm, V, H, B, w, dbm.Hyperparams(base_epsilon=1e-3), visible=dbm.LINEAR, seed=2)
    data = cm.CUDAMatrix(x)
    sig = lambda z: 1 / (1 + np.exp(-np.clip(z, -700, 700)))
    others, rows = np.arange(2 * B) != 7, np.arange(V) != 3
    assert np.abs(eng.Inference(data).T - sig(w.T.astype(np.float64) @ x))[:, others].max() < 1e-5
    eng.TrainOneBatch(0, data.slice(0, B))
    v = get(eng.v_neg).astype(np.float64)
    want = (x[:, :B] @ sig(w.T.astype(np.float64) @ x[:, :B]).T - v @ sig(w.T.astype(np.float64) @ v).T)[rows]
    assert relerr(get(eng.suff_W)[rows], want) < 1e-5
    assert cm.read_status() == 0


@pytest.mark.parametrize("largest", [0.0, 10.0, 1e4, 1e8])
def test_one_large_weight_leaves_the_other_units_exact(cm, largest):
    """One weight of any size, in a model that would go on half-precision planes: every other unit's representation against float64
    to 3e-7 (1.3e-7 without it), whether the engine was made with it or loads it, and planes again once it is gone."""
    rng = np.random.default_rng(0)
    V, H, B = 784, 512, 256
    w = (0.05 * rng.standard_normal((V, H))).astype(np.float32)
    x = (rng.random((V, 4 * B)) < 0.3).astype(np.float32)
    plain, odd = w.copy(), w.copy()
    odd[3, 7] += np.float32(largest)
    sig = lambda z: 1 / (1 + np.exp(-np.clip(z, -700, 700)))
    others, data = np.arange(H) != 7, cm.CUDAMatrix(x)
    made = FusedRBM(cm, V, H, B, odd, dbm.Hyperparams(), binary_data=True, seed=1)
    loads = FusedRBM(cm, V, H, B, plain, dbm.Hyperparams(), binary_data=True, seed=1)
    assert loads.f16
    loads.W.overwrite(np.asfortranarray(odd))
    loads.refresh_weight_aux()
    for eng in (made, loads):
        assert eng.f16 == (largest < 64)
        assert np.abs(eng.Inference(data).T - sig(odd.T.astype(np.float64) @ x))[others].max() < 3e-7
    results = []
    for eng in (made, loads):
        cm.CUDAMatrix.init_random(1)
        eng.TrainOneBatch(0, data.slice(0, B))
        results.append(get(eng.W))
        eng.W.overwrite(np.asfortranarray(plain))
        eng.refresh_weight_aux()
        assert eng.f16 and bool(eng._programs) == (largest < 64)      # (what is recorded stays while the form does)
        assert np.abs(eng.Inference(data).T - sig(plain.T.astype(np.float64) @ x + get(eng.bh))).max() < 3e-7
        eng.TrainOneBatch(1, data.slice(0, B))
        assert np.isfinite(get(eng.W)).all()
    np.testing.assert_array_equal(*results)
    assert cm.read_status() == 0


def test_representations_on_a_device_that_is_nearly_full(cm, monkeypatch):
    """Without memory for states of several minibatches, or for planes of a fresh exponent, they go one by one, from fp32 operands."""
    rng = np.random.default_rng(1)
    V, H, B = 784, 512, 256
    w = (0.05 * rng.standard_normal((V, H))).astype(np.float32)
    w[0, 0] = 0.9999                       # (grows past 1: another exponent would be fresh)
    x = (rng.random((V, 4 * B)) < 0.3).astype(np.float32)
    x[0] = 1
    eng = FusedRBM(cm, V, H, B, w, dbm.Hyperparams(base_epsilon=0.1), binary_data=True, seed=1)
    data = cm.CUDAMatrix(x)
    eng.TrainOneBatch(0, data.slice(0, B))
    now, fresh = get(eng.W_scale)[0, :2]
    assert eng.f16 and now != fresh

    def full(*_, **__):
        raise cm.CUDAMatException("no memory")
    for name in ("carve", "empty_aux"):
        monkeypatch.setattr(cm, name, full)
    w, b = get(eng.W).astype(np.float64), get(eng.bh)
    assert np.abs(eng.Inference(data).T - 1 / (1 + np.exp(-(w.T @ x + b)))).max() < 1e-5
    monkeypatch.undo()
    assert np.abs(eng.Inference(data).T - 1 / (1 + np.exp(-(w.T @ x + b)))).max() < 1e-5
    assert cm.read_status() == 0


def _launches(cm, step):
    """Kernels of an update, recorded as a graph behind two that were not."""
    import torch
    from cuda.bindings import runtime
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph(keep_graph=True)
    cm.cuda_sync_threads()
    cm._lib.b200_set_stream(stream.cuda_stream)
    try:
        for n in range(2):
            step(n)
        cm.cuda_sync_threads()
        with torch.cuda.graph(graph, stream=stream):
            step(2)
    finally:
        cm._lib.b200_set_stream(None)
    raw = runtime.cudaGraph_t(graph.raw_cuda_graph())
    _, nodes, _ = runtime.cudaGraphGetNodes(raw, runtime.cudaGraphGetNodes(raw, 0)[2])
    assert all(runtime.cudaGraphNodeGetType(x)[1] == runtime.cudaGraphNodeType.cudaGraphNodeTypeKernel for x in nodes)
    return len(nodes)


@pytest.mark.parametrize("config,launches", [(0, 5), (1, 5), (2, 9), (3, 44)])
def test_launches_of_an_update_are_counted(cm, config, launches):
    """The configurations at their full size: what the engine says, what the library issues, what the launch lists hold."""
    from deepnet_b200.fused_dbm import FusedDBM
    cfg = configs.build(config, cases=256)
    B, dims, weights = cfg["batchsize"], [l["numdims"] for l in cfg["layers"]], [e["weight"] for e in cfg["edges"]]
    if config == 3:
        eng = FusedDBM(cm, dims, B, weights, cfg["hyperparams"], seed=1)
    else:
        eng = FusedRBM(cm, dims[0], dims[1], B, weights[0], cfg["hyperparams"], visible=cfg["layers"][0]["activation"],
                       binary_data=config != 1, seed=1)
    data = cm.CUDAMatrix(cfg["data"][:, :B])
    assert _launches(cm, lambda n: eng.TrainOneBatch(n, data)) == eng.kernel_launches == launches


@pytest.mark.parametrize("V,H,B,k,sample", [(1024, 512, 256, 1, False), (1024, 513, 300, 3, True), (1001, 777, 1100, 2, True),
                                            (100, 100, 20, 1, False), (1000, 100, 1100, 1, False)])
def test_launches_on_either_side_of_the_lines_are_counted(cm, V, H, B, k, sample):
    """Weights whose planes one block rewrites and more, up to 1024 cases and more, planes and fp32 operands."""
    rng = np.random.default_rng(0)
    eng = FusedRBM(cm, V, H, B, (0.01 * rng.standard_normal((V, H))).astype(np.float32),
                   dbm.Hyperparams(gibbs_steps=k, sample_input=sample), binary_data=True, seed=1)
    data = cm.CUDAMatrix((rng.random((V, B)) < 0.3).astype(np.float32))
    assert _launches(cm, lambda n: eng.TrainOneBatch(n, data)) == eng.kernel_launches


def test_work_side_by_side(cm):
    """Two chains of products beside each other and what follows the join, recorded and call by call: the bits of one stream.  An
    operation that fails between fork and join leaves the thread on the library stream."""
    rng = np.random.default_rng(3)
    f = lambda *s: rng.random(s).astype(np.float32)
    w, xs, b = cm.CUDAMatrix(0.05 * f(2048, 2048)), [cm.CUDAMatrix(f(2048, 200)) for _ in range(2)], cm.CUDAMatrix(f(2048, 1))
    results = []
    for X, beside in ((cm.Immediate(), False), (cm.Immediate(), True), (cm.Program(), True)):
        out = [[cm.empty((2048, 200)) for _ in range(4)] for _ in range(2)]
        total = cm.empty((2048, 1))
        if beside:
            X.branch(0)
        for k in range(4):
            for side in (0, 1):
                if beside and side:
                    X.branch(1)
                X.fused_gemm(cm.split_passes(w.T, out[side][k - 1] if k else xs[side]), out=out[side][k], bias=b, activation=1)
                if beside and side:
                    X.branch(2)
        if beside:
            X.branch(3)
        X.row_sum_diff(out[0][3], out[1][3], total)
        if isinstance(X, cm.Program):
            X.run()
        results.append([get(m) for o in out for m in o] + [get(total)])
    for other in results[1:]:
        for a, c in zip(results[0], other):
            np.testing.assert_array_equal(a, c)
    stream = cm._lib.b200_get_stream()
    bad = cm.Program()
    bad.branch(0)
    bad.branch(1)
    bad.copy(xs[0], b)
    bad.branch(3)
    with pytest.raises(cm.CUDAMatException):
        bad.run()
    assert cm._lib.b200_get_stream() == stream
    np.testing.assert_array_equal(get(cm.empty((2048, 200)).assign(xs[0])), get(xs[0]))
    assert cm.read_status() == 0


def test_representations_leave_while_the_next_minibatch_is_computed(cm):
    """Several pieces a minibatch and a ragged last one, an even and an odd number of minibatches, and the staging area taken by
    someone else (plain copies): the rows are the products', bit for bit."""
    rng = np.random.default_rng(4)
    V, H, B = 300, 701, 250
    w = (rng.standard_normal((V, H)) * 0.05).astype(np.float32)
    eng = FusedRBM(cm, V, H, B, w, dbm.Hyperparams(), binary_data=True, seed=1)
    for n in (4, 3, 1):
        x = (rng.random((V, n * B)) < 0.3).astype(np.float32)
        data = cm.CUDAMatrix(x)
        with cm.RowsOut() as taken:
            assert taken.held
            want = eng.Inference(data)
        got = eng.Inference(data)
        np.testing.assert_array_equal(got, want)
        np.testing.assert_array_equal(get(eng.h_pos).T, got[(n - 1) * B:])
        assert np.abs(got - 1 / (1 + np.exp(-(x.T.astype(np.float64) @ w)))).max() < 1e-5
    assert cm.read_status() == 0


@pytest.mark.parametrize("once", [False, True])
@pytest.mark.parametrize("sizes,B,mf,gibbs", [((60, 40), 20, 3, 1), ((61, 40, 33), 7, 1, 2), ((60, 44, 32), 20, 2, 1), ((64, 40, 100), 33, 3, 2),
                                              ((50, 41, 33, 20), 12, 3, 1), ((40, 36, 30, 26, 20, 17), 9, 2, 1),
                                              ((48, 20, 24), 1025, 2, 1), ((64, 1040, 20), 1028, 2, 1)])
def test_dbm_of_any_depth_matches_oracle(cm, oracle, sizes, B, mf, gibbs, once, monkeypatch):
    """Two to six layers (biases beyond the fourth in a launch of their own), one to three mean-field sweeps with W1'data in every
    sweep and multiplied once, odd sizes, cases past what the bias launch takes and products that find what is added in their
    output."""
    from deepnet_b200.fused_dbm import FusedDBM
    monkeypatch.setattr(FusedDBM, "_data_once", lambda self: once and self.L > 2 and self.hyp.mf_steps > 1)
    rng = np.random.default_rng(sum(sizes) + B)
    hyp = dbm.Hyperparams(base_epsilon=0.05, initial_momentum=0.5, final_momentum=0.9, momentum_change_steps=10, mf_steps=mf,
                          gibbs_steps=gibbs)
    names = ["l%d" % i for i in range(len(sizes))]
    w = [(rng.standard_normal((sizes[i], sizes[i + 1])) * 0.1).astype(np.float32) for i in range(len(sizes) - 1)]
    layers = [dict(name=n, activation=dbm.LOGISTIC, numdims=d, is_input=i == 0) for i, (n, d) in enumerate(zip(names, sizes))]
    edges = [dict(node1=names[i], node2=names[i + 1], weight=w[i]) for i in range(len(w))]
    data = (rng.random((sizes[0], 2 * B)) < 0.3).astype(np.float32)
    cfg = dict(layers=layers, edges=edges, hyperparams=hyp, batchsize=B, optimizer=dbm.PCD, seed=4, data=data)
    mo, lo = run_driver(oracle, cfg, 2 * B, 2)
    eng = FusedDBM(cm, list(sizes), B, w, hyp, seed=4)
    dev, lg = cm.CUDAMatrix(data), []
    for step in range(2):
        eng.TrainOneBatch(step, dev.slice(step * B, (step + 1) * B))
        lg.append(eng.read_loss())
    np.testing.assert_allclose(lg, lo, rtol=1e-5)
    for i, e in enumerate(mo.edge):
        assert relerr(get(eng.W[i]), get(e.params["weight"])) < TOL
    for j, l in enumerate(mo.layer):
        assert relerr(get(eng.pos[j]), get(l.pos_state)) < TOL, l.name
        if j > 0:
            np.testing.assert_array_equal(get(eng.neg_sample[j]), get(l.neg_sample))
        assert np.abs(get(eng.b[j]) - get(l.params["bias"])).max() < 1e-6
    assert cm.read_status() == 0


def test_dbm_multiplies_the_data_once_only_where_that_pays(cm):
    """us an update, in every sweep / once: 784-500-1000, 100 cases, 10 sweeps 328 / 298; 64-64-64 193 / 211; 256-256-1500, 16 cases
    262 / 292; 500-2048-500, 1030 cases 772 / 896."""
    from deepnet_b200.fused_dbm import FusedDBM

    def once(sizes, B, mf):
        w = [np.zeros((sizes[i], sizes[i + 1]), np.float32) for i in range(len(sizes) - 1)]
        eng = FusedDBM(cm, sizes, B, w, dbm.Hyperparams(mf_steps=mf, gibbs_steps=1))
        return eng._data_once()

    assert once([784, 500, 1000], 100, 10) and once([784, 500, 1000], 100, 3) and once([1500, 256, 256], 16, 3)
    assert not once([784, 500, 1000], 100, 2) and not once([784, 500], 100, 10) and not once([64, 64, 64], 100, 10)
    assert not once([256, 256, 1500], 16, 10) and not once([500, 2048, 500], 1030, 10)


def test_recorded_operations_equal_the_calls(cm):
    """Every operation of the vocabulary that no engine records today, recorded and replayed, against its call: same bits."""
    rng = np.random.default_rng(12)
    f = lambda *shape: rng.random(shape).astype(np.float32) + 0.1
    V, H, B = 33, 20, 9
    host = dict(m=f(V, B), n=f(V, B), h=f(H, B), g=f(H, B), nn=np.floor(9 * f(1, B)), b=f(V + H, 1), db=f(V + H, 1), w=f(V, H), d=f(V, H),
                s=f(V, H))
    results = []
    for recorded in (False, True):
        d = {k: cm.CUDAMatrix(v) for k, v in host.items()}
        t = [cm.empty(shape) for shape in ((V, B), (1, B), (V, B), (V, B), (V + H, 1), (1, 1), (V, B), (V, B))]
        cm.CUDAMatrix.init_random(5)
        X = cm.Program() if recorded else cm.Immediate()
        X.softmax_scaled(d["m"], d["nn"], t[0])
        X.sum(d["m"], 0, t[1])
        X.add_sums(t[1], d["n"], 0, 0.5)
        X.add_scalar(t[1], 1e-3)
        X.div_by_row(d["n"], t[1], t[2])
        X.sigmoid(d["m"], t[3])
        X.rbm_bias_update(d["m"], d["n"], d["h"], d["g"], t[4], d["b"], d["db"], t[5], 1.0 / B, 0.5, 0.1)
        X.momentum_update(d["w"], d["d"], None, d["s"], 1.0 / B, 0.9, 0.2, l2=1e-3, l1=1e-4)
        X.sample_bernoulli(d["m"], t[6])
        X.copy(t[6], t[7])
        X.assign_scalar(t[6], 2.0)
        if recorded:
            assert len(X) == 11
            X.run()
        results.append([get(x) for x in t + [d["b"], d["db"], d["w"], d["d"]]] + [cm.CUDAMatrix.rnd_state.calls])
    for a, b in zip(*results):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_allclose(results[0][0].sum(axis=0), host["nn"][0], rtol=1e-5)
    assert results[0][-1] == 1 and results[0][5][0, 0] > 0
