"""DBN stacking (deepnet/dbn.py:202-209) and the representation writer (deepnet/dbm.py:365-398,
extract_rbm_representation.py, DataWriter of deepnet/datahandler.py:636-746): host logic on the CPU
restatement here, the fused forms on the device against it."""
import glob
import os

import numpy as np
import pytest

from deepnet_b200 import configs, dbm, dbn


def get(m):
    return np.array(m.asarray(), copy=True)


def test_get_bytes():
    assert dbn.get_bytes("2K") == 2048 and dbn.get_bytes("1.5M") == int(1.5 * 1024 ** 2) and dbn.get_bytes("123") == 123


def test_shard_writer_names_sizes_and_order(tmp_path):
    rng = np.random.default_rng(0)
    a, b = rng.standard_normal((250, 6)).astype(np.float32), rng.standard_normal((250, 2)).astype(np.float32)
    # 8 floats per case, 4 bytes each: 3200 bytes hold 100 cases -> three shards of 100, 100, 50
    w = dbn.ShardWriter(["h", "y"], str(tmp_path), "3200", [6, 2], 250)
    for s in range(0, 250, 30):                      # minibatches that straddle shard boundaries
        w.submit([a[s:s + 30], b[s:s + 30]])
    assert w.commit() == [250, 250]
    files = sorted(os.path.basename(f) for f in glob.glob(str(tmp_path / "h-*")))
    assert files == ["h-00001-of-00003.npy", "h-00002-of-00003.npy", "h-00003-of-00003.npy"]
    got = np.concatenate([np.load(str(tmp_path / f)) for f in files])
    np.testing.assert_array_equal(got, a)
    np.testing.assert_array_equal(np.concatenate([np.load(f) for f in sorted(glob.glob(str(tmp_path / "y-*")))]), b)
    assert [len(np.load(str(tmp_path / f))) for f in files] == [100, 100, 50]


def _stack(backend, fused_top, steps=3):
    """A 2-layer stack: a fixed lower RBM layer below a top RBM trained with CD-1 on its output."""
    cfg = configs.build(0, cases=300, dims_scale=0.25)
    B = cfg["batchsize"]
    V, H1 = cfg["layers"][0]["numdims"], cfg["layers"][1]["numdims"]
    H2 = 64
    rng = np.random.default_rng(12)
    w1 = cfg["edges"][0]["weight"]
    b1 = (rng.standard_normal(H1) * 0.1).astype(np.float32)
    w2 = (rng.standard_normal((H1, H2)) * 0.01).astype(np.float32)
    hyp = cfg["hyperparams"]
    data = backend.CUDAMatrix(cfg["data"])
    if fused_top:
        from deepnet_b200.fused_rbm import FusedRBM
        top = FusedRBM(backend, H1, H2, B, w2, hyp, seed=cfg["seed"])        # real-valued inputs: not binary
        net = dbn.DBN(backend, [(w1, b1, dbm.LOGISTIC)], top, B, binary_data=True)
        for step in range(steps):
            net.TrainOneBatch(step, data.slice(step * B, (step + 1) * B))
        rep = net.Represent(data)
        return get(top.W), top.read_loss(), rep
    # the reference's form: upward net call by call, the top RBM through the call-by-call driver
    layers = [dict(name="v", activation=dbm.LOGISTIC, numdims=H1, is_input=True),
              dict(name="h", activation=dbm.LOGISTIC, numdims=H2)]
    m = dbm.DBM(backend, layers, [dict(node1="v", node2="h", weight=w2)], hyp, B, dbm.CD, seed=cfg["seed"])
    up = dbn.UpwardNet(backend, [(w1, b1, dbm.LOGISTIC)], B, fused=False)
    loss = 0.0
    for step in range(steps):
        m.SetBatch([up.forward(data.slice(step * B, (step + 1) * B))])
        loss += m.TrainOneBatch(step)[0]
    reps = []
    for i in range(300 // B):
        m.SetBatch([up.forward(data.slice(i * B, (i + 1) * B))])
        m.PositivePhase(train=False)
        reps.append(get(m.GetLayerByName("h").state).T)
    return get(m.edge[0].params["weight"]), loss, np.concatenate(reps, axis=0)


def test_stacked_training_and_extraction_on_the_cpu_restatement(oracle, tmp_path):
    W, loss, rep = _stack(oracle, fused_top=False)
    assert np.isfinite(loss) and rep.shape == (300, 64) and 0 < rep.min() and rep.max() < 1
    # the representation of the whole set, sharded and described for the next stage
    B = 100
    batches = [rep[i:i + B] for i in range(0, 300, B)]
    entries = dbn.extract_representations(lambda b: [b], {"train": (batches, 300)}, ["hidden2"], [64], str(tmp_path),
                                          "rbm2", memory="1G")
    assert entries == [("hidden2_train", os.path.join("train", "hidden2-*-of-*.npy"), 300, 64)]
    got = np.load(str(tmp_path / "train" / "hidden2-00001-of-00001.npy"))
    np.testing.assert_array_equal(got, rep)
    text = open(str(tmp_path / "data.pbtxt")).read()
    assert 'name: "hidden2_train"' in text and "size: 300" in text and "dimensions: 64" in text


@pytest.mark.gpu
def test_stacked_training_on_the_device_matches_the_cpu_restatement(cm, oracle):
    Wg, lg, rg = _stack(cm, fused_top=True)
    Wo, lo, ro = _stack(oracle, fused_top=False)
    assert abs(lg - lo) < 1e-5 * lo
    assert np.abs(Wg - Wo).max() / np.abs(Wo).max() < 1e-5
    assert np.abs(rg - ro).max() < 1e-5
    # the call-by-call upward net on the device equals the fused one
    Wc, lc, rc = _stack(cm, fused_top=False)
    assert np.abs(rc - ro).max() < 1e-5 and abs(lc - lo) < 1e-5 * lo
    assert cm.read_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,acts,B,exact", [((784, 500, 1000), "LL", 2048, True), ((784, 500, 1000), "LL", 2048, False),
                                                ((61, 33, 70), "LL", 20, True), ((301, 203, 77, 45), "LNL", 333, False),
                                                ((1001, 515, 130, 33), "LLN", 517, True)])
def test_upward_net_on_half_precision_planes(cm, sizes, acts, B, exact):
    """0/1 and real data, odd layers, a linear layer between logistic ones (its states have no planes): every layer's states
    against float64, 1e-5 of the largest."""
    rng = np.random.default_rng(B)
    specs = [((0.1 * rng.standard_normal((sizes[i], sizes[i + 1]))).astype(np.float32), rng.standard_normal(sizes[i + 1]).astype(np.float32),
              dbm.LOGISTIC if a == "L" else dbm.LINEAR) for i, a in enumerate(acts)]
    net = dbn.UpwardNet(cm, specs, B)
    x = (rng.random((sizes[0], B)) < 0.3 if exact else rng.standard_normal((sizes[0], B))).astype(np.float32)
    for _ in range(2):
        top = net.forward(cm.CUDAMatrix(x), exact_input=exact)
    assert top is net.layers[-1]["state"]
    want = x.astype(np.float64)
    for (w, b, act), l in zip(specs, net.layers):
        want = w.T.astype(np.float64) @ want + b[:, None]
        want = 1 / (1 + np.exp(-want)) if act == dbm.LOGISTIC else want
        assert np.abs(np.array(l["state"].asarray()) - want).max() < 1e-5 * max(1.0, np.abs(want).max())
    assert cm.read_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("largest", [1, 3, 4, 255, 2047])
def test_upward_net_takes_counts_for_exact_input(cm, largest):
    """A net that splits its data into planes, on 0/1 data and on counts, which the weights bring back to ordinary size: the
    logistic against float64."""
    rng = np.random.default_rng(largest)
    V, H, B = 1024, 2048, 512
    w = (0.05 / largest * rng.standard_normal((V, H))).astype(np.float32)
    net = dbn.UpwardNet(cm, [(w, np.zeros(H, np.float32), dbm.LOGISTIC)], B)
    assert net._data_aux is not None
    x = (rng.integers(1, largest + 1, (V, B)) * (rng.random((V, B)) < 0.1)).astype(np.float32)
    got = np.array(net.forward(cm.CUDAMatrix(x), exact_input=True).asarray())
    assert np.abs(got - 1 / (1 + np.exp(-(w.T.astype(np.float64) @ x)))).max() < 1e-5
    assert cm.read_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("V,H,B", [(1024, 2048, 512), (70, 40, 20)])
def test_upward_net_takes_a_transposed_minibatch(cm, V, H, B):
    """Whether or not the net splits its data into planes."""
    rng = np.random.default_rng(V)
    w = (0.05 * rng.standard_normal((V, H))).astype(np.float32)
    net = dbn.UpwardNet(cm, [(w, np.zeros(H, np.float32), dbm.LOGISTIC)], B)
    assert (net._data_aux is not None) == (V == 1024)
    x = (rng.random((V, B)) < 0.3).astype(np.float32)
    want = 1 / (1 + np.exp(-(w.T.astype(np.float64) @ x)))
    for exact in (True, False):
        for m in (cm.CUDAMatrix(np.ascontiguousarray(x.T)).T, cm.CUDAMatrix(x)):
            assert np.abs(np.array(net.forward(m, exact_input=exact).asarray()) - want).max() < 1e-5
    assert cm.read_status() == 0


@pytest.mark.gpu
def test_upward_net_without_layers_hands_the_data_on(cm):
    """A deep belief network whose top model sees the data itself."""
    data = cm.CUDAMatrix(np.ones((6, 4), np.float32))
    for exact in (False, True):
        assert dbn.UpwardNet(cm, [], 4).forward(data, exact_input=exact) is data


@pytest.mark.gpu
@pytest.mark.parametrize("act,largest", [(dbm.LINEAR, 0.0), (dbm.LOGISTIC, 0.0), (dbm.LOGISTIC, 1e4), (dbm.LOGISTIC, 1e8)])
def test_units_of_an_upward_net_do_not_share_their_precision(cm, act, largest):
    """Weights of a linear layer's units ten orders apart: every unit against float64, 1e-5 of its own largest state.  One
    weight of any size in a logistic layer: every other unit's logistic to 1e-6."""
    rng = np.random.default_rng(6)
    V, H, H2, B = 300, 200, 100, 64
    w = (0.1 * rng.standard_normal((V, H))).astype(np.float32)
    w2 = (0.1 * rng.standard_normal((H, H2))).astype(np.float32)
    if act == dbm.LINEAR:
        w2 *= (10.0 ** -np.linspace(0, 10, H2)).astype(np.float32)
    w2[5, 9] += np.float32(largest)
    net = dbn.UpwardNet(cm, [(w, np.zeros(H, np.float32), dbm.LOGISTIC), (w2, np.zeros(H2, np.float32), act)], B)
    x = rng.standard_normal((V, B)).astype(np.float32)
    got = np.array(net.forward(cm.CUDAMatrix(x)).asarray())
    want = w2.T.astype(np.float64) @ (1 / (1 + np.exp(-(w.T.astype(np.float64) @ x))))
    if act == dbm.LINEAR:
        assert (np.abs(got - want).max(axis=1) < 1e-5 * np.abs(want).max(axis=1)).all()
    else:
        others = np.arange(H2) != 9
        assert np.abs(got - 1 / (1 + np.exp(-np.clip(want, -700, 700))))[others].max() < 1e-6
    assert cm.read_status() == 0
