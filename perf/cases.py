"""The work a user of this framework has it do, as cases that can be timed and compared.

A case is one call (or one training update) through the public entry points, on inputs a user's
program would have in hand.  The kinds:

  rbm        `FusedRBM.TrainOneBatch`: one CD-k update of a binary or Gaussian-binary RBM
  softmax    the same for a replicated-softmax RBM over word counts (multinomial draws fed upward)
  dbm        `FusedDBM.TrainOneBatch`: one PCD update of a deep Boltzmann machine
  feed       `DeviceFeed.Get` (shuffled, bit-packed data set on the device) and the CD update on what it gives
  driver     `dbm.DBM.TrainOneBatch`: the reference's call sequence, one library call per reference call
  represent  `UpwardNet.forward`: a minibatch through the fixed lower layers of a deep belief network
  infer      `FusedRBM.Inference`: hidden representation and reconstruction error, returned to the host
  ais        `ais_binary_rbm`: partition function of a trained RBM by annealed importance sampling

Matrices handed back are the engine's own device buffers, seen as torch tensors.
"""
import ctypes as ct
import math

import numpy as np
import torch

from deepnet_b200 import ais, b200mat as cm, dbm
from deepnet_b200.datahandler import DeviceFeed
from deepnet_b200.dbn import UpwardNet
from deepnet_b200.fused_dbm import FusedDBM
from deepnet_b200.fused_rbm import FusedRBM

MINIBATCHES = 4      # resident minibatches a training case cycles through


def listed():
    return [
        # the first RBM everybody trains: binary 28 x 28 images, CD-1, minibatches of 100
        dict(name="rbm_784x500", kind="rbm", V=784, H=500, B=100, k=1, visible="LOGISTIC"),
        # layer and batch sizes as feature sets have them, not multiples of anything; CD-3, binary draws fed upward
        dict(name="rbm_odd", kind="rbm", V=1357, H=601, B=203, k=3, visible="LOGISTIC", sample_input=True),
        # dense real-valued features with an overcomplete hidden layer
        dict(name="gauss_1024x4096", kind="rbm", V=1024, H=4096, B=256, k=1, visible="LINEAR"),
        # text: word counts over a 10 000 word vocabulary
        dict(name="softmax_10000x512", kind="softmax", V=10000, H=512, B=100),
        # two hidden layers, 10 mean-field sweeps and 5 Gibbs sweeps an update
        dict(name="dbm_784_500_1000", kind="dbm", V=784, H=500, H2=1000, B=100, mf=10, gibbs=5),
        # the large binary model: CD-10, 4096 cases a GPU
        dict(name="rbm_8192", kind="rbm", V=8192, H=8192, B=4096, k=10, visible="LOGISTIC"),
        # an ordinary mid-sized model trained from the device-resident data set
        dict(name="feed_2048", kind="feed", V=2048, H=2048, B=512, k=1),
        # the drop-in backend: the reference's dbm.py driving the matrix library call by call
        dict(name="driver_784x500", kind="driver", V=784, H=500, B=100, k=1, visible="LOGISTIC"),
        # the same on the Gaussian-binary model, where the calls are not tiny
        dict(name="driver_1024x4096", kind="driver", V=1024, H=4096, B=256, k=1, visible="LINEAR"),
        # lower layers of a DBN feeding the RBM above
        dict(name="represent_2048", kind="represent", V=784, H=500, H2=1000, B=2048),
        # representations of a held-out set written out for the next RBM, with the reconstruction error
        dict(name="infer_1000x1000", kind="infer", V=1000, H=1000, B=250, batches=8),
        # log Z of a trained model: 100 chains, 100 inverse temperatures
        dict(name="ais_784x500", kind="ais", V=784, H=500, B=100, steps=100),
    ]


def draw(rng):
    """One more case of the same kinds and ranges."""
    def size(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        # layer sizes people choose: any number, or a round one
        step = rng.choice([1, 1, 4, 10, 50, 64])
        return max(lo, min(hi, n // step * step))

    kind = rng.choice(["rbm", "rbm", "rbm", "softmax", "dbm", "feed", "driver", "represent", "infer", "ais"])
    if kind == "rbm":
        visible = rng.choice(["LOGISTIC", "LOGISTIC", "LINEAR"])
        return dict(kind=kind, V=size(64, 4096), H=size(64, 4096), B=size(16, 1024), k=rng.choice([1, 1, 2, 5, 10]),
                    visible=visible, sample_input=visible == "LOGISTIC" and rng.random() < 0.3)
    if kind == "softmax":
        return dict(kind=kind, V=size(400, 10000), H=size(32, 1024), B=size(16, 200))
    if kind == "dbm":
        return dict(kind=kind, V=size(64, 1500), H=size(64, 1000), H2=size(64, 1500), B=size(16, 256),
                    mf=rng.choice([3, 5, 10]), gibbs=rng.choice([1, 3, 5]))
    if kind == "feed":
        return dict(kind=kind, V=size(64, 4096), H=size(64, 4096), B=size(32, 1024), k=1)
    if kind == "driver":
        return dict(kind=kind, V=size(64, 2048), H=size(64, 4096), B=size(16, 512), k=1,
                    visible=rng.choice(["LOGISTIC", "LINEAR"]))
    if kind == "represent":
        return dict(kind=kind, V=size(64, 4096), H=size(64, 4096), H2=size(64, 4096), B=size(64, 4096))
    if kind == "infer":
        return dict(kind=kind, V=size(64, 2048), H=size(64, 2048), B=size(50, 500), batches=rng.randint(2, 8))
    return dict(kind=kind, V=size(64, 1024), H=size(64, 1024), B=size(20, 500), steps=rng.randint(20, 100))


# -- inputs ---------------------------------------------------------------------------------
class _Memory(object):
    def __init__(self, mat):
        self.mat = mat                       # a tensor over the memory keeps its matrix (and so the memory) alive
        ptr = ct.cast(mat.mat.data_device, ct.c_void_p).value
        self.__cuda_array_interface__ = dict(shape=(mat.mat.size[1], mat.mat.size[0]), typestr="<f4", data=(ptr, False),
                                             strides=None, version=3)


def tensor(mat):
    """The device memory of a matrix as a torch tensor (cols x rows: the matrix is column-major)."""
    return torch.as_tensor(_Memory(mat), device="cuda")


class _Inputs(object):
    """Everything a case is made of, from its seed."""

    def __init__(self, seed):
        self.host = np.random.default_rng(seed)
        self.dev = torch.Generator(device="cuda")
        self.dev.manual_seed(seed)

    def weights(self, rows, cols, sigma):
        return (torch.randn(cols, rows, generator=self.dev, device="cuda") * sigma).cpu().numpy().T

    def biases(self, n, sigma):
        return (self.host.standard_normal((n, 1)) * sigma).astype(np.float32)

    def binary(self, dims, cases):
        """x_ij ~ Bernoulli(p_i), p_i ~ Beta(0.3, 2): cases x dims."""
        p = torch.from_numpy(self.host.beta(0.3, 2.0, size=dims).astype(np.float32)).cuda()
        return (torch.rand(cases, dims, generator=self.dev, device="cuda") < p).float()

    def gaussian(self, dims, cases, latent=64):
        """x = A z + noise, every dimension with zero mean and unit variance: cases x dims."""
        a = torch.randn(latent, dims, generator=self.dev, device="cuda") / math.sqrt(latent)
        z = torch.randn(cases, latent, generator=self.dev, device="cuda")
        x = z @ a + 0.1 * torch.randn(cases, dims, generator=self.dev, device="cuda")
        return (x - x.mean(0)) / x.std(0)

    def counts(self, vocab, cases):
        """Documents of Poisson(100) + 1 words, words by Zipf(1.07) over a shuffled vocabulary: cases x vocab."""
        p = torch.arange(1, vocab + 1, dtype=torch.float64, device="cuda") ** -1.07
        p = (p / p.sum()).float()[torch.from_numpy(self.host.permutation(vocab)).cuda()]
        lengths = torch.from_numpy(self.host.poisson(100, size=cases) + 1).cuda()
        longest = int(lengths.max())
        words = torch.multinomial(p, cases * longest, replacement=True, generator=self.dev).view(cases, longest)
        used = (torch.arange(longest, device="cuda") < lengths[:, None]).float()
        return torch.zeros(cases, vocab, device="cuda").scatter_add_(1, words, used)


def matrix(x):
    """A device matrix holding the (cases x dims) tensor x, one case a column."""
    m = cm.empty((x.shape[1], x.shape[0]))
    cm.cuda_sync_threads()
    tensor(m).copy_(x)
    torch.cuda.synchronize()
    return m


def prepare(case, seed):
    kind, V, H, B = case["kind"], case["V"], case["H"], case["B"]
    r = _Inputs(seed)
    s = dict(kind=kind, step=0)
    if kind in ("rbm", "softmax", "feed"):
        visible = {"softmax": dbm.REPLICATED_SOFTMAX, "feed": dbm.LOGISTIC}.get(kind) or case["visible"]
        hyp = dbm.Hyperparams(base_epsilon={dbm.LOGISTIC: 0.05, dbm.LINEAR: 0.0005}.get(visible, 0.001),
                              initial_momentum=0.5, final_momentum=0.9, momentum_change_steps=3000,
                              gibbs_steps=case.get("k", 1),
                              sample_input=visible == dbm.REPLICATED_SOFTMAX or bool(case.get("sample_input")))
        edge = hyp.copy(apply_l2_decay=True, l2_decay=2e-4)
        w = r.weights(V, H, 0.001 if visible == dbm.LINEAR else 0.01)
        eng = FusedRBM(cm, V, H, B, w, hyp, edge_hyperparams=edge, visible=visible, binary_data=visible != dbm.LINEAR,
                       seed=seed)
        s["engine"] = eng
        n = MINIBATCHES * B
        if kind == "feed":
            s["feed"] = DeviceFeed(cm, [r.binary(V, n).cpu().numpy()], randomize=True, binary=[True], seed=seed,
                                   aux_mode=(2 if eng.f16 else 1) if eng.state_aux else 0)
        else:
            x = {dbm.LOGISTIC: r.binary, dbm.LINEAR: r.gaussian, dbm.REPLICATED_SOFTMAX: r.counts}[visible](V, n)
            s["data"] = matrix(x)
            s["batches"] = [s["data"].slice(i * B, (i + 1) * B) for i in range(MINIBATCHES)]
        s["out"] = [tensor(m) for m in (eng.W, eng.dW, eng.b, eng.db, eng.loss_acc)]
    elif kind == "dbm":
        sizes = [V, H, case["H2"]]
        hyp = dbm.Hyperparams(base_epsilon=0.005, initial_momentum=0.5, final_momentum=0.9, momentum_change_steps=3000,
                              mf_steps=case["mf"], gibbs_steps=case["gibbs"])
        eng = FusedDBM(cm, sizes, B, [r.weights(sizes[i], sizes[i + 1], 0.01) for i in range(2)], hyp, seed=seed)
        s["engine"] = eng
        s["data"] = matrix(r.binary(V, MINIBATCHES * B))
        s["batches"] = [s["data"].slice(i * B, (i + 1) * B) for i in range(MINIBATCHES)]
        s["out"] = [tensor(m) for m in eng.W + eng.dW + eng.b + eng.db + [eng.loss_acc]]
    elif kind == "driver":
        linear = case["visible"] == dbm.LINEAR
        hyp = dbm.Hyperparams(base_epsilon=0.0005 if linear else 0.05, initial_momentum=0.5, final_momentum=0.9,
                              momentum_change_steps=3000, gibbs_steps=case["k"])
        edge = hyp.copy(apply_l2_decay=True, l2_decay=2e-4)
        layers = [dict(name="v", activation=case["visible"], numdims=V, is_input=True),
                  dict(name="h", activation=dbm.LOGISTIC, numdims=H)]
        edges = [dict(node1="v", node2="h", weight=r.weights(V, H, 0.001 if linear else 0.01), hyperparams=edge)]
        net = dbm.DBM(cm, layers, edges, hyp, B, dbm.CD, seed=seed)
        s["net"] = net
        s["data"] = matrix((r.gaussian if linear else r.binary)(V, MINIBATCHES * B))
        s["batches"] = [s["data"].slice(i * B, (i + 1) * B) for i in range(MINIBATCHES)]
        s["out"] = [tensor(p.params[n]) for p, n in ((net.edge[0], "weight"), (net.layer[0], "bias"), (net.layer[1], "bias"))]
        s["out"] += [tensor(p.gradient_history) for p in (net.edge[0], net.layer[0], net.layer[1])]
    elif kind == "represent":
        sizes = [V, H, case["H2"]]
        specs = [(r.weights(sizes[i], sizes[i + 1], 0.05), r.biases(sizes[i + 1], 0.5), dbm.LOGISTIC) for i in range(2)]
        s["net"] = UpwardNet(cm, specs, B)
        s["data"] = matrix(r.binary(V, B))
        s["out"] = [tensor(l["state"]) for l in s["net"].layers]
    elif kind == "infer":
        hyp = dbm.Hyperparams()
        s["engine"] = FusedRBM(cm, V, H, B, r.weights(V, H, 0.05), hyp, binary_data=True, bias_v=r.biases(V, 0.5),
                               bias_h=r.biases(H, 0.5), seed=seed)
        s["data"] = matrix(r.binary(V, case["batches"] * B))
    else:
        s["weight"], s["hidden"], s["visible"] = r.weights(V, H, 0.05), r.biases(H, 0.5), r.biases(V, 0.5)
        s["chains"], s["schedule"], s["seed"] = B, np.linspace(0.0, 1.0, case["steps"] + 1), seed
    cm.cuda_sync_threads()
    return s


def run(s):
    kind = s["kind"]
    if kind == "represent":
        s["net"].forward(s["data"], exact_input=True)
        return s["out"]
    if kind == "infer":
        return s["engine"].Inference(s["data"], input_recon=True)
    if kind == "ais":
        return ais.ais_binary_rbm(cm, s["weight"], s["hidden"], s["visible"], s["chains"], s["schedule"], seed=s["seed"])
    step = s["step"]
    s["step"] = step + 1
    if kind == "feed":
        batch = s["feed"].Get(s["engine"].B)[0]
        s["engine"].TrainOneBatch(step, batch, s["feed"].last_aux)
        return s["out"]
    batch = s["batches"][step % MINIBATCHES]
    if kind == "driver":
        s["net"].SetBatch([batch])
        return [s["out"], s["net"].TrainOneBatch(step)]
    s["engine"].TrainOneBatch(step, batch)
    return s["out"]


# -- what a pass cannot do without, and how far two correct implementations lie apart -------------
def work(case):
    kind, V, H, B = case["kind"], case["V"], case["H"], case["B"]
    if kind in ("rbm", "softmax", "driver", "feed"):
        data = V * B / 8.0 if kind == "feed" else 4.0 * V * B
        # W, its history and the biases read and written; the minibatch read
        return dict(bytes=16.0 * (V * H + V + H) + data, flops=(3 + 2 * case.get("k", 1)) * 2.0 * V * H * B)
    if kind == "dbm":
        H2, n = case["H2"], V * H + H * case["H2"]
        per_case = case["mf"] * (V * H + 2 * H * H2) + V * H + case["gibbs"] * (2 * V * H + 2 * H * H2) + 2 * n
        # parameters as above; the persistent particles of every layer read and written
        return dict(bytes=16.0 * (n + V + H + H2) + 4.0 * V * B + 8.0 * (V + H + H2) * B, flops=2.0 * per_case * B)
    if kind == "represent":
        H2 = case["H2"]
        return dict(bytes=4.0 * (V * H + H * H2 + H + H2 + B * (V + H + H2)), flops=2.0 * B * (V * H + H * H2))
    if kind == "infer":
        n = case["batches"] * B
        return dict(bytes=4.0 * (V * H + V + H + n * (V + H)), flops=4.0 * n * V * H)
    return dict(bytes=4.0 * (V * H + V + H + B), flops=4.0 * case["steps"] * B * V * H)


def tolerance(case):
    # Measured between the library's own forms of a product (tensor cores in three operand forms, split or
    # not along the inner dimension, and fp32 on CUDA cores), one and three passes; about four times that.
    kind = case["kind"]
    if kind in ("represent", "infer"):
        return {"rel": 1e-5, "max": 5e-5}                  # fp32-grade products: 2.6e-6, 1.3e-5 seen
    # A draw u < p falls on the other side where two correct probabilities straddle u: about one draw in 10^7.
    # From there one case's chain goes its own way, which shows in the gradient history.
    if kind == "ais":
        return {"rel": 2e-3, "max": 2e-2}                  # one chain of a hundred, its log weight off by about 1 %
    if kind == "dbm":
        return {"rel": 1.5e-2, "max": 5e-2}                # 3.7e-3, 1.2e-2 seen (bias history of the top layer)
    return {"rel": 1e-3, "max": 0.15}                      # 2e-4, 3.5e-2 seen (CD-10 at 8192 x 8192)


def exact(case, seed):
    """What `run` returns, in 64 bits, for the kinds that draw nothing."""
    kind, V, H, B = case["kind"], case["V"], case["H"], case["B"]
    r = _Inputs(seed)

    def layer(x, w, b):
        w, b = (torch.from_numpy(np.ascontiguousarray(a)).cuda().double() for a in (w, b))
        return torch.sigmoid(x @ w + b.view(1, -1))

    if kind == "represent":
        sizes = [V, H, case["H2"]]
        params = [(r.weights(sizes[i], sizes[i + 1], 0.05), r.biases(sizes[i + 1], 0.5)) for i in range(2)]
        low = layer(r.binary(V, B).double(), *params[0])
        return [low, layer(low, *params[1])]
    if kind == "infer":
        w, bv, bh = r.weights(V, H, 0.05), r.biases(V, 0.5), r.biases(H, 0.5)
        x = r.binary(V, case["batches"] * B).double()
        h = layer(x, w, bh)
        return h, float(((layer(h, w.T, bv) - x) ** 2).sum())
    return None                                            # the others end in random draws
