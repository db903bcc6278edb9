"""PCD training of a deep Boltzmann machine (a chain of logistic layers) on fused kernels.

Same arithmetic and random stream as `dbm.DBM.TrainOneBatch` with the PCD optimizer
(deepnet/dbm.py:118-181 mean-field positive phase and particle initialisation, :183-238
Gibbs sweeps on persistent particles, :240-261 updates), but a layer update - the products
with BOTH neighbouring layers, bias, logistic, Bernoulli draw - is one `fused_gemm` call whose
pass list mixes the two inner dimensions, and positive-minus-negative edge statistics are one
call per edge.  Split-TF32 as in fused_rbm: a real-valued matrix x is multiplied as
x.y plus correction terms over its low part x - tf32(x), which the kernel derives from x itself;
a binary one (data, samples) has no low part.
"""
import ctypes as ct
import os

import numpy as np

from .dbm import Parameter
from .fused_rbm import LossReadback


class FusedDBM(LossReadback):
    def __init__(self, cm, sizes, batchsize, weights, hyperparams, seed=0):
        """sizes = [visible, hidden1, ...]; weights[i] is sizes[i] x sizes[i+1]."""
        self.cm, self.sizes, self.B, self.hyp = cm, list(sizes), batchsize, hyperparams
        self.L = len(sizes)
        cm.CUDAMatrix.init_random(seed)
        z = lambda r, c: cm.empty((r, c))
        B = batchsize
        self.W, self.W_aux, self.dW, self.suff_W = [], [], [], []
        for i, w in enumerate(weights):
            w = np.asarray(w, np.float32)
            assert w.shape == (sizes[i], sizes[i + 1])
            self.W.append(cm.CUDAMatrix(w))
            self.W_aux.append(self.W[-1].split_bf16(cm.empty_aux(w.shape)))   # bfloat16 parts, rewritten by the update
            self.dW.append(z(*w.shape))
            self.suff_W.append(z(*w.shape))
        self.b = [z(n, 1) for n in sizes]
        self.db = [z(n, 1) for n in sizes]
        self.suff_b = [z(n, 1) for n in sizes]
        self.pos = [z(n, B) for n in sizes]
        self.neg = [z(n, B) for n in sizes]
        self.neg_sample = [z(n, B) for n in sizes]
        self.from_data = z(sizes[1], B)           # W[0]' data and bias of the positive phase
        self.loss_acc = z(1, 1)
        self._sched = Parameter(cm, hyperparams)
        self.kernel_launches = 0
        # the step is recorded once per (Gibbs sweeps, first step) and replayed with one library call;
        # B200_RBM_PROGRAM=0 issues every operation through its own call instead
        self.use_program = os.environ.get("B200_RBM_PROGRAM", "1") != "0"
        self._programs = {}
        self._batch = cm.CUDAMatrix._from_mat(cm.cudamat())

    def _data_once(self):
        """Whether W[0]' data is multiplied once a positive phase, not in every sweep together with W[1]'s product.  It costs a launch
        (3 us) and, each sweep, the reading of the result; a sweep saves about a microsecond for every slab of K its product is
        shallower.  Measured, us an update with one Gibbs sweep, in every sweep / once: 784-500-1000, 100 cases, 10 mean-field
        sweeps 328 / 298, 3 sweeps 152 / 151; 64-64-64 193 / 211; 256-256-1500, 16 cases 262 / 292; 500-2048-500, 1030 cases 772 /
        896 (wide layers: tcgen05 products, the result is copied to the output first)."""
        if self.L < 3 or self.hyp.mf_steps < 2:
            return False
        V, H, above = self.sizes[:3]
        slabs = lambda k: (k + 31) // 32
        depth = lambda s: self.cm.product_depth(H, self.B, s)
        saved = depth(slabs(V) + slabs(above)) - depth(slabs(above))
        return (saved >= 2 and (self.hyp.mf_steps - 1) * saved >= 6
                and (H * self.B <= 1 << 20 or (V >= 1024 and V >= 2 * above)))

    def _update_layer(self, X, j, below, above, out, sample, add=None):
        """state_j = sigmoid(W[j-1]' below + W[j] above + b_j) (deepnet/dbm.py:82-105), optional draw; `add` stands for what the
        layer gets from below and its bias.  below / above = (state, exact): exact states (0/1) have no low part."""
        P = self.cm.split_passes
        passes = []
        if below is not None:
            passes += P(self.W[j - 1].T, below[0], exact_b=below[1], a_aux=self.W_aux[j - 1])
        if above is not None:
            passes += P(self.W[j], above[0], exact_b=above[1], a_aux=self.W_aux[j])
        X.fused_gemm(passes, out=out, sample=sample, bias=self.b[j] if add is None else None, activation=1, add=add)
        self.kernel_launches += 1

    def TrainOneBatch(self, step, data):
        cm, hyp = self.cm, self.hyp
        gibbs = hyp.gibbs_steps
        if hyp.start_step_up_cd_after > 0 and hyp.start_step_up_cd_after < step:
            gibbs = hyp.gibbs_steps + 1 + (step - hyp.start_step_up_cd_after) // hyp.step_up_cd_after
        mom, eps = self._sched.GetMomentumAndEpsilon(step)
        l2 = hyp.l2_decay if hyp.apply_l2_decay else 0.0
        l1 = hyp.l1_decay if (hyp.apply_l1_decay and step > hyp.apply_l1decay_after) else 0.0
        if not self.use_program:
            self.kernel_launches = 0
            self._issue(cm.Immediate(), data, gibbs, step == 0, mom, eps, l2, l1)
            return
        key = (gibbs, step == 0)
        rec = self._programs.get(key)
        if rec is None:
            prog = cm.Program()
            self.kernel_launches = 0
            handles = self._issue(prog, self._batch, gibbs, step == 0, mom, eps, l2, l1)
            rec = self._programs[key] = (prog, handles, self.kernel_launches)
        prog, (bias_ops, weight_ops, first), self.kernel_launches = rec
        ct.memmove(ct.byref(self._batch.mat), ct.byref(data.mat), ct.sizeof(data.mat))
        self._batch.mat.owns_data = 0
        self._batch_owner = data
        prog.set_floats(first, f1=mom, f2=eps, f3=mom, f4=eps, f5=l2, f6=l1)
        for i in bias_ops:
            prog.set_floats(i, f1=mom, f2=eps)
        for i in weight_ops:
            prog.set_floats(i, f1=mom, f2=eps, f3=l2, f4=l1)
        prog.run()

    def _issue(self, X, data, gibbs, first_step, mom, eps, l2, l1):
        cm, L = self.cm, self.L
        pos, neg, ns = self.pos, self.neg, self.neg_sample
        once = self._data_once()

        def positive():
            """Data clamped, hidden layers start at zero, mean-field sweeps; one operation at a time."""
            for j in range(1, L):
                X.assign_scalar(pos[j], 0)
            # W[0]' data (and the bias) is the same in every sweep
            if once:
                X.fused_gemm(cm.split_passes(self.W[0].T, data, exact_b=True, a_aux=self.W_aux[0]), out=self.from_data, bias=self.b[1])
                self.kernel_launches += 1
                yield
            for sweep in range(self.hyp.mf_steps):
                for j in range(1, L):
                    below = (data, True) if j == 1 else (pos[j - 1], False)
                    above = (pos[j + 1], False) if j < L - 1 else None
                    if sweep == 0 and j == 1:      # (the layer above is zero)
                        above = None
                    if j > 1 or not once:
                        self._update_layer(X, j, below, above, pos[j], None)
                    elif sweep == 0:
                        X.sigmoid(self.from_data, pos[1])
                        self.kernel_launches += 1
                    else:
                        self._update_layer(X, j, None, above, pos[j], None, add=self.from_data)
                    yield
            # PCD reports the reconstruction of the input from the first hidden layer (deepnet/dbm.py:163-166)
            self._update_layer(X, 0, None, (pos[1], False), pos[0], None)
            X.sq_diff(pos[0], data, self.loss_acc)
            yield

        def negative():
            """Gibbs sweeps on the particles, neighbours' samples as input; one layer at a time."""
            for _ in range(gibbs):
                for j in range(L):
                    # the visible "sample" is its mean (sample_input off), so it carries a low part
                    below = None if j == 0 else ((neg[0], False) if j == 1 else (ns[j - 1], True))
                    above = (ns[j + 1], True) if j < L - 1 else None
                    self._update_layer(X, j, below, above, neg[j], ns[j] if j > 0 else None)
                    yield

        if first_step:       # particles start from the positive states (deepnet/dbm.py:169-181, 270-271)
            for _ in positive():
                pass
            for j in range(L):
                X.copy(pos[j], neg[j])
                X.sample_bernoulli(neg[j], ns[j])
            for _ in negative():
                pass
        else:
            # The phases share nothing but W and the biases, and a layer's product leaves most of the device idle: they run side
            # by side (784-500-1000, 100 cases, 10 sweeps and 5: 426 -> 321 us; 2048-2048-2048, 256 cases, 10 and 1: 673 -> 582).
            # The draws keep the order they had: the positive phase makes none.
            X.branch(0)
            try:
                a, b = positive(), negative()
                more = [True, True]
                while any(more):
                    if more[0]:
                        more[0] = next(a, 0) is None
                    if more[1]:
                        X.branch(1)
                        more[1] = next(b, 0) is None
                        X.branch(2)
            finally:
                X.branch(3)
        # ---- statistics pos - neg and updates (the visible positive state is the data)
        for i in range(L - 1):
            # the difference of two nearly equal products: TF32 correction terms; the data are exact
            P = cm.split_passes
            p = P(data if i == 0 else pos[i], pos[i + 1].T, exact_a=(i == 0), terms="tf32")
            n = P(neg[i], neg[i + 1].T, negate=1, terms="tf32")
            X.fused_gemm(p + n, out=self.suff_W[i])
        self.kernel_launches += (L - 1) + 1 + (L - 1) + (2 * L if first_step else 0)
        inv_b = 1.0 / self.B
        layers = [(data if j == 0 else pos[j], neg[j], self.suff_b[j], self.b[j], self.db[j]) for j in range(L)]
        # the first four layers' biases go with the first weights (past 1024 cases in launches of their own)
        first = X.update_all(layers[:4], self.W[0], self.dW[0], self.suff_W[0], self.W_aux[0], inv_b, mom, eps, mom, eps, l2=l2,
                             l1=l1)
        bias_ops = [X.bias_updates(layers[j:j + 4], inv_b, mom, eps) for j in range(4, L, 4)]
        weight_ops = [X.momentum_update(self.W[i], self.dW[i], None, self.suff_W[i], inv_b, mom, eps, l2=l2, l1=l1,
                                        w_aux=self.W_aux[i]) for i in range(1, L - 1)]
        self.kernel_launches += (len(bias_ops) if self.B <= 1024 else 2 * L) + L - 1
        return bias_ops, weight_ops, first

    def read_loss(self, reset=True):
        v = float(np.array(self.loss_acc.asarray())[0, 0])
        if reset:
            self.loss_acc.assign(0)
        return v
