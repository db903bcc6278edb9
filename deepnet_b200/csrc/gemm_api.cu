// C entry points built on the fused matrix product: the reference `dot`
// (cudamat/cudamat.cu:1671-1696) and the fused calls that replace whole groups of
// reference operations on the contrastive-divergence path (deepnet/dbm.py:64-115,
// deepnet/edge.py:222-246, deepnet/parameter.py:80-106).
#include "gemm.cuh"

using namespace b200;

namespace {

int g_path = 0;       // 0 auto; one kernel only: 1 tcgen05, 2 CUDA cores, 3 the one-launch kernel, 4 tcgen05 behind aligned copies
int g_dot_mode = 0;   // 0: fp32-grade (three TF32 terms), 1: single TF32 term
constexpr long kTcMinWork = 1L << 21;  // below this many multiply-adds `dot` multiplies full fp32 operands

inline int lead(const cudamat* m) { return m->is_trans ? m->size[1] : m->size[0]; }
inline int nonlead(const cudamat* m) { return m->is_trans ? m->size[0] : m->size[1]; }
inline GemmOperand operand(const cudamat* m, int part, const cudamat* aux = nullptr) {
  GemmOperand o;
  o.ptr = m->data_device;
  o.ld = m->size[0];
  o.trans = m->is_trans;
  o.part = part;
  o.aux = aux ? aux->data_device : nullptr;
  o.lda = aux ? aux->size[0] : 0;
  o.row0 = 0;
  return o;
}
// An aux handle holds aux_rows(rows) x cols floats.
inline bool aux_shape_ok(const cudamat* aux, const cudamat* m) {
  return aux->on_device && aux->size[0] == aux_rows(m->size[0]) && aux->size[1] == m->size[1];
}

// Where the tcgen05 kernel needs aligned copies of its operands first: the one-launch kernel (gemm_small.cu) up to so many
// slabs of 32 of K that an SM has to walk.  Measured (one launch against copies + product + finish): 8 slabs 20.0 against
// 26.6 us (1021 x 255, K = 1021), 11 slabs 25.1 against 26.3 (601 x 203, K = 1357), 14 slabs 32.7 against 28.9 (1357 x 601,
// two pairs of K = 203).
constexpr int kSmallDepth = 11;

// `dot` on operands TMA cannot address and `dot` of little work multiply full fp32 operands with rounding adds (k_gemm_simt,
// and in one launch gemm_small's fp32 form): a 0/1 selection returns the selected entries bit for bit, integer
// products below 2^24 are exact, an infinity keeps its meaning.  Split TF32 holds 22 or 23 bits of an operand, which shows
// while K is short.  Relative error against float64, 201 x 101 outputs, normal operands (0/1 against normal):
//   K       k_gemm_simt         one launch, fp32    one launch, split   split, aligned copies
//   1       2.5e-8  (0)         2.5e-8  (0)         7.9e-8  (2.9e-8)    4.0e-7  (1.2e-7)
//   16      7.3e-8  (3.6e-8)    7.3e-8  (3.6e-8)    1.4e-7  (6.2e-8)    4.0e-7  (1.4e-7)
//   100     1.8e-7  (7.9e-8)    1.0e-7  (5.9e-8)    2.4e-7  (9.4e-8)    4.3e-7  (1.5e-7)
//   400     3.6e-7  (1.4e-7)    1.4e-7  (7.5e-8)    2.4e-7  (1.0e-7)    4.3e-7  (1.6e-7)
//   600     4.5e-7  (1.8e-7)    1.3e-7  (8.2e-8)    2.4e-7  (1.1e-7)    4.3e-7  (1.6e-7)
//   4001    1.1e-6  (4.4e-7)    2.9e-7  (1.3e-7)    2.6e-7  (1.2e-7)    4.5e-7  (1.9e-7)
// The fp32 form costs what the split costs to within a fifth (us): 201 x 101, K = 1001: 183.6 / 10.8 / 9.8 / 14.8; 1021 x
// 255, K = 1021: 191 / 22.7 / 20.0 / 26.6.  From K = 600 on the split behind aligned copies is no less exact than
// k_gemm_simt was on random operands, and deeper products take it (2047 x 511, K = 2047: 433 / 149 / 127 / 46).
constexpr int kPackedDotK = 600;

// TF32 terms of odd matrices that the tcgen05 kernel's truncating adds do not suit: chunks of 32 keep the error of long sums
// below that of k_gemm_simt, which ran them and rounds every addition, but not that of short ones, nor, ever, with an exact
// operand (0/1).  They take one launch, a short single pair in its fp32 form.  Relative error against float64:
//                                      k_gemm_simt  copies, tcgen05  one launch, split  one launch, fp32
//   one pair, K = 64                   3.7e-7       4.3e-7           2.5e-7             1.1e-7
//   the same, positive operands        2.7e-7       3.7e-7           2.3e-7             0.7e-7
//   positive operands, K = 400         3.8e-7       3.7e-7           2.0e-7             0.6e-7
//   0/1 and positive operand, K = 65   8.0e-8       1.2e-7           8.4e-8             4.2e-8
//   the same, K = 801                  8.0e-8       1.2e-7           9.0e-8             1.05e-7   (an ulp: 1.2e-7)
//   difference of two of K = 32        1.9e-6       2.0e-6           0.6e-6
//   difference of two of K = 64        2.7e-6       2.2e-6           1.5e-6
enum { kAnyLength, kOneLaunchFp32, kOneLaunch };
int short_tf32(const GemmProblem& g) {
  long k = 0;
  int pairs = 0, low = 0;
  for (int q = 0; q < g.npass; q++) {
    const int pa = g.pass[q].a.part, pb = g.pass[q].b.part;
    if (pa == kPartX && pb == kPartX) {
      k += g.pass[q].k;
      pairs++;
    }
    if (pa == kPartLo32 || pb == kPartLo32) low++;
  }
  if (!low) return kAnyLength;
  if (pairs == 1 && k < 400) return kOneLaunchFp32;
  return k < 128 || (pairs == 1 && low == 1) ? kOneLaunch : kAnyLength;
}

__global__ void __launch_bounds__(256) k_copy(const float* x, float* y, long n, bool vec) {
  grid_dependents_launch();
  grid_dependency_wait();
  const long tid = (long)blockIdx.x * blockDim.x + threadIdx.x, nth = (long)gridDim.x * blockDim.x;
  if (vec) {
    for (long i = tid; i < n / 4; i += nth) reinterpret_cast<float4*>(y)[i] = reinterpret_cast<const float4*>(x)[i];
  } else {
    for (long i = tid; i < n; i += nth) y[i] = x[i];
  }
}

// The one-launch kernel reads the matrix that is added where it lies; the others, whose products are long, find it in the
// output.  (A kernel, not cudaMemcpyAsync: the launches around it stay dependent.)
int prior_to_output(GemmProblem& g) {
  const long n = (long)g.M * g.N;
  if (!g.prior || n == 0) return 0;
  const bool vec = n % 4 == 0 && (((uintptr_t)g.prior | (uintptr_t)g.epi.out) & 15) == 0;
  long blocks = ((vec ? n / 4 : n) + 255) / 256;
  if (blocks > (long)sm_count() * 8) blocks = (long)sm_count() * 8;
  if (launch_dependent(k_copy, dim3((unsigned)blocks), dim3(256), 0, stream(), g.prior, g.epi.out, n, vec) != cudaSuccess)
    return set_error(cudaGetErrorString(cudaGetLastError()));
  g.prior = nullptr;
  return check_launch();
}

// A product takes the same way with a matrix to add as without.
int run(GemmProblem& g) {
  auto after_copy = [&](int (*kernel)(const GemmProblem&)) {
    const int err = prior_to_output(g);
    return err ? err : kernel(g);
  };
  if (product_is_scattered(g.epi.out)) return after_copy(gemm_tc);   // (fails loudly when the tensor-core kernel cannot take it)
  if (g_path == 2) return after_copy(gemm_simt);
  if (g_path == 3) return gemm_small(g, kSmallSplit);
  if (g_path == 4) return after_copy(gemm_tc_packed);
  const bool tc = gemm_tc_supported(g);
  int r = ERROR_UNSUPPORTED;
  if (g_path == 0 && tc) {
    if (small_beats_tc(g)) r = gemm_small(g, kSmallSplit);
  } else if (g_path == 0) {
    const int tf32 = short_tf32(g), depth = small_depth(g);
    if (tf32 == kOneLaunchFp32) r = gemm_small(g, kSmallFp32Parts);
    if (r == ERROR_UNSUPPORTED && depth > 0 && (depth <= kSmallDepth || tf32 != kAnyLength)) r = gemm_small(g, kSmallSplit);
  }
  if (r != ERROR_UNSUPPORTED) return r;
  // (unsupported: more operand pairs or tiles than one tensor-core launch carries)
  if (tc) r = after_copy(gemm_tc);
  else if (g_path == 0) r = after_copy(gemm_tc_packed);
  if (r != ERROR_UNSUPPORTED || g_path == 1) return r;
  r = gemm_small(g, kSmallSplit);
  return r != ERROR_UNSUPPORTED ? r : after_copy(gemm_simt);
}

// hi may be null: the tensor core itself drops the low 13 mantissa bits of an fp32
// operand, so the matrix x can stand in for its own high part and only lo is stored.
__global__ void __launch_bounds__(256) k_split(const float* x, float* hi, float* lo, long n, bool vec) {
  grid_dependents_launch();
  grid_dependency_wait();
  const long tid = (long)blockIdx.x * blockDim.x + threadIdx.x, nth = (long)gridDim.x * blockDim.x;
  if (vec) {
    const long n4 = n >> 2;
    for (long i = tid; i < n4; i += nth) {
      const float4 v = reinterpret_cast<const float4*>(x)[i];
      float4 h, l;
      split_tf32(v.x, h.x, l.x); split_tf32(v.y, h.y, l.y); split_tf32(v.z, h.z, l.z); split_tf32(v.w, h.w, l.w);
      if (hi) reinterpret_cast<float4*>(hi)[i] = h;
      reinterpret_cast<float4*>(lo)[i] = l;
    }
    for (long i = (n4 << 2) + tid; i < n; i += nth) {
      float h, l;
      split_tf32(x[i], h, l);
      if (hi) hi[i] = h;
      lo[i] = l;
    }
  } else {
    for (long i = tid; i < n; i += nth) {
      float h, l;
      split_tf32(x[i], h, l);
      if (hi) hi[i] = h;
      lo[i] = l;
    }
  }
}

// aux matrix of x (rows x cols, contiguous columns): both bfloat16 planes in one pass.
__global__ void __launch_bounds__(256) k_split_aux(const float* x, uint16_t* aux, int rows, int lda, long n,
                                                   bool vec) {
  grid_dependents_launch();
  grid_dependency_wait();
  const long tid = (long)blockIdx.x * blockDim.x + threadIdx.x, nth = (long)gridDim.x * blockDim.x;
  if (vec) {   // rows % 4 == 0: four consecutive elements share a column
    for (long i = tid; i < (n >> 2); i += nth) {
      const float4 v = reinterpret_cast<const float4*>(x)[i];
      const long e = i << 2, c = e / rows, r = e - c * rows;
      ushort4 l, b;
      split_aux(v.x, l.x, b.x); split_aux(v.y, l.y, b.y); split_aux(v.z, l.z, b.z); split_aux(v.w, l.w, b.w);
      uint16_t* dst = aux + c * 2 * lda + r;
      *reinterpret_cast<ushort4*>(dst) = l;
      *reinterpret_cast<ushort4*>(dst + lda) = b;
    }
  } else {
    for (long i = tid; i < n; i += nth) {
      const long c = i / rows, r = i - c * rows;
      uint16_t l, b;
      split_aux(x[i], l, b);
      aux[c * 2 * lda + r] = l;
      aux[c * 2 * lda + lda + r] = b;
    }
  }
}

// aux matrix of x in scaled half-precision form (split_f16): scale = 2^(*exp_dev + exp_const).
// `only_if` (optional): a device flag; the kernel returns at once when it is zero.
__global__ void __launch_bounds__(256) k_split_f16(const float* x, uint16_t* aux, int rows, int lda, long n, bool vec,
                                                   const float* exp_dev, int exp_const, const float* only_if) {
  grid_dependents_launch();
  grid_dependency_wait();
  if (only_if && *only_if == 0.0f) return;
  const float scale = exp2f((exp_dev ? *exp_dev : 0.0f) + (float)exp_const);
  const long tid = (long)blockIdx.x * blockDim.x + threadIdx.x, nth = (long)gridDim.x * blockDim.x;
  if (vec) {
    for (long i = tid; i < (n >> 2); i += nth) {
      const float4 v = reinterpret_cast<const float4*>(x)[i];
      const long e = i << 2, c = e / rows, r = e - c * rows;
      ushort4 l, h;
      split_f16(v.x, scale, l.x, h.x); split_f16(v.y, scale, l.y, h.y);
      split_f16(v.z, scale, l.z, h.z); split_f16(v.w, scale, l.w, h.w);
      uint16_t* dst = aux + c * 2 * lda + r;
      *reinterpret_cast<ushort4*>(dst) = l;
      *reinterpret_cast<ushort4*>(dst + lda) = h;
    }
  } else {
    for (long i = tid; i < n; i += nth) {
      const long c = i / rows, r = i - c * rows;
      uint16_t l, h;
      split_f16(x[i], scale, l, h);
      aux[c * 2 * lda + r] = l;
      aux[c * 2 * lda + lda + r] = h;
    }
  }
}

// aux holds aux_rows(rows) floats per column.
int launch_split_aux(const float* x, float* aux, int rows, long n) {
  if (n == 0) return 0;
  const bool vec = (rows % 4 == 0) && ((((uintptr_t)x) & 15) == 0) && ((((uintptr_t)aux) & 7) == 0);
  long blocks = ((vec ? n / 4 : n) + 255) / 256;
  if (blocks > (long)sm_count() * 8) blocks = (long)sm_count() * 8;
  if (blocks < 1) blocks = 1;
  if (launch_dependent(k_split_aux, dim3((unsigned)blocks), dim3(256), 0, stream(), x, reinterpret_cast<uint16_t*>(aux), rows,
                       aux_rows(rows), n, vec) != cudaSuccess)
    return set_error(cudaGetErrorString(cudaGetLastError()));
  return check_launch();
}

int launch_split(const float* x, float* hi, float* lo, long n) {
  if (n == 0) return 0;
  const bool vec = (((uintptr_t)x | (uintptr_t)hi | (uintptr_t)lo) & 15) == 0;
  long blocks = ((vec ? (n + 3) / 4 : n) + 255) / 256;
  if (blocks > (long)sm_count() * 8) blocks = (long)sm_count() * 8;
  (void)launch_dependent(k_split, dim3((unsigned)blocks), dim3(256), 0, stream(), x, hi, lo, n, vec);
  return check_launch();
}

// One pass of the parameter update, in the order the reference issues its calls
// (deepnet/dbm.py:242,254 then deepnet/parameter.py:89-106).  Products and sums are
// rounded separately (no fused multiply-add) so the result equals the call sequence's.
__device__ __forceinline__ void update_one(float& w, float& d, float g, float suff, float ninv_batch, float momentum,
                                           float neps, float l2, float l1) {
  g = __fadd_rn(g, __fmul_rn(suff, ninv_batch));
  d = __fmul_rn(d, momentum);
  if (l2 != 0.0f) d = __fadd_rn(d, __fmul_rn(w, l2));
  if (l1 != 0.0f) d = __fadd_rn(d, w == 0.0f ? 0.0f : (w > 0.0f ? l1 : -l1));
  d = __fadd_rn(d, g);
  w = __fadd_rn(w, __fmul_rn(d, neps));
}

// What ends an update beside the weights, in one launch: for every unit r of up to four layers
//   suff[r] = sum_c pos[r, c] - neg[r, c]   (deepnet/layer.py:202-213), then the parameter update of the biases,
// and, with `acc`, acc[0] += sum (pos - neg)^2 of the first, the reconstruction error of deepnet/logistic_layer.py:48-52
// (the visible rows are being read anyway).  A block owns 32 rows whole (32 lanes of cases, four rows a thread, folded in
// order), so the sums need no second pass; the error's partial sums (doubles) are folded by the block that finishes last, in
// order.  Latency bound at the sizes it is used for.  Four launches before: 784 + 500 units, 100 cases: 10.6 -> 4 us; with 8
// lanes of cases and one row a thread the walk over 512 cases stood behind the weights' blocks (2048 x 2048: 22.2 -> 13.9 us).
constexpr int kTailLanes = 32, kTailThreads = 8 * kTailLanes;
constexpr int kTailLayers = 4;
struct TailLayer {
  const float *pos, *neg;
  float *suff, *b, *db;
  int rows, block0;        // first block
};
struct TailArgs {
  TailLayer l[kTailLayers];
  int layers, cases;
  double* part;
  unsigned* counter;
  float *acc, ninv_batch, momentum, neps;
};
__device__ __forceinline__ void bias_tail(const TailArgs& a) {
  __shared__ float sums[kTailLanes][33];
  __shared__ double sq[kTailThreads / 32];
  __shared__ bool is_last;
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3, cases = a.cases;
  int which = 0;
  while (which + 1 < a.layers && (int)blockIdx.x >= a.l[which + 1].block0) which++;
  const TailLayer l = a.l[which];
  const int r0 = 32 * ((int)blockIdx.x - l.block0), r = r0 + 4 * tx;
  const bool err = which == 0 && a.acc != nullptr;
  const int err_blocks = (a.l[0].rows + 31) / 32;
  float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  double e = 0.0;
  const bool vec = l.rows % 4 == 0 && (((uintptr_t)l.pos | (uintptr_t)l.neg) & 15) == 0;
  auto difference = [&](int c) {
    const long o = (long)c * l.rows + r;
    if (vec) {
      const float4 p = *reinterpret_cast<const float4*>(l.pos + o), n = *reinterpret_cast<const float4*>(l.neg + o);
      return make_float4(p.x - n.x, p.y - n.y, p.z - n.z, p.w - n.w);
    }
    return make_float4(l.pos[o] - l.neg[o], r + 1 < l.rows ? l.pos[o + 1] - l.neg[o + 1] : 0.0f,
                       r + 2 < l.rows ? l.pos[o + 2] - l.neg[o + 2] : 0.0f, r + 3 < l.rows ? l.pos[o + 3] - l.neg[o + 3] : 0.0f);
  };
  auto add = [&](const float4& d) {
    s[0] += d.x;
    s[1] += d.y;
    s[2] += d.z;
    s[3] += d.w;
    if (err) e += ((double)d.x * d.x + (double)d.y * d.y) + ((double)d.z * d.z + (double)d.w * d.w);
  };
  if (r < l.rows) {
    int c = ty;
    for (; c + 3 * kTailLanes < cases; c += 4 * kTailLanes) {   // eight loads in flight
      float4 d[4];
#pragma unroll
      for (int i = 0; i < 4; i++) d[i] = difference(c + i * kTailLanes);
#pragma unroll
      for (int i = 0; i < 4; i++) add(d[i]);
    }
    for (; c < cases; c += kTailLanes) add(difference(c));
  }
#pragma unroll
  for (int i = 0; i < 4; i++) sums[ty][4 * tx + i] = s[i];
  if (err) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if ((threadIdx.x & 31) == 0) sq[threadIdx.x >> 5] = e;
  }
  __syncthreads();
  {
    const int row = threadIdx.x & 31, first = threadIdx.x >> 5;   // lanes first, first + 8, ...
    float t = 0.0f;
#pragma unroll
    for (int j = 0; j < kTailLanes; j += 8) t += sums[first + j][row];
    sums[first][row] = t;    // (the only thread that reads it before the barrier)
  }
  __syncthreads();
  if (threadIdx.x < 32 && r0 + (int)threadIdx.x < l.rows) {
    const int row = r0 + (int)threadIdx.x;
    float t = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; j++) t += sums[j][threadIdx.x];
    l.suff[row] = t;
    float w = l.b[row], d = l.db[row];
    update_one(w, d, 0.0f, t, a.ninv_batch, a.momentum, a.neps, 0.0f, 0.0f);
    l.b[row] = w;
    l.db[row] = d;
  }
  if (!err) return;
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int j = 0; j < kTailThreads / 32; j++) t += sq[j];
    a.part[blockIdx.x] = t;
    __threadfence();
    is_last = atomicAdd(a.counter, 1u) == (unsigned)(err_blocks - 1);
  }
  __syncthreads();
  if (!is_last || threadIdx.x >= 32) return;
  __threadfence();
  double t = 0.0;
  for (int i = threadIdx.x; i < err_blocks; i += 32) t += __ldcg(a.part + i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (threadIdx.x == 0) {
    *a.acc += (float)t;
    *a.counter = 0u;
  }
}
__global__ void __launch_bounds__(kTailThreads) k_bias_tail(const __grid_constant__ TailArgs a) {
  grid_dependents_launch();
  grid_dependency_wait();
  bias_tail(a);
}

// One block walks all cases of its 32 rows: past this many cases the launches that also split the cases are faster.
constexpr int kTailCases = 1024;

}  // namespace

extern "C" {
int row_sum_diff(cudamat* a, cudamat* b, cudamat* target);
int add_sq_diff(cudamat* a, cudamat* b, cudamat* acc);
int momentum_update(cudamat* w, cudamat* delta, cudamat* grad, cudamat* suff, cudamat* w_aux, cudamat* w_scale,
                    float inv_batch, float momentum, float eps, float l2, float l1);
}

// Bias statistics (positive minus negative) and bias update of up to four layers and, with sq_acc, the squared
// difference of the first layer's states.
struct b200_bias_layers {
  cudamat *pos[kTailLayers], *neg[kTailLayers], *suff[kTailLayers], *b[kTailLayers], *db[kTailLayers];
  cudamat* sq_acc;
  int layers;
};
// Checks the layers; blocks: of the one launch, 0 where the sums take launches of their own.
static int plan_bias_tail(b200_bias_layers* t, float inv_batch, float momentum, float eps, TailArgs& a, int& blocks) {
  blocks = 0;
  if (!t || t->layers < 1 || t->layers > kTailLayers) return ERROR_UNSUPPORTED;
  const int n = t->layers;
  bool empty = false;
  for (int i = 0; i < n; i++) {
    for (cudamat* m : {t->pos[i], t->neg[i], t->suff[i], t->b[i], t->db[i]}) {
      if (!m) return ERROR_GENERIC;
      if (!m->on_device) return ERROR_NOT_ON_DEVICE;
      if (m->is_trans) return ERROR_TRANSPOSED;
    }
    const long rows = t->pos[i]->size[0];
    if (!same_shape(t->pos[i], t->neg[i]) || t->pos[i]->size[1] != t->pos[0]->size[1] || numel(t->suff[i]) != rows ||
        numel(t->b[i]) != rows || numel(t->db[i]) != rows)
      return ERROR_INCOMPATIBLE_DIMENSIONS;
    empty = empty || rows == 0;
  }
  if (t->sq_acc && !t->sq_acc->on_device) return ERROR_NOT_ON_DEVICE;
  if (t->sq_acc && numel(t->sq_acc) < 1) return ERROR_INCOMPATIBLE_DIMENSIONS;
  a.cases = t->pos[0]->size[1];
  if (a.cases > kTailCases || a.cases == 0 || empty) return 0;
  a.layers = n;
  for (int i = 0; i < n; i++) {
    a.l[i] = {t->pos[i]->data_device, t->neg[i]->data_device, t->suff[i]->data_device, t->b[i]->data_device,
              t->db[i]->data_device, t->pos[i]->size[0], blocks};
    blocks += (a.l[i].rows + 31) / 32;
  }
  a.part = nullptr;
  a.counter = nullptr;
  a.acc = nullptr;
  a.ninv_batch = -inv_batch;
  a.momentum = momentum;
  a.neps = -eps;
  if (t->sq_acc) {
    a.acc = t->sq_acc->data_device;
    a.part = (double*)workspace(1, (size_t)((a.l[0].rows + 31) / 32 + 1) * sizeof(double));
    a.counter = (unsigned*)workspace_zeroed(3, 4096 * sizeof(unsigned));   // (the first counter: add_sq_diff's, zero between calls)
    if (!a.part || !a.counter) return CUDA_ERROR;
  }
  return 0;
}
extern "C" int bias_updates(b200_bias_layers* t, float inv_batch, float momentum, float eps) {
  TailArgs a;
  int blocks = 0;
  int err = plan_bias_tail(t, inv_batch, momentum, eps, a, blocks);
  if (err) return err;
  if (blocks == 0) {
    const int n = t->layers;
    err = t->sq_acc ? add_sq_diff(t->neg[0], t->pos[0], t->sq_acc) : 0;
    for (int i = 0; i < n && !err; i++) err = row_sum_diff(t->pos[i], t->neg[i], t->suff[i]);
    for (int i = 0; i < n && !err; i++)
      err = momentum_update(t->b[i], t->db[i], nullptr, t->suff[i], nullptr, nullptr, inv_batch, momentum, eps, 0.0f, 0.0f);
    return err;
  }
  if (launch_dependent(k_bias_tail, dim3((unsigned)blocks), dim3(kTailThreads), 0, stream(), a) != cudaSuccess)
    return set_error(cudaGetErrorString(cudaGetLastError()));
  return check_launch();
}

// The same for an RBM whose biases, histories and statistics are packed [visible | hidden].
extern "C" int rbm_bias_update(cudamat* v_pos, cudamat* v_neg, cudamat* h_pos, cudamat* h_neg, cudamat* suff, cudamat* b,
                               cudamat* db, cudamat* sq_acc, float inv_batch, float momentum, float eps) {
  cudamat* all[7] = {v_pos, v_neg, h_pos, h_neg, suff, b, db};
  for (int i = 0; i < 7; i++) {
    if (!all[i]->on_device) return ERROR_NOT_ON_DEVICE;
    if (all[i]->is_trans) return ERROR_TRANSPOSED;
  }
  const int V = v_pos->size[0], H = h_pos->size[0];
  if (numel(suff) != (long)V + H || !same_shape(suff, b) || !same_shape(suff, db)) return ERROR_INCOMPATIBLE_DIMENSIONS;
  cudamat half[6];       // suff, b, db of either layer
  for (int i = 0; i < 3; i++) {
    half[i] = half[3 + i] = *all[4 + i];
    half[i].size[0] = V;
    half[3 + i].size[0] = H;
    half[i].size[1] = half[3 + i].size[1] = 1;
    half[3 + i].data_device += V;
  }
  b200_bias_layers t = {{v_pos, h_pos}, {v_neg, h_neg}, {half, half + 3}, {half + 1, half + 4}, {half + 2, half + 5}, sq_acc, 2};
  return bias_updates(&t, inv_batch, momentum, eps);
}

namespace {

// kAux: 0 no aux, 1 bfloat16 parts, 2 scaled half-precision form.  For 2 the aux is written with
// the exponent the parameter has carried so far (`scale` = {exponent, copy, max |w| bits, redo flag})
// and the largest |w| of the new parameter is gathered into scale[2]; k_update_scale then checks
// that this exponent still fits the new parameter (it does unless the weights grew eightfold or
// shrank by more than half in one update) and only otherwise sets the flag that makes a second
// pass (k_split_f16) rewrite the aux with a new exponent.  One pass over the weights in the
// common case: 24 bytes per weight instead of 28.
template <bool kHasGrad, int kAux>
__device__ __forceinline__ void update_weights(float* w, float* delta, float* grad, const float* suff, uint16_t* w_aux,
                                               float* scale, int rows, int lda, long n, bool vec, float ninv_batch,
                                               float momentum, float neps, float l2, float l1, int block, int blocks) {
  const long tid = (long)block * blockDim.x + threadIdx.x, nth = (long)blocks * blockDim.x;
  float wmax = 0.0f;
  const float f16_scale = kAux == 2 ? exp2f(scale[0]) : 1.0f;
  if (vec) {   // n % 4 == 0, and with an aux rows % 4 == 0: four consecutive elements share a column
    for (long i = tid; i < (n >> 2); i += nth) {
      float4 W = reinterpret_cast<float4*>(w)[i];
      float4 D = reinterpret_cast<float4*>(delta)[i];
      const float4 S = __ldcs(reinterpret_cast<const float4*>(suff) + i);   // (read for the last time: leaves the L2 first)
      float4 G = make_float4(0, 0, 0, 0);
      if (kHasGrad) G = reinterpret_cast<float4*>(grad)[i];
      update_one(W.x, D.x, G.x, S.x, ninv_batch, momentum, neps, l2, l1);
      update_one(W.y, D.y, G.y, S.y, ninv_batch, momentum, neps, l2, l1);
      update_one(W.z, D.z, G.z, S.z, ninv_batch, momentum, neps, l2, l1);
      update_one(W.w, D.w, G.w, S.w, ninv_batch, momentum, neps, l2, l1);
      reinterpret_cast<float4*>(w)[i] = W;
      reinterpret_cast<float4*>(delta)[i] = D;
      if (kHasGrad) reinterpret_cast<float4*>(grad)[i] = make_float4(0, 0, 0, 0);
      if (kAux == 1) {
        const long e = i << 2, c = e / rows, r = e - c * rows;
        ushort4 L, B;
        split_aux(W.x, L.x, B.x); split_aux(W.y, L.y, B.y); split_aux(W.z, L.z, B.z); split_aux(W.w, L.w, B.w);
        uint16_t* dst = w_aux + c * 2 * lda + r;
        *reinterpret_cast<ushort4*>(dst) = L;
        *reinterpret_cast<ushort4*>(dst + lda) = B;
      }
      if (kAux == 2) {
        wmax = fmaxf(fmaxf(wmax, fmaxf(fabsf(W.x), fabsf(W.y))), fmaxf(fabsf(W.z), fabsf(W.w)));
        const long e = i << 2, c = e / rows, r = e - c * rows;
        ushort4 L, Hh;
        split_f16(W.x, f16_scale, L.x, Hh.x); split_f16(W.y, f16_scale, L.y, Hh.y);
        split_f16(W.z, f16_scale, L.z, Hh.z); split_f16(W.w, f16_scale, L.w, Hh.w);
        uint16_t* dst = w_aux + c * 2 * lda + r;
        *reinterpret_cast<ushort4*>(dst) = L;
        *reinterpret_cast<ushort4*>(dst + lda) = Hh;
      }
    }
  } else {
    for (long i = tid; i < n; i += nth) {
      float W = w[i], D = delta[i];
      update_one(W, D, kHasGrad ? grad[i] : 0.0f, suff[i], ninv_batch, momentum, neps, l2, l1);
      w[i] = W; delta[i] = D;
      if (kHasGrad) grad[i] = 0.0f;
      if (kAux == 1) {
        const long c = i / rows, r = i - c * rows;
        uint16_t L, B;
        split_aux(W, L, B);
        w_aux[c * 2 * lda + r] = L;
        w_aux[c * 2 * lda + lda + r] = B;
      }
      if (kAux == 2) {
        wmax = fmaxf(wmax, fabsf(W));
        const long c = i / rows, r = i - c * rows;
        uint16_t L, Hh;
        split_f16(W, f16_scale, L, Hh);
        w_aux[c * 2 * lda + r] = L;
        w_aux[c * 2 * lda + lda + r] = Hh;
      }
    }
  }
  if (kAux == 2) {
    // Non-negative floats order like their bit patterns.  One atomic a block, and only by blocks that raise the maximum: one a
    // warp, all on one word, took 15 us of the 33 of a 2048 x 2048 update.
    __shared__ unsigned warp_max[8];
    const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(wmax));
    if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned b = warp_max[0];
      for (int i = 1; i < 8; i++) b = max(b, warp_max[i]);
      unsigned* const at = reinterpret_cast<unsigned*>(scale) + 2;
      if (b > *(volatile unsigned*)at) atomicMax(at, b);
    }
  }
}

template <bool kHasGrad, int kAux>
__global__ void __launch_bounds__(256) k_update(float* w, float* delta, float* grad, const float* suff,
                                                uint16_t* w_aux, float* scale, int rows, int lda, long n, bool vec,
                                                float ninv_batch, float momentum, float neps, float l2, float l1) {
  grid_dependents_launch();
  grid_dependency_wait();
  update_weights<kHasGrad, kAux>(w, delta, grad, suff, w_aux, scale, rows, lda, n, vec, ninv_batch, momentum, neps, l2, l1,
                                 (int)blockIdx.x, (int)gridDim.x);
}

// The biases' blocks and the weights' in one launch: neither needs the other, and one after the other the first, bound by
// latency, stood before the second, bound by memory.  784 x 500, 100 cases: update 51.1 -> 48.6 us; 2048 x 2048, 512: 180.5 -> 172.8.
struct UpdateArgs {
  float *w, *delta;
  const float* suff;
  uint16_t* w_aux;
  int rows, lda;
  long n;
  bool vec;
  float ninv_batch, momentum, neps, l2, l1;
  float* scale;            // of the scaled half-precision form
  unsigned* done;          // blocks that have finished, zero between calls
};

// The exponent after an update in scaled half-precision form, see k_update_scale; true: the planes have to be rewritten.
__device__ __forceinline__ bool update_scale(float* scale) {
  const float m = __uint_as_float(__ldcg(reinterpret_cast<unsigned*>(scale) + 2));
  bool redo = false;
  float want = scale[0];
  if (m > 0.0f && m < 3.0e38f) {
    want = f16_exponent(m);
    const float d = scale[0] - want;
    if (d < -1.0f || d > 2.0f) {
      scale[0] = want;
      redo = true;
    }
  }
  scale[1] = want;
  reinterpret_cast<unsigned*>(scale)[2] = 0u;
  return redo;
}

// Weights whose planes one block rewrites alone; of more of them a launch of its own, which returns at once unless it has to.
constexpr long kRedoByOneBlock = 1L << 19;

// kAux 2: the block that finishes last decides on the exponent, and rewrites the planes in the rare update that has to (weights
// grown eightfold or halved since it was chosen): one or two launches less.
template <int kAux>
__global__ void __launch_bounds__(256) k_update_all(const __grid_constant__ TailArgs a, const __grid_constant__ UpdateArgs u,
                                                    int tail_blocks) {
  grid_dependents_launch();
  grid_dependency_wait();
  if ((int)blockIdx.x < tail_blocks) {
    bias_tail(a);
    return;
  }
  const int block = (int)blockIdx.x - tail_blocks, blocks = (int)gridDim.x - tail_blocks;
  update_weights<false, kAux>(u.w, u.delta, nullptr, u.suff, u.w_aux, u.scale, u.rows, u.lda, u.n, u.vec, u.ninv_batch, u.momentum,
                              u.neps, u.l2, u.l1, block, blocks);
  if (kAux == 2) {
    __shared__ int redo;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      redo = 0;
      if (atomicAdd(u.done, 1u) == (unsigned)(blocks - 1)) {
        __threadfence();
        redo = update_scale(u.scale) ? 1 : 0;
        u.scale[3] = redo ? 1.0f : 0.0f;
        *u.done = 0u;
      }
    }
    __syncthreads();
    if (!redo || u.n > kRedoByOneBlock) return;
    const float s = exp2f(u.scale[0]);
    for (long i0 = threadIdx.x; i0 < u.n; i0 += 8 * 256) {
      float w[8];
#pragma unroll
      for (int j = 0; j < 8; j++) w[j] = i0 + 256 * j < u.n ? __ldcg(u.w + i0 + 256 * j) : 0.0f;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const long i = i0 + 256 * j, c = i / u.rows, r = i - c * u.rows;
        if (i >= u.n) break;
        uint16_t l, h;
        split_f16(w[j], s, l, h);
        u.w_aux[c * 2 * u.lda + r] = l;
        u.w_aux[c * 2 * u.lda + u.lda + r] = h;
      }
    }
  }
}

// After an update in scaled half-precision form.  The exponent wanted for the new parameter puts
// the largest |w| * 2^e in (2^12, 2^13] (the fp16 limit is just under 2^16).  The aux was written
// with the exponent carried so far; it stands while the largest scaled magnitude stays within
// (2^11, 2^15].  Otherwise the wanted exponent, which scale[1] names in any case, is stored and scale[3] tells the second pass to
// rewrite the aux.  The maximum starts over.  A parameter that is all zero (or not finite) keeps
// its exponent.
__global__ void k_update_scale(float* scale) {
  grid_dependents_launch();
  grid_dependency_wait();
  scale[3] = update_scale(scale) ? 1.0f : 0.0f;
}

}  // namespace

namespace b200 {
int rewrite_f16_planes_if(const float* x, uint16_t* aux, int rows, long n, const float* exp_dev, const float* only_if) {
  if (n == 0) return 0;
  const bool svec = (rows % 4 == 0) && ((((uintptr_t)x) & 15) == 0);
  long sblocks = ((svec ? n / 4 : n) + 255) / 256;
  if (sblocks > (long)sm_count() * 8) sblocks = (long)sm_count() * 8;
  if (sblocks < 1) sblocks = 1;
  if (launch_dependent(k_split_f16, dim3((unsigned)sblocks), dim3(256), 0, stream(), x, aux, rows, aux_rows(rows), n, svec,
                       exp_dev, 0, only_if) != cudaSuccess)
    return set_error(cudaGetErrorString(cudaGetLastError()));
  return check_launch();
}
}  // namespace b200

// One term of a fused product: op(a) is M x k, op(b) is k x N (handles carry is_trans).
// a_part / b_part choose what of each fp32 matrix the term multiplies (kPartX, kPartLo32:
// a TF32 product; kPartLo16, kPartB16: a bfloat16 product); both of one width.  a_aux / b_aux:
// the aux matrix of a / b (or null): its bfloat16 parts are then read from there.
struct b200_pass {
  cudamat* a;
  cudamat* b;
  int negate;
  int a_part, b_part;
  cudamat* a_aux;
  cudamat* b_aux;
  // Row windows of the STORED matrices (0, 0 = all rows): a_rows > 0 restricts a (not transposed) to
  // rows [a_row0, a_row0 + a_rows), a panel of the output's rows; b_rows > 0 restricts b (transposed)
  // likewise, a panel of the output's columns.  Offsets are multiples of 8.
  int a_row0, a_rows, b_row0, b_rows;
};
// out = act(alpha * sum_p (+/-) op(a_p).op(b_p) + beta * out + bias (x) col_scale)
struct b200_fused_gemm {
  int npass;
  b200_pass pass[kMaxPass];
  float alpha, beta;
  cudamat* bias;       // M x 1 or null
  cudamat* col_scale;  // 1 x N or null
  int activation;      // 0 identity, 1 logistic
  cudamat* out;        // M x N or null
  cudamat* out_aux;    // aux matrix of the result, or null
  cudamat* sample;     // Bernoulli(result), or null
  cudamat* sample_aux; // aux matrix of the draw, or null
  // scaled half-precision operands (parts kPartF16Lo / kPartF16Hi): the terms carry a factor
  // 2^(*scale_exp + scale_exp_const) (scale_exp: 1 x 1 device matrix or null), divided out of alpha;
  // aux_f16 != 0: out_aux / sample_aux are written in that form with exponent aux_exp
  cudamat* scale_exp;
  int scale_exp_const;
  int aux_f16;
  int aux_exp;
};

extern "C" {

// 0 auto (by size and alignment), 1 the tcgen05 kernel only (ERROR_UNSUPPORTED where TMA cannot address an
// operand), 2 CUDA cores only, 3 the one-launch kernel only, 4 the
// tcgen05 kernel behind aligned copies of its operands only.
int b200_set_gemm_path(int path) {
  g_path = path;
  return 0;
}
// Precision of `dot`: 0 = fp32-grade (three TF32 terms over x and x - tf32(x)),
// 1 = one TF32 term (about 1e-3 relative).
int b200_set_dot_precision(int mode) {
  g_dot_mode = mode;
  return 0;
}

// hi = x with the low 13 mantissa bits cleared (optional, may be null), lo = x - hi.
int split_tf32(cudamat* x, cudamat* hi, cudamat* lo) {
  if (!x->on_device || (hi && !hi->on_device) || !lo->on_device) return ERROR_NOT_ON_DEVICE;
  if ((hi && !same_shape(x, hi)) || !same_shape(x, lo)) return ERROR_INCOMPATIBLE_DIMENSIONS;
  return launch_split(x->data_device, hi ? hi->data_device : nullptr, lo->data_device, numel(x));
}

// aux = the bfloat16 planes of x (see split_aux in common.cuh); aux holds aux_rows(rows) x cols floats.
int split_bf16(cudamat* x, cudamat* aux) {
  if (!x->on_device || !aux->on_device) return ERROR_NOT_ON_DEVICE;
  if (x->is_trans || aux->is_trans) return ERROR_TRANSPOSED;
  if (!aux_shape_ok(aux, x)) return ERROR_INCOMPATIBLE_DIMENSIONS;
  return launch_split_aux(x->data_device, aux->data_device, x->size[0], numel(x));
}

// aux = x in scaled half-precision form, scale 2^(*exp_dev + exp_const) (exp_dev: 1 x 1 device matrix or null).
int split_f16(cudamat* x, cudamat* aux, cudamat* exp_dev, int exp_const) {
  if (!x->on_device || !aux->on_device || (exp_dev && !exp_dev->on_device)) return ERROR_NOT_ON_DEVICE;
  if (x->is_trans || aux->is_trans) return ERROR_TRANSPOSED;
  if (!aux_shape_ok(aux, x)) return ERROR_INCOMPATIBLE_DIMENSIONS;
  const long n = numel(x);
  if (n == 0) return 0;
  const int rows = x->size[0];
  const bool vec = (rows % 4 == 0) && ((((uintptr_t)x->data_device) & 15) == 0);
  long blocks = ((vec ? n / 4 : n) + 255) / 256;
  if (blocks > (long)sm_count() * 8) blocks = (long)sm_count() * 8;
  if (blocks < 1) blocks = 1;
  if (launch_dependent(k_split_f16, dim3((unsigned)blocks), dim3(256), 0, stream(), x->data_device,
                       reinterpret_cast<uint16_t*>(aux->data_device), rows, aux_rows(rows), n, vec,
                       exp_dev ? exp_dev->data_device : nullptr, exp_const, nullptr) != cudaSuccess)
    return set_error(cudaGetErrorString(cudaGetLastError()));
  return check_launch();
}

// The same with add (M x N, or null) added to every output before the activation (beta 0, out given): what a layer gets from a
// neighbour that stands still is multiplied once.
int fused_gemm_add(rnd_struct* rnd_state, b200_fused_gemm* f, cudamat* add) {
  if (f->npass <= 0 || f->npass > kMaxPass) return ERROR_UNSUPPORTED;
  GemmProblem g;
  g.npass = f->npass;
  g.tf32_operands = 1;
  g.M = f->pass[0].a_rows > 0 ? f->pass[0].a_rows : lead(f->pass[0].a);
  g.N = f->pass[0].b_rows > 0 ? f->pass[0].b_rows : nonlead(f->pass[0].b);
  for (int q = 0; q < f->npass; q++) {
    const cudamat *a = f->pass[q].a, *b = f->pass[q].b;
    const b200_pass& ps = f->pass[q];
    if (!a->on_device || !b->on_device) return ERROR_NOT_ON_DEVICE;
    // a window selects rows of the stored matrix that run along M (a as stored) or N (b transposed)
    if (ps.a_rows > 0 && (a->is_trans || ps.a_row0 < 0 || (ps.a_row0 & 7) || ps.a_row0 + ps.a_rows > a->size[0])) return ERROR_UNSUPPORTED;
    if (ps.b_rows > 0 && (!b->is_trans || ps.b_row0 < 0 || (ps.b_row0 & 7) || ps.b_row0 + ps.b_rows > b->size[0])) return ERROR_UNSUPPORTED;
    const int m_q = ps.a_rows > 0 ? ps.a_rows : lead(a), n_q = ps.b_rows > 0 ? ps.b_rows : nonlead(b);
    if (m_q != g.M || n_q != g.N || nonlead(a) != lead(b)) return ERROR_INCOMPATIBLE_DIMENSIONS;
    const int pa = f->pass[q].a_part, pb = f->pass[q].b_part;
    if (pa < 0 || pa >= kNumParts || pb < 0 || pb >= kNumParts) return ERROR_UNSUPPORTED;
    // both operands of a term of one kind: fp32-wide, bfloat16, or scaled half precision (aux only)
    if (part_is_16bit(pa) != part_is_16bit(pb) || part_is_f16(pa) != part_is_f16(pb)) return ERROR_UNSUPPORTED;
    if (part_is_f16(pa) && (!f->pass[q].a_aux || !f->pass[q].b_aux)) return ERROR_UNSUPPORTED;
    const cudamat *xa = f->pass[q].a_aux, *xb = f->pass[q].b_aux;
    if ((xa && !aux_shape_ok(xa, a)) || (xb && !aux_shape_ok(xb, b))) return ERROR_INCOMPATIBLE_DIMENSIONS;
    g.pass[q].a = operand(a, pa, xa);
    g.pass[q].b = operand(b, pb, xb);
    if (ps.a_rows > 0) g.pass[q].a.row0 = ps.a_row0;
    if (ps.b_rows > 0) g.pass[q].b.row0 = ps.b_row0;
    g.pass[q].k = nonlead(a);
    g.pass[q].negate = f->pass[q].negate;
  }
  GemmEpilogue& e = g.epi;
  e.alpha = f->alpha;
  e.beta = f->beta;
  e.bias = nullptr;
  e.col_scale = nullptr;
  e.activation = f->activation;
  e.out = e.out_aux = e.sample = e.sample_aux = nullptr;
  e.ldo = g.M;
  e.ld_aux = aux_rows(g.M);
  e.aux_f16 = f->aux_f16;
  e.aux_exp = f->aux_exp;
  e.scale_exp = nullptr;
  e.scale_exp_const = f->scale_exp_const;
  if (f->scale_exp) {
    if (!f->scale_exp->on_device) return ERROR_NOT_ON_DEVICE;
    e.scale_exp = f->scale_exp->data_device;
  }
  e.col0 = rng_col0();
  cudamat* outs[4] = {f->out, f->out_aux, f->sample, f->sample_aux};
  for (int i = 0; i < 4; i++) {
    if (!outs[i]) continue;
    if (!outs[i]->on_device) return ERROR_NOT_ON_DEVICE;
    if (outs[i]->is_trans) return ERROR_TRANSPOSED;
    const int want_rows = (i & 1) ? e.ld_aux : g.M;   // aux handles hold the rounded-up rows
    if (outs[i]->size[0] != want_rows || outs[i]->size[1] != g.N) return ERROR_INCOMPATIBLE_DIMENSIONS;
  }
  if (f->out) e.out = f->out->data_device;
  if (f->out_aux) e.out_aux = f->out_aux->data_device;
  if (f->sample) e.sample = f->sample->data_device;
  if (f->sample_aux) e.sample_aux = f->sample_aux->data_device;
  if (e.beta != 0.0f && !e.out) return ERROR_UNSUPPORTED;
  if (add) {
    if (!add->on_device) return ERROR_NOT_ON_DEVICE;
    if (add->is_trans) return ERROR_TRANSPOSED;
    if (add->size[0] != g.M || add->size[1] != g.N) return ERROR_INCOMPATIBLE_DIMENSIONS;
    if (e.beta != 0.0f || !e.out) return ERROR_UNSUPPORTED;
    e.beta = 1.0f;
    if (add->data_device != e.out) g.prior = add->data_device;
  }
  if (f->bias) {
    if (!f->bias->on_device) return ERROR_NOT_ON_DEVICE;
    if (numel(f->bias) != g.M) return ERROR_INCOMPATIBLE_DIMENSIONS;
    e.bias = f->bias->data_device;
  }
  if (f->col_scale) {
    if (!f->col_scale->on_device) return ERROR_NOT_ON_DEVICE;
    if (numel(f->col_scale) != g.N || !f->bias) return ERROR_INCOMPATIBLE_DIMENSIONS;
    e.col_scale = f->col_scale->data_device;
  }
  e.key = make_philox_key(0, 0);
  if (f->sample || f->sample_aux) {
    if (!rnd_state) return ERROR_GENERIC;
    e.key = make_philox_key(rnd_state->seed, rnd_state->calls);
    rnd_state->calls += 1;
  }
  return run(g);
}
int fused_gemm(rnd_struct* rnd_state, b200_fused_gemm* f) { return fused_gemm_add(rnd_state, f, nullptr); }

// cudamat/cudamat.cu:1671-1696: target = beta * target + alpha * op(mat1) . op(mat2).
int dot(cudamat* mat1, cudamat* mat2, cudamat* target, float beta, float alpha) {
  if (!mat1->on_device || !mat2->on_device || !target->on_device) return ERROR_NOT_ON_DEVICE;
  if (lead(mat1) != lead(target) || nonlead(mat2) != nonlead(target) || nonlead(mat1) != lead(mat2))
    return ERROR_INCOMPATIBLE_DIMENSIONS;
  if (target->is_trans) return ERROR_TRANSPOSED;
  const int m = lead(mat1), k = lead(mat2), n = nonlead(mat2);
  GemmProblem g;
  g.M = m;
  g.N = n;
  g.tf32_operands = 0;  // on CUDA cores `dot` multiplies full fp32 operands
  GemmEpilogue& e = g.epi;
  e.alpha = alpha;
  e.beta = beta;
  e.bias = e.col_scale = nullptr;
  e.activation = 0;
  e.out = target->data_device;
  e.out_aux = e.sample = e.sample_aux = nullptr;
  e.ldo = m;
  e.ld_aux = aux_rows(m);
  e.aux_f16 = e.aux_exp = e.scale_exp_const = 0;
  e.scale_exp = nullptr;
  e.col0 = 0;
  e.key = make_philox_key(0, 0);
  g.npass = 1;
  g.pass[0].a = operand(mat1, kPartX);
  g.pass[0].b = operand(mat2, kPartX);
  g.pass[0].k = k;
  g.pass[0].negate = 0;
  if (m == 0 || n == 0) return 0;
  if (k == 0) {  // empty inner dimension: target = beta * target
    g.pass[0].k = 0;
    return gemm_simt(g);
  }
  // fp32-grade: x = tf32(x) + lo with lo = x - tf32(x); lo.x + x.lo + x.x, small terms first,
  // every term a TF32 product (the kernel derives lo from the staged tile of x).  The cheaper
  // bfloat16 correction terms are a few times less accurate (2^-18 against 2^-20 per term),
  // which shows when a caller subtracts two nearly equal products, as the positive and
  // negative statistics are.
  GemmProblem f = g;
  f.npass = 3;
  const int pa[3] = {kPartLo32, kPartX, kPartX}, pb[3] = {kPartX, kPartLo32, kPartX};
  for (int q = 0; q < 3; q++) {
    f.pass[q].a = operand(mat1, pa[q]);
    f.pass[q].b = operand(mat2, pb[q]);
    f.pass[q].k = k;
    f.pass[q].negate = 0;
  }
  f.tf32_operands = 1;
  if (g_path == 2) return gemm_simt(g);
  if (g_path == 4) return gemm_tc_packed(f);
  const bool tc = gemm_tc_supported(g);
  if (g_path == 1) return tc ? gemm_tc(g_dot_mode == 1 ? g : f) : ERROR_UNSUPPORTED;
  // Operands TMA cannot address and little work: fp32 multiply-adds of the full operands.
  if (!tc || (long)m * n * k < kTcMinWork) {
    if (g_path == 0 && !tc && k >= kPackedDotK && g_dot_mode != 1 && beta == 0.0f && small_depth(f) > kSmallDepth) {
      int r = gemm_tc_packed(f);
      if (r == 0) r = recompute_nonfinite(f);
      if (r != ERROR_UNSUPPORTED) return r;
    }
    const int r = gemm_small(f, kSmallFp32);
    return r != ERROR_UNSUPPORTED || g_path == 3 ? r : gemm_simt(g);
  }
  if (g_path == 3 || (g_dot_mode != 1 && small_beats_tc(f))) {
    const int r = gemm_small(f, kSmallIeee);
    if (r != ERROR_UNSUPPORTED || g_path == 3) return r;
  }
  return gemm_tc(g_dot_mode == 1 ? g : f);
}

// deepnet/dbm.py:242,254 + deepnet/parameter.py:80-106 in one pass over the parameter:
//   grad += suff * (-inv_batch); delta = momentum*delta + l2*w + l1*sign(w) + grad;
//   w -= eps * delta; grad = 0; and, when w_aux is given, the aux matrix of the new w: its
//   bfloat16 parts, or with w_scale (1 x 4 device matrix {exponent, the one a fresh start would take, max |w| bits, -}) its
//   scaled half-precision form, written in the same pass with the exponent carried so far; a
//   second pass rewrites it only when the new w no longer fits that exponent.
// grad may be null (treated as zero and not written).  20 bytes of traffic per element
// without grad and aux; +8 with grad, +4 with either aux (+8 more in an update that changes the exponent).
// The update restricted to columns [col0, col0 + ncols) of the parameter (and of delta, grad, suff,
// w_aux): the statistics of a data-parallel update arrive panel by panel (each after its own
// all-reduce) and every panel is updated as it arrives.  In scaled half-precision form all panels
// use the exponent carried so far; the check of that exponent against the new parameter (and, if it
// no longer fits, the rewrite of the whole aux) runs with the panel that ends at the last column.
int momentum_update_columns(cudamat* w, cudamat* delta, cudamat* grad, cudamat* suff, cudamat* w_aux, cudamat* w_scale,
                            int col0, int ncols, float inv_batch, float momentum, float eps, float l2, float l1) {
  if (!w->on_device || !delta->on_device || !suff->on_device) return ERROR_NOT_ON_DEVICE;
  if (!same_shape(w, delta) || !same_shape(w, suff)) return ERROR_INCOMPATIBLE_DIMENSIONS;
  if (grad && (!grad->on_device || !same_shape(w, grad))) return ERROR_INCOMPATIBLE_DIMENSIONS;
  if (w_aux && (w->is_trans || !aux_shape_ok(w_aux, w))) return ERROR_INCOMPATIBLE_DIMENSIONS;
  if (w_scale && (!w_aux || !w_scale->on_device || numel(w_scale) < 4)) return ERROR_INCOMPATIBLE_DIMENSIONS;
  if (w->is_trans && !(col0 == 0 && ncols == w->size[1])) return ERROR_TRANSPOSED;
  if (col0 < 0 || ncols < 0 || col0 + ncols > w->size[1]) return ERROR_INCOMPATIBLE_DIMENSIONS;
  const int rows = w->size[0];
  const long n = (long)rows * ncols, first = (long)rows * col0;
  const bool last_panel = col0 + ncols == w->size[1];
  float* sp = w_scale ? w_scale->data_device : nullptr;
  uint16_t* ap = w_aux ? reinterpret_cast<uint16_t*>(w_aux->data_device) : nullptr;
  const int mode = !w_aux ? 0 : (w_scale ? 2 : 1);
  const int lda = aux_rows(rows);
  if (n > 0) {
    float *wp = w->data_device + first, *dp = delta->data_device + first, *gp = grad ? grad->data_device + first : nullptr;
    const float* sfp = suff->data_device + first;
    uint16_t* app = ap ? ap + (long)col0 * 2 * lda : nullptr;
    uintptr_t bits = (uintptr_t)wp | (uintptr_t)dp | (uintptr_t)sfp;
    if (gp) bits |= (uintptr_t)gp;
    if (app) bits |= (uintptr_t)app;
    const bool vec = (bits & 15) == 0 && n % 4 == 0 && (!w_aux || rows % 4 == 0);
    long blocks = ((vec ? n / 4 : n) + 255) / 256;
    if (blocks > (long)sm_count() * 8) blocks = (long)sm_count() * 8;
    if (blocks < 1) blocks = 1;
#define LAUNCH_UPDATE(G, A)                                                                                          \
  (void)launch_dependent(k_update<G, A>, dim3((unsigned)blocks), dim3(256), 0, stream(), wp, dp, gp, sfp, app, sp, rows, lda, n, \
                         vec, -inv_batch, momentum, -eps, l2, l1)
    if (grad) {
      if (mode == 2) LAUNCH_UPDATE(true, 2);
      else if (mode == 1) LAUNCH_UPDATE(true, 1);
      else LAUNCH_UPDATE(true, 0);
    } else {
      if (mode == 2) LAUNCH_UPDATE(false, 2);
      else if (mode == 1) LAUNCH_UPDATE(false, 1);
      else LAUNCH_UPDATE(false, 0);
    }
#undef LAUNCH_UPDATE
    const int err = check_launch();
    if (err) return err;
  }
  if (mode != 2 || !last_panel) return 0;
  (void)launch_dependent(k_update_scale, dim3(1), dim3(1), 0, stream(), sp);
  int err = check_launch();
  if (err) return err;
  const long total = numel(w);
  if (total == 0) return 0;
  const bool svec = (rows % 4 == 0) && ((((uintptr_t)w->data_device) & 15) == 0);
  long sblocks = ((svec ? total / 4 : total) + 255) / 256;
  if (sblocks > (long)sm_count() * 8) sblocks = (long)sm_count() * 8;
  if (sblocks < 1) sblocks = 1;
  // (returns at once unless the exponent had to change)
  (void)launch_dependent(k_split_f16, dim3((unsigned)sblocks), dim3(256), 0, stream(), w->data_device, ap, rows, lda, total, svec,
                         sp, 0, sp + 3);
  return check_launch();
}

int momentum_update(cudamat* w, cudamat* delta, cudamat* grad, cudamat* suff, cudamat* w_aux, cudamat* w_scale,
                    float inv_batch, float momentum, float eps, float l2, float l1) {
  return momentum_update_columns(w, delta, grad, suff, w_aux, w_scale, 0, w->size[1], inv_batch, momentum, eps, l2, l1);
}

// bias_updates and momentum_update of a weight matrix with its bfloat16 parts, in one launch where the biases take one; with
// w_scale its scaled half-precision form (see momentum_update).
int update_all_scaled(b200_bias_layers* t, cudamat* w, cudamat* delta, cudamat* suff, cudamat* w_aux, cudamat* w_scale,
                      float inv_batch, float mom_b, float eps_b, float mom_w, float eps_w, float l2, float l1) {
  if (!w->on_device || !delta->on_device || !suff->on_device || !w_aux->on_device) return ERROR_NOT_ON_DEVICE;
  if (w->is_trans || delta->is_trans || suff->is_trans) return ERROR_TRANSPOSED;
  if (!same_shape(w, delta) || !same_shape(w, suff) || !aux_shape_ok(w_aux, w)) return ERROR_INCOMPATIBLE_DIMENSIONS;
  if (w_scale && !w_scale->on_device) return ERROR_NOT_ON_DEVICE;
  if (w_scale && numel(w_scale) < 4) return ERROR_INCOMPATIBLE_DIMENSIONS;
  TailArgs a;
  int tail = 0;
  int err = plan_bias_tail(t, inv_batch, mom_b, eps_b, a, tail);
  if (err) return err;
  const long n = numel(w);
  if (tail == 0 || n == 0) {
    err = bias_updates(t, inv_batch, mom_b, eps_b);
    return err ? err : momentum_update(w, delta, nullptr, suff, w_aux, w_scale, inv_batch, mom_w, eps_w, l2, l1);
  }
  UpdateArgs u = {w->data_device, delta->data_device, suff->data_device, reinterpret_cast<uint16_t*>(w_aux->data_device),
                  w->size[0], aux_rows(w->size[0]), n, false, -inv_batch, mom_w, -eps_w, l2, l1,
                  w_scale ? w_scale->data_device : nullptr, nullptr};
  if (w_scale) {
    unsigned* const counters = (unsigned*)workspace_zeroed(3, 4096 * sizeof(unsigned));
    if (!counters) return CUDA_ERROR;
    u.done = counters + 1;                     // (the first one is the squared error's)
  }
  u.vec = (((uintptr_t)u.w | (uintptr_t)u.delta | (uintptr_t)u.suff | (uintptr_t)u.w_aux) & 15) == 0 && u.rows % 4 == 0;
  long blocks = ((u.vec ? n / 4 : n) + 255) / 256;
  if (blocks > (long)sm_count() * 8) blocks = (long)sm_count() * 8;
  if (launch_dependent(w_scale ? k_update_all<2> : k_update_all<1>, dim3((unsigned)(tail + blocks)), dim3(256), 0, stream(), a, u,
                       tail) != cudaSuccess)
    return set_error(cudaGetErrorString(cudaGetLastError()));
  err = check_launch();
  return err || !w_scale || n <= kRedoByOneBlock ? err : rewrite_f16_planes_if(u.w, u.w_aux, u.rows, n, u.scale, u.scale + 3);
}
int update_all(b200_bias_layers* t, cudamat* w, cudamat* delta, cudamat* suff, cudamat* w_aux, float inv_batch, float mom_b,
               float eps_b, float mom_w, float eps_w, float l2, float l1) {
  return update_all_scaled(t, w, delta, suff, w_aux, nullptr, inv_batch, mom_b, eps_b, mom_w, eps_w, l2, l1);
}

}  // extern "C"

namespace {

__device__ __forceinline__ float log_1_plus_exp(float x) { return x > 0 ? x + log1pf(expf(-x)) : log1pf(expf(x)); }

// What an annealing step does between its two products (deepnet/ais.py:156-166), one block per chain: with x the
// hidden pre-activations W'v + a,
//   w += sum_j [log(1 + exp(s x_j)) - log(1 + exp(s0 x_j))] + ds b'v,   h ~ Bernoulli(sigmoid(s x))
// and, by the first block, the visible bias of the next product, s b.  Nine calls of the matrix API otherwise.
// Latency bound (500 x 100: 200 KB).
__global__ void __launch_bounds__(256) k_ais_hidden(const float* x, const float* b, const float* v, float* w, float* h,
                                                    float* sb, int H, int V, int col0, float s0, float s, float ds,
                                                    PhiloxKey key) {
  __shared__ float red[2][8];
  grid_dependents_launch();
  grid_dependency_wait();
  const int c = blockIdx.x, gc = c + col0;
  float gain = 0.0f, bv = 0.0f;
  for (int j = threadIdx.x; j < H; j += 256) {
    const float t = x[(long)c * H + j], ts = t * s;
    gain += log_1_plus_exp(ts) - log_1_plus_exp(t * s0);
    const uint4 r = philox4x32_10((uint32_t)j, (uint32_t)(gc >> 2), key);
    h[(long)c * H + j] = word_to_uniform(pick_word(r, gc & 3)) < sigmoid_accurate(ts) ? 1.0f : 0.0f;
  }
  for (int i = threadIdx.x; i < V; i += 256) {
    bv = fmaf(b[i], v[(long)c * V + i], bv);
    if (c == 0) sb[i] = s * b[i];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    gain += __shfl_xor_sync(0xffffffffu, gain, o);
    bv += __shfl_xor_sync(0xffffffffu, bv, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = gain;
    red[1][threadIdx.x >> 5] = bv;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; i++) {
      gain += red[0][i];
      bv += red[1][i];
    }
    w[c] = (w[c] + gain) + ds * bv;
  }
}

}  // namespace

// The annealing steps 1 .. n - 1 of `schedule` for a binary RBM (deepnet/ais.py:152-170), in one launch where that is
// faster (chains.cu), else three launches a step, issued from here: w V x H (w_aux its bfloat16 parts), a H x 1, b V x 1, v_state / v_sample V x B, h_pre / h_sample H x B,
// sb V x 1 scratch, weights 1 x B (added to).  Two sampling calls a step, in the order of the reference's calls.
extern "C" int ais_binary_steps(rnd_struct* rnd_state, cudamat* w, cudamat* w_aux, cudamat* a, cudamat* b, cudamat* v_state,
                                cudamat* v_sample, cudamat* h_pre, cudamat* h_sample, cudamat* sb, cudamat* weights,
                                const double* schedule, int n) {
  if (!rnd_state || !schedule) return ERROR_GENERIC;
  cudamat* all[10] = {w, w_aux, a, b, v_state, v_sample, h_pre, h_sample, sb, weights};
  for (int i = 0; i < 10; i++) {
    if (!all[i]->on_device) return ERROR_NOT_ON_DEVICE;
    if (all[i]->is_trans) return ERROR_TRANSPOSED;
  }
  const int V = w->size[0], H = w->size[1], B = v_state->size[1];
  if (!aux_shape_ok(w_aux, w) || numel(a) != H || numel(b) != V || numel(sb) != V || numel(weights) != B ||
      v_state->size[0] != V || !same_shape(v_state, v_sample) || h_pre->size[0] != H || h_pre->size[1] != B ||
      !same_shape(h_pre, h_sample))
    return ERROR_INCOMPATIBLE_DIMENSIONS;
  if ((long)V * H * B == 0) return 0;
  if (g_path == 0) {
    const AisChains c = {w->data_device, a->data_device, b->data_device, v_state->data_device, v_sample->data_device,
                         h_pre->data_device, h_sample->data_device, sb->data_device, weights->data_device,
                         V, H, B, schedule, n, rnd_state->seed, rnd_state->calls};
    const int err = ais_chains(c);
    if (err == 0) rnd_state->calls += 2ull * (n - 1);
    if (err != ERROR_UNSUPPORTED) return err;
  }
  cudamat wt = *w;
  wt.is_trans = 1;
  b200_fused_gemm up = {}, down = {};
  // the samples are exact: lo16(w) . b16(x) and w . x
  auto product = [](b200_fused_gemm& f, cudamat* m, cudamat* aux, cudamat* x) {
    f.npass = 2;
    f.alpha = 1.0f;
    for (int q = 0; q < 2; q++) {
      f.pass[q].a = m;
      f.pass[q].b = x;
      f.pass[q].a_aux = aux;
      f.pass[q].a_part = q ? kPartX : kPartLo16;
      f.pass[q].b_part = q ? kPartX : kPartB16;
    }
  };
  product(up, &wt, w_aux, v_sample);
  up.bias = a;
  up.out = h_pre;
  product(down, w, w_aux, h_sample);
  down.bias = sb;
  down.activation = 1;
  down.out = v_state;
  down.sample = v_sample;
  for (int i = 1; i < n; i++) {
    int err = fused_gemm(rnd_state, &up);
    if (err) return err;
    const float s0 = (float)schedule[i - 1], s = (float)schedule[i];
    const PhiloxKey key = make_philox_key(rnd_state->seed, rnd_state->calls++);
    if (launch_dependent(k_ais_hidden, dim3((unsigned)B), dim3(256), 0, stream(), h_pre->data_device, b->data_device,
                         v_state->data_device, weights->data_device, h_sample->data_device, sb->data_device, H, V, rng_col0(),
                         s0, s, (float)(schedule[i] - schedule[i - 1]), key) != cudaSuccess)
      return set_error(cudaGetErrorString(cudaGetLastError()));
    down.alpha = s;
    err = fused_gemm(rnd_state, &down);
    if (err) return err;
  }
  return check_launch();
}
