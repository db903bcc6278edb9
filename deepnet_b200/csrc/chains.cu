// All steps of annealed importance sampling of a binary RBM in one launch.
//
// Given W the chains never meet, so nothing but W has to be shared between them.  A cluster of thread blocks takes a few
// chains through ALL of their steps; a block owns a share of the columns of W (of the hidden units):
//   up    x_j = sum_i W_ij v_i for its own j: whole sums, from the full visible states every block holds;
//   down  partial sums over its own j of W_ij h_j for every i, left in its shared memory; after a cluster barrier the block
//         that owns unit i adds the blocks' sums through distributed shared memory, in rank order (the same bits every run),
//         finishes its units and stores their states into every block's copy.
// Two cluster barriers a step, no launch, no grid-wide wait, and W read from L2 once per cluster; the columns that do not
// fit in shared memory are read from L2 in every step.
//
// Products run on mma.sync bfloat16 with W in three parts of eight bits, w = h + m + l exactly (made in registers from
// the fp32 value, by truncation); the states are 0 or 1, so that h.s + m.s + l.s are exact products.  The tensor core's
// accumulator, which truncates, is added to an fp32 register after 32 of K.  tcgen05 has no use here: 8 or 16 chains a
// cluster are the short side of every product.  mma.sync bfloat16 multiplies 1024 pairs a clock and SM (TF32 512, fp32
// multiply-adds 128).  States a caller starts from may be anything: where bfloat16 does not hold them the first product is
// taken in doubles.
// Bound by instruction issue (the split of W) and the latency of the exchange.  784 x 500, 100 chains, clocks of a step:
// up 4850, hidden units 3200, down 6140, visible units 3900, barriers 2000: 10.5 us, against 25 as two products and a
// kernel between them (three launches; 36 with the products as they were).  The steps are a millisecond of a call of
// `ais_binary_rbm` with a hundred of them; the rest is the caller's set-up.
#include <cmath>
#include <initializer_list>
#include <type_traits>

#include "gemm.cuh"

namespace b200 {

namespace {

constexpr int kChainThreads = 512, kChainWarps = kChainThreads / 32;
constexpr int kChainSmem = 222 * 1024;      // (the rest: what the kernel declares itself)

__device__ __forceinline__ void chain_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t chain_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t chain_peer(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float2 ld_peer2(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void st_peer(uint32_t addr, uint2 v) {
  asm volatile("st.shared::cluster.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(v.x), "r"(v.y) : "memory");
}
__device__ __forceinline__ void st_peer(uint32_t addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ uint32_t chain_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint2 b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y));
}
// x = h + m + l exactly, eight bits each (truncation: a finite value has finite parts); two values to a register, the first in
// the low half.
__device__ __forceinline__ void split3(float x, float y, uint32_t& h, uint32_t& m, uint32_t& l) {
  const uint32_t xh = __float_as_uint(x), yh = __float_as_uint(y);
  const float xr = x - __uint_as_float(xh & 0xffff0000u), yr = y - __uint_as_float(yh & 0xffff0000u);
  const uint32_t xm = __float_as_uint(xr), ym = __float_as_uint(yr);
  const float xl = xr - __uint_as_float(xm & 0xffff0000u), yl = yr - __uint_as_float(ym & 0xffff0000u);
  h = __byte_perm(xh, yh, 0x7632);
  m = __byte_perm(xm, ym, 0x7632);
  l = __byte_perm(__float_as_uint(xl), __float_as_uint(yl), 0x7632);
}

inline __host__ __device__ int chain_pad(int n, int to) { return (n + to - 1) / to * to; }

// How the chains of a call are spread out.
struct ChainSpread {
  int blocks, clusters;    // blocks of a cluster, clusters
  int resident;            // columns of W a block keeps in shared memory
  int B, col0;             // chains, first global column (random stream)
};

// The block's place among the others, and its chains.
struct ChainCluster {
  int rank, blocks;
  int c0, n;                       // first chain, chains of the cluster

  __device__ __forceinline__ void set_up(const ChainSpread& s) {
    rank = (int)chain_rank();
    blocks = s.blocks;
    const int cl = (int)blockIdx.x / blocks;
    c0 = (int)((long)s.B * cl / s.clusters);
    n = (int)((long)s.B * (cl + 1) / s.clusters) - c0;
  }
};

// 0/1 states of up to N chains over K units as bfloat16, [chain][row]; rows 32 or 96 bytes apart modulo 128, so that a
// warp's reads of eight chains x 32 bytes meet no bank conflict.
template <int N>
struct ChainStates {
  uint16_t* p;
  int row;
  static inline __host__ __device__ int row_of(int K) { return chain_pad(K, 32) + 16; }
  static inline __host__ __device__ int floats(int K) { return N * row_of(K) / 2; }
  __device__ __forceinline__ void set_up(float* at, int K) {
    p = reinterpret_cast<uint16_t*>(at);
    row = row_of(K);
  }
  __device__ __forceinline__ uint16_t* at(int chain, int k) const { return p + chain * row + k; }
  __device__ __forceinline__ void put(int chain, int k, float x) const { *at(chain, k) = x != 0.0f ? 0x3f80 : 0; }
  __device__ __forceinline__ void clear() const {
    uint32_t* w = reinterpret_cast<uint32_t*>(p);
    for (int i = threadIdx.x; i < N * row / 2; i += kChainThreads) w[i] = 0u;
  }
  // the states of chains [0, n) from columns of K units, eight loads in flight per thread; true where a thread met one that
  // bfloat16 does not hold
  __device__ __forceinline__ bool load(const float* x, int n, int K) const {
    const int items = n * K;
    bool rounded = false;
    for (int i0 = threadIdx.x; i0 < items; i0 += 8 * kChainThreads) {
      float y[8];
#pragma unroll
      for (int u = 0; u < 8; u++) y[u] = i0 + u * kChainThreads < items ? x[i0 + u * kChainThreads] : 0.0f;
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int i = i0 + u * kChainThreads, c = i / K;
        if (i < items) {
          const uint16_t b = float_to_bf16(y[u]);
          *at(c, i - c * K) = b;
          rounded |= !(bf16_to_float(b) == y[u]);
        }
      }
    }
    return rounded;
  }
  // units [4 q0, 4 (q0 + nq)) of n chains from this block's copy into the others'
  __device__ __forceinline__ void share(const ChainCluster& k, int n, int q0, int nq) const {
    for (int it = threadIdx.x; it < n * nq; it += kChainThreads) {
      const int c = it / nq, q = it - c * nq;
      const uint16_t* from = at(c, 4 * (q0 + q));
      const uint2 v = *reinterpret_cast<const uint2*>(from);
      const uint32_t a = chain_addr(from);
#pragma unroll 8
      for (int r = 0; r < k.blocks; r++)
        if (r != k.rank) st_peer(chain_peer(a, r), v);
    }
  }
};
// The order of a down product's K: a lane's four units of sixteen, which are four apart, lie side by side.
__device__ __forceinline__ int down_order(int j) { return (j & ~15) | ((j & 3) << 2) | ((j >> 2) & 3); }

// The block's columns [j0, j0 + nj) of a matrix W of V rows, the first R of them in shared memory: column j at j Vs, its
// 16-byte chunk q at q ^ swizzle(j), which keeps the reads of both products free of bank conflicts.
template <int NT>
struct ChainShare {
  static constexpr int N = 8 * NT, NS = N + 1;
  float* sw;
  const float* gw;         // first own column in global memory
  int V, Vs, nj, j0, R;
  int tiles, split;        // of the up product: 16 columns each, parts of the rows

  static inline __host__ __device__ int column(int V) { return chain_pad(V, 32); }
  // floats of the up product's sums
  static inline __host__ __device__ int sums(int cols) {
    const int tiles = (cols + 15) / 16;
    return chain_pad((tiles > kChainWarps ? tiles : kChainWarps) * 16 * NS, 4);
  }
  __device__ __forceinline__ static int swizzle(int j) { return ((j & 1) << 2) | (j & 2); }

  __device__ __forceinline__ void set_up(const float* w, int V_, int first, int count, int resident, float* smem) {
    V = V_;
    Vs = column(V);
    j0 = first;
    nj = count;
    R = resident < nj ? resident : nj;
    gw = w + (long)j0 * V;
    sw = smem;
    tiles = (nj + 15) >> 4;
    split = tiles == 0 ? 1 : min(max(kChainWarps / tiles, 1), Vs >> 5);
  }
  // copies the resident columns (zero below the last row and, where all are resident, up to whole tiles of columns); a wait and
  // a barrier follow
  template <bool kVec>
  __device__ __forceinline__ void load() const {
    const uint32_t dst = chain_addr(sw);
    const int chunks = Vs >> 2, filled = (R + 15) & ~15;
    for (int c = threadIdx.x >> 5; c < filled; c += kChainWarps) {
      const float* col = gw + (long)min(c, R - 1) * V;
      for (int q = threadIdx.x & 31; q < chunks; q += 32) {
        const uint32_t at = dst + 4u * (uint32_t)(c * Vs + 4 * (q ^ swizzle(c)));
        if (kVec) {
          const bool in = 4 * q < V && c < R;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(in ? col + 4 * q : col), "r"(in ? 16 : 0) : "memory");
        } else {
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const bool in = 4 * q + i < V && c < R;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(at + 4u * i), "l"(in ? col + 4 * q + i : col), "r"(in ? 4 : 0) : "memory");
          }
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // four rows from i on of a column in global memory (rows past the last: zero)
  template <bool kVec>
  __device__ __forceinline__ float4 rows(const float* col, int i) const {
    if (kVec) return i < V ? __ldg(reinterpret_cast<const float4*>(col + i)) : make_float4(0, 0, 0, 0);
    float4 x;
    x.x = i < V ? __ldg(col + i) : 0.0f;
    x.y = i + 1 < V ? __ldg(col + i + 1) : 0.0f;
    x.z = i + 2 < V ? __ldg(col + i + 2) : 0.0f;
    x.w = i + 3 < V ? __ldg(col + i + 3) : 0.0f;
    return x;
  }

  template <bool kVec, bool kShared>
  __device__ __forceinline__ void up_tile(const ChainStates<N>& v, int tile, int kb0, int kb1, float (&acc)[NT][4]) const {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    // (columns past the last: the last one in global memory, zeros in shared memory; their sums are not read)
    const int ja = 16 * tile + g, f = swizzle(ja);
    const float* const wa = kShared ? sw + ja * Vs : gw + (long)min(ja, nj - 1) * V;
    const float* const wb = kShared ? wa + 8 * Vs : gw + (long)min(ja + 8, nj - 1) * V;
    const uint16_t* const vs = v.at(g, 4 * t);
    float4 x[2][2], ahead[2][2];      // [k16 step][row g, row g + 8]; from global memory one block of rows ahead
    auto fetch = [&](int kb, float4 (&y)[2][2]) {
#pragma unroll
      for (int s = 0; s < 2; s++) {
        if (kShared) {
          const int at = 32 * kb + 4 * ((4 * s + t) ^ f);
          y[s][0] = *reinterpret_cast<const float4*>(wa + at);
          y[s][1] = *reinterpret_cast<const float4*>(wb + at);
        } else {
          y[s][0] = rows<kVec>(wa, 32 * kb + 16 * s + 4 * t);
          y[s][1] = rows<kVec>(wb, 32 * kb + 16 * s + 4 * t);
        }
      }
    };
    if (!kShared && kb0 < kb1) fetch(kb0, ahead);
#pragma unroll 1
    for (int kb = kb0; kb < kb1; kb++) {
      if (kShared) {
        fetch(kb, x);
      } else {
#pragma unroll
        for (int s = 0; s < 2; s++) {
          x[s][0] = ahead[s][0];
          x[s][1] = ahead[s][1];
        }
        if (kb + 1 < kb1) fetch(kb + 1, ahead);
      }
      float d[NT][4] = {};
#pragma unroll
      for (int s = 0; s < 2; s++) {
        uint32_t h[4], m[4], l[4];
        split3(x[s][0].x, x[s][0].y, h[0], m[0], l[0]);
        split3(x[s][1].x, x[s][1].y, h[1], m[1], l[1]);
        split3(x[s][0].z, x[s][0].w, h[2], m[2], l[2]);
        split3(x[s][1].z, x[s][1].w, h[3], m[3], l[3]);
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {   // small terms first
          const uint2 b = *reinterpret_cast<const uint2*>(vs + 8 * nt * v.row + 32 * kb + 16 * s);
          mma_bf16(d[nt], l, b);
          mma_bf16(d[nt], m, b);
          mma_bf16(d[nt], h, b);
        }
      }
#pragma unroll
      for (int nt = 0; nt < NT; nt++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[nt][i] += d[nt][i];
    }
  }
  // W'v of the own columns.  sum[(s tiles 16 + j) NS + chain]: over the s-th part of the rows.  The caller synchronises before
  // and after.
  template <bool kVec>
  __device__ __forceinline__ void up(const ChainStates<N>& v, float* sum) const {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, blocks_k = Vs >> 5;
    for (int u = threadIdx.x >> 5; u < tiles * split; u += kChainWarps) {
      const int tile = u % tiles, s = u / tiles;
      const int kb0 = blocks_k * s / split, kb1 = blocks_k * (s + 1) / split;
      float acc[NT][4] = {};
      if (min(16 * tile + 16, nj) <= R) up_tile<kVec, true>(v, tile, kb0, kb1, acc);
      else up_tile<kVec, false>(v, tile, kb0, kb1, acc);
      float* to = sum + ((s * tiles + tile) * 16 + g) * NS + 2 * t;
#pragma unroll
      for (int nt = 0; nt < NT; nt++) {
        to[8 * nt] = acc[nt][0];
        to[8 * nt + 1] = acc[nt][1];
        to[8 * nt + 8 * NS] = acc[nt][2];
        to[8 * nt + 8 * NS + 1] = acc[nt][3];
      }
    }
  }
  __device__ __forceinline__ float up_sum(const float* sum, int j, int c) const {
    float x = 0.0f;
    for (int s = 0; s < split; s++) x += sum[(s * tiles * 16 + j) * NS + c];
    return x;
  }

  // The same sums from states v (chains V apart) that bfloat16 does not hold, whole and in doubles: what a caller may start
  // from, once a launch.
  __device__ __forceinline__ void up_exact(const float* v, int n, float* sum) const {
    sums_in_doubles(gw, v, sum, V, nj, n, split, tiles * 16 * NS);
  }
  static __device__ __noinline__ void sums_in_doubles(const float* w, const float* v, float* sum, int V, int nj, int n, int split,
                                                      int part) {
    for (int it = threadIdx.x; it < nj * n; it += kChainThreads) {
      const int c = it / nj, j = it - c * nj;
      double x = 0.0;
      for (int i = 0; i < V; i++) x += (double)w[(long)j * V + i] * v[(long)c * V + i];
      for (int s = 0; s < split; s++) sum[s * part + j * NS + c] = s ? 0.0f : (float)x;
    }
  }

  template <bool kVec, bool kShared>
  __device__ __forceinline__ void down_steps(const ChainStates<N>& hs, int unit, int ks0, int ks1, float (&acc)[2][NT][4]) const {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const float* const w = kShared ? sw + t * Vs + 32 * unit + 4 * (g ^ swizzle(t)) : gw;
    const uint16_t* const hs0 = hs.at(g, 4 * t);
#pragma unroll 1
    for (int k0 = ks0; k0 < ks1; k0 += 2) {
      float d[2][NT][4] = {};
#pragma unroll
      for (int s = 0; s < 2; s++) {
        if (k0 + s >= ks1) break;
        float4 x[4];
#pragma unroll
        for (int r = 0; r < 4; r++) {   // (columns past the last: their states are zero)
          const int j = 16 * (k0 + s) + 4 * r;
          x[r] = kShared ? *reinterpret_cast<const float4*>(w + j * Vs) : rows<kVec>(w + (long)min(j + t, nj - 1) * V, 32 * unit + 4 * g);
        }
        uint2 b[NT];
#pragma unroll
        for (int nt = 0; nt < NT; nt++) b[nt] = *reinterpret_cast<const uint2*>(hs0 + 8 * nt * hs.row + 16 * (k0 + s));
#pragma unroll
        for (int a = 0; a < 2; a++) {   // rows 4g, 4g + 1 of the unit's 32, then 4g + 2, 4g + 3
          uint32_t h[4], m[4], l[4];
          split3(a ? x[0].z : x[0].x, a ? x[1].z : x[1].x, h[0], m[0], l[0]);
          split3(a ? x[0].w : x[0].y, a ? x[1].w : x[1].y, h[1], m[1], l[1]);
          split3(a ? x[2].z : x[2].x, a ? x[3].z : x[3].x, h[2], m[2], l[2]);
          split3(a ? x[2].w : x[2].y, a ? x[3].w : x[3].y, h[3], m[3], l[3]);
#pragma unroll
          for (int nt = 0; nt < NT; nt++) {
            mma_bf16(d[a][nt], l, b[nt]);
            mma_bf16(d[a][nt], m, b[nt]);
            mma_bf16(d[a][nt], h, b[nt]);
          }
        }
      }
#pragma unroll
      for (int a = 0; a < 2; a++)
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
          for (int i = 0; i < 4; i++) acc[a][nt][i] += d[a][nt][i];
    }
  }
  // W h over the own columns, h in down_order: partial sums of every quad of rows, part[quad (N + 1) + chain].
  template <bool kVec>
  __device__ __forceinline__ void down(const ChainStates<N>& hs, float4* part) const {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int steps = (nj + 15) >> 4, in_smem = R == nj ? steps : R >> 4;
    for (int u = threadIdx.x >> 5; u < (Vs >> 5); u += kChainWarps) {
      float acc[2][NT][4] = {};
      down_steps<kVec, true>(hs, u, 0, in_smem, acc);
      if (in_smem < steps) down_steps<kVec, false>(hs, u, in_smem, steps, acc);
      float4* const to = part + (8 * u + g) * (N + 1) + 2 * t;
#pragma unroll
      for (int nt = 0; nt < NT; nt++) {
        to[8 * nt] = make_float4(acc[0][nt][0], acc[0][nt][2], acc[1][nt][0], acc[1][nt][2]);
        to[8 * nt + 1] = make_float4(acc[0][nt][1], acc[0][nt][3], acc[1][nt][1], acc[1][nt][3]);
      }
    }
  }
};

// The visible layer, whose units the blocks share out by quads: the block's own quads, and the partial sums of all.
template <int NT>
struct ChainLayer {
  static constexpr int N = 8 * NT;
  int V, q0, nq;
  float4* part;            // [quad][N + 1]
  static inline __host__ __device__ int per_block(int V, int blocks) { return ((V + 3) / 4 + blocks - 1) / blocks; }
  static inline __host__ __device__ int floats(int V) { return chain_pad(V, 32) * (N + 1); }
  __device__ __forceinline__ void set_up(const ChainCluster& k, int V_, float* at) {
    V = V_;
    const int per = per_block(V, k.blocks), quads = (V + 3) / 4;
    q0 = min(k.rank * per, quads);
    nq = min(quads, q0 + per) - q0;
    part = reinterpret_cast<float4*>(at);
  }
  // f(item, chain, unit, x, y): units (unit even) and unit + 1, of which the second may lie past the last; x, y: the sums of
  // all blocks (with_sums), in rank order.  A thread gets the same items every time.
  template <typename F>
  __device__ __forceinline__ void each(const ChainCluster& k, bool with_sums, F f) const {
    for (int it = threadIdx.x; it < 2 * nq * k.n; it += kChainThreads) {
      const int half = it & 1, c = (it >> 1) % k.n, q = q0 + (it >> 1) / k.n, unit = 4 * q + 2 * half;
      if (unit >= V) continue;
      float x = 0.0f, y = 0.0f;
      if (with_sums) {
        const uint32_t from = chain_addr(reinterpret_cast<const float2*>(part + q * (N + 1) + c) + half);
#pragma unroll 1
        for (int r0 = 0; r0 < k.blocks; r0 += 8) {     // (clusters have 8 or 16 blocks)
          float2 p[8];
#pragma unroll
          for (int r = 0; r < 8; r++) p[r] = ld_peer2(chain_peer(from, r0 + r));
#pragma unroll
          for (int r = 0; r < 8; r++) {
            x += p[r].x;
            y += p[r].y;
          }
        }
      }
      f(it, c, unit, x, y);
    }
  }
};

__device__ __forceinline__ float draw_of(int row, int col, const PhiloxKey& key, float p) {
  return word_to_uniform(pick_word(philox4x32_10((uint32_t)row, (uint32_t)(col >> 2), key), col & 3)) < p ? 1.0f : 0.0f;
}
__device__ __forceinline__ float log_1_plus_exp(float x) { return fmaxf(x, 0.0f) + log1pf(expf(-fabsf(x))); }

constexpr int kAisBatch = 256;      // inverse temperatures that travel with a launch
struct AisArgs {
  ChainSpread s;
  AisChains a;
  unsigned long long call0;
  int steps;
  float beta[kAisBatch + 1];     // beta[0]: of the step before the first
  float dbeta[kAisBatch];
};

// Shared memory: the log weights' terms (doubles: per hidden unit and per pair of visible units), visible states, hidden
// states, the visible layer's partial sums, the up product's sums, hidden biases, the share of W.
template <int NT>
struct AisShared {
  static constexpr int N = 8 * NT;
  int gains, v, h, part, sum, bh, w;      // offsets in floats; w: the end of the rest
  inline __host__ __device__ AisShared(int V, int H, int blocks) {
    const int cols = (H + blocks - 1) / blocks;
    gains = 0;
    v = gains + chain_pad(2 * N * (cols + 2 * ChainLayer<NT>::per_block(V, blocks)), 4);
    h = v + ChainStates<N>::floats(V);
    part = h + ChainStates<N>::floats(cols);
    sum = part + ChainLayer<NT>::floats(V);
    bh = sum + ChainShare<NT>::sums(cols);
    w = bh + chain_pad(cols, 4);
  }
};

// The annealing steps of deepnet/ais.py:152-170 at the temperatures beta[1 .. steps].  The log weights' terms are kept per
// unit in doubles and summed once, at the end.
template <int NT, bool kVec>
__global__ void __launch_bounds__(kChainThreads, 1) k_ais_chains(const __grid_constant__ AisArgs args) {
  extern __shared__ float4 chain_smem[];
  constexpr int N = 8 * NT;
  __shared__ double total[16][N];        // by rank: the block's share of every chain's log weight, in the leader
  float* const smem = reinterpret_cast<float*>(chain_smem);
  const AisChains& p = args.a;
  const int V = p.V, H = p.H;
  const AisShared<NT> at(V, H, args.s.blocks);
  ChainCluster k;
  k.set_up(args.s);
  const int j0 = (int)((long)H * k.rank / k.blocks), nj = (int)((long)H * (k.rank + 1) / k.blocks) - j0;
  const int n = k.n, c0 = k.c0, gc0 = c0 + args.s.col0;
  ChainStates<N> vs, hs;
  vs.set_up(smem + at.v, V);
  hs.set_up(smem + at.h, (H + k.blocks - 1) / k.blocks);
  ChainLayer<NT> visible;
  visible.set_up(k, V, smem + at.part);
  float* const sum = smem + at.sum;
  float* const bh = smem + at.bh;
  ChainShare<NT> w;
  w.set_up(p.w, V, j0, nj, args.s.resident, smem + at.w);
  double* const hgain = reinterpret_cast<double*>(smem + at.gains);   // (an entry belongs to a thread)
  double* const vgain = hgain + nj * N;
  vs.clear();
  hs.clear();
  grid_dependents_launch();
  grid_dependency_wait();
  w.template load<kVec>();
  for (int j = threadIdx.x; j < nj; j += kChainThreads) bh[j] = p.a[j0 + j];
  __syncthreads();
  const bool rounded = __syncthreads_or(vs.load(p.v_sample + (long)c0 * V, n, V));
  for (int it = threadIdx.x; it < nj * n; it += kChainThreads) hgain[it] = 0.0;
  for (int it = threadIdx.x; it < 2 * visible.nq * n; it += kChainThreads) vgain[it] = 0.0;
  // b'v of the states the chains start from
  visible.each(k, false, [&](int it, int c, int i, float, float) {
    const float* v = p.v_state + (long)(c0 + c) * V + i;
    vgain[it] = (double)args.dbeta[0] * (p.b[i] * v[0] + (i + 1 < V ? p.b[i + 1] * v[1] : 0.0f));
  });
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  chain_cluster_sync();    // (also: every block of the cluster is there before anyone stores into it)
  for (int step = 0; step < args.steps; step++) {
    const bool last = step == args.steps - 1;
    const float s0 = args.beta[step], s = args.beta[step + 1];
    if (step == 0 && rounded) w.up_exact(p.v_sample + (long)c0 * V, n, sum);
    else w.template up<kVec>(vs, sum);
    __syncthreads();
    {
      const PhiloxKey key = make_philox_key(p.seed, args.call0 + 2ull * step);
      for (int it = threadIdx.x; it < nj * n; it += kChainThreads) {
        const int c = it / nj, j = it - c * nj;
        const float x = w.up_sum(sum, j, c) + bh[j], xs = x * s;
        hgain[it] += (double)(log_1_plus_exp(xs) - log_1_plus_exp(x * s0));
        const float d = draw_of(j0 + j, gc0 + c, key, sigmoid_accurate(xs));
        hs.put(c, down_order(j), d);
        if (last) {
          const long to = (long)(c0 + c) * H + j0 + j;
          p.h_pre[to] = x;
          p.h_sample[to] = d;
        }
      }
    }
    __syncthreads();
    w.template down<kVec>(hs, visible.part);
    chain_cluster_sync();
    {
      const PhiloxKey key = make_philox_key(p.seed, args.call0 + 2ull * step + 1);
      visible.each(k, true, [&](int it, int c, int i, float x, float y) {
        const bool two = i + 1 < V;
        const float bx = p.b[i], by = two ? p.b[i + 1] : 0.0f;
        x = sigmoid_accurate(s * x + s * bx);
        y = sigmoid_accurate(s * y + s * by);
        const float dx = draw_of(i, gc0 + c, key, x), dy = two ? draw_of(i + 1, gc0 + c, key, y) : 0.0f;
        if (!last) {
          vgain[it] += (double)args.dbeta[step + 1] * (bx * x + by * y);
        } else {
          const long to = (long)(c0 + c) * V + i;
          p.v_state[to] = x;
          p.v_sample[to] = dx;
          if (two) {
            p.v_state[to + 1] = y;
            p.v_sample[to + 1] = dy;
          }
        }
        vs.put(c, i, dx);
        vs.put(c, i + 1, dy);
      });
    }
    __syncthreads();
    vs.share(k, n, visible.q0, visible.nq);
    chain_cluster_sync();
  }
  // the log weights: a warp per chain, then the blocks in order
  for (int c = threadIdx.x >> 5; c < n; c += kChainWarps) {
    double g = 0.0;
    for (int j = threadIdx.x & 31; j < nj; j += 32) g += hgain[c * nj + j];
    for (int q = threadIdx.x & 31; q < 2 * visible.nq; q += 32) g += vgain[((q >> 1) * n + c) * 2 + (q & 1)];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
    if ((threadIdx.x & 31) == 0) st_peer(chain_peer(chain_addr(&total[k.rank][c]), 0), g);
  }
  chain_cluster_sync();
  if (k.rank == 0 && (int)threadIdx.x < n) {
    double g = 0.0;
    for (int r = 0; r < k.blocks; r++) g += total[r][threadIdx.x];
    p.weights[c0 + threadIdx.x] = (float)(p.weights[c0 + threadIdx.x] + g);
  }
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < V; i += kChainThreads) p.sb[i] = args.beta[args.steps] * p.b[i];
}

// ---- host side ------------------------------------------------------------------
// f(std::integral_constant<int, NT>) of the instance that takes n chains a cluster.
constexpr int kMaxChains = 16;
constexpr int kMaxUnits = 1 << 16;   // of a layer: far more than shared memory takes, and sizes that stay within an int
template <typename F>
int with_chains(int n, F f) {
  return n <= 8 ? f(std::integral_constant<int, 1>{}) : f(std::integral_constant<int, 2>{});
}

cudaLaunchConfig_t chain_config(int clusters, int blocks, size_t smem, cudaLaunchAttribute (&at)[2]) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(clusters * blocks));
  cfg.blockDim = dim3(kChainThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream();
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)blocks;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = dependent_launch_enabled() ? 2 : 1;
  return cfg;
}

template <typename K>
int allow_chains(K kernel) {
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kChainSmem) == cudaSuccess &&
      cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess)
    return 0;
  return set_error(cudaGetErrorString(cudaGetLastError()));
}

// Clusters of 8 or 16 blocks that the device runs at the same time; 0: none.
int clusters_at_once(int blocks) {
  static int room[64][2] = {{0}};      // (computed twice by two threads: the same value)
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int& r = room[dev][blocks == 16];
  if (!r) {
    auto kernel = k_ais_chains<2, true>;
    int n = 0;
    if (allow_chains(kernel) == 0) {
      cudaLaunchAttribute at[2];
      cudaLaunchConfig_t cfg = chain_config(1, blocks, kChainSmem, at);
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) n = 0;
    }
    cudaGetLastError();
    clear_error();
    r = n > 0 ? n : -1;
  }
  return r > 0 ? r : 0;
}

struct ChainPlan {
  ChainSpread s;
  size_t smem;
  int n;               // the most chains of a cluster
  float us;            // estimate
};

// Spreads B chains.  The estimate, in us, is fitted to 1700 runs of 21 models (16 x 24 to 4000 x 1000) and 1 to 1500 chains
// with either cluster and up to eight waves: rms error 5 %, at most 17 %.
bool plan_chains(int V, int H, int B, int steps, ChainPlan& best) {
  best.us = 1e30f;
  if (V > kMaxUnits || H > kMaxUnits) return false;
  for (int blocks : {8, 16}) {
    const int room = clusters_at_once(blocks);
    if (!room) continue;
    for (int waves = 1; waves <= 16; waves++) {
      const long most = (long)waves * room;
      const int clusters = (int)(most < B ? most : B), n = (B + clusters - 1) / clusters;
      if (n > kMaxChains) continue;
      ChainPlan c = {};
      c.s.B = B;
      c.s.blocks = blocks;
      c.s.clusters = clusters;
      c.n = n;
      with_chains(n, [&](auto k) {
        constexpr int NT = decltype(k)::value;
        const size_t other = 4 * (size_t)AisShared<NT>(V, H, blocks).w;
        if (other > (size_t)kChainSmem) return 0;
        const size_t column = 4 * (size_t)ChainShare<NT>::column(V);
        const int all = ((H + blocks - 1) / blocks + 15) & ~15;        // (whole tiles of columns)
        long res = (long)((kChainSmem - other) / column);
        res = res < all ? res & ~15L : all;
        c.s.resident = (int)res;
        c.smem = other + column * res;
        // thousands of quads of weights of a block, of weights it reads from L2; its hidden units, the visible units
        const float weights = 1e-3f * all * (column / 16), from_l2 = 1e-3f * (all - res) * (column / 4);
        const float hidden = (float)((H + blocks - 1) / blocks) * n / 512.0f, visible = (float)V * n / 4096.0f;
        const float step = 2.35f + 0.047f * blocks + (NT == 1 ? 0.367f : 0.438f) * weights + 0.047f * from_l2 + 0.89f * hidden + 1.15f * visible;
        c.us = 8.0f + waves * (6.0f + steps * step);      // (beyond the set-up of the products)
        if (c.us < best.us) best = c;
        return 0;
      });
    }
  }
  return best.us < 1e30f;
}

template <typename K>
int launch_chains(K kernel, const ChainPlan& plan, const AisArgs& args) {
  const int err = allow_chains(kernel);
  if (err) return err;
  cudaLaunchAttribute at[2];
  cudaLaunchConfig_t cfg = chain_config(plan.s.clusters, plan.s.blocks, plan.smem, at);
  if (cudaLaunchKernelEx(&cfg, kernel, args) != cudaSuccess) return set_error(cudaGetErrorString(cudaGetLastError()));
  return check_launch();
}

// What a step takes as two products and a kernel between them, in us: fitted to the same models and up to 2048 chains, rms error
// 11 %, at most 35 %.
float products_us(int V, int H, int B) {
  const float vh = (float)V * H;
  return 14.7f + 2.8e-3f * (V + H) + 0.77e-6f * vh + 0.96e-3f * sqrtf(vh * B) + 6.8e-6f * (V + H) * B;
}

}  // namespace

static int g_ais_form = 0;    // 0: by the estimates; 1: one launch or none; 2: the products (tests)

// Whether all steps go in one launch: where they come out a tenth ahead.  Of 270 sets of models and chains, 1 to 100 steps each,
// that was never more than 3 % behind the products; at the line 784 x 500 takes (us a step, one launch
// / products) 26.5 / 30.5 with 250 chains, 28.8 / 38.6 with 350, 43.1 / 39.4 with 500, 85.9 / 49.5 with 1000.
static bool in_one_launch(int V, int H, int B, int steps, ChainPlan& plan) {
  if (V <= 0 || H <= 0 || B <= 0 || steps < 1 || g_ais_form == 2) return false;
  const int typical = steps < kAisBatch ? steps : kAisBatch;
  return plan_chains(V, H, B, typical, plan) && (g_ais_form == 1 || 1.1f * plan.us <= typical * products_us(V, H, B));
}

int ais_chains(const AisChains& a) {
  const int steps = a.n - 1;
  ChainPlan plan;
  if (!in_one_launch(a.V, a.H, a.B, steps, plan)) return g_ais_form == 1 ? set_error("the steps do not go in one launch") : ERROR_UNSUPPORTED;
  const bool vec = a.V % 4 == 0 && ((uintptr_t)a.w & 15) == 0;
  AisArgs p = {plan.s, a, 0, 0, {}, {}};
  p.s.col0 = rng_col0();
  for (int first = 0; first < steps; first += kAisBatch) {
    p.steps = steps - first < kAisBatch ? steps - first : kAisBatch;
    p.call0 = a.call0 + 2ull * first;
    for (int i = 0; i <= p.steps; i++) p.beta[i] = (float)a.schedule[first + i];
    for (int i = 0; i < p.steps; i++) p.dbeta[i] = (float)(a.schedule[first + i + 1] - a.schedule[first + i]);
    const int err = with_chains(plan.n, [&](auto k) {
      constexpr int NT = decltype(k)::value;
      return vec ? launch_chains(k_ais_chains<NT, true>, plan, p) : launch_chains(k_ais_chains<NT, false>, plan, p);
    });
    if (err) return err;
  }
  return 0;
}

}  // namespace b200

// Test hook: 0 the faster form of ais_binary_steps, 1 all steps in one launch (an error where they do not go), 2 three launches a
// step.
extern "C" int b200_test_ais_form(int form) {
  if (form < 0 || form > 2) return ERROR_UNSUPPORTED;
  b200::g_ais_form = form;
  return 0;
}
// 1: ais_binary_steps takes one launch for n inverse temperatures of B chains.
extern "C" int b200_test_ais_in_one_launch(int V, int H, int B, int n) {
  b200::ChainPlan plan;
  return b200::in_one_launch(V, H, B, n - 1, plan) ? 1 : 0;
}
