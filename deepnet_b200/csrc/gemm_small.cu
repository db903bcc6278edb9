// fp32-grade product for the sizes at which a launch, not the tensor pipe, sets the time, and for
// operands TMA cannot address (leading dimensions that are not multiples of four floats).
//
// A CTA owns a 64 x 64 tile of the output and walks its share of K in slabs of 32 through a ring of
// cp.async stages: 16-byte copies where the operand's columns allow them, 4-byte copies otherwise, so
// every leading dimension and offset takes the same kernel.  Eight warps: four cover the tile (32 x 32
// each), twice, for the two halves of every slab.  A staged tile keeps the operand's own direction; which
// row, column and k an mma slot stands for is free as long as both sides agree, so a lane takes rows
// 4g .. 4g + 3 and k = 8t .. 8t + 7 and every fragment read is 16 bytes, without bank conflicts behind the
// swizzles below.
// The parts are made in registers: hi = x rounded to TF32 (11 significant bits), lo = x - hi (exact, at
// most 12 bits, of which the tensor core reads 11), and a . b = lo.hi + hi.lo + hi.hi on mma.sync TF32:
// 2^-21 per term at worst (lo.lo is left out: 2^-22, and a bit of either lo: 2^-23 each).
// The tensor core truncates when it accumulates: after two slabs its accumulator is added to
// the running sum with ordinary rounding and starts over.
// The other form of the kernel multiplies full fp32 operands on CUDA cores from the same staged tiles: `dot` where
// every bit of a short product counts.  A lane keeps the 4 x 8 outputs that its mma products end in; a slab takes
// up to a fifth longer (500 x 100, K = 784: 11.2 us against 10.0; 1024 x 256, K = 1024: 20.3 against 16.7).
//
// Few tiles and a long K are cut along K over the CTAs of a thread-block cluster (2, 4 or 8): each
// leaves its partial tile in its own shared memory, and every CTA of the cluster sums one share of
// the tile over all of them through distributed shared memory, in rank order (the same bits every
// run), and runs the epilogue for that share.  One launch a product: no partials in global memory, no
// finishing kernel.  mma.sync rather than tcgen05: the smallest tcgen05 tile is 128 rows, its operands
// need TMA's alignment (or a pass through shared memory), and setting up tensor memory, barriers and
// roles costs more than these products compute.
//
// Bound by instruction issue (the split of the operands and the copies, not the products): a CTA walks a slab in
// 1.05 us (two terms) or 1.35 (three) alone on its SM, in 1.1 or 1.5 beside another.  Measured, with the error against 64 bits of a logistic layer:
//   500 x 100, K = 784       15.1 us (tcgen05 product + finishing launch, 2.0e-7) -> 10.0 us (5.5e-8)
//   784 x 500, 2 x K = 100   19.2 us                                               -> 12.8 us
//   1024 x 256, K = 1024     23.6 us                                               -> 15.5 us
//   601 x 203, K = 1357      519 us (CUDA cores, 2.4e-7)                           -> 24.2 us (6.0e-8)
#include <initializer_list>

#include "gemm.cuh"

namespace b200 {

namespace {

constexpr int SM_T = 64;              // rows and columns of a tile
constexpr int SK = 32;                // K per slab
constexpr int kStages = 4;
constexpr int kTileFloats = SM_T * SK;
constexpr int kSmallThreads = 256;
constexpr int kSmallSmem = kStages * 2 * kTileFloats * 4;
constexpr int kPartFloats = SM_T * SM_T;      // one partial tile, [n][m]
static_assert(kPartFloats * 4 <= kSmallSmem, "the partial tile reuses the ring");
constexpr int kMaxPairs = 4;

struct SmallOperand {
  const float* p;      // first element the product reads
  int ld;
  int kmajor;          // 1: K is the contiguous direction
  int vec;             // 16-byte copies
  int exact;           // no low part wanted (the operand is read as TF32)
};
struct SmallPair {
  SmallOperand a, b;
  int k, negate;
  int slab0;           // first slab of this pair in the product's list
};
struct SmallParams {
  SmallPair pair[kMaxPairs];
  int npairs, slabs, splits;
  int M, N, tiles_m;
  int ieee;            // non-finite results are computed again: in plain fp32 (`dot` keeps the meaning of inf), else as
                       // the tcgen05 kernel's parts give them
  const float* prior;  // what beta multiplies
  GemmEpilogue e;
};

__device__ __forceinline__ void cp16(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory"); }

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address of this CTA's shared location in CTA `rank` of the cluster, and a read through it.
__device__ __forceinline__ uint32_t peer_smem(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float ld_peer(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}

__device__ __forceinline__ void mma_tf32_16x8x8(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Where a staged tile keeps its elements (in floats).  K-major: rows of 32, 16-byte chunk c of row r at
// c ^ (r / 4 mod 8).  Rows-major: rows of 64 for every k, chunk c at c ^ 2 (k / 8 mod 4).  Partial tiles
// ([n][m], rows of 64) are kept like the latter, with n in the place of k.
__device__ __forceinline__ int at_k(int r, int k) { return r * SK + (((k >> 2) ^ ((r >> 2) & 7)) << 2) + (k & 3); }
__device__ __forceinline__ int at_m(int k, int r) { return k * SM_T + (((r >> 2) ^ (((k >> 3) & 3) << 1)) << 2) + (r & 3); }

// One operand's copies as a thread issues them, slab after slab: where its first copy comes from, what lies
// inside, and how far the next ones are.  Set up once per pair of matrices.
struct Stager {
  const float* src;      // of the thread's first copy in the next slab
  int step, slab;        // floats from one copy to the next, from one slab to the next
  int k, K;              // K index of that copy, end of K
  int left;              // rows left from the thread's first row
  uint32_t dst;          // byte offset of the first copy inside the tile
  bool kmajor, vec;

  // rows [r0, r0 + 64) of an operand of R rows, from k0 on
  __device__ __forceinline__ void start(const SmallOperand& o, int r0, int R, int k0, int K_) {
    const int t = threadIdx.x;
    kmajor = o.kmajor;
    vec = o.vec;
    K = K_;
    const int ld = o.ld;
    int r, kk;
    if (kmajor) {
      r = vec ? t >> 3 : t >> 5;          // 8 chunks or 32 elements a row
      kk = vec ? 4 * (t & 7) : t & 31;
      src = o.p + (long)(r0 + r) * ld + k0 + kk;
      step = (vec ? 32 : 8) * ld;
      slab = SK;
      dst = 4u * (uint32_t)at_k(r, kk);
    } else {
      r = vec ? 4 * (t & 15) : t & 63;    // 16 chunks or 64 elements per k
      kk = vec ? t >> 4 : t >> 6;
      src = o.p + (long)(k0 + kk) * ld + r0 + r;
      step = (vec ? 16 : 4) * ld;
      slab = SK * ld;
      dst = 4u * (uint32_t)at_m(kk, r);
    }
    k = k0 + kk;
    left = R - r0 - r;
  }
  // Copies the tile of the next slab to `tile`; what lies outside the operand becomes zero (a copy of no bytes
  // reads nothing).
  __device__ __forceinline__ void copy(uint32_t tile) {
    const float* s = src;
    if (kmajor) {
      if (vec) {
        const int in_k = min(max(K - k, 0), 4) * 4;
#pragma unroll
        for (int i = 0; i < 2; i++) {     // (32 rows on: the same swizzle)
          cp16(tile + dst + i * (32 * SK * 4), s, 32 * i < left ? in_k : 0);
          s += step;
        }
      } else {
        const int in_k = k < K ? 4 : 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {     // 8 rows on: r / 4 grows by 2 (its bit 0 is the first row's own)
          cp4(tile + (dst ^ (((2u * i) & 7u) * 16u)) + i * (8 * SK * 4), s, 8 * i < left ? in_k : 0);
          s += step;
        }
      }
    } else if (vec) {
      const int in_r = min(max(left, 0), 4) * 4;
#pragma unroll
      for (int i = 0; i < 2; i++) {       // 16 values of k on: (k / 8) mod 4 changes by 2, the chunk by 4
        cp16(tile + ((dst + i * (16 * SM_T * 4)) ^ (i * 64u)), s, k + 16 * i < K ? in_r : 0);
        s += step;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; i++) {       // 4 values of k on: k / 8 is i / 2 (the first k is below 4)
        cp4(tile + (dst ^ ((i >> 1) * 32u)) + i * (4 * SM_T * 4), s, (left > 0 && k + 4 * i < K) ? 4 : 0);
        s += step;
      }
    }
    src += slab;
    k += SK;
  }
};

// x = hi + lo, hi rounded to TF32, lo of 12 significant bits at most.  An exact operand is used as it is: the tensor
// core drops the low 13 bits.
template <bool kExact>
__device__ __forceinline__ void split_parts(float x, uint32_t& hi, uint32_t& lo) {
  hi = __float_as_uint(x);
  if (!kExact) {
    hi = (hi + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi));
  }
}

// Half a slab of one operand for a warp: x[i][c] = element of row 4g + i at k = 8t + 4 * half + c.  `tile` points
// at the lane's first chunk (a K-major tile holds its next rows 32 floats apart, a rows-major one its next k 64
// apart, under the same swizzle).
template <bool kKMajor>
__device__ __forceinline__ void read_half(const float* tile, float (&x)[4][4]) {
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float4 v = *reinterpret_cast<const float4*>(tile + i * (kKMajor ? SK : SM_T));
    if (kKMajor) { x[i][0] = v.x; x[i][1] = v.y; x[i][2] = v.z; x[i][3] = v.w; }
    else { x[0][i] = v.x; x[1][i] = v.y; x[2][i] = v.z; x[3][i] = v.w; }
  }
}

// Half a slab for a warp: its 32 x 32 outputs over 16 values of K.  One instance per pair of directions and of
// exact operands: with the directions read at run time the two ways of a fragment into its registers met in moves.
// mma slots: rows g, g + 8 of product i = rows 4g + 2i, 4g + 2i + 1; column g of product n = column 4g + n; k slots
// t, t + 4 = the lane's k values 2j, 2j + 1.
template <bool kAK, bool kBK, bool kEA, bool kEB>
__device__ __forceinline__ void half_slab(const float* ta, const float* tb, float (&part)[2][4][4]) {
  float xa[4][4], xb[4][4];
  read_half<kAK>(ta, xa);
  read_half<kBK>(tb, xb);
#pragma unroll
  for (int j = 0; j < 2; j++) {
    uint32_t ah[2][4], al[2][4], bh[4][2], bl[4][2];
#pragma unroll
    for (int n = 0; n < 4; n++)
#pragma unroll
      for (int c = 0; c < 2; c++) split_parts<kEB>(xb[n][2 * j + c], bh[n][c], bl[n][c]);
#pragma unroll
    for (int i = 0; i < 2; i++) {
#pragma unroll
      for (int c = 0; c < 4; c++) split_parts<kEA>(xa[2 * i + (c & 1)][2 * j + (c >> 1)], ah[i][c], al[i][c]);
      if (!kEA) {
#pragma unroll
        for (int n = 0; n < 4; n++) mma_tf32_16x8x8(part[i][n], al[i], bh[n]);
      }
      if (!kEB) {
#pragma unroll
        for (int n = 0; n < 4; n++) mma_tf32_16x8x8(part[i][n], ah[i], bl[n]);
      }
#pragma unroll
      for (int n = 0; n < 4; n++) mma_tf32_16x8x8(part[i][n], ah[i], bh[n]);
    }
  }
}

// Half a slab of full fp32 multiply-adds: the lane's 4 rows x 8 columns (the ones its mma products end in) over 16
// values of K, in order.  `rows` and `cols`: the lane's first row and column in the tile.  12 reads of 16 bytes,
// without bank conflicts, to 128 multiply-adds.
template <bool kAK, bool kBK>
__device__ __forceinline__ void half_slab_fp32(const float* sa, const float* sb, int rows, int cols, int half,
                                               float (&acc)[2][4][4]) {
#pragma unroll
  for (int kc = 0; kc < 4; kc++) {
    const int k = 16 * half + 4 * kc;
    float a[4][4], b[8][4];      // [row][k], [column][k]
    read_half<kAK>(sa + (kAK ? at_k(rows, k) : at_m(k, rows)), a);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      float x[4][4];
      read_half<kBK>(sb + (kBK ? at_k(cols + 4 * h, k) : at_m(k, cols + 4 * h)), x);
#pragma unroll
      for (int n = 0; n < 4; n++)
#pragma unroll
        for (int c = 0; c < 4; c++) b[4 * h + n][c] = x[n][c];
    }
#pragma unroll
    for (int c = 0; c < 4; c++)
#pragma unroll
      for (int r = 0; r < 4; r++)
#pragma unroll
        for (int n = 0; n < 8; n++) {
          float& s = acc[r >> 1][n & 3][2 * (r & 1) + (n >> 2)];
          s = fmaf(a[r][c], b[n][c], s);
        }
  }
}

// The sum of one output element as a chain of fp32 multiply-adds.
__device__ __noinline__ float element_fp32(const SmallParams& p, int m, int n) {
  float acc = 0.0f;
  for (int q = 0; q < p.npairs; q++) {
    const SmallPair& pr = p.pair[q];
    for (int k = 0; k < pr.k && !isnan(acc); k++) {   // (NaN stays)
      const float a = pr.a.kmajor ? pr.a.p[(long)m * pr.a.ld + k] : pr.a.p[(long)k * pr.a.ld + m];
      const float b = pr.b.kmajor ? pr.b.p[(long)n * pr.b.ld + k] : pr.b.p[(long)k * pr.b.ld + n];
      acc = fmaf(pr.negate ? -a : a, b, acc);
    }
  }
  return acc;
}

// The same of the parts as the tcgen05 kernel takes them, by truncation: an operand so near the largest float that it
// rounds to an infinity stays finite, an infinity (whose low part is not a number) gives NaN.
__device__ __noinline__ float element_truncated(const SmallParams& p, int m, int n) {
  float acc = 0.0f;
  for (int q = 0; q < p.npairs; q++) {
    const SmallPair& pr = p.pair[q];
    for (int k = 0; k < pr.k && !isnan(acc); k++) {
      const float a = pr.a.kmajor ? pr.a.p[(long)m * pr.a.ld + k] : pr.a.p[(long)k * pr.a.ld + m];
      const float b = pr.b.kmajor ? pr.b.p[(long)n * pr.b.ld + k] : pr.b.p[(long)k * pr.b.ld + n];
      const float ah = __uint_as_float(__float_as_uint(a) & 0xffffe000u), bh = __uint_as_float(__float_as_uint(b) & 0xffffe000u);
      const float s = pr.negate ? -1.0f : 1.0f;
      if (!pr.a.exact) acc = fmaf(s * (a - ah), bh, acc);
      if (!pr.b.exact) acc = fmaf(s * ah, b - bh, acc);
      acc = fmaf(s * ah, bh, acc);
    }
  }
  return acc;
}

// Two CTAs per SM: with one, the next product's CTAs could not become resident before this one's end, and the
// dependent launch would hide nothing (500 x 100, K = 784: 15.8 us at one CTA per SM and no spills, 10.9 at two).
template <bool kFp32>
__global__ void __launch_bounds__(kSmallThreads, 2) k_gemm_small(const __grid_constant__ SmallParams p) {
  extern __shared__ float4 smem4[];
  float* const smem = reinterpret_cast<float*>(smem4);
  const uint32_t smem_base = (uint32_t)__cvta_generic_to_shared(smem);
  const int S = p.splits;
  const int tile = blockIdx.x / S, rank = blockIdx.x - tile * S;   // (the CTAs of a cluster are neighbours in x)
  const int tn = tile / p.tiles_m, tm = tile - tn * p.tiles_m;
  const int m0 = tm * SM_T, n0 = tn * SM_T;
  const int warp = threadIdx.x >> 5, wm = (warp & 1) * 32, wn = ((warp >> 1) & 1) * 32, half = warp >> 2;
  const int first = (int)((long)p.slabs * rank / S), last = (int)((long)p.slabs * (rank + 1) / S);
  grid_dependents_launch();
  grid_dependency_wait();

  Stager ca, cb;
  int lq = -1, lnext = first;   // the pair being copied, and the slab at which the next one starts
  auto issue = [&](int s) {
    if (s < last) {
      if (s >= lnext) {
        do {
          lq++;
          lnext = lq + 1 < p.npairs ? p.pair[lq + 1].slab0 : p.slabs;
        } while (s >= lnext);
        const SmallPair& pr = p.pair[lq];
        const int k0 = (s - pr.slab0) * SK;
        ca.start(pr.a, m0, p.M, k0, pr.k);
        cb.start(pr.b, n0, p.N, k0, pr.k);
      }
      const uint32_t st = smem_base + (uint32_t)((s - first) % kStages) * (2 * kTileFloats * 4);
      ca.copy(st);
      cb.copy(st + kTileFloats * 4);
    }
    cp_commit();   // (an empty group keeps the count of groups in step)
  };
  float acc[2][4][4] = {}, part[2][4][4] = {};
#pragma unroll 1
  for (int s = 0; s < kStages - 1; s++) issue(first + s);
  const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
  int offa = 0, offb = 0;       // where the lane's fragments start in a tile
  int q = -1, qnext = first;
  int form = 0;                 // directions and exact operands of the pair
  float sign = 1.0f;
#pragma unroll 1
  for (int s = first; s < last; s++) {
    cp_wait<kStages - 2>();
    __syncthreads();      // slab s has landed for everyone; the stage of slab s - 1 is free
    issue(s + kStages - 1);
    if (s >= qnext) {
      do {
        q++;
        qnext = q + 1 < p.npairs ? p.pair[q + 1].slab0 : p.slabs;
      } while (s >= qnext);
      const SmallPair& pr = p.pair[q];
      const bool ak = pr.a.kmajor, bk = pr.b.kmajor;
      form = (ak ? 8 : 0) + (bk ? 4 : 0) + (pr.a.exact ? 2 : 0) + (pr.b.exact ? 1 : 0);
      sign = pr.negate ? -1.0f : 1.0f;
      offa = ak ? at_k(wm + 4 * g, 8 * t + 4 * half) : at_m(8 * t + 4 * half, wm + 4 * g);
      offb = kTileFloats + (bk ? at_k(wn + 4 * g, 8 * t + 4 * half) : at_m(8 * t + 4 * half, wn + 4 * g));
    }
    const float* sa = smem + (size_t)((s - first) % kStages) * (2 * kTileFloats);
    if constexpr (kFp32) {   // (one pair, not negated)
      const float* sb = sa + kTileFloats;
      switch (form >> 2) {
        case 0: half_slab_fp32<false, false>(sa, sb, wm + 4 * g, wn + 8 * t, half, acc); break;
        case 1: half_slab_fp32<false, true>(sa, sb, wm + 4 * g, wn + 8 * t, half, acc); break;
        case 2: half_slab_fp32<true, false>(sa, sb, wm + 4 * g, wn + 8 * t, half, acc); break;
        case 3: half_slab_fp32<true, true>(sa, sb, wm + 4 * g, wn + 8 * t, half, acc); break;
      }
      continue;
    }
    const float *ta = sa + offa, *tb = sa + offb;
    switch (form) {
#define B200_HALF_SLAB(F) case F: half_slab<((F) & 8) != 0, ((F) & 4) != 0, ((F) & 2) != 0, ((F) & 1) != 0>(ta, tb, part); break;
      B200_HALF_SLAB(0) B200_HALF_SLAB(1) B200_HALF_SLAB(2) B200_HALF_SLAB(3)
      B200_HALF_SLAB(4) B200_HALF_SLAB(5) B200_HALF_SLAB(6) B200_HALF_SLAB(7)
      B200_HALF_SLAB(8) B200_HALF_SLAB(9) B200_HALF_SLAB(10) B200_HALF_SLAB(11)
      B200_HALF_SLAB(12) B200_HALF_SLAB(13) B200_HALF_SLAB(14) B200_HALF_SLAB(15)
#undef B200_HALF_SLAB
    }
    // into the running sum after two slabs, and where the sign may change or the share ends
    if (((s - first) & 1) || s + 1 == last || s + 1 == qnext) {
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int n = 0; n < 4; n++)
#pragma unroll
          for (int c = 0; c < 4; c++) {
            acc[i][n][c] = fmaf(sign, part[i][n][c], acc[i][n][c]);
            part[i][n][c] = 0.0f;
          }
    }
  }
  cp_wait<0>();
  __syncthreads();

  // the CTA's partial tile, [n][m]: the second half's sums through shared memory into the first's
  {
    // columns 2t + h of product n: tile column 4 (2t + h) + n, rows 4g .. 4g + 3 (4h + n < 8: one swizzle)
    float4* const at = reinterpret_cast<float4*>(smem + at_m(wn + 8 * t, wm + 4 * g));
    if (half == 1) {
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int n = 0; n < 4; n++)
          at[(4 * h + n) * (SM_T / 4)] = make_float4(acc[0][n][h], acc[0][n][2 + h], acc[1][n][h], acc[1][n][2 + h]);
    }
    __syncthreads();
    if (half == 0) {
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int n = 0; n < 4; n++) {
          const float4 o = at[(4 * h + n) * (SM_T / 4)];
          at[(4 * h + n) * (SM_T / 4)] =
              make_float4(acc[0][n][h] + o.x, acc[0][n][2 + h] + o.y, acc[1][n][h] + o.z, acc[1][n][2 + h] + o.w);
        }
    }
  }
  if (S > 1) cluster_barrier();
  else __syncthreads();

  // This CTA's share of the tile: one row of four columns (they share one Philox block) per thread and round.
  const GemmEpilogue e = p.e;
  const bool draw = e.sample != nullptr || e.sample_aux != nullptr;
  const float alpha = e.alpha * exp2f(-((e.scale_exp ? *e.scale_exp : 0.0f) + (float)e.scale_exp_const));
  const float aux_scale = exp2f((float)e.aux_exp);
  const int shift = (n0 + e.col0) & 3;         // 0 unless the shard's first column is not a multiple of four
  const int nitems = SM_T * (SM_T / 4) / S;
#pragma unroll 1
  for (int it = threadIdx.x; it < nitems; it += kSmallThreads) {
    const int item = rank * nitems + it;
    const int ml = item & (SM_T - 1), nl = (item >> 6) * 4;
    const int m = m0 + ml, n = n0 + nl;
    if (m >= p.M || n >= p.N) continue;
    const float bias = e.bias ? e.bias[m] : 0.0f;
    const int at = at_m(nl, ml);     // the four columns are SM_T apart (nl is a multiple of four: one swizzle)
    float x[4];
    if (S == 1) {
#pragma unroll
      for (int j = 0; j < 4; j++) x[j] = smem[at + j * SM_T];
    } else {   // four neighbours' reads at a time: each takes a fifth of a microsecond
#pragma unroll
      for (int j = 0; j < 4; j++) x[j] = 0.0f;
#pragma unroll 1
      for (int r0 = 0; r0 < S; r0 += 4) {
        float v[4][4];
#pragma unroll
        for (int r = 0; r < 4; r++) {
          const uint32_t peer = peer_smem(smem_base, r0 + r < S ? r0 + r : 0);
#pragma unroll
          for (int j = 0; j < 4; j++) v[r][j] = r0 + r < S ? ld_peer(peer + 4u * (uint32_t)(at + j * SM_T)) : 0.0f;
        }
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
          for (int j = 0; j < 4; j++) x[j] += v[r][j];
      }
    }
    const int ncols = min(4, p.N - n);
    if ((!kFp32 || !p.ieee) && !isfinite((x[0] + x[1]) + (x[2] + x[3]))) {   // (a finite sum has finite terms)
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (j < ncols && !isfinite(x[j])) x[j] = p.ieee ? element_fp32(p, m, n + j) : element_truncated(p, m, n + j);
    }
    const long off = (long)n * e.ldo + m;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      x[j] *= alpha;
      if (e.beta != 0.0f && j < ncols) x[j] += e.beta * p.prior[off + (long)j * e.ldo];
      if (e.bias) x[j] += (e.col_scale && j < ncols) ? bias * e.col_scale[n + j] : bias;
      if (e.activation == 1) x[j] = sigmoid_accurate(x[j]);
    }
    if (e.out) {
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (j < ncols) e.out[off + (long)j * e.ldo] = x[j];
    }
    const long word = 2L * n * e.ld_aux + m;   // 16-bit word of plane 0
    if (e.out_aux) {
      uint16_t* const oa = reinterpret_cast<uint16_t*>(e.out_aux);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        uint16_t lo, hi;
        if (e.aux_f16) split_f16(x[j], aux_scale, lo, hi);
        else split_aux(x[j], lo, hi);
        if (j < ncols) {
          oa[word + 2L * j * e.ld_aux] = lo;
          oa[word + 2L * j * e.ld_aux + e.ld_aux] = hi;
        }
      }
    }
    if (draw) {
      const uint32_t blk = (uint32_t)((n + e.col0) >> 2);
      uint4 w = philox4x32_10((uint32_t)m, blk, e.key);
      if (shift) {
        const uint4 w2 = philox4x32_10((uint32_t)m, blk + 1u, e.key);
        w = shift == 1 ? make_uint4(w.y, w.z, w.w, w2.x)
                       : (shift == 2 ? make_uint4(w.z, w.w, w2.x, w2.y) : make_uint4(w.w, w2.x, w2.y, w2.z));
      }
      const uint16_t one = e.aux_f16 ? __half_as_ushort(__float2half_rn(aux_scale)) : (uint16_t)0x3f80;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const bool on = word_to_uniform(pick_word(w, j)) < x[j];
        if (j < ncols) {
          if (e.sample) e.sample[off + (long)j * e.ldo] = on ? 1.0f : 0.0f;
          if (e.sample_aux)
            reinterpret_cast<uint16_t*>(e.sample_aux)[word + 2L * j * e.ld_aux + e.ld_aux] = on ? one : (uint16_t)0;
        }
      }
    }
  }
  if (S > 1) cluster_barrier();   // nobody leaves while its partial tile may still be read
}

inline bool same_matrix(const GemmOperand& a, const GemmOperand& b) {
  return a.ptr == b.ptr && a.ld == b.ld && a.trans == b.trans && a.row0 == b.row0;
}

SmallOperand small_operand(const GemmOperand& o, bool kmajor, bool exact) {
  SmallOperand s;
  s.p = o.ptr + o.row0;
  s.ld = o.ld;
  s.kmajor = kmajor;
  s.vec = o.ld % 4 == 0 && ((uintptr_t)s.p & 15) == 0;
  s.exact = exact;
  return s;
}

// Gathers the term list into pairs of matrices: consecutive terms over one pair have to spell out its
// product once (x.x, with the low part of either side or without).  False: another kind of list.
bool gather_pairs(const GemmProblem& g, SmallParams& p) {
  p.npairs = 0;
  p.slabs = 0;
  int q = 0;
  while (q < g.npass) {
    const GemmPass& f = g.pass[q];
    if (f.k <= 0 || f.a.ld > (1 << 24) || f.b.ld > (1 << 24)) return false;   // (a slab's step is kept in 32 bits)
    int xx = 0, la = 0, lb = 0;
    for (; q < g.npass; q++) {
      const GemmPass& t = g.pass[q];
      if (!same_matrix(t.a, f.a) || !same_matrix(t.b, f.b) || t.k != f.k || t.negate != f.negate || xx) break;
      const int pa = t.a.part, pb = t.b.part;
      if (pa == kPartX && pb == kPartX) xx++;
      else if ((pa == kPartLo32 && pb == kPartX) || (pa == kPartLo16 && pb == kPartB16)) la++;
      else if ((pa == kPartX && pb == kPartLo32) || (pa == kPartB16 && pb == kPartLo16)) lb++;
      else return false;
    }
    if (xx != 1 || la > 1 || lb > 1 || p.npairs == kMaxPairs) return false;
    SmallPair& s = p.pair[p.npairs++];
    s.a = small_operand(f.a, f.a.trans != 0, la == 0);
    s.b = small_operand(f.b, f.b.trans == 0, lb == 0);
    s.k = f.k;
    s.negate = f.negate;
    s.slab0 = p.slabs;
    p.slabs += (f.k + SK - 1) / SK;
  }
  return p.npairs > 0;
}

// Tiles and splits; returns the CTAs.  Cut along K while the CTAs would not fill the device twice over (two are
// resident per SM) and every share keeps two slabs.
long cut_up(const GemmProblem& g, SmallParams& p) {
  p.M = g.M;
  p.N = g.N;
  p.tiles_m = (g.M + SM_T - 1) / SM_T;
  const long tiles = (long)p.tiles_m * ((g.N + SM_T - 1) / SM_T);
  p.splits = 1;
  while (p.splits < 8 && tiles * p.splits * 2 <= sm_count() * 2L && p.slabs >= p.splits * 4) p.splits *= 2;
  return tiles * p.splits;
}

// Slabs of K that one SM walks.
int walked_slabs(const GemmProblem& g, SmallParams& p) {
  const long ctas = cut_up(g, p), room = 2L * sm_count();
  const long depth = (p.slabs + p.splits - 1) / p.splits * ((ctas + room - 1) / room);
  return depth < (1 << 30) ? (int)depth : 1 << 30;
}

int allow_shared_memory() {
  static bool attr_set[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return set_error("cudaGetDevice failed");
  if (!attr_set[dev]) {   // (setting it twice from two threads does no harm)
    for (void (*kernel)(SmallParams) : {k_gemm_small<true>, k_gemm_small<false>})
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem) != cudaSuccess)
        return set_error("cudaFuncSetAttribute(max dynamic shared memory) failed");
    attr_set[dev] = true;
  }
  return 0;
}

// CTAs of clusters of `splits` that are resident at the same time (two per SM, less what the clusters leave over in every
// group of SMs that shares them: 296 CTAs in clusters of four took two waves).
long resident_ctas(int splits) {
  static long room[9] = {0};   // (computed twice by two threads: the same value)
  const long all = 2L * sm_count();
  if (splits == 1) return all;
  if (!room[splits]) {
    if (allow_shared_memory()) return all;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)splits);
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = kSmallSmem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)splits;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_gemm_small<false>, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      return all;
    }
    room[splits] = (long)n * splits;
  }
  return room[splits] < all ? room[splits] : all;
}

// Recomputes what came out non-finite (nothing, as a rule: one read of the result).
__global__ void __launch_bounds__(256) k_recompute_nonfinite(const __grid_constant__ SmallParams p) {
  grid_dependents_launch();
  grid_dependency_wait();
  const long items = (long)p.M * p.N;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < items; i += (long)gridDim.x * blockDim.x) {
    const int n = (int)(i / p.M), m = (int)(i - (long)n * p.M);
    float* const at = p.e.out + (long)n * p.e.ldo + m;
    if (!isfinite(*at)) *at = p.e.alpha * element_fp32(p, m, n);
  }
}

}  // namespace

int recompute_nonfinite(const GemmProblem& g) {
  SmallParams p;
  if (g.M <= 0 || g.N <= 0 || !gather_pairs(g, p)) return ERROR_UNSUPPORTED;
  p.M = g.M;
  p.N = g.N;
  p.e = g.epi;
  long blocks = ((long)g.M * g.N + 255) / 256;
  if (blocks > (long)sm_count() * 8) blocks = (long)sm_count() * 8;
  if (launch_dependent(k_recompute_nonfinite, dim3((unsigned)blocks), dim3(256), 0, stream(), p) != cudaSuccess)
    return set_error(cudaGetErrorString(cudaGetLastError()));
  return check_launch();
}

int small_depth(const GemmProblem& g) {
  SmallParams p;
  if (g.M <= 0 || g.N <= 0 || !gather_pairs(g, p)) return 0;
  return walked_slabs(g, p);
}

// Whether a product that both kernels take goes in one launch here.  The other side is estimated as the tcgen05 kernel with tiles
// of 256 columns wherever N > 128, fitted (as this one) to about 150 products of 64 x 32 to 4096 x 1024 outputs and K from 16 to
// 4096.  Narrower tiles since made it faster than that by up to a third, yet the line stays: what lies between is three to five
// times as exact here, where additions round and the terms are split TF32.  Logistic layer on 0/1 input, us and relative
// error against float64, here / there:
//   1024 x 256, K = 2048    23.7, 6.3e-8 / 17.2, 2.5e-7       500 x 1000, K = 784    20.8, 5.4e-8 / 16.0, 1.8e-7
//   1024 x 1024, K = 384    19.3, 5.0e-8 / 11.9, 1.3e-7       1024 x 1024, K = 128   10.3, 4.7e-8 /  8.8, 8.8e-8
// On the line's other sides: 2048 x 2048, two pairs of K = 32: 27.1 us here (several waves), 14.9 there; 500 x 100, K = 2800: 18.1
// here, 16.9 there.
bool small_beats_tc(const GemmProblem& g) {
  SmallParams p;
  if (g.M <= 0 || g.N <= 0 || !gather_pairs(g, p)) return false;
  const GemmEpilogue& e = g.epi;
  const bool act = e.bias || e.activation != 0 || e.sample || e.out_aux || e.sample_aux;
  const long ctas = cut_up(g, p);
  const int sms = sm_count();
  // here: a start and an end per wave of two CTAs per SM, and the walk over K; a rows-major operand's slab takes 0.1 more
  const long room = resident_ctas(p.splits);
  const float waves = (float)((ctas + room - 1) / room);
  float walk = 0.0f;
  int shortest = 1 << 30;
  for (int q = 0; q < p.npairs; q++) {
    const SmallPair& s = p.pair[q];
    const int slabs = (s.k + SK - 1) / SK, terms = 3 - (s.a.exact != 0) - (s.b.exact != 0);
    const float per_slab = ctas > sms ? 0.3f + 0.41f * terms : 0.45f + 0.3f * terms;
    walk += slabs * (per_slab + 0.1f * ((s.a.kmajor ? 0 : 1) + (s.b.kmajor ? 0 : 1)));
    shortest = slabs < shortest ? slabs : shortest;
  }
  const float one = waves * ((act ? 6.5f : 5.0f) + walk / p.splits);
  // there: tiles of 128 rows x up to 256 columns; K is cut (and a second launch finishes) when the tiles fill less than half
  // of the SMs and every pair has 8 slabs
  const bool wide = g.N > 128;
  const long tc_ctas = wide && g.M > 128 ? 2L * ((g.M + 255) / 256) * ((g.N + 255) / 256)
                                         : (long)((g.M + 127) / 128) * (wide ? (g.N + 255) / 256 : 1);
  const float n = (float)p.slabs;
  float tc;
  if (tc_ctas * 2 <= sms && shortest >= 8) {
    tc = wide ? (act ? 18.3f : 19.5f) + 0.13f * n : (act ? 9.8f : 11.3f) + 0.07f * n;
    const float second = wide ? 5.0f - 0.08f * n : 4.0f - 0.03f * n;   // of another pair, hidden behind a long K
    if (p.npairs > 1 && second > 0.0f) tc += second;
  } else {
    tc = act ? (wide ? 39.0f : 17.0f) + 0.3f * n : (wide ? 12.0f : 7.5f) + 0.87f * n;
  }
  return one < tc + 1.0f;
}

// ieee: results that come out non-finite are computed again in plain fp32, so that an infinity in an operand
// means what it means there (its low part is not a number).
int gemm_small(const GemmProblem& g, SmallForm form) {
  SmallParams p;
  if (g.M <= 0 || g.N <= 0 || !gather_pairs(g, p)) return ERROR_UNSUPPORTED;
  const bool fp32 = form == kSmallFp32 || form == kSmallFp32Parts;
  if (fp32 && (p.npairs != 1 || p.pair[0].negate)) return ERROR_UNSUPPORTED;
  p.ieee = form == kSmallIeee || form == kSmallFp32;
  p.e = g.epi;
  p.prior = g.prior ? g.prior : g.epi.out;
  const long ctas = cut_up(g, p);
  if (ctas > 0x7fffffffL) return ERROR_UNSUPPORTED;
  void (*const kernel)(SmallParams) = fp32 ? k_gemm_small<true> : k_gemm_small<false>;
  const int err = allow_shared_memory();
  if (err) return err;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(kSmallThreads);
  cfg.dynamicSmemBytes = kSmallSmem;
  cfg.stream = stream();
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)p.splits;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = dependent_launch_enabled() ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, kernel, p) != cudaSuccess) return set_error(cudaGetErrorString(cudaGetLastError()));
  return check_launch();
}

}  // namespace b200

// Slabs of 32 of K that an SM walks in the one-launch kernel for an m x n product of so many slabs.
extern "C" int b200_product_depth(int m, int n, int slabs) {
  if (m <= 0 || n <= 0 || slabs <= 0) return 0;
  b200::GemmProblem g;
  g.M = m;
  g.N = n;
  b200::SmallParams p;
  p.slabs = slabs;
  return b200::walked_slabs(g, p);
}
