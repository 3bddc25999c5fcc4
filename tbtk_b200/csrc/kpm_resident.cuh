// The whole recursion of a small matrix in one launch, on chip.
//
// Why: a step of a matrix of up to some ten thousand rows is microseconds of
// launch latency, dependent memory round trips and a nearly empty grid (4-6
// us per step at 2k-64k rows), whatever the step kernel.  Here a cluster of
// 1-16 blocks owns COLS sources: each block keeps its rows' matrix entries
// and both vectors of its rows in shared memory, a gather of another block's
// row is a distributed-shared-memory load, and one cluster barrier ends a
// step.  Clusters of different sources are independent, so the grid may be
// larger than what fits the device at once.
//
// Layout of a block's shared memory (the same offsets in every block):
//   x[2][rows + 4][COLS]  j_n and j_{n-1} of the block's rows, in turn; the
//                      row after the last stays zero
//   val[chunks*32]     the values 2H/s of the block's SELL-32 slices
//   adr[chunks*32]     per entry the shared::cluster address of its column's
//                      row in x[0] (x[1] lies `delta` bytes behind); padding
//                      points at the zero row
//   bnd[slices + 1]    chunk bounds of the slices
//   first[rows]        a flagged row's first target, else kNoEntry
//   tcol, tout[cap]    the block's targets: column in the group, output slot
//   stage[kResRing][cap]  their moments, dsum[kResRing][warps][2*COLS] the
//                      warps' doubling sums, flushed every kResRing steps
// When a warp owns at most one slice of at most kResRegs chunks, the entries
// live in registers instead (REG) and a step reads only vectors.
//
// No step touches global memory: the release of a cluster barrier waits for
// a block's stores to reach the L2 cache, and its acquire drops the cached
// copies of what was loaded (one moment stored and three target words loaded
// per step measured 0.4 us a step).
//
// Arithmetic and entry order per element are those of the step kernels
// (Exact64 for FP64, Wide64 otherwise; real vectors likewise), so stored
// vectors and directly gathered moments are bit-identical to theirs.  The
// doubling terms are summed per warp, block and cluster in a fixed order.
#pragma once

#include "kpm_kernels.cuh"

namespace tbtkkpm {

constexpr uint32_t kNoEntry = 0xffffffffu;
constexpr uint32_t kPadMark = 1;  // in the address of a padding entry (SKIP)
constexpr int kResWarps = 16;   // most warps of a block
constexpr int kResRegs = 10;    // chunks of a slice kept in registers
constexpr uint32_t kResMaxCluster = 16;
constexpr uint32_t kResRing = 16;    // steps between flushes of moments and sums
constexpr uint32_t kResTargets = 64; // most targets of a block staged (else stored step by step)
constexpr size_t kResSmem = 227 * 1024;

struct ResidentArgs {
  Sell A;
  uint32_t spb;         // slices per block
  uint32_t chunks;      // most chunks of a block
  uint32_t Bp;          // columns of the global buffers, a multiple of COLS
  void *x, *y;          // j_{n0-1}, j_{n0-2} on entry; j_{n1}, j_{n1-1} on exit if `keep`
  uint32_t n0, n1;      // steps n0..n1
  uint32_t keep;
  Targets tg;
  uint32_t cap;         // most targets of a block and group, at most kResTargets
  double *part;         // [n - n0][group][block of the cluster][2*COLS] doubling sums
};

// Offsets of a block's shared memory.
struct ResLayout {
  uint32_t val, adr, bnd, first, tcol, tout, stage, dsum, nt, bytes;
};
__host__ __device__ inline ResLayout resident_layout(uint32_t spb, uint32_t chunks, uint32_t cap,
                                                     uint32_t warps, uint32_t cols, uint32_t esz,
                                                     uint32_t vsz, bool reg, bool dots) {
  ResLayout L;
  const uint32_t ent = reg ? 0 : chunks * 32;
  L.val = (2 * (spb * 32 + 4) * cols * esz + 15) / 16 * 16;
  L.stage = L.val + ent * vsz;
  L.dsum = L.stage + kResRing * cap * 16;
  L.adr = L.dsum + (dots ? kResRing * warps * 2 * cols * 8 : 0);
  L.bnd = L.adr + ent * 4;
  L.first = L.bnd + (reg ? 0 : (spb + 1) * 4);
  L.tcol = L.first + spb * 32 * 4;
  L.tout = L.tcol + cap * 4;
  L.nt = L.tout + cap * 4;
  L.bytes = L.nt + 4;
  return L;
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <bool CL> __device__ __forceinline__ void block_or_cluster_wait() {
  if constexpr (CL) cluster_wait();
  else __syncthreads();
}

// BYTES bytes of (distributed) shared memory at a.
template <int BYTES, bool CL> __device__ __forceinline__ void res_load(uint32_t a, uint32_t *w) {
  if constexpr (BYTES == 4) {
    if constexpr (CL) asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(w[0]) : "r"(a));
    else asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[0]) : "r"(a));
  } else if constexpr (BYTES == 8) {
    if constexpr (CL)
      asm volatile("ld.shared::cluster.v2.u32 {%0, %1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "r"(a));
    else asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "r"(a));
  } else {
    static_assert(BYTES % 16 == 0, "4, 8 or a multiple of 16 bytes");
#pragma unroll
    for (int i = 0; i < BYTES / 16; i++) {
      if constexpr (CL)
        asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(w[4 * i]), "=r"(w[4 * i + 1]), "=r"(w[4 * i + 2]), "=r"(w[4 * i + 3])
                     : "r"(a + 16 * i));
      else
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(w[4 * i]), "=r"(w[4 * i + 1]), "=r"(w[4 * i + 2]), "=r"(w[4 * i + 3])
                     : "r"(a + 16 * i));
    }
  }
}

// A staged target's column word: the column in the group, and kTargetNew on
// the first target of a row.
constexpr uint32_t kTargetNew = 0x80000000u, kTargetCol = 0x7fffffffu;
__device__ __forceinline__ bool first_of(const uint32_t *tcol, uint32_t t) {
  return (tcol[t] & kTargetNew) != 0;
}

// A padding entry adds nothing, not even to the sign of a zero: for a real
// kind its value is -0 and its row is the zero row, whose product -0 leaves
// any sum as it is; a complex product's four zeros cannot all be -0, so the
// complex kinds drop its result (SKIP).
//
// How a vector kind computes: value and accumulator types, one product added,
// the value as stored and its doubling terms.
template <typename V> struct ResKind;
template <> struct ResKind<double2> {  // FP64, the reference's operations
  static constexpr bool SKIP = true;
  using Val = double2;
  using Acc = double2;
  __device__ __forceinline__ static double2 unpack(const uint32_t *w) {
    return make_double2(__hiloint2double((int)w[1], (int)w[0]), __hiloint2double((int)w[3], (int)w[2]));
  }
  __device__ __forceinline__ static Val value(const Sell &A, uint64_t i) { return A.val[i]; }
  __device__ __forceinline__ static Val none() { return make_double2(0, 0); }
  __device__ __forceinline__ static Val half(Val v) { return make_double2(v.x * 0.5, v.y * 0.5); }
  __device__ __forceinline__ static Acc zero() { return make_double2(0, 0); }
  __device__ __forceinline__ static Acc minus(double2 y) { return make_double2(-y.x, -y.y); }
  __device__ __forceinline__ static Acc mac(Acc a, Val v, double2 x) { return cmac<true>(a, v, x); }
  __device__ __forceinline__ static double2 stored(Acc a) { return a; }
  __device__ __forceinline__ static double2 moment(Acc a) { return a; }
  __device__ __forceinline__ static double term(double2, double2) { return 0; }
};
template <> struct ResKind<double> {  // FP64 of a real matrix
  static constexpr bool SKIP = false;
  using Val = double;
  using Acc = double;
  __device__ __forceinline__ static double unpack(const uint32_t *w) {
    return __hiloint2double((int)w[1], (int)w[0]);
  }
  __device__ __forceinline__ static Val value(const Sell &A, uint64_t i) { return A.vre[i]; }
  __device__ __forceinline__ static Val none() { return -0.0; }
  __device__ __forceinline__ static Val half(Val v) { return v * 0.5; }
  __device__ __forceinline__ static Acc zero() { return 0; }
  __device__ __forceinline__ static Acc minus(double y) { return -y; }
  __device__ __forceinline__ static Acc mac(Acc a, Val v, double x) {
    return __dadd_rn(a, __dmul_rn(v, x));
  }
  __device__ __forceinline__ static double stored(Acc a) { return a; }
  __device__ __forceinline__ static double2 moment(Acc a) { return make_double2(a, 0.0); }
  __device__ __forceinline__ static double term(double, double) { return 0; }
};
template <> struct ResKind<float2> {  // complex64 vectors, FP64 arithmetic
  static constexpr bool SKIP = true;
  using Val = double2;
  using Acc = double2;
  __device__ __forceinline__ static float2 unpack(const uint32_t *w) {
    return make_float2(__uint_as_float(w[0]), __uint_as_float(w[1]));
  }
  __device__ __forceinline__ static Val value(const Sell &A, uint64_t i) { return A.val[i]; }
  __device__ __forceinline__ static Val none() { return make_double2(0, 0); }
  __device__ __forceinline__ static Val half(Val v) { return make_double2(v.x * 0.5, v.y * 0.5); }
  __device__ __forceinline__ static Acc zero() { return make_double2(0, 0); }
  __device__ __forceinline__ static Acc minus(float2 y) {
    return make_double2(-(double)y.x, -(double)y.y);
  }
  __device__ __forceinline__ static Acc mac(Acc a, Val v, float2 x) {
    return cmac<false>(a, v, make_double2(x.x, x.y));
  }
  __device__ __forceinline__ static float2 stored(Acc a) {
    return make_float2(__double2float_rn(a.x), __double2float_rn(a.y));
  }
  __device__ __forceinline__ static double2 moment(Acc a) { return a; }
  __device__ __forceinline__ static double term(float2 a, float2 b) {
    return (double)fmaf(a.x, b.x, a.y * b.y);
  }
};
template <> struct ResKind<float> {  // real float vectors, FP64 arithmetic
  static constexpr bool SKIP = false;
  using Val = double;
  using Acc = double;
  __device__ __forceinline__ static float unpack(const uint32_t *w) {
    return __uint_as_float(w[0]);
  }
  __device__ __forceinline__ static Val value(const Sell &A, uint64_t i) { return A.vre[i]; }
  __device__ __forceinline__ static Val none() { return -0.0; }
  __device__ __forceinline__ static Val half(Val v) { return v * 0.5; }
  __device__ __forceinline__ static Acc zero() { return 0; }
  __device__ __forceinline__ static Acc minus(float y) { return -(double)y; }
  __device__ __forceinline__ static Acc mac(Acc a, Val v, float x) { return fma(v, (double)x, a); }
  __device__ __forceinline__ static float stored(Acc a) { return __double2float_rn(a); }
  __device__ __forceinline__ static double2 moment(Acc a) { return make_double2(a, 0.0); }
  __device__ __forceinline__ static double term(float a, float b) { return (double)fmaf(a, b, 0.0f); }
};

// The address of column c's row in x[0] (kPad: the block's zero row, marked
// with SKIP).
template <typename V, int COLS, bool CL>
__device__ __forceinline__ uint32_t res_address(uint32_t c, uint32_t xbase, uint32_t rows, uint32_t spb,
                                                uint32_t rank) {
  constexpr uint32_t BYTES = (uint32_t)sizeof(V) * COLS;
  uint32_t owner = rank, local = rows;
  if (c != kPad) {
    owner = (c >> 5) / spb;
    local = c - owner * rows;
  }
  const uint32_t a = xbase + local * BYTES;
  return (CL ? map_rank(a, owner) : a) | (c == kPad && ResKind<V>::SKIP ? kPadMark : 0u);
}

// Adds the first L of a row's entries (a, v) to acc: gathers first, then the
// products in order.  START: j_1 = (H/s) j_0 takes half of each value.
template <typename V, int COLS, bool START, bool CL, int L, int G>
__device__ __forceinline__ void res_round(const uint32_t (&a)[G], const typename ResKind<V>::Val (&v)[G],
                                          uint32_t off, typename ResKind<V>::Acc (&acc)[COLS]) {
  using K = ResKind<V>;
  constexpr int W = (int)sizeof(V) / 4;
  uint32_t w[L][W * COLS];
#pragma unroll
  for (int g = 0; g < L; g++) res_load<4 * W * COLS, CL>((K::SKIP ? a[g] & ~kPadMark : a[g]) + off, w[g]);
#pragma unroll
  for (int g = 0; g < L; g++) {
    typename K::Val u = v[g];
    if constexpr (START) u = K::half(u);
#pragma unroll
    for (int j = 0; j < COLS; j++) {
      const typename K::Acc t = K::mac(acc[j], u, K::unpack(w[g] + j * W));
      if (!K::SKIP || !(a[g] & kPadMark)) acc[j] = t;
    }
  }
}

// The same for the unrolled width that covers `len` entries (warp-uniform).
template <typename V, int COLS, bool START, bool CL, int G>
__device__ __forceinline__ void res_entries(uint32_t len, const uint32_t (&a)[G],
                                            const typename ResKind<V>::Val (&v)[G], uint32_t off,
                                            typename ResKind<V>::Acc (&acc)[COLS]) {
  if (len <= 4) res_round<V, COLS, START, CL, 4>(a, v, off, acc);
  else if (len == 5) res_round<V, COLS, START, CL, 5>(a, v, off, acc);
  else if (G > 7 && len <= 7) res_round<V, COLS, START, CL, G < 7 ? G : 7>(a, v, off, acc);
  else res_round<V, COLS, START, CL, G>(a, v, off, acc);
}

// Steps n0..n1 of one group of COLS columns per cluster.  CL: clusters of
// more than one block (blocks of one use plain shared memory and
// __syncthreads).
template <typename V, int COLS, bool DOTS, bool REG, bool CL>
__global__ void __launch_bounds__(32 * kResWarps, 1)
kpm_resident(ResidentArgs R) {
  using K = ResKind<V>;
  using Val = typename K::Val;
  using Acc = typename K::Acc;
  constexpr int BYTES = (int)sizeof(V) * COLS;
  constexpr int G = REG ? kResRegs : (sizeof(Val) * COLS <= 16 && BYTES <= 8 ? 9 : 5);  // gathers in flight
  extern __shared__ __align__(16) unsigned char res_smem[];
  const uint32_t warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank = 0, C = 1;
  if constexpr (CL) {
    rank = cluster_rank();
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(C));
  }
  const uint32_t group = blockIdx.x / C, groups = gridDim.x / C, c0 = group * COLS;
  const uint32_t rows = R.spb * 32;
  const ResLayout LY = resident_layout(R.spb, R.chunks, R.cap, warps, COLS, sizeof(V), sizeof(Val), REG, DOTS);
  V *xs = reinterpret_cast<V *>(res_smem);
  const uint32_t half = (rows + 4) * COLS, delta = half * (uint32_t)sizeof(V);
  Val *val = reinterpret_cast<Val *>(res_smem + LY.val);
  double2 *stage = reinterpret_cast<double2 *>(res_smem + LY.stage);
  double *dsum = reinterpret_cast<double *>(res_smem + LY.dsum);
  uint32_t *adr = reinterpret_cast<uint32_t *>(res_smem + LY.adr);
  uint32_t *bnd = reinterpret_cast<uint32_t *>(res_smem + LY.bnd);
  uint32_t *first = reinterpret_cast<uint32_t *>(res_smem + LY.first);
  uint32_t *tcol = reinterpret_cast<uint32_t *>(res_smem + LY.tcol);
  uint32_t *tout = reinterpret_cast<uint32_t *>(res_smem + LY.tout);
  uint32_t &s_nt = *reinterpret_cast<uint32_t *>(res_smem + LY.nt);
  const uint32_t s0 = min(rank * R.spb, R.A.nslices), s1 = min(s0 + R.spb, R.A.nslices), ns = s1 - s0;
  const uint32_t cb0 = __ldg(R.A.slice_ptr + s0), nch = __ldg(R.A.slice_ptr + s1) - cb0;
  const uint32_t xbase = (uint32_t)__cvta_generic_to_shared(xs);
  const uint32_t ta = target_first(R.tg, s0 * 32), tb = target_first(R.tg, s1 * 32);
  if (threadIdx.x == 0) s_nt = 0;
  // the block's rows of both vectors
  const V *gx = static_cast<const V *>(R.x), *gy = static_cast<const V *>(R.y);
  for (uint32_t i = threadIdx.x; i < rows + 4; i += blockDim.x) {
    const uint64_t r = (uint64_t)s0 * 32 + i;
    const bool live = i < ns * 32 && r < R.A.N;
#pragma unroll
    for (int j = 0; j < COLS; j++) {
      V a{}, b{};
      if (live) {
        a = gx[r * R.Bp + c0 + j];
        b = gy[r * R.Bp + c0 + j];
      }
      xs[(size_t)i * COLS + j] = a;
      xs[half + (size_t)i * COLS + j] = b;
    }
    if (i < rows) first[i] = kNoEntry;
  }
  __syncthreads();
  // The block's targets in this group, and the first one of each row.  Up to
  // `cap` of them are staged, in row order; more are stored step by step
  // instead (staged false, first[] counts in R.tg).  All threads look: one
  // alone took 0.1 us a target of the block's rows, whatever its column (2.6
  // ms before 64 sources with 512 targets each could start).
  for (uint32_t t = ta + threadIdx.x; t < tb; t += blockDim.x) {
    if (__ldg(R.tg.col + t) - c0 >= (uint32_t)COLS) continue;
    const uint32_t k = atomicAdd(&s_nt, 1u);
    if (k < R.cap) tout[k] = t;
    atomicMin(&first[__ldg(R.tg.row + t) - s0 * 32], t);
  }
  __syncthreads();
  const uint32_t nt = s_nt;
  const bool staged = nt <= R.cap;
  static_assert(kResTargets <= 64, "two targets per thread of a warp");
  uint32_t mine[2], rank_of[2];
  if (staged) {
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const uint32_t k = threadIdx.x + u * blockDim.x;
      mine[u] = k < nt ? tout[k] : kNoEntry;
      rank_of[u] = 0;
      if (k < nt)
        for (uint32_t j = 0; j < nt; j++) rank_of[u] += tout[j] < mine[u] ? 1u : 0u;
    }
  }
  __syncthreads();
  if (staged) {
    bool lead[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      lead[u] = false;
      if (mine[u] == kNoEntry) continue;
      lead[u] = first[__ldg(R.tg.row + mine[u]) - s0 * 32] == mine[u];
      tcol[rank_of[u]] = (__ldg(R.tg.col + mine[u]) - c0) | (lead[u] ? kTargetNew : 0u);
      tout[rank_of[u]] = __ldg(R.tg.out + mine[u]);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; u++)
      if (lead[u]) first[__ldg(R.tg.row + mine[u]) - s0 * 32] = rank_of[u];
  }
  uint32_t radr[REG ? kResRegs : 1];
  Val rval[REG ? kResRegs : 1];
  uint32_t rlen = 0;
  if constexpr (REG) {
    const uint32_t s = s0 + warp;
    const uint32_t cb = s < s1 ? __ldg(R.A.slice_ptr + s) : 0, ce = s < s1 ? __ldg(R.A.slice_ptr + s + 1) : 0;
    rlen = ce - cb;
#pragma unroll
    for (int g = 0; g < kResRegs; g++) {
      radr[g] = res_address<V, COLS, CL>(kPad, xbase, rows, R.spb, rank);
      rval[g] = K::none();
      if (cb + g < ce) {
        const uint64_t slot = (uint64_t)(cb + g) * 32 + lane;
        const uint32_t c = R.A.col[slot];
        radr[g] = res_address<V, COLS, CL>(c, xbase, rows, R.spb, rank);
        if (c != kPad) rval[g] = K::value(R.A, slot);
      }
    }
  } else {
    for (uint32_t i = threadIdx.x; i < nch * 32; i += blockDim.x) {
      const uint64_t slot = (uint64_t)cb0 * 32 + i;
      const uint32_t c = R.A.col[slot];
      adr[i] = res_address<V, COLS, CL>(c, xbase, rows, R.spb, rank);
      val[i] = c != kPad ? K::value(R.A, slot) : K::none();
    }
    for (uint32_t i = threadIdx.x; i <= ns; i += blockDim.x) bnd[i] = __ldg(R.A.slice_ptr + s0 + i) - cb0;
  }
  if constexpr (CL) cluster_arrive();
  block_or_cluster_wait<CL>();
  bool flagged = false;  // some row of this warp has a target
  for (uint32_t s = warp; s < ns; s += warps) flagged |= first[s * 32 + lane] != kNoEntry;
  flagged = __any_sync(0xffffffffu, flagged);

  uint32_t p = 0;  // x[p] holds j_{n-1}, x[p ^ 1] holds j_{n-2} and takes j_n
  for (uint32_t n = R.n0; n <= R.n1; n++) {
    const uint32_t off = p ? delta : 0u, slot = (n - R.n0) % kResRing;
    const V *xc = xs + (p ? half : 0u);
    V *yc = xs + (p ? 0u : half);
    double dn[DOTS ? COLS : 1], dp[DOTS ? COLS : 1];
#pragma unroll
    for (int j = 0; j < (DOTS ? COLS : 1); j++) dn[j] = dp[j] = 0.0;
    for (uint32_t s = warp; s < ns; s += warps) {
      const uint32_t i = s * 32 + lane;
      Acc acc[COLS];
#pragma unroll
      for (int j = 0; j < COLS; j++) acc[j] = n == 1 ? K::zero() : K::minus(yc[(size_t)i * COLS + j]);
      if constexpr (REG) {
        if (n == 1) res_entries<V, COLS, true, CL>(rlen, radr, rval, off, acc);
        else res_entries<V, COLS, false, CL>(rlen, radr, rval, off, acc);
      } else {
        const uint32_t cb = bnd[s], ce = bnd[s + 1];
        for (uint32_t k = cb; k < ce; k += G) {
          uint32_t a[G];
          Val v[G];
          const uint32_t pad = res_address<V, COLS, CL>(kPad, xbase, rows, R.spb, rank);
#pragma unroll
          for (int g = 0; g < G; g++) {
            a[g] = pad;
            v[g] = K::none();
            if (k + g < ce) {
              a[g] = adr[(k + g) * 32 + lane];
              v[g] = val[(k + g) * 32 + lane];
            }
          }
          if (n == 1) res_entries<V, COLS, true, CL>(ce - k, a, v, off, acc);
          else res_entries<V, COLS, false, CL>(ce - k, a, v, off, acc);
        }
      }
#pragma unroll
      for (int j = 0; j < COLS; j++) {
        const V o = K::stored(acc[j]);
        if constexpr (DOTS) {
          dn[j] += K::term(o, o);
          dp[j] += K::term(o, xc[(size_t)i * COLS + j]);
        }
        yc[(size_t)i * COLS + j] = o;
      }
      if (flagged) {
        const uint32_t f = first[i];
        if (f != kNoEntry) {
          if (staged) {
            for (uint32_t t = f; t < nt; t++) {
              if (t > f && first_of(tcol, t)) break;
#pragma unroll
              for (int j = 0; j < COLS; j++)
                if ((tcol[t] & kTargetCol) == (uint32_t)j) stage[slot * R.cap + t] = K::moment(acc[j]);
            }
          } else {
            const uint32_t r = s0 * 32 + i;
            // a row's targets are in column order
            for (uint32_t t = f; t < R.tg.count && __ldg(R.tg.row + t) == r; t++) {
              const uint32_t c = __ldg(R.tg.col + t) - c0;
              if (c >= (uint32_t)COLS) break;
#pragma unroll
              for (int j = 0; j < COLS; j++)
                if (c == (uint32_t)j)
                  R.tg.mu[(uint64_t)__ldg(R.tg.out + t) * R.tg.ld + n] = K::moment(acc[j]);
            }
          }
        }
      }
    }
    if constexpr (CL) cluster_arrive();
    if constexpr (DOTS) {
      // while the other blocks arrive: the warp's sums, in a fixed tree order
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int j = 0; j < COLS; j++) {
          dn[j] += __shfl_xor_sync(0xffffffffu, dn[j], o);
          dp[j] += __shfl_xor_sync(0xffffffffu, dp[j], o);
        }
      if (lane == 0) {
#pragma unroll
        for (int j = 0; j < COLS; j++) {
          dsum[(slot * warps + warp) * 2 * COLS + 2 * j] = dn[j];
          dsum[(slot * warps + warp) * 2 * COLS + 2 * j + 1] = dp[j];
        }
      }
    }
    block_or_cluster_wait<CL>();
    p ^= 1;
    if (slot + 1 == kResRing || n == R.n1) {
      // flush the last slot + 1 steps: moments, and the block's doubling sums
      // (the warps summed in order)
      __syncthreads();
      const uint32_t nf = n - slot, cnt = slot + 1;
      if (staged)
        for (uint32_t q = threadIdx.x; q < cnt * nt; q += blockDim.x) {
          const uint32_t t = q / cnt, d = q % cnt;
          R.tg.mu[(uint64_t)tout[t] * R.tg.ld + nf + d] = stage[d * R.cap + t];
        }
      if constexpr (DOTS)
        for (uint32_t q = threadIdx.x; q < cnt * 2 * COLS; q += blockDim.x) {
          const uint32_t d = q / (2 * COLS), e = q % (2 * COLS);
          double sum = 0;
          for (uint32_t w = 0; w < warps; w++) sum += dsum[(d * warps + w) * 2 * COLS + e];
          R.part[(((uint64_t)(nf + d - R.n0) * groups + group) * C + rank) * 2 * COLS + e] = sum;
        }
      __syncthreads();
    }
  }
  if (!R.keep) return;
  V *ox = static_cast<V *>(R.x), *oy = static_cast<V *>(R.y);
  const V *xc = xs + (p ? half : 0u), *yc = xs + (p ? 0u : half);
  for (uint32_t i = threadIdx.x; i < ns * 32; i += blockDim.x) {
    const uint64_t r = (uint64_t)s0 * 32 + i;
    if (r >= R.A.N) continue;
#pragma unroll
    for (int j = 0; j < COLS; j++) {
      ox[r * R.Bp + c0 + j] = xc[(size_t)i * COLS + j];
      oy[r * R.Bp + c0 + j] = yc[(size_t)i * COLS + j];
    }
  }
}

// Locality of a matrix's entries for the estimates of resident.cu: out[0] those
// not within two columns of the row before's entry of the same place,
// out[1 + 2c] those of them and out[2 + 2c] the others that another block owns
// when 2^c blocks share the slices.  A warp per slice.
static __global__ void __launch_bounds__(256)
k_locality(Sell A, uint32_t *out) {
  const uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (s >= A.nslices) return;
  const uint32_t k0 = __ldg(A.slice_ptr + s), k1 = __ldg(A.slice_ptr + s + 1);
  uint32_t n[11];
#pragma unroll
  for (int i = 0; i < 11; i++) n[i] = 0;
  for (uint32_t k = k0; k < k1; k++) {
    const uint32_t c = __ldg(A.col + (uint64_t)k * 32 + lane);
    const uint32_t before = __shfl_up_sync(0xffffffffu, c, 1);
    const bool live = c != kPad;
    const bool scattered = lane == 0 || before == kPad || c + 2 < before || c > before + 2;
    n[0] += __popc(__ballot_sync(0xffffffffu, live && scattered));
#pragma unroll
    for (int i = 0; i < 5; i++) {
      const uint32_t spb = (A.nslices + (1u << i) - 1) >> i;
      const bool away = live && (c >> 5) / spb != s / spb;
      n[1 + 2 * i] += __popc(__ballot_sync(0xffffffffu, away && scattered));
      n[2 + 2 * i] += __popc(__ballot_sync(0xffffffffu, away && !scattered));
    }
  }
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < 11; i++)
      if (n[i]) atomicAdd(out + i, n[i]);
}

// The doubled moments of steps n0.. from the blocks' sums of kpm_resident (as
// kpm_dots_finalize): one warp per (step, column), the sums in a fixed order.
static __global__ void __launch_bounds__(256)
kpm_resident_dots(uint32_t n0, uint32_t steps, uint32_t B, uint32_t groups, uint32_t cols, uint32_t parts,
                  const double *__restrict__ part, const uint32_t *__restrict__ col_out, double2 *mu,
                  uint32_t ld, uint32_t M) {
  const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t lane = threadIdx.x & 31;
  if (w >= (uint64_t)steps * B) return;
  const uint32_t c = (uint32_t)(w % B), i = (uint32_t)(w / B), m = n0 + i;
  const uint32_t slot = col_out[c];
  if (slot == kPad) return;
  const double *q = part + ((uint64_t)i * groups + c / cols) * parts * 2 * cols + 2 * (c % cols);
  double a = 0, b = 0;
  for (uint32_t k = lane; k < parts; k += 32) {
    a += q[(uint64_t)k * 2 * cols];
    b += q[(uint64_t)k * 2 * cols + 1];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if (lane) return;
  double2 *row = mu + (uint64_t)slot * ld;
  const double2 mu0 = row[0], mu1 = row[1];
  if (2 * m < M) row[2 * m] = make_double2(2.0 * a - mu0.x, -mu0.y);
  if (m >= 2 && 2 * m - 1 < M) row[2 * m - 1] = make_double2(2.0 * b - mu1.x, -mu1.y);
}

}  // namespace tbtkkpm
