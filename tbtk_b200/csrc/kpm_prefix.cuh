// FP64 head of a mixed-precision doubling run.
//
// The doubling identities mu_{2m} = 2<j_m|j_m> - mu_0 and
// mu_{2m-1} = 2<j_m|j_{m-1}> - mu_1 (the moments of the reference's
// recursion, Lib/src/Solver/ChebyshevExpander.cpp:150-190, taken from half
// as many steps) pick up the FP32 rounding of the recursion vectors through
// whole-vector dot products.  The rounding that matters is that of the first
// few dozen steps, while j_n still sits on the few rows around its source
// with entries of order one: with those steps in FP64 the largest relative
// LDOS error of the doubling path drops about fourfold (1.6e-6 -> 3.9e-7 on
// 1000-point windows of s = 12, M = 512-4096 square and honeycomb lattices).
//
// So one block per source computes j_0 .. j_q in FP64 on the rows they reach
// (the ball of radius q around the source in the matrix graph, which needs a
// structurally symmetric pattern), writes the moments of those steps, and the
// FP32 recursion starts from j_{q-1}, j_q rounded once.  The rows live in a
// per-block open-addressing table (row -> local index) in shared memory; every
// probe loop is bounded by the table size.  When the ball outgrows the table
// the block stops at the last complete step and reports it.  The dot products
// are summed in 64-bit fixed point (2^-61 units), so the moments do not depend
// on the order in which rows entered the table.
//
// A step is a chain of dependent loads and table probes, so they are spread
// thin: a row's entries are looked up only while it is new, one thread per
// entry; their local indices and values then lie in scratch, [entry][row],
// read together and coalesced; the three vectors of a real matrix lie in
// shared memory; 1024 threads share the rows.  Every entry looked up in every
// step by 256 threads took 0.59 ms for 32 steps on a square lattice and 1.4 ms
// on a Rashba lattice.
#pragma once

#include "kpm_kernels.cuh"

#include <algorithm>
#include <vector>

namespace tbtkkpm {

constexpr uint32_t kPrefixSteps = 32;      // FP64 steps of a doubling run's head
constexpr uint32_t kPrefixRows = 6144;     // rows of one source's ball
constexpr uint32_t kPrefixSlots = 8192;    // hash slots (power of two, above the rows)
constexpr uint32_t kPrefixSlotBits = 13;
constexpr uint32_t kPrefixEmpty = 0xffffffffu;
constexpr int kPrefixBlock = 1024;
constexpr int kPrefixWidth = 10;           // most entries of a row kept in scratch
constexpr uint16_t kPrefixNone = 0xffffu;  // an entry whose column is not in the ball
constexpr double kPrefixFix = 2305843009213693952.0;          // 2^61
constexpr double kPrefixUnit = 1.0 / 2305843009213693952.0;   // 2^-61
// shared memory of a block: key[slots] u32 | rows[rows] u32 | index[slots] u16
// | the vectors of a real matrix, v[3][rows] doubles (j_{n-1}, j_n, j_{n+1} in
// rotation)
constexpr size_t kPrefixTable = (size_t)kPrefixSlots * 4 + (size_t)kPrefixRows * 4 + (size_t)kPrefixSlots * 2;
__host__ __device__ constexpr size_t prefix_smem(bool real) { return kPrefixTable + (real ? 3 * (size_t)kPrefixRows * 8 : 0); }
// global scratch of a source: values [lists][rows], complex vectors
// v[3][rows], local indices [lists][rows] u16, with `lists` the widest slice of
// up to kPrefixWidth entries among the sources' matrices: 0.31 MB on a square
// lattice, 1.29 on a Rashba one
__host__ __device__ constexpr size_t prefix_scratch(bool real, uint32_t lists) {
  return (size_t)lists * kPrefixRows * ((real ? 8 : 16) + 2) + (real ? 0 : 3 * (size_t)kPrefixRows * 16);
}

struct PrefixJob {
  const uint32_t *slice_ptr;  // the source's matrix (SELL-32 of 2H/s)
  const uint32_t *scol;
  const double2 *sval;
  uint32_t site;        // source row (and the moments' target row)
  uint32_t steps;       // j_0 .. j_steps wanted
  uint32_t M;           // doubled moments written for n < M
  uint32_t ld;          // direct moments written for n < ld
  double2 *mu;          // doubled-moment row
  double2 *mu_direct;   // direct-moment row
  void *x_cur, *x_prev; // [rows][W] buffers that take j_q and j_{q-1}
  uint32_t W, col;      // row stride and column of the source
  uint32_t real;        // buffers hold real floats (else complex64)
  uint32_t width;       // the matrix's widest slice
};

// Result of one source: the last step computed (q) and the rows used.
struct PrefixResult {
  uint32_t q, count;
};

__device__ __forceinline__ uint32_t prefix_hash(uint32_t row) {
  return (row * 2654435761u) >> (32 - kPrefixSlotBits);
}

__device__ __forceinline__ int prefix_find(const uint32_t *key, const uint16_t *index, uint32_t row) {
  uint32_t h = prefix_hash(row);
  for (uint32_t p = 0; p < kPrefixSlots; p++) {
    const uint32_t k = key[h];
    if (k == row) return (int)index[h];
    if (k == kPrefixEmpty) return -1;
    h = (h + 1) & (kPrefixSlots - 1);
  }
  return -1;
}

// Element of a source's vectors: double for a real matrix (the complex sums
// then only add zeros to the real parts), double2 otherwise.
template <bool REAL> struct PrefixVec {
  using T = double;
  __device__ __forceinline__ static T value(double2 a) { return a.x; }
  __device__ __forceinline__ static T zero() { return 0.0; }
  __device__ __forceinline__ static T one() { return 1.0; }
  __device__ __forceinline__ static T mac(T acc, T a, T b) { return fma(a, b, acc); }
  __device__ __forceinline__ static T half(T a) { return a * 0.5; }
  __device__ __forceinline__ static T minus(T a, T b) { return a - b; }
  __device__ __forceinline__ static double dot(T a, T b) { return a * b; }
  __device__ __forceinline__ static double2 wide(T a) { return make_double2(a, 0.0); }
};
template <> struct PrefixVec<false> {
  using T = double2;
  __device__ __forceinline__ static T value(double2 a) { return a; }
  __device__ __forceinline__ static T zero() { return make_double2(0.0, 0.0); }
  __device__ __forceinline__ static T one() { return make_double2(1.0, 0.0); }
  __device__ __forceinline__ static T mac(T acc, T a, T b) { return cmac<false>(acc, a, b); }
  __device__ __forceinline__ static T half(T a) { return make_double2(a.x * 0.5, a.y * 0.5); }
  __device__ __forceinline__ static T minus(T a, T b) { return make_double2(a.x - b.x, a.y - b.y); }
  __device__ __forceinline__ static double dot(T a, T b) { return fma(a.x, b.x, a.y * b.y); }
  __device__ __forceinline__ static double2 wide(T a) { return a; }
};

// Enters `row` into the table unless present and returns its slot if it is
// new (its local index is given out afterwards), kPrefixSlots if it was there,
// kPrefixSlots + 1 when no slot is free.
__device__ __forceinline__ uint32_t prefix_enter(uint32_t *key, uint32_t row) {
  uint32_t h = prefix_hash(row);
  for (uint32_t p = 0; p < kPrefixSlots; p++) {
    const uint32_t prev = atomicCAS(key + h, kPrefixEmpty, row);
    if (prev == row) return kPrefixSlots;
    if (prev == kPrefixEmpty) return h;
    h = (h + 1) & (kPrefixSlots - 1);
  }
  return kPrefixSlots + 1;
}

// One block per source (prefix_smem bytes of dynamic shared memory).
// j_1 = (H/s) j_0 takes half of the stored 2H/s (exact), later steps
// j_{n+1} = (2H/s) j_n - j_{n-1}; every product and sum in FP64 (fma), rows
// in the matrix's entry order.  With q >= 2 steps done, the block writes
// j_q and j_{q-1} into its column of the two recursion buffers (zero
// elsewhere beforehand), rounded once to FP32.
template <bool REAL>
__global__ void __launch_bounds__(kPrefixBlock, 1)
kpm_prefix(const PrefixJob *__restrict__ jobs, char *scratch, uint32_t lists, PrefixResult *res) {
  using V = PrefixVec<REAL>;
  using T = typename V::T;
  constexpr int L = 5;  // entries loaded together
  extern __shared__ __align__(16) unsigned char prefix_mem[];
  __shared__ uint32_t s_count, s_over;
  __shared__ long long red[2][kPrefixBlock / 32];
  const PrefixJob &J = jobs[blockIdx.x];
  uint32_t *key = reinterpret_cast<uint32_t *>(prefix_mem);
  uint32_t *rows = key + kPrefixSlots;
  uint16_t *index = reinterpret_cast<uint16_t *>(rows + kPrefixRows);
  char *mine = scratch + (size_t)blockIdx.x * prefix_scratch(REAL, lists);
  T *val = reinterpret_cast<T *>(mine);
  T *v = REAL ? reinterpret_cast<T *>(index + kPrefixSlots) : val + (size_t)lists * kPrefixRows;
  uint16_t *nbr = reinterpret_cast<uint16_t *>(val + (size_t)(lists + (REAL ? 0 : 3)) * kPrefixRows);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool listed = J.width <= lists;
  for (uint32_t i = threadIdx.x; i < kPrefixSlots; i += kPrefixBlock) key[i] = kPrefixEmpty;
  if (threadIdx.x == 0) {
    s_count = 0;
    s_over = 0;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    index[prefix_enter(key, J.site)] = 0;
    rows[0] = J.site;
    s_count = 1;
    v[0] = V::one();
    v[kPrefixRows] = v[2 * kPrefixRows] = V::zero();
    if (J.M > 0) J.mu[0] = make_double2(1.0, 0.0);
    if (J.ld > 0) J.mu_direct[0] = make_double2(1.0, 0.0);
  }
  __syncthreads();
  uint32_t f0 = 0, f1 = 1, q = 0;
  double2 mu1 = make_double2(0.0, 0.0);
  for (uint32_t n = 0; n < J.steps; n++) {
    // Rows of the next ball: neighbours of the last step's new rows.  A new
    // row gets the next local index and zero values in all three vectors; a
    // warp takes the indices of its lanes' new rows at once.  Past kPrefixRows,
    // or with no free slot, s_over is set instead, and the step, which is then
    // dropped, ends at a warp's next look at it, before the table is full.
    auto enter = [&](uint32_t c) {  // a column per lane, or kPad
      const uint32_t at = c != kPad ? prefix_enter(key, c) : kPrefixSlots;
      if (at > kPrefixSlots) s_over = 1;
      const uint32_t fresh = __ballot_sync(0xffffffffu, at < kPrefixSlots);
      uint32_t base = 0;
      if (lane == 0 && fresh) base = atomicAdd(&s_count, (uint32_t)__popc(fresh));
      const uint32_t id = __shfl_sync(0xffffffffu, base, 0) + __popc(fresh & ((1u << lane) - 1u));
      if (at < kPrefixSlots) {
        if (id < kPrefixRows) {
          index[at] = (uint16_t)id;
          rows[id] = c;
          v[id] = v[kPrefixRows + id] = v[2 * kPrefixRows + id] = V::zero();
        } else {
          s_over = 1;
        }
      }
    };
    auto over = [&]() { return __any_sync(0xffffffffu, *(volatile uint32_t *)&s_over != 0); };
    if (listed) {
      // a thread per (row, entry): at most kPrefixRows * kPrefixWidth of them
      const uint32_t count = (f1 - f0) * J.width;
      for (uint32_t b = 32 * warp; b < count && !over(); b += kPrefixBlock) {
        const uint32_t t = b + lane, i = f0 + t / J.width, k = t % J.width;
        uint32_t c = kPad;
        if (t < count) {
          const uint32_t r = rows[i], s = r >> 5;
          const uint32_t cb = __ldg(J.slice_ptr + s), ce = __ldg(J.slice_ptr + s + 1);
          if (cb + k < ce) c = __ldg(J.scol + (uint64_t)(cb + k) * 32 + (r & 31));
        }
        enter(c);
      }
    } else {
      // A warp per row up to the row's own last entry: one long row of the
      // matrix makes J.width thousands where a row of the ball has a few (a
      // row of 5000 entries outside the ball: walking J.width positions per
      // row took 3.7 ms a head, this 0.41).
      for (uint32_t i = f0 + warp; i < f1; i += kPrefixBlock / 32) {
        const uint32_t r = rows[i], s = r >> 5;
        const uint32_t cb = __ldg(J.slice_ptr + s), ce = __ldg(J.slice_ptr + s + 1);
        for (uint32_t k = cb; k < ce && !over(); k += 32) {
          const uint32_t c =
              lane < ce - k ? __ldg(J.scol + ((uint64_t)k + lane) * 32 + (r & 31)) : kPad;
          enter(c);
          if (__any_sync(0xffffffffu, c == kPad)) break;
        }
      }
    }
    __syncthreads();
    if (s_over) break;
    const uint32_t cnt = s_count;
    // The entries of the rows from f0 on: the neighbours of the rows before
    // f1 are all in the table by now, of the newest only some (the others are
    // zero), so those are looked up once more next step.
    if (listed) {
      const uint32_t look = (cnt - f0) * J.width;
      for (uint32_t t = threadIdx.x; t < look; t += kPrefixBlock) {
        const uint32_t i = f0 + t / J.width, k = t % J.width;
        const uint32_t r = rows[i], s = r >> 5;
        const uint32_t cb = __ldg(J.slice_ptr + s), ce = __ldg(J.slice_ptr + s + 1);
        int j = -1;
        if (cb + k < ce) {
          const uint64_t slot = (uint64_t)(cb + k) * 32 + (r & 31);
          const uint32_t c = __ldg(J.scol + slot);
          const double2 a = __ldg(J.sval + slot);
          if (c != kPad) j = prefix_find(key, index, c);
          if (j >= 0) val[(size_t)k * kPrefixRows + i] = V::value(a);
        }
        nbr[(size_t)k * kPrefixRows + i] = j < 0 ? kPrefixNone : (uint16_t)j;
      }
      __syncthreads();
    }
    const T *x = v + (size_t)(n % 3) * kPrefixRows;
    const T *y = v + (size_t)((n + 2) % 3) * kPrefixRows;
    T *out = v + (size_t)((n + 1) % 3) * kPrefixRows;
    long long sa = 0, sb = 0;
    for (uint32_t i = threadIdx.x; i < cnt; i += kPrefixBlock) {
      T acc = V::zero();
      if (listed) {
        for (uint32_t k = 0; k < J.width; k += L) {
          uint16_t nb[L];
          T a[L];
#pragma unroll
          for (int g = 0; g < L; g++) {
            nb[g] = kPrefixNone;
            if (k + g < J.width) {
              nb[g] = nbr[(size_t)(k + g) * kPrefixRows + i];
              a[g] = val[(size_t)(k + g) * kPrefixRows + i];
            }
          }
#pragma unroll
          for (int g = 0; g < L; g++)
            if (nb[g] != kPrefixNone) acc = V::mac(acc, a[g], x[nb[g]]);
        }
      } else {
        const uint32_t r = rows[i], s = r >> 5, l = r & 31;
        const uint32_t cb = __ldg(J.slice_ptr + s), ce = __ldg(J.slice_ptr + s + 1);
        for (uint32_t k = cb; k < ce; k++) {
          const uint64_t slot = (uint64_t)k * 32 + l;
          const uint32_t c = __ldg(J.scol + slot);
          if (c == kPad) break;  // padding ends a row
          const int j = prefix_find(key, index, c);
          if (j >= 0) acc = V::mac(acc, V::value(__ldg(J.sval + slot)), x[j]);
        }
      }
      acc = n == 0 ? V::half(acc) : V::minus(acc, y[i]);
      out[i] = acc;
      sa += __double2ll_rn(V::dot(acc, acc) * kPrefixFix);
      sb += __double2ll_rn(V::dot(acc, x[i]) * kPrefixFix);
    }
    for (int o = 16; o > 0; o >>= 1) {
      sa += __shfl_down_sync(0xffffffffu, sa, o);
      sb += __shfl_down_sync(0xffffffffu, sb, o);
    }
    if (lane == 0) {
      red[0][warp] = sa;
      red[1][warp] = sb;
    }
    __syncthreads();
    if (warp == 0) {
      long long ta = red[0][lane], tb = red[1][lane];
      for (int o = 16; o > 0; o >>= 1) {
        ta += __shfl_down_sync(0xffffffffu, ta, o);
        tb += __shfl_down_sync(0xffffffffu, tb, o);
      }
      if (lane == 0) {
        const uint32_t m = n + 1;
        const double2 d = V::wide(out[0]);  // the source row has local index 0
        if (m < J.ld) J.mu_direct[m] = d;
        if (m == 1) {
          mu1 = d;
          if (J.M > 1) J.mu[1] = d;
        }
        const double a = (double)ta * kPrefixUnit, b = (double)tb * kPrefixUnit;
        if (2 * m < J.M) J.mu[2 * m] = make_double2(2.0 * a - 1.0, -0.0);
        if (m >= 2 && 2 * m - 1 < J.M) J.mu[2 * m - 1] = make_double2(2.0 * b - mu1.x, -mu1.y);
      }
    }
    q = n + 1;
    f0 = f1;
    f1 = cnt;
  }
  __syncthreads();
  const uint32_t count = min(s_count, kPrefixRows);
  if (threadIdx.x == 0) res[blockIdx.x] = {q, count};
  if (q < 2) return;
  const T *cur = v + (size_t)(q % 3) * kPrefixRows;
  const T *prev = v + (size_t)((q - 1) % 3) * kPrefixRows;
  for (uint32_t i = threadIdx.x; i < count; i += kPrefixBlock) {
    const uint64_t o = (uint64_t)rows[i] * J.W + J.col;
    const double2 c = V::wide(cur[i]), p = V::wide(prev[i]);
    if (REAL || J.real) {
      static_cast<float *>(J.x_cur)[o] = __double2float_rn(c.x);
      static_cast<float *>(J.x_prev)[o] = __double2float_rn(p.x);
    } else {
      static_cast<float2 *>(J.x_cur)[o] = make_float2(__double2float_rn(c.x), __double2float_rn(c.y));
      static_cast<float2 *>(J.x_prev)[o] = make_float2(__double2float_rn(p.x), __double2float_rn(p.y));
    }
  }
}

// Structural symmetry of a CSR pattern (every (r, c) has a (c, r)), which
// the ball of kpm_prefix relies on.  Rows longer than kPrefixRows count as a
// failure (their scan is not done and such a ball would not fit anyway).
static __global__ void k_pattern_check(uint32_t N, const uint32_t *__restrict__ rowptr,
                                       const uint32_t *__restrict__ col, unsigned *flag) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= N) return;
  const uint32_t e0 = rowptr[r], e1 = rowptr[r + 1];
  if (e1 - e0 > kPrefixRows) {
    atomicOr(flag, 1u);
    return;
  }
  for (uint32_t e = e0; e < e1; e++) {
    const uint32_t c = col[e];
    if (c >= N) {
      atomicOr(flag, 1u);
      return;
    }
    const uint32_t f0 = rowptr[c], f1 = rowptr[c + 1];
    if (f1 - f0 > kPrefixRows) {
      atomicOr(flag, 1u);
      return;
    }
    bool found = false;
    for (uint32_t f = f0; f < f1 && !found; f++) found = col[f] == r;
    if (!found) {
      atomicOr(flag, 1u);
      return;
    }
  }
}

}  // namespace tbtkkpm

#include "kpm_host.h"

namespace tbtkkpm {

// Runs the FP64 head of `jobs` on stream st, those with real buffers apart from
// the others; every source with q >= 2 leaves j_q and j_{q-1} in its buffers.
// res[i] receives the steps source i reached and its rows.  A launch takes as
// many sources as run at once, a block per SM, and the next one reuses their
// scratch; fewer when that cannot be allocated.  Returns after the stream has
// passed the last launch.
static int run_fp64_head(cudaStream_t st, int device, const std::vector<PrefixJob> &jobs, Workspace &ws,
                         std::vector<PrefixResult> &res) {
  const size_t nj = jobs.size();
  res.assign(nj, PrefixResult{0, 0});
  if (nj == 0) return 0;
  std::vector<uint32_t> order(nj);  // the real jobs first
  size_t nreal = 0;
  for (size_t i = 0; i < nj; i++)
    if (jobs[i].real) order[nreal++] = (uint32_t)i;
  for (size_t i = 0, k = nreal; i < nj; i++)
    if (!jobs[i].real) order[k++] = (uint32_t)i;
  std::vector<PrefixJob> sorted(nj);
  uint32_t lists[2] = {0, 0};  // complex, real
  for (size_t i = 0; i < nj; i++) {
    sorted[i] = jobs[order[i]];
    uint32_t &l = lists[i < nreal];
    if (sorted[i].width <= (uint32_t)kPrefixWidth) l = std::max(l, sorted[i].width);
  }
  int rc;
  if ((rc = ws.head_jobs.reserve(sizeof(PrefixJob) * nj)) || (rc = ws.head_res.reserve(sizeof(PrefixResult) * nj)))
    return rc;
  const size_t most = std::max(nreal, nj - nreal);
  size_t chunk = std::min<size_t>(most, std::max(sm_count(device), 1));
  for (;; chunk = (chunk + 1) / 2) {
    rc = ws.head.reserve(std::max(nreal ? prefix_scratch(true, lists[1]) * std::min(nreal, chunk) : 0,
                                  nreal < nj ? prefix_scratch(false, lists[0]) * std::min(nj - nreal, chunk) : 0));
    if (!rc) break;
    cudaGetLastError();
    if (chunk == 1) return rc;
  }
  cudaError_t e = cudaFuncSetAttribute(kpm_prefix<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)prefix_smem(true));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kpm_prefix<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)prefix_smem(false));
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(ws.head_jobs.ptr, sorted.data(), sizeof(PrefixJob) * nj, cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return cuda_fail(e, "fp64 head: jobs");
  uint64_t launches = 0;
  for (size_t j0 = 0; j0 < nj; launches++) {
    const bool real = j0 < nreal;
    const size_t n = std::min((real ? nreal : nj) - j0, chunk);
    auto kern = real ? kpm_prefix<true> : kpm_prefix<false>;
    kern<<<(unsigned)n, kPrefixBlock, prefix_smem(real), st>>>(ws.head_jobs.as<PrefixJob>() + j0, ws.head.as<char>(),
                                                               lists[real], ws.head_res.as<PrefixResult>() + j0);
    j0 += n;
  }
  count_launches(launches);
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "fp64 head: launch");
  std::vector<PrefixResult> got(nj);
  e = cudaMemcpyAsync(got.data(), ws.head_res.ptr, sizeof(PrefixResult) * nj, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cuda_fail(e, "fp64 head");
  for (size_t i = 0; i < nj; i++) res[order[i]] = got[i];
  return 0;
}

}  // namespace tbtkkpm
