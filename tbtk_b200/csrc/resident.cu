// Launches of the on-chip recursion of small matrices (kpm_resident.cuh) and
// the rule that decides when it runs and in which shape.
#include "tbtkkpm.h"
#include "kpm_host.h"
#include "kpm_resident.cuh"

#include <algorithm>
#include <cmath>
#include <mutex>

namespace tbtkkpm {

namespace {

using ResFn = void (*)(ResidentArgs);

template <typename V, int COLS, bool DOTS> ResFn pick_kernel(bool reg, bool cl) {
  if (reg) return cl ? kpm_resident<V, COLS, DOTS, true, true> : kpm_resident<V, COLS, DOTS, true, false>;
  return cl ? kpm_resident<V, COLS, DOTS, false, true> : kpm_resident<V, COLS, DOTS, false, false>;
}

template <typename V, int MAX, bool DOTS> ResFn pick_cols(uint32_t cols, bool reg, bool cl) {
  if constexpr (MAX >= 4)
    if (cols == 4) return pick_kernel<V, 4, DOTS>(reg, cl);
  if constexpr (MAX >= 2)
    if (cols == 2) return pick_kernel<V, 2, DOTS>(reg, cl);
  return pick_kernel<V, 1, DOTS>(reg, cl);
}

ResFn kernel_of(const ResidentPlan &p) {
  const bool cl = p.cluster > 1;
  switch (p.kind) {
    case kVecF64C: return pick_cols<double2, 1, false>(p.cols, p.reg, cl);
    case kVecF64R: return pick_cols<double, 2, false>(p.cols, p.reg, cl);
    case kVecC64:
      return p.dots ? pick_cols<float2, 2, true>(p.cols, p.reg, cl) : pick_cols<float2, 2, false>(p.cols, p.reg, cl);
    default:
      return p.dots ? pick_cols<float, 4, true>(p.cols, p.reg, cl) : pick_cols<float, 4, false>(p.cols, p.reg, cl);
  }
}

uint32_t max_cols(int kind) { return kind == kVecF32 ? 4 : kind == kVecF64C ? 1 : 2; }

}  // namespace

size_t vec_elem_size(int kind) {
  return kind == kVecF64C ? 16 : kind == kVecF32 ? 4 : 8;
}

static size_t value_size(int kind) { return kind == kVecF64C || kind == kVecC64 ? 16 : 8; }

// Fills the shape-dependent fields; false when a block's share does not fit.
static bool shape_resident(const tbtkkpm_matrix *m, const uint32_t *trow, const uint32_t *tcol, uint32_t T,
                           ResidentPlan &p) {
  const std::vector<uint32_t> &sp = m->host_slice_ptr;
  p.spb = (m->nslices + p.cluster - 1) / p.cluster;
  p.chunks = 0;
  for (uint32_t s = 0; s < m->nslices; s += p.spb)
    p.chunks = std::max(p.chunks, sp[std::min(s + p.spb, m->nslices)] - sp[s]);
  p.warps = std::min<uint32_t>(p.spb, kResWarps);
  // most targets of one block and group of columns
  std::vector<uint32_t> count((size_t)p.cluster * p.groups, 0u);
  p.cap = 0;
  for (uint32_t t = 0; t < T; t++)
    p.cap = std::max(p.cap, ++count[(size_t)(trow[t] / (p.spb * 32)) * p.groups + tcol[t] / p.cols]);
  if (p.cap > kResTargets) p.cap = 0;
  p.reg = p.spb <= p.warps && m->widest_slice <= (uint32_t)kResRegs;
  // (also keeps the layout's 32-bit offsets from wrapping)
  if (!p.reg && (uint64_t)p.chunks * 32 * (value_size(p.kind) + 4) > kResSmem) return false;
  p.smem = resident_layout(p.spb, p.chunks, p.cap, p.warps, p.cols, (uint32_t)vec_elem_size(p.kind),
                           (uint32_t)value_size(p.kind), p.reg, p.dots).bytes;
  return p.smem <= kResSmem;
}

static int kernel_attributes(ResFn fn, uint32_t cluster) {
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResSmem);
  if (e == cudaSuccess && cluster > 8)
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e == cudaSuccess ? TBTKKPM_OK : cuda_fail(e, "recursion: on-chip kernel");
}

static void launch_config(const ResidentPlan &p, cudaStream_t st, cudaLaunchConfig_t &cfg,
                          cudaLaunchAttribute &at) {
  cfg = cudaLaunchConfig_t{};
  cfg.gridDim = dim3(p.groups * p.cluster);
  cfg.blockDim = dim3(32 * p.warps);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = st;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = p.cluster;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = p.cluster > 1 ? 1 : 0;
}

// Groups that run at once.
static uint32_t resident_groups(const ResidentPlan &p, int device) {
  ResFn fn = kernel_of(p);
  int n = 0;
  cudaError_t e = cudaSuccess;
  if (kernel_attributes(fn, p.cluster)) return 0;
  if (p.cluster == 1) {
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, 32 * p.warps, p.smem);
    n *= sm_count(device);
  } else {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    launch_config(p, nullptr, cfg, at);
    e = cudaOccupancyMaxActiveClusters(&n, fn, &cfg);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return (uint32_t)std::max(n, 0);
}

// Microseconds of a step of `waves` waves of groups, fitted (1400 batches of 1 to
// 128 sources on square, Rashba, honeycomb and cubic lattices of 50 to 80k rows,
// all shapes) to nine in ten times within 13%, all within a third.  A fixed
// part (for a cluster more than half of it the barrier's release and a
// distributed-shared-memory round trip), the entries of a block, which cost
// shared-memory wavefronts unless they live in registers, more where several
// blocks share an SM, and the doubling sums.  Measured for FP64 real / complex,
// one source: 0.65 / 0.83 us at 512 rows, 0.74 / 0.93 at 1800, 0.80 / 1.2 at
// 8192; a batch of 128 sources of 1800 rows 2.1 / 4.3.
// A load from another block costs 1.3 ns a block and SM where the lanes of a
// warp reach scattered rows, a tenth of that where they reach neighbours
// (measured on the same lattices with their rows renumbered at random, where
// the estimate without it was a quarter of the time: 11k rows of 9 entries 11.2
// us a step, launched 6.2).
static double wave_us(const tbtkkpm_matrix *m, const ResidentPlan &p, uint32_t groups_at_once, uint32_t sms) {
  static const double base[2][4] = {{0.74, 0.45, 0.45, 0.52}, {0.49, 0.34, 0.64, 0.35}};
  static const double entry_ns[2][4] = {{0.168, 0.129, 0.205, 0.135}, {0.122, 0.044, 0.073, 0.044}};
  static const double wider[2][2] = {{1.26, 1.88}, {1.87, 3.78}};  // two and four columns
  static const double column[4] = {0.0, 0.09, 0.22, 0.086};
  const int reg = p.reg ? 1 : 0;
  const double blocks = std::min(std::ceil((double)p.groups * p.cluster / sms),
                                 (double)groups_at_once * p.cluster / sms);
  const double per_entry = entry_ns[reg][p.kind] * (p.cols == 1 ? 1.0 : wider[reg][p.cols == 4]) +
                           0.1 * std::max(blocks - 1, 0.0);
  double us = base[reg][p.kind] + (p.cluster > 1 ? 0.295 : 0.0) + 32e-3 * p.chunks * per_entry +
              column[p.kind] * (p.cols - 1);
  if (p.dots) us += 0.18 * (1 + 0.4 * (p.cols - 1));
  if (p.cap == 0) us += 1.2;  // moments stored step by step
  int c = 0;
  while ((1u << c) < p.cluster) c++;
  us += 1e-3 * m->nnz / p.cluster * (1.3 * m->far_scattered[c] + 0.13 * m->far_next[c]) * std::max(blocks, 1.0);
  return us * ((p.groups + groups_at_once - 1) / groups_at_once);
}

// The same for a dependent step of the launched kernels, by padded width:
// launch, round trips, rows and entries of the columns.  Nine in ten times
// within 14%, all within a third.  Measured at 1800 / 16k / 51k rows: FP64
// real, one source 3.2 / 3.2 / 2.6 us, 16 sources 3.9 / 4.4 / 5.9, 128 4.3 /
// 10.8 / 29; doubling steps, real, 1 source 2.9 / 2.9 / 3.1, 16 4.4 / 5.3 / 6.7,
// 128 6.5 / 11.8 / 23.
static double launch_us(const tbtkkpm_matrix *m, int kind, bool dots, uint32_t B) {
  struct Fit { double fixed, doubling, row, entry; };  // us, us per doubled width, ps per row and entry
  static const Fit direct[4] = {{2.7, 0.22, 2.3, 0.94}, {2.65, 0.25, 1.1, 0.45}, {2.81, 0.28, 0, 0.78}, {2.39, 0.26, 0.09, 0.42}};
  static const Fit doubled[2] = {{3.06, 0.38, 0, 0.87}, {2.73, 0.41, 0.74, 0.41}};
  const Fit &f = dots ? doubled[kind - kVecC64] : direct[kind];
  int log2w = 0;
  while ((1u << log2w) < B) log2w++;
  const double us = f.fixed + f.doubling * log2w +
                    1e-6 * (double)(1u << log2w) * (f.row * m->N + f.entry * 32.0 * m->chunks);
  // Scattered entries and long rows, which those lattices do not have, bring
  // it towards the register-staged step's, not all the way, since few batches
  // should leave the launched step for a slower one (6 of 575 do by more than a
  // tenth, at most 1.6 times; of 575 the choice is 3 to 8% from the better path on
  // average).
  const double share = std::max((m->scattered - 0.4) / 0.5, ((double)m->nnz / m->N - 10) / 20);
  if (share <= 0) return us;
  const int cls = kind <= kVecF64R ? 0 : kind == kVecC64 ? 1 + dots : 3 + dots;
  return us + 0.8 * std::min(share, 1.0) * std::max(register_us(m, cls, 1u << log2w) - us, 0.0);
}

int plan_resident(tbtkkpm_matrix *m, int kind, bool dots, uint32_t B, const uint32_t *trow,
                  const uint32_t *tcol, uint32_t T, ResidentPlan &out) {
  out = ResidentPlan{};
  if (m->nslices > kResMaxSlices || m->nslices == 0 || B == 0) return TBTKKPM_OK;
  // a handle with a wait bound of its own runs the steps whose waits it bounds
  if (m->wait_limit != TBTKKPM_WAIT_DEFAULT) return TBTKKPM_OK;
  if (m->host_slice_ptr.size() != (size_t)m->nslices + 1) {
    std::vector<uint32_t> sp((size_t)m->nslices + 1);
    ScratchBufs<1> scratch(m->stream);
    DevBuf &n = scratch.b[0];
    uint32_t hn[11];
    int rc = n.reserve(sizeof hn);
    if (rc) return rc;
    Sell A{};
    A.slice_ptr = m->slice_ptr.as<uint32_t>();
    A.col = m->scol.as<uint32_t>();
    A.N = m->N;
    A.nslices = m->nslices;
    cudaError_t e = cudaMemsetAsync(n.ptr, 0, sizeof hn, m->stream);
    if (e == cudaSuccess) {
      k_locality<<<(m->nslices + 7) / 8, 256, 0, m->stream>>>(A, n.as<uint32_t>());
      count_launches(1);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(sp.data(), m->slice_ptr.ptr, 4 * sp.size(), cudaMemcpyDeviceToHost, m->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(hn, n.ptr, sizeof hn, cudaMemcpyDeviceToHost, m->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    if (e != cudaSuccess) return cuda_fail(e, "recursion: slice bounds");
    const double all = (double)std::max<uint64_t>(m->nnz, 1);
    m->scattered = hn[0] / all;
    for (int i = 0; i < 5; i++) {
      m->far_scattered[i] = hn[1 + 2 * i] / all;
      m->far_next[i] = hn[2 + 2 * i] / all;
    }
    m->host_slice_ptr = std::move(sp);
  }
  // Below the launched step by a margin for the error of both estimates.  Over
  // those 1400 batches the rule's choice is within 5% of the launched step or
  // faster but for four (at most 1.16), and 0.6% from the best shape on average;
  // estimates of the steps before they were dependent launches sent batches on
  // chip that were up to 1.5 times faster launched (16k to 50k rows, 2-128
  // sources).
  double best = 0.95 * launch_us(m, kind, dots, B);
  for (uint32_t C = 1; C <= kResMaxCluster; C *= 2)
    for (uint32_t cols = 1; cols <= std::min(max_cols(kind), 2 * B - 1); cols *= 2) {
      ResidentPlan p{};
      p.kind = kind;
      p.dots = dots;
      p.cluster = C;
      p.cols = cols;
      p.groups = (B + cols - 1) / cols;
      if (!shape_resident(m, trow, tcol, T, p)) continue;
      if (wave_us(m, p, p.groups, p.groups * p.cluster) >= best) continue;  // at least that
      const uint64_t key = ((((uint64_t)kind * 2 + dots) * 32 + C) * 8 + cols) << 32 | p.smem;
      auto it = m->resident_groups.find(key);
      if (it == m->resident_groups.end()) {
        if (m->resident_groups.size() > 256) m->resident_groups.clear();
        it = m->resident_groups.emplace(key, resident_groups(p, m->device)).first;
      }
      if (it->second == 0) continue;
      const double us = wave_us(m, p, it->second, (uint32_t)sm_count(m->device));
      if (us >= best) continue;
      best = us;
      p.ok = true;
      out = p;
    }
  return TBTKKPM_OK;
}

int launch_resident(cudaStream_t st, int device, const ResidentPlan &p, const ResidentArgs &a) {
  ResFn fn = kernel_of(p);
  int rc = kernel_attributes(fn, p.cluster);
  if (rc) return rc;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at;
  launch_config(p, st, cfg, at);
  cudaError_t e = cudaLaunchKernelEx(&cfg, fn, a);
  if (e != cudaSuccess) return cuda_fail(e, "recursion: on-chip launch");
  count_launches(1);
  return TBTKKPM_OK;
}

void launch_resident_dots(cudaStream_t st, const ResidentPlan &p, uint32_t n0, uint32_t steps, uint32_t B,
                          const double *part, const uint32_t *col_out, double2 *mu, uint32_t ld, uint32_t M) {
  const uint64_t threads = (uint64_t)steps * B * 32;
  kpm_resident_dots<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(
      n0, steps, B, p.groups, p.cols, p.cluster, part, col_out, mu, ld, M);
  count_launches(1);
}

}  // namespace tbtkkpm
