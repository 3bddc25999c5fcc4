// Launches of the on-chip recursion of small matrices (kpm_resident.cuh) and
// the rule that decides when it runs and in which shape.
#include "tbtkkpm.h"
#include "kpm_host.h"
#include "kpm_resident.cuh"

#include <algorithm>
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

// Microseconds of a step of one wave of groups, fitted to slopes over 200 to
// 2000 moments on square, Rashba and honeycomb lattices of 128 to 32k rows:
// a fixed part (for a cluster more than half of it the barrier's release and
// a distributed-shared-memory round trip) and the entries of a block, which
// cost shared-memory wavefronts unless they live in registers.  Measured for
// FP64 real / complex, one source: 0.43 / 0.67 us at 512 rows, 0.56 / 0.71 at
// 1800, 0.65 / 0.85 at 8192; doubling steps 0.61 / 0.71 / 0.79; a batch of 128
// sources of 1800 rows 1.7 / 3.6.
static double wave_us(const ResidentPlan &p) {
  static const double block0[4] = {0.42, 0.30, 0.45, 0.32}, reg0[4] = {0.68, 0.56, 0.72, 0.58};
  static const double smem_ns[4] = {0.22, 0.14, 0.18, 0.15}, reg_ns[4] = {0.07, 0.04, 0.08, 0.045};
  const double fixed = (p.cluster == 1 ? block0[p.kind] : p.reg ? reg0[p.kind] : 0.45) + (p.dots ? 0.17 : 0.0);
  const double per_entry = (p.reg ? reg_ns : smem_ns)[p.kind] * 1e-3 *
                           (p.cols == 1 ? 1.0 : p.cols == 2 ? 1.15 : 1.5);
  return fixed + 32.0 * p.chunks * per_entry;
}

// The same for a step of the launched kernels: launch latency, dependent
// round trips and the fewest bytes at 5 TB/s (us measured at 2k-64k rows: 4.1
// to 5.1 for one source, 6.2 to 10 for a batch; the doubling step is two
// launches, 10.3 to 37).
static double launch_us(const tbtkkpm_matrix *m, int kind, bool dots, uint32_t B) {
  const double bytes = 32.0 * m->chunks * (value_size(kind) + 4) + 3.0 * m->N * B * vec_elem_size(kind);
  return (B == 1 ? 4.0 : 5.5) + (dots ? 3.0 : 0.0) + bytes / 5e6;
}

int plan_resident(tbtkkpm_matrix *m, int kind, bool dots, uint32_t B, const uint32_t *trow,
                  const uint32_t *tcol, uint32_t T, ResidentPlan &out) {
  out = ResidentPlan{};
  if (m->nslices > kResMaxSlices || m->nslices == 0 || B == 0) return TBTKKPM_OK;
  // a handle with a wait bound of its own runs the steps whose waits it bounds
  if (m->wait_limit != TBTKKPM_WAIT_DEFAULT) return TBTKKPM_OK;
  if (m->host_slice_ptr.size() != (size_t)m->nslices + 1) {
    std::vector<uint32_t> sp((size_t)m->nslices + 1);
    cudaError_t e = cudaMemcpyAsync(sp.data(), m->slice_ptr.ptr, 4 * sp.size(), cudaMemcpyDeviceToHost,
                                    m->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    if (e != cudaSuccess) return cuda_fail(e, "recursion: slice bounds");
    m->host_slice_ptr = std::move(sp);
  }
  // a tenth below the launched step, for the error of both estimates
  double best = 0.9 * launch_us(m, kind, dots, B);
  for (uint32_t C = 1; C <= kResMaxCluster; C *= 2)
    for (uint32_t cols = 1; cols <= std::min(max_cols(kind), 2 * B - 1); cols *= 2) {
      ResidentPlan p{};
      p.kind = kind;
      p.dots = dots;
      p.cluster = C;
      p.cols = cols;
      p.groups = (B + cols - 1) / cols;
      if (!shape_resident(m, trow, tcol, T, p)) continue;
      if (wave_us(p) >= best) continue;
      const uint64_t key = ((((uint64_t)kind * 2 + dots) * 32 + C) * 8 + cols) << 32 | p.smem;
      auto it = m->resident_groups.find(key);
      if (it == m->resident_groups.end()) {
        if (m->resident_groups.size() > 256) m->resident_groups.clear();
        it = m->resident_groups.emplace(key, resident_groups(p, m->device)).first;
      }
      if (it->second == 0) continue;
      const uint32_t waves = (p.groups + it->second - 1) / it->second;
      const double us = wave_us(p) * (waves == 1 ? 1.0 : 1.1 * waves);
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
