// Launchers of the batched stage kernels, shared by the exact translation
// unit (clv_batch.cu) and the tolerance-arithmetic one (clv_fast.cu): each
// instantiates the kernels of its own arithmetic (clv::exact or clv::fast).
#pragma once
#include <algorithm>
#include <string>

#include "clv_batch.cuh"

namespace clv_host {
int set_error(int code, const std::string& msg);
int check_cuda(const char* where);
}  // namespace clv_host

namespace clv {
inline namespace CLV_ARITH {
namespace batch_launch {

// the current device (launch set-up is cached per device), or -1
constexpr int kMaxDevices = 64;
inline int current_device() {
  int d = 0;
  return (cudaGetDevice(&d) == cudaSuccess && d >= 0 && d < kMaxDevices) ? d : -1;
}

template <class real, bool BULK, int BS, int MINB>
int launch_stage(const Params& p, const BatchArgs<real>& a, int step, int grid, cudaStream_t s) {
  auto kern = batch_stage_kernel<real, BULK, BS, MINB>;
  if (grid <= 0) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, BS, 0);
    grid = sms * (per_sm > 0 ? per_sm : 1);
  }
  kern<<<grid, BS, 0, s>>>(p, a, step);
  return clv_host::check_cuda("batch_stage_kernel");
}

// the register caps are offered in FP32 only (FP64 spills heavily under
// them): 128 registers a thread (512 threads per SM) or, for 64- and
// 128-thread blocks, 168 (384 threads per SM)
template <class real> constexpr int capped_minb(int bs) { return sizeof(real) == 4 ? 512 / bs : 1; }
template <class real> constexpr int capped168_minb(int bs) { return sizeof(real) == 4 ? 384 / bs : 1; }

template <class real, bool BULK>
int stage_bs(const Params& p, const BatchArgs<real>& a, int step, int bs, int grid, int cap,
             cudaStream_t s) {
  if (cap && sizeof(real) == 8) return clv_host::set_error(CLV_ERR_INVALID, "batch: max_registers is FP32 only");
  if (cap == 168 && bs == 256)
    return clv_host::set_error(CLV_ERR_INVALID, "batch: max_registers 168 needs 64- or 128-thread blocks");
  if (bs == 64 && cap == 168) return launch_stage<real, BULK, 64, capped168_minb<real>(64)>(p, a, step, grid, s);
  if (bs == 128 && cap == 168) return launch_stage<real, BULK, 128, capped168_minb<real>(128)>(p, a, step, grid, s);
  if (bs == 64)
    return cap ? launch_stage<real, BULK, 64, capped_minb<real>(64)>(p, a, step, grid, s)
               : launch_stage<real, BULK, 64, 1>(p, a, step, grid, s);
  if (bs == 128)
    return cap ? launch_stage<real, BULK, 128, capped_minb<real>(128)>(p, a, step, grid, s)
               : launch_stage<real, BULK, 128, 1>(p, a, step, grid, s);
  if (bs == 256)
    return cap ? launch_stage<real, BULK, 256, capped_minb<real>(256)>(p, a, step, grid, s)
               : launch_stage<real, BULK, 256, 1>(p, a, step, grid, s);
  return clv_host::set_error(CLV_ERR_INVALID, "batch: block_size must be 64, 128 or 256");
}

// resident blocks per SM of the stage kernel of one launch shape (this also
// loads the kernel and, for the tiled one, raises its shared-memory limit, so
// that a later stream capture needs neither)
template <class real, bool BULK>
int occupancy(int bs, int cap, int* n) {
  const void* f = nullptr;
  if (bs == 64) f = cap == 168 ? (const void*)batch_stage_kernel<real, BULK, 64, capped168_minb<real>(64)>
                 : cap ? (const void*)batch_stage_kernel<real, BULK, 64, capped_minb<real>(64)>
                       : (const void*)batch_stage_kernel<real, BULK, 64, 1>;
  else if (bs == 128) f = cap == 168 ? (const void*)batch_stage_kernel<real, BULK, 128, capped168_minb<real>(128)>
                     : cap ? (const void*)batch_stage_kernel<real, BULK, 128, capped_minb<real>(128)>
                           : (const void*)batch_stage_kernel<real, BULK, 128, 1>;
  else f = cap ? (const void*)batch_stage_kernel<real, BULK, 256, capped_minb<real>(256)>
               : (const void*)batch_stage_kernel<real, BULK, 256, 1>;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, f, bs, 0) != cudaSuccess)
    return clv_host::check_cuda("batch_occupancy");
  return 0;
}
// resident blocks an SM (the pointers of the event at hand take registers: at
// five blocks the FP32 kernel spills 150 bytes)
constexpr int kPatchBlocks = 4;
// the (2+1)D stage by patches: its two kernels, loaded, and their resident
// blocks per SM
template <class real, bool BULK> int occupancy_patch(int* n) {
  typedef PatchWide<real, BULK> W;
  typedef PatchSmem<real, BULK, W::TX, W::TY> SM;
  auto k1 = batch_patch_kernel<real, BULK, W::TX, W::TY, W::NT, kPatchBlocks, 1>;
  auto k2 = batch_patch_kernel<real, BULK, W::TX, W::TY, W::NT, kPatchBlocks, 2>;
  for (auto k : {k1, k2})
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SM)) != cudaSuccess)
      return clv_host::check_cuda("cudaFuncSetAttribute(batch_patch_kernel)");
  int a = 0, b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k1, W::NT, sizeof(SM)) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k2, W::NT, sizeof(SM)) != cudaSuccess)
    return clv_host::check_cuda("batch_occupancy_tiled");
  *n = std::min(a, b);
  return 0;
}
// A persistent grid: the patches of `grid` strips of (rows - 4) x chunk cells, at
// most the blocks that fit the GPU at once (<= 0: those). One patch is short work
// and blocks of one wave pick up where they leave off; with a block for every few
// patches the waves' ends cost 15 %. Launch shapes count strips: taken as blocks,
// four events of 121 x 121 to 151 x 149 ran on 108 of 592 blocks, 1.81 ms for 20
// steps against 1.00.
template <class real, bool BULK>
int stage_patch(const Params& p, const BatchArgs<real>& a, int step, int rows, int chunk, int grid, cudaStream_t s) {
  typedef PatchWide<real, BULK> W;
  typedef PatchSmem<real, BULK, W::TX, W::TY> SM;
  static int resident[kMaxDevices] = {};  // per device; also: its launch attributes are set
  const int dev = current_device();
  if (dev < 0) return clv_host::check_cuda("cudaGetDevice");
  if (!resident[dev]) {
    int n = 0;
    const int rc = occupancy_patch<real, BULK>(&n);
    if (rc) return rc;
    resident[dev] = sm_count() * std::max(1, n);
  }
  const long long patches = ((long long)grid * (rows - 4) * chunk + W::TX * W::TY - 1) / (W::TX * W::TY);
  const int g = grid > 0 ? (int)std::min<long long>(patches, resident[dev]) : resident[dev];
  if (step == 1) batch_patch_kernel<real, BULK, W::TX, W::TY, W::NT, kPatchBlocks, 1><<<g, W::NT, sizeof(SM), s>>>(p, a, 1, chunk);
  else batch_patch_kernel<real, BULK, W::TX, W::TY, W::NT, kPatchBlocks, 2><<<g, W::NT, sizeof(SM), s>>>(p, a, 2, chunk);
  return clv_host::check_cuda("batch_patch_kernel");
}
template <class real>
int stage_tiled(const Params& p, const BatchArgs<real>& a, int step, int rows, int chunk, int grid, cudaStream_t s) {
  return p.flags & FLAG_BULK ? stage_patch<real, true>(p, a, step, rows, chunk, grid, s)
                             : stage_patch<real, false>(p, a, step, rows, chunk, grid, s);
}
template <class real> int occupancy_tiled(bool bulk, int* n) {
  return bulk ? occupancy_patch<real, true>(n) : occupancy_patch<real, false>(n);
}

}  // namespace batch_launch
}  // namespace CLV_ARITH
}  // namespace clv
