// Bulk-evolution diagnostics on the device (pyvisc/bulkinfo.py,
// pyvisc/bulkinfo_h5.py, kernel_bulkinfo.cl).
//
// bulk_slices_kernel restates bulkinfo.py's get_ed and get_pimn kernels
// (bulkinfo.py:62-117): the lines through the grid centre along x, y and
// eta_s, the planes k = NZ/2, j = NY/2 and i = NX/2 of (e, vx, vy, veta), and
// pi^{xx}, pi^{yy}, pi^{tx} "in the transverse plane" with get_pimn's own
// index oid = i*NY*(NZ/2) + j*(NZ/2) + NZ/2, which is not the cell
// (i, j, NZ/2) of the plane (for NZ = 1 it is cell 0 everywhere); the index
// is kept as the reference computes it.
//
// bulk_sums_kernel replaces the host sums the reference makes after copying
// the whole state to the host (bulkinfo.py:184-257): per eta_s slice the
// momentum-anisotropy sums of T^{xx}, T^{yy}, T^{tx} (ecc_vs_rapidity,
// bulkinfo.py:259-271), and in the plane k = NZ/2 the sums behind eccp, the
// viscous eccp, <v_r> and the mid-rapidity entropy (bulkinfo.py:184-257, with
// their floors e >= 1e-10 and v^2 <= 0.999999 and their vz = 0 in the plane).
// One block per slice reduces in a fixed order in double, so the results do
// not depend on scheduling. The equation of state is the run's table.
//
// bulk_lab_kernel is kernel_bulkinfo.cl:18-45 (total_energy_and_entropy)
// with the sums over all cells (bulkinfo_h5.py:264-277) done per block in a
// fixed order.
#pragma once
#include <cooperative_groups.h>

#include "clv_device.cuh"

namespace clv {

constexpr int BULK_SUM_THREADS = 256;
// per-slice sums: Txx, Tyy, T0x (with veta)
constexpr int BULK_NSLICE = 3;
// plane sums: Txx, Tyy, T0x (veta = 0), u0 e v_r, u0 e, u0 s, pi^xx + pi^yy, pi^xx - pi^yy
constexpr int BULK_NPLANE = 8;

// one thread per output cell: the lines x0, y0, z0, then the planes xy, xz, yz
// (201x201x61: 6.8 us; with one block for all of them 694)
template <class real>
__global__ void bulk_slices_kernel(Params p, const real* ev, real* out) {
  const int NX = p.nx, NY = p.ny, NZ = p.nz;
  const long long ld = p.ld;
  const long long n = (long long)NX + NY + NZ + (long long)NX * NY + (long long)NX * NZ + (long long)NY * NZ;
  const long long d = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= n) return;
  int i = NX / 2, j = NY / 2, k = NZ / 2;
  long long q = d;
  if (q < NX) i = (int)q;
  else if ((q -= NX) < NY) j = (int)q;
  else if ((q -= NY) < NZ) k = (int)q;
  else if ((q -= NZ) < (long long)NX * NY) { i = (int)(q / NY); j = (int)(q % NY); }
  else if ((q -= (long long)NX * NY) < (long long)NX * NZ) { i = (int)(q / NZ); k = (int)(q % NZ); }
  else { q -= (long long)NX * NZ; j = (int)(q / NZ); k = (int)(q % NZ); }
  const long long I = ((long long)i * NY + j) * NZ + k;
#pragma unroll
  for (int c = 0; c < 4; c++) out[4 * d + c] = ev[c * ld + I];
}

// get_pimn, bulkinfo.py:103-117 (pi planes 4 = xx, 7 = yy, 1 = tx)
template <class real>
__global__ void bulk_pimn_kernel(Params p, const real* pi, real* pixx, real* piyy, real* pitx) {
  const int gx = blockIdx.y;
  const int gy = blockIdx.x * blockDim.x + threadIdx.x;
  if (gx >= p.nx || gy >= p.ny) return;
  const int NY = p.ny, NZ = p.nz;
  const long long oid = (long long)gx * NY * (NZ / 2) + (long long)gy * (NZ / 2) + NZ / 2;
  const long long nid = (long long)gx * NY + gy;
  pixx[nid] = pi[4 * p.ld + oid];
  piyy[nid] = pi[7 * p.ld + oid];
  pitx[nid] = pi[1 * p.ld + oid];
}

template <int N> __device__ void block_sum(double (&v)[N], double (*sh)[BULK_SUM_THREADS]) {
  const int t = threadIdx.x;
#pragma unroll
  for (int q = 0; q < N; q++) sh[q][t] = v[q];
  __syncthreads();
  for (int s = BULK_SUM_THREADS / 2; s > 0; s >>= 1) {
    if (t < s)
#pragma unroll
      for (int q = 0; q < N; q++) sh[q][t] += sh[q][t + s];
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < N; q++) v[q] = sh[q][0];
}

// the reference's host floors: e >= 1e-10, v^2 > 1 -> 0.999999
__device__ __forceinline__ double floor_ed(double e) { return e < 1.0E-10 ? 1.0E-10 : e; }
__device__ __forceinline__ double u0_of(double vr2) { return 1.0 / sqrt(1.0 - (vr2 > 1.0 ? 0.999999 : vr2)); }

// A cluster of BULK_CLUSTER blocks takes BULK_KL neighbouring slices: a block's
// threads are BULK_KL lanes along eta_s (eight floats are one 32-byte sector)
// times rows of (i, j) columns, the blocks take the columns in turn, and the
// partial sums are added through distributed shared memory in a fixed order.
// (One block a slice read one float of every sector it touched and left the
// chip to NZ blocks of 256 threads: 201x201x61 FP32 204 us, 96 this way.) out[3k .. 3k+2] per slice; the slice
// k = NZ/2 also gives out[3 NZ .. 3 NZ + 7] (pi terms only when pi != nullptr).
constexpr int BULK_CLUSTER = 8, BULK_KL = 8, BULK_ROWS = 64;
constexpr int BULK_NS = BULK_NSLICE + BULK_NPLANE;

template <class real>
__global__ void __cluster_dims__(BULK_CLUSTER, 1, 1) __launch_bounds__(BULK_KL * BULK_ROWS)
    bulk_sums_kernel(Params p, const real* ev, const real* pi, double* out) {
  __shared__ double sh[BULK_NS][BULK_KL][BULK_ROWS / 4 + 1];  // one partial sum of four rows each
  __shared__ double tot[BULK_NS][BULK_KL];
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned int rank = cluster.block_rank();
  const int lane = threadIdx.x % BULK_KL, row = threadIdx.x / BULK_KL;
  const int k = (blockIdx.x / BULK_CLUSTER) * BULK_KL + lane;
  const int NX = p.nx, NY = p.ny, NZ = p.nz;
  const long long ld = p.ld;
  const bool plane = (k == NZ / 2);
  double s[BULK_NS];
#pragma unroll
  for (int q = 0; q < BULK_NS; q++) s[q] = 0.0;
  if (k < NZ) {
    for (int id = (int)rank * BULK_ROWS + row; id < NX * NY; id += BULK_CLUSTER * BULK_ROWS) {
      const long long I = (long long)id * NZ + k;
      const double ed = floor_ed((double)ev[I]);
      const double vx = ev[ld + I], vy = ev[2 * ld + I], vz = ev[3 * ld + I];
      const double pre = (double)eosP<real>(p, (real)ed);
      const double u0 = u0_of(vx * vx + vy * vy + vz * vz);
      s[0] += (ed + pre) * u0 * u0 * vx * vx + pre;
      s[1] += (ed + pre) * u0 * u0 * vy * vy + pre;
      s[2] += (ed + pre) * u0 * u0 * vx;
      if (plane) {
        const double w0 = u0_of(vx * vx + vy * vy);
        s[3] += (ed + pre) * w0 * w0 * vx * vx + pre;
        s[4] += (ed + pre) * w0 * w0 * vy * vy + pre;
        s[5] += (ed + pre) * w0 * w0 * vx;
        s[6] += w0 * ed * sqrt(vx * vx + vy * vy);
        s[7] += w0 * ed;
        s[8] += w0 * (double)eos_comp<real>(p, (real)ed, 3);
        if (pi) {
          const int i = id / NY, j = id % NY;
          const long long oid = (long long)i * NY * (NZ / 2) + (long long)j * (NZ / 2) + NZ / 2;
          const double xx = pi[4 * ld + oid], yy = pi[7 * ld + oid];
          s[9] += xx + yy;
          s[10] += xx - yy;
        }
      }
    }
  }
  // the four rows of a warp by shuffles (lanes 0-7, 8-15, ...), then the
  // block's warps, then the cluster's blocks
#pragma unroll
  for (int q = 0; q < BULK_NS; q++) {
    s[q] += __shfl_down_sync(0xffffffffu, s[q], 16);
    s[q] += __shfl_down_sync(0xffffffffu, s[q], 8);
    if ((threadIdx.x & 31) < BULK_KL) sh[q][lane][row / 4] = s[q];
  }
  __syncthreads();
  for (int t = threadIdx.x; t < BULK_NS * BULK_KL; t += blockDim.x) {
    const int q = t / BULK_KL, l = t % BULK_KL;
    double a = 0.0;
    for (int r = 0; r < BULK_ROWS / 4; r++) a += sh[q][l][r];
    tot[q][l] = a;
  }
  cluster.sync();
  if (rank == 0)
    for (int t = threadIdx.x; t < BULK_NS * BULK_KL; t += blockDim.x) {
      const int q = t / BULK_KL, l = t % BULK_KL;
      const int kk = (blockIdx.x / BULK_CLUSTER) * BULK_KL + l;
      double a = 0.0;
      for (int r = 0; r < BULK_CLUSTER; r++) a += *cluster.map_shared_rank(&tot[q][l], r);
      if (kk >= NZ) continue;
      if (q < BULK_NSLICE) out[BULK_NSLICE * kk + q] = a;
      else if (kk == NZ / 2) out[BULK_NSLICE * NZ + q - BULK_NSLICE] = a;
    }
  cluster.sync();  // the other blocks' shared memory is read until here
}

// kernel_bulkinfo.cl:18-45 summed: block b adds cells [b*chunk, (b+1)*chunk)
// into part[2b], part[2b+1] (lab-frame energy and entropy density)
template <class real>
__global__ void __launch_bounds__(BULK_SUM_THREADS) bulk_lab_kernel(Params p, const real* ev, real tau, long long chunk,
                                                                     double* part) {
  __shared__ double sh[2][BULK_SUM_THREADS];
  // cosh and sinh of eta_s depend on the slice alone: once a block, not once a cell
  constexpr int NZTAB = 512;
  __shared__ real s_ch[NZTAB], s_sh[NZTAB];
  const bool tab = p.nz <= NZTAB;
  if (tab)
    for (int k = threadIdx.x; k < p.nz; k += BULK_SUM_THREADS) {
      const real etas = (k - p.nz / 2) * (real)p.DZ;
      s_ch[k] = cosh(etas);
      s_sh[k] = sinh(etas);
    }
  __syncthreads();
  const long long N = (long long)p.nx * p.ny * p.nz;
  const long long lo = blockIdx.x * chunk, hi = min(N, lo + chunk);
  const long long ld = p.ld;
  double s[2] = {0.0, 0.0};
  for (long long I = lo + threadIdx.x; I < hi; I += BULK_SUM_THREADS) {
    const int K = (int)(I % p.nz);
    real ed = ev[I], vx = ev[ld + I], vy = ev[2 * ld + I], vz = ev[3 * ld + I];
    real pr = eosP<real>(p, ed);
    real u0 = gamma3<real>(vx, vy, vz);
    real etas = (K - p.nz / 2) * (real)p.DZ;
    real cosh_etas = tab ? s_ch[K] : cosh(etas);
    real sinh_etas = tab ? s_sh[K] : sinh(etas);
    real ed_lab = (ed + pr) * u0 * u0 * (cosh_etas + vz * sinh_etas) - pr * cosh_etas;
    real s_lab = u0 * eos_comp<real>(p, ed, 3);
    s[0] += (double)ed_lab;
    s[1] += (double)s_lab;
  }
  block_sum<2>(s, sh);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = s[0];
    part[2 * blockIdx.x + 1] = s[1];
  }
}

}  // namespace clv
