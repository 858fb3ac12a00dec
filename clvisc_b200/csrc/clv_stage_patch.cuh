// Fused Runge-Kutta stage for (2+1)D grids (one cell along eta) by patches.
//
// A block owns a patch of TX x TY cells and evaluates, each once: the record
// of every cell of the patch and its 2-cell halo, the limited slopes, the face
// fluxes, and the update. The phases are separated by barriers and each
// spreads its items over all threads of the block; nothing is carried from one
// plane to the next, so a block's work is short (the marching kernel of
// clv_stage_tiled2d.cuh runs chunk + 4 dependent planes) and a small grid
// becomes many independent blocks: a single (2+1)D event is bound by the
// latency of one thread's chain, not by the chip's throughput. Against the
// per-cell kernel a cell costs 1.9-2.3 records, 2.4 slopes and 2.2 faces in
// place of 9, 6 and 4.
// Records, slopes and faces are the functions of clv_stage_tiled2d.cuh: the
// exact build's results are the per-cell kernel's bit for bit, the FP32
// tolerance build's are the strips'.
#pragma once
#include "clv_stage_tiled2d.cuh"

namespace clv {

template <int TX, int TY> struct PatchGeom {
  static constexpr int CX = TX + 4, CY = TY + 4, NC = CX * CY;  // records (corners unused)
  static constexpr int NSX = (TX + 2) * TY, NSY = TX * (TY + 2);  // slopes along x and y
  static constexpr int NFX = (TX + 1) * TY, NFY = TX * (TY + 1);  // faces
};
template <class real, bool BULK, int TX, int TY> struct PatchSmem {
  typedef PatchGeom<TX, TY> G;
  typedef Rec2L<real, BULK> L;
  __align__(16) real C[L::RG][G::NC][L::U];
  __align__(16) real S[L::CG][G::NSX + G::NSY][L::U];  // slopes, then (there are fewer) face fluxes
};

// Patch shapes. FP32: 8 x 16 cells on 128 threads, four or five blocks an SM;
// where that leaves SMs without a block (fewer patches than SMs: a single event
// below about 150 x 150 cells), 4 x 8 cells on 96 threads. FP64: 8 x 8 on 64.
// B200, 20 steps of one event, tolerance build, FP32: 301 x 301 0.70 ms (one
// thread a cell 1.30, strips that march 2.2), 145 x 145 0.59 (0.72), 121 x 121 0.39
// (0.66), 61 x 61 0.37 (0.61); FP64 301 x 301 1.57 (2.30). Measured against each
// other with another record, the shapes were: 301 x 301 8 x 16 0.67, 8 x 8 0.88,
// 4 x 8 0.93; 61 x 61 4 x 8 0.36, 8 x 16 0.43; FP64 64 threads 1.57, 96 1.92.
template <class real, bool BULK> struct PatchWide {
  static constexpr int TX = 8, TY = sizeof(real) == 4 ? 16 : 8, NT = sizeof(real) == 4 ? 128 : 64;
  static constexpr int MINB = sizeof(real) == 4 ? (BULK ? 4 : 5) : 4;
};
struct PatchSmall {  // FP32
  static constexpr int TX = 4, TY = 8, NT = 96, MINB = 5;
};

inline namespace CLV_ARITH {

// The patch at (i0, j0) of the event (gd, b); first: a strip starts at i0. Every
// thread of the block calls it (it holds barriers).
template <class real, bool BULK, int TX, int TY, int NT, int STAGE>
__device__ __forceinline__ void patch2d(const Params& p, const GridDims& gd, const ViscBuffers<real>& b, int step_,
                                        const TauConst<real>& tc, int i0, int j0, PatchSmem<real, BULK, TX, TY>& s,
                                        bool first = false) {
  typedef Rec2<BULK> R;
  typedef Rec2L<real, BULK> L;
  typedef PatchGeom<TX, TY> G;
  constexpr int NP = L::NP, CP = L::CP, RG = L::RG, CG = L::CG, NC = R::NCOMP;
  constexpr int NS = G::NSX + G::NSY, NF = G::NFX + G::NFY;
  const int step = arith_step<real, STAGE>(step_);
  const real tau = tc.tau;
  const Recips<real>& rc = recips<real>(p);
  const long long ld = gd.ld;
  const int t = threadIdx.x;
  real* const C = &s.C[0][0][0];
  real* const S = &s.S[0][0][0];
  real* const F = S;

  // records of the patch and its halo (rows x0-2 .. x0+TX+1, consecutive
  // threads along y), the four 2 x 2 corners left out
  for (int q = t; q < G::NC; q += NT) {
    const int r = q / G::CY, c = q % G::CY;
    if ((r < 2 || r >= TX + 2) && (c < 2 || c >= TY + 2)) continue;
    real rec[NP];
    rec2_make<real, BULK>(p, gd, b, tau, i0 - 2 + r, j0 - 2 + c, rec);
    grp_store<real, RG>(C, G::NC, q, rec);
  }
  __syncthreads();
  // slopes: along x at rows 1 .. TX+2 of the record array, along y at columns
  // 1 .. TY+2
  for (int q = t; q < NS; q += NT) {
    const bool x = q < G::NSX;
    const int qq = x ? q : q - G::NSX;
    const int cm = x ? (qq / TY + 1) * G::CY + (qq % TY + 2) : (qq / (TY + 2) + 2) * G::CY + (qq % (TY + 2) + 1);
    const int d = x ? G::CY : 1;
    real rl[NP], rm[NP], rr[NP], sl[CP];
    grp_load<real, RG>(C, G::NC, cm - d, rl);
    grp_load<real, RG>(C, G::NC, cm, rm);
    grp_load<real, RG>(C, G::NC, cm + d, rr);
    rec2_slopes<real, BULK, true>(rl, rm, rr, sl, first && x && qq / TY == 0);
    grp_store<real, CG>(S, NS, q, sl);
  }
  __syncthreads();
  // faces: face f of a row (or column) lies between its slope slots f and f+1.
  // They take the slopes' place, so a thread holds its two or three until all
  // slopes have been read: the space of a second array keeps one block more an
  // SM.
  constexpr int NIT = (NF + NT - 1) / NT;
  real f[NIT][CP];
#pragma unroll
  for (int it = 0; it < NIT; it++) {
    const int q = t + it * NT;
    if (q < NF) {
      const bool x = q < G::NFX;
      const int qq = x ? q : q - G::NFX;
      const int r = x ? qq / TY : qq / (TY + 1), c = x ? qq % TY : qq % (TY + 1);
      const int cl = x ? (r + 1) * G::CY + (c + 2) : (r + 2) * G::CY + (c + 1);
      const int s0 = x ? q : G::NSX + r * (TY + 2) + c;
      real rl[NP], rr[NP], sl[CP], sr[CP];
      grp_load<real, RG>(C, G::NC, cl, rl);
      grp_load<real, RG>(C, G::NC, cl + (x ? G::CY : 1), rr);
      grp_load<real, CG>(S, NS, s0, sl);
      grp_load<real, CG>(S, NS, s0 + (x ? TY : 1), sr);
      rec2_face<real, BULK, true>(p, tau, x ? 0 : 1, rl, sl, rr, sr, f[it]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < NIT; it++)
    if (t + it * NT < NF) grp_store<real, CG>(F, NF, t + it * NT, f[it]);
  __syncthreads();
  // update
  for (int q = t; q < TX * TY; q += NT) {
    const int r = q / TY, c = q % TY;
    if (i0 + r >= gd.nx || j0 + c >= gd.ny) continue;
    const long long I = (long long)(i0 + r) * gd.ny + (j0 + c);
    const int cs = (r + 2) * G::CY + (c + 2);
    real S4[4], S10[11], pc[11], pin[5], grad[3][4];
    CellIn<real> cin;
    rec2_cell<real, BULK>(p, gd, b, step, tc, I, C, G::NC, cs, cin, pc, pin, S4, S10);
    // flux differences in the reference's order x, y (eta: one cell, none)
#pragma unroll
    for (int a = 0; a < 2; a++) {
      real Fm[CP], Fp[CP];
      const int fm = a == 0 ? r * TY + c : G::NFX + r * (TY + 1) + c;
      grp_load<real, CG>(F, NF, fm, Fm);
      grp_load<real, CG>(F, NF, fm + (a == 0 ? TY : 1), Fp);
      rec2_flux<real, BULK>(Fp, Fm, a == 0 ? (real)p.DX : (real)p.DY, a == 0 ? rc.DX : rc.DY, S4, S10);
    }
    {
      real um[4], ux0[4], ux1[4], uy0[4], uy1[4], n[NP];
      grp_load<real, RG>(C, G::NC, cs, n);
      rec2_umu<real, BULK>(n, um);
      grp_load<real, RG>(C, G::NC, cs - G::CY, n);
      rec2_umu<real, BULK, true>(n, ux0);
      grp_load<real, RG>(C, G::NC, cs + G::CY, n);
      rec2_umu<real, BULK>(n, ux1);
      grp_load<real, RG>(C, G::NC, cs - 1, n);
      rec2_umu<real, BULK>(n, uy0);
      grp_load<real, RG>(C, G::NC, cs + 1, n);
      rec2_umu<real, BULK>(n, uy1);
      rec2_grad<real, BULK>(p, tc, cin, um, ux0, ux1, uy0, uy1, grad);
    }
    real pinew[11];
    cell_in_ev1<real>(p, b, I, ld, cin);
    real pstart[R::NPI];  // pi at the start of the step: at stage 1 the stage input's
    rec2_start<real, BULK, STAGE>(b, I, ld, pc, pstart);
    pi_update<real, false, BULK>(p, b, step, tc, I, ld, cin, pc, grad, S10, pinew,
                                 [&](int m, real u) { return pstart[m] * u; });
    ev_update<real, true, BULK>(p, b, step, tc, I, ld, cin, pin, S4, pinew);
    if (b.write_src) {
#pragma unroll
      for (int m = 0; m < 4; m++) b.src[m * ld + I] = S4[m];
#pragma unroll
      for (int m = 0; m < R::NPI; m++) b.src[(4 + m) * ld + I] = S10[m];
    }
  }
  (void)NC;
}

// single event, grid (ceil(NY / TY), ceil(NX / TX)); STAGE as in
// visc_stage_tiled_kernel
template <class real, bool BULK, int TX, int TY, int NT, int MINB, int STAGE>
__global__ void __launch_bounds__(NT, MINB)
    visc_stage_patch_kernel(Params p, ViscBuffers<real> b, int step, TauConst<real> tc) {
  after_previous();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PatchSmem<real, BULK, TX, TY>& s = *reinterpret_cast<PatchSmem<real, BULK, TX, TY>*>(smem_raw);
  const GridDims gd{p.nx, p.ny, p.nz, p.ld};
  patch2d<real, BULK, TX, TY, NT, STAGE>(p, gd, b, step, tc, blockIdx.y * TX, blockIdx.x * TY, s);
}

// launches the stage on the patches of a single event; a cudaError_t
template <class real, bool BULK, class Shape>
cudaError_t launch_patch_shape(const Params& p, const ViscBuffers<real>& v, int step, const TauConst<real>& tc,
                               cudaStream_t s) {
  constexpr int TX = Shape::TX, TY = Shape::TY, NT = Shape::NT, MINB = Shape::MINB;
  typedef PatchSmem<real, BULK, TX, TY> SM;
  const int kind = stage_kind(v, step);
  auto kern = kind == 1   ? visc_stage_patch_kernel<real, BULK, TX, TY, NT, MINB, 1>
              : kind == 2 ? visc_stage_patch_kernel<real, BULK, TX, TY, NT, MINB, 2>
                          : visc_stage_patch_kernel<real, BULK, TX, TY, NT, MINB, 0>;
  static bool configured[3][64] = {};  // the attribute is per device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) return e != cudaSuccess ? e : cudaErrorInvalidDevice;
  if (!configured[kind][dev]) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SM));
    if (e != cudaSuccess) return e;
    configured[kind][dev] = true;
  }
  return launch_early(kern, dim3((p.ny + TY - 1) / TY, (p.nx + TX - 1) / TX), NT, sizeof(SM), s, p, v, step, tc);
}
template <class real, bool BULK>
cudaError_t launch_patch(const Params& p, const ViscBuffers<real>& v, int step, const TauConst<real>& tc,
                         cudaStream_t s) {
  typedef PatchWide<real, BULK> W;
  if constexpr (sizeof(real) == 4) {
    const long long wide = (long long)((p.ny + W::TY - 1) / W::TY) * ((p.nx + W::TX - 1) / W::TX);
    if (wide < sm_count()) return launch_patch_shape<real, BULK, PatchSmall>(p, v, step, tc, s);
  }
  return launch_patch_shape<real, BULK, W>(p, v, step, tc, s);
}
// grid.y of the patch launches: patches of 4 cells along x
inline bool patch_fits(const Params& p) { return p.nz == 1 && (p.nx + 3) / 4 <= 65535; }

}  // namespace CLV_ARITH
}  // namespace clv
