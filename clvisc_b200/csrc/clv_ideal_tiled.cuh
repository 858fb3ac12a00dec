// Tiled Runge-Kutta stage of the ideal step ((3+1)D grids).
//
// Same arithmetic as ideal_stage_kernel (clv_stage.cuh), which evaluates the
// equation of state 13 times and the characteristic speed 6 times a cell. Here
// a CTA owns a TJ x TK tile of (j, k) columns and marches along i (the scheme
// of clv_stage_tiled.cuh with a record of nine values): the record (e, v,
// P(e), T^{tau mu}) of a cell, its limited slope in each direction and the
// flux through a face are computed once. A cell's flux difference subtracts
// its minus face from its plus face, exactly the two values the per-cell
// kernel forms, and each record, slope and face is that kernel's expression:
// the same bits.
//
// The plane's records sit in shared memory with their 2-cell halo; the own
// column's records of the two planes ahead, its x slope and its x face stay in
// registers (nine values a record: no second shared copy as the viscous kernel
// needs), so FP32 keeps three CTAs of 256 threads an SM (85 registers, 30 KB).
// Bound by the latency of a plane's chain, as the viscous kernel: 201x201x61
// FP32, one stage, 390 us against 608 with a thread a cell. (2+1)D grids take
// 8 x 8 patches below: 101 x 101 FP64, 20 steps with the maximum read after
// each, 1.19 ms against 1.61 (evolve's single library call included).
#pragma once
#include "clv_smem16.cuh"
#include "clv_stage_patch.cuh"
#include "clv_stage_tiled.cuh"

namespace clv {

// record: e, vx, vy, vz, P(e), T0..T3, padded to whole 16-byte groups
enum { IR_E = 0, IR_VX, IR_VY, IR_VZ, IR_PR, IR_T, IR_N = IR_T + 4 };

template <class real, int TJ, int TK> struct IdealSmem {
  typedef TileGeom<TJ, TK> G;
  static constexpr int U = Smem16<real>::U;
  static constexpr int NP = Smem16<real>::pad(IR_N), RG = NP / U, SG = 4 / U;
  __align__(16) real C[RG][G::NC][U];    // plane i with its halo
  __align__(16) real SY[SG][G::NSY][U];  // y slopes, then y face fluxes
  __align__(16) real SZ[SG][G::NSZ][U];  // z slopes, then z face fluxes
};

inline namespace CLV_ARITH {

template <class real, int NP>
__device__ __forceinline__ void ideal_record(const Params& p, const real* ev, int i, int j, int k, real r[NP]) {
  i = min(max(i, 0), p.nx - 1);
  j = min(max(j, 0), p.ny - 1);
  k = min(max(k, 0), p.nz - 1);
  const Idx32 I{((unsigned int)i * p.ny + j) * p.nz + k};
  const long long ld = p.ld;
#pragma unroll
  for (int c = 0; c < 4; c++) r[IR_E + c] = plane_at(ev, c * ld, I);
  r[IR_PR] = eosP<real>(p, r[IR_E]);
  real u0 = gamma3<real>(r[IR_VX], r[IR_VY], r[IR_VZ]);
  real A = (r[IR_E] + r[IR_PR]) * u0;
  real u4[4] = {(real)1.0f * u0, r[IR_VX] * u0, r[IR_VY] * u0, r[IR_VZ] * u0};
#pragma unroll
  for (int c = 0; c < 4; c++) {
    real g0 = c == 0 ? (real)1.0f : (real)0.0f;
    r[IR_T + c] = A * u4[c] - g0 * r[IR_PR];
  }
#pragma unroll
  for (int c = IR_N; c < NP; c++) r[c] = 0.0f;
}

template <class real>
__device__ __forceinline__ void ideal_slopes(const real* L, const real* M, const real* R, real out[4]) {
#pragma unroll
  for (int c = 0; c < 4; c++) out[c] = slope<real>(L[IR_T + c], M[IR_T + c], R[IR_T + c]);
}

// kt1d, helper.h:199-262, for the face between records L and R along axis a
template <class real>
__device__ __forceinline__ void ideal_face(const Params& p, int a, const real* L, const real* sL, const real* R,
                                           const real* sR, real F[4]) {
  real h[4];
#pragma unroll
  for (int c = 0; c < 4; c++) h[c] = 0.5f * (L[IR_E + c] + R[IR_E + c]);
  const real vh = a == 0 ? h[1] : (a == 1 ? h[2] : h[3]);
  const real lam = max_speed<real>(p, h[0], h[1], h[2], h[3], vh);
  const real pr_half = 0.5f * (L[IR_PR] + R[IR_PR]);
#pragma unroll
  for (int c = 0; c < 4; c++) {
    real AL = L[IR_T + c] + 0.5f * sL[c];
    real AR = R[IR_T + c] - 0.5f * sR[c];
    real g0 = c == 0 ? (real)1.0f : (real)0.0f;
    real ga = c == a + 1 ? (real)-1.0f : (real)0.0f;
    real Jp = (AR + pr_half * g0) * vh - pr_half * ga;
    real Jm = (AL + pr_half * g0) * vh - pr_half * ga;
    F[c] = 0.5f * (Jp + Jm) - 0.5f * lam * (AR - AL);
  }
}

// Christoffel terms, kernel_ideal.cl:125-143
template <class real> __device__ __forceinline__ void ideal_christoffel(const Params& p, const real* own, real S[4]) {
  real ed = own[IR_E], vz = own[IR_VZ];
  real pressure = own[IR_PR];
  real u0 = gamma3<real>(own[IR_VX], own[IR_VY], vz);
  real Tzz_tilde = (ed + pressure) * u0 * u0 * vz * vz + pressure;
  real Ttz_tilde = (ed + pressure) * u0 * u0 * vz;
  if (!(p.flags & FLAG_RIEMANN)) {
    S[0] = S[0] - Tzz_tilde;
    S[1] = S[1] - (real)0.0f;
    S[2] = S[2] - (real)0.0f;
    S[3] = S[3] - Ttz_tilde;
  }
}
// flux difference along axis a into the sources
template <class real>
__device__ __forceinline__ void ideal_flux(const Params& p, const TauConst<real>& tc, int a, const real Fp[4],
                                           const real Fm[4], real S[4]) {
  const Recips<real>& rc = recips<real>(p);
  const real D = a == 0 ? (real)p.DX : (a == 1 ? (real)p.DY : (real)p.DZ);
  const real rD = a == 0 ? rc.DX : (a == 1 ? rc.DY : rc.DZ);
#pragma unroll
  for (int c = 0; c < 4; c++) {
    real src = Fp[c];
    src -= Fm[c];
    if (p.flags & FLAG_RIEMANN) S[c] = S[c] - div_by<real>(src, D, rD);
    else if (a < 2) S[c] = S[c] - div_by<real>(tc.tau * src, D, rD);
    else S[c] = S[c] - div_by<real>(tc.tau * src, tc.dzt, tc.rdzt);
  }
}

template <class real, int TJ, int TK, int MINB>
__global__ void __launch_bounds__(TJ * TK, MINB)
    ideal_stage_tiled_kernel(Params p, IdealBuffers<real> b, int step, TauConst<real> tc, int chunk) {
  typedef TileGeom<TJ, TK> G;
  typedef IdealSmem<real, TJ, TK> SM;
  constexpr int NP = SM::NP, RG = SM::RG, SG = SM::SG;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SM& s = *reinterpret_cast<SM*>(smem_raw);
  real* const C = &s.C[0][0][0];
  real* const SY = &s.SY[0][0][0];
  real* const SZ = &s.SZ[0][0][0];
  const int tid = threadIdx.x;
  const int tj = tid / TK, tk = tid % TK;
  const int k0 = blockIdx.x * TK, j0 = blockIdx.y * TJ;
  const int i0 = blockIdx.z * chunk;
  const int i1 = min(i0 + chunk, p.nx);
  const int jj = j0 + tj, kk = k0 + tk;
  const bool inside = (jj < p.ny) && (kk < p.nz);
  const int cself = (tj + 2) * G::CZ + (tk + 2);
  const long long ld = p.ld;

  // records of the centre plane's halo (rows and columns a stencil reads)
  auto halo = [&](int i) {
    constexpr int NHY = 4 * TK, NHZ = 4 * TJ;
    for (int q = tid; q < NHY + NHZ; q += TJ * TK) {
      int r, c;
      if (q < NHY) {
        const int rr = q / TK;
        r = rr < 2 ? rr : TJ + rr;
        c = 2 + q % TK;
      } else {
        const int qq = q - NHY, cc = qq / TJ;
        c = cc < 2 ? cc : TK + cc;
        r = 2 + qq % TJ;
      }
      real t[NP];
      ideal_record<real, NP>(p, b.ev_st, i, j0 - 2 + r, k0 - 2 + c, t);
      grp_store<real, RG>(C, G::NC, r * G::CZ + c, t);
    }
  };

  typename KeyT<real>::type best = 0;  // maximum energy density of this thread's cells
  // x window of the own column: plane i in C, i+1 in ra
  real ra[NP], s_cur[4], F_prev[4];
  {
    real r0[NP], r1[NP], r2[NP], s_prev[4];
    ideal_record<real, NP>(p, b.ev_st, i0 - 2, jj, kk, r0);
    ideal_record<real, NP>(p, b.ev_st, i0 - 1, jj, kk, r1);
    ideal_record<real, NP>(p, b.ev_st, i0, jj, kk, r2);
    ideal_record<real, NP>(p, b.ev_st, i0 + 1, jj, kk, ra);
    grp_store<real, RG>(C, G::NC, cself, r2);
    ideal_slopes<real>(r0, r1, r2, s_prev);
    ideal_slopes<real>(r1, r2, ra, s_cur);
    ideal_face<real>(p, 0, r1, s_prev, r2, s_cur, F_prev);
  }
  halo(i0);
  __syncthreads();

  for (int i = i0; i < i1; i++) {
    // slopes of plane i in y and z, and of plane i+1 along x
    for (int q = tid; q < G::NSY + G::NSZ; q += TJ * TK) {
      const bool y = q < G::NSY;
      const int qq = y ? q : q - G::NSY;
      const int cm = y ? (qq / TK + 1) * G::CZ + (qq % TK + 2) : (qq / (TK + 2) + 2) * G::CZ + (qq % (TK + 2) + 1);
      const int d = y ? G::CZ : 1;
      real rl[NP], rm[NP], rr[NP], sl[4];
      grp_load<real, RG>(C, G::NC, cm - d, rl);
      grp_load<real, RG>(C, G::NC, cm, rm);
      grp_load<real, RG>(C, G::NC, cm + d, rr);
      ideal_slopes<real>(rl, rm, rr, sl);
      grp_store<real, SG>(y ? SY : SZ, y ? G::NSY : G::NSZ, qq, sl);
    }
    real own[NP], rb[NP], s_next[4], Fx[4];
    ideal_record<real, NP>(p, b.ev_st, i + 2, jj, kk, rb);
    grp_load<real, RG>(C, G::NC, cself, own);
    ideal_slopes<real>(own, ra, rb, s_next);
    ideal_face<real>(p, 0, own, s_cur, ra, s_next, Fx);
    __syncthreads();

    // face fluxes: the tile's outer row and column first, each stored at once
    // (its slope slots are read by that thread alone)
    real Fy[4], Fz[4];
    {
      real rn[NP], sa[4], sb[4];
      if (tid < TK + TJ) {
        const bool y = tid < TK;
        const int q = y ? tid : tid - TK;
        const int c0 = y ? G::CZ + q + 2 : (q + 2) * G::CZ + 1;
        const int slot = y ? q : q * (TK + 2);
        real* const dst = y ? SY : SZ;
        const int n = y ? G::NSY : G::NSZ;
        real rl[NP], F[4];
        grp_load<real, RG>(C, G::NC, c0, rl);
        grp_load<real, RG>(C, G::NC, c0 + (y ? G::CZ : 1), rn);
        grp_load<real, SG>(dst, n, slot, sa);
        grp_load<real, SG>(dst, n, slot + (y ? TK : 1), sb);
        ideal_face<real>(p, y ? 1 : 2, rl, sa, rn, sb, F);
        grp_store<real, SG>(dst, n, slot, F);
      }
      const int sy = (tj + 1) * TK + tk, sz = tj * (TK + 2) + (tk + 1);
      grp_load<real, RG>(C, G::NC, cself + G::CZ, rn);
      grp_load<real, SG>(SY, G::NSY, sy, sa);
      grp_load<real, SG>(SY, G::NSY, sy + TK, sb);
      ideal_face<real>(p, 1, own, sa, rn, sb, Fy);
      grp_load<real, RG>(C, G::NC, cself + 1, rn);
      grp_load<real, SG>(SZ, G::NSZ, sz, sa);
      grp_load<real, SG>(SZ, G::NSZ, sz + 1, sb);
      ideal_face<real>(p, 2, own, sa, rn, sb, Fz);
    }
    __syncthreads();
    grp_store<real, SG>(SY, G::NSY, (tj + 1) * TK + tk, Fy);
    grp_store<real, SG>(SZ, G::NSZ, tj * (TK + 2) + (tk + 1), Fz);
    __syncthreads();

    if (inside) {
      const long long I = ((long long)i * p.ny + jj) * p.nz + kk;
      real S[4];
#pragma unroll
      for (int c = 0; c < 4; c++) S[c] = (step == 1) ? (real)0.0f : b.src[c * ld + I];
      ideal_christoffel<real>(p, own, S);
#pragma unroll
      for (int a = 0; a < 3; a++) {
        real Fp[4], Fm[4];
        if (a == 1) grp_load<real, SG>(SY, G::NSY, tj * TK + tk, Fm);
        if (a == 2) grp_load<real, SG>(SZ, G::NSZ, tj * (TK + 2) + tk, Fm);
#pragma unroll
        for (int c = 0; c < 4; c++) {
          Fp[c] = a == 0 ? Fx[c] : (a == 1 ? Fy[c] : Fz[c]);
          if (a == 0) Fm[c] = F_prev[c];
        }
        ideal_flux<real>(p, tc, a, Fp, Fm, S);
      }
      // at stage 1 the stage input is d_ev[1] itself: its pressure is the record's
      const real e = ideal_update_ev<real>(p, b, step, tc, I, S, b.ev1 == b.ev_st ? own : nullptr);
      if (e == e) {
        const auto key = fkey(e);
        best = key > best ? key : best;
      }
    }
#pragma unroll
    for (int c = 0; c < 4; c++) {
      F_prev[c] = Fx[c];
      s_cur[c] = s_next[c];
    }
    __syncthreads();
    if (i + 1 < i1) {
      grp_store<real, RG>(C, G::NC, cself, ra);
#pragma unroll
      for (int c = 0; c < NP; c++) ra[c] = rb[c];
      halo(i + 1);
      __syncthreads();
    }
  }
  if (b.edmax_key) key_commit<real>(b.edmax_key, best);
}

// (2+1)D grids (one cell along eta): a block takes a patch of TX x TY cells,
// records with their halo, slopes, faces and update in turn (the scheme of
// clv_stage_patch.cuh). Small grids are bound by the length of one thread's
// chain, which drops from 9 records, 6 slopes and 4 faces a cell to 2.0, 2.5
// and 2.3.
template <class real, int TX, int TY> struct IdealPatchSmem {
  typedef PatchGeom<TX, TY> G;
  static constexpr int U = Smem16<real>::U;
  static constexpr int NP = Smem16<real>::pad(IR_N), RG = NP / U, SG = 4 / U;
  __align__(16) real C[RG][G::NC][U];
  __align__(16) real S[SG][G::NSX + G::NSY][U];
  __align__(16) real F[SG][G::NFX + G::NFY][U];
};

template <class real, int TX, int TY, int NT>
__global__ void __launch_bounds__(NT)
    ideal_stage_patch_kernel(Params p, IdealBuffers<real> b, int step, TauConst<real> tc) {
  after_previous();
  typedef PatchGeom<TX, TY> G;
  typedef IdealPatchSmem<real, TX, TY> SM;
  constexpr int NP = SM::NP, RG = SM::RG, SG = SM::SG, NS = G::NSX + G::NSY, NF = G::NFX + G::NFY;
  __shared__ SM s;
  real* const C = &s.C[0][0][0];
  real* const S_ = &s.S[0][0][0];
  real* const F = &s.F[0][0][0];
  const int t = threadIdx.x;
  const int i0 = blockIdx.y * TX, j0 = blockIdx.x * TY;

  for (int q = t; q < G::NC; q += NT) {
    const int r = q / G::CY, c = q % G::CY;
    if ((r < 2 || r >= TX + 2) && (c < 2 || c >= TY + 2)) continue;
    real rec[NP];
    ideal_record<real, NP>(p, b.ev_st, i0 - 2 + r, j0 - 2 + c, 0, rec);
    grp_store<real, RG>(C, G::NC, q, rec);
  }
  __syncthreads();
  for (int q = t; q < NS; q += NT) {
    const bool x = q < G::NSX;
    const int qq = x ? q : q - G::NSX;
    const int cm = x ? (qq / TY + 1) * G::CY + (qq % TY + 2) : (qq / (TY + 2) + 2) * G::CY + (qq % (TY + 2) + 1);
    const int d = x ? G::CY : 1;
    real rl[NP], rm[NP], rr[NP], sl[4];
    grp_load<real, RG>(C, G::NC, cm - d, rl);
    grp_load<real, RG>(C, G::NC, cm, rm);
    grp_load<real, RG>(C, G::NC, cm + d, rr);
    ideal_slopes<real>(rl, rm, rr, sl);
    grp_store<real, SG>(S_, NS, q, sl);
  }
  __syncthreads();
  for (int q = t; q < NF; q += NT) {
    const bool x = q < G::NFX;
    const int qq = x ? q : q - G::NFX;
    const int r = x ? qq / TY : qq / (TY + 1), c = x ? qq % TY : qq % (TY + 1);
    const int cl = x ? (r + 1) * G::CY + (c + 2) : (r + 2) * G::CY + (c + 1);
    const int sl0 = x ? q : G::NSX + r * (TY + 2) + c;
    real rl[NP], rr[NP], sl[4], sr[4], f[4];
    grp_load<real, RG>(C, G::NC, cl, rl);
    grp_load<real, RG>(C, G::NC, cl + (x ? G::CY : 1), rr);
    grp_load<real, SG>(S_, NS, sl0, sl);
    grp_load<real, SG>(S_, NS, sl0 + (x ? TY : 1), sr);
    ideal_face<real>(p, x ? 0 : 1, rl, sl, rr, sr, f);
    grp_store<real, SG>(F, NF, q, f);
  }
  __syncthreads();
  for (int q = t; q < TX * TY; q += NT) {
    const int r = q / TY, c = q % TY;
    if (i0 + r >= p.nx || j0 + c >= p.ny) continue;
    const long long I = (long long)(i0 + r) * p.ny + (j0 + c);
    real own[NP], S[4];
    grp_load<real, RG>(C, G::NC, (r + 2) * G::CY + (c + 2), own);
#pragma unroll
    for (int m = 0; m < 4; m++) S[m] = (step == 1) ? (real)0.0f : b.src[m * p.ld + I];
    ideal_christoffel<real>(p, own, S);
#pragma unroll
    for (int a = 0; a < 2; a++) {
      const int fm = a == 0 ? r * TY + c : G::NFX + r * (TY + 1) + c;
      real Fp[4], Fm[4];
      grp_load<real, SG>(F, NF, fm, Fm);
      grp_load<real, SG>(F, NF, fm + (a == 0 ? TY : 1), Fp);
      ideal_flux<real>(p, tc, a, Fp, Fm, S);
    }
    const real e = ideal_update_ev<real>(p, b, step, tc, I, S, b.ev1 == b.ev_st ? own : nullptr);
    if (b.edmax_key) key_max<real>(b.edmax_key, e);
  }
}

}  // namespace CLV_ARITH
}  // namespace clv
