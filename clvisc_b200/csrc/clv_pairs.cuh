// Pairs of FP32 components for the tolerance build's tiled stage kernels: the
// record layout, limiter and face flux on the two-lane FP32 instructions of
// sm_100 (add, mul, fma .f32x2).
#pragma once
#include "clv_device.cuh"

namespace clv {

// The tolerance build in FP32 keeps another record (same 20 values a cell):
// u^i and u^0 in one group (the velocity gradients read only that one), the
// densities u0*pi^{mu nu} in place of pi^{mu nu} (three of four readers want
// the product; 1/u0 gives pi back) and 1/u0 in place of e (which the cell
// update alone reads, from the field). Its slopes and faces work on pairs of
// neighbouring components with the two-lane FP32 instructions (add, mul, fma
// .f32x2 of sm_100), which halves the issue slots of a kernel that is bound by
// instruction issue and latency: 3.06k instructions a cell and stage before, with
// the scalar forms, 2.35k after.
enum { PK_UX = 0, PK_UY, PK_UZ, PK_U0, PK_RU, PK_PR, PK_Q, PK_U = PK_Q + 4 };

inline namespace CLV_ARITH {
template <class real> struct Pairs { static constexpr bool on = CLV_FAST && sizeof(real) == 4; };
#if CLV_FAST
// ---- pairs of FP32 components (tolerance build)
__device__ __forceinline__ float2 pair_at(const float* v) { return make_float2(v[0], v[1]); }
__device__ __forceinline__ float2 pair_sub(float2 a, float2 b) {  // a - b, exactly rounded as a scalar subtraction
  return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);
}
// 1/TH times the limited slope of slope() at the middle of three pairs: with
// a, b the one-sided differences and t = (a + b)/(2 TH), the one of a, b, t
// nearest zero when all have one sign, else zero. The sign tests of the scalar
// form become min and max: max(min(a,b,t), min(max(a,b,t), 0)). Four two-lane
// operations and four min/max a component against six scalar operations, a
// compare and a select. TH is folded into the face's coefficients.
__device__ __forceinline__ float limit3(float a, float b, float t) {
  return fmaxf(fminf(fminf(a, b), t), fminf(fmaxf(fmaxf(a, b), t), 0.0f));
}
__device__ __forceinline__ void pair_limit(float2 l, float2 m, float2 r, float* out) {
  const float kt = 0.5f / CLV_THETA;
  const float2 a = pair_sub(r, m), b = pair_sub(m, l);
  const float2 t = __fmul2_rn(pair_sub(r, l), make_float2(kt, kt));
  out[0] = limit3(a.x, b.x, t.x);
  out[1] = limit3(a.y, b.y, t.y);
}
// the 20 values of a record (21 with Pi) from (e, v), pi and the pressure of
// the flux (P(e), plus Pi with the bulk sector)
template <int NPI>
__device__ __forceinline__ void pair_record(float tau, float e, float vx, float vy, float vz, float pr,
                                            const float* pi, float* r) {
  const float q = cmax<float>(1.0f - vx * vx - vy * vy - vz * vz, Acu<float>::v);  // as gamma3
  const float g = rsqrt(q);
  const float A = (e + pr) * g;
  r[PK_U0] = g;
  r[PK_UX] = vx * g;
  r[PK_UY] = vy * g;
  r[PK_UZ] = vz * g;
  r[PK_RU] = q * g;
  r[PK_PR] = pr;
  r[PK_Q] = tau * (A * g - pr + pi[0]);
#pragma unroll
  for (int c = 1; c < 4; c++) r[PK_Q + c] = tau * (A * r[c - 1] + pi[c]);
#pragma unroll
  for (int m = 0; m < NPI; m++) r[PK_U + m] = g * pi[m];
}
// face_flux in the weighted form (below) on pairs. th*pi at the face comes
// from the densities: th (u0 pi)_L / u0_L + th (u0 pi)_R / u0_R.
template <int NC>
__device__ __forceinline__ void pair_face(float tau, int a, const float* L, const float* sL,
                                          const float* R, const float* sR, float* F) {
  // a may be known at run time only: selects, no indexing
  const float ul = a == 0 ? L[PK_UX] : (a == 1 ? L[PK_UY] : L[PK_UZ]);
  const float ur = a == 0 ? R[PK_UX] : (a == 1 ? R[PK_UY] : R[PK_UZ]);
  const float vs = ul * L[PK_RU] + ur * R[PK_RU];  // v_L + v_R
  const float vh = 0.5f * vs;
  const float cp = 0.25f * vs + 0.5f, cm = 0.25f * vs - 0.5f;
  const float hp = (0.5f * CLV_THETA) * cp, hm = (-0.5f * CLV_THETA) * cm;
  const float th = 0.5f * tau;
  const float pt = th * (L[PK_PR] + R[PK_PR]);
  const float rl = th * L[PK_RU], rr = th * R[PK_RU];
  const float2 rl2 = make_float2(rl, rl), rr2 = make_float2(rr, rr);
  float ps[10];  // th * (pi_L + pi_R); unused components drop out
#pragma unroll
  for (int m = 0; m < 10; m += 2) {
    const float2 t = __ffma2_rn(rl2, pair_at(L + PK_U + m), __fmul2_rn(rr2, pair_at(R + PK_U + m)));
    ps[m] = t.x;
    ps[m + 1] = t.y;
  }
  float k[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const float pa = a == 0 ? ps[pidx(1, c)] : (a == 1 ? ps[pidx(2, c)] : ps[pidx(3, c)]);
    k[c] = pa - vh * ps[c];
    if (c == 0) k[c] += pt * vh;
    k[c] += c == a + 1 ? pt : 0.0f;
  }
  const float2 cm2 = make_float2(cm, cm), cp2 = make_float2(cp, cp), hm2 = make_float2(hm, hm),
               hp2 = make_float2(hp, hp);
#pragma unroll
  for (int c = 0; c < NC; c += 2) {
    const float2 qr = pair_at(R + PK_Q + c);
    float2 f = c < 4 ? __ffma2_rn(cm2, qr, pair_at(k + c)) : __fmul2_rn(cm2, qr);
    f = __ffma2_rn(hm2, pair_at(sR + c), f);
    f = __ffma2_rn(cp2, pair_at(L + PK_Q + c), f);
    f = __ffma2_rn(hp2, pair_at(sL + c), f);
    F[c] = f.x;
    F[c + 1] = f.y;
  }
}
#endif
}  // namespace CLV_ARITH
}  // namespace clv
