// Cooper-Frye smooth spectra dN/(dY pt dpt dphi) of one hadron species on the
// freeze-out surface (CLSmoothSpec/src/kernel_spec.cl:4-141 for ideal
// surfaces, kernel_spec_csc.cl:4-101 with the viscous correction delta f).
//
// Layout: block (c, k) takes the rapidity Y[k] and the c-th contiguous chunk
// of surface elements; its NPT x NPHI threads each own one (pt, phi) point.
// Elements pass through shared memory in tiles. What depends on the element
// and the rapidity alone is folded there once into the coefficients of three
// linear and quadratic forms in (mt, px, py), in 16-byte groups:
//   u.p    = mt (ch u0 - sh u3) - px u1 - py u2
//   p.dS   = mt (ch S0 - sh S3) - px S1 - py S2
//   p.pi.p = mt^2 c0 - mt px c1 - mt py c2 + px^2 c3 + px py c4 + py^2 c5
// with c0 = ch^2 pi00 + sh^2 pi33 - 2 ch sh pi03, c1 = 2 (ch pi01 - sh pi03),
// c2 = 2 (ch pi02 - sh pi13), c3 = pi11, c4 = 2 pi12, c5 = pi22: the
// reference's contraction (kernel_spec_csc.cl:58-70), which has pi^{03} and
// pi^{13} where the p_3 p_1 and p_3 p_2 terms take pi^{13} and pi^{23} (kept).
// A thread then needs 12 multiply-adds, three broadcast 16-byte reads, one
// exponential and the distribution function (in double, as the reference
// computes it with delta f) an element: the issue of these bounds the kernel.
// 40 000 viscous elements, 15 x 48 momenta, 41 rapidities: 6.64 ms with the
// contractions per thread, 1.73 ms folded.
// Each thread sums its point over the chunk in double, in element order;
// spectra_finish adds the chunks in order, so the result does not depend on
// scheduling.
#pragma once
#include "clv_device.cuh"

namespace clv {

constexpr int SPEC_TILE = 128;

struct SpecHadron {
  double mass, gspin, fermi_boson, muB;
};

// exp(x / T) from x times the scale spec_scale<real>(T): FP32 takes the base-2
// exponential, with log2(e) in the scale. The scale goes into the coefficients
// of u.p in double, so that each is rounded once: a rounding of the scale
// would move every element's exponential the same way.
__device__ __forceinline__ float spec_exp(float x) { return exp2f(x); }
__device__ __forceinline__ double spec_exp(double x) { return exp(x); }
// the argument of spec_exp from which the result is infinite
__device__ __forceinline__ float spec_overflow(float) { return 128.0f; }
__device__ __forceinline__ double spec_overflow(double) { return 710.0; }
template <class real> __device__ __forceinline__ double spec_scale(real t) {
  return (sizeof(real) == 4 ? 1.4426950408889634 : 1.0) / (double)t;
}

// MAXT: the largest block (736 threads: the reference's 15 x 48 points, two
// blocks an SM; else 1024)
template <class real, bool VISCOUS, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT <= 736 && sizeof(real) == 4 ? 2 : 1)
    spectra_kernel(const real* sf, const real* pisf, long long n, long long chunk, SpecHadron h, real tfrz, real tcoeff,
                   const real* Y, const real* Pt, const real* cphi, const real* sphi, int npt, int nphi, double* part) {
  constexpr int NV = VISCOUS ? 12 : 6;
  __shared__ __align__(16) real s_c[SPEC_TILE][VISCOUS ? 12 : 8];
  const int c = blockIdx.x, k = blockIdx.y, ny = gridDim.y;
  const int tid = threadIdx.x;
  const int nthr = blockDim.x;
  const bool active = tid < npt * nphi;
  const int l = active ? tid / nphi : 0, m = active ? tid % nphi : 0;
  const real fb = (real)h.fermi_boson;
  // dof = gspin / (2 pi)^3 (kernel_spec.cl:30)
  const double dof = (double)(real)(h.gspin / ((2.0 * 3.14159265358979323846) * (2.0 * 3.14159265358979323846) *
                                               (2.0 * 3.14159265358979323846)));
  const real rapidity = Y[k];
  const real mass = (real)h.mass, pt = Pt[l];
  const real mt = sqrt(mass * mass + pt * pt);
  const real px = pt * cphi[m], py = pt * sphi[m];
  const double sc = spec_scale(tfrz), dpt = pt;
  const real emt = (real)(sqrt((double)mass * (double)mass + dpt * dpt) * sc), emu = (real)(-(double)(real)h.muB * sc);
  const real epx = (real)(-dpt * (double)cphi[m] * sc), epy = (real)(-dpt * (double)sphi[m] * sc);
  const unsigned int lanes = __ballot_sync(0xffffffffu, active);
  double acc = 0.0;
  const long long lo = (long long)c * chunk, hi = min(n, lo + chunk);
  for (long long t0 = lo; t0 < hi; t0 += SPEC_TILE) {
    const int nt = (int)min((long long)SPEC_TILE, hi - t0);
    bool finite = true;  // this thread's elements
    __syncthreads();
    for (int e = tid; e < nt; e += nthr) {
      const real* S = sf + (t0 + e) * 8;
      const real vx = S[4], vy = S[5], vh = S[6];
      const real ch = cosh(rapidity - S[7]), sh = sinh(rapidity - S[7]);
      real g;
      if (VISCOUS)  // kernel_spec_csc.cl:55-57
        g = (real)1.0f / sqrt(cmax<real>((real)1.0E-15f, (real)(1.0f - vx * vx - vy * vy - vh * vh)));
      else  // kernel_spec.cl:40
        g = (real)(1.0 / sqrt(cmax<double>(1.0E-30, 1.0 - vx * vx - vy * vy - vh * vh)));
      real v[NV];
      v[0] = g * fma(-sh, vh, ch);
      v[1] = g * vx;
      v[2] = g * vy;
      v[3] = fma(ch, S[0], -(sh * S[3]));
      v[4] = S[1];
      v[5] = S[2];
      if (VISCOUS) {
        const real* P = pisf + (t0 + e) * 10;
        v[6] = tcoeff * fma(ch, fma(ch, P[0], (real)-2.0f * sh * P[3]), sh * sh * P[9]);
        v[7] = tcoeff * (real)2.0f * fma(ch, P[1], -(sh * P[3]));
        v[8] = tcoeff * (real)2.0f * fma(ch, P[2], -(sh * P[6]));
        v[9] = tcoeff * P[4];
        v[10] = tcoeff * (real)2.0f * P[5];
        v[11] = tcoeff * P[7];
      }
#pragma unroll
      for (int q = 0; q < NV; q++) {
        s_c[e][q] = v[q];
        finite = finite && isfinite(v[q]);
      }
    }
    const real cut = __syncthreads_and(finite) ? spec_overflow(mt) : (real)INFINITY;
    if (!active) continue;
#pragma unroll 2
    for (int e = 0; e < nt; e++) {
      const real* v = s_c[e];
      const real x = fma(emt, v[0], fma(epx, v[1], fma(epy, v[2], emu)));
      // where the exponential overflows for the whole warp every term is an
      // exact zero (a finite element over infinity): a third to a half of the
      // (element, Y, pt) combinations lie that far apart in rapidity
      if (__all_sync(lanes, x >= cut)) continue;
      const real pdsig = fma(mt, v[3], fma(-px, v[4], -(py * v[5])));
      const real ex = spec_exp(x);
      if constexpr (!VISCOUS) {  // kernel_spec.cl:41-55
        acc += (double)(pdsig / (ex + fb));
      } else {  // kernel_spec_csc.cl:58-78
        double feq = 1.0 / ((double)ex + (double)fb);
        const real pl = fma(mt, v[6], -fma(px, v[7], py * v[8]));
        const real p2pi = fma(mt, pl, fma(px, fma(px, v[9], py * v[10]), py * (py * v[11])));
        const double df = feq * fma(-(double)fb, feq, 1.0) * (double)p2pi;
        feq += fabs(df) > feq ? (df > 0 ? 1.0 : (df < 0 ? -1.0 : 0.0)) * feq * 0.999 : df;
        acc = fma((double)pdsig, feq, acc);
      }
    }
  }
  if (active) part[((long long)c * ny + k) * (npt * nphi) + tid] = dof * acc;
}

template <class real>
__global__ void spectra_finish_kernel(const double* part, int nchunk, long long npoint, real* out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= npoint) return;
  double s = 0.0;
  for (int c = 0; c < nchunk; c++) s += part[(long long)c * npoint + i];
  out[i] = (real)s;
}

}  // namespace clv
