// Freeze-out hypersurface finder (kernel_hypersf.cl:98-660) with
// deterministic output order.
//
// The reference appends surface elements with atomic_inc, so their order
// changes from run to run. Here a first pass marks the coarse cubes that emit
// an element, a block scan turns the marks into offsets, and the element pass
// writes cube q's element at (elements already in the buffer) + (number of
// emitting cubes before q in (i, j, k) order). The element count and the
// per-element arithmetic are those of the reference kernel.
#pragma once
#include "clv_device.cuh"

namespace clv {

template <class real> struct R4 { real x, y, z, w; };  // (tau, x, y, eta) / dSigma components
template <class real> __device__ __forceinline__ R4<real> add4(R4<real> a, R4<real> b) { return {a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w}; }
template <class real> __device__ __forceinline__ R4<real> sub4(R4<real> a, R4<real> b) { return {a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w}; }
template <class real> __device__ __forceinline__ R4<real> scl4(real s, R4<real> a) { return {s * a.x, s * a.y, s * a.z, s * a.w}; }
template <class real> __device__ __forceinline__ R4<real> mul4s(R4<real> a, real s) { return {a.x * s, a.y * s, a.z * s, a.w * s}; }
template <class real> __device__ __forceinline__ R4<real> div4(R4<real> a, real s) { return {a.x / s, a.y / s, a.z / s, a.w / s}; }
template <class real> __device__ __forceinline__ real dotr4(R4<real> a, R4<real> b) {
  real r = a.x * b.x;
  r = r + a.y * b.y;
  r = r + a.z * b.z;
  r = r + a.w * b.w;
  return r;
}
// corner n of the unit 4-cube: (tau, x, y, eta) bits (3, 0, 1, 2) (kernel_hypersf.cl:33-54)
template <class real> __device__ __forceinline__ R4<real> cube_corner(int n) {
  return R4<real>{(real)((n >> 3) & 1), (real)(n & 1), (real)((n >> 1) & 1), (real)((n >> 2) & 1)};
}

template <class real> struct SurfPiece {
  int id[4];
  R4<real> center, norm;
};

// kernel_hypersf.cl:98-122
template <class real>
__device__ SurfPiece<real> construct_hypersf(int id0, int id1, int id2, int id3, const R4<real>* ints, R4<real> mc) {
  SurfPiece<real> s;
  s.id[0] = id0; s.id[1] = id1; s.id[2] = id2; s.id[3] = id3;
  s.center = scl4<real>(0.25f, add4(add4(add4(ints[id0], ints[id1]), ints[id2]), ints[id3]));
  R4<real> vo = sub4(s.center, mc);
  R4<real> a = sub4(ints[id1], ints[id0]);
  R4<real> b = sub4(ints[id2], ints[id0]);
  R4<real> c = sub4(ints[id3], ints[id0]);
  R4<real> n;
  n.x = a.y * (b.z * c.w - b.w * c.z) + a.z * (b.w * c.y - b.y * c.w) + a.w * (b.y * c.z - b.z * c.y);
  n.y = -(a.x * (b.z * c.w - b.w * c.z) + a.z * (b.w * c.x - b.x * c.w) + a.w * (b.x * c.z - b.z * c.x));
  n.z = a.x * (b.y * c.w - b.w * c.y) + a.y * (b.w * c.x - b.x * c.w) + a.w * (b.x * c.y - b.y * c.x);
  n.w = -(a.x * (b.y * c.z - b.z * c.y) + a.y * (b.z * c.x - b.x * c.z) + a.z * (b.x * c.y - b.y * c.x));
  real projection = dotr4(vo, n);
  if (projection < 0) n = R4<real>{-n.x, -n.y, -n.z, -n.w};
  s.norm = n;
  return s;
}

// kernel_hypersf.cl:126-132 (the 32-bit product wraps as on any GPU)
template <class real> __device__ __forceinline__ real sf_rand(int* seed) {
  const int a = 16807;
  const int m = 2147483647;
  int prod = (int)((unsigned int)(*seed) * (unsigned int)a);
  *seed = (int)(((long long)prod) % m);
  return (*seed) / ((real)m);
}

template <class real> __device__ R4<real> mass_center(const R4<real>* ints, int n) {  // :226-232
  R4<real> c{0.0f, 0.0f, 0.0f, 0.0f};
  for (int i = 0; i < n; i++) c = add4(c, ints[i]);
  return div4(c, (real)n);
}

// :135-159. The reference builds the piece (i, j, k, l) inside the m loop;
// it depends only on the intersections and their centre, which change only
// at a hit, after which the m loop ends, so it is built once per (i, j, k, l)
// here: the same values, n - l - 1 times fewer constructions.
template <class real> __device__ void tiny_move_if_coplanar(R4<real>* ints, int n, R4<real>* mc, int gid) {
  int seed = (int)(32117u * (unsigned int)(gid + 1));
  for (int i = 0; i < n - 4; i++)
    for (int j = i + 1; j < n - 3; j++)
      for (int k = j + 1; k < n - 2; k++)
        for (int l = k + 1; l < n - 1; l++) {
          const SurfPiece<real> sf = construct_hypersf(i, j, k, l, ints, *mc);
          for (int m = l + 1; m < n; m++) {
            if (dotr4(sf.norm, sub4(ints[m], sf.center)) == 0.0f) {
              for (int q = 0; q < n; q++) {
                real r0 = sf_rand<real>(&seed), r1 = sf_rand<real>(&seed), r2 = sf_rand<real>(&seed),
                     r3 = sf_rand<real>(&seed);
                R4<real> sh{(r0 - 0.5f) * 1.0E-7f, (r1 - 0.5f) * 1.0E-7f, (r2 - 0.5f) * 1.0E-7f, (r3 - 0.5f) * 1.0E-7f};
                ints[q] = add4(ints[q], sh);
              }
              *mc = mass_center(ints, n);
              break;
            }
          }
        }
}

template <class real> __device__ bool on_convex_hull(const SurfPiece<real>& sf, const R4<real>* ints, int n) {  // :163-176
  for (int q = 0; q < n; q++) {
    if (q != sf.id[0] && q != sf.id[1] && q != sf.id[2] && q != sf.id[3]) {
      if (dotr4(sub4(ints[q], sf.center), sf.norm) >= 0.0f) return false;
    }
  }
  return true;
}

// :195-223 with contribution_from (:180-192)
template <class real> __device__ R4<real> energy_flow(const real ed[16], real efrz) {
  R4<real> vl{0.0f, 0.0f, 0.0f, 0.0f}, vh{0.0f, 0.0f, 0.0f, 0.0f};
  real elsum = 0.0f, ehsum = 0.0f;
#pragma unroll
  for (int n = 0; n < 2; n++)
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 2; j++)
#pragma unroll
        for (int k = 0; k < 2; k++) {
          int id = 8 * n + 4 * k + 2 * j + i;
          real dek = efrz - ed[id];
          real adek = fabs(dek);
          R4<real> w = mul4s(R4<real>{(real)n, (real)i, (real)j, (real)k}, adek);
          if (dek > 0.0f) {
            elsum += adek;
            vl = add4(vl, w);
          } else {
            ehsum += adek;
            vh = add4(vh, w);
          }
        }
  if (fabs(elsum) > Acu<real>::v) vl = div4(vl, elsum);
  if (fabs(ehsum) > Acu<real>::v) vh = div4(vh, ehsum);
  return sub4(vl, vh);
}

// :237-266
template <class real> __device__ R4<real> calc_area(R4<real>* ints, R4<real> flow, int n, int gid) {
  R4<real> mc = mass_center(ints, n);
  R4<real> area{0.0f, 0.0f, 0.0f, 0.0f};
  if (n == 4) {
    SurfPiece<real> sf = construct_hypersf(0, 1, 2, 3, ints, mc);
    if (dotr4(flow, sf.norm) < 0.0f) sf.norm = R4<real>{-sf.norm.x, -sf.norm.y, -sf.norm.z, -sf.norm.w};
    area = sf.norm;
  } else if (n > 4) {
    tiny_move_if_coplanar(ints, n, &mc, gid);
    for (int i = 0; i < n - 3; i++)
      for (int j = i + 1; j < n - 2; j++)
        for (int k = j + 1; k < n - 1; k++)
          for (int l = k + 1; l < n; l++) {
            SurfPiece<real> sf = construct_hypersf(i, j, k, l, ints, mc);
            // both tests are pure: the cheap one first (the reference
            // evaluates the hull test first; the sum is the same)
            if (dotr4(sf.norm, flow) > 0.0f && on_convex_hull(sf, ints, n)) area = add4(area, sf.norm);
          }
  }
  return div4(area, (real)6.0f);
}

// :269-314
template <class real>
__device__ __forceinline__ void ints_between(real el, real er, int cl, int cr, real efrz, R4<real>* all, int* n) {
  real dE1 = efrz - el;
  real dE2 = efrz - er;
  real dE12 = el - er;
  if (dE1 * dE2 < 0) {
    real ratio = fabs(dE1) / fabs(dE12);
    all[*n] = add4(scl4<real>(ratio, cube_corner<real>(cr)), scl4<real>((real)(1 - ratio), cube_corner<real>(cl)));
    *n += 1;
  }
}
template <class real> __device__ void all_intersections(const real ed[16], real efrz, R4<real>* all, int* n) {
  *n = 0;
  for (int s = 0; s < 16; s += 4) {
    ints_between(ed[s + 0], ed[s + 1], s + 0, s + 1, efrz, all, n);
    ints_between(ed[s + 0], ed[s + 2], s + 0, s + 2, efrz, all, n);
    ints_between(ed[s + 2], ed[s + 3], s + 2, s + 3, efrz, all, n);
    ints_between(ed[s + 1], ed[s + 3], s + 1, s + 3, efrz, all, n);
  }
  for (int s = 0; s < 16; s += 8) {
    ints_between(ed[s + 0], ed[s + 4], s + 0, s + 4, efrz, all, n);
    ints_between(ed[s + 1], ed[s + 5], s + 1, s + 5, efrz, all, n);
    ints_between(ed[s + 2], ed[s + 6], s + 2, s + 6, efrz, all, n);
    ints_between(ed[s + 3], ed[s + 7], s + 3, s + 7, efrz, all, n);
  }
  for (int s = 0; s < 8; s++) ints_between(ed[s + 0], ed[s + 8], s + 0, s + 8, efrz, all, n);
}

struct CubeGrid {
  int nx, ny, nz;  // coarse cube counts per axis
};
__host__ __device__ inline CubeGrid cube_grid(const Params& p) {
  return CubeGrid{(p.nx - 1) / p.nxskip + 1, (p.ny - 1) / p.nyskip + 1, (p.nz - 1) / p.nzskip + 1};
}
__device__ __forceinline__ long long corner_cell(const Params& p, int i, int j, int k, int q) {
  int ii = (i + (q & 1)) * p.nxskip, jj = (j + ((q >> 1) & 1)) * p.nyskip, kk = (k + ((q >> 2) & 1)) * p.nzskip;
  return ((long long)ii * p.ny + jj) * p.nz + kk;
}
// centroid weight of corner q (kernel_hypersf.cl:329-348)
template <class real> __device__ __forceinline__ real corner_weight(R4<real> mc, int q) {
  real a = (q & 8) ? mc.x : (real)(1.0f - mc.x);
  real b = (q & 1) ? mc.y : (real)(1.0f - mc.y);
  real c = (q & 2) ? mc.z : (real)(1.0f - mc.z);
  real d = (q & 4) ? mc.w : (real)(1.0f - mc.w);
  return a * b * c * d;
}

// energy densities of the 16 corners; false when the cube is outside the
// grid (kernel_hypersf.cl:536)
template <class real>
__device__ __forceinline__ bool load_cube(const Params& p, const real* ev_old, const real* ev_new, int i, int j, int k,
                                          real ed[16]) {
  if (!((i + 1) * p.nxskip < p.nx && (j + 1) * p.nyskip < p.ny && (k + 1) * p.nzskip < p.nz)) return false;
#pragma unroll
  for (int q = 0; q < 8; q++) {
    long long c = corner_cell(p, i, j, k, q);
    ed[q] = ev_old[c];
    ed[8 + q] = ev_new[c];
  }
  return true;
}
template <class real> __device__ __forceinline__ bool crosses(const real ed[16], real efrz) {  // :562-571
  return !((ed[0] - efrz) * (ed[15] - efrz) > 0 && (ed[1] - efrz) * (ed[14] - efrz) > 0 &&
           (ed[2] - efrz) * (ed[13] - efrz) > 0 && (ed[3] - efrz) * (ed[12] - efrz) > 0 &&
           (ed[4] - efrz) * (ed[11] - efrz) > 0 && (ed[5] - efrz) * (ed[10] - efrz) > 0 &&
           (ed[6] - efrz) * (ed[9] - efrz) > 0 && (ed[7] - efrz) * (ed[8] - efrz) > 0);
}

// pass 1: does cube q emit an element?  (visc: mass centre not NaN, :604)
template <class real>
__global__ void hsf_mark_kernel(Params p, const real* ev_old, const real* ev_new, int visc, uint8_t* mark,
                                int* block_count) {
  const CubeGrid g = cube_grid(p);
  const long long nc = (long long)g.nx * g.ny * g.nz;
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int emit = 0;
  if (q < nc) {
    int k = (int)(q % g.nz), j = (int)((q / g.nz) % g.ny), i = (int)(q / ((long long)g.ny * g.nz));
    real ed[16];
    const real efrz = p.EFRZ;
    if (load_cube(p, ev_old, ev_new, i, j, k, ed) && crosses(ed, efrz)) {
      emit = 1;
      if (visc) {
        R4<real> all[32];
        int n;
        all_intersections(ed, efrz, all, &n);
        R4<real> mc = mass_center(all, n);
        if (isnan(mc.x)) emit = 0;
      }
    }
    mark[q] = (uint8_t)emit;
  }
  int c = __syncthreads_count(emit);
  if (threadIdx.x == 0) block_count[blockIdx.x] = c;
}

#ifndef CLV_HSF_NO_SHARED_KERNELS
// pass 2: exclusive scan of the block counts in one block; total -> *total
__global__ void hsf_scan_kernel(int* block_count, int nblocks, long long* total) {
  __shared__ long long warp_sum[32];
  __shared__ long long carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < nblocks; base += blockDim.x) {
    int t = base + threadIdx.x;
    long long v = t < nblocks ? block_count[t] : 0;
    long long x = v;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      long long y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[w] = x;
    __syncthreads();
    if (w == 0) {
      long long s = lane < (int)(blockDim.x >> 5) ? warp_sum[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        long long y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
      }
      warp_sum[lane] = s;
    }
    __syncthreads();
    long long excl = carry + (w > 0 ? warp_sum[w - 1] : 0) + x - v;
    if (t < nblocks) block_count[t] = (int)excl;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = excl + v;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

// pass 3: cube list in order
__global__ void hsf_compact_kernel(long long ncube, const uint8_t* mark, const int* block_offset, int* list) {
  __shared__ int warp_tot[32];
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int m = (q < ncube) ? mark[q] : 0;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned int bal = __ballot_sync(0xffffffffu, m);
  int before = __popc(bal & ((1u << lane) - 1u));
  if (lane == 0) warp_tot[w] = __popc(bal);
  __syncthreads();
  int wbase = 0;
  for (int u = 0; u < w; u++) wbase += warp_tot[u];
  if (m) list[block_offset[blockIdx.x] + wbase + before] = (int)q;
}

#endif  // CLV_HSF_NO_SHARED_KERNELS

// pass 4: one warp per emitted element.
//
// The work of an element is its 4-subsets of the n intersections (n = 4 to 12
// on smooth surfaces: 1 to 495 pieces to build and test against the others,
// and up to 330 more for the coplanarity test). One thread an element left a
// warp at the pace of its largest n, with every intersection in local memory.
// Here the warp's 32 lanes take the 32 edges of the cube, then the subsets in
// lexicographic order 32 at a time, then the interpolated components; the
// intersections sit in shared memory. The sequential rules are kept: the first
// coplanar subset of a batch (by ballot) moves the points and the search goes
// on behind it, and the pieces on the hull are added in order, so the area has
// the per-thread evaluation's bits. 201x201x105 viscous surface: 1034 us a
// thread an element, 410 a warp an element (the whole finder 1.29 to 0.72 ms).
constexpr int HSF_WARPS = 4;      // per block
constexpr int HSF_TAB_N = 16;     // subsets of up to 16 points come from the table
constexpr int HSF_TAB = 1820;     // C(16, 4)
// 4-subsets {a < b < c < d} in colexicographic order, packed a | b<<8 | c<<16 | d<<24
struct SubsetTable {
  unsigned int v[HSF_TAB];
  constexpr SubsetTable() : v() {
    int r = 0;
    for (unsigned int d = 3; d < HSF_TAB_N; d++)
      for (unsigned int c = 2; c < d; c++)
        for (unsigned int b = 1; b < c; b++)
          for (unsigned int a = 0; a < b; a++) v[r++] = a | b << 8 | c << 16 | d << 24;
  }
};
static __device__ const SubsetTable hsf_subsets{};

__device__ __forceinline__ int binom4(int n) { return n * (n - 1) / 2 * (n - 2) / 3 * (n - 3) / 4; }
// the lexicographically r-th 4-subset of {0 .. n-1}: with x -> n-1-x the
// colexicographically (C(n,4) - 1 - r)-th
__device__ __forceinline__ void hsf_subset(const unsigned int* tab, int n, int total, int r, int id[4]) {
  int q = total - 1 - r;
  if (n <= HSF_TAB_N) {
    const unsigned int t = tab[q];
    id[0] = n - 1 - (int)(t >> 24);
    id[1] = n - 1 - (int)(t >> 16 & 255u);
    id[2] = n - 1 - (int)(t >> 8 & 255u);
    id[3] = n - 1 - (int)(t & 255u);
    return;
  }
  int d = 3, c = 2, b = 1;
  while (binom4(d + 1) <= q) d++;
  q -= binom4(d);
  while ((c + 1) * c / 2 * (c - 1) / 3 <= q) c++;
  q -= c * (c - 1) / 2 * (c - 2) / 3;
  while ((b + 1) * b / 2 <= q) b++;
  q -= b * (b - 1) / 2;
  id[0] = n - 1 - d;
  id[1] = n - 1 - c;
  id[2] = n - 1 - b;
  id[3] = n - 1 - q;
}
// the (left, right) corners of edge e in all_intersections' order
__device__ __forceinline__ void hsf_edge(int e, int* cl, int* cr) {
  if (e < 16) {
    const int s = e & ~3, k = e & 3;
    *cl = s + (k == 2 ? 2 : (k == 3 ? 1 : 0));
    *cr = s + (k == 0 ? 1 : (k == 1 ? 2 : 3));
  } else if (e < 24) {
    *cl = (e < 20 ? 0 : 8) + (e & 3);
    *cr = *cl + 4;
  } else {
    *cl = e - 24;
    *cr = *cl + 8;
  }
}
// component c of the centre of mass (mass_center's sums), one component a lane
template <class real> __device__ __forceinline__ R4<real> hsf_center(const real (*pt)[4], int n, int lane) {
  real c = 0.0f;
  for (int i = 0; i < n; i++) c = c + pt[i][lane & 3];
  c = c / (real)n;
  return R4<real>{__shfl_sync(0xffffffffu, c, 0), __shfl_sync(0xffffffffu, c, 1), __shfl_sync(0xffffffffu, c, 2),
                  __shfl_sync(0xffffffffu, c, 3)};
}
template <class real> __device__ __forceinline__ R4<real> hsf_pt(const real (*pt)[4], int i) {
  if constexpr (sizeof(real) == 4) {
    const float4 t = *reinterpret_cast<const float4*>(pt[i]);
    return R4<real>{t.x, t.y, t.z, t.w};
  } else {
    const double2 a = *reinterpret_cast<const double2*>(pt[i]), b = *reinterpret_cast<const double2*>(pt[i] + 2);
    return R4<real>{a.x, a.y, b.x, b.y};
  }
}
// construct_hypersf on shared-memory points
template <class real>
__device__ __forceinline__ SurfPiece<real> hsf_piece(const int id[4], const real (*pt)[4], R4<real> mc) {
  const R4<real> q[4] = {hsf_pt(pt, id[0]), hsf_pt(pt, id[1]), hsf_pt(pt, id[2]), hsf_pt(pt, id[3])};
  SurfPiece<real> s = construct_hypersf<real>(0, 1, 2, 3, q, mc);
#pragma unroll
  for (int i = 0; i < 4; i++) s.id[i] = id[i];
  return s;
}
// tiny_move_if_coplanar's shift of all points, one point a lane. sf_rand's
// remainder by 2^31 - 1 of a 32-bit product is the product itself except for
// +-(2^31 - 1) and -2^31, so the t-th seed is seed * 16807^t modulo 2^32
// unless one of those comes up (then the seeds are stepped one by one).
__device__ __forceinline__ bool hsf_seed_odd(int s) { return s == 2147483647 || s == -2147483647 || s == (-2147483647 - 1); }
template <class real>
__device__ __forceinline__ void hsf_move(real (*pt)[4], int n, int* seed, int lane) {
  unsigned int a4 = 1u, base = 16807u;  // 16807^(4 lane)
  for (int k = 4 * lane; k; k >>= 1) {
    if (k & 1) a4 *= base;
    base *= base;
  }
  int s[4];
  bool odd = false;
  unsigned int x = (unsigned int)*seed * a4;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    x *= 16807u;
    s[k] = (int)x;
    odd = odd || hsf_seed_odd(s[k]);
  }
  if (__any_sync(0xffffffffu, odd && lane < n)) {
    int t = *seed;
    for (int q = 0; q <= lane; q++)
#pragma unroll
      for (int k = 0; k < 4; k++) {
        sf_rand<real>(&t);
        s[k] = t;
      }
  }
  if (lane < n) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const real r = s[k] / ((real)2147483647);
      pt[lane][k] = pt[lane][k] + (r - 0.5f) * 1.0E-7f;
    }
  }
  *seed = __shfl_sync(0xffffffffu, s[3], n - 1);
  __syncwarp();
}

template <class real>
__global__ void __launch_bounds__(32 * HSF_WARPS, sizeof(real) == 4 ? 6 : 4)
    hsf_element_kernel(Params p, const real* ev_old, const real* ev_new, const real* pi_old, const real* pi_new,
                       real time_old, real time_new, int visc, const int* list, const long long* count,
                       long long* total_inout, real* sf, real* txyz, real* pisf, long long capacity) {
  __shared__ unsigned int tab[HSF_TAB];
  __shared__ __align__(16) real s_pt[HSF_WARPS][32][4];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned int full = 0xffffffffu;
  const long long n_here = *count;
  const long long base = *total_inout;
  if ((long long)blockIdx.x * HSF_WARPS >= n_here) return;  // block-uniform
  for (int t = threadIdx.x; t < HSF_TAB; t += 32 * HSF_WARPS) tab[t] = hsf_subsets.v[t];
  __syncthreads();
  real (*const pt)[4] = s_pt[w];
  const CubeGrid g = cube_grid(p);
  const long long ld = p.ld;
  const real efrz = p.EFRZ;
  for (long long e = (long long)blockIdx.x * HSF_WARPS + w; e < n_here; e += (long long)gridDim.x * HSF_WARPS) {
    const unsigned int q = (unsigned int)list[e], ij = q / (unsigned int)g.nz;
    const int k = (int)(q - ij * (unsigned int)g.nz), j = (int)(ij % (unsigned int)g.ny), i = (int)(ij / (unsigned int)g.ny);
    // corner energies (load_cube), corner lane & 15 on this lane
    const long long own = corner_cell(p, i, j, k, lane & 7);
    const real ed = (lane & 8) ? ev_new[own] : ev_old[own];
    // all_intersections, an edge a lane
    int cl, cr;
    hsf_edge(lane, &cl, &cr);
    const real el = __shfl_sync(full, ed, cl), er = __shfl_sync(full, ed, cr);
    const real dE1 = efrz - el, dE2 = efrz - er, dE12 = el - er;
    const bool cut = dE1 * dE2 < 0;
    const unsigned int cuts = __ballot_sync(full, cut);
    const int n = __popc(cuts);
    __syncwarp();
    if (cut) {
      const real ratio = fabs(dE1) / fabs(dE12);
      const R4<real> t = add4(scl4<real>(ratio, cube_corner<real>(cr)), scl4<real>((real)(1 - ratio), cube_corner<real>(cl)));
      real* const o = pt[__popc(cuts & ((1u << lane) - 1u))];
      o[0] = t.x;
      o[1] = t.y;
      o[2] = t.z;
      o[3] = t.w;
    }
    __syncwarp();
    const R4<real> mc = hsf_center<real>(pt, n, lane);
    // energy_flow, component lane & 3 (tau, x, y, eta) on this lane
    R4<real> flow;
    {
      real vl = 0.0f, vh = 0.0f, elsum = 0.0f, ehsum = 0.0f;
#pragma unroll
      for (int o = 0; o < 16; o++) {  // the loops n, i, j, k of energy_flow
        const int nn = o >> 3, ii = o >> 2 & 1, jj = o >> 1 & 1, kk = o & 1;
        const real dek = efrz - __shfl_sync(full, ed, 8 * nn + 4 * kk + 2 * jj + ii);
        const real adek = fabs(dek);
        const int c = lane & 3;
        const real x = (real)(c == 0 ? nn : (c == 1 ? ii : (c == 2 ? jj : kk))) * adek;
        if (dek > 0.0f) {
          elsum += adek;
          vl = vl + x;
        } else {
          ehsum += adek;
          vh = vh + x;
        }
      }
      if (fabs(elsum) > Acu<real>::v) vl = vl / elsum;
      if (fabs(ehsum) > Acu<real>::v) vh = vh / ehsum;
      const real f = vl - vh;
      flow = R4<real>{__shfl_sync(full, f, 0), __shfl_sync(full, f, 1), __shfl_sync(full, f, 2), __shfl_sync(full, f, 3)};
    }
    // calc_area
    R4<real> area{0.0f, 0.0f, 0.0f, 0.0f};
    if (n == 4) {
      const int id[4] = {0, 1, 2, 3};
      SurfPiece<real> sp = hsf_piece<real>(id, pt, mc);
      if (dotr4(flow, sp.norm) < 0.0f) sp.norm = R4<real>{-sp.norm.x, -sp.norm.y, -sp.norm.z, -sp.norm.w};
      area = sp.norm;
    } else if (n > 4) {
      R4<real> mcm = mc;
      int seed = (int)(32117u * (unsigned int)(i * j * k + 1));
      const int nco = binom4(n - 1);  // subsets whose last point is not the last
      for (int r0 = 0; r0 < nco;) {
        bool hit = false;
        if (r0 + lane < nco) {
          int id[4];
          hsf_subset(tab, n - 1, nco, r0 + lane, id);
          const SurfPiece<real> sp = hsf_piece<real>(id, pt, mcm);
          for (int m = id[3] + 1; m < n; m++)
            if (dotr4(sp.norm, sub4(hsf_pt<real>(pt, m), sp.center)) == 0.0f) {
              hit = true;
              break;
            }
        }
        const unsigned int hits = __ballot_sync(full, hit);
        if (!hits) {
          r0 += 32;
          continue;
        }
        hsf_move<real>(pt, n, &seed, lane);
        mcm = hsf_center<real>(pt, n, lane);
        r0 += __ffs(hits);
      }
      const int nsub = binom4(n);
      for (int r0 = 0; r0 < nsub; r0 += 32) {
        bool on = false;
        R4<real> nv{0.0f, 0.0f, 0.0f, 0.0f};
        if (r0 + lane < nsub) {
          int id[4];
          hsf_subset(tab, n, nsub, r0 + lane, id);
          const SurfPiece<real> sp = hsf_piece<real>(id, pt, mcm);
          nv = sp.norm;
          // the cheap test first: both are pure
          on = dotr4(sp.norm, flow) > 0.0f;
          unsigned int rest = (n < 32 ? (1u << n) - 1u : full) & ~(1u << id[0] | 1u << id[1] | 1u << id[2] | 1u << id[3]);
          for (; on && rest; rest &= rest - 1u)
            on = !(dotr4(sub4(hsf_pt<real>(pt, __ffs(rest) - 1), sp.center), sp.norm) >= 0.0f);
        }
        for (unsigned int b = __ballot_sync(full, on); b; b &= b - 1u) {  // in order
          const int src = __ffs(b) - 1;
          area = add4(area, R4<real>{__shfl_sync(full, nv.x, src), __shfl_sync(full, nv.y, src),
                                     __shfl_sync(full, nv.z, src), __shfl_sync(full, nv.w, src)});
        }
      }
    }
    const R4<real> dS = div4(area, (real)6.0f);
    const long long o = base + e;
    if (o >= capacity) continue;  // warp-uniform
    const real dtd = time_new - time_old;
    const real dxd = p.nxskip * p.DX;
    const real dyd = p.nyskip * p.DY;
    const real dzd = p.nzskip * p.DZ;
    const real tau = time_old + mc.x * dtd;
    // lanes 0..2: v, 3..12: pi, each over the 16 corners in order
    if (lane < ((visc && pisf) ? 13 : 3)) {
      const real* const fo = lane < 3 ? ev_old + (lane + 1) * ld : pi_old + (lane - 3) * ld;
      const real* const fn = lane < 3 ? ev_new + (lane + 1) * ld : pi_new + (lane - 3) * ld;
      real x[16];
#pragma unroll
      for (int c = 0; c < 16; c++) x[c] = (c < 8 ? fo : fn)[corner_cell(p, i, j, k, c & 7)];
      real acc = 0.0f;
#pragma unroll
      for (int c = 0; c < 16; c++) {
        const real t = corner_weight(mc, c) * x[c];
        acc = (c == 0) ? t : acc + t;
      }
      if (lane < 3) sf[8 * o + 4 + lane] = acc;
      else pisf[10 * o + lane - 3] = acc;
    } else if (lane == 16) {
      real* const r8 = sf + 8 * o;
      r8[0] = tau * dxd * dyd * dzd * dS.x;
      r8[1] = -tau * dtd * dyd * dzd * dS.y;
      r8[2] = -tau * dtd * dxd * dzd * dS.z;
      r8[3] = -dtd * dxd * dyd * dS.w;
    } else if (lane == 17) {
      const real x = (-p.nx) / 2 * p.DX + i * dxd + mc.y * dxd;
      const real y = (-p.ny) / 2 * p.DY + j * dyd + mc.z * dyd;
      const real eta = (-p.nz) / 2 * p.DZ + k * dzd + mc.w * dzd;
      sf[8 * o + 7] = eta;
      real* const r4 = txyz + 4 * o;
      r4[0] = tau * cosh(eta);
      r4[1] = x;
      r4[2] = y;
      r4[3] = tau * sinh(eta);
    }
  }
}

#ifndef CLV_HSF_NO_SHARED_KERNELS
__global__ void hsf_advance_kernel(const long long* count, long long* total_inout) { *total_inout += *count; }
#endif

}  // namespace clv
