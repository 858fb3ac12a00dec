// Test-only kernel: the tolerance build's EOS lookup on given energy densities.
#define CLV_FAST 1
#include "../../clvisc_b200/csrc/clv_device.cuh"

template <class real> __global__ void lookup(clv::Params p, const real* e, int n, real* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) clv::eos_texel4<real>(p, e[i], out + 4 * i);
}

// host pointers; the table's recorded sizes as clv_params has them
template <class real>
int run(const float* table, int nrow, int ncol, float start, float step, int num, float top, float inner, const real* e,
        int n, real* out) {
  clv::Params p = {};
  float* t;
  real *de, *dout;
  cudaMalloc(&t, sizeof(float) * 4 * nrow * ncol);
  cudaMalloc(&de, sizeof(real) * n);
  cudaMalloc(&dout, sizeof(real) * 4 * n);
  cudaMemcpy(t, table, sizeof(float) * 4 * nrow * ncol, cudaMemcpyHostToDevice);
  cudaMemcpy(de, e, sizeof(real) * n, cudaMemcpyHostToDevice);
  p.eos = t;
  p.eos_start = start;
  p.eos_step = step;
  p.eos_num = num;
  p.eos_nrow = nrow;
  p.eos_ncol = ncol;
  p.eos_last = nrow * ncol - 1;
  p.eos_top = top;
  p.eos_inner = inner;
  const float epr = step * ncol;
  p.rf.eos_step = 1.0f / step;
  p.rf.eos_epr = 1.0f / epr;
  p.rd.eos_step = 1.0 / (double)step;
  p.rd.eos_epr = 1.0 / (double)epr;
  lookup<real><<<(n + 127) / 128, 128>>>(p, de, n, dout);
  cudaMemcpy(out, dout, sizeof(real) * 4 * n, cudaMemcpyDeviceToHost);
  cudaFree(t);
  cudaFree(de);
  cudaFree(dout);
  return (int)cudaGetLastError();
}
extern "C" int run_f64(const float* table, int nrow, int ncol, float start, float step, int num, float top, float inner,
                       const double* e, int n, double* out) {
  return run<double>(table, nrow, ncol, start, step, num, top, inner, e, n, out);
}
