// Host entry points over the scalar device functions, for tests/test_gpu_scalars.py.
#include "../../alf_gb300/csrc/arith.cuh"

template <class F>
__global__ void k_each(int n, F f) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) f(i);
}
// f(i) for i < n over managed buffers; the first CUDA error, or 0
template <class F>
static int each(int n, F f) {
  k_each<<<304, 256>>>(n, f);
  const cudaError_t e = cudaGetLastError();
  return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
template <class T>
struct Buf {  // a device copy of a host array, written back by out()
  T* d = nullptr;
  T* h;
  size_t n;
  Buf(const T* host, int count) : h(const_cast<T*>(host)), n((size_t)count * sizeof(T)) {
    cudaMalloc(&d, n);
    cudaMemcpy(d, h, n, cudaMemcpyHostToDevice);
  }
  ~Buf() { cudaFree(d); }
  void out() { cudaMemcpy(h, d, n, cudaMemcpyDeviceToHost); }
};

extern "C" int chk_df_make(const double* x, float* hi, float* lo, double* back, int n) {
  Buf<double> bx(x, n), bb(back, n);
  Buf<float> bh(hi, n), bl(lo, n);
  const double* px = bx.d;
  double* pb = bb.d;
  float *ph = bh.d, *pl = bl.d;
  const int rc = each(n, [=] __device__(int i) {
    const dff v = df_make(px[i]);
    ph[i] = v.h;
    pl[i] = v.l;
    pb[i] = df_wide(v);
  });
  bh.out(); bl.out(); bb.out();
  return rc;
}

// out: [5][n] the approximation, this library's and CUDA's reciprocal of x, this library's and CUDA's root of |x|
extern "C" int chk_roots(const double* x, double* out, int n) {
  Buf<double> bx(x, n), bo(out, 5 * n);
  const double* p = bx.d;
  double* o = bo.d;
  const long long m = n;
  const int rc = each(n, [=] __device__(int i) {
    const double y = p[i], t = fabs(y);
    o[i] = alf_rcp_seed(y); o[m + i] = alf_rcp(y); o[2 * m + i] = 1.0 / y;
    o[3 * m + i] = alf_sqrt_n(t, rsqrt(t)); o[4 * m + i] = sqrt(t);
  });
  bo.out();
  return rc;
}
