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
