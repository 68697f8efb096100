// Q of a QR factorisation applied to columns (ZUNMQR 'L', 'N'), or formed (ZUNGQR), reflector by
// reflector in reverse order, in one launch over all panels of 32 reflectors.
#pragma once
#include "arith.cuh"

struct QApplyParams {
  const zd* V; long long ldv, sV;  // reflectors below the diagonal (unit diagonal implied)
  const zd* tau; long long sT;
  zd* C; long long ldc, sC;
  int N;                           // rows, columns and reflectors
  int init;                        // C starts as the identity (explicit Q)
};

static inline size_t qap_smem_bytes(int N, int zb) { return ((size_t)((N + 31) / 32) * 32 * 32 + 32) * zb; }

// The reflectors n - 1 .. 0 of a staged panel on CW columns of NB active row blocks each, held bottom up
// (x[.][i]: block i from the last); v: lane's entry of the last block of reflector 0.  The next
// reflector is loaded while the FP64 pipe works on this one.
ALF_DEV bool qap_zero(double t) { return (__double_as_longlong(t) << 1) == 0; }
ALF_DEV bool qap_zero(zd t) { return qap_zero(t.x) && qap_zero(t.y); }
template <class A, int NB, int QW, int CW>
ALF_DEV void qap_panel(typename A::Z (&x)[CW][QW], const typename A::Z* v, int ldv, const typename A::Z* tq, int n) {
  typedef typename A::Z Z;
  constexpr int P = A::kReal ? 1 : 2;
  constexpr int per = 32 / (CW * P);  // lanes that hold one total
  Z vn[NB], tn = tq[n - 1];
#pragma unroll
  for (int i = 0; i < NB; ++i) vn[i] = v[(n - 1) * ldv - 32 * i];
#pragma unroll 1
  for (int k = n - 1; k >= 0; --k) {
    Z vq[NB];
    const Z t = tn;
#pragma unroll
    for (int i = 0; i < NB; ++i) vq[i] = vn[i];
    if (k > 0) {
      tn = tq[k - 1];
#pragma unroll
      for (int i = 0; i < NB; ++i) vn[i] = v[(k - 1) * ldv - 32 * i];
    }
    if (qap_zero(t)) continue;  // uniform
    Z s[CW];
#pragma unroll
    for (int u = 0; u < CW; ++u) s[u] = A::zero();
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
      for (int u = 0; u < CW; ++u) s[u] = A::mac(s[u], A::conj(vq[i]), x[u][i]);
    double d[CW * P];
#pragma unroll
    for (int u = 0; u < CW; ++u) {
      d[u * P] = A::re(s[u]);
      if (P == 2) d[u * P + P - 1] = A::im(s[u]);
    }
    const double tot = warp_sum_packed<CW * P>(d);
    Z f[CW];
    if constexpr (A::kReal) {
      const Z g = A::neg(A::mul(t, tot));  // each lane for its column
#pragma unroll
      for (int u = 0; u < CW; ++u) f[u] = CW == 1 ? g : A::shfl(g, u * per);
    } else {
      const int my = threadIdx.x & 31 & ~(2 * per - 1);
      const Z g = A::neg(A::mul(t, A::mkz(__shfl_sync(0xffffffffu, tot, my), __shfl_sync(0xffffffffu, tot, my + per))));
#pragma unroll
      for (int u = 0; u < CW; ++u) f[u] = CW == 1 ? g : A::shfl(g, 2 * u * per);
    }
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
      for (int u = 0; u < CW; ++u) x[u][i] = A::mac(x[u][i], vq[i], f[u]);
  }
}
template <class A, int NB, int QW, int CW>
ALF_DEV void qap_dispatch(int nb, typename A::Z (&x)[CW][QW], const typename A::Z* v, int ldv, const typename A::Z* tq, int n) {
  if (nb == NB) qap_panel<A, NB, QW, CW>(x, v, ldv, tq, n);
  else if constexpr (NB > 1) qap_dispatch<A, NB - 1, QW, CW>(nb, x, v, ldv, tq, n);
}

// A warp holds CW columns in registers from the last reflector to the first (lane l: rows l + 32 i); the
// CTA's warps share a panel, staged in shared memory with its unit diagonal and zeros written out.
// The FP64 pipe bounds it (an instruction of one warp holds its sub-partition ~64 cycles): 2 r products
// per column and reflector of r 32-row blocks, and 5 (one or two columns) or 6 (four) additions of
// the packed reduction and one factor per warp.  Compact WY in FP64 would save most of those too, but
// doubled the error of G (4 x 4 Hubbard model, beta = 2, against the oracle).
// Measured, one Q of real matrices, a launch per panel -> this: N = 256, two 400 -> 238 us, 32 1740 ->
// 1213 us (two columns per warp); N = 576, two (all columns) 2490 -> 1336 us.
// grid (ceil(N / (CW warps)), B), the columns with the most reflectors first; dynamic shared memory
// qap_smem_bytes; N <= 32 QW.
template <class A, int QW, int CW>
__global__ void __launch_bounds__(256) k_q_apply(QApplyParams p) {
  typedef typename A::Z Z;
  const int b = blockIdx.y, N = p.N, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int cb = (int)(gridDim.x - 1 - blockIdx.x) * nw * CW, c = cb + warp * CW;
  const int nblk = (N + 31) >> 5;
  extern __shared__ __align__(16) unsigned char qap_raw[];
  Z* tq = reinterpret_cast<Z*>(qap_raw);  // [k]
  Z* Vs = tq + 32;                        // [k][32 blocks]
  const zd* V = p.V + b * p.sV;
  zd* col = p.C + b * p.sC + (long long)c * p.ldc;
  Z x[CW][QW];  // blocks bottom up, so that a panel's active ones come first
#pragma unroll
  for (int u = 0; u < CW; ++u)
#pragma unroll
    for (int i = 0; i < QW; ++i) {
      const int r = 32 * (nblk - 1 - i) + lane;
      x[u][i] = A::zero();
      if (c + u < N && r >= 0 && r < N) x[u][i] = p.init ? (r == c + u ? A::one() : A::zero()) : A::mk(col[r + u * p.ldc]);
    }
  // an explicit column is e_c until its own reflector's panel (a CTA's columns, 32 at most and a power of
  // two, are of one panel)
  for (int pn = p.init ? cb >> 5 : nblk - 1; pn >= 0; --pn) {
    const int j0 = 32 * pn, ldv = 32 * (nblk - pn);
    __syncthreads();
    for (int k = warp; k < 32; k += 2 * nw) {  // two reflectors at a time, their loads in flight together
      const zd* v = V + (long long)(j0 + k) * p.ldv + j0;
#pragma unroll 8
      for (int r = lane; r < ldv; r += 32)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int ku = k + u * nw;
          Vs[ku * ldv + r] = r == ku ? A::one() : (r > ku && j0 + r < N && j0 + ku < N ? A::mk(v[r + u * nw * p.ldv]) : A::zero());
        }
    }
    if (threadIdx.x < 32) tq[lane] = j0 + lane < N ? A::mk(p.tau[b * p.sT + j0 + lane]) : A::zero();
    __syncthreads();
    if (c < N) qap_dispatch<A, QW, QW, CW>(nblk - pn, x, Vs + ldv - 32 + lane, ldv, tq, min(32, N - j0));
  }
#pragma unroll
  for (int u = 0; u < CW; ++u)
    if (c + u < N) {
#pragma unroll
      for (int i = 0; i < QW; ++i) {
        const int r = 32 * (nblk - 1 - i) + lane;
        if (r >= 0 && r < N) col[r + u * p.ldc] = A::wide(x[u][i]);
      }
    }
}
