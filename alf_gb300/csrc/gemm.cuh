// Batched complex128 GEMM on the FP64 tensor path (mma.sync m8n8k4 f64, DMMA).
//
//   C = alpha * rs .* ( op(A) * diag(ks) * op(B) ) .* cs + beta * C
//
// with op in {N, T, C}, either operand optionally real (the ZLARCM/ZLACRM case
// of ALF's dense hopping products, Libraries/Modules/Mat_subroutines_mod.F90:1225-1418),
// an optional K-dimension gather on either operand (ZLAPMR/ZLAPMT row/column
// permutations folded into the load), an optional "stored upper triangular"
// mask (ZTRMM with R kept above the Householder vectors), per-batch K read from
// device memory (delayed-update flushes whose rank differs per chain), and a
// row/column scaling epilogue (the D scalings of CGR, Prog/cgr1_mod.F90:233-236).
#pragma once
#include <type_traits>

#include "common.cuh"

enum { OP_N = 0, OP_T = 1, OP_C = 2 };

struct GemmParams {
  int m, n, k;
  const void* A; long long lda, sA; int opA, realA, triA;
  const void* B; long long ldb, sB; int opB, realB, triB;
  zd* C; long long ldc, sC;
  zd alpha, beta;
  const zd* ks; long long sKS; int ksOnA, ksConj, ksInv;
  const zd* rs; long long sRS; int rsInv;
  const zd* cs; long long sCS; int csInv;
  const int* permA; long long sPA;
  const int* permB; long long sPB;
  const int* kdyn;  // per-batch K (<= k) or null
  int batch;
  int modA, modB;   // if > 0, operand batch index = b % mod (an operand shared across chains)
};

static inline GemmParams gemm_defaults() {
  GemmParams p;
  memset(&p, 0, sizeof(p));
  p.alpha = zmk(1.0, 0.0);
  p.beta = zmk(0.0, 0.0);
  p.batch = 1;
  return p;
}

ALF_DEV void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// alpha rs v cs + beta C of a real product.
ALF_DEV double gemm_real_out(const GemmParams& p, double v, const zd* rs, int row, const zd* cs, int col, bool usebeta,
                             const zd* cp) {
  if (rs) v = p.rsInv ? v / rs[row].x : rs[row].x * v;
  if (cs) v = p.csInv ? v / cs[col].x : v * cs[col].x;
  v *= p.alpha.x;
  return usebeta ? fma(p.beta.x, cp->x, v) : v;
}

ALF_DEV zd gemm_cplx_out(const GemmParams& p, zd v, const zd* rs, int row, const zd* cs, int col, bool usebeta,
                         const zd* cp) {
  if (rs) v = p.rsInv ? zdiv(v, rs[row]) : zmul(rs[row], v);
  if (cs) v = p.csInv ? zdiv(v, cs[col]) : zmul(v, cs[col]);
  v = zmul(p.alpha, v);
  return usebeta ? zadd(v, zmul(p.beta, *cp)) : v;
}

// Product on 16 x 16 tiles: four 8 x 8 quadrants times WK slices of K, one warp each, and a warp each
// for the real and the imaginary part of a complex product.  A DMMA holds its sub-partition ~577 cycles, so what counts is how evenly the
// m n K / 256 DMMAs (two or four times as many complex) are dealt to the 608 sub-partitions; the
// operands (KC K steps staged at once) come from L2.  RE: every operand and the output are real
// (complex128 storage with zero imaginary parts, or float64).
// grid (ceil(n/16), ceil(m/16), batch), 128 WK threads real, 256 WK complex.
template <int WK, bool RE>
__global__ void __launch_bounds__((RE ? 128 : 256) * WK) k_gemm16(GemmParams p) {
  constexpr int NP = RE ? 1 : 2, KC = RE ? 64 : 32, NT = 128 * NP * WK, AE = 16 * KC / NT, QW = 4 * NP;
  __shared__ double As[NP][KC][20], Bs[NP][KC][20];
  __shared__ double red[WK > 1 ? WK - 1 : 1][QW][64];
  const int b = blockIdx.z, m0 = blockIdx.y * 16, n0 = blockIdx.x * 16;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int qm = (warp & 1) * 8, qn = ((warp >> 1) & 1) * 8, im = RE ? 0 : (warp >> 2) & 1, sl = warp / QW;
  const int g = lane >> 2, t = lane & 3;
  const int K = p.kdyn ? min(p.kdyn[b], p.k) : p.k;
  const int bA = p.modA > 0 ? b % p.modA : b, bB = p.modB > 0 ? b % p.modB : b;
  const void* A = p.realA ? (const void*)((const double*)p.A + bA * p.sA) : (const void*)((const zd*)p.A + bA * p.sA);
  const void* B = p.realB ? (const void*)((const double*)p.B + bB * p.sB) : (const void*)((const zd*)p.B + bB * p.sB);
  const zd* ks = p.ks ? p.ks + b * p.sKS : nullptr;
  const int* pA = p.permA ? p.permA + b * p.sPA : nullptr;
  const int* pB = p.permB ? p.permB + b * p.sPB : nullptr;
  typedef typename std::conditional<RE, double, zd>::type E;  // a staged element
  auto ld = [](const void* X, int isreal, int op, long long e) -> E {
    if constexpr (RE) {
      return isreal ? ((const double*)X)[e] : ((const zd*)X)[e].x;
    } else {
      if (isreal) return zmk(((const double*)X)[e], 0.0);
      zd v = ((const zd*)X)[e];
      if (op == OP_C) v.y = -v.y;
      return v;
    }
  };
  auto scl = [&](E v, int k) -> E {
    if constexpr (RE) {
      return p.ksInv ? v / ks[k].x : v * ks[k].x;
    } else {
      zd s = ks[k];
      if (p.ksConj) s.y = -s.y;
      return p.ksInv ? zdiv(v, s) : zmul(v, s);
    }
  };
  auto put = [&](double (*X)[KC][20], int kk, int i, E v) {
    if constexpr (RE) {
      X[0][kk][i] = v;
    } else {
      X[0][kk][i] = v.x;
      X[NP - 1][kk][i] = v.y;
    }
  };
  // the warp's part: real  Ar Br - Ai Bi,  imaginary  Ar Bi + Ai Br
  const bool first = RE || !im || !p.realB, second = !RE && !p.realA && (im || !p.realB);
  const int sgn = im ? 0 : (int)0x80000000u;
  double d0 = 0.0, d1 = 0.0;
  for (int k0 = 0; k0 < K; k0 += KC) {
    E ra[AE], rb[AE];
#pragma unroll
    for (int r = 0; r < AE; ++r) {
      const int e = tid + r * NT;
      const int i = p.opA == OP_N ? e % 16 : e / KC, kk = p.opA == OP_N ? e / 16 : e % KC;
      E v = E();
      if (m0 + i < p.m && k0 + kk < K) {
        const int kq = pA ? pA[k0 + kk] : k0 + kk;
        const long long rr = p.opA == OP_N ? m0 + i : kq, cc = p.opA == OP_N ? kq : m0 + i;
        if (!(p.triA && rr > cc)) v = ld(A, p.realA, p.opA, rr + cc * p.lda);
        if (ks && p.ksOnA) v = scl(v, k0 + kk);
      }
      ra[r] = v;
      const int j = p.opB == OP_N ? e / KC : e % 16, kb = p.opB == OP_N ? e % KC : e / 16;
      v = E();
      if (n0 + j < p.n && k0 + kb < K) {
        const int kq = pB ? pB[k0 + kb] : k0 + kb;
        const long long rr = p.opB == OP_N ? kq : n0 + j, cc = p.opB == OP_N ? n0 + j : kq;
        if (!(p.triB && rr > cc)) v = ld(B, p.realB, p.opB, rr + cc * p.ldb);
        if (ks && !p.ksOnA) v = scl(v, k0 + kb);
      }
      rb[r] = v;
    }
    if (k0) __syncthreads();
#pragma unroll
    for (int r = 0; r < AE; ++r) {
      const int e = tid + r * NT;
      if (p.opA == OP_N) put(As, e / 16, e % 16, ra[r]);
      else put(As, e % KC, e / KC, ra[r]);
      if (p.opB == OP_N) put(Bs, e % KC, e / KC, rb[r]);
      else put(Bs, e / 16, e % 16, rb[r]);
    }
    __syncthreads();
    const int kend = min(KC, K - k0);
    for (int k4 = 4 * sl; k4 < kend; k4 += 4 * WK) {
      if (first) dmma(d0, d1, As[0][k4 + t][qm + g], Bs[im][k4 + t][qn + g]);
      if (second) {
        const double a = As[NP - 1][k4 + t][qm + g];
        dmma(d0, d1, __hiloint2double(__double2hiint(a) ^ sgn, __double2loint(a)), Bs[NP - 1 - im][k4 + t][qn + g]);
      }
    }
  }
  if (WK > 1) {
    if (sl > 0) { red[sl - 1][warp % QW][2 * lane] = d0; red[sl - 1][warp % QW][2 * lane + 1] = d1; }
    __syncthreads();
    if (sl == 0) {
#pragma unroll
      for (int s = 0; s < WK - 1; ++s) { d0 += red[s][warp][2 * lane]; d1 += red[s][warp][2 * lane + 1]; }
    }
  }
  if (!RE) {  // the imaginary parts join the real parts' warps
    if (WK > 1) __syncthreads();
    if (sl == 0 && im) { red[0][warp][2 * lane] = d0; red[0][warp][2 * lane + 1] = d1; }
    __syncthreads();
  }
  if (sl > 0 || im) return;
  const zd* rs = p.rs ? p.rs + b * p.sRS : nullptr;
  const zd* cs = p.cs ? p.cs + b * p.sCS : nullptr;
  const bool usebeta = p.beta.x != 0.0 || (!RE && p.beta.y != 0.0);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int row = m0 + qm + g, col = n0 + qn + 2 * t + h;
    if (row >= p.m || col >= p.n) continue;
    zd* cp = p.C + b * p.sC + row + (long long)col * p.ldc;
    if constexpr (RE) {
      *cp = zmk(gemm_real_out(p, h ? d1 : d0, rs, row, cs, col, usebeta, cp), 0.0);
    } else {
      *cp = gemm_cplx_out(p, zmk(h ? d1 : d0, red[0][warp + 4][2 * lane + h]), rs, row, cs, col, usebeta, cp);
    }
  }
}

// WK, the slices of K: two or four fill the sub-partitions when there are few tiles.  Measured, complex
// products of B matrices, one / two slices: N = 72, B = 4 (100 tiles) 31 / 29 us, N = 128, B = 16 (1024) 328 /
// 293, N = 256, B = 8 (2048) 1124 / 1129.  64 x 64 tiles, which read a quarter as often, took 418, 664 and
// 1289 us, and were ahead (by 9% at most) only where their last wave happens to be full.  One chain's
// wrap of a real model (two products, two flavours): N = 16 14.7 us, N = 256 248 us.
template <bool RE>
static inline cudaError_t launch_zgemm_as(const GemmParams& p, cudaStream_t st) {
  const dim3 grid((p.n + 15) / 16, (p.m + 15) / 16, p.batch);
  const long long t16 = (long long)grid.x * grid.y * grid.z;
  constexpr int nt = RE ? 128 : 256;
  if constexpr (RE) {
    if (t16 * 2 <= 152 && p.k > 8) {
      k_gemm16<4, RE><<<grid, 4 * nt, 0, st>>>(p);
      return cudaGetLastError();
    }
  }
  if (t16 <= (RE ? 2 : 8) * 152 && p.k > 4) k_gemm16<2, RE><<<grid, 2 * nt, 0, st>>>(p);
  else k_gemm16<1, RE><<<grid, nt, 0, st>>>(p);
  return cudaGetLastError();
}

static inline cudaError_t launch_zgemm(const GemmParams& p, cudaStream_t st, int real) {
  if (p.m <= 0 || p.n <= 0 || p.batch <= 0) return cudaSuccess;
  return real ? launch_zgemm_as<true>(p, st) : launch_zgemm_as<false>(p, st);
}
