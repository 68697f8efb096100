// Exact ZGEQP3 (ZLAQP2: dynamic column pivoting with norm downdates,
// Prog/QDRP_decompose_mod.F90:60-101) on one thread-block cluster per matrix, columns dealt
// cyclically to the CTAs (column c -> CTA c % CL) and kept in shared memory.
#pragma once
#include "common.cuh"
#include "arith.cuh"
#include "linalg.cuh"

#define QRC_WORK 256                 // threads that carry FP64 work: two warps per sub-partition
#define QRC_THREADS (QRC_WORK + 32)  // and one warp of integer bookkeeping

struct QRColsParams {
  const zd* Ain;             // input (may equal A)
  zd* A; long long lda, sA;  // output: R above the diagonal, reflectors below
  int N;
  const double* colscale; long long sCS;
  zd* tau; long long sT;
  int* jpvt; long long sP;
  double* D; long long sD;
  QRInfo* info;
};

struct QRCand {  // a CTA's best remaining column, read by its peers
  unsigned long long key;  // squared norm's bits + 1 (0: NaN or none)
  int pos, col;            // its position in the pivoted order, its original index
};

// Column stride: 64 bytes past a multiple of 128, so that the row segments of neighbouring
// columns start on different banks.
static inline __host__ __device__ int qrc_ld(int N, int zb) {
  const int per = 128 / zb;
  return (N + per - 1) / per * per + per / 2;
}
static inline size_t qrc_smem_bytes(int N, int CL, int zb) {
  const size_t nc = (size_t)((N + CL - 1) / CL);
  return nc * qrc_ld(N, zb) * zb + ((size_t)N + 3 * nc + 2) * zb + (3 * nc) * 8 + (3 * nc) * sizeof(int) + 64;
}

template <class Z>
ALF_DEV Z qrc_peer(const Z* p, unsigned rank) {  // a value in a peer CTA's shared memory
  const uint32_t a = dsmem_addr(p, rank);
  double v[sizeof(Z) / 8];
#pragma unroll
  for (int i = 0; i < (int)sizeof(Z) / 8; ++i) v[i] = dsmem_ld_f64(a + 8 * i);
  Z z;
  memcpy(&z, v, sizeof(Z));
  return z;
}

template <class Z>
ALF_DEV Z qrc_shfl_xor(Z v, int o, unsigned m) {  // xor shuffle among the lanes of m
  unsigned w[sizeof(Z) / 4];
  memcpy(w, &v, sizeof(Z));
#pragma unroll
  for (int i = 0; i < (int)sizeof(Z) / 4; ++i) w[i] = __shfl_xor_sync(m, w[i], o);
  memcpy(&v, w, sizeof(Z));
  return v;
}

// Largest key of the warp, the smallest position on ties: integer reductions only.
ALF_DEV void qrc_argmax(unsigned long long& key, int& pos, int& col) {
  const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32));
  const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32) == hi ? (unsigned)key : 0u);
  const unsigned long long best = ((unsigned long long)hi << 32) | lo;
  const int bp = (int)__reduce_min_sync(0xffffffffu, key == best ? (unsigned)pos : 0x7fffffffu);
  const unsigned who = __ballot_sync(0xffffffffu, key == best && pos == bp);
  key = best;
  pos = bp;
  col = __shfl_sync(0xffffffffu, col, __ffs(who) - 1);
}

// The FP64 pipe takes one warp instruction per sub-partition every ~64 cycles, with nothing in
// flight beside it, so a step's cost is the FP64 instructions on its longest sub-partition plus
// the cluster exchange.  Columns in a CTA make every dot product and norm local: per step the
// CTAs exchange one candidate column each (16 bytes) and read the chosen one (N - j values);
// rows in a CTA would exchange a partial sum of every column.  Columns are never moved: a
// column keeps its slot and its position in the pivoted order is tracked beside it, a finished
// one leaves the list of active columns.  The update uses the unscaled column x:
// f = conj(tau) a_j - (x^H a) / beta (tau and scal = 1 / (alpha - beta) give conj(tau scal) =
// -1 / beta), a_j -= f, a_i -= x_i (scal f).  Norms are kept squared and compared as integers.
// Arithmetic A: ArD or ArRe.  Grid (CL, B), QRC_THREADS threads, one cluster barrier per step.
// Measured (GB300, one QR): two 256 x 256 matrices 3.41 ms with rows in the CTAs (k_qrp_rows) ->
// 2.23 ms complex, 1.17 ms real; 32 of them 5.70 -> 1.64 ms (real); two 576 x 576 21.9 -> 4.9 ms
// (real).  Per step at N = 256 (16 CTAs, cycles): barrier 1260, candidates 490, the column 900, dot
// products 2240, scalars 1700, update 2000; eight warps hide each other's loads (four: 1.26 ms).
template <class A>
__global__ void __launch_bounds__(QRC_THREADS) k_qrp_cols(QRColsParams p) {
  typedef typename A::Z Z;
  const unsigned rank = cluster_ctarank(), CL = cluster_nctarank();
  const int b = blockIdx.y, N = p.N, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nc = (N + (int)CL - 1) / (int)CL;                 // slots per CTA
  const int nmine = (N - (int)rank + (int)CL - 1) / (int)CL;  // columns rank, rank + CL, ...
  const int ld = qrc_ld(N, (int)sizeof(Z));
  extern __shared__ __align__(16) unsigned char qrc_raw[];
  Z* cols = reinterpret_cast<Z*>(qrc_raw);  // [nc][ld]
  Z* xb = cols + (size_t)nc * ld;           // [N] the chosen column
  Z* dsh = xb + N;                          // [nc + 1] x^H a of the active columns, x^H x last
  Z* gsh = dsh + nc + 1;                    // [nc] scal f
  Z* scl = gsh + nc;                        // [nc] scal of finished columns
  double* vn1 = reinterpret_cast<double*>(scl + nc + 1);  // [nc] squared norms, -1: to be recomputed
  double* tv2 = vn1 + nc;                                 // [nc] tol3z times the last exact squared norm
  double* bet = tv2 + nc;                                 // [nc] beta of finished columns
  int* pos = reinterpret_cast<int*>(bet + nc);            // [nc] position in the pivoted order
  int* act = pos + nc;                                    // [nc] active slots
  int* fin = act + nc;                                    // [nc] step at which a column was chosen
  __shared__ __align__(16) QRCand cand[2];
  const double tol3z = 1.0536712127723509e-08;  // sqrt(dlamch('Epsilon'))
  const zd* Ab = p.Ain + b * p.sA;
  zd* Ob = p.A + b * p.sA;

  for (int lc = warp; lc < nmine; lc += QRC_THREADS / 32) {
    const int c = (int)rank + lc * (int)CL;
    const double s = p.colscale ? p.colscale[b * p.sCS + c] : 1.0;
    for (int i = lane; i < N; i += 32) {
      zd v = Ab[i + c * p.lda];
      if (p.colscale) v = zscale(v, s);
      cols[(size_t)lc * ld + i] = A::mk(v);
    }
    if (lane == 0) { pos[lc] = c; act[lc] = lc; }
  }
  int nact = nmine;
  __syncthreads();

  // Entries 0 .. ne - 1 by groups of L = 1 << lL lanes, QRC_WORK / L groups: the lane count with
  // the fewest FP64 instructions, ceil(ne / groups) rounds of rows / L products and lL additions.
  auto pick = [&](int ne, int rows) {
    int best = 0x7fffffff, bl = 3;
    for (int l = 1; l <= 5; ++l) {
      const int cost = (((ne << l) + QRC_WORK - 1) / QRC_WORK) * (((rows + (1 << l) - 1) >> l) + l);
      if (cost < best) { best = cost; bl = l; }
    }
    return bl;
  };
  // squared norms over the rows i >= i0 of the active columns (flagged ones only)
  auto norms = [&](int i0, bool flagged, int lL) {
    const int L = 1 << lL, lg = tid & (L - 1);
    for (int t = tid >> lL; t < nact; t += QRC_WORK >> lL) {
      const int lc = act[t];
      if (flagged && !(vn1[lc] < 0.0)) continue;
      const Z* a = cols + (size_t)lc * ld;
      double s = 0.0;
      for (int i = i0 + lg; i < N; i += L) s += A::abs2(a[i]);
      const unsigned gm = (L == 32 ? 0xffffffffu : ((1u << L) - 1u) << (lane & ~(L - 1)));
      for (int o = 1; o < L; o <<= 1) s += __shfl_xor_sync(gm, s, o);
      __syncwarp(gm);  // every lane of the group has read the flag
      if (lg == 0) { vn1[lc] = s; tv2[lc] = tol3z * s; }
    }
  };
  // the CTA's candidate for the next step (the bookkeeping warp)
  auto post = [&](int par) {
    unsigned long long key = 0;
    int bp = 0x7fffffff, bc = -1;
    for (int t = lane; t < nact; t += 32) {
      const int lc = act[t];
      const unsigned long long v = (unsigned long long)__double_as_longlong(vn1[lc]) & 0x7fffffffffffffffull;
      const unsigned long long k = v > 0x7ff0000000000000ull ? 0ull : v + 1ull;
      const int ps = pos[lc];
      if (k > key || (k == key && ps < bp)) { key = k; bp = ps; bc = (int)rank + lc * (int)CL; }
    }
    qrc_argmax(key, bp, bc);
    if (lane == 0) { cand[par].key = key; cand[par].pos = bp; cand[par].col = bc; }
  };
  int lL = pick(nact, N);
  if (warp < QRC_WORK / 32) norms(0, false, lL);
  __syncthreads();
  if (warp == QRC_WORK / 32) post(0);

  int sign = 1;
  for (int j = 0; j < N; ++j) {
    __syncwarp();
    cluster_sync();  // candidates posted, columns updated
    // the winner, by every warp for itself
    unsigned long long key = 0;
    int pw = 0x7fffffff, w = -1;
    if (lane < (int)CL) {
      const QRCand q = qrc_peer(&cand[j & 1], lane);
      key = q.key; pw = q.pos; w = q.col;
    }
    qrc_argmax(key, pw, w);
    const unsigned owner = (unsigned)w % CL;
    const int lw = w / (int)CL;
    if (pw != j) sign = -sign;
    for (int i = j + tid; i < N; i += QRC_THREADS) xb[i] = qrc_peer(cols + (size_t)lw * ld + i, owner);
    if (warp == QRC_WORK / 32) {  // positions and the active list
      for (int t = lane; t < nact; t += 32) {
        const int lc = act[t];
        if (pos[lc] == j) pos[lc] = pw;
      }
      __syncwarp();
      if (rank == owner) {
        int at = -1;
        for (int t = lane; t < nact; t += 32)
          if (act[t] == lw) at = t;
        if (at >= 0) { act[at] = act[nact - 1]; fin[lw] = j; }
      }
      if (rank == 0 && lane == 0) p.jpvt[b * p.sP + j] = w + 1;
    }
    if (rank == owner) --nact;
    lL = pick(nact + 1, N - j - 1);
    __syncthreads();
    const int L = 1 << lL, lg = tid & (L - 1);
    if (warp < QRC_WORK / 32) {  // x^H a over the rows i > j
      const unsigned gm = (L == 32 ? 0xffffffffu : ((1u << L) - 1u) << (lane & ~(L - 1)));
      for (int t = tid >> lL; t <= nact; t += QRC_WORK >> lL) {
        const Z* a = t < nact ? cols + (size_t)act[t] * ld : xb;
        Z s0 = A::zero(), s1 = s0;
        int i = j + 1 + lg;
#pragma unroll 4
        for (; i + L < N; i += 2 * L) {
          s0 = A::mac(s0, A::conj(xb[i]), a[i]);
          s1 = A::mac(s1, A::conj(xb[i + L]), a[i + L]);
        }
        if (i < N) s0 = A::mac(s0, A::conj(xb[i]), a[i]);
        s0 = A::add(s0, s1);
        for (int o = 1; o < L; o <<= 1) s0 = A::add(s0, qrc_shfl_xor(s0, o, gm));
        if (lg == 0) dsh[t] = s0;
      }
    }
    __syncthreads();
    // ZLARFG and the per-column scalars, one thread per active column
    int need = 0;
    const Z alpha = xb[j];
    const double xn2 = A::re(dsh[nact]);
    const bool trivial = __double_as_longlong(xn2) == 0 && A::rzero_p(A::im(alpha));
    if (warp < QRC_WORK / 32 && (tid < nact || (tid == 0 && rank == owner)) && !trivial) {
      const double ar = A::re(alpha);
      const double t2 = A::abs2add(alpha, xn2);
      double s, ib, iy = 0.0, yy;
      if (alf_normal(t2)) {
        ib = alf_rsqrt_n(t2);
        s = t2 * ib;
        s = fma(fma(-s, s, t2), alf_half(ib), s);
      } else {
        s = sqrt(t2);
        ib = 1.0 / s;
      }
      const double beta = -copysign(s, ar);
      ib = -copysign(ib, ar);
      const Z tau = A::mkz(fma(-ar, ib, 1.0), -A::im(alpha) * ib);  // (beta - alpha) / beta
      const Z y = A::sub(alpha, A::mkz(beta, 0.0));
      yy = A::kReal ? A::re(y) : A::abs2(y);
      iy = alf_normal(yy) ? alf_rcp_n(yy) : 1.0 / yy;
      const Z scal = A::kReal ? A::mkz(iy, 0.0) : A::scale(A::conj(y), iy);
      for (int t = tid; t < nact; t += QRC_WORK) {
        const int lc = act[t];
        Z* a = cols + (size_t)lc * ld + j;
        const Z f = A::mac(A::scale(dsh[t], -ib), A::conj(tau), *a);
        const Z an = A::sub(*a, f);
        *a = an;
        gsh[t] = A::mul(scal, f);
        const double v1 = vn1[lc];
        if (__double_as_longlong(v1) != 0) {
          const double rest = A::abs2sub(v1, an);
          if (__double_as_longlong(rest) <= __double_as_longlong(tv2[lc])) { need = 1; vn1[lc] = -1.0; }
          else vn1[lc] = rest;
        }
      }
      if (tid == 0 && rank == owner) {
        scl[lw] = scal;
        bet[lw] = beta;
        p.tau[b * p.sT + j] = A::wide(tau);
        p.D[b * p.sD + j] = fabs(beta);
      }
    } else if (warp < QRC_WORK / 32 && trivial) {  // H = I: the norms alone change
      for (int t = tid; t < nact; t += QRC_WORK) {
        const int lc = act[t];
        const double v1 = vn1[lc];
        if (__double_as_longlong(v1) != 0) {
          const double rest = A::abs2sub(v1, cols[(size_t)lc * ld + j]);
          if (__double_as_longlong(rest) <= __double_as_longlong(tv2[lc])) { need = 1; vn1[lc] = -1.0; }
          else vn1[lc] = rest;
        }
      }
      if (tid == 0 && rank == owner) {
        scl[lw] = A::one();
        bet[lw] = A::re(alpha);
        p.tau[b * p.sT + j] = zmk(0.0, 0.0);
        p.D[b * p.sD + j] = fabs(A::re(alpha));
      }
    }
    const bool recompute = __syncthreads_or(need);
    if (warp < QRC_WORK / 32) {
      if (!trivial)
        for (int t = tid >> lL; t < nact; t += QRC_WORK >> lL) {
          Z* a = cols + (size_t)act[t] * ld;
          const Z ng = A::neg(gsh[t]);
#pragma unroll 4
          for (int i = j + 1 + lg; i < N; i += L) a[i] = A::mac(a[i], xb[i], ng);
        }
    } else if (!recompute) {
      post((j + 1) & 1);
    }
    if (recompute) {  // ZLAQP2's tol3z test: exact norms of the flagged columns
      __syncthreads();
      if (warp < QRC_WORK / 32) norms(j + 1, true, lL);
      __syncthreads();
      if (warp == QRC_WORK / 32) post((j + 1) & 1);
    }
  }
  __syncwarp();
  cluster_sync();  // no CTA leaves while its shared memory may still be read
  for (int lc = warp; lc < nmine; lc += QRC_THREADS / 32) {
    const int j = fin[lc];
    const Z sc = scl[lc];
    const Z* a = cols + (size_t)lc * ld;
    for (int i = lane; i < N; i += 32) {
      Z v = a[i];
      if (i == j) v = A::mkz(bet[lc], 0.0);
      else if (i > j) v = A::mul(sc, v);
      Ob[i + j * p.lda] = A::wide(v);
    }
  }
  if (rank == 0 && tid == 0) p.info[b].psign = sign;
}
