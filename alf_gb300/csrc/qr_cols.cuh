// Exact ZGEQP3 (ZLAQP2: dynamic column pivoting with norm downdates,
// Prog/QDRP_decompose_mod.F90:60-101) on one thread-block cluster per matrix, columns dealt
// cyclically to the CTAs (column c -> CTA c % CL) and kept in shared memory.
#pragma once
#include "common.cuh"
#include "arith.cuh"
#include "linalg.cuh"

#define QRC_WORK 256                 // threads that carry FP64 work: two warps per sub-partition
#define QRC_THREADS (QRC_WORK + 32)  // and one warp for a step's scalars (FP64) and its exchange
#ifndef QRC_WAIT_CYCLES
#define QRC_WAIT_CYCLES (1ll << 31)  // a wait's limit in SM cycles: one second
#endif

struct QRColsParams {
  const zd* Ain;             // input (may equal A)
  zd* A; long long lda, sA;  // output: R above the diagonal, reflectors below
  int N;
  const double* colscale; long long sCS;
  zd* tau; long long sT;
  int* jpvt; long long sP;
  double* D; long long sD;
  QRInfo* info;
  int* err;                  // may be null: bit 4 is set if a peer's data does not come
};

struct __align__(16) QRCand {  // a CTA's best remaining column
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
  return (nc + 2) * qrc_ld(N, zb) * zb + 3 * nc * zb + (3 * nc) * 8 + (4 * nc) * sizeof(int) + 64;
}

ALF_DEV uint32_t qrc_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// Wait for a phase of an mbarrier of this CTA; gives up after QRC_WAIT_CYCLES.
ALF_DEV bool qrc_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
ALF_DEV bool qrc_wait(uint32_t bar, uint32_t parity) {
  if (qrc_try(bar, parity)) return true;
  const long long t0 = clock64();
  while (!qrc_try(bar, parity))
    if (clock64() - t0 > QRC_WAIT_CYCLES) return false;
  return true;
}
ALF_DEV void qrc_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// 16 bytes into a peer's shared memory, counted on the peer's mbarrier.
ALF_DEV void qrc_push16(uint32_t dst, uint32_t bar, const QRCand& q) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
               "r"((unsigned)q.key), "r"((unsigned)(q.key >> 32)), "r"((unsigned)q.pos), "r"((unsigned)q.col), "r"(bar)
               : "memory");
}
// A run of shared memory (16-byte aligned, a multiple of 16 bytes) into a peer's, the same way.
ALF_DEV void qrc_push(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(src),
      "r"(bytes), "r"(bar)
      : "memory");
}
ALF_DEV void qrc_fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
ALF_DEV void qrc_bar_work() { asm volatile("bar.sync 1, %0;" ::"n"(QRC_WORK) : "memory"); }
ALF_DEV void qrc_bar_arrive() { asm volatile("bar.arrive 2, %0;" ::"n"(QRC_THREADS) : "memory"); }
ALF_DEV void qrc_bar_join() { asm volatile("bar.sync 2, %0;" ::"n"(QRC_THREADS) : "memory"); }

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

// Sums and updates over the entries i, i + L, .. < N, the next ones loaded while the FP64 pipe holds
// the current: one warp on a sub-partition has nobody else to hide its loads.
template <class A>
ALF_DEV typename A::Z qrc_dot(const typename A::Z* x, const typename A::Z* a, int i, int L, int N) {  // x^H a
  typedef typename A::Z Z;
  Z s = A::zero();
  if (i >= N) return s;
  Z u = x[i], v = a[i];
  while (true) {
    i += L;
    const Z cu = u, cv = v;
    if (i < N) { u = x[i]; v = a[i]; }
    s = A::mac(s, A::conj(cu), cv);
    if (i >= N) return s;
  }
}
template <class A>
ALF_DEV double qrc_norm2(const typename A::Z* a, int i, int L, int N) {
  double s = 0.0;
  if (i >= N) return s;
  typename A::Z v = a[i];
  while (true) {
    i += L;
    const typename A::Z cv = v;
    if (i < N) v = a[i];
    s = A::abs2add(cv, s);
    if (i >= N) return s;
  }
}
template <class A>
ALF_DEV void qrc_axpy(typename A::Z* a, const typename A::Z* x, typename A::Z g, int i, int L, int N) {  // a += x g
  typedef typename A::Z Z;
  if (i >= N) return;
  Z u = x[i], v = a[i];
  while (true) {
    const int c = i;
    i += L;
    const Z cu = u, cv = v;
    if (i < N) { u = x[i]; v = a[i]; }
    a[c] = A::mac(cv, cu, g);
    if (i >= N) return;
  }
}

// The FP64 pipe takes one warp instruction per sub-partition every ~64 cycles, with nothing in
// flight beside it, so a step's cost is the FP64 instructions on its longest sub-partition plus
// the cluster exchange.  Columns in a CTA make every dot product and norm local: per step the
// CTAs exchange one candidate column each (16 bytes) and the chosen one (N - j values).  Columns are
// never moved: a column keeps its slot and its position in the pivoted order is tracked beside it, a
// finished one leaves the list of active columns.  The update uses the unscaled column x:
// f = conj(tau) a_j - (x^H a) / beta (tau and scal = 1 / (alpha - beta) give conj(tau scal) =
// -1 / beta), a_j -= f, a_i -= x_i (scal f).  Norms are kept squared and compared as integers.
//
// Eight warps carry the columns.  A ninth runs what is serial beside them: ZLARFG's scalars while
// they form the dot products, and the exchange while they update.  The norms a step leaves behind are
// known before its update is applied, so each CTA pushes its best column's norm to its peers then
// and updates that column first; the ninth warp collects the candidates, and the winner's CTA pushes
// the column into every peer's shared memory while the rest of the update goes on.  No cluster barrier:
// an mbarrier per message, two of each in turn (a CTA posts step j + 1 only when it has read the
// candidates and the column of step j - 1, so two are enough).
// Arithmetic A: ArD or ArRe.  Grid (CL, B), QRC_THREADS threads.
// Measured (GB300, one QR): two 256 x 256 matrices 3.41 ms with rows in the CTAs (k_qrp_rows), 1.17 ms
// with columns, a cluster barrier and everything in sequence, 0.82 ms this (complex 2.23 -> 1.67); 32 of
// them 5.70, 1.64, 1.40 (real); two 576 x 576 21.9, 4.9, 3.7.  A step at N = 256 (16 CTAs), cycles: dot
// products and scalars beside them 2700, per-column scalars 1000, update and exchange 2400, barriers 300.
template <class A>
__global__ void __launch_bounds__(QRC_THREADS) k_qrp_cols(QRColsParams p) {
  typedef typename A::Z Z;
  constexpr int ZB = (int)sizeof(Z), ZA = 16 / ZB;  // ZA elements per 16 bytes
  const unsigned rank = cluster_ctarank(), CL = cluster_nctarank();
  const int b = blockIdx.y, N = p.N, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nc = (N + (int)CL - 1) / (int)CL;                 // slots per CTA
  const int nmine = (N - (int)rank + (int)CL - 1) / (int)CL;  // columns rank, rank + CL, ...
  const int ld = qrc_ld(N, ZB);
  extern __shared__ __align__(16) unsigned char qrc_raw[];
  Z* cols = reinterpret_cast<Z*>(qrc_raw);  // [nc][ld]
  Z* xb = cols + (size_t)nc * ld;           // [2][ld] the chosen column of step j in xb[j & 1]
  Z* dsh = xb + 2 * ld;                     // [nc] x^H a of the active columns
  Z* gsh = dsh + nc;                        // [nc] scal f
  Z* scl = gsh + nc;                        // [nc] scal of finished columns
  double* vn1 = reinterpret_cast<double*>(scl + nc);  // [nc] squared norms, -1: to be recomputed
  double* tv2 = vn1 + nc;                             // [nc] tol3z times the last exact squared norm
  double* bet = tv2 + nc;                             // [nc] beta of finished columns
  int* pos = reinterpret_cast<int*>(bet + nc);        // [nc] position in the pivoted order
  int* actb = pos + nc;                               // [2][nc] active slots at step j in actb[j & 1]
  int* fin = actb + 2 * nc;                           // [nc] step at which a column was chosen
  __shared__ QRCand cand[2][16];                      // the CTAs' candidates, pushed by them
  __shared__ QRCand wc[QRC_WORK / 32];                // the warps' candidates: col is the index in the active list
  __shared__ __align__(8) unsigned long long mb[4];   // cand[0], cand[1], xb[0], xb[1] complete
  // step j: own slot chosen or -1, active columns, lanes; dead: 1 + the step whose exchange gave up, gone:
  // some CTA of the cluster has given up
  __shared__ struct { int lw, nact, lanes, dead, gone; } st;
  __shared__ struct { Z tau, scal; double ib; int trivial; } rf;  // the reflector of step j
  const double tol3z = 1.0536712127723509e-08;  // sqrt(dlamch('Epsilon'))
  const zd* Ab = p.Ain + b * p.sA;
  zd* Ob = p.A + b * p.sA;
  const bool work = warp < QRC_WORK / 32;
  const int lgC = 31 - __clz((int)CL);  // CL is a power of two
  // work threads in the order of the dot products' columns: warps 1 2 3 5 6 7 0 4
  const int tidw = (warp % 4 == 0 ? 6 + warp / 4 : warp / 4 * 3 + warp % 4 - 1) * 32 + lane;

  if (tid == 0) {
    for (int i = 0; i < 4; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(qrc_smem(mb + i)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    st.dead = st.gone = 0;
  }
  for (int lc = warp; lc < nmine; lc += QRC_THREADS / 32) {
    const int c = (int)rank + lc * (int)CL;
    const double s = p.colscale ? p.colscale[b * p.sCS + c] : 1.0;
    for (int i = lane; i < N; i += 32) {
      zd v = Ab[i + c * p.lda];
      if (p.colscale) v = zscale(v, s);
      cols[(size_t)lc * ld + i] = A::mk(v);
    }
    if (lane == 0) { pos[lc] = c; actb[lc] = lc; fin[lc] = c; }
  }
  __syncwarp();
  cluster_sync();  // every CTA's mbarriers are ready

  // The lane count L = 1 << l per column with the fewest FP64 instructions on a sub-partition: ne
  // columns fill ne L / 32 warps, each with rows / L products and, for a sum, l additions.  The ninth
  // warp keeps sub-partition 0 busy beside them (`own` instructions), so its two work warps come last.
  auto pick = [&](int ne, int rows, int adds, int own) {  // one warp
    const int l = 1 + lane % 5;
    const int W = ((ne << l) + 31) >> 5, full = W >> 3, rem = W & 7;
    const int r = (A::kReal ? 1 : 4) * ((rows + (1 << l) - 1) >> l) + adds * l;
    const int cost = max((2 * full + (rem > 3 ? 2 : (rem > 0 ? 1 : 0))) * r, (2 * full + (rem == 7 ? 1 : 0)) * r + own);
    return (int)(__reduce_min_sync(0xffffffffu, (unsigned)min(cost, 0xfffffff) * 8u + (unsigned)l) & 7u);
  };
  // lane counts of step j with ne active columns, dot products | updates << 4
  auto lanes_of = [&](int ne, int j) {
    constexpr int c = A::kReal ? 1 : 2;
    return pick(ne, N - j - 1, c, (A::kReal ? 17 : 21) + c * ((N - j + 30) >> 5)) | pick(ne, N - j - 1, 0, 0) << 4;
  };
  // squared norms over the rows i >= i0 of the active columns (flagged ones only)
  auto norms = [&](const int* act, int nact, int i0, bool flagged, int lL) {
    const int L = 1 << lL, lg = tid & (L - 1);
    for (int t = tid >> lL; t < nact; t += QRC_WORK >> lL) {
      const int lc = act[t];
      if (flagged && !(vn1[lc] < 0.0)) continue;
      const Z* a = cols + (size_t)lc * ld;
      double s = qrc_norm2<A>(a, i0 + lg, L, N);
      const unsigned gm = (L == 32 ? 0xffffffffu : ((1u << L) - 1u) << (lane & ~(L - 1)));
      for (int o = 1; o < L; o <<= 1) s += __shfl_xor_sync(gm, s, o);
      __syncwarp(gm);  // every lane of the group has read the flag
      if (lg == 0) { vn1[lc] = s; tv2[lc] = tol3z * s; }
    }
  };
  // the warp's best active column (thread t: entry t; warps with entries, and the first)
  auto candidate = [&](const int* act, int nact) {
    unsigned long long key = 0;
    int bp = 0x7fffffff, bt = -1;
    if (tid < nact) {
      const int lc = act[tid];
      const unsigned long long v = (unsigned long long)__double_as_longlong(vn1[lc]) & 0x7fffffffffffffffull;
      key = v > 0x7ff0000000000000ull ? 0ull : v + 1ull;
      bp = pos[lc];
      bt = tid;
    }
    qrc_argmax(key, bp, bt);
    QRCand q;
    q.key = key; q.pos = bp; q.col = bt;
    if (lane == 0) wc[warp] = q;
    return q;
  };
  auto post = [&](QRCand q, const int* act, int par) {  // to the peers, by one warp
    if (q.col >= 0) q.col = (int)rank + (act[q.col] << lgC);
    if (lane < (int)CL && lane != (int)rank) qrc_push16(dsmem_addr(&cand[par][rank], lane), dsmem_addr(mb + par, lane), q);
  };
  auto best = [&](int nact) {  // the CTA's, known to every thread; col: index in the active list or -1
    QRCand q;
    q.key = 0; q.pos = 0x7fffffff; q.col = -1;
    for (int k = 0; 32 * k < nact; ++k) {
      const QRCand o = wc[k];
      if (o.key > q.key || (o.key == q.key && o.pos < q.pos)) q = o;
    }
    return q;
  };
  int sign = 1;
  // The ninth warp: the exchange that opens step j, with the CTA's candidate q (posted already or not);
  // join: its column is being updated.
  auto exchange = [&](QRCand q, int j, int nact, int ln0, int ln1, bool posted, bool join) {
    const int par = j & 1;
    const uint32_t cbar = qrc_smem(mb + par), xbar = qrc_smem(mb + 2 + par);
    int* an = actb + par * nc;
    const int* act = j == 0 ? an : actb + (par ^ 1) * nc;  // of step j - 1
    if (!posted) post(q, act, par);
    if (lane == 0) qrc_expect(cbar, 16u * (CL - 1));
    const int last = nact > 0 ? act[nact - 1] : 0;
    if (join) qrc_bar_join();
    qrc_fence_async();  // the column as the work warps left it, for the copy engine
    if (q.col >= 0) q.col = (int)rank + (act[q.col] << lgC);
    const int i0 = j & ~(ZA - 1);
    const uint32_t bytes = (uint32_t)((N - i0 + ZA - 1) & ~(ZA - 1)) * ZB;
    bool armed = false, ok = __all_sync(0xffffffffu, qrc_wait(cbar, (unsigned)(j >> 1) & 1u));
    if (ok) {
      unsigned long long key = 0;
      int pw = 0x7fffffff, w = -1;
      if (lane < (int)CL) {
        if (lane != (int)rank) q = cand[par][lane];
        key = q.key; pw = q.pos; w = q.col;
      }
      qrc_argmax(key, pw, w);
      const bool own = (w & ((int)CL - 1)) == (int)rank;
      const int lw = w >> lgC;
      armed = true;
      if (own) {
        const uint32_t src = qrc_smem(cols + (size_t)lw * ld + i0);
        if (lane < (int)CL && lane != (int)rank)
          qrc_push(dsmem_addr(xb + par * ld + i0, lane), src, bytes, dsmem_addr(mb + 2 + par, lane));
        if (lane == 0) qrc_expect(xbar, 0);
      } else if (lane == 0) {
        qrc_expect(xbar, bytes);
      }
      for (int t = lane; t < nact; t += 32) {  // positions and the active list
        const int lc = act[t];
        if (pos[lc] == j) pos[lc] = pw;
        if (j > 0 || (own && lc == lw)) an[t] = own && lc == lw ? last : lc;  // past the new end: never read
      }
      if (pw != j) sign = -sign;
      if (lane == 0) {
        if (own) fin[lw] = j;
        st.lw = own ? lw : -1;
        st.nact = nact - (own ? 1 : 0); st.lanes = own ? ln1 : ln0;
        if (rank == 0) p.jpvt[b * p.sP + j] = w + 1;
      }
      ok = __all_sync(0xffffffffu, qrc_wait(xbar, (unsigned)(j >> 1) & 1u));
    }
    if (!ok) {
      if (lane < (int)CL) asm volatile("st.shared::cluster.u32 [%0], 1;" ::"r"(dsmem_addr(&st.gone, lane)) : "memory");
      if (lane == 0) {
        st.dead = j + 1;
        if (!armed) qrc_expect(xbar, bytes);  // what may still come: this step's messages, the next candidates
        qrc_expect(qrc_smem(mb + (par ^ 1)), 16u * (CL - 1));
        if (p.err) atomicOr(p.err, 4);
      }
    }
  };

  if (work) {
    const int l0 = 31 - __clz(max(2, min(32, QRC_WORK / max(1, nmine))));
    norms(actb, nmine, 0, false, l0);
    qrc_bar_work();
    if (warp * 32 < nmine || warp == 0) candidate(actb, nmine);
  }
  __syncthreads();
  if (!work) exchange(best(nmine), 0, nmine, lanes_of(nmine, 0), lanes_of(nmine - 1, 0), false, false);

  for (int j = 0; j < N; ++j) {
    __syncthreads();
    if (st.dead) break;
    const int lw = st.lw, nact = st.nact, lL = st.lanes & 15, lU = st.lanes >> 4;
    const int* act = actb + (j & 1) * nc;
    const Z* x = lw >= 0 ? cols + (size_t)lw * ld : xb + (j & 1) * ld;
    if (work) {  // x^H a over the rows i > j
      const int L = 1 << lL, lg = tid & (L - 1);
      const unsigned gm = (L == 32 ? 0xffffffffu : ((1u << L) - 1u) << (lane & ~(L - 1)));
      for (int t = tidw >> lL; t < nact; t += QRC_WORK >> lL) {
        const Z* a = cols + (size_t)act[t] * ld;
        Z s0 = qrc_dot<A>(x, a, j + 1 + lg, L, N);
        for (int o = 1; o < L; o <<= 1) s0 = A::add(s0, qrc_shfl_xor(s0, o, gm));
        if (lg == 0) dsh[t] = s0;
      }
    }
    double t2 = 0.0, ib = 0.0;
    bool plain = false;  // H = I
    Z alpha = A::zero();
    if (!work) {  // ZLARFG: with s = |beta|, 1 / beta = ib, tau = 1 - alpha ib, scal = 1 / (alpha - beta) = -ib / tau
      const double xn2 = warp_sum(qrc_norm2<A>(x, j + 1 + lane, 32, N));
      alpha = x[j];
      plain = __double_as_longlong(xn2) == 0 && A::rzero_p(A::im(alpha));
      Z tau = A::zero(), scal = A::one();
      if (!plain) {
        const double ar = A::re(alpha);
        t2 = A::abs2add(alpha, xn2);
        if (alf_normal(t2)) {
          ib = -copysign(rsqrt(t2), ar);
          tau = A::mkz(fma(-ar, ib, 1.0), -A::im(alpha) * ib);  // 1 <= |tau|^2 <= 4
          if constexpr (A::kReal) scal = -ib * alf_rcp_n(tau);
          else scal = A::scale(A::conj(tau), -ib * alf_rcp_n(A::abs2(tau)));
        } else {
          const double s = sqrt(t2);
          ib = -copysign(1.0 / s, ar);
          tau = A::mkz(fma(-ar, ib, 1.0), -A::im(alpha) * ib);
          const Z y = A::sub(alpha, A::mkz(-copysign(s, ar), 0.0));
          const double iy = 1.0 / (A::kReal ? A::re(y) : A::abs2(y));
          scal = A::kReal ? A::mkz(iy, 0.0) : A::scale(A::conj(y), iy);
        }
      }
      if (lane == 0) {
        rf.tau = tau; rf.scal = scal; rf.ib = ib; rf.trivial = plain;
        if (lw >= 0) {
          scl[lw] = scal;
          p.tau[b * p.sT + j] = A::wide(tau);
        }
      }
    }
    if (j + 1 < N) __syncthreads();
    int ln0 = 0, ln1 = 0;  // of the next step, without and with this CTA's column chosen
    if (!work && j + 1 < N) { ln0 = lanes_of(nact, j + 1); ln1 = lanes_of(nact - 1, j + 1); }
    if (!work && lw >= 0) {  // beta, needed at the end only
      double beta = A::re(alpha);
      if (!plain) {
        const double s = alf_normal(t2) ? alf_sqrt_n(t2, fabs(ib)) : sqrt(t2);
        beta = -copysign(s, beta);
      }
      if (lane == 0) {
        bet[lw] = beta;
        p.D[b * p.sD + j] = fabs(beta);
      }
    }
    if (j + 1 == N) break;
    // the per-column scalars, one thread per active column, and the norms the update leaves
    const bool trivial = rf.trivial;
    int need = 0;
    if (work && (warp * 32 < nact || warp == 0)) {
      Z f = A::zero();
      if (tid < nact) {
        const int lc = act[tid];
        Z* a = cols + (size_t)lc * ld + j;
        Z an = *a;
        if (!trivial) {  // H = I otherwise: the norms alone change
          f = A::mac(A::scale(dsh[tid], -rf.ib), A::conj(rf.tau), an);
          an = A::sub(an, f);
          *a = an;
        }
        const double v1 = vn1[lc];
        if (__double_as_longlong(v1) != 0) {
          const double rest = A::abs2sub(v1, an);
          if (__double_as_longlong(rest) <= __double_as_longlong(tv2[lc])) { need = 1; vn1[lc] = -1.0; }
          else vn1[lc] = rest;
        }
      }
      const QRCand q = candidate(act, nact);
      if (nact <= 32 && !__any_sync(0xffffffffu, need)) post(q, act, (j + 1) & 1);  // one warp has them all
      if (tid < nact && !trivial) gsh[tid] = A::mul(rf.scal, f);
    }
    const bool recompute = __syncthreads_or(need);
    auto update = [&](int skip) {
      const int L = 1 << lU, lg = lane & (L - 1);
      if (!trivial)
        for (int t = tidw >> lU; t < nact; t += QRC_WORK >> lU)
          if (t != skip) qrc_axpy<A>(cols + (size_t)act[t] * ld, x, A::neg(gsh[t]), j + 1 + lg, L, N);
    };
    if (recompute) {  // ZLAQP2's tol3z test: exact norms of the flagged columns first
      if (work) {
        update(-1);
        qrc_bar_work();
        norms(act, nact, j + 1, true, lL);
        qrc_bar_work();
        if (warp * 32 < nact || warp == 0) candidate(act, nact);
      }
      __syncthreads();
    }
    const QRCand q = best(nact);
    if (!work) {
      exchange(q, j + 1, nact, ln0, ln1, !recompute && nact <= 32, !recompute);
    } else if (!recompute) {
      if (!trivial && q.col >= 0) {
        Z* a = cols + (size_t)act[q.col] * ld;
        const Z ng = A::neg(gsh[q.col]);
        for (int i = j + 1 + tid; i < N; i += QRC_WORK) a[i] = A::mac(a[i], x[i], ng);
      }
      qrc_bar_arrive();
      update(q.col);
    }
  }
  __syncwarp();
  cluster_sync();  // no CTA leaves while a peer may still write to it
  if (st.gone) {
    // Nothing is sent any more.  A CTA that gave up waits until what its peers had sent has landed in its
    // shared memory (a message that was never sent costs the limit), and none leaves before.  No column is
    // written, but the pivots stay indices: the kernels that run before the host reads the error use them.
    if (rank == 0 && st.dead)
      for (int i = tid; i < N; i += QRC_THREADS) p.jpvt[b * p.sP + i] = i + 1;
    if (rank == 0 && tid == QRC_WORK) p.info[b].psign = sign;
    if (st.dead && tid < 3) {
      const int s = st.dead - 1 + (tid == 1);
      qrc_wait(qrc_smem(mb + (tid == 2 ? 2 : 0) + (s & 1)), (unsigned)(s >> 1) & 1u);
    }
    __syncwarp();
    cluster_sync();
    return;
  }
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
  if (rank == 0 && tid == QRC_WORK) p.info[b].psign = sign;
}
