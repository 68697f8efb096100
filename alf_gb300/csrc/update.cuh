// Sequential single-vertex Metropolis updates with a delayed (submatrix) update.
//
// Reference: Upgrade2 (Prog/upgrade_mod.F90:105-302) called from WRAPGRUP /
// WRAPGRDO (Prog/Wrapgr_mod.F90:115-147, 198-236), for diagonal single-site
// vertices (Op%N = 1): the Mz and SU(N) Hubbard operators.
//
// Within one time slice the vertex exponentials are diagonal similarity
// transforms: G_ii is unchanged by them and the Sherman-Morrison update
// G <- G - x_i G(:,i) (e_i - G(i,:)), x_i = Delta_i / (1 + Delta_i (1 - G_ii)),
// has the same form in the frame of the slice-start matrix G0, so the scalings
// are applied once at the end of the slice by the hopping GEMMs.
//
// A block of nq consecutive visits touches only the sites Sblk of its
// vertices.  The kernel keeps Ghat = G(Sblk, Sblk) in shared memory and applies
// every accepted Sherman-Morrison update to Ghat only; each visit's ratio is
// then Upgrade2's Mat(1,1) = 1 + Delta (1 - Ghat_jj) read directly.  The effect
// on the full matrix is the sum of the same updates over the accepted sites S,
//   G = G0 - G0(:,S) Y,
// applied by one rank-m GEMM flush; the kernel leaves the coefficients from which
// k_flush_xy forms Y by two triangular substitutions (below), without an inverse.
//
// G is complex128 in both precision forms.  The per-flavour determinants
// Mat(1,1) (or the 2x2 determinant of a two-site vertex), the Ghat rank-1 updates
// and the coefficients run in FP64 (plain form) or double-float (mixed form,
// dfloat.cuh, ~2^-46 relative rounding), real ones on models that are real.  The accumulation of the Metropolis ratio (the
// product over flavours, exp(Z1 alpha), the N_SUN power and the gamma ratio), the
// weight test and the phase are FP64 in both forms.  GB300's FP64 dependent
// latency (63-76 cycles, ~560 for a division) sets the cost of every visit, so
// the chain avoids divisions and square roots: the Metropolis test is
// division-free, the reciprocal is one step of an iteration (arith.cuh), and the phase stays
// unnormalised until the block ends.
#pragma once
#include "common.cuh"
#include "arith.cuh"

#define UPD_KMAX 32
#define UPD_THREADS 256

struct VertexDev {
  // per chain: K = F*M entries, index k = nf*M + n
  const int* site;       // site of eigen-index 0 (P(1), 0-based)
  const int* site2;      // site of eigen-index 1, or -1
  const int8_t* nsite;   // positions of the vertex: its non-zero eigenvalues (1 or 2)
  const int8_t* type;    // 1 or 2
  long long sK;          // per-chain stride in entries (F*M)
};
struct UpdTab;

struct UpdParams {
  int N, F, M, L, NSUN;
  int nt1;        // slice, 1-based
  int dir;        // 0: up pass (n = pos), 1: down pass (n = M-1-pos)
  int q0, nq;     // visit positions q0 .. q0+nq-1 of this slice
  int visit_base; // visit index (within the sweep) of position 0 of this slice
  int nChains;
  const void* G; long long sG;  // [chain][F][N][N] complex128
  VertexDev V;
  const UpdTab* tab;    // [chain][F*M][5][3]
  int8_t* fields;       // [chain][L][M]
  const double* draws; long long sDraws;  // [chain][6*M*L] or null
  const unsigned long long* rngkey;      // [chain]
  const unsigned long long* rngctr;      // [chain] counter of draw 0 of this sweep
  zd* phase;            // [chain]
  int* m_out;           // [chain], then [chain][F] (per-GEMM-batch rank)
  zd* W;                // [chain][2][UPD_KMAX][UPD_KMAX]  C, x and P of the accepted positions
  int* sites_out;       // [chain][UPD_KMAX]  accepted sites, accept order
  long long* cnt;       // [chain][4] n_prop, n_acc, n_prop_eff, n_acc_eff
  int8_t* rec_acc; zd* rec_ratio; long long sRec;
  FieldTables ft;
  // vector vertices (a single-site vertex on a site of a rotated pair: in the rotated basis its
  // one position is the real unit vector u = c_a e_a + c_b e_b); null when the model has none
  const int* vsite2;    // [chain][F*M] site b of a vector vertex, -1 otherwise
  const double* vcoef;  // [chain][F*M][2] (c_a, c_b)
  int* sites2_out;      // [chain][UPD_KMAX] accepted positions: site b or -1
  double* coef_out;     // [chain][UPD_KMAX][2]
  // optional: the block submatrix Ghat = G(P, P) over this block's positions P, staged by
  // k_sub_stage while the previous block's flush still runs ([chain][F][KMAX][KMAX], row a =
  // position a); null: read from G
  const zd* Gsub;
};

// Positions of the block of visits q0 .. q0 + nq - 1 (slice order dir) of chain c: the site of
// every non-zero eigenvalue, in the order k_update numbers them (exclusive prefix sum of the
// vertex sizes over the visits).  Warp-level: every lane of the calling warp takes part;
// returns the position count, writes pos[0 .. np).
ALF_DEV int block_positions(const VertexDev& V, int c, int M, int dir, int q0, int nq, int* pos) {
  const int lane = threadIdx.x & 31;
  const int* site = V.site + (long long)c * V.sK;
  const int* site2 = V.site2 + (long long)c * V.sK;
  const int8_t* nsite = V.nsite + (long long)c * V.sK;
  int w = 0, n = 0;
  if (lane < nq) {
    n = dir == 0 ? q0 + lane : M - 1 - (q0 + lane);
    w = nsite[n];
  }
  int incl = w;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  const int p0 = incl - w;
  for (int I = 0; I < w; ++I) pos[p0 + I] = I ? site2[n] : site[n];
  return __shfl_sync(0xffffffffu, incl, 31);
}

// Snapshot of G over the positions of the next block, taken beside the current block's visits, before its flush
// writes G: Gsnap[chain][f][a][l] = G(P_a, P_l).  Also stores the positions (pos[chain][KMAX],
// npos[chain]).  grid (chains * F), 256 threads.
__global__ void k_sub_gather(const zd* G, long long sG, int N, int F, int M, VertexDev V, int dir, int q0, int nq,
                             zd* Gsnap, int* pos, int* npos) {
  const int b = blockIdx.x, c = b / F, f = b % F, tid = threadIdx.x;
  __shared__ int sp[UPD_KMAX];
  __shared__ int snp;
  if (tid < 32) {
    const int np = block_positions(V, c, M, dir, q0, nq, sp);
    if (tid == 0) snp = np;
  }
  __syncthreads();
  const int np = snp;
  if (f == 0) {
    for (int a = tid; a < np; a += 256) pos[(long long)c * UPD_KMAX + a] = sp[a];
    if (tid == 0) npos[c] = np;
  }
  const zd* Gf = G + (long long)c * sG + (long long)f * N * N;
  zd* out = Gsnap + (long long)b * UPD_KMAX * UPD_KMAX;
  for (int e = tid; e < np * np; e += 256) {
    const int a = e / np, l = e % np;
    out[a * UPD_KMAX + l] = Gf[sp[a] + (long long)sp[l] * N];
  }
}

// The next block's submatrix after the current block's accepted updates, from the snapshot
// and the flush operands: Gsub(a, l) = Gsnap(a, l) - sum_k X(P_a, k) Y(k, P_l), k < m (the same
// Woodbury form the flush applies to all of G).
// grid (ceil(KMAX / 8), chains * F), block (32, 8): (l, a).
template <class A>
__global__ void k_sub_stage(const zd* Gsnap, const int* pos, const int* npos, const int* m_in, int N, int F,
                            const zd* X, const zd* Y, zd* Gsub) {
  typedef typename A::Z Z;
  const int b = blockIdx.y, c = b / F, f = b % F;
  const int l = threadIdx.x, a = blockIdx.x * 8 + threadIdx.y;
  const int np = npos[c], m = m_in[c];
  if (a >= np || l >= np) return;
  const long long o = (long long)b * UPD_KMAX * UPD_KMAX + a * UPD_KMAX + l;
  const int pa = pos[(long long)c * UPD_KMAX + a], pl = pos[(long long)c * UPD_KMAX + l];
  const long long xy = ((long long)c * 2 + f) * N * UPD_KMAX;
  Z acc = A::zero();
  for (int k = 0; k < m; ++k) acc = A::mac(acc, A::mk(X[xy + pa + (long long)k * N]), A::mk(Y[xy + k + (long long)pl * UPD_KMAX]));
  Gsub[o] = A::wide(A::sub(A::mk(Gsnap[o]), acc));
}

ALF_DEV int nranf3(double r) {
  // nint(r*3 + 0.5) clamped to [1,3] (random_wrap_mod.F90:159-168); no contraction.
  double y = __dadd_rn(__dmul_rn(r, 3.0), 0.5);
  int v = (int)round(y);
  return v < 1 ? 1 : (v > 3 ? 3 : v);
}

// Per-visit transition data, precomputed per (vertex k, old field s, flip choice):
//   myexp_I = exp(Z E_I), dlt_I = myexp_I - 1, expal = exp(Z alpha),  Z = g (phi(s_new) - phi(s_old))
// for the eigen-indices I = 0, 1 (Upgrade2's Mat(I,I) = myexp_I - dlt_I G(P_I,P_I),
// upgrade_mod.F90:140-190).
struct UpdTab {
  zd myexp[2], dlt[2], expal;
};

// One CTA of UPD_THREADS threads per chain.  Dynamic shared memory:
//   Gh[F][KMAX][KMAX+1]  the block Ghat over the block's positions, updated in place
//   Tc[F][KMAX][KMAX]    x_q Ghat(:, q) of every position q at its step (0 on the rows up to q)
// A position is one non-zero eigenvalue of a vertex (its site in the diagonal basis);
// single-site vertices have one, two-site vertices two consecutive positions whose
// joint ratio is Upgrade2's 2x2 determinant, computed as D_a (1 + Delta_b (1 - G'_bb))
// with G' after the tentative Sherman-Morrison update of position a; an accepted
// two-site vertex is applied as two rank-1 updates, the second decided with the first.
//
// One block barrier per position v.  Between two barriers, with the previous position's decision
// and Tc column known, four parts run on different sub-partitions (an FP64 instruction holds its
// sub-partition ~64 cycles, so the chain per position is counted in them):
//   warp 0       the ratio and its test, from the diagonal element (scalars only)
//   warp 1 + f   flavour f's column v, 1 / D and Tc(v), whether or not v is accepted
//   the others   the previous position's rank-1 update of the columns beyond v
// Column v is not written back: nothing reads it after its own step (the column that follows the
// first position of a pair is left out of that step's update and takes two at its own step).
// The flush needs no inverse of Gamma: the accepted updates are G0 - sum_l x_l u_l w_l^T with
//   w_l = b_l + sum_{k<l} C_lk w_k,  C_lk = x_k u_k(s_l),      b_l = e_{s_l} - G0(s_l, :)
//   u_l = G0(:, s_l) + sum_{k<l} u_k P_kl,  P_kl = x_k G^{(k-1)}(s_k, s_l),
// so G0 - X Y with X = G0(:, S), Y = (1 - P)^-1 diag(x) (1 - C)^-1 b: two triangular
// substitutions per column in k_flush_xy.  C, P and x are entries of Tc and Ghat.
// Measured, 32 positions, two flavours: FP64 complex 105 us, double-float 79 us (one warp for the
// chain, Gauss-Jordan at the end) -> 28 us real, 65 us complex, 59 us double-float (with about 8 us of
// timing events).
template <class A>
__global__ void __launch_bounds__(UPD_THREADS) k_update(UpdParams p) {
  typedef typename A::Z Z;
  constexpr int KM = UPD_KMAX, LD = UPD_KMAX + 1, NW = UPD_THREADS / 32;
  constexpr bool FOLD = A::kReal && !A::kDoubleFloat;  // K joins a position's factors (FP64)
  const int c = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = p.N, F = p.F, M = p.M, nq = p.nq;
  extern __shared__ __align__(16) unsigned char upd_raw[];
  Z* Gh = reinterpret_cast<Z*>(upd_raw);  // [F][KM][LD]
  Z* Tc = Gh + 2 * KM * LD;               // [F][KM][KM]
  // per position
  __shared__ Z s_mye[2][KM], s_dlt[2][KM], s_rD[2][KM];
  __shared__ Z s_myk[2][FOLD ? KM : 1], s_dlk[2][FOLD ? KM : 1];  // real FP64: K folded in
  __shared__ int s_psite[KM], s_pvis[KM], s_pkind[KM], s_acc[KM], s_accq[NW][KM];
  __shared__ int s_psite2[KM];      // vector positions: site b, else -1
  __shared__ double s_pc[KM][2];    // vector positions: (c_a, c_b)
  // per visit (FP64 in both forms: the ratio accumulation)
  __shared__ zd s_K[KM];
  __shared__ double s_u2[KM], s_gr[KM];
  __shared__ int s_vtx[KM], s_snew[KM], s_prop[KM];

  const double2* G = reinterpret_cast<const double2*>(p.G) + (long long)c * p.sG;
  const int* site = p.V.site + (long long)c * p.V.sK;
  const int* site2 = p.V.site2 + (long long)c * p.V.sK;
  const int8_t* nsite = p.V.nsite + (long long)c * p.V.sK;
  const int8_t* ty = p.V.type + (long long)c * p.V.sK;
  const UpdTab* tab = p.tab + (long long)c * p.V.sK * 15;
  int8_t* fl = p.fields + (long long)c * p.L * M + (long long)(p.nt1 - 1) * M;
  const long long NN = (long long)N * N;

  // Positions (every warp, lane q = visit): an exclusive prefix sum of the vertex sizes.
  const int q = lane;
  int w = 0, n = 0;
  if (q < nq) {
    const int pos = p.q0 + q;
    n = p.dir == 0 ? pos : M - 1 - pos;
    w = nsite[n];
  }
  int incl = w;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  const int p0 = incl - w, np = __shfl_sync(0xffffffffu, incl, 31);
  if (warp == 1 && q < nq) {
    const int vb = p.vsite2 ? p.vsite2[(long long)c * p.V.sK + n] : -1;
    for (int I = 0; I < w; ++I) {
      s_psite[p0 + I] = I ? site2[n] : site[n];
      s_pvis[p0 + I] = q;
      s_pkind[p0 + I] = (w == 2) ? (I ? 2 : 1) : 0;  // 0 single, 1 first of a pair, 2 second
      s_psite2[p0 + I] = (w == 1) ? vb : -1;
      if (vb >= 0) {
        s_pc[p0 + I][0] = p.vcoef[2 * ((long long)c * p.V.sK + n)];
        s_pc[p0 + I][1] = p.vcoef[2 * ((long long)c * p.V.sK + n) + 1];
      }
    }
  }
  if (warp == 0 && q < nq) {
    // each vertex is visited once per block, so its old field is the field at block start and
    // every visit's proposal, draws and transition factors are known
    s_vtx[q] = n;
    const int v = p.visit_base + p.q0 + q;
    const int so = fl[n], tp = ty[n];
    double u0, u1, uu2;
    if (p.draws) {
      const double* d = p.draws + (long long)c * p.sDraws + 3ll * v;
      u0 = d[0]; u1 = d[1]; uu2 = d[2];
    } else {
      unsigned long long key = p.rngkey[c], ctr = p.rngctr[c] + 3ull * v;
      u0 = alf_uniform(key, ctr); u1 = alf_uniform(key, ctr + 1); uu2 = alf_uniform(key, ctr + 2);
    }
    const int ch = (tp == 1) ? 0 : nranf3(u0) - 1;
    const int sn = (tp == 1) ? -so : (int)p.ft.flip[so + 2][ch];
    const UpdTab* e = tab + ((long long)n * 5 + so + 2) * 3 + ch;
    s_snew[q] = sn;
    s_prop[q] = 1.5 > u1;  // T0_proposal (Wrapgr_mod.F90:123,133); always true
    // real models compare the weight with it bit by bit: one zero, and one NaN, which no weight is above
    long long ub = __double_as_longlong(uu2);
    if ((ub & 0x7fffffffffffffffll) > 0x7ff0000000000000ll) ub = 0x7ff8000000000000ll;
    if ((ub << 1) == 0) ub = 0;
    s_u2[q] = __longlong_as_double(ub);
    const double gr = p.ft.grat[tp - 1][so + 2][sn + 2];
    s_gr[q] = gr;
    zd K = e->expal;
    if (F == 2) K = zmul(K, e[(long long)M * 15].expal);
    // [prod_f exp(Z1 alpha)]^N_SUN gamma'/gamma: with N_SUN = 1 the gamma ratio joins K
    if (p.NSUN == 1) K = zscale(K, gr);
    s_K[q] = K;
    for (int f = 0; f < F; ++f)
      for (int I = 0; I < w; ++I) {
        const Z me = A::mk(e[(long long)f * M * 15].myexp[I]), dl = A::mk(e[(long long)f * M * 15].dlt[I]);
        s_mye[f][p0 + I] = me;
        s_dlt[f][p0 + I] = dl;
        // real FP64: K joins the first flavour's factor of a single position (the last factor of a pair)
        if (FOLD && I == w - 1) {
          s_myk[f][p0 + I] = f == 0 ? A::mul(me, A::mk(K)) : me;
          s_dlk[f][p0 + I] = f == 0 ? A::mul(dl, A::mk(K)) : dl;
        }
      }
  }
  if (warp != 0) {
    asm volatile("bar.sync 1, 224;" ::: "memory");  // positions (warps 1..7); warp 0 joins below
    if (p.Gsub) {
      for (int a = warp - 1; a < np; a += NW - 1)
        if (lane < np)
          for (int f = 0; f < F; ++f)
            Gh[(f * KM + a) * LD + lane] = A::mk(p.Gsub[(((long long)c * F + f) * KM + a) * KM + lane]);
    } else {
      for (int l = warp - 1; l < np; l += NW - 1)  // lane = row: consecutive sites are contiguous in G
        if (lane < np)
          for (int f = 0; f < F; ++f) {
            zd g;
            if (p.vsite2 && (s_psite2[lane] >= 0 || s_psite2[l] >= 0)) {
              // Ghat(a, l) = v_a^T G v_l over the (up to two) sites of each position
              const int ia[2] = {s_psite[lane], s_psite2[lane]}, il[2] = {s_psite[l], s_psite2[l]};
              const double ca[2] = {s_psite2[lane] >= 0 ? s_pc[lane][0] : 1.0, s_psite2[lane] >= 0 ? s_pc[lane][1] : 0.0};
              const double cl[2] = {s_psite2[l] >= 0 ? s_pc[l][0] : 1.0, s_psite2[l] >= 0 ? s_pc[l][1] : 0.0};
              g = zmk(0.0, 0.0);
              for (int x = 0; x < 2; ++x)
                for (int y = 0; y < 2; ++y)
                  if (ia[x] >= 0 && il[y] >= 0 && ca[x] != 0.0 && cl[y] != 0.0)
                    g = zadd(g, zscale(G[f * NN + ia[x] + (long long)il[y] * N], ca[x] * cl[y]));
            } else {
              g = G[f * NN + s_psite[lane] + (long long)s_psite[l] * N];
            }
            Gh[(f * KM + lane) * LD + l] = A::mk(g);
          }
    }
  }
  __syncthreads();

  // scalar state of warp 0 (identical in all lanes)
  zd ph = p.phase[c];  // FP64, kept unnormalised within a block (only its direction enters the weight)
  long long n_prop = 0;
  int nacc = 0;
  const int fo = (F == 2) ? (lane & 1) : 0;  // flavour of this lane's scalar work
  for (int v = 0; v < np; ++v) {
    const int kind = s_pkind[v];
    const int q = v - 1, qs = v > 0 ? q : 0;
    const int acc = v > 0 ? s_acc[q] : 0;
    if (warp == 0) {
      int a = 0;
      if (kind == 2) {  // second position: decided with the first
        a = acc;
        if (lane == 0) s_acc[v] = a;
      } else {
        const int vi = s_pvis[v], prop = s_prop[vi];
        zd Rt = zmk(0.0, 0.0);
        // Mat(1,1) = myexp - Delta G(P,P), and for the first position of a pair the 2x2
        // determinant D_a (myexp_b - Delta_b G'_bb); the real FP64 form has K in its last factor
        Z Rm;
        if (kind == 0) {
          const Z me = FOLD ? s_myk[fo][v] : s_mye[fo][v], dl = FOLD ? s_dlk[fo][v] : s_dlt[fo][v];
          Z g = Gh[(fo * KM + v) * LD + v];
          const Z tq = Tc[(fo * KM + qs) * KM + v], row = Gh[(fo * KM + qs) * LD + v];
          if (acc) g = A::mac(g, tq, row);
          Rm = A::mac(me, A::neg(dl), g);
        } else {
          const int w = v + 1, ra = v + ((lane >> 1) & 1), rb = v + ((lane >> 2) & 1);
          const Z me = FOLD ? s_myk[fo][w] : s_mye[fo][w], dl = FOLD ? s_dlk[fo][w] : s_dlt[fo][w];
          Z g = Gh[(fo * KM + ra) * LD + rb];
          if (acc) g = A::mac(g, Tc[(fo * KM + q) * KM + ra], Gh[(fo * KM + q) * LD + rb]);
          const Z gvv = A::shfl(g, fo), gwv = A::shfl(g, fo + 2), gvw = A::shfl(g, fo + 4), gww = A::shfl(g, fo + 6);
          const Z D = A::mac(s_mye[fo][v], A::neg(s_dlt[fo][v]), gvv);
          const Z xm = A::mul(s_dlt[fo][v], A::rcp(D));
          const Z gp = A::mac(gww, A::mul(xm, gwv), gvw);
          Rm = A::mul(D, A::mac(me, A::neg(dl), gp));
        }
        if (prop) {
          // the ratio is accumulated in FP64: flavour product, exp(Z1 alpha), N_SUN power
          if (A::kReal) {
            // the weight |Re(phase R) / Re(phase)| (Wrapgr_mod.F90:141-143) of a real ratio is |R|;
            // non-negative numbers compare like their bits
            double r = A::wide(Rm).x;
            if (F == 2) r *= __shfl_xor_sync(0xffffffffu, r, 1);
            if (!FOLD) r *= s_K[vi].x;
            if (p.NSUN != 1) {
              double rp = r;
              for (int e = 1; e < p.NSUN; ++e) rp *= r;
              r = rp * s_gr[vi];
            }
            Rt.x = r;
            const long long rb = __double_as_longlong(r) & 0x7fffffffffffffffll;
            // an infinite weight is a NaN in complex products (infinity times zero), so not accepted either
            a = rb < 0x7ff0000000000000ll && rb > __double_as_longlong(s_u2[vi]);
            if (a && __double_as_longlong(r) < 0) ph = zmk(alf_flip(ph.x), alf_flip(ph.y));
          } else {
            const zd Rm64 = A::wide(Rm);
            Rt = (F == 2) ? zmul(ArD::shfl(Rm64, 0), ArD::shfl(Rm64, 1)) : Rm64;
            Rt = zmul(Rt, s_K[vi]);
            if (p.NSUN != 1) {
              zd Rp = Rt;
              for (int e = 1; e < p.NSUN; ++e) Rp = zmul(Rp, Rt);
              Rt = zscale(Rp, s_gr[vi]);
            }
            // division-free
            const double num = fabs(ph.x * Rt.x - ph.y * Rt.y);
            const double den = fabs(ph.x) * s_u2[vi];
            a = num > den;
            if (a) ph = zmul(ph, Rt);
          }
        }
        n_prop += prop;
        nacc += a;
        if (lane == 0) {
          s_acc[v] = a;
          if (p.rec_acc) {
            const long long r = (long long)c * p.sRec + p.visit_base + p.q0 + vi;
            p.rec_acc[r] = (int8_t)a;
            p.rec_ratio[r] = Rt;
          }
        }
      }
    } else if (warp <= F) {
      const int f = warp - 1;
      Z* Gf = Gh + f * KM * LD;
      Z* Tf = Tc + f * KM * KM;
      const Z dl = s_dlt[f][v], me = s_mye[f][v], tq = Tf[qs * KM + lane];
      Z col = (lane < np) ? Gf[lane * LD + v] : A::zero();
      Z row = Gf[qs * LD + v];
      if (kind == 2) {  // the update before the pair's first position was left out of this column
        if (v > 1 && s_acc[v - 2] && lane > v - 2 && lane < np)
          col = A::mac(col, Tf[(v - 2) * KM + lane], Gf[(v - 2) * LD + v]);
        row = A::shfl(col, q);
        if (lane == q) Gf[q * LD + v] = col;
      }
      if (acc) col = A::mac(col, tq, row);  // Tc is zero on the rows up to its position
      const Z D = A::mac(me, A::neg(dl), A::shfl(col, v));
      const Z dc = A::mul(dl, col);
      const Z r = A::rcp(D);
      Tf[v * KM + lane] = (lane > v && lane < np) ? A::mul(dc, r) : A::zero();
      if (lane == 0) s_rD[f][v] = r;
    } else if (acc) {
      // Ghat(a,b) += x Ghat(a,q) Ghat(q,b), rows a > q, columns b > v (b > v + 1 if v opens a pair)
      const int b = lane;
      if (b > v + (kind == 1) && b < np)
        for (int f = 0; f < F; ++f) {
          const Z row = Gh[(f * KM + q) * LD + b];
          const Z* Tq = Tc + (f * KM + q) * KM;
          Z* g = Gh + f * KM * LD + b;
          const int ws = F + 1, st = NW - ws;  // first of these warps, and how many
          int a = v + (warp - ws);
          for (; a + st < np; a += 2 * st) {
            const Z g0 = g[a * LD], g1 = g[(a + st) * LD], t0 = Tq[a], t1 = Tq[a + st];
            g[a * LD] = A::mac(g0, t0, row);
            g[(a + st) * LD] = A::mac(g1, t1, row);
          }
          if (a < np) g[a * LD] = A::mac(g[a * LD], Tq[a], row);
        }
    }
    __syncthreads();
  }
  // accepted positions in order (every warp for itself)
  const int myacc = lane < np ? s_acc[lane] : 0;
  const unsigned mask = __ballot_sync(0xffffffffu, myacc);
  const int m = __popc(mask), my = __popc(mask & ((1u << lane) - 1u));
  if (warp == 0 && lane == 0) {
    p.m_out[c] = m;
    for (int f = 0; f < F; ++f) p.m_out[p.nChains + c * F + f] = m;
    if (m > 0) p.phase[c] = A::kReal ? ph : ArD::unit(ph);
    unsigned long long* cn = reinterpret_cast<unsigned long long*>(p.cnt) + 4ll * c;
    atomicAdd(cn, (unsigned long long)n_prop);
    atomicAdd(cn + 1, (unsigned long long)nacc);
    atomicAdd(cn + 2, (unsigned long long)nq);
    atomicAdd(cn + 3, (unsigned long long)nacc);
  }
  if (warp == NW - 1 && myacc) {
    p.sites_out[(long long)c * KM + my] = s_psite[lane];
    if (p.sites2_out) {
      p.sites2_out[(long long)c * KM + my] = s_psite2[lane];
      if (s_psite2[lane] >= 0) {
        p.coef_out[2 * ((long long)c * KM + my)] = s_pc[lane][0];
        p.coef_out[2 * ((long long)c * KM + my) + 1] = s_pc[lane][1];
      }
    }
    if (s_pkind[lane] != 2) fl[s_vtx[s_pvis[lane]]] = (int8_t)s_snew[s_pvis[lane]];
  }
  // W(l, k): C_lk below the diagonal, x_l on it, P_lk above
  if (myacc) s_accq[warp][my] = lane;
  __syncwarp();
  const int qk = s_accq[warp][lane];  // the lane-th accepted position (lane < m)
  for (int l = warp; l < m; l += NW) {
    const int ql = __shfl_sync(0xffffffffu, qk, l);
    if (lane < m)
      for (int f = 0; f < F; ++f) {
        const Z x = A::mul(s_dlt[f][ql], s_rD[f][ql]);
        const Z w = lane < l ? Tc[(f * KM + qk) * KM + ql] : (lane == l ? x : A::mul(x, Gh[(f * KM + ql) * LD + qk]));
        p.W[(((long long)c * 2 + f) * KM + l) * KM + lane] = A::wide(w);
      }
  }
}

// zb: bytes of one element in the kernel's arithmetic (16 complex or double-float, 8 real)
constexpr size_t upd_smem_bytes(size_t zb = 16) { return 2ull * UPD_KMAX * (2 * UPD_KMAX + 1) * zb; }

// Flush operands for G = G0 - X Y (one launch, spread over the GPU, in the precision form's
// arithmetic, double-float in the mixed form on complex models):
//   X(:, l) = G0 v_l
//   Y = (1 - P)^-1 diag(x) (1 - C)^-1 b,  b(l, :) = v_l^T - v_l^T G0
// with v_l = e_{s_l}, or c_a e_a + c_b e_b for a vector position (sites2 / coefs, may be null), and
// C, x, P as k_update leaves them in W.  One warp per column of Y (two columns when m <= 16),
// lane = l: two substitutions, one shuffle and one multiply-add per accepted position each.
// grid (ceil(N/8), chains*flavours), 256 threads.
// X: [chain][2][N][KMAX] col-major (ld N); Y: [chain][2][KMAX][N] col-major (ld KMAX).
template <class A>
__global__ void __launch_bounds__(256) k_flush_xy(const zd* Gv, long long sG, int N, int F, const int* m_in,
                                                  const int* sites, const zd* W, zd* X, zd* Y,
                                                  const int* sites2 = nullptr, const double* coefs = nullptr) {
  typedef typename A::Z Z;
  const int b = blockIdx.y, c = b / F, f = b % F;
  const int m = m_in[c];
  if (m == 0) return;
  const int cpw = m <= 16 ? 2 : 1;  // columns per warp
  const int col0 = blockIdx.x * 8 * cpw;
  if (col0 >= N) return;
  __shared__ Z Ws[UPD_KMAX][UPD_KMAX + 1];
  __shared__ int st[UPD_KMAX];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int l = tid; l < m; l += 256) st[l] = sites[(long long)c * UPD_KMAX + l];
  for (int e = tid; e < m * UPD_KMAX; e += 256)
    if ((e & 31) < m) Ws[e >> 5][e & 31] = A::mk(W[((long long)c * 2 + f) * UPD_KMAX * UPD_KMAX + e]);
  __syncthreads();
  const zd* Gf = Gv + (long long)c * sG + (long long)f * N * N;
  const long long xy = ((long long)c * 2 + f) * N * UPD_KMAX;
  for (int e = tid; e < m * 8 * cpw; e += 256) {  // rows col0 .. of X
    const int l = e / (8 * cpw), r = col0 + e % (8 * cpw);
    if (r >= N) continue;
    const int s = st[l], s2 = sites2 ? sites2[(long long)c * UPD_KMAX + l] : -1;
    zd x = Gf[r + (long long)s * N];
    if (s2 >= 0)
      x = zadd(zscale(x, coefs[2 * ((long long)c * UPD_KMAX + l)]),
               zscale(Gf[r + (long long)s2 * N], coefs[2 * ((long long)c * UPD_KMAX + l) + 1]));
    X[xy + r + (long long)l * N] = x;
  }
  const int wd = 32 / cpw, l = lane & (wd - 1);
  const int col = col0 + warp * cpw + lane / wd;
  Z y = A::zero();
  if (col < N && l < m) {
    const int s = st[l], s2 = sites2 ? sites2[(long long)c * UPD_KMAX + l] : -1;
    zd g = Gf[s + (long long)col * N];
    double e = s == col ? 1.0 : 0.0;
    if (s2 >= 0) {
      const double ca = coefs[2 * ((long long)c * UPD_KMAX + l)], cb = coefs[2 * ((long long)c * UPD_KMAX + l) + 1];
      g = zadd(zscale(g, ca), zscale(Gf[s2 + (long long)col * N], cb));
      e = (s == col ? ca : 0.0) + (s2 == col ? cb : 0.0);
    }
    y = A::mk(zsub(zmk(e, 0.0), g));
  }
  const int base = lane & ~(wd - 1);
  const int lr = l < m ? l : 0;
  for (int k = 0; k + 1 < m; ++k) {
    const Z yk = A::shfl(y, base + k);
    if (l > k && l < m) y = A::mac(y, Ws[lr][k], yk);
  }
  y = A::mul(y, Ws[lr][lr]);
  for (int k = m - 1; k > 0; --k) {
    const Z yk = A::shfl(y, base + k);
    if (l < k) y = A::mac(y, Ws[lr][k], yk);
  }
  if (col < N && l < m) Y[xy + l + (long long)col * UPD_KMAX] = A::wide(y);
}
