// Small per-slice and per-stabilisation kernels.
#pragma once
#include "common.cuh"
#include "linalg.cuh"

// Diagonal product of all single-site vertex exponentials of slice nt1 (1-based):
//   S(i) = prod_{n: P(n)=i} E_exp(1, s(n,nt1)),  Sinv(i) = prod E_exp(1, -s(n,nt1)).
// This is Op_mmultR / Op_Wrapup for diagonal operators (Operator_mod.F90:686-693,
// 776-781) for every vertex of the slice at once.  grid (B), block 256.
// sptr/slist: per (chain, flavour) the positions (vertex n, eigen-index I) of each site
// in ascending order, coded 2n + I (CSR, built at upload); Eexp: [k][I][s+2].
__global__ void k_slice_scale(const int8_t* fields, int L, int M, int N, int F, int nt1, const int* sptr,
                              const int* slist, const zd* Eexp, zd* S, zd* Sinv) {
  const int b = blockIdx.x, c = b / F, f = b % F;
  const int8_t* fl = fields + (long long)c * L * M + (long long)(nt1 - 1) * M;
  const int* ptr = sptr + (long long)b * (N + 1);
  const int* lst = slist + (long long)b * 2 * M;
  const zd* ee = Eexp + ((long long)c * F * M + (long long)f * M) * 10;
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    zd s = zmk(1.0, 0.0), si = zmk(1.0, 0.0);
    for (int e = ptr[i]; e < ptr[i + 1]; ++e) {
      const int code = lst[e], n = code >> 1, I = code & 1;
      const int sp = fl[n];
      s = zmul(s, ee[(long long)(2 * n + I) * 5 + sp + 2]);
      si = zmul(si, ee[(long long)(2 * n + I) * 5 - sp + 2]);
    }
    S[(long long)b * N + i] = s;
    Sinv[(long long)b * N + i] = si;
  }
}

// G(i,j) <- S(i) G(i,j) Sinv(j)  (deferred vertex wraps of one slice), grid (ceil(N*N/256), B)
__global__ void k_apply_scale(zd* G, const zd* S, const zd* Sinv, int N) {
  const int b = blockIdx.y;
  const long long NN = (long long)N * N;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < NN; e += (long long)gridDim.x * blockDim.x) {
    int i = e % N, j = e / N;
    zd* g = G + b * NN + e;
    *g = zmul(zmul(S[(long long)b * N + i], *g), Sinv[(long long)b * N + j]);
  }
}

// U = I, V = I, D = 1, det(U) = 1 (reset_UDV_state, udv_state_mod.F90:320-345)
__global__ void k_udv_reset(zd* U, zd* V, double* D, zd* detU, int N) {
  const int b = blockIdx.y;
  const long long NN = (long long)N * N;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < NN; e += (long long)gridDim.x * blockDim.x) {
    int i = e % N, j = e / N;
    zd v = zmk(i == j ? 1.0 : 0.0, 0.0);
    U[b * NN + e] = v;
    V[b * NN + e] = v;
    if (e < N) D[(long long)b * N + e] = 1.0;
    if (e == 0) detU[b] = zmk(1.0, 0.0);
  }
}

// decompose_UDV_state phase handling (udv_state_mod.F90:481-492): phase = prod R_ii *
// pivot sign (conjugated on the L side); R(1,:) /= phase; det(U) = det(Q) * phase.
__global__ void k_decomp_phase(zd* R, long long ldr, int N, const QRInfo* info, int left, zd* phase_out, zd* detU) {
  const int b = blockIdx.x;
  __shared__ zd s_beta;
  if (threadIdx.x == 0) {
    zd ph = info[b].prodR;
    if (info[b].psign < 0) ph = zneg(ph);
    if (left) ph = zconj(ph);
    phase_out[b] = ph;
    detU[b] = zmul(info[b].detQ, ph);
    s_beta = zdiv(zmk(1.0, 0.0), ph);
  }
  __syncthreads();
  zd* Rb = R + (long long)b * ldr * N;
  for (int j = threadIdx.x; j < N; j += blockDim.x) Rb[(long long)j * ldr] = zmul(s_beta, Rb[(long long)j * ldr]);
}

// U(:,1) *= phase
__global__ void k_scale_col0(zd* U, int N, const zd* phase) {
  const int b = blockIdx.x;
  zd* u = U + (long long)b * N * N;
  zd ph = phase[b];
  for (int r = threadIdx.x; r < N; r += blockDim.x) u[r] = zmul(u[r], ph);
}

// COMPARE_C (mymats_mod.F90:683-704) with the NaN test of Control_PrecisionG
// (control_mod.F90:219-263).  grid (CMP_BLOCKS, B), block 256; out[b] = {xmax, xmean},
// zeroed by the caller.  The maximum is taken over |d|^2 as an integer on the IEEE bit
// pattern (non-negative doubles order like their bits) and rooted once; the mean adds
// FP32 square roots per element (a diagnostic) in FP64 partial sums.  Per element this
// costs five FP64-pipe instructions instead of a hypot.
#define CMP_BLOCKS 32
__global__ void __launch_bounds__(256) k_compare(const zd* A, const zd* Bm, int N, double* out, int* err) {
  const int b = blockIdx.y;
  const long long NN = (long long)N * N;
  const zd* a = A + b * NN;
  const zd* c = Bm + b * NN;
  unsigned long long mx = 0ull;
  float sm = 0.f;
  int nan = 0;
  for (long long e = blockIdx.x * 256ll + threadIdx.x; e < NN; e += 256ll * CMP_BLOCKS) {
    const zd x = a[e], y = c[e];
    const unsigned long long bits[4] = {(unsigned long long)__double_as_longlong(x.x),
                                        (unsigned long long)__double_as_longlong(x.y),
                                        (unsigned long long)__double_as_longlong(y.x),
                                        (unsigned long long)__double_as_longlong(y.y)};
#pragma unroll
    for (int t = 0; t < 4; ++t) nan |= (bits[t] & 0x7fffffffffffffffull) > 0x7ff0000000000000ull;
    const double dx = x.x - y.x, dy = x.y - y.y;
    const double d2 = fma(dx, dx, dy * dy);
    const unsigned long long u = (unsigned long long)__double_as_longlong(d2);
    mx = u > mx ? u : mx;
    sm += sqrtf(__double2float_rn(d2));
  }
  __shared__ unsigned long long rm[8];
  __shared__ float rs[8];
  __shared__ int rn[8];
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long om = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = om > mx ? om : mx;
    sm += __shfl_xor_sync(0xffffffffu, sm, o);
  }
  nan = __any_sync(0xffffffffu, nan);
  if ((threadIdx.x & 31) == 0) { rm[threadIdx.x >> 5] = mx; rs[threadIdx.x >> 5] = sm; rn[threadIdx.x >> 5] = nan; }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long m = 0ull;
    double s = 0.0;
    int nn = 0;
    for (int w = 0; w < 8; ++w) { m = rm[w] > m ? rm[w] : m; s += (double)rs[w]; nn |= rn[w]; }
    if (m > 0x7ff0000000000000ull) nn = 1;
    atomicMax(reinterpret_cast<unsigned long long*>(out + 2 * b), m);  // |d|^2 bits; rooted by k_stab_finish
    atomicAdd(out + 2 * b + 1, s / (double)NN);
    if (nn) atomicOr(err, 1);
  }
}

// Op_phase angle sum (Operator_mod.F90:160-181): sum over n, nt of Im(g alpha phi).
__global__ void k_opphase(const int8_t* fields, int L, int M, int F, const zd* g, const zd* alpha, const int8_t* type,
                          FieldTables ft, double* out) {
  const int b = blockIdx.x, c = b / F, f = b % F;
  const int8_t* fl = fields + (long long)c * L * M;
  const long long k0 = (long long)c * F * M + (long long)f * M;
  double s = 0.0;
  for (long long e = threadIdx.x; e < (long long)L * M; e += blockDim.x) {
    int n = e % M;
    int sp = fl[e];
    zd ga = zmul(g[k0 + n], alpha[k0 + n]);
    s += ga.y * ft.phi[type[(long long)c * F * M + n] - 1][sp + 2];
  }
  __shared__ double r[8];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) r[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += r[w];
    out[b] = t;
  }
}

// Phase and precision bookkeeping after CGR on all flavours of a chain
// (main.F90:734-753, control_mod.F90:207-320).  stat layout per chain:
// [0] ncg [1] xmeanG_sum [2] xmaxG [3] xmaxP [4] ncg_tau [5] xmean_tau_sum [6] xmax_tau [7] sweeps
struct StabFinishParams {
  int C, F, NSUN, nvar, compare, init;
  const zd* detUR; const zd* detUL;   // [B]
  const QRInfo* info;                 // [B]
  const double* opang;                // [B]
  const double* cmp;                  // [B][2]
  zd* phase;                          // [C]
  double* stat;                       // [C][8]
  int* err;
  zd* rec_phase;                      // [C] slot for this point or null
};

__global__ void k_stab_finish(StabFinishParams p) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= p.C) return;
  zd Z = zmk(1.0, 0.0);
  double* st = p.stat + 8ll * c;
  for (int f = 0; f < p.F; ++f) {
    const int b = c * p.F + f;
    zd ph = zmul(p.detUR[b], zconj(p.detUL[b]));  // conj(det(U_R^H U_L))
    ph = zscale(ph, 1.0 / zabs(ph));
    if (p.info[b].psign < 0) ph = zneg(ph);
    zd q = zmul(p.info[b].prodR, p.info[b].detQ);
    if (p.nvar != 1) q = zconj(q);
    ph = zmul(ph, q);
    double s, co;
    sincos(p.opang[b], &s, &co);
    ph = zmul(ph, zmk(co, s));
    Z = zmul(Z, ph);
    if (p.compare) {
      double xmax = sqrt(p.cmp[2 * b]), xmean = p.cmp[2 * b + 1];  // k_compare leaves max |d|^2
      st[0] += 1.0;
      if (xmax > 10.0) atomicOr(p.err, 2);
      if (xmax > st[2]) st[2] = xmax;
      st[1] += xmean;
    }
  }
  zd Zp = Z;
  for (int e = 1; e < p.NSUN; ++e) Zp = zmul(Zp, Z);
  if (p.compare) {
    double X = zabs(zsub(Zp, p.phase[c]));
    if (X > st[3]) st[3] = X;
  }
  p.phase[c] = Zp;
  if (p.rec_phase) p.rec_phase[c] = Zp;
}

__global__ void k_real_to_complex(const double* a, zd* out, long long n) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) out[i] = zmk(a[i], 0.0);
}
__global__ void k_real_to_complex2(const double* a, const double* b, zd* oa, zd* ob, long long n) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) {
    oa[i] = zmk(a[i], 0.0);
    ob[i] = zmk(b[i], 0.0);
  }
}
__global__ void k_count_sweep(double* stat, int C) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < C) stat[8 * c + 7] += 1.0;
}

// G <- W G W^T for the block-diagonal real orthogonal W with the 2x2 block U (column-major)
// on every site pair: the rotated-basis G of two-site vertices back to the original basis.
// Rows: grid (ceil(N*npairs/256), B); columns: the same grid.
__global__ void k_rot_rows(zd* G, int N, const int* pairs, int npairs, double u00, double u10, double u01,
                           double u11) {
  const long long NN = (long long)N * N, b = blockIdx.y;
  const long long e = blockIdx.x * 256ll + threadIdx.x;
  if (e >= (long long)N * npairs) return;
  const int j = e % N, pr = e / N;
  zd* g = G + b * NN + (long long)j * N;
  const int a = pairs[2 * pr], c = pairs[2 * pr + 1];
  const zd x = g[a], y = g[c];
  g[a] = zadd(zscale(x, u00), zscale(y, u01));
  g[c] = zadd(zscale(x, u10), zscale(y, u11));
}
__global__ void k_rot_cols(zd* G, int N, const int* pairs, int npairs, double u00, double u10, double u01,
                           double u11) {
  const long long NN = (long long)N * N, b = blockIdx.y;
  const long long e = blockIdx.x * 256ll + threadIdx.x;
  if (e >= (long long)N * npairs) return;
  const int i = e % N, pr = e / N;
  zd* g = G + b * NN;
  const int a = pairs[2 * pr], c = pairs[2 * pr + 1];
  const zd x = g[i + (long long)a * N], y = g[i + (long long)c * N];
  g[i + (long long)a * N] = zadd(zscale(x, u00), zscale(y, u01));
  g[i + (long long)c * N] = zadd(zscale(x, u10), zscale(y, u11));
}


// Equal-time scalar observables of the Hubbard-type models at one ham%Obser call site
// (Hamiltonian_Hubbard_smod.F90:695-801; kinetic term as Predefined_Hoppings_Compute_Kin,
// Predefined_Hop_mod.F90:1905-1959), accumulated per chain:
//   GRC(i,j) = delta_ij - G(j,i),  ZP = Phase / Re(Phase),  ZS = sign(Re(Phase))
//   Kin  = N_SUN sum_f sum_ij H_f(i,j) GRC_f(i,j) = N_SUN sum_f [tr H_f - sum_ij H_f(i,j) G_f(j,i)]
//   Pot  = sum_i U_i GRC_1(i,i) GRC_dec(i,i)   (dec = 2 for two flavours, else 1)
//   Part = N_SUN sum_f sum_i GRC_f(i,i),  Ener = Kin + Pot
// acc[c] += {ZP ZS Kin, ZP ZS Pot, ZP ZS Part, ZP ZS Ener} (complex), ZS, 1.
// HT holds H_f transposed (HT_f[j + i N] = H_f(i,j)), so sum_ij H(i,j) G(j,i) is the
// elementwise sum over the two column-major arrays.  A cluster of CTAs (256 threads) per chain, each
// with its stretch of the elements and sites, the partial sums added in a fixed order.  The FP64 pipe
// bounds it: the kinetic sum is F N^2 multiply-adds (twice that in complex arithmetic) at 32 per 64
// cycles and sub-partition.  N = 64, four chains: one CTA per chain, complex, 19.6 us; this 10.9 us, most
// of it the latency of the final weights.
template <bool RE>
__global__ void __launch_bounds__(256) k_obs_scal(const zd* G, const zd* phase, const double* HT, const double* trH,
                                                  const double* U, int N, int F, int nsun, double* acc) {
  const int c = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ncl = gridDim.x, rank = blockIdx.x;  // one cluster per chain
  const long long NN = (long long)N * N;
  double kr = 0.0, ki = 0.0, pr = 0.0, pi = 0.0;
  for (int f = 0; f < F; ++f) {
    const zd* g = G + ((long long)c * F + f) * NN;
    const double* ht = HT + (long long)f * NN;
    for (long long e = rank * 256 + tid; e < NN; e += 256 * ncl) {
      const zd v = g[e];
      kr = fma(ht[e], v.x, kr);
      if (!RE) ki = fma(ht[e], v.y, ki);
    }
  }
  // Pot and Part need the diagonals of both flavours at the same site
  double rr = 0.0, ri = 0.0;
  for (int i = rank * 256 + tid; i < N; i += 256 * ncl) {
    const zd g1 = G[((long long)c * F) * NN + i + (long long)i * N];
    const zd a = zmk(1.0 - g1.x, RE ? 0.0 : -g1.y);  // GRC_1(i,i)
    zd b = a;
    if (F == 2) {
      const zd g2 = G[((long long)c * F + 1) * NN + i + (long long)i * N];
      b = zmk(1.0 - g2.x, RE ? 0.0 : -g2.y);
      rr += b.x;
      if (!RE) ri += b.y;
    }
    rr += a.x;
    if (!RE) ri += a.y;
    const zd ab = RE ? zmk(a.x * b.x, 0.0) : zmul(a, b);
    pr = fma(U[i], ab.x, pr);
    if (!RE) pi = fma(U[i], ab.y, pi);
  }
  double v[6] = {kr, ki, pr, pi, rr, ri};
#pragma unroll
  for (int q = 0; q < 6; ++q)
    if (!RE || q % 2 == 0) v[q] = warp_sum(v[q]);
  __shared__ double wsum[6][8], csum[6];
  if (lane == 0)
    for (int q = 0; q < 6; ++q) wsum[q][warp] = v[q];
  __syncthreads();
  double sq = 0.0;  // thread q < 6: total of v[q] over this CTA, then over the cluster
  if (tid < 6) {
    for (int w = 0; w < 8; ++w) sq += wsum[tid][w];
    csum[tid] = sq;
  }
  if (ncl > 1) {
    cluster_sync();
    if (rank == 0 && tid < 6)
      for (int r = 1; r < ncl; ++r) sq += dsmem_ld_f64(dsmem_addr(&csum[tid], r));
    cluster_sync();  // no CTA leaves while its sums may still be read
  }
  if (rank == 0 && warp == 0) {
    double s[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) s[q] = __shfl_sync(0xffffffffu, sq, q);
    if (tid != 0) return;
    double trh = 0.0;
    for (int f = 0; f < F; ++f) trh += trH[f];
    const zd kin = zmk(nsun * (trh - s[0]), -nsun * s[1]);
    const zd pot = zmk(s[2], s[3]);
    const zd part = zmk(nsun * s[4], nsun * s[5]);  // s[4], s[5]: sum_f sum_i GRC_f(i,i)
    const zd ph = phase[c];
    const double zs = ph.x > 0.0 ? 1.0 : (ph.x < 0.0 ? -1.0 : 0.0);
    const zd zpzs = ph.x != 0.0 ? zscale(zmk(1.0, ph.y / ph.x), zs) : zmk(0.0, 0.0);
    const zd o[4] = {kin, pot, part, zadd(kin, pot)};
    double* a = acc + 10ll * c;
    for (int q = 0; q < 4; ++q) {
      const zd w = zmul(o[q], zpzs);
      a[2 * q] += w.x;
      a[2 * q + 1] += w.y;
    }
    a[8] += zs;
    a[9] += 1.0;
  }
}

// ---- explicit vertex wraps of one phase (models with vector vertices) --------------------------
// A phase is a range [n0, n1) of vertices with pairwise disjoint supports in the rotated basis.
// Vertex n acts on its support with the block
//   kind 0 (one site a):            e_0
//   kind 1 (pair (a, b), diagonal): diag(e_0, e_1)
//   kind 2 (pair (a, b), vector u): I + (e_0 - 1) u u^T,  u = (c_a, c_b) real, |u| = 1
// where e_m = E_exp(m, s) of the vertex's field s (Op%E_exp of Operator_mod.F90:472-529), with
// s -> -s for the inverse (inv) and every entry conjugated for the adjoint (cj; the blocks
// are symmetric).  fl points at the slice's fields of chain 0 ([chain] stride fstride).
struct VtxPhase {
  const int8_t* fl; long long fstride;
  const int8_t* kind; const int* site; const int* site2; const double* coef;  // [chain][F*M]
  const zd* Eexp;                                                              // [chain][F*M][2][5]
  long long sK;                                                                // F * M
  int F, M, N, n0, n1, inv, cj;
};

ALF_DEV void vtx_block(const VtxPhase& p, int b, int n, int* a, int* c, zd m[4], int* two) {
  const int ch = b / p.F, f = b % p.F;
  const long long k = (long long)ch * p.sK + (long long)f * p.M + n;
  int s = p.fl[(long long)ch * p.fstride + n];
  if (p.inv) s = -s;
  const zd* ee = p.Eexp + k * 10;
  const zd e0 = ee[s + 2];
  const int kd = p.kind[k];
  *a = p.site[k];
  *two = kd != 0;
  if (kd == 0) {
    m[0] = e0;
  } else if (kd == 1) {
    *c = p.site2[k];
    m[0] = e0; m[1] = zmk(0.0, 0.0); m[2] = zmk(0.0, 0.0); m[3] = ee[5 + s + 2];
  } else {
    *c = p.site2[k];
    const double ua = p.coef[2 * k], ub = p.coef[2 * k + 1];
    const zd d = zmk(e0.x - 1.0, e0.y);
    m[0] = zadd(zmk(1.0, 0.0), zscale(d, ua * ua));
    m[1] = zscale(d, ua * ub);  // (b, a) entry
    m[2] = m[1];                 // (a, b) entry
    m[3] = zadd(zmk(1.0, 0.0), zscale(d, ub * ub));
  }
  if (p.cj)
    for (int e = 0; e < 4; ++e) m[e] = zconj(m[e]);
}

// X <- E X (rows of every vertex's support), grid (ceil(N * (n1 - n0) / 256), B)
__global__ void k_vtx_rows(zd* X, long long sX, VtxPhase p) {
  const int b = blockIdx.y;
  const long long e = blockIdx.x * 256ll + threadIdx.x;
  const int nv = p.n1 - p.n0;
  if (e >= (long long)p.N * nv) return;
  const int j = (int)(e % p.N), n = p.n0 + (int)(e / p.N);
  int a = 0, c = 0, two = 0;
  zd m[4];
  vtx_block(p, b, n, &a, &c, m, &two);
  zd* col = X + b * sX + (long long)j * p.N;
  if (!two) { col[a] = zmul(m[0], col[a]); return; }
  const zd xa = col[a], xc = col[c];
  col[a] = zadd(zmul(m[0], xa), zmul(m[2], xc));
  col[c] = zadd(zmul(m[1], xa), zmul(m[3], xc));
}

// X <- X E (columns of every vertex's support), grid (ceil(N * (n1 - n0) / 256), B)
__global__ void k_vtx_cols(zd* X, long long sX, VtxPhase p) {
  const int b = blockIdx.y;
  const long long e = blockIdx.x * 256ll + threadIdx.x;
  const int nv = p.n1 - p.n0;
  if (e >= (long long)p.N * nv) return;
  const int i = (int)(e % p.N), n = p.n0 + (int)(e / p.N);
  int a = 0, c = 0, two = 0;
  zd m[4];
  vtx_block(p, b, n, &a, &c, m, &two);
  zd* Xb = X + b * sX;
  if (!two) { Xb[i + (long long)a * p.N] = zmul(Xb[i + (long long)a * p.N], m[0]); return; }
  const zd xa = Xb[i + (long long)a * p.N], xc = Xb[i + (long long)c * p.N];
  Xb[i + (long long)a * p.N] = zadd(zmul(xa, m[0]), zmul(xc, m[1]));
  Xb[i + (long long)c * p.N] = zadd(zmul(xa, m[2]), zmul(xc, m[3]));
}

// copy of one slice's fields of every chain (the fields before the slice's updates)
__global__ void k_copy_fields(const int8_t* fields, int L, int M, int nt1, int8_t* out) {
  const int c = blockIdx.y;
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < M; n += gridDim.x * blockDim.x)
    out[(long long)c * M + n] = fields[(long long)c * L * M + (long long)(nt1 - 1) * M + n];
}

// ---- checkerboard hopping: bond operators --------------------------------------------------
// The bonds [fam[q], fam[q + 1]) of a family are disjoint two-site operators (P [F][ncheck][2], E [F][ncheck][4]
// real, column-major 2 x 2); batch entry b uses flavour b % F.  The RealExpOpT lmult / rmult of
// each bond (Prog/OpTTypes_mod.F90:135-304): rows (X <- E X) or columns (X <- X E), family by family.
// X(i, j) is multiplied by rs0(i) (conjugated with conj0) and cs0(j) before and rs1(i), cs1(j) after
// (null: not).
//
// Row operators act within a column of X and column operators within a row, so a CTA holds its T columns
// (rows) in shared memory through all families and the scalings: one launch where each family and
// the scaling took one of ~4 us, most of it launch and memory latency (N = 36, eight matrices, four
// families and the scaling: 20 us, this 6.7).  The next family's bonds are loaded ahead.
// Arithmetic A: ArD or ArRe.  grid (ceil(N / T), B), shared memory T N values.
struct BondScale {
  const zd *rs0 = nullptr, *cs0 = nullptr, *rs1 = nullptr, *cs1 = nullptr;
  int conj0 = 0;
};
template <class A, bool ROWS>
__global__ void __launch_bounds__(256) k_bonds(zd* X, int N, int F, const int* P, const double* E, int ncheck,
                                               const int* fam, int nfam, int reverse, int T, BondScale sc) {
  typedef typename A::Z Z;
  const int b = blockIdx.y, t0 = blockIdx.x * T, nt = min(T, N - t0), tid = threadIdx.x, nth = blockDim.x;
  const int2* Pf = reinterpret_cast<const int2*>(P) + (long long)(b % F) * ncheck;
  const double2* Ef = reinterpret_cast<const double2*>(E) + 2ll * (b % F) * ncheck;
  zd* Xb = X + (long long)b * N * N;
  const long long bN = (long long)b * N;
  extern __shared__ __align__(16) unsigned char bonds_raw[];
  Z* tile = reinterpret_cast<Z*>(bonds_raw);  // [t][operator index]
  auto bond = [&](int q, int e, int2& ac, double2& m02, double2& m13) {  // entry e of family q: bond e / nt
    const int f = reverse ? nfam - 1 - q : q, b0 = fam[f];
    if (e >= (fam[f + 1] - b0) * nt) { ac = make_int2(-1, 0); return; }
    const int k = b0 + e / nt;
    const double2 u = Ef[2 * k], v = Ef[2 * k + 1];
    ac = Pf[k];
    m02 = make_double2(u.x, ROWS ? v.x : u.y);  // of the first site's new value
    m13 = make_double2(ROWS ? u.y : v.x, v.y);
  };
  int2 ac, an;
  double2 p0, p1, n0, n1;
  bond(0, tid, an, n0, n1);
  for (int e = tid; e < N * nt; e += nth) {
    const int t = ROWS ? e / N : e % nt, o = ROWS ? e % N : e / nt, i = ROWS ? o : t0 + t, j = ROWS ? t0 + t : o;
    zd v = Xb[i + (long long)j * N];
    Z z = A::mk(v);
    if (sc.rs0) z = A::mul(sc.conj0 ? A::conj(A::mk(sc.rs0[bN + i])) : A::mk(sc.rs0[bN + i]), z);
    if (sc.cs0) z = A::mul(z, A::mk(sc.cs0[bN + j]));
    tile[t * N + o] = z;
  }
  __syncthreads();
  for (int q = 0; q < nfam; ++q) {
    ac = an; p0 = n0; p1 = n1;
    if (q + 1 < nfam) bond(q + 1, tid, an, n0, n1);
    for (int e = tid; ac.x >= 0; bond(q, e, ac, p0, p1)) {
      Z* x = tile + (e % nt) * N;
      const Z xa = x[ac.x], xc = x[ac.y];
      x[ac.x] = A::add(A::scale(xa, p0.x), A::scale(xc, p0.y));
      x[ac.y] = A::add(A::scale(xa, p1.x), A::scale(xc, p1.y));
      e += nth;
    }
    __syncthreads();
  }
  for (int e = tid; e < N * nt; e += nth) {
    const int t = ROWS ? e / N : e % nt, o = ROWS ? e % N : e / nt, i = ROWS ? o : t0 + t, j = ROWS ? t0 + t : o;
    Z z = tile[t * N + o];
    if (sc.rs1) z = A::mul(A::mk(sc.rs1[bN + i]), z);
    if (sc.cs1) z = A::mul(z, A::mk(sc.cs1[bN + j]));
    Xb[i + (long long)j * N] = A::wide(z);
  }
}
