// Device-side lattice-resolved observables: the predefined equal-time and time-displaced
// measurements that ham%Obser / ham%ObserT run with the Green functions of the sweep
// (Prog/Predefined_Obs_mod.F90:137-330 equal time: Green, SpinMz (SpinZ, SpinXY, SpinT), Den;
// :330-600 time displaced; N_FL = 1 models: Green, SpinSUN, Den), accumulated per chain as
// Obs_Latt(imj, nt, no_I, no_J), Obs_Latt0(no), the measurement count and the sign sum, the
// arrays Print_bin_Latt normalises (Prog/observables_mod.F90:355-500).
//
// A contribution of the site pair (i, j) goes to R = imj(cell(i), cell(j)) and the orbitals
// (orb(i), orb(j)).  One CTA owns one output (R, no_I, no_J) and sums over the cells I, with
// J = jof(I, R) the cell at distance R from I, in a fixed order: no atomics, the same result for the
// same G.  Weights w = ZP ZS = Phase / Re(Phase) sign(Re(Phase)).
//
// The FP64 pipe bounds both kernels (an instruction of one warp holds its sub-partition ~64 cycles), so
// the pairs are dealt to as many warps as there are: a thread per pair of one output, the reduction
// packed (each step halves the values a lane still carries), and real arithmetic (ArRe) on real
// models, about 20 FP64 instructions a pair instead of 110.  A thread per output summing serially over
// the cells took, equal time, 8 x 8 sites, four chains: 209 us, 12 x 12 cells of two sites 511 us (time
// displaced 579); this, 7.9 and 12.5 us (13.0).
#pragma once
#include "arith.cuh"

struct LattObsParams {
  int N, F, nsun, ncell, norb, nnames;
  int L1;                // time slices of the accumulator: 1 (equal time) or Ltrot + 1
  const int* site_of;    // [ncell][norb] site of (cell, orbital)
  const int* jof;        // [ncell][ncell] jof[I ncell + R]: the cell J with imj(I, J) = R
  const zd* phase;       // [chain]
  zd* acc;               // [chain][nnames][ncell][L1][norb][norb]
  zd* acc0;              // [chain][nnames][norb]
  double* cnt;           // [chain][2]: measurements, sum of ZS
};

ALF_DEV zd lobs_weight(zd ph, double* zs) {
  const double s = ph.x > 0.0 ? 1.0 : (ph.x < 0.0 ? -1.0 : 0.0);
  *zs = s;
  return zmk(ph.x / ph.x * s, ph.y / ph.x * s);  // (Phase / Re Phase) ZS
}

// Totals of NV values over the CTA's 128 threads, known to the threads of warp 0 when it returns.
template <class A, int NV>
ALF_DEV void lobs_cta_sum(typename A::Z (&v)[NV]) {
  constexpr int P = A::kReal ? 1 : 2, M = NV * P <= 2 ? 2 : (NV * P <= 4 ? 4 : (NV * P <= 8 ? 8 : 16));
  __shared__ double red[4][M];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double x[M];
#pragma unroll
  for (int q = 0; q < M; ++q) x[q] = 0.0;
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    x[q * P] = A::re(v[q]);
    if (P == 2) x[q * P + P - 1] = A::im(v[q]);
  }
  const double s = warp_sum_packed<M>(x);
  if (lane % (32 / M) == 0) red[warp][lane / (32 / M)] = s;
  __syncthreads();
  if (warp != 0) return;
  double t = 0.0;
  if (lane < M) t = ((red[0][lane] + red[1][lane]) + red[2][lane]) + red[3][lane];
#pragma unroll
  for (int q = 0; q < NV; ++q)
    v[q] = A::mkz(__shfl_sync(0xffffffffu, t, q * P), P == 2 ? __shfl_sync(0xffffffffu, t, q * P + P - 1) : 0.0);
}

// Equal time, G = [chain][F][N][N] column-major in the callback's frame.
// grid (ncell norb^2 + norb, chains), 128 threads: CTAs past the outputs form Obs_Latt0.
template <class A>
__global__ void __launch_bounds__(128) k_obs_latt_eq(const zd* G, LattObsParams p) {
  typedef typename A::Z V;
  const int c = blockIdx.y, no = p.norb, t = blockIdx.x, tid = threadIdx.x;
  const long long NN = (long long)p.N * p.N;
  const zd* G0 = G + (long long)c * p.F * NN;
  const zd* G1 = G0 + (p.F == 2 ? NN : 0);
  const double ns = (double)p.nsun;
  const int nout = p.ncell * no * no;
  auto at = [&](const zd* X, int i, int j) { return A::mk(X[i + (long long)j * p.N]); };
  auto hole = [&](const zd* X, int i, int j) {  // delta_ij - X(i, j)
    return A::sub(A::mkz(i == j ? 1.0 : 0.0, 0.0), at(X, i, j));
  };
  if (t < nout) {
    const int R = t / (no * no), oi = (t / no) % no, oj = t % no;
    V s[5];  // Green, same-flavour and cross-flavour exchange, density and spin pairs
#pragma unroll
    for (int q = 0; q < 5; ++q) s[q] = A::zero();
    for (int I = tid; I < p.ncell; I += 128) {
      const int i = p.site_of[I * no + oi], J = p.jof[I * p.ncell + R], j = p.site_of[J * no + oj];
      const V g0 = at(G0, i, j), c0 = hole(G0, j, i), ci0 = hole(G0, i, i), cj0 = hole(G0, j, j);
      s[0] = A::add(s[0], c0);
      s[1] = A::mac(s[1], c0, g0);
      if (p.F == 1) {
        s[3] = A::mac(s[3], ci0, cj0);
        continue;
      }
      const V g1 = at(G1, i, j), c1 = hole(G1, j, i), ci1 = hole(G1, i, i), cj1 = hole(G1, j, j);
      s[0] = A::add(s[0], c1);
      s[1] = A::mac(s[1], c1, g1);
      if (p.nsun == 1) {
        s[2] = A::mac(A::mac(s[2], c0, g1), c1, g0);
        s[4] = A::mac(s[4], A::sub(ci1, ci0), A::sub(cj1, cj0));
      }
      s[3] = A::mac(s[3], A::add(ci0, ci1), A::add(cj0, cj1));
    }
    lobs_cta_sum<A, 5>(s);
    if (tid < p.nnames) {
      double zs;
      const zd w = lobs_weight(p.phase[c], &zs);
      const V zz = A::add(s[1], s[4]), den = A::add(A::scale(s[3], ns * ns), A::scale(s[1], ns));
      V o;
      if (tid == 0) o = A::scale(s[0], ns);                                   // Green
      else if (p.F == 1) o = tid == 1 ? A::scale(s[1], ns) : den;            // SpinSUN, Den
      else if (tid == 4) o = den;                                             // Den
      else if (p.nsun != 1) o = A::zero();
      else if (tid == 3) o = A::scale(A::add(A::scale(s[2], 2.0), zz), 1.0 / 3.0);  // SpinT
      else o = tid == 1 ? zz : s[2];                                          // SpinZ, SpinXY
      zd* a = p.acc + ((long long)c * p.nnames + tid) * nout + t;  // L1 = 1
      *a = zadd(*a, zmul(A::wide(o), w));
    }
    return;
  }
  const int o = t - nout;  // Obs_Latt0 of orbital o: sum over the cells
  V s[2] = {A::zero(), A::zero()};  // up + down, down - up
  for (int I = tid; I < p.ncell; I += 128) {
    const int i = p.site_of[I * no + o];
    const V ci0 = hole(G0, i, i);
    s[0] = A::add(s[0], ci0);
    if (p.F == 1) continue;
    const V ci1 = hole(G1, i, i);
    s[0] = A::add(s[0], ci1);
    s[1] = A::add(s[1], A::sub(ci1, ci0));
  }
  lobs_cta_sum<A, 2>(s);
  double zs;
  if (tid == 0) {
    const zd w = lobs_weight(p.phase[c], &zs);
    zd* a0 = p.acc0 + (long long)c * p.nnames * no;
    const zd zi = zmul(zscale(A::wide(s[0]), ns), w);
    zd* den = a0 + (p.F == 1 ? 2 : 4) * no + o;
    *den = zadd(*den, zi);
    if (p.F != 1 && p.nsun == 1) {
      const zd dz = zmul(A::wide(s[1]), w);
      a0[1 * no + o] = zadd(a0[1 * no + o], dz);
      a0[3 * no + o] = zadd(a0[3 * no + o], zscale(dz, 0.57735026918962576451));  // 1/sqrt(3)
    }
    if (o == 0) {
      p.cnt[2 * c] += 1.0;
      p.cnt[2 * c + 1] += zs;
    }
  }
}

// Time displaced at slice nt, Q = [chain][4][F][N][N] = [GT0, G0T, G00, GTT].
// grid (ncell norb^2 + norb, chains), 128 threads.
template <class A>
__global__ void __launch_bounds__(128) k_obs_latt_tau(const zd* Q, int nt, LattObsParams p) {
  typedef typename A::Z V;
  const int c = blockIdx.y, no = p.norb, F = p.F, t = blockIdx.x, tid = threadIdx.x;
  const long long NN = (long long)p.N * p.N;
  const zd* q = Q + (long long)c * 4 * F * NN;
  const zd *GT0 = q, *G0T = q + F * NN, *G00 = q + 2 * F * NN, *GTT = q + 3 * F * NN;
  const double ns = (double)p.nsun;
  const int nout = p.ncell * no * no;
  const long long per_name = (long long)p.ncell * p.L1 * no * no;
  auto at = [&](const zd* X, int f, int i, int j) { return A::mk(X[f * NN + i + (long long)j * p.N]); };
  auto occ = [&](const zd* X, int f, int i) { return A::sub(A::one(), at(X, f, i, i)); };
  if (t < nout) {
    const int R = t / (no * no), oi = (t / no) % no, oj = t % no;
    V s[5];  // Green, same-flavour and cross-flavour exchange, density and spin pairs
#pragma unroll
    for (int k = 0; k < 5; ++k) s[k] = A::zero();
    for (int I = tid; I < p.ncell; I += 128) {
      const int i = p.site_of[I * no + oi], J = p.jof[I * p.ncell + R], j = p.site_of[J * no + oj];
      const V a0 = at(GT0, 0, i, j), b0 = at(G0T, 0, j, i), ti0 = occ(GTT, 0, i), zj0 = occ(G00, 0, j);
      s[0] = A::add(s[0], a0);
      s[1] = A::mac(s[1], b0, a0);
      if (F == 1) {
        s[3] = A::mac(s[3], ti0, zj0);
        continue;
      }
      const V a1 = at(GT0, 1, i, j), b1 = at(G0T, 1, j, i), ti1 = occ(GTT, 1, i), zj1 = occ(G00, 1, j);
      s[0] = A::add(s[0], a1);
      s[1] = A::mac(s[1], b1, a1);
      s[2] = A::mac(A::mac(s[2], b0, a1), b1, a0);
      s[4] = A::mac(s[4], A::sub(at(GTT, 0, i, i), at(GTT, 1, i, i)), A::sub(at(G00, 0, j, j), at(G00, 1, j, j)));
      s[3] = A::mac(s[3], A::add(ti0, ti1), A::add(zj0, zj1));
    }
    lobs_cta_sum<A, 5>(s);
    if (tid < p.nnames) {
      double zs;
      const zd w = lobs_weight(p.phase[c], &zs);
      const V zz = A::sub(s[4], s[1]), den = A::sub(A::scale(s[3], ns * ns), A::scale(s[1], ns));
      V o;
      if (tid == 0) o = F == 1 ? s[0] : A::scale(s[0], 0.5);                          // Green
      else if (F == 1) o = tid == 1 ? A::neg(A::scale(s[1], ns)) : den;              // SpinSUN, Den
      else if (tid == 4) o = den;                                                     // Den
      else if (tid == 3) o = A::scale(A::sub(zz, A::scale(s[2], 2.0)), 1.0 / 3.0);  // SpinT
      else o = tid == 1 ? zz : A::neg(s[2]);                                          // SpinZ, SpinXY
      zd* a = p.acc + ((long long)c * p.nnames + tid) * per_name + ((long long)R * p.L1 + nt) * no * no + oi * no + oj;
      *a = zadd(*a, zmul(A::wide(o), w));
    }
    return;
  }
  const int o = t - nout;
  V s[2] = {A::zero(), A::zero()};  // up + down, up - down of GTT
  for (int I = tid; I < p.ncell; I += 128) {
    const int i = p.site_of[I * no + o];
    s[0] = A::add(s[0], occ(GTT, 0, i));
    if (F == 1) continue;
    s[0] = A::add(s[0], occ(GTT, 1, i));
    s[1] = A::add(s[1], A::sub(at(GTT, 0, i, i), at(GTT, 1, i, i)));
  }
  lobs_cta_sum<A, 2>(s);
  if (tid == 0) {
    double zs;
    const zd w = lobs_weight(p.phase[c], &zs);
    zd* a0 = p.acc0 + (long long)c * p.nnames * no;
    zd* den = a0 + (F == 1 ? 2 : 4) * no + o;
    *den = zadd(*den, zmul(zscale(A::wide(s[0]), ns), w));
    if (F != 1) {
      const zd dz = zmul(A::wide(s[1]), w);
      a0[1 * no + o] = zsub(a0[1 * no + o], dz);
      a0[3 * no + o] = zsub(a0[3 * no + o], zscale(dz, 0.57735026918962576451));
    }
    if (o == 0 && nt == 0) {
      p.cnt[2 * c] += 1.0;
      p.cnt[2 * c + 1] += zs;
    }
  }
}
