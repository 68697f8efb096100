// FP64-accurate real GEMM on the BF16 tensor cores (tcgen05 + TMA), by exact digit
// slicing (the Ozaki scheme: T. Ozaki, T. Ogita, S. Oishi, S. M. Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numer. Algorithms 59, 2012).
//
// Every row of the M-side operand A (and every row of the N-side operand B, i.e. every
// output column) is scaled by a power of two 2^-e, rounded to b S - 1 bits below the row's
// largest entry and cut into S digits of b bits in balanced form, x = 2^e sum_s d_s 2^(-b s),
// |d_s| <= 2^(b-1).  The digits are integers, exact in BF16 (b <= 8).  For each anti-diagonal
// D = s + t <= S + 2 of the digit products, sum_{s+t=D} A_s B_t is accumulated on the
// tensor cores in FP32; b and S are chosen so that every partial sum is an integer of at most
// 2^24, so these accumulations are exact.  The diagonals are combined exactly (two 64-bit words) and
// rounded once to FP64.  What is lost: the operands' rounding, 2^-(b S) of the row scale per entry
// (S b = 56: 55 bits and a sign, FP64 entries near their row's maximum keep all their bits; 63 in the FP64
// form), and the dropped diagonals D >= S + 3, K S 2^(2b-2) 2^(-b(S+3)) of the scales at most (below 2^-58
// for digits of random sign).  Both are against the largest entries of a row of A and of a row of B: the
// error is normwise, and an output far below them has fewer digits of its own than an FP64 product leaves
// it.  Measured with 62 bits (N(0, 1) entries, K = 16 .. 448), of max|A_i.| max|B_j.|: 2^-51.8 .. 2^-50.2
// where a plain FP64 product has 2^-49.8 .. 2^-47.0; where the sum cancels 2^-62 (2^-50); of entries spread
// over 2^40 2^-53 (2^-50), but of (|A||B|)_ij 2^-33 at K = 16 (2^-50).  Green functions of sweeps are no
// further off than with FP64 products, also element by element.  FP32 products (2^-24) are not enough
// there (they are amplified by the stabilisation interval).  Balanced digits carry one bit more per product than signed magnitudes:
// 43 digit products at K = 256 (S = 8, b = 7) for the 53 of nine 6-bit magnitudes.
// Complex products are real GEMMs on interleaved real/imaginary rows
// (k_oz_slice modes) with the complex element assembled in the epilogue; real models use plain
// rows (OZ_REAL, OZ_OUT_REALZ).  The first S' digits of an S-digit slicing are the element rounded
// to S' digits, so a product may use a prefix of a buffer's slices (SbA /
// SbB give the buffers' own slice counts): fewer slices trade accuracy, 2^-(b S'), for
// (S' + 1)(S' + 2)/2 - 2 instead of (S + 1)(S + 2)/2 - 2 digit products.
//
//   k_oz_slice  FP64 -> BF16 digit slices [batch][S][Rpad][Kpad] (K contiguous) and the
//               row exponents, integer arithmetic only (the FP64 pipe is 1/64 of FP32)
//   k_oz_gemm   one CTA per 128 x BN output tile: per 64-wide K chunk, the chunk's B slices (double
//               buffered) and its A slices (ring of stages) come by TMA with 128-byte swizzle; an MMA
//               warp issues, per A slice and K step, one tcgen05.mma (M = 128, N = up to 256,
//               K = 16, BF16 -> FP32) against all B slices at once, into S + 1 TMEM accumulators (one
//               per diagonal, the MMA's column base offset by the A slice index), and
//               tcgen05.commit releases the buffers; eight warps read TMEM back
//               (tcgen05.ld 32x32b), combine, round, and write complex128/float64.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"

enum { OZ_REAL = 0, OZ_CROWS = 1, OZ_CKA = 2, OZ_CKB = 3 };
enum { OZ_OUT_COLS = 0, OZ_OUT_ROWS = 1, OZ_OUT_REAL = 2, OZ_OUT_CPLX = 3, OZ_OUT_REALZ = 4 };
#define OZ_KC 64          // K chunk of one TMA box (128 bytes of BF16)
#define OZ_BM 128         // MMA M
#ifndef OZ_TARGET_BITS
#define OZ_TARGET_BITS 54  // digits x bits per slice > this (an FP64 mantissa, one guard bit and a sign)
#endif

// ---------------------------------------------------------------------------------------
// Slicing
// ---------------------------------------------------------------------------------------
struct OzSliceParams {
  const void* src;          // complex128 (OZ_C*) or float64 (OZ_REAL)
  int mode;                 // OZ_*
  long long sr, sk, sb;     // source element strides: row, k, batch
  int modb;                 // source batch = b % modb when > 0
  const zd* ks; long long sks;  // optional real per-k scale (real part; complex k index)
  int conj;                 // OZ_CROWS: negate imaginary parts
  int srows;                // source rows (complex rows for OZ_C*)
  int Kc;                   // source K extent (complex k for OZ_C*)
  const int* kdyn;          // optional per-batch valid source K (entries beyond are zero)
  const int* perm; long long sperm;  // optional K remap (OZ_CROWS, OZ_REAL): element (i, k) is source (i, perm[k])
  int tri, trans;           // tri: zero the strictly lower triangle of the source in storage
                            // coordinates (row, col) = trans ? (k', i) : (i, k'), k' the remapped k
  const zd* rsc; long long srsc; int rinv;  // optional real per-row scale (real part), or its inverse
  int kvalid;               // > 0: source k >= kvalid are zero (with kdyn: the smaller bound)
  int unitlow, doff;        // OZ_CROWS: the source is a unit lower trapezoid (Householder vectors of a
                            // QR panel): storage (r, c) is 0 for r < c + doff, 1 for r == c + doff
  int S, bits;
  unsigned long long cadd;  // sum_s 2^(bits s + bits - 1), set by oz_launch_slice
  int Rpad, Kpad;
  unsigned short* out;      // BF16 bits, [batch][S][Rpad][Kpad]
  int* expo;                // [batch][Rpad]
  int* err;                 // bit 0: non-finite input
};

struct OzNum {
  unsigned long long m;  // value = (-1)^neg m 2^e2; m == 0: zero
  int e2, neg;
};

ALF_DEV OzNum oz_decode(double x, int* bad) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  const int E = (int)((u >> 52) & 0x7ff);
  OzNum r;
  r.neg = (int)(u >> 63);
  if (E == 0 || E == 0x7ff) {  // zero, subnormal (below 2^-1022: 0 here), inf / NaN (flagged)
    if (E == 0x7ff) *bad = 1;
    r.m = 0; r.e2 = 0;
    return r;
  }
  r.m = ((u & 0xfffffffffffffull) | 0x10000000000000ull) << 11;
  r.e2 = E - 1086;
  return r;
}

// x s as (m, e2, neg) with the product of the two 64-bit mantissas truncated to its high
// word (error < 2^-62 relative); s == nullptr: x alone.
ALF_DEV OzNum oz_num(double x, const double* s, int* bad) {
  OzNum n = oz_decode(x, bad);
  if (s && n.m) {
    const OzNum t = oz_decode(*s, bad);
    if (!t.m) { n.m = 0; return n; }
    n.m = __umul64hi(n.m, t.m);  // >= 2^62
    n.e2 += t.e2 + 64;
    n.neg ^= t.neg;
  }
  return n;
}



// Upper bound e with |x s| < 2^e from the exponent fields alone (one above the tight bound
// when the mantissa product stays below 2); x or s zero: -100000.
ALF_DEV int oz_ebound(double x, const double* s) {
  const int ex = (int)((__double_as_longlong(x) >> 52) & 0x7ff);
  if (ex == 0 || ex == 0x7ff) return -100000;
  int e = ex - 1022;
  if (s) {
    const int es = (int)((__double_as_longlong(*s) >> 52) & 0x7ff);
    if (es == 0 || es == 0x7ff) return -100000;
    e += es - 1022;
  }
  return e;
}

// Digits of one element pair of one logical row, one 32-bit word (two BF16) per slice: the value
// rounded to v = x s 2^(b S - 1 - e), |v| <= 2^(b S - 1); with C = sum_s 2^(b s + b - 1) added, the b-bit
// fields of v + C (the top one unmasked) are the balanced digits plus 2^(b-1).  A field f as
// float: 2^23 + f in FP32 is exact, subtracting 2^23 + 2^(b-1) leaves the digit, whose low 16
// bits are zero.
ALF_DEV void oz_write_pair(const OzSliceParams& p, unsigned* o, double x0, double x1, const double* s0,
                           const double* s1, int e, int* bad) {
  const int bS = p.bits * p.S;
  const unsigned mask = (1u << p.bits) - 1u;
  const float off = 8388608.0f + (float)(1 << (p.bits - 1));
  const size_t sstride = (size_t)p.Rpad * p.Kpad / 2;
  unsigned long long v[2];
  const double xs[2] = {x0, x1};
  const double* ss[2] = {s0, s1};
  const unsigned long long C = p.cadd;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const OzNum n = oz_num(xs[u], ss[u], bad);
    v[u] = C;
    if (n.m) {
      const int sh = e - n.e2 - bS;  // |x s| 2^(bS - 1 - e) = m 2^(-sh - 1), rounded (sh >= 0: |x s| < 2^e, bS <= 63)
      const unsigned long long r = sh >= 64 ? 0ull : ((n.m >> sh) + 1ull) >> 1;
      v[u] = n.neg ? C - r : C + r;
    }
  }
  const unsigned l0 = (unsigned)v[0], h0 = (unsigned)(v[0] >> 32);
  const unsigned l1 = (unsigned)v[1], h1 = (unsigned)(v[1] >> 32);
  for (int s = 0; s < p.S; ++s) {
    const int sh = p.bits * (p.S - 1 - s);
    const unsigned ms = s ? mask : 2u * mask + 1u;
    const unsigned a = (sh >= 32 ? (h0 >> (sh - 32)) : __funnelshift_r(l0, h0, sh)) & ms;
    const unsigned c = (sh >= 32 ? (h1 >> (sh - 32)) : __funnelshift_r(l1, h1, sh)) & ms;
    const float f0 = __uint_as_float(0x4B000000u + a) - off, f1 = __uint_as_float(0x4B000000u + c) - off;
    o[(size_t)s * sstride] = __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
  }
}

// One CTA per source row (one or two logical rows), one thread per pair of consecutive k:
// the row exponent(s) by a block reduction of exponent-field bounds, then the S digits of
// both elements of the pair (K contiguous).  Logical rows: OZ_REAL row i; OZ_CROWS 2 i + c
// (c = 0 real, 1 imaginary part of source row i); OZ_CKA row i with K = 2 Kc ([Re | Im]);
// OZ_CKB 2 j + c with K = 2 Kc: row 2j [Re Y(:, j); -Im Y(:, j)], row 2j + 1 [Im Y(:, j);
// Re Y(:, j)].  Padding rows of `out` are never written (zero from allocation); every
// k < Kl of a written row is (and k = Kl when Kl is odd), entries beyond kdyn as zeros.
// grid (srows, batch), blockDim = 32 ceil(Kl / 64) <= 256
__global__ void __launch_bounds__(256) k_oz_slice(OzSliceParams p) {
  __shared__ int red[2][8];
  const int b = blockIdx.y, i = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool two = p.mode == OZ_CROWS || p.mode == OZ_CKB;
  const int Kl = (p.mode == OZ_CKA || p.mode == OZ_CKB) ? 2 * p.Kc : p.Kc;
  const int bs = p.modb > 0 ? b % p.modb : b;
  const double* srd = (const double*)p.src + (size_t)bs * p.sb;
  const zd* srz = (const zd*)p.src + (size_t)bs * p.sb;
  const zd* ks = p.ks ? p.ks + (size_t)b * p.sks : nullptr;
  int kd = p.kdyn ? min(p.kdyn[b], p.Kc) : p.Kc;
  if (p.kvalid > 0) kd = min(kd, p.kvalid);
  double x0[2] = {0.0, 0.0}, x1[2] = {0.0, 0.0}, sc[2] = {1.0, 1.0};
  const int k0 = 2 * tid;
  double rs_row = 1.0;  // per-row scale (an output row / column scale of the product)
  if (p.rsc) {
    rs_row = p.rsc[(size_t)b * p.srsc + i].x;
    if (p.rinv) rs_row = 1.0 / rs_row;
  }
  const bool scaled = ks != nullptr || p.rsc != nullptr;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int k = k0 + u;
    if (k >= Kl) continue;
    switch (p.mode) {
      case OZ_REAL:
        if (k < kd) {
          const int kq = p.perm ? p.perm[(size_t)b * p.sperm + k] : k;
          if (p.tri && (p.trans ? kq > i : i > kq)) break;
          x0[u] = srd[i * p.sr + kq * p.sk];
        }
        break;
      case OZ_CROWS:
        if (k < kd) {
          const int kq = p.perm ? p.perm[(size_t)b * p.sperm + k] : k;
          if (p.tri && (p.trans ? kq > i : i > kq)) break;  // below the diagonal of an upper triangle
          if (p.unitlow) {
            const int r = p.trans ? kq : i, cc = (p.trans ? i : kq) + p.doff;
            if (r < cc) break;
            if (r == cc) { x0[u] = 1.0; break; }
          }
          const zd z = srz[i * p.sr + kq * p.sk];
          x0[u] = z.x; x1[u] = p.conj ? -z.y : z.y;
        }
        break;
      case OZ_CKA: {
        const int kc = k < p.Kc ? k : k - p.Kc;
        if (kc < kd) { const zd z = srz[i * p.sr + kc * p.sk]; x0[u] = k < p.Kc ? z.x : z.y; }
      } break;
      default: {
        const int kc = k < p.Kc ? k : k - p.Kc;
        if (kc < kd) {
          const zd z = srz[i * p.sr + kc * p.sk];
          x0[u] = k < p.Kc ? z.x : -z.y;
          x1[u] = k < p.Kc ? z.y : z.x;
        }
      } break;
    }
    if (ks) sc[u] = ks[k].x;
    if (p.rsc) sc[u] = rs_row;
  }
  int e0 = max(oz_ebound(x0[0], scaled ? &sc[0] : nullptr), oz_ebound(x0[1], scaled ? &sc[1] : nullptr));
  int e1 = two ? max(oz_ebound(x1[0], scaled ? &sc[0] : nullptr), oz_ebound(x1[1], scaled ? &sc[1] : nullptr))
               : -100000;
  e0 = __reduce_max_sync(0xffffffffu, e0);
  e1 = __reduce_max_sync(0xffffffffu, e1);
  if (lane == 0) { red[0][warp] = e0; red[1][warp] = e1; }
  __syncthreads();
  const int nw = blockDim.x >> 5;
  for (int w = 0; w < nw; ++w) { e0 = max(e0, red[0][w]); e1 = max(e1, red[1][w]); }
  if (e0 == -100000) e0 = 0;
  if (e1 == -100000) e1 = 0;
  const int r0 = two ? 2 * i : i;
  if (tid == 0) {  // the digits' scale is 2^(e + 1): v carries the sign in its top digit
    p.expo[(size_t)b * p.Rpad + r0] = e0 + 1;
    if (two) p.expo[(size_t)b * p.Rpad + r0 + 1] = e1 + 1;
  }
  if (k0 >= Kl) return;
  int bad = 0;
  unsigned* o = reinterpret_cast<unsigned*>(p.out + ((size_t)b * p.S * p.Rpad + r0) * p.Kpad + k0);
  oz_write_pair(p, o, x0[0], x0[1], scaled ? &sc[0] : nullptr, scaled ? &sc[1] : nullptr, e0, &bad);
  if (two)
    oz_write_pair(p, o + p.Kpad / 2, x1[0], x1[1], scaled ? &sc[0] : nullptr, scaled ? &sc[1] : nullptr, e1, &bad);
  if (bad && p.err) atomicOr(p.err, 1);
}

static inline cudaError_t oz_launch_slice(const OzSliceParams& p, int batch, cudaStream_t st) {
  const int Kl = (p.mode == OZ_CKA || p.mode == OZ_CKB) ? 2 * p.Kc : p.Kc;
  if (Kl > 512) return cudaErrorInvalidValue;
  OzSliceParams q = p;
  q.cadd = 0;
  for (int s = 0; s < p.S; ++s) q.cadd += 1ull << (p.bits * s + p.bits - 1);
  k_oz_slice<<<dim3(p.srows, batch), 32 * ((Kl + 63) / 64), 0, st>>>(q);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------
// tcgen05 / TMA / mbarrier primitives
// ---------------------------------------------------------------------------------------
ALF_DEV uint32_t oz_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

ALF_DEV void oz_mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
ALF_DEV void oz_mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
ALF_DEV bool oz_mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
#ifndef OZ_WAIT_CYCLES
#define OZ_WAIT_CYCLES (1ll << 31)  // a wait's limit in SM cycles: one second
#endif
// Bounded wait: gives up after OZ_WAIT_CYCLES and returns false.
ALF_DEV bool oz_mbar_wait(uint32_t bar, uint32_t parity) {
  if (oz_mbar_try(bar, parity)) return true;
  const long long t0 = clock64();
  while (!oz_mbar_try(bar, parity))
    if (clock64() - t0 > OZ_WAIT_CYCLES) return false;
  return true;
}
// The same for a converged warp: one answer for all its lanes.
ALF_DEV bool oz_mbar_wait_w(uint32_t bar, uint32_t parity) {
  return __all_sync(0xffffffffu, oz_mbar_wait(bar, parity)) != 0;
}
ALF_DEV void oz_tma_2d(uint32_t dst, const CUtensorMap* tm, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"((unsigned long long)tm), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
// Shared-memory matrix descriptor: K-major operand in the canonical 128-byte-swizzled
// layout (8-row x 128-byte atoms, atoms 1024 bytes apart along M/N), as written by TMA
// with CU_TENSOR_MAP_SWIZZLE_128B.  Fields: start >> 4 [0,14), leading byte offset >> 4
// [16,30) (unused for this layout), stride byte offset >> 4 [32,46), version 1 [46,48),
// swizzle mode 2 = 128 B [61,64).
ALF_DEV uint64_t oz_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3ffffu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// Instruction descriptor, kind::f16: FP32 accumulator [4,6) = 1, A and B BF16 [7,10) =
// [10,13) = 1, both K-major, N >> 3 at [17,23), M >> 4 at [24,29).
ALF_DEV uint32_t oz_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(OZ_BM >> 4) << 24);
}
ALF_DEV void oz_mma_acc(uint32_t dtmem, uint64_t ad, uint64_t bd, uint32_t idesc) {  // D += A B
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.eq.u32 p, 0, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtmem),
      "l"(ad), "l"(bd), "r"(idesc)
      : "memory");
}
ALF_DEV void oz_mma(uint32_t dtmem, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtmem),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
      : "memory");
}
// One lane of the converged warp (the same one each time).
ALF_DEV bool oz_elect() {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok));
  return ok != 0;
}
ALF_DEV void oz_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
ALF_DEV void oz_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
ALF_DEV void oz_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

// (zh 2^sh + zl) 2^sc rounded to the nearest FP64 (ties to even), 0 < sh < 64, |sum| < 2^95: integer
// arithmetic without branches.
ALF_DEV double oz_round(long long zh, long long zl, int sh, int sc) {
  // the 96-bit sum and its magnitude
  unsigned long long lo = ((unsigned long long)zh << sh) + (unsigned long long)zl;
  int w2 = (int)(zh >> (64 - sh)) + (int)(zl >> 63) + (lo < (unsigned long long)zl ? 1 : 0);
  const int neg = w2 >> 31;
  const unsigned long long nl = (unsigned long long)(long long)neg;
  lo = (lo ^ nl) - nl;
  unsigned a2 = (unsigned)((w2 ^ neg) + (neg && lo == 0ull ? 1 : 0));
  unsigned a1 = (unsigned)(lo >> 32), a0 = (unsigned)lo;
  // leading word to the top, then the leading bit; what falls off is kept as a sticky bit
  int T = 0;
  if (!a2) { a2 = a1; a1 = a0; a0 = 0u; T = 32; }
  if (!a2) { a2 = a1; a1 = 0u; T += 32; }
  const int n = __clz(a2);  // 32 only for zero
  const unsigned mh = __funnelshift_lc(a1, a2, n);
  unsigned ml = __funnelshift_lc(a0, a1, n);
  ml |= ((a0 << (n & 31)) != 0u) ? 1u : 0u;
  // 53 bits with the implicit one, rounded; a carry out of them raises the exponent by itself
  const unsigned rem = ml & 0x7ffu;
  unsigned long long r = (((unsigned long long)mh << 32) | ml) >> 11;
  r += (rem > 0x400u || (rem == 0x400u && (r & 1ull))) ? 1ull : 0ull;
  const int be = 95 - T - n + sc + 1023;
  unsigned long long u = ((unsigned long long)(unsigned)(be - 1) << 52) + r;
  if (be <= 0 || !a2) u = 0ull;
  if (be >= 2047 && a2) u = 0x7ff0000000000000ull;
  return __longlong_as_double((long long)(u | ((unsigned long long)(unsigned)neg << 63)));
}

// ---------------------------------------------------------------------------------------
// GEMM
// ---------------------------------------------------------------------------------------
struct OzGemmParams {
  int M, N;                  // logical rows of A and of B (valid extents)
  int nkc, S, bits, nst;     // K chunks (Kpad / 64), slices, bits per slice, ring stages
  int nd;                    // diagonals accumulated: s + t < nd (0-based digit indices), nd = S + 1
  int lg, pair;              // diagonals in the low word (ND - lg even); two diagonals fit 32 bits (oz_words)
  int Kv;                    // K steps of 16 that hold digits (the rest of Kpad is zero)
  int RpadA, RpadB;
  int modA, modB;            // operand batch = b % mod when > 0
  const int* expA; const int* expB;
  int omode, osub;           // OZ_OUT_*; osub 1: out -= A B, -1: out += A B (OZ_OUT_CPLX, OZ_OUT_REALZ)
  void* out; long long ldr, ldc, sout;  // element strides (float64 for _REAL, complex128 otherwise)
  int* err;                  // bit 2: a bounded wait gave up
  const zd* rsc; long long srsc;  // optional real scale of output row m (real part used), per batch
  const zd* csc; long long scsc;  // optional real scale of output column n (OZ_OUT_ROWS; real part), per batch
  int SbA, SbB;              // slices per batch entry in the A / B slice buffers (>= S: the first S are used)
  // k_oz_gemm<BN, true>: the grid is smaller than the tile count and each CTA takes tiles
  // blockIdx.x, blockIdx.x + gridDim.x, ... of the tiles_n x tiles_m x tiles_b tiles (N-tile
  // fastest); <BN, false>: one tile per CTA at (blockIdx.x, blockIdx.y, blockIdx.z)
  int persist, tiles_n, tiles_m, tiles_b;
};

static inline size_t oz_smem_bytes(int bn, int S, int nkc, int nst) {
  return (size_t)S * (nkc > 1 ? 2 : 1) * bn * 128 + (size_t)nst * OZ_BM * 128 + 256 + 1024;
}

template <int HB>
ALF_DEV void oz_tmem_ld_async(uint32_t taddr, uint32_t (&r)[HB]);
template <>
ALF_DEV void oz_tmem_ld_async<16>(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
template <>
ALF_DEV void oz_tmem_ld_async<8>(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
// Waits for the warp's TMEM loads; the registers are tied to the wait so that their uses stay behind it.
template <int HB>
ALF_DEV void oz_tmem_wait(uint32_t (&r)[HB], uint32_t (&q)[HB]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < HB; ++j) asm volatile("" : "+r"(r[j]), "+r"(q[j]));
}

// 256 threads.  Warp 0, one elected lane issuing, is the TMA producer (per K chunk the B slices into one of two
// buffers, then the A slices into the ring, as they free up), warp 1 issues the MMAs the same way and
// commits each buffer back to the producer; then all eight warps read TMEM: warp w takes TMEM
// lanes 32 (w % 4) .. + 31 (its sub-partition's) and columns (w / 4) BN/2 .. + BN/2 - 1.
// Holding one chunk's B slices instead of all of them leaves room, at 16-wide tiles, for two CTAs per
// SM, whose epilogues and main loops overlap.  Measured (K = 256, real): 32 matrices N = 256, 16-wide
// pairs 64 us, 32-wide with nine stages 67 us; two matrices 16 us and 19 us (start: 32-wide tiles with all B
// slices resident and one issuing thread, 105 us per real half of a complex product).  The ring's depth
// (2 .. 9) makes no difference: a chunk of 4 K steps takes ~450 cycles to issue.
// <16, true> has 104 registers a thread: two CTAs leave 12,288 of the SM's, what a CTA of the real visits in
// double-float takes (48 a thread), so the next block's visits start beside a flush.  With 105 (allocated as
// 112) they waited for it: 16 chains of 16 x 16, mixed, 317 ms a sweep for 306.
template <int BN, bool PERSIST = false>
__global__ void __launch_bounds__(256, BN == 16 ? 2 : 1) k_oz_gemm(const __grid_constant__ CUtensorMap tmA,
                                                    const __grid_constant__ CUtensorMap tmB, OzGemmParams p) {
  constexpr int HB = BN / 2;  // columns per epilogue thread
  extern __shared__ unsigned char oz_raw[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wu = __shfl_sync(0xffffffffu, warp, 0);  // warp index, uniform for the compiler
  const int S = p.S, nkc = p.nkc, NST = p.nst, ND = p.nd, NB = nkc > 1 ? 2 : 1;
  const uint32_t raw = oz_smem(oz_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t sB = base;                                      // [NB][S][BN rows x 128 B]
  const uint32_t sA = sB + (uint32_t)(NB * S * BN * 128);        // [NST][128 rows x 128 B]
  const uint32_t sBar = sA + (uint32_t)(NST * OZ_BM * 128);      // full[NST], empty[NST], bfull[2], bempty[2], done
  unsigned char* gbar = oz_raw + (sBar - raw);
  const uint32_t full0 = sBar, empty0 = sBar + 8u * NST, bfull0 = sBar + 16u * NST, bempty0 = bfull0 + 16,
                 done = bfull0 + 32;  // tslot, abort flag and consumed count follow
  uint32_t* tslot = reinterpret_cast<uint32_t*>(gbar + 16 * NST + 40);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gbar + 16 * NST + 44);
  volatile int* consumed_sh = reinterpret_cast<volatile int*>(gbar + 16 * NST + 48);
  const uint32_t cons = done + 16;  // shared address of *consumed_sh
  int ncols = 32;
  while (ncols < ND * BN) ncols <<= 1;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(oz_smem(tslot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 32) {
    for (int i = 0; i < NST; ++i) { oz_mbar_init(full0 + 8u * i, 1); oz_mbar_init(empty0 + 8u * i, 1); }
    for (int i = 0; i < 2; ++i) { oz_mbar_init(bfull0 + 8u * i, 1); oz_mbar_init(bempty0 + 8u * i, 1); }
    oz_mbar_init(done, 1);
    *abort_flag = 0;
    *consumed_sh = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  oz_fence_before();
  __syncthreads();
  oz_fence_after();
  const uint32_t tbase = *tslot;
  const int total = S * nkc;
  const uint32_t chunkA = OZ_BM * 128, chunkB = BN * 128;
  const int ntile = PERSIST ? p.tiles_n * p.tiles_m * p.tiles_b : 1;
  // stage and round of each A chunk and of each B chunk follow their counts over all tiles of this
  // CTA, kept as running (stage, round) pairs by the producer (p*) and the MMA issuer (m*); done
  // completes once per tile (parity = tile iteration & 1)
  int pst = 0, pround = 0, mst = 0, mround = 0, pbst = 0, pbround = 0, mbst = 0, mbround = 0;
  int it = 0;
  for (int tix = PERSIST ? (int)blockIdx.x : 0; tix < ntile; tix += PERSIST ? (int)gridDim.x : 1, ++it) {
  int b, m0, n0;
  if (PERSIST) {
    n0 = (tix % p.tiles_n) * BN;
    m0 = ((tix / p.tiles_n) % p.tiles_m) * OZ_BM;
    b = tix / (p.tiles_n * p.tiles_m);
  } else {
    b = blockIdx.z; m0 = blockIdx.y * OZ_BM; n0 = blockIdx.x * BN;
  }
  const int bA = p.modA > 0 ? b % p.modA : b, bB = p.modB > 0 ? b % p.modB : b;
  const uint32_t tpar = (uint32_t)(it & 1);

  // Both loops run on whole warps, with one elected lane issuing: in a one-thread branch the
  // compiler cannot keep the descriptors in uniform registers, and an MMA took ~325 cycles to issue.
  if (wu == 0) {  // producer
    const int rowA0 = bA * p.SbA * p.RpadA + m0, rowB0 = bB * p.SbB * p.RpadB + n0;
    const int g0 = it * total, gb0 = it * nkc;  // counts of this tile's first A and B chunk
    int loaded = 0, bloaded = 0;
    bool ok = true;
    for (int kc = 0; ok && kc < nkc; ++kc) {
      if (pbround > 0 && !oz_mbar_wait_w(bempty0 + 8u * pbst, (uint32_t)((pbround - 1) & 1))) { ok = false; break; }
      if (__any_sync(0xffffffffu, *abort_flag)) break;
      if (oz_elect()) {
        oz_mbar_expect_tx(bfull0 + 8u * pbst, (uint32_t)S * chunkB);
        for (int t = 0; t < S; ++t)
          oz_tma_2d(sB + (uint32_t)(pbst * S + t) * chunkB, &tmB, kc * OZ_KC, rowB0 + t * p.RpadB, bfull0 + 8u * pbst);
      }
      __syncwarp();
      ++bloaded;
      if (++pbst == NB) { pbst = 0; ++pbround; }
      for (int s = 0; s < S; ++s) {
        if (pround > 0 && !oz_mbar_wait_w(empty0 + 8u * pst, (uint32_t)((pround - 1) & 1))) { ok = false; break; }
        if (__any_sync(0xffffffffu, *abort_flag)) break;
        if (oz_elect()) {
          oz_mbar_expect_tx(full0 + 8u * pst, chunkA);
          oz_tma_2d(sA + (uint32_t)pst * chunkA, &tmA, kc * OZ_KC, rowA0 + s * p.RpadA, full0 + 8u * pst);
        }
        __syncwarp();
        ++loaded;
        if (++pst == NST) { pst = 0; ++pround; }
      }
      if (__any_sync(0xffffffffu, *abort_flag)) break;
    }
    if (!ok && lane == 0) { atomicOr(p.err, 4); *abort_flag = 1; }
    __syncwarp();
    if (__any_sync(0xffffffffu, *abort_flag)) {  // let every copy issued by this warp land before the CTA exits
      for (int q = gb0 + max(0, bloaded - NB); q < gb0 + bloaded; ++q) oz_mbar_wait(bfull0 + 8u * (uint32_t)(q % NB), (uint32_t)((q / NB) & 1));
      for (int q = g0 + *consumed_sh; q < g0 + loaded; ++q)
        oz_mbar_wait(full0 + 8u * (uint32_t)(q % NST), (uint32_t)((q / NST) & 1));
    }
  } else if (wu == 1) {  // MMA issuer
    oz_fence_after();  // the previous tile's TMEM reads are done (barrier below)
    bool ok = true;
    // descriptors differ only in the start-address field: advance them by (bytes >> 4)
    const uint64_t dA0 = oz_desc(sA), dB0 = oz_desc(sB);
    constexpr int TMAX = 256 / BN;  // B blocks per MMA (N <= 256)
    int q = 0;
    for (int kc = 0; ok && kc < nkc; ++kc) {
      if (!oz_mbar_wait_w(bfull0 + 8u * mbst, (uint32_t)(mbround & 1))) { ok = false; break; }
      const uint64_t dBk = dB0 + (uint64_t)((uint32_t)(mbst * S) * chunkB >> 4);
      const int nkk = min(OZ_KC / 16, p.Kv - kc * (OZ_KC / 16));
      for (int s = 0; s < S; ++s) {
        if (!oz_mbar_wait_w(full0 + 8u * mst, (uint32_t)(mround & 1))) { ok = false; break; }
        oz_fence_after();
        // A_s times the contiguous blocks B_0 .. B_{nt-1} of this K chunk in one MMA (N = nt BN),
        // into TMEM columns (s + t) BN: each product lands in its diagonal's accumulator.  In the
        // first K step s = 0 writes the diagonals 0 .. S - 1 and the last block of s = 1 diagonal S;
        // everything else accumulates.
        const uint64_t dA = dA0 + (uint64_t)(((uint32_t)mst * chunkA) >> 4);
        const int nt = min(S, ND - s), n1 = min(TMAX, nt), n2 = nt - n1;  // at most two MMAs per K step
        const uint32_t d1 = tbase + (uint32_t)(s * BN), d2 = d1 + (uint32_t)(n1 * BN);
        const uint32_t i1 = oz_idesc(n1 * BN), i2 = oz_idesc(n2 * BN);
        const uint64_t dB2 = dBk + (uint64_t)((uint32_t)n1 * chunkB >> 4);
        const bool start = kc == 0 && s < 2;
        if (oz_elect()) {
          if (start) {
            for (int kk = 0; kk < nkk; ++kk) {
              const int tw = (kk == 0 && s == 1) ? nt - 1 : nt;  // blocks that share one accumulate flag
              for (int t0 = 0; t0 < tw; t0 += TMAX) {
                const int n = min(TMAX, tw - t0);
                oz_mma(tbase + (uint32_t)((s + t0) * BN), dA + 2u * kk,
                       dBk + (uint64_t)((uint32_t)t0 * chunkB >> 4) + 2u * kk, oz_idesc(n * BN),
                       (kk == 0 && s == 0) ? 0u : 1u);
              }
              if (tw < nt)
                oz_mma(tbase + (uint32_t)((s + tw) * BN), dA + 2u * kk,
                       dBk + (uint64_t)((uint32_t)tw * chunkB >> 4) + 2u * kk, oz_idesc(BN), 0u);
            }
          } else if (n2) {
#pragma unroll
            for (int kk = 0; kk < OZ_KC / 16; ++kk)
              if (kk < nkk) {
                oz_mma_acc(d1, dA + 2u * kk, dBk + 2u * kk, i1);
                oz_mma_acc(d2, dA + 2u * kk, dB2 + 2u * kk, i2);
              }
          } else {
#pragma unroll
            for (int kk = 0; kk < OZ_KC / 16; ++kk)
              if (kk < nkk) oz_mma_acc(d1, dA + 2u * kk, dBk + 2u * kk, i1);
          }
          oz_commit(empty0 + 8u * mst);
          asm volatile("st.shared.u32 [%0], %1;" ::"r"(cons), "r"(q + 1) : "memory");
          if (s == S - 1) oz_commit(bempty0 + 8u * mbst);
        }
        __syncwarp();
        ++q;
        if (++mst == NST) { mst = 0; ++mround; }
      }
      if (!ok) break;
      if (++mbst == NB) { mbst = 0; ++mbround; }
    }
    if (!ok && lane == 0) { atomicOr(p.err, 4); *abort_flag = 1; }
    __syncwarp();
    if (oz_elect()) oz_commit(done);  // arrives when every MMA issued above has completed
    __syncwarp();
  }
  // the exponents of this thread's outputs, while the products run
  const int quarter = warp & 3, c0 = (warp >> 2) * HB, m = m0 + 32 * quarter + lane;
  const int ea = (m < p.M) ? p.expA[(size_t)bA * p.RpadA + m] : 0;
  int eb[HB];
#pragma unroll
  for (int j = 0; j < HB; ++j) {
    const int n = n0 + c0 + j;
    eb[j] = (n < p.N) ? p.expB[(size_t)bB * p.RpadB + n] : 0;
  }
  double old[HB];  // real outputs that are updated: read while the products run too
  const bool upd = p.omode == OZ_OUT_REALZ && p.osub != 0;
  if (upd) {
    const zd* o = (const zd*)p.out + (size_t)b * p.sout;
#pragma unroll
    for (int j = 0; j < HB; ++j)
      old[j] = (m < p.M && n0 + c0 + j < p.N) ? o[m * p.ldr + (n0 + c0 + j) * p.ldc].x : 0.0;
  }
  const bool mine_ok = oz_mbar_wait(done, tpar);
  oz_fence_after();
  const bool done_ok = __syncthreads_and(mine_ok) != 0;  // one answer for the CTA: TMEM loads are warp-wide
  if (!done_ok && tid == 0) { atomicOr(p.err, 4); *abort_flag = 1; }
  if (done_ok && !*abort_flag) {
    // The diagonals in two exact 64-bit words, the last lg of them in the low one.
    long long Zh[HB], Zl[HB];
#pragma unroll
    for (int j = 0; j < HB; ++j) { Zh[j] = 0; Zl[j] = 0; }
    const int lg = p.lg;
    const uint32_t tcol = tbase + ((uint32_t)(32 * quarter) << 16) + (uint32_t)c0;
    // The diagonals d, d + 1 first meet in one 32-bit word where it holds them (p.pair).
    auto f2i = [](uint32_t u) { return __float2int_rn(__uint_as_float(u)); };
    double v[HB];
    for (int d = 0; d < ND; d += 2) {  // two diagonals' loads in flight
      uint32_t r0[HB], r1[HB];
      const bool two = d + 1 < ND;
      oz_tmem_ld_async<HB>(tcol + (uint32_t)(d * BN), r0);
      if (two) oz_tmem_ld_async<HB>(tcol + (uint32_t)((d + 1) * BN), r1);
      oz_tmem_wait<HB>(r0, r1);
      if (two && p.pair) {
        if (d < ND - lg) {
#pragma unroll
          for (int j = 0; j < HB; ++j) Zh[j] = (Zh[j] << (2 * p.bits)) + (long long)((f2i(r0[j]) << p.bits) + f2i(r1[j]));
        } else {
#pragma unroll
          for (int j = 0; j < HB; ++j) Zl[j] = (Zl[j] << (2 * p.bits)) + (long long)((f2i(r0[j]) << p.bits) + f2i(r1[j]));
        }
      } else {
        if (d < ND - lg) {
#pragma unroll
          for (int j = 0; j < HB; ++j) Zh[j] = (Zh[j] << p.bits) + (long long)f2i(r0[j]);
        } else {
#pragma unroll
          for (int j = 0; j < HB; ++j) Zl[j] = (Zl[j] << p.bits) + (long long)f2i(r0[j]);
        }
        if (two && d + 1 < ND - lg) {
#pragma unroll
          for (int j = 0; j < HB; ++j) Zh[j] = (Zh[j] << p.bits) + (long long)f2i(r1[j]);
        } else if (two) {
#pragma unroll
          for (int j = 0; j < HB; ++j) Zl[j] = (Zl[j] << p.bits) + (long long)f2i(r1[j]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < HB; ++j) v[j] = oz_round(Zh[j], Zl[j], p.bits * lg, ea + eb[j] - p.bits * (ND + 1));
    if (p.rsc && m < p.M) {
      const double s = p.rsc[(size_t)b * p.srsc + m].x;
#pragma unroll
      for (int j = 0; j < HB; ++j) v[j] *= s;
    }
    if (p.csc) {  // OZ_OUT_ROWS, OZ_OUT_REALZ: real column n is output column n
#pragma unroll
      for (int j = 0; j < HB; ++j) {
        const int n = n0 + c0 + j;
        if (n < p.N) v[j] *= p.csc[(size_t)b * p.scsc + n].x;
      }
    }
    if (p.omode == OZ_OUT_REALZ) {  // real result, complex128 storage
      zd* o = (zd*)p.out + (size_t)b * p.sout;
      if (m < p.M)
#pragma unroll
        for (int j = 0; j < HB; ++j)
          if (n0 + c0 + j < p.N) {
            const double x = !upd ? v[j] : (p.osub > 0 ? old[j] - v[j] : old[j] + v[j]);
            o[m * p.ldr + (n0 + c0 + j) * p.ldc] = zmk(x, 0.0);
          }
    } else
    if (p.omode == OZ_OUT_REAL) {
      double* o = (double*)p.out + (size_t)b * p.sout;
      if (p.ldc == 1 && !p.osub && !(p.ldr & 1) && !(p.sout & 1) && n0 + c0 + HB <= p.N) {  // rows: 16-byte stores
        if (m < p.M) {
          double2* w = reinterpret_cast<double2*>(o + m * p.ldr + n0 + c0);
#pragma unroll
          for (int j = 0; j < HB / 2; ++j) w[j] = make_double2(v[2 * j], v[2 * j + 1]);
        }
      } else if (m < p.M)
#pragma unroll
        for (int j = 0; j < HB; ++j)
          if (n0 + c0 + j < p.N) {
            double* w = o + m * p.ldr + (n0 + c0 + j) * p.ldc;
            *w = p.osub ? *w - v[j] : v[j];
          }
    } else if (p.omode == OZ_OUT_COLS) {  // real column 2 j + c -> complex column j
      zd* o = (zd*)p.out + (size_t)b * p.sout;
      if (m < p.M)
#pragma unroll
        for (int j = 0; j < HB / 2; ++j) {
          const int jc = (n0 + c0) / 2 + j;
          if (2 * jc < p.N) {
            zd* w = o + m * p.ldr + jc * p.ldc;
            zd x = zmk(v[2 * j], v[2 * j + 1]);
            if (p.osub) { const zd g = *w; x = zmk(g.x - x.x, g.y - x.y); }
            *w = x;
          }
        }
    } else if (p.omode == OZ_OUT_CPLX) {
      // complex x complex: rows 2i / 2i+1 hold Re / Im of A's row i, columns 2j / 2j+1 Re / Im
      // of op(B)'s column j; C(i, j) = (ReA ReB - ImA ImB) + i (ReA ImB + ImA ReB).  The lane
      // pair of rows 2i, 2i+1 exchanges halves: even lanes finish the first HQ complex columns
      // of the thread's HB real columns, odd lanes the other HQ.
      zd* o = (zd*)p.out + (size_t)b * p.sout;
      const int i = m >> 1, c = m & 1;
      constexpr int HQ = HB / 4;
      double mine[HB / 2], got[HB / 2];
#pragma unroll
      for (int q2 = 0; q2 < HQ; ++q2) {
        // static register indices: select the value, not the index
        const double lo0 = v[2 * q2], lo1 = v[2 * q2 + 1], hi0 = v[2 * (HQ + q2)], hi1 = v[2 * (HQ + q2) + 1];
        got[2 * q2] = __shfl_xor_sync(0xffffffffu, c ? lo0 : hi0, 1);  // what the partner finishes
        got[2 * q2 + 1] = __shfl_xor_sync(0xffffffffu, c ? lo1 : hi1, 1);
        mine[2 * q2] = c ? hi0 : lo0;
        mine[2 * q2 + 1] = c ? hi1 : lo1;
      }
      if (2 * i < p.M)
#pragma unroll
        for (int q2 = 0; q2 < HQ; ++q2) {
          const int jc = (n0 + c0) / 2 + (c ? HQ + q2 : q2);
          if (2 * jc < p.N) {
            // even lane: mine = (ReA ReB, ReA ImB), got = (ImA ReB, ImA ImB); odd lane the reverse
            const double rr = c ? got[2 * q2] : mine[2 * q2], ri = c ? got[2 * q2 + 1] : mine[2 * q2 + 1];
            const double ir = c ? mine[2 * q2] : got[2 * q2], ii = c ? mine[2 * q2 + 1] : got[2 * q2 + 1];
            zd x = zmk(rr - ii, ri + ir);
            zd* w = o + i * p.ldr + jc * p.ldc;
            if (p.osub > 0) { const zd g = *w; x = zmk(g.x - x.x, g.y - x.y); }
            else if (p.osub < 0) { const zd g = *w; x = zmk(g.x + x.x, g.y + x.y); }
            *w = x;
          }
        }
    } else {  // OZ_OUT_ROWS: real row 2 i + c -> complex row i; even lanes write the first HB/2 columns
      zd* o = (zd*)p.out + (size_t)b * p.sout;
      const int i = m >> 1, c = m & 1;
      double u[HB / 2], w2[HB / 2];
#pragma unroll
      for (int j = 0; j < HB / 2; ++j) {
        const double send = c ? v[j] : v[HB / 2 + j];  // odd lanes send their first half, even their second
        const double got = __shfl_xor_sync(0xffffffffu, send, 1);
        u[j] = c ? got : v[j];                         // real part of column (c ? HB/2 + j : j)
        w2[j] = c ? v[HB / 2 + j] : got;               // imaginary part
      }
      if (2 * i < p.M)
#pragma unroll
        for (int j = 0; j < HB / 2; ++j) {
          const int n = n0 + c0 + (c ? HB / 2 : 0) + j;
          if (n < p.N) {
            zd* w = o + i * p.ldr + n * p.ldc;
            zd x = zmk(u[j], w2[j]);
            if (p.osub) { const zd g = *w; x = zmk(g.x - x.x, g.y - x.y); }
            *w = x;
          }
        }
    }
  }
  oz_fence_before();
  if (tid == 0) *consumed_sh = 0;  // the next tile's chunk count (read by the producer on abort)
  __syncthreads();  // TMEM reads and the shared B blocks are free for the next tile
  if (*abort_flag || !done_ok) break;
  }  // tiles
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(ncols) : "memory");
}

// ---------------------------------------------------------------------------------------
// Host helpers
// ---------------------------------------------------------------------------------------
typedef CUresult (*oz_encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static inline oz_encode_fn oz_encoder() {
  static oz_encode_fn fn = nullptr;
  if (!fn) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (oz_encode_fn)f;
  }
  return fn;
}

// 2-D map over a slice buffer [rows_total][Kpad] of BF16, box 64 x box_rows, 128-byte swizzle.
static inline int oz_tmap(CUtensorMap* m, void* base, int Kpad, long long rows_total, int box_rows) {
  oz_encode_fn enc = oz_encoder();
  if (!enc) return 1;
  const cuuint64_t dims[2] = {(cuuint64_t)Kpad, (cuuint64_t)rows_total};
  const cuuint64_t strides[1] = {(cuuint64_t)Kpad * 2};
  const cuuint32_t box[2] = {OZ_KC, (cuuint32_t)box_rows};
  const cuuint32_t es[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
                 CUDA_SUCCESS
             ? 0
             : 1;
}

// Digit width and count for a K extent: every diagonal partial sum stays an integer of at most
// 2^24 (S pairs, each at most K 4^(b-1)), and target < S b <= 63.
static inline int oz_pick(int Kpad, int* bits, int* S, int target = OZ_TARGET_BITS) {
  for (int b = 8; b >= 4; --b) {
    const int s = (target + b) / b;
    const double bound = (double)s * Kpad * (double)(1 << (2 * (b - 1)));
    if (s * b <= 63 && bound <= 16777216.0) { *bits = b; *S = s; return 0; }
  }
  return 1;
}

// The words of the epilogue: ND - lg diagonals (an even number) in the high one, |acc| <= 2^24 and
// lg b <= 40 keep each below 2^62; pair: |acc| (2^b + 1) < 2^31.
static inline void oz_words(int Kpad, int bits, int S, int nd, int* lg, int* pair) {
  *lg = (nd + 1) / 2;
  if ((nd - *lg) & 1) --*lg;
  *pair = (double)S * Kpad * (double)(1 << (2 * (bits - 1))) * ((1 << bits) + 1) < 2147483648.0;
}

static inline int oz_roundup(int x, int m) { return (x + m - 1) / m * m; }

// Tile width and ring depth.  pairs: 16-wide tiles (32-wide where the accumulators of two CTAs fit
// TMEM) with shared memory for two CTAs per SM; else the widest tile whose accumulators fit TMEM
// (512 columns), 16 with narrow, with the deepest ring.  1 when none fits.
static inline int oz_pick_tile(int S, int nkc, int* bn, int* nst, int narrow = 0, int pairs = 0) {
  const size_t cap = pairs ? 113 * 1024 : 232448;
  const int tcols = pairs ? 256 : 512;
  for (int w = narrow ? 16 : 32; w >= 16; w -= 16) {
    if ((S + 1) * w > tcols) continue;
    for (int st = 10; st >= 2; --st)
      if (oz_smem_bytes(w, S, nkc, st) <= cap) { *bn = w; *nst = st; return 0; }
  }
  return 1;
}
