// FP64 complex GEMM by residue arithmetic on the 5th-generation tensor cores
// (tcgen05 kind::i8): the Ozaki scheme II idea (Ozaki, Uchino, Imamura,
// arXiv:2504.08009) for complex operands.
//
//  1. Every row a_i of op(A) and column b_j of op(B) is scaled by a power of two and
//     rounded to Gaussian integers with ||a'_i||_2, ||b'_j||_2 <= 2^58.  By Cauchy-Schwarz
//     the real and imaginary parts of c'_ij = sum_k a'_ik b'_kj are below 2^116, so c' is
//     determined by its residues modulo P = product of the 16 moduli below (2^117.7).
//  2. Each modulus p has a square root of -1, iota: u = x + iota y and v = x - iota y map
//     the Gaussian integers mod p onto two copies of the integers mod p, in which the
//     complex product is two real ones (not four).  All residues are int8, the sums over K
//     exact in int32: 32 real int8 GEMMs of M x N x K.
//  3. The 32 residues of an output give Re c' / P and Im c' / P as fractions modulo 1
//     (Chinese remainder theorem), then the product with P and the power-of-two scales; or,
//     where both lines were integers up to a power of two, the exact integers c', rounded once.
//
// Accuracy: the roundings of step 1 are below 2^-58 of the row's (column's) 2-norm per
// component, so an element of C is off by about 0.58 2^-57 ||a_i|| ||b_j||, and by its own
// rounding.  An FP64 sum is off by up to (n + 1) 2^-53 S for its n nonzero terms, S =
// sum_k |a_ik| |b_kj|, which is less where the large elements of one line meet the small
// ones of the other.  So S is bounded from below for every element by one more int8 product,
// of the magnitudes (plane NPL - 1 below), and an element of which it does not follow that
// the FP64 bound holds is summed in FP64 in the reconstruction:
//   by Cauchy-Schwarz over the n terms, with lines of norm >= 2^57 and elements off by
//   2^-1/2, the error is at most sqrt(n / 2) 2^-56 ||a_i|| ||b_j||; it meets the FP64 bound
//   when S >= ||a_i|| ||b_j|| 2^-3.5 / sqrt(n).  n is at least nnz(a_i) + nnz(b_j) - K.
// Unstructured lines have S = 0.8 ||a_i|| ||b_j||, a flat line times one that a single element
// dominates still ||a_i|| ||b_j|| / sqrt(K).  A line with one nonzero element (the identity
// level of an environment) gives plain FP64 products, as exact as on the FP64 tensor cores,
// and lines that lose nothing in step 1 (integers, permutations) a correctly rounded result.
// Rows or columns with a NaN or an Inf are recognised and their elements computed as plain
// FP64 sums.
//
// The four kernels: partial row norms, residue and magnitude planes, the int8 GEMMs, the
// reconstruction.  Measured (B200): 6144 x 4096 x 1024 1.15 ms = 31 + 149 + 635 + 332 us
// (6.50 ms on the FP64 tensor cores), 4096 x 1024 x 6144 1.09 ms = 79 + 425 + 528 + 58 us
// (6.57 ms); the magnitudes and the checks cost 6 and 3 % of that.  With operands graded so
// that every element is summed in FP64, 6144 x 4096 x 1024 takes 12.4 ms; with an identity and
// noise of 1e-17 as one operand 2.9 ms.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <utility>

#include "gemm_modular.h"
#include "split_gemm.h"

namespace imps {
namespace {

constexpr int NMOD = 16;
constexpr int NRES = 2 * NMOD;   // residue planes: u of every modulus, then v
constexpr int NPL = NRES + 1;    // and the magnitudes
constexpr int BETA_BITS = 58;    // the integer operands' lines have 2-norm <= 2^58
constexpr int EXP_NONFINITE = 1 << 20;

// odd, pairwise coprime, at most 241, each with a square root of -1 (all prime factors 1 mod 4)
constexpr int kMod[NMOD] = {241, 233, 229, 221, 205, 197, 193, 181, 173, 157, 149, 137, 113, 109, 101, 97};

struct ModTables {
  // residue of a 64-bit integer: dp4a weights 256^j and iota 256^j mod p of its 8 bytes
  int wa_lo[NMOD], wa_hi[NMOD], wb_lo[NMOD], wb_hi[NMOD];
  // constants that take out the 2^62 bias of both integers (off_v relative to off_u), or the
  // 2^31 bias of an int32 sum; off_u and off_s carry the 1.5 2^23 of mod_byte
  int off_u[NMOD], off_v[NMOD], off_s[NMOD];
  int p[NMOD];
  float inv[NMOD];
  // CRT weights as fractions of P: the first 32 bits as an integer, the next 40 as a double;
  // re multiplies u + v, im multiplies u - v
  unsigned re1[NMOD], im1[NMOD];
  double re2[NMOD], im2[NMOD];
  unsigned re1_0, im1_0;           // -256 times the sums of the weights (see k_mod_join)
  double re2_0, im2_0;
  double P;
  // the weights as integers in [0, P), in three pieces w0 + 2^39 w1 + 2^78 w2, -256 times their
  // sums, P in the same pieces and 2^78 / P
  double re3[NMOD][3], im3[NMOD][3], re3_0[3], im3_0[3], p3[3], inv_p2;
};

constexpr int mod_pow(int b, int e, int p) {
  int r = 1;
  for (int i = 0; i < e; ++i) r = r * b % p;
  return r;
}
constexpr int mod_inv(int a, int p) {
  for (int x = 1; x < p; ++x)
    if (a * x % p == 1) return x;
  return 0;
}
constexpr int mod_iota(int p) {
  for (int x = 1; x < p; ++x)
    if ((x * x + 1) % p == 0) return x;
  return 0;
}
constexpr int kMagicBits = 0x4B400000;   // 1.5 2^23 as a float: its mantissa holds an integer
constexpr int centred(int x, int p) { return x > p / 2 ? x - p : x; }

// The part of g / p below 2^-32, to 2^-72: sums of 16 of them times 9-bit integers are exact
// in a double (so that vanishing residues give a zero), and what is dropped is 2^-8 of the
// rounding of the operands.
constexpr double low_weight(int g, int p) {
  const unsigned long long rem = ((unsigned long long)g << 32) % (unsigned)p;
  return (double)((((rem << 41) / (unsigned)p) + 1) >> 1) / 4722366482869645213696.0;   // 2^72
}

// 39 bits each of an integer below 2^118.  Sums of 16 of them times integers below 2^9 stay
// below 2^53, so three such sums are exact in doubles.
constexpr void pieces(unsigned __int128 x, double (&w)[3]) {
  w[0] = (double)(unsigned long long)(x & (((unsigned __int128)1 << 39) - 1));
  w[1] = (double)(unsigned long long)((x >> 39) & (((unsigned __int128)1 << 39) - 1));
  w[2] = (double)(unsigned long long)(x >> 78);
}

constexpr ModTables make_tables() {
  ModTables t{};
  unsigned __int128 P = 1;
  for (int i = 0; i < NMOD; ++i) P *= (unsigned)kMod[i];
  t.P = (double)(P >> 32) * 4294967296.0;   // the dropped 32 of 118 bits are below 2^-85 of it
  pieces(P, t.p3);
  t.inv_p2 = 302231454903657293676544.0 / t.P;   // 2^78 / P
  for (int i = 0; i < NMOD; ++i) {
    const int p = kMod[i], io = mod_iota(p);
    unsigned w[4] = {0, 0, 0, 0};
    for (int j = 0; j < 8; ++j) {
      const int a = mod_pow(256 % p, j, p), b = a * io % p;
      w[j / 4] |= (unsigned)(centred(a, p) & 255) << (8 * (j % 4));
      w[2 + j / 4] |= (unsigned)(centred(b, p) & 255) << (8 * (j % 4));
    }
    t.wa_lo[i] = (int)w[0];
    t.wa_hi[i] = (int)w[1];
    t.wb_lo[i] = (int)w[2];
    t.wb_hi[i] = (int)w[3];
    const int bias = mod_pow(2, 62, p), ib = bias * io % p;
    const int ou = centred((2 * p - bias - ib) % p, p), ov = centred((p - bias + ib) % p, p);
    t.off_u[i] = ou + kMagicBits;
    t.off_v[i] = ov - ou;
    t.off_s[i] = centred(p - mod_pow(2, 31, p), p) + kMagicBits;
    t.p[i] = p;
    t.inv[i] = 1.0f / (float)p;
    // (P / p)^-1 / 2 and (P / p)^-1 / (2 iota) mod p, as fractions of p
    int q = 1;
    for (int j = 0; j < NMOD; ++j)
      if (j != i) q = q * (kMod[j] % p) % p;
    const int g = mod_inv(q * 2 % p, p), h = mod_inv(q * 2 % p * io % p, p);
    t.re1[i] = (unsigned)(((unsigned long long)g << 32) / (unsigned)p);
    t.im1[i] = (unsigned)(((unsigned long long)h << 32) / (unsigned)p);
    t.re2[i] = low_weight(g, p);
    t.im2[i] = low_weight(h, p);
    t.re1_0 -= 256u * t.re1[i];
    t.im1_0 -= 256u * t.im1[i];
    t.re2_0 -= 256.0 * t.re2[i];
    t.im2_0 -= 256.0 * t.im2[i];
    pieces(P / (unsigned)p * (unsigned)g, t.re3[i]);
    pieces(P / (unsigned)p * (unsigned)h, t.im3[i]);
    for (int k = 0; k < 3; ++k) {
      t.re3_0[k] -= 256.0 * t.re3[i][k];
      t.im3_0[k] -= 256.0 * t.im3[i][k];
    }
  }
  return t;
}
// In unrolled code the constants of modulus I are immediates (a cold constant cache costs a
// short kernel microseconds); the GEMM's epilogue, which meets one modulus per tile, reads
// them from constant memory.
constexpr ModTables kT = make_tables();
__constant__ ModTables kTab = make_tables();

// ---------------------------------------------------------------------------
// Operands
// ---------------------------------------------------------------------------
// One side of the product: `lines` rows of op(A) or columns of op(B), each of K elements.
struct ModOperand {
  const double2* X;
  int64_t ld;
  int lines, K;
  int kcontig;        // element (l, k) at X[k + ld l], else at X[l + ld k]
  int conj;
  int8_t* planes;     // NPL planes of lines x Kp
  int64_t Kp;
  double* part;       // per K chunk and line: sum of squares, then max |re|, |im|
  int nchunk, kchunk;
  int* count;         // per K chunk and line: nonzero elements, the largest k of one, lowest bit
  int4* info;         // per line: the scale's exponent, nonzero elements, the last one's k,
                      // whether all elements are integers in the scale
  int nblocks_norm, nblocks_split;
};

__device__ __forceinline__ double2 load_elem(const ModOperand& o, int l, int k) {
  double2 v = o.kcontig ? o.X[k + o.ld * l] : o.X[l + o.ld * k];
  if (o.conj) v.y = -v.y;
  return v;
}

// A bound from below for the exponents of all set bits of a set of doubles: from the least
// exponent of a nonzero one and the zeros below all their mantissas.  (Whole numbers below 2^b
// come out no lower than 2^-b, which is low enough for the scale of a line up to b = 26, i.e.
// wherever a sum of such products is itself a double.)
struct LowBits {
  unsigned any = 0u, least = 0xffffffffu;
  __device__ __forceinline__ void add(double x) {
    const unsigned lo = (unsigned)__double2loint(x), hi = (unsigned)__double2hiint(x) & 0x7fffffffu;
    any |= lo;
    least = min(least, hi - (lo == 0u ? 1u : 0u));   // zero: the largest
  }
  __device__ __forceinline__ int bound() const {
    if (least == 0xffffffffu) return 4096;
    return (int)(least >> 20) - 1075 + (any ? __ffs((int)any) - 1 : 32);
  }
};
// 2^e in the double range, and x 2^e for any |e| <= 1100
__device__ __forceinline__ double pow2(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }
__device__ __forceinline__ double scale2(double x, int e) { return x * pow2(e / 2) * pow2(e - e / 2); }

// Whether a sum of squares has left (or may have left) the double range; m is the largest element
__device__ __forceinline__ bool squares_lost(double s, double m) {
  return m > 0.0 && !isinf(m) && !isnan(s) && !(s > 1e-280 && s < 1e280);
}

// Partial sums of squares and maxima of every line over the K chunks (a fixed order, so
// that the scales do not depend on timing).  Blocks [0, a.nblocks_norm) serve a.  A chunk
// whose squares leave the double range is summed again in units of 2^e > its largest element
// (frexp), and the sum stored with a minus sign.
__global__ void __launch_bounds__(256) k_mod_norms(const ModOperand a, const ModOperand b) {
  grid_enter();
  __shared__ double ss[4][64], sm[4][64];
  __shared__ int sn[4][64], sk[4][64], sb[4][64];
  const bool first = (int)blockIdx.x < a.nblocks_norm;
  const ModOperand& o = first ? a : b;
  const int blk = first ? blockIdx.x : blockIdx.x - a.nblocks_norm;
  const int chunk = blk % o.nchunk, grp = blk / o.nchunk;
  const int k0 = chunk * o.kchunk, k1 = min(o.K, k0 + o.kchunk);
  double* psum = o.part + (int64_t)chunk * o.lines;
  double* pmax = o.part + (int64_t)(o.nchunk + chunk) * o.lines;
  int* pnnz = o.count + (int64_t)chunk * o.lines;
  int* plast = o.count + (int64_t)(o.nchunk + chunk) * o.lines;
  int* plow = o.count + (int64_t)(2 * o.nchunk + chunk) * o.lines;
  double s = 0.0, m = 0.0;
  int nz = 0, last = 0;
  LowBits bits;
  auto add = [&](double2 v, int k) {
    s = fma(v.x, v.x, fma(v.y, v.y, s));
    m = fmax(m, fmax(fabs(v.x), fabs(v.y)));
    // nonzero (a NaN too), by integer instructions beside the FP64 ones
    if (((unsigned)(__double2hiint(v.x) | __double2hiint(v.y)) << 1 | __double2loint(v.x) | __double2loint(v.y)) != 0u) {
      ++nz;
      last = k;
    }
    bits.add(v.x);
    bits.add(v.y);
  };
  auto add_scaled = [&](double2 v, int e) {
    v.x = scale2(v.x, -e);
    v.y = scale2(v.y, -e);
    s = fma(v.x, v.x, fma(v.y, v.y, s));
  };
  if (o.kcontig) {
    // eight lanes a line, 32 lines a block
    const int l = grp * 32 + (threadIdx.x >> 3);
    if (l < o.lines)
      for (int k = k0 + (threadIdx.x & 7); k < k1; k += 8) add(o.X[k + o.ld * l], k);
    int low = bits.bound();
    const unsigned mine = 0xffu << (threadIdx.x & 24);
#pragma unroll
    for (int d = 4; d >= 1; d >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, d);
      m = fmax(m, __shfl_xor_sync(0xffffffffu, m, d));
      nz += __shfl_xor_sync(0xffffffffu, nz, d);
      last = max(last, __shfl_xor_sync(0xffffffffu, last, d));
      low = min(low, __shfl_xor_sync(0xffffffffu, low, d));
    }
    if (squares_lost(s, m)) {   // the same for the line's eight lanes
      int e;
      frexp(m, &e);
      s = 0.0;
      for (int k = k0 + (threadIdx.x & 7); k < k1; k += 8) add_scaled(o.X[k + o.ld * l], e);
#pragma unroll
      for (int d = 4; d >= 1; d >>= 1) s += __shfl_xor_sync(mine, s, d);
      s = -s;
    }
    if (l < o.lines && (threadIdx.x & 7) == 0) {
      psum[l] = s;
      pmax[l] = m;
      pnnz[l] = nz;
      plast[l] = last;
      plow[l] = low;
    }
  } else {
    const int tl = threadIdx.x & 63, tk = threadIdx.x >> 6, l = grp * 64 + tl;
    if (l < o.lines)
      for (int k = k0 + tk; k < k1; k += 4) add(o.X[l + o.ld * k], k);
    ss[tk][tl] = s;
    sm[tk][tl] = m;
    sn[tk][tl] = nz;
    sk[tk][tl] = last;
    sb[tk][tl] = bits.bound();
    __syncthreads();
    double t = (ss[0][tl] + ss[1][tl]) + (ss[2][tl] + ss[3][tl]);
    m = fmax(fmax(sm[0][tl], sm[1][tl]), fmax(sm[2][tl], sm[3][tl]));
    const bool lost = squares_lost(t, m);
    if (__syncthreads_or(lost)) {
      if (lost) {
        int e;
        frexp(m, &e);
        s = 0.0;
        for (int k = k0 + tk; k < k1; k += 4) add_scaled(o.X[l + o.ld * k], e);
        ss[tk][tl] = s;
      }
      __syncthreads();
      if (lost) t = -((ss[0][tl] + ss[1][tl]) + (ss[2][tl] + ss[3][tl]));
    }
    if (tk == 0 && l < o.lines) {
      psum[l] = t;
      pmax[l] = m;
      pnnz[l] = (sn[0][tl] + sn[1][tl]) + (sn[2][tl] + sn[3][tl]);
      plast[l] = max(max(sk[0][tl], sk[1][tl]), max(sk[2][tl], sk[3][tl]));
      plow[l] = min(min(sb[0][tl], sb[1][tl]), min(sb[2][tl], sb[3][tl]));
    }
  }
}

// The scale of a line from its chunks' partial results, by eight lanes together (q of them): x 2^e
// rounds to integers of 2-norm in [2^57, 2^58] (the rounding adds at most sqrt(K / 2), far
// below the 2^0.6 that 2^116 leaves under P / 2).  frac: that norm as a fraction of 2^58.
__device__ __forceinline__ int4 line_info(const ModOperand& o, int l, int q, double& frac) {
  double s = 0.0, m = 0.0;
  int nz = 0, last = 0, low = 4096;
  bool lost = false;
  if (l < o.lines)
    for (int c = q; c < o.nchunk; c += 8) {
      const double t = o.part[(int64_t)c * o.lines + l];
      lost = lost || t < 0.0;
      s += t;
      m = fmax(m, o.part[(int64_t)(o.nchunk + c) * o.lines + l]);
      nz += o.count[(int64_t)c * o.lines + l];
      last = max(last, o.count[(int64_t)(o.nchunk + c) * o.lines + l]);
      low = min(low, o.count[(int64_t)(2 * o.nchunk + c) * o.lines + l]);
    }
#pragma unroll
  for (int d = 4; d >= 1; d >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, d);
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, d));
    nz += __shfl_xor_sync(0xffffffffu, nz, d);
    last = max(last, __shfl_xor_sync(0xffffffffu, last, d));
    low = min(low, __shfl_xor_sync(0xffffffffu, low, d));
  }
  frac = 1.0;
  // a NaN does not pass fmax but does reach the sum of squares
  const bool nonfinite = isnan(s) || isinf(m);
  int unit = 0;
  if (__any_sync(0xffffffffu, lost)) {   // all chunks of such a line in units of 2^unit > m
    const unsigned mine = 0xffu << (threadIdx.x & 24);
    lost = (__ballot_sync(0xffffffffu, lost) & mine) != 0u && !nonfinite;
    if (lost) {
      frexp(m, &unit);
      s = 0.0;
      for (int c = q; c < o.nchunk; c += 8) {
        const double t = o.part[(int64_t)c * o.lines + l], mc = o.part[(int64_t)(o.nchunk + c) * o.lines + l];
        int ec = 0;
        if (t < 0.0) frexp(mc, &ec);
        // (a plain sum beside one that left the range is no larger than 2^930; what underflows
        // here is nothing to the result)
        s += scale2(scale2(fabs(t), max(ec - unit, -1100)), max(ec - unit, -1100));
      }
#pragma unroll
      for (int d = 4; d >= 1; d >>= 1) s += __shfl_xor_sync(mine, s, d);
    }
  }
  int e = 0;
  if (nonfinite) {
    e = EXP_NONFINITE;
  } else if (m > 0.0) {
    frac = frexp(sqrt(s) * (1.0 + 1e-12), &e);
    e = BETA_BITS - (e + unit);
  }
  return make_int4(e, nz, last, low + e >= 0);
}

__device__ __forceinline__ int dp4a_us(unsigned a, int b, int c) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
// The residue of s mod p nearest zero (in [-p/2 - 1, p/2 + 1]) in the low byte of the
// result; sb = s + kMagicBits, |s| < 2^22.  (kMagicBits is 0 mod 256, so it needs no care.)
__device__ __forceinline__ int mod_byte(int sb, int p, float inv) {
  const float f = __int_as_float(sb) - 12582912.0f;
  return sb - __float_as_int(fmaf(f, inv, 12582912.0f)) * p;
}
// low bytes of four words
__device__ __forceinline__ unsigned pack4(int r0, int r1, int r2, int r3) {
  return __byte_perm(__byte_perm(r0, r1, 0x0040), __byte_perm(r2, r3, 0x0040), 0x5410);
}

// Magnitudes: element k of a line as q = floor(mag_units max(|re|, |im|)) <= 127, in units of
// 16 / 127 of the line's root mean square, so that sum_k q_ik q_kj is at most
// 127^2 K / 256 S / (||a_i|| ||b_j||), with S as above.  (Larger elements are cut off, which
// keeps it a lower bound; the usual ones have eight levels.)  The GEMM's epilogue keeps the
// sum's exponent and three bits of its mantissa in a byte.
constexpr float MAG_TOP = 127.0f, MAG_RMS = 16.0f;
__device__ __forceinline__ uint32_t mag_byte(int sum) {
  const int bits = __float_as_int(__int2float_rz(sum));   // sum >= 0
  return (uint32_t)max(0, (bits >> 20) - (127 << 3));
}
__device__ __forceinline__ float mag_sum(uint32_t byte) { return byte ? __int_as_float((int)(byte + (127 << 3)) << 20) : 0.0f; }
// Whether a sum (its byte) shows the FP64 bound for n terms: sum >= 127^2 K / 256 2^-3.5 / sqrt(n)
// (and the roundings of the magnitudes, below 2^-10 in all); limit = mag_limit(K)
__device__ __forceinline__ float mag_limit(int K) {
  const float t = MAG_TOP * MAG_TOP / (MAG_RMS * MAG_RMS) * 0.0885f * (float)K;
  return t * t;
}
__device__ __forceinline__ bool mag_shows(uint32_t byte, int n, float limit) {
  const float t = mag_sum(byte);
  return t * t * (float)max(n, 1) >= limit;
}
__device__ __forceinline__ float mag_units(int K, double frac) {   // for max(|re|, |im|) / 2^32
  return MAG_TOP / MAG_RMS * sqrtf((float)K) / (float)frac * 0x1p-26f;
}

// The u and v bytes of 8 integers modulo modulus I into its two planes.
template <int I>
__device__ __forceinline__ void split_modulus(const unsigned (&xlo)[8], const unsigned (&xhi)[8],
                                              const unsigned (&ylo)[8], const unsigned (&yhi)[8], int8_t* out,
                                              int64_t plane) {
  constexpr int wal = kT.wa_lo[I], wah = kT.wa_hi[I], wbl = kT.wb_lo[I], wbh = kT.wb_hi[I];
  constexpr int offu = kT.off_u[I], offv = kT.off_v[I], p = kT.p[I];
  constexpr float inv = kT.inv[I];
  int u[8], v[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int sx = dp4a_us(xhi[c], wah, dp4a_us(xlo[c], wal, offu));
    const int sy = dp4a_us(yhi[c], wbh, dp4a_us(ylo[c], wbl, 0));
    u[c] = mod_byte(sx + sy, p, inv);
    v[c] = mod_byte(sx - sy + offv, p, inv);
  }
  *reinterpret_cast<uint2*>(out + plane * I) = make_uint2(pack4(u[0], u[1], u[2], u[3]), pack4(u[4], u[5], u[6], u[7]));
  *reinterpret_cast<uint2*>(out + plane * (NMOD + I)) =
      make_uint2(pack4(v[0], v[1], v[2], v[3]), pack4(v[4], v[5], v[6], v[7]));
}
template <int... I>
__device__ __forceinline__ void split_moduli(const unsigned (&xlo)[8], const unsigned (&xhi)[8],
                                             const unsigned (&ylo)[8], const unsigned (&yhi)[8], int8_t* out,
                                             int64_t plane, std::integer_sequence<int, I...>) {
  (split_modulus<I>(xlo, xhi, ylo, yhi, out, plane), ...);
}

// Residue planes.  A block covers SPL_LINES lines x 64 k of the padded extent, transposed
// through shared memory; a thread turns 8 consecutive k of a line into 8 bytes of each plane.
// Bound by its integer instructions (about 250 a complex element) and the 32 plane bytes;
// small blocks let one's loads run beside another's arithmetic.
constexpr int SPL_LINES = 16, SPL_NT = SPL_LINES * 8;
__global__ void __launch_bounds__(SPL_NT, 1024 / SPL_NT) k_mod_split(const ModOperand a, const ModOperand b) {
  grid_enter();
  __shared__ double2 tile[SPL_LINES][65];
  const bool first = (int)blockIdx.x < a.nblocks_split;
  const ModOperand& o = first ? a : b;
  const int blk = first ? blockIdx.x : blockIdx.x - a.nblocks_split;
  const int nk = (int)(o.Kp / 64);
  const int k0 = (blk % nk) * 64, l0 = (blk / nk) * SPL_LINES;
  const int tid = threadIdx.x;
  const int ll = tid >> 3, kq = tid & 7;
  if (o.kcontig) {
    const int kx = tid & 63, ly = tid >> 6;
#pragma unroll
    for (int r = 0; r < SPL_LINES; r += SPL_NT / 64) {
      const int l = l0 + r + ly, k = k0 + kx;
      tile[r + ly][kx] = (l < o.lines && k < o.K) ? o.X[k + o.ld * l] : make_double2(0.0, 0.0);
    }
  } else {
    const int lx = tid % SPL_LINES, ky = tid / SPL_LINES;
#pragma unroll
    for (int r = 0; r < 64; r += 8) {
      const int l = l0 + lx, k = k0 + r + ky;
      tile[lx][r + ky] = (l < o.lines && k < o.K) ? o.X[l + o.ld * k] : make_double2(0.0, 0.0);
    }
  }
  double frac;
  const int4 info = line_info(o, l0 + ll, kq, frac);
  if (k0 == 0 && kq == 0 && l0 + ll < o.lines) o.info[l0 + ll] = info;
  __syncthreads();
  if (l0 + ll >= o.lines) return;
  const int e = info.x == EXP_NONFINITE ? 0 : info.x, eh = e / 2;
  const double s1 = pow2(eh), s2 = pow2(e - eh);
  const float unit = mag_units(o.K, frac);
  unsigned xlo[8], xhi[8], ylo[8], yhi[8], q[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const double2 v = tile[ll][8 * kq + c];
    const unsigned long long nx = (unsigned long long)__double2ll_rn(v.x * s1 * s2) + (1ull << 62);
    const unsigned long long ny = (unsigned long long)__double2ll_rn((o.conj ? -v.y : v.y) * s1 * s2) + (1ull << 62);
    xlo[c] = (unsigned)nx;
    xhi[c] = (unsigned)(nx >> 32);
    ylo[c] = (unsigned)ny;
    yhi[c] = (unsigned)(ny >> 32);
    // (the floors of both components, one less in magnitude where negative: a lower bound)
    const int hx = (int)xhi[c] - (1 << 30), hy = (int)yhi[c] - (1 << 30);
    const int h = max(max(hx, -1 - hx), max(hy, -1 - hy));
    q[c] = (unsigned)__float_as_int(__fadd_rz(fminf((float)h * unit, MAG_TOP), 8388608.0f));
  }
  int8_t* out = o.planes + (int64_t)(l0 + ll) * o.Kp + k0 + 8 * kq;
  const int64_t plane = (int64_t)o.lines * o.Kp;
  *reinterpret_cast<uint2*>(out + plane * NRES) =
      make_uint2(pack4((int)q[0], (int)q[1], (int)q[2], (int)q[3]), pack4((int)q[4], (int)q[5], (int)q[6], (int)q[7]));
  split_moduli(xlo, xhi, ylo, yhi, out, plane, std::make_integer_sequence<int, NMOD>{});
}

// ---------------------------------------------------------------------------
// The int8 GEMMs: CTA pairs (cta_group::2) on 256 x 256 tiles
// ---------------------------------------------------------------------------
// A tile's A rows and B rows are split over the two CTAs (128 each), so a K stage of 128
// bytes brings 32 KB into each SM for 2 x 128 x 256 x 128 multiply-adds: 64 bytes a clock at
// the full int8 rate, half of what 128 x 128 tiles of single CTAs need from L2.  Warp 0
// loads (TMA, no multicast; both CTAs' bytes arrive at the leader's barrier), warp 1 of the
// leader issues the MMAs and warps 2-17 of both reduce the int32 sums modulo p and write
// them as bytes (blocks of 16 columns, so that a warp's rows are contiguous) while the next
// tile's MMAs run into the other TMEM buffer.
constexpr int GT = 256;                    // tile rows and columns
constexpr int HALF = 128;                  // rows of A and of B in each CTA
constexpr int GKB = 128;                   // K bytes a stage
constexpr int GSTAGES = 6;
constexpr int GSTAGE_BYTES = 2 * HALF * GKB;
constexpr int GBUF = 2;
constexpr int GEPI = 16;
constexpr int GTHREADS = 32 * (2 + GEPI);
constexpr int GSMEM = GSTAGES * GSTAGE_BYTES + 1024 + 512;
constexpr long long GDRAIN = 2000000000LL;

struct ModGemmArgs {
  int num_m, num_n, kblocks;
  int M;                // rows written
  int64_t ldo;          // columns of the output planes (a multiple of 32, >= N)
  uint8_t* out;         // NPL planes of ldo / 16 column blocks of M rows of 16 bytes
  int* err;
  long long wait_cycles;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded: false (and the error flag raised) after `limit` cycles
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* err, long long limit) {
  if (mbar_try(bar, parity)) return true;
  const long long t0 = clock64();
  unsigned spins = 0;
  while (!mbar_try(bar, parity)) {
    ++spins;
    if (spins != 1u && (spins & 255u) != 0u) continue;
    if (spins != 1u && *err) return false;
    if (clock64() - t0 > limit) {
      atomicExch((int*)err, 1);
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ void mbar_drain(uint64_t* bar, uint32_t parity) {
  const long long t0 = clock64();
  while (!mbar_try(bar, parity) && clock64() - t0 < GDRAIN) {
  }
}
__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// the leader's copy of a barrier, as a shared::cluster address
__device__ __forceinline__ uint32_t leader_addr(const void* p) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
  return a;
}
__device__ __forceinline__ void tma_load_pair(void* dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
// K-major shared-memory descriptor, 128B swizzle, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// kind::i8: s32 = s8 x s8, both K-major, M = N = 256 over the pair
constexpr uint32_t GIDESC = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(GT >> 3) << 17) | ((uint32_t)(GT >> 4) << 24);

__device__ __forceinline__ void mma_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(GIDESC), "r"(acc));
}
// arrives at the barrier of both CTAs when the MMAs issued so far have retired
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// What each role of a pair got done, told to both CTAs: the stages that the two producers
// filled and that the MMA thread has read
enum : uint32_t { DONE_FILL0, DONE_FILL1, DONE_MMA, DONE_SLOTS };
__device__ __forceinline__ void publish(uint32_t* slot, uint32_t n) {
#pragma unroll
  for (uint32_t r = 0; r < 2; ++r) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(slot)), "r"(r));
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(n) : "memory");
  }
}
// The end of both CTAs, by all their threads.  Every commit of the leader arrives at the
// barriers of both, so each CTA stays until its own copies have completed: the `empty` phases
// of the last stages read, the `tfull` phases of the last tiles (kblocks stages each) and
// `drain`.  With every stage read nothing is in flight then.
// After a wait that gave up, the leader completes each outstanding phase of the `full`
// barriers (an arrival for a stage that only its peer filled, the peer's bytes for one that
// only it filled) and waits for the copies; the peer stays until then.
struct PairBars {
  uint64_t *full, *empty, *tfull, *drain;
};
__device__ __forceinline__ void leave_pair(const PairBars& b, uint32_t nst, uint32_t nbuf, uint32_t bytes,
                                           const uint32_t* done, uint32_t rank, uint32_t total, uint32_t kblocks) {
  uint64_t* full = b.full;
  __syncthreads();
  cluster_sync();   // the leader has committed for the last time and its MMAs have retired
  if (threadIdx.x == 0) {
    const uint32_t nread = done[DONE_MMA], tiles = nread / kblocks;
    for (uint32_t i = nread > nst ? nread - nst : 0; i < nread; ++i) mbar_drain(&b.empty[i % nst], (i / nst) & 1);
    for (uint32_t i = tiles > nbuf ? tiles - nbuf : 0; i < tiles; ++i) mbar_drain(&b.tfull[i % nbuf], (i / nbuf) & 1);
    mbar_drain(b.drain, 0);
  }
  if (done[DONE_MMA] == total) return;
  const uint32_t n0 = done[DONE_FILL0], n1 = done[DONE_FILL1];
  if (rank == 0 && threadIdx.x == 0) {
    const uint32_t end = max(n0, n1);
    for (uint32_t i = end > nst ? end - nst : 0; i < end; ++i) {
      uint64_t* bar = &full[i % nst];
      if (i >= n0) mbar_expect(bar, bytes);
      if (i >= n1)
        asm volatile("mbarrier.complete_tx.relaxed.cluster.shared::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                     : "memory");
      mbar_drain(bar, (i / nst) & 1);
    }
  }
  __syncwarp();
  cluster_sync();
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GTHREADS, 1)
    k_mod_gemm(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const ModGemmArgs g) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + GSTAGES * GSTAGE_BYTES);
  uint64_t* full = bars;                               // leader: both CTAs' bytes of a stage
  uint64_t* empty = bars + GSTAGES;                    // each CTA: the stage's MMAs have retired
  uint64_t* tfull = bars + 2 * GSTAGES;                // each CTA: a tile's sums are in TMEM
  uint64_t* tempty = bars + 2 * GSTAGES + GBUF;        // leader: both CTAs have read them
  uint64_t* drain = bars + 2 * GSTAGES + 2 * GBUF;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * GSTAGES + 2 * GBUF + 1);
  uint32_t* done = tmem_slot + 1;                      // [DONE_SLOTS]
  volatile int* err = g.err;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  if (threadIdx.x == 0) {
    for (int s = 0; s < GSTAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < GBUF; ++b) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], 2 * GEPI);
    }
    mbar_init(drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  grid_enter();
  const uint32_t tmem = *tmem_slot;
  const int per = g.num_m * g.num_n, ntiles = per * NPL;
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      uint32_t nfilled = 0;
      for (int t = pair; t < ntiles && ok; t += npairs) {
        const int pl = t / per, mb = (t % per) % g.num_m, nb = (t % per) / g.num_m;
        for (int kb = 0; kb < g.kblocks && ok; ++kb) {
          ok = mbar_wait(&empty[stage], phase ^ 1, err, g.wait_cycles);
          if (!ok) break;
          uint8_t* base = smem + stage * GSTAGE_BYTES;
          if (rank == 0) mbar_expect(&full[stage], 2 * GSTAGE_BYTES);
          const uint32_t bar = leader_addr(&full[stage]);
          tma_load_pair(base, &mapA, bar, kb * GKB, mb * GT + (int)rank * HALF, pl);
          tma_load_pair(base + HALF * GKB, &mapB, bar, kb * GKB, nb * GT + (int)rank * HALF, pl);
          ++nfilled;
          if (++stage == GSTAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      publish(&done[DONE_FILL0 + rank], nfilled);
    }
  } else if (warp == 1) {
    if (rank == 0 && lane == 0) {
      int stage = 0, n = 0;
      uint32_t phase = 0, nread = 0;
      bool ok = true;
      for (int t = pair; t < ntiles && ok; t += npairs, ++n) {
        const int buf = n % GBUF;
        ok = mbar_wait(&tempty[buf], ((n / GBUF) & 1) ^ 1, err, g.wait_cycles);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int kb = 0; kb < g.kblocks && ok; ++kb) {
          ok = mbar_wait(&full[stage], phase, err, g.wait_cycles);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a0 = smem_u32(smem + stage * GSTAGE_BYTES);
          const uint64_t da = make_desc(a0), db = make_desc(a0 + HALF * GKB);
#pragma unroll
          for (int kk = 0; kk < GKB / 32; ++kk)
            mma_pair(tmem + (uint32_t)(buf * GT), da + (uint64_t)(kk * 2), db + (uint64_t)(kk * 2),
                     (kb == 0 && kk == 0) ? 0u : 1u);
          commit_pair(&empty[stage]);
          ++nread;
          if (++stage == GSTAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        commit_pair(&tfull[buf]);
      }
      commit_pair(drain);
      mbar_drain(drain, 0);
      publish(&done[DONE_MMA], nread);
    }
  } else {
    constexpr int ECOLS = GT / (GEPI / 4);   // columns of a warp
    const int q = warp & 3, h = (warp - 2) / 4;
    int n = 0;
    for (int t = pair; t < ntiles; t += npairs, ++n) {
      const int pl = t / per, mb = (t % per) % g.num_m, nb = (t % per) / g.num_m;
      const int mi = pl % NMOD;
      const int p = kTab.p[mi], wgt = kTab.wa_lo[mi], off = kTab.off_s[mi];
      const float inv = kTab.inv[mi];
      const uint32_t flip = pl < NRES ? 0x80808080u : 0u;   // residues are stored with an offset of 128
      const int buf = n % GBUF;
      if (!mbar_wait(&tfull[buf], (n / GBUF) & 1, err, g.wait_cycles)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int row = mb * GT + (int)rank * HALF + q * 32 + lane;
      uint8_t* orow = g.out + (int64_t)pl * g.M * g.ldo + (int64_t)row * 16;
#pragma unroll 1
      for (int ch = 0; ch < ECOLS / 32; ++ch) {
        uint32_t r[32];
        tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * GT + h * ECOLS + ch * 32), r);
        if (ch == ECOLS / 32 - 1) {
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0)
            // (not .release.cluster, which would wait for this warp's stores of the last chunk;
            // the fence above orders the reads of TMEM)
            asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(leader_addr(&tempty[buf])) : "memory");
        }
        const int col = nb * GT + h * ECOLS + ch * 32;
        if (row < g.M && col < g.ldo) {
          uint32_t w[8];
          if (pl < NRES) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              r[j] = (uint32_t)mod_byte(dp4a_us(r[j] ^ 0x80000000u, wgt, off), p, inv);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = mag_byte((int)r[j]);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) w[j] = pack4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]) ^ flip;
          uint8_t* o = orow + (int64_t)col * g.M;   // column block col / 16
          *reinterpret_cast<uint4*>(o) = make_uint4(w[0], w[1], w[2], w[3]);
          *reinterpret_cast<uint4*>(o + (int64_t)16 * g.M) = make_uint4(w[4], w[5], w[6], w[7]);
        }
      }
    }
  }
  // no CTA leaves, and no TMEM is released, while the pair's MMAs or copies are in flight
  const uint32_t mine = pair < ntiles ? (uint32_t)((ntiles - pair + npairs - 1) / npairs) : 0u;
  leave_pair(PairBars{full, empty, tfull, drain}, GSTAGES, GBUF, (uint32_t)GSTAGE_BYTES, done, rank,
             mine * (uint32_t)g.kblocks, (uint32_t)g.kblocks);
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem));
  }
}

// ---------------------------------------------------------------------------
// Reconstruction
// ---------------------------------------------------------------------------
struct ModJoinArgs {
  int M, N, K;
  int64_t ldo;
  const uint8_t* res;
  const int4 *ia, *ib;
  const int* err;       // set when a wait of the GEMMs (or of a product before) gave up
  double2 alpha, beta;
  double2* C;
  int64_t ldc;
};

template <int I>
__device__ __forceinline__ void join_modulus(unsigned wu, unsigned wv, unsigned (&x1)[4], unsigned (&y1)[4],
                                             double (&x2)[4], double (&y2)[4]) {
  constexpr unsigned re1 = kT.re1[I], im1 = kT.im1[I];
  constexpr double re2 = kT.re2[I], im2 = kT.im2[I];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const unsigned u = __byte_perm(wu, 0, 0x4440 + e), v = __byte_perm(wv, 0, 0x4440 + e);
    const unsigned sp = u + v, sm = u - v + 256u;
    x1[e] += sp * re1;
    y1[e] += sm * im1;
    x2[e] = fma(__hiloint2double(0x43300000, (int)sp) - 4503599627370496.0, re2, x2[e]);
    y2[e] = fma(__hiloint2double(0x43300000, (int)sm) - 4503599627370496.0, im2, y2[e]);
  }
}
template <int... I>
__device__ __forceinline__ void join_moduli(const unsigned (&wu)[NMOD], const unsigned (&wv)[NMOD], unsigned (&x1)[4],
                                            unsigned (&y1)[4], double (&x2)[4], double (&y2)[4],
                                            std::integer_sequence<int, I...>) {
  (join_modulus<I>(wu[I], wv[I], x1, y1, x2, y2), ...);
}

// The integer nearest zero that is w0 + 2^39 w1 + 2^78 w2 modulo P (|w| < 2^53), rounded once.
// It is below 2^116.1 by the operands' scales, so taking the multiple of P from w2 alone is
// safe.  The leading two pieces are added with their exact remainder; when the result is a
// double it comes out exactly.
__device__ __forceinline__ double crt_value(const double (&w)[3]) {
  const double q = rint(w[2] * kTab.inv_p2);
  const double h = fma(-q, kTab.p3[2], w[2]) * 0x1p39, m = fma(-q, kTab.p3[1], w[1]), l = fma(-q, kTab.p3[0], w[0]);
  const double s = h + m, b = s - h;
  const double r = (h - (s - b)) + (m - b);
  return fma(s, 0x1p39, fma(r, 0x1p39, l));
}
// The columns `which` of a thread's four (its bytes at src) from exact sums.  Products of whole
// numbers come here; three double multiply-adds per modulus and component where the fractions
// need one (146 us more for 6144 x 4096, were it done for all).
__device__ __noinline__ void exact_elements(const ModJoinArgs& g, int m0, int n0, unsigned which, double2 (*tile)[65]) {
  const int r = threadIdx.x >> 2, c4 = (threadIdx.x & 3) * 4;
  const uint8_t* src = g.res + (int64_t)n0 * g.M + (int64_t)(m0 + r) * 16 + c4;
  const int64_t plane = (int64_t)g.M * g.ldo;
  const int ea = g.ia[m0 + r].x;
#pragma unroll 1
  for (int e = 0; e < 4; ++e) {
    if (!(which >> e & 1)) continue;
    double x[3], y[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      x[k] = kTab.re3_0[k];
      y[k] = kTab.im3_0[k];
    }
#pragma unroll 4
    for (int i = 0; i < NMOD; ++i) {
      const int u = src[plane * i + e], v = src[plane * (NMOD + i) + e];
      const double sp = (double)(u + v), sm = (double)(u - v + 256);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        x[k] = fma(sp, kTab.re3[i][k], x[k]);
        y[k] = fma(sm, kTab.im3[i][k], y[k]);
      }
    }
    const int t = max(-(ea + g.ib[n0 + c4 + e].x), -2000), th = t / 2;
    const double s1 = pow2(th), s2 = pow2(t - th);
    tile[c4 + e][r] = make_double2(crt_value(x) * s1 * s2, crt_value(y) * s1 * s2);
  }
}

// Elements of a 64 x 16 tile that residues do not give to the accuracy of FP64, as plain FP64
// sums: `bad` marks those of this thread's four columns c4 .. c4 + 3 of row r.  All threads of
// the block call it.  A few elements take a warp each; from 32 on the block forms the whole
// tile on the FP64 tensor cores, K stages of 16 through shared memory.  An element's sum does
// not depend on timing.
constexpr int RD_K = 16, RD_FEW = 32;
__device__ __forceinline__ void dmma_8x8x4(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}
__device__ __noinline__ void fp64_elements(const ModOperand& a, const ModOperand& b, int M, int N, int K, int m0, int n0,
                                           unsigned bad, double2 (*tile)[65]) {
  __shared__ double2 as[RD_K][66], bs[RD_K][18];   // strides of 2 mod 8: fragment reads without bank conflicts
  __shared__ unsigned mask[64];                    // bits: columns of a row to be replaced
  __shared__ unsigned short list[RD_FEW];
  __shared__ int count;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r = tid >> 2, c4 = (tid & 3) * 4;
  if (tid == 0) count = 0;
  if (tid < 64) mask[tid] = 0u;
  __syncthreads();
  if (bad) {
    atomicOr(&mask[r], bad << c4);
    int at = atomicAdd(&count, __popc(bad));
    for (int e = 0; e < 4; ++e)
      if (bad >> e & 1) {
        if (at < RD_FEW) list[at] = (unsigned short)(r << 4 | (c4 + e));
        ++at;
      }
  }
  __syncthreads();
  const int n = count;
  if (n <= RD_FEW) {
    for (int i = warp; i < n; i += 8) {
      const int er = list[i] >> 4, ec = list[i] & 15;
      double2 s = make_double2(0.0, 0.0);
#pragma unroll 4
      for (int k = lane; k < K; k += 32) {
        const double2 x = load_elem(a, m0 + er, k), y = load_elem(b, n0 + ec, k);
        s.x = fma(-x.y, y.y, fma(x.x, y.x, s.x));
        s.y = fma(x.y, y.x, fma(x.x, y.y, s.y));
      }
#pragma unroll
      for (int d = 16; d >= 1; d >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, d);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, d);
      }
      if (lane == 0) tile[ec][er] = s;
    }
    __syncthreads();
    return;
  }
  // a warp's 8 rows x 16 columns, in the order of sums of the FP64 tensor-core kernel
  const int ak = a.kcontig ? tid & 15 : tid >> 6, al = a.kcontig ? tid >> 4 : tid & 63;
  const int bk = b.kcontig ? tid & 15 : tid >> 4, bl = b.kcontig ? tid >> 4 : tid & 15;
  const int dk = a.kcontig ? 0 : 4, dl = a.kcontig ? 16 : 0;
  double2 pa[4], pb;
  auto fetch = [&](int k0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = k0 + ak + dk * q, l = m0 + al + dl * q;
      pa[q] = k < K && l < M ? load_elem(a, l, k) : make_double2(0.0, 0.0);
    }
    pb = k0 + bk < K && n0 + bl < N ? load_elem(b, n0 + bl, k0 + bk) : make_double2(0.0, 0.0);
  };
  double re[2][2] = {}, im[2][2] = {};
  const int fr = lane >> 2, fk = lane & 3;
  fetch(0);
  for (int k0 = 0; k0 < K; k0 += RD_K) {
#pragma unroll
    for (int q = 0; q < 4; ++q) as[ak + dk * q][al + dl * q] = pa[q];
    bs[bk][bl] = pb;
    __syncthreads();
    if (k0 + RD_K < K) fetch(k0 + RD_K);
#pragma unroll
    for (int kb = 0; kb < RD_K; kb += 4) {
      const double2 x = as[kb + fk][8 * warp + fr];
      const double2 y[2] = {bs[kb + fk][fr], bs[kb + fk][8 + fr]};
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        dmma_8x8x4(re[j], x.x, y[j].x);
        dmma_8x8x4(im[j], x.x, y[j].y);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        dmma_8x8x4(re[j], -x.y, y[j].y);
        dmma_8x8x4(im[j], x.y, y[j].x);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int row = 8 * warp + fr, col = 8 * j + 2 * fk + e;
      if (mask[row] >> col & 1) tile[col][row] = make_double2(re[j][e], im[j][e]);
    }
  __syncthreads();
}

// A block joins a 64 x 16 tile of C: a thread reads 4 columns of a row from the planes
// and sums the CRT fractions of its 4 elements, modulo 1 in 32-bit integers for their
// leading bits, in FP64 below; the tile goes through shared memory so that C is written
// along its columns.  The stored bytes are residues + 128, so u + v and u - v + 256 exceed
// the sums meant by 256 each, which the accumulators' starting values take out.  Per
// element: 32 integer and 32 double multiply-adds, 32 conversions by exponent trick and
// 49 bytes of memory traffic.
template <bool BETA>
__global__ void __launch_bounds__(256, 3)
    k_mod_join(const __grid_constant__ ModJoinArgs g, const __grid_constant__ ModOperand a,
               const __grid_constant__ ModOperand b) {
  grid_enter();
  __shared__ double2 tile[16][65];
  const int tid = threadIdx.x;
  const int r = tid >> 2, c4 = (tid & 3) * 4;
  const int m0 = blockIdx.x * 64, n0 = blockIdx.y * 16;
  const int row = m0 + r;
  // a product that gave up leaves NaNs, for callers that wait without asking for the status
  const bool gave_up = *(const volatile int*)g.err != 0;
  unsigned bad = 0, whole = 0;   // columns to be summed in FP64, columns of whole numbers
  if (row < g.M) {
    const uint8_t* src = g.res + (int64_t)n0 * g.M + (int64_t)row * 16 + c4;
    const int64_t plane = (int64_t)g.M * g.ldo;
    constexpr unsigned re1_0 = kT.re1_0, im1_0 = kT.im1_0;
    constexpr double re2_0 = kT.re2_0, im2_0 = kT.im2_0, P = kT.P;
    unsigned x1[4], y1[4];
    double x2[4], y2[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      x1[e] = re1_0;
      y1[e] = im1_0;
      x2[e] = re2_0;
      y2[e] = im2_0;
    }
    // all 32 loads in flight before the first use
    unsigned wu[NMOD], wv[NMOD];
#pragma unroll
    for (int i = 0; i < NMOD; ++i) {
      wu[i] = __ldcs(reinterpret_cast<const unsigned*>(src + plane * i));
      wv[i] = __ldcs(reinterpret_cast<const unsigned*>(src + plane * (NMOD + i)));
    }
    const unsigned wm = __ldcs(reinterpret_cast<const unsigned*>(src + plane * NRES));
    join_moduli(wu, wv, x1, y1, x2, y2, std::make_integer_sequence<int, NMOD>{});
    const int4 ia = g.ia[row];
    const int ea = ia.x, na = ia.y;
    const float limit = mag_limit(g.K);
    unsigned one = 0;   // columns whose sum has one term
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int4 ib = g.ib[min(n0 + c4 + e, g.N - 1)];
      const int eb = ib.x, nb = ib.y;
      const bool finite = ea != EXP_NONFINITE && eb != EXP_NONFINITE, single = na == 1 || nb == 1;
      if (finite && !single && ia.w && ib.w) whole |= 1u << e;
      else if (!finite || (na > 0 && nb > 0 && !single && !mag_shows(__byte_perm(wm, 0, 0x4440 + e), na + nb - g.K, limit)))
        bad |= 1u << e;
      else if (single) one |= 1u << e;
      const int t = finite ? max(-(ea + eb), -2000) : 0, th = t / 2;
      const double s1 = pow2(th), s2 = pow2(t - th);
      tile[c4 + e][r] = make_double2(fma((double)(int)x1[e], 0x1p-32, x2[e]) * P * s1 * s2,
                                     fma((double)(int)y1[e], 0x1p-32, y2[e]) * P * s1 * s2);
    }
    const int live = min(4, g.N - n0 - c4);   // (columns past the last one were read in its place)
    const unsigned in = live > 0 ? (1u << live) - 1u : 0u;
    bad &= gave_up ? 0u : in;
    one &= in;
    whole &= in;
    if (one) {
      double2 x[4], y[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int col = min(n0 + c4 + e, g.N - 1), k = na == 1 ? ia.z : g.ib[col].z;
        x[e] = load_elem(a, row, k);
        y[e] = load_elem(b, col, k);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (one >> e & 1)
          tile[c4 + e][r] = make_double2(fma(-x[e].y, y[e].y, x[e].x * y[e].x), fma(x[e].y, y[e].x, x[e].x * y[e].y));
    }
  }
  if (whole) exact_elements(g, m0, n0, whole, tile);
  if (__syncthreads_or(bad)) fp64_elements(a, b, g.M, g.N, g.K, m0, n0, bad, tile);
  const int tr = tid & 63;
  if (m0 + tr >= g.M) return;
#pragma unroll
  for (int c = tid >> 6; c < 16; c += 4) {
    if (n0 + c >= g.N) break;
    const double2 v = tile[c][tr];
    double2 o = make_double2(g.alpha.x * v.x - g.alpha.y * v.y, g.alpha.x * v.y + g.alpha.y * v.x);
    if (gave_up) o.x = o.y = __longlong_as_double(0x7ff8000000000000ll);
    double2* p = g.C + (m0 + tr) + g.ldc * (int64_t)(n0 + c);
    if (BETA) {
      const double2 z = *p;
      o.x += g.beta.x * z.x - g.beta.y * z.y;
      o.y += g.beta.x * z.y + g.beta.y * z.x;
    }
    *p = o;
  }
}

int64_t up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

}  // namespace

bool zgemm_modular(Context* ctx, Op opA, Op opB, int M, int N, int K, cplx alpha, const dcplx* A, int64_t lda,
                   const dcplx* B, int64_t ldb, cplx beta, dcplx* C, int64_t ldc, double t_fp64) {
  // int32 sums of K products of residues <= 122 stay below 2^31; planes of 64 MiB at most
  if (M < 64 || N < 64 || K < 64 || K > 131072) return false;
  // Modelled times in us, fitted to both engines on a B200: 16 for the four launches, the
  // operands' and outputs' elements, and the waves of tiles (2.7 of epilogue at least).  The
  // lines cross near 0.6 GFLOP for square products (events around one call, which add some 8:
  // 448 x 448 x 448 taken by the FP64 tensor cores in 36, 512 x 512 x 512 41 here against 50
  // there; 502 x 251 x 1255 47 against 64, 1255 x 502 x 251 49 against 70, 300 x 300 x 1200 48
  // against 47) and far later for a short K, whose outputs dominate (4096 x 960 x 64: 165
  // against 88).
  const int64_t tiles = (int64_t)((M + GT - 1) / GT) * ((N + GT - 1) / GT) * NPL, npair = ctx->num_sms / 2;
  const double t_here = 16.0 + 15.4e-6 * ((double)M + N) * K + 14.8e-6 * M * (double)N +
                        (double)((tiles + npair - 1) / npair) * std::max(2.7, 3.2 / 1024 * K);
  if (t_here > 0.9 * t_fp64) return false;
  if (ctx->capturing()) return false;   // its error flag needs a synchronisation
  const int64_t Kp = up(K, GKB);
  const size_t pa = (size_t)NPL * M * Kp, pb = (size_t)NPL * N * Kp;
  if (pa > ((size_t)NPL << 26) || pb > ((size_t)NPL << 26)) return false;
  // the output's planes of one column panel within 32 MiB each (panels that stay in L2 were no
  // faster: 1.47 ms against 1.21 ms for 6144 x 4096 x 1024, the GEMMs' last waves)
  int64_t np = ((int64_t)1 << 25) / M / GT * GT;
  if (np < GT) return false;
  np = std::min<int64_t>(np, N);
  const int64_t ldo = up(np, 32);
  const size_t pc = (size_t)NPL * M * ldo;
  const int nchunk = std::max(1, std::min(16, K / 64));
  const size_t tail = (size_t)(M + N) * (nchunk * (2 * sizeof(double) + 3 * sizeof(int)) + sizeof(int4));
  auto at = [](size_t x) { return (x + 1023) / 1024 * 1024; };
  uint8_t* base = static_cast<uint8_t*>(ctx->optional_buf("gemm_modular", at(pa) + at(pb) + at(pc) + tail + 4096));
  if (!base) return false;
  int8_t* planesA = reinterpret_cast<int8_t*>(base);
  int8_t* planesB = reinterpret_cast<int8_t*>(base + at(pa));
  uint8_t* res = base + at(pa) + at(pb);
  int4* info = reinterpret_cast<int4*>(res + at(pc));
  double* part = reinterpret_cast<double*>(info + M + N);
  int* count = reinterpret_cast<int*>(part + (size_t)(M + N) * 2 * nchunk);

  ModOperand a{}, b{};
  a.X = A;
  a.ld = lda;
  a.lines = M;
  a.kcontig = opA != OP_N;
  a.conj = opA == OP_C;
  a.planes = planesA;
  a.part = part;
  a.count = count;
  a.info = info;
  b.X = B;
  b.ld = ldb;
  b.lines = N;
  b.kcontig = opB == OP_N;
  b.conj = opB == OP_C;
  b.planes = planesB;
  b.part = part + (size_t)M * 2 * nchunk;
  b.count = count + (size_t)M * 3 * nchunk;
  b.info = info + M;
  for (ModOperand* o : {&a, &b}) {
    o->K = K;
    o->Kp = Kp;
    o->nchunk = nchunk;
    o->kchunk = (K + nchunk - 1) / nchunk;
    o->nblocks_norm = (o->lines + (o->kcontig ? 31 : 63)) / (o->kcontig ? 32 : 64) * nchunk;
    o->nblocks_split = (int)(Kp / 64) * ((o->lines + SPL_LINES - 1) / SPL_LINES);
  }
  ScopedTimer tm(ctx, "zgemm_modular", 8.0 * M * (double)N * K);
  launch_kernel(ctx, k_mod_norms, a.nblocks_norm + b.nblocks_norm, 256, 0, a, b);
  launch_kernel(ctx, k_mod_split, a.nblocks_split + b.nblocks_split, SPL_NT, 0, a, b);
  static DeviceOnce attr;
  attr.run(ctx->device, [] {
    IMPS_CUDA(cudaFuncSetAttribute(k_mod_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, GSMEM));
  });
  const CUtensorMap mapA = plane_map(planesA, Kp, M, NPL, GKB, HALF);
  ctx->n_kernels += 2;
  for (int64_t n0 = 0; n0 < N; n0 += np) {
    const int nn = (int)std::min<int64_t>(np, N - n0);
    const CUtensorMap mapB = plane_map(planesB + n0 * Kp, Kp, nn, NPL, GKB, HALF, (int64_t)N * Kp);
    ModGemmArgs g;
    g.num_m = (M + GT - 1) / GT;
    g.num_n = (nn + GT - 1) / GT;
    g.kblocks = (int)(Kp / GKB);
    g.M = M;
    g.ldo = ldo;
    g.out = res;
    g.err = ctx->err_dev;
    g.wait_cycles = ctx->wait_cycles;
    const int pairs = std::min(g.num_m * g.num_n * NPL, ctx->num_sms / 2);
    launch_kernel(ctx, k_mod_gemm, 2 * pairs, GTHREADS, GSMEM, mapA, mapB, g);
    ModJoinArgs j;
    j.M = M;
    j.N = nn;
    j.K = K;
    j.ldo = ldo;
    j.res = res;
    j.ia = a.info;
    j.ib = b.info + n0;
    j.err = ctx->err_dev;
    j.alpha = make_double2(alpha.real(), alpha.imag());
    j.beta = make_double2(beta.real(), beta.imag());
    j.C = C + ldc * n0;
    j.ldc = ldc;
    ModOperand bj = b;
    bj.X = b.kcontig ? B + ldb * n0 : B + n0;
    const dim3 grid((M + 63) / 64, (nn + 15) / 16);
    if (beta != cplx(0.0, 0.0)) launch_kernel(ctx, k_mod_join<true>, grid, 256, 0, j, a, bj);
    else launch_kernel(ctx, k_mod_join<false>, grid, 256, 0, j, a, bj);
    ctx->n_kernels += 2;
  }
  IMPS_CUDA(cudaPeekAtLastError());
  ctx->n_gemm++;
  ctx->err_later = true;   // the bounded waits' flag is read at the next synchronisation
  return true;
}

}  // namespace imps
