// gsks_sliced.cuh -- shared pieces of the FP64 form on the tensor cores
// (gsks_sliced.cu): the operand format, the 2^-y evaluation in integers and
// the FP64 kernel functions on assembled distances.
#pragma once
#include <cstddef>
#include <cstdint>
#include "gsks_internal.cuh"

namespace gsks {
namespace sliced {

constexpr int BM = 128;              // targets per tile (TMEM lanes)
constexpr int BN = 32;               // sources per tile
constexpr int NS = 6;                // slices per coordinate
constexpr int SB = 9;                // bits per slice (balanced digits, |d| <= 256)
constexpr int KRES = 64;             // largest padded k of the target-resident layout, and the k-run of one accumulation
constexpr int KST = 32;              // k-chunk of one streamed stage beyond it
constexpr int KMAX = 1024;           // largest padded k
constexpr int RMAX = 4;              // right-hand sides of one sweep
constexpr int ELIM = 450;            // largest magnitude of a sliced point's exponent
// A point's exponent word where x.y goes through FP64 (dot_cols): the exponent plus
// EBIAS (twice of which leaves a double's high word unchanged), what the point's digits
// do not promise for its inner products (held_bits), and the class of its length.
constexpr int EBIAS = 2048;
constexpr int EMASK = 12, EMASK_K = 8;  // up to 8 coordinates: a bit for each large one
constexpr int NOT_COARSE = 1 << 20, NOT_LARGE = 1 << 21, NOT_DENSE = 1 << 22;
constexpr int NOT_HELD = NOT_COARSE | NOT_LARGE | NOT_DENSE;   // also of a point without digits
constexpr int NORM_GIVEN = 1 << 23;     // the point's norm, as given, is not that of its coordinates
constexpr int ECLASS = 24;
constexpr int ETAB = 2048;           // entries of the 2^-f table

// Metadata of a source tile, one block of shared memory: the norms (FP64, or
// the integers of the fixed-point Gaussian), bandwidths, exponents,
// what the digits of all its points do not promise (NOT_HELD's bits), and the weight columns.
struct ColMeta {
  double bb[BN];
  uint64_t hj[BN];      // FP64 bits, or (fixed-point form) the mantissa
  int e[BN];
  int flag;
  int pad[3];
  double w[RMAX][BN];
};
__host__ __device__ constexpr size_t colmeta_bytes(int nr) { return offsetof(ColMeta, w) + (size_t)nr * BN * 8; }
static_assert(colmeta_bytes(1) % 16 == 0 && sizeof(ColMeta) % 16 == 0, "ColMeta is copied by the bulk-copy engine");

// ---------------------------------------------------------------------------
// 2^-(i / ETAB) in units of 2^-63, i = 0 .. ETAB - 1, plus EXP_BIAS: half of 2^-53 for
// exp2_neg's last shift and the mean of its floors.  (In units of 2^-64 the first entry has
// no room for the half: values just below 1, all of a wide Gaussian's, were 0.6 2^-53 too
// small in the mean.)  Products of the eleven constants 2^(-2^b / ETAB) in 64-bit fixed
// point, evaluated by the compiler.
constexpr uint64_t mulhi64c(uint64_t a, uint64_t b)
{
  const uint64_t al = a & 0xffffffffu, ah = a >> 32, bl = b & 0xffffffffu, bh = b >> 32;
  const uint64_t m = ah * bl + ((al * bl) >> 32);
  const uint64_t n = al * bh + (m & 0xffffffffu);
  return ah * bh + (m >> 32) + (n >> 32);
}
constexpr uint64_t EXP_BIAS = 640;
struct ExpTable {
  uint64_t v[ETAB];
  constexpr ExpTable() : v()
  {
    constexpr uint64_t c[11] = {0xffe9d2b2f7db2756, 0xffd3a751c0f7e10c, 0xffa756521c8daed2, 0xff4ecb59511ec8a5,
                                0xfe9e115c7b8f884c, 0xfd3e0c0cf486c175, 0xfa83b2db722a033a, 0xf5257d152486cc2c,
                                0xeac0c6e7dd24392f, 0xd744fccad69d6af4, 0xb504f333f9de6484};
    v[0] = (1ull << 63) + EXP_BIAS;
    for (int i = 1; i < ETAB; i++) {
      uint64_t p = 0;
      bool first = true;
      for (int b = 0; b < 11; b++)
        if (i >> b & 1) {
          p = first ? c[b] : mulhi64c(p, c[b]);
          first = false;
        }
      v[i] = (p >> 1) + EXP_BIAS;
    }
  }
};

// a b + c with a 32 x 32 -> 64 bit product: one instruction (64 per SM cycle,
// the rate of a 32-bit multiply).
__device__ __forceinline__ uint64_t madw(uint32_t a, uint32_t b, uint64_t c)
{
  uint64_t d;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}
__device__ __forceinline__ long long madws(int a, int b, long long c)
{
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint32_t mulhi(uint32_t a, uint32_t b)
{
  return (uint32_t)(madw(a, b, 0) >> 32);
}

// Two consecutive 64-bit words of shared memory (16-byte aligned address).
__device__ __forceinline__ void lds2(uint32_t addr, long long &a, long long &b)
{
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr));
}
__device__ __forceinline__ void lds2(uint32_t addr, double &a, double &b)
{
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(a), "=d"(b) : "r"(addr));
}

__device__ __forceinline__ void lds1(uint32_t addr, double &a)
{
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(a) : "r"(addr));
}

// 2^-y for y = z 2^-F, |z| >= 2^32, |y| < 1021, to about one unit in the last place:
// y = n + (i + phi) / 2048, 2^-y = 2^-n T[i] (1 - P), P = 1 - 2^(-phi / 2048)
// (the table-driven scheme of P. T. P. Tang, ACM TOMS 15 (1989), in integers).
// FP64 instructions issue at 1/32 of the integer rate here (2 against 64 per
// SM cycle, measured): an FP64 exponential of about 18 of them takes 9 SM
// cycles a value, these about 27 integer ones less than half a cycle.
//   phi = f 2^-32 + flo 2^(11 - F); P in units of 2^-75: ln2 (f 2^32 + ...) with
//   ln2 2^32 rounded up (2977044472), less q in units of 2^-55: z^2/2 - z^3/6 +
//   z^4/24, z = ln2 phi / 2048, and the excess of the first constant; the
//   fourth power replaced by its best cubic on [0, 1] (error 2^-7 of 20 2^-55).
// Against 50 decimals (the integer steps run on the host, F = 43 .. 62, y up to 1000): at
// most 1.4 2^-53 relative, rms 0.43 2^-53 (correctly rounded: 1 and 0.43); below 2^-11 rms
// 0.30, mean 0.03 or less.  y = 0 gives 1.
struct ExpFrame {
  int s;                  // F - 43, 0 .. 19
  uint32_t mask, mul;     // 2^s - 1, ln2 2^(32 - s) (flo in units of P)
  uint32_t tab;           // shared-memory address of the table
  uint32_t half;          // half a unit of z, in units of P, where z was rounded down (else 0)
};
__device__ __forceinline__ ExpFrame exp_frame(int F, uint32_t tab)
{
  ExpFrame f;
  f.s = F - 43;
  f.mask = (1u << f.s) - 1u;
  f.mul = (2977044472u >> f.s) + (f.s ? (2977044472u >> (f.s - 1)) & 1u : 0u);
  f.tab = tab;
  f.half = 0;
  return f;
}
// (The table's contents never change, so its load may move freely.)
__device__ __forceinline__ double exp2_neg(uint64_t z, const ExpFrame &E)
{
  const uint32_t hi = (uint32_t)(z >> 32), lo = (uint32_t)z;
  const int v = (int)hi >> E.s;
  const uint32_t f = __funnelshift_r(lo, hi, E.s);    // v = n 2048 + i, phi's upper 32 bits
  uint64_t t;
  asm("ld.shared.u64 %0, [%1];" : "=l"(t) : "r"(E.tab + (v & (ETAB - 1)) * 8));
  const uint64_t lin = madw(lo & E.mask, E.mul, madw(f, 2977044472u, E.half));
  const uint32_t q = mulhi(f, mulhi(f, 2063529957u - mulhi(f, 232762u)) + 744u);
  const uint64_t p = (uint64_t)madws((int)q, -(1 << 20), (long long)lin) >> 11;   // P in units of 2^-64
  const uint32_t th = (uint32_t)(t >> 32), tl = (uint32_t)t, ph = (uint32_t)(p >> 32), pl = (uint32_t)p;
  const uint64_t s = madw(th, ph, 0) + mulhi(th, pl) + mulhi(tl, ph);      // T P, units of 2^-63
  const uint64_t m = (t - s) >> 10;                                        // [2^52, 2^53], units of 2^-53
  return __hiloint2double((int)((uint32_t)(m >> 32) + (1021u << 20)) - (v >> 11) * (1 << 20), (int)(uint32_t)m);
}

// High 64 bits of a 64 x 64 bit product, less at most 2 units (three of the four
// partial products).
__device__ __forceinline__ uint64_t mulhi64(uint64_t a, uint64_t b)
{
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
  return madw(ah, bh, 0) + mulhi(ah, bl) + mulhi(al, bh);
}

// d^-(P / 2) for d = D 2^-F, D >= 2^32, as 2^-y, y = (P / 2) log2 d, in integers:
// D = m 2^lz', m in [1, 2) 2^63; j = 2048 log2 m to the nearest integer from the
// SFU's logarithm; r = m T[j] - 1 (T of exp2_neg: a power of two of j / 2048, so
// its logarithm needs no table), |r| < 2^-12.4; log2 d = E + j / 2048 + log2(1 +
// r), ln(1 + r) = r - r^2 (1/2 - r / 3 + r^2 / 4).
// (The general pow, or binary powering with its division, takes 16 to 20 FP64
// instructions, 8 to 10 SM cycles a value; this about 35 integer ones and
// exp2_neg.)  The error of y is about Q 2^-55, Q = P log2(e) / 2, to be compared
// with the distance's own: P / 2 times its rounding, 2^-53 (|x|^2 + |y|^2) / d2.
struct PowFrame {
  int p8;                 // P 2^8: y's part from E + j / 2048, in units of 2^-52
  uint32_t qh, ql;        // Q 2^56 (P <= 128: qh below 2^31)
  int pad;
};
// E: exp_frame_floor(52).  ok: y in (-1000, 1000).
__device__ __forceinline__ double pow_neg_half(uint64_t D, int F, const PowFrame &Q, const ExpFrame &E, bool &ok)
{
  const int lz = __clz((int)(D >> 32));
  const uint64_t m = D << lz;
  const uint32_t mh = (uint32_t)(m >> 32);
  float l;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(__uint_as_float(0x3f800000u | ((mh >> 8) & 0x7fffffu))));
  const int j = __float_as_int(fmaf(l, 2048.0f, 12582912.0f)) - 0x4B400000;       // 0 .. 2048
  const int J = (63 - F - lz) * 2048 + j;
  uint64_t t;
  asm("ld.shared.u64 %0, [%1];" : "=l"(t) : "r"(E.tab + (j & (ETAB - 1)) * 8));
  t = (j & (ETAB - 1)) ? 2 * (t - EXP_BIAS) - 225 : ~0ull;   // units of 2^-64 (225: the mean of the floors of r)
  // j = 2048: T[0] / 2, m just below 2
  const uint64_t pr = mulhi64(m, j == ETAB ? t >> 1 : t);                         // (1 + r) 2^63
  const long long r = (long long)(pr ^ 0x8000000000000000ull);
  const int rs = (int)(r >> 20);                                                  // units of 2^-43
  const uint32_t r2 = (uint32_t)(madws(rs, rs, 0) >> 32);                         // 2^-54
  const uint32_t c = (uint32_t)(madws(rs, -349525, (long long)1 << 62) >> 32) + (r2 >> 25);   // 1/2 - r / 3 + r^2 / 4, 2^-31
  const long long u = r - (long long)(madw(r2, c, 0) >> 22);
  const long long qu = madws((int)(u >> 32), (int)Q.qh, (long long)mulhi((uint32_t)u, Q.qh)) +
                       (madws((int)(u >> 32), (int)(Q.ql >> 1), 0) >> 31);        // Q u, units of 2^-55
  const long long y = (qu >> 3) + ((long long)((uint64_t)(uint32_t)(J * Q.p8) << 32));   // 2^-52
  ok = (uint32_t)((int)(y >> 32) + (1000 << 20)) < (2000u << 20);
  return exp2_neg((uint64_t)y, E);
}

// 2^-y outside exp2_neg's range (y negative, beyond 1021, or no number).
__device__ __noinline__ inline double exp2_neg_wide(double y) { return exp2(-y); }

constexpr uint32_t EXP_END = 1021u << 21;   // high word of 1021 2^53

// 2^-y for an FP64 y (given as y 2^53).
__device__ __forceinline__ double exp2_neg64(double y53, uint32_t tab)
{
  const long long z = __double2ll_rn(y53);
  if ((uint32_t)(z >> 32) - 1u >= EXP_END - 1u) {          // y below 2^-21 (or negative), or 1021 and more
    // y above 1088 (high word of 1088 2^53): 0 in FP64 as well
    if ((uint32_t)(__double2hiint(y53) - 0x43e10000) < 0x7ff00001u - 0x43e10000u) return 0.0;
    return exp2_neg_wide(y53 * 0x1p-53);
  }
  return exp2_neg((uint64_t)z, ExpFrame{10, 1023u, 2907270u, tab, 0});
}

// exp2_neg for y up to 1088 (deep: y is 1021 or more): beyond 1021 the value is formed
// 2^512 too large and rounded into the subnormal range by one multiplication.
__device__ __forceinline__ double exp2_neg_deep(uint64_t z, bool deep, const ExpFrame &E)
{
  double v = exp2_neg(deep ? z - ((uint64_t)512 << (E.s + 43)) : z, E);
  if (deep) v *= 0x1p-512;
  return v;
}

// 2^-y for y = D 2^-F h_i h_j with the (positive) factors as 64-bit mantissas (Mi,
// Mj, leading bit set) and the sum ex of their exponents (value = M 2^(ex - 63)):
// D normalised, two products, one shift.  zh: the high word of y 2^53, saturated
// (the value holds for zh in [1, 1088 2^21)).  E: exp_frame_floor(53).
__device__ __forceinline__ double exp2_neg_scaled(uint64_t D, int F, uint64_t Mi, uint64_t Mj, int ex, const ExpFrame &E,
                                                  uint32_t &zh)
{
  const int lz = __clzll((long long)D);
  const uint64_t t = mulhi64(mulhi64(D << lz, Mi), Mj);   // in [2^61, 2^64)
  const int s = F + lz - ex - 55;                          // y 2^53 = t 2^-s
  const uint64_t z = s < 0 ? t << 1 : t >> min(s, 63);     // (s < 0: y at least 512)
  zh = s < -1 || (s < 0 && (t >> 63)) ? 0xffffffffu : (uint32_t)(z >> 32);
  return exp2_neg_deep(z, zh >= 1021u << 21, E);
}
// Frames of a z rounded down (pow_neg_half 52, exp2_neg_scaled 53): its mean error, half a
// unit, is taken out (values were 0.7 2^-53 too large in the mean).
__device__ __forceinline__ ExpFrame exp_frame_floor(int F, uint32_t tab)
{
  return F == 52 ? ExpFrame{9, 511u, 5814540u, tab, 2907270u} : ExpFrame{10, 1023u, 2907270u, tab, 1453635u};
}

// (double)w: the conversion instruction issues to the FP64 pipe (2 per SM cycle),
// these about a dozen integer ones take a third of its time.  Rounds to nearest,
// ties away.
__device__ __forceinline__ double to_double(long long w)
{
  const uint64_t a = (uint64_t)(w < 0 ? -w : w);
  const int lz = __clzll((long long)a);
  const uint64_t m = ((a << (lz & 63)) >> 1) + 512u;        // [2^62, 2^63] + half of 2^-52
  const uint32_t hi = (uint32_t)(m >> 42) + ((1085u - (uint32_t)lz) << 20);
  const uint32_t sg = (uint32_t)(w >> 32) & 0x80000000u;
  return a ? __hiloint2double((int)(hi + sg), (int)(uint32_t)(m >> 10)) : 0.0;
}

// v^p, p = 2, 3 or 4, by 64-bit products of mantissas (an FP64 product issues at 2
// per SM cycle; these three take about 14 to 20 integer instructions), to about
// half a unit more than correct rounding.  ok: v^p lies well inside the normal
// range (else the value does not hold).
template <int P>
__device__ __forceinline__ double pow_int(double v, bool &ok)
{
  const uint64_t b = (uint64_t)__double_as_longlong(v);
  const int e = (int)(b >> 52 & 0x7ff) - 1023;
  ok = (uint32_t)(e + 200) < 400u;
  const uint64_t m = (b | 0x10000000000000ull) << 11;       // [1, 2) 2^63
  uint64_t q = mulhi64(m, m);                               // [1, 4) 2^62
  int up = 1;                                               // q = value 2^(63 - up)
  if (P == 3) { q = mulhi64(q, m); up = 2; }
  if (P == 4) { q = mulhi64(q, q); up = 3; }
  const int lz = __clz((int)(q >> 32));                     // 0 .. up
  const uint64_t r = ((q << lz) >> 1) + 512u;
  const uint32_t hi = (uint32_t)(r >> 42) + (uint32_t)(P * e + up - lz + 1022) * (1u << 20);
  const uint32_t sg = P == 3 ? (uint32_t)(b >> 32) & 0x80000000u : 0u;
  return __hiloint2double((int)(hi + sg), (int)(uint32_t)(r >> 10));
}

}  // namespace sliced
}  // namespace gsks
