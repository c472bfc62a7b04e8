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
constexpr int EFLAG = 1 << 20;       // exponent of a point whose inner products are formed directly
constexpr int ELIM = 450;            // largest magnitude of a sliced point's exponent
constexpr int ETAB = 2048;           // entries of the 2^-f table

// Metadata of a source tile, one block of shared memory: the norms (FP64, or
// the integers of the fixed-point Gaussian), bandwidths, exponents, whether the
// tile holds a point with EFLAG, and the weight columns.
struct ColMeta {
  double bb[BN];
  double hj[BN];
  int e[BN];
  int flag;
  int pad[3];
  double w[RMAX][BN];
};
__host__ __device__ constexpr size_t colmeta_bytes(int nr) { return offsetof(ColMeta, w) + (size_t)nr * BN * 8; }
static_assert(colmeta_bytes(1) % 16 == 0 && sizeof(ColMeta) % 16 == 0, "ColMeta is copied by the bulk-copy engine");

// ---------------------------------------------------------------------------
// 2^-(i / ETAB) in units of 2^-64, i = 0 .. ETAB - 1 (the first one unit short
// of 1), plus 1300: half of 2^-53 for exp2_neg's last shift and the mean of its
// floors.  Products of the eleven constants 2^(-2^b / ETAB) in 64-bit fixed point,
// evaluated by the compiler.
constexpr uint64_t mulhi64c(uint64_t a, uint64_t b)
{
  const uint64_t al = a & 0xffffffffu, ah = a >> 32, bl = b & 0xffffffffu, bh = b >> 32;
  const uint64_t m = ah * bl + ((al * bl) >> 32);
  const uint64_t n = al * bh + (m & 0xffffffffu);
  return ah * bh + (m >> 32) + (n >> 32);
}
struct ExpTable {
  uint64_t v[ETAB];
  constexpr ExpTable() : v()
  {
    constexpr uint64_t c[11] = {0xffe9d2b2f7db2756, 0xffd3a751c0f7e10c, 0xffa756521c8daed2, 0xff4ecb59511ec8a5,
                                0xfe9e115c7b8f884c, 0xfd3e0c0cf486c175, 0xfa83b2db722a033a, 0xf5257d152486cc2c,
                                0xeac0c6e7dd24392f, 0xd744fccad69d6af4, 0xb504f333f9de6484};
    v[0] = ~0ull;
    for (int i = 1; i < ETAB; i++) {
      uint64_t p = 0;
      bool first = true;
      for (int b = 0; b < 11; b++)
        if (i >> b & 1) {
          p = first ? c[b] : mulhi64c(p, c[b]);
          first = false;
        }
      v[i] = p + 1300;
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

// 2^-y for y = z 2^-F, 2^-21 <= y < 1021, to about one unit in the last place:
// y = n + (i + phi) / 2048, 2^-y = 2^-n T[i] (1 - P), P = 1 - 2^(-phi / 2048)
// (the table-driven scheme of P. T. P. Tang, ACM TOMS 15 (1989), in integers).
// FP64 instructions issue at 1/32 of the integer rate here (2 against 64 per
// SM cycle, measured): an FP64 exponential of about 18 of them takes 9 SM
// cycles a value, these about 27 integer ones less than half a cycle.
//   phi = f 2^-32 + flo 2^(11 - F); P in units of 2^-75: ln2 (f 2^32 + ...) with
//   ln2 2^32 rounded up (2977044472), less q in units of 2^-55: z^2/2 - z^3/6 +
//   z^4/24, z = ln2 phi / 2048, and the excess of the first constant; the
//   fourth power replaced by its best cubic on [0, 1] (error 2^-7 of 20 2^-55).
// Against exp2l over y in [2^-21, 1000]: at most 1.6 2^-53 relative, rms 0.45
// 2^-53 (correctly rounded: 1 and 0.43).  y = 0 gives 1 - 2^-53: callers treat
// it apart.
struct ExpFrame {
  int s;                  // F - 43, 0 .. 19
  uint32_t mask, mul;     // 2^s - 1, ln2 2^(32 - s) (flo in units of P)
  uint32_t tab;           // shared-memory address of the table
};
__device__ __forceinline__ ExpFrame exp_frame(int F, uint32_t tab)
{
  ExpFrame f;
  f.s = F - 43;
  f.mask = (1u << f.s) - 1u;
  f.mul = (2977044472u >> f.s) + (f.s ? (2977044472u >> (f.s - 1)) & 1u : 0u);
  f.tab = tab;
  return f;
}
// (The table's contents never change, so its load may move freely.)
__device__ __forceinline__ double exp2_neg(uint64_t z, const ExpFrame &E)
{
  const uint32_t hi = (uint32_t)(z >> 32), lo = (uint32_t)z;
  const uint32_t v = hi >> E.s, f = __funnelshift_r(lo, hi, E.s);          // n 2048 + i, phi's upper 32 bits
  uint64_t t;
  asm("ld.shared.u64 %0, [%1];" : "=l"(t) : "r"(E.tab + (v & (ETAB - 1)) * 8));
  const uint64_t lin = madw(lo & E.mask, E.mul, madw(f, 2977044472u, 0));
  const uint32_t q = mulhi(f, mulhi(f, 2063529957u - mulhi(f, 232762u)) + 744u);
  const uint64_t p = (uint64_t)madws((int)q, -(1 << 20), (long long)lin) >> 11;   // P in units of 2^-64
  const uint32_t th = (uint32_t)(t >> 32), tl = (uint32_t)t, ph = (uint32_t)(p >> 32), pl = (uint32_t)p;
  const uint64_t s = madw(th, ph, 0) + mulhi(th, pl) + mulhi(tl, ph);      // T P
  const uint64_t m = (t - s) >> 11;                                        // [2^52, 2^53], units of 2^-53
  return __hiloint2double((int)((uint32_t)(m >> 32) + (1021u << 20) - (v >> 11) * (1u << 20)), (int)(uint32_t)m);
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
  return exp2_neg((uint64_t)z, ExpFrame{10, 1023u, 2907270u, tab});
}

}  // namespace sliced
}  // namespace gsks
