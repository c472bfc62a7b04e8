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
constexpr int BN = 64;               // sources per tile
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
// the integers of the fixed-point Gaussian), bandwidths, exponents, whether a
// half tile holds a point with EFLAG, and the weight columns.
struct ColMeta {
  double bb[BN];
  double hj[BN];
  int e[BN];
  int flag[2];
  int pad[2];
  double w[RMAX][BN];
};
__host__ __device__ constexpr size_t colmeta_bytes(int nr) { return offsetof(ColMeta, w) + (size_t)nr * BN * 8; }
static_assert(colmeta_bytes(1) % 16 == 0, "ColMeta is copied by the bulk-copy engine");

// ---------------------------------------------------------------------------
// 2^-(i / ETAB) in units of 2^-53, i = 0 .. ETAB - 1 (2^53 down to just above
// 2^52): products of the eleven constants 2^(-2^b / ETAB) in 64-bit fixed
// point, evaluated by the compiler.
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
    v[0] = 1ull << 53;
    for (int i = 1; i < ETAB; i++) {
      uint64_t p = 0;
      bool first = true;
      for (int b = 0; b < 11; b++)
        if (i >> b & 1) {
          p = first ? c[b] : mulhi64c(p, c[b]);
          first = false;
        }
      v[i] = (p + (1ull << 10)) >> 11;
    }
  }
};

__device__ __forceinline__ uint64_t mulw(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
__device__ __forceinline__ uint32_t mulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }

// 2^-y for y = z 2^-53, 0 <= y < 1021, to about one unit in the last place:
// y = n + (i + phi) / 2048, 2^-y = 2^-n T[i] (1 - P), P = 1 - 2^(-phi / 2048)
// by its series to the fourth order (the table-driven scheme of P. T. P. Tang,
// ACM TOMS 15 (1989), in integers).  FP64 instructions issue at 1/32 of the
// integer rate here (2 against 64 per SM cycle, measured): an FP64 exponential
// of about 18 of them takes 9 SM cycles a value, these about 28 integer ones
// less than half a cycle.
//   phi = f 2^-32 + flo 2^-42; P in units of 2^-75: ln2 (f 2^32 + ...) with
//   ln2 2^32 rounded up (2977044472; the excess, 739 2^-55 phi, goes to q);
//   q in units of 2^-55: z^2/2 - z^3/6 + z^4/24, z = ln2 phi / 2048.  The
//   addend 736 of T P rounds its last shift (1024) less the mean of q's floors.
// Against exp2l over y in [0, 1000]: at most 2.3 2^-53 relative, rms 0.6 2^-53.
constexpr uint32_t EXP_END = 1021u << 21;   // high word of y = 1021

__device__ __forceinline__ double exp2_neg(uint64_t z, const uint64_t *__restrict__ tab)
{
  const uint32_t hi = (uint32_t)(z >> 32), lo = (uint32_t)z;
  const uint64_t t = tab[(hi >> 10) & (ETAB - 1)];
  const uint32_t f = __funnelshift_l(lo, hi, 22);
  const uint64_t lin = mulw(f, 2977044472u) + mulw(lo & 1023u, 2907270u);
  uint32_t q = 232801u - mulhi(f, 20u);
  q = 2063529982u - mulhi(f, q);
  q = mulhi(f, q) + 739u;
  q = mulhi(f, q);
  const uint64_t P = lin - mulw(q, 1u << 20);
  const uint32_t th = (uint32_t)(t >> 32), tl = (uint32_t)t, ph = (uint32_t)(P >> 32), pl = (uint32_t)P;
  const uint64_t s = mulw(th, ph) + (uint64_t)mulhi(th, pl) + (uint64_t)mulhi(tl, ph) + 736u;   // T P, units of 2^-64
  const uint64_t m = t - (s >> 11);                        // [2^52, 2^53], units of 2^-53
  const uint32_t top = (uint32_t)(m >> 32) + (1021u << 20) - ((hi >> 21) << 20);
  return __hiloint2double((int)top, (int)(uint32_t)m);
}

// 2^-y outside exp2_neg's range (y negative, beyond 1021, or no number).
__device__ __noinline__ inline double exp2_neg_wide(double y) { return exp2(-y); }

// 2^-y for an FP64 y (given as y 2^53).
__device__ __forceinline__ double exp2_neg64(double y53, const uint64_t *__restrict__ tab)
{
  const long long z = __double2ll_rn(y53);
  if ((uint32_t)(z >> 32) >= EXP_END) {          // (negative z too)
    // y above 1088 (high word of 1088 2^53): 0 in FP64 as well
    if ((uint32_t)(__double2hiint(y53) - 0x43e10000) < 0x7ff00001u - 0x43e10000u) return 0.0;
    return exp2_neg_wide(y53 * 0x1p-53);
  }
  return exp2_neg((uint64_t)z, tab);
}

}  // namespace sliced
}  // namespace gsks
