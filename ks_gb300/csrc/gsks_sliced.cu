// gsks_sliced.cu -- the FP64 form on the tensor cores (sm_103a).
//
// FP64 instructions issue at 2 per SM cycle on this GPU, 1/64 of the FP32 rate
// and 1/32 of the integer rate, so a kernel that forms its inner products with
// DFMA is bound by that pipe at k + 12 .. k + 40 instructions a pair whatever
// else it does (gsks_fp64.cu: 6.9e9 pairs/s at k = 64).  Here the inner
// products run on the 5th-generation tensor cores, exactly, after the scheme
// of Ozaki, Ogita, Oishi and Rump (Numerical Algorithms 59, 2012):
//
//   x_p = 2^e (d0 2^-8 + d1 2^-17 + ... + d5 2^-53),  e the row's exponent,
//         six balanced digits |d| <= 256, stored as FP16 integers (the
//         row's largest coordinate is held to its last bit, every other one to
//         2^-54 of 2^e);
//   the products of digits i and j, i + j = l <= 5, are integers; their sums
//         over 64 coordinates stay within 2^24 and are exact in the FP32
//         accumulator of level l (levels 4 and 5 may round their last bit on
//         rows of nothing but extreme digits);
//   W = sum over l of acc_l 2^-9l as one 64-bit integer, formed with integer
//         instructions.  What is left out (levels 6 and beyond) is of the size
//         2^-54 of 2^(e_i + e_j), below the rounding of the norms' own sum.
//
// One conversion then gives x.y in FP64, and the kernel functions follow as in
// gsks_fp64.cu.  The Gaussian kernel goes further: with the bandwidth folded
// into the coordinates and all points on one exponent, the exponent y of its
// value 2^-y is |x|^2 + |y|^2 - W in integers, 2^-y comes from exp2_neg
// (integers too), and the weighted sum is the one FP64 instruction a pair.
//
// Preparation: scan_kernel (Gaussian only: the points' largest coordinate and
// the range of their norms), slice_kernel (the digits, written as tile images
// in the layout the MMA reads, one block per 32 points).  Then sliced_tiles,
// one persistent CTA of 18 warps per SM over items (target tile of 128, run of
// source tiles of 64):
//   warp 0       bulk copies: the target tile resident for k <= 64 (96 KB at
//                k = 64), source tiles through two stages; beyond k = 64 both
//                operands in 32-wide chunks
//   warp 1       MMA issue: 21 tcgen05.mma (M 128, N 64) per 16 coordinates
//                into six accumulators (384 TMEM columns)
//   warps 2..17  epilogue: each 32 rows x 16 columns; the accumulators become
//                16 integers W per thread, the tensor memory is handed back,
//                and the kernel values are formed while the next tile's
//                products run
// Each epilogue group writes its own row sums, one per (row, run, group);
// fp64_reduce adds them in a fixed order (deterministic).  Every wait is
// bounded, as in gsks_split.cu.
#include "gsks.h"
#include "gsks_internal.cuh"
#include "gsks_host.h"
#include "gsks_sm100.cuh"
#include "gsks_sliced.cuh"

#include <cuda_fp16.h>
#include <algorithm>
#include <cmath>

namespace gsks {
namespace sliced {

using namespace sm100;

constexpr int GROUPS = 4;                        // column groups of the epilogue
constexpr int COLS = BN / GROUPS;                // columns per thread and tile
constexpr int EPI_WARPS = 4 * GROUPS;
constexpr int NTHREADS = 32 * (2 + EPI_WARPS);
constexpr int NMETA = 3;                         // source metadata slots
constexpr int NSTAGE = 2;                        // operand stages
constexpr uint32_t TMEM_COLS = 512;              // six accumulators of 64 columns (allocation: a power of two)
constexpr size_t SMEM_MAX = 232448;
constexpr long long WAIT_LIMIT = 1LL << 32;      // clock cycles (~2 s) per wait

static __device__ const ExpTable g_exp_table = ExpTable();

// What the Gaussian's fixed-point form needs, per call (written by
// slice_kernel): all points on the exponent e, y = A + B - W in units of 2^-F.
struct CallParam {
  int fixed;             // the fixed-point form applies
  int e, F;
  int shl;               // 53 - F: y to units of 2^-53
  int lim, end;          // high words of 1021 2^F and (at most 2^31 - 1) of 1088 2^F
  double alpha, ah, al;  // alpha^2 = ah + al
};

// One block's share of the scan: largest |coordinate| (as ordered bits), the
// norms' range, whether anything is not finite.
struct ScanPart {
  unsigned long long maxabs;
  double nmin, nmax;
  int bad, pad;
};
constexpr int SCAN_MAX = 256;

struct SliceArgs {
  int m, n, k, kpad, kt, nrhs, nr;
  const double *XA, *XA2, *hi; const int *amap; int nxa;
  const double *XB, *XB2, *hj; const int *bmap; int nxb;
  const double *w; const int *wmap;
  double scal;
  uint8_t *imgA, *imgB;
  double *row_aa, *row_hi; int *row_e;
  const ScanPart *scan; int nscan;
  CallParam *cp;
  int *next_item;
  int *err;
};

// k coordinates are processed in chunks: the whole padded k when the target
// tile stays resident, KST beyond.
__host__ __device__ inline int kchunk(int kpad) { return kpad <= KRES ? kpad : KST; }
__host__ __device__ inline size_t op_bytes(int rows, int kpad) { return (size_t)NS * rows * kpad * 2; }
__host__ __device__ inline size_t btile_bytes(int kpad, int nr) { return op_bytes(BN, kpad) + colmeta_bytes(nr); }
// Bits of W below 2^-52 of 2^(e_i + e_j): what 64 bits leave for k coordinates
// (|x.y| <= k 2^(e_i + e_j), and sums of norms four times that; three at most,
// for combine's multipliers).
__host__ __device__ inline int guard_bits(int kpad)
{
  int g = 3;
  for (int k = 32; k < kpad; k *= 2) g--;
  return g;
}

__device__ __forceinline__ int pool_index(const int *map, int pos, int npool, int *err)
{
  int p = map ? map[pos] : pos;
  if (npool >= 0 && (p < 0 || p >= npool)) { atomicOr(err, DEVERR_MAP_RANGE); p = 0; }
  return p;
}

// ---------------------------------------------------------------------------
// Largest |coordinate| and norm range of the gathered points (one warp per
// point): HBM-bound, 8 k bytes a point.
__global__ void __launch_bounds__(256) scan_kernel(SliceArgs a, ScanPart *__restrict__ part)
{
  __shared__ unsigned long long s_mx[8];
  __shared__ double s_lo[8], s_hi[8];
  __shared__ int s_bad[8];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  unsigned long long mx = 0;
  double lo = 1e300, hi = -1e300;
  bool bad = false;
  for (int i = blockIdx.x * 8 + wp; i < a.m + a.n; i += gridDim.x * 8) {
    const bool A = i < a.m;
    const int p = A ? pool_index(a.amap, i, a.nxa, a.err) : pool_index(a.bmap, i - a.m, a.nxb, a.err);
    const double *x = (A ? a.XA : a.XB) + (size_t)p * a.k;
    for (int c = lane; c < a.k; c += 32)
      mx = max(mx, (unsigned long long)__double_as_longlong(x[c]) & 0x7fffffffffffffffull);
    const double nn = A ? a.XA2[p] : a.XB2[p];
    bad |= !(nn >= 0.0 && nn < 1e300);
    lo = fmin(lo, nn);
    hi = fmax(hi, nn);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  bad = __any_sync(0xffffffffu, bad);
  if (lane == 0) { s_mx[wp] = mx; s_lo[wp] = lo; s_hi[wp] = hi; s_bad[wp] = bad; }
  __syncthreads();
  if (threadIdx.x == 0) {
    ScanPart r{0, 1e300, -1e300, 0, 0};
    for (int q = 0; q < 8; q++) {
      r.maxabs = max(r.maxabs, s_mx[q]);
      r.nmin = fmin(r.nmin, s_lo[q]);
      r.nmax = fmax(r.nmax, s_hi[q]);
      r.bad |= s_bad[q];
    }
    part[blockIdx.x] = r;
  }
}

// The Gaussian's frame from the points' range.  The form applies when every
// value is finite, the exponent leaves 33 <= F, the norms fit their points,
// and an absolute error of a few 2^-F in y is no more than FP64's own rounding
// of the pairs' norms: F >= 52, or every norm sum at least 2^(52 - F).
__device__ CallParam call_param(const ScanPart &s, double scal, int kpad)
{
  CallParam c;
  c.fixed = 0; c.e = 0; c.F = 0; c.shl = 0; c.lim = 0; c.end = 0;
  const double c2 = -scal * 1.4426950408889634;     // y = c2 d^2
  c.alpha = sqrt(c2);
  c.ah = c.alpha * c.alpha;
  c.al = fma(c.alpha, c.alpha, -c.ah);
  const double mx = __longlong_as_double((long long)s.maxabs) * c.alpha;
  if (!(c2 > 0.0 && c2 < 1e100) || s.bad || !(mx < 0x1p30)) return c;
  int e = max(0, (guard_bits(kpad) - 1) / 2);       // F at most 53
  while (mx >= ldexp(1.0, e)) e++;
  c.e = e;
  c.F = 51 + guard_bits(kpad) - 2 * e;
  if (c.F < 33 || c.F > 53) return c;
  if (s.nmax * c.ah > (double)kpad * ldexp(1.0, 2 * e)) return c;
  if (c.F < 52 && 2.0 * s.nmin * c.ah < ldexp(1.0, 52 - c.F)) return c;
  c.shl = 53 - c.F;
  c.lim = (int)(1021u << (c.F - 32));
  c.end = (int)min(1088u << (c.F - 32), 0x7fffffffu);
  c.fixed = 1;
  return c;
}

// Digits of eight coordinates as six 16-byte rows of FP16 integers.
// x = 2^(e - 53) X, |X| < 2^53; X plus 256 in every digit but the first splits
// into fields; 1024 + field is an FP16 bit pattern.
__device__ __forceinline__ void slice8(const double (&v)[8], int e, bool live, uint4 (&out)[NS])
{
  uint32_t f[NS][8];
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const uint64_t b = (uint64_t)__double_as_longlong(v[q]);
    const int fld = (int)(b >> 52) & 0x7ff;
    const int sh = e + 1022 - fld;
    uint64_t X = (b & 0xfffffffffffffull) | 0x10000000000000ull;
    X = (live && fld != 0 && sh <= 54) ? (X + ((1ull << sh) >> 1)) >> sh : 0ull;
    if ((long long)b < 0) X = 0ull - X;
    X += 0x1008040201ull << 8;     // 256 (1 + 2^9 + 2^18 + 2^27 + 2^36)
#pragma unroll
    for (int s = 1; s < NS; s++) f[s][q] = (uint32_t)(X >> (SB * (NS - 1 - s))) & 511u;
    f[0][q] = (uint32_t)((int)((long long)X >> (SB * (NS - 1))) + 256);
  }
  const __half2 bias = __floats2half2_rn(1280.f, 1280.f);
#pragma unroll
  for (int s = 0; s < NS; s++) {
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const uint32_t u = (f[s][2 * q] | (f[s][2 * q + 1] << 16)) + 0x64006400u;
      __half2 h = __hsub2(*(const __half2 *)&u, bias);
      w[q] = *(uint32_t *)&h;
    }
    out[s] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// One block per 32 points: lane = point, warp = group of eight coordinates
// (then every eighth group).  Reads 64 bytes a thread, writes 16-byte row
// segments, consecutive points side by side (512 contiguous bytes a warp).
__global__ void __launch_bounds__(256) slice_kernel(SliceArgs a)
{
  __shared__ uint32_t s_max[8][32];
  __shared__ CallParam s_cp;
  __shared__ ScanPart s_part[8];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int nbA = (a.m + BM - 1) / BM * (BM / 32);
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.next_item = 0;
  bool fixed = false;
  if (a.nscan > 0) {
    // every block folds the scan's partials (at most one per thread)
    ScanPart r{0, 1e300, -1e300, 0, 0};
    if ((int)threadIdx.x < a.nscan) r = a.scan[threadIdx.x];
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      r.maxabs = max(r.maxabs, __shfl_xor_sync(0xffffffffu, r.maxabs, o));
      r.nmin = fmin(r.nmin, __shfl_xor_sync(0xffffffffu, r.nmin, o));
      r.nmax = fmax(r.nmax, __shfl_xor_sync(0xffffffffu, r.nmax, o));
      r.bad |= __shfl_xor_sync(0xffffffffu, r.bad, o);
    }
    if (lane == 0) s_part[wp] = r;
    __syncthreads();
    if (threadIdx.x == 0) {
      r = s_part[0];
      for (int q = 1; q < 8; q++) {
        r.maxabs = max(r.maxabs, s_part[q].maxabs);
        r.nmin = fmin(r.nmin, s_part[q].nmin);
        r.nmax = fmax(r.nmax, s_part[q].nmax);
        r.bad |= s_part[q].bad;
      }
      s_cp = call_param(r, a.scal, a.kpad);
      if (blockIdx.x == 0) *a.cp = s_cp;
    }
    __syncthreads();
    fixed = s_cp.fixed != 0;
  } else if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.cp->fixed = 0;
  }

  const int side = (int)blockIdx.x >= nbA;
  const int blk = side ? blockIdx.x - nbA : blockIdx.x;
  const int rows = side ? BN : BM, per = rows / 32;       // rows per tile, blocks per tile
  const int tile = blk / per, r = (blk - tile * per) * 32 + lane;
  const int pt = tile * rows + r;
  const bool valid = pt < (side ? a.n : a.m);
  const int p = valid ? (side ? pool_index(a.bmap, pt, a.nxb, a.err) : pool_index(a.amap, pt, a.nxa, a.err)) : 0;
  const double *x = (side ? a.XB : a.XA) + (size_t)p * a.k;
  const double mul = fixed ? s_cp.alpha : 1.0;
  const int kgs = a.kpad / 8, kc = kchunk(a.kpad), gpc = kc / 8;
  const bool wide = (a.k & 1) == 0 && ((uintptr_t)(side ? a.XB : a.XA) & 15) == 0;

  auto load8 = [&](int kg, double (&v)[8]) {
    const int c0 = kg * 8;
    if (valid && wide && c0 + 8 <= a.k) {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const double2 d = __ldg((const double2 *)(x + c0) + q);
        v[2 * q] = d.x; v[2 * q + 1] = d.y;
      }
    } else {
#pragma unroll
      for (int q = 0; q < 8; q++) v[q] = (valid && c0 + q < a.k) ? __ldg(x + c0 + q) : 0.0;
    }
  };

  double v[8];
  uint32_t mh = 0;
  for (int kg = wp; kg < kgs; kg += 8) {
    load8(kg, v);
    if (!fixed) {
#pragma unroll
      for (int q = 0; q < 8; q++)
        mh = max(mh, ((uint32_t)__double2hiint(v[q]) & 0x7fffffffu) | (__double2loint(v[q]) != 0 ? 1u : 0u));
    }
  }
  int e = fixed ? s_cp.e : 0;
  bool flag = false;
  if (!fixed) {
    s_max[wp][lane] = mh;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; q++) mh = max(mh, s_max[q][lane]);
    if (mh) {
      const int fld = (int)(mh >> 20);
      e = fld - 1022;                     // |x_p| < 2^e
      flag = fld == 0 || fld == 0x7ff || e > ELIM || e < -ELIM;
      if (flag) e = 0;
    }
  }
  uint8_t *base = side ? a.imgB + (size_t)tile * btile_bytes(a.kpad, a.nr) : a.imgA + (size_t)tile * op_bytes(BM, a.kpad);
  const bool once = kgs <= 8;             // each thread's only group is still in registers
  for (int kg = wp; kg < kgs; kg += 8) {
    if (!once) load8(kg, v);
    if (fixed) {
#pragma unroll
      for (int q = 0; q < 8; q++) v[q] *= mul;
    }
    uint4 out[NS];
    slice8(v, e, !flag, out);
    const int c = kg / gpc, kgc = kg - c * gpc;
    uint8_t *dst = base + (size_t)c * op_bytes(rows, kc) + (size_t)kgc * rows * 16 + (size_t)r * 16;
#pragma unroll
    for (int s = 0; s < NS; s++) *(uint4 *)(dst + (size_t)s * rows * kc * 2) = out[s];
  }

  if (wp == 0) {
    const bool norms = kt_uses_norms(a.kt), varbw = a.kt == KS_GAUSSIAN_VAR_BANDWIDTH;
    double nn = (valid && norms) ? (side ? a.XB2[p] : a.XA2[p]) : 0.0;
    if (fixed) {
      const double y = fma(nn, s_cp.ah, nn * s_cp.al) * ldexp(1.0, s_cp.F);
      nn = __longlong_as_double(__double2ll_rn(y));
    }
    const double h = (valid && varbw) ? (side ? a.hj[p] : a.hi[p]) : 0.0;
    if (!side) {
      a.row_aa[pt] = nn;
      a.row_hi[pt] = h;
      a.row_e[pt] = flag ? EFLAG : e;
    } else {
      ColMeta *cm = (ColMeta *)(base + op_bytes(BN, a.kpad));
      cm->bb[r] = nn;
      cm->hj[r] = h;
      cm->e[r] = flag ? EFLAG : e;
      const bool any = __any_sync(0xffffffffu, flag);
      if (lane == 0) { cm->flag[r >> 5] = any ? 1 : 0; cm->pad[r >> 5] = 0; }
      const size_t wi = valid ? (size_t)(a.wmap ? a.wmap[pt] : pt) * a.nrhs : 0;
      for (int q = 0; q < a.nr; q++) cm->w[q][r] = (valid && q < a.nrhs) ? a.w[wi + q] : 0.0;
    }
  }
}

// ---------------------------------------------------------------------------
struct TileArgs {
  int m, n, k, kpad, nrhs;
  int ntm, ntn, nsc, chunk_tiles;   // items = ntm * nsc, chunk_tiles source tiles each
  const uint8_t *imgA, *imgB;
  const double *row_aa, *row_hi; const int *row_e;
  const double *XA, *XB;            // pools and maps, for the points with EFLAG
  const int *amap, *bmap;
  int nxa, nxb;
  KParams kp;
  const CallParam *cp;
  double *partial;                  // [nrhs][nsc][GROUPS][ldp]
  int ldp;
  int *err, *next_item;
  long long wait_limit;
};

struct SlicedSmem {
  uint64_t a_full, a_empty;
  uint64_t b_full[NSTAGE], b_empty[NSTAGE];
  uint64_t m_full[NMETA], m_empty[NMETA];
  uint64_t t_full, t_empty;
  uint64_t drain;
  uint32_t tmem_base;
  int abort;
  int never;             // stays 0: an abort flag for the drain waits
  int islot[2];          // the current items (-1: no work left), by item parity
};

struct SmemLayout {
  bool resident;
  int kc, nch;               // k-chunk, chunks per tile
  size_t a_chunk, b_chunk;   // operand bytes of one chunk
  size_t a_region, stage, meta, table;
};
__host__ __device__ inline SmemLayout smem_layout(int kpad, int nr, bool table)
{
  SmemLayout L;
  L.kc = kchunk(kpad);
  L.nch = kpad / L.kc;
  L.resident = L.nch == 1;
  L.a_chunk = op_bytes(BM, L.kc);
  L.b_chunk = op_bytes(BN, L.kc);
  L.a_region = L.resident ? L.a_chunk : 0;
  L.stage = L.b_chunk + (L.resident ? 0 : L.a_chunk);
  L.meta = colmeta_bytes(nr);
  L.table = table ? ETAB * sizeof(uint64_t) : 0;
  return L;
}
inline size_t smem_bytes(const SmemLayout &L)
{
  return 1024 + L.a_region + NSTAGE * L.stage + NMETA * L.meta + L.table + sizeof(SlicedSmem) + 64;
}
static_assert(1024 + NS * (size_t)BM * KRES * 2 + NSTAGE * NS * (size_t)BN * KRES * 2 +
                      NMETA * colmeta_bytes(RMAX) + ETAB * 8 + sizeof(SlicedSmem) + 64 <= SMEM_MAX,
              "sliced_tiles shared memory (resident)");
static_assert(1024 + NSTAGE * NS * (size_t)(BM + BN) * KST * 2 + NMETA * colmeta_bytes(RMAX) +
                      ETAB * 8 + sizeof(SlicedSmem) + 64 <= SMEM_MAX,
              "sliced_tiles shared memory (streaming)");

// a 2^s sign-extended to 64 bits, m = 2^s: one integer multiply (a 64-bit
// shift of a sign-extended value would be three instructions).
__device__ __forceinline__ long long mulw_s(int a, int m)
{
  long long d;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(d) : "r"(a), "r"(m));
  return d;
}

// W of one pair from its six level sums, with g guard bits (2 or more when
// k <= 64; possibly negative beyond).
template <bool STREAM>
__device__ __forceinline__ long long combine(const uint32_t (&r)[NS], int g)
{
  int a[NS];
#pragma unroll
  for (int l = 0; l < NS; l++) a[l] = __float2int_rn(__uint_as_float(r[l]));
  long long w = mulw_s(a[1], 1 << (27 + g)) + mulw_s(a[2], 1 << (18 + g)) + mulw_s(a[3], 1 << (9 + g));
  if constexpr (!STREAM) {
    // |a4| 2^g <= 5 2^22 2^2 at k = 64, 5 2^21 2^3 at k = 32: 32 bits hold it
    w += (long long)((a[4] << g) + ((a[5] + (1 << (8 - g))) >> (9 - g)));
    return w + ((long long)(a[0] << (4 + g)) << 32);
  } else {
    const long long v = mulw_s(a[4], 512) + a[5];
    w += (v + (1ll << (8 - g))) >> (9 - g);
    return w + ((long long)a[0] << (36 + g));
  }
}

// 4 consecutive 32-bit columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t &a, uint32_t &b, uint32_t &c, uint32_t &d)
{
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(a), "=r"(b), "=r"(c), "=r"(d)
               : "r"(taddr)
               : "memory");
}

__device__ __noinline__ double pow_call(double x, const KParams &kp) { return pow_class(x, kp); }
__device__ __noinline__ double tanh_call(double x) { return tanh(x); }
__device__ __noinline__ double dot_direct(const double *__restrict__ x, const double *__restrict__ y, int k)
{
  double s = 0.0;
  for (int p = 0; p < k; p++) s = fma(x[p], y[p], s);
  return s;
}

// |x_i - y_j|^2 from the pool coordinates.  For points that agree to about
// 2^-39 of their norms |x|^2 + |y|^2 - 2 x.y leaves only the rounding of the
// given norms, which the DFMA form's own rounding cancels when the norms were
// summed in the same order (coincident points: exactly); an exact x.y does
// not, so such pairs are formed directly.
__device__ __noinline__ double near_d2(const TileArgs &a, int i, int j, double d2)
{
  if (!(fabs(d2) < 1e308)) return d2;   // infinite norms or coordinates
  int pa = a.amap ? a.amap[i] : i, pb = a.bmap ? a.bmap[j] : j;
  if (a.nxa >= 0 && (pa < 0 || pa >= a.nxa)) pa = 0;   // flagged by slice_kernel
  if (a.nxb >= 0 && (pb < 0 || pb >= a.nxb)) pb = 0;
  if (pa == pb && a.XA == a.XB) return 0.0;
  const double *x = a.XA + (size_t)pa * a.k, *y = a.XB + (size_t)pb * a.k;
  double s = 0.0;
  for (int p = 0; p < a.k; p++) { const double d = x[p] - y[p]; s = fma(d, d, s); }
  return s;
}

// Row side of a pair.
struct RowMeta {
  double aa, hi;
  int e;
};

// Kernel value from the inner product: the functions of kfun64, with the
// exponentials through exp2_neg and the comparisons of rare cases on the
// doubles' high words (an FP64 comparison costs as much as an FP64 add).
template <int KT>
__device__ __forceinline__ double kvalue(const TileArgs &a, int i, int j, double dot, const RowMeta &am, double bb,
                                         double hj, double cfold, const uint64_t *__restrict__ tab)
{
  const KParams &kp = a.kp;
  double d2 = 0.0;
  bool near = false;
  if constexpr (kt_uses_norms(KT)) {
    d2 = fma(-2.0, dot, am.aa) + bb;
    // d2 at most about 2^-39 of the larger norm, by the high words
    near = __double2hiint(d2) <= max(__double2hiint(am.aa), __double2hiint(bb)) - (39 << 20);
    if (KT != KS_LAPLACE && near && i < a.m) d2 = near_d2(a, i, j, d2);
  }
  if constexpr (KT == KS_GAUSSIAN || KT == KS_GAUSSIAN_VAR_BANDWIDTH) {
    // max(d2, 0), also of NaN (fmax): anything not in (0, inf] becomes 0
    if ((uint32_t)__double2hiint(d2) > 0x7ff00000u) d2 = 0.0;
    if constexpr (KT == KS_GAUSSIAN) return exp2_neg64(d2 * cfold, tab);
    else return exp2_neg64((d2 * cfold) * hj, tab);
  } else if constexpr (KT == KS_POLYNOMIAL) {
    const double c = fma(dot, kp.scal, kp.cons);
    if (kp.powe == 2.0) return c * c;
    if (kp.powe == 3.0) return (c * c) * c;
    if (kp.powe == 4.0) { const double q = c * c; return q * q; }
    return pow_call(c, kp);
  } else if constexpr (KT == KS_LAPLACE) {
    // coincidence only where the high words allow it (coinc < 2^-40)
    if (near || __double2hiint(d2) < 0x3cd203b0) {
      if (d2 < fmax(1e-15, kp.coinc * (am.aa + bb))) d2 = 1.79e308;
    }
    return pow_call(d2, kp) * kp.scal;
  } else if constexpr (KT == KS_TANH) {
    return tanh_call(fma(dot, kp.scal, kp.cons));
  } else if constexpr (KT == KS_MULTIQUADRATIC) {
    return d2 + kp.cons;
  } else {
    // d2 < 1 by the high word (NaN and inf: no)
    if (__double2hiint(d2) >= 0x3ff00000 || (uint32_t)__double2hiint(d2) > 0xfff00000u) return 0.0;
    const double t = 1.0 - d2;
    return KT == KS_QUARTIC ? (15.0 / 16.0) * t * t : 0.75 * t;
  }
}

template <int KT, int NR, bool STREAM>
__global__ void __launch_bounds__(NTHREADS, 1) sliced_tiles(TileArgs a)
{
  constexpr bool TABLE = KT == KS_GAUSSIAN || KT == KS_GAUSSIAN_VAR_BANDWIDTH;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *sm = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const SmemLayout L = smem_layout(a.kpad, NR, TABLE);
  uint8_t *sA = sm, *sStage = sm + L.a_region, *sMeta = sStage + NSTAGE * L.stage;
  uint64_t *sTab = (uint64_t *)(sMeta + NMETA * L.meta);
  SlicedSmem *S = (SlicedSmem *)((uint8_t *)sTab + L.table);
  volatile int *abort = &S->abort;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int items = a.ntm * a.nsc;

  if (threadIdx.x == 0) {
    mbar_init(&S->a_full, 1);
    mbar_init(&S->a_empty, 1 + EPI_WARPS);
    for (int s = 0; s < NSTAGE; s++) { mbar_init(&S->b_full[s], 1); mbar_init(&S->b_empty[s], 1); }
    for (int s = 0; s < NMETA; s++) { mbar_init(&S->m_full[s], 1); mbar_init(&S->m_empty[s], EPI_WARPS); }
    mbar_init(&S->t_full, 1);
    mbar_init(&S->t_empty, EPI_WARPS);
    mbar_init(&S->drain, 1);
    S->abort = 0;
    S->never = 0;
    fence_mbar_init();
  }
  if (warp == 0) { tmem_alloc(&S->tmem_base, TMEM_COLS); tmem_relinquish(); }
  if constexpr (TABLE)
    for (int i = threadIdx.x; i < ETAB; i += NTHREADS) sTab[i] = g_exp_table.v[i];
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = S->tmem_base;

  if (warp == 0) {
    // ---------------- producer ----------------
    if (lane == 0) {
      int g = 0, tt = 0, a_issued = -1;
      int b_last[NSTAGE], m_last[NMETA];
      for (int s = 0; s < NSTAGE; s++) b_last[s] = -1;
      for (int s = 0; s < NMETA; s++) m_last[s] = -1;
      bool stop = false;
      int item = blockIdx.x;
      const size_t bt = btile_bytes(a.kpad, NR);
      for (int it = 0; !*abort && !stop; it++) {
        if (it > 0 && !mbar_wait(&S->a_empty, (it - 1) & 1, abort, a.wait_limit)) break;
        if (item >= items) {
          S->islot[it & 1] = -1;
          mbar_arrive(&S->a_full);
          break;
        }
        S->islot[it & 1] = item;
        const int next = atomicAdd(a.next_item, 1) + (int)gridDim.x;
        const int ti = item % a.ntm, sc = item / a.ntm;
        const int t0 = sc * a.chunk_tiles, t1 = min(a.ntn, t0 + a.chunk_tiles);
        const uint8_t *imgA = a.imgA + (size_t)ti * op_bytes(BM, a.kpad);
        if (L.resident) {
          mbar_arrive_expect_tx(&S->a_full, (uint32_t)L.a_chunk);
          bulk_g2s(sA, imgA, (uint32_t)L.a_chunk, &S->a_full);
        } else {
          mbar_arrive(&S->a_full);
        }
        a_issued = it;
        for (int tj = t0; tj < t1 && !stop; tj++, tt++) {
          const uint8_t *imgB = a.imgB + (size_t)tj * bt;
          for (int c = 0; c < L.nch; c++, g++) {
            const int st = g % NSTAGE, u = g / NSTAGE;
            if (u > 0 && !mbar_wait(&S->b_empty[st], (u - 1) & 1, abort, a.wait_limit)) { stop = true; break; }
            uint8_t *dst = sStage + st * L.stage;
            mbar_arrive_expect_tx(&S->b_full[st], (uint32_t)L.stage);
            bulk_g2s(dst, imgB + (size_t)c * L.b_chunk, (uint32_t)L.b_chunk, &S->b_full[st]);
            if (!L.resident)
              bulk_g2s(dst + L.b_chunk, imgA + (size_t)c * L.a_chunk, (uint32_t)L.a_chunk, &S->b_full[st]);
            b_last[st] = u;
          }
          if (stop) break;
          const int ms = tt % NMETA, mu = tt / NMETA;
          if (mu > 0 && !mbar_wait(&S->m_empty[ms], (mu - 1) & 1, abort, a.wait_limit)) break;
          mbar_arrive_expect_tx(&S->m_full[ms], (uint32_t)L.meta);
          bulk_g2s(sMeta + ms * L.meta, imgB + op_bytes(BN, a.kpad), (uint32_t)L.meta, &S->m_full[ms]);
          m_last[ms] = mu;
        }
        item = next;
      }
      // On an abort, let the copies already issued land before the CTA exits.
      if (*abort) {
        volatile int *nev = &S->never;
        if (a_issued >= 0) mbar_wait(&S->a_full, a_issued & 1, nev, 1LL << 28);
        for (int s = 0; s < NSTAGE; s++)
          if (b_last[s] >= 0) mbar_wait(&S->b_full[s], b_last[s] & 1, nev, 1LL << 28);
        for (int s = 0; s < NMETA; s++)
          if (m_last[s] >= 0) mbar_wait(&S->m_full[s], m_last[s] & 1, nev, 1LL << 28);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (whole warp, one elected lane issues) ----------------
    const unsigned full = 0xffffffffu;
    const uint32_t idesc = idesc_f16_f32(BM, BN);
    const uint64_t ablk = (uint64_t)(BM * L.kc * 2) >> 4, bblk = (uint64_t)(BN * L.kc * 2) >> 4;   // one slice
    const uint64_t astep = (2 * BM * 16) >> 4, bstep = (2 * BN * 16) >> 4;                         // 16 coordinates
    const int nks = L.kc / 16, gch = STREAM ? KRES / KST : 1;   // chunks per accumulation
    int g = 0, tg = 0;
    bool stop = false;
    for (int it = 0; !stop; it++) {
      if (!__all_sync(full, *abort == 0 && mbar_wait(&S->a_full, it & 1, abort, a.wait_limit))) break;
      const int item = __shfl_sync(full, ((volatile int *)S->islot)[it & 1], 0);
      if (item < 0) break;
      const int sc = item / a.ntm, t0 = sc * a.chunk_tiles, t1 = min(a.ntn, t0 + a.chunk_tiles);
      for (int tj = t0; tj < t1 && !stop; tj++) {
        for (int c = 0; c < L.nch; c++, g++) {
          const bool first = c % gch == 0, last = c % gch == gch - 1;
          if (first) {
            if (tg > 0 && !__all_sync(full, mbar_wait(&S->t_empty, (tg - 1) & 1, abort, a.wait_limit))) { stop = true; break; }
            tg++;
          }
          const int st = g % NSTAGE;
          if (!__all_sync(full, mbar_wait(&S->b_full[st], (g / NSTAGE) & 1, abort, a.wait_limit))) { stop = true; break; }
          tc_fence_after();
          const uint32_t sb = smem_addr(sStage + st * L.stage);
          const uint32_t sa = L.resident ? smem_addr(sA) : sb + (uint32_t)L.b_chunk;
          const uint64_t dA = desc_noswizzle(sa, BM * 16, 128), dB = desc_noswizzle(sb, BN * 16, 128);
          if (elect_one()) {
#pragma unroll
            for (int s = 0; s < KRES / 16; s++) {
              if (s < nks) {
                const uint64_t As = dA + (uint64_t)s * astep, Bs = dB + (uint64_t)s * bstep;
#pragma unroll
                for (int l = 0; l < NS; l++)
#pragma unroll
                  for (int i = 0; i <= l; i++)
                    umma_f16(tmem + l * BN, As + i * ablk, Bs + (l - i) * bblk, idesc,
                             (i > 0 || s > 0 || !first) ? 1u : 0u);
              }
            }
            umma_commit(&S->b_empty[st]);
            if (last) umma_commit(&S->t_full);
          }
          __syncwarp();
        }
      }
      if (elect_one()) umma_commit(&S->a_empty);
      __syncwarp();
    }
    if (elect_one()) umma_commit(&S->drain);
    __syncwarp();
    mbar_wait(&S->drain, 0, &S->never, 1LL << 30);
  } else {
    // ---------------- epilogue ----------------
    const int grp = (warp - 2) >> 2, qd = warp & 3;
    const int row = qd * 32 + lane, c0 = grp * COLS;
    const uint32_t tT = tmem + ((uint32_t)(qd * 32) << 16) + c0;
    const int gb = guard_bits(a.kpad);
    const CallParam cp = *a.cp;
    const bool fixed = KT == KS_GAUSSIAN && cp.fixed != 0;
    int g = 0, tg = 0;
    for (int it = 0; !*abort; it++) {
      if (!mbar_wait(&S->a_full, it & 1, abort, a.wait_limit)) break;
      const int item = ((volatile int *)S->islot)[it & 1];
      if (item < 0) break;
      __syncwarp();
      if (lane == 0) mbar_arrive(&S->a_empty);
      const int ti = item % a.ntm, sc = item / a.ntm;
      const int t0 = sc * a.chunk_tiles, t1 = min(a.ntn, t0 + a.chunk_tiles);
      const int i = ti * BM + row;
      RowMeta am;
      am.aa = a.row_aa[i];
      am.hi = a.row_hi[i];
      am.e = a.row_e[i];
      const bool rflag = am.e == EFLAG;
      const bool anyrow = __any_sync(0xffffffffu, rflag);
      // the exponent of 2^-y per unit of d2, in units of 2^-53 (variable bandwidth: times h_i)
      double cfold = 0.0;
      if constexpr (KT == KS_GAUSSIAN) cfold = -a.kp.scal * (1.4426950408889634 * 0x1p53);
      if constexpr (KT == KS_GAUSSIAN_VAR_BANDWIDTH) cfold = am.hi * (0.5 * 1.4426950408889634 * 0x1p53);
      double racc[NR];
#pragma unroll
      for (int r = 0; r < NR; r++) racc[r] = 0.0;
      bool ok = true;
      for (int tj = t0; tj < t1; tj++, g++) {
        long long W[COLS];
        // accumulators -> integers; the tensor memory is free again after the last load
        const int ngr = STREAM ? a.kpad / KRES : 1;
        for (int c = 0; c < ngr; c++, tg++) {
          if (!mbar_wait(&S->t_full, tg & 1, abort, a.wait_limit)) { ok = false; break; }
          tc_fence_after();
#pragma unroll
          for (int q = 0; q < COLS; q += 4) {
            uint32_t r[4][NS];
#pragma unroll
            for (int l = 0; l < NS; l++) tmem_ld4(tT + l * BN + q, r[0][l], r[1][l], r[2][l], r[3][l]);
            tmem_ld_wait();
#pragma unroll
            for (int s = 0; s < 4; s++) {
              const long long w = combine<STREAM>(r[s], gb);
              W[q + s] = STREAM && c > 0 ? W[q + s] + w : w;
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&S->t_empty);
        }
        if (!ok) break;
        const int ms = g % NMETA;
        if (!mbar_wait(&S->m_full[ms], (g / NMETA) & 1, abort, a.wait_limit)) { ok = false; break; }
        const ColMeta *cm = (const ColMeta *)(sMeta + ms * L.meta);
        const int nv = min(COLS, a.n - tj * BN - c0);   // valid columns of this group
        if (fixed) {
          const long long A = __double_as_longlong(am.aa);
#pragma unroll
          for (int c = 0; c < COLS; c++) {
            long long y = A + __double_as_longlong(cm->bb[c0 + c]) - W[c];
            if (y <= (A >> 38) && c < nv && i < a.m)
              y = __double2ll_rn(near_d2(a, i, tj * BN + c0 + c, 0.0) * cp.ah * ldexp(1.0, cp.F));
            double kv;
            if ((int)(y >> 32) < cp.lim) kv = exp2_neg((uint64_t)y << cp.shl, sTab);
            else if ((int)(y >> 32) >= cp.end) kv = 0.0;
            else kv = exp2_neg_wide((double)y * ldexp(1.0, -cp.F));
#pragma unroll
            for (int r = 0; r < NR; r++)
              if (r == 0 || r < a.nrhs) racc[r] = fma(kv, cm->w[r][c0 + c], racc[r]);
          }
        } else {
          const bool slow = anyrow || cm->flag[c0 >> 5] != 0;
#pragma unroll
          for (int c = 0; c < COLS; c++) {
            const int ej = cm->e[c0 + c];
            double dot = (double)W[c];
            dot = __hiloint2double(__double2hiint(dot) + (W[c] != 0 ? (am.e + ej - 52 - gb) << 20 : 0),
                                   __double2loint(dot));
            if (slow && (rflag || ej == EFLAG) && c < nv && i < a.m) {
              const int j = tj * BN + c0 + c;
              int pa = a.amap ? a.amap[i] : i, pb = a.bmap ? a.bmap[j] : j;
              if (a.nxa >= 0 && (pa < 0 || pa >= a.nxa)) pa = 0;   // flagged by slice_kernel
              if (a.nxb >= 0 && (pb < 0 || pb >= a.nxb)) pb = 0;
              dot = dot_direct(a.XA + (size_t)pa * a.k, a.XB + (size_t)pb * a.k, a.k);
            }
            if (c < nv) {
              const double kv = kvalue<KT>(a, i, tj * BN + c0 + c, dot, am, cm->bb[c0 + c], cm->hj[c0 + c], cfold, sTab);
#pragma unroll
              for (int r = 0; r < NR; r++)
                if (r == 0 || r < a.nrhs) racc[r] = fma(kv, cm->w[r][c0 + c], racc[r]);
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&S->m_empty[ms]);
      }
      if (!ok) break;
      if (i < a.m) {
#pragma unroll
        for (int r = 0; r < NR; r++)
          if (r == 0 || r < a.nrhs) a.partial[(((size_t)r * a.nsc + sc) * GROUPS + grp) * a.ldp + i] = racc[r];
      }
    }
  }

  __syncthreads();
  if (*abort && threadIdx.x == 0) atomicOr(a.err, DEVERR_TIMEOUT);
  if (warp == 0) { tc_fence_after(); tmem_dealloc(tmem, TMEM_COLS); }
}

template <int KT, int NR, bool STREAM>
cudaError_t launch_t(const TileArgs &a, int grid, cudaStream_t s)
{
  const size_t smem = smem_bytes(smem_layout(a.kpad, NR, KT == KS_GAUSSIAN || KT == KS_GAUSSIAN_VAR_BANDWIDTH));
  // The attribute is per function and device; raised once to the most any launch takes.
  static bool raised[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !raised[dev]) {
    const cudaError_t e =
        cudaFuncSetAttribute(sliced_tiles<KT, NR, STREAM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) raised[dev] = true;
  }
  sliced_tiles<KT, NR, STREAM><<<grid, NTHREADS, smem, s>>>(a);
  return cudaGetLastError();
}

template <int KT>
cudaError_t launch_k(const TileArgs &a, int grid, int nr, cudaStream_t s)
{
  const bool stream = a.kpad > KRES;
  if (nr > 1) return stream ? launch_t<KT, RMAX, true>(a, grid, s) : launch_t<KT, RMAX, false>(a, grid, s);
  return stream ? launch_t<KT, 1, true>(a, grid, s) : launch_t<KT, 1, false>(a, grid, s);
}

cudaError_t launch_tiles(const TileArgs &a, int grid, int nr, cudaStream_t s)
{
  switch (a.kp.type) {
    case KS_GAUSSIAN: return launch_k<KS_GAUSSIAN>(a, grid, nr, s);
    case KS_GAUSSIAN_VAR_BANDWIDTH: return launch_k<KS_GAUSSIAN_VAR_BANDWIDTH>(a, grid, nr, s);
    case KS_POLYNOMIAL: return launch_k<KS_POLYNOMIAL>(a, grid, nr, s);
    case KS_LAPLACE: return launch_k<KS_LAPLACE>(a, grid, nr, s);
    case KS_TANH: return launch_k<KS_TANH>(a, grid, nr, s);
    case KS_QUARTIC: return launch_k<KS_QUARTIC>(a, grid, nr, s);
    case KS_MULTIQUADRATIC: return launch_k<KS_MULTIQUADRATIC>(a, grid, nr, s);
    default: return launch_k<KS_EPANECHNIKOV>(a, grid, nr, s);
  }
}

}  // namespace sliced

// Padded k: a multiple of the MMA's k-step up to KRES, of KRES beyond.
static int sliced_kpad(int k)
{
  return k <= sliced::KRES ? (k + 15) / 16 * 16 : (k + sliced::KRES - 1) / sliced::KRES * sliced::KRES;
}

bool sliced_takes(int k) { return sliced_kpad(k) <= sliced::KMAX; }

int enqueue_sliced(Ctx *c, const ks_t *ker, int m, int n, int k, double *u, const int *umap,
                   const double *XA, const double *XA2, const int *amap, int nxa,
                   const double *XB, const double *XB2, const int *bmap, int nxb,
                   const double *w, const int *wmap, const double *hi, const double *hj,
                   cudaStream_t s, bool stream_ordered_alloc, int nrhs)
{
  using namespace sliced;
  const int nr = nrhs > 1 ? RMAX : 1;
  const int kpad = sliced_kpad(k);
  const int ntm = (m + BM - 1) / BM, ntn = (n + BN - 1) / BN, sms = std::max(1, c->num_sms);
  // Runs of source tiles: the slowest CTA's work, waves x (run + one tile of
  // per-item overhead), over up to 16 items per SM (as enqueue_split).
  int nsc = 1, chunk = ntn;
  {
    const int cmax = (int)std::min<long long>(ntn, std::max<long long>(1, (16LL * sms + ntm - 1) / ntm));
    long long best = -1;
    for (int q = 1; q <= cmax; q++) {
      const int ch = (ntn + q - 1) / q;
      if ((ntn + ch - 1) / ch != q) continue;
      const long long cost = (((long long)ntm * q + sms - 1) / sms) * (ch + 1);
      if (best < 0 || cost < best) { best = cost; nsc = q; chunk = ch; }
    }
  }
  const int ldp = ntm * BM;
  const bool scan = ker->type == KS_GAUSSIAN;
  const int nscan = scan ? (int)std::min<long long>(SCAN_MAX, ((long long)m + n + 7) / 8) : 0;

  auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const size_t o_cp = 0;
  const size_t o_next = o_cp + al(sizeof(CallParam));
  const size_t o_scan = o_next + al(4);
  const size_t o_a = o_scan + al((size_t)nscan * sizeof(ScanPart));
  const size_t o_b = o_a + al((size_t)ntm * op_bytes(BM, kpad));
  const size_t o_aa = o_b + al((size_t)ntn * btile_bytes(kpad, nr));
  const size_t o_hi = o_aa + al((size_t)ldp * 8);
  const size_t o_e = o_hi + al((size_t)ldp * 8);
  const size_t o_p = o_e + al((size_t)ldp * 4);
  const size_t total = o_p + al((size_t)nrhs * nsc * GROUPS * ldp * 8);
  uint8_t *ws = nullptr;
  if (stream_ordered_alloc) {
    const cudaError_t e = cudaMallocAsync((void **)&ws, total, s);
    if (e != cudaSuccess) return cuda_status(e, "sliced workspace");
  } else {
    if (!c->dwork.ensure(total)) return GSKS_ERR_ALLOC;
    ws = (uint8_t *)c->dwork.p;
  }

  SliceArgs p{};
  p.m = m; p.n = n; p.k = k; p.kpad = kpad; p.kt = ker->type; p.nrhs = nrhs; p.nr = nr;
  p.XA = XA; p.XA2 = XA2; p.hi = hi; p.amap = amap; p.nxa = nxa;
  p.XB = XB; p.XB2 = XB2; p.hj = hj; p.bmap = bmap; p.nxb = nxb;
  p.w = w; p.wmap = wmap; p.scal = ker->scal;
  p.imgA = ws + o_a; p.imgB = ws + o_b;
  p.row_aa = (double *)(ws + o_aa); p.row_hi = (double *)(ws + o_hi); p.row_e = (int *)(ws + o_e);
  p.scan = (const ScanPart *)(ws + o_scan); p.nscan = nscan;
  p.cp = (CallParam *)(ws + o_cp);
  p.next_item = (int *)(ws + o_next);
  p.err = err_word(c);
  if (scan) scan_kernel<<<nscan, 256, 0, s>>>(p, (ScanPart *)(ws + o_scan));
  slice_kernel<<<ntm * (BM / 32) + ntn * (BN / 32), 256, 0, s>>>(p);

  TileArgs a{};
  a.m = m; a.n = n; a.k = k; a.kpad = kpad; a.nrhs = nrhs;
  a.ntm = ntm; a.ntn = ntn; a.nsc = nsc; a.chunk_tiles = chunk;
  a.imgA = p.imgA; a.imgB = p.imgB;
  a.row_aa = p.row_aa; a.row_hi = p.row_hi; a.row_e = p.row_e;
  a.XA = XA; a.XB = XB; a.amap = amap; a.bmap = bmap; a.nxa = nxa; a.nxb = nxb;
  a.kp = make_kparams(ker, hi, hj);
  a.kp.coinc = coincidence_eps(k);
  a.cp = p.cp;
  a.partial = (double *)(ws + o_p);
  a.ldp = ldp;
  a.err = p.err;
  a.next_item = p.next_item;
  a.wait_limit = WAIT_LIMIT;
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = launch_tiles(a, std::min(ntm * nsc, sms), nr, s);
  if (e == cudaSuccess) {
    fp64_reduce_launch(m, nsc * GROUPS, ldp, nrhs, (long long)nsc * GROUPS * ldp, a.partial, u, umap, s);
    e = cudaGetLastError();
  }
  if (stream_ordered_alloc) cudaFreeAsync(ws, s);
  if (e != cudaSuccess) return cuda_status(e, "sliced launch");
  note_launches(scan ? 4 : 3);
  return GSKS_OK;
}

}  // namespace gsks
