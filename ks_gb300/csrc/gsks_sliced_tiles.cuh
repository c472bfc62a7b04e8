// gsks_sliced_tiles.cuh -- the kernels of the FP64 form on the tensor cores, shared by
// the single call (gsks_sliced.cu) and the batched form (gsks_sliced_list.cu).
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
//         2^-54 of 2^e: held_bits says where that is not enough);
//   the products of digits i and j, i + j = l <= 6, are integers; their sums
//         over 64 coordinates stay within 2^24 and are exact in the FP32
//         accumulator of level l up to 3 (beyond, rows of nothing but extreme
//         digits may round their last bit);
//   W = sum over l of acc_l 2^-9l as one 64-bit integer, formed with integer
//         instructions, one rounding per 64 coordinates.  What is left out
//         (levels 7 and beyond) is at most k 2^-61 of 2^(e_i + e_j).
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
// source tiles of 32):
//   warp 0       bulk copies: the target tile resident for k <= 64 (96 KB at
//                k = 64), source tiles through four stages; beyond k = 64 two
//                source tiles and the targets in 32-wide chunks
//   warp 1       MMA issue: the source slices lie stacked along N, so that
//                target slice i times slices 0 .. 6 - i (0 .. 5 for i = 0) is one
//                tcgen05.mma of N = 32 (7 - i) whose columns are the accumulators of
//                levels i .. 6: six instructions per 16 coordinates, each target
//                slice read once (21 of N = 64 read it six times over and took
//                4032 SM cycles of shared-memory bandwidth per 64 columns at
//                k = 64 where these take 2816)
//   warps 2..17  epilogue, in two halves of eight, each with an accumulator
//                buffer (224 TMEM columns) of its own: a half turns its
//                accumulators into integers W (bound by the float-to-integer
//                conversions, 16 per SM cycle) while the other forms kernel
//                values (bound by the FP64 pipe) and the tensor cores fill the
//                buffer handed back
// A work item's row sums (the four groups' in order) go to one partial per (row,
// run) -- with several right-hand sides one per group too -- and the last of a
// row's runs to arrive adds them in run order (deterministic).  Every wait is
// bounded, as in gsks_split.cu; no wait is on another CTA.  The batched form
// (LISTED) runs the same kernels over tables of tiles and items from many tasks,
// each with its own descriptor and frame: one launch per kernel type, in two streams
// that start after slice_kernel, so that a type's blocks get in as the one's before it in
// the other stream run out of items.  (One kernel with every type's epilogue spilled 800
// bytes a thread and took 1.5 times as long.)
#pragma once
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

constexpr int GROUPS = 4;                        // epilogue groups of four warps
constexpr int HALVES = 2;                        // accumulator buffers, each with two of the groups
constexpr int COLS = BN * HALVES / GROUPS;       // columns per thread and tile
constexpr int EPI_WARPS = 4 * GROUPS;
constexpr int HALF_WARPS = EPI_WARPS / HALVES;
constexpr int NTHREADS = 32 * (2 + EPI_WARPS);
constexpr int NMETA = 4;                         // source metadata slots
constexpr int NSTAGE_RES = 4, NSTAGE_STR = 2;    // operand stages (resident, streaming)
constexpr uint32_t TMEM_COLS = 512;              // two buffers of up to seven accumulators (allocation: a power of two)
// Levels formed.  With six the products left out were the largest part of the error
// wherever the points do not lie in one orthant far from the origin: the error's rms in
// units of 2^-53 of the conditioned sum, six levels -> seven (DFMA): Laplace of normal
// points, k = 16, 4.5 -> 0.5 (0.5); tanh of sparse rows, k = 33, 2.4 -> 0.7 (0.2);
// polynomial of rows with one large coordinate, k = 1000, 4.5 -> 1.3 (1.3).  The seventh
// costs 8 % where the streamed images bound the kernel (8192 x 12000, k = 1024: 4.30 ->
// 4.65 ms), 1 to 3 % elsewhere (65536 x 65536, k = 64: 13.84 -> 14.01 ms).
constexpr int LV = NS + 1;
constexpr size_t SMEM_MAX = 232448;
constexpr long long WAIT_LIMIT = 1LL << 32;      // clock cycles (~2 s) per wait

static __device__ const ExpTable g_exp_table = ExpTable();

// What the fixed-point form of the Gaussian, variable-bandwidth Gaussian and
// Laplace kernels needs, per call or task: all points on the exponent e, their
// distance (the Gaussian: its exponent y) A + B - W in units of 2^-F.
struct CallParam {
  int fixed;             // the fixed-point form applies
  int e, F;
  int pre;               // left shift of y where F is below 43 (exp2_neg's least), else 0
  int lim, end;          // high words of 1021 2^F and 1088 2^F, at most 2^31 - 1
  int small;             // high word of 2^51, or 0: two norms below it, the pair is formed directly
  int pad;
  double alpha, ah, al;  // coordinates are scaled by alpha; alpha^2 = ah + al
  double pad2;
  PowFrame pw;           // Laplace
};

// One task of the list form (copied into shared memory with its items): the
// kernel and the Gaussian's frame from the task's own points.
struct __align__(16) TaskParam {
  KParams kp;
  CallParam cp;
};
static_assert(sizeof(TaskParam) % 16 == 0, "TaskParam is copied by the bulk-copy engine");

// One work item of the list form: target tile a_tile (list positions ia ..
// ia + rows - 1), source tiles b0 .. b1 - 1 (positions jb .. jb + cols - 1); the
// row sums go to partial[out + row].
struct Item {
  int a_tile, rows, ia, b0, b1, jb, cols, task;
  long long out;
};

// One task's target and source list positions.
struct TaskGeo {
  int a0, m, b0, n;
};

// One block's share of the scan, by high words (one reduction instruction each;
// small calls wait for this code to be fetched): the largest |coordinate|, the
// least and the largest norm (all ones: a value the form does not take).
struct ScanPart {
  uint32_t maxabs, nmin, nmax, pad;
};
constexpr int NTYPES = 8;           // kernel types (ks_type), each with a work counter in the list form
constexpr int SCAN_MAX = 256;
// Coordinates up to which every block of slice_kernel scans all points itself
// (32 loads a thread) instead of a launch of its own.
constexpr long long SCAN_SELF = 8192;

struct SliceArgs {
  int m, n, k, kpad, kt, nrhs, nr;
  const double *XA, *XA2, *hi; const int *amap; int nxa;
  const double *XB, *XB2, *hj; const int *bmap; int nxb;
  const double *w; const int *wmap;
  CallParam frame;         // kernel_frame of the call
  uint8_t *imgA, *imgB;
  double *row_aa; uint64_t *row_hi; int *row_e, *row_n;
  const ScanPart *scan; int nscan;   // partials; 0: few points, -1: no Gaussian
  CallParam *cp;
  int *next_item;
  int *err;
  // list form: tile t of a side packs list positions tiles[t].x .. + tiles[t].y - 1
  // of task tile_task[t]
  const int2 *tilesA, *tilesB;
  const int *taskA, *taskB;
  const TaskParam *tp;
  int nta;                 // target tiles
};

// k coordinates are processed in chunks: the whole padded k when the target
// tile stays resident, KST beyond.
__host__ __device__ inline int kchunk(int kpad) { return kpad <= KRES ? kpad : KST; }
__host__ __device__ inline size_t op_bytes(int rows, int kpad) { return (size_t)NS * rows * kpad * 2; }
__host__ __device__ inline size_t btile_bytes(int kpad, int nr) { return op_bytes(BN, kpad) + colmeta_bytes(nr); }
// Bits of W below 2^-52 of 2^(e_i + e_j): what 64 bits leave for k coordinates
// (|x.y| < k 2^(e_i + e_j), and with a frame sums of norms four times that;
// three at most, for combine's multipliers).
__host__ __device__ inline int guard_bits(int kpad, bool framed)
{
  int g = 3;
  for (int k = framed ? 32 : 128; k < kpad; k *= 2) g--;
  return g;
}

__device__ __forceinline__ int pool_index(const int *map, int pos, int npool, int *err)
{
  int p = map ? map[pos] : pos;
  if (npool >= 0 && (p < 0 || p >= npool)) { atomicOr(err, DEVERR_MAP_RANGE); p = 0; }
  return p;
}

__device__ __forceinline__ int pool_clamp(const int *map, int pos, int npool)
{
  const int p = map ? map[pos] : pos;
  return npool >= 0 && (uint32_t)p >= (uint32_t)npool ? 0 : p;
}

// ---------------------------------------------------------------------------
// A block's fold of its threads' scan values (256 threads, every thread calls;
// the result in every thread).
__device__ __forceinline__ ScanPart scan_fold(ScanPart r)
{
  __shared__ ScanPart part[8];
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  r.maxabs = __reduce_max_sync(full, r.maxabs);
  r.nmin = __reduce_min_sync(full, r.nmin);
  r.nmax = __reduce_max_sync(full, r.nmax);
  if (lane == 0) part[threadIdx.x >> 5] = r;
  __syncthreads();
  r = part[lane & 7];
  r.maxabs = __reduce_max_sync(full, r.maxabs);
  r.nmin = __reduce_min_sync(full, r.nmin);
  r.nmax = __reduce_max_sync(full, r.nmax);
  return r;
}

// Scan values of points first, first + step, ... of a target list (m positions
// of amap from a0) followed by a source list (n of bmap from b0), with the
// bandwidth factors hi, hj of the variable-bandwidth kernel: the block's
// threads take one coordinate of every (256 / k)-th point (a point at a time for
// long rows), U of them in flight.
// (Map entries out of range read point 0, as in slice_kernel, which flags them: a
// flag here would keep the loads from being issued together.)
template <int U>
__device__ __forceinline__ ScanPart scan_points(const SliceArgs &a, int a0, int m, int b0, int n, const double *hi,
                                                const double *hj, int first, int step)
{
  ScanPart r{0, ~0u, 0, 0};
  const int lanes = min(a.k, 256), per = 256 / lanes, c0 = threadIdx.x % lanes, sub = threadIdx.x / lanes;
  if (sub < per) {
#pragma unroll
    for (int side = 0; side < 2; side++) {
      const int cnt = side ? n : m, npool = side ? a.nxb : a.nxa;
      const int *__restrict__ map = side ? a.bmap : a.amap;
      const int at = side ? b0 : a0;
      const double *__restrict__ X = side ? a.XB : a.XA, *__restrict__ X2 = side ? a.XB2 : a.XA2;
      const double *__restrict__ h = side ? hj : hi;
      for (int i0 = first * per + sub; i0 < cnt; i0 += U * step * per) {
        uint32_t xh[U], nh[U];
#pragma unroll
        for (int e = 0; e < U; e++) {       // (past the end: the last point again)
          const int p = pool_clamp(map, at + min(i0 + e * step * per, cnt - 1), npool);
          xh[e] = (uint32_t)__double2hiint(X[(size_t)p * a.k + c0]) & 0x7fffffffu;
          for (int c = c0 + lanes; c < a.k; c += lanes)
            xh[e] = max(xh[e], (uint32_t)__double2hiint(X[(size_t)p * a.k + c]) & 0x7fffffffu);
          nh[e] = (uint32_t)__double2hiint(X2[p]);
          if (h) {            // bandwidth factors: within 2^-300 .. 2^300
            if ((uint32_t)__double2hiint(h[p]) - (723u << 20) >= 600u << 20) nh[e] = ~0u;
          }
        }
#pragma unroll
        for (int e = 0; e < U; e++) {
          r.maxabs = max(r.maxabs, xh[e]);
          r.nmin = min(r.nmin, nh[e]);
          r.nmax = max(r.nmax, nh[e]);
        }
      }
    }
  }
  return r;
}

// Largest |coordinate| and norm range of the call's points: HBM-bound, 8 k bytes
// a point.
static __global__ void __launch_bounds__(256) scan_kernel(SliceArgs a, ScanPart *__restrict__ part)
{
  launch_dependents();
  const ScanPart r = scan_fold(scan_points<4>(a, 0, a.m, 0, a.n, a.hi, a.hj, blockIdx.x, gridDim.x));
  if (threadIdx.x == 0) part[blockIdx.x] = r;
}

inline __device__ CallParam call_param(const ScanPart &s, CallParam c, int kt, int kpad);

// The same over one task's points, one block per task with a frame.
static __global__ void __launch_bounds__(256) list_scan_kernel(SliceArgs a, int ntask, const TaskGeo *__restrict__ tg,
                                                        TaskParam *__restrict__ tp)
{
  const int t = blockIdx.x;
  launch_dependents();
  if (t == 0 && threadIdx.x < NTYPES) a.next_item[threadIdx.x] = 0;
  if (t >= ntask || tp[t].cp.alpha == 0.0) return;
  const TaskGeo G = tg[t];
  const KParams &kp = tp[t].kp;
  const bool vb = kp.type == KS_GAUSSIAN_VAR_BANDWIDTH;
  const ScanPart r = scan_fold(scan_points<8>(a, G.a0, G.m, G.b0, G.n, vb ? kp.hi : nullptr, vb ? kp.hj : nullptr, 0, 1));
  if (threadIdx.x == 0) tp[t].cp = call_param(r, tp[t].cp, tp[t].kp.type, a.kpad);
}

// The frame from the points' range.  The form applies when every value is
// finite, the exponent leaves 33 <= F and the norms fit their points.  An error
// of a few 2^-F is no more than FP64's own rounding of a pair's norms where
// their sum is at least 2^(52 - F); a Gaussian's y with F >= 52 needs no more
// than that anyway.  Pairs of two smaller norms are formed directly; where there
// may be many (a norm 64 times smaller) the form does not apply.
// c: what the kernel alone sets (kernel_frame), the rest filled in.
inline __device__ CallParam call_param(const ScanPart &s, CallParam c, int kt, int kpad)
{
  auto pow2 = [](int e) { return __hiloint2double((1023 + e) << 20, 0); };
  c.fixed = 0;
  // (upper bounds of the largest values, a lower one of the least norm)
  if (c.alpha == 0.0 || s.maxabs >= 0x7fe00000u || s.nmax >= 0x7fe00000u) return c;
  const double mx = __hiloint2double((int)s.maxabs + 1, 0) * c.alpha;
  if (!(mx < 0x1p30)) return c;
  // e as low as the points allow (mx < 2^e), F = 51 + g - 2 e at most 62
  const int g = guard_bits(kpad, true);
  c.e = max((g - 11 + 1) / 2, (__double2hiint(mx) >> 20) - 1022);
  c.F = 51 + g - 2 * c.e;
  if (c.F < 33) return c;
  const double nmin = __hiloint2double((int)s.nmin, 0), nmax = __hiloint2double((int)s.nmax + 1, 0);
  if (nmax * c.ah > (double)kpad * pow2(2 * c.e)) return c;
  const bool relative = kt != KS_GAUSSIAN || c.F < 52;
  if (relative && nmin * c.ah < pow2(45 - c.F)) return c;
  c.small = relative ? 1 << 19 : 0;
  if (kt != KS_GAUSSIAN && c.F < 43) return c;
  c.pre = max(0, 43 - c.F);
  c.lim = c.F < 54 ? (int)(1021u << (c.F - 32)) : 0x7fffffff;
  c.end = c.F < 53 ? (int)(1088u << (c.F - 32)) : 0x7fffffff;
  c.fixed = 1;
  return c;
}

// The part of the frame that the kernel alone sets (alpha 0: no fixed-point
// form).  Gaussian: y = alpha^2 d2.  Laplace: exponents up to 64 (P <= 128 keeps
// pow_neg_half's products in 32 bits).
inline CallParam kernel_frame(const KParams &kp)
{
  CallParam c{};
  if (kp.type == KS_GAUSSIAN) {
    const double c2 = -kp.scal * 1.4426950408889634;
    if (!(c2 > 0x1p-300 && c2 < 0x1p300)) return c;
    c.alpha = sqrt(c2);
    c.ah = c.alpha * c.alpha;
    c.al = fma(c.alpha, c.alpha, -c.ah);
  } else if (kp.type == KS_GAUSSIAN_VAR_BANDWIDTH) {
    c.alpha = c.ah = 1.0;
  } else if (kp.type == KS_LAPLACE) {
    const double P = -2.0 * kp.powe;
    if (!(P >= 1.0 && P <= 128.0 && P == rint(P))) return c;
    c.alpha = c.ah = 1.0;
    c.pw.p8 = (int)P << 8;
    const uint64_t q = (uint64_t)(0.5L * P * 1.442695040888963407359924681001892137L * 0x1p56L);
    c.pw.qh = (uint32_t)(q >> 32);
    c.pw.ql = (uint32_t)q;
  }
  return c;
}
__host__ __device__ constexpr bool has_frame(int kt)
{
  return kt == KS_GAUSSIAN || kt == KS_GAUSSIAN_VAR_BANDWIDTH || kt == KS_LAPLACE;
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
    // to nearest, ties to even: points on a grid of 2^-54 (uniform generators)
    // have a tie in every second coordinate, and rounding these up showed as a
    // bias of x.y
    X = (live && fld != 0 && sh <= 54) ? (X + ((1ull << sh) >> 1) - (sh > 0 ? ~(X >> sh) & 1ull : 0ull)) >> sh : 0ull;
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

// What decides how well a point's digits hold its inner products (x.y of the kernels
// without norms).  With x_p = xi_p 2^e the error of W is about 2^-54 of 2^(e_i + e_j)
// (|xi|^2 + |eta|^2)^1/2, rms: nothing beside sum |x_p y_p| of ordinary points, all of it
// where the large coordinates of one point meet zeros or small ones of the other
// ((1e20, 1) and (1e-20, 1)).  Sound without a look at W are pairs of
//   coarse points: 26 bits below 2^e (three digits) hold every coordinate; W is exact;
//   large ones (k up to 128: one or two roundings to W's unit): every coordinate that is
//     not 0 is at least 2^-3, so that |xi_p eta_p| >= 2^-6 for each p that both have;
//   dense ones: three quarters of the coordinates or more are at least 2^-5, so that half
//     of them are in both points;
//   any with a coordinate of at least 2^-3 in both (k up to 8, whose points often have a
//     small one: a mask of them.  Polynomial, 16384 x 16384 normal points, k = 7: 4.8 -> 2.6 ms).
// Of other pairs dot_cols forms those with a small W directly: |W| < 2^-4 2^c, c the larger
// class, 2^c >= |xi| (and the share of W's own roundings in long rows).
struct HeldStat {
  int large3, large5;       // coordinates of at least 2^-3, 2^-5
  int count;                // that are not 0
  int sq;                   // |xi|^2 2^16, rounded down
  int fine;                 // one needs more than 26 bits
  int mask;                 // the first eight of at least 2^-3
};
__device__ __forceinline__ void held_stat(const double (&v)[8], int e, bool first, HeldStat &t)
{
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const uint64_t b = (uint64_t)__double_as_longlong(v[q]) & 0x7fffffffffffffffull;
    const uint64_t M = (b & 0xfffffffffffffull) | 0x10000000000000ull;
    const int sh = e + 1022 - (int)(b >> 52);          // 0 and more; xi = M 2^-(53 + sh)
    const int top = sh < 8 ? (int)(M >> (45 + sh)) : 0;
    t.large3 += sh < 3;
    if (first) t.mask |= sh < 3 ? 1 << q : 0;
    t.large5 += sh < 5;
    t.count += b != 0;
    t.sq += top * top;
    t.fine |= b != 0 && (sh > 25 || (M & ((1ull << (27 + sh)) - 1)) != 0);
  }
}
// The bits and class of a point's exponent word.
__device__ __forceinline__ int held_bits(const HeldStat &t, int k, int kpad)
{
  int c = t.sq <= 1 << 16 ? 0 : (17 - __clz(t.sq - 1)) / 2;            // 4^c >= |xi|^2
  c = max(c, kpad > 512 ? 3 : kpad > 256 ? 1 : 0);
  return (t.fine ? NOT_COARSE : 0) | (t.large3 < t.count || kpad > 128 ? NOT_LARGE : 0) |
         (4 * t.large5 < 3 * k ? NOT_DENSE : 0) | (k <= EMASK_K ? t.mask << EMASK : 0) | c << ECLASS;
}

// One block per 32 points: lane = point, each warp a group of eight coordinates
// (then every eighth one; the list form's blocks have no more warps than groups).  Reads 64 bytes a thread, writes 16-byte row
// segments, consecutive points side by side (512 contiguous bytes a warp).
static __global__ void __launch_bounds__(256) slice_kernel(SliceArgs a)
{
  __shared__ uint32_t s_max[8][32];
  __shared__ HeldStat s_held[8][32];
  __shared__ double s_norm[8][32];
  __shared__ CallParam s_cp;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int nbA = a.nta * (BM / 32);
  launch_dependents();
  wait_primary();
  const bool listed = a.tp != nullptr;
  bool fixed = false;
  if (!listed && blockIdx.x == 0 && threadIdx.x == 0) *a.next_item = 0;
  if (listed) {
    // (below, from the tile's task)
  } else if (a.nscan >= 0) {
    // every block folds the scan's partials (at most one per thread) or, for
    // few points, scans them all itself
    ScanPart r{0, ~0u, 0, 0};
    if (a.nscan == 0) r = scan_points<2>(a, 0, a.m, 0, a.n, a.hi, a.hj, 0, 1);
    else if ((int)threadIdx.x < a.nscan) r = a.scan[threadIdx.x];
    r = scan_fold(r);
    if (threadIdx.x == 0) {
      s_cp = call_param(r, a.frame, a.kt, a.kpad);
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
  int pt = tile * rows + r, kt = a.kt;     // position in the call's maps
  bool valid = pt < (side ? a.n : a.m);
  const int slot = pt;                     // row of the metadata
  const double *hv = side ? a.hj : a.hi;
  if (listed) {
    const int2 tl = side ? a.tilesB[tile] : a.tilesA[tile];
    const TaskParam *T = a.tp + (side ? a.taskB[tile] : a.taskA[tile]);
    pt = tl.x + r;
    valid = r < tl.y;
    kt = T->kp.type;
    hv = side ? T->kp.hj : T->kp.hi;
    if (has_frame(kt)) {
      if (threadIdx.x == 0) s_cp = T->cp;
      __syncthreads();
      fixed = s_cp.fixed != 0;
    }
  }
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

  double v[8], norm = 0.0;
  uint32_t mh = 0;
  const int nw = blockDim.x >> 5;
  const bool dots = !kt_uses_norms(kt);
  for (int kg = wp; kg < kgs; kg += nw) {
    load8(kg, v);
    if (!dots) {
#pragma unroll
      for (int q = 0; q < 8; q++) norm = fma(v[q], v[q], norm);
    }
    if (!fixed) {
#pragma unroll
      for (int q = 0; q < 8; q++)
        mh = max(mh, ((uint32_t)__double2hiint(v[q]) & 0x7fffffffu) | (__double2loint(v[q]) != 0 ? 1u : 0u));
    }
  }
  int e = fixed ? s_cp.e : 0;
  bool flag = false;
  s_max[wp][lane] = mh;
  s_norm[wp][lane] = norm;
  __syncthreads();
  if (!fixed) {
#pragma unroll
    for (int q = 0; q < 8; q++)
      if (q < nw) mh = max(mh, s_max[q][lane]);
    if (mh) {
      const int fld = (int)(mh >> 20);
      e = fld - 1022;                     // |x_p| < 2^e
      flag = fld == 0 || fld == 0x7ff || e > ELIM || e < -ELIM;
      if (flag) e = 0;
    }
  }
  uint8_t *base = side ? a.imgB + (size_t)tile * btile_bytes(a.kpad, a.nr) : a.imgA + (size_t)tile * op_bytes(BM, a.kpad);
  const bool once = kgs <= nw;             // each thread's only group is still in registers
  HeldStat held{};
  for (int kg = wp; kg < kgs; kg += nw) {
    if (!once) load8(kg, v);
    if (fixed) {
#pragma unroll
      for (int q = 0; q < 8; q++) v[q] *= mul;
    }
    if (dots) held_stat(v, e, kg == 0, held);
    uint4 out[NS];
    slice8(v, e, !flag, out);
    const int c = kg / gpc, kgc = kg - c * gpc;
    // targets: slice, then k-group, row; sources: k-group, then slice, row
    uint8_t *dst = base + (size_t)c * op_bytes(rows, kc) + (size_t)kgc * (side ? NS : 1) * rows * 16 + (size_t)r * 16;
    const size_t step = side ? (size_t)rows * 16 : (size_t)rows * kc * 2;
#pragma unroll
    for (int s = 0; s < NS; s++) *(uint4 *)(dst + s * step) = out[s];
  }

  if (dots) {
    s_held[wp][lane] = held;
    __syncthreads();
  }
  if (wp == 0) {
    int bits = flag ? NOT_HELD : 0;
    if (dots && !flag && mh) {                // (points of zeros only: W is exact)
      for (int q = 1; q < nw; q++) {
        const HeldStat &t = s_held[q][lane];
        held.large3 += t.large3; held.large5 += t.large5; held.count += t.count; held.sq += t.sq; held.fine |= t.fine;
      }
      bits = held_bits(held, a.k, a.kpad);
    }
    const bool norms = !dots, varbw = kt == KS_GAUSSIAN_VAR_BANDWIDTH;
    double nn = (valid && norms) ? (side ? a.XB2[p] : a.XA2[p]) : 0.0;
    if (norms) {
      // the point's own norm summed in any order, or another one
      for (int q = 1; q < nw; q++) norm += s_norm[q][lane];
      if (!(fabs(norm - nn) <= norm * ((double)(a.k + 16) * 0x1p-52) + 0x1p-1060)) bits |= NORM_GIVEN;
    }
    if (fixed) {
      const double y = fma(nn, s_cp.ah, nn * s_cp.al) * ldexp(1.0, s_cp.F);
      nn = __longlong_as_double(__double2ll_rn(y));
    }
    const double h = (valid && varbw) ? hv[p] : 0.0;
    uint64_t hb = (uint64_t)__double_as_longlong(h);
    if (fixed && varbw) {
      // the factor (a row's times log2(e) / 2) as a 64-bit mantissa and an
      // exponent; the words are kept as integers (as FP64 some would be NaN)
      const double f = valid ? h : 1.0;
      hb = (uint64_t)__double_as_longlong(side ? f : f * (0.5 * 1.4426950408889634));
      e = (int)(hb >> 52) - 1023;
      hb = (hb | 0x10000000000000ull) << 11;
    }
    if (!side) {
      a.row_aa[slot] = nn;
      a.row_hi[slot] = hb;
      a.row_e[slot] = fixed ? (e & 0xfffff) | bits : (e + EBIAS) | bits;
      if (a.row_n) a.row_n[slot] = 0;
    } else {
      ColMeta *cm = (ColMeta *)(base + op_bytes(BN, a.kpad));
      cm->bb[r] = nn;
      cm->hj[r] = hb;
      cm->e[r] = fixed ? e : (e + EBIAS) | bits;
      const int any = (int)__reduce_or_sync(0xffffffffu, (unsigned)bits) & (NOT_HELD | NORM_GIVEN);
      if (lane == 0) { cm->flag = any; cm->pad[0] = cm->pad[1] = cm->pad[2] = 0; }
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
  const double *row_aa; const uint64_t *row_hi; const int *row_e;
  const double *XA, *XB, *XA2, *XB2;   // pools and maps, for pairs formed directly
  const int *amap, *bmap;
  int nxa, nxb;
  KParams kp;
  const CallParam *cp;
  double *partial;                  // [nsc][ldp]; several right-hand sides: [nrhs][nsc][GROUPS][ldp]
  int *row_n;                       // arrivals per row (nullptr: the list form)
  double *u; const int *umap;
  int ldp;
  int *err, *next_item;
  long long wait_limit;
  int stall;                        // test hook: the producer issues nothing (the waits run out)
  // list form
  const Item *tab;
  int ntab;
  const TaskParam *tp;
};

// Geometry of a work item: target tile, source tiles, list positions of its
// first row and column and how many are valid, the partial offset of row 0.
template <bool LISTED>
__device__ __forceinline__ Item item_geo(const TileArgs &a, int item)
{
  if constexpr (LISTED) return a.tab[item];
  Item g;
  g.a_tile = item % a.ntm;
  const int sc = item / a.ntm;
  g.b0 = sc * a.chunk_tiles;
  g.b1 = min(a.ntn, g.b0 + a.chunk_tiles);
  g.ia = g.a_tile * BM;
  g.rows = min(BM, a.m - g.ia);
  g.jb = g.b0 * BN;
  g.cols = a.n - g.jb;
  g.task = 0;
  g.out = (long long)sc * a.ldp + g.ia;
  return g;
}

struct __align__(16) SlicedSmem {
  uint64_t a_full, a_empty;
  uint64_t b_full[NSTAGE_RES], b_empty[NSTAGE_RES];
  uint64_t m_full[NMETA], m_empty[NMETA];
  uint64_t t_full[HALVES], t_empty[HALVES];
  uint64_t r_full[2], r_empty[2];       // row-sum exchange of the epilogue groups, by item parity
  uint64_t drain;
  double rsum[2][GROUPS - 1][BM];       // row sums of groups 1 .., by item parity
  TaskParam tslot[2];                   // list form: the items' task parameters, by item parity
  uint32_t tmem_base;
  int abort;
  int never;             // stays 0: an abort flag for the drain waits
  int islot[2];          // the current items (-1: no work left), by item parity
};

struct SmemLayout {
  bool resident;
  int kc, nch;               // k-chunk, chunks per tile
  int nstage;
  size_t a_chunk, b_chunk;   // operand bytes of one chunk (one source tile)
  size_t a_region, stage, meta, table;
};
__host__ __device__ inline SmemLayout smem_layout(int kpad, int nr, bool table)
{
  SmemLayout L;
  L.kc = kchunk(kpad);
  L.nch = kpad / L.kc;
  L.resident = L.nch == 1;
  L.nstage = L.resident ? NSTAGE_RES : NSTAGE_STR;
  L.a_chunk = op_bytes(BM, L.kc);
  L.b_chunk = op_bytes(BN, L.kc);
  L.a_region = L.resident ? L.a_chunk : 0;
  L.stage = L.resident ? L.b_chunk : L.a_chunk + HALVES * L.b_chunk;
  L.meta = colmeta_bytes(nr);
  L.table = table ? ETAB * sizeof(uint64_t) : 0;
  return L;
}
inline size_t smem_bytes(const SmemLayout &L)
{
  return 1024 + L.a_region + L.nstage * L.stage + NMETA * L.meta + L.table + sizeof(SlicedSmem) + 64;
}
static_assert(1024 + NS * (size_t)BM * KRES * 2 + NSTAGE_RES * NS * (size_t)BN * KRES * 2 + NMETA * colmeta_bytes(RMAX) +
                      ETAB * 8 + sizeof(SlicedSmem) + 64 <= SMEM_MAX,
              "sliced_tiles shared memory (resident)");
static_assert(1024 + NSTAGE_STR * NS * (size_t)(BM + HALVES * BN) * KST * 2 + NMETA * colmeta_bytes(RMAX) +
                      ETAB * 8 + sizeof(SlicedSmem) + 64 <= SMEM_MAX,
              "sliced_tiles shared memory (streaming)");

// The high word that takes the bias of combine's level 0 back out.
template <int SIGN>
__device__ __forceinline__ uint32_t combine_bias(int g) { return 0u - 0x4B400000u * (uint32_t)(SIGN * (1 << (4 + g))); }
// w + SIGN W of one pair, from its level sums, with g guard bits: four
// 32 x 32 + 64 bit multiply-adds and one into the high word.  Levels 4 to 6
// join in FP32 (their last bits lie below W's or near its last one).  Level 0, at
// most 2^22 over 64 coordinates, becomes an integer by adding 1.5 2^23 to it (w
// starts with combine_bias in its high word); the others, up to 2^24, need the
// conversion instruction.
template <int SIGN>
__device__ __forceinline__ long long combine(const uint32_t (&r)[LV], int g, long long w)
{
  const float f4 = SIGN * __int_as_float((127 + g) << 23), f5 = SIGN * __int_as_float((118 + g) << 23);   // 2^g, 2^(g-9)
  float v = fmaf(__uint_as_float(r[5]), f5, __uint_as_float(r[4]) * f4);
  v = fmaf(__uint_as_float(r[6]), SIGN * __int_as_float((109 + g) << 23), v);   // 2^(g-18)
  w = madws(__float2int_rn(v), 1, w);
  w = madws(__float2int_rn(__uint_as_float(r[3])), SIGN * (1 << (9 + g)), w);
  w = madws(__float2int_rn(__uint_as_float(r[2])), SIGN * (1 << (18 + g)), w);
  w = madws(__float2int_rn(__uint_as_float(r[1])), SIGN * (1 << (27 + g)), w);
  const int hi = (int)(w >> 32) + __float_as_int(__uint_as_float(r[0]) + 12582912.0f) * (SIGN * (1 << (4 + g)));
  return (long long)(((uint64_t)(uint32_t)hi << 32) | (uint32_t)w);
}

// 4 consecutive 32-bit columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t &a, uint32_t &b, uint32_t &c, uint32_t &d)
{
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(a), "=r"(b), "=r"(c), "=r"(d)
               : "r"(taddr)
               : "memory");
}

static __device__ __noinline__ double pow_call(double x, const KParams &kp) { return pow_class(x, kp); }
static __device__ __noinline__ double tanh_call(double x) { return tanh(x); }
static __device__ __noinline__ double dot_direct(const double *__restrict__ x, const double *__restrict__ y, int k)
{
  double s = 0.0;
  for (int p = 0; p < k; p++) s = fma(x[p], y[p], s);
  return s;
}
// x.y of a row with two others, in the order of the DFMA kernels, eight coordinates' loads at
// a time (each lane has rows of its own: whole 32-byte sectors).
static __device__ __noinline__ double2 dot_direct2(const double *__restrict__ x, const double *__restrict__ y0,
                                                   const double *__restrict__ y1, int k)
{
  double s0 = 0.0, s1 = 0.0;
  int p = 0;
  if ((k & 1) == 0 && (((uintptr_t)x | (uintptr_t)y0 | (uintptr_t)y1) & 15) == 0) {
    for (; p + 8 <= k; p += 8) {
      double2 a[4], b[4], c[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        a[q] = __ldg((const double2 *)(x + p) + q);
        b[q] = __ldg((const double2 *)(y0 + p) + q);
        c[q] = __ldg((const double2 *)(y1 + p) + q);
      }
#pragma unroll
      for (int q = 0; q < 4; q++) {
        s0 = fma(a[q].y, b[q].y, fma(a[q].x, b[q].x, s0));
        s1 = fma(a[q].y, c[q].y, fma(a[q].x, c[q].x, s1));
      }
    }
  }
#pragma unroll 4
  for (; p < k; p++) {
    const double v = __ldg(x + p);
    s0 = fma(v, __ldg(y0 + p), s0);
    s1 = fma(v, __ldg(y1 + p), s1);
  }
  return make_double2(s0, s1);
}

// |x_i - y_j|^2 from the pool coordinates.  For points that agree to about
// 2^-39 of their norms |x|^2 + |y|^2 - 2 x.y leaves only the rounding of the
// given norms, which the DFMA form's own rounding cancels when the norms were
// summed in the same order (coincident points: exactly); an exact x.y does
// not, so such pairs are formed directly.
static __device__ __noinline__ double near_d2(const TileArgs &a, int i, int j, double d2)
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

// The same from norms that are not the points' own: as given.
static __device__ __noinline__ double given_d2(const TileArgs &a, int i, int j)
{
  const int pa = pool_clamp(a.amap, i, a.nxa), pb = pool_clamp(a.bmap, j, a.nxb);   // flagged by slice_kernel
  const double *x = a.XA + (size_t)pa * a.k, *y = a.XB + (size_t)pb * a.k;
  double s = 0.0;
#pragma unroll 1   // (what a function called here needs in registers, every caller sets aside)
  for (int p = 0; p < a.k; p++) s = fma(x[p], y[p], s);
  return fma(-2.0, s, a.XA2[pa]) + a.XB2[pb];
}

// Row side of a pair: metadata, and the row's position in the call's maps (-1:
// a padding row).
struct RowMeta {
  double aa, hi;
  int e, i;
};

// Kernel value from the inner product: the functions of kfun64, with the
// exponentials through exp2_neg and the comparisons of rare cases on the
// doubles' high words (an FP64 comparison costs as much as an FP64 add).
// cfold: y 2^53 per unit of d2 (Gaussian), times h_i (variable bandwidth).
template <int KT>
__device__ __forceinline__ double kvalue(const TileArgs &a, const KParams &kp, int j, double dot, const RowMeta &am,
                                         double bb, double hj, double cfold, uint32_t tab, const ColMeta *cm)
{
  double d2 = 0.0;
  bool near = false;
  if constexpr (kt_uses_norms(KT)) {
    d2 = fma(-2.0, dot, am.aa) + bb;
    // d2 at most about 2^-39 of the larger norm, by the high words
    near = __double2hiint(d2) <= max(__double2hiint(am.aa), __double2hiint(bb)) - (39 << 20);
    if (KT != KS_LAPLACE && near && am.i >= 0 && !((am.e | cm->flag) & NORM_GIVEN)) d2 = near_d2(a, am.i, j, d2);
  }
  if constexpr (KT == KS_GAUSSIAN || KT == KS_GAUSSIAN_VAR_BANDWIDTH) {
    // max(d2, 0), also of NaN (fmax): anything not in (0, inf] becomes 0
    if ((uint32_t)__double2hiint(d2) > 0x7ff00000u) d2 = 0.0;
    if constexpr (KT == KS_GAUSSIAN) return exp2_neg64(d2 * cfold, tab);
    else return exp2_neg64((d2 * cfold) * hj, tab);
  } else if constexpr (KT == KS_POLYNOMIAL) {
    const double c = fma(dot, kp.scal, kp.cons);
    if (kp.pmode == POW_INT && kp.pint >= 2 && kp.pint <= 4) {
      bool ok;
      const double v = kp.pint == 2 ? pow_int<2>(c, ok) : kp.pint == 3 ? pow_int<3>(c, ok) : pow_int<4>(c, ok);
      if (ok) return v;
    }
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

// Where a thread stands in an item: its row's position in the call's maps (-1: a
// padding row), and for a tile its first column's position and how many are
// valid.  Formed anew where it is needed (the common path does not).
struct Place {
  int i, j0, nv;
};
template <bool LISTED>
__device__ __forceinline__ Place place_of(const TileArgs &a, int item, int row, int tj, int c0)
{
  const Item g = item_geo<LISTED>(a, item);
  const int done = (tj - g.b0) * BN + c0;
  return Place{row < g.rows ? g.ia + row : -1, g.jb + done, min(COLS, g.cols - done)};
}

// A pair's distance where the fixed-point one does not do: nearly coincident
// points (D at most about 2^-38 of the norms), two small norms.
__device__ __forceinline__ double direct_d2(const TileArgs &a, const CallParam &cp, long long D, long long A, int i, int j,
                                            bool given)
{
  if (D <= (A >> 38) || (cp.small && (int)(A >> 32) < cp.small)) return given ? given_d2(a, i, j) : near_d2(a, i, j, 0.0);
  return (double)D * ldexp(1.0, -cp.F);
}

// The fixed-point value of a pair outside the common range.  j: the column's
// position (-1: a padding column).  A's top bit: one of the norms
// is not its point's own (NORM_GIVEN).
template <int KT>
__device__ __noinline__ double rare_value(const TileArgs &a, const KParams &kp, const CallParam &cp, uint32_t tab,
                                          long long y, long long A, int i, int j)
{
  if (i < 0 || j < 0) return 0.0;   // padding: its weight is 0
  const bool given = A < 0;
  A &= 0x7fffffffffffffffll;
  if constexpr (KT == KS_GAUSSIAN) {
    if (y <= (A >> 38) || (cp.small && (int)(A >> 32) < cp.small))
      y = __double2ll_rn((given ? given_d2(a, i, j) : near_d2(a, i, j, 0.0)) * cp.ah * ldexp(1.0, cp.F));
    if (y <= 0) return 1.0;
    if ((int)(y >> 32) >= cp.end) return 0.0;
    return exp2_neg_deep((uint64_t)y << cp.pre, (int)(y >> 32) >= cp.lim, exp_frame(max(cp.F, 43), tab));
  } else {
    double d2 = direct_d2(a, cp, y, A, i, j, given);
    if constexpr (KT == KS_LAPLACE) {
      // (two coincident points have the same norm)
      if (d2 < fmax(1e-15, kp.coinc * 2.0 * ((double)A * ldexp(1.0, -cp.F)))) d2 = 1.79e308;
      return pow_call(d2, kp);      // the row's sum is multiplied by scal
    } else {
      const int pa = pool_clamp(a.amap, i, a.nxa), pb = pool_clamp(a.bmap, j, a.nxb);   // flagged by slice_kernel
      return exp2_neg64(((fmax(d2, 0.0) * (0.5 * 1.4426950408889634 * 0x1p53)) * kp.hi[pa]) * kp.hj[pb], tab);
    }
  }
}

// One thread's columns of a tile in the fixed-point form: W holds the distance D
// (the Gaussian: y); A: the row's norm in the same units; i0: its metadata.
// Columns outside the common range are left for a loop in which each lane takes
// a column of its own, since their loads take long.
template <int KT, int NR, bool LISTED>
__device__ __forceinline__ void fixed_cols(const TileArgs &a, const KParams &kp, const CallParam &cp, const ExpFrame &E,
                                           long long (&W)[COLS], long long A, const ColMeta *cm, uint32_t cmS, int item,
                                           int row, int i0, int tj, int c0, double (&sum)[NR])
{
  const uint32_t wS = cmS + (uint32_t)offsetof(ColMeta, w);
  const int lim = cp.lim;
  uint32_t mask = 0;
  // a row of small norm: its columns of small norm too (bb >= 0)
  if ((int)(A >> 32) < cp.small) {
#pragma unroll 1
    for (int c = 0; c < COLS; c++)
      if (__double2hiint(cm->bb[c0 + c]) < cp.small) mask |= 1u << c;
  }
  if constexpr (KT == KS_GAUSSIAN) {
    // straight-line code where every y of the thread's columns lies in [2^32,
    // 1021 2^F): independent chains for the schedulers
    bool rare = mask != 0;
#pragma unroll
    for (int c = 0; c < COLS; c++) rare |= (uint32_t)((int)(W[c] >> 32) - 1) >= (uint32_t)(lim - 1);
    if (cp.pre && !rare) {
#pragma unroll
      for (int c = 0; c < COLS; c++) W[c] <<= cp.pre;
    }
    if (!rare) {
#pragma unroll
      for (int c = 0; c < COLS; c += 2) {
        const double k0 = exp2_neg((uint64_t)W[c], E), k1 = exp2_neg((uint64_t)W[c + 1], E);
#pragma unroll
        for (int r = 0; r < NR; r++) {
          if (r > 0 && r >= a.nrhs) continue;
          double w0, w1;
          lds2(wS + (r * BN + c) * 8, w0, w1);
          sum[r] = fma(k1, w1, fma(k0, w0, sum[r]));
        }
      }
      return;
    }
    // the columns in the range (values of 1088 and more are 0, times w)
    const int yend = cp.end;
#pragma unroll
    for (int c = 0; c < COLS; c += 2) {
      double kv[2];
      bool good[2];
#pragma unroll
      for (int s = 0; s < 2; s++) {
        const int yh = (int)(W[c + s] >> 32);
        good[s] = yh > 0 && !(mask >> (c + s) & 1u);
        kv[s] = exp2_neg_deep((uint64_t)W[c + s] << cp.pre, yh >= lim, E);
        kv[s] = yh < yend ? kv[s] : 0.0;
        mask = good[s] ? mask : mask | (1u << (c + s));
      }
#pragma unroll
      for (int r = 0; r < NR; r++) {
        if (r > 0 && r >= a.nrhs) continue;
        double w0, w1;
        lds2(wS + (r * BN + c) * 8, w0, w1);
        if (good[0]) sum[r] = fma(kv[0], w0, sum[r]);
        if (good[1]) sum[r] = fma(kv[1], w1, sum[r]);
      }
    }
  } else {
    uint64_t Mi = 0;
    int ei = 0;
    if constexpr (KT == KS_GAUSSIAN_VAR_BANDWIDTH) {
      Mi = a.row_hi[i0];
      ei = a.row_e[i0] << 12 >> 12;
    }
    const PowFrame pw = cp.pw;
    const int F = cp.F;
#pragma unroll
    for (int c = 0; c < COLS; c += 2) {
      double kv[2];
      bool good[2];
#pragma unroll
      for (int s = 0; s < 2; s++) {
        const long long D = W[c + s];
        good[s] = (int)(D >> 32) > 0 && !(mask >> (c + s) & 1u);
        if constexpr (KT == KS_LAPLACE) {
          bool ok;
          kv[s] = pow_neg_half((uint64_t)D, F, pw, E, ok);
          good[s] = good[s] && ok;
        } else {
          uint32_t zh;
          kv[s] = exp2_neg_scaled((uint64_t)D, F, Mi, cm->hj[c0 + c + s],
                                  ei + cm->e[c0 + c + s], E, zh);
          if (good[s] && zh >= 1088u << 21) kv[s] = 0.0;      // beyond 2^-1088: 0, times w
          else good[s] = good[s] && zh > 0;
        }
        mask = good[s] ? mask : mask | (1u << (c + s));
      }
#pragma unroll
      for (int r = 0; r < NR; r++) {
        if (r > 0 && r >= a.nrhs) continue;
        double w0, w1;
        lds2(wS + (r * BN + c) * 8, w0, w1);
        if (good[0]) sum[r] = fma(kv[0], w0, sum[r]);
        if (good[1]) sum[r] = fma(kv[1], w1, sum[r]);
      }
    }
  }
  if (!mask) return;
  const Place P = place_of<LISTED>(a, item, row, tj, c0);
  // (the row's place in the metadata, formed anew)
  if ((a.row_e[item_geo<LISTED>(a, item).a_tile * BM + row] | cm->flag) & NORM_GIVEN)
    A = (long long)((uint64_t)A | 0x8000000000000000ull);
  for (; mask; mask &= mask - 1) {
    const int c = __ffs(mask) - 1;
    long long y = W[0];
#pragma unroll
    for (int q = 1; q < COLS; q++) y = c == q ? W[q] : y;
    const double kv = rare_value<KT>(a, kp, cp, E.tab, y, A, P.i, c < P.nv ? P.j0 + c : -1);
#pragma unroll
    for (int r = 0; r < NR; r++) {
      if (r > 0 && r >= a.nrhs) continue;
      double w0;
      lds1(wS + (r * BN + c) * 8, w0);
      sum[r] = fma(kv, w0, sum[r]);
    }
  }
}

// A call's copy of kvalue, for the pairs formed directly.
template <int KT>
__device__ __noinline__ double kvalue_call(const TileArgs &a, const KParams &kp, double dot)
{
  return kvalue<KT>(a, kp, 0, dot, RowMeta{}, 0.0, 0.0, 0.0, 0, nullptr);
}

// The columns that dot_cols left (a bit each; the whole warp calls).  Few pairs among the
// lanes: four at a time, each by eight lanes, since a lane on its own waits for its loads at
// every eighth coordinate (one point of a 65536-point tile row held its warp, and with it
// the tile, for 20 000 cycles a tile).  Many: each lane its own, two at a time.
template <int KT, int NR>
__device__ __noinline__ void direct_cols(const TileArgs &a, const KParams &kp, int i, const ColMeta *cm, int c0,
                                         int j0, uint32_t direct, double (&sum)[NR])
{
  const unsigned full = 0xffffffffu;
  const int total = (int)__reduce_add_sync(full, __popc(direct));
  if (total == 0) return;
  const int trips = ((int)__reduce_max_sync(full, __popc(direct)) + 1) / 2;
  const double *x = a.XA + (direct ? (size_t)pool_clamp(a.amap, i, a.nxa) * a.k : 0);
  if (total > trips * min(32, 4 + a.k / 4)) {
    while (direct) {
      const int ca = __ffs(direct) - 1;
      direct &= direct - 1;
      const int cb = direct ? __ffs(direct) - 1 : -1;
      direct &= direct - 1;
      const double *y0 = a.XB + (size_t)pool_clamp(a.bmap, j0 + ca, a.nxb) * a.k;
      const double *y1 = cb < 0 ? y0 : a.XB + (size_t)pool_clamp(a.bmap, j0 + cb, a.nxb) * a.k;
      const double2 dot = dot_direct2(x, y0, y1, a.k);
      const double ka = kvalue_call<KT>(a, kp, dot.x), kb = cb < 0 ? 0.0 : kvalue_call<KT>(a, kp, dot.y);
#pragma unroll
      for (int r = 0; r < NR; r++) {
        if (r > 0 && r >= a.nrhs) continue;
        sum[r] = fma(ka, cm->w[r][c0 + ca], sum[r]);
        if (cb >= 0) sum[r] = fma(kb, cm->w[r][c0 + cb], sum[r]);
      }
    }
    return;
  }
  const int lane = threadIdx.x & 31, sub = lane & 7;
  for (int left = total; left > 0; left -= 4) {
    int src = 0, col = 0, mine[4];               // my group's pair; my own pairs, by group
#pragma unroll
    for (int g = 0; g < 4; g++) {
      const unsigned b = __ballot_sync(full, direct != 0);
      const int l = b ? __ffs(b) - 1 : 0, c = __shfl_sync(full, __ffs(direct) - 1, l);
      mine[g] = b && lane == l ? c : -1;
      if (b && lane == l) direct &= direct - 1;
      if (g == lane >> 3) { src = l; col = b ? c : -1; }
    }
    const double *xs = (const double *)__shfl_sync(full, (unsigned long long)x, src);
    double s = 0.0;
    const double *y = a.XB + (col >= 0 ? (size_t)pool_clamp(a.bmap, j0 + col, a.nxb) * a.k : 0);
    if (col >= 0) {
#pragma unroll 8
      for (int p = sub; p < a.k; p += 8) s = fma(__ldg(xs + p), __ldg(y + p), s);
    }
#pragma unroll
    for (int d = 4; d; d >>= 1) s += __shfl_xor_sync(full, s, d);
    // (an overflow's sign is that of the sum in order; two partial sums' may cancel to NaN)
    if (!(fabs(s) <= 1.79e308)) s = dot_direct(xs, y, a.k);
    const double kv = kvalue_call<KT>(a, kp, s);
#pragma unroll
    for (int g = 0; g < 4; g++) {
      const double kg = __shfl_sync(full, kv, 8 * g);
      if (mine[g] < 0) continue;
#pragma unroll
      for (int r = 0; r < NR; r++)
        if (r == 0 || r < a.nrhs) sum[r] = fma(kg, cm->w[r][c0 + mine[g]], sum[r]);
    }
  }
}

// One thread's columns of a tile through x.y in FP64; W holds SIGN W.  slow: the digits
// of the rows and of the tile's points do not promise every x.y (NOT_HELD).  A pair of a
// point without digits is formed directly; for the kernels without norms, pairs whose W is
// too small for their digits are left to direct_cols.
template <int KT, int NR, int SIGN>
__device__ __forceinline__ void dot_cols(const TileArgs &a, const KParams &kp, const long long (&W)[COLS],
                                         const RowMeta &am, const ColMeta *cm, int c0, const Place &P, int gb, bool slow,
                                         uint32_t tab, double (&sum)[NR])
{
  constexpr bool DOTS = !kt_uses_norms(KT);
  double cfold = 0.0;
  if (KT == KS_GAUSSIAN) cfold = -kp.scal * (1.4426950408889634 * 0x1p53);
  if (KT == KS_GAUSSIAN_VAR_BANDWIDTH) cfold = am.hi * (0.5 * 1.4426950408889634 * 0x1p53);
  uint32_t direct = 0;
  if (DOTS && slow && am.i >= 0) {
#pragma unroll
    for (int c = 0; c < COLS; c++) {
      const int ej = cm->e[c0 + c];
      // (a point without digits: W = 0)
      const int lim = 1 << (16 + gb + (max(am.e, ej) >> ECLASS));          // 2^-4 2^class, high word
      if (c < P.nv && ((am.e | ej) & NOT_HELD) == NOT_HELD &&
          !(am.e & ej & (((1 << EMASK_K) - 1) << EMASK)) &&
          (uint32_t)((int)(W[c] >> 32) + lim) < 2u * (uint32_t)lim)
        direct |= 1u << c;
    }
  }
#pragma unroll
  for (int c = 0; c < COLS; c++) {
    if (c < P.nv && (!DOTS || !(direct >> c & 1u))) {
      const int ej = cm->e[c0 + c], j = P.j0 + c;
      double dot = to_double(SIGN * W[c]);
      dot = __hiloint2double(__double2hiint(dot) + (W[c] != 0 ? (int)((uint32_t)(am.e + ej - 52 - gb) << 20) : 0),
                             __double2loint(dot));
      if (!DOTS && slow && ((am.e | ej) & NOT_HELD) == NOT_HELD && am.i >= 0) {
        const int pa = pool_clamp(a.amap, am.i, a.nxa), pb = pool_clamp(a.bmap, j, a.nxb);   // flagged by slice_kernel
        dot = dot_direct(a.XA + (size_t)pa * a.k, a.XB + (size_t)pb * a.k, a.k);
      }
      const double kv = kvalue<KT>(a, kp, j, dot, am, cm->bb[c0 + c],
                                    __longlong_as_double((long long)cm->hj[c0 + c]), cfold, tab, cm);
#pragma unroll
      for (int r = 0; r < NR; r++)
        if (r == 0 || r < a.nrhs) sum[r] = fma(kv, cm->w[r][c0 + c], sum[r]);
    }
  }
  if (DOTS && slow) {
    double t[NR];           // (of its own: sum stays in registers)
#pragma unroll
    for (int r = 0; r < NR; r++) t[r] = sum[r];
    direct_cols<KT, NR>(a, kp, am.i, cm, c0, P.j0, direct, t);
#pragma unroll
    for (int r = 0; r < NR; r++) sum[r] = t[r];
  }
}

constexpr bool uses_table(int kt) { return has_frame(kt); }

// A thread's partial sums of row i are stored; the last of the row's parts
// (count in all) adds them in order into u.  (A reduction kernel of its own cost
// a launch: 3 us of a 40 us call.)
template <int NR>
__device__ __forceinline__ void row_done(const TileArgs &a, int i, int parts)
{
  if (parts > 1) {
    __threadfence();
    if (atomicAdd(&a.row_n[i], 1) != parts - 1) return;
    __threadfence();
  }
  const size_t q = (size_t)(a.umap ? a.umap[i] : i) * (NR > 1 ? a.nrhs : 1);
#pragma unroll
  for (int r = 0; r < NR; r++) {
    if (r > 0 && r >= a.nrhs) continue;
    double s = 0.0;
    for (int c = 0; c < parts; c++) s += __ldcg(&a.partial[((size_t)r * parts + c) * a.ldp + i]);
    a.u[q + r] += s;
  }
}

// G: guard bits of the resident layouts (3; with a frame and k > 32: 2), -1: streaming.
template <int KT, int NR, int G, bool LISTED>
__global__ void __launch_bounds__(NTHREADS, 1) sliced_tiles(TileArgs a)
{
  constexpr uint32_t TBUF = LV * BN;                // columns of one accumulator buffer
  constexpr bool STREAM = G < 0;
  constexpr bool TABLE = uses_table(KT);
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *sm = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const SmemLayout L = smem_layout(a.kpad, NR, TABLE);
  uint8_t *sA = sm, *sStage = sm + L.a_region, *sMeta = sStage + L.nstage * L.stage;
  uint64_t *sTab = (uint64_t *)(sMeta + NMETA * L.meta);
  SlicedSmem *S = (SlicedSmem *)((uint8_t *)sTab + L.table);
  volatile int *abort = &S->abort;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int items = LISTED ? a.ntab : a.ntm * a.nsc;

  if (threadIdx.x == 0) {
    mbar_init(&S->a_full, 1);
    mbar_init(&S->a_empty, 1 + EPI_WARPS);
    for (int s = 0; s < NSTAGE_RES; s++) { mbar_init(&S->b_full[s], 1); mbar_init(&S->b_empty[s], 1); }
    for (int s = 0; s < NMETA; s++) { mbar_init(&S->m_full[s], 1); mbar_init(&S->m_empty[s], HALF_WARPS); }
    for (int h = 0; h < HALVES; h++) { mbar_init(&S->t_full[h], 1); mbar_init(&S->t_empty[h], HALF_WARPS); }
    for (int b = 0; b < 2; b++) {   // one arrive per thread: groups 1 .. fill, group 0 empties
      mbar_init(&S->r_full[b], 32 * 4 * (GROUPS - 1));
      mbar_init(&S->r_empty[b], 32 * 4);
    }
    mbar_init(&S->drain, 1);
    S->abort = 0;
    S->never = 0;
    fence_mbar_init();
  }
  if (warp == 0) { tmem_alloc(&S->tmem_base, TMEM_COLS); tmem_relinquish(); }
  if constexpr (TABLE)
    for (int i = threadIdx.x; i < ETAB; i += NTHREADS) sTab[i] = g_exp_table.v[i];
  wait_primary();   // slice_kernel's results from here on
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = S->tmem_base;

  if (warp == 0) {
    // ---------------- producer ----------------
    if (lane == 0 && !a.stall) {
      int g = 0, tt = 0, a_issued = -1;
      int b_last[NSTAGE_RES], m_last[NMETA];
      for (int s = 0; s < NSTAGE_RES; s++) b_last[s] = -1;
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
        const Item G_ = item_geo<LISTED>(a, item);
        const int t0 = G_.b0, t1 = G_.b1;
        const uint8_t *imgA = a.imgA + (size_t)G_.a_tile * op_bytes(BM, a.kpad);
        // (a task slot was last read for item it - 2, which every epilogue warp
        // has finished once it arrived on a_empty for item it - 1)
        const uint32_t tp_bytes = LISTED ? (uint32_t)sizeof(TaskParam) : 0u;
        const uint32_t a_bytes = STREAM ? 0u : (uint32_t)L.a_chunk;
        if (a_bytes + tp_bytes) mbar_arrive_expect_tx(&S->a_full, a_bytes + tp_bytes);
        else mbar_arrive(&S->a_full);
        if (a_bytes) bulk_g2s(sA, imgA, a_bytes, &S->a_full);
        if (tp_bytes) bulk_g2s(&S->tslot[it & 1], a.tp + G_.task, tp_bytes, &S->a_full);
        a_issued = it;
        // resident: a stage per source tile; streaming: a stage per k-chunk of
        // the targets and of two source tiles
        const int step = STREAM ? HALVES : 1;
        for (int tj = t0; tj < t1 && !stop; tj += step) {
          const uint8_t *imgB = a.imgB + (size_t)tj * bt;
          const int nt = min(step, t1 - tj);
          // the metadata first: the epilogue waits for it before it takes the
          // first accumulators, which the copies below wait for in turn
          for (int q = 0; q < nt && !stop; q++, tt++) {
            const int ms = tt % NMETA, mu = tt / NMETA;
            if (mu > 0 && !mbar_wait(&S->m_empty[ms], (mu - 1) & 1, abort, a.wait_limit)) { stop = true; break; }
            mbar_arrive_expect_tx(&S->m_full[ms], (uint32_t)L.meta);
            bulk_g2s(sMeta + ms * L.meta, imgB + q * bt + op_bytes(BN, a.kpad), (uint32_t)L.meta, &S->m_full[ms]);
            m_last[ms] = mu;
          }
          for (int c = 0; c < L.nch && !stop; c++, g++) {
            const int st = g % L.nstage, u = g / L.nstage;
            if (u > 0 && !mbar_wait(&S->b_empty[st], (u - 1) & 1, abort, a.wait_limit)) { stop = true; break; }
            uint8_t *dst = sStage + st * L.stage;
            mbar_arrive_expect_tx(&S->b_full[st], (uint32_t)((STREAM ? L.a_chunk : 0) + nt * L.b_chunk));
            if (STREAM) {
              bulk_g2s(dst, imgA + (size_t)c * L.a_chunk, (uint32_t)L.a_chunk, &S->b_full[st]);
              dst += L.a_chunk;
            }
            for (int q = 0; q < nt; q++)
              bulk_g2s(dst + q * L.b_chunk, imgB + q * bt + (size_t)c * L.b_chunk, (uint32_t)L.b_chunk, &S->b_full[st]);
            b_last[st] = u;
          }
        }
        item = next;
      }
      // On an abort, let the copies already issued land before the CTA exits.
      if (*abort) {
        volatile int *nev = &S->never;
        if (a_issued >= 0) mbar_wait(&S->a_full, a_issued & 1, nev, 1LL << 28);
        for (int s = 0; s < NSTAGE_RES; s++)
          if (b_last[s] >= 0) mbar_wait(&S->b_full[s], b_last[s] & 1, nev, 1LL << 28);
        for (int s = 0; s < NMETA; s++)
          if (m_last[s] >= 0) mbar_wait(&S->m_full[s], m_last[s] & 1, nev, 1LL << 28);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (whole warp, one elected lane issues) ----------------
    const unsigned full = 0xffffffffu;
    const uint64_t ablk = (uint64_t)(BM * L.kc * 2) >> 4;                           // one target slice
    const uint64_t astep = (2 * BM * 16) >> 4, bstep = (2 * NS * BN * 16) >> 4;     // 16 coordinates
    const int nks = L.kc / 16, gch = STREAM ? KRES / KST : 1;                       // chunks per accumulation
    int g = 0, use[HALVES] = {0, 0};
    bool stop = false;
    for (int it = 0; !stop; it++) {
      if (!__all_sync(full, *abort == 0 && mbar_wait(&S->a_full, it & 1, abort, a.wait_limit))) break;
      const int item = __shfl_sync(full, ((volatile int *)S->islot)[it & 1], 0);
      if (item < 0) break;
      const Item G_ = item_geo<LISTED>(a, item);
      const int t0 = G_.b0, t1 = G_.b1;
      const int step = STREAM ? HALVES : 1;
      for (int tj = t0; tj < t1 && !stop; tj += step) {
        for (int c = 0; c < L.nch && !stop; c++, g++) {
          const bool first = c % gch == 0, last = c % gch == gch - 1;
          const int st = g % L.nstage;
          if (!__all_sync(full, mbar_wait(&S->b_full[st], (g / L.nstage) & 1, abort, a.wait_limit))) { stop = true; break; }
          const uint32_t sb = smem_addr(sStage + st * L.stage);
          const uint64_t dA = desc_noswizzle(STREAM ? sb : smem_addr(sA), BM * 16, 128);
#pragma unroll
          for (int q = 0; q < (STREAM ? HALVES : 1); q++) {
            if (tj + q >= t1) continue;
            const int h = STREAM ? q : (tj - t0) & 1;      // the accumulator buffer
            if (first) {
              const int u = h ? use[1]++ : use[0]++;
              if (u > 0 && !__all_sync(full, mbar_wait(&S->t_empty[h], (u - 1) & 1, abort, a.wait_limit))) { stop = true; break; }
            }
            tc_fence_after();
            const uint64_t dB = desc_noswizzle(sb + (STREAM ? (uint32_t)(L.a_chunk + q * L.b_chunk) : 0u), NS * BN * 16, 128);
            if (elect_one()) {
#pragma unroll
              for (int s = 0; s < KRES / 16; s++) {
                if (s < nks) {
#pragma unroll
                  for (int i = 0; i < NS; i++) {
                    // (level 6 starts in slice 1, whose first instruction adds to
                    // levels 1 .. 5: its own first product goes before)
                    int n = i > 0 ? NS + 1 - i : NS;
                    if (i == 1 && s == 0 && first) {
                      umma_f16(tmem + h * TBUF + NS * BN, dA + ablk, dB + (uint64_t)(NS - 1) * BN, idesc_f16_f32(BM, BN), 0u);
                      n = NS - 1;
                    }
                    umma_f16(tmem + h * TBUF + i * BN, dA + (uint64_t)s * astep + i * ablk, dB + (uint64_t)s * bstep,
                             idesc_f16_f32(BM, BN * n), (i > 0 || s > 0 || !first) ? 1u : 0u);
                  }
                }
              }
              if (last) umma_commit(&S->t_full[h]);
            }
            __syncwarp();
          }
          if (stop) break;
          if (elect_one()) umma_commit(&S->b_empty[st]);
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
    const int grp = (warp - 2) >> 2, qd = warp & 3, half = grp >> 1;
    const int row = qd * 32 + lane, c0 = (grp & 1) * COLS;
    const uint32_t tT = tmem + ((uint32_t)(qd * 32) << 16) + half * TBUF + c0;
    constexpr bool FRAMED = has_frame(KT);
    constexpr int SIGN = FRAMED ? -1 : 1;           // W or -W
    const uint32_t tabS = smem_addr(sTab);
    int tbase = 0, tg = 0;                          // tiles before this item, accumulations taken
    // All lanes of a warp go on or none does: a lane that saw another role's abort
    // while its neighbours' phase completed would leave them at the next vote or load
    // of tensor memory.
    auto wait = [&](uint64_t *bar, int parity) {
      return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort, a.wait_limit)) != 0;
    };
    for (int it = 0;; it++) {
      if (!wait(&S->a_full, it & 1)) break;
      const int item = ((volatile int *)S->islot)[it & 1];
      if (item < 0) break;
      __syncwarp();
      if (lane == 0) mbar_arrive(&S->a_empty);
      int t0, t1, i0;
      {
        const Item g = item_geo<LISTED>(a, item);
        t0 = g.b0; t1 = g.b1; i0 = g.a_tile * BM + row;
      }
      const KParams &kp = LISTED ? S->tslot[it & 1].kp : a.kp;
      const CallParam &cp = LISTED ? S->tslot[it & 1].cp : *a.cp;
      const bool fixed = FRAMED && cp.fixed != 0;
      // (without the frame's norms the sum of many coordinates leaves two bits more)
      const int gb = G >= 0 ? G : guard_bits(a.kpad, fixed);
      const uint32_t bias = combine_bias<SIGN>(gb);
      const ExpFrame E = KT == KS_GAUSSIAN ? exp_frame(max(fixed ? cp.F : 43, 43), tabS)
                                           : exp_frame_floor(KT == KS_LAPLACE ? 52 : 53, tabS);
      const long long arow = __double_as_longlong(a.row_aa[i0]);
      const int unheld = (int)__reduce_or_sync(0xffffffffu, (unsigned)a.row_e[i0]);
      double racc[NR];
#pragma unroll
      for (int r = 0; r < NR; r++) racc[r] = 0.0;
      bool ok = true;
      for (int tj = t0 + half; tj < t1; tj += HALVES) {
        const int tt = tbase + tj - t0, ms = tt % NMETA;
        if (!wait(&S->m_full[ms], (tt / NMETA) & 1)) { ok = false; break; }
        const ColMeta *cm = (const ColMeta *)(sMeta + ms * L.meta);
        const uint32_t cmS = smem_addr(cm) + c0 * 8;   // the group's first column
        // Accumulators -> W (the fixed form: y = A + B - W), four columns at a
        // time; the tensor memory is free again after the last load.
        long long W[COLS];
        const int ngr = STREAM ? a.kpad / KRES : 1;
        for (int c = 0; c < ngr; c++, tg++) {
          if (!wait(&S->t_full[half], tg & 1)) { ok = false; break; }
          tc_fence_after();
#pragma unroll
          for (int q = 0; q < COLS; q += 4) {
            uint32_t r[4][LV];
#pragma unroll
            for (int l = 0; l < LV; l++) tmem_ld4(tT + l * BN + q, r[0][l], r[1][l], r[2][l], r[3][l]);
            const long long b0 = (long long)((uint64_t)bias << 32);
            long long w0[4] = {b0, b0, b0, b0};
            if (STREAM && c > 0) {
#pragma unroll
              for (int s = 0; s < 4; s++) w0[s] += W[q + s];
            } else if (FRAMED && fixed) {
              lds2(cmS + q * 8, w0[0], w0[1]);
              lds2(cmS + q * 8 + 16, w0[2], w0[3]);
#pragma unroll
              for (int s = 0; s < 4; s++) w0[s] += arow + b0;
            }
            tmem_ld_wait();
#pragma unroll
            for (int s = 0; s < 4; s++) W[q + s] = combine<SIGN>(r[s], gb, w0[s]);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&S->t_empty[half]);
        }
        if (!ok) break;
        // the tile's sum first: a chain of 16 and one of the tiles, not one of
        // all the row's columns (its rounding)
        double tsum[NR];
#pragma unroll
        for (int r = 0; r < NR; r++) tsum[r] = 0.0;
        if (FRAMED && fixed) {
          if constexpr (FRAMED)
            fixed_cols<KT, NR, LISTED>(a, kp, cp, E, W, arow, cm, cmS, item, row, i0, tj, c0, tsum);
        } else {
          const Place P = place_of<LISTED>(a, item, row, tj, c0);
          const RowMeta am{__longlong_as_double(arow), __longlong_as_double((long long)a.row_hi[i0]), a.row_e[i0], P.i};
          const bool slow = ((unheld | cm->flag) & NOT_HELD) == NOT_HELD;
          dot_cols<KT, NR, SIGN>(a, kp, W, am, cm, c0, P, gb, slow, tabS, tsum);
        }
#pragma unroll
        for (int r = 0; r < NR; r++)
          if (r == 0 || r < a.nrhs) racc[r] += tsum[r];
        __syncwarp();
        if (lane == 0) mbar_arrive(&S->m_empty[ms]);
      }
      if (!ok) break;
      tbase += t1 - t0;
      const Item g = item_geo<LISTED>(a, item);
      if (KT == KS_LAPLACE && fixed) {
#pragma unroll
        for (int r = 0; r < NR; r++) racc[r] *= kp.scal;
      }
      if constexpr (NR > 1) {
        // every group writes its own partials; the reduction adds them in order
        const int sc = item / a.ntm;
        if (row < g.rows) {
#pragma unroll
          for (int r = 0; r < NR; r++)
            if (r < a.nrhs) a.partial[(((size_t)r * a.nsc + sc) * GROUPS + grp) * a.ldp + g.ia + row] = racc[r];
          row_done<NR>(a, g.ia + row, a.nsc * GROUPS);
        }
      } else {
        // the groups' row sums in group order, through a slot per item parity:
        // groups 1 .. write theirs and arrive on r_full, group 0 waits, adds
        // and arrives on r_empty
        const int rb = it & 1, ru = it >> 1;   // slot, and its earlier uses
        if (grp > 0) {
          if (ru > 0 && !wait(&S->r_empty[rb], (ru - 1) & 1)) break;
          S->rsum[rb][grp - 1][row] = racc[0];
          mbar_arrive(&S->r_full[rb]);
        } else {
          if (!wait(&S->r_full[rb], ru & 1)) break;
          double s = racc[0];
          for (int q = 0; q < GROUPS - 1; q++) s += S->rsum[rb][q][row];
          mbar_arrive(&S->r_empty[rb]);
          if (row < g.rows) {
            a.partial[g.out + row] = s;
            if (!LISTED) row_done<1>(a, g.ia + row, a.nsc);
          }
        }
      }
    }
  }

  __syncthreads();
  if (*abort && threadIdx.x == 0) atomicOr(a.err, DEVERR_TIMEOUT);
  if (warp == 0) { tc_fence_after(); tmem_dealloc(tmem, TMEM_COLS); }
}

// dependent: slice_kernel is the launch just before this one on s.
template <int KT, int NR, int G, bool LISTED>
cudaError_t launch_t(const TileArgs &a, int grid, cudaStream_t s, bool dependent)
{
  const size_t smem = smem_bytes(smem_layout(a.kpad, NR, uses_table(KT)));
  // The attribute is per function and device; raised once to the most any launch takes.
  static bool raised[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !raised[dev]) {
    const cudaError_t e =
        cudaFuncSetAttribute(sliced_tiles<KT, NR, G, LISTED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) raised[dev] = true;
  }
  if (dependent) return launch_after(sliced_tiles<KT, NR, G, LISTED>, grid, NTHREADS, smem, s, a);
  sliced_tiles<KT, NR, G, LISTED><<<grid, NTHREADS, smem, s>>>(a);
  return cudaGetLastError();
}

template <int KT, int NR, bool LISTED>
cudaError_t launch_g(const TileArgs &a, int grid, cudaStream_t s, bool dependent = true)
{
  if (a.kpad > KRES) return launch_t<KT, NR, -1, LISTED>(a, grid, s, dependent);
  if constexpr (!has_frame(KT)) return launch_t<KT, NR, 3, LISTED>(a, grid, s, dependent);
  else return a.kpad > 32 ? launch_t<KT, NR, 2, LISTED>(a, grid, s, dependent) : launch_t<KT, NR, 3, LISTED>(a, grid, s, dependent);
}

}  // namespace sliced

// Padded k: a multiple of the MMA's k-step up to KRES, of KRES beyond.
static inline int sliced_kpad(int k)
{
  return k <= sliced::KRES ? (k + 15) / 16 * 16 : (k + sliced::KRES - 1) / sliced::KRES * sliced::KRES;
}

}  // namespace gsks
