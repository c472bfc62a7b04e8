// gsks_sliced_list.cu -- the FP64 form on the tensor cores: the batched form.  The
// kernels and what they rest on: gsks_sliced_tiles.cuh.
#include "gsks_sliced_tiles.cuh"

#include <climits>
#include <cstring>
#include <vector>

namespace gsks {
namespace sliced {

static_assert(KS_EPANECHNIKOV < NTYPES, "one work counter per kernel type");

static cudaError_t launch_type(int type, const TileArgs &a, int grid, cudaStream_t s, bool dependent)
{
  switch (type) {
    case KS_GAUSSIAN: return launch_g<KS_GAUSSIAN, 1, true>(a, grid, s, dependent);
    case KS_GAUSSIAN_VAR_BANDWIDTH: return launch_g<KS_GAUSSIAN_VAR_BANDWIDTH, 1, true>(a, grid, s, dependent);
    case KS_POLYNOMIAL: return launch_g<KS_POLYNOMIAL, 1, true>(a, grid, s, dependent);
    case KS_LAPLACE: return launch_g<KS_LAPLACE, 1, true>(a, grid, s, dependent);
    case KS_TANH: return launch_g<KS_TANH, 1, true>(a, grid, s, dependent);
    case KS_QUARTIC: return launch_g<KS_QUARTIC, 1, true>(a, grid, s, dependent);
    case KS_MULTIQUADRATIC: return launch_g<KS_MULTIQUADRATIC, 1, true>(a, grid, s, dependent);
    default: return launch_g<KS_EPANECHNIKOV, 1, true>(a, grid, s, dependent);
  }
}

}  // namespace sliced

// ---------------------------------------------------------------------------
// Batched form: every task's targets and sources in tiles of their own; an item
// is (task, target tile, chunk of source tiles), its row sums go to
// partial[pbase[t] + sc m_t + r], the layout the list merge reads.
// sliced_list_plan builds the tile and item tables of a fixed set of lists on
// the device, sliced_list_run evaluates them (launches only).
int sliced_list_plan(SlicedListPlan &Pl, const KParams *kps, int ntask, int k, const int *hoff_a, const int *hoff_b,
                     const long long *pbase, int chunk, cudaStream_t s)
{
  using namespace sliced;
  if (chunk % BN) return GSKS_ERR_ARG;
  const int kpad = sliced_kpad(k), chunk_tiles = chunk / BN;
  std::vector<int> ota(ntask + 1, 0), otb(ntask + 1, 0);
  std::vector<long long> oit(ntask + 1, 0);
  for (int t = 0; t < ntask; t++) {
    const int m = hoff_a[t + 1] - hoff_a[t], n = hoff_b[t + 1] - hoff_b[t];
    const bool live = m > 0 && n > 0;
    const int ca = live ? (m + BM - 1) / BM : 0, cb = live ? (n + BN - 1) / BN : 0;
    ota[t + 1] = ota[t] + ca;
    otb[t + 1] = otb[t] + cb;
    oit[t + 1] = oit[t] + (long long)ca * ((cb + chunk_tiles - 1) / chunk_tiles);
  }
  if (oit[ntask] > INT32_MAX) return GSKS_ERR_TOO_LARGE;
  std::vector<int2> ta(ota[ntask]), tb(otb[ntask]);
  std::vector<int> ta_task(ota[ntask]), tb_task(otb[ntask]), rank(oit[ntask]);
  std::vector<Item> items(oit[ntask]);
  std::vector<TaskGeo> tg(ntask);
  std::vector<TaskParam> tp(ntask);
#pragma omp parallel for schedule(dynamic, 64) if (ntask > 512)
  for (int t = 0; t < ntask; t++) {
    const int m = hoff_a[t + 1] - hoff_a[t], n = hoff_b[t + 1] - hoff_b[t];
    tg[t] = TaskGeo{hoff_a[t], m, hoff_b[t], n};
    memset(&tp[t], 0, sizeof(TaskParam));
    tp[t].kp = kps[t];
    tp[t].cp = kernel_frame(kps[t]);
    if (m <= 0 || n <= 0) continue;
    for (int q = ota[t]; q < ota[t + 1]; q++) {
      const int i0 = (q - ota[t]) * BM;
      ta[q] = make_int2(hoff_a[t] + i0, std::min(BM, m - i0));
      ta_task[q] = t;
    }
    for (int q = otb[t]; q < otb[t + 1]; q++) {
      const int j0 = (q - otb[t]) * BN;
      tb[q] = make_int2(hoff_b[t] + j0, std::min(BN, n - j0));
      tb_task[q] = t;
    }
    long long q = oit[t];
    for (int b0 = otb[t]; b0 < otb[t + 1]; b0 += chunk_tiles)
      for (int i0 = 0; i0 < m; i0 += BM, q++) {
        Item it{};
        it.a_tile = ota[t] + i0 / BM;
        it.rows = std::min(BM, m - i0);
        it.ia = hoff_a[t] + i0;
        it.b0 = b0;
        it.b1 = std::min(otb[t + 1], b0 + chunk_tiles);
        it.jb = hoff_b[t] + (b0 - otb[t]) * BN;
        it.cols = std::min(hoff_b[t + 1] - it.jb, chunk);
        it.task = t;
        it.out = pbase[t] + (long long)((b0 - otb[t]) / chunk_tiles) * m + i0;
        items[q] = it;
        rank[q] = kps[t].type * (chunk_tiles + 1) + chunk_tiles - (it.b1 - it.b0);
      }
  }
  {
    // by kernel type, the most source tiles first, ties in build order: a
    // counting sort
    std::vector<size_t> start((size_t)NTYPES * (chunk_tiles + 1) + 1, 0);
    for (const int c : rank) start[(size_t)c + 1]++;
    for (size_t b = 0; b + 1 < start.size(); b++) start[b + 1] += start[b];
    for (int t = 0; t <= NTYPES; t++) Pl.first[t] = (int)start[(size_t)t * (chunk_tiles + 1)];
    std::vector<Item> sorted(items.size());
    for (size_t i = 0; i < items.size(); i++) sorted[start[rank[i]]++] = items[i];
    items.swap(sorted);
  }
  auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
  Pl.ntask = ntask; Pl.k = k; Pl.kpad = kpad;
  Pl.n_ta = (int)ta.size(); Pl.n_tb = (int)tb.size(); Pl.n_items = (int)items.size();
  Pl.any_frame = false;
  for (int t = 0; t < ntask && !Pl.any_frame; t++) Pl.any_frame = has_frame(kps[t].type);
  const size_t rows = (size_t)Pl.n_ta * BM;
  Pl.o_next = 0;
  Pl.o_ta = al(NTYPES * 4);
  Pl.o_tat = Pl.o_ta + al(ta.size() * sizeof(int2));
  Pl.o_tb = Pl.o_tat + al(ta.size() * 4);
  Pl.o_tbt = Pl.o_tb + al(tb.size() * sizeof(int2));
  Pl.o_items = Pl.o_tbt + al(tb.size() * 4);
  Pl.o_tg = Pl.o_items + al(items.size() * sizeof(Item));
  Pl.o_tp = Pl.o_tg + al(tg.size() * sizeof(TaskGeo));
  Pl.o_aa = Pl.o_tp + al(tp.size() * sizeof(TaskParam));
  Pl.o_hi = Pl.o_aa + al(rows * 8);
  Pl.o_e = Pl.o_hi + al(rows * 8);
  Pl.o_a = Pl.o_e + al(rows * 4);
  Pl.o_b = Pl.o_a + al((size_t)Pl.n_ta * op_bytes(BM, kpad));
  const size_t total = Pl.o_b + al((size_t)Pl.n_tb * btile_bytes(kpad, 1));
  if (!Pl.ws.ensure(total)) return GSKS_ERR_ALLOC;
  uint8_t *ws = (uint8_t *)Pl.ws.p;
  auto up = [&](size_t off, const void *src, size_t bytes) {
    return bytes == 0 || cudaMemcpyAsync(ws + off, src, bytes, cudaMemcpyHostToDevice, s) == cudaSuccess;
  };
  if (!(up(Pl.o_ta, ta.data(), ta.size() * sizeof(int2)) && up(Pl.o_tat, ta_task.data(), ta_task.size() * 4) &&
        up(Pl.o_tb, tb.data(), tb.size() * sizeof(int2)) && up(Pl.o_tbt, tb_task.data(), tb_task.size() * 4) &&
        up(Pl.o_items, items.data(), items.size() * sizeof(Item)) && up(Pl.o_tg, tg.data(), tg.size() * sizeof(TaskGeo)) &&
        up(Pl.o_tp, tp.data(), tp.size() * sizeof(TaskParam))))
    return cuda_status(cudaGetLastError(), "sliced list tables");
  // the host vectors above die here: the copies must have left them
  const cudaError_t e = cudaStreamSynchronize(s);
  return e == cudaSuccess ? GSKS_OK : cuda_status(e, "sliced list tables");
}

int sliced_list_run(const SlicedListPlan &Pl, Ctx *c, const double *XA, const double *XA2, const int *a_idx, int nxa,
                    const double *XB, const double *XB2, const int *b_idx, int nxb, const double *w, const int *w_idx,
                    double *partial, int *err, cudaStream_t s, int *launches)
{
  using namespace sliced;
  if (Pl.n_items == 0) return GSKS_OK;
  uint8_t *ws = (uint8_t *)Pl.ws.p;
  TaskParam *tp = (TaskParam *)(ws + Pl.o_tp);
  SliceArgs p{};
  p.k = Pl.k; p.kpad = Pl.kpad; p.nrhs = 1; p.nr = 1;
  p.XA = XA; p.XA2 = XA2; p.amap = a_idx; p.nxa = nxa;
  p.XB = XB; p.XB2 = XB2; p.bmap = b_idx; p.nxb = nxb;
  p.w = w; p.wmap = w_idx;
  p.imgA = ws + Pl.o_a; p.imgB = ws + Pl.o_b;
  p.row_aa = (double *)(ws + Pl.o_aa); p.row_hi = (uint64_t *)(ws + Pl.o_hi); p.row_e = (int *)(ws + Pl.o_e);
  p.next_item = (int *)(ws + Pl.o_next);
  p.err = err;
  p.tilesA = (const int2 *)(ws + Pl.o_ta); p.taskA = (const int *)(ws + Pl.o_tat);
  p.tilesB = (const int2 *)(ws + Pl.o_tb); p.taskB = (const int *)(ws + Pl.o_tbt);
  p.tp = tp;
  p.nta = Pl.n_ta;
  // (also clears the work counter)
  list_scan_kernel<<<Pl.any_frame ? Pl.ntask : 1, 256, 0, s>>>(p, Pl.ntask, (const TaskGeo *)(ws + Pl.o_tg), tp);
  cudaError_t e = launch_after(slice_kernel, Pl.n_ta * (BM / 32) + Pl.n_tb * (BN / 32), 32 * std::min(8, Pl.kpad / 8), 0, s, p);
  TileArgs a{};
  a.k = Pl.k; a.kpad = Pl.kpad; a.nrhs = 1; a.ntm = 1;
  a.imgA = p.imgA; a.imgB = p.imgB;
  a.row_aa = p.row_aa; a.row_hi = p.row_hi; a.row_e = p.row_e;
  a.XA = XA; a.XB = XB; a.XA2 = XA2; a.XB2 = XB2; a.amap = a_idx; a.bmap = b_idx; a.nxa = nxa; a.nxb = nxb;
  a.partial = partial;
  a.err = err;
  a.next_item = p.next_item;
  a.wait_limit = tl_split_wait > 0 ? tl_split_wait : WAIT_LIMIT;
  a.stall = tl_split_stall;
  a.tp = tp;
  if (e == cudaSuccess) e = cudaGetLastError();
  // Several types: every other one in the thread's second stream, which waits for
  // slice_kernel by an event, so that each launch follows it in full.
  int types = 0, kernels = 0;
  for (int t = 0; t < NTYPES; t++) types += Pl.first[t + 1] > Pl.first[t];
  const bool fork = types > 1 && e == cudaSuccess;
  if (fork) {
    e = cudaEventRecord(c->fork, s);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(c->side, c->fork, 0);
    if (e != cudaSuccess) return cuda_status(e, "sliced list launch");
  }
  for (int t = 0; t < NTYPES && e == cudaSuccess; t++) {
    a.ntab = Pl.first[t + 1] - Pl.first[t];
    if (!a.ntab) continue;
    a.tab = (const Item *)(ws + Pl.o_items) + Pl.first[t];
    a.next_item = p.next_item + t;
    e = launch_type(t, a, std::min(a.ntab, std::max(1, c->num_sms)), kernels++ & 1 ? c->side : s, !fork);
  }
  if (fork) {   // (after a failed launch too: a capture of s must not end with side left in it)
    const cudaError_t r = cudaEventRecord(c->join, c->side), w = cudaStreamWaitEvent(s, c->join, 0);
    if (e == cudaSuccess) e = r != cudaSuccess ? r : w;
  }
  if (e != cudaSuccess) return cuda_status(e, "sliced list launch");
  *launches += 2 + kernels;
  return GSKS_OK;
}

}  // namespace gsks
