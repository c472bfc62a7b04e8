// gsks_sliced.cu -- the FP64 form on the tensor cores: single calls.  The kernels and
// what they rest on: gsks_sliced_tiles.cuh.
#include "gsks_sliced_tiles.cuh"

namespace gsks {
namespace sliced {

template <int KT>
cudaError_t launch_k(const TileArgs &a, int grid, int nr, cudaStream_t s)
{
  return nr > 1 ? launch_g<KT, RMAX, false>(a, grid, s) : launch_g<KT, 1, false>(a, grid, s);
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
  const int ntp = (ntn + 1) / 2;   // pairs of source tiles (one for each half of the epilogue)
  // Runs of source tiles, in pairs: the slowest CTA's work, waves x (run + one
  // pair of per-item overhead), over up to 16 items per SM (as enqueue_split).
  int nsc = 1, chunk = ntp;
  {
    const int cmax = (int)std::min<long long>(ntp, std::max<long long>(1, (16LL * sms + ntm - 1) / ntm));
    long long best = -1;
    for (int q = 1; q <= cmax; q++) {
      const int ch = (ntp + q - 1) / q;
      if ((ntp + ch - 1) / ch != q) continue;
      const long long cost = (((long long)ntm * q + sms - 1) / sms) * (ch + 1);
      if (best < 0 || cost < best) { best = cost; nsc = q; chunk = ch; }
    }
  }
  const int ldp = ntm * BM;
  const KParams kp = make_kparams(ker, hi, hj);
  const CallParam frame = kernel_frame(kp);
  const bool framed = frame.alpha != 0.0, scan = framed && ((long long)m + n) * k > SCAN_SELF;
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
  const size_t o_n = o_e + al((size_t)ldp * 4);
  const size_t o_p = o_n + al((size_t)ldp * 4);
  const int nparts = nr > 1 ? nsc * GROUPS : nsc;          // partials per row and column
  const size_t total = o_p + al((size_t)nrhs * nparts * ldp * 8);
  // (a capturing stream would only record the allocation, to fail with the graph)
  if (total > c->total_mem) return GSKS_ERR_ALLOC;
  uint8_t *ws = nullptr;
  // (a synchronous call keeps its workspace for the next one, but no large one)
  const bool from_pool = stream_ordered_alloc || total > SYNC_KEEP;
  if (from_pool) {
    const cudaError_t e = stream_alloc(c, (void **)&ws, total, s);
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      return GSKS_ERR_ALLOC;
    }
    if (e != cudaSuccess) return cuda_status(e, "sliced workspace");
  } else {
    if (!c->dwork.ensure(total)) return GSKS_ERR_ALLOC;
    ws = (uint8_t *)c->dwork.p;
  }

  SliceArgs p{};
  p.m = m; p.n = n; p.k = k; p.kpad = kpad; p.kt = ker->type; p.nrhs = nrhs; p.nr = nr;
  const bool varbw = ker->type == KS_GAUSSIAN_VAR_BANDWIDTH;
  p.XA = XA; p.XA2 = XA2; p.hi = varbw ? hi : nullptr; p.amap = amap; p.nxa = nxa;
  p.XB = XB; p.XB2 = XB2; p.hj = varbw ? hj : nullptr; p.bmap = bmap; p.nxb = nxb;
  p.w = w; p.wmap = wmap;
  p.nta = ntm;
  p.imgA = ws + o_a; p.imgB = ws + o_b;
  p.row_aa = (double *)(ws + o_aa); p.row_hi = (uint64_t *)(ws + o_hi); p.row_e = (int *)(ws + o_e);
  p.row_n = (int *)(ws + o_n);
  p.scan = (const ScanPart *)(ws + o_scan); p.nscan = framed ? nscan : -1;
  p.frame = frame;
  p.cp = (CallParam *)(ws + o_cp);
  p.next_item = (int *)(ws + o_next);
  p.err = err_word(c);
  const int blocks = ntm * (BM / 32) + ntn * (BN / 32);
  cudaError_t e = cudaSuccess;
  if (scan) {
    scan_kernel<<<nscan, 256, 0, s>>>(p, (ScanPart *)(ws + o_scan));
    e = launch_after(slice_kernel, blocks, 256, 0, s, p);
  } else {
    slice_kernel<<<blocks, 256, 0, s>>>(p);
  }

  TileArgs a{};
  a.m = m; a.n = n; a.k = k; a.kpad = kpad; a.nrhs = nrhs;
  a.ntm = ntm; a.ntn = ntn; a.nsc = nsc; a.chunk_tiles = 2 * chunk;
  a.imgA = p.imgA; a.imgB = p.imgB;
  a.row_aa = p.row_aa; a.row_hi = p.row_hi; a.row_e = p.row_e;
  a.XA = XA; a.XB = XB; a.XA2 = XA2; a.XB2 = XB2; a.amap = amap; a.bmap = bmap; a.nxa = nxa; a.nxb = nxb;
  a.kp = kp;
  a.kp.coinc = coincidence_eps(k);
  a.cp = p.cp;
  a.partial = (double *)(ws + o_p);
  a.row_n = p.row_n;
  a.u = u; a.umap = umap;
  a.ldp = ldp;
  a.err = p.err;
  a.next_item = p.next_item;
  a.wait_limit = tl_split_wait > 0 ? tl_split_wait : WAIT_LIMIT;
  a.stall = tl_split_stall;
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) e = launch_tiles(a, std::min(ntm * nsc, sms), nr, s);
  if (from_pool) cudaFreeAsync(ws, s);
  if (e != cudaSuccess) return cuda_status(e, "sliced launch");
  note_launches(scan ? 3 : 2);
  return GSKS_OK;
}

}  // namespace gsks
