// Host orchestration of the CSR product and the C ABI entry points.
//
// Flow of one product C = A·B on one stream (compare nsp_spgemm_kernel_hash,
// nsp/src/nsp.cu:2448-2488, which creates 11 streams, calls cudaMalloc and
// cudaFree for its scratch on every call, and synchronises the host 4-6 times):
//   1. B row-order check (skipped with opts.assume_sorted)
//   2. intermediate products per row -> symbolic bins          (host sync #1)
//   3. bin permutation (skipped when one bin holds every row)
//   4. one persistent kernel per non-empty symbolic bin
//   5. single-pass scan row_nz -> C.rowptr, numeric-bin histogram (host sync #2)
//   6. C.col / C.val allocated (unless provided)
//   7. bin permutation + one persistent kernel per non-empty numeric bin
// Scratch comes from a library-owned stream-ordered memory pool, so repeated
// calls do not call cudaMalloc for it.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

#include "common.cuh"
#include "internal.h"
#include "spgemm_host.h"

namespace nspb {

thread_local int g_last_cuda = 0;

const DevInfo &dev_info() {
  static std::mutex mu;
  static DevInfo infos[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  std::lock_guard<std::mutex> lock(mu);
  DevInfo &d = infos[dev];
  if (d.device < 0) {
    cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&d.smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    size_t free_b = 0;
    if (cudaMemGetInfo(&free_b, &d.total_mem) != cudaSuccess) {
      cudaGetLastError();
      d.total_mem = 0;
    }
    d.device = dev;
  }
  return d;
}

// Pinned staging for the two small device->host reads of a call.
HostStage *host_stage() {
  struct Holder {
    HostStage *p = nullptr;
    ~Holder() {
      if (p) cudaFreeHost(p);
    }
  };
  static thread_local Holder h;
  if (!h.p) {
    void *q = nullptr;
    if (cudaMallocHost(&q, sizeof(HostStage)) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    h.p = static_cast<HostStage *>(q);
  }
  return h.p;
}

static size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

// Lanes per row group from the mean length of the B rows the products read
// and of A's rows. Measured on B200 (one call, C allocated inside): 32 lanes
// win from a mean B row of 8 entries up (random, AMG and stencil products).
// Below that, when A has enough rows to fill the GPU with smaller groups, 8
// lanes win on short A rows (7-point Laplacian 128^3, 7 entries a row: 3.38 ms
// with 8 lanes, 3.87 with 16, 5.11 with 32) and 16 on longer ones, which 8
// lanes stage in too many rounds (27-point stencil 96^3 times its smoothed
// aggregation prolongator, 27 A entries a row and B rows of 4.5: 3.53 ms with
// 16 lanes, 4.61 with 8, 4.00 with 32).
static int pick_lanes(double mean_b_row, double mean_a_row, int a_rows) {
  if (mean_b_row < 7.5 && a_rows >= 65536) return mean_a_row <= 8.0 ? 8 : 16;
  return 32;
}

// ---- a call --------------------------------------------------------------------
int Call::init(const nspb_csr_in *a, const nspb_csr_in *b, const nspb_opts *o) {
  nspb_default_opts(&opts);
  if (o) opts = *o;
  s = static_cast<cudaStream_t>(opts.stream);
  if (!a || !b) return NSPB_ERR_INVALID;
  if (a->nrows < 0 || a->ncols < 0 || b->nrows < 0 || b->ncols < 0) return NSPB_ERR_INVALID;
  if (a->ncols != b->nrows) return NSPB_ERR_INVALID;
  if (a->nnz < 0 || b->nnz < 0 || a->nnz > INT32_MAX || b->nnz > INT32_MAX) return NSPB_ERR_INVALID;
  if ((a->nrows > 0 && !a->rowptr) || (b->nrows > 0 && !b->rowptr)) return NSPB_ERR_INVALID;
  if ((a->nnz > 0 && (!a->col || !a->val)) || (b->nnz > 0 && (!b->col || !b->val)))
    return NSPB_ERR_INVALID;
  const int want = fp32_inputs(opts.precision) ? NSPB_F32 : NSPB_F64;
  if (opts.precision != NSPB_PREC_FP64 && !fp32_inputs(opts.precision)) return NSPB_ERR_INVALID;
  if ((a->nnz > 0 && a->val_type != want) || (b->nnz > 0 && b->val_type != want))
    return NSPB_ERR_INVALID;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return NSPB_ERR_NO_DEVICE;
  }
  auto fill = [&](CsrDev &d, const nspb_csr_in *m) {
    d.nrows = m->nrows;
    d.ncols = m->ncols;
    d.nnz = m->nnz;
    d.rpt = m->rowptr;
    d.col = m->col;
    if (m->val_type == NSPB_F32) d.val32 = static_cast<const float *>(m->val);
    else d.val = static_cast<const double *>(m->val);
  };
  fill(A, a);
  fill(B, b);
  n = A.nrows;
  t64 = ProdTable<double>{};
  t64.one = Operands<double>{A.rpt, A.col, A.val, B.rpt, B.col, B.val, B.ncols, B.nrows, nullptr};
  t32 = ProdTable<float>{};
  t32.one = Operands<float>{A.rpt, A.col, A.val32, B.rpt, B.col, B.val32, B.ncols, B.nrows, nullptr};
  info = ProdInfo{n, B.ncols, 1, B.nrows, B.nrows, false};
  lim = bin_limits(opts.sym_fill_pct, opts.num_fill_pct);
  a_nnz = A.nnz;
  b_nnz = B.nnz;
  table = false;
  ops = nullptr;
  if (opts.timing) {
    timing = true;
    for (auto &e : ev) cudaEventCreate(&e);
  }
  if (opts.group_lanes == 8 || opts.group_lanes == 16 || opts.group_lanes == 32) {
    lanes = opts.group_lanes;
  } else {
    // until the intermediate products are counted (symbolic): B's mean row
    const double avg = B.nrows > 0 ? (double)B.nnz / (double)B.nrows : 0.0;
    lanes = pick_lanes(avg, A.nrows > 0 ? (double)A.nnz / (double)A.nrows : 0.0, A.nrows);
  }
  return NSPB_OK;
}

void Call::set_table(const ProdTable<double> &d, const ProdTable<float> &f, const ProdInfo &pi,
                     int64_t total_a_nnz) {
  t64 = d;
  t32 = f;
  info = pi;
  n = pi.n;
  a_nnz = total_a_nnz;
  table = true;
  ops = reinterpret_cast<const Operands<void> *>(d.ops);
  A = CsrDev{};
  B = CsrDev{};
  A.nrows = pi.n;
  A.nnz = total_a_nnz;
  B.ncols = pi.max_ncols;
  if (!(opts.group_lanes == 8 || opts.group_lanes == 16 || opts.group_lanes == 32)) lanes = 32;
}

size_t Call::scratch_bytes() {
  allow_runs = runs_wanted();  // no tables, and fewer counters to clear and read, without
  const size_t nn = (size_t)std::max(n, 1);
  off_row_nz = 0;
  off_perm = align256(off_row_nz + (nn + 1) * 4);
  off_slots = align256(off_perm + nn * 4);
  off_counters = off_slots;
  if (allow_runs) off_counters = align256(off_slots + kRunTableRest * (kRunSlots + 64) * 4);
  off_tiles = align256(off_counters + counter_bytes() +
                       (allow_runs ? kRunTableZeroed * kRunSlots * 4 : 0));
  const size_t tiles = (size_t)scan_tiles(n);
  ws_bytes = align256(off_tiles + tiles * 8);
  return ws_bytes;
}

int Call::alloc_scratch() {
  scratch_bytes();
  if (ext_ws) {
    if (ws_bytes > ext_bytes) return NSPB_ERR_CAPACITY;
    ws = ext_ws;
    ws_external = true;
  } else {
    int st = scratch_alloc(reinterpret_cast<void **>(&ws), ws_bytes, s);
    if (st) return st;
  }
  row_nz = reinterpret_cast<int *>(ws + off_row_nz);
  perm = reinterpret_cast<int *>(ws + off_perm);
  ctr = reinterpret_cast<DevCounters *>(ws + off_counters);
  tile_state = reinterpret_cast<unsigned long long *>(ws + off_tiles);
  if (allow_runs) {
    rtab.head = &ctr->run;
    rtab.rep = reinterpret_cast<unsigned long long *>(ctr + 1);
    rtab.prog_of = reinterpret_cast<int *>(ws + off_slots);
    rtab.brep = rtab.rep + kRunSlots;
    rtab.bcount = reinterpret_cast<int *>(rtab.brep + kRunSlots);
    rtab.count = rtab.bcount + kRunSlots;
    int *rest = rtab.prog_of;
    for (int **p : {&rtab.run_of, &rtab.slot_of, &rtab.first, &rtab.bslot, &rtab.brow, &rtab.brows, &rtab.bplace, &rtab.btiles[0],
                    &rtab.btiles[1]})
      *p = rest += kRunSlots + 64;
  }
  // counters, pattern table and scan tile states are contiguous: one memset clears them
  cudaError_t e = cudaMemsetAsync(ws + off_counters, 0, ws_bytes - off_counters, s);
  if (e != cudaSuccess) return cuda_fail(e);
  return NSPB_OK;
}

Call::~Call() {
  if (ws && !ws_external) scratch_free(ws, s);
  if (map_block) scratch_free(map_block, s);
  drop_runs();
  for (auto &e : ev)
    if (e) cudaEventDestroy(e);
}

int Call::cuda_fail(cudaError_t e) {
  g_last_cuda = (int)e;
  cudaGetLastError();
  return NSPB_ERR_CUDA;
}

cudaError_t Call::order_block_bins(const int *key, int kind, const int *counts, int first,
                                   int end, const BinOffsets &off) {
  RowLists lists{};
  for (int b = first; b < end; ++b)
    if (counts[b] > 1) {
      lists.off[lists.n] = off.v[b];
      lists.count[lists.n] = counts[b];
      ++lists.n;
    }
  if (lists.n == 0) return cudaSuccess;
  ++launches;
  return launch_order_rows(key, kind, lists, perm, s);
}

int Call::fetch_counters() {
  HostStage *hs = stage ? stage : host_stage();
  if (!hs) return NSPB_ERR_ALLOC;
  cudaError_t e = cudaMemcpyAsync(&hs->c, ctr, counter_bytes(), cudaMemcpyDeviceToHost, s);
  if (e != cudaSuccess) return cuda_fail(e);
  e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(e);
  h = hs->c;
  if (h.err) return NSPB_ERR_DEVICE;
  return NSPB_OK;
}

static BinOffsets offsets_of(const int *counts, int nb, int *nonempty, int *total) {
  BinOffsets o;
  int acc = 0, ne = 0;
  for (int b = 0; b < 16; ++b) {
    o.v[b] = acc;
    if (b < nb) {
      acc += counts[b];
      ne += counts[b] > 0;
    }
  }
  *nonempty = ne;
  *total = acc;
  return o;
}

// Row runs are looked for when the caller leaves the choice of the row kernels
// to the library and A's rows are short enough on average for runs to hold
// most of them. The search and the programs cost a chain of ten small launches,
// so small products do without, unless row_kernel is 8: those of fewer than
// about 24 million intermediate products (A's entries times B's mean row), or 8
// million where B's rows are so short that the row-group kernels leave most
// lanes idle. Measured, runs against none: 27-point 40^3 (42 M) 379 vs 497 us,
// 30^3 (17 M) 297 vs 333, 24^3 (8.5 M) 280 vs 244, R (A P) of 80^3 (28 M) 507
// vs 519, of 60^3 (11 M) 404 vs 262; B's rows of 4.5 and 7: A P of 48^3 (12 M)
// 341 vs 390, of 40^3 (7.4 M) 310 vs 284, 7-point 64^3 (12.5 M) 286 vs 406,
// 64 x 50 x 50 (7.6 M) 249 vs 314, 32^3 (1.5 M) 222 vs 170.
// The symbolic and the numeric step in calls of their own (two_calls) search
// twice, and need more: 14 million where B's rows are shorter than 8, 26 million
// up to 16 if A's have at most 64 entries, 40 million otherwise. Both calls, runs against what came before
// them: A P of 44^3 (9.8 M) 585 vs 460, of 52^3 (16.6 M) 649 vs 672; 7-point
// 12.5 M 515 vs 497, 17.9 M 605 vs 646; R (A P) of 80^3 873 vs 818, 15-point
// 26.6 M 539 vs 657; 27-point 31 M 566 vs 523, 43 M 608 vs 686, 7-point 30^3 of
// 3 unknowns a node (34 M) 738 vs 654.
bool Call::runs_wanted() const {
  if (!allow_runs || family() != 0 || (opts.row_kernel & kNoRowTemplates)) return false;
  if (n < 2 * kRunMin || a_nnz > (int64_t)kRunMaxA * n || (table && !info.bdel)) return false;
  if ((opts.row_kernel & 0xff) == 8) return true;
  if (info.brows <= 0) return false;
  const double mean = (double)b_nnz / (double)info.brows;
  // rows of far more products than a run may have (14^3 27-point grid of 3
  // unknowns a node, both calls: 945 us, with the search 1010)
  if (!table && mean * (double)a_nnz > 1.5 * kRunMaxIp * (double)n) return false;
  const double least = mean < 8.0 ? (two_calls ? 14e6 : 8e6)
                       : !two_calls ? 24e6
                       : mean < 16.0 && a_nnz <= 64LL * n ? 26e6 : 40e6;
  return (double)a_nnz * mean >= least;
}

int Call::alloc_runs() {
  const size_t cap = (size_t)run_capacity(n) * sizeof(RowRun);
  const size_t o_found = align256((size_t)n), o_runs = align256(o_found + cap);
  const size_t o_slot = align256(o_runs + cap), o_list = align256(o_slot + (size_t)n * 4);
  const size_t o_del = align256(o_list + (size_t)n * 4);
  const size_t bytes = o_del + (table ? 0 : (size_t)kMaxLag * std::max(B.nrows, 1) * sizeof(int2));
  int st = scratch_alloc(reinterpret_cast<void **>(&run_block), bytes, s);
  if (st) return st;
  member = reinterpret_cast<unsigned char *>(run_block);
  found = reinterpret_cast<RowRun *>(run_block + o_found);
  runs = reinterpret_cast<RowRun *>(run_block + o_runs);
  bunch_slot = reinterpret_cast<int *>(run_block + o_slot);
  bunch_list = reinterpret_cast<int *>(run_block + o_list);
  if (!table) t64.one.bdel = t32.one.bdel = reinterpret_cast<int2 *>(run_block + o_del);
  return NSPB_OK;
}

int Call::build_programs() {
  for (int c = 0; c < 2; ++c) nruns[c] = run_block ? h.run.nruns[c] : 0;
  use_runs = nruns[0] + nruns[1] > 0;
  nprog = nbunch = 0;
  if (!use_runs) return NSPB_OK;
  nprog = h.run.nprog;
  // the rows left over, where the runs took most of the row-group rows
  long long taken = 0, left = 0;
  for (int b = 0; b < kSymGroupBins; ++b) {
    taken += h.sym_sub[b];
    left += h.sym_counts[b] - h.sym_sub[b];
  }
  int st;
  cudaError_t e;
  if (left > 0 && taken >= left) {
    e = launch_bunch_find(structure_of(t64), member, n, lim, row_nz, rtab, bunch_slot, bunch_list,
                          ctr->sym_sub, s);
    if (e != cudaSuccess) return cuda_fail(e);
    launches += 3;
    if ((st = fetch_counters())) return st;
    nbunch = h.run.nbunch;
  }
  if ((st = scratch_alloc(&progs, (size_t)(nprog + nbunch) * run_prog_bytes(), s))) return st;
  e = launch_run_progs(structure_of(t64), found, rtab, nprog, nbunch, fp32_inputs(opts.precision),
                       progs, &ctr->err, s);
  if (e != cudaSuccess) return cuda_fail(e);
  ++launches;
  return NSPB_OK;
}

// The rows of runs and bunches get their counts (nz) and leave the numeric bins.
cudaError_t Call::count_runs(int *nz, const int *crpt) {
  cudaError_t e = launch_run_counts(found, h.run.nfound, runs, (int)run_capacity(n), rtab, progs, nz,
                                    crpt, lim, ctr->num_sub, s);
  if (e == cudaSuccess)
    e = launch_bunch_counts(rtab, nprog, nbunch, bunch_list, progs, nz, crpt, lim, ctr->num_sub, s);
  launches += 1 + (nbunch > 0);
  return e;
}

void Call::drop_runs() {
  if (run_block) scratch_free(run_block, s);
  if (progs) scratch_free(progs, s);
  run_block = nullptr;
  progs = nullptr;
  t64.one.bdel = t32.one.bdel = nullptr;
  use_runs = false;
  nruns[0] = nruns[1] = 0;
  nprog = nbunch = 0;
}

// same: B is A, whose order the row walk of k_rowinfo checks.
cudaError_t Call::check_b(bool same) {
  if (run_block) {
    ++launches;
    return launch_brow_delta(structure_of(t64), info, b_nnz, ctr->lag_count,
                             opts.assume_sorted || same ? nullptr : &ctr->flags, s);
  }
  if (opts.assume_sorted || same) return cudaSuccess;
  ++launches;
  return table ? launch_check_sorted_table(ops, info.nprod, info.max_brows, &ctr->flags, s)
               : launch_check_sorted(B, &ctr->flags, s);
}

// Steps 1-5: C.rowptr and nnz(C). crpt must hold n+1 ints.
int Call::symbolic(int *crpt, int64_t *nnz_out) {
  cudaError_t e;
  if (n == 0) {
    e = cudaMemsetAsync(crpt, 0, sizeof(int), s);
    if (e != cudaSuccess) return cuda_fail(e);
    *nnz_out = 0;
    return NSPB_OK;
  }
  int st = alloc_scratch();
  if (st) return st;
  mark(0);
  // B = A (the same arrays): the row walk of k_rowinfo checks B's order too
  const bool same = !table && A.rpt == B.rpt && A.col == B.col && A.nrows == B.nrows &&
                    A.nnz == B.nnz;
  if (runs_wanted() && alloc_runs()) drop_runs();  // no memory for them: every row on its own
  if ((e = check_b(same)) != cudaSuccess) return cuda_fail(e);
  RunScan scan;
  if (run_block) scan = RunScan{member, ctr->lag_count, info.brows, false, same};
  // perm is free until the bins are permuted: it holds the long-row list here
  if ((e = launch_rowinfo(structure_of(t64), n, a_nnz, lim, row_nz, nullptr, ctr->sym_counts,
                          &ctr->total_ip,
                          !opts.assume_sorted && same ? &ctr->flags : nullptr, perm,
                          &ctr->long_rows, scan, s)) != cudaSuccess)
    return cuda_fail(e);
  if (run_block) {
    if ((e = launch_run_find(structure_of(t64), member, n, lim, row_nz, found, rtab,
                             ctr->sym_sub, s)) != cudaSuccess)
      return cuda_fail(e);
    launches += 2;
  }
  ++launches;
  mark(1);
  if ((st = fetch_counters())) return st;
  b_sorted = opts.assume_sorted || !(h.flags & B_UNSORTED);
  intprod = (int64_t)h.total_ip;
  products = (double)intprod;
  if ((st = build_programs()) == NSPB_ERR_ALLOC) {  // no memory for them: without runs
    drop_runs();
    allow_runs = false;
    if (!ws_external) scratch_free(ws, s);
    ws = nullptr;
    return symbolic(crpt, nnz_out);
  }
  if (st) return st;
  int todo[16];  // rows of each bin to be counted: those that no run serves
  for (int b = 0; b < 16; ++b) todo[b] = h.sym_counts[b] - (use_runs ? h.sym_sub[b] : 0);
  // the mean length of the B rows actually read, weighted by how often A reads
  // them: a block-diagonal batch mixes products whose B rows differ
  if (!(opts.group_lanes == 8 || opts.group_lanes == 16 || opts.group_lanes == 32) && a_nnz > 0)
    lanes = pick_lanes((double)intprod / (double)a_nnz, (double)a_nnz / (double)n, n);
  if (a_nnz > 0) info.mean_b = (double)intprod / (double)a_nnz;
  int nonempty = 0, binned = 0;
  BinOffsets off = offsets_of(todo, kSymBins, &nonempty, &binned);
  const bool direct = nonempty == 1 && binned == n;
  // entry maps: a stride of the bin's row limit (products) per row
  long long map_bin_off[kSymGroupBins] = {};
  int map_stride[kSymGroupBins] = {};
  use_map = false;
  if (binned > 0 && map_wanted()) {
    long long total = 0;
    for (int b = 0; b < kSymGroupBins; ++b) {
      // quads of the map take at most 4/3 of a byte per product, plus alignment
      map_stride[b] = (int)(((long long)lim.sym[b] * 3 / 2 + 16 + 15) & ~15LL);
      map_bin_off[b] = total;
      total += (long long)todo[b] * map_stride[b];
    }
    const size_t head = align256((size_t)n * 4);
    // row templates of one product check B rows by their shift bits
    const bool shift_bits = !(opts.row_kernel & kNoRowTemplates) && !table;
    const size_t bits = shift_bits ? align256(((size_t)B.nrows / 32 + 1) * 4) : 0;
    // at most an eighth of the device's memory (C is allocated after this phase)
    if ((head + bits + (size_t)total) * 8 <= dev_info().total_mem &&
        scratch_alloc(&map_block, head + bits + (size_t)total, s) == NSPB_OK) {
      map_off = static_cast<unsigned *>(map_block);
      bshift = shift_bits ? reinterpret_cast<unsigned *>(static_cast<unsigned char *>(map_block) +
                                                         head)
                          : nullptr;
      map = static_cast<unsigned char *>(map_block) + head + bits;
      use_map = true;
      if (bshift) {
        e = run_block ? launch_shift_bits(t64.one.bdel, B.nrows, bshift, s)
                      : launch_brow_shift(B.rpt, B.col, B.nrows, bshift, s);
        if (e != cudaSuccess) return cuda_fail(e);
        ++launches;
      }
    }
  }
  mark(2);
  if (!direct && binned > 0) {
    if ((e = launch_perm(row_nz, n, 0, off, lim, nullptr, ctr->cursor_sym, perm, s)) != cudaSuccess)
      return cuda_fail(e);
    ++launches;
    if ((e = order_block_bins(row_nz, 0, todo, kSymGroupBins, kSymBins, off)) != cudaSuccess)
      return cuda_fail(e);
  }
  // flat product lists unless the B rows fill the lanes of a row group; rows of
  // at most 48 products, which leave most of a warp of the flat kernel idle,
  // also stay with row groups of 8 lanes (5-point 1000^2 renumbered 165 us
  // against 255; 300,000 rows of 25 products 58 and 86, of 4 products 26 and 69)
  const bool flat = family() == 0 && (double)intprod < 0.75 * (double)lanes * (double)a_nnz;
  const int flat_from = lanes == 8 ? 2 : 0;
  for (int b = 0; b < kSymBins; ++b) {
    const int c = todo[b];
    if (c <= 0) continue;
    const int *rows = direct ? nullptr : perm + off.v[b];
    if (use_map) {
      MapArgs m;
      m.map = map;
      m.bin_off = map_bin_off[b];
      m.stride = map_stride[b];
      m.map_off = map_off;
      m.flags = &ctr->flags;
      m.chunk = template_run();
      m.bshift = bshift;
      e = launch_symbolic_map(b, lanes, structure_of(t64), rows, c, row_nz, &ctr->err, m, s);
    } else if (b < kSymGroupBins && flat && b >= flat_from) {
      e = launch_symbolic_flat(b, structure_of(t64), rows, c, row_nz, &ctr->err, s);
    } else {
      e = launch_symbolic_bin(b, lanes, b_sorted, structure_of(t64), info, rows, c, row_nz,
                              &ctr->err, &ctr->ticket[b], s);
    }
    if (e != cudaSuccess) return cuda_fail(e);
    ++launches;
  }
  if (use_runs) {
    if ((e = count_runs(row_nz, nullptr)) != cudaSuccess) return cuda_fail(e);
  }
  mark(3);
  if ((e = launch_scan(row_nz, n, crpt, &ctr->total_nnz, tile_state, &ctr->tile_ctr, lim,
                       ctr->num_counts, &ctr->err, s)) != cudaSuccess)
    return cuda_fail(e);
  ++launches;
  mark(4);
  if ((st = fetch_counters())) return st;
  num_counts_ready = true;
  for (int b = 0; b < 16; ++b) run_rows[b] = use_runs ? h.num_sub[b] : 0;
  if (use_map && (h.flags & MAP_OVERFLOW)) {  // a row outgrew its stride: no map
    use_map = false;
    scratch_free(map_block, s);
    map_block = nullptr;
    map = nullptr;
    map_off = nullptr;
    bshift = nullptr;
  }
  if (h.total_nnz > INT32_MAX) return NSPB_ERR_OVERFLOW;
  *nnz_out = h.total_nnz;
  return NSPB_OK;
}

// Step 7 (the numeric-bin histogram must be in h.num_counts).
int Call::numeric(const int *crpt, int *ccol, double *cval) {
  cudaError_t e;
  if (n == 0) return NSPB_OK;
  int nonempty = 0, binned = 0;
  int todo[16];  // rows of each bin that no run serves
  for (int b = 0; b < 16; ++b) todo[b] = h.num_counts[b] - run_rows[b];
  BinOffsets off = offsets_of(todo, kNumBins, &nonempty, &binned);
  if (binned == 0 && !use_runs) return NSPB_OK;
  const bool direct = nonempty == 1 && binned == n;
  mark(5);
  if (!direct && binned > 0) {
    if ((e = launch_perm(crpt, n, 1, off, lim, use_runs ? member : nullptr, ctr->cursor_num, perm,
                         s)) != cudaSuccess)
      return cuda_fail(e);
    ++launches;
    if ((e = order_block_bins(crpt, 1, todo, use_flat() ? kNumLong : kNumGroupBins, kNumBins,
                              off)) != cudaSuccess)
      return cuda_fail(e);
  }
  // fp32 inputs: rows of at most nmax A entries accumulate in fp32 pairs, the
  // others (every row in the wide mode) in fp64 from exact products
  const bool comp = fp32_inputs(opts.precision);
  const int nmax = opts.precision == NSPB_PREC_FP32_COMP ? comp_nmax(opts.comp_tol) : 0;
  const bool staged = use_staged();
  auto hash_bin = [&](int b, int g, const int *rows, int c, int *ticket, int tshift,
                      const int *dcount) {
    return comp ? launch_numeric_comp_bin(b, g, b_sorted, b_sorted, t32, info, crpt, ccol, cval,
                                          rows, c, nmax, &ctr->redo_count, &ctr->max_comp_deg,
                                          &ctr->err, ticket, tshift, dcount, s)
                : launch_numeric_bin(b, g, b_sorted, b_sorted, t64, info, crpt, ccol, cval, rows,
                                     c, &ctr->err, ticket, tshift, dcount, s);
  };
  if (use_runs) {
    const int cap = (int)run_capacity(n);
    // pairs for the rows that the row-group kernels sum in pairs
    const int pair_a = b_sorted ? nmax : 0, pair_c = lim.num[kNumGroupBins - 1];
    e = comp ? launch_numeric_comp_run(t32, runs, nruns, cap, progs, crpt, ccol, cval, pair_a,
                                       pair_c, &ctr->redo_count, &ctr->max_comp_deg, &ctr->err,
                                       &ctr->ticket[30], s)
             : launch_numeric_run(t64, runs, nruns, cap, progs, crpt, ccol, cval, &ctr->err,
                                  &ctr->ticket[30], s);
    if (e != cudaSuccess) return cuda_fail(e);
    launches += (nruns[0] > 0) + (nruns[1] > 0);
    if (nbunch > 0) {
      e = comp ? launch_numeric_comp_bunch(t32, rtab, nprog, nbunch, bunch_list, progs, crpt, ccol,
                                           cval, pair_a, pair_c, &ctr->redo_count, &ctr->max_comp_deg,
                                           &ctr->err, &ctr->ticket[28], s)
               : launch_numeric_bunch(t64, rtab, nprog, nbunch, bunch_list, progs, crpt, ccol, cval,
                                      &ctr->err, &ctr->ticket[28], s);
      if (e != cudaSuccess) return cuda_fail(e);
      launches += 2;
    }
  }
  // Rows with more products than their flat list holds go to the hash kernel
  // of their own bin (of bin 3 for the smaller ones): with one kernel for all
  // rows of up to 512 entries and one for the others, 10,000 rows of 996 entries
  // and 1296 products took 608 us there, 298 in their own. Where products exceed
  // the entries by 5% at most there can be few such rows, and two launches do.
  // Bin b's are listed from off.v[b] on (row_nz is free by now).
  const bool apart = h.total_ip == 0 || products > 1.05 * (double)h.total_nnz;
  constexpr int kFlatFirst = 3;
  auto over_bin = [&](int b) {
    if (!apart) return b < kNumGroupBins ? kNumGroupBins - 1 : kNumLong - 1;
    return std::max(b, kFlatFirst);
  };
  auto over_at = [&](int bin) {
    if (!apart) return off.v[bin < kNumGroupBins ? 0 : kNumGroupBins];
    return off.v[bin == kFlatFirst ? 0 : bin];
  };
  const bool flat = use_flat();
  const bool few = info.mean_b * (double)a_nnz <= 12.0 * (double)n;
  int flat_rows[kNumLong] = {};
  for (int b = 0; b < kNumBins; ++b) {
    const int c = todo[b];
    if (c <= 0) continue;
    const int *rows = direct ? nullptr : perm + off.v[b];
    int *ticket = &ctr->ticket[16 + b];
    const int tshift = opts.num_table_shift == 1 ? 1 : 0;
    if (use_map && b < kMapNumBins) {
      // cp.async of the next row's A entries pays on short A rows (7-point
      // Laplacian 128^3: numeric 1.47 -> 1.16 ms) and costs on long ones
      // (27-point stencil 128^3: 6.63 -> 7.42 ms, L1 data pipe saturated)
      const bool pref = !table && a_nnz <= 12LL * n;
      const int run = template_run();
      e = comp ? launch_numeric_comp_map(b, lanes, t32, map, map_off, crpt, ccol, cval, rows, c,
                                         pref, run, bshift, nmax, &ctr->redo_count,
                                         &ctr->max_comp_deg, &ctr->err, s)
               : launch_numeric_map(b, lanes, t64, map, map_off, crpt, ccol, cval, rows, c, pref,
                                    run, bshift, &ctr->err, s);
      if (e != cudaSuccess) return cuda_fail(e);
      ++launches;
      continue;
    }
    if (b < kNumGroupBins && b_sorted && staged) {
      const int rg_shift = (opts.row_kernel & 0xff) == 3 ? -1 : 0;  // tables 2x, else 4x
      e = comp ? launch_numeric_comp_rg(b, lanes, rg_shift, rg_depth(), t32, crpt, ccol, cval,
                                        rows, c, nmax, &ctr->redo_count, &ctr->max_comp_deg,
                                        &ctr->err, s)
               : launch_numeric_rg(b, lanes, rg_shift, rg_depth(), t64, crpt, ccol, cval, rows,
                                   c, &ctr->err, s);
      if (e != cudaSuccess) return cuda_fail(e);
      ++launches;
      continue;
    }
    // rows of at most 16 entries and few products on average: row groups of 8
    // lanes (300,000 rows of 4 products 93 us, from flat lists 161; 1 M of 9 380
    // and 526; the short rows of a power-law 300,000^2 of mean 6 170 and 126)
    // Rows of up to 512 entries are ahead in their hash kernels from about 1.25
    // products an entry on: lists and hash kernels, 20 M products, d entries a
    // row of A and B, at 1.29, 1.39 and 1.48 products an entry: d = 12 579 and
    // 557, 566 and 507, 570 and 498 us, d = 16 568 and 508, 568 and 470, 578 and
    // 460, d = 20 620 and 650, 618 and 610, 652 and 615; d = 60, rows of 2400 to
    // 2800 entries, 729 and 815, 733 and 794, 728 and 758.
    if (b < kNumLong && flat && !(b == 0 && lanes == 8 && few) &&
        (b >= kNumGroupBins || products < 1.25 * (double)h.total_nnz)) {
      const int o = over_bin(b);
      int *over = row_nz + over_at(o);
      e = comp ? launch_numeric_comp_flat(b, b_sorted, t32, crpt, ccol, cval, rows, c, nmax,
                                          &ctr->redo_count, &ctr->max_comp_deg, over,
                                          &ctr->over[o], &ctr->err, s)
               : launch_numeric_flat(b, t64, crpt, ccol, cval, rows, c, over, &ctr->over[o],
                                     &ctr->err, s);
      if (e != cudaSuccess) return cuda_fail(e);
      ++launches;
      flat_rows[o] += c;
      continue;
    }
    if ((e = hash_bin(b, lanes, rows, c, ticket, tshift, nullptr)) != cudaSuccess)
      return cuda_fail(e);
    ++launches;
  }
  for (int b = 0; b < kNumLong; ++b) {
    if (flat_rows[b] == 0) continue;
    if ((e = hash_bin(b, apart ? lanes : 32, row_nz + over_at(b), flat_rows[b],
                      &ctr->ticket[16 + b], 0, &ctr->over[b])) != cudaSuccess)
      return cuda_fail(e);
    ++launches;
  }
  mark(6);
  return NSPB_OK;
}

// The symbolic phase records entry maps when the numeric phase of the same
// call can use them: B rows strictly increasing, every row with
// products in a row-group symbolic bin, column offsets within 24 bits, and
// row_kernel 7 (maps), or 0 (automatic) when the B rows the products read
// fill at least 3/4 of a row group's lanes on average. The map costs the
// symbolic pass a fixed amount per B row and saves the numeric pass a hash
// probe per product. Measured on B200 (full product, maps vs staged walk):
// 27-point stencil 128^3 12.9 vs 14.3 ms and 96^3 5.3 vs 5.9 ms (B rows of
// 27 on 32 lanes), 7-point Laplacian 128^3 2.13 vs 2.28 ms (7 on 8 lanes);
// slower on smoothed-aggregation products, 3.3 vs 2.5 ms for A*P of the
// 96^3 stencil (4.5 on 16 lanes), and on random products of 4..32 entries
// a row, 3.2 vs 3.0 ms (18 on 32 lanes, against the hash-sort kernels).
bool Call::map_wanted() const {
  const int k = family();
  if (!allow_map || !(k == 0 || k == 7)) return false;
  if (!b_sorted || n <= 0 || a_nnz <= 0) return false;
  if (info.max_ncols > kMapMaxCols) return false;
  for (int b = kSymGroupBins; b < kSymBins; ++b)
    if (h.sym_counts[b] > 0) return false;
  if (k == 7) return true;
  return (double)intprod >= 0.75 * (double)lanes * (double)a_nnz;
}

// Numeric bins and B order for a two-call numeric step.
int Call::prepare_numeric(const int *crpt, int64_t nnz) {
  if (n == 0) return NSPB_OK;
  two_calls = true;
  int st = alloc_scratch();
  if (st) return st;
  cudaError_t e;
  if (runs_wanted() && alloc_runs()) drop_runs();
  if ((e = check_b(false)) != cudaSuccess) return cuda_fail(e);
  if (run_block) {
    // the runs again (the symbolic phase was another call's); operands without
    // structure skip the row walk
    const bool same = !table && A.rpt == B.rpt && A.col == B.col && A.nrows == B.nrows &&
                      A.nnz == B.nnz;
    const RunScan scan{member, ctr->lag_count, info.brows, true, same};
    if ((e = launch_rowinfo(structure_of(t64), n, a_nnz, lim, row_nz, nullptr, ctr->sym_counts,
                            &ctr->total_ip, nullptr, perm, &ctr->long_rows, scan, s)) !=
            cudaSuccess ||
        (e = launch_run_find(structure_of(t64), member, n, lim, row_nz, found, rtab,
                             ctr->sym_sub, s)) != cudaSuccess)
      return cuda_fail(e);
    launches += 3;
  }
  // The products, where they are not counted, are A's entries times B's mean row,
  // or times the mean row that some of A's entries read where that is clearly
  // longer (A may read B's long rows above all; the shorter mean would send rows
  // to lists that they outgrow: 20,000 rows of 10 of B's 400 rows of 60 among
  // 20,000 of one entry, both calls 414 us, 373 before the lists).
  const double plain = info.brows > 0 ? (double)b_nnz / (double)info.brows : 0.0;
  ReadSample rs;
  if (!table && family() == 0 && a_nnz > 32768 && plain * (double)a_nnz < 1.25 * (double)nnz)
    rs = ReadSample{A.rpt, A.col, B.rpt, 1024 * std::min(n / 1024 + (n % 1024 > 0), 16),
                    &ctr->read_sum};
  if ((e = launch_num_hist(crpt, n, lim, ctr->num_counts, rs, s)) != cudaSuccess)
    return cuda_fail(e);
  ++launches;
  if ((st = fetch_counters())) return st;
  b_sorted = opts.assume_sorted || !(h.flags & B_UNSORTED);
  num_counts_ready = true;
  const double read = rs.samples ? (double)h.read_sum / (double)rs.samples : 0.0;
  const double each = read > 1.5 * plain ? read : plain;
  products = h.total_ip ? (double)h.total_ip : each * (double)a_nnz;
  if (a_nnz > 0) info.mean_b = products / (double)a_nnz;
  if ((st = build_programs()) == NSPB_ERR_ALLOC) drop_runs();
  else if (st) return st;
  if (use_runs) {
    if ((e = count_runs(nullptr, crpt)) != cudaSuccess) return cuda_fail(e);
    if ((st = fetch_counters())) return st;
    for (int b = 0; b < 16; ++b) run_rows[b] = h.num_sub[b];
  }
  return NSPB_OK;
}

// Largest A-row degree n whose Dot2 error bound gamma_n^2 (gamma_n =
// n u / (1 - n u), u = 2^-24, Ogita, Rump and Oishi 2005) stays within tol,
// relative to sum |a_ik b_kj|; fp32 pairs then add within tol of the exact sum.
int comp_nmax(double tol) {
  if (!(tol > 0.0)) tol = 1e-10;
  const double u = 0x1.0p-24, r = std::sqrt(tol);
  return (int)std::floor(r / (u * (1.0 + r)));
}

double comp_bound(int n) {
  if (n <= 0) return 0.0;
  const double u = 0x1.0p-24, g = n * u / (1.0 - n * u);
  return g * g + 0x1.0p-53;
}

int Call::finish(nspb_stats *stats) {
  if ((opts.check_errors || opts.precision == NSPB_PREC_FP32_COMP) && n > 0) {
    int st = fetch_counters();
    if (st) return st;
  }
  if (stats) {
    stats->intprod = intprod;
    stats->nnz = h.total_nnz;
    for (int b = 0; b < 16; ++b) {
      stats->sym_bins[b] = b < kSymBins ? h.sym_counts[b] : 0;
      stats->num_bins[b] = b < kNumBins ? h.num_counts[b] : 0;
    }
    stats->b_sorted = b_sorted ? 1 : 0;
    stats->rows_redone = opts.precision == NSPB_PREC_FP32_COMP ? h.redo_count : 0;
    stats->max_row_err = opts.precision == NSPB_PREC_FP32_COMP ? comp_bound(h.max_comp_deg) : 0.0;
    stats->launches = launches;
    stats->entry_map = use_map ? 1 : 0;
    stats->ms_rowinfo = stats->ms_symbolic = stats->ms_scan = stats->ms_numeric = 0.f;
    if (timing && n > 0) {
      cudaStreamSynchronize(s);
      auto span = [&](int a, int b) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, ev[a], ev[b]) != cudaSuccess) {
          cudaGetLastError();
          ms = 0.f;
        }
        return ms;
      };
      stats->ms_rowinfo = span(0, 1);
      stats->ms_symbolic = span(2, 3);
      stats->ms_scan = span(3, 4);
      stats->ms_numeric = span(5, 6);
    }
  }
  return NSPB_OK;
}

}  // namespace nspb

using namespace nspb;

extern "C" {

const char *nspb_version(void) { return "nspb 0.1 (sm_100a)"; }

const char *nspb_strerror(int status) {
  switch (status) {
    case NSPB_OK: return "success";
    case NSPB_ERR_INVALID: return "invalid argument";
    case NSPB_ERR_OVERFLOW: return "nnz(C) or a row count exceeds int32";
    case NSPB_ERR_ALLOC: return "allocation failed";
    case NSPB_ERR_CUDA: return "CUDA runtime error";
    case NSPB_ERR_DEVICE: return "device error word set (bounded probe or wait exhausted)";
    case NSPB_ERR_NO_DEVICE: return "no CUDA device";
    case NSPB_ERR_UNSUPPORTED: return "unsupported";
    case NSPB_ERR_CAPACITY: return "output capacity too small";
    case NSPB_ERR_IO: return "file could not be opened, read or written";
    default: return "unknown status";
  }
}

int nspb_last_cuda_error(void) { return g_last_cuda; }

void nspb_default_opts(nspb_opts *o) {
  if (!o) return;
  std::memset(o, 0, sizeof(*o));
  o->precision = NSPB_PREC_FP64;
  o->comp_tol = 1e-10;
}

int nspb_device_sm_count(int *sms) {
  int ndev = 0;
  if (!sms) return NSPB_ERR_INVALID;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return NSPB_ERR_NO_DEVICE;
  }
  *sms = dev_info().sms;
  return NSPB_OK;
}

int nspb_spgemm_symbolic(const nspb_csr_in *A, const nspb_csr_in *B, nspb_csr_out *C,
                         const nspb_opts *opts, nspb_stats *stats) {
  if (!C) return NSPB_ERR_INVALID;
  Call call;
  int st = call.init(A, B, opts);
  if (st) return st;
  call.allow_map = false;  // the numeric phase runs in another call
  call.two_calls = true;
  bool own_rpt = false;
  if (!C->rowptr) {
    if ((st = alloc_out(reinterpret_cast<void **>(&C->rowptr), ((size_t)call.n + 1) * 4))) return st;
    own_rpt = true;
  }
  int64_t nnz = 0;
  st = call.symbolic(C->rowptr, &nnz);
  if (!st) st = call.finish(stats);
  if (st) {
    if (own_rpt) {
      cudaStreamSynchronize(call.s);
      cudaFree(C->rowptr);
      C->rowptr = nullptr;
    }
    return st;
  }
  C->nrows = A->nrows;
  C->ncols = B->ncols;
  C->nnz = nnz;
  return NSPB_OK;
}

int nspb_spgemm_numeric(const nspb_csr_in *A, const nspb_csr_in *B, nspb_csr_out *C,
                        const nspb_opts *opts, nspb_stats *stats) {
  if (!C || !C->rowptr) return NSPB_ERR_INVALID;
  Call call;
  int st = call.init(A, B, opts);
  if (st) return st;
  if (C->nnz < 0 || C->nnz > INT32_MAX) return NSPB_ERR_INVALID;
  if ((C->col || C->val) && (!C->col || !C->val)) return NSPB_ERR_INVALID;
  if (C->col && C->capacity < C->nnz) return NSPB_ERR_CAPACITY;
  if ((st = call.prepare_numeric(C->rowptr, C->nnz))) return st;
  call.h.total_nnz = C->nnz;
  bool own = false;
  if (!C->col) {
    if ((st = alloc_out(reinterpret_cast<void **>(&C->col), (size_t)C->nnz * 4))) return st;
    if ((st = alloc_out(reinterpret_cast<void **>(&C->val), (size_t)C->nnz * 8))) {
      cudaFree(C->col);
      C->col = nullptr;
      return st;
    }
    own = true;
    C->capacity = C->nnz;
  }
  st = call.numeric(C->rowptr, C->col, C->val);
  if (!st) st = call.finish(stats);
  if (st && own) {
    cudaStreamSynchronize(call.s);
    cudaFree(C->col);
    cudaFree(C->val);
    C->col = nullptr;
    C->val = nullptr;
  }
  return st;
}

int nspb_spgemm(const nspb_csr_in *A, const nspb_csr_in *B, nspb_csr_out *C,
                const nspb_opts *opts, nspb_stats *stats) {
  if (!C) return NSPB_ERR_INVALID;
  if ((C->col || C->val) && (!C->col || !C->val)) return NSPB_ERR_INVALID;
  Call call;
  int st = call.init(A, B, opts);
  if (st) return st;
  bool own_rpt = false, own_cv = false;
  if (!C->rowptr) {
    if ((st = alloc_out(reinterpret_cast<void **>(&C->rowptr), ((size_t)call.n + 1) * 4))) return st;
    own_rpt = true;
  }
  int64_t nnz = 0;
  st = call.symbolic(C->rowptr, &nnz);
  if (!st) {
    if (!C->col) {
      st = alloc_out(reinterpret_cast<void **>(&C->col), (size_t)nnz * 4);
      if (!st) {
        st = alloc_out(reinterpret_cast<void **>(&C->val), (size_t)nnz * 8);
        if (st) {
          cudaFree(C->col);
          C->col = nullptr;
        }
      }
      own_cv = !st;
      if (!st) C->capacity = nnz;
    } else if (C->capacity < nnz) {
      st = NSPB_ERR_CAPACITY;
    }
  }
  if (!st) st = call.numeric(C->rowptr, C->col, C->val);
  if (!st) st = call.finish(stats);
  if (st) {
    cudaStreamSynchronize(call.s);
    if (own_cv) {
      cudaFree(C->col);
      cudaFree(C->val);
      C->col = nullptr;
      C->val = nullptr;
    }
    if (own_rpt) {
      cudaFree(C->rowptr);
      C->rowptr = nullptr;
    }
    return st;
  }
  C->nrows = A->nrows;
  C->ncols = B->ncols;
  C->nnz = nnz;
  return NSPB_OK;
}

int nspb_intprod(const nspb_csr_in *A, const nspb_csr_in *B, int64_t *d_row_ip, int64_t *total,
                 void *stream) {
  nspb_opts o;
  nspb_default_opts(&o);
  o.stream = stream;
  o.assume_sorted = 1;
  // values are not read: accept either value type
  o.precision = (A && A->val_type == NSPB_F32) ? NSPB_PREC_FP32_COMP : NSPB_PREC_FP64;
  Call call;
  int st = call.init(A, B, &o);
  if (st) return st;
  if (call.n == 0) {
    if (total) *total = 0;
    return NSPB_OK;
  }
  if ((st = call.alloc_scratch())) return st;
  cudaError_t e = launch_rowinfo(structure_of(call.t64), call.n, call.a_nnz, call.lim, call.row_nz,
                                 d_row_ip, call.ctr->sym_counts,
                                 &call.ctr->total_ip, nullptr, call.perm, &call.ctr->long_rows,
                                 RunScan(), call.s);
  if (e != cudaSuccess) return call.cuda_fail(e);
  if ((st = call.fetch_counters())) return st;
  if (total) *total = (int64_t)call.h.total_ip;
  return NSPB_OK;
}

}  // extern "C"
