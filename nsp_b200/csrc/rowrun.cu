// Row runs: rows of C that repeat one pattern at a fixed distance.
//
// Reference counterparts (amavliut/nsp): none. The reference hashes every row
// twice (nsp/src/nsp.cu:477-1130 and :1307-2440) whatever its neighbours hold.
//
// On structured grids, row i of A is row i - s with every column moved by
// sigma, and the B rows that it reads are those of row i - s moved by one
// column shift: A*A of a stencil has s = sigma = 1, A*P of an aggregation
// with aggregates of three nodes has s = sigma = 3, R*(A P) has s = 1 and
// sigma = 3. The products of such a row fall on entries of C exactly as those
// of row i - s do. Rows linked in this way form runs (k_rowinfo finds the
// links, k_run_list the runs); nothing here assumes a grid, every link is
// checked on the columns themselves.
//
// Runs of one pattern share a program (k_run_key finds the patterns by hash
// and compares them exactly, k_run_prog writes the programs): the products of
// a row sorted once by (column, walk order), which gives the rows' count and
// columns and tells what to add to each entry. The rows of a run need no hash
// table, no map and no sort in either phase. In the numeric phase
// (k_num_run) lanes are rows; a warp takes some entries of C for 32 rows and
// sums each entry's products in registers, in A-row order from zero, so values
// equal the hash kernels' bit for bit.
#include "common.cuh"
#include "internal.h"
#include "launch_util.h"

#include <cuda_pipeline.h>

#include <algorithm>

namespace nspb {

// ---- column shifts of B's rows ----------------------------------------------------
// bdel[(g-1) * nb + k]: the shift that moves B row k - g onto row k, or
// kNoShift, and the length of row k. For g > 1 the g rows before k must also take as many entries as
// the g rows before those, so that along a chain k, k+g, k+2g, ... the rows
// start at equal distances in memory (for g = 1 equal lengths give that).
// The order of the rows is checked on the way (flags).
// A thread a row over columns staged in shared memory (common.cuh): a group
// of lanes a row took 200 instructions of a warp a row, 571 us on the 27-point
// 128^3 stencil.
template <bool MULTI>
__global__ void __launch_bounds__(kTileThreads)
    k_brow_delta(const ProdTable<void> src, int tile, int *__restrict__ lag_count,
                 int *__restrict__ flags) {
  __shared__ int s_cnt[kMaxLag];
  __shared__ int cols[kTileWords];
  __shared__ int rp[kTileThreads + 2 * kMaxLag + 1];  // row starts from row r0 - 6 on
  __shared__ int s_long[kTileThreads], s_nlong;       // rows too long for one thread
  constexpr int kHalo = 2 * kMaxLag;
  if (threadIdx.x < kMaxLag) s_cnt[threadIdx.x] = 0;
  const Operands<void> o = MULTI ? src.ops[blockIdx.y] : src.one;
  const int nb = o.brows;
  int mine[kMaxLag] = {0, 0, 0};
  int bad = 0;
  for (long long first = (long long)blockIdx.x * tile; first < nb;
       first += (long long)gridDim.x * tile) {
    const int r0 = (int)first, nr = min(tile, nb - r0);
    __syncthreads();  // the last tile is read
    if (threadIdx.x == 0) s_nlong = 0;
    for (int i = threadIdx.x; i <= nr + kHalo; i += kTileThreads)
      rp[i] = __ldg(o.brpt + max(r0 - kHalo + i, 0));
    __syncthreads();
    const int e0 = rp[kHalo - min(kMaxLag, r0)], e1 = rp[nr + kHalo];
    const bool staged = e1 - e0 <= kTileCols;
    const int skew = tile_skew(rp[nr / 2 + kHalo + 1] - rp[nr / 2 + kHalo]);
    if (staged) {
      tile_stage(o.bcol, e0, e1, skew, cols);
      __syncthreads();
    }
    with_cols(staged, skew, cols, e0, o.bcol, [&](auto col) {
      const int q = threadIdx.x;
      if (q >= nr) return;
      const int k = r0 + q;
      const int *p = rp + q + kHalo;  // p[-g]: start of row k - g
      const int s0 = p[0], len = p[1] - s0;
      const int walk = len > kShiftMaxLen ? 0 : len;
      if (len > kShiftMaxLen) s_long[atomicAdd(&s_nlong, 1)] = q;  // its order: the block, below
      bool ok[kMaxLag];
      int at[kMaxLag], d[kMaxLag];  // start of the row compared with, shift
#pragma unroll
      for (int g = 1; g <= kMaxLag; ++g) {
        bool x = k >= g && len <= kShiftMaxLen && p[1 - g] - p[-g] == len;
        if (g > 1) x = x && k >= 2 * g && s0 - p[-g] == p[-g] - p[-2 * g];
        if (x && len > 0) {  // most rows that are no shift differ at the ends already
          d[g - 1] = col(s0) - col(p[-g]);
          x = col(s0 + len - 1) - col(p[-g] + len - 1) == d[g - 1];
        } else {
          d[g - 1] = kAnyShift;
        }
        ok[g - 1] = x;
        at[g - 1] = p[-g];
      }
      int prev = -1, wrong = 0;
      if (ok[0] || ok[1] || ok[2]) {
        // a lag that is out is compared with the row itself
#pragma unroll
        for (int g = 0; g < kMaxLag; ++g)
          if (!ok[g]) at[g] = s0;
        int off[kMaxLag] = {0, 0, 0};
#pragma unroll 4
        for (int e = 0; e < walk; ++e) {
          const int c = col(s0 + e);
          wrong |= c <= prev;
          prev = c;
#pragma unroll
          for (int g = 0; g < kMaxLag; ++g) off[g] |= (c - col(at[g] + e)) ^ d[g];
        }
#pragma unroll
        for (int g = 0; g < kMaxLag; ++g) ok[g] = ok[g] && (off[g] == 0 || walk == 0);
      } else {
#pragma unroll 4
        for (int e = 0; e < walk; ++e) {
          const int c = col(s0 + e);
          wrong |= c <= prev;
          prev = c;
        }
      }
      bad |= wrong;
#pragma unroll
      for (int g = 0; g < kMaxLag; ++g) {
        o.bdel[(long long)g * nb + k] = make_int2(ok[g] ? d[g] : kNoShift, len);
        mine[g] += ok[g];
      }
    });
    if (!flags) continue;
    __syncthreads();
    for (int i = 0; i < s_nlong; ++i) {
      const int s0 = rp[s_long[i] + kHalo], s1 = rp[s_long[i] + kHalo + 1];
#pragma unroll 4
      for (int e = s0 + 1 + (int)threadIdx.x; e < s1; e += kTileThreads)
        bad |= __ldg(o.bcol + e) <= __ldg(o.bcol + e - 1);
    }
  }
#pragma unroll
  for (int g = 0; g < kMaxLag; ++g) {
    int v = mine[g];
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) v += __shfl_xor_sync(0xffffffffu, v, w);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&s_cnt[g], v);
  }
  if (__syncthreads_or(bad) && flags && threadIdx.x == 0) atomicOr(flags, B_UNSORTED);
  if (threadIdx.x < kMaxLag && s_cnt[threadIdx.x])
    atomicAdd(lag_count + 1 + threadIdx.x, s_cnt[threadIdx.x]);
}

cudaError_t launch_brow_delta(const ProdTable<void> &t, const ProdInfo &info, int64_t b_nnz,
                              int *lag_count, int *flags, cudaStream_t s) {
  if (info.brows <= 0) return cudaSuccess;
  const int tile = tile_rows((double)b_nnz / (double)info.brows);
  const bool multi = t.prod_of_row != nullptr;
  const int gx = (int)std::min<long long>(((long long)info.max_brows + tile - 1) / tile,
                                          (long long)dev_info().sms * 16);
  const dim3 grid(gx, multi ? info.nprod : 1);
  auto kern = multi ? k_brow_delta<true> : k_brow_delta<false>;
  kern<<<grid, kTileThreads, 0, s>>>(t, tile, lag_count, flags);
  return cudaGetLastError();
}

// ---- the runs ---------------------------------------------------------------------
// Rows linked with one (s, sigma) form a run: the first of them, or the row
// that it is linked to when that row has no link of its own and no shorter
// distance claims it, starts it. Runs end at multiples of kRunBlock rows, so
// that a block finds them alone and no run grows past kRunBlock rows. How many
// links follow each row comes from pointer doubling (a walk by the first row's
// thread took 59 us on the 27-point 128^3 stencil).
constexpr int kRunBlock = 512;

__global__ void __launch_bounds__(kRunBlock)
    k_run_list(unsigned char *__restrict__ codes, int n, RowRun *__restrict__ found,
               int *__restrict__ nfound) {
  __shared__ unsigned char code[kRunBlock];
  __shared__ short links[2][kRunBlock];  // rows of the code from here on, doubling
  __shared__ RowRun run[kRunBlock / kRunMin + 1];
  __shared__ int s_n, s_base;
  const int t = threadIdx.x;
  const int b0 = blockIdx.x * kRunBlock;
  const int cnt = min(kRunBlock, n - b0);
  const int c = t < cnt ? codes[b0 + t] : 0;
  code[t] = (unsigned char)c;
  links[0][t] = c ? 1 : 0;
  if (t == 0) s_n = 0;
  const int s = c & 3;
  int side = 0;
  const bool any = __syncthreads_or(c);
  for (int w = 1; any && w < kRunBlock; w <<= 1, side ^= 1) {
    int v = links[side][t];
    const int j = t + s * w;
    if (c && v == w && j < cnt && code[j] == c) v += links[side][j];
    links[side ^ 1][t] = (short)v;
    __syncthreads();
  }
  if (c && !(t >= s && code[t - s] == c)) {
    int first = t, len = links[side][t];
    if (t >= s && code[t - s] == 0) {
      bool mine = true;
      for (int g = 1; g < s; ++g) mine = mine && (code[t - s + g] & 3) != g;
      if (mine) {
        first = t - s;
        ++len;
      }
    }
    if (len >= kRunMin)
      run[atomicAdd(&s_n, 1)] = RowRun{b0 + first, s | (c >> 2 & 3) << 2 | len << 4, -1, 0};
  }
  __syncthreads();
  if (t == 0 && s_n) s_base = atomicAdd(nfound, s_n);
  if (c) codes[b0 + t] = 0;  // the members' flags are set by k_run_key
  __syncthreads();
  if (t < s_n) found[s_base + t] = run[t];
}

// ---- the programs -----------------------------------------------------------------
// Two sizes of the numeric kernel: rows of few products leave little to share
// out among 16 warps, and many small blocks hide the waits between their steps.
// WARPS compute, LOOK warps look up tiles.
template <int CLASS>
struct RunCfg;
template <>
struct RunCfg<0> {  // rows of at most kRunSmallIp products
  static constexpr int WARPS = 8, LOOK = 2, SMEM = 50 * 1024, MINB = 4;
};
template <>
struct RunCfg<1> {
  static constexpr int WARPS = 16, LOOK = 1, SMEM = 110000, MINB = 2;
};
constexpr int kRunSmallIp = 256;
constexpr int kRunRows = 128;  // most rows of a tile

// A program as k_run_prog leaves it in global memory. The words, one per
// product:
//   x = byte of the staged B values that row 0 multiplies | the distance from
//       one row's to the next << 17 (elements; 0 where `step` gives it)
//   y = byte of the A entry in its row | rank of the entry of C << 11 |
//       segment of B << 22 | last product of its entry << 31
// Entries are dealt to the warps by descending product count, alternately
// forwards and backwards, so that warps get nearly equal shares.
struct RunProg {
  int na, p, n;          // A entries, products and entries of a row
  int rows;              // most rows of a tile
  int parts;             // warps that share a row group
  int segs;              // segments of B a tile stages
  int t0;                // first A entry with products
  int step;              // distance of all words from one row to the next, or -1
  int belems;            // elements of the staged B area
  int w0[16], w1[16];    // words of each part
  unsigned char seg0[kRunMaxA], seg1[kRunMaxA];  // first and last A entry of a segment
  int dst[kRunMaxA];     // its place
  int rel[kRunMaxIp];    // columns of the row less the first product's
  uint2 word[kRunMaxIp + 32];
  // bunches: the A entry of every product, products before every A entry
  unsigned char term[kRunMaxIp];
  short before[kRunMaxA + 1];
};
static_assert(kRunMaxA <= 128 && kRunMaxIp < 2048, "fields of a program word");

size_t run_prog_bytes() { return sizeof(RunProg); }

// One A entry of a run's first row: its B row, where that starts and how long
// it is, and the distance to the start of the row sigma on.
struct RunTerm {
  int k, bs, len, pl;
};
__device__ __forceinline__ RunTerm run_term(const Operands<void> &o, int e, int sigma) {
  RunTerm r;
  r.k = __ldg(o.acol + e);
  r.bs = __ldg(o.brpt + r.k);
  r.len = __ldg(o.brpt + r.k + 1) - r.bs;
  r.pl = __ldg(o.brpt + r.k + sigma) - r.bs;
  return r;
}
// Entries t - 1 and t may share a segment of B: their B rows lie near each
// other and move by the same distance from row to row, so that their places
// keep their distance in every tile.
constexpr int kSegReach = 512;
__device__ __forceinline__ bool run_near(int k, int pl, int pk, int ppl) {
  return k >= pk && k - pk <= kSegReach && pl == ppl;
}

__device__ __forceinline__ unsigned run_mix(unsigned a, unsigned b) {
  a = (a ^ (b * 0x9e3779b1u)) * 0x85ebca6bu;
  a ^= a >> 15;
  a *= 0xc2b2ae35u;
  return a ^ (a >> 16);
}

// An entry of a table of representatives.
__device__ __forceinline__ unsigned long long run_entry(unsigned hash, int index) {
  return (unsigned long long)hash << 32 | (unsigned)(index + 1);
}

// Patterns of the runs: a warp a run hashes everything that its program
// depends on and looks for a run with the same pattern in a table of
// representatives; a run that finds one is compared with it, value by value.
// Runs that find no place in the table are dropped (prog -1) and their rows
// computed like any others. Runs kept take a place in their pattern, and their
// rows are marked and taken out of the symbolic bins.
template <bool MULTI>
__global__ void __launch_bounds__(256)
    k_run_key(const ProdTable<void> src, RowRun *__restrict__ found, const BinLimits lim,
              unsigned char *__restrict__ member, int *__restrict__ row_nz, const RunTable rt,
              int *__restrict__ sym_sub) {
  __shared__ int hist[kSymBins];
  if (threadIdx.x < kSymBins) hist[threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int total = rt.head->nfound;
  for (int q = (blockIdx.x * 256 + threadIdx.x) >> 5; q < total; q += gridDim.x * 8) {
    const RowRun rd = found[q];
    const int s = rd.meta & 3, sigma = rd.meta >> 2 & 3, len = rd.meta >> 4;
    Operands<void> o;
    const int lr = prod_row<MULTI>(src, rd.row0, o);
    const int a0 = __ldg(o.arpt + lr), na = __ldg(o.arpt + lr + 1) - a0;
    // hash and product count; a lane takes an A entry and its B row
    unsigned h = 0;
    int P = 0, cb = 0;
    bool have = false;
    for (int c = 0; c < na; c += 32) {
      const int t = c + lane;
      RunTerm r{0, 0, 0, 0}, p{0, 0, 0, 0};
      if (t < na) r = run_term(o, a0 + t, sigma);
      p.k = __shfl_up_sync(0xffffffffu, r.k, 1);
      p.bs = __shfl_up_sync(0xffffffffu, r.bs, 1);
      p.pl = __shfl_up_sync(0xffffffffu, r.pl, 1);
      if (t < na && lane == 0 && t > 0) p = run_term(o, a0 + t - 1, sigma);
      const unsigned some = __ballot_sync(0xffffffffu, r.len > 0);
      if (some && !have) {
        cb = __ldg(o.bcol + __shfl_sync(0xffffffffu, r.bs, __ffs(some) - 1));
        have = true;
      }
      if (t < na) {
        unsigned w = run_mix((unsigned)r.len, (unsigned)r.pl);
        if (t > 0 && run_near(r.k, r.pl, p.k, p.pl))
          w = run_mix(w, (unsigned)(r.k - p.k) * 31u + (unsigned)(r.bs - p.bs));
        h += run_mix(w, (unsigned)t + 1u);
#pragma unroll 4
        for (int e = 0; e < r.len; ++e)
          h += run_mix((unsigned)(__ldg(o.bcol + r.bs + e) - cb), (unsigned)(t * 2048 + e) + 0x10000u);
        P += r.len;
      }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      h += __shfl_xor_sync(0xffffffffu, h, d);
      P += __shfl_xor_sync(0xffffffffu, P, d);
    }
    h = run_mix(h, (unsigned)na * 4u + (unsigned)sigma);
    int slot = -1;
    for (int tries = 0; tries < 16 && slot < 0; ++tries) {
      const int at = (int)((h + (unsigned)tries) & (kRunSlots - 1));
      unsigned long long entry = 0;
      if (lane == 0) {
        entry = *(volatile unsigned long long *)(rt.rep + at);
        if (entry == 0) entry = atomicCAS(rt.rep + at, 0ull, run_entry(h, q));
      }
      entry = __shfl_sync(0xffffffffu, entry, 0);
      if (entry == 0) {  // the first of its pattern
        slot = at;
        if (lane == 0) {
          const int p = atomicAdd(&rt.head->nprog, 1);
          rt.prog_of[at] = p;
          rt.run_of[p] = q;
          rt.slot_of[p] = at | (P > kRunSmallIp) << 16;
        }
        break;
      }
      // the same pattern as the representative's?
      if ((unsigned)(entry >> 32) != h) continue;
      const int rep = (int)(unsigned)entry;
      const RowRun other{found[rep - 1].row0, found[rep - 1].meta, 0, 0};
      if ((other.meta >> 2 & 3) != sigma) continue;
      Operands<void> o2;
      const int lr2 = prod_row<MULTI>(src, other.row0, o2);
      const int a2 = __ldg(o2.arpt + lr2);
      if (__ldg(o2.arpt + lr2 + 1) - a2 != na) continue;
      bool diff = false;
      int cb2 = 0;
      bool have2 = false;
      for (int c = 0; c < na && !diff; c += 32) {
        const int t = c + lane;
        RunTerm r{0, 0, 0, 0}, r2{0, 0, 0, 0};
        if (t < na) {
          r = run_term(o, a0 + t, sigma);
          r2 = run_term(o2, a2 + t, sigma);
          diff = r.len != r2.len || r.pl != r2.pl;
          if (t > 0) {
            const RunTerm p = run_term(o, a0 + t - 1, sigma), p2 = run_term(o2, a2 + t - 1, sigma);
            const bool near = run_near(r.k, r.pl, p.k, p.pl);
            diff |= near != run_near(r2.k, r2.pl, p2.k, p2.pl);
            diff |= near && (r.k - p.k != r2.k - p2.k || r.bs - p.bs != r2.bs - p2.bs);
          }
        }
        const unsigned some = __ballot_sync(0xffffffffu, r2.len > 0);
        if (some && !have2) {
          cb2 = __ldg(o2.bcol + __shfl_sync(0xffffffffu, r2.bs, __ffs(some) - 1));
          have2 = true;
        }
        if (!diff) {
#pragma unroll 4
          for (int e = 0; e < r.len; ++e)
            diff |= __ldg(o.bcol + r.bs + e) - cb != __ldg(o2.bcol + r2.bs + e) - cb2;
        }
        diff = __any_sync(0xffffffffu, diff);
      }
      if (!diff) slot = at;
    }
    if (lane == 0) {
      const int large = P > kRunSmallIp;
      found[q].prog = slot;
      if (slot >= 0) {
        atomicAdd(&rt.head->nruns[large], 1);
        found[q].place = atomicAdd(rt.count + slot, 1);
        const int ub = row_nz[rd.row0];
        if (ub > 0) atomicAdd(&hist[sym_bin(ub, lim)], len);
      }
    }
    if (slot < 0) continue;
    __syncwarp();
    for (int m = lane; m < len; m += 32) {
      member[rd.row0 + s * m] = 1;
      row_nz[rd.row0 + s * m] = 0;
    }
  }
  __syncthreads();
  if (threadIdx.x < kSymBins && hist[threadIdx.x])
    atomicAdd(&sym_sub[threadIdx.x], hist[threadIdx.x]);
}

cudaError_t launch_run_find(const ProdTable<void> &t, unsigned char *codes, int n,
                            const BinLimits &lim, int *row_nz, RowRun *found,
                            const RunTable &rt, int *sym_sub, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_run_list<<<(n + kRunBlock - 1) / kRunBlock, kRunBlock, 0, s>>>(codes, n, found,
                                                                   &rt.head->nfound);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int cap = (int)run_capacity(n);
  const int grid = std::max(1, std::min((cap + 7) / 8, dev_info().sms * 8));
  auto kern = t.prod_of_row ? k_run_key<true> : k_run_key<false>;
  kern<<<grid, 256, 0, s>>>(t, found, lim, codes, row_nz, rt, sym_sub);
  return cudaGetLastError();
}

// ---- bunches ------------------------------------------------------------------------
// Rows that no run took (the ends of grid lines above all) still share their
// patterns with many others, at no fixed distance. They are grouped by pattern
// alone, with the same hash, table and exact comparison as the runs, and
// computed by the same programs, each row's B values staged on their own. On
// the 27-point 128^3 stencil the 65,536 rows at the ends of its lines took 297
// us in k_sym_map and 305 us in k_num_map, a fifth of the product.
//
// Rows without structure all differ: hashing 1.6 M of them on a 7-point grid
// took 1.6 ms of 7.5, and 4096 programs for one row each 0.9 ms more on a
// 27-point one. The search therefore ends after kBunchNew rows that met no
// earlier row's pattern (the grids and their aggregation products have 27 to
// 730 patterns).
constexpr int kBunchNew = 2048;
constexpr int kBunchBits = 19;  // place of a row in its slot; slots take the bits above
static_assert(kRunSlots <= 1 << (31 - kBunchBits), "slot and place in one int");

template <bool MULTI>
__global__ void __launch_bounds__(256, MULTI ? 5 : 8)
    k_bunch_key(const ProdTable<void> src, const unsigned char *__restrict__ member, int n,
                const int *__restrict__ row_nz, const RunTable rt, int *__restrict__ slot_of) {
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * 8;
  int seen = 0;  // of the last eight rows: looked at, and << 8 those that met no pattern; -1: no more
  for (int base = ((blockIdx.x * 256 + threadIdx.x) >> 5) * 32; base < n; base += warps * 32) {
    const int mine = base + lane;
    int my_slot = -1;
    unsigned todo =
        __ballot_sync(0xffffffffu, seen >= 0 && mine < n && !member[mine] && row_nz[mine] > 0);
    while (todo) {
      const int w = __ffs(todo) - 1;
      todo &= todo - 1u;
      const int row = base + w;
      Operands<void> o;
      const int lr = prod_row<MULTI>(src, row, o);
      const int a0 = __ldg(o.arpt + lr), na = __ldg(o.arpt + lr + 1) - a0;
      if (na > kRunMaxA) continue;
      unsigned h = 0;
      int P = 0, cb = 0;
      bool have = false;
      for (int c = 0; c < na; c += 32) {
        const int t = c + lane;
        int bs = 0, len = 0;
        if (t < na) {
          const int k = __ldg(o.acol + a0 + t);
          bs = __ldg(o.brpt + k);
          len = run_len(__ldg(o.brpt + k + 1) - bs);
        }
        // a row of too many products is left before its columns are read
        int total = len;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) total += __shfl_xor_sync(0xffffffffu, total, d);
        P += total;
        if (P > kRunMaxIp) {
          P = kRunMaxIp + 1;
          break;
        }
        const unsigned some = __ballot_sync(0xffffffffu, len > 0);
        if (some && !have) {
          cb = __ldg(o.bcol + __shfl_sync(0xffffffffu, bs, __ffs(some) - 1));
          have = true;
        }
        if (t < na) {
          h += run_mix((unsigned)len, (unsigned)t + 1u);
#pragma unroll 4
          for (int e = 0; e < len; ++e)
            h += run_mix((unsigned)(__ldg(o.bcol + bs + e) - cb),
                         (unsigned)(t * 2048 + e) + 0x10000u);
        }
      }
      if (P <= 0 || P > kRunMaxIp) continue;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) h += __shfl_xor_sync(0xffffffffu, h, d);
      int prod = 0;
      if constexpr (MULTI) prod = __ldg(src.prod_of_row + row);
      h = run_mix(h, (unsigned)na + (unsigned)prod * 0x9e37u);
      int slot = -1;
      for (int tries = 0; tries < 16 && slot < 0; ++tries) {
        const int at = (int)((h + (unsigned)tries) & (kRunSlots - 1));
        unsigned long long entry = 0;
        if (lane == 0) {
          entry = *(volatile unsigned long long *)(rt.brep + at);
          if (entry == 0) entry = atomicCAS(rt.brep + at, 0ull, run_entry(h, row));
        }
        entry = __shfl_sync(0xffffffffu, entry, 0);
        if (entry == 0) {
          slot = at;
          seen += 0x100;
          break;
        }
        if ((unsigned)(entry >> 32) != h) continue;
        const int rep = (int)(unsigned)entry;
        Operands<void> o2;
        const int lr2 = prod_row<MULTI>(src, rep - 1, o2);
        if constexpr (MULTI)
          if (__ldg(src.prod_of_row + rep - 1) != prod) continue;
        const int a2 = __ldg(o2.arpt + lr2);
        if (__ldg(o2.arpt + lr2 + 1) - a2 != na) continue;
        bool diff = false, have2 = false;
        int cb2 = 0;
        for (int c = 0; c < na && !diff; c += 32) {
          const int t = c + lane;
          int bs = 0, len = 0, bs2 = 0, len2 = 0;
          if (t < na) {
            const int k = __ldg(o.acol + a0 + t), k2 = __ldg(o2.acol + a2 + t);
            bs = __ldg(o.brpt + k);
            len = run_len(__ldg(o.brpt + k + 1) - bs);
            bs2 = __ldg(o2.brpt + k2);
            len2 = run_len(__ldg(o2.brpt + k2 + 1) - bs2);
            diff = len != len2;
          }
          const unsigned some = __ballot_sync(0xffffffffu, len2 > 0);
          if (some && !have2) {
            cb2 = __ldg(o2.bcol + __shfl_sync(0xffffffffu, bs2, __ffs(some) - 1));
            have2 = true;
          }
          if (!diff) {
#pragma unroll 4
            for (int e = 0; e < len; ++e)
              diff |= __ldg(o.bcol + bs + e) - cb != __ldg(o2.bcol + bs2 + e) - cb2;
          }
          diff = __any_sync(0xffffffffu, diff);
        }
        if (!diff) slot = at;
      }
      int place = 0;
      seen += slot < 0 ? 0x101 : 1;
      if ((seen & 0xff) == 8) {
        if (seen >= 0x100) {
          int before = 0;
          if (lane == 0) before = atomicAdd(&rt.head->bnew, seen >> 8);
          seen = __shfl_sync(0xffffffffu, before, 0) >= kBunchNew ? -1 : 0;
          if (seen < 0) todo = 0;
        } else {
          seen = 0;
        }
      }
      if (slot >= 0) {
        if (lane == 0) place = atomicAdd(rt.bcount + slot, 1);
        place = __shfl_sync(0xffffffffu, place, 0);
      }
      if (lane == w && slot >= 0 && place < (1 << kBunchBits)) my_slot = slot << kBunchBits | place;
    }
    if (mine < n) slot_of[mine] = my_slot;
  }
}

// Used slots become bunches, in slot order; one block, kRunSlots / 1024 slots a
// thread. Where there are more than kBunchAll patterns, those of fewer than
// kBunchMin rows are left to the other kernels: a program takes as long as those
// need for about 24 rows (0.2 us).
constexpr int kBunchAll = 1024, kBunchMin = 24;

__global__ void __launch_bounds__(1024) k_bunch_plan(const RunTable rt) {
  constexpr int kPer = kRunSlots / 1024;
  __shared__ int s_rows[32], s_num[32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  int c[kPer], used = 0;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    c[i] = min(rt.bcount[t * kPer + i], 1 << kBunchBits);
    used += c[i] > 0;
  }
  used = __reduce_add_sync(0xffffffffu, used);
  if (lane == 0) s_num[warp] = used;
  __syncthreads();
  const bool many = __reduce_add_sync(0xffffffffu, s_num[lane]) > kBunchAll;
  __syncthreads();  // s_num
  int rows = 0, num = 0;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    if (many && c[i] < kBunchMin) {
      rt.bslot[t * kPer + i] = -1;
      c[i] = 0;
    }
    rows += c[i];
    num += c[i] > 0;
  }
  const int own_rows = rows, own_num = num;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, rows, d), b = __shfl_up_sync(0xffffffffu, num, d);
    if (lane >= d) {
      rows += a;
      num += b;
    }
  }
  if (lane == 31) {
    s_rows[warp] = rows;
    s_num[warp] = num;
  }
  __syncthreads();
  for (int w = 0; w < warp; ++w) {
    rows += s_rows[w];
    num += s_num[w];
  }
  if (t == 1023) rt.head->nbunch = num;
  int place = rows - own_rows, b = num - own_num;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    if (c[i] == 0) continue;
    const int slot = t * kPer + i;
    rt.bslot[slot] = place;
    rt.brow[b] = (int)(unsigned)rt.brep[slot] - 1;
    rt.brows[b] = c[i];
    rt.bplace[b] = place;
    place += c[i];
    ++b;
  }
}

__global__ void __launch_bounds__(256)
    k_bunch_list(const int *__restrict__ slot_of, int n, const RunTable rt, const BinLimits lim,
                 unsigned char *__restrict__ member, int *__restrict__ row_nz,
                 int *__restrict__ list, int *__restrict__ sym_sub) {
  __shared__ int hist[kSymBins];
  if (threadIdx.x < kSymBins) hist[threadIdx.x] = 0;
  __syncthreads();
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
    const int v = slot_of[i];
    if (v < 0) continue;
    const int first = rt.bslot[v >> kBunchBits];
    if (first < 0) continue;
    list[first + (v & ((1 << kBunchBits) - 1))] = i;
    member[i] = 1;
    const int ub = row_nz[i];
    if (ub > 0) atomicAdd(&hist[sym_bin(ub, lim)], 1);
    row_nz[i] = 0;
  }
  __syncthreads();
  if (threadIdx.x < kSymBins && hist[threadIdx.x])
    atomicAdd(&sym_sub[threadIdx.x], hist[threadIdx.x]);
}

cudaError_t launch_bunch_find(const ProdTable<void> &t, unsigned char *member, int n,
                              const BinLimits &lim, int *row_nz, const RunTable &rt, int *slot,
                              int *list, int *sym_sub, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int grid = std::min((n + 255) / 256, dev_info().sms * 8);
  auto kern = t.prod_of_row ? k_bunch_key<true> : k_bunch_key<false>;
  kern<<<grid, 256, 0, s>>>(t, member, n, row_nz, rt, slot);
  k_bunch_plan<<<1, 1024, 0, s>>>(rt);
  k_bunch_list<<<grid, 256, 0, s>>>(slot, n, rt, lim, member, row_nz, list, sym_sub);
  return cudaGetLastError();
}

// Bytes of shared memory: the program and the columns of its rows; then a tile
// but for its B values: entries of C and A values, with room for copies that
// start and end on 16-byte boundaries.
__host__ __device__ constexpr int run_fixed(int n, int p) {
  return ((8 * (p + 32) + 4 * n + 15) & ~15);
}
__host__ __device__ constexpr long long run_out(int rows, int n) {
  return ((long long)rows * (n | 1) * 8 + 16 + 15) & ~15LL;
}
// bytes of one staged A row where rows are copied one by one
__host__ __device__ constexpr int run_arow(int na, int vsz) { return (na * vsz + 16 + 15) & ~15; }
__host__ __device__ constexpr long long run_tile(int rows, int n, int na, int vsz) {
  return run_out(rows, n) + (long long)rows * run_arow(na, vsz) + 16;
}

// A bunch's rows are staged one by one: their B values in walk order, a row's
// A values, and where each of its B rows starts.
__host__ __device__ constexpr int bunch_row(int n, int na, int p, int vsz) {
  return (n | 1) * 8 + ((na | 1) + (p | 1)) * vsz + 4 * na;
}

// One block a program: that of run run_of[b], or of bunch b - nprog.
constexpr int kProgThreads = 512;
template <bool MULTI>
__global__ void __launch_bounds__(kProgThreads, 3)
    k_run_prog(const ProdTable<void> src, const RowRun *__restrict__ found,
               const RunTable rt, int nprog, int vsz, RunProg *__restrict__ progs,
               int *__restrict__ err) {
  __shared__ unsigned long long keys[2048];
  __shared__ int tk[kRunMaxA], tbs[kRunMaxA], tlen[kRunMaxA], tpl[kRunMaxA], tpre[kRunMaxA + 1];
  __shared__ int toff[kRunMaxA];
  __shared__ short hstart[kRunMaxIp + 1], ooff[kRunMaxIp], byrank[kRunMaxIp], sq[kRunMaxIp];
  __shared__ unsigned char ow[kRunMaxIp];
  __shared__ unsigned char tseg[kRunMaxA];
  __shared__ int s_scan[kProgThreads / 32], s_w0[16], s_int[6];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int W = kProgThreads / 32;
  RunProg &out = progs[blockIdx.x];
  const bool bunch = (int)blockIdx.x >= nprog;
  RowRun rd{0, 0, 0, 0};
  if (bunch) rd.row0 = rt.brow[blockIdx.x - nprog];
  else rd = found[rt.run_of[blockIdx.x]];
  const int sigma = bunch ? 0 : rd.meta >> 2 & 3;
  Operands<void> o;
  const int lr = prod_row<MULTI>(src, rd.row0, o);
  const int a0 = __ldg(o.arpt + lr), na = __ldg(o.arpt + lr + 1) - a0;
  if (na <= 0 || na > kRunMaxA) {  // not a row of a run: the operands changed
    if (tid == 0) {
      atomicOr(err, ERR_CAPACITY);
      out.na = out.p = out.n = 0;
    }
    return;
  }
  if (tid < na) {
    const RunTerm r = run_term(o, a0 + tid, sigma);
    tk[tid] = r.k;
    tbs[tid] = r.bs;
    tlen[tid] = run_len(r.len);
    tpl[tid] = r.pl;
  }
  __syncthreads();
  if (warp == 0) {
    int run = 0, first = na;
    for (int c = 0; c < na; c += 32) {
      const int t = c + lane;
      const int v = t < na ? tlen[t] : 0;
      int incl = v;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += u;
      }
      if (t < na) tpre[t] = run + incl - v;
      run += __shfl_sync(0xffffffffu, incl, 31);
      const unsigned m = __ballot_sync(0xffffffffu, v > 0);
      if (first == na && m) first = c + __ffs(m) - 1;
    }
    if (lane == 0) {
      tpre[na] = run;
      s_int[0] = run;
      s_int[1] = first;
    }
  }
  __syncthreads();
  const int P = s_int[0], t0 = s_int[1];
  if (P <= 0 || P > kRunMaxIp) {
    if (tid == 0) {
      atomicOr(err, ERR_CAPACITY);
      out.na = out.p = out.n = 0;
    }
    return;
  }
  if (!bunch) {  // runs are listed by program, the classes apart
    int before = 0;
    for (int p = tid; p < (int)blockIdx.x; p += kProgThreads) {
      const int v = rt.slot_of[p];
      if ((v >> 16) == (P > kRunSmallIp)) before += rt.count[v & 0xffff];
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) before += __shfl_xor_sync(0xffffffffu, before, d);
    if (lane == 0) s_scan[warp] = before;
    __syncthreads();
    if (tid == 0) {
      int sum = 0;
      for (int w = 0; w < W; ++w) sum += s_scan[w];
      rt.first[blockIdx.x] = sum;
    }
    __syncthreads();
  }
  // -- the products sorted by (column, walk order)
  const int cb = __ldg(o.bcol + tbs[t0]);
  int p2 = 1;
  while (p2 < P) p2 <<= 1;
  for (int t = warp; t < na; t += W)
    for (int e = lane; e < tlen[t]; e += 32) {
      const unsigned c = (unsigned)(__ldg(o.bcol + tbs[t] + e) - cb) ^ 0x80000000u;
      keys[tpre[t] + e] = (unsigned long long)c << 32 | (unsigned)(tpre[t] + e);
    }
  for (int i = P + tid; i < p2; i += kProgThreads) keys[i] = ~0ull;
  __syncthreads();
  for (int k = 2; k <= p2; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = tid; i < p2; i += kProgThreads) {
        const int x = i ^ j;
        if (x > i) {
          const unsigned long long u = keys[i], v = keys[x];
          if ((u > v) == ((i & k) == 0)) {
            keys[i] = v;
            keys[x] = u;
          }
        }
      }
      __syncthreads();
    }
  // -- entries: heads of equal columns, numbered by a scan over the block
  int n = 0;
  for (int base = 0; base < P; base += kProgThreads) {
    const int i = base + tid;
    const bool head =
        i < P && (i == 0 || (unsigned)(keys[i] >> 32) != (unsigned)(keys[i - 1] >> 32));
    const unsigned m = __ballot_sync(0xffffffffu, head);
    if (lane == 0) s_scan[warp] = __popc(m);
    __syncthreads();
    int before = n, all = 0;
    for (int w = 0; w < W; ++w) {
      const int v = s_scan[w];
      if (w < warp) before += v;
      all += v;
    }
    const int q = before + __popc(m & (0xffffffffu >> (31 - lane))) - 1;
    if (i < P) {
      sq[i] = (short)q;
      if (head) {
        hstart[q] = (short)i;
        out.rel[q] = (int)((unsigned)(keys[i] >> 32) ^ 0x80000000u);
      }
    }
    n += all;
    __syncthreads();
  }
  if (tid == 0) hstart[n] = (short)P;
  __syncthreads();
  // -- rows of a tile: the most that fit, whole row groups of 32 where it is
  // more than one; segments of B and the place of every A entry's B row
  const bool large = P > kRunSmallIp;
  const int warps = large ? RunCfg<1>::WARPS : RunCfg<0>::WARPS;
  if (warp == 0) {
    const int smem = large ? RunCfg<1>::SMEM : RunCfg<0>::SMEM;
    if (bunch) {
      const int room = smem - run_fixed(n, P) - 64 - ((P + 15) & ~15) - 2 * (kRunMaxA + 2);
      int most = min(room / (bunch_row(n, na, P, vsz) + 8), kRunRows);
      if (most > 32) most &= ~31;
      if (lane == 0) {
        s_int[2] = 0;
        s_int[3] = max(most, 1);
        s_int[4] = P | 1;
        s_int[5] = 0;
      }
    }
    const int unit = 16 / vsz;
    auto layout = [&](int L, bool write) {  // elements of B; segments in s_int[2]
      const int span = (L - 1) * sigma + 1;
      int x = 0, pk = 0, ppl = 0, segs = 0, total = 0;
      for (int c = 0; c < na; c += 32) {
        const int t = c + lane;
        const int k = t < na ? tk[t] : 0, pl = t < na ? tpl[t] : 0;
        int k1 = __shfl_up_sync(0xffffffffu, k, 1), l1 = __shfl_up_sync(0xffffffffu, pl, 1);
        if (lane == 0) {
          k1 = pk;
          l1 = ppl;
        }
        const bool brk = t < na && (t == 0 || !run_near(k, pl, k1, l1) || k - k1 >= span);
        // a segment's place less its start in memory changes where one begins,
        // by what lies between it and the end of the segment before
        int dx = 0;
        if (brk) dx = tbs[t] - (t == 0 ? 0 : tbs[t - 1] + (L - 1) * tpl[t - 1] + tlen[t - 1]);
        const int own = t < na ? (L - 1) * pl + tlen[t] : 0;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, dx, d);
          if (lane >= d) dx += u;
        }
        const unsigned bm = __ballot_sync(0xffffffffu, brk);
        const int g = segs + __popc(bm & (0xffffffffu >> (31 - lane))) - 1;
        if (t < na) {
          // segments start on 16-byte boundaries, with room for a copy that
          // starts and ends on one
          const int off = tbs[t] - (x + dx) + 3 * unit * g;
          const bool last = t == na - 1;
          if (write) {
            toff[t] = off;
            tseg[t] = (unsigned char)g;
            if (brk) {
              out.seg0[g] = (unsigned char)t;
              out.dst[g] = off & ~(unit - 1);
            }
            if (last || !run_near(tk[t + 1], tpl[t + 1], k, pl) || tk[t + 1] - k >= span)
              out.seg1[g] = (unsigned char)t;
          }
          if (last) total = off + own + 3 * unit;
        }
        segs += __popc(bm);
        x += __shfl_sync(0xffffffffu, dx, 31);
        pk = __shfl_sync(0xffffffffu, k, 31);
        ppl = __shfl_sync(0xffffffffu, pl, 31);
      }
      if (lane == 0) s_int[2] = segs;
      return __shfl_sync(0xffffffffu, total, (na - 1) & 31);
    };
    auto fits = [&](int L) {
      const long long fixed = run_fixed(n, P) + run_tile(L, n, na, vsz);
      if (fixed > smem) return false;
      return fixed + (long long)layout(L, false) * vsz <= smem;
    };
    if (!bunch) {
      bool near = true;
      for (int t = lane; t < na; t += 32) near = near && run_step_fits(tpl[t], 2);
      // lo fits, hi does not
      int lo = 1, hi = __all_sync(0xffffffffu, near) ? kRunRows + 1 : 2;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (fits(mid)) lo = mid; else hi = mid;
      }
      if (lo > 32) lo &= ~31;
      const int total = layout(lo, true);
      bool one = true;
      for (int t = lane; t < na; t += 32) one = one && tpl[t] == tpl[0];
      one = __all_sync(0xffffffffu, one);
      if (lane == 0) {
        s_int[3] = lo;
        s_int[4] = lo == 1 ? 0 : one ? tpl[0] : -1;
        s_int[5] = total;
      }
    }
  }
  // -- entries by descending product count, dealt to the parts
  for (int q = tid; q < n; q += kProgThreads) {
    const int c = hstart[q + 1] - hstart[q];
    int r = 0;
    for (int u = 0; u < n; ++u) {
      const int cu = hstart[u + 1] - hstart[u];
      r += cu > c || (cu == c && u < q);
    }
    byrank[r] = (short)q;
  }
  __syncthreads();
  const int L = s_int[3], segs = s_int[2];
  const int parts = warps / ((L + 31) / 32);
  if (tid < parts) {
    int off = 0;
    for (int round = 0; round * parts < n; ++round) {
      const int r = round * parts + ((round & 1) ? parts - 1 - tid : tid);
      if (r < n) {
        const int q = byrank[r];
        ow[q] = (unsigned char)tid;
        ooff[q] = (short)off;
        off += hstart[q + 1] - hstart[q];
      }
    }
    s_scan[tid] = off;
  }
  __syncthreads();
  if (tid == 0) {
    int at = 0;
    for (int w = 0; w < 16; ++w) {
      const int c = w < parts ? s_scan[w] : 0;
      s_w0[w] = at;
      out.w0[w] = at;
      out.w1[w] = at + c;
      at = (at + c + 1) & ~1;  // 16-byte boundaries
    }
    out.na = na;
    out.p = P;
    out.n = n;
    out.rows = L;
    out.parts = parts;
    out.segs = segs;
    out.t0 = t0;
    out.step = s_int[4];
    out.belems = s_int[5];
  }
  for (int i = tid; i < P + 32; i += kProgThreads) out.word[i] = make_uint2(0u, 0u);
  if (tid <= na) out.before[tid] = (short)tpre[tid];
  __syncthreads();
  for (int i = tid; i < P; i += kProgThreads) {
    const int p = (int)(unsigned)keys[i], q = sq[i];
    int lo = 0, hi = na;  // the A entry of product p: tpre[t] <= p < tpre[t + 1]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (tpre[mid] <= p) lo = mid; else hi = mid;
    }
    while (tpre[lo + 1] <= p) ++lo;
    if (bunch) {
      out.term[p] = (unsigned char)lo;
      out.word[s_w0[ow[q]] + ooff[q] + (i - hstart[q])] =
          make_uint2((unsigned)(p * vsz),
                     (unsigned)(lo * vsz) | (unsigned)q << 11 |
                         (i + 1 == hstart[q + 1] ? 0x80000000u : 0u));
      continue;
    }
    const int g = tseg[lo];
    // a place counts from its segment's 16-byte boundary; the copy's start
    // within the boundary is added tile by tile
    const int place = toff[lo] - toff[out.seg0[g]] + (toff[out.seg0[g]] & ~(16 / vsz - 1)) + p - tpre[lo];
    const unsigned stride = L > 1 && s_int[4] < 0 ? (unsigned)tpl[lo] : 0u;
    out.word[s_w0[ow[q]] + ooff[q] + (i - hstart[q])] =
        make_uint2((unsigned)(place * vsz) | stride << 17,
                   (unsigned)(lo * vsz) | (unsigned)q << 11 | (unsigned)g << 22 |
                       (i + 1 == hstart[q + 1] ? 0x80000000u : 0u));
  }
}

cudaError_t launch_run_progs(const ProdTable<void> &t, const RowRun *found, const RunTable &rt,
                             int nprog, int nbunch, bool fp32, void *progs, int *err,
                             cudaStream_t s) {
  if (nprog + nbunch <= 0) return cudaSuccess;
  auto kern = t.prod_of_row ? k_run_prog<true> : k_run_prog<false>;
  kern<<<nprog + nbunch, kProgThreads, 0, s>>>(t, found, rt, nprog, fp32 ? 4 : 8,
                                               static_cast<RunProg *>(progs), err);
  return cudaGetLastError();
}

// The list of the runs (small ones from the front of `runs`, large ones from
// the back), by program; with row_nz their rows get their count there; they
// are counted as numeric-bin rows that no bin needs (by crpt, what k_perm goes
// by, when row_nz is null).
__global__ void __launch_bounds__(256)
    k_run_counts(const RowRun *__restrict__ found, int nfound, RowRun *__restrict__ runs, int cap,
                 const RunTable rt, const RunProg *__restrict__ progs, int *__restrict__ row_nz,
                 const int *__restrict__ crpt, const BinLimits lim, int *__restrict__ num_sub) {
  __shared__ int hist[kNumBins];
  if (threadIdx.x < kNumBins) hist[threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int q = (blockIdx.x * 256 + threadIdx.x) >> 5; q < nfound; q += gridDim.x * 8) {
    RowRun rd = found[q];
    if (rd.prog < 0) continue;
    const int s = rd.meta & 3, len = rd.meta >> 4;
    const int p = rt.prog_of[rd.prog];
    const int n = progs[p].n;
    if (lane == 0) {
      const int at = rt.first[p] + rd.place;
      rd.prog = p;
      runs[rt.slot_of[p] >> 16 ? cap - 1 - at : at] = rd;
    }
    if (row_nz) {
      if (lane == 0 && n > 0) atomicAdd(&hist[num_bin(n, lim)], len);
      for (int m = lane; m < len; m += 32) row_nz[rd.row0 + s * m] = n;
    } else {
      for (int m = lane; m < len; m += 32) {
        const int row = rd.row0 + s * m;
        const int v = crpt[row + 1] - crpt[row];
        if (v > 0) atomicAdd(&hist[num_bin(v, lim)], 1);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < kNumBins && hist[threadIdx.x])
    atomicAdd(&num_sub[threadIdx.x], hist[threadIdx.x]);
}

cudaError_t launch_run_counts(const RowRun *found, int nfound, RowRun *runs, int cap,
                              const RunTable &rt, const void *progs, int *row_nz, const int *crpt,
                              const BinLimits &lim, int *num_sub, cudaStream_t s) {
  if (nfound <= 0) return cudaSuccess;
  const int grid = std::min((nfound + 7) / 8, dev_info().sms * 8);
  k_run_counts<<<grid, 256, 0, s>>>(found, nfound, runs, cap, rt,
                                    static_cast<const RunProg *>(progs), row_nz, crpt, lim, num_sub);
  return cudaGetLastError();
}

// The same for the rows of the bunches; blockIdx.y is the bunch. The first
// block also adds up the tiles of every bunch, by class.
__global__ void __launch_bounds__(256)
    k_bunch_counts(const RunTable rt, int nprog, const int *__restrict__ list,
                   const RunProg *__restrict__ progs, int *__restrict__ row_nz,
                   const int *__restrict__ crpt, const BinLimits lim, int *__restrict__ num_sub) {
  const int b = blockIdx.y;
  if (blockIdx.x == 0 && b == 0) {
    __shared__ int part[2][256];
    const int nb = gridDim.y, per = (nb + 255) / 256, first = (int)threadIdx.x * per;
    int sum[2] = {0, 0};
    auto tiles = [&](int i, int c) {
      const RunProg &pg = progs[nprog + i];
      return pg.n > 0 && (pg.p > kRunSmallIp) == (c == 1) ? (rt.brows[i] + pg.rows - 1) / pg.rows : 0;
    };
    for (int i = first; i < min(first + per, nb); ++i)
      for (int c = 0; c < 2; ++c) sum[c] += tiles(i, c);
    for (int c = 0; c < 2; ++c) part[c][threadIdx.x] = sum[c];
    __syncthreads();
    for (int c = 0; c < 2; ++c) {
      int at = 0;
      for (int i = 0; i < (int)threadIdx.x; ++i) at += part[c][i];
      for (int i = first; i < min(first + per, nb); ++i) {
        rt.btiles[c][i] = at;
        at += tiles(i, c);
      }
      if (first < nb && first + per >= nb) rt.btiles[c][nb] = at;
    }
  }
  const int n = progs[nprog + b].n, rows = rt.brows[b];
  const int *rl = list + rt.bplace[b];
  int mine = 0;
  for (int i = blockIdx.x * 256 + threadIdx.x; i < rows; i += gridDim.x * 256) {
    if (row_nz) {
      row_nz[rl[i]] = n;
    } else {
      const int v = crpt[rl[i] + 1] - crpt[rl[i]];
      if (v == n) ++mine;
      else if (v > 0) atomicAdd(&num_sub[num_bin(v, lim)], 1);
    }
  }
  if (row_nz) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && n > 0) atomicAdd(&num_sub[num_bin(n, lim)], rows);
  } else {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, d);
    if ((threadIdx.x & 31) == 0 && mine && n > 0) atomicAdd(&num_sub[num_bin(n, lim)], mine);
  }
}

cudaError_t launch_bunch_counts(const RunTable &rt, int nprog, int nbunch, const int *list,
                                const void *progs, int *row_nz, const int *crpt,
                                const BinLimits &lim, int *num_sub, cudaStream_t s) {
  if (nbunch <= 0) return cudaSuccess;
  k_bunch_counts<<<dim3(8, nbunch), 256, 0, s>>>(rt, nprog, list,
                                                  static_cast<const RunProg *>(progs), row_nz,
                                                  crpt, lim, num_sub);
  return cudaGetLastError();
}

// ---- numeric phase of the runs ----------------------------------------------------
// One block a run, taken from a ticket counter; a run is computed in tiles of
// up to the program's rows. Lane l of a row group of 32 computes row l of it;
// the warps share the row groups and the entries of C.
//
// The tile's A values and the B rows that it reads are staged in shared
// memory by bulk copies (cp.async.bulk): consecutive A entries whose B rows
// touch share one contiguous segment of B (9 segments of 34 rows serve the 27
// A entries of 32 rows of a 27-point stencil). A copy starts on the 16-byte
// boundary at or before its first value; how far into it that value lies
// changes from tile to tile and is added to the program's words. A staged
// value is read where it is used, a lane per row: odd row lengths spread the
// lanes over all banks. One or two warps more only look up what tiles need
// (their run, the places of their rows), each for runs of its own, and start
// the copies of the next tile as soon as the others have computed the one
// before, while they write it out. With the look-ups left to the computing
// warps they took as long as the sums (5,700 of 14,200 cycles a tile of the
// 27-point stencil); with one warp for them the chain of five dependent loads a
// run bound the tiles of few products (7-point 149 x 131 x 97: 377 us, 311 with
// two; a second warp gains nothing where a run has several large tiles). Runs
// are listed by program, so that a block seldom changes it: the parts of
// another program lie elsewhere, and its tile has to wait for the last one to
// be written out. Where the rows of C
// lie one after the other (s = 1, an odd count) their values leave by one bulk
// copy too.
//
// What bounds it: shared-memory wavefronts (L1 data pipe 74% on the 27-point
// 80^3 stencil) and issue. Two 8-byte reads a product are four wavefronts for
// 32 products; the whole kernel takes 8.8, with the program words, the sums and
// columns written out, and the idle lanes of partial row groups. The entry-map
// kernel takes 16.5, a read-modify-write of a value slot a product.
constexpr int kCopyWait = 1 << 20;  // polls before a wait gives up

__device__ __forceinline__ unsigned smem_u32(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long *b, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned long long *b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long *b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ bool mbar_wait(unsigned long long *b, unsigned parity) {
  for (int i = 0; i < kCopyWait; ++i) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n"
        " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.b32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
// 16-byte aligned addresses, a multiple of 16 bytes
__device__ __forceinline__ void copy_in(void *dst, const void *src, unsigned bytes,
                                        unsigned long long *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void copy_out(void *dst, const void *src, unsigned bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(
                   __cvta_generic_to_global(dst)),
               "r"(smem_u32(src)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void proxy_fence() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// The bytes of `count` values from p on with both ends moved out to 16-byte
// boundaries, and how many values lie before the first.
template <typename VT>
struct CopySpan {
  const unsigned char *src;
  unsigned bytes;
  int lead;
  __device__ __forceinline__ CopySpan(const VT *p, int count) {
    const size_t a = reinterpret_cast<size_t>(p), a0 = a & ~(size_t)15;
    src = reinterpret_cast<const unsigned char *>(a0);
    lead = (int)((a - a0) / sizeof(VT));
    bytes = (unsigned)(((a + (size_t)count * sizeof(VT) + 15) & ~(size_t)15) - a0);
  }
};

// Where the parts of a tile lie in shared memory (program words, then the
// columns of its rows, entries of C, A values, B values).
template <typename VT>
struct RunSmem {
  uint2 *prog;
  int *rel;
  double *out;
  VT *as, *bs;
  __device__ __forceinline__ RunSmem(unsigned char *base, int na, int p, int n, int rows) {
    prog = reinterpret_cast<uint2 *>(base);
    rel = reinterpret_cast<int *>(prog + p + 32);
    unsigned char *at = base + run_fixed(n, p);
    out = reinterpret_cast<double *>(at);
    at += run_out(rows, n);
    as = reinterpret_cast<VT *>(at);
    at += rows * run_arow(na, sizeof(VT)) + 16;
    bs = reinterpret_cast<VT *>(at);
  }
};

// Words [w0, w1) of a program for one row: al its A values, b_of a word's B
// value, ol the row's entries of C.
template <typename VT, bool COMP, typename F>
__device__ __forceinline__ void run_walk(const uint2 *prog, int w0, int w1, const char *al,
                                         bool pair, bool write, double *ol, F &&b_of) {
  auto a_of = [&](uint2 w) { return *reinterpret_cast<const VT *>(al + (w.y & 0x7ffu)); };
  auto rank = [](unsigned y) { return y >> 11 & 0x7ffu; };
  if (!COMP || !pair) {
    double acc = 0.0;
    auto step = [&](unsigned y, VT a, VT b) {
      acc = __dadd_rn(acc, __dmul_rn((double)a, (double)b));
      if ((int)y < 0) {
        if (write) ol[rank(y)] = acc;
        acc = 0.0;
      }
    };
    int p = w0;
    for (; p + 4 <= w1; p += 4) {
      const uint4 u = *reinterpret_cast<const uint4 *>(prog + p);
      const uint4 v = *reinterpret_cast<const uint4 *>(prog + p + 2);
      const uint2 q0 = make_uint2(u.x, u.y), q1 = make_uint2(u.z, u.w);
      const uint2 q2 = make_uint2(v.x, v.y), q3 = make_uint2(v.z, v.w);
      const VT x0 = a_of(q0), x1 = a_of(q1), x2 = a_of(q2), x3 = a_of(q3);
      const VT y0 = b_of(q0), y1 = b_of(q1), y2 = b_of(q2), y3 = b_of(q3);
      step(u.y, x0, y0);
      step(u.w, x1, y1);
      step(v.y, x2, y2);
      step(v.w, x3, y3);
    }
    for (; p < w1; ++p) {
      const uint2 w = prog[p];
      step(w.y, a_of(w), b_of(w));
    }
  } else {
    // error-free fp32 pairs, started from the entry's first product
    bool fresh = true;
    float2 sc = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int p = w0; p < w1; ++p) {
      const uint2 w = prog[p];
      const float a = (float)a_of(w), b = (float)b_of(w);
      if (fresh) {
        const float ph = __fmul_rn(a, b);
        sc = make_float2(ph, __fmaf_rn(a, b, -ph));
      } else {
        comp_add(sc, a, b);
      }
      fresh = (int)w.y < 0;
      if (fresh && write) ol[rank(w.y)] = (double)sc.x + (double)sc.y;
    }
  }
}

// Compensated mode: whether rows of na A entries and n entries of C sum in fp32
// pairs. The rows that the other kernels sum in pairs, so that a row's sums and
// its bound do not depend on whether it is in a run: those of the row-group
// bins (at most comp.most entries), over B rows without repeated columns
// (comp.nmax is 0 otherwise), where an entry has at most na products.
__device__ __forceinline__ bool run_pairs(const CompArgs &comp, int na, int n) {
  return na <= comp.nmax && n <= comp.most;
}

// What the look-up warp leaves for a tile.
struct RunTile {
  int prog;   // -1: no more tiles
  int cnt;    // rows
  int bulk_c; // the rows of C lie one after the other
  int pad;
  int c0[kRunRows];  // start of each row of C, or -1: not this program's row
  int cb[kRunRows];  // column of its first product
  int ao[kRunRows];  // place of its first A value
  unsigned char lead[kRunMaxA];  // values before each segment's first
};

template <int CLASS, typename VT, bool COMP, bool MULTI>
__global__ void __launch_bounds__((RunCfg<CLASS>::WARPS + RunCfg<CLASS>::LOOK) * 32, RunCfg<CLASS>::MINB)
    k_num_run(const ProdTable<VT> src, const RowRun *__restrict__ runs, int nruns,
              const RunProg *__restrict__ progs, const int *__restrict__ crpt,
              int *__restrict__ ccol, double *__restrict__ cval, int *__restrict__ err,
              CompArgs comp, int *__restrict__ ticket) {
  constexpr int WARPS = RunCfg<CLASS>::WARPS, THREADS = WARPS * 32;
  extern __shared__ __align__(16) unsigned char smem_run[];
  __shared__ __align__(8) unsigned long long s_full, s_done, s_free[2];
  __shared__ RunTile s_tile[2];
  __shared__ unsigned char held[kRunMaxA];  // the leads that the words hold
  __shared__ int s_lost, s_stop, s_tiles, s_ended;  // tiles announced, look-up warps that have ended
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    s_tiles = s_ended = 0;
    mbar_init(&s_full, 1);        // a tile's data and values are there
    mbar_init(&s_done, 1);        // it is computed: the next one's values may come
    mbar_init(&s_free[0], WARPS); // it is written out: its data may be replaced
    mbar_init(&s_free[1], WARPS);
    s_lost = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  if (warp >= WARPS) {
    // -- the look-up warps
    int next = 0;
    bool lost = false;
    int max_deg = 0, redo = 0;
    if (lane == 0) next = atomicAdd(ticket, 1);
    for (;;) {
      const int at = __shfl_sync(0xffffffffu, next, 0);
      if (at >= nruns || lost) break;
      if (lane == 0) next = atomicAdd(ticket, 1);
      const RowRun rd = CLASS ? runs[-1 - at] : runs[at];
      const int s = rd.meta & 3, sigma = rd.meta >> 2 & 3, len = rd.meta >> 4;
      const RunProg &pg = progs[rd.prog];
      const int na = pg.na, n = pg.n, L = pg.rows, segs = pg.segs;
      if (n <= 0) {
        if (lane == 0) atomicOr(err, ERR_COUNT);
        continue;
      }
      Operands<VT> op;
      const int lr0 = prod_row<MULTI>(src, rd.row0, op);
      const int a0 = __ldg(op.arpt + lr0);
      const RunSmem<VT> sm(smem_run, na, pg.p, n, L);
      constexpr int kPer = kRunMaxA / 32;  // segments a lane looks after
      int k0[kPer], k1[kPer], dst[kPer];
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const int g = lane + 32 * i;
        if (g < segs) {
          k0[i] = __ldg(op.acol + a0 + pg.seg0[g]);
          k1[i] = __ldg(op.acol + a0 + pg.seg1[g]);
          dst[i] = pg.dst[g];
        }
      }
      const int kf = __ldg(op.acol + a0 + pg.t0);
      const bool whole_a = s == 1 && (na & 1);  // the tile's A rows are staged as they lie
      const int arow = run_arow(na, sizeof(VT)) / (int)sizeof(VT);
      const bool bulk_c = s == 1 && (n & 1) && (reinterpret_cast<size_t>(cval) & 15) == 0;
      if (COMP) {
        if (run_pairs(comp, na, n)) max_deg = max(max_deg, na);
        else redo += len;
      }
      for (int r0 = 0; r0 < len && !lost; r0 += L) {
        const int cnt = min(L, len - r0);
        const int adv = sigma * r0, reach = sigma * (r0 + cnt - 1) + 1;
        int b0[kPer], b1[kPer];
#pragma unroll
        for (int i = 0; i < kPer; ++i)
          if (lane + 32 * i < segs) {
            b0[i] = __ldg(op.brpt + k0[i] + adv);
            b1[i] = __ldg(op.brpt + k1[i] + reach);
          }
        // rows of the tile: a lane each, in turns of 32
        int c0[kRunRows / 32], cb[kRunRows / 32], as[kRunRows / 32];
        bool in_line = bulk_c;
        int c_first = 0;
#pragma unroll
        for (int i = 0; i < kRunRows / 32; ++i) {
          const int l = lane + 32 * i;
          if (32 * i < cnt) {
            const int lc = min(l, cnt - 1);
            const int row = rd.row0 + s * (r0 + lc);
            c0[i] = __ldg(crpt + row);
            const bool fits = __ldg(crpt + row + 1) - c0[i] == n;
            if (!fits) {
              atomicOr(err, ERR_COUNT);
              c0[i] = -1;
            }
            cb[i] = __ldg(op.bcol + __ldg(op.brpt + kf + sigma * (r0 + lc)));
            as[i] = s == 1 ? a0 + (r0 + lc) * na : __ldg(op.arpt + lr0 + s * (r0 + lc));
            if (i == 0) c_first = __shfl_sync(0xffffffffu, c0[0], 0);
            in_line = in_line && c0[i] >= 0 && c0[i] == c_first + lc * n;
          }
        }
        in_line = __all_sync(0xffffffffu, in_line);
        // everything is looked up: this is the block's next tile
        int t = 0;
        if (lane == 0) t = atomicAdd(&s_tiles, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        RunTile &tile = s_tile[t & 1];
        if (t >= 2 && !mbar_wait(&s_free[t & 1], (unsigned)((t >> 1) - 1) & 1u)) lost = true;
        unsigned bytes = 0;
#pragma unroll
        for (int i = 0; i < kPer; ++i)
          if (lane + 32 * i < segs) {
            const CopySpan<VT> c(op.bval + b0[i], b1[i] - b0[i]);
            if (b1[i] > b0[i]) bytes += c.bytes;
            tile.lead[lane + 32 * i] = (unsigned char)c.lead;
          }
        const CopySpan<VT> ca(op.aval + a0 + r0 * na, cnt * na);
        if (whole_a && lane == 0) bytes += ca.bytes;
#pragma unroll
        for (int i = 0; i < kRunRows / 32; ++i) {
          const int l = lane + 32 * i;
          if (l < cnt) {
            const CopySpan<VT> c(op.aval + as[i], na);
            if (!whole_a) bytes += c.bytes;
            tile.c0[l] = c0[i];
            tile.cb[l] = cb[i];
            tile.ao[l] = whole_a ? ca.lead + l * na : l * arow + c.lead;
          }
        }
        if (lane == 0) {
          tile.prog = rd.prog;
          tile.cnt = cnt;
          tile.bulk_c = in_line;
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) bytes += __shfl_xor_sync(0xffffffffu, bytes, d);
        if (t >= 1) {
          if (!mbar_wait(&s_done, (unsigned)(t - 1) & 1u)) lost = true;
          // another program has its parts elsewhere: the last tile must be out
          if (!lost && *(volatile int *)&s_tile[(t - 1) & 1].prog != rd.prog &&
              !mbar_wait(&s_free[(t - 1) & 1], (unsigned)((t - 1) >> 1) & 1u))
            lost = true;
        }
        lost = __any_sync(0xffffffffu, lost);
        if (lost) break;
        __syncwarp();
        if (lane == 0) mbar_expect(&s_full, bytes);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kPer; ++i)
          if (lane + 32 * i < segs && b1[i] > b0[i]) {
            const CopySpan<VT> c(op.bval + b0[i], b1[i] - b0[i]);
            copy_in(sm.bs + dst[i], c.src, c.bytes, &s_full);
          }
        if (whole_a) {
          if (lane == 0) copy_in(sm.as, ca.src, ca.bytes, &s_full);
        } else {
#pragma unroll
          for (int i = 0; i < kRunRows / 32; ++i) {
            const int l = lane + 32 * i;
            if (l < cnt) {
              const CopySpan<VT> c(op.aval + as[i], na);
              copy_in(sm.as + l * arow, c.src, c.bytes, &s_full);
            }
          }
        }
      }
    }
    // no more tiles: the computing warps end on a tile without a program, which
    // the last look-up warp announces once the last tile's values have arrived
    // (two arrivals in one phase of s_full are one too many)
    int ended = 0;
    if (lane == 0) ended = atomicAdd(&s_ended, 1);
    ended = __shfl_sync(0xffffffffu, ended, 0);
    const int t = *(volatile int *)&s_tiles;
    const bool last = ended == RunCfg<CLASS>::LOOK - 1;
    if (last && !lost && t >= 1 && !mbar_wait(&s_done, (unsigned)(t - 1) & 1u)) lost = true;
    if (last && !lost && t >= 2 && !mbar_wait(&s_free[t & 1], (unsigned)((t >> 1) - 1) & 1u))
      lost = true;
    if (lost) {
      if (lane == 0) {
        atomicExch(&s_lost, 1);
        atomicOr(err, ERR_WAIT);
      }
    } else if (last && lane == 0) {
      s_tile[t & 1].prog = -1;
      mbar_expect(&s_full, 0);
    }
    if (COMP && lane == 0) {
      if (max_deg) atomicMax(comp.max_deg, max_deg);
      if (redo) atomicAdd(comp.redo, redo);
    }
    return;
  }

  // -- the computing warps
  // lanes leave a poll loop one by one: the warp comes together first
  auto meet = [] {
    __syncwarp();
    asm volatile("barrier.sync 1, %0;" ::"n"(THREADS) : "memory");
  };
  // thread 0's view of the flag, for all (read again only two barriers later). A
  // wait that ran out in another warp alone, while thread 0 still saw the tile
  // arrive, stops the block a tile later; a vote of all warps here
  // (barrier.red.or) cost 0.6% of the 27-point 128^3 product, 2 to 4% of this
  // kernel on aggregation products.
  auto one_view = [&](bool yes) {
    if (tid == 0) *(volatile int *)&s_stop = yes;
    meet();
    return *(volatile int *)&s_stop != 0;
  };
  int cur = -1;  // the program in shared memory
  int na = 0, P = 0, n = 0, parts = 1, pstep = 0, w0 = 0, w1 = 0, rg = 0;
  RunSmem<VT> sm(smem_run, 0, 0, 0, 0);
  for (int t = 0;; ++t) {
    // one lane polls; the others then find the phase complete
    if (lane == 0 && !mbar_wait(&s_full, (unsigned)t & 1u)) s_lost = 1;
    __syncwarp();
    if (!*(volatile int *)&s_lost && !mbar_wait(&s_full, (unsigned)t & 1u)) s_lost = 1;
    const RunTile &tile = s_tile[t & 1];
    if (run_gives_up([&] { return tid == 0 && *(volatile int *)&s_lost != 0; }, one_view)) {
      if (tid == 0) atomicOr(err, ERR_WAIT);
      break;
    }
    if (tile.prog < 0) break;
    const int cnt = tile.cnt;
    if (tile.prog != cur) {
      cur = tile.prog;
      const RunProg &pg = progs[cur];
      na = pg.na;
      P = pg.p;
      n = pg.n;
      parts = pg.parts;
      pstep = pg.step;
      rg = warp / parts;
      const bool works = rg < (pg.rows + 31) / 32;
      w0 = works ? pg.w0[warp - rg * parts] : 0;
      w1 = works ? pg.w1[warp - rg * parts] : 0;
      sm = RunSmem<VT>(smem_run, na, P, n, pg.rows);
      for (int i = tid; i < P + 32; i += THREADS) {
        uint2 w = pg.word[i];
        w.x += (unsigned)tile.lead[w.y >> 22 & 0x7fu] * (unsigned)sizeof(VT);
        sm.prog[i] = w;
      }
      for (int i = tid; i < n; i += THREADS) sm.rel[i] = pg.rel[i];
    } else {
      for (int i = tid; i < P + 32; i += THREADS) {
        const int g = (int)(sm.prog[i].y >> 22 & 0x7fu);
        const int d = (int)tile.lead[g] - (int)held[g];
        if (d) sm.prog[i].x += (unsigned)(d * (int)sizeof(VT));
      }
    }
    meet();
    if (tid < kRunMaxA) held[tid] = tile.lead[tid];
    const int npad = n | 1;
    const int c_lead = tile.bulk_c ? tile.c0[0] & 1 : 0;  // C's values leave from where they go
    double *out0 = sm.out + c_lead;
    if (rg * 32 < cnt) {
      const int l = rg * 32 + lane;
      const int ll = min(l, cnt - 1);
      const bool write = l < cnt;
      const bool pair = COMP && run_pairs(comp, na, n);
      const char *al = reinterpret_cast<const char *>(sm.as + tile.ao[ll]);
      double *ol = out0 + (size_t)ll * npad;
      const char *bl = reinterpret_cast<const char *>(sm.bs + (pstep > 0 ? pstep : 0) * ll);
      const int lb = ll * (int)sizeof(VT);
      if (pstep >= 0)
        run_walk<VT, COMP>(sm.prog, w0, w1, al, pair, write, ol,
                           [&](uint2 w) { return *reinterpret_cast<const VT *>(bl + w.x); });
      else
        run_walk<VT, COMP>(sm.prog, w0, w1, al, pair, write, ol, [&](uint2 w) {
          return *reinterpret_cast<const VT *>(bl + (w.x & 0x1ffffu) + (w.x >> 17) * lb);
        });
    }
    proxy_fence();
    meet();
    if (tid == 0) mbar_arrive(&s_done);
    // the finished rows, while the next tile's values arrive
    const bool bulk_c = tile.bulk_c;
    if (bulk_c && warp == 1) {
      const int c00 = tile.c0[0];
      const int total = cnt * n, last = (c_lead + total) & ~1;  // values up to a boundary
      const int from = c_lead ? 2 : 0;                           // from one on, in `out`
      if (lane == 0) {
        if (last > from)
          copy_out(cval + c00 - c_lead + from, sm.out + from, (unsigned)(last - from) * 8u);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
      if (lane == 1 && c_lead) cval[c00] = sm.out[1];
      if (lane == 2 && last < c_lead + total && last >= from)
        cval[c00 - c_lead + last] = sm.out[last];
    }
    const int gw = n <= 4 ? 4 : n <= 8 ? 8 : n <= 16 ? 16 : 32;
    for (int l = tid / gw; l < cnt; l += THREADS / gw) {
      const int c0 = tile.c0[l], cb = tile.cb[l];
      if (c0 < 0) continue;
      int *cc = ccol + c0;
      for (int q = tid & (gw - 1); q < n; q += gw) __stcs(cc + q, sm.rel[q] + cb);
      if (!bulk_c) {
        double *cv = cval + c0;
        const double *ov = out0 + (size_t)l * npad;
        for (int q = tid & (gw - 1); q < n; q += gw) __stcs(cv + q, ov[q]);
      }
    }
    if (bulk_c && warp == 1 && lane == 0)
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncwarp();
    proxy_fence();
    if (lane == 0) mbar_arrive(&s_free[t & 1]);
  }
  if (tid == 32) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

template <int CLASS, typename VT, bool COMP>
static cudaError_t run_num_run(const ProdTable<VT> &t, const RowRun *runs, int nruns,
                               const void *progs, const int *crpt, int *ccol, double *cval,
                               int *err, CompArgs comp, int *ticket, cudaStream_t s) {
  if (nruns <= 0) return cudaSuccess;
  using C = RunCfg<CLASS>;
  auto kern = t.prod_of_row ? k_num_run<CLASS, VT, COMP, true> : k_num_run<CLASS, VT, COMP, false>;
  const int threads = (C::WARPS + C::LOOK) * 32;
  const int grid = persistent_grid((const void *)kern, threads, C::SMEM, nruns, 1);
  if (grid <= 0) return cudaErrorInvalidConfiguration;
  kern<<<grid, threads, C::SMEM, s>>>(t, runs, nruns, static_cast<const RunProg *>(progs),
                                            crpt, ccol, cval, err, comp, ticket);
  return cudaGetLastError();
}

template <typename VT, bool COMP>
static cudaError_t run_num_runs(const ProdTable<VT> &t, const RowRun *runs, const int (&nruns)[2],
                                int cap, const void *progs, const int *crpt, int *ccol,
                                double *cval, int *err, CompArgs comp, int *ticket,
                                cudaStream_t s) {
  cudaError_t e = run_num_run<1, VT, COMP>(t, runs + cap, nruns[1], progs, crpt, ccol, cval, err,
                                           comp, ticket + 1, s);
  if (e != cudaSuccess) return e;
  return run_num_run<0, VT, COMP>(t, runs, nruns[0], progs, crpt, ccol, cval, err, comp, ticket, s);
}

cudaError_t launch_numeric_run(const ProdTable<double> &t, const RowRun *runs,
                               const int (&nruns)[2], int cap, const void *progs, const int *crpt,
                               int *ccol, double *cval, int *err, int *ticket, cudaStream_t s) {
  return run_num_runs<double, false>(t, runs, nruns, cap, progs, crpt, ccol, cval, err,
                                     CompArgs{0, nullptr, nullptr}, ticket, s);
}

cudaError_t launch_numeric_comp_run(const ProdTable<float> &t, const RowRun *runs,
                                    const int (&nruns)[2], int cap, const void *progs,
                                    const int *crpt, int *ccol, double *cval, int nmax, int most,
                                    int *redo, int *max_deg, int *err, int *ticket,
                                    cudaStream_t s) {
  return run_num_runs<float, true>(t, runs, nruns, cap, progs, crpt, ccol, cval, err,
                                   CompArgs{nmax, redo, max_deg, false, most}, ticket, s);
}

// ---- numeric phase of the bunches --------------------------------------------------
// As k_num_run, but a tile's rows lie anywhere: each row's B values are staged
// in walk order (product p at place p), a warp a row. Few rows come here (those
// at the ends of grid lines); 14 rows of a 27-point stencil fill a block's
// shared memory. Bound by the look-ups of a tile's rows, which two to four
// blocks an SM overlap.
template <int CLASS, typename VT, bool COMP, bool MULTI>
__global__ void __launch_bounds__(RunCfg<CLASS>::WARPS * 32, RunCfg<CLASS>::MINB)
    k_num_bunch(const ProdTable<VT> src, const RunTable rt, int nprog, int nbunch,
                const int *__restrict__ list, const RunProg *__restrict__ progs,
                const int *__restrict__ crpt, int *__restrict__ ccol, double *__restrict__ cval,
                int *__restrict__ err, CompArgs comp, int *__restrict__ ticket) {
  constexpr int WARPS = RunCfg<CLASS>::WARPS, THREADS = WARPS * 32;
  extern __shared__ __align__(16) unsigned char smem_bunch[];
  __shared__ int s_next, s_bunch;
  __shared__ int s_c0[kRunRows], s_cb[kRunRows];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int *tiles = rt.btiles[CLASS];  // before each bunch
  const int all = __ldg(tiles + nbunch);
  int cur = -1, redo = 0, max_deg = 0;
  for (;;) {
    __syncthreads();  // the last tile is written out
    if (tid == 0) s_next = atomicAdd(ticket, 1);
    __syncthreads();
    const int at = s_next;
    if (at >= all) break;
    for (int i = tid; i < nbunch; i += THREADS)
      if (__ldg(tiles + i) <= at && at < __ldg(tiles + i + 1)) s_bunch = i;
    __syncthreads();
    const int b = s_bunch;
    const RunProg &pg = progs[nprog + b];
    const int na = pg.na, P = pg.p, n = pg.n, L = pg.rows, parts = pg.parts;
    const int r0 = (at - __ldg(tiles + b)) * L, cnt = min(L, rt.brows[b] - r0);
    const int *rl = list + rt.bplace[b] + r0;
    uint2 *prog = reinterpret_cast<uint2 *>(smem_bunch);
    int *rel = reinterpret_cast<int *>(prog + P + 32);
    double *out = reinterpret_cast<double *>(smem_bunch + run_fixed(n, P));
    VT *As = reinterpret_cast<VT *>(out + (size_t)L * (n | 1));
    VT *Bs = As + (size_t)L * (na | 1);
    int *from = reinterpret_cast<int *>(Bs + (size_t)L * (P | 1));  // B row start - its place
    unsigned char *term = reinterpret_cast<unsigned char *>(from + (size_t)L * na);
    short *before = reinterpret_cast<short *>(term + ((P + 15) & ~15));
    if (b != cur) {
      cur = b;
      for (int i = tid; i < P + 32; i += THREADS) prog[i] = pg.word[i];
      for (int i = tid; i < n; i += THREADS) rel[i] = pg.rel[i];
      for (int i = tid; i < P; i += THREADS) term[i] = pg.term[i];
      for (int i = tid; i <= na; i += THREADS) before[i] = pg.before[i];
    }
    const bool pair = COMP && run_pairs(comp, na, n);
    if (COMP && tid == 0) {
      if (pair) max_deg = max(max_deg, na);
      else redo += cnt;
    }
    __syncthreads();
    Operands<VT> op;  // every row of a bunch is of one product
    prod_row<MULTI>(src, rl[0], op);
    const int first = MULTI ? __ldg(src.row_off + __ldg(src.prod_of_row + rl[0])) : 0;
    for (int l = warp; l < cnt; l += WARPS) {
      const int row = rl[l];
      const int a0 = __ldg(op.arpt + row - first);
      for (int t = lane; t < na; t += 32) {
        const int b0 = __ldg(op.brpt + __ldg(op.acol + a0 + t));
        from[l * na + t] = b0 - before[t];
        As[l * (na | 1) + t] = __ldg(op.aval + a0 + t);
        if (t == pg.t0) s_cb[l] = __ldg(op.bcol + b0);
      }
      if (lane == 0) {
        const int c0 = __ldg(crpt + row);
        const bool fits = __ldg(crpt + row + 1) - c0 == n;
        if (!fits) atomicOr(err, ERR_COUNT);
        s_c0[l] = fits ? c0 : -1;
      }
      __syncwarp();
      VT *bl = Bs + (size_t)l * (P | 1);
#pragma unroll 4
      for (int p = lane; p < P; p += 32)
        __pipeline_memcpy_async(bl + p, op.bval + from[l * na + term[p]] + p, sizeof(VT));
    }
    __pipeline_commit();
    __pipeline_wait_prior(0);
    __syncthreads();
    const int rg = warp / parts, part = warp - rg * parts;
    if (rg * 32 < cnt && rg < (L + 31) / 32) {
      const int l = rg * 32 + lane, ll = min(l, cnt - 1);
      const char *bl = reinterpret_cast<const char *>(Bs + (size_t)ll * (P | 1));
      run_walk<VT, COMP>(prog, pg.w0[part], pg.w1[part],
                         reinterpret_cast<const char *>(As + ll * (na | 1)), pair, l < cnt,
                         out + (size_t)ll * (n | 1),
                         [&](uint2 w) { return *reinterpret_cast<const VT *>(bl + w.x); });
    }
    __syncthreads();
    const int gw = n <= 4 ? 4 : n <= 8 ? 8 : n <= 16 ? 16 : 32;
    for (int l = tid / gw; l < cnt; l += THREADS / gw) {
      const int c0 = s_c0[l], cb = s_cb[l];
      if (c0 < 0) continue;
      for (int q = tid & (gw - 1); q < n; q += gw) {
        __stcs(ccol + c0 + q, rel[q] + cb);
        __stcs(cval + c0 + q, out[(size_t)l * (n | 1) + q]);
      }
    }
  }
  if (COMP && tid == 0) {
    if (max_deg) atomicMax(comp.max_deg, max_deg);
    if (redo) atomicAdd(comp.redo, redo);
  }
}

template <int CLASS, typename VT, bool COMP>
static cudaError_t run_num_bunch(const ProdTable<VT> &t, const RunTable &rt, int nprog, int nbunch,
                                 const int *list, const void *progs, const int *crpt, int *ccol,
                                 double *cval, int *err, CompArgs comp, int *ticket,
                                 cudaStream_t s) {
  using C = RunCfg<CLASS>;
  auto kern = t.prod_of_row ? k_num_bunch<CLASS, VT, COMP, true> : k_num_bunch<CLASS, VT, COMP, false>;
  // how many tiles there are is known on the device only
  const int grid = persistent_grid((const void *)kern, C::WARPS * 32, C::SMEM, INT32_MAX, 1);
  if (grid <= 0) return cudaErrorInvalidConfiguration;
  kern<<<grid, C::WARPS * 32, C::SMEM, s>>>(t, rt, nprog, nbunch, list,
                                            static_cast<const RunProg *>(progs), crpt, ccol, cval,
                                            err, comp, ticket);
  return cudaGetLastError();
}

cudaError_t launch_numeric_bunch(const ProdTable<double> &t, const RunTable &rt, int nprog,
                                 int nbunch, const int *list, const void *progs, const int *crpt,
                                 int *ccol, double *cval, int *err, int *ticket, cudaStream_t s) {
  if (nbunch <= 0) return cudaSuccess;
  const CompArgs none{0, nullptr, nullptr};
  cudaError_t e = run_num_bunch<1, double, false>(t, rt, nprog, nbunch, list, progs, crpt, ccol,
                                                  cval, err, none, ticket + 1, s);
  if (e != cudaSuccess) return e;
  return run_num_bunch<0, double, false>(t, rt, nprog, nbunch, list, progs, crpt, ccol, cval, err,
                                         none, ticket, s);
}

cudaError_t launch_numeric_comp_bunch(const ProdTable<float> &t, const RunTable &rt, int nprog,
                                      int nbunch, const int *list, const void *progs,
                                      const int *crpt, int *ccol, double *cval, int nmax, int most,
                                      int *redo, int *max_deg, int *err, int *ticket,
                                      cudaStream_t s) {
  if (nbunch <= 0) return cudaSuccess;
  const CompArgs comp{nmax, redo, max_deg, false, most};
  cudaError_t e = run_num_bunch<1, float, true>(t, rt, nprog, nbunch, list, progs, crpt, ccol,
                                                cval, err, comp, ticket + 1, s);
  if (e != cudaSuccess) return e;
  return run_num_bunch<0, float, true>(t, rt, nprog, nbunch, list, progs, crpt, ccol, cval, err,
                                       comp, ticket, s);
}

}  // namespace nspb
