// Numeric phase of rows whose products hardly meet: sort the products.
//
// Where almost every intermediate product is an entry of C of its own (random
// and power-law matrices), a hash table does work for nothing: it is cleared,
// probed, and compacted again before its entries are sorted. k_num_flat takes
// the row's products as one flat list (flat.cuh), with the loads of up to K
// products a thread in flight at once, and gives each product its place in
// the sorted row directly: a bit per narrow bucket of columns (32 and more
// buckets a product), and a count of the bits before it. The few products
// that share a bucket go to a second and third bitmap and are put in order
// afterwards by (column, place in the list); a row with more than that in one
// bucket is sorted by wide buckets, with a rank inside each. Products of one
// column come out side by side in the order of A's entries and are added in
// that order, so a sum is the sequential one, bit for bit, also in rows of
// more than 512 entries, which the hash kernels add in any order.
//
// Bound: instruction issue (62% of the slots) and shared-memory wavefronts
// (61% of the data pipe), at 58% occupancy by registers; DRAM is at 10%. A
// block a row keeps the rows' latencies apart; four warps and five products a
// thread for 257..512 entries (259 us): with two warps and ten products the
// unrolled code no longer fits the instruction cache (377 us), with eight warps
// and three products every warp's work for the row as a whole weighs more (343).
// Measured on 100003 x 80021 x 120011 with 4..32 entries a row (rows of 257..512
// entries, 48800 of them): hash table, compaction and bucket sort 694 us;
// products in wide buckets with a rank 322 us; bitmaps 259 us. All rows of that
// product 1160 -> 490 us; of 20 such products of 1000..40000 rows in one call
// 4370 -> 2090 us. Where C's row is one row of B, in order already (a diagonal
// times B), nothing is sorted: 27-point 64^3 rows scaled, in two calls, 480 -> 389
// us, the columns of a stencil crowd the narrow buckets.
#include "flat.cuh"
#include "internal.h"
#include "launch_util.h"

#include <algorithm>

namespace nspb {

// W warps a row, K products a thread: a row of at most 32 * W * (K - K / 5)
// entries may have a quarter more products than that.
template <int W, int K>
struct FlatCfg {
  static constexpr int TH = 32 * W;              // threads a row
  static constexpr int ROWS = W == 1 ? 4 : 1;    // rows a block
  static constexpr int CAP = TH * K;             // products a row
  static constexpr int WORDS = TH * 4;           // of a bitmap
  static constexpr int LEV = W >= 8 ? 3 : 2;     // bitmaps
  static constexpr int PER = K - K / 5;          // wide buckets a thread, at most
  static constexpr int CH = CAP / 32;
  static constexpr int O_KEY = CAP * 8;
  static constexpr int O_AUX = O_KEY + (CAP + 4) * 4;
  static constexpr int O_MAP = O_AUX + CAP * 4;  // bitmaps and ranks, or the wide buckets
  static constexpr int MAP = (LEV + 1) * WORDS * 4;
  static_assert(MAP >= (TH * PER + 4) * 4, "the wide buckets share the bitmaps' room");
  static constexpr int O_FIRST = O_MAP + MAP;
  static constexpr int O_RED = O_FIRST + (((CH + 1) * 4 + 15) & ~15);
  static constexpr int BYTES = (O_RED + (2 * W + 3) * 4 + 15) & ~15;
  static constexpr int SMEM = BYTES * ROWS;
  static constexpr int MINB = K > 5 ? 2 : W > 8 ? 3 : 1280 / (TH * ROWS);
};

// A product on its way: its value, or (compensated mode) its two factors.
template <typename VT>
struct FlatVal {
  double v;
  __device__ __forceinline__ void set(double a, VT b) { v = __dmul_rn(a, (double)b); }
};
template <>
struct FlatVal<float> {
  float2 v;
  __device__ __forceinline__ void set(double a, float b) { v = make_float2((float)a, b); }
};

// Sum of the products [q, end) of one column, in order.
__device__ __forceinline__ double flat_sum(const FlatVal<double> *v, int q, int end, bool) {
  double s = __dadd_rn(0.0, v[q].v);
  for (++q; q < end; ++q) s = __dadd_rn(s, v[q].v);
  return s;
}
__device__ __forceinline__ double flat_sum(const FlatVal<float> *v, int q, int end, bool pair) {
  if (pair) {
    float2 sc = make_float2(0.f, 0.f);
    for (; q < end; ++q) comp_add(sc, v[q].v.x, v[q].v.y);
    return (double)sc.x + (double)sc.y;
  }
  double s = 0.0;
  for (; q < end; ++q) s = __dadd_rn(s, __dmul_rn((double)v[q].v.x, (double)v[q].v.y));
  return s;
}

template <int W, int K, typename VT, bool MULTI>
__global__ void __launch_bounds__(FlatCfg<W, K>::TH *FlatCfg<W, K>::ROWS, FlatCfg<W, K>::MINB)
    k_num_flat(const ProdTable<VT> src, const int *__restrict__ crpt, int *__restrict__ ccol,
               double *__restrict__ cval, const int *__restrict__ rows, int count,
               int *__restrict__ over, int *__restrict__ n_over, int *__restrict__ err,
               CompArgs comp) {
  using C = FlatCfg<W, K>;
  using FV = FlatVal<VT>;
  constexpr bool COMP = sizeof(VT) == 4;
  extern __shared__ __align__(16) unsigned char smem_flat[];
  const int g = W == 1 ? threadIdx.x >> 5 : 0;
  const int tid = W == 1 ? threadIdx.x & 31 : threadIdx.x;
  const int lane = threadIdx.x & 31, warp = W == 1 ? 0 : threadIdx.x >> 5;
  unsigned char *sb = smem_flat + g * C::BYTES;
  FV *svals = reinterpret_cast<FV *>(sb);
  int *skey = reinterpret_cast<int *>(sb + C::O_KEY);
  int *aux = reinterpret_cast<int *>(sb + C::O_AUX);
  unsigned *maps = reinterpret_cast<unsigned *>(sb + C::O_MAP);
  int *before = reinterpret_cast<int *>(maps + C::LEV * C::WORDS);
  int *cnt = reinterpret_cast<int *>(maps);  // wide buckets
  unsigned *mask = reinterpret_cast<unsigned *>(sb + C::O_FIRST);  // once the tables are read
  unsigned *red = reinterpret_cast<unsigned *>(sb + C::O_RED);     // 2 * W, then the ends
  int *ends = reinterpret_cast<int *>(red + 2 * W);                // first, last column, crowded
  const FlatTab ft{skey, aux, reinterpret_cast<double *>(sb),
                   reinterpret_cast<unsigned short *>(mask), red};

  int my_max_deg = 0, my_redo = 0;
  const int step = gridDim.x * C::ROWS;
  int r = blockIdx.x * C::ROWS + g;
  int row = 0;
  if (r < count) row = rows ? rows[r] : r;
  for (; r < count; r += step) {
    const int this_row = row;
    if (r + step < count) row = rows ? __ldg(rows + r + step) : r + step;
    Operands<VT> op;
    const int lr = prod_row<MULTI>(src, this_row, op);
    const int a0 = op.arpt[lr], a1 = op.arpt[lr + 1];
    const int c0 = crpt[this_row];
    const int n = crpt[this_row + 1] - c0;
    int ne;
    const int total = flat_entries<W, VT>(ft, op.acol, op.aval, op.brpt, a0, a1, C::CAP, tid, warp,
                                          lane, &ne);
    if (total > C::CAP) {  // more products than this kernel holds: listed for the hash kernels
      if (tid == 0) over[atomicAdd(n_over, 1)] = this_row;
      flat_sync<W>();
      continue;
    }
#pragma unroll
    for (int q = 0; q < C::LEV; ++q)
      reinterpret_cast<uint4 *>(maps)[q * C::TH + tid] = make_uint4(0u, 0u, 0u, 0u);
    if (tid == 0) {
      ends[0] = 0x7fffffff;
      ends[1] = -1;
      ends[2] = 0;
    }
    flat_sync<W>();  // walk tables, bitmaps
    const bool dup = total != n;  // more products than entries: some share a column
    int col[K];
    FV val[K];
    // this thread's products: i * TH + tid where i * TH <= last; the warp has
    // any where warp_has(i). Places past the row's last product repeat it.
    const int last = total - 1 - tid;
    auto warp_has = [&](int i) { return (i * W + warp) * 32 < total; };
#pragma unroll
    for (int i = 0; i < K; ++i)
      if (warp_has(i)) {
        const int t = flat_entry(ft, (i * W + warp) * 32, lane, ne);
        const int j = min(i * C::TH + tid, total - 1) + ft.shift[t];
        col[i] = __ldg(op.bcol + j);
        val[i].set(ft.a[t], __ldg(op.bval + j));
      }
    // one B row in order is the row of C already (rows of one warp)
    bool copy = false;
    if constexpr (W == 1) {
      if (ne == 1) {
        copy = true;
        int prev = -1;
#pragma unroll
        for (int i = 0; i < K; ++i)
          if (warp_has(i)) {
            const int left = __shfl_up_sync(0xffffffffu, col[i], 1);
            copy = copy && (i * C::TH > last || (lane > 0 ? left : prev) < col[i]);
            prev = __shfl_sync(0xffffffffu, col[i], 31);
          }
        copy = __all_sync(0xffffffffu, copy);
      }
    }
    int mn = 0x7fffffff, mx = -1;
#pragma unroll
    for (int i = 0; i < K; ++i)
      if (warp_has(i)) {
        mn = min(mn, col[i]);
        mx = max(mx, col[i]);
      }
    mn = __reduce_min_sync(0xffffffffu, mn);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if constexpr (W > 1) {
      if (lane == 0) {
        atomicMin(ends, mn);
        atomicMax(ends + 1, mx);
      }
    }
    flat_sync<W>();  // the tables are read: their room takes keys and values
    if constexpr (W > 1) {
      mn = ends[0];
      mx = ends[1];
    }
    const float range = (float)((long long)mx - mn + 1);
    float scale = (float)(C::WORDS * 32) / range;
    for (int q = tid; q <= C::CH; q += C::TH) mask[q] = 0u;
    // narrow buckets, 32 and more for a product: a bit each. The first
    // product of a bucket sets it in the first bitmap, the next in the second.
    int at[K];  // bucket | bitmap << 20, then the place
#pragma unroll
    for (int i = 0; i < K; ++i)
      if (!copy && i * C::TH <= last) {
        const int b = bucket_of(col[i], mn, scale, C::WORDS * 32);
        const unsigned bit = 1u << (b & 31);
        int lev = 0;
        while (atomicOr(maps + lev * C::WORDS + (b >> 5), bit) & bit)
          if (++lev == C::LEV) {
            ends[2] = 1;  // more products in a bucket than bitmaps
            break;
          }
        at[i] = b | lev << 20;
      }
    flat_sync<W>();
    if (copy) {
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (i * C::TH <= last) {
          skey[i * C::TH + tid] = col[i];
          svals[i * C::TH + tid] = val[i];
        }
      if (tid == 0) skey[total] = 0x7fffffff;
    } else if (ends[2] == 0) {
      // products before each word
      uint4 x = reinterpret_cast<const uint4 *>(maps)[tid];
      int4 c = make_int4(__popc(x.x), __popc(x.y), __popc(x.z), __popc(x.w));
#pragma unroll
      for (int q = 1; q < C::LEV; ++q) {
        x = reinterpret_cast<const uint4 *>(maps)[q * C::TH + tid];
        c.x += __popc(x.x);
        c.y += __popc(x.y);
        c.z += __popc(x.z);
        c.w += __popc(x.w);
      }
      unsigned tot;
      const int ex = (int)flat_scan<W>((unsigned)(c.x + c.y + c.z + c.w), red + W, warp, lane, &tot);
      reinterpret_cast<int4 *>(before)[tid] =
          make_int4(ex, ex + c.x, ex + c.x + c.y, ex + c.x + c.y + c.z);
      if (tid == 0) skey[total] = 0x7fffffff;  // past the last key
      flat_sync<W>();
      unsigned many = 0;  // products that share their bucket
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (i * C::TH <= last) {
          const int w = (at[i] & 0xfffff) >> 5, lev = at[i] >> 20;
          const unsigned bit = 1u << (at[i] & 31);
          int place = before[w];
          unsigned second = 0;
#pragma unroll
          for (int q = 0; q < C::LEV; ++q) {
            const unsigned m = maps[q * C::WORDS + w];
            place += __popc(m & (bit - 1u));
            if (q == 1) second = m & bit;
          }
          if (second) {
            many |= 1u << i;
            // (column, place in the list), for the others of the bucket
            *reinterpret_cast<unsigned long long *>(svals + place + lev) =
                (unsigned long long)col[i] << 13 | (unsigned)(i * C::TH + tid);
          } else {
            skey[place] = col[i];
            svals[place] = val[i];
          }
          at[i] = place | lev << 20;
        }
      flat_sync<W>();
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (many >> i & 1u) {
          const int place = at[i] & 0xfffff;
          const unsigned long long mine =
              (unsigned long long)col[i] << 13 | (unsigned)(i * C::TH + tid);
          at[i] = place;
          // up to LEV products: those of a bucket lie side by side
          const int b = bucket_of(col[i], mn, scale, C::WORDS * 32);
          int size = 2;
          if (C::LEV > 2) size += maps[(C::LEV - 1) * C::WORDS + (b >> 5)] >> (b & 31) & 1u;
          bool later = false;  // an earlier product has the same column
          for (int u = 0; u < size; ++u) {
            const unsigned long long o = reinterpret_cast<unsigned long long *>(svals)[place + u];
            at[i] += o < mine;
            later |= o < mine && o >> 13 == mine >> 13;
          }
          if (later) atomicOr(mask + (at[i] >> 5), 1u << (at[i] & 31));
        }
      flat_sync<W>();
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (many >> i & 1u) {
          skey[at[i]] = col[i];
          svals[at[i]] = val[i];
        }
    } else {
      // columns in few places of their range: wide buckets, about one a
      // product, and a rank inside each
      const int per = min(C::PER, (total + C::TH - 1) / C::TH);
      const int nb = per * C::TH;
      scale = (float)nb / range;
      for (int q = tid; q < nb; q += C::TH) cnt[q] = 0;
      flat_sync<W>();
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (i * C::TH <= last) {
          const int b = bucket_of(col[i], mn, scale, nb);
          at[i] = b << 13 | atomicAdd(cnt + b, 1);
        }
      flat_sync<W>();
      int local[C::PER], sum = 0;
#pragma unroll
      for (int q = 0; q < C::PER; ++q) {
        local[q] = q < per ? cnt[tid * per + q] : 0;
        sum += local[q];
      }
      unsigned tot;
      int ex = (int)flat_scan<W>((unsigned)sum, red + W, warp, lane, &tot);
#pragma unroll
      for (int q = 0; q < C::PER; ++q) {
        if (q < per) cnt[tid * per + q] = ex;
        ex += local[q];
      }
      if (tid == 0) {
        cnt[nb] = total;
        skey[total] = 0x7fffffff;
      }
      flat_sync<W>();
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (i * C::TH <= last) {
          const int q = cnt[at[i] >> 13] + (at[i] & 0x1fff);
          skey[q] = col[i];
          aux[q] = i * C::TH + tid;
        }
      flat_sync<W>();
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (i * C::TH <= last) {
          const int b = at[i] >> 13, p = i * C::TH + tid;
          const int st = cnt[b], en = cnt[b + 1];
          int place = st;
          bool later = false;
          for (int u = st; u < en; ++u) {
            const int x = skey[u];
            if (x == col[i]) {
              const bool o = aux[u] < p;
              place += o;
              later |= o;
            } else {
              place += x < col[i];
            }
          }
          at[i] = place;
          if (later) atomicOr(mask + (place >> 5), 1u << (place & 31));
        }
      flat_sync<W>();
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (i * C::TH <= last) {
          skey[at[i]] = col[i];
          svals[at[i]] = val[i];
        }
    }
    flat_sync<W>();
    const bool pair = COMP && comp.owned && W * K <= 20 && a1 - a0 <= comp.nmax;
    // C is written once and not read here again: streaming stores
    bool wrong = false;  // symbolic/numeric disagreement
    if (!dup) {
      for (int q = tid; q < total; q += C::TH) {
        const int key = skey[q];
        wrong |= skey[q + 1] == key;
        __stcs(ccol + c0 + q, key);
        __stcs(cval + c0 + q, flat_sum(svals, q, q + 1, pair));
      }
    } else {
      // consecutive words of places for each warp; marked places are added to
      // the one before them
      const int words = (total + 31) >> 5, mine = (words + W - 1) / W, w0 = warp * mine;
      int marked = 0, all = 0;  // before this warp's words, and in the row
      for (int w = lane; w < words; w += 32) {
        const int c = __popc(mask[w]);
        all += c;
        if (w < w0) marked += c;
      }
      all = __reduce_add_sync(0xffffffffu, all);
      if constexpr (W > 1) marked = __reduce_add_sync(0xffffffffu, marked);
      wrong = total - all != n;
      for (int w = w0; w < min(w0 + mine, words) && !wrong; ++w) {
        const int q = w * 32 + lane;
        const unsigned m = mask[w];
        if (q < total && !(m >> lane & 1u)) {
          const int pos = q - marked - __popc(m & ((1u << lane) - 1u));
          const int key = skey[q];
          int end = q + 1;
          if ((lane < 31 ? m >> (lane + 1) : mask[w + 1]) & 1u)
            while (skey[end] == key) ++end;
          __stcs(ccol + c0 + pos, key);
          __stcs(cval + c0 + pos, flat_sum(svals, q, end, pair));
        }
        marked += __popc(m);
      }
    }
    if (wrong) atomicOr(err, ERR_COUNT);
    if (COMP) {
      if (pair) my_max_deg = max(my_max_deg, a1 - a0);
      else ++my_redo;
    }
    flat_sync<W>();
  }
  if (COMP && tid == 0) {
    if (my_max_deg) atomicMax(comp.max_deg, my_max_deg);
    if (my_redo) atomicAdd(comp.redo, my_redo);
  }
}

template <int W, int K, typename VT>
static cudaError_t run_num_flat(const ProdTable<VT> &t, const int *crpt, int *ccol, double *cval,
                                const int *rows, int count, int *over, int *n_over, int *err,
                                CompArgs comp, cudaStream_t s) {
  using C = FlatCfg<W, K>;
  auto kern = t.prod_of_row ? k_num_flat<W, K, VT, true> : k_num_flat<W, K, VT, false>;
  const int threads = C::TH * C::ROWS;
  const int grid = persistent_grid((const void *)kern, threads, C::SMEM, count, C::ROWS);
  if (grid <= 0) return cudaErrorInvalidConfiguration;
  kern<<<grid, threads, C::SMEM, s>>>(t, crpt, ccol, cval, rows, count, over, n_over, err, comp);
  return cudaGetLastError();
}

// Rows of at most 16 << bin entries.
template <typename VT>
static cudaError_t flat_bin(int bin, const ProdTable<VT> &t, const int *crpt, int *ccol,
                            double *cval, const int *rows, int count, int *over, int *n_over,
                            int *err, CompArgs comp, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
#define NSPB_FB(W, K) \
  run_num_flat<W, K, VT>(t, crpt, ccol, cval, rows, count, over, n_over, err, comp, s)
  switch (bin) {
    case 0:
    case 1: return NSPB_FB(1, 2);
    case 2:
    case 3: return NSPB_FB(1, 5);
    case 4: return NSPB_FB(2, 5);
    case 5: return NSPB_FB(4, 5);
    case 6: return NSPB_FB(8, 5);
    case 7: return NSPB_FB(16, 5);
    default: return NSPB_FB(16, 10);
  }
#undef NSPB_FB
}

cudaError_t launch_numeric_flat(int bin, const ProdTable<double> &t, const int *crpt, int *ccol,
                                double *cval, const int *rows, int count, int *over, int *n_over,
                                int *err, cudaStream_t s) {
  return flat_bin<double>(bin, t, crpt, ccol, cval, rows, count, over, n_over, err,
                          CompArgs{0, nullptr, nullptr, false}, s);
}

cudaError_t launch_numeric_comp_flat(int bin, bool owned, const ProdTable<float> &t,
                                     const int *crpt, int *ccol, double *cval, const int *rows,
                                     int count, int nmax, int *redo, int *max_deg, int *over,
                                     int *n_over, int *err, cudaStream_t s) {
  return flat_bin<float>(bin, t, crpt, ccol, cval, rows, count, over, n_over, err,
                         CompArgs{nmax, redo, max_deg, owned}, s);
}

}  // namespace nspb
