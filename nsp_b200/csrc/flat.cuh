// The products of one A row as one flat list, spread evenly over the W warps
// that share the row.
#pragma once

#include "common.cuh"

namespace nspb {

template <int W>
__device__ __forceinline__ void flat_sync() {
  if constexpr (W == 1) __syncwarp();
  else __syncthreads();
}

// Exclusive scan of one value per thread over the W warps of a row; *total:
// the sum. red: W values, not in use by another call without a barrier
// between the two. Contains one barrier (none for W = 1).
template <int W>
__device__ __forceinline__ unsigned flat_scan(unsigned v, unsigned *red, int warp, int lane,
                                              unsigned *total) {
  unsigned incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if constexpr (W == 1) {
    *total = __shfl_sync(0xffffffffu, incl, 31);
    return incl - v;
  } else {
    if (lane == 31) red[warp] = incl;
    __syncthreads();
    const unsigned mine = lane < W ? red[lane] : 0u;
    *total = __reduce_add_sync(0xffffffffu, mine);
    return incl - v + __reduce_add_sync(0xffffffffu, lane < warp ? mine : 0u);
  }
}

// Walk tables of a row: its non-empty A entries in order, with the place of
// each one's first product, the distance from a product's place to its B
// entry, the A value, and for each 32 products the entry of the first one.
struct FlatTab {
  int *start, *shift;
  double *a;  // unused without values
  unsigned short *first;
  unsigned *red;  // 2 * W
};

// Fills the tables of the A row [a0, a1) with at most `cap` products; returns
// the row's products, or a number above cap when it has more (the tables are
// then not to be used). *entries: its non-empty A entries. The caller's next
// barrier makes the tables visible. Lengths are clamped to cap + 1 so that the
// packed scan (22 bits of products, 10 of entries) cannot overflow: at most
// 512 threads and 5120 products.
template <int W, typename VT>
__device__ __forceinline__ int flat_entries(const FlatTab &ft, const int *acol, const VT *aval,
                                            const int *brpt, int a0, int a1, int cap, int tid,
                                            int warp, int lane, int *entries) {
  constexpr int TH = 32 * W;
  static_assert(TH <= 512, "the packed scan holds 10 bits of entries");
  int total = 0, ne = 0;
  // start and (clamped) length of the B row of entry base + tid, and its A value
  auto load = [&](int base, int &s0, double &av) {
    if (base + tid >= a1) return 0;
    const int k = ld_stream(acol + base + tid);
    if (aval) av = ldv_stream(aval + base + tid);
    s0 = __ldg(brpt + k);
    return min(__ldg(brpt + k + 1) - s0, cap + 1);
  };
  auto enter = [&](unsigned ex, int len, int s0, double av) {
    const int p = total + (int)(ex & 0x3fffffu), t = ne + (int)(ex >> 22);
    if (len > 0 && p + len <= cap) {
      ft.start[t] = p;
      ft.shift[t] = s0 - p;
      if (aval) ft.a[t] = av;
      for (int c = (p + 31) >> 5; c << 5 < p + len; ++c) ft.first[c] = (unsigned short)t;
    }
  };
  // one warp has them all: the others wait for the sums instead of scanning
  // zeros beside it (random 100003 x 80021 x 120011, the whole product: 878 -> 857 us)
  if (W > 1 && a1 - a0 <= 32) {
    if (warp == 0) {
      int s0 = 0;
      double av = 0.0;
      const int len = load(a0, s0, av);
      unsigned sum;
      const unsigned ex = flat_scan<1>((unsigned)len | (len > 0 ? 1u << 22 : 0u), ft.red, 0, lane,
                                       &sum);
      enter(ex, len, s0, av);
      if (lane == 0) ft.red[0] = sum;
    }
    __syncthreads();
    const unsigned sum = ft.red[0];
    *entries = (int)(sum >> 22);
    return (int)(sum & 0x3fffffu);
  }
  for (int base = a0;; base += TH) {
    int s0 = 0;
    double av = 0.0;
    const int len = load(base, s0, av);
    unsigned sum;
    const unsigned ex = flat_scan<W>((unsigned)len | (len > 0 ? 1u << 22 : 0u), ft.red, warp, lane,
                                     &sum);
    enter(ex, len, s0, av);
    total += (int)(sum & 0x3fffffu);
    ne += (int)(sum >> 22);
    if (total > cap || base + TH >= a1) break;
    flat_sync<W>();  // red
  }
  *entries = ne;
  return total;
}

// The table entry of product p0 + lane (p0 a multiple of 32 and a product of
// the row; past the row's last product: its last entry). The whole warp calls
// it with one p0.
__device__ __forceinline__ int flat_entry(const FlatTab &ft, int p0, int lane, int ne) {
  const int t0 = ft.first[p0 >> 5];
  const int s = t0 + 1 + lane < ne ? ft.start[t0 + 1 + lane] - p0 : 32;
  const unsigned m = __reduce_or_sync(0xffffffffu, s < 32 ? 1u << s : 0u);
  return t0 + __popc(m & (0xffffffffu >> (31 - lane)));
}

}  // namespace nspb
