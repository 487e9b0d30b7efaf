// Symbolic phase of rows of up to 3072 intermediate products: the row's
// products as one flat list (flat.cuh), each inserted into a hash table of
// the row's own in shared memory.
//
// The row-group kernel (k_sym_group) takes one B row a step, a lane an entry:
// with B rows of 4..32 entries half its lanes idle, and one step's loads are
// in flight at a time. Here all lanes have a product, and all products of a
// thread are loaded before the first is inserted. Bound: issue and latency of
// the inserts; the table has at least twice the products, so that most take
// one exchange (reading the slot first made it slower: 121 -> 134 us below; so did twelve
// products a thread with half the warps, 150, and three with twice the warps, 157).
// Measured, row-group kernel -> this one: rows of 385..768 products of a random
// product (4..32 entries a row) 163 -> 121 us, all rows of it 366 -> 250; 20
// such products in one call 1151 -> 861; power-law 1M, rows of up to 3072
// products 2700 -> 930; R (A P) of 50^3 146 -> 40; 7-point 32^3 36 -> 24.
// Where B's rows fill three quarters of the lanes and the columns repeat, the
// row group is faster: 27-point 40 x 33 x 25, counted alone, 65 -> 76 us.
#include "flat.cuh"
#include "internal.h"
#include "launch_util.h"

namespace nspb {

// W warps a row, K products a thread; a table of 2^LOG2T slots, at least twice
// the products.
template <int W, int K, int LOG2T>
struct SymFlatCfg {
  static constexpr int TH = 32 * W;
  static constexpr int ROWS = W == 1 ? 4 : 1;  // rows a block
  static constexpr int CAP = TH * K;
  static constexpr int T = 1 << LOG2T;
  static constexpr int O_START = T * 4;
  static constexpr int O_SHIFT = O_START + CAP * 4;
  static constexpr int O_FIRST = O_SHIFT + CAP * 4;
  static constexpr int O_RED = O_FIRST + ((CAP / 16 + 15) & ~15);
  static constexpr int BYTES = (O_RED + 2 * W * 4 + 15) & ~15;
  static constexpr int SMEM = BYTES * ROWS;
  static constexpr int MINB = W >= 16 ? 3 : 1536 / (TH * ROWS);
};

template <int W, int K, int LOG2T, bool MULTI>
__global__ void __launch_bounds__(SymFlatCfg<W, K, LOG2T>::TH *SymFlatCfg<W, K, LOG2T>::ROWS,
                                  SymFlatCfg<W, K, LOG2T>::MINB)
    k_sym_flat(const ProdTable<void> src, const int *__restrict__ rows, int count,
               int *__restrict__ row_nz, int *__restrict__ err) {
  using C = SymFlatCfg<W, K, LOG2T>;
  extern __shared__ __align__(16) unsigned char smem_sf[];
  const int g = W == 1 ? threadIdx.x >> 5 : 0;
  const int tid = W == 1 ? threadIdx.x & 31 : threadIdx.x;
  const int lane = threadIdx.x & 31, warp = W == 1 ? 0 : threadIdx.x >> 5;
  unsigned char *sb = smem_sf + g * C::BYTES;
  int *table = reinterpret_cast<int *>(sb);
  unsigned *red = reinterpret_cast<unsigned *>(sb + C::O_RED);
  const FlatTab ft{reinterpret_cast<int *>(sb + C::O_START),
                   reinterpret_cast<int *>(sb + C::O_SHIFT), nullptr,
                   reinterpret_cast<unsigned short *>(sb + C::O_FIRST), red};
  const int step = gridDim.x * C::ROWS;
  int r = blockIdx.x * C::ROWS + g;
  int row = 0;
  if (r < count) row = rows ? rows[r] : r;
  for (; r < count; r += step) {
    const int this_row = row;
    if (r + step < count) row = rows ? __ldg(rows + r + step) : r + step;
    Operands<void> op;
    const int lr = prod_row<MULTI>(src, this_row, op);
    const int a0 = op.arpt[lr], a1 = op.arpt[lr + 1];
#pragma unroll
    for (int q = 0; q < (C::T / 4 + C::TH - 1) / C::TH; ++q)
      if (C::T / 4 % C::TH == 0 || q * C::TH + tid < C::T / 4)
        reinterpret_cast<int4 *>(table)[q * C::TH + tid] =
            make_int4(kEmpty, kEmpty, kEmpty, kEmpty);
    int ne;
    const int total = flat_entries<W, double>(ft, op.acol, nullptr, op.brpt, a0, a1, C::CAP, tid,
                                              warp, lane, &ne);
    flat_sync<W>();  // walk tables, hash table
    int nz = 0;
    if (total <= C::CAP) {
      int col[K];
      const int last = total - 1 - tid;
#pragma unroll
      for (int i = 0; i < K; ++i)
        if ((i * W + warp) * 32 < total) {
          const int t = flat_entry(ft, (i * W + warp) * 32, lane, ne);
          col[i] = __ldg(op.bcol + min(i * C::TH + tid, total - 1) + ft.shift[t]);
        }
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (i * C::TH <= last) {
          unsigned h = hash_slot<LOG2T>(col[i]);
#pragma unroll 1
          for (int q = 0;; ++q) {
            const int old = atomicCAS(table + h, kEmpty, col[i]);
            nz += old == kEmpty;
            if (old == kEmpty || old == col[i]) break;
            if (q == C::T) {
              atomicOr(err, ERR_PROBE);
              break;
            }
            h = (h + 1u) & (C::T - 1u);
          }
        }
    } else {  // many products of few columns (a narrow C): B row by B row
      for (int j = a0 + warp; j < a1; j += W) {
        const int k = __ldg(op.acol + j);
        for (int e = __ldg(op.brpt + k) + lane; e < __ldg(op.brpt + k + 1); e += 32)
          nz += sym_insert<LOG2T>(table, __ldg(op.bcol + e), err);
      }
    }
    nz = __reduce_add_sync(0xffffffffu, nz);
    if constexpr (W == 1) {
      if (lane == 0) row_nz[this_row] = nz;
      __syncwarp();
    } else {
      if (lane == 0) red[W + warp] = (unsigned)nz;
      __syncthreads();
      if (warp == 0) {
        nz = (int)__reduce_add_sync(0xffffffffu, lane < W ? red[W + lane] : 0u);
        if (lane == 0) row_nz[this_row] = nz;
      }
    }
  }
}

template <int W, int K, int LOG2T>
static cudaError_t run_sym_flat(const ProdTable<void> &t, const int *rows, int count, int *row_nz,
                                int *err, cudaStream_t s) {
  using C = SymFlatCfg<W, K, LOG2T>;
  auto kern = t.prod_of_row ? k_sym_flat<W, K, LOG2T, true> : k_sym_flat<W, K, LOG2T, false>;
  const int threads = C::TH * C::ROWS;
  const int grid = persistent_grid((const void *)kern, threads, C::SMEM, count, C::ROWS);
  if (grid <= 0) return cudaErrorInvalidConfiguration;
  kern<<<grid, threads, C::SMEM, s>>>(t, rows, count, row_nz, err);
  return cudaGetLastError();
}

// Bin b holds rows of at most 24 << b columns (more with a fuller sym_fill_pct)
// and, unless C is that narrow, products.
cudaError_t launch_symbolic_flat(int bin, const ProdTable<void> &t, const int *rows, int count,
                                 int *row_nz, int *err, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  switch (bin) {
    case 0: return run_sym_flat<1, 1, 6>(t, rows, count, row_nz, err, s);
    case 1: return run_sym_flat<1, 2, 7>(t, rows, count, row_nz, err, s);
    case 2: return run_sym_flat<1, 3, 8>(t, rows, count, row_nz, err, s);
    case 3: return run_sym_flat<1, 6, 9>(t, rows, count, row_nz, err, s);
    case 4: return run_sym_flat<2, 6, 10>(t, rows, count, row_nz, err, s);
    case 5: return run_sym_flat<4, 6, 11>(t, rows, count, row_nz, err, s);
    case 6: return run_sym_flat<8, 6, 12>(t, rows, count, row_nz, err, s);
    default: return run_sym_flat<16, 6, 13>(t, rows, count, row_nz, err, s);
  }
}

}  // namespace nspb
