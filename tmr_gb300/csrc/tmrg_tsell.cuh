// Tiled sliced ELL: a square sparse matrix stored for repeated products with
// a gathered vector.  TS_ROWS consecutive rows form a tile (one block of the
// product kernels); a tile lists its distinct columns once, ascending, and
// its entries name them by a 16-bit place in that list.  The product loads
// the tile's vector values into shared memory, a few per row instead of one
// per entry (27-point rows numbered along a Morton curve: 2 to 3), and an
// entry is its value and two bytes instead of its value and four.  Inside a
// tile rows are ordered by length, longest first, and each 32 rows form a
// slice stored entry-major, so a warp's k-th entries are one run of memory;
// an entry's place in its row is that of the CSR matrix.
#pragma once

#include "tmrg_prims.cuh"

namespace tmrg {

constexpr int TS_ROWS = 256;
constexpr int TS_SLICES = TS_ROWS / 32;
// Distinct columns a tile may have, the space of its sorted list (a power of
// two) and the slots of the hash table that finds them.  Rows numbered along
// a curve have 600 to 900; the second size is for rows numbered with less
// locality (many small blocks) and ends where the products' input, four FP64
// components a column, fills the shared memory.
struct TsSize {
  int cols, list, slots;
};
constexpr TsSize TS_SIZES[2] = {{2048, 2048, 4096}, {7000, 8192, 16384}};

struct TSellView {
  long long n;
  const unsigned *uoff;  // per tile: its columns in ucol
  const int *ucol;
  const int *row;        // per position: the row (-1: none) and its length
  const uint16_t *len;
  const unsigned *soff;  // per slice: its entries, in units of 32
  const uint16_t *idx;
};
struct TSell {
  bool ok = false;
  long long n = 0, tiles = 0, entries = 0;  // entries with the slices' padding
  int maxu = 0;                             // most columns of a tile
  DBuf<unsigned> uoff, soff;
  DBuf<int> ucol, row;
  DBuf<uint16_t> len, idx;
  TSellView view() const { return TSellView{n, uoff.p, ucol.p, row.p, len.p, soff.p, idx.p}; }
};

// Pass 1, one block per tile: the distinct columns (ascending, at tile *
// Z.list of `tmp`) and their number, the row order and the slice sizes.
// state[0]: some tile has too many columns, state[1]: the most columns.
static __global__ void __launch_bounds__(TS_ROWS)
    k_ts_columns(long long n, TsSize Z, const int *__restrict__ rp, const int *__restrict__ ci,
                 int *tmp, unsigned *ucount, int *row, uint16_t *len, unsigned *ssize, int *state) {
  extern __shared__ __align__(16) int ts_smem[];
  int *tab = ts_smem, *cols = ts_smem + Z.slots;
  __shared__ int slen[TS_ROWS];
  __shared__ int s_n, s_stop;
  const int t = threadIdx.x;
  const long long r0 = (long long)blockIdx.x * TS_ROWS;
  for (int i = t; i < Z.slots; i += TS_ROWS) tab[i] = -1;
  const long long r = r0 + t;
  const int a = r < n ? rp[r] : 0, b = r < n ? rp[r + 1] : 0;
  slen[t] = r < n ? b - a : -1;
  if (t == 0) {
    s_n = 0;
    s_stop = *(volatile int *)state;  // some tile has too many: all for nothing
  }
  __syncthreads();
  if (s_stop) return;
  // the tile's entries are one run; threads take them in turn
  const int e0 = rp[min(n, r0)], e1 = rp[min(n, r0 + TS_ROWS)];
  for (int e = e0 + t; e < e1 && *(volatile int *)&s_n <= Z.cols; e += TS_ROWS) {
    const int c = __ldg(ci + e);
    unsigned h = ((unsigned)c * 0x9E3779B1u) >> 16 & (unsigned)(Z.slots - 1);
    // an empty slot always ends a probe: threads stop adding past Z.cols
    for (int it = 0; it < Z.slots; it++) {
      int was = *(volatile int *)(tab + h);
      if (was == -1) {
        was = atomicCAS(tab + h, -1, c);
        if (was == -1) atomicAdd(&s_n, 1);
      }
      if (was == -1 || was == c) break;
      if (*(volatile int *)&s_n > Z.cols) break;
      h = (h + 1) & (unsigned)(Z.slots - 1);
    }
  }
  // row order: longest first, equal lengths in row order
  int place = 0;
  for (int k = 0; k < TS_ROWS; k++) {
    const int l = slen[k];
    place += l > slen[t] || (l == slen[t] && k < t);
  }
  const long long q = r0 + place;
  row[q] = r < n ? (int)r : -1;
  len[q] = r < n ? (uint16_t)min(b - a, 65535) : 0;
  // a slice's size is that of its first (longest) row
  if ((place & 31) == 0) ssize[q >> 5] = (unsigned)max(slen[t], 0);
  __syncthreads();
  const int m = s_n;
  if (t == 0) {
    ucount[blockIdx.x] = (unsigned)min(m, Z.cols);
    if (m > Z.cols) atomicOr(state, 1);
    atomicMax(state + 1, min(m, Z.cols));
  }
  if (m > Z.cols) return;  // uniform
  // the taken slots to the front, then a bitonic sort padded with INT_MAX
  __shared__ int s_at;
  if (t == 0) s_at = 0;
  int p2 = 32;
  while (p2 < m) p2 <<= 1;
  for (int i = t; i < p2; i += TS_ROWS) cols[i] = 0x7fffffff;
  __syncthreads();
  for (int i = t; i < Z.slots; i += TS_ROWS) {
    const int c = tab[i];
    const unsigned w = __ballot_sync(0xffffffffu, c >= 0);
    int o = 0;
    if ((t & 31) == 0 && w) o = atomicAdd(&s_at, __popc(w));
    o = __shfl_sync(0xffffffffu, o, 0);
    if (c >= 0) cols[o + __popc(w & ((1u << (t & 31)) - 1u))] = c;
  }
  __syncthreads();
  for (int k = 2; k <= p2; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = t; i < p2; i += TS_ROWS) {
        const int o = i ^ j;
        if (o > i) {
          const int x = cols[i], y = cols[o];
          if ((x > y) == ((i & k) == 0)) {
            cols[i] = y;
            cols[o] = x;
          }
        }
      }
      __syncthreads();
    }
  for (int i = t; i < m; i += TS_ROWS) tmp[(long long)blockIdx.x * Z.list + i] = cols[i];
}
// Pass 2, one block per tile: the column list in place and every entry's
// place in it.
static __global__ void __launch_bounds__(TS_ROWS)
    k_ts_index(int list, const int *__restrict__ rp, const int *__restrict__ ci,
               const int *__restrict__ tmp, const unsigned *__restrict__ uoff,
               const int *__restrict__ row, const unsigned *__restrict__ soff, int *ucol,
               uint16_t *idx) {
  extern __shared__ __align__(16) int ts_smem[];
  int *cols = ts_smem;
  const int t = threadIdx.x;
  const unsigned u0 = uoff[blockIdx.x];
  const int m = (int)(uoff[blockIdx.x + 1] - u0);
  for (int i = t; i < m; i += TS_ROWS) {
    const int c = tmp[(long long)blockIdx.x * list + i];
    cols[i] = c;
    ucol[u0 + i] = c;
  }
  __syncthreads();
  const long long q = (long long)blockIdx.x * TS_ROWS + t;
  const int r = row[q];
  const int p0 = r >= 0 ? rp[r] : 0, len = r >= 0 ? rp[r + 1] - p0 : 0;
  const unsigned s0 = soff[q >> 5], size = soff[(q >> 5) + 1] - s0;
  uint16_t *out = idx + (long long)s0 * 32 + (t & 31);
  for (unsigned k = 0; k < size; k++) {
    int lo = 0;
    if ((int)k < len) {
      const int c = __ldg(ci + p0 + k);
      int hi = m;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (cols[mid] < c)
          lo = mid + 1;
        else
          hi = mid;
      }
    }
    out[(long long)k * 32] = (uint16_t)lo;
  }
}
// Values of the entries (0 in the padding), from CSR.
template <typename S, typename T>
__global__ void __launch_bounds__(TS_ROWS)
    k_ts_values(const int *__restrict__ rp, const S *__restrict__ vals,
                const int *__restrict__ row, const unsigned *__restrict__ soff, T *out) {
  const long long q = (long long)blockIdx.x * TS_ROWS + threadIdx.x;
  const int r = row[q];
  const int p0 = r >= 0 ? rp[r] : 0, len = r >= 0 ? rp[r + 1] - p0 : 0;
  const unsigned s0 = soff[q >> 5], size = soff[(q >> 5) + 1] - s0;
  T *o = out + (long long)s0 * 32 + (threadIdx.x & 31);
  for (unsigned k = 0; k < size; k++)
    o[(long long)k * 32] = (int)k < len ? (T)__ldg(vals + p0 + k) : T(0);
}

// Builds the structure; false (nothing kept) where a tile has more columns
// than the larger size.
inline bool tsell_build(TSell &M, long long n, const int *rp, const int *ci, cudaStream_t s) {
  M = TSell();
  if (n <= 0) return false;
  const long long tiles = (n + TS_ROWS - 1) / TS_ROWS;
  const unsigned g = (unsigned)tiles;
  for (const TsSize &Z : TS_SIZES) {
    const int smem = (Z.slots + Z.list) * (int)sizeof(int);
    TMRG_CUDA(cudaFuncSetAttribute(k_ts_columns, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (TS_SIZES[1].slots + TS_SIZES[1].list) * (int)sizeof(int)));
    DBuf<int> tmp((size_t)tiles * Z.list, s), state(2, s);
    state.zero();
    M.uoff.alloc(tiles + 1, s);
    M.soff.alloc(tiles * TS_SLICES + 1, s);
    M.row.alloc(tiles * TS_ROWS, s);
    M.len.alloc(tiles * TS_ROWS, s);
    launch(k_ts_columns, g, TS_ROWS, smem, s, n, Z, rp, ci, tmp.p, M.uoff.p, M.row.p, M.len.p,
           M.soff.p, state.p);
    exclusive_scan<unsigned>(M.uoff.p, M.uoff.p, tiles, s);
    exclusive_scan<unsigned>(M.soff.p, M.soff.p, tiles * TS_SLICES, s);
    const unsigned *pv[4] = {M.uoff.p + tiles, M.soff.p + tiles * TS_SLICES,
                             (const unsigned *)state.p, (const unsigned *)state.p + 1};
    unsigned hv[4];
    read_scalars(pv, hv, s);
    if (hv[2]) continue;
    M.n = n;
    M.tiles = tiles;
    M.entries = 32LL * hv[1];
    M.maxu = (int)hv[3];
    M.ucol.alloc((size_t)hv[0] + 1, s);
    M.idx.alloc((size_t)M.entries + 1, s);
    launch(k_ts_index, g, TS_ROWS, Z.list * sizeof(int), s, Z.list, rp, ci, (const int *)tmp.p,
           (const unsigned *)M.uoff.p, (const int *)M.row.p, (const unsigned *)M.soff.p,
           M.ucol.p, M.idx.p);
    M.ok = true;
    return true;
  }
  M = TSell();
  return false;
}
template <typename S, typename T>
inline void tsell_values(const TSell &M, const int *rp, const S *vals, DBuf<T> &out,
                         cudaStream_t s) {
  out.alloc((size_t)M.entries + 1, s);
  launch((k_ts_values<S, T>), (unsigned)M.tiles, TS_ROWS, 0, s, rp, vals, (const int *)M.row.p,
         (const unsigned *)M.soff.p, out.p);
}

}  // namespace tmrg
