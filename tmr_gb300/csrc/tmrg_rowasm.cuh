// Assembly of a sparse matrix from element matrices by rows: the mass matrix
// of the density filter and the Helmholtz operator of linear elements on
// octree (8-node) and quadtree (4-node) forests, dependent nodes condensed
// onto the independent nodes they interpolate.
#pragma once

#include <algorithm>

#include "tmrg_prims.cuh"

namespace tmrg {

constexpr int FMAXK = 27;  // distinct independent nodes one element touches

struct ElemCtx {
  const int *conn;
  const int *dptr, *dconn;
  const double *dw;
  int *err;
  int npe;  // 8 (octree) or 4 (quadtree)
};

// Merged element block: distinct nodes U[0..K) in first-appearance order
// and L[u][v] summed over (a, b, p, q) in loop order, from the element's
// entries ent.direct(e, a, b).
template <typename Entry>
__device__ int element_block(const ElemCtx &c, const Entry &ent, long long e, int *U,
                             double (*L)[FMAXK]) {
  const int npe = c.npe;
  const int *ec = c.conn + e * npe;
  int ni[8][4];
  double nw[8][4];
  int nc[8];
  int K = 0;
  for (int a = 0; a < npe; a++) {
    int g = ec[a];
    if (g >= 0) {
      nc[a] = 1;
      ni[a][0] = g;
      nw[a][0] = 1.0;
    } else {
      int d = -g - 1;
      int p0 = c.dptr[d], p1 = c.dptr[d + 1];
      nc[a] = p1 - p0;
      if (nc[a] > 4) {
        atomicExch(c.err, 1);
        nc[a] = 4;
      }
      for (int p = 0; p < nc[a]; p++) {
        ni[a][p] = c.dconn[p0 + p];
        nw[a][p] = c.dw[p0 + p];
      }
    }
    for (int p = 0; p < nc[a]; p++) {
      int u = 0;
      while (u < K && U[u] != ni[a][p]) u++;
      if (u == K) {
        if (K == FMAXK) {
          atomicExch(c.err, 1);
          return K;
        }
        U[K++] = ni[a][p];
      }
    }
  }
  if (!L) return K;
  for (int u = 0; u < K; u++)
    for (int v = 0; v < K; v++) L[u][v] = 0.0;
  for (int a = 0; a < npe; a++)
    for (int b = 0; b < npe; b++) {
      const double mab = ent.direct(e, a, b);
      for (int p = 0; p < nc[a]; p++) {
        int u = 0;
        while (U[u] != ni[a][p]) u++;
        double t = __dmul_rn(mab, nw[a][p]);
        for (int q = 0; q < nc[b]; q++) {
          int v = 0;
          while (U[v] != ni[b][q]) v++;
          L[u][v] = __dadd_rn(L[u][v], __dmul_rn(t, nw[b][q]));
        }
      }
    }
  return K;
}

// ---------------------------------------------------------------------
// The matrix by rows.  Sorting every block entry by (row, column) moves K^2
// records of 20 bytes per element through 5 or more passes; here only the K
// block rows of an element are sorted, by their node, and a row adds its
// block rows into a hash table in shared memory, element after element (the
// order of the sums is that of the sorted entries, hence the same bits).
// An element without dependent nodes needs no stored block: its entry for
// corners a and b is ent.regular(e, a ^ b).
// Bound by the probes and the rank pass of the small rows (1.9 ms for 2.56M
// rows of 27 columns) and by local memory in the hanging elements' blocks
// (0.8 ms); building this filter with its restrictions and filtering once
// went from 23.0 to 13.1 ms, 14.9 of the 23.0 the sort and its passes.
struct RowAsm {
  const int *conn;
  int npe;
  const unsigned *hoff;     // per element: place among the hanging ones
  const unsigned *ucnt;     // per hanging element: first of its distinct nodes,
  const unsigned *boff;     // and of its block
  const int *unode;
  const double *block;
  const unsigned *srp;      // per node: its block rows in `slot`,
  const uint32_t *slot;     // element << 5 | block row, elements ascending
  __device__ __forceinline__ bool hanging(unsigned e) const {
    return hoff[e + 1] != hoff[e];
  }
  __device__ __forceinline__ int nodes(unsigned e) const {
    if (!hanging(e)) return npe;
    const unsigned h = hoff[e];
    return (int)(ucnt[h + 1] - ucnt[h]);
  }
};
// Elements with a stored block: those with a dependent node, or with one
// node twice (a collapsed block), or all of them (`all`).
static __global__ void k_fa_hanging(long long ne, int npe, const int *__restrict__ conn, int all,
                             unsigned *flag) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  bool h = all != 0;
  int g[8];
#pragma unroll
  for (int a = 0; a < 8; a++) {
    g[a] = a < npe ? __ldg(conn + e * npe + a) : 0;
    if (a < npe) h |= g[a] < 0;
#pragma unroll
    for (int b = 0; b < a; b++) h |= a < npe && g[a] == g[b];
  }
  flag[e] = h ? 1u : 0u;
}
static __global__ void k_fa_list(long long ne, const unsigned *__restrict__ hoff, unsigned *list) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < ne && hoff[e + 1] != hoff[e]) list[hoff[e]] = (unsigned)e;
}
// total: entries of all blocks, which the 32-bit places of the scan must hold.
template <typename Entry>
__global__ void k_fa_count(long long nh, ElemCtx c, Entry ent,
                           const unsigned *__restrict__ list,
                           unsigned *ucnt, unsigned *bcnt, unsigned long long *total) {
  const long long h = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned kk = 0;
  if (h < nh) {
    int U[FMAXK];
    const int K = element_block(c, ent, list[h], U, nullptr);
    kk = (unsigned)(K * K);
    ucnt[h] = (unsigned)K;
    bcnt[h] = kk;
  }
  kk = __reduce_add_sync(0xffffffffu, kk);
  if ((threadIdx.x & 31) == 0 && kk) atomicAdd(total, (unsigned long long)kk);
}
template <typename Entry>
__global__ void __launch_bounds__(64)
    k_fa_blocks(long long nh, ElemCtx c, Entry ent, const unsigned *__restrict__ list,
                const unsigned *__restrict__ uoff, const unsigned *__restrict__ boff, int *unode,
                double *block) {
  const long long h = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= nh) return;
  int U[FMAXK];
  double L[FMAXK][FMAXK];
  const int K = element_block(c, ent, list[h], U, L);
  const unsigned u0 = uoff[h], b0 = boff[h];
  for (int u = 0; u < K; u++) {
    unode[u0 + u] = U[u];
    for (int v = 0; v < K; v++) block[b0 + u * K + v] = L[u][v];
  }
}
// Block rows of every element (soff: their scanned counts) by node.
static __global__ void k_fa_slot_count(long long ne, RowAsm A, unsigned *cnt) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < ne) cnt[e] = (unsigned)A.nodes((unsigned)e);
}
static __global__ void k_fa_slots(long long ne, RowAsm A, const unsigned *__restrict__ soff,
                           uint32_t *keys, uint32_t *vals) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  const unsigned o = soff[e];
  const int K = (int)(soff[e + 1] - o);
  const int *U = A.hanging((unsigned)e) ? A.unode + A.ucnt[A.hoff[e]] : A.conn + e * A.npe;
  for (int u = 0; u < K; u++) {
    keys[o + u] = (uint32_t)U[u];
    vals[o + u] = (uint32_t)e << 5 | (uint32_t)u;
  }
}
// first[j] = first sorted block row of a node >= j
static __global__ void k_fa_starts(long long n, long long E, const uint32_t *__restrict__ keys,
                            unsigned *first) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i > E) return;
  const long long k = i < E ? (long long)keys[i] : n;
  for (long long j = i ? (long long)keys[i - 1] + 1 : 0; j <= k; j++) first[j] = (unsigned)i;
}
// Entries each row has to add; rows with more than FA_SMALL go to `large`.
constexpr int FA_SMALL = 64;         // 8 elements of 8 nodes
// A large row's table: slots and rows per block of the first attempt, and of
// the one that follows where some row has more columns (in a 2:1 balanced
// forest none has).
constexpr int FA_LARGE = 512, FA_LARGE_WARPS = 4;
constexpr int FA_HUGE = 8192, FA_HUGE_WARPS = 1;
constexpr size_t FA_SLOT_BYTES = sizeof(double) + sizeof(int) + sizeof(uint16_t);
static __global__ void k_fa_candidates(long long n, RowAsm A, unsigned *cand, unsigned *large,
                                unsigned *nlarge) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned t = 0;
  if (i < n) {
    for (unsigned p = A.srp[i]; p < A.srp[i + 1]; p++) t += (unsigned)A.nodes(A.slot[p] >> 5);
    cand[i] = t;
  }
  const unsigned m = __ballot_sync(0xffffffffu, t > FA_SMALL);
  if (m == 0u) return;
  const int lane = threadIdx.x & 31, lead = __ffs(m) - 1;
  unsigned o = 0;
  if (lane == lead) o = atomicAdd(nlarge, (unsigned)__popc(m));
  o = __shfl_sync(0xffffffffu, o, lead);
  if (t > FA_SMALL) large[o + __popc(m & ((1u << lane) - 1u))] = (unsigned)i;
}
// One row by G lanes (the whole warp calls it) over a table of `slots` slots (a
// power of two): the sorted columns and sums go to col / val, their number
// is returned; *err = FA_FULL when the row has more columns than the table.
constexpr int FA_FULL = 2;
template <int G, typename Entry>
__device__ __forceinline__ int assemble_row(const RowAsm &A, const Entry &ent, long long row,
                                            bool have, int slots, int *tcol, double *tval,
                                            uint16_t *tidx, int *col, double *val, int *err) {
  const int lane = threadIdx.x & 31, l = lane & (G - 1);
  for (int i = l; i < slots; i += G) {
    tcol[i] = -1;
    tval[i] = 0.0;
  }
  __syncwarp();
  const unsigned p0 = have ? A.srp[row] : 0, p1 = have ? A.srp[row + 1] : 0;
  unsigned steps = p1 - p0;
#pragma unroll
  for (int o = G; o < 32; o <<= 1) steps = max(steps, __shfl_xor_sync(0xffffffffu, steps, o));
  bool full = false;
  for (unsigned k = 0; k < steps; k++) {
    const bool on = p0 + k < p1;
    unsigned e = 0, u = 0;
    int K = 0;
    bool hang = false;
    if (on) {
      const unsigned s = __ldg(A.slot + p0 + k);
      e = s >> 5;
      u = s & 31u;
      hang = A.hanging(e);
      K = A.npe;
    }
    const int *U = A.conn + (long long)e * A.npe;
    const double *B = nullptr;
    if (hang) {
      const unsigned h = A.hoff[e], u0 = A.ucnt[h];
      K = (int)(A.ucnt[h + 1] - u0);
      U = A.unode + u0;
      B = A.block + A.boff[h] + u * K;
    }
    for (int v = l; v < K; v += G) {  // an element's nodes are distinct
      const int c = __ldg(U + v);
      double m;
      if (hang) {
        m = __ldg(B + v);
      } else {
        m = ent.regular(e, u ^ (unsigned)v);
      }
      unsigned h = ((unsigned)c * 0x9E3779B1u) >> 16 & (unsigned)(slots - 1);
      int it = 0;
      for (; it < slots; it++) {
        int was = *(volatile int *)(tcol + h);
        if (was == -1) was = atomicCAS(tcol + h, -1, c);
        if (was == -1 || was == c) break;
        h = (h + 1) & (unsigned)(slots - 1);
      }
      if (it == slots)
        full = true;
      else
        tval[h] = __dadd_rn(tval[h], m);
    }
    __syncwarp();
  }
  if (full) atomicExch(err, FA_FULL);
  // the taken slots, then each one's rank among their columns
  int n = 0;
  const unsigned gmask = G == 32 ? 0xffffffffu : ((1u << G) - 1u) << (lane & ~(G - 1));
  for (int i = l; i < slots; i += G) {
    const bool taken = tcol[i] >= 0;
    const unsigned m = __ballot_sync(0xffffffffu, taken) & gmask;
    if (taken) tidx[n + __popc(m & ((1u << lane) - 1u))] = (uint16_t)i;
    n += __popc(m);
  }
  __syncwarp();
  for (int i = l; i < n; i += G) {
    const int s = tidx[i], c = tcol[s];
    int r = 0;
    for (int j = 0; j < n; j++) r += tcol[tidx[j]] < c;
    col[r] = c;
    val[r] = tval[s];
  }
  return n;
}
// Rows of at most FA_SMALL entries: 8 lanes each (7-8 elements of 8 nodes
// keep every lane busy).
template <typename Entry>
__global__ void __launch_bounds__(128)
    k_fa_rows_small(long long n, RowAsm A, Entry ent, const unsigned *__restrict__ coff, int *col,
                    double *val, int *len, int *err) {
  __shared__ int tcol[16][FA_SMALL];
  __shared__ double tval[16][FA_SMALL];
  __shared__ uint16_t tidx[16][FA_SMALL];
  const int g = threadIdx.x >> 3;
  const long long row = (long long)blockIdx.x * 16 + g;
  const unsigned o = row < n ? coff[row] : 0, o1 = row < n ? coff[row + 1] : 0;
  const bool have = row < n && o1 - o <= FA_SMALL;
  const int m = assemble_row<8>(A, ent, row, have, FA_SMALL, tcol[g], tval[g], tidx[g], col + o,
                                val + o, err);
  if (have && (threadIdx.x & 7) == 0) len[row] = m;
}
// The others: a warp each, `warps` rows per block.
template <typename Entry>
__global__ void __launch_bounds__(FA_LARGE_WARPS * 32)
    k_fa_rows_large(const unsigned *__restrict__ nlarge, const unsigned *__restrict__ list,
                    int slots, int warps, RowAsm A, Entry ent,
                    const unsigned *__restrict__ coff, int *col, double *val, int *len,
                    int *err) {
  extern __shared__ __align__(16) unsigned char fa_smem[];
  const int w = threadIdx.x >> 5;
  double *tval = (double *)fa_smem + (size_t)w * slots;
  int *tcol = (int *)((double *)fa_smem + (size_t)warps * slots) + (size_t)w * slots;
  uint16_t *tidx = (uint16_t *)((int *)((double *)fa_smem + (size_t)warps * slots) +
                                (size_t)warps * slots) + (size_t)w * slots;
  const unsigned m = *nlarge;
  for (unsigned i = blockIdx.x * warps + w; i < m; i += gridDim.x * warps) {
    const long long row = list[i];
    const unsigned o = coff[row];
    const int c =
        assemble_row<32>(A, ent, row, true, slots, tcol, tval, tidx, col + o, val + o, err);
    if ((threadIdx.x & 31) == 0) len[row] = c;
    __syncwarp();
  }
}
// Rows from their places to CSR, 8 lanes per row.
static __global__ void k_fa_compact(long long n, const unsigned *__restrict__ coff,
                             const int *__restrict__ rp, const int *__restrict__ col,
                             const double *__restrict__ val, int *ocol, double *oval) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long row = t >> 3;
  if (row >= n) return;
  const unsigned o = coff[row];
  const int p0 = rp[row], m = rp[row + 1] - p0;
  for (int k = (int)(t & 7); k < m; k += 8) {
    ocol[p0 + k] = col[o + k];
    oval[p0 + k] = val[o + k];
  }
}

// The n x n matrix of the elements' entries as CSR (columns ascending).  `all`:
// every element stores its block.  Anything but ASM_DONE leaves nothing in the
// outputs.
enum AsmResult {
  ASM_DONE,
  ASM_NODES,    // an element touches more than FMAXK nodes
  ASM_ENTRIES,  // 2^32 element-matrix entries or more
  ASM_PLACES    // too many elements for their 32-bit places, or a row of more
                // than FA_HUGE columns: assemble_entries has no such limit
};
template <typename Entry>
inline AsmResult assemble_rows(const ElemCtx &c, const Entry &ent, long long n, long long ne, bool all,
                          DBuf<int> &rowptr, DBuf<int> &colidx, DBuf<double> &vals,
                          long long &nnz, cudaStream_t s) {
  if (ne >= (1LL << 27)) return ASM_PLACES;
  const int cb = bits_for(n + 1);
  RowAsm A{};
  A.conn = c.conn;
  A.npe = c.npe;
  // hanging elements: their distinct nodes and blocks
  DBuf<unsigned> hoff(ne + 1, s);
  launch(k_fa_hanging, blocks_for(ne, 256), 256, 0, s, ne, c.npe, c.conn, (int)all, hoff.p);
  exclusive_scan<unsigned>(hoff.p, hoff.p, ne, s);
  const long long nh = read_scalar(hoff.p + ne, s);
  DBuf<unsigned> list(nh + 1, s), ucnt(nh + 1, s), boff(nh + 1, s);
  launch(k_fa_list, blocks_for(ne, 256), 256, 0, s, ne, (const unsigned *)hoff.p, list.p);
  DBuf<unsigned long long> total(1, s);
  total.zero();
  launch(k_fa_count<Entry>, blocks_for(nh, 128), 128, 0, s, nh, c, ent, (const unsigned *)list.p,
         ucnt.p, boff.p, total.p);
  exclusive_scan<unsigned>(ucnt.p, ucnt.p, nh, s);
  exclusive_scan<unsigned>(boff.p, boff.p, nh, s);
  const unsigned *tw = (const unsigned *)total.p;  // low word first
  const unsigned *hp[5] = {ucnt.p + nh, boff.p + nh, tw, tw + 1, (const unsigned *)c.err};
  unsigned hv[5];
  read_scalars(hp, hv, s);
  // rows, each at its number of entries before equal columns are added
  const long long E = (ne - nh) * c.npe * c.npe + ((long long)hv[3] << 32 | hv[2]);
  if (hv[4]) return ASM_NODES;
  if (E >= (1LL << 32)) return ASM_ENTRIES;
  DBuf<int> unode((size_t)hv[0] + 1, s);
  DBuf<double> block((size_t)hv[1] + 1, s);
  launch(k_fa_blocks<Entry>, blocks_for(nh, 64), 64, 0, s, nh, c, ent, (const unsigned *)list.p,
         (const unsigned *)ucnt.p, (const unsigned *)boff.p, unode.p, block.p);
  list.release();
  A.hoff = hoff.p;
  A.ucnt = ucnt.p;
  A.boff = boff.p;
  A.unode = unode.p;
  A.block = block.p;
  // block rows sorted by node, elements ascending
  DBuf<unsigned> soff(ne + 1, s);
  launch(k_fa_slot_count, blocks_for(ne, 256), 256, 0, s, ne, A, soff.p);
  exclusive_scan<unsigned>(soff.p, soff.p, ne, s);
  const long long ns = (long long)(ne - nh) * c.npe + hv[0];
  DBuf<uint32_t> skey(ns, s), slot(ns, s);
  launch(k_fa_slots, blocks_for(ne, 256), 256, 0, s, ne, A, (const unsigned *)soff.p, skey.p,
         slot.p);
  soff.release();
  radix_sort(skey, &slot, ns, cb, s);
  DBuf<unsigned> srp(n + 1, s);
  launch(k_fa_starts, blocks_for(ns + 1, 256), 256, 0, s, n, ns, (const uint32_t *)skey.p, srp.p);
  skey.release();
  A.srp = srp.p;
  A.slot = slot.p;
  DBuf<unsigned> coff(n + 1, s), large(n + 1, s), nlarge(1, s);
  nlarge.zero();
  launch(k_fa_candidates, blocks_for(n, 256), 256, 0, s, n, A, coff.p, large.p, nlarge.p);
  exclusive_scan<unsigned>(coff.p, coff.p, n, s);
  DBuf<int> col(E + 1, s);
  DBuf<double> val(E + 1, s);
  rowptr.alloc(n + 1, s);
  DBuf<int> ncol(n + 1, s);
  launch(k_fa_rows_small<Entry>, blocks_for(n, 16), 128, 0, s, n, A, ent,
         (const unsigned *)coff.p, col.p, val.p, ncol.p, c.err);
  auto rows = [&](int slots, int warps) {
    const size_t smem = FA_SLOT_BYTES * slots * warps;
    TMRG_CUDA(cudaFuncSetAttribute(k_fa_rows_large<Entry>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)(FA_SLOT_BYTES * FA_HUGE * FA_HUGE_WARPS)));
    launch(k_fa_rows_large<Entry>, std::min(blocks_for(n, warps), 152u * 8), warps * 32, smem, s,
           (const unsigned *)nlarge.p, (const unsigned *)large.p, slots, warps, A, ent,
           (const unsigned *)coff.p, col.p, val.p, ncol.p, c.err);
    exclusive_scan<int>(ncol.p, rowptr.p, n, s);
    const int *pv[2] = {rowptr.p + n, c.err};
    int hv2[2];
    read_scalars(pv, hv2, s);
    nnz = hv2[0];
    return hv2[1];
  };
  int err = rows(FA_LARGE, FA_LARGE_WARPS);
  if (err == FA_FULL) {
    TMRG_CUDA(cudaMemsetAsync(c.err, 0, sizeof(int), s));
    err = rows(FA_HUGE, FA_HUGE_WARPS);
  }
  if (err) {
    rowptr.release();
    return err == FA_FULL ? ASM_PLACES : ASM_NODES;
  }
  colidx.alloc(nnz + 1, s);
  vals.alloc(nnz + 1, s);
  launch(k_fa_compact, blocks_for(n * 8, 256), 256, 0, s, n, (const unsigned *)coff.p,
         (const int *)rowptr.p, (const int *)col.p, (const double *)val.p, colidx.p,
         vals.p);
  return ASM_DONE;
}

// The block entries of every element as records (row << cb | column, place,
// value) for a sort, and their number in E.
template <typename Entry>
__global__ void k_fa_entry_count(long long ne, ElemCtx c, Entry ent, long long *cnt) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  int U[FMAXK];
  const int K = element_block(c, ent, e, U, nullptr);
  cnt[e] = K * K;
}
template <typename Entry>
__global__ void __launch_bounds__(64)
    k_fa_entries(long long ne, ElemCtx c, Entry ent, int cb, const long long *__restrict__ off,
                 uint64_t *keys, uint32_t *perm, double *vals) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  int U[FMAXK];
  double L[FMAXK][FMAXK];
  const int K = element_block(c, ent, e, U, L);
  long long o = off[e];
  for (int u = 0; u < K; u++)
    for (int v = 0; v < K; v++, o++) {
      keys[o] = (uint64_t)(uint32_t)U[u] << cb | (uint64_t)(uint32_t)U[v];
      perm[o] = (uint32_t)o;
      vals[o] = L[u][v];
    }
}
template <typename Entry>
inline AsmResult assemble_entries(const ElemCtx &c, const Entry &ent, long long ne, int cb,
                                  DBuf<uint64_t> &keys, DBuf<uint32_t> &perm, DBuf<double> &vals,
                                  long long &E, cudaStream_t s) {
  DBuf<long long> cnt(ne + 1, s);
  launch(k_fa_entry_count<Entry>, blocks_for(ne, 128), 128, 0, s, ne, c, ent, cnt.p);
  exclusive_scan<long long>(cnt.p, cnt.p, ne, s);
  const unsigned *w = (const unsigned *)(cnt.p + ne);  // low word first
  const unsigned *pv[3] = {w, w + 1, (const unsigned *)c.err};
  unsigned hv[3];
  read_scalars(pv, hv, s);
  E = (long long)hv[1] << 32 | hv[0];
  if (hv[2]) return ASM_NODES;
  if (E >= (1LL << 32)) return ASM_ENTRIES;
  keys.alloc(E, s);
  perm.alloc(E, s);
  vals.alloc(E, s);
  launch(k_fa_entries<Entry>, blocks_for(ne, 64), 64, 0, s, ne, c, ent, cb,
         (const long long *)cnt.p, keys.p, perm.p, vals.p);
  return ASM_DONE;
}

}  // namespace tmrg
