// Matrix density filter (TMRMatrixFilter.cpp:30-235) on the GPU.
//
// Setup: the consistent mass matrix M of the trilinear (octree) or
// bilinear (quadtree) elements of an order-2 forest, with dependent nodes
// condensed onto the independent nodes they interpolate.  Each element's
// matrix, expanded through the dependent-node weights, is a dense block
// over its distinct independent nodes; a row of M adds the block rows of
// the elements around its node in element order (assemble_rows).  Orders
// 3 and 4 sort the blocks' entries by (row, column) instead.  Then
// D = M 1, Ainv = 1/(1 + r^2/D^(2/3)), B = Ainv r^2/(D^(2/3) D) (in 2-D
// Ainv = 1/(1 + r^2/D), B = Ainv r^2/(D D)) and Tinv = 1/(F~ 1).
//
// Apply: Horner's recurrence out = B.(M out) + t1 (forward) or
// out = M(B.out) + t1 (transpose), one fused kernel per term over up to four
// of the interleaved design components, so M is read once per term.
#include <string.h>

#include <algorithm>
#include <mutex>
#include <string>

#include "tmrg_quad.h"
#include "tmrg_rowasm.cuh"
#include "tmrg_tree.cuh"
#include "tmrg_tsell.cuh"

namespace tmrg {

struct FilterCtx {
  const int *conn;
  const int *dptr, *dconn;
  const double *dw;
  double block_len;
  const int16_t *lev;
  int *err;
  int npe, dim;  // 8 and 3 (octree) or 4 and 2 (quadtree)
};

// The entries of M (assemble_rows): the exact mass of the linear element
// (corner a = i + 2j + 4k), the 1-D entries s/3 and s/6 multiplied over the
// directions, nd of which differ.  A side is block_len over a power of two,
// so an element's entry is the unit block's with a smaller exponent.
struct MassEntry {
  double block_len;
  const int16_t *lev;
  int dim;
  unsigned long long m0;  // bits of the unit block's entry, nd = 0
  __device__ __forceinline__ double direct(long long e, int a, int b) const {
    const double side = block_len / (double)(1 << lev[e]);
    const double s2 = __dmul_rn(side, side);
    const int nd = __popc((unsigned)(a ^ b));
    return dim == 3 ? __ddiv_rn(__dmul_rn(s2, side), 27.0 * (double)(1 << nd))
                    : __ddiv_rn(s2, 9.0 * (double)(1 << nd));
  }
  __device__ __forceinline__ double regular(unsigned e, unsigned x) const {
    return __longlong_as_double((long long)(
        m0 - ((unsigned long long)(dim * __ldg(lev + e) + __popc(x)) << 52)));
  }
};

// Sum each run of equal (row, col) keys in element order.
__global__ void k_fe_reduce(long long E, const uint64_t *__restrict__ keys,
                            const uint32_t *__restrict__ perm,
                            const double *__restrict__ v,
                            const unsigned *__restrict__ pos, int cb,
                            int *cols, double *out, int *rowcnt) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= E || pos[i + 1] == pos[i]) return;
  uint64_t k = keys[i];
  double s = v[perm[i]];
  for (long long j = i + 1; j < E && keys[j] == k; j++) s = __dadd_rn(s, v[perm[j]]);
  unsigned o = pos[i];
  cols[o] = (int)(k & ((1ULL << cb) - 1));
  out[o] = s;
  atomicAdd(rowcnt + (k >> cb), 1);
}
__global__ void k_fe_first(long long E, const uint64_t *__restrict__ keys,
                           unsigned *flag) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < E) flag[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1u : 0u;
}

// ---------------------------------------------------------------------
// Orders 3 and 4 (the quadratic and cubic Bernstein hexahedra the
// reference's matrix creator picks, TMRMatrixCreator.h:80-85): one warp per
// element.  The element's expansion list (each node, dependent nodes
// through their CSR rows) is staged in shared memory; its distinct
// independent nodes U are numbered in first-appearance order; then
//   T[a][v] = sum over entries (b, w) with node U[v] of M_e[a][b] w
// (entries in list order) and the merged block row u is
//   L[u][v] = sum over entries (a, w) with node U[u] of w T[a][v]
// (entries in list order), written as K x K (row, column, value) triplets
// that the common sort-and-sum pass adds up in element order.  M_e[a][b] =
// ((s^3 m[ia][ib]) m[ja][jb]) m[ka][kb] with m the 1-D Bernstein mass on
// [0, 1] (exact on axis-aligned cubes).  The sums run in a different
// order than the per-pair loop of the order-2 kernel; the results agree to
// rounding.
struct FGen {
  int o, npe;
  int cap;    // staged entries per warp
  int kcap;   // distinct nodes per element
  int tcols;  // columns of T in shared memory (0 in the count pass)
  double m1[4][4];
};
constexpr int FG_WARPS = 2;

// Shared-memory layout of one warp (bytes, 8-aligned).
struct FGLayout {
  size_t node, w, a, u, ord, U, ust, T, total;
};
__host__ __device__ inline FGLayout fg_layout(const FGen &g) {
  FGLayout L;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    size_t r = o;
    o += (bytes + 7) & ~(size_t)7;
    return r;
  };
  L.w = take(sizeof(double) * g.cap);
  L.T = take(sizeof(double) * (size_t)g.npe * g.tcols);
  L.node = take(sizeof(int) * g.cap);
  L.U = take(sizeof(int) * g.kcap);
  L.u = take(sizeof(uint16_t) * g.cap);
  L.ord = take(sizeof(uint16_t) * g.cap);
  L.ust = take(sizeof(uint16_t) * (g.kcap + 1));
  L.a = take(g.cap);
  L.total = o;
  return L;
}

// Expansion list and distinct nodes of element e; returns K (0 with the
// error flag set when the element outgrows the stage).
__device__ int fg_stage(const FilterCtx &c, const FGen &g, long long e, unsigned char *sm,
                        const FGLayout &L) {
  const int lane = threadIdx.x & 31;
  int *s_node = (int *)(sm + L.node);
  double *s_w = (double *)(sm + L.w);
  uint8_t *s_a = (uint8_t *)(sm + L.a);
  uint16_t *s_u = (uint16_t *)(sm + L.u), *s_first = (uint16_t *)(sm + L.ord);
  int *s_U = (int *)(sm + L.U);
  const int *ec = c.conn + e * g.npe;
  int total = 0;
  for (int a0 = 0; a0 < g.npe; a0 += 32) {
    const int a = a0 + lane;
    int gv = 0, len = 0, d0 = 0;
    if (a < g.npe) {
      gv = __ldg(ec + a);
      if (gv >= 0) {
        len = 1;
      } else {
        d0 = __ldg(c.dptr - gv - 1);
        len = __ldg(c.dptr - gv) - d0;
      }
    }
    int incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const int off = total + incl - len;
    if (off + len <= g.cap) {
      for (int p = 0; p < len; p++) {
        s_node[off + p] = gv >= 0 ? gv : __ldg(c.dconn + d0 + p);
        s_w[off + p] = gv >= 0 ? 1.0 : __ldg(c.dw + d0 + p);
        s_a[off + p] = (uint8_t)a;
      }
    }
    total += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (total > g.cap) {
    if (lane == 0) atomicExch(c.err, 1);
    return 0;
  }
  __syncwarp();
  // first occurrence of each entry's node
  for (int i = lane; i < total; i += 32) {
    const int nd = s_node[i];
    int j = 0;
    while (s_node[j] != nd) j++;
    s_first[i] = (uint16_t)j;
  }
  __syncwarp();
  int K = 0;
  for (int i0 = 0; i0 < total; i0 += 32) {
    const int i = i0 + lane;
    const bool first = i < total && s_first[i] == i;
    const unsigned m = __ballot_sync(0xffffffffu, first);
    if (first) {
      const int k = K + __popc(m & ((1u << lane) - 1u));
      if (k < g.kcap) s_U[k] = s_node[i];
      s_u[i] = (uint16_t)k;
    }
    K += __popc(m);
  }
  if (K > g.kcap) {
    if (lane == 0) atomicExch(c.err, 1);
    return 0;
  }
  __syncwarp();
  for (int i = lane; i < total; i += 32)
    if (s_first[i] != i) s_u[i] = s_u[s_first[i]];
  __syncwarp();
  return K | (total << 16);
}

// Largest expansion list of an element (sizes the stage).
__global__ void k_fe_gen_emax(long long ne, FilterCtx c, int npe, int *emax) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  const int *ec = c.conn + e * npe;
  int t = 0;
  for (int a = 0; a < npe; a++) {
    const int gv = __ldg(ec + a);
    t += gv >= 0 ? 1 : __ldg(c.dptr - gv) - __ldg(c.dptr - gv - 1);
  }
  atomicMax(emax, t);
}
// Pass 0: K^2 triplets per element (and the largest K).
__global__ void __launch_bounds__(FG_WARPS * 32)
    k_fe_gen_count(long long ne, FilterCtx c, FGen g, long long *cnt, int *kmax) {
  extern __shared__ __align__(16) unsigned char fg_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long e = (long long)blockIdx.x * FG_WARPS + warp;
  if (e >= ne) return;
  const FGLayout L = fg_layout(g);
  const int r = fg_stage(c, g, e, fg_smem + warp * L.total, L);
  const int K = r & 0xffff;
  if (lane == 0) {
    cnt[e] = (long long)K * K;
    atomicMax(kmax, K);
  }
}
// Pass 1: the triplets at offs[e].
__global__ void __launch_bounds__(FG_WARPS * 32)
    k_fe_gen_write(long long ne, FilterCtx c, FGen g, int cb, const long long *__restrict__ offs,
                   uint64_t *keys, uint32_t *perm, double *vals) {
  extern __shared__ __align__(16) unsigned char fg_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long e = (long long)blockIdx.x * FG_WARPS + warp;
  if (e >= ne) return;
  const FGLayout L = fg_layout(g);
  unsigned char *sm = fg_smem + warp * L.total;
  const int r = fg_stage(c, g, e, sm, L);
  const int K = r & 0xffff, total = r >> 16;
  if (K == 0) return;
  const double *s_w = (const double *)(sm + L.w);
  const uint8_t *s_a = (const uint8_t *)(sm + L.a);
  const uint16_t *s_u = (const uint16_t *)(sm + L.u);
  uint16_t *s_ord = (uint16_t *)(sm + L.ord), *s_ust = (uint16_t *)(sm + L.ust);
  const int *s_U = (const int *)(sm + L.U);
  double *T = (double *)(sm + L.T);
  const int o = g.o, npe = g.npe;
  const double side = c.block_len / (double)(1 << c.lev[e]);
  const double s3 = __dmul_rn(__dmul_rn(side, side), side);
  // T = M_e W over the K distinct nodes; lanes own rows a
  for (int a = lane; a < npe; a += 32)
    for (int v = 0; v < K; v++) T[a * K + v] = 0.0;
  for (int i = 0; i < total; i++) {
    const int b = s_a[i], v = s_u[i];
    const double wb = s_w[i];
    const int ib = b % o, jb = (b / o) % o, kb = b / (o * o);
    for (int a = lane; a < npe; a += 32) {
      const int ia = a % o, ja = (a / o) % o, ka = a / (o * o);
      const double mab =
          __dmul_rn(__dmul_rn(__dmul_rn(s3, g.m1[ia][ib]), g.m1[ja][jb]), g.m1[ka][kb]);
      T[a * K + v] = __fma_rn(mab, wb, T[a * K + v]);
    }
  }
  // entries ordered by distinct node (stable), and each node's first slot
  for (int i = lane; i < total; i += 32) {
    const int ui = s_u[i];
    int pos = 0;
    for (int j = 0; j < total; j++) {
      const int uj = s_u[j];
      pos += (uj < ui) || (uj == ui && j < i);
    }
    s_ord[pos] = (uint16_t)i;
  }
  __syncwarp();
  for (int p = lane; p < total; p += 32) {
    const int up = s_u[s_ord[p]];
    if (p == 0 || s_u[s_ord[p - 1]] != up) s_ust[up] = (uint16_t)p;
  }
  if (lane == 0) s_ust[K] = (uint16_t)total;
  __syncwarp();
  // row u of the merged block: lanes own columns v
  const long long base = offs[e];
  for (int u = 0; u < K; u++) {
    const int p0 = s_ust[u], p1 = s_ust[u + 1];
    const uint64_t rk = (uint64_t)(uint32_t)s_U[u] << cb;
    for (int v = lane; v < K; v += 32) {
      double acc = 0.0;
      for (int p = p0; p < p1; p++) {
        const int i = s_ord[p];
        acc = __fma_rn(s_w[i], T[s_a[i] * K + v], acc);
      }
      const long long q = base + (long long)u * K + v;
      keys[q] = rk | (uint64_t)(uint32_t)s_U[v];
      perm[q] = (uint32_t)q;
      vals[q] = acc;
    }
  }
}

// D, Ainv, B (TMRMatrixFilter.cpp:121-147).
__global__ void k_fe_scalings(long long n, int dim, const int *__restrict__ rp,
                              const double *__restrict__ vals, double r,
                              double *Ainv, double *B) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double D = 0.0;
  for (int p = rp[i]; p < rp[i + 1]; p++) D = __dadd_rn(D, vals[p]);
  if (D == 0.0) {
    Ainv[i] = 1.0;
    B[i] = 0.0;
  } else if (dim == 2) {
    double rr = __dmul_rn(r, r);
    double a = __ddiv_rn(1.0, __dadd_rn(1.0, __ddiv_rn(rr, D)));
    Ainv[i] = a;
    B[i] = __ddiv_rn(__dmul_rn(__dmul_rn(a, r), r), __dmul_rn(D, D));
  } else {
    double t = pow(D, 2.0 / 3.0);
    double rr = __dmul_rn(r, r);
    double a = __ddiv_rn(1.0, __dadd_rn(1.0, __ddiv_rn(rr, t)));
    Ainv[i] = a;
    B[i] = __ddiv_rn(__dmul_rn(__dmul_rn(a, r), r), __dmul_rn(t, D));
  }
}
__global__ void k_fe_tinv(long long n, const double *__restrict__ y, double *T) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) T[i] = (y[i] != 0.0) ? __ddiv_rn(1.0, y[i]) : 0.0;
}
__global__ void k_fe_ones(long long n, double *a, double *b) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = b[i] = 1.0;
}
template <typename T>
__global__ void k_to_f32(long long n, const double *__restrict__ a, T *b) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = (T)a[i];
}

// ---------------------------------------------------------------------
__device__ __forceinline__ double fmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double fadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
// The Horner terms accumulate M x with fused multiply-adds: half the FP64
// instructions (a scarce pipe on GB300) and one rounding per term.
__device__ __forceinline__ double ffma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float ffma(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// four values from shared memory, 16 bytes a load
__device__ __forceinline__ void lds4(const float *p, float (&v)[4]) {
  const float4 q = *(const float4 *)p;
  v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
}
__device__ __forceinline__ void lds4(const double *p, double (&v)[4]) {
  const double2 a = ((const double2 *)p)[0], b = ((const double2 *)p)[1];
  v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
}

// t1 = s . in ; returns t1 (the first Horner iterate).
template <typename T>
__global__ void k_fe_scale(long long n, int vpn, const T *__restrict__ s,
                           const T *__restrict__ in, T *out) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * vpn) return;
  out[i] = fmul(s[i / vpn], in[i]);
}

// One Horner term over all components:
//   forward:   y = B.(M x) + t1
//   transpose: y = M(B.x) + t1
// then y *= post (the final Tinv or Ainv) when post != nullptr.
// ---------------------------------------------------------------------
// Sliced-ELL copy of M (see Filter): per slice the longest row length,
// then per position its row's entries at soff[slice] + 32 k + lane (CSR
// order; the tail of a shorter row holds column = row, value 0, never
// read).
__global__ void k_sell_len(long long npos, long long n, const int *__restrict__ perm,
                           const int *__restrict__ rp, int *srl, long long *ssz) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npos) return;
  int len = 0;
  if (p < n) {
    const int row = perm[p];
    len = rp[row + 1] - rp[row];
  }
  srl[p] = len;
  // slice length: the longest row of the 32 positions (one warp)
  int m = len;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((p & 31) == 0) ssz[p >> 5] = 32LL * m;
}
template <typename T>
__global__ void k_sell_fill(long long npos, long long n, const int *__restrict__ perm,
                            const int *__restrict__ rp, const int *__restrict__ cols,
                            const T *__restrict__ vals, const long long *__restrict__ soff,
                            int *scol, T *sval) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npos) return;
  const long long sl = p >> 5;
  const int L = (int)((soff[sl + 1] - soff[sl]) >> 5);
  const long long base = soff[sl] + (p & 31);
  const int row = p < n ? perm[p] : 0;
  const int p0 = p < n ? rp[row] : 0, len = p < n ? rp[row + 1] - p0 : 0;
  for (int k = 0; k < L; k++) {
    scol[base + 32LL * k] = k < len ? cols[p0 + k] : row;
    sval[base + 32LL * k] = k < len ? vals[p0 + k] : T(0);
  }
}

// One Horner term on the sliced copy: thread p <-> row sperm[p], its
// entries in CSR order (the same FMA sequence as k_fe_step).
template <typename T, int VPN, bool TR>
__global__ void __launch_bounds__(256)
    k_fe_sell(long long n, int vpn_rt, const int *__restrict__ perm, const int *__restrict__ srl,
              const long long *__restrict__ soff, const int *__restrict__ scol,
              const T *__restrict__ sval, const T *__restrict__ B, const T *__restrict__ t1,
              const T *__restrict__ x, T *__restrict__ y, const T *__restrict__ post) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const long long i = perm[p];
  const int len = srl[p];
  const long long base = soff[p >> 5] + (p & 31);
  const int vpn = VPN > 0 ? VPN : vpn_rt;
  T acc[VPN > 0 ? VPN : 4];
  for (int c0 = 0; c0 < vpn; c0 += (VPN > 0 ? VPN : 4)) {
    const int nc = (VPN > 0) ? VPN : min(4, vpn - c0);
#pragma unroll
    for (int v = 0; v < (VPN > 0 ? VPN : 4); v++) acc[v] = T(0);
#pragma unroll 4
    for (int k = 0; k < len; k++) {
      const int j = __ldg(scol + base + 32LL * k);
      const T m = __ldg(sval + base + 32LL * k);
      const T bj = TR ? __ldg(B + j) : T(1);
#pragma unroll
      for (int v = 0; v < (VPN > 0 ? VPN : 4); v++) {
        if (v < nc) {
          T xv = __ldg(x + (long long)j * vpn + c0 + v);
          if (TR) xv = fmul(bj, xv);
          acc[v] = ffma(m, xv, acc[v]);
        }
      }
    }
    const T bi = TR ? T(1) : B[i];
    const T pi = post ? post[i] : T(1);
#pragma unroll
    for (int v = 0; v < (VPN > 0 ? VPN : 4); v++) {
      if (v < nc) {
        const long long o = i * vpn + c0 + v;
        T r = TR ? fadd(acc[v], t1[o]) : fadd(fmul(bi, acc[v]), t1[o]);
        if (post) r = fmul(r, pi);
        y[o] = r;
      }
    }
  }
}

// The same term on the tiled copy (TSell): a block loads its tile's distinct
// input values into shared memory, the transpose scaled by B there (once per
// value instead of once per entry), and its rows read them by 16-bit places.
// FIRST: the term's input is pre.in, formed as it is loaded, and t1 = pre.in
// is written for the terms that follow.  The same multiplies and FMAs per
// row, in CSR order, as k_fe_sell after k_fe_scale: the same bits.  VPN
// components a time (of vpn, from c0).  Three components sit three values
// apart: consecutive places meet no bank twice (padded to four, a 16-byte
// load each, the FP32 terms took 127 us instead of 110).
//
// Measured with 2.56M rows of 27 and three components, against sliced ELL
// with 32-bit columns and gathers through L1: FP64 forward 336 -> 342 us a
// term, transpose 645 -> 357 us, both at the FP64 pipe's 0.6 T FMA/s (the
// transpose no longer multiplies every entry's input by B); FP32 120 -> 109 and
// 144 -> 110 us, 3.8 TB/s, bound by the shared-memory reads (3 per entry).
template <typename T, int VPN, bool TR, bool FIRST>
__global__ void __launch_bounds__(TS_ROWS)
    k_fe_tile(TSellView M, int vpn, int c0, const T *__restrict__ val, const T *__restrict__ B,
              const T *__restrict__ pre, T *t1, const T *__restrict__ x, T *__restrict__ y,
              const T *__restrict__ post) {
  extern __shared__ __align__(16) unsigned char fe_smem[];
  T *sx = (T *)fe_smem;
  const int t = threadIdx.x;
  const unsigned u0 = M.uoff[blockIdx.x];
  const int m = (int)(M.uoff[blockIdx.x + 1] - u0);
  for (int i = t; i < m; i += TS_ROWS) {
    const long long j = __ldg(M.ucol + u0 + i);
    const T sc = FIRST ? __ldg(pre + j) : T(1);
    const T bj = TR ? __ldg(B + j) : T(1);
    const T *xj = x + j * vpn + c0;
#pragma unroll
    for (int v = 0; v < VPN; v++) {
      T xv = __ldg(xj + v);
      if (FIRST) xv = fmul(sc, xv);
      if (TR) xv = fmul(bj, xv);
      sx[i * VPN + v] = xv;
    }
  }
  __syncthreads();
  const long long q = (long long)blockIdx.x * TS_ROWS + t;
  const int i = M.row[q];
  if (i < 0) return;
  const int len = M.len[q];
  const long long base = (long long)M.soff[q >> 5] * 32 + (t & 31);
  const uint16_t *ip = M.idx + base;
  const T *vp = val + base;
  T acc[VPN];
#pragma unroll
  for (int v = 0; v < VPN; v++) acc[v] = T(0);
#pragma unroll 4
  for (int k = 0; k < len; k++) {
    const T *xv = sx + (int)__ldg(ip + 32LL * k) * VPN;
    const T mv = __ldg(vp + 32LL * k);
    if constexpr (VPN == 4) {
      T xr[4];
      lds4(xv, xr);
#pragma unroll
      for (int v = 0; v < VPN; v++) acc[v] = ffma(mv, xr[v], acc[v]);
    } else {
#pragma unroll
      for (int v = 0; v < VPN; v++) acc[v] = ffma(mv, xv[v], acc[v]);
    }
  }
  const T bi = TR ? T(1) : B[i];
  const T si = FIRST ? pre[i] : T(1);
  const T pi = post ? post[i] : T(1);
#pragma unroll
  for (int v = 0; v < VPN; v++) {
    const long long o = (long long)i * vpn + c0 + v;
    T tv;
    if (FIRST) {
      tv = fmul(si, __ldg(x + o));
      t1[o] = tv;
    } else {
      tv = t1[o];
    }
    T r = TR ? fadd(acc[v], tv) : fadd(fmul(bi, acc[v]), tv);
    if (post) r = fmul(r, pi);
    y[o] = r;
  }
}

template <typename T>
static const T *sell_vals(const Filter &F);
template <>
const double *sell_vals<double>(const Filter &F) {
  return F.sval.p;
}
template <>
const float *sell_vals<float>(const Filter &F) {
  return F.sval32.p;
}

// One Horner term (all vpn components) on the sliced copy of M.
template <typename T, bool TR>
static void launch_sell(const Filter &F, int vpn, const T *B, const T *t1, const T *x, T *y,
                        const T *post, cudaStream_t s) {
  const long long n = F.n;
  const unsigned g = blocks_for(n, 256);
  // compulsory traffic of one term: M (value + column), B, t1, one read of
  // x and one write of y (all vpn components)
  prof_bytes((long long)(sizeof(T) + 4) * F.nnz + 4 * (n + 1) + (long long)sizeof(T) * n +
             3LL * sizeof(T) * n * vpn + (post ? (long long)sizeof(T) * n : 0));
  prof_flops(2LL * vpn * F.nnz);
  const T *sv = sell_vals<T>(F);
#define TMRG_SELL(V)                                                                         \
  launch((k_fe_sell<T, V, TR>), g, 256, 0, s, n, vpn, (const int *)F.sperm.p,               \
         (const int *)F.srl.p, (const long long *)F.soff.p, (const int *)F.scol.p, sv, B, t1, \
         x, y, post)
  switch (vpn) {
    case 1: TMRG_SELL(1); break;
    case 2: TMRG_SELL(2); break;
    case 3: TMRG_SELL(3); break;
    case 4: TMRG_SELL(4); break;
    default: TMRG_SELL(0);
  }
#undef TMRG_SELL
}

template <typename T>
static const T *tile_vals(const Filter &F);
template <>
const double *tile_vals<double>(const Filter &F) {
  return F.tval.p;
}
template <>
const float *tile_vals<float>(const Filter &F) {
  return F.tval32.p;
}
// One Horner term on the tiled copy, VPN components from c0.
template <typename T, int VPN>
static void launch_tile_term(const Filter &F, bool tr, bool first, int vpn, int c0, const T *B,
                             const T *pre, T *t1, const T *x, T *y, const T *post,
                             cudaStream_t s) {
  const size_t smem = sizeof(T) * VPN * (size_t)F.tiled.maxu;
  const unsigned g = (unsigned)F.tiled.tiles;
  const TSellView M = F.tiled.view();
  // compulsory traffic of one term: M (value + place), the input, t1 and y
  // once, B
  prof_bytes((long long)(sizeof(T) + 2) * F.nnz + (long long)sizeof(T) * F.n * (3LL * VPN + 1));
  prof_flops(2LL * VPN * F.nnz);
  // the limit is the kernel's, for all threads: that of the largest tile
#define TMRG_TILE(TR, FIRST)                                                                 \
  do {                                                                                       \
    if (smem > 48 * 1024)                                                                    \
      TMRG_CUDA(cudaFuncSetAttribute(k_fe_tile<T, VPN, TR, FIRST>,                           \
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,            \
                                     (int)(sizeof(T) * VPN * TS_SIZES[1].cols)));            \
    launch((k_fe_tile<T, VPN, TR, FIRST>), g, TS_ROWS, smem, s, M, vpn, c0, tile_vals<T>(F), B, \
           pre, t1, x, y, post);                                                             \
  } while (0)
  if (tr) {
    if (first) TMRG_TILE(true, true); else TMRG_TILE(true, false);
  } else {
    if (first) TMRG_TILE(false, true); else TMRG_TILE(false, false);
  }
#undef TMRG_TILE
}
// applyFilter / applyTranspose on the tiled copy (F.N > 0); t1 and tmp hold
// n * vpn values.  Where `in` and `out` overlap t1 is formed before any term
// writes.
template <typename T>
static void horner_tiled(const Filter &F, bool tr, int vpn, const T *in, T *out, T *t1, T *tmp,
                         const T *Ainv, const T *B, const T *Tinv, cudaStream_t s) {
  const long long len = F.n * vpn;
  const T *pre = tr ? Tinv : Ainv, *post = tr ? Ainv : Tinv;
  const T *x = in;
  bool first = true;
  if (overlap(in, sizeof(T) * len, out, sizeof(T) * len)) {
    prof_bytes(2LL * sizeof(T) * len + (long long)sizeof(T) * F.n);
    launch(k_fe_scale<T>, blocks_for(len, 256), 256, 0, s, F.n, vpn, pre, in, t1);
    x = t1;
    first = false;
  }
  for (int k = 0; k < F.N; k++, first = false) {
    const T *last = k == F.N - 1 ? post : nullptr;
    T *y = ((F.N - 1 - k) % 2 == 0) ? out : tmp;
    for (int c0 = 0; c0 < vpn; c0 += 4) {
      const int nc = std::min(4, vpn - c0);
      if (nc == 1)
        launch_tile_term<T, 1>(F, tr, first, vpn, c0, B, pre, t1, x, y, last, s);
      else if (nc == 2)
        launch_tile_term<T, 2>(F, tr, first, vpn, c0, B, pre, t1, x, y, last, s);
      else if (nc == 3)
        launch_tile_term<T, 3>(F, tr, first, vpn, c0, B, pre, t1, x, y, last, s);
      else
        launch_tile_term<T, 4>(F, tr, first, vpn, c0, B, pre, t1, x, y, last, s);
    }
    x = y;
  }
}

template <typename T>
static void horner_generic(Filter &F, bool tr, int vpn, const T *in, T *out, const T *Ainv,
                           const T *B, const T *Tinv);

// applyFilter / applyTranspose (TMRMatrixFilter.cpp:191-235).
template <typename T>
static void horner(Filter &F, bool tr, int vpn, const T *in, T *out, const T *Ainv,
                   const T *B, const T *Tinv) {
  const long long len = F.n * vpn;
  if (len == 0) return;
  if (F.tiled.ok && F.N > 0) {
    DBuf<T> t1(len, F.s), tmp(F.N > 1 ? len : 0, F.s);
    horner_tiled<T>(F, tr, vpn, in, out, t1.p, tmp.p, Ainv, B, Tinv, F.s);
    return;
  }
  horner_generic<T>(F, tr, vpn, in, out, Ainv, B, Tinv);
}

template <typename T>
static void horner_generic(Filter &F, bool tr, int vpn, const T *in, T *out, const T *Ainv,
                           const T *B, const T *Tinv) {
  cudaStream_t s = F.s;
  long long n = F.n, len = n * vpn;
  DBuf<T> t1(len, s), tmp(len, s);
  const T *pre = tr ? Tinv : Ainv;
  const T *post = tr ? Ainv : Tinv;
  prof_bytes(2LL * sizeof(T) * len + (long long)sizeof(T) * n);
  launch(k_fe_scale<T>, blocks_for(len, 256), 256, 0, s, n, vpn, pre, in, t1.p);
  if (F.N == 0) {
    prof_bytes(2LL * sizeof(T) * len + (long long)sizeof(T) * n);
    launch(k_fe_scale<T>, blocks_for(len, 256), 256, 0, s, n, vpn, post,
           (const T *)t1.p, out);
    return;
  }
  // ping-pong so that the last term lands in `out`
  const T *x = t1.p;
  for (int k = 0; k < F.N; k++) {
    bool last = (k == F.N - 1);
    T *y = ((F.N - 1 - k) % 2 == 0) ? out : tmp.p;
    if (tr)
      launch_sell<T, true>(F, vpn, B, t1.p, x, y, last ? post : nullptr, s);
    else
      launch_sell<T, false>(F, vpn, B, t1.p, x, y, last ? post : nullptr, s);
    x = y;
  }
}

void filter_apply(Filter &F, bool tr, int vpn, const double *in, double *out) {
  Stage st(tr ? "tmrg_filter_apply_transpose" : "tmrg_filter_apply");
  horner<double>(F, tr, vpn, in, out, F.Ainv.p, F.B.p, F.Tinv.p);
}
void filter_apply_f32(Filter &F, bool tr, int vpn, const float *in, float *out) {
  horner<float>(F, tr, vpn, in, out, F.Ainv32.p, F.B32.p, F.Tinv32.p);
}

// ---------------------------------------------------------------------
// Allocation-free apply.  Some callers cannot allocate device memory at
// the point where they filter: a framework whose caching allocator owns
// the GPU's memory, or a section that must not call cudaMalloc/cudaFree
// because those can synchronise the device.  This variant takes its two
// Horner work vectors (t1 and the ping-pong term) from a static device
// array instead of the stream-ordered pool.
//
// The array holds 2 x FILTER_STATIC_MAX doubles (16 MiB) and stays
// resident on every GPU that loads the library until the process exits.
// Every call shares it and it keeps the last call's contents; nothing in
// it has to start at zero (each call writes t1 and every Horner term in
// full before reading them).  Calls that overlap on the GPU (different
// streams, or different filters sharing a device) race on the array.
constexpr long long FILTER_STATIC_MAX = 1LL << 20;
static __device__ __align__(256) double g_filter_static[2 * FILTER_STATIC_MAX];

// Device address of the array on the current device, looked up once per
// device: in host code `g_filter_static` names a host-side stand-in, not
// device memory.  The first call on a device performs the lookup, so it
// should come before any stream capture.
static double *filter_static_scratch() {
  static std::mutex mu;
  static double *addr[256] = {nullptr};
  int dev = 0;
  TMRG_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 256) throw Error(TMRG_ERR_ARG, "device ordinal out of range");
  std::lock_guard<std::mutex> lk(mu);
  if (!addr[dev]) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_filter_static);
    if (e != cudaSuccess)
      throw Error(TMRG_ERR_CUDA, std::string("cudaGetSymbolAddress(filter scratch): ") +
                                     cudaGetErrorString(e));
    addr[dev] = (double *)p;
  }
  return addr[dev];
}

void filter_apply_static(Filter &F, bool tr, int vpn, const double *in, double *out) {
  const long long n = F.n, len = n * vpn;
  if (len > FILTER_STATIC_MAX)
    throw Error(TMRG_ERR_ARG,
                "allocation-free filter apply: " + std::to_string(len) +
                    " values (nodes x vpn) exceed the static scratch limit of " +
                    std::to_string(FILTER_STATIC_MAX));
  Stage st(tr ? "tmrg_filter_apply_static_transpose" : "tmrg_filter_apply_static");
  double *t1 = filter_static_scratch();
  double *tmp = t1 + FILTER_STATIC_MAX;
  if (n == 0) return;
  cudaStream_t s = F.s;
  if (F.tiled.ok && F.N > 0) {
    horner_tiled<double>(F, tr, vpn, in, out, t1, tmp, F.Ainv.p, F.B.p, F.Tinv.p, s);
    return;
  }
  const double *pre = tr ? F.Tinv.p : F.Ainv.p;
  const double *post = tr ? F.Ainv.p : F.Tinv.p;
  prof_bytes(2LL * sizeof(double) * len + (long long)sizeof(double) * n);
  launch(k_fe_scale<double>, blocks_for(len, 256), 256, 0, s, n, vpn, pre, in, t1);
  if (F.N == 0) {
    prof_bytes(2LL * sizeof(double) * len + (long long)sizeof(double) * n);
    launch(k_fe_scale<double>, blocks_for(len, 256), 256, 0, s, n, vpn, post,
           (const double *)t1, out);
    return;
  }
  const double *x = t1;
  for (int k = 0; k < F.N; k++) {
    bool last = (k == F.N - 1);
    double *y = ((F.N - 1 - k) % 2 == 0) ? out : tmp;
    if (tr)
      launch_sell<double, true>(F, vpn, F.B.p, t1, x, y, last ? post : nullptr, s);
    else
      launch_sell<double, false>(F, vpn, F.B.p, t1, x, y, last ? post : nullptr, s);
    x = y;
  }
}

// What the filter needs from an octree or quadtree forest (nodes created).
struct FSource {
  cudaStream_t s;
  int order, npe, dim;
  long long ne, nn;
  const int *econn, *dptr, *dconn;
  const double *dw;
  const int16_t *level;
};
static void filter_build(const FSource &f, double len, double r, int N, Filter &F);

// 1-D Bernstein mass of degree p on [0, 1]:
// C(p, i) C(p, j) / ((2p + 1) C(2p, i + j)), one division.
static double bernstein_mass_1d(int p, int i, int j) {
  double ci = 1.0, cj = 1.0, c2 = 1.0;
  for (int k = 1; k <= i; k++) ci = ci * (p - k + 1) / k;
  for (int k = 1; k <= j; k++) cj = cj * (p - k + 1) / k;
  for (int k = 1; k <= i + j; k++) c2 = c2 * (2 * p - k + 1) / k;
  return (ci * cj) / ((2 * p + 1) * c2);
}

void filter_create(Forest &f, double len, double r, int N, Filter &F) {
  Stage st("tmrg_filter_create");
  if (f.order < 2 || f.order > 4)
    throw Error(TMRG_ERR_UNSUPPORTED,
                "matrix filter: forests of order 2-4 (the element bases the reference's "
                "matrix creator provides)");
  forest_create_nodes(f);
  filter_build(FSource{f.s, f.order, f.order * f.order * f.order, 3, f.n, f.num_owned,
                       f.econn.p, f.dep_ptr.p, f.dep_conn.p, f.dep_w.p, f.level.p},
               len, r, N, F);
}
void filter_create_quad(QForest &f, double len, double r, int N, Filter &F) {
  Stage st("tmrg_filter_create");
  if (f.order != 2)
    throw Error(TMRG_ERR_UNSUPPORTED, "matrix filter: order-2 forests only");
  qforest_create_nodes(f);
  filter_build(FSource{f.s, 2, 4, 2, f.n, f.num_owned, f.econn.p, f.dep_ptr.p, f.dep_conn.p,
                       f.dep_w.p, f.level.p},
               len, r, N, F);
}

// M from its E block entries: sorted by (row, column), equal ones summed in
// element order.
static void sum_entries(DBuf<uint64_t> &keys, DBuf<uint32_t> &perm, DBuf<double> &ev, long long E,
                        int cb, Filter &F) {
  cudaStream_t s = F.s;
  const long long n = F.n;
  radix_sort(keys, &perm, E, 2 * cb, s);
  DBuf<unsigned> pos(E + 1, s);
  launch(k_fe_first, blocks_for(E, 256), 256, 0, s, E, (const uint64_t *)keys.p,
         pos.p);
  exclusive_scan<unsigned>(pos.p, pos.p, E, s);
  const long long nnz = read_scalar(pos.p + E, s);
  F.nnz = nnz;
  F.colidx.alloc(nnz + 1, s);
  F.vals.alloc(nnz + 1, s);
  F.rowptr.alloc(n + 1, s);
  F.rowptr.zero();
  launch(k_fe_reduce, blocks_for(E, 256), 256, 0, s, E, (const uint64_t *)keys.p,
         (const uint32_t *)perm.p, (const double *)ev.p, (const unsigned *)pos.p,
         cb, F.colidx.p, F.vals.p, F.rowptr.p);
  keys.release();
  perm.release();
  ev.release();
  pos.release();
  exclusive_scan<int>(F.rowptr.p, F.rowptr.p, n, s);
}

// The entries of orders 3 and 4.
static void assemble_sorted(const FSource &f, const FilterCtx &c, int cb, Filter &F) {
  cudaStream_t s = f.s;
  const long long ne = f.ne;
  long long E = 0;
  DBuf<uint64_t> keys;
  DBuf<uint32_t> perm;
  DBuf<double> ev;
  FGen g{};
  g.o = f.order;
  g.npe = f.npe;
  for (int i = 0; i < g.o; i++)
    for (int j = 0; j < g.o; j++) g.m1[i][j] = bernstein_mass_1d(g.o - 1, i, j);
  DBuf<int> mx(2, s);
  mx.zero();
  launch(k_fe_gen_emax, blocks_for(ne, 256), 256, 0, s, ne, c, g.npe, mx.p);
  const int emax = read_scalar(mx.p, s);
  // count pass: the list and its distinct nodes (at most the list length)
  g.cap = std::max(32, emax);
  g.kcap = g.cap;
  g.tcols = 0;
  const size_t sm_c = fg_layout(g).total * FG_WARPS;
  if (g.cap > 65535 || sm_c > 200 * 1024)
    throw Error(TMRG_ERR_UNSUPPORTED, "matrix filter: an element expands to " +
                                          std::to_string(emax) + " entries");
  DBuf<long long> cnt(ne + 1, s);
  TMRG_CUDA(cudaFuncSetAttribute(k_fe_gen_count, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sm_c));
  launch(k_fe_gen_count, blocks_for(ne, FG_WARPS), FG_WARPS * 32, sm_c, s, ne, c, g, cnt.p,
         mx.p + 1);
  const int kmax = read_scalar(mx.p + 1, s);
  if (read_scalar(c.err, s))
    throw Error(TMRG_ERR_UNSUPPORTED, "matrix filter: an element touches too many nodes");
  exclusive_scan<long long>(cnt.p, cnt.p, ne, s);
  E = read_scalar(cnt.p + ne, s);
  if (E >= (1LL << 32))
    throw Error(TMRG_ERR_ARG, "matrix filter: more than 2^32 element-matrix entries");
  // write pass: T over the largest number of distinct nodes
  g.kcap = std::max(1, kmax);
  g.tcols = g.kcap;
  const size_t smem = fg_layout(g).total * FG_WARPS;
  if (smem > 227 * 1024)
    throw Error(TMRG_ERR_UNSUPPORTED, "matrix filter: an element touches " +
                                          std::to_string(kmax) + " independent nodes");
  keys.alloc(E, s);
  perm.alloc(E, s);
  ev.alloc(E, s);
  TMRG_CUDA(cudaFuncSetAttribute(k_fe_gen_write, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
  launch(k_fe_gen_write, blocks_for(ne, FG_WARPS), FG_WARPS * 32, smem, s, ne, c, g, cb,
         (const long long *)cnt.p, keys.p, perm.p, ev.p);
  sum_entries(keys, perm, ev, E, cb, F);
}

// Block entries (of elements without dependent nodes) up to which a linear mesh's
// are sorted: a few passes over little, where the rows' tables take 25 launches.
// The whole filter by the sort against by rows: 450 octants 0.82 and 0.88 ms, 10K
// 0.92 and 1.00, 27K 1.032 and 1.035, 53K 1.35 and 1.20; quadrants 7.9K 0.45 and
// 0.52, 109K 0.65 and 0.67, 468K 1.44 and 1.13.
constexpr long long FE_SORT_MAX = 2000000;

static void filter_build(const FSource &f, double len, double r, int N, Filter &F) {
  cudaStream_t s = f.s;
  F.s = s;
  F.N = N;
  F.r = r;
  const long long n = f.nn, ne = f.ne;
  F.n = n;
  DBuf<int> err(1, s);
  err.zero();
  FilterCtx c{f.econn, f.dptr, f.dconn, f.dw, len, f.level, err.p, f.npe, f.dim};
  const int cb = bits_for(n + 1);
  if (2 * cb > 64) throw Error(TMRG_ERR_KEY_RANGE, "filter key range");
  if (f.order == 2) {
    MassEntry ent{len, f.level, f.dim, 0};
    const double m0 = f.dim == 3 ? len * len * len / 27.0 : len * len / 9.0;
    memcpy(&ent.m0, &m0, sizeof(m0));
    // near the ends of the exponent's range an entry of a deep level might
    // not be the scaled one (3 x 30 levels and nd <= 3)
    const int ex = (int)((ent.m0 >> 52) & 0x7ff);
    const ElemCtx ec{c.conn, c.dptr, c.dconn, c.dw, c.err, c.npe};
    AsmResult res = ASM_PLACES;
    if (ne * c.npe * c.npe > FE_SORT_MAX)
      res = assemble_rows(ec, ent, n, ne, ex < 128 || ex == 0x7ff, F.rowptr, F.colidx, F.vals,
                          F.nnz, s);
    if (res == ASM_PLACES) {
      DBuf<uint64_t> keys;
      DBuf<uint32_t> perm;
      DBuf<double> ev;
      long long E = 0;
      err.zero();
      res = assemble_entries(ec, ent, ne, cb, keys, perm, ev, E, s);
      if (res == ASM_DONE) sum_entries(keys, perm, ev, E, cb, F);
    }
    if (res == ASM_NODES)
      throw Error(TMRG_ERR_INTERNAL, "matrix filter: element touches too many nodes");
    if (res == ASM_ENTRIES)
      throw Error(TMRG_ERR_ARG, "matrix filter: more than 2^32 element-matrix entries");
  } else {
    assemble_sorted(f, c, cb, F);
  }
  if (read_scalar(err.p, s))
    throw Error(TMRG_ERR_INTERNAL, "matrix filter: element touches too many nodes");
  F.Ainv.alloc(n, s);
  F.B.alloc(n, s);
  F.Tinv.alloc(n, s);
  launch(k_fe_scalings, blocks_for(n, 256), 256, 0, s, n, f.dim, (const int *)F.rowptr.p,
         (const double *)F.vals.p, r, F.Ainv.p, F.B.p);
  // the copy the Horner steps read: tiled, or sliced with 32-bit columns
  // where a tile has too many
  if (tsell_build(F.tiled, n, F.rowptr.p, F.colidx.p, s)) {
    tsell_values(F.tiled, F.rowptr.p, (const double *)F.vals.p, F.tval, s);
    tsell_values(F.tiled, F.rowptr.p, (const double *)F.vals.p, F.tval32, s);
  } else {
    const long long nsl = (n + 31) / 32;
    F.npos = nsl * 32;
    F.sperm.alloc(std::max(1LL, n), s);
    F.srl.alloc(std::max(1LL, F.npos), s);
    F.soff.alloc(nsl + 1, s);
    if (n) len_order(n, (const int *)F.rowptr.p, F.sperm.p, s);
    launch(k_sell_len, blocks_for(F.npos, 256), 256, 0, s, F.npos, n, (const int *)F.sperm.p,
           (const int *)F.rowptr.p, F.srl.p, F.soff.p);
    exclusive_scan<long long>(F.soff.p, F.soff.p, nsl, s);
    F.nsell = read_scalar(F.soff.p + nsl, s);
    F.scol.alloc(std::max(1LL, F.nsell), s);
    F.sval.alloc(std::max(1LL, F.nsell), s);
    launch((k_sell_fill<double>), blocks_for(F.npos, 256), 256, 0, s, F.npos, n,
           (const int *)F.sperm.p, (const int *)F.rowptr.p, (const int *)F.colidx.p,
           (const double *)F.vals.p, (const long long *)F.soff.p, F.scol.p, F.sval.p);
  }
  // Tinv = 1 / (F~ 1) with Tinv = 1 during the evaluation.
  {
    DBuf<double> ones(n, s), y(n, s);
    launch(k_fe_ones, blocks_for(n, 256), 256, 0, s, n, ones.p, F.Tinv.p);
    filter_apply(F, false, 1, ones.p, y.p);
    launch(k_fe_tinv, blocks_for(n, 256), 256, 0, s, n, (const double *)y.p,
           F.Tinv.p);
    TMRG_CUDA(cudaStreamSynchronize(s));
  }
  if (!F.tiled.ok) {
    F.sval32.alloc(std::max(1LL, F.nsell), s);
    launch(k_to_f32<float>, blocks_for(F.nsell, 256), 256, 0, s, F.nsell,
           (const double *)F.sval.p, F.sval32.p);
  }
  F.Ainv32.alloc(n, s);
  F.B32.alloc(n, s);
  F.Tinv32.alloc(n, s);
  launch(k_to_f32<float>, blocks_for(n, 256), 256, 0, s, n,
         (const double *)F.Ainv.p, F.Ainv32.p);
  launch(k_to_f32<float>, blocks_for(n, 256), 256, 0, s, n,
         (const double *)F.B.p, F.B32.p);
  launch(k_to_f32<float>, blocks_for(n, 256), 256, 0, s, n,
         (const double *)F.Tinv.p, F.Tinv32.p);
  TMRG_CUDA(cudaStreamSynchronize(s));
}

}  // namespace tmrg
