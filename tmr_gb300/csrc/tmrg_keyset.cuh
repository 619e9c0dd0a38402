// A set of 64-bit keys in device memory (open addressing, linear probing)
// with the list of its members in the order they were added: the families
// of the 2:1 balance.  Forest operations that only need "is this family
// there yet" use it instead of sorting every generation of candidates.
#pragma once

#include "tmrg_prims.cuh"

namespace tmrg {

// No octant key is all ones (the level field holds at most 30).
constexpr unsigned long long KEYSET_EMPTY = ~0ULL;
// A probe that has not ended after this many slots sets `overflow` (the
// table is kept at most two thirds full, where runs are tens of slots).
constexpr int KEYSET_PROBES = 1024;
// count[g]: members added in generation g (one launch per generation)
constexpr int KEYSET_GENS = 40;

struct KeySet {
  unsigned long long *tab;
  int shift;         // 64 - log2(table size)
  uint64_t *list;    // members in the order added
  unsigned cap;      // entries the list holds
  unsigned *count;   // [KEYSET_GENS], then the overflow flag, then a leaf counter

  __device__ __forceinline__ unsigned slot(uint64_t k) const {
    return (unsigned)((k * 0x9E3779B97F4A7C15ULL) >> shift);
  }
  __device__ __forceinline__ unsigned *overflow() const { return count + KEYSET_GENS; }
  __device__ __forceinline__ unsigned *counter() const { return count + KEYSET_GENS + 1; }
  // The set overflowed and is given up.  A whole warp asks and gets one answer.
  __device__ __forceinline__ bool full() const {
    return __any_sync(0xffffffffu, __ldcg(overflow()) != 0u);
  }
  // True when `k` was not in the set (it is now).
  __device__ __forceinline__ bool insert(uint64_t k) const {
    const unsigned mask = 0xffffffffu >> (shift - 32);
    unsigned s = slot(k);
    for (int i = 0; i < KEYSET_PROBES; i++) {
      unsigned long long v = __ldcg(tab + s);
      if (v == KEYSET_EMPTY) {
        v = atomicCAS(tab + s, KEYSET_EMPTY, (unsigned long long)k);
        if (v == KEYSET_EMPTY) return true;
      }
      if (v == (unsigned long long)k) return false;
      s = (s + 1) & mask;
    }
    atomicOr(overflow(), 1u);
    return false;
  }
  // Membership, once no kernel adds any more.
  __device__ __forceinline__ bool contains(uint64_t k) const {
    const unsigned mask = 0xffffffffu >> (shift - 32);
    unsigned s = slot(k);
    for (int i = 0; i < KEYSET_PROBES; i++) {
      const unsigned long long v = __ldg(tab + s);
      if (v == (unsigned long long)k) return true;
      if (v == KEYSET_EMPTY) return false;
      s = (s + 1) & mask;
    }
    return false;
  }
  // Members before generation g.
  __device__ __forceinline__ unsigned before(int g) const {
    unsigned t = 0;
    for (int i = 0; i < g; i++) t += count[i];
    return min(t, cap);
  }
  // Adds one key per lane where `on`, new members appended as generation g
  // from list position `base` = before(g); a whole warp calls it.  True once the
  // list has no room for what the warp adds: the set is given up then, and a
  // caller that goes on would fill the table (KEYSET_PROBES steps a key).
  __device__ __forceinline__ bool add(uint64_t k, bool on, int g, unsigned base) const {
    const bool fresh = on && insert(k);
    const unsigned m = __ballot_sync(0xffffffffu, fresh);
    if (m == 0u) return false;
    const int lane = threadIdx.x & 31, lead = __ffs(m) - 1;
    unsigned o = 0;
    if (lane == lead) o = atomicAdd(count + g, (unsigned)__popc(m));
    o = __shfl_sync(0xffffffffu, o, lead) + base;
    const unsigned at = o + __popc(m & ((1u << lane) - 1u));
    if (fresh && at < cap) list[at] = k;
    const bool none = o + __popc(m) > cap;
    if (none && lane == lead) atomicOr(overflow(), 1u);
    return none;
  }
};

// The buffers of a KeySet for up to `cap` members.
struct KeySetBuf {
  DBuf<unsigned long long> tab;
  DBuf<uint64_t> list;
  DBuf<unsigned> count;
  KeySet set{};
  KeySetBuf(long long cap, cudaStream_t s) {
    int lg = 10;
    while ((1LL << lg) * 2 < 3 * cap) lg++;
    tab.alloc((size_t)1 << lg, s);
    tab.fill_bytes(0xff);
    list.alloc((size_t)cap, s);
    count.alloc(KEYSET_GENS + 2, s);
    count.zero();
    set = KeySet{tab.p, 64 - lg, list.p, (unsigned)cap, count.p};
  }
};

}  // namespace tmrg
