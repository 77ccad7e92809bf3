// The record side of the NN-descent join (base_index.hpp:328-371), shared by the join over FP32 rows
// (join_fp32.cu), over byte rows (bytes.cu) and on the tensor cores (join_tc.cu): which of a pair's two sides becomes
// a pool-insert record, and where the record goes.
#pragma once
#include "internal.cuh"

namespace efg {

// A record, 16 bytes: candidate id, distance bits (together the little-endian (dist, id) key), source
// node << 1 | side, target node.
__device__ __forceinline__ uint64_t rec_key(const uint4& r) { return ((uint64_t)r.y << 32) | r.x; }

// The records of one join.  Every record takes its slot from its target's count as it is found, so
// the pair distances are neither stored nor walked a second time: the first W of a target go to its
// bucket, later ones (hub nodes) to one overflow list with their slots.  W follows the expected
// records per node and a memory bound; with W = 0 every record takes the list.  What this replaced --
// all pair distances stored and per-target counts first, then a scan and a second walk over the
// pairs that placed the records -- moved 8 bytes per pair (2.84 G pairs at 1M x 128, 8 iterations)
// for 0.22 records per pair and spent 35 ms in the second walk alone.
struct RecordSink {
  uint32_t* cnt;               // records per target
  uint4* bucket;               // n x W records
  uint4* ovf;                  // overflow records
  uint32_t* ovf_slot;          // and their slots within their target
  unsigned long long* ovf_n;   // overflow records found (may exceed ovf_cap: the join runs again)
  uint64_t ovf_cap;
  uint32_t W;
  // With little memory (W = 0, ovf_cap = 0) a join counts its records first; its second run has their
  // places, off[t] .. off[t + 1] of ovf for target t: 16 bytes a record and no more.
  const uint64_t* off;
};

// A record whose slot lies past its target's bucket.  (Not inlined: rare, and its code would be
// repeated at every place that makes records.)  One atomic for the lanes that come together: half of the
// records of 1M x 960 with K = 100 are hubs' (260M an iteration), and one address takes 1.5 G atomics a second.
static __device__ __noinline__ void place_overflow(const RecordSink& s, uint32_t t, uint32_t slot, float d,
                                                   uint32_t cand, uint32_t aux) {
  const uint32_t mask = __activemask(), lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
  unsigned long long o = 0;
  if (lane == leader) o = atomicAdd(s.ovf_n, (unsigned long long)__popc(mask));
  o = __shfl_sync(mask, o, leader) + __popc(mask & ((1u << lane) - 1));
  if (s.off) {
    const uint64_t at = s.off[t] + slot;
    if (at < s.off[t + 1]) s.ovf[at] = make_uint4(cand, __float_as_uint(d), aux, t);
    return;
  }
  if (o < s.ovf_cap) {
    s.ovf[o] = make_uint4(cand, __float_as_uint(d), aux, t);
    s.ovf_slot[o] = slot;
  }
}

// Writes a record to slot `slot` (taken from cnt[t]) of target t.
__device__ __forceinline__ void place_record(const RecordSink& s, uint32_t t, uint32_t slot, float d, uint32_t cand,
                                             uint32_t aux) {
  if (slot < s.W) s.bucket[(uint64_t)t * s.W + slot] = make_uint4(cand, __float_as_uint(d), aux, t);
  else place_overflow(s, t, slot, d, cand, aux);
}

}  // namespace efg
