// NN-descent kNN-graph build: leaf-merge initial graph, then `epochs` x (join, update).
//
// Reference (ZJULearning/efanna):
//   initGraph's merge + pool seeding   algorithm/kdtreeub_index.hpp:1000-1081, 1367-1424
//   Point / InsertIntoKnn / insert      algorithm/base_index.hpp:24-93
//   join                                algorithm/base_index.hpp:328-371
//   update                              algorithm/base_index.hpp:373-437
//   refineGraph                         algorithm/base_index.hpp:438-481
//
// Order independence.  The reference applies neighbour-list inserts in whatever order its
// OpenMP threads reach them; its results depend on that order only through ties and through the
// rank an insert lands at.  Here every insert aimed at node t is first materialised as a record
// (dist, candidate, source node, side), the records of t are applied in ascending order of that
// tuple with exactly the reference's insert semantics (radius test, InsertIntoKnn with its
// equal-distance duplicate check and overflow slot, L growth, radius update, rank-based `found`),
// and everything else (reverse-list sampling, initial extra candidates, random fills) comes from
// counter hashes.  A build is therefore a pure function of (data, params), reproduced bit-for-bit
// by the oracle's canonical mode.
//
// Device state (n nodes, pool capacity P = L + 1):
//   pd[n*P]  pool distances           pid[n*P] pool ids, bit 31 = the "new" flag
//   Lc[n], Range[n], radius[n], radiusM[n], found[n]
//   new_ids/old_ids[n*cap] + counts   the sampled lists the next join reads
// Pool slots past L stay zero (dist 0, id 0) until written, as the reference's freshly
// allocated pools are; update() reads pool[L].dist as the next radius either way.
#include <algorithm>
#include <cfloat>
#include <vector>

#include "join.cuh"
#include "scan.cuh"
#include "warpsort.cuh"

namespace efg {

static constexpr uint32_t FLAG = 0x80000000u;
static constexpr uint32_t IDM = 0x7FFFFFFFu;

struct NNDev {
  uint64_t n = 0;
  uint32_t P = 0, cap = 0;
  DevBuf<float> pd, radius, radiusM;
  DevBuf<uint32_t> pid, Lc, Range, new_ids, new_cnt, old_ids, old_cnt;
  DevBuf<uint8_t> found;
  // scratch
  DevBuf<uint64_t> task_len, off64, scan64;
  DevBuf<uint32_t> cnt, cursor, rcnt, rcur, roff, rbuf, scan32;
  DevBuf<float> bound;
  DevBuf<unsigned long long> totals;  // pairs, records, overflow records, nodes larger than a tile
  DevBuf<uint32_t> jctr;              // node counters: the merge's, the join's (up to three launches)
  DevBuf<uint4> bucket, ovf, ovfrec;  // join records: per-target buckets, overflow list, hub targets' records
  DevBuf<uint32_t> ovf_slot;
  // tensor-core join: BF16 rows (hi, lo), FP32 norms, flags {inexact, error}, nodes left to FP32
  DevBuf<__nv_bfloat16> jhi, jlo;
  DevBuf<float> jnorm;
  DevBuf<int> jflag;  // inexact, error, not integers
  DevBuf<uint32_t> jmid, jbig;  // nodes of 129-256 rows, and larger ones (FP32: of many pairs); count in word 0
  uint32_t jterms = 0;  // 0: not prepared; 1 or 3 products per value
  bool jexact = false;  // the tensor cores' distances are exact (integers, squared norms below 2^22)
  uint32_t W = 0;          // records per bucket
  uint64_t bucket_cap = 0, ovf_cap = 0, last_ovf = 0;  // last_ovf: the last iteration's overflow records
  bool scarce = false;  // memory for buckets and lists fell short: every join counts, then places, its records
  // every buffer from the stream's pool: only the build's stream uses them
  explicit NNDev(cudaStream_t s) {
    each([s](auto& b) { b.on(s); });
  }
  ~NNDev() {
    each([](auto& b) { b.release(); });
  }
  NNDev(const NNDev&) = delete;
  NNDev& operator=(const NNDev&) = delete;
  // Gives the record buffers back (their contents are lost); the build goes on in 16 bytes a record, with
  // every join run twice.
  void run_scarce() {
    bucket.release();
    ovf.release();
    ovf_slot.release();
    ovfrec.release();
    W = 0;
    ovf_cap = last_ovf = 0;
    scarce = true;
  }
  // Room in b, at the record buffers' cost when there is no other (while they hold nothing).
  template <typename B>
  int room(B& b, uint64_t count) {
    if (b.reserve(count) == EFG_OK) return EFG_OK;
    run_scarce();
    return b.reserve(count);
  }
  template <typename F>
  void each(F f) {
    auto all = [&](auto&... b) { (f(b), ...); };
    all(pd, radius, radiusM, pid, Lc, Range, new_ids, new_cnt, old_ids, old_cnt, found, task_len, off64, scan64,
        cnt, cursor, bound, rcnt, rcur, roff, rbuf, scan32, totals, jctr, bucket, ovf, ovfrec, ovf_slot,
        jhi, jlo, jnorm, jflag, jmid, jbig);
  }
};

static int nn_alloc(NNDev& S, uint64_t n, uint32_t L, uint32_t cap) {
  S.n = n;
  S.P = L + 1;
  S.cap = cap;
  uint64_t np = n * S.P;
  EFG_TRY(S.pd.reserve(np));
  EFG_TRY(S.pid.reserve(np));
  EFG_TRY(S.Lc.reserve(n));
  EFG_TRY(S.Range.reserve(n));
  EFG_TRY(S.radius.reserve(n));
  EFG_TRY(S.radiusM.reserve(n));
  EFG_TRY(S.found.reserve(n));
  EFG_TRY(S.new_ids.reserve(n * cap));
  EFG_TRY(S.old_ids.reserve(n * cap));
  EFG_TRY(S.new_cnt.reserve(n));
  EFG_TRY(S.old_cnt.reserve(n));
  return EFG_OK;
}

// Warp-cooperative partial squared distance between rows a and b (lane owns float4 chunks).
__device__ __forceinline__ float lane_l2_rows(const float* __restrict__ base, uint32_t ld4, uint32_t a, uint32_t b) {
  const float4* ra = reinterpret_cast<const float4*>(base) + (uint64_t)a * ld4;
  const float4* rb = reinterpret_cast<const float4*>(base) + (uint64_t)b * ld4;
  uint32_t lane = threadIdx.x & 31;
  float acc = 0.f;
  for (uint32_t c = lane; c < ld4; c += 32) {
    float4 x = __ldg(ra + c), y = __ldg(rb + c);
    float d0 = x.x - y.x, d1 = x.y - y.y, d2 = x.z - y.z, d3 = x.w - y.w;
    acc += d0 * d0;
    acc += d1 * d1;
    acc += d2 * d2;
    acc += d3 * d3;
  }
  return acc;
}

// =============================================================================================
// Initial graph: leaf merge (mergeSubGraphs) and pool seeding.
// =============================================================================================

struct TreeView {
  const DNode* nodes;
  const int32_t *left, *right, *level, *tree;
  const uint32_t *start, *end;
  const uint32_t* leaves;
  uint64_t n;
};

// Merge tasks: internal nodes of the graph trees at depth >= ml.  len = size of the smaller child.
__global__ void merge_task_len_kernel(TreeView tv, uint64_t nnodes, uint32_t trees_build, int32_t ml,
                                      uint64_t* __restrict__ len) {
  uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nnodes) return;
  uint64_t l = 0;
  if (tv.left[v] >= 0 && (uint32_t)tv.tree[v] < trees_build && tv.level[v] >= ml) {
    int32_t L = tv.left[v], R = tv.right[v];
    uint64_t nl = tv.end[L] - tv.start[L], nr = tv.end[R] - tv.start[R];
    l = nl < nr ? nl : nr;
  }
  len[v] = l;
}

__global__ void min_leaf_level_kernel(TreeView tv, uint64_t nnodes, uint32_t trees_build, int32_t* __restrict__ out) {
  uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nnodes) return;
  if (tv.left[v] < 0 && (uint32_t)tv.tree[v] < trees_build) atomicMin(out, tv.level[v]);
}

// Byte rows for the leaf merge's distances (rows null: FP32 rows).
struct ByteRows {
  const uint8_t* rows;
  const uint32_t* norm;
  uint32_t chunks, gshift;  // 16-byte chunks per row; 2^gshift >= chunks lanes take one row
};

// Routed points: descend the larger child to a leaf (SearchToLeaf, kdtreeub_index.hpp:1012-1021) and
// compare with each leaf point.  pass 0 counts records per target, pass 1 writes them: key = (dist
// bits << 32) | candidate.  With task_d set, pass 0 also keeps each task's point, leaf and distances
// (maxl per task), and merge_emit_kernel writes the records from them instead of a second routing pass.
// A warp routes 32 consecutive tasks at once, one per lane (search and descent are chains of dependent
// loads: the lanes run theirs side by side), then the whole warp computes each task's leaf distances in
// turn.  Bound: the latency of the leaf rows' reads, one task's at a time per warp; byte rows bring
// a leaf of ten points in one pass of four 16-byte loads per lane (8 lanes per row at 128 dimensions).
template <int PASS, bool BYTES>
__global__ void __launch_bounds__(256, 3) merge_route_kernel(const float* __restrict__ base, uint32_t ld4,
                                   const ByteRows br, TreeView tv,
                                   const uint64_t* __restrict__ task_off, uint64_t nnodes, uint64_t ntasks,
                                   uint32_t* __restrict__ cnt, const uint64_t* __restrict__ off,
                                   uint32_t* __restrict__ cursor, uint64_t* __restrict__ keys,
                                   unsigned long long* __restrict__ ndist, uint32_t* __restrict__ task_p,
                                   int32_t* __restrict__ task_leaf, float* __restrict__ task_d, uint32_t maxl) {
  const uint64_t gwarp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t lane = threadIdx.x & 31;
  unsigned long long local = 0;
  const float* fb = base;
  for (uint64_t wb = gwarp * 32; wb < ntasks; wb += nwarps * 32) {
    const uint64_t myw = wb + lane;
    uint32_t myp = 0, mls = 0, mle = 0;
    uint64_t mt = 0;
    // node owning task wb, the last v with task_off[v] <= wb: 32 probes at a time
    uint64_t lo = 0, hi = nnodes;
    while (hi - lo > 1) {
      const uint64_t step = (hi - lo + 32) / 33;
      const uint64_t probe = lo + (lane + 1) * step;
      const uint32_t le = __popc(__ballot_sync(0xffffffffu, probe < hi && task_off[probe] <= wb));
      const uint64_t nlo = lo + le * step;
      hi = nlo + step < hi ? nlo + step : hi;
      lo = nlo;
    }
    if (myw < ntasks) {
      // the lane's own task: a few nodes further
      uint64_t step = 1;
      hi = lo + 1;
      while (hi < nnodes && task_off[hi] <= myw) {
        lo = hi;
        hi += step;
        step *= 2;
      }
      if (hi > nnodes) hi = nnodes;
      while (hi - lo > 1) {
        uint64_t mid = (lo + hi) >> 1;
        if (task_off[mid] <= myw) lo = mid;
        else hi = mid;
      }
      const uint64_t v = lo;
      int32_t L = tv.left[v], R = tv.right[v];
      uint64_t nl = tv.end[L] - tv.start[L], nr = tv.end[R] - tv.start[R];
      int32_t cur = nl < nr ? R : L;
      int32_t small = nl < nr ? L : R;
      mt = (uint64_t)tv.tree[v];
      myp = tv.leaves[mt * tv.n + tv.start[small] + (myw - task_off[v])];
      DNode nd = tv.nodes[cur];
      while (nd.left >= 0) {
        float x = __ldg(fb + (uint64_t)myp * (ld4 * 4) + nd.div_dim);
        cur = x < nd.div_val ? nd.left : nd.right;
        nd = tv.nodes[cur];
      }
      mls = (uint32_t)(-(nd.left + 1));
      mle = (uint32_t)nd.right;
      if (PASS == 0 && task_d) {
        task_p[myw] = myp;
        task_leaf[myw] = cur;
      }
    }
    const uint32_t ntask = ntasks - wb < 32 ? (uint32_t)(ntasks - wb) : 32u;
    for (uint32_t j = 0; j < ntask; ++j) {
      const uint64_t w = wb + j;
      const uint32_t p = __shfl_sync(0xffffffffu, myp, j);
      const uint32_t ls = __shfl_sync(0xffffffffu, mls, j), le = __shfl_sync(0xffffffffu, mle, j);
      const uint64_t t = __shfl_sync(0xffffffffu, mt, j);
      const uint32_t* ll = tv.leaves + t * tv.n;
      if (BYTES) {
        const uint32_t G = 1u << br.gshift, rpi = 32u >> br.gshift, sub = lane >> br.gshift, cl = lane & (G - 1);
        const bool on = cl < br.chunks;
        const uint4 zero = make_uint4(0, 0, 0, 0);
        const uint4* row4 = reinterpret_cast<const uint4*>(br.rows);
        const uint4 y = on ? __ldg(row4 + (uint64_t)p * br.chunks + cl) : zero;
        const uint32_t np = __ldg(br.norm + p);
        const uint32_t span = min(4 * rpi, 32u);
        for (uint32_t i0 = ls; i0 < le; i0 += span) {
          const uint32_t m = min(span, le - i0);  // leaf points of this pass, point i with lane i
          const uint32_t q = lane < m ? ll[i0 + lane] : 0u;
          const uint32_t nq = lane < m ? __ldg(br.norm + q) : 0u;
          uint4 x[4];
          uint32_t dot[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const uint32_t r = u * rpi + sub, id = __shfl_sync(0xffffffffu, q, r < m ? r : 0u);
            x[u] = on && r < m ? __ldg(row4 + (uint64_t)id * br.chunks + cl) : zero;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            dot[u] = __dp4a(x[u].x, y.x, __dp4a(x[u].y, y.y, __dp4a(x[u].z, y.z, __dp4a(x[u].w, y.w, 0u))));
          for (uint32_t o = G >> 1; o > 0; o >>= 1) {
#pragma unroll
            for (int u = 0; u < 4; ++u) dot[u] += __shfl_xor_sync(0xffffffffu, dot[u], o);
          }
          uint32_t mine = 0;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const uint32_t v = __shfl_sync(0xffffffffu, dot[u], (lane & (rpi - 1)) << br.gshift);
            if (lane / rpi == (uint32_t)u) mine = v;
          }
          const float d = (float)(np + nq - 2 * mine);
          local += m;
          if (PASS == 0) {
            if (lane < m) {
              if (task_d) task_d[w * maxl + (i0 - ls) + lane] = d;
              atomicAdd(&cnt[q], 1u);
            }
            if (lane == 0) atomicAdd(&cnt[p], m);
          } else {
            uint32_t b = lane == 0 ? atomicAdd(&cursor[p], m) : 0u;
            b = __shfl_sync(0xffffffffu, b, 0);
            if (lane < m) {
              keys[off[q] + atomicAdd(&cursor[q], 1u)] = pack_key(d, p);
              keys[off[p] + b + lane] = pack_key(d, q);
            }
          }
        }
        continue;
      }
      const float4* rp = reinterpret_cast<const float4*>(base) + (uint64_t)p * ld4;
      for (uint32_t i0 = ls; i0 < le; i0 += 8) {  // eight leaf points at a time, their loads in flight together
        const uint32_t cnt8 = min(8u, le - i0);
        uint32_t qq[8];
        float acc[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          qq[u] = ll[i0 + min((uint32_t)u, cnt8 - 1)];
          acc[u] = 0.f;
        }
        for (uint32_t c = lane; c < ld4; c += 32) {
          float4 y = __ldg(rp + c);
          float4 x[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) x[u] = __ldg(reinterpret_cast<const float4*>(base) + (uint64_t)qq[u] * ld4 + c);
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            float d0 = x[u].x - y.x, d1 = x[u].y - y.y, d2 = x[u].z - y.z, d3 = x[u].w - y.w;
            acc[u] += d0 * d0;
            acc[u] += d1 * d1;
            acc[u] += d2 * d2;
            acc[u] += d3 * d3;
          }
        }
        const float d = reduce8_rows(acc, lane);  // lanes 4r .. 4r+3: leaf point r's distance
        const uint32_t r = lane >> 2;
        uint32_t q = qq[0];
#pragma unroll
        for (int u = 1; u < 8; ++u)
          if (r == (uint32_t)u) q = qq[u];
        local += cnt8;
        const bool put = (lane & 3) == 0 && r < cnt8;
        if (PASS == 0) {
          if (put) {
            if (task_d) task_d[w * maxl + (i0 - ls) + r] = d;
            atomicAdd(&cnt[q], 1u);
          }
          if (lane == 0) atomicAdd(&cnt[p], cnt8);
        } else {
          uint32_t b = lane == 0 ? atomicAdd(&cursor[p], cnt8) : 0u;
          b = __shfl_sync(0xffffffffu, b, 0);
          if (put) {
            keys[off[q] + atomicAdd(&cursor[q], 1u)] = pack_key(d, p);
            keys[off[p] + b + r] = pack_key(d, q);
          }
        }
      }
    }
  }
  if (PASS == 0 && lane == 0 && local) atomicAdd(ndist, local);
}

// Records of the leaf merge from what pass 0 kept: one thread per task, whose own records (the point
// with every leaf point) take their slots by one atomic.
__global__ void merge_emit_kernel(TreeView tv, uint64_t ntasks, const uint32_t* __restrict__ task_p,
                                  const int32_t* __restrict__ task_leaf, const float* __restrict__ task_d,
                                  uint32_t maxl, const uint64_t* __restrict__ off, uint32_t* __restrict__ cursor,
                                  uint64_t* __restrict__ keys) {
  for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < ntasks;
       w += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t p = task_p[w];
    const int32_t leaf = task_leaf[w];
    const DNode nd = tv.nodes[leaf];
    const uint32_t* ll = tv.leaves + (uint64_t)tv.tree[leaf] * tv.n;
    const uint32_t ls = (uint32_t)(-(nd.left + 1)), le = (uint32_t)nd.right;
    const uint64_t mine = off[p] + atomicAdd(&cursor[p], le - ls);
    for (uint32_t i0 = ls; i0 < le; i0 += 4) {  // four atomics in flight
      uint32_t q[4], slot[4];
      float d[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i0 + u < le) {
          q[u] = ll[i0 + u];
          d[u] = task_d[w * maxl + (i0 + u - ls)];
        }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i0 + u < le) slot[u] = atomicAdd(&cursor[q[u]], 1u);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i0 + u < le) {
          keys[off[q[u]] + slot[u]] = pack_key(d[u], p);
          keys[mine + (i0 + u - ls)] = pack_key(d[u], q[u]);
        }
    }
  }
}

// Largest leaf of the forest (points per leaf).
__global__ void max_leaf_kernel(TreeView tv, uint64_t nnodes, uint32_t* __restrict__ out) {
  uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nnodes) return;
  if (tv.left[v] < 0) atomicMax(out, (uint32_t)(tv.end[v] - tv.start[v]));
}

// Position of x in the ascending warp-distributed list t (number of elements < x), or -1 if an
// element equals x.
// Every lane must call this (fixed five shuffle steps, no lane-dependent trip count).
__device__ __forceinline__ int warp_find(uint64_t t, uint64_t x) {
  int pos = 0;  // number of elements < x (branchless lower bound over 32 sorted lanes)
#pragma unroll
  for (int step = 16; step > 0; step >>= 1) {
    uint64_t v = __shfl_sync(0xffffffffu, t, pos + step - 1);
    if (v < x) pos += step;
  }
  uint64_t at = __shfl_sync(0xffffffffu, t, pos < 32 ? pos : 31);
  return (pos < 32 && at == x) ? -1 : pos;
}

// Folds one batch (one key per lane, ~0 = none) into the running ascending list of distinct keys.
__device__ __forceinline__ uint64_t fold_distinct(uint64_t run, uint64_t x) {
  uint32_t lane = threadIdx.x & 31;
  uint32_t same = __match_any_sync(0xffffffffu, x);
  if ((same & ((1u << lane) - 1)) != 0) x = ~0ULL;  // keep the lowest lane of each equal group
  int found_at = warp_find(run, x);
  if (x != ~0ULL && found_at < 0) x = ~0ULL;
  x = warp_sort32(x);
  return warp_merge_min32(run, x);
}

// Keys waiting to be folded into a warp's running list: those below the list's `rank`-th key, which
// few are once the list has settled (of 494 records per node about 70 in all), so a fold -- a match, a
// sort and a merge of 32 -- runs for every 32 of them and not for every 32 records (15.5 ms of the
// 1M x 128 build without the queue).
struct FoldQueue {
  uint64_t* q;  // 64 keys in shared memory
  uint32_t n, rank;
  uint64_t run, limit;
  __device__ __forceinline__ FoldQueue(uint64_t* mem, uint32_t rank_) : q(mem), n(0), rank(rank_), run(~0ULL), limit(~0ULL) {}
  __device__ __forceinline__ void fold(uint32_t m) {  // the first m <= 32
    const uint32_t lane = threadIdx.x & 31;
    __syncwarp();
    const uint64_t x = lane < m ? q[lane] : ~0ULL;
    const uint64_t rest = lane + 32 < n ? q[lane + 32] : ~0ULL;
    run = fold_distinct(run, x);
    limit = __shfl_sync(0xffffffffu, run, rank - 1);
    __syncwarp();
    if (lane + 32 < n) q[lane] = rest;
    n -= m;
    __syncwarp();
  }
  __device__ __forceinline__ void push(uint64_t x) {  // one key per lane, ~0 = none
    const uint32_t lane = threadIdx.x & 31;
    const bool take = x < limit;
    const uint32_t bal = __ballot_sync(0xffffffffu, take);
    if (take) q[n + __popc(bal & ((1u << lane) - 1))] = x;
    n += __popc(bal);
    if (n >= 32) fold(32);
  }
  __device__ __forceinline__ void finish() {
    if (n) fold(n);
  }
};

// One warp per node: S best distinct (dist, id) keys, S extra join candidates, pool seeding.
__global__ void __launch_bounds__(256) init_select_kernel(const float* __restrict__ base, uint32_t ld4, uint64_t n, uint32_t S, uint32_t P,
                                   uint32_t cap, uint64_t seed, const uint32_t* __restrict__ cnt,
                                   const uint64_t* __restrict__ off, const uint64_t* __restrict__ keys,
                                   float* __restrict__ pd, uint32_t* __restrict__ pid, uint32_t* __restrict__ Lc,
                                   uint32_t* __restrict__ Range, float* __restrict__ radius,
                                   float* __restrict__ radiusM, uint8_t* __restrict__ found,
                                   uint32_t* __restrict__ new_ids, uint32_t* __restrict__ new_cnt,
                                   uint32_t* __restrict__ old_cnt) {
  uint64_t t = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  uint32_t lane = threadIdx.x & 31;
  if (t >= n) return;
  const uint64_t* R = keys + off[t];
  uint32_t B = cnt[t];
  __shared__ uint64_t queue[8][64];
  // 1. the S smallest distinct keys
  FoldQueue best(queue[threadIdx.x >> 5], S);
  for (uint32_t b = 0; b < B; b += 32) best.push(b + lane < B ? R[b + lane] : ~0ULL);
  best.finish();
  uint64_t run = best.run;
  uint32_t nvalid = __popc(__ballot_sync(0xffffffffu, run != ~0ULL));
  // 2. top up to S distinct with counter-hash random ids (kdtreeub_index.hpp:1399-1405)
  if (nvalid < S) {
    CRng g(hash4(seed, TAG_TOPUP, t, 0, 0));
    uint32_t guard = 0;
    while (nvalid < S && guard < 1000000u) {
      ++guard;
      uint32_t rid = g.next() % (uint32_t)n;
      float d = warp_sum(lane_l2_rows(base, ld4, (uint32_t)t, rid));
      uint64_t x = lane == 0 ? pack_key(d, rid) : ~0ULL;
      run = fold_distinct(run, x);
      nvalid = __popc(__ballot_sync(0xffffffffu, run != ~0ULL));
    }
  }
  uint64_t kth = __shfl_sync(0xffffffffu, run, S - 1);
  // 3. extras: S of the distinct keys beyond the S best, by smallest (hash, id); needs >= 2S
  FoldQueue more(queue[threadIdx.x >> 5], 2 * S);
  if (kth != ~0ULL) {
    const uint64_t hkey = mix64(mix64(seed ^ (TAG_EXTRA * 0x9E3779B97F4A7C15ULL)) ^ t);  // hash4's first two steps
    for (uint32_t b = 0; b < B; b += 32) {
      uint64_t x = ~0ULL;
      if (b + lane < B) {
        uint64_t k = R[b + lane];
        if (k > kth) {
          uint32_t c = (uint32_t)k;
          x = ((mix64(mix64(hkey ^ c)) >> 32) << 32) | c;
        }
      }
      more.push(x);
    }
    more.finish();
  }
  const uint64_t hrun = more.run;
  uint32_t nh = __popc(__ballot_sync(0xffffffffu, hrun != ~0ULL));
  uint32_t extra = 0;  // lane l < S holds extra id l
  if (nh >= 2 * S) {
    extra = (uint32_t)hrun;
  } else if (lane == 0) {
    // GenRandom(2S) (kdtreeub_index.hpp:1121-1135) on a counter stream; keep positions S..2S-1
    uint32_t addr[32];
    uint32_t size = 2 * S, N = (uint32_t)n;
    CRng g(hash4(seed, TAG_GENRAND, t, 0, 0));
    for (uint32_t i = 0; i < size; ++i) addr[i] = g.next() % (N - size);
    for (uint32_t i = 1; i < size; ++i) {  // insertion sort
      uint32_t v = addr[i];
      int j = (int)i - 1;
      while (j >= 0 && addr[j] > v) {
        addr[j + 1] = addr[j];
        --j;
      }
      addr[j + 1] = v;
    }
    for (uint32_t i = 1; i < size; ++i)
      if (addr[i] <= addr[i - 1]) addr[i] = addr[i - 1] + 1;
    uint32_t offr = g.next() % N;
    for (uint32_t i = 0; i < S; ++i) new_ids[t * cap + S + i] = (addr[S + i] + offr) % N;
  }
  // 4. seed the pool and the first new list (lane j < S holds the j-th best key)
  uint64_t prow = t * P;
  uint64_t mine = run;
  for (uint32_t j = lane; j < P; j += 32) {
    float dd = 0.f;
    uint32_t ii = 0;
    if (j < S) {
      dd = key_dist(mine);
      ii = key_id(mine) | FLAG;
    }
    pd[prow + j] = dd;
    pid[prow + j] = ii;
  }
  if (lane < S) new_ids[t * cap + lane] = key_id(run);
  if (nh >= 2 * S && lane < S) new_ids[t * cap + S + lane] = extra;
  if (lane == 0) {
    Lc[t] = S;
    Range[t] = S;
    radius[t] = FLT_MAX;
    radiusM[t] = 0.f;
    found[t] = 0;
    new_cnt[t] = 2 * S;
    old_cnt[t] = 0;
  }
}

// =============================================================================================
// Join.
// =============================================================================================

// bound[t]: the largest distance any insert aimed at node t can still be accepted at during this join:
// max(radius, pool[L-1].dist).  Inserts beyond it are rejected by Neighbor::insert whatever the order
// (the radius never rises above it), so their records need not be materialised.  total: the pairs of
// the nodes' joins, new x new with p < q and new x old.
__global__ void __launch_bounds__(256) bound_kernel(uint64_t n, uint32_t P, const float* __restrict__ pd,
                                                    const uint32_t* __restrict__ Lc, const float* __restrict__ radius,
                                                    const uint32_t* __restrict__ new_cnt,
                                                    const uint32_t* __restrict__ old_cnt, float* __restrict__ bound,
                                                    unsigned long long* __restrict__ total) {
  __shared__ unsigned long long wsum[8];
  uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long pairs = 0;
  if (t < n) {
    float r = radius[t];
    float w = pd[t * P + Lc[t] - 1];
    bound[t] = r > w ? r : w;
    uint64_t a = new_cnt[t], b = old_cnt[t];
    pairs = a * (a - (a > 0 ? 1 : 0)) / 2 + a * b;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
  if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = pairs;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) pairs += wsum[w];
    if (pairs) atomicAdd(total, pairs);
  }
}

// Targets with more records than a bucket holds: their record counts (0 for the others), whose scan
// places their records in one exactly sized array.
__global__ void hub_len_kernel(uint64_t n, uint32_t W, const uint32_t* __restrict__ cnt, uint64_t* __restrict__ len) {
  uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) len[t] = cnt[t] > W ? cnt[t] : 0;
}

// The bucket's share of those targets' records (a warp per target) ...
__global__ void hub_copy_kernel(uint64_t n, uint32_t W, const uint32_t* __restrict__ cnt,
                                const uint64_t* __restrict__ off, const uint4* __restrict__ bucket,
                                uint4* __restrict__ out) {
  const uint64_t t = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (t >= n || cnt[t] <= W) return;
  for (uint32_t b = threadIdx.x & 31; b < W; b += 32) out[off[t] + b] = bucket[t * W + b];
}

// ... and the overflow list's.
__global__ void hub_scatter_kernel(uint64_t m, const uint4* __restrict__ ovf, const uint32_t* __restrict__ slot,
                                   const uint64_t* __restrict__ off, uint4* __restrict__ out) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const uint4 r = ovf[i];
  out[off[r.w] + slot[i]] = r;
}

__device__ __forceinline__ K96 rec_k96(const uint4& r) { return K96{rec_key(r), r.z}; }

// A target's P-th smallest distance over distinct ids of its pool and the records found so far lowers
// its bound: P entries at or below it fill the pool and its overflow slot, after which the radius is at
// most that distance, so a record beyond it is rejected whatever else arrives.  A pair's distance is the
// same wherever it is computed (the caller sees to that), so equal ids have equal keys.  The 64 smallest
// keys, whatever order the records arrived in, are kept over chunks of 32; targets of more records than
// a bucket holds keep their bound.  A warp per target.
constexpr uint32_t TIGHTEN_MAX_P = 48;
__global__ void __launch_bounds__(256) tighten_kernel(uint64_t n, uint32_t P, uint32_t W,
                                                      const uint32_t* __restrict__ cnt,
                                                      const uint4* __restrict__ bucket, const float* __restrict__ pd,
                                                      const uint32_t* __restrict__ pid,
                                                      const uint32_t* __restrict__ Lc, float* __restrict__ bound) {
  const uint64_t t = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t lane = threadIdx.x & 31;
  if (t >= n) return;
  const uint32_t L = Lc[t], B = cnt[t];
  if (L + B < P || B > W) return;
  uint64_t v[2] = {~0ull, ~0ull};  // the 64 smallest, ascending over v[0] then v[1]
  for (uint32_t b = 0; b < L + B; b += 32) {
    const uint32_t e = b + lane;
    uint64_t x = ~0ull;
    if (e < L) x = pack_key(pd[t * P + e], pid[t * P + e] & IDM);
    else if (e < L + B) x = rec_key(bucket[t * W + e - L]);
    const uint64_t worst = __shfl_sync(0xffffffffu, v[1], 31);
    if (__all_sync(0xffffffffu, x >= worst)) continue;
    x = warp_sort32(x);
    // v[1] and x, both ascending: the 32 smallest into v[1], then with v[0] likewise
    v[1] = warp_merge_min32(v[1], x);
    const uint64_t hi = shfl_idx(v[1], 31 - lane);  // bitonic split of v[0] (ascending) and v[1] reversed
    uint64_t lo0 = lt(hi, v[0]) ? hi : v[0], hi0 = lt(hi, v[0]) ? v[0] : hi;
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) {
      const bool lower = (lane & j) == 0;
      uint64_t y = shfl_xor(lo0, j);
      lo0 = (lower == lt(y, lo0)) ? y : lo0;
      y = shfl_xor(hi0, j);
      hi0 = (lower == lt(y, hi0)) ? y : hi0;
    }
    v[0] = lo0;
    v[1] = hi0;
  }
  uint32_t seen = 0;  // distinct keys before this register
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    uint64_t prev = __shfl_up_sync(0xffffffffu, v[r], 1);
    const uint64_t last = __shfl_sync(0xffffffffu, v[0], 31);
    if (lane == 0) prev = r == 0 ? ~v[0] : last;
    const uint32_t m = __ballot_sync(0xffffffffu, v[r] != ~0ull && v[r] != prev);
    const uint32_t mine = seen + __popc(m & ((2u << lane) - 1));
    if ((m >> lane & 1u) && mine == P) bound[t] = fminf(bound[t], key_dist(v[r]));
    seen += __popc(m);
  }
}

constexpr uint32_t MERGE_WARPS = 4;  // warps per merge block

// Records sorted at a time (a window): 64 for pools of up to 64 entries, which reject soon after as
// many, 256 for larger ones.
template <int NS>
struct Merge {
  static constexpr uint32_t WIN = NS <= 2 ? 64 : 256;
  static constexpr uint32_t WARP_BYTES = WIN * 12 + NS * 32 * 8;
};

// The pool of one node in a warp's shared memory, entries [0, L) ascending, slot P - 1 the overflow
// slot, with Neighbor::insert / InsertIntoKnn applied to it (base_index.hpp:37-61).
template <int NS>
struct Pool {
  float* pd;
  uint32_t* pid;
  uint8_t* found;
  uint32_t P, check_k, L;
  float rad;
  bool any_dist, rejected;
  K96 rej;

  // One record as the reference applies it; true when it is rejected (every later one is too).
  __device__ __forceinline__ bool apply(const K96 r) {
    const uint32_t lane = threadIdx.x & 31;
    const float d = key_dist(r.k);
    const uint32_t cand = key_id(r.k);
    if (d > rad) {
      rejected = true;
      rej = r;
      return true;
    }
    float v[NS], up[NS];
    uint32_t id[NS], upid[NS], i = 0, dup = 0;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const uint32_t e = s * 32 + lane;
      v[s] = pd[e];
      id[s] = pid[e];
      up[s] = e ? pd[e - 1] : 0.f;
      upid[s] = e ? pid[e - 1] : 0u;
      i += __popc(__ballot_sync(0xffffffffu, e < L && v[s] <= d));  // entries of [0, L) with dist <= d
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const uint32_t e = s * 32 + lane;
      dup |= __ballot_sync(0xffffffffu, (any_dist ? e < L : (e < i && v[s] == d)) && (id[s] & IDM) == cand);
    }
    uint32_t rank = L + 1;
    if (!dup) {  // [i, L) moves up by one; entry L (<= P - 1) receives entry L - 1
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const uint32_t e = s * 32 + lane;
        if (e > i && e <= L) {
          pd[e] = up[s];
          pid[e] = upid[s];
        } else if (e == i) {
          pd[e] = d;
          pid[e] = cand | FLAG;
        }
      }
      __syncwarp();
      rank = i;
      if (L + 1 < P) ++L;
      else rad = pd[L - 1];
    }
    if ((r.a & 1u) == 0 && rank < check_k && lane == 0) found[r.a >> 1] = 1;
    __syncwarp();
    return false;
  }

  // Up to 32 ascending records, one per lane (lanes >= m hold none); true when one is rejected.
  //
  // The records that land strictly inside the pool are placed at once: with `j` of the records before
  // it inserted and `pa` entries at or below its distance, a record's rank is pa + j (earlier records
  // are no larger, so all of them precede it), and an entry moves up by the records placed before it.
  // Duplicates are recognised among the entries and, as equal neighbours (with any_dist: equal ids),
  // among the records.  From the first record on for which this does not hold -- one that is rejected,
  // lands in the overflow slot, or whose duplicate may have left the pool -- they are applied one by one.
  __device__ __forceinline__ bool apply_batch(const K96 r, uint32_t m) {
    const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1;
    const float d = key_dist(r.k);
    const uint32_t cand = key_id(r.k);
    uint32_t pa = 0;  // entries with dist <= d
    {
      uint32_t hi = L;
      while (__any_sync(0xffffffffu, pa < hi)) {
        if (pa < hi) {
          const uint32_t mid = (pa + hi) >> 1;
          if (pd[mid] <= d) pa = mid + 1;
          else hi = mid;
        }
      }
    }
    bool dup = false;
    uint32_t at = 0;  // (any_dist) the duplicate entry
    if (any_dist) {
      for (uint32_t e = 0; e < L; e += 4) {
        const uint4 q = *reinterpret_cast<const uint4*>(pid + e);
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if ((w[c] & IDM) == cand && e + c < L) {
            dup = true;
            at = e + c;
          }
      }
      const uint32_t same = __match_any_sync(0xffffffffu, lane < m ? cand : ~lane);  // (ids are < 2^30)
      dup |= (same & below) != 0;
    } else {
      for (uint32_t e = pa; e > 0 && pd[e - 1] == d; --e)
        if ((pid[e - 1] & IDM) == cand) {
          dup = true;
          break;
        }
      __syncwarp();
      const uint64_t prev = __shfl_up_sync(0xffffffffu, r.k, 1);
      dup |= lane > 0 && prev == r.k;
    }
    const uint32_t valid = m >= 32 ? 0xffffffffu : (1u << m) - 1;
    const uint32_t j = __popc(__ballot_sync(0xffffffffu, !dup) & valid & below);
    const bool accept = d <= rad || j >= P - L;  // (the radius is an inner entry's after an insert at capacity)
    const bool ok = accept && pa + j < P - 1 && at + j < P - 1;
    const uint32_t bad = ~__ballot_sync(0xffffffffu, ok) & valid;
    const uint32_t f = bad ? __ffs(bad) - 1 : m;
    const bool mine = lane < f;
    if (mine && (r.a & 1u) == 0 && (dup ? min(L + j, P - 1) + 1 : pa + j) < check_k) found[r.a >> 1] = 1;
    const uint32_t J = __popc(__ballot_sync(0xffffffffu, mine && !dup));
    if (J) {
      const uint32_t pos = pa + j, end = min(L + J, P);
      uint32_t before = 0;
      float nv[NS];
      uint32_t ni[NS];
#pragma unroll
      for (int s = 0; s < NS; ++s) {  // slot x takes entry x - (records placed below x)
        const uint32_t word = __reduce_or_sync(0xffffffffu, mine && !dup && pos / 32 == (uint32_t)s ? 1u << (pos & 31) : 0u);
        const uint32_t x = s * 32 + lane;
        const uint32_t src = x < end ? x - min(x, before + __popc(word & below)) : x;
        nv[s] = pd[src];
        ni[s] = pid[src];
        before += __popc(word);
      }
      __syncwarp();
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        pd[s * 32 + lane] = nv[s];
        pid[s * 32 + lane] = ni[s];
      }
      __syncwarp();
      if (mine && !dup) {
        pd[pos] = d;
        pid[pos] = cand | FLAG;
      }
      __syncwarp();
      if (J >= P - L) rad = pd[P - 2];
      L = min(L + J, P - 1);
    }
    for (uint32_t u = f; u < m; ++u)
      if (apply(shfl_idx(r, u))) return true;
    return false;
  }
};

// Sorts m <= 32 NR records of the warp's window (keys wk, aux wa) in registers.
template <int NR>
__device__ __forceinline__ void sort_window(uint64_t* wk, uint32_t* wa, uint32_t m) {
  const uint32_t lane = threadIdx.x & 31;
  K96 v[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const uint32_t e = r * 32 + lane;
    v[r] = e < m ? K96{wk[e], wa[e]} : k96_max();
  }
  warp_sort_regs<NR>(v);
  __syncwarp();
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    wk[r * 32 + lane] = v[r].k;
    wa[r * 32 + lane] = v[r].a;
  }
  __syncwarp();
}

// Next 32 records of distance bits g in ascending (key, aux) order after `last`.  With `single` a lone id's
// copies count as its first record: a pass without sorting finds whether there is one id.
// (Not inlined: rare, and the code around its place runs for every node.)
static __device__ __noinline__ K96 next_batch(const uint4* __restrict__ rec, uint32_t B, uint32_t g, K96 last, bool first,
                                              bool single) {
  const uint32_t lane = threadIdx.x & 31;
  if (single) {
    K96 mn = k96_max();
    uint32_t mx = 0;
    for (uint32_t b = lane; b < B; b += 32) {
      if (rec[b].y != g) continue;
      const K96 y = rec_k96(rec[b]);
      if (!first && !lt(last, y)) continue;
      if (lt(y, mn)) mn = y;
      mx = max(mx, key_id(y.k));
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    mn = shfl_idx(warp_sort32(mn), 0);
    if (is_max(mn) || key_id(mn.k) == mx) return lane == 0 ? mn : k96_max();
  }
  K96 run = k96_max(), worst = run;  // the 32 smallest so far, and the largest of them
  for (uint32_t b = 0; b < B; b += 32) {
    K96 x = k96_max();
    if (b + lane < B) {
      const uint4 q = rec[b + lane];
      const K96 y = rec_k96(q);
      if (q.y == g && (first || lt(last, y))) x = y;
    }
    if (__all_sync(0xffffffffu, !lt(x, worst))) continue;
    x = warp_sort32(x);
    run = warp_merge_min32(run, x);
    worst = shfl_idx(run, 31);
  }
  return run;
}

// The records of distance bits g after `last`, for a pool full up to that distance (entries [0, P - 1), the
// radius and the last of them at it): each of them lands in the overflow slot or is a duplicate, so the
// last one that is none stays there, at a rank of P - 1 (a duplicate's is P; check_k is not P).
static __device__ __noinline__ void overflow_ties(const uint4* __restrict__ rec, uint32_t B, uint32_t g, K96 last,
                                                  bool first, float* pd, uint32_t* pid, uint32_t P, bool any_dist,
                                                  bool mark, uint8_t* __restrict__ found) {
  const uint32_t lane = threadIdx.x & 31;
  const float d = __uint_as_float(g);
  for (uint64_t limit = 1ull << 32; limit;) {  // the largest id below `limit`
    uint64_t mx = 0;                           // (+ 1; 0: none)
    for (uint32_t b = lane; b < B; b += 32) {
      const uint4 q = rec[b];
      if (q.y != g) continue;
      const K96 y = rec_k96(q);
      if (!first && !lt(last, y)) continue;
      if (q.x < limit) mx = max(mx, (uint64_t)q.x + 1);
      if (mark && limit == 1ull << 32 && !(q.z & 1u)) found[q.z >> 1] = 1;
    }
    const uint32_t top = __reduce_max_sync(0xffffffffu, (uint32_t)mx);  // (ids are < 2^30)
    if (!top) break;
    const uint32_t cand = top - 1;
    bool dup = false;
    for (uint32_t e = lane; e + 1 < P; e += 32) dup |= (any_dist || pd[e] == d) && (pid[e] & IDM) == cand;
    if (!__any_sync(0xffffffffu, dup)) {
      if (lane == 0) {
        pd[P - 1] = d;
        pid[P - 1] = cand | FLAG;
      }
      break;
    }
    limit = cand;
  }
  __syncwarp();
}

// One warp per target node: applies its records in ascending (dist, id, source, side) order until one
// is rejected.  The records are taken a window at a time: those below a distance chosen (by
// interpolation and bisection on the distance bits) so that at most WIN and, as a rule, at least half
// as many fall below it, sorted in registers and applied 32 at once (Pool::apply_batch); a pool of 30
// is done after one window of the 78 records per node and iteration that 1M x 128 has.  More than WIN
// records at one distance are pulled 32 at a time; from a pool of check_k entries on without the copies of
// a pair (found again from every common neighbour), which change nothing there: they are duplicates, or
// land in the overflow slot again, at a rank of check_k or more.  Once the pool is full up to their
// distance the rest of them are settled by one scan (overflow_ties: 100k rows of 16 kinds 64 ms, 1714 ms
// with all of them pulled).  A record equal to an earlier one in all four fields changes nothing, so the
// windows need not keep its copies apart.
// The reference rejects a candidate whose id sits among the entries of equal distance; a pair's
// distance is the same wherever the reference computes it, so that finds every repeat.  With
// any_dist a repeat is found at any distance: the tensor-core join's distances can differ in the
// last bits from the FP32 ones a pool entry was inserted with, and an equal-distance test would
// let the id in twice.
// Bound: instruction issue and the latency of the record reads.  (Hubs are the tail: one of 4800 records at
// 30 distances took 21M cycles with all copies pulled in order, 8 of its iteration's 10.8 ms.)  Sorting every record in shared memory
// and inserting them one by one took 40 ms of the 1M x 128 build's 8 iterations and 65 ms of 6
// iterations at 100k x 960 (P = 201).
template <int NS>
__global__ void __launch_bounds__(MERGE_WARPS * 32) merge_kernel(
    uint64_t n, uint32_t P, uint32_t check_k, bool any_dist, const uint32_t* __restrict__ cnt, uint32_t W,
    const uint4* __restrict__ bucket, const uint64_t* __restrict__ hub_off, const uint4* __restrict__ hub,
    float* __restrict__ pd, uint32_t* __restrict__ pid, uint32_t* __restrict__ Lc, float* __restrict__ radius,
    uint8_t* __restrict__ found, uint32_t* __restrict__ next_node, unsigned long long* __restrict__ nrec) {
  constexpr uint32_t WIN = Merge<NS>::WIN;
  extern __shared__ __align__(16) unsigned char merge_smem[];
  const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1;
  unsigned char* mine = merge_smem + (size_t)(threadIdx.x >> 5) * Merge<NS>::WARP_BYTES;
  uint64_t* wk = reinterpret_cast<uint64_t*>(mine);
  Pool<NS> pool;
  pool.pd = reinterpret_cast<float*>(mine + WIN * 8);
  pool.pid = reinterpret_cast<uint32_t*>(pool.pd + NS * 32);
  uint32_t* wa = pool.pid + NS * 32;
  pool.found = found;
  pool.P = P;
  pool.check_k = check_k;
  pool.any_dist = any_dist;
  unsigned long long records = 0;
  for (;;) {  // nodes taken from a shared counter as warps come free (their record counts differ)
    uint32_t tt = 0;
    if (lane == 0) tt = atomicAdd(next_node, 1u);
    const uint64_t t = __shfl_sync(0xffffffffu, tt, 0);
    if (t >= n) {
      if (lane == 0 && records) atomicAdd(nrec, records);
      return;
    }
    const uint32_t B = cnt[t];
    if (B == 0) continue;
    records += B;
    const uint4* rec = B <= W ? bucket + t * W : hub + hub_off[t];  // (the hub array holds targets of B > W)
    const uint64_t prow = t * P;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const uint32_t e = s * 32 + lane;
      pool.pd[e] = e < P ? pd[prow + e] : 0.f;
      pool.pid[e] = e < P ? pid[prow + e] : 0u;
    }
    pool.L = Lc[t];
    pool.rad = radius[t];
    pool.rejected = false;
    __syncwarp();

    uint32_t tlo = 0;  // every record below these distance bits is done
    bool stop = false, ties = false, first = true;  // ties: more than WIN records at distance bits tlo
    K96 last{0, 0};
    while (!stop) {
      uint32_t thi = 0xffffffffu, total = B;
      if (!ties && (B > WIN || tlo)) {
        uint32_t mn = 0xffffffffu, mx = 0;
        total = 0;
        for (uint32_t b = lane; b < B; b += 32) {
          const uint32_t q = rec[b].y;
          if (q >= tlo) {
            mn = min(mn, q);
            mx = max(mx, q);
            ++total;
          }
        }
        mn = __reduce_min_sync(0xffffffffu, mn);
        mx = __reduce_max_sync(0xffffffffu, mx);
        total = __reduce_add_sync(0xffffffffu, total);
        if (total == 0) break;
        if (total > WIN) {
          uint32_t lo = mn, hi = mx + 1, clo = 0, chi = total;  // records in [tlo, lo) and [tlo, hi)
          for (uint32_t it = 0; hi - lo > 1 && (clo == 0 || (clo < WIN / 2 && it < 8)); ++it) {
            uint32_t mid = lo + (hi - lo) / 2;
            if (!(it & 1)) mid = lo + (uint32_t)((float)(hi - lo) * ((float)(WIN * 3 / 4 - clo) / (float)(chi - clo)));
            mid = min(max(mid, lo + 1), hi - 1);
            uint32_t c = 0;
            for (uint32_t b = lane; b < B; b += 32) {
              const uint32_t q = rec[b].y;
              c += q >= tlo && q < mid;
            }
            c = __reduce_add_sync(0xffffffffu, c);
            if (c <= WIN) {
              lo = mid;
              clo = c;
            } else {
              hi = mid;
              chi = c;
            }
          }
          thi = lo;
          total = clo;
          ties = clo == 0;
          if (ties) tlo = lo;
        }
      }
      if (ties) {  // the next 32 of them
        const bool quiet = pool.L >= check_k;
        const float dt = __uint_as_float(tlo);
        if (pool.L == P - 1 && pool.rad == dt && pool.pd[P - 2] == dt && check_k != P) {  // nothing left but its last
          overflow_ties(rec, B, tlo, last, first, pool.pd, pool.pid, P, any_dist, check_k > P, found);
          ties = false;
          first = true;
          ++tlo;
          continue;
        }
        const K96 batch = next_batch(rec, B, tlo, last, first, quiet);
        total = __popc(__ballot_sync(0xffffffffu, !is_max(batch)));
        first = total == 0;
        if (first) {
          ties = false;
          ++tlo;
          continue;
        }
        last = shfl_idx(batch, total - 1);
        if (quiet) last.a = 0xffffffffu;  // past all its copies
        wk[lane] = batch.k;
        wa[lane] = batch.a;
        __syncwarp();
      } else {  // the records of [tlo, thi), sorted
        if (tlo == 0 && thi == 0xffffffffu) {
          for (uint32_t b = lane; b < B; b += 32) {
            const K96 y = rec_k96(rec[b]);
            wk[b] = y.k;
            wa[b] = y.a;
          }
        } else {
          uint32_t at = 0;
          for (uint32_t b = 0; b < B; b += 32) {
            const uint4 q = b + lane < B ? rec[b + lane] : make_uint4(0, 0xffffffffu, 0, 0);
            const bool take = b + lane < B && q.y >= tlo && q.y < thi;
            const uint32_t bal = __ballot_sync(0xffffffffu, take);
            if (take) {
              const uint32_t o = at + __popc(bal & below);
              wk[o] = rec_key(q);
              wa[o] = q.z;
            }
            at += __popc(bal);
          }
        }
        __syncwarp();
        if (WIN == 64 && total <= 32) sort_window<1>(wk, wa, total);
        else if (total <= 64) sort_window<2>(wk, wa, total);
        else if (WIN > 64) sort_window<(WIN > 64 ? 8 : 1)>(wk, wa, total);
      }
      for (uint32_t b = 0; b < total && !stop; b += 32) {
        const K96 batch = b + lane < total ? K96{wk[b + lane], wa[b + lane]} : k96_max();
        stop = pool.apply_batch(batch, min(32u, total - b));
      }
      if (ties) continue;
      if (thi == 0xffffffffu) break;
      tlo = thi;
    }
    if (pool.rejected && P < check_k) {
      // every record from `rej` on was rejected with rank P < check_k
      for (uint32_t b = lane; b < B; b += 32) {
        const K96 y = rec_k96(rec[b]);
        if (!lt(y, pool.rej) && (y.a & 1u) == 0) found[y.a >> 1] = 1;
      }
    }
    __syncwarp();
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const uint32_t e = s * 32 + lane;
      if (e < P) {
        pd[prow + e] = pool.pd[e];
        pid[prow + e] = pool.pid[e];
      }
    }
    if (lane == 0) {
      Lc[t] = pool.L;
      radius[t] = pool.rad;
    }
    __syncwarp();
  }
}

// =============================================================================================
// Update.
// =============================================================================================

// radius = pool[L].dist (the overflow slot); Range grows by up to S new entries for found nodes;
// radiusM = pool[Range-1].dist.  (update(), base_index.hpp:374-395)
__global__ void update_range_kernel(uint64_t n, uint32_t P, uint32_t S, const float* __restrict__ pd,
                                    const uint32_t* __restrict__ pid, const uint32_t* __restrict__ Lc,
                                    uint32_t* __restrict__ Range, float* __restrict__ radius,
                                    float* __restrict__ radiusM, const uint8_t* __restrict__ found) {
  uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  uint64_t row = t * P;
  radius[t] = pd[row + P - 1];
  uint32_t R = Range[t];
  if (found[t]) {
    uint32_t L = Lc[t];
    uint32_t maxl = R + S < L ? R + S : L;
    uint32_t c = 0, l = 0;
    while (l < maxl && c < S) {
      if (pid[row + l] & FLAG) ++c;
      ++l;
    }
    R = l;
    Range[t] = R;
  }
  radiusM[t] = pd[row + R - 1];
}

// Forward lists of node t (pool order) and reverse-edge counts per target; a warp per node, an entry per
// lane, so that the pool's rows are read in lines and the targets' radii and counts side by side.
// PASS 0: counts; PASS 1: writes reverse edges and clears the new flags.
template <int PASS>
__global__ void __launch_bounds__(256) update_lists_kernel(
    uint64_t n, uint32_t P, uint32_t cap, const float* __restrict__ pd, uint32_t* __restrict__ pid,
    const uint32_t* __restrict__ Range, const float* __restrict__ radiusM, uint32_t* __restrict__ new_ids,
    uint32_t* __restrict__ new_cnt, uint32_t* __restrict__ old_ids, uint32_t* __restrict__ old_cnt,
    uint32_t* __restrict__ rcnt, const uint32_t* __restrict__ roff, uint32_t* __restrict__ rcur,
    uint32_t* __restrict__ rbuf) {
  const uint64_t t = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1;
  if (t >= n) return;
  const uint64_t row = t * P;
  const uint32_t R = Range[t];
  uint32_t cn = 0, co = 0;
  for (uint32_t l0 = 0; l0 < R; l0 += 32) {
    const uint32_t l = l0 + lane;
    const bool in = l < R;
    const uint32_t v = in ? pid[row + l] : 0u, id = v & IDM;
    const bool isnew = in && (v & FLAG), isold = in && !(v & FLAG);
    const bool rev = in && pd[row + l] > radiusM[id];
    const uint64_t slot = isnew ? id : n + id;  // the target's new or old reverse list
    if (PASS == 0) {
      const uint32_t bn = __ballot_sync(0xffffffffu, isnew), bo = __ballot_sync(0xffffffffu, isold);
      if (isnew) new_ids[t * cap + cn + __popc(bn & below)] = id;
      if (isold) old_ids[t * cap + co + __popc(bo & below)] = id;
      cn += __popc(bn);
      co += __popc(bo);
      if (rev) atomicAdd(&rcnt[slot], 1u);
    } else {
      if (rev) rbuf[roff[slot] + atomicAdd(&rcur[slot], 1u)] = (uint32_t)t;
      if (isnew) pid[row + l] = id;  // flag cleared
    }
  }
  if (PASS == 0 && lane == 0) {
    new_cnt[t] = cn;
    old_cnt[t] = co;
  }
}

// One warp per (target, list): the reverse sources, sorted by id, or -- when more than `rcap` --
// the rcap sources with the smallest (hash, id), in that order; appended to the list.
__global__ void update_reverse_kernel(uint64_t n, uint32_t cap, uint32_t rcap, uint64_t seed, uint32_t iter,
                                      const uint32_t* __restrict__ rcnt, const uint32_t* __restrict__ roff,
                                      const uint32_t* __restrict__ rbuf, uint32_t* __restrict__ new_ids,
                                      uint32_t* __restrict__ new_cnt, uint32_t* __restrict__ old_ids,
                                      uint32_t* __restrict__ old_cnt) {
  uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  uint32_t lane = threadIdx.x & 31;
  if (w >= 2 * n) return;
  uint64_t t = w % n;
  bool is_old = w >= n;
  uint32_t* ids = (is_old ? old_ids : new_ids) + t * cap;
  uint32_t* cntp = (is_old ? old_cnt : new_cnt) + t;
  const uint32_t B = rcnt[w], c0 = *cntp, o0 = roff[w];  // (three loads in flight)
  if (B == 0) return;
  const uint32_t* src = rbuf + o0;
  bool sample = rcap && B > rcap;
  if (B <= 32 && !sample) {  // each source's rank counted: 8 iterations of 1M x 128 in 6.6 ms, 8.2 with a sort
    const uint32_t v = lane < B ? src[lane] : 0xffffffffu;
    uint32_t rank = 0;
#pragma unroll 4
    for (uint32_t i = 0; i < B; ++i) {
      const uint32_t o = __shfl_sync(0xffffffffu, v, i);
      rank += o < v || (o == v && i < lane);
    }
    if (lane < B) ids[c0 + rank] = v;
    if (lane == 0) *cntp = c0 + B;
    return;
  }
  uint32_t take = sample ? rcap : B;
  uint64_t tag = is_old ? TAG_ROLD : TAG_RNEW;
  uint64_t last = 0;
  bool first = true;
  uint32_t done = 0;
  while (done < take) {
    uint64_t run = ~0ULL;
    for (uint32_t b = 0; b < B; b += 32) {
      uint64_t x = ~0ULL;
      if (b + lane < B) {
        uint32_t sv = src[b + lane];
        uint64_t k = sample ? (((hash4(seed, tag, iter, t, sv) >> 32) << 32) | sv) : (uint64_t)sv;
        if (first || k > last) x = k;
      }
      if (__all_sync(0xffffffffu, x == ~0ULL)) continue;
      x = warp_sort32(x);
      run = warp_merge_min32(run, x);
    }
    first = false;
    // a source listed twice (a pool holding an id twice) leaves fewer distinct keys than take:
    // the list ends at the last one
    uint32_t got = min(32u, take - done);
    got = min(got, (uint32_t)__popc(__ballot_sync(0xffffffffu, run != ~0ULL)));
    if (lane < got) ids[c0 + done + lane] = (uint32_t)run;
    if (got == 0) break;
    last = __shfl_sync(0xffffffffu, run, got - 1);
    done += got;
  }
  if (lane == 0) *cntp = c0 + done;
}

__global__ void export_graph_kernel(uint64_t n, uint32_t P, uint32_t K, const uint32_t* __restrict__ pid,
                                    uint32_t* __restrict__ gids, uint64_t* __restrict__ gptr) {
  uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g < n * K) gids[g] = pid[(g / K) * P + (g % K)] & IDM;
  if (g <= n) gptr[g] = g * K;
}

// =============================================================================================
// Host drivers.
// =============================================================================================

static unsigned blocks_for(uint64_t threads, int per_block) {
  return (unsigned)((threads + per_block - 1) / per_block);
}

__global__ void widen_kernel(const uint32_t* __restrict__ in, uint64_t* __restrict__ out, uint64_t n) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = in[i];
}

static int merge_level_check(efg_index* idx, int32_t* min_level) {
  Forest& F = idx->forest;
  TreeView tv{F.nodes.p, F.n_left.p, F.n_right.p, F.n_level.p, F.n_tree.p, F.n_start.p, F.n_end.p, F.leaves.p, F.n};
  LocalBuf<int32_t> d(idx->stream);
  EFG_TRY(d.reserve(1));
  int32_t big = 0x7fffffff;
  EFG_CUDA(cudaMemcpyAsync(d.p, &big, 4, cudaMemcpyHostToDevice, idx->stream));
  min_leaf_level_kernel<<<blocks_for(F.nnodes, 256), 256, 0, idx->stream>>>(tv, F.nnodes, idx->bp.trees_build, d.p);
  EFG_CUDA(cudaGetLastError());
  EFG_CUDA(cudaMemcpyAsync(min_level, d.p, 4, cudaMemcpyDeviceToHost, idx->stream));
  EFG_CUDA(cudaStreamSynchronize(idx->stream));
  return EFG_OK;
}

// The first join keeps every pair of the seeded lists, 2 S (2S - 1) records per node on average (380 for
// S = 10), of which a pool of P - 1 takes a few dozen.  Where an eighth of the nodes leaves more than P
// entries per target it runs in parts: of every FIRST_STEP nodes those from one entry of FIRST_PARTS to the
// next, the targets' bounds tightened in between (1M x 128: 8.7 ms; in two parts, 1 and 7, 10.9 ms with
// half as many records again).  On the tensor cores only where their distances are exact: else an id may be
// found at two distances, and would count twice.
constexpr uint32_t FIRST_STEP = 8, FIRST_PARTS[] = {0, 1, 3, 8};
static uint64_t first_mean(const efg_build_params& bp) { return 2ull * bp.S * (2 * bp.S - 1); }
static bool first_in_parts(const efg_index* idx, const NNDev& S) {
  const efg_build_params& bp = idx->bp;
  const bool exact = idx->build_precision != EFG_PRECISION_BF16 || S.jexact;
  return exact && S.P <= TIGHTEN_MAX_P && first_mean(bp) / FIRST_STEP + bp.S >= S.P + S.P / 4;
}

// The tensor-core join's rows, and whether its distances are exact (once per build; nothing in FP32).
static int prepare_tc(efg_index* idx, NNDev& S) {
  if (idx->build_precision != EFG_PRECISION_BF16 || S.jterms) return EFG_OK;
  cudaStream_t s = idx->stream;
  const uint64_t n = S.n, W = (idx->dim + 63) / 64 * 64;
  EFG_TRY(S.jhi.reserve(n * W));
  EFG_TRY(S.jlo.reserve(n * W));
  EFG_TRY(S.jnorm.reserve(n));
  EFG_TRY(S.jflag.reserve(3));
  EFG_TRY(S.jmid.reserve(n + 1));
  EFG_TRY(tc_join_prepare(idx->d_base, n, idx->dim, idx->ld, S.jhi.p, S.jlo.p, S.jnorm.p, S.jflag.p, s));
  int flags[3] = {0, 0, 0};
  EFG_CUDA(cudaMemcpyAsync(flags, S.jflag.p, 12, cudaMemcpyDeviceToHost, s));
  EFG_CUDA(cudaStreamSynchronize(s));
  S.jterms = flags[0] ? 3 : 1;
  S.jexact = !flags[0] && !flags[2];
  return EFG_OK;
}

// Bucket width: about the records a node receives in the first join, or five pools' worth where pools
// are large (later joins then bring more), then (see the end of an iteration) three times the last
// iteration's mean as far as the buffer reaches -- it grows only when the mean itself nears its width:
// a GB costs about 0.8 ms to allocate and free, more than some overflowing hubs do -- within a quarter
// of the memory free at the start; the rest goes to the overflow list.
static int first_width(efg_index* idx, NNDev& S) {
  if (S.W || S.scarce) return EFG_OK;
  EFG_TRY(prepare_tc(idx, S));  // (the first join in parts or not: up to twice the records)
  const efg_build_params& bp = idx->bp;
  size_t free_b = 0, total_b = 0;
  EFG_CUDA(cudaMemGetInfo(&free_b, &total_b));
  S.bucket_cap = std::max<uint64_t>(1, (uint64_t)free_b / 4 / sizeof(uint4) / S.n);
  const uint64_t mean = first_mean(bp);
  const uint64_t expect = first_in_parts(idx, S) ? mean / FIRST_STEP + 6 * S.P
                                                 : std::max<uint64_t>(mean + mean / 4, S.P > 64 ? 5 * S.P : 0);
  S.W = (uint32_t)std::min<uint64_t>(S.bucket_cap, expect + 32);
  // (a list above an eighth of the free memory grows to its size only when a join finds that many)
  S.ovf_cap = std::max<uint64_t>(std::min<uint64_t>(S.n * (expect / 4 + 8), (uint64_t)free_b / 8 / 20), 1 << 16);
  if (S.ovf.reserve(S.ovf_cap) != EFG_OK || S.ovf_slot.reserve(S.ovf_cap) != EFG_OK) S.run_scarce();
  return EFG_OK;
}

static int nnd_init_device(efg_index* idx, NNDev& S) {
  Forest& F = idx->forest;
  cudaStream_t s = idx->stream;
  const efg_build_params& bp = idx->bp;
  if (F.ntrees < bp.trees_build) return fail(EFG_ERR_STATE, "fewer trees than trees_build");
  int32_t minlev = 0;
  EFG_TRY(merge_level_check(idx, &minlev));
  idx->bstats.max_merge_depth = -1;
  if (minlev < (int32_t)bp.merge_level) {
    idx->bstats.max_merge_depth = minlev - 1;
    return fail(EFG_ERR_MERGE_LEVEL,
                "merge level deeper than tree, max merge deepth is" + std::to_string(minlev - 1));
  }
  uint64_t n = idx->n;
  uint32_t ld4 = idx->ld / 4;
  uint32_t cap = std::max(bp.L, 2 * bp.S) + bp.reverse_cap;
  EFG_TRY(nn_alloc(S, n, bp.L, cap));
  TreeView tv{F.nodes.p, F.n_left.p, F.n_right.p, F.n_level.p, F.n_tree.p, F.n_start.p, F.n_end.p, F.leaves.p, F.n};
  // task offsets over nodes
  EFG_TRY(S.task_len.reserve(F.nnodes + 1));
  EFG_TRY(S.off64.reserve(std::max<uint64_t>(F.nnodes, n) + 1));
  EFG_TRY(S.scan64.reserve(scan_tmp_elems<uint64_t>(std::max<uint64_t>(F.nnodes, n)) + 1));
  merge_task_len_kernel<<<blocks_for(F.nnodes, 256), 256, 0, s>>>(tv, F.nnodes, bp.trees_build,
                                                                   (int32_t)bp.merge_level, S.task_len.p);
  EFG_CUDA(cudaGetLastError());
  EFG_TRY(device_scan<uint64_t>(S.task_len.p, F.nnodes, S.off64.p, S.scan64.p, s));
  uint64_t ntasks = 0;
  EFG_CUDA(cudaMemcpyAsync(&ntasks, S.off64.p + F.nnodes, 8, cudaMemcpyDeviceToHost, s));
  EFG_CUDA(cudaStreamSynchronize(s));
  // per-target record counts -> offsets
  EFG_TRY(S.cnt.reserve(n));
  EFG_TRY(S.cursor.reserve(n));
  LocalBuf<uint64_t> cnt64(s), off64(s);
  EFG_TRY(cnt64.reserve(n));
  EFG_TRY(off64.reserve(n + 1));
  LocalBuf<unsigned long long> nd(s);
  EFG_TRY(nd.reserve(1));
  EFG_CUDA(cudaMemsetAsync(S.cnt.p, 0, n * 4, s));
  EFG_CUDA(cudaMemsetAsync(S.cursor.p, 0, n * 4, s));
  EFG_CUDA(cudaMemsetAsync(nd.p, 0, 8, s));
  unsigned rgrid = (unsigned)std::min<uint64_t>(blocks_for(ntasks * 32, 256), 152ull * 64);
  // what pass 0 keeps for the record pass: the point, the leaf and maxl distances per task (when
  // that stays within 4 GiB; otherwise pass 1 routes again)
  uint32_t maxl = 0;
  {
    LocalBuf<uint32_t> ml(s);
    EFG_TRY(ml.reserve(1));
    EFG_CUDA(cudaMemsetAsync(ml.p, 0, 4, s));
    max_leaf_kernel<<<blocks_for(F.nnodes, 256), 256, 0, s>>>(tv, F.nnodes, ml.p);
    EFG_CUDA(cudaMemcpyAsync(&maxl, ml.p, 4, cudaMemcpyDeviceToHost, s));
    EFG_CUDA(cudaStreamSynchronize(s));
  }
  const bool keep = ntasks && maxl && ntasks * (uint64_t)(maxl + 2) * 4 <= (4ull << 30);
  LocalBuf<uint32_t> task_p(s);
  LocalBuf<int32_t> task_leaf(s);
  LocalBuf<float> task_d(s);
  if (keep) {
    EFG_TRY(task_p.reserve(ntasks));
    EFG_TRY(task_leaf.reserve(ntasks));
    EFG_TRY(task_d.reserve(ntasks * maxl));
  }
  EFG_TRY(make_bytes(idx));
  ByteRows br{nullptr, nullptr, 0, 0};
  if (idx->bytes_state == 1) {
    br = ByteRows{idx->bytes.p, idx->bnorm.p, idx->ldb / 16, 0};
    while ((1u << br.gshift) < br.chunks) ++br.gshift;
  }
  if (ntasks) {
    auto route = br.rows ? merge_route_kernel<0, true> : merge_route_kernel<0, false>;
    route<<<rgrid, 256, 0, s>>>(idx->d_base, ld4, br, tv, S.off64.p, F.nnodes, ntasks, S.cnt.p, nullptr, nullptr,
                                nullptr, nd.p, task_p.p, task_leaf.p, task_d.p, maxl);
    EFG_CUDA(cudaGetLastError());
  }
  widen_kernel<<<blocks_for(n, 256), 256, 0, s>>>(S.cnt.p, cnt64.p, n);
  EFG_CUDA(cudaGetLastError());
  EFG_TRY(device_scan<uint64_t>(cnt64.p, n, off64.p, S.scan64.p, s));
  uint64_t nrec = 0;
  unsigned long long ndist = 0;
  EFG_CUDA(cudaMemcpyAsync(&nrec, off64.p + n, 8, cudaMemcpyDeviceToHost, s));
  EFG_CUDA(cudaMemcpyAsync(&ndist, nd.p, 8, cudaMemcpyDeviceToHost, s));
  EFG_CUDA(cudaStreamSynchronize(s));
  idx->bstats.merge_distances = ndist;
  // the leaf merge's records in the join's bucket buffer, allocated once for both
  EFG_TRY(first_width(idx, S));
  if (S.bucket.reserve(std::max<uint64_t>(n * S.W, nrec / 2 + 1)) != EFG_OK) EFG_TRY(S.room(S.bucket, nrec / 2 + 1));
  uint64_t* rec_key_buf = reinterpret_cast<uint64_t*>(S.bucket.p);
  if (keep) {
    merge_emit_kernel<<<(unsigned)std::min<uint64_t>(blocks_for(ntasks, 256), 152ull * 64), 256, 0, s>>>(
        tv, ntasks, task_p.p, task_leaf.p, task_d.p, maxl, off64.p, S.cursor.p, rec_key_buf);
    EFG_CUDA(cudaGetLastError());
  } else if (ntasks) {
    auto route = br.rows ? merge_route_kernel<1, true> : merge_route_kernel<1, false>;
    route<<<rgrid, 256, 0, s>>>(idx->d_base, ld4, br, tv, S.off64.p, F.nnodes, ntasks, nullptr, off64.p, S.cursor.p,
                                rec_key_buf, nullptr, nullptr, nullptr, nullptr, 0);
    EFG_CUDA(cudaGetLastError());
  }
  init_select_kernel<<<blocks_for(n * 32, 256), 256, 0, s>>>(
      idx->d_base, ld4, n, bp.S, S.P, cap, bp.seed, S.cnt.p, off64.p, rec_key_buf, S.pd.p, S.pid.p, S.Lc.p,
      S.Range.p, S.radius.p, S.radiusM.p, S.found.p, S.new_ids.p, S.new_cnt.p, S.old_cnt.p);
  EFG_CUDA(cudaGetLastError());
  EFG_CUDA(cudaStreamSynchronize(s));
  return EFG_OK;
}

static int nnd_iterate_device(efg_index* idx, NNDev& S, uint32_t iter, uint64_t* pairs_out, uint64_t* recs_out) {
  cudaStream_t s = idx->stream;
  const efg_build_params& bp = idx->bp;
  uint64_t n = S.n;
  // ---- join
  const bool tc = idx->build_precision == EFG_PRECISION_BF16;
  EFG_TRY(prepare_tc(idx, S));
  EFG_TRY(first_width(idx, S));
  if (S.scarce) S.bucket.release();  // (the leaf merge's records)
  EFG_TRY(S.room(S.off64, n + 1));
  EFG_TRY(S.room(S.scan64, scan_tmp_elems<uint64_t>(2 * n) + 1));
  EFG_TRY(S.room(S.task_len, n + 1));
  EFG_TRY(S.room(S.cnt, 2 * n));
  EFG_TRY(S.room(S.bound, n));
  EFG_TRY(S.room(S.totals, 4));
  EFG_TRY(S.room(S.jctr, 8));
  if (!tc) EFG_TRY(make_bytes(idx));
  if (tc || idx->bytes_state != 1) EFG_TRY(S.room(S.jbig, n + 1));
  if (!S.scarce && S.bucket.reserve(n * S.W) != EFG_OK) S.run_scarce();
  int sms = 152, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  EFG_CUDA(cudaMemsetAsync(S.found.p, 0, n, s));
  uint64_t npairs = 0, novf = 0, large = 0;
  if (!S.scarce && S.last_ovf + S.last_ovf / 4 > S.ovf_cap) {  // lists that fill up grow before a join has to run again
    const uint64_t want = S.last_ovf + S.last_ovf / 2;
    if (S.ovf.reserve(want) == EFG_OK && S.ovf_slot.reserve(want) == EFG_OK) S.ovf_cap = want;
    else if (S.ovf.reserve(S.ovf_cap) != EFG_OK || S.ovf_slot.reserve(S.ovf_cap) != EFG_OK) S.run_scarce();
  }
  bool counted = false;  // (scarce memory) the records of the second run have their places
  for (;;) {  // again when the overflow list was too short for its records, and with scarce memory
    EFG_CUDA(cudaMemsetAsync(S.totals.p, 0, 32, s));
    EFG_CUDA(cudaMemsetAsync(S.cnt.p, 0, n * 4, s));
    EFG_CUDA(cudaMemsetAsync(S.jctr.p, 0, 32, s));
    bound_kernel<<<blocks_for(n, 256), 256, 0, s>>>(n, S.P, S.pd.p, S.Lc.p, S.radius.p, S.new_cnt.p, S.old_cnt.p,
                                                    S.bound.p, S.totals.p);
    EFG_CUDA(cudaGetLastError());
    const RecordSink sink{S.cnt.p, S.bucket.p, counted ? S.ovfrec.p : S.ovf.p, S.ovf_slot.p, S.totals.p + 2, S.ovf_cap,
                          S.W, counted ? S.off64.p : nullptr};
    if (tc) EFG_CUDA(cudaMemsetAsync(S.jflag.p + 1, 0, 4, s));
    auto join = [&](const NodeSet& set) -> int {
      EFG_CUDA(cudaMemsetAsync(S.jctr.p + 1, 0, 12, s));
      if (!tc && idx->bytes_state == 1)
        return join_bytes(idx->bytes.p, idx->bnorm.p, n, idx->ldb, S.cap, S.P, bp.check_k, S.new_ids.p, S.new_cnt.p,
                          S.old_ids.p, S.old_cnt.p, S.bound.p, sink, S.found.p, S.jctr.p + 1, set, s);
      EFG_CUDA(cudaMemsetAsync(S.jbig.p, 0, 4, s));
      if (!tc)
        return join_fp32(idx->d_base, n, idx->ld, S.cap, S.P, bp.check_k, S.new_ids.p, S.new_cnt.p, S.old_ids.p,
                         S.old_cnt.p, S.bound.p, sink, S.found.p, S.jctr.p + 1, S.jbig.p, set, s);
      EFG_CUDA(cudaMemsetAsync(S.jmid.p, 0, 4, s));
      return tc_join(S.jhi.p, S.jlo.p, S.jnorm.p, n, idx->dim, S.jterms, S.cap, S.P, bp.check_k, S.new_ids.p,
                     S.new_cnt.p, S.old_ids.p, S.old_cnt.p, S.bound.p, sink, S.found.p, S.jctr.p + 1, S.jmid.p,
                     S.jbig.p, S.totals.p + 3, S.jflag.p + 1, set, s);
    };
    if (iter == 0 && !S.scarce && first_in_parts(idx, S)) {
      for (uint32_t p = 0; p + 1 < sizeof(FIRST_PARTS) / 4; ++p) {
        if (p) {
          tighten_kernel<<<blocks_for(n * 32, 256), 256, 0, s>>>(n, S.P, S.W, S.cnt.p, S.bucket.p, S.pd.p, S.pid.p,
                                                                 S.Lc.p, S.bound.p);
          EFG_CUDA(cudaGetLastError());
        }
        EFG_TRY(join(NodeSet{FIRST_STEP, FIRST_PARTS[p], FIRST_PARTS[p + 1] - FIRST_PARTS[p]}));
      }
    } else {
      EFG_TRY(join(NodeSet{1, 0, 1}));
    }
    unsigned long long tot[4] = {0, 0, 0, 0};
    EFG_CUDA(cudaMemcpyAsync(tot, S.totals.p, 32, cudaMemcpyDeviceToHost, s));
    int jerr = 0;  // the tensor-core join's error word
    if (tc) EFG_CUDA(cudaMemcpyAsync(&jerr, S.jflag.p + 1, 4, cudaMemcpyDeviceToHost, s));
    EFG_CUDA(cudaStreamSynchronize(s));
    if (jerr & 4) return fail(EFG_ERR_ARG, "tensor-core join: a join list holds an id >= n");
    if (jerr) return fail(EFG_ERR_DEVICE_LIMIT, "tensor-core join: a wait ran out on the device");
    npairs = tot[0];
    large = tot[3];
    if (counted) {
      if (tot[2] != novf) return fail(EFG_ERR_STATE, "NN-descent: a join's two runs found different records");
      break;
    }
    novf = tot[2];
    if (!S.scarce && novf > S.ovf_cap) {
      ++idx->bstats.join_reruns;
      S.ovf_cap = novf + novf / 4;
      if (S.ovf.reserve(S.ovf_cap) != EFG_OK || S.ovf_slot.reserve(S.ovf_cap) != EFG_OK) S.run_scarce();
      continue;
    }
    if (novf == 0) break;
    // one array for the hub targets' records (scarce: for all of them, which the second run writes)
    hub_len_kernel<<<blocks_for(n, 256), 256, 0, s>>>(n, S.W, S.cnt.p, S.task_len.p);
    EFG_CUDA(cudaGetLastError());
    EFG_TRY(device_scan<uint64_t>(S.task_len.p, n, S.off64.p, S.scan64.p, s));
    uint64_t hub_total = 0;
    EFG_CUDA(cudaMemcpyAsync(&hub_total, S.off64.p + n, 8, cudaMemcpyDeviceToHost, s));
    EFG_CUDA(cudaStreamSynchronize(s));
    if (S.scarce) {
      EFG_TRY(S.ovfrec.reserve(hub_total));
      counted = true;
      continue;
    }
    if (S.ovfrec.reserve(hub_total) != EFG_OK) {
      S.run_scarce();
      continue;
    }
    hub_copy_kernel<<<blocks_for(n * 32, 256), 256, 0, s>>>(n, S.W, S.cnt.p, S.off64.p, S.bucket.p, S.ovfrec.p);
    EFG_CUDA(cudaGetLastError());
    hub_scatter_kernel<<<blocks_for(novf, 256), 256, 0, s>>>(novf, S.ovf.p, S.ovf_slot.p, S.off64.p, S.ovfrec.p);
    EFG_CUDA(cudaGetLastError());
    break;
  }
  S.last_ovf = novf;
  idx->bstats.join_large_nodes += large;
  auto launch_merge = [&](auto kern, uint32_t warp_bytes) -> int {
    const size_t msmem = (size_t)MERGE_WARPS * warp_bytes;
    EFG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)msmem));
    int per = 1;
    EFG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, MERGE_WARPS * 32, msmem));
    const unsigned grid = (unsigned)std::min<uint64_t>(blocks_for(n * 32, MERGE_WARPS * 32),
                                                       (uint64_t)sms * std::max(per, 1));
    kern<<<grid, MERGE_WARPS * 32, msmem, s>>>(n, S.P, bp.check_k, tc, S.cnt.p, S.W, S.bucket.p, S.off64.p,
                                               S.ovfrec.p, S.pd.p, S.pid.p, S.Lc.p, S.radius.p, S.found.p,
                                               S.jctr.p, S.totals.p + 1);
    return EFG_OK;
  };
  if (S.P <= 32) EFG_TRY(launch_merge(merge_kernel<1>, Merge<1>::WARP_BYTES));
  else if (S.P <= 64) EFG_TRY(launch_merge(merge_kernel<2>, Merge<2>::WARP_BYTES));
  else if (S.P <= 128) EFG_TRY(launch_merge(merge_kernel<4>, Merge<4>::WARP_BYTES));
  else EFG_TRY(launch_merge(merge_kernel<8>, Merge<8>::WARP_BYTES));
  EFG_CUDA(cudaGetLastError());
  // ---- update
  update_range_kernel<<<blocks_for(n, 256), 256, 0, s>>>(n, S.P, bp.S, S.pd.p, S.pid.p, S.Lc.p, S.Range.p,
                                                         S.radius.p, S.radiusM.p, S.found.p);
  EFG_CUDA(cudaGetLastError());
  EFG_TRY(S.room(S.rcnt, 2 * n));  // (the records have been merged)
  EFG_TRY(S.room(S.rcur, 2 * n));
  EFG_TRY(S.room(S.roff, 2 * n + 1));
  EFG_TRY(S.room(S.scan32, scan_tmp_elems<uint32_t>(2 * n) + 1));
  EFG_CUDA(cudaMemsetAsync(S.rcnt.p, 0, 2 * n * 4, s));
  EFG_CUDA(cudaMemsetAsync(S.rcur.p, 0, 2 * n * 4, s));
  update_lists_kernel<0><<<blocks_for(n * 32, 256), 256, 0, s>>>(n, S.P, S.cap, S.pd.p, S.pid.p, S.Range.p, S.radiusM.p,
                                                            S.new_ids.p, S.new_cnt.p, S.old_ids.p, S.old_cnt.p,
                                                            S.rcnt.p, nullptr, nullptr, nullptr);
  EFG_CUDA(cudaGetLastError());
  EFG_TRY(device_scan<uint32_t>(S.rcnt.p, 2 * n, S.roff.p, S.scan32.p, s));
  uint32_t nrev = 0;
  EFG_CUDA(cudaMemcpyAsync(&nrev, S.roff.p + 2 * n, 4, cudaMemcpyDeviceToHost, s));
  EFG_CUDA(cudaStreamSynchronize(s));
  EFG_TRY(S.room(S.rbuf, (uint64_t)nrev + 1));
  update_lists_kernel<1><<<blocks_for(n * 32, 256), 256, 0, s>>>(n, S.P, S.cap, S.pd.p, S.pid.p, S.Range.p, S.radiusM.p,
                                                            S.new_ids.p, S.new_cnt.p, S.old_ids.p, S.old_cnt.p,
                                                            S.rcnt.p, S.roff.p, S.rcur.p, S.rbuf.p);
  EFG_CUDA(cudaGetLastError());
  update_reverse_kernel<<<blocks_for(2 * n * 32, 256), 256, 0, s>>>(n, S.cap, bp.reverse_cap, bp.seed, iter, S.rcnt.p,
                                                                    S.roff.p, S.rbuf.p, S.new_ids.p, S.new_cnt.p,
                                                                    S.old_ids.p, S.old_cnt.p);
  EFG_CUDA(cudaGetLastError());
  unsigned long long nrec = 0;
  EFG_CUDA(cudaMemcpyAsync(&nrec, S.totals.p + 1, 8, cudaMemcpyDeviceToHost, s));
  EFG_CUDA(cudaStreamSynchronize(s));
  const uint64_t avg = nrec / n, have = S.bucket.cap / n;
  if (!S.scarce)
    S.W = (uint32_t)std::max<uint64_t>(
        1, std::min<uint64_t>({S.bucket_cap, 3 * avg + 64, std::max<uint64_t>(have, avg + avg / 4 + 32)}));
  if (pairs_out) *pairs_out = npairs;
  if (recs_out) *recs_out = nrec;
  return EFG_OK;
}

int build_graph_device(efg_index* idx) {
  NvtxRange range("efg: build graph");
  cudaStream_t s = idx->stream;
  idx->bstats = efg_build_stats{};
  idx->graph.release();
  ScopedEvents<4> evs;
  cudaEvent_t* ev = evs.e;
  cudaEventRecord(ev[0], s);
  {
    NvtxRange r("efg: build trees");
    EFG_TRY(build_forest(idx, idx->bp.trees));
  }
  cudaEventRecord(ev[1], s);
  NNDev S(idx->stream);
  int rc;
  {
    NvtxRange r("efg: leaf-merge init");
    rc = nnd_init_device(idx, S);
  }
  if (rc != EFG_OK) {
      return rc;
  }
  cudaEventRecord(ev[2], s);
  uint64_t pairs = 0, recs = 0;
  for (uint32_t it = 0; it < idx->bp.epochs; ++it) {
    uint64_t p = 0, r = 0;
    NvtxRange range_it("efg: nn-descent iteration");
    rc = nnd_iterate_device(idx, S, it, &p, &r);
    if (rc != EFG_OK) {
          return rc;
    }
    pairs += p;
    recs += r;
  }
  // export gs: first K pool ids of every node (refineGraph, base_index.hpp:469-479)
  uint64_t n = idx->n;
  uint32_t K = idx->bp.K;
  Graph& g = idx->graph;
  EFG_TRY(g.ids.reserve(n * K));
  EFG_TRY(g.ptr.reserve(n + 1));
  export_graph_kernel<<<blocks_for(n * K + 1, 256), 256, 0, s>>>(n, S.P, K, S.pid.p, g.ids.p, g.ptr.p);
  EFG_CUDA(cudaGetLastError());
  cudaEventRecord(ev[3], s);
  EFG_CUDA(cudaStreamSynchronize(s));
  g.n = n;
  g.nnz = n * K;
  g.fixed_k = K;
  g.max_deg = K;
  g.valid = true;
  float a = 0, b = 0, c = 0;
  cudaEventElapsedTime(&a, ev[0], ev[1]);
  cudaEventElapsedTime(&b, ev[1], ev[2]);
  cudaEventElapsedTime(&c, ev[2], ev[3]);
  idx->bstats.trees_ms = a;
  idx->bstats.init_ms = b;
  idx->bstats.refine_ms = c;
  idx->bstats.total_ms = a + b + c;
  idx->bstats.join_pairs = pairs;
  idx->bstats.join_records = recs;
  return EFG_OK;
}

// ---- host-state entry points (state-level parity) ----------------------------------------------

static int state_to_device(efg_index* idx, NNDev& S, const efg_nnd_host_state* st) {
  if (st->n != idx->n || st->L != idx->bp.L) return fail(EFG_ERR_ARG, "state does not match the index");
  EFG_TRY(nn_alloc(S, st->n, st->L, st->cap));
  EFG_CUDA(cudaStreamSynchronize(idx->stream));  // the copies below run on the default stream
  uint64_t n = st->n, np = n * S.P;
  std::vector<uint32_t> pid(np);
  for (uint64_t i = 0; i < np; ++i) pid[i] = st->pool_id[i] | (st->pool_flag[i] ? FLAG : 0u);
  EFG_CUDA(cudaMemcpy(S.pd.p, st->pool_dist, np * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(S.pid.p, pid.data(), np * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(S.Lc.p, st->Lcur, n * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(S.Range.p, st->Range, n * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(S.radius.p, st->radius, n * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(S.radiusM.p, st->radiusM, n * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(S.found.p, st->found, n, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(S.new_ids.p, st->new_ids, n * st->cap * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(S.new_cnt.p, st->new_cnt, n * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(S.old_ids.p, st->old_ids, n * st->cap * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(S.old_cnt.p, st->old_cnt, n * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaStreamSynchronize(0));
  return EFG_OK;
}

static int state_to_host(NNDev& S, efg_nnd_host_state* st) {
  uint64_t n = S.n, np = n * S.P;
  std::vector<uint32_t> pid(np);
  EFG_CUDA(cudaMemcpy(st->pool_dist, S.pd.p, np * 4, cudaMemcpyDeviceToHost));
  EFG_CUDA(cudaMemcpy(pid.data(), S.pid.p, np * 4, cudaMemcpyDeviceToHost));
  for (uint64_t i = 0; i < np; ++i) {
    st->pool_id[i] = pid[i] & IDM;
    st->pool_flag[i] = (pid[i] & FLAG) ? 1 : 0;
  }
  EFG_CUDA(cudaMemcpy(st->Lcur, S.Lc.p, n * 4, cudaMemcpyDeviceToHost));
  EFG_CUDA(cudaMemcpy(st->Range, S.Range.p, n * 4, cudaMemcpyDeviceToHost));
  EFG_CUDA(cudaMemcpy(st->radius, S.radius.p, n * 4, cudaMemcpyDeviceToHost));
  EFG_CUDA(cudaMemcpy(st->radiusM, S.radiusM.p, n * 4, cudaMemcpyDeviceToHost));
  EFG_CUDA(cudaMemcpy(st->found, S.found.p, n, cudaMemcpyDeviceToHost));
  EFG_CUDA(cudaMemcpy(st->new_ids, S.new_ids.p, n * S.cap * 4, cudaMemcpyDeviceToHost));
  EFG_CUDA(cudaMemcpy(st->new_cnt, S.new_cnt.p, n * 4, cudaMemcpyDeviceToHost));
  EFG_CUDA(cudaMemcpy(st->old_ids, S.old_ids.p, n * S.cap * 4, cudaMemcpyDeviceToHost));
  EFG_CUDA(cudaMemcpy(st->old_cnt, S.old_cnt.p, n * 4, cudaMemcpyDeviceToHost));
  return EFG_OK;
}

int nnd_init_host(efg_index* idx, efg_nnd_host_state* st) {
  if (idx->forest.ntrees == 0) return fail(EFG_ERR_STATE, "no trees");
  if (st->n != idx->n || st->L != idx->bp.L) return fail(EFG_ERR_ARG, "state does not match the index");
  uint32_t need = std::max(idx->bp.L, 2 * idx->bp.S) + idx->bp.reverse_cap;
  if (st->cap != need) return fail(EFG_ERR_ARG, "state list capacity must be " + std::to_string(need));
  NNDev S(idx->stream);
  int rc = nnd_init_device(idx, S);
  if (rc == EFG_OK) rc = state_to_host(S, st);
  return rc;
}

int nnd_iterate_host(efg_index* idx, efg_nnd_host_state* st, uint32_t iter, uint64_t* pairs) {
  uint32_t need = std::max(idx->bp.L, 2 * idx->bp.S) + idx->bp.reverse_cap;
  if (st->cap < need) return fail(EFG_ERR_ARG, "state list capacity too small");
  NNDev S(idx->stream);
  int rc = state_to_device(idx, S, st);
  uint64_t p = 0, r = 0;
  if (rc == EFG_OK) rc = nnd_iterate_device(idx, S, iter, &p, &r);
  if (rc == EFG_OK) rc = state_to_host(S, st);
  if (pairs) *pairs = p;
  return rc;
}

}  // namespace efg
