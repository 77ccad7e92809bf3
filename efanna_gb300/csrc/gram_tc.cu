// Exact k-NN screening on the fifth-generation tensor cores (tcgen05, sm_103a).
//
// Matrix::brute_force_search (general/matrix.hpp:57-68) ranks every base row by its squared L2
// distance to the query.  Written as ||q||^2 + ||x||^2 - 2 q.x, the distances of a block of
// queries against a block of base rows are one dense Gram contraction, which this file runs as
// BF16 tcgen05.mma tiles accumulated in FP32 in tensor memory (TMEM):
//
//   * queries and base rows are converted once per call to BF16 rows padded to a multiple of 64
//     values (128 bytes, one 128-byte-swizzle row), together with their FP32 squared norms.  Data
//     whose values BF16 holds exactly (the integer-valued configurations: values in [0, 255]) use
//     one product per tile, and then every product and every FP32 partial sum is an exact integer
//     below 2^24, so the screened distances equal the exact ones.  Other data are split as
//     x = hi + lo (two BF16 values) and each tile accumulates hi.hi + hi.lo + lo.hi, which leaves
//     an error near 2^-16 of |q.x| instead of 2^-8.
//   * tc_screen_kernel: a CTA owns one work item at a time, 128 or 256 queries (the MMA's M, one TMEM
//     lane each; one or two accumulators) against one chunk of base rows, walked in tiles of 128 rows
//     (N).  The queries' blocks stay in shared memory where they fit; warp 0 streams the base's
//     k-blocks into a ring of stages with cp.async.bulk.tensor (TMA, 128-byte swizzle), warp 1 issues
//     the MMAs (K = 16 each) into double-buffered accumulators, and sixteen warps in two sets read
//     the finished ones with tcgen05.ld and screen them.
//   * every query has an upper bound on its K2-th distance (K2 = k + 16) from cheap passes of the
//     same kernel over samples; the pass over the whole base appends the few values under it to the
//     query's candidate buffer, and select_kernel sorts them and re-ranks the K2 smallest in FP64.
//   * tc_knn_kernel, for the queries whose candidates overran their buffers (many rows at nearly one
//     distance): per-(query, chunk) sorted lists of K2 keys in shared memory, as the FP32 kernel writes
//     them (distance.cu), ranked by the same merge kernel.
//
// Every wait on an mbarrier is bounded: a wait that runs out sets an error word and the CTA leaves its
// loops, drains its tensor-core work and frees its TMEM; the host turns the word into
// EFG_ERR_DEVICE_LIMIT.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <mutex>
#include <vector>

#include "internal.cuh"
#include "tcgen05.cuh"

namespace efg {

int bf_merge_launch(const float* base, uint32_t dim, uint32_t ld, const float* q, uint64_t nq, uint32_t qld,
                    uint32_t k, uint32_t K2, uint32_t nchunks, const uint64_t* part, int32_t* ids, float* dists,
                    cudaStream_t s);

namespace {

constexpr uint32_t TM = 128;           // queries per tile (MMA M, TMEM lanes)
constexpr uint32_t TN = 128;           // base rows per tile (MMA N, TMEM columns per accumulator)
constexpr uint32_t TKB = 64;           // BF16 values per k-block: one 128-byte swizzle row
constexpr uint32_t PART = TM * TKB * 2;  // bytes of one 128 x 64 BF16 operand block (16 KiB)
constexpr uint32_t GRP = 16;           // values per screening group (one any-hit vote)
// warp 0 TMA, warp 1 MMA (+TMEM), then EW screening warps: 4 (each thread one query, all 128
// columns of a tile) or 8 (two threads per query, 64 columns each, two warps per scheduler)
template <int EW>
constexpr uint32_t kThreads = 64 + 32 * EW;
constexpr uint32_t MAX_STAGES = 8;
constexpr uint32_t TMEM_COLS = 2 * TN;  // two FP32 accumulators of 128 columns

constexpr uint32_t IDESC = tc::idesc_bf16(TM, TN);
using namespace tc;

struct TcArgs {
  const float* qnorm;  // nq FP32 squared norms
  const float* xnorm;  // squared norms of the base rows, +inf past n (rounded up to a tile)
  const float* qbound; // per query an upper bound of its K2-th distance, or null (+inf)
  uint64_t* part;      // nq x nchunks x K2 keys
  const uint32_t* qid; // the queries' numbers in the call (exclude_self), or null: 0, 1, ...
  int* err;
  uint64_t n, chunk, first_row;
  uint32_t nq, qtiles, nchunks, K2, kblocks, terms, stages, exclude_self;
  uint32_t o_list, o_scr, o_xn;  // byte offsets of the lists, scratch and norm copies in dynamic shared memory
};

__device__ __forceinline__ void tmem_ld64(uint32_t taddr, uint32_t (&r)[64]) {
  tmem_ld16(taddr, r);
  tmem_ld16(taddr + 16, r + 16);
  tmem_ld16(taddr + 32, r + 32);
  tmem_ld16(taddr + 48, r + 48);
}

// Inserts a key into a thread's sorted list of at most K2 keys (a full list drops its last key).
// Lists are slot-major with a stride of LS (the screening threads), so the threads of a warp touch
// consecutive words.
template <uint32_t LS>
__device__ __forceinline__ void insert_key(uint64_t* list, uint32_t t, uint32_t K2, uint32_t& lcnt, uint64_t key) {
  if (lcnt == K2 && key >= list[(K2 - 1) * LS + t]) return;
  uint32_t j = lcnt < K2 ? lcnt : K2 - 1;
  while (j > 0) {
    const uint64_t prev = list[(j - 1) * LS + t];
    if (prev <= key) break;
    list[j * LS + t] = prev;
    --j;
  }
  list[j * LS + t] = key;
  if (lcnt < K2) ++lcnt;
}

template <int EW>
__global__ void __launch_bounds__(kThreads<EW>, 1)
    tc_knn_kernel(const __grid_constant__ CUtensorMap mq_hi, const __grid_constant__ CUtensorMap mq_lo,
                  const __grid_constant__ CUtensorMap mx_hi, const __grid_constant__ CUtensorMap mx_lo,
                  const TcArgs a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[MAX_STAGES], bar_empty[MAX_STAGES], bar_tfull[2], bar_tempty[2],
      bar_drain;
  __shared__ uint32_t tmem_base_sh;
  __shared__ int abort_sh;

  // stages start on a 1024-byte boundary (the swizzle pattern repeats every 1024 bytes)
  const uint32_t raw = smem_addr(smem_raw);
  const uint32_t pad = ((raw + 1023u) & ~1023u) - raw;
  unsigned char* smem = smem_raw + pad;
  const uint32_t sbase = raw + pad;
  const uint32_t stage_bytes = 2 * PART;  // a query block and a base block
  const uint32_t steps = a.kblocks * a.terms;  // stages per tile
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < a.stages; ++s) {
      mbar_init(smem_addr(&bar_full[s]), 1);
      mbar_init(smem_addr(&bar_empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_addr(&bar_tfull[b]), 1);
      mbar_init(smem_addr(&bar_tempty[b]), 32 * EW);
    }
    mbar_init(smem_addr(&bar_drain), 1);
    abort_sh = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // the whole warp allocates the two accumulators
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_sh)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_sh;
  volatile int* abort_flag = &abort_sh;
  const uint32_t items = a.qtiles * a.nchunks;
  bool mma_issued = false;

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer (one lane)
    if (lane == 0) {
      uint32_t s = 0, ph = 0;
      bool ok = true;
      for (uint32_t w = blockIdx.x; ok && w < items; w += gridDim.x) {
        const uint32_t chunk = w / a.qtiles, qt = w % a.qtiles;
        const uint64_t r0 = (uint64_t)chunk * a.chunk, r1 = min(a.n, r0 + a.chunk);
        const uint32_t ntiles = (uint32_t)((r1 - r0 + TN - 1) / TN);
        for (uint32_t t = 0; ok && t < ntiles; ++t) {
          for (uint32_t step = 0; step < steps; ++step) {
            if (!mbar_wait(smem_addr(&bar_empty[s]), ph ^ 1u, abort_flag, a.err)) {
              ok = false;
              break;
            }
            const uint32_t kb = step / a.terms, term = step - kb * a.terms;  // term 0 (hi,hi), 1 (hi,lo), 2 (lo,hi)
            const uint32_t fb = smem_addr(&bar_full[s]);
            mbar_expect_tx(fb, stage_bytes);
            const uint32_t st = sbase + s * stage_bytes;
            const int x = (int)(kb * TKB), yq = (int)(qt * TM), yx = (int)(r0 + (uint64_t)t * TN);
            tma_load_2d(st, term == 2 ? &mq_lo : &mq_hi, fb, x, yq);
            tma_load_2d(st + PART, term == 1 ? &mx_lo : &mx_hi, fb, x, yx);
            if (++s == a.stages) {
              s = 0;
              ph ^= 1u;
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer (one lane)
    if (lane == 0) {
      uint32_t s = 0, ph = 0, tcount = 0;
      bool ok = true;
      for (uint32_t w = blockIdx.x; ok && w < items; w += gridDim.x) {
        const uint32_t chunk = w / a.qtiles;
        const uint64_t r0 = (uint64_t)chunk * a.chunk, r1 = min(a.n, r0 + a.chunk);
        const uint32_t ntiles = (uint32_t)((r1 - r0 + TN - 1) / TN);
        for (uint32_t t = 0; ok && t < ntiles; ++t, ++tcount) {
          const uint32_t b = tcount & 1u, tph = (tcount >> 1) & 1u;
          if (!mbar_wait(smem_addr(&bar_tempty[b]), tph ^ 1u, abort_flag, a.err)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + b * TN;
          for (uint32_t step = 0; step < steps; ++step) {
            if (!mbar_wait(smem_addr(&bar_full[s]), ph, abort_flag, a.err)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t st = sbase + s * stage_bytes;
            const uint64_t dq = sw128_desc(st), dx = sw128_desc(st + PART);
#pragma unroll
            for (uint32_t j = 0; j < TKB / 16; ++j) {  // K = 16 per MMA: 32 bytes further along the row
              const uint64_t o = (uint64_t)(2 * j);
              umma_bf16(d_tmem, dq + o, dx + o, IDESC, (step | j) != 0 ? 1u : 0u);
            }
            mma_issued = true;
            umma_commit(smem_addr(&bar_empty[s]));  // frees the stage when these MMAs have read it
            if (++s == a.stages) {
              s = 0;
              ph ^= 1u;
            }
          }
          if (!ok) break;
          umma_commit(smem_addr(&bar_tfull[b]));  // accumulator b holds tile t
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- screening (warps 2 ..)
    constexpr uint32_t CH = EW / 4;             // column parts of a tile (threads per query)
    constexpr uint32_t CPT = TN / CH;           // columns per thread per tile
    constexpr uint32_t LS = 32 * EW;            // list stride: all screening threads
    const uint32_t ew = warp - 2;
    const uint32_t quad = warp & 3u;            // TMEM lanes 32 * quad .. + 31
    const uint32_t et = quad * 32 + lane;       // this thread's query within the tile
    const uint32_t cp = ew / 4;                 // its column part: columns cp * CPT ..
    const uint32_t lt = cp * TM + et;           // its list
    uint64_t* list = reinterpret_cast<uint64_t*>(smem + a.o_list);
    // this thread's copy of a group's 16 values, float4 slot j4 stored at j4 ^ ((lane >> 1) & 3): the
    // eight threads of a quarter warp then write eight different 16-byte bank groups
    float* scr = reinterpret_cast<float*>(smem + a.o_scr) + (ew * 32 + lane) * GRP;
    const uint32_t sw = (lane >> 1) & 3u;
    // base-row norms of the current and the next tile, one copy per warp (warp-local hand-over)
    float* xw = reinterpret_cast<float*>(smem + a.o_xn) + ew * 2 * TN;
    uint32_t tcount = 0;
    bool ok = true;
    for (uint32_t w = blockIdx.x; ok && w < items; w += gridDim.x) {
      const uint32_t chunk = w / a.qtiles, qt = w % a.qtiles;
      const uint64_t r0 = (uint64_t)chunk * a.chunk, r1 = min(a.n, r0 + a.chunk);
      const uint32_t ntiles = (uint32_t)((r1 - r0 + TN - 1) / TN);
      const uint32_t q = qt * TM + et;
      const bool qvalid = q < a.nq;
      const float qn = qvalid ? a.qnorm[q] : 0.f;
      const uint64_t self = a.exclude_self && qvalid ? a.first_row + (a.qid ? a.qid[q] : q) : ~0ull;
      uint32_t lcnt = 0;
      // distance bound: the K2-th key's once the list is full; a thread past the queries accepts nothing
      float thr = qvalid ? (a.qbound ? a.qbound[q] : INFINITY) : -1.f;
      // the group test compares xn - 2 q.x against thr - qn, widened by a few ulps so that it never
      // rejects what the exact test (d = xn - 2 q.x + qn <= thr) accepts
      auto bound = [&](float t) { return qvalid ? t - qn + (fabsf(t) + qn) * 4.8e-7f : -INFINITY; };
      float lim = bound(thr);
      reinterpret_cast<float4*>(xw + (tcount & 1u) * TN)[lane] =
          __ldg(reinterpret_cast<const float4*>(a.xnorm + r0) + lane);
      __syncwarp();
      for (uint32_t t = 0; t < ntiles; ++t, ++tcount) {
        const uint32_t b = tcount & 1u, tph = (tcount >> 1) & 1u;
        const uint64_t row0 = r0 + (uint64_t)t * TN;
        const bool more = t + 1 < ntiles;
        float4 xnext = make_float4(0.f, 0.f, 0.f, 0.f);
        if (more) xnext = __ldg(reinterpret_cast<const float4*>(a.xnorm + row0 + TN) + lane);  // in flight meanwhile
        // every lane waits; the vote keeps the warp together for the warp-wide TMEM loads
        ok = __all_sync(0xffffffffu, mbar_wait(smem_addr(&bar_tfull[b]), tph, abort_flag, a.err));
        if (!ok) break;
        tc_fence_after();
        const bool edge = row0 + TN > r1 || (self >= row0 && self < row0 + TN);
        const uint32_t taddr = tmem_base + ((quad * 32u) << 16) + b * TN + cp * CPT;
        const float* xs = xw + (tcount & 1u) * TN + cp * CPT;
        uint32_t va[64], vb[64];
        tmem_ld64(taddr, va);
        tmem_wait();
        if (CPT == 128) tmem_ld64(taddr + 64, vb);  // the second half arrives while the first is screened
#pragma unroll
        for (uint32_t half = 0; half < CPT / 64; ++half) {
          if (half == 1) tmem_wait();
          const uint32_t* v = half == 0 ? va : vb;
#pragma unroll
          for (uint32_t g = 0; g < 64 / GRP; ++g) {
            const float4* x4 = reinterpret_cast<const float4*>(xs + half * 64 + g * GRP);
            // any value of the group under the bound? (four independent chains)
            bool h0 = false, h1 = false, h2 = false, h3 = false;
#pragma unroll
            for (uint32_t j4 = 0; j4 < GRP / 4; ++j4) {
              const float4 xn = x4[j4];
              const uint32_t o = g * GRP + 4 * j4;
              h0 |= fmaf(-2.f, __uint_as_float(v[o + 0]), xn.x) <= lim;
              h1 |= fmaf(-2.f, __uint_as_float(v[o + 1]), xn.y) <= lim;
              h2 |= fmaf(-2.f, __uint_as_float(v[o + 2]), xn.z) <= lim;
              h3 |= fmaf(-2.f, __uint_as_float(v[o + 3]), xn.w) <= lim;
            }
            const bool hit = h0 | h1 | h2 | h3;
            if (__any_sync(0xffffffffu, hit)) {
              // the group's values under the bound, as a mask; this thread's values to its scratch
              uint32_t m = 0;
              if (hit) {
#pragma unroll
                for (uint32_t j4 = 0; j4 < GRP / 4; ++j4) {
                  const float4 xn = x4[j4];
                  const uint32_t o = g * GRP + 4 * j4;
                  m |= (fmaf(-2.f, __uint_as_float(v[o + 0]), xn.x) <= lim ? 1u : 0u) << (4 * j4);
                  m |= (fmaf(-2.f, __uint_as_float(v[o + 1]), xn.y) <= lim ? 2u : 0u) << (4 * j4);
                  m |= (fmaf(-2.f, __uint_as_float(v[o + 2]), xn.z) <= lim ? 4u : 0u) << (4 * j4);
                  m |= (fmaf(-2.f, __uint_as_float(v[o + 3]), xn.w) <= lim ? 8u : 0u) << (4 * j4);
                  reinterpret_cast<float4*>(scr)[j4 ^ sw] =
                      make_float4(__uint_as_float(v[o]), __uint_as_float(v[o + 1]), __uint_as_float(v[o + 2]),
                                  __uint_as_float(v[o + 3]));
                }
              }
              // one marked value per lane per round: the exact test, straight into the sorted list
              while (__any_sync(0xffffffffu, m != 0u)) {
                if (m != 0u) {
                  const uint32_t j = __ffs(m) - 1;
                  m &= m - 1;
                  const float val = scr[(((j >> 2) ^ sw) << 2) | (j & 3u)];
                  const uint32_t c = half * 64 + g * GRP + j;
                  const float d = fmaxf(fmaf(-2.f, val, xs[c]) + qn, 0.f);
                  const uint64_t row = row0 + cp * CPT + c;
                  if (d <= thr && (!edge || (row < r1 && row != self))) {
                    insert_key<LS>(list, lt, a.K2, lcnt, ((uint64_t)__float_as_uint(d) << 32) | (uint32_t)row);
                    if (lcnt == a.K2) {
                      thr = __uint_as_float((uint32_t)(list[(a.K2 - 1) * LS + lt] >> 32));
                      lim = bound(thr);
                    }
                  }
                }
              }
            }
          }
        }
        tc_fence_before();
        mbar_arrive(smem_addr(&bar_tempty[b]));  // accumulator b may be overwritten
        if (more) reinterpret_cast<float4*>(xw + ((tcount + 1) & 1u) * TN)[lane] = xnext;
        __syncwarp();
      }
      if (!ok) break;
      if (qvalid) {  // list part cp of this (query, chunk): the merge sees CH lists per chunk
        uint64_t* dst = a.part + ((uint64_t)q * a.nchunks * CH + chunk * CH + cp) * a.K2;
        for (uint32_t i = 0; i < a.K2; ++i) dst[i] = i < lcnt ? list[i * LS + lt] : ~0ull;
      }
    }
  }

  // ------------------------------------------------------------------------------ teardown
  __syncthreads();
  if (warp == 1) {
    if (lane == 0 && mma_issued) {  // every MMA this thread issued has finished before TMEM is freed
      umma_commit(smem_addr(&bar_drain));
      unsigned long long t0 = clock64();
      while (!mbar_try_wait(smem_addr(&bar_drain), 0)) {
        if (clock64() - t0 > WAIT_CYCLES) {
          atomicOr(a.err, 2);
          break;
        }
      }
    }
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS)
                 : "memory");
  }
}

// Rows floor(i * n / S) of the converted base (hi, lo, norm) into S contiguous sample rows (a warp
// per row, 16-byte copies; W BF16 values per row).
__global__ void sample_rows_kernel(const uint4* __restrict__ hi, const uint4* __restrict__ lo,
                                   const float* __restrict__ norms, uint64_t n, uint32_t W, uint32_t S,
                                   uint4* __restrict__ shi, uint4* __restrict__ slo, float* __restrict__ snorms) {
  const uint32_t lane = threadIdx.x & 31, w16 = W / 8;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < S; i += nw) {
    const uint64_t r = i * n / S;
    for (uint32_t c = lane; c < w16; c += 32) {
      shi[i * w16 + c] = hi[r * w16 + c];
      slo[i * w16 + c] = lo[r * w16 + c];
    }
    if (lane == 0) snorms[i] = norms[r];
  }
}

// Per query the distance of the rank-th smallest key over its L sorted lists of `stride` keys (L <=
// 16, ~0 padded), widened by `rel` (the split form's passes may round differently); +inf when the
// lists hold fewer keys; never above the query's previous bound `prev` (when given).
__global__ void bound_kernel(const uint64_t* __restrict__ lists, uint64_t nq, uint32_t L, uint32_t stride,
                             uint32_t rank, float rel, const float* __restrict__ prev, float* __restrict__ out) {
  for (uint64_t qi = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; qi < nq; qi += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t* a = lists + qi * L * stride;
    uint32_t pos[16];
    for (uint32_t l = 0; l < L; ++l) pos[l] = 0;
    uint64_t key = ~0ull;
    for (uint32_t r = 0; r < rank; ++r) {  // merge walk up to the rank-th key
      uint32_t best = 0;
      key = ~0ull;
      for (uint32_t l = 0; l < L; ++l) {
        const uint64_t h = pos[l] < stride ? a[l * stride + pos[l]] : ~0ull;
        if (h < key) {
          key = h;
          best = l;
        }
      }
      if (key == ~0ull) break;
      pos[best] += 1;
    }
    const float d = __uint_as_float((uint32_t)(key >> 32));
    float bnd = key == ~0ull ? INFINITY : d + d * rel;
    if (prev) bnd = fminf(bnd, prev[qi]);
    out[qi] = bnd;
  }
}


// ==============================================================================================
// Screening against a bound: every query whose candidates fit its buffer.
//
// With an upper bound on each query's K2-th distance, screening only has to find the values under it
// and append them to the query's buffer; lists, and their divergent insertions, are left to the few.
// The bound comes from cheap passes of the same kernel:
//   * MIN pass over a sample: the rows fall into groups, every thread keeps its groups' minima, and the
//     largest minimum of at least K2 disjoint groups bounds the K2-th distance (no list, two
//     instructions per value);
//   * append pass over n / 16 rows with that bound, whose K2-th key is a tight one: about 16 K2 values of
//     the whole base lie under it.
//
// Data movement is what bounds a Gram tile here: 128 x 128 x 64 products take 256 cycles and read 32 KB.
// So a work item keeps its query blocks in shared memory (where they fit) and takes two query tiles at
// a time (256 queries, 512 TMEM columns with two buffers), which reads each base block once per 256
// queries: 32 KB per 1024 cycles at 128 dimensions instead of 64 KB per 512.  The screening warps spend
// one packed FMA and one three-input minimum per two values.
constexpr uint32_t SW_ = 16;                    // screening warps: eight per accumulator buffer
constexpr uint32_t STH = 64 + 32 * SW_;         // threads
constexpr uint32_t CAND_MAX = 4096;             // candidates a query's buffer can hold
// Bytes of candidate buffers: more queries than they serve (262,144 at k = 1, 131,072 at k = 10, 65,536 from
// k = 27 on, far more than keep the chip busy) are taken in blocks.
constexpr uint64_t CAND_BYTES = 2ull << 30;

struct ScreenArgs {
  const float* qnorm;     // nq FP32 squared norms
  const float* xnorm;     // of the rows, +inf past the last up to a whole tile
  const uint32_t* qbound; // bits of an upper bound of each query's rank-th distance, or null (+inf)
  uint32_t* qmax;         // MIN pass: bits of the bound, combined by atomicMax (zero on entry)
  uint32_t* cnt;          // append pass: candidates per query (may exceed cap)
  uint64_t* buf;          // nq x cap keys
  int* err;
  uint64_t n, first_row;
  uint32_t ntiles, chunk_tiles, nchunks, qgroups, nq, cap, kblocks, stages, exclude_self;
  uint32_t group_tiles;   // MIN pass: a thread's tiles (every other one) per group of its 64 columns (0: groups of
                          // 16 columns); a chunk holds a multiple of 2 group_tiles
  // MIN_STRIDED: rows `stride` apart fill a box of 2^box_shift columns (row i stride + u is column i of box
  // u, for i < rows_box; the others are empty), so that every group reaches over the whole base; W values
  // per row.
  uint32_t stride, box_shift, rows_box, W;
  uint32_t split, resident;
  float rel;              // the bound is widened by this much (passes of the split form may round differently)
  uint32_t stage_bytes, o_x, o_scr, o_xn, o_queue;
};

__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// PASS: values under the bound appended, groups' minima of rows in order, or of strided rows.
enum { APPEND = 0, MIN_ROWS = 1, MIN_STRIDED = 2 };
template <int NT, int PASS>
__global__ void __launch_bounds__(STH, 1)
    tc_screen_kernel(const __grid_constant__ CUtensorMap mq_hi, const __grid_constant__ CUtensorMap mq_lo,
                     const __grid_constant__ CUtensorMap mx_hi, const __grid_constant__ CUtensorMap mx_lo,
                     const ScreenArgs a) {
  constexpr uint32_t COLS = 2 * NT * TN;  // two buffers of NT accumulators
  constexpr bool MINP = PASS != APPEND;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[MAX_STAGES], bar_empty[MAX_STAGES], bar_tfull[2], bar_tempty[2], bar_q,
      bar_qfree, bar_drain;
  __shared__ uint32_t tmem_base_sh;
  __shared__ int abort_sh;
  const uint32_t raw = smem_addr(smem_raw);
  const uint32_t pad = ((raw + 1023u) & ~1023u) - raw;
  unsigned char* smem = smem_raw + pad;
  const uint32_t sbase = raw + pad;
  const uint32_t parts = a.split ? 2u : 1u;  // hi, or hi and lo blocks
  // (the shuffle tells the compiler that the warp index is the same in all lanes)
  const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < a.stages; ++s) {
      mbar_init(smem_addr(&bar_full[s]), 1);
      mbar_init(smem_addr(&bar_empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_addr(&bar_tfull[b]), 1);
      mbar_init(smem_addr(&bar_tempty[b]), 16 * SW_);
    }
    mbar_init(smem_addr(&bar_q), 1);
    mbar_init(smem_addr(&bar_qfree), 1);
    mbar_init(smem_addr(&bar_drain), 1);
    abort_sh = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_sh)),
                 "r"(COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_sh;
  volatile int* abort_flag = &abort_sh;
  const uint32_t items = a.qgroups * a.nchunks;
  bool mma_issued = false;

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer (one lane)
    if (lane == 0) {
      uint32_t s = 0, ph = 0, it = 0;
      bool ok = true;
      for (uint32_t w = blockIdx.x; ok && w < items; w += gridDim.x, ++it) {
        const uint32_t chunk = w / a.qgroups, qg = w % a.qgroups;
        const uint32_t t0 = chunk * a.chunk_tiles, t1 = min(a.ntiles, t0 + a.chunk_tiles);
        const int yq = (int)(qg * NT * TM);
        if (a.resident) {  // the item's query blocks, once the previous item's products have read theirs
          if (!mbar_wait(smem_addr(&bar_qfree), (it & 1u) ^ 1u, abort_flag, a.err)) break;
          const uint32_t qb = smem_addr(&bar_q);
          mbar_expect_tx(qb, NT * a.kblocks * parts * PART);
          for (uint32_t i = 0; i < NT * a.kblocks; ++i) {
            const int x = (int)((i % a.kblocks) * TKB), y = yq + (int)((i / a.kblocks) * TM);
            tma_load_2d(sbase + i * parts * PART, &mq_hi, qb, x, y);
            if (a.split) tma_load_2d(sbase + (i * parts + 1) * PART, &mq_lo, qb, x, y);
          }
        }
        for (uint32_t t = t0; ok && t < t1; ++t) {
          for (uint32_t kb = 0; kb < a.kblocks; ++kb) {
            if (!mbar_wait(smem_addr(&bar_empty[s]), ph ^ 1u, abort_flag, a.err)) {
              ok = false;
              break;
            }
            const uint32_t fb = smem_addr(&bar_full[s]);
            mbar_expect_tx(fb, a.stage_bytes);
            const uint32_t st = sbase + a.o_x + s * a.stage_bytes;
            const int x = (int)(kb * TKB), yx = (int)(t * TN);
            if (PASS == MIN_STRIDED) {
              for (uint32_t c = 0; c < TN; c += 1u << a.box_shift) {
                const int xb = x + (int)(((t * TN + c) >> a.box_shift) * a.W);
                tma_load_2d(st + c * TKB * 2, &mx_hi, fb, xb, 0);
                if (a.split) tma_load_2d(st + PART + c * TKB * 2, &mx_lo, fb, xb, 0);
              }
            } else {
              tma_load_2d(st, &mx_hi, fb, x, yx);
              if (a.split) tma_load_2d(st + PART, &mx_lo, fb, x, yx);
            }
            if (!a.resident)
              for (uint32_t i = 0; i < NT; ++i) {
                const uint32_t dst = st + (1 + i) * parts * PART;
                tma_load_2d(dst, &mq_hi, fb, x, yq + (int)(i * TM));
                if (a.split) tma_load_2d(dst + PART, &mq_lo, fb, x, yq + (int)(i * TM));
              }
            if (++s == a.stages) {
              s = 0;
              ph ^= 1u;
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    // The whole warp walks the loops, so that descriptors and addresses stay in uniform registers, and one
    // elected lane issues.  With the loops inside one lane's branch every tcgen05.mma cost about 144
    // cycles of issue, more than twice its 64 cycles in the tensor cores.
    {
      uint32_t s = 0, ph = 0, tcount = 0, it = 0;
      bool ok = true;
      const bool one = elect_one();
      for (uint32_t w = blockIdx.x; ok && w < items; w += gridDim.x, ++it) {
        const uint32_t chunk = w / a.qgroups;
        const uint32_t t0 = chunk * a.chunk_tiles, t1 = min(a.ntiles, t0 + a.chunk_tiles);
        if (a.resident && !warp_wait(smem_addr(&bar_q), it & 1u, abort_flag, a.err)) break;
        tc_fence_after();
        for (uint32_t t = t0; ok && t < t1; ++t, ++tcount) {
          const uint32_t b = tcount & 1u, tph = (tcount >> 1) & 1u;
          if (!warp_wait(smem_addr(&bar_tempty[b]), tph ^ 1u, abort_flag, a.err)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + b * NT * TN;
          for (uint32_t kb = 0; kb < a.kblocks; ++kb) {
            if (!warp_wait(smem_addr(&bar_full[s]), ph, abort_flag, a.err)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t st = sbase + a.o_x + s * a.stage_bytes;
            const uint64_t xh = sw128_desc(st), xl = sw128_desc(st + PART);
            const uint32_t qa = a.resident ? sbase + kb * parts * PART : st + parts * PART;
            const uint32_t qstep = a.resident ? a.kblocks * parts * PART : parts * PART;
            const uint32_t free_bar = smem_addr(&bar_empty[s]), done_bar = smem_addr(&bar_tfull[b]);
            const bool last = kb + 1 == a.kblocks;
            if (one) {
#pragma unroll
              for (uint32_t i = 0; i < NT; ++i) {
                const uint64_t qh = sw128_desc(qa + i * qstep), ql = sw128_desc(qa + i * qstep + PART);
#pragma unroll
                for (uint32_t j = 0; j < TKB / 16; ++j) {  // K = 16 per MMA: 32 bytes further along the row
                  const uint64_t o = (uint64_t)(2 * j);
                  umma_bf16(d_tmem + i * TN, qh + o, xh + o, IDESC, (kb | j) != 0 ? 1u : 0u);
                  if (a.split) {
                    umma_bf16(d_tmem + i * TN, qh + o, xl + o, IDESC, 1u);
                    umma_bf16(d_tmem + i * TN, ql + o, xh + o, IDESC, 1u);
                  }
                }
              }
              umma_commit(free_bar);               // frees the stage when these MMAs have read it
              if (last) umma_commit(done_bar);     // buffer b holds the tile
            }
            mma_issued = true;
            __syncwarp();
            if (++s == a.stages) {
              s = 0;
              ph ^= 1u;
            }
          }
        }
        if (ok && a.resident && one) umma_commit(smem_addr(&bar_qfree));
        __syncwarp();
      }
      if (one && mma_issued) umma_commit(smem_addr(&bar_drain));  // by the lane that issued them
    }
  } else {
    // ---------------------------------------------------------------- screening (warps 2 ..)
    // eight warps screen the tiles of one accumulator buffer, eight the other's: a tile's chain of waiting,
    // TMEM reads and tests takes longer than its products, and two run side by side this way
    const uint32_t ew = warp - 2, quad = warp & 3u, half = (ew >> 2) & 1u, b = ew >> 3;  // TMEM lanes 32 quad ..,
    const uint32_t taddr0 = tmem_base + ((quad * 32u) << 16) + b * NT * TN + half * 64;  // columns 64 half ..
    float* scr = reinterpret_cast<float*>(smem + a.o_scr) + (ew * 32 + lane) * GRP;
    const uint32_t sw = (lane >> 1) & 3u;  // (the copy of a group's 16 values: float4 slot j at j ^ sw)
    float* xw = reinterpret_cast<float*>(smem + a.o_xn) + ew * 2 * 64;  // norms of 64 rows, this tile's and the next
    const uint64_t m2 = pack2(__float_as_uint(-2.f), __float_as_uint(-2.f));
    // candidates on their way to the queries' buffers: 32 slots are taken at once, an atomic per lane
    // (one at a time their latency held the warp at every hit: 4.6 of 7.0 ms at 10k x 1M x 128)
    uint64_t* queue_key = reinterpret_cast<uint64_t*>(smem + a.o_queue) + ew * 64;
    uint32_t* queue_q = reinterpret_cast<uint32_t*>(smem + a.o_queue + SW_ * 64 * 8) + ew * 64;
    uint32_t queued = 0;
    auto flush = [&](uint32_t m) {
      __syncwarp();
      if (lane < m) {
        const uint32_t qq = queue_q[lane];
        const uint32_t pos = atomicAdd(&a.cnt[qq], 1u);
        if (pos < a.cap) a.buf[(uint64_t)qq * a.cap + pos] = queue_key[lane];
      }
      const uint64_t rk = lane + 32 < queued ? queue_key[lane + 32] : 0;
      const uint32_t rq = lane + 32 < queued ? queue_q[lane + 32] : 0;
      __syncwarp();
      if (lane + 32 < queued) {
        queue_key[lane] = rk;
        queue_q[lane] = rq;
      }
      queued -= m;
      __syncwarp();
    };
    // norms of this lane's two of the 64 columns from col on, where the rows are not in order
    auto strided_norms = [&](uint32_t col) -> float2 {
      const uint32_t c = col + 2 * lane, u = c >> a.box_shift, i = c & ((1u << a.box_shift) - 1);  // (both in one box)
      return make_float2(i < a.rows_box ? __ldg(a.xnorm + (uint64_t)i * a.stride + u) : INFINITY,
                         i + 1 < a.rows_box ? __ldg(a.xnorm + (uint64_t)(i + 1) * a.stride + u) : INFINITY);
    };
    uint32_t tcount = 0;
    bool ok = true;
    for (uint32_t w = blockIdx.x; ok && w < items; w += gridDim.x) {
      const uint32_t chunk = w / a.qgroups, qg = w % a.qgroups;
      const uint32_t t0 = chunk * a.chunk_tiles, t1 = min(a.ntiles, t0 + a.chunk_tiles);
      float qn[NT], thr[NT], lim[NT], gmin[NT], gmax[NT];
      uint32_t qi[NT];
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        qi[i] = (qg * NT + i) * TM + quad * 32 + lane;
        const bool valid = qi[i] < a.nq;
        qn[i] = valid ? a.qnorm[qi[i]] : 0.f;
        const float b = !MINP && valid && a.qbound ? __uint_as_float(a.qbound[qi[i]]) : INFINITY;
        thr[i] = !valid ? -1.f : b < INFINITY ? b + b * a.rel : INFINITY;
        // the group test compares xn - 2 q.x against thr - qn, widened by a few ulps so that it never
        // rejects what the exact test (d = xn - 2 q.x + qn <= thr) accepts
        lim[i] = valid ? thr[i] - qn[i] + (fabsf(thr[i]) + qn[i]) * 4.8e-7f : -INFINITY;
        gmin[i] = INFINITY;
        gmax[i] = -INFINITY;
      }
      const uint32_t first = t0 + ((tcount & 1u) ^ b);  // this buffer's tiles: first, first + 2, ...
      const uint32_t item_end = tcount + (t1 - t0);
      uint32_t flip = 0, in_group = 0;
      if (first < t1)
        reinterpret_cast<float2*>(xw)[lane] =
            PASS == MIN_STRIDED ? strided_norms(first * TN + half * 64)
                             : __ldg(reinterpret_cast<const float2*>(a.xnorm + (uint64_t)first * TN + half * 64) + lane);
      __syncwarp();
      for (uint32_t t = first; t < t1; t += 2, flip ^= 1u) {
        const uint32_t tph = ((tcount + (t - t0)) >> 1) & 1u;
        const uint64_t row0 = (uint64_t)t * TN + half * 64;
        float2 xnext = make_float2(0.f, 0.f);
        if (t + 2 < t1)  // in flight meanwhile
          xnext = PASS == MIN_STRIDED ? strided_norms((uint32_t)row0 + 2 * TN)
                                   : __ldg(reinterpret_cast<const float2*>(a.xnorm + row0 + 2 * TN) + lane);
        ok = __all_sync(0xffffffffu, mbar_wait(smem_addr(&bar_tfull[b]), tph, abort_flag, a.err));
        if (!ok) break;
        tc_fence_after();
        const float* xs = xw + flip * 64;
#pragma unroll
        for (int i = 0; i < NT; ++i) {
          uint32_t v[32];
#pragma unroll
          for (uint32_t g = 0; g < 64 / GRP; ++g) {
            if (g % 2 == 0) {  // 32 columns at a time (64 would not leave 16 warps their registers)
              tmem_ld16(taddr0 + i * TN + g * GRP, v);
              tmem_ld16(taddr0 + i * TN + g * GRP + 16, v + 16);
              tmem_wait();
            }
            const ulonglong2* x2 = reinterpret_cast<const ulonglong2*>(xs + g * GRP);
            float m0 = INFINITY, m1 = INFINITY;
#pragma unroll
            for (uint32_t j = 0; j < GRP / 4; ++j) {
              const ulonglong2 xn = x2[j];
              const uint32_t o = (g % 2) * GRP + 4 * j;
              float p0, p1, p2, p3;
              unpack2(fma2(m2, pack2(v[o], v[o + 1]), xn.x), p0, p1);
              unpack2(fma2(m2, pack2(v[o + 2], v[o + 3]), xn.y), p2, p3);
              m0 = min3(m0, p0, p1);
              m1 = min3(m1, p2, p3);
            }
            const float m = fminf(m0, m1);
            if (MINP) {
              if (a.group_tiles) gmin[i] = fminf(gmin[i], m);
              else gmax[i] = fmaxf(gmax[i], m);
            } else if (__any_sync(0xffffffffu, m <= lim[i])) {
              // the group's values under the bound, as a mask; this thread's values to its scratch
              uint32_t hits = 0;
              if (m <= lim[i]) {
#pragma unroll
                for (uint32_t j = 0; j < GRP / 4; ++j) {
                  const float4 xn = reinterpret_cast<const float4*>(xs + g * GRP)[j];
                  const uint32_t o = (g % 2) * GRP + 4 * j;
                  hits |= (fmaf(-2.f, __uint_as_float(v[o + 0]), xn.x) <= lim[i] ? 1u : 0u) << (4 * j);
                  hits |= (fmaf(-2.f, __uint_as_float(v[o + 1]), xn.y) <= lim[i] ? 2u : 0u) << (4 * j);
                  hits |= (fmaf(-2.f, __uint_as_float(v[o + 2]), xn.z) <= lim[i] ? 4u : 0u) << (4 * j);
                  hits |= (fmaf(-2.f, __uint_as_float(v[o + 3]), xn.w) <= lim[i] ? 8u : 0u) << (4 * j);
                  reinterpret_cast<float4*>(scr)[j ^ sw] =
                      make_float4(__uint_as_float(v[o]), __uint_as_float(v[o + 1]), __uint_as_float(v[o + 2]),
                                  __uint_as_float(v[o + 3]));
                }
              }
              // one marked value per lane per round: the exact test, then the warp's queue
              const uint64_t self = a.exclude_self ? a.first_row + qi[i] : ~0ull;
              while (__any_sync(0xffffffffu, hits != 0)) {
                uint64_t key = 0;
                bool take = false;
                if (hits) {
                  const uint32_t j = __ffs(hits) - 1;
                  hits &= hits - 1;
                  const float val = scr[(((j >> 2) ^ sw) << 2) | (j & 3u)];
                  const float d = fmaxf(fmaf(-2.f, val, xs[g * GRP + j]) + qn[i], 0.f);
                  const uint64_t row = row0 + g * GRP + j;
                  key = ((uint64_t)__float_as_uint(d) << 32) | (uint32_t)row;
                  take = d <= thr[i] && row < a.n && row != self;
                }
                const uint32_t bal = __ballot_sync(0xffffffffu, take);
                if (take) {
                  const uint32_t e = queued + __popc(bal & ((1u << lane) - 1));
                  queue_key[e] = key;
                  queue_q[e] = qi[i];
                }
                queued += __popc(bal);
                if (queued >= 32) flush(32);
              }
              __syncwarp();
            }
          }
        }
        tc_fence_before();
        mbar_arrive(smem_addr(&bar_tempty[b]));  // buffer b may be overwritten
        if (t + 2 < t1) reinterpret_cast<float2*>(xw + (flip ^ 1u) * 64)[lane] = xnext;
        if (MINP && a.group_tiles && ++in_group == a.group_tiles) {
          in_group = 0;
#pragma unroll
          for (int i = 0; i < NT; ++i) {
            gmax[i] = fmaxf(gmax[i], gmin[i]);
            gmin[i] = INFINITY;
          }
        }
        __syncwarp();
      }
      if (!ok) break;
      tcount = item_end;
      if (MINP) {
#pragma unroll
        for (int i = 0; i < NT; ++i)
          if (qi[i] < a.nq) atomicMax(&a.qmax[qi[i]], __float_as_uint(fmaxf(gmax[i] + qn[i], 0.f)));
      }
    }
    if (!MINP && queued) flush(queued);
  }

  // ------------------------------------------------------------------------------ teardown
  __syncthreads();
  if (warp == 1) {
    if (lane == 0 && mma_issued) {  // every MMA has finished before TMEM is freed
      unsigned long long t0 = clock64();
      while (!mbar_try_wait(smem_addr(&bar_drain), 0)) {
        if (clock64() - t0 > WAIT_CYCLES) {
          atomicOr(a.err, 2);
          break;
        }
      }
    }
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(COLS) : "memory");
  }
}

// Sample rows in a scattered order: the base falls into S strata of n / S (per) rows, and row i of the sample is a
// row of stratum (i * step) mod S, step prime to S, so that every leading part of the sample is spread
// over the base too.  Which row of the stratum is hashed: the first one of each would be of one class where
// classes alternate with a period that divides n / S (2^20 rows of 16 classes in turn, 10k queries: 54.9
// ms with nearly all queries in the lists, 5.8 ms this way).  A warp per row, 16-byte copies, W BF16
// values per row; lo may be null.
__global__ void scatter_sample_kernel(const uint4* __restrict__ hi, const uint4* __restrict__ lo,
                                      const float* __restrict__ norms, uint64_t n, uint32_t W, uint32_t S,
                                      uint32_t step, uint32_t per, uint4* __restrict__ shi, uint4* __restrict__ slo,
                                      float* __restrict__ snorms) {
  const uint32_t lane = threadIdx.x & 31, w16 = W / 8;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < S; i += nw) {
    const uint64_t p = i * step % S, r = p * n / S + __umulhi((uint32_t)mix64(p), per);
    for (uint32_t c = lane; c < w16; c += 32) {
      shi[i * w16 + c] = hi[r * w16 + c];
      if (lo) slo[i * w16 + c] = lo[r * w16 + c];
    }
    if (lane == 0) snorms[i] = norms[r];
  }
}

// FP32 rows -> BF16 hi (and, with lo, lo = x - hi) rows of W values (zero padded), squared norms (+inf
// for the rows up to norm_rows), and a flag set when some lo is not zero.  A warp per row of the rows
// r * step; a lane four values at a time.  hi null: only the flag.
__global__ void split_bf16_kernel(const float* __restrict__ src, uint64_t rows, uint64_t step, uint32_t dim,
                                  uint64_t ld, uint32_t W, uint2* __restrict__ hi, uint2* __restrict__ lo,
                                  float* __restrict__ norms, uint64_t norm_rows, int* __restrict__ inexact) {
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t lane = threadIdx.x & 31;
  bool any_lo = false;
  for (uint64_t r = (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * step; r < norm_rows; r += nw * step) {
    if (r >= rows) {
      if (lane == 0) norms[r] = INFINITY;
      continue;
    }
    float acc = 0.f;
    for (uint32_t c = lane; c < W / 4; c += 32) {
      float x[4] = {0.f, 0.f, 0.f, 0.f};
      if (4 * c + 3 < dim) {
        const float4 f = __ldg(reinterpret_cast<const float4*>(src + r * ld) + c);
        x[0] = f.x;
        x[1] = f.y;
        x[2] = f.z;
        x[3] = f.w;
      } else {
        for (uint32_t j = 0; 4 * c + j < dim; ++j) x[j] = src[r * ld + 4 * c + j];
      }
      __nv_bfloat16 h[4], l[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        h[j] = __float2bfloat16_rn(x[j]);
        l[j] = __float2bfloat16_rn(x[j] - __bfloat162float(h[j]));
        any_lo |= __bfloat162float(l[j]) != 0.f;
        acc = fmaf(x[j], x[j], acc);
      }
      if (hi) hi[r * (W / 4) + c] = *reinterpret_cast<const uint2*>(h);
      if (lo) lo[r * (W / 4) + c] = *reinterpret_cast<const uint2*>(l);
    }
    acc = warp_sum(acc);
    if (lane == 0 && hi) norms[r] = acc;
  }
  if (__any_sync(0xffffffffu, any_lo) && lane == 0) atomicOr(inexact, 1);
}

// One CTA per query: the query's candidates sorted in shared memory.  With `ids` the K2 smallest are
// re-ranked in FP64 and the first k written; else the rank-th distance becomes the query's bound (when
// the buffer holds that many, and all of them).  A query whose final buffer was too short is left to the
// lists: its number (q0 the first's) goes to over_list, which *over counts.
__global__ void __launch_bounds__(256) select_kernel(const uint64_t* __restrict__ buf, const uint32_t* __restrict__ cnt,
                                                     uint32_t cap, uint32_t rank, uint32_t* __restrict__ qbound,
                                                     const float* __restrict__ base, uint32_t dim, uint32_t ld,
                                                     const float* __restrict__ q, uint32_t qld, uint32_t k,
                                                     int32_t* __restrict__ ids, float* __restrict__ dists,
                                                     int* __restrict__ over, uint32_t* __restrict__ over_list,
                                                     uint32_t q0) {
  extern __shared__ __align__(16) uint64_t keys[];  // next_pow2(candidates), then K2 distances
  const uint64_t qi = blockIdx.x;
  const uint32_t m = cnt[qi], lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (m > cap) {
    if (threadIdx.x == 0 && ids) over_list[atomicAdd(over, 1)] = q0 + (uint32_t)qi;
    return;
  }
  if (!ids && m < rank) return;
  const uint32_t p2 = next_pow2(m < 2 ? 2 : m);
  for (uint32_t i = threadIdx.x; i < p2; i += 256) keys[i] = i < m ? buf[qi * cap + i] : ~0ull;
  __syncthreads();
  for (uint32_t s = 2; s <= p2; s <<= 1)
    for (uint32_t j = s >> 1; j > 0; j >>= 1) {
      for (uint32_t i = threadIdx.x; i < p2 / 2; i += 256) {
        const uint32_t lo = ((i & ~(j - 1)) << 1) | (i & (j - 1)), hi = lo | j;
        const uint64_t x = keys[lo], y = keys[hi];
        if ((x > y) == ((lo & s) == 0)) {
          keys[lo] = y;
          keys[hi] = x;
        }
      }
      __syncthreads();
    }
  if (!ids) {
    if (threadIdx.x == 0) qbound[qi] = min(qbound[qi], (uint32_t)(keys[rank - 1] >> 32));
    return;
  }
  // FP64 distances of the first `rank` (= K2) keys, then their places by (distance, id)
  const uint32_t K2 = min(rank, m);
  double* d64 = reinterpret_cast<double*>(keys + cap);
  const float* qr = q + qi * qld;
  for (uint32_t i = warp; i < K2; i += 8) {
    const float* br = base + (uint64_t)(uint32_t)keys[i] * ld;
    double acc = 0.0;
    for (uint32_t c = lane; c < dim; c += 32) {
      const double t = (double)br[c] - (double)qr[c];
      acc += t * t;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) d64[i] = acc;
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < K2; i += 256) {
    const double d = d64[i];
    const uint32_t id = (uint32_t)keys[i];
    uint32_t place = 0;
    for (uint32_t j = 0; j < K2; ++j) place += d64[j] < d || (d64[j] == d && (uint32_t)keys[j] < id);
    if (place < k) {
      ids[qi * k + place] = (int32_t)id;
      if (dists) dists[qi * k + place] = (float)d;
    }
  }
  for (uint32_t i = K2 + threadIdx.x; i < k; i += 256) {  // (fewer rows than k)
    ids[qi * k + i] = -1;
    if (dists) dists[qi * k + i] = INFINITY;
  }
}

// The listed queries' operands and FP32 rows, one after another (a warp per query), and their results back
// to their places.
__global__ void gather_queries_kernel(const uint32_t* __restrict__ list, uint64_t m, const uint4* __restrict__ hi,
                                      const uint4* __restrict__ lo, const float* __restrict__ norms,
                                      const float* __restrict__ q, uint32_t W, uint32_t dim, uint64_t qld, uint32_t gld,
                                      uint4* __restrict__ ghi, uint4* __restrict__ glo, float* __restrict__ gnorms,
                                      float* __restrict__ gq) {
  const uint32_t lane = threadIdx.x & 31, w16 = W / 8;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < m; i += nw) {
    const uint64_t r = list[i];
    for (uint32_t c = lane; c < w16; c += 32) {
      ghi[i * w16 + c] = hi[r * w16 + c];
      if (lo) glo[i * w16 + c] = lo[r * w16 + c];
    }
    for (uint32_t c = lane; c < gld; c += 32) gq[i * gld + c] = c < dim ? q[r * qld + c] : 0.f;
    if (lane == 0) gnorms[i] = norms[r];
  }
}

__global__ void scatter_results_kernel(const uint32_t* __restrict__ list, uint64_t m, uint32_t k,
                                       const int32_t* __restrict__ gi, const float* __restrict__ gd,
                                       int32_t* __restrict__ ids, float* __restrict__ dists) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < m; i += nw) {
    const uint64_t r = list[i];
    for (uint32_t c = lane; c < k; c += 32) {
      ids[r * k + c] = gi[i * k + c];
      if (dists) dists[r * k + c] = gd[i * k + c];
    }
  }
}

}  // namespace

thread_local efg_knn_stats g_knn_stats = {};

// Largest k the tensor-core path serves (the per-thread lists of K2 = k + 16 keys and the buffers
// must fit in shared memory beside two pipeline stages of the split form).
uint32_t tc_knn_max_k() { return 104; }

namespace {

// Converted operands of one call and what the list path needs of them.
struct Operands {
  const __nv_bfloat16 *xh, *xl, *qh, *ql;
  const float *xn, *qn;
  int* flags;
  uint32_t terms;
};

int knn_lists(const float* base, uint64_t n, uint32_t dim, uint32_t ld, const float* q, uint64_t nq, uint32_t qld,
              uint32_t k, int exclude_self, uint64_t first_row, int32_t* ids, float* dists, cudaStream_t s,
              const Operands& op, const uint32_t* qid);

uint32_t next_prime(uint32_t x) {  // the least prime >= x
  for (x = std::max(x, 2u);; ++x) {
    bool prime = true;
    for (uint32_t d = 2; (uint64_t)d * d <= x && prime; ++d) prime = x % d != 0;
    if (prime) return x;
  }
}

// Stream-ordered memory of one call.
struct CallBuf {
  cudaStream_t s;
  std::vector<void*> p;
  explicit CallBuf(cudaStream_t st) : s(st) {}
  ~CallBuf() {
    for (void* x : p)
      if (x) cudaFreeAsync(x, s);
  }
  template <typename T>
  int get(T** out, uint64_t count) {
    void* x = nullptr;
    EFG_CUDA(cudaMallocAsync(&x, count * sizeof(T), s));
    p.push_back(x);
    *out = reinterpret_cast<T*>(x);
    return EFG_OK;
  }
  void drop(void* x) {
    for (void*& y : p)
      if (y == x) {
        cudaFreeAsync(x, s);
        y = nullptr;
      }
  }
};

}  // namespace

int brute_force_knn_tc(const float* base, uint64_t n, uint32_t dim, uint32_t ld, const float* q, uint64_t nq,
                       uint32_t qld, uint32_t k, int exclude_self, uint64_t first_row, int32_t* ids, float* dists,
                       cudaStream_t s, int force_split, uint64_t cand_bytes) {
  if (nq == 0) return EFG_OK;
  if (n >= (1ull << 31) || nq >= (1ull << 31)) return fail(EFG_ERR_ARG, "tensor-core k-NN: more than 2^31 rows");
  if (k > tc_knn_max_k()) return fail(EFG_ERR_ARG, "tensor-core k-NN: k above " + std::to_string(tc_knn_max_k()));
  const uint32_t K2 = (uint32_t)std::min<uint64_t>(k + 16, n);
  const uint32_t W = (dim + TKB - 1) / TKB * TKB, kblocks = W / TKB;
  const uint64_t ntiles = (n + TN - 1) / TN;
  int dev = 0, sms = 148, smem_max = 0;
  EFG_CUDA(cudaGetDevice(&dev));
  EFG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  EFG_CUDA(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  // start, then bounds, screening and selection of each block of queries, end
  struct Events {
    std::vector<cudaEvent_t> e;
    size_t n = 0;  // recorded
    ~Events() {
      for (cudaEvent_t x : e) cudaEventDestroy(x);
    }
    int make() {
      cudaEvent_t x;
      EFG_CUDA(cudaEventCreate(&x));
      e.push_back(x);
      return EFG_OK;
    }
    int record(cudaStream_t st) {
      if (n == e.size()) EFG_TRY(make());
      EFG_CUDA(cudaEventRecord(e[n++], st));
      return EFG_OK;
    }
  } ev;
  for (int i = 0; i < 5; ++i) EFG_TRY(ev.make());  // (one block's)
  CallBuf mem(s);

  // operands: BF16 rows, norms, flags {inexact, error, a buffer too short}.  A thin sample tells whether
  // the low parts are wanted, so that data BF16 holds are converted without them.
  __nv_bfloat16 *xh, *xl = nullptr, *qh, *ql = nullptr;
  float *xn, *qn;
  int* flags;
  EFG_TRY(mem.get(&xh, n * W));
  EFG_TRY(mem.get(&qh, nq * W));
  EFG_TRY(mem.get(&xn, ntiles * TN));
  EFG_TRY(mem.get(&qn, nq));
  EFG_TRY(mem.get(&flags, 4));
  EFG_CUDA(cudaMemsetAsync(flags, 0, 16, s));
  EFG_TRY(ev.record(s));
  auto blocks = [&](uint64_t warps) { return (unsigned)((std::min<uint64_t>(warps, (uint64_t)sms * 64) + 7) / 8); };
  const uint64_t thin = std::max<uint64_t>(1, n / 1024);
  split_bf16_kernel<<<blocks(n / thin + 1), 256, 0, s>>>(base, n, thin, dim, ld, W, nullptr, nullptr, nullptr, n, flags);
  split_bf16_kernel<<<blocks(nq), 256, 0, s>>>(q, nq, 1, dim, qld, W, nullptr, nullptr, nullptr, nq, flags);
  EFG_CUDA(cudaGetLastError());
  int hflags[4] = {0, 0, 0, 0};
  EFG_CUDA(cudaMemcpyAsync(hflags, flags, 16, cudaMemcpyDeviceToHost, s));
  EFG_CUDA(cudaStreamSynchronize(s));
  bool split = force_split || hflags[0];
  for (;;) {
    if (split) {
      EFG_TRY(mem.get(&xl, n * W));
      EFG_TRY(mem.get(&ql, nq * W));
    }
    split_bf16_kernel<<<blocks(ntiles * TN), 256, 0, s>>>(base, n, 1, dim, ld, W, (uint2*)xh, (uint2*)xl, xn,
                                                          ntiles * TN, flags);
    split_bf16_kernel<<<blocks(nq), 256, 0, s>>>(q, nq, 1, dim, qld, W, (uint2*)qh, (uint2*)ql, qn, nq, flags);
    EFG_CUDA(cudaGetLastError());
    if (split) break;
    EFG_CUDA(cudaMemcpyAsync(hflags, flags, 16, cudaMemcpyDeviceToHost, s));
    EFG_CUDA(cudaStreamSynchronize(s));
    if (!hflags[0]) break;
    split = true;  // the sample missed it
  }
  const uint32_t terms = split ? 3u : 1u, parts = split ? 2u : 1u;

  EFG_TRY(ev.record(s));

  // Candidate buffers, and the block of queries they serve at a time (in whole query groups; fewer where
  // memory is short).  rank = K2, + 1 with exclude_self (a sample may hold the query itself).
  const uint32_t rank = K2 + (exclude_self ? 1u : 0u);
  uint32_t cap = 1024;  // three times the 16 x rank expected under a bound from n / 16 rows
  while (cap < 48 * rank && cap < CAND_MAX) cap *= 2;
  constexpr uint64_t QGROUP = 2 * TM;
  const uint64_t most = std::max<uint64_t>(1, (cand_bytes ? cand_bytes : CAND_BYTES) / (8 * cap) / QGROUP) * QGROUP;
  uint64_t QB = nq;
  if (nq > most) {  // blocks of about one size
    const uint64_t nb = (nq + most - 1) / most;
    QB = round_up((nq + nb - 1) / nb, QGROUP);
  }
  uint32_t *qbound, *cnt;
  uint64_t* buf;
  EFG_TRY(mem.get(&qbound, nq));
  EFG_TRY(mem.get(&cnt, 2 * nq));
  uint32_t* over_list = cnt + nq;  // queries whose buffer was too short
  for (;;) {
    const int rc = mem.get(&buf, QB * cap);
    if (rc == EFG_OK) break;
    if (rc != EFG_ERR_NOMEM || QB <= QGROUP) return rc;
    QB = round_up(QB / 2, QGROUP);
  }
  const uint64_t qtiles = (QB + TM - 1) / TM;

  // Query tiles per item, and whether their blocks stay in shared memory: two tiles unless that would
  // leave a tile empty for a few queries (300 queries: three tiles as three items, not two pairs) or the
  // stages would not fit; resident with at least three stages of base blocks beside them, else streamed
  // with those.
  const uint32_t scratch = 32 * SW_ * GRP * 4, norms_b = SW_ * 2 * 64 * 4, queue_b = SW_ * 64 * 12;
  const int64_t room = (int64_t)smem_max - 1024 - 1024 - scratch - norms_b - queue_b;  // alignment pad, barriers
  uint32_t NT = qtiles >= 8 || qtiles % 2 == 0 ? 2u : 1u, qbytes, stage_bytes, stages;
  bool resident;
  for (;; NT = 1) {
    qbytes = NT * kblocks * parts * PART;
    resident = (int64_t)qbytes + 3 * (int64_t)(parts * PART) <= room;
    stage_bytes = resident ? parts * PART : (1 + NT) * parts * PART;
    stages = (uint32_t)std::min<int64_t>(MAX_STAGES, (room - (resident ? qbytes : 0)) / stage_bytes);
    if (stages >= 2 || NT == 1) break;
  }
  CUtensorMap mqh, mql, mxh, mxl;
  EFG_TRY(make_map(&mxh, xh, n, W));
  EFG_TRY(make_map(&mxl, split ? xl : xh, n, W));

  unsigned grid = 0;
  uint32_t nchunks = 1, qgroups = 0;
  uint64_t chunk_tiles = 1, q0 = 0, nqb = 0;  // the block: its first query, its queries (and their groups, maps)
  // One pass of the block's queries over `rows` rows (maps, norms): the chunk count that keeps the SMs busiest, time ~ waves x
  // (tiles per item, and about two for an item's start); chunks of whole groups for the MIN pass.
  auto pass = [&](bool minp, const CUtensorMap& mh, const CUtensorMap& ml, const float* xnorm, uint64_t rows,
                  uint32_t group_tiles, const uint32_t* qbound, uint32_t* qmax, uint32_t* cnt, uint64_t* buf,
                  uint32_t cap, int excl, uint32_t stride = 0, uint32_t box_shift = 0) -> int {
    ScreenArgs a;
    a.stride = stride;
    a.box_shift = box_shift;
    a.rows_box = stride ? (uint32_t)std::min<uint64_t>(1u << box_shift, n / stride) : 0;
    a.W = W;
    const uint64_t tiles = (rows + TN - 1) / TN, unit = std::max<uint32_t>(1, 2 * group_tiles);
    const uint64_t units = (tiles + unit - 1) / unit;
    double best = 1e300;
    for (uint64_t nc = 1; nc <= std::min<uint64_t>(units, 512); ++nc) {
      const uint64_t ct = (units + nc - 1) / nc * unit, real = (tiles + ct - 1) / ct;
      const uint64_t waves = (qgroups * real + sms - 1) / sms;
      const double cost = (double)waves * (double)(ct + 2) + 0.001 * (double)real;
      if (cost < best) {
        best = cost;
        chunk_tiles = ct;
        nchunks = (uint32_t)real;
      }
    }
    a.qnorm = qn + q0;
    a.xnorm = xnorm;
    a.qbound = qbound;
    a.qmax = qmax;
    a.cnt = cnt;
    a.buf = buf;
    a.err = flags + 1;
    a.n = rows;
    a.first_row = first_row + q0;
    a.ntiles = (uint32_t)tiles;
    a.chunk_tiles = (uint32_t)chunk_tiles;
    a.nchunks = nchunks;
    a.qgroups = qgroups;
    a.nq = (uint32_t)nqb;
    a.cap = cap;
    a.kblocks = kblocks;
    a.stages = stages;
    a.exclude_self = excl ? 1u : 0u;
    a.group_tiles = group_tiles;
    a.split = split ? 1u : 0u;
    a.resident = resident ? 1u : 0u;
    a.rel = split ? 1e-5f : 0.f;
    a.stage_bytes = stage_bytes;
    a.o_x = resident ? qbytes : 0;
    a.o_scr = a.o_x + stages * stage_bytes;
    a.o_xn = a.o_scr + scratch;
    a.o_queue = a.o_xn + norms_b;
    const size_t smem = 1024 + (size_t)a.o_queue + queue_b;
    auto kern = NT == 2 ? (!minp    ? tc_screen_kernel<2, APPEND>
                           : stride ? tc_screen_kernel<2, MIN_STRIDED>
                                    : tc_screen_kernel<2, MIN_ROWS>)
                        : (!minp    ? tc_screen_kernel<1, APPEND>
                           : stride ? tc_screen_kernel<1, MIN_STRIDED>
                                    : tc_screen_kernel<1, MIN_ROWS>);
    EFG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    grid = (unsigned)std::min<uint64_t>((uint64_t)qgroups * nchunks, (uint64_t)sms);
    kern<<<grid, STH, smem, s>>>(mqh, mql, mh, ml, a);
    EFG_CUDA(cudaGetLastError());
    return EFG_OK;
  };

  // 1. bounds: how, and the sample
  const size_t sel_smem = (size_t)cap * 8 + (size_t)rank * 8;
  EFG_CUDA(cudaFuncSetAttribute(select_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sel_smem));
  // Rows of the append pass's sample: n / 16 up to 2^20 of them, more for bases so large that the values
  // under the bound of 2^20 rows, n / 2^20 x rank and six deviations, would not fit a buffer (from 23
  // million rows at k = 100; 2000 queries over 45M x 8: 144 ms with all of them in the lists, 40.7 this way).
  const double spread = (double)rank * (1 + 6 / std::sqrt((double)rank));
  uint64_t S1 = std::min<uint64_t>(n / 16, std::max<uint64_t>(1u << 20, (uint64_t)((double)n * spread / cap) + TN)) / TN * TN;
  const uint64_t gtiles = (rank + 3) / 4 * 2;                          // tiles that hold `rank` groups of 64 columns, an even number
  uint32_t S = 0, gt = 0;  // rows of the last bound pass (0: no bounds); tiles per group
  CUtensorMap m0h, m0l, m1h, m1l;  // of the MIN pass and the append pass
  uint64_t min_rows = 0;
  const float* min_norms = xn;
  uint32_t min_stride = 0, box_shift = 0;
  const bool sampled = S1 >= gtiles * TN;
  if (sampled) {
    gt = 1;  // up to a third of the sample for the MIN pass
    while (gt < 16 && gtiles * (2 * gt) * TN * 3 <= S1) gt *= 2;
    // Values of the sample under the MIN pass's bound: a share p of them, where all of the `rank` groups of
    // 64 gt columns have one below it; (1 - p)^(64 gt) rank nq = 1 / 32 says what their buffers must hold.
    // Queries that overrun them go through the lists after all (k = 100, 10k queries at 1M x 960: 167 ms when
    // all did, 65 ms), so the sample is cut while the base's expected candidates (six deviations
    // up) still fit, else the groups doubled.
    const double tail = std::log(32.0 * (double)rank * (double)nq);
    while ((double)S1 * tail > (double)cap * 64 * gt) {
      const uint64_t cut = (uint64_t)((double)cap * 64 * gt / tail) / TN * TN;
      const double expect = (double)n / (double)std::max<uint64_t>(cut, 1) * spread;
      if (cut >= gtiles * gt * TN && expect <= (double)cap) S1 = cut;
      else if (gtiles * (2 * gt) * TN <= S1) gt *= 2;
      else break;
    }
    __nv_bfloat16 *bh, *bl = nullptr;
    float* bn;
    EFG_TRY(mem.get(&bh, S1 * W));
    if (split) EFG_TRY(mem.get(&bl, S1 * W));
    EFG_TRY(mem.get(&bn, S1));
    uint32_t step = (uint32_t)((double)S1 * 0.6180339887) | 1u;
    auto gcd = [](uint64_t x, uint64_t y) {
      while (y) {
        const uint64_t r = x % y;
        x = y;
        y = r;
      }
      return x;
    };
    while (gcd(step, S1) != 1) step += 2;
    scatter_sample_kernel<<<blocks(S1), 256, 0, s>>>((const uint4*)xh, (const uint4*)xl, xn, n, W, (uint32_t)S1, step,
                                                     (uint32_t)(n / S1), (uint4*)bh, (uint4*)bl, bn);
    EFG_CUDA(cudaGetLastError());
    min_rows = gtiles * gt * TN;
    min_norms = bn;
    EFG_TRY(make_map(&m0h, bh, min_rows, W));
    EFG_TRY(make_map(&m0l, split ? bl : bh, min_rows, W));
    EFG_TRY(make_map(&m1h, bh, S1, W));
    EFG_TRY(make_map(&m1l, split ? bl : bh, S1, W));
    S = (uint32_t)S1;
  } else if (n >= 16ull * (rank + 8)) {  // a small base: groups of it all (the last tile may be partly empty)
    const uint64_t full = n / TN;
    // groups of 16 columns, or of 64 columns x gt tiles
    while (full / (gt ? 4 * gt : 2) * 4 >= rank) gt = gt ? 2 * gt : 1;
    if (gt || full * 8 >= rank) {
      // Boxes of 64 or 16 rows (one of a group's) whose rows are a prime number apart, the least that spreads
      // them over the whole base: groups of neighbouring rows would give bounds that let a whole class
      // through where rows come class by class, a multiple of its period where classes alternate (20k x
      // 128 in four classes, 10k queries: 4.2 ms with all of them in the lists, 1.3 ms this way).
      min_rows = gt ? full / (2 * gt) * (2 * gt) * TN : full * TN;
      box_shift = gt ? 6 : 4;
      const uint32_t box = 1u << box_shift;
      min_stride = next_prime((uint32_t)((n + box - 1) / box));
      EFG_TRY(make_map(&m0h, xh, std::min<uint64_t>(box, n / min_stride), min_stride * W, box));
      EFG_TRY(make_map(&m0l, split ? xl : xh, std::min<uint64_t>(box, n / min_stride), min_stride * W, box));
      S = (uint32_t)min_rows;
    }
  }

  double tile_rows = 0;  // queries' rows in the tiles
  for (q0 = 0; q0 < nq; q0 += QB) {
    nqb = std::min(QB, nq - q0);
    qgroups = (uint32_t)(((nqb + TM - 1) / TM + NT - 1) / NT);
    tile_rows += (double)(qgroups * NT * TM);
    EFG_TRY(make_map(&mqh, qh + q0 * W, nqb, W));
    EFG_TRY(make_map(&mql, (split ? ql : qh) + q0 * W, nqb, W));
    if (q0) EFG_TRY(ev.record(s));
    if (S) {
      EFG_CUDA(cudaMemsetAsync(qbound, 0, nqb * 4, s));
      EFG_TRY(pass(true, m0h, m0l, min_norms, min_rows, gt, nullptr, qbound, nullptr, nullptr, 0, 0, min_stride, box_shift));
    }
    if (sampled) {
      EFG_CUDA(cudaMemsetAsync(cnt, 0, nqb * 4, s));
      EFG_TRY(pass(false, m1h, m1l, min_norms, S1, 0, qbound, nullptr, cnt, buf, cap, 0));
      select_kernel<<<(unsigned)nqb, 256, sel_smem, s>>>(buf, cnt, cap, rank, qbound, nullptr, 0, 0, nullptr, 0, 0,
                                                         nullptr, nullptr, nullptr, nullptr, 0);
      EFG_CUDA(cudaGetLastError());
    }
    // 2. the whole base, 3. the candidates' order
    EFG_TRY(ev.record(s));
    EFG_CUDA(cudaMemsetAsync(cnt, 0, nqb * 4, s));
    EFG_TRY(pass(false, mxh, mxl, xn, n, 0, S ? qbound : nullptr, nullptr, cnt, buf, cap, exclude_self));
    EFG_TRY(ev.record(s));
    select_kernel<<<(unsigned)nqb, 256, sel_smem, s>>>(buf, cnt, cap, K2, nullptr, base, dim, ld, q + q0 * qld, qld, k,
                                                       ids + q0 * k, dists ? dists + q0 * k : nullptr, flags + 2,
                                                       over_list, (uint32_t)q0);
    EFG_CUDA(cudaGetLastError());
  }
  EFG_TRY(ev.record(s));
  EFG_CUDA(cudaMemcpyAsync(hflags, flags, 16, cudaMemcpyDeviceToHost, s));
  EFG_CUDA(cudaStreamSynchronize(s));
  if (hflags[1]) return fail(EFG_ERR_DEVICE_LIMIT, "tensor-core k-NN: a pipeline wait ran out (error word " +
                                                       std::to_string(hflags[1]) + ")");
  const uint64_t over = (uint64_t)hflags[2];
  efg_knn_stats lists = {};
  if (over) {
    mem.drop(buf);
    // more values under a bound than a buffer holds (many rows at nearly one distance): sorted lists for
    // these queries, gathered unless they are all of the call's
    Operands op{xh, split ? xl : xh, qh, split ? ql : qh, xn, qn, flags, terms};
    if (over == nq) {
      EFG_TRY(knn_lists(base, n, dim, ld, q, nq, qld, k, exclude_self, first_row, ids, dists, s, op, nullptr));
    } else {
      __nv_bfloat16 *gh, *gl = nullptr;
      float *gn, *gq, *gd = nullptr;
      int32_t* gi;
      const uint32_t gld = (uint32_t)round_up(dim, 4);
      EFG_TRY(mem.get(&gh, over * W));
      if (split) EFG_TRY(mem.get(&gl, over * W));
      EFG_TRY(mem.get(&gn, over));
      EFG_TRY(mem.get(&gq, over * gld));
      EFG_TRY(mem.get(&gi, over * k));
      if (dists) EFG_TRY(mem.get(&gd, over * k));
      gather_queries_kernel<<<blocks(over), 256, 0, s>>>(over_list, over, (const uint4*)qh, (const uint4*)ql, qn, q, W,
                                                         dim, qld, gld, (uint4*)gh, (uint4*)gl, gn, gq);
      EFG_CUDA(cudaGetLastError());
      op.qh = gh;
      op.ql = split ? gl : gh;
      op.qn = gn;
      EFG_TRY(knn_lists(base, n, dim, ld, gq, over, gld, k, exclude_self, first_row, gi, gd, s, op, over_list));
      scatter_results_kernel<<<blocks(over), 256, 0, s>>>(over_list, over, k, gi, gd, ids, dists);
      EFG_CUDA(cudaGetLastError());
      EFG_CUDA(cudaStreamSynchronize(s));  // (a call has its results when it returns)
    }
    lists = g_knn_stats;
  }
  double ms[4] = {0, 0, 0, 0};
  for (size_t i = 0; i + 1 < ev.n; ++i) {
    float t = 0;
    cudaEventElapsedTime(&t, ev.e[i], ev.e[i + 1]);
    ms[i ? 1 + (i - 1) % 3 : 0] += t;
  }
  g_knn_stats.convert_ms = ms[0];
  g_knn_stats.bound_ms = ms[1] + lists.bound_ms;
  g_knn_stats.screen_ms = ms[2] + lists.screen_ms;
  g_knn_stats.merge_ms = ms[3] + lists.merge_ms;
  g_knn_stats.sample_rows = S;
  g_knn_stats.screen_flops = 2.0 * (double)nq * (double)n * (double)dim;
  g_knn_stats.tile_flops = 2.0 * tile_rows * (double)(ntiles * TN) * (double)W * (double)terms + lists.tile_flops;
  g_knn_stats.terms = terms;
  g_knn_stats.stages = stages;
  g_knn_stats.nchunks = nchunks;
  g_knn_stats.ctas = grid;
  g_knn_stats.list_queries = (uint32_t)over;
  return EFG_OK;
}

namespace {

// The same result with sorted lists of K2 keys per (query, chunk), whatever the number of values under a
// bound: for queries whose candidate buffers were too short (qid: their numbers in the call, or null for all).
int knn_lists(const float* base, uint64_t n, uint32_t dim, uint32_t ld, const float* q, uint64_t nq, uint32_t qld,
              uint32_t k, int exclude_self, uint64_t first_row, int32_t* ids, float* dists, cudaStream_t s,
              const Operands& op, const uint32_t* qid) {
  const uint32_t K2 = (uint32_t)std::min<uint64_t>(k + 16, n);
  const uint32_t W = (dim + TKB - 1) / TKB * TKB;
  const uint32_t kblocks = W / TKB;
  const uint64_t qtiles = (nq + TM - 1) / TM;
  int dev = 0, sms = 148;
  EFG_CUDA(cudaGetDevice(&dev));
  EFG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  int smem_max = 0;
  EFG_CUDA(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const __nv_bfloat16 *xh = op.xh, *xl = op.xl, *qh = op.qh, *ql = op.ql;
  const float *xn = op.xn, *qn = op.qn;
  int* flags = op.flags;
  const uint32_t terms = op.terms;
  uint64_t* part = nullptr;
  float *sn = nullptr, *qbound = nullptr;
  auto release = [&] {
    cudaFreeAsync(sn, s);
    cudaFreeAsync(qbound, s);
    cudaFreeAsync(part, s);
  };
  struct Guard {
    decltype(release)& f;
    ~Guard() { f(); }
  } guard{release};
  cudaEvent_t ev[5] = {};
  struct EvGuard {
    cudaEvent_t* e;
    ~EvGuard() {
      for (int i = 0; i < 5; ++i)
        if (e[i]) cudaEventDestroy(e[i]);
    }
  } evguard{ev};
  for (auto& e : ev) EFG_CUDA(cudaEventCreate(&e));
  EFG_CUDA(cudaEventRecord(ev[0], s));
  int hflags[2] = {0, 0};

  // shared memory: pipeline stages, then the per-thread lists, scratch and norm copies
  const uint32_t stage_bytes = 2 * PART;
  // screening warps: eight (two threads per query) while their lists fit, else four
  auto warps_for = [](uint32_t K2l) { return K2l <= 48 ? 8u : 4u; };
  auto layout = [&](uint32_t K2l, uint32_t& stages, uint32_t& o_list, uint32_t& o_scr, uint32_t& o_xn,
                    size_t& smem) -> bool {
    const uint32_t ew = warps_for(K2l);
    const uint32_t lists = 32 * ew * K2l * 8, scratch = 32 * ew * GRP * 4, norms = ew * 2 * TN * 4;
    const int64_t room = (int64_t)smem_max - 1024 - 2048 - lists - scratch - norms;  // alignment pad, barriers
    stages = (uint32_t)std::min<int64_t>(MAX_STAGES, std::max<int64_t>(0, room / stage_bytes));
    o_list = stages * stage_bytes;
    o_scr = o_list + lists;
    o_xn = o_scr + scratch;
    smem = 1024 + (size_t)o_xn + norms;
    return stages >= 2;
  };
  auto launch = [&](const CUtensorMap& mq_h, const CUtensorMap& mq_l, const CUtensorMap& mx_h,
                    const CUtensorMap& mx_l, const float* xnorm, uint64_t rows, uint64_t chunk_rows,
                    uint32_t nch, uint32_t K2l, const float* qb, uint64_t* out, int excl, unsigned* grid_out) -> int {
    TcArgs a;
    uint32_t stages, o_list, o_scr, o_xn;
    size_t smem;
    if (!layout(K2l, stages, o_list, o_scr, o_xn, smem))
      return fail(EFG_ERR_ARG, "tensor-core k-NN: k too large for shared memory");
    a.qnorm = qn;
    a.xnorm = xnorm;
    a.qbound = qb;
    a.part = out;
    a.qid = qid;
    a.err = flags + 1;
    a.n = rows;
    a.chunk = chunk_rows;
    a.first_row = first_row;
    a.nq = (uint32_t)nq;
    a.qtiles = (uint32_t)qtiles;
    a.nchunks = nch;
    a.K2 = K2l;
    a.kblocks = kblocks;
    a.terms = terms;
    a.stages = stages;
    a.exclude_self = excl ? 1u : 0u;
    a.o_list = o_list;
    a.o_scr = o_scr;
    a.o_xn = o_xn;
    const unsigned grid = (unsigned)std::min<uint64_t>(qtiles * nch, (uint64_t)sms);
    if (warps_for(K2l) == 8) {
      EFG_CUDA(cudaFuncSetAttribute(tc_knn_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      tc_knn_kernel<8><<<grid, kThreads<8>, smem, s>>>(mq_h, mq_l, mx_h, mx_l, a);
    } else {
      EFG_CUDA(cudaFuncSetAttribute(tc_knn_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      tc_knn_kernel<4><<<grid, kThreads<4>, smem, s>>>(mq_h, mq_l, mx_h, mx_l, a);
    }
    EFG_CUDA(cudaGetLastError());
    if (grid_out) *grid_out = grid;
    g_knn_stats.stages = stages;
    return EFG_OK;
  };
  {
    uint32_t st, o1, o2, o3;
    size_t sm;
    if (!layout(K2 + 1, st, o1, o2, o3, sm)) return fail(EFG_ERR_ARG, "tensor-core k-NN: k too large for shared memory");
  }

  CUtensorMap mqh, mql, mxh, mxl;
  EFG_TRY(make_map(&mqh, qh, nq, W));
  EFG_TRY(make_map(&mql, ql, nq, W));
  EFG_TRY(make_map(&mxh, xh, n, W));
  EFG_TRY(make_map(&mxl, xl, n, W));

  // 1. bounds from strided samples of the base: the rank-th distance of a sample bounds the whole
  // base's (rank = K2, + 1 with exclude_self: a sample may hold the query itself).  Nested samples
  // growing 8x, each holding the previous one (strides that divide), each pass starting from the
  // previous bound so that it only admits about 8 x rank candidates.
  EFG_CUDA(cudaEventRecord(ev[1], s));
  const uint32_t rank = K2 + (exclude_self ? 1u : 0u);
  const uint32_t CHb = warps_for(rank) / 4;
  uint32_t S = 0;  // rows of the last bound pass
  auto bound_pass = [&](uint32_t rows, const float* prev, float* out) -> int {
    __nv_bfloat16 *bh = nullptr, *bl = nullptr;
    float* bn = nullptr;
    uint64_t* lists = nullptr;
    struct Free {
      cudaStream_t s;
      void* p[4];
      ~Free() {
        for (void* x : p) cudaFreeAsync(x, s);
      }
    } fr{s, {nullptr, nullptr, nullptr, nullptr}};
    // chunks: enough items for the SMs, at most 16 lists per query, at least 1024 rows each
    uint32_t nch = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((sms + qtiles - 1) / qtiles, 16 / CHb));
    nch = std::min<uint32_t>(nch, std::max<uint32_t>(1, rows / 1024));
    const uint32_t crow = (rows / nch + TN - 1) / TN * TN;
    nch = (rows + crow - 1) / crow;
    EFG_CUDA(cudaMallocAsync((void**)&bh, (uint64_t)rows * W * 2, s));
    fr.p[0] = bh;
    EFG_CUDA(cudaMallocAsync((void**)&bl, (uint64_t)rows * W * 2, s));
    fr.p[1] = bl;
    EFG_CUDA(cudaMallocAsync((void**)&bn, (uint64_t)rows * 4, s));
    fr.p[2] = bn;
    EFG_CUDA(cudaMallocAsync((void**)&lists, nq * nch * CHb * rank * 8, s));
    fr.p[3] = lists;
    sample_rows_kernel<<<(unsigned)std::min<uint64_t>((rows + 7) / 8, (uint64_t)sms * 8), 256, 0, s>>>(
        reinterpret_cast<const uint4*>(xh), reinterpret_cast<const uint4*>(xl), xn, n, W, rows,
        reinterpret_cast<uint4*>(bh), reinterpret_cast<uint4*>(bl), bn);
    EFG_CUDA(cudaGetLastError());
    CUtensorMap mbh, mbl;
    EFG_TRY(make_map(&mbh, bh, rows, W));
    EFG_TRY(make_map(&mbl, bl, rows, W));
    EFG_TRY(launch(mqh, mql, mbh, mbl, bn, rows, crow, nch, rank, prev, lists, 0, nullptr));
    bound_kernel<<<(unsigned)std::min<uint64_t>((nq + 127) / 128, 4096), 128, 0, s>>>(
        lists, nq, nch * CHb, rank, rank, terms == 1 ? 0.f : 1e-5f, prev, out);
    EFG_CUDA(cudaGetLastError());
    S = rows;
    return EFG_OK;
  };
  // sample sizes: S0 = 64 x rank (at least 2048) and 8x steps up to n / 16, each a multiple of the
  // previous one (so each sample holds the previous one) and of the tile height
  uint32_t S0 = 2048;
  while (S0 < 64 * rank) S0 *= 2;
  if (n / 16 >= S0) {
    EFG_CUDA(cudaMallocAsync((void**)&qbound, nq * 4, s));
    EFG_CUDA(cudaMallocAsync((void**)&sn, nq * 4, s));
    EFG_TRY(bound_pass(S0, nullptr, qbound));
    uint64_t last = S0;
    const uint64_t cap = std::min<uint64_t>(n / 16, 1u << 20);
    for (uint64_t Si = last * 8; Si <= cap; Si *= 8) {
      EFG_TRY(bound_pass((uint32_t)Si, qbound, sn));
      std::swap(sn, qbound);
      last = Si;
    }
    if (cap / last >= 2) {  // the largest multiple of the last sample within n / 16
      EFG_TRY(bound_pass((uint32_t)(cap / last * last), qbound, sn));
      std::swap(sn, qbound);
    }
  }

  // 2. the whole base in (query tile, base chunk) items: the chunk count that keeps the SMs busiest.
  // Time ~ waves x (tiles per item, and about two for an item's start and its lists' write), plus a
  // little per list in the merge.  A few queries need many chunks (300 queries are three query
  // tiles), so what bounds the count is the merge's 256 lists per query, not the keys in them: a
  // bound of 4096 keys per query left 300 queries x 150k rows (k = 100) as three items on three SMs,
  // 23.3 ms of screening against 0.40 ms in 147 items.
  uint64_t best_nc = 1;
  double best_cost = 1e300;
  const uint32_t CH = warps_for(K2) / 4;  // lists per (query, chunk)
  const uint64_t max_nc = std::max<uint64_t>(1, std::min<uint64_t>(256 / CH, (n + TN - 1) / TN));
  for (uint64_t nc = 1; nc <= max_nc; ++nc) {
    const uint64_t chunk = ((n + nc - 1) / nc + TN - 1) / TN * TN;
    const uint64_t real = (n + chunk - 1) / chunk, itm = qtiles * real;
    const uint64_t waves = (itm + sms - 1) / sms;
    const double cost = (double)waves * (double)(chunk / TN + 2) + 0.02 * (double)(real * qtiles);
    if (cost < best_cost) {
      best_cost = cost;
      best_nc = real;
    }
  }
  const uint64_t chunk = ((n + best_nc - 1) / best_nc + TN - 1) / TN * TN;
  const uint32_t nchunks = (uint32_t)((n + chunk - 1) / chunk);
  EFG_CUDA(cudaMallocAsync((void**)&part, nq * nchunks * CH * K2 * 8, s));
  EFG_CUDA(cudaEventRecord(ev[2], s));
  unsigned grid = 0;
  EFG_TRY(launch(mqh, mql, mxh, mxl, xn, n, chunk, nchunks, K2, S ? qbound : nullptr, part, exclude_self, &grid));
  EFG_CUDA(cudaEventRecord(ev[3], s));
  EFG_TRY(bf_merge_launch(base, dim, ld, q, nq, qld, k, K2, nchunks * CH, part, ids, dists, s));
  EFG_CUDA(cudaEventRecord(ev[4], s));
  EFG_CUDA(cudaMemcpyAsync(hflags, flags, 8, cudaMemcpyDeviceToHost, s));
  EFG_CUDA(cudaStreamSynchronize(s));
  float ms[4] = {0, 0, 0, 0};
  for (int i = 0; i < 4; ++i) cudaEventElapsedTime(&ms[i], ev[i], ev[i + 1]);
  g_knn_stats.convert_ms = ms[0];
  g_knn_stats.bound_ms = ms[1];
  g_knn_stats.screen_ms = ms[2];
  g_knn_stats.merge_ms = ms[3];
  g_knn_stats.sample_rows = S;
  g_knn_stats.screen_flops = 2.0 * (double)nq * (double)n * (double)dim;
  g_knn_stats.tile_flops = 2.0 * (double)(qtiles * TM) * (double)(nchunks * chunk) * (double)W * (double)terms;
  g_knn_stats.terms = terms;
  g_knn_stats.nchunks = nchunks;
  g_knn_stats.ctas = grid;
  if (hflags[1]) return fail(EFG_ERR_DEVICE_LIMIT, "tensor-core k-NN: a pipeline wait ran out (error word " +
                                                        std::to_string(hflags[1]) + ")");
  return EFG_OK;
}

}  // namespace

}  // namespace efg
