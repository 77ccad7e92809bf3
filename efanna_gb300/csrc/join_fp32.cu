// The NN-descent join in FP32 (InitIndex::join, base_index.hpp:328-371): the squared distances of
// every pair new[p] x new[p + 1 ..] and new[p] x old of a node's lists, and their records.
#include <algorithm>

#include "join.cuh"

namespace efg {
namespace {

// One warp per node, nodes taken from a shared counter as warps come free (pair counts differ by an
// order of magnitude, so a fixed assignment leaves most warps of a block idle behind its longest node).
// New entries are taken two at a time: x0 = new[p] pairs with Y = new[p+1..] + old, x1 = new[p+1]
// with Y[1..], so every candidate row loaded serves both; four rows per pass, the 2 x 4 sums
// reduced together.
__global__ void __launch_bounds__(256, 4) join_fp32_kernel(
    const float* __restrict__ base, uint32_t ld4, uint32_t cap, uint32_t P, uint32_t check_k,
    const uint32_t* __restrict__ new_ids, const uint32_t* __restrict__ new_cnt, const uint32_t* __restrict__ old_ids,
    const uint32_t* __restrict__ old_cnt, const float* __restrict__ bound, const RecordSink sink,
    uint8_t* __restrict__ found, uint32_t* __restrict__ next_node, uint32_t count, uint32_t step, uint32_t skip) {
  const uint32_t lane = threadIdx.x & 31;
  for (;;) {
    uint32_t ii = 0;
    if (lane == 0) ii = atomicAdd(next_node, 1u);
    const uint32_t k = __shfl_sync(0xffffffffu, ii, 0);
    if (k >= count) return;
    const uint64_t i = skip ? (uint64_t)k + k / (step - 1) + 1 : (uint64_t)k * step;
    const uint32_t nn = new_cnt[i], no = old_cnt[i];
    if (nn == 0) continue;
    const uint32_t* nw = new_ids + i * cap;
    const uint32_t* od = old_ids + i * cap;
    bool found_drop = false;
    for (uint32_t p = 0; p < nn; p += 2) {
      const bool two = p + 1 < nn;
      const uint32_t x0 = nw[p], x1 = two ? nw[p + 1] : x0;
      const uint32_t nl = nn - 1 - p;  // new-list candidates of x0
      const uint32_t m = nl + no;      // Y positions (x1 takes positions 1..m-1)
      const float4* r0 = reinterpret_cast<const float4*>(base) + (uint64_t)x0 * ld4;
      const float4* r1 = reinterpret_cast<const float4*>(base) + (uint64_t)x1 * ld4;
      for (uint32_t cb = 0; cb < m; cb += 32) {
        const uint32_t cm = min(32u, m - cb);
        // lane l's candidate (position cb + l; the last one repeated past cm), loaded once per
        // chunk and handed to the passes by shuffles
        const uint32_t cl = cb + min(lane, cm - 1);
        const uint32_t cand = cl < nl ? nw[p + 1 + cl] : od[cl - nl];
        float mine0 = 0.f, mine1 = 0.f;
        for (uint32_t u0 = 0; u0 < cm; u0 += 4) {
          float acc[8];  // [0..4): x0 against rows u0..u0+3, [4..8): x1 against them
          const float4* ry[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint32_t yu = __shfl_sync(0xffffffffu, cand, min(u0 + u, cm - 1));
            ry[u] = reinterpret_cast<const float4*>(base) + (uint64_t)yu * ld4;
            acc[u] = 0.f;
            acc[u + 4] = 0.f;
          }
          for (uint32_t c4 = lane; c4 < ld4; c4 += 32) {
            const float4 a = __ldg(r0 + c4), b = __ldg(r1 + c4);
            float4 yv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) yv[u] = __ldg(ry[u] + c4);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              float d0 = a.x - yv[u].x, d1 = a.y - yv[u].y, d2 = a.z - yv[u].z, d3 = a.w - yv[u].w;
              acc[u] += d0 * d0;
              acc[u] += d1 * d1;
              acc[u] += d2 * d2;
              acc[u] += d3 * d3;
              float e0 = b.x - yv[u].x, e1 = b.y - yv[u].y, e2 = b.z - yv[u].z, e3 = b.w - yv[u].w;
              acc[u + 4] += e0 * e0;
              acc[u + 4] += e1 * e1;
              acc[u + 4] += e2 * e2;
              acc[u + 4] += e3 * e3;
            }
          }
          // lanes 4r .. 4r+3 end with sum r: r < 4 x0's row u0+r, r >= 4 x1's row u0+r-4; row
          // u's sums move to lane u0 + u
          const float tot = reduce8_rows(acc, lane);
          const uint32_t u = (lane - u0) & 3;
          const float d0 = __shfl_sync(0xffffffffu, tot, u * 4), d1 = __shfl_sync(0xffffffffu, tot, (u + 4) * 4);
          if (lane - u0 < 4u) {
            mine0 = d0;
            mine1 = d1;
          }
        }
        const uint32_t c = cb + lane;
        if (lane < cm) {
          const bool my_new = c < nl;
          found_drop |= join_pair_records(sink, i, x0, cand, my_new, mine0, P, check_k, bound);
          if (two && c >= 1)  // x1's candidate c - 1 (new exactly when x0's candidate c is)
            found_drop |= join_pair_records(sink, i, x1, cand, my_new, mine1, P, check_k, bound);
        }
      }
    }
    if (__any_sync(0xffffffffu, found_drop) && lane == 0) found[i] = 1;
  }
}

}  // namespace

int join_fp32(const float* base, uint64_t n, uint32_t ld, uint32_t cap, uint32_t P, uint32_t check_k,
              const uint32_t* new_ids, const uint32_t* new_cnt, const uint32_t* old_ids, const uint32_t* old_cnt,
              const float* bound, const RecordSink& sink, uint8_t* found, uint32_t* counter, uint32_t step,
              uint32_t skip, cudaStream_t s) {
  const uint64_t first = (n + step - 1) / step, count = skip ? n - first : first;  // nodes k * step, or the others
  if (count == 0) return EFG_OK;
  int dev = 0, sms = 152, per = 1;
  EFG_CUDA(cudaGetDevice(&dev));
  EFG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  EFG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, join_fp32_kernel, 256, 0));
  const unsigned grid = (unsigned)std::min<uint64_t>((count + 7) / 8, (uint64_t)sms * std::max(per, 1));
  join_fp32_kernel<<<grid, 256, 0, s>>>(base, ld / 4, cap, P, check_k, new_ids, new_cnt, old_ids, old_cnt, bound, sink,
                                        found, counter, (uint32_t)count, step, skip);
  EFG_CUDA(cudaGetLastError());
  return EFG_OK;
}

}  // namespace efg
