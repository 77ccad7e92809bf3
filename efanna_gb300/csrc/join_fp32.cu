// The NN-descent join in FP32 (InitIndex::join, base_index.hpp:328-371): the squared distances of
// every pair new[p] x new[p + 1 ..] and new[p] x old of a node's lists, and their records.
//
// New entries are taken two at a time: x0 = new[p] pairs with Y = new[p+1..] + old, x1 = new[p+1] with
// Y[1..], so every candidate row loaded serves both.  Eight lanes share a candidate row (lane cl its
// chunks cl, cl + 8, cl + 16, cl + 24 of each 512 bytes), so a warp has eight rows in flight with eight
// loads per lane, x0 and x1 stay in registers up to 128 dimensions, and the 16 sums of a pass need four
// shuffles.  The sum of a pair is the one the library's other kernels form with a whole warp per row
// (lane l adds chunks l, l + 32, ..., then the lanes fold by an xor butterfly 16, 8, 4, 2, 1), bit for
// bit: the folds 16 and 8 are between a lane's own four partial sums.
// Of a pass's results lane pairs hold one pair each, one lane per side of the record; the record is
// written after the next pass's loads are issued, so its slot's atomic does not hold them up.
//
// Nodes of many pairs go to a list that whole CTAs take afterwards, a node's new entries dealt to
// their warps: on data with hub nodes one warp's longest node was most of an iteration (20k x 100:
// 1.6 ms of an iteration's 1.6 ms).
#include <algorithm>

#include "join.cuh"

namespace efg {
namespace {

constexpr uint32_t JW = 8;         // warps per CTA
constexpr uint64_t JBIG = 2048;    // pairs above which a node goes to the list

struct JoinFp32Args {
  const float* base;
  const uint32_t *new_ids, *new_cnt, *old_ids, *old_cnt;
  const float* bound;
  RecordSink sink;
  uint8_t* found;
  uint32_t* next_node;
  uint32_t* big;               // big[0]: nodes listed, then their ids
  NodeSet set;
  uint32_t count;  // of its nodes
  uint32_t ld4, cap, P, check_k;
};

__device__ __forceinline__ void sq_chunk(float& acc, const float4& x, const float4& y) {
  const float d0 = x.x - y.x, d1 = x.y - y.y, d2 = x.z - y.z, d3 = x.w - y.w;
  acc += d0 * d0;
  acc += d1 * d1;
  acc += d2 * d2;
  acc += d3 * d3;
}

// A record whose slot has been taken but not yet written.
struct Pending {
  uint32_t t, slot, cand, aux;
  float d;
  bool has;
  __device__ __forceinline__ void take(const RecordSink& s, uint32_t t_, uint32_t cand_, uint32_t aux_, float d_) {
    has = true;
    t = t_;
    cand = cand_;
    aux = aux_;
    d = d_;
    slot = atomicAdd(&s.cnt[t_], 1u);
  }
  __device__ __forceinline__ void write(const RecordSink& s) {
    if (has) place_record(s, t, slot, d, cand, aux);
    has = false;
  }
};

// New entries p0, p0 + pstep, ... (two each) of one node, by one warp: rows of at most 32 chunks.
__device__ __forceinline__ void join_node_one(const JoinFp32Args& a, uint64_t i, uint32_t nn, uint32_t no, uint32_t p0,
                                          uint32_t pstep, Pending& pend) {
  const uint32_t lane = threadIdx.x & 31, cl = lane & 7, g = lane >> 3;
  const uint32_t* nw = a.new_ids + i * a.cap;
  const uint32_t* od = a.old_ids + i * a.cap;
  const float4* base4 = reinterpret_cast<const float4*>(a.base);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  bool drop = false;
  for (uint32_t p = p0; p < nn; p += pstep) {
    const bool two = p + 1 < nn;
    const uint32_t x0 = nw[p], x1 = two ? nw[p + 1] : x0;
    const float b0 = a.bound[x0], b1 = a.bound[x1];
    const uint32_t nl = nn - 1 - p;  // new-list candidates of x0
    const uint32_t m = nl + no;      // Y positions (x1 takes positions 1..m-1)
    const float4* r0 = base4 + (uint64_t)x0 * a.ld4;
    const float4* r1 = base4 + (uint64_t)x1 * a.ld4;
    float4 xa[4], xb[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t c = cl + 8 * k;
      xa[k] = c < a.ld4 ? __ldg(r0 + c) : zero;
      xb[k] = c < a.ld4 ? __ldg(r1 + c) : zero;
    }
    for (uint32_t cb = 0; cb < m; cb += 32) {
      const uint32_t cm = min(32u, m - cb);
      // lane l's candidate (position cb + l; the last one repeated past cm) and its bound
      const uint32_t pos = cb + min(lane, cm - 1);
      const uint32_t cand = pos < nl ? nw[p + 1 + pos] : od[pos - nl];
      const float cbound = a.bound[cand];
      for (uint32_t u0 = 0; u0 < cm; u0 += 8) {  // rows u0 + g and u0 + 4 + g
        const uint32_t ya = __shfl_sync(0xffffffffu, cand, min(u0 + g, cm - 1));
        const uint32_t yb = __shfl_sync(0xffffffffu, cand, min(u0 + 4 + g, cm - 1));
        const float4* ra = base4 + (uint64_t)ya * a.ld4;
        const float4* rb = base4 + (uint64_t)yb * a.ld4;
        float s[2][2][4];  // row, x, partial sum
#pragma unroll
        for (int k = 0; k < 4; ++k) s[0][0][k] = s[0][1][k] = s[1][0][k] = s[1][1][k] = 0.f;
        float4 va[4], vb[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t c = cl + 8 * k;
          va[k] = c < a.ld4 ? __ldg(ra + c) : zero;
          vb[k] = c < a.ld4 ? __ldg(rb + c) : zero;
        }
        pend.write(a.sink);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          sq_chunk(s[0][0][k], xa[k], va[k]);
          sq_chunk(s[0][1][k], xb[k], va[k]);
          sq_chunk(s[1][0][k], xa[k], vb[k]);
          sq_chunk(s[1][1][k], xb[k], vb[k]);
        }
        float v[2][2];
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int x = 0; x < 2; ++x) v[r][x] = (s[r][x][0] + s[r][x][2]) + (s[r][x][1] + s[r][x][3]);
        // lane bit 2 keeps the row, bit 1 the x; bit 0 the record's side
        const bool hi4 = cl & 4, hi2 = cl & 2;
        float h[2];
#pragma unroll
        for (int x = 0; x < 2; ++x)
          h[x] = (hi4 ? v[1][x] : v[0][x]) + __shfl_xor_sync(0xffffffffu, hi4 ? v[0][x] : v[1][x], 4);
        float d = (hi2 ? h[1] : h[0]) + __shfl_xor_sync(0xffffffffu, hi2 ? h[0] : h[1], 2);
        d += __shfl_xor_sync(0xffffffffu, d, 1);
        const uint32_t row = u0 + (hi4 ? 4 + g : g), c = cb + row;
        const uint32_t y = hi4 ? yb : ya, x = hi2 ? x1 : x0;
        const float by = __shfl_sync(0xffffffffu, cbound, min(row, cm - 1)), bx = hi2 ? b1 : b0;
        const bool my_new = c < nl;
        const bool ok = row < cm && (!hi2 || (two && c >= 1)) && !(my_new && y == x);
        // side 0: candidate b into node a = the smaller id of two new entries, else x; side 1: a into b
        const bool swap = my_new && y < x, side = cl & 1;
        const bool into_x = swap == side;
        const bool in = d <= (into_x ? bx : by);
        drop |= ok && !side && !in;
        if (ok && in) pend.take(a.sink, into_x ? x : y, into_x ? y : x, (uint32_t)(i << 1) | (side ? 1u : 0u), d);
      }
    }
  }
  if (a.P < a.check_k && __any_sync(0xffffffffu, drop) && lane == 0) a.found[i] = 1;
}

// The same for longer rows: x0 and x1 are read again with every pass, so a pass takes sixteen rows (six
// loads for eight pairs per lane and chunk), one of the lane's four partial sums at a time; its 32 pairs
// end one to a lane, which makes both sides' records.
__device__ __forceinline__ void join_node_long(const JoinFp32Args& a, uint64_t i, uint32_t nn, uint32_t no,
                                               uint32_t p0, uint32_t pstep, Pending& pend, Pending& pend1) {
  const uint32_t lane = threadIdx.x & 31, cl = lane & 7, g = lane >> 3;
  const uint32_t* nw = a.new_ids + i * a.cap;
  const uint32_t* od = a.old_ids + i * a.cap;
  const float4* base4 = reinterpret_cast<const float4*>(a.base);
  bool drop = false;
  for (uint32_t p = p0; p < nn; p += pstep) {
    const bool two = p + 1 < nn;
    const uint32_t x0 = nw[p], x1 = two ? nw[p + 1] : x0;
    const float b0 = a.bound[x0], b1 = a.bound[x1];
    const uint32_t nl = nn - 1 - p, m = nl + no;
    const float4* r0 = base4 + (uint64_t)x0 * a.ld4;
    const float4* r1 = base4 + (uint64_t)x1 * a.ld4;
    for (uint32_t cb = 0; cb < m; cb += 32) {
      const uint32_t cm = min(32u, m - cb);
      const uint32_t pos = cb + min(lane, cm - 1);
      const uint32_t cand = pos < nl ? nw[p + 1 + pos] : od[pos - nl];
      const float cbound = a.bound[cand];
      for (uint32_t u0 = 0; u0 < cm; u0 += 16) {  // rows u0 + 4 r + g, r < 4
        const float4* ry[4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
          ry[r] = base4 + (uint64_t)__shfl_sync(0xffffffffu, cand, min(u0 + 4 * r + g, cm - 1)) * a.ld4;
        float v[8], w[8];  // [x * 4 + r]
#pragma unroll
        for (int half = 0; half < 2; ++half) {  // partial sums 0 + 2, then 1 + 3
          float s[8];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            float t[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) t[e] = 0.f;
#pragma unroll 2
            for (uint32_t c = cl + 8 * (half + 2 * k); c < a.ld4; c += 32) {
              const float4 xa = __ldg(r0 + c), xb = __ldg(r1 + c);
              float4 y[4];
#pragma unroll
              for (int r = 0; r < 4; ++r) y[r] = __ldg(ry[r] + c);
#pragma unroll
              for (int r = 0; r < 4; ++r) {
                sq_chunk(t[r], xa, y[r]);
                sq_chunk(t[4 + r], xb, y[r]);
              }
            }
            if (half == 0 && k == 0) {
              pend.write(a.sink);
              pend1.write(a.sink);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) s[e] = k == 0 ? t[e] : s[e] + t[e];
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            if (half == 0) w[e] = s[e];
            else v[e] = w[e] + s[e];
          }
        }
        // lane bit 2 keeps the x, bits 1 and 0 the row
        const bool hi4 = cl & 4, hi2 = cl & 2, hi1 = cl & 1;
        float h[4], q[2];
#pragma unroll
        for (int r = 0; r < 4; ++r)
          h[r] = (hi4 ? v[4 + r] : v[r]) + __shfl_xor_sync(0xffffffffu, hi4 ? v[r] : v[4 + r], 4);
#pragma unroll
        for (int r = 0; r < 2; ++r)
          q[r] = (hi2 ? h[2 + r] : h[r]) + __shfl_xor_sync(0xffffffffu, hi2 ? h[r] : h[2 + r], 2);
        const float d = (hi1 ? q[1] : q[0]) + __shfl_xor_sync(0xffffffffu, hi1 ? q[0] : q[1], 1);
        const uint32_t row = u0 + 4 * (cl & 3) + g, c = cb + row;
        const uint32_t y = __shfl_sync(0xffffffffu, cand, min(row, cm - 1)), x = hi4 ? x1 : x0;
        const float by = __shfl_sync(0xffffffffu, cbound, min(row, cm - 1)), bx = hi4 ? b1 : b0;
        const bool my_new = c < nl;
        const bool ok = row < cm && (!hi4 || (two && c >= 1)) && !(my_new && y == x);
        const bool swap = my_new && y < x;  // side 0: the larger id into the smaller id's node
        const bool into_x = ok && d <= bx, into_y = ok && d <= by;
        drop |= ok && !(swap ? into_y : into_x);
        if (into_x) pend.take(a.sink, x, y, (uint32_t)(i << 1) | (swap ? 1u : 0u), d);
        if (into_y) pend1.take(a.sink, y, x, (uint32_t)(i << 1) | (swap ? 0u : 1u), d);
      }
    }
  }
  if (a.P < a.check_k && __any_sync(0xffffffffu, drop) && lane == 0) a.found[i] = 1;
}

template <bool ONE>
__device__ __forceinline__ void join_node(const JoinFp32Args& a, uint64_t i, uint32_t nn, uint32_t no, uint32_t p0,
                                          uint32_t pstep, Pending& pend, Pending& pend1) {
  if (ONE) join_node_one(a, i, nn, no, p0, pstep, pend);
  else join_node_long(a, i, nn, no, p0, pstep, pend, pend1);
}

// A warp per node, nodes taken from a shared counter as warps come free.
template <bool ONE>
__global__ void __launch_bounds__(JW * 32, 2) join_fp32_kernel(const JoinFp32Args a) {
  const uint32_t lane = threadIdx.x & 31;
  Pending pend, pend1;
  pend.has = pend1.has = false;
  for (;;) {
    uint32_t kk = 0;
    if (lane == 0) kk = atomicAdd(a.next_node, 1u);
    const uint32_t k = __shfl_sync(0xffffffffu, kk, 0);
    if (k >= a.count) break;
    const uint64_t i = a.set.node(k);
    const uint32_t nn = a.new_cnt[i], no = a.old_cnt[i];
    if (nn == 0) continue;
    if ((uint64_t)nn * (nn / 2 + no) > JBIG) {
      if (lane == 0) a.big[1 + atomicAdd(a.big, 1u)] = (uint32_t)i;
      continue;
    }
    join_node<ONE>(a, i, nn, no, 0, 2, pend, pend1);
  }
  pend.write(a.sink);
  pend1.write(a.sink);
}

// A CTA per listed node.
template <bool ONE>
__global__ void __launch_bounds__(JW * 32, 2) join_fp32_big_kernel(const JoinFp32Args a) {
  __shared__ uint32_t next;
  Pending pend, pend1;
  pend.has = pend1.has = false;
  const uint32_t n = a.big[0];
  for (;;) {
    if (threadIdx.x == 0) next = atomicAdd(a.next_node + 1, 1u);
    __syncthreads();
    const uint32_t k = next;
    __syncthreads();
    if (k >= n) break;
    const uint64_t i = a.big[1 + k];
    join_node<ONE>(a, i, a.new_cnt[i], a.old_cnt[i], 2 * (threadIdx.x >> 5), 2 * JW, pend, pend1);
  }
  pend.write(a.sink);
  pend1.write(a.sink);
}

}  // namespace

int join_fp32(const float* base, uint64_t n, uint32_t ld, uint32_t cap, uint32_t P, uint32_t check_k,
              const uint32_t* new_ids, const uint32_t* new_cnt, const uint32_t* old_ids, const uint32_t* old_cnt,
              const float* bound, const RecordSink& sink, uint8_t* found, uint32_t* counters, uint32_t* big,
              const NodeSet& set, cudaStream_t s) {
  JoinFp32Args a;
  a.base = base;
  a.new_ids = new_ids;
  a.new_cnt = new_cnt;
  a.old_ids = old_ids;
  a.old_cnt = old_cnt;
  a.bound = bound;
  a.sink = sink;
  a.found = found;
  a.next_node = counters;
  a.big = big;
  a.set = set;
  a.count = (uint32_t)set.count(n);
  a.ld4 = ld / 4;
  a.cap = cap;
  a.P = P;
  a.check_k = check_k;
  if (a.count == 0) return EFG_OK;
  const bool one = a.ld4 <= 32;
  auto kern = one ? join_fp32_kernel<true> : join_fp32_kernel<false>;
  auto kern_big = one ? join_fp32_big_kernel<true> : join_fp32_big_kernel<false>;
  int dev = 0, sms = 152, per = 1;
  EFG_CUDA(cudaGetDevice(&dev));
  EFG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  EFG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, JW * 32, 0));
  const unsigned full = (unsigned)sms * std::max(per, 1);
  kern<<<(unsigned)std::min<uint64_t>((a.count + JW - 1) / JW, full), JW * 32, 0, s>>>(a);
  EFG_CUDA(cudaGetLastError());
  kern_big<<<full, JW * 32, 0, s>>>(a);
  EFG_CUDA(cudaGetLastError());
  return EFG_OK;
}

}  // namespace efg
