// Byte rows of a base whose values are all integers in [0, 255] (SIFT-like descriptors), and the
// NN-descent join over them.
//
// Distances between such rows are integers, and with at most 258 dimensions below 2^24, so FP32
// arithmetic gives them exactly in any order: ||x||^2 + ||y||^2 - 2 x.y in 32-bit integers is the same
// number.  A byte row is a quarter of an FP32 row (one 128-byte line at 128 dimensions, and a base of
// a million rows about fits L2) and __dp4a does four products per instruction.
#include <algorithm>

#include "join.cuh"

namespace efg {
namespace {

// Sets *flag when some value of the rows r0, r0 + step, ... is not an integer in [0, 255].
__global__ void not_bytes_kernel(const float* __restrict__ base, uint64_t n, uint32_t ld4, uint64_t step,
                                 int* __restrict__ flag) {
  const uint64_t rows = (n + step - 1) / step, total = rows * ld4;
  bool bad = false;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t r = i / ld4;
    const float4 x = __ldg(reinterpret_cast<const float4*>(base) + r * step * ld4 + (i - r * ld4));
    bad |= !is_byte(x.x) || !is_byte(x.y) || !is_byte(x.z) || !is_byte(x.w);
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(flag, 1);
}

// FP32 rows -> byte rows of ldb bytes (zero padded) and their squared norms; a warp per row.
__global__ void to_bytes_kernel(const float* __restrict__ base, uint64_t n, uint32_t ld4, uint32_t ldb,
                                uint8_t* __restrict__ out, uint32_t* __restrict__ norm) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n; r += nw) {
    uint32_t acc = 0;
    for (uint32_t c = lane; c < ldb / 4; c += 32) {
      uint32_t w = 0;
      if (c < ld4) {
        const float4 x = __ldg(reinterpret_cast<const float4*>(base) + r * ld4 + c);
        w = (uint32_t)x.x | (uint32_t)x.y << 8 | (uint32_t)x.z << 16 | (uint32_t)x.w << 24;
      }
      reinterpret_cast<uint32_t*>(out + r * ldb)[c] = w;
      acc = __dp4a(w, w, acc);
    }
    acc = __reduce_add_sync(0xffffffffu, acc);
    if (lane == 0) norm[r] = acc;
  }
}

constexpr uint32_t BW = 4;       // warps per CTA
constexpr uint32_t BROWS = 64;   // rows per tile
constexpr uint32_t QUEUE = 256;  // records made at a time (a round of 32 blocks has 1024 at most)
constexpr uint32_t BBLOCK = 32;  // new entries per tile of a node with more rows

struct JoinBytesArgs {
  const uint8_t* rows;
  const uint32_t* norm;
  const uint32_t *new_ids, *new_cnt, *old_ids, *old_cnt;
  const float* bound;
  RecordSink sink;
  uint8_t* found;
  uint32_t* next_node;
  NodeSet set;
  uint32_t count;           // of its nodes
  uint32_t chunks, cmagic;  // 16-byte chunks per row, and ceil(2^16 / chunks) for the division by it
  uint32_t stride;          // of a row in shared memory: an odd number of chunks, in bytes
  uint32_t cap, P, check_k;
};

__device__ __forceinline__ uint4 lds_u4(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}

// Row r of a tile sits in slot (r % 4) * 16 + r / 4: the four rows of a block of four are 16 slots apart
// and eight blocks' rows eight consecutive slots, which an odd stride spreads over the banks.
__device__ __forceinline__ uint32_t row_slot(uint32_t r) { return (r & 3u) * (BROWS / 4) + (r >> 2); }

// The join (InitIndex::join, base_index.hpp:328-371), a warp per node: the node's rows (new entries
// first, then old ones; a node of more than 64 rows tile by tile) go to shared memory once, then a lane
// computes the distances of a 4 x 4 block of pairs, on or above the diagonal of (new groups x all
// groups).  The pairs that make records (a fifth of them) are queued and their records made by whole warps.
// Bound: instruction issue (half of all slots) and the latency of a node's chain (lists, rows, records'
// slots), which 16 warps per SM overlap; products are 64 __dp4a per 16-byte chunk and block.  The 1M x 128
// build's joins: 34.0 ms (28.2 since the first one runs in three parts and overflowing lanes share an atomic),
// 46.7 with each lane making the records of its own pairs, four at a time (half as
// many instructions again), and 37.1 with 48 rows a tile and 20 warps per SM.
__global__ void __launch_bounds__(BW * 32, 4) join_bytes_kernel(const JoinBytesArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(16) uint32_t id_all[BW][BROWS], norm_all[BW][BROWS], bound_all[BW][BROWS];
  __shared__ uint32_t blk_all[BW][32];
  __shared__ uint16_t queue_all[BW][QUEUE];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t* id_sh = id_all[warp];
  uint32_t* norm_sh = norm_all[warp];
  uint32_t* bound_sh = bound_all[warp];
  uint32_t* blk_sh = blk_all[warp];
  uint16_t* queue = queue_all[warp];
  const uint32_t rows0 = (uint32_t)__cvta_generic_to_shared(smem) + warp * BROWS * a.stride;
  uint32_t* dot_sh = reinterpret_cast<uint32_t*>(smem + BW * BROWS * a.stride) + warp * 512;
  uint32_t nk = 0;
  if (lane == 0) nk = atomicAdd(a.next_node, 1u);
  for (;;) {
    const uint32_t k = __shfl_sync(0xffffffffu, nk, 0);
    if (k >= a.count) return;
    if (lane == 0) nk = atomicAdd(a.next_node, 1u);  // the next node's, in flight meanwhile
    const uint64_t node = a.set.node(k);
    const uint32_t nn = a.new_cnt[node], T = nn + a.old_cnt[node];
    bool drop = false;
    // tiles: A new entries from a0 with C entries from c0 on; the first of a block (tri) also covers the
    // pairs within the block
    uint32_t a0 = 0, A = T <= BROWS ? nn : min(BBLOCK, nn), c0 = A;
    bool tri = true;
    while (a0 < nn) {
      const uint32_t C = min(BROWS - A, T - c0), R = A + C;
      for (uint32_t r = lane; r < R; r += 32) {
        const uint32_t e = r < A ? a0 + r : c0 + (r - A);
        const uint32_t id = e < nn ? a.new_ids[node * a.cap + e] : a.old_ids[node * a.cap + e - nn];
        id_sh[r] = id;
        norm_sh[r] = a.norm[id];
        bound_sh[r] = __float2uint_rd(a.bound[id]);  // (distances are integers)
      }
      __syncwarp();
      for (uint32_t e = lane; e < R * a.chunks; e += 32) {
        const uint32_t r = (e * a.cmagic) >> 16, c = e - r * a.chunks;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(rows0 + row_slot(r) * a.stride + c * 16),
                     "l"(a.rows + ((uint64_t)id_sh[r] * a.chunks + c) * 16)
                     : "memory");
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
      // blocks (gx, gy): new group gx with group gy >= gx, or with the candidates' groups
      const uint32_t GX = (A + 3) / 4, GY = (R + 3) / 4, g0 = tri ? 0 : A / 4;
      const uint32_t nb = tri ? GX * GY - GX * (GX - 1) / 2 : GX * (GY - g0);
      for (uint32_t b0 = 0; b0 < nb; b0 += 32) {
        const uint32_t b = b0 + lane;
        uint32_t gx = 0, gy = 0;
        if (b >= nb) {  // (computed for nothing)
        } else if (tri) {
          uint32_t r = b;
          while (r >= GY - gx) {
            r -= GY - gx;
            ++gx;
          }
          gy = gx + r;
        } else {
          gx = b / (GY - g0);
          gy = g0 + b - gx * (GY - g0);
        }
        uint32_t acc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0;
        uint32_t xa = rows0 + gx * a.stride, ya = rows0 + gy * a.stride;
        const uint32_t quarter = (BROWS / 4) * a.stride;
        for (uint32_t c = 0; c < a.chunks; ++c, xa += 16, ya += 16) {
          uint4 x[4], y[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) x[i] = lds_u4(xa + i * quarter);
#pragma unroll
          for (int i = 0; i < 4; ++i) y[i] = lds_u4(ya + i * quarter);
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint32_t s = acc[i * 4 + j];
              s = __dp4a(x[i].x, y[j].x, s);
              s = __dp4a(x[i].y, y[j].y, s);
              s = __dp4a(x[i].z, y[j].z, s);
              s = __dp4a(x[i].w, y[j].w, s);
              acc[i * 4 + j] = s;
            }
        }
        // which of the 16 pairs make a record: bit q = 4 i + j for x's node, 16 + q for y's
        uint32_t put = 0;
        {
          const uint4 xn = *reinterpret_cast<const uint4*>(norm_sh + gx * 4), yn = *reinterpret_cast<const uint4*>(norm_sh + gy * 4);
          const uint4 xb = *reinterpret_cast<const uint4*>(bound_sh + gx * 4), yb = *reinterpret_cast<const uint4*>(bound_sh + gy * 4);
          const uint32_t nx[4] = {xn.x, xn.y, xn.z, xn.w}, ny[4] = {yn.x, yn.y, yn.z, yn.w};
          const uint32_t bx[4] = {xb.x, xb.y, xb.z, xb.w}, by[4] = {yb.x, yb.y, yb.z, yb.w};
#pragma unroll
          for (int q = 0; q < 16; ++q) {
            acc[q] = nx[q / 4] + ny[q % 4] - 2 * acc[q];
            put |= (acc[q] <= bx[q / 4] ? 1u << q : 0u) | (acc[q] <= by[q % 4] ? 0x10000u << q : 0u);
          }
        }
        // pairs of the tile: rows x < A, columns y < R, above the diagonal or past the new entries
        uint32_t ok = 0;
        if (b < nb) {
          const uint32_t na = min(A - gx * 4, 4u), ny = min(R - gy * 4, 4u), y0 = tri ? 0 : max(A, gy * 4) - gy * 4;
          ok = (0xffffu >> (16 - 4 * na)) & (0x1111u * ((1u << ny) - (1u << y0)));
          if (tri && gx == gy) ok &= 0x08ceu;  // j > i
        }
        put &= ok | ok << 16;
        // the distances to shared memory: the records are made by whole warps, a lane each, from a queue of
        // (block, pair, side) -- made by the lanes that found them, a lane's 32 chances had each to be tried
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(dot_sh + (i * 32 + lane) * 4) =
              make_uint4(acc[i * 4], acc[i * 4 + 1], acc[i * 4 + 2], acc[i * 4 + 3]);
        blk_sh[lane] = gx * 4 | gy * 4 << 16;
        if (a.P < a.check_k) {  // a pair whose first side is rejected
          for (uint32_t q = 0; q < 16; ++q) {
            const uint32_t rx = gx * 4 + q / 4, ry = gy * 4 + q % 4;
            if (!(ok >> q & 1u)) continue;
            const bool my_new = (ry < A ? a0 + ry : c0 + (ry - A)) < nn;
            const uint32_t x = id_sh[rx], y = id_sh[ry];
            drop |= !(my_new && y == x) && !(put >> (my_new && y < x ? 16 + q : q) & 1u);
          }
        }
        while (__any_sync(0xffffffffu, put != 0)) {
          uint32_t end = __popc(put);
          uint32_t at = end;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= (uint32_t)o) end += y;
          }
          at = end - at;
          for (; put && at < QUEUE; put &= put - 1) queue[at++] = (uint16_t)(lane << 5 | (__ffs(put) - 1));
          const uint32_t total = min(__shfl_sync(0xffffffffu, end, 31), QUEUE);
          __syncwarp();
          for (uint32_t r = lane; r < total; r += 32) {
            const uint32_t code = queue[r], src = code >> 5, q = code & 15u, blk = blk_sh[src];
            const uint32_t rx = (blk & 0xffffu) + q / 4, ry = (blk >> 16) + q % 4;
            const float d = (float)dot_sh[(q / 4 * 32 + src) * 4 + q % 4];
            const bool to_y = code & 16u;
            const uint32_t x = id_sh[rx], y = id_sh[ry];
            const bool my_new = (ry < A ? a0 + ry : c0 + (ry - A)) < nn;
            if (my_new && y == x) continue;
            // side 0: the larger id into the smaller id's node (an old y into x's)
            const uint32_t t = to_y ? y : x, cand = to_y ? x : y, side = to_y != (my_new && y < x) ? 1u : 0u;
            const uint32_t aux = (uint32_t)(node << 1) | side;
            place_record(a.sink, t, atomicAdd(&a.sink.cnt[t], 1u), d, cand, aux);
          }
          __syncwarp();
        }
      }
      __syncwarp();  // the tile's rows are no longer read
      c0 += C;
      tri = false;
      if (c0 >= T) {  // the next block of new entries
        a0 += A;
        A = min(BBLOCK, nn - min(a0, nn));
        c0 = a0 + A;
        tri = true;
      }
    }
    if (a.P < a.check_k && __any_sync(0xffffffffu, drop) && lane == 0) a.found[node] = 1;
  }
}

}  // namespace

// The byte rows of an index's base, made on first use (the base does not change): idx->bytes_state is
// 1 when they exist, 2 when the base does not fit them.
int make_bytes(efg_index* idx) {
  if (idx->bytes_state) return EFG_OK;
  if (idx->dim > 258) {  // 258 * 255^2 < 2^24
    idx->bytes_state = 2;
    return EFG_OK;
  }
  int dev = 0, sms = 152;
  EFG_CUDA(cudaGetDevice(&dev));
  EFG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  LocalBuf<int> flag(idx->stream);
  EFG_TRY(flag.reserve(1));
  EFG_CUDA(cudaMemsetAsync(flag.p, 0, 4, idx->stream));
  // a thin sample first: other data are known by it
  for (uint64_t step : {std::max<uint64_t>(1, idx->n / 1024), (uint64_t)1}) {
    not_bytes_kernel<<<sms * 8, 256, 0, idx->stream>>>(idx->d_base, idx->n, idx->ld / 4, step, flag.p);
    EFG_CUDA(cudaGetLastError());
    int bad = 0;
    EFG_CUDA(cudaMemcpyAsync(&bad, flag.p, 4, cudaMemcpyDeviceToHost, idx->stream));
    EFG_CUDA(cudaStreamSynchronize(idx->stream));
    if (bad) {
      idx->bytes_state = 2;
      return EFG_OK;
    }
  }
  idx->ldb = (uint32_t)round_up(idx->dim, 16);
  if (idx->bytes.reserve(idx->n * idx->ldb) != EFG_OK || idx->bnorm.reserve(idx->n) != EFG_OK) {
    idx->bytes.release();  // no room: the FP32 rows serve as well
    idx->bnorm.release();
    idx->bytes_state = 2;
    return EFG_OK;
  }
  to_bytes_kernel<<<sms * 8, 256, 0, idx->stream>>>(idx->d_base, idx->n, idx->ld / 4, idx->ldb, idx->bytes.p,
                                                    idx->bnorm.p);
  EFG_CUDA(cudaGetLastError());
  EFG_CUDA(cudaStreamSynchronize(idx->stream));
  idx->bytes_state = 1;
  return EFG_OK;
}

int join_bytes(const uint8_t* rows, const uint32_t* norm, uint64_t n, uint32_t ldb, uint32_t cap, uint32_t P,
               uint32_t check_k, const uint32_t* new_ids, const uint32_t* new_cnt, const uint32_t* old_ids,
               const uint32_t* old_cnt, const float* bound, const RecordSink& sink, uint8_t* found, uint32_t* counter,
               const NodeSet& set, cudaStream_t s) {
  JoinBytesArgs a;
  a.rows = rows;
  a.norm = norm;
  a.new_ids = new_ids;
  a.new_cnt = new_cnt;
  a.old_ids = old_ids;
  a.old_cnt = old_cnt;
  a.bound = bound;
  a.sink = sink;
  a.found = found;
  a.next_node = counter;
  a.set = set;
  a.count = (uint32_t)set.count(n);
  a.chunks = ldb / 16;  // <= 17
  a.cmagic = (65536 + a.chunks - 1) / a.chunks;  // exact for e < 64 * 17 (error e / 65536 * (chunks - 1) < 1 / chunks)
  a.stride = (a.chunks | 1) * 16;
  a.cap = cap;
  a.P = P;
  a.check_k = check_k;
  if (a.count == 0) return EFG_OK;
  int dev = 0, sms = 152, per = 1;
  EFG_CUDA(cudaGetDevice(&dev));
  EFG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const size_t smem = (size_t)BW * (BROWS * a.stride + 2048);
  EFG_CUDA(cudaFuncSetAttribute(join_bytes_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  EFG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, join_bytes_kernel, BW * 32, smem));
  const unsigned grid = (unsigned)std::min<uint64_t>((a.count + BW - 1) / BW, (uint64_t)sms * std::max(per, 1));
  join_bytes_kernel<<<grid, BW * 32, smem, s>>>(a);
  EFG_CUDA(cudaGetLastError());
  return EFG_OK;
}

}  // namespace efg
