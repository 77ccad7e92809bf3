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
constexpr uint32_t BBLOCK = 32;  // new entries per tile of a node with more rows

struct JoinBytesArgs {
  const uint8_t* rows;
  const uint32_t* norm;
  const uint32_t *new_ids, *new_cnt, *old_ids, *old_cnt;
  const float* bound;
  RecordSink sink;
  uint8_t* found;
  uint32_t* next_node;
  uint32_t count, step, skip;
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
// groups).  Bound: the latency of a node's chain (lists, rows, records' slots), which 20 warps per SM
// overlap, and the records' atomics; products are 64 __dp4a per 16-byte chunk and block.
__global__ void __launch_bounds__(BW * 32, 5) join_bytes_kernel(const JoinBytesArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint32_t id_all[BW][BROWS], norm_all[BW][BROWS];
  __shared__ float bound_all[BW][BROWS];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t* id_sh = id_all[warp];
  uint32_t* norm_sh = norm_all[warp];
  float* bound_sh = bound_all[warp];
  const uint32_t rows0 = (uint32_t)__cvta_generic_to_shared(smem) + warp * BROWS * a.stride;
  uint32_t* dot_sh = reinterpret_cast<uint32_t*>(smem + BW * BROWS * a.stride) + warp * 512;
  uint32_t nk = 0;
  if (lane == 0) nk = atomicAdd(a.next_node, 1u);
  for (;;) {
    const uint32_t k = __shfl_sync(0xffffffffu, nk, 0);
    if (k >= a.count) return;
    if (lane == 0) nk = atomicAdd(a.next_node, 1u);  // the next node's, in flight meanwhile
    const uint64_t node = a.skip ? (uint64_t)k + k / (a.step - 1) + 1 : (uint64_t)k * a.step;
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
        bound_sh[r] = a.bound[id];
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
      for (uint32_t b = lane; b < nb; b += 32) {
        uint32_t gx = 0, gy = 0;
        if (tri) {
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
        // the lane's 16 products through shared memory, so that the record code below exists once per
        // column and not 16 times: unrolled over the rows too it outgrew the instruction cache
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(dot_sh + (i * 32 + lane) * 4) =
              make_uint4(acc[i * 4], acc[i * 4 + 1], acc[i * 4 + 2], acc[i * 4 + 3]);
#pragma unroll 1
        for (uint32_t i = 0; i < 4; ++i) {
          const uint32_t rx = gx * 4 + i;
          if (rx >= A) break;
          const uint32_t x = id_sh[rx], nx = norm_sh[rx];
          const float bx = bound_sh[rx];
          const uint4 dv = *reinterpret_cast<const uint4*>(dot_sh + (i * 32 + lane) * 4);
          const uint32_t dot[4] = {dv.x, dv.y, dv.z, dv.w};
          // four pairs' slots first, then their records: the atomics' latencies overlap
          uint32_t slot[8], ta[8];
          float dd[4];
          uint32_t put = 0;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t ry = gy * 4 + j;
            const bool pair = ry < R && (tri ? ry > rx : ry >= A);
            const uint32_t y = id_sh[ry];
            const float by = bound_sh[ry];
            const bool my_new = (ry < A ? a0 + ry : c0 + (ry - A)) < nn;
            dd[j] = (float)(nx + norm_sh[ry] - 2 * dot[j]);
            const bool ok = pair && !(my_new && y == x);
            const bool swap = my_new && y < x;  // side 0: the larger id into the smaller id's node
            const bool in0 = dd[j] <= (swap ? by : bx), in1 = dd[j] <= (swap ? bx : by);
            put |= (ok && in0 ? 1u : 0u) << (2 * j) | (ok && in1 ? 2u : 0u) << (2 * j);
            drop |= ok && !in0;
            ta[2 * j] = swap ? y : x;
            ta[2 * j + 1] = swap ? x : y;
          }
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (put >> q & 1u) slot[q] = atomicAdd(&a.sink.cnt[ta[q]], 1u);
          uint32_t over = 0;
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (put >> q & 1u) {
              if (slot[q] < a.sink.W)
                a.sink.bucket[(uint64_t)ta[q] * a.sink.W + slot[q]] =
                    make_uint4(ta[q ^ 1], __float_as_uint(dd[q >> 1]), (uint32_t)(node << 1) | (q & 1), ta[q]);
              else over |= 1u << q;
            }
          if (over) {
#pragma unroll
            for (int q = 0; q < 8; ++q)
              if (over >> q & 1u)
                place_overflow(a.sink, ta[q], slot[q], dd[q >> 1], ta[q ^ 1], (uint32_t)(node << 1) | (q & 1));
          }
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
  EFG_TRY(idx->bytes.reserve(idx->n * idx->ldb));
  EFG_TRY(idx->bnorm.reserve(idx->n));
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
               uint32_t step, uint32_t skip, cudaStream_t s) {
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
  a.step = step;
  a.skip = skip;
  const uint64_t first = (n + step - 1) / step;  // nodes k * step
  a.count = (uint32_t)(skip ? n - first : first);
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
