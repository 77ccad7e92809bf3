// Randomised truncated KD-trees, built level-synchronously for all trees at once.
//
// Reference: buildTrees / the tree part of initGraph (algorithm/kdtreeub_index.hpp:1192-1276,
// 1295-1363), meanSplit (:902-953), selectDivision (:974-999), planeSplit (:954-973),
// DFSbuild (:1138-1167).  Per node, as in the reference:
//   * mean and variance over the first min(101, count) ids of the node's id range, summed in id
//     order (FP32, no fused multiply-add);
//   * the split dimension is one of the (up to) 5 largest variances, ranked by (variance desc,
//     dimension asc) — the order selectDivision's insertion produces — picked at random;
//   * the cut is the mean in that dimension; ids with value < cut, == cut, > cut are laid out in
//     that order and the split index follows meanSplit's balancing rule;
//   * while fewer than 1100 nodes are active (all trees together) every active node is split and
//     children with more than S ids stay active (the BFS phase); afterwards nodes split while they
//     hold more than TNS ids (the DFS phase).
// Where the reference draws from std::rand()/mt19937 and partitions with Hoare swaps, this build
// uses a Feistel permutation per tree, a counter hash for the split choice and a stable
// three-way partition, so the trees are a pure function of (data, seed): the oracle's canonical
// mode builds identical trees.
//
// Layout during the build: ids[t*n + pos] (tree-major leaf lists, double-buffered),
// owner[t*n + pos] = node holding position pos; node records in structure-of-arrays form.
#include <algorithm>
#include <vector>

#include "scan.cuh"

namespace efg {

static constexpr int T_SAMPLE = 101;  // SAMPLE_NUM + 1 (kdtreeub_index.hpp:912)
static constexpr int T_RAND_DIM = 5;  // RAND_DIM (kdtreeub_index.hpp:1102)

struct NodeArrays {
  uint32_t *start, *end;
  int32_t *tree, *level, *left, *right, *dim, *split_at;  // split_at = level + 1 when split
  float* val;
};

__global__ void perm_init_kernel(uint32_t* ids, int32_t* owner, uint64_t n, uint32_t ntrees, uint64_t seed) {
  uint64_t total = n * ntrees;
  for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < total; g += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t t = (uint32_t)(g / n), i = (uint32_t)(g % n);
    ids[g] = feistel_perm(i, (uint32_t)n, hash4(seed, TAG_PERM, t, 0, 0));
    owner[g] = (int32_t)t;  // node t is tree t's root
  }
}

__global__ void roots_init_kernel(NodeArrays na, uint32_t ntrees, uint64_t n) {
  uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntrees) return;
  na.start[t] = 0;
  na.end[t] = (uint32_t)n;
  na.tree[t] = (int32_t)t;
  na.level[t] = 0;
  na.left[t] = na.right[t] = -1;
  na.dim[t] = -1;
  na.val[t] = 0.f;
  na.split_at[t] = 0;
}

// Four consecutive values of a row, from FP32 rows or from byte rows (ldw floats or bytes per row).
__device__ __forceinline__ float4 row_quad(const float* __restrict__ rows, uint32_t ldw, uint32_t id, uint32_t q) {
  return __ldg(reinterpret_cast<const float4*>(rows + (uint64_t)id * ldw) + q);
}
__device__ __forceinline__ float4 row_quad(const uint8_t* __restrict__ rows, uint32_t ldw, uint32_t id, uint32_t q) {
  const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(rows + (uint64_t)id * ldw) + q);
  // byte b as the low mantissa bits of 2^23: exact, and off the conversion unit
  float4 v;
  v.x = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440)) - 8388608.f;
  v.y = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7441)) - 8388608.f;
  v.z = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7442)) - 8388608.f;
  v.w = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7443)) - 8388608.f;
  return v;
}

// Takes the T_RAND_DIM best of the warp's candidates (c per lane; taken[i]: not one) in selectDivision's
// rank order, value descending, then index ascending; lane r returns the r-th (value -1, index
// 0x7fffffff when there are fewer).  Variances are not negative, so their bits order like them.
template <int C>
__device__ __forceinline__ void warp_top(const float (&val)[C], const int32_t (&idx)[C], bool (&taken)[C],
                                         float& out_v, int32_t& out_i) {
  const uint32_t lane = threadIdx.x & 31;
  out_v = -1.0f;
  out_i = 0x7fffffff;
#pragma unroll
  for (int r = 0; r < T_RAND_DIM; ++r) {
    uint32_t key = 0;  // best value's bits + 1 (0: no candidate left)
#pragma unroll
    for (int c = 0; c < C; ++c)
      if (!taken[c]) key = max(key, __float_as_uint(val[c]) + 1u);
    const uint32_t best = __reduce_max_sync(0xffffffffu, key);
    if (best == 0) break;
    uint32_t who = 0x7fffffffu;
#pragma unroll
    for (int c = 0; c < C; ++c)
      if (!taken[c] && __float_as_uint(val[c]) + 1u == best) who = min(who, (uint32_t)idx[c]);
    const uint32_t win = __reduce_min_sync(0xffffffffu, who);
#pragma unroll
    for (int c = 0; c < C; ++c) taken[c] |= (uint32_t)idx[c] == win;
    if (lane == (uint32_t)r) {
      out_v = __uint_as_float(best - 1u);
      out_i = (int32_t)win;
    }
  }
}

// Statistics, split dimension and cut value of the active nodes: `wpn` warps of a block of eight per
// node, each over its blocks of 128 dimensions, a lane four of them (one 16-byte load per row, or one
// 4-byte load from byte rows); the sums of a dimension run in id order in one lane, eight rows in
// flight.  Bound: the latency of the dependent sums at the top levels (few nodes), the row reads below.
// With one warp per node and one dimension per lane this took 15.3 ms of the 1M x 128 build's trees
// (8 trees, 27 levels) and 27.3 ms at 100k x 960.
template <typename Row>
__global__ void __launch_bounds__(256) split_stats_kernel(
    const Row* __restrict__ rows, uint32_t ldw, uint32_t dim, uint64_t n, const uint32_t* __restrict__ ids,
    NodeArrays na, const int32_t* __restrict__ active, uint32_t nactive, uint32_t wpn, int32_t level, int phaseB,
    uint32_t tns, uint64_t seed, uint32_t* __restrict__ split_flag) {
  extern __shared__ float smean[];  // (8 / wpn) * dim
  __shared__ float cand_v[8][T_RAND_DIM];
  __shared__ int32_t cand_i[8][T_RAND_DIM];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t slot = warp / wpn, part = warp - slot * wpn;
  const uint32_t a = blockIdx.x * (8 / wpn) + slot;
  const bool here = a < nactive;
  float* mean = smean + (size_t)slot * dim;
  const int32_t v = here ? active[a] : 0;
  const uint32_t s = here ? na.start[v] : 0, count = here ? na.end[v] - s : 0;
  const int32_t t = here ? na.tree[v] : 0;
  const bool split = here && !(phaseB && count <= tns);  // else a DFSbuild leaf (kdtreeub_index.hpp:1142-1149)
  if (split) {
    const uint32_t* seg = ids + (uint64_t)t * n + s;
    const uint32_t cnt = min((uint32_t)T_SAMPLE, count);
    const float inv = __fdiv_rn(1.0f, (float)cnt);
    uint32_t sid[4];  // lane l: sample ids l, l + 32, l + 64, l + 96
#pragma unroll
    for (int j = 0; j < 4; ++j) sid[j] = j * 32 + lane < cnt ? __ldg(seg + j * 32 + lane) : 0u;
    float bv = -1.0f;  // lane r: the best r-th of this warp's dimensions so far
    int32_t bi = 0x7fffffff;
    for (uint32_t kb = part * 128; kb < dim; kb += wpn * 128) {
      const uint32_t k = kb + lane * 4;
      const bool in = k < dim;
      const uint32_t q = in ? k / 4 : 0;
      float4 m = make_float4(0.f, 0.f, 0.f, 0.f), var = m;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t jc = cnt > j * 32u ? min(32u, cnt - j * 32u) : 0u;
        for (uint32_t u0 = 0; u0 < jc; u0 += 8) {
          float4 x[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) x[u] = row_quad(rows, ldw, __shfl_sync(0xffffffffu, sid[j], min(u0 + u, jc - 1)), q);
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (u0 + u < jc) {
              m.x = __fadd_rn(m.x, x[u].x);
              m.y = __fadd_rn(m.y, x[u].y);
              m.z = __fadd_rn(m.z, x[u].z);
              m.w = __fadd_rn(m.w, x[u].w);
            }
        }
      }
      m.x = __fmul_rn(m.x, inv);
      m.y = __fmul_rn(m.y, inv);
      m.z = __fmul_rn(m.z, inv);
      m.w = __fmul_rn(m.w, inv);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t jc = cnt > j * 32u ? min(32u, cnt - j * 32u) : 0u;
        for (uint32_t u0 = 0; u0 < jc; u0 += 8) {
          float4 x[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) x[u] = row_quad(rows, ldw, __shfl_sync(0xffffffffu, sid[j], min(u0 + u, jc - 1)), q);
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (u0 + u < jc) {
              const float d0 = __fsub_rn(x[u].x, m.x), d1 = __fsub_rn(x[u].y, m.y);
              const float d2 = __fsub_rn(x[u].z, m.z), d3 = __fsub_rn(x[u].w, m.w);
              var.x = __fadd_rn(var.x, __fmul_rn(d0, d0));
              var.y = __fadd_rn(var.y, __fmul_rn(d1, d1));
              var.z = __fadd_rn(var.z, __fmul_rn(d2, d2));
              var.w = __fadd_rn(var.w, __fmul_rn(d3, d3));
            }
        }
      }
      const float mk[4] = {m.x, m.y, m.z, m.w};
      float cv[5] = {var.x, var.y, var.z, var.w, bv};
      int32_t ci[5];
      bool taken[5];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const bool is = in && k + c < dim;
        if (is) mean[k + c] = mk[c];
        ci[c] = (int32_t)(k + c);
        taken[c] = !is;
      }
      ci[4] = bi;
      taken[4] = bi == 0x7fffffff;
      warp_top<5>(cv, ci, taken, bv, bi);
    }
    if (lane < T_RAND_DIM) {
      cand_v[warp][lane] = bv;
      cand_i[warp][lane] = bi;
    }
  }
  __syncthreads();
  if (!here || part != 0) return;
  if (!split) {
    if (lane == 0) {
      na.dim[v] = -1;
      split_flag[a] = 0;
    }
    return;
  }
  // the node's best over its warps' (at most 40 candidates)
  float cv[2];
  int32_t ci[2];
  bool taken[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const uint32_t e = c * 32 + lane, w = e / T_RAND_DIM;
    const bool is = w < wpn;
    cv[c] = is ? cand_v[warp + w][e - w * T_RAND_DIM] : -1.0f;
    ci[c] = is ? cand_i[warp + w][e - w * T_RAND_DIM] : 0x7fffffff;
    taken[c] = ci[c] == 0x7fffffff;
  }
  float tv;
  int32_t ti;
  warp_top<2>(cv, ci, taken, tv, ti);
  const int num = __popc(__ballot_sync(0xffffffffu, lane < T_RAND_DIM && ti != 0x7fffffff));
  const uint32_t rnd = (uint32_t)(hash4(seed, TAG_DIM, (uint64_t)t, (uint64_t)level, (uint64_t)s) % (uint64_t)num);
  const int32_t cutdim = __shfl_sync(0xffffffffu, ti, rnd);
  if (lane == 0) {
    na.dim[v] = cutdim;
    na.val[v] = mean[cutdim];
    na.split_at[v] = level + 1;
    split_flag[a] = 1;
  }
}

// Packed class counters per position: (is_less << 32) | is_equal, zero outside split nodes.
__global__ void classify_kernel(const float* __restrict__ base, uint32_t ld, uint64_t n, uint32_t ntrees,
                                const uint32_t* __restrict__ ids, const int32_t* __restrict__ owner, NodeArrays na,
                                int32_t level, uint64_t* __restrict__ flags) {
  uint64_t total = n * ntrees;
  for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < total; g += (uint64_t)gridDim.x * blockDim.x) {
    int32_t v = owner[g];
    uint64_t f = 0;
    if (na.split_at[v] == level + 1) {
      float x = __ldg(base + (uint64_t)ids[g] * ld + na.dim[v]);
      float c = na.val[v];
      if (x < c) f = 1ULL << 32;
      else if (x <= c) f = 1ULL;
    }
    flags[g] = f;
  }
}

// One thread per active node: split index, children, and the next level's activity flags.
__global__ void finish_nodes_kernel(NodeArrays na, uint64_t n, const int32_t* __restrict__ active, uint32_t nactive,
                                    const uint32_t* __restrict__ child_off, const uint64_t* __restrict__ pref,
                                    int32_t base_node, int32_t level, int phaseB, uint32_t S,
                                    uint32_t* __restrict__ mids, uint32_t* __restrict__ next_flag,
                                    int32_t* __restrict__ next_cand) {
  uint32_t a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= nactive) return;
  int32_t v = active[a];
  next_flag[2 * a] = next_flag[2 * a + 1] = 0;
  if (na.split_at[v] != level + 1) return;
  uint32_t s = na.start[v], e = na.end[v], count = e - s;
  uint64_t g0 = (uint64_t)na.tree[v] * n + s, g1 = g0 + count;
  uint64_t d = pref[g1] - pref[g0];
  uint32_t nless = (uint32_t)(d >> 32), neq = (uint32_t)(d & 0xffffffffu);
  uint32_t lim1 = nless, lim2 = nless + neq;
  uint32_t index;  // meanSplit's split-index rule (kdtreeub_index.hpp:942-950)
  if (lim1 > count / 2) index = lim1;
  else if (lim2 < count / 2) index = lim2;
  else index = count / 2;
  if ((lim1 == count) || (lim2 == 0)) index = count / 2;
  mids[a] = index;
  int32_t L = base_node + 2 * (int32_t)child_off[a], R = L + 1;
  na.left[v] = L;
  na.right[v] = R;
  int32_t t = na.tree[v];
  na.start[L] = s;
  na.end[L] = s + index;
  na.start[R] = s + index;
  na.end[R] = e;
  na.tree[L] = na.tree[R] = t;
  na.level[L] = na.level[R] = level + 1;
  na.left[L] = na.right[L] = na.left[R] = na.right[R] = -1;
  na.dim[L] = na.dim[R] = 0;  // value-initialised Node (kdtreeub_index.hpp:1249)
  na.val[L] = na.val[R] = 0.f;
  na.split_at[L] = na.split_at[R] = 0;
  next_cand[2 * a] = L;
  next_cand[2 * a + 1] = R;
  if (phaseB) {
    next_flag[2 * a] = next_flag[2 * a + 1] = 1;
  } else {
    next_flag[2 * a] = index > S;
    next_flag[2 * a + 1] = count - index > S;
  }
}

// Stable three-way scatter of the ids of split nodes; owner[] switches to the children.
__global__ void scatter_kernel(uint64_t n, uint32_t ntrees, const uint32_t* __restrict__ ids_in,
                               uint32_t* __restrict__ ids_out, int32_t* __restrict__ owner, NodeArrays na,
                               int32_t level, const uint64_t* __restrict__ pref) {
  uint64_t total = n * ntrees;
  for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < total; g += (uint64_t)gridDim.x * blockDim.x) {
    int32_t v = owner[g];
    uint32_t id = ids_in[g];
    if (na.split_at[v] != level + 1) {
      ids_out[g] = id;
      continue;
    }
    uint32_t s = na.start[v], count = na.end[v] - s;
    uint64_t g0 = (uint64_t)na.tree[v] * n + s;
    uint64_t pg = pref[g] - pref[g0], pt = pref[g0 + count] - pref[g0];
    uint32_t rl = (uint32_t)(pg >> 32), re = (uint32_t)pg, nl = (uint32_t)(pt >> 32), ne = (uint32_t)pt;
    uint32_t off = (uint32_t)(g - g0);
    uint64_t fg = pref[g + 1] - pref[g];
    uint32_t np;
    if (fg >> 32) np = rl;
    else if (fg & 0xffffffffu) np = nl + re;
    else np = nl + ne + (off - rl - re);
    ids_out[g0 + np] = id;
    uint32_t mid = na.end[na.left[v]] - s;
    owner[g] = off < mid ? na.left[v] : na.right[v];
  }
}

__global__ void compact_kernel(const uint32_t* __restrict__ flag, const uint32_t* __restrict__ pos,
                               const int32_t* __restrict__ cand, uint32_t m, int32_t* __restrict__ out) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < m && flag[i]) out[pos[i]] = cand[i];
}

__global__ void to_dnodes_kernel(NodeArrays na, uint32_t nnodes, DNode* __restrict__ out) {
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nnodes) return;
  DNode d;
  d.div_dim = na.dim[v];
  d.div_val = na.val[v];
  if (na.left[v] >= 0) {
    d.left = na.left[v];
    d.right = na.right[v];
  } else {
    d.left = -(int32_t)na.start[v] - 1;
    d.right = (int32_t)na.end[v];
  }
  out[v] = d;
}

// Leaves per subtree for the nodes [lo, hi) of one level; deeper levels are already done.
// Children's leaf counts next to each node, so that the search descent gets them with the node.
__global__ void child_counts_kernel(const DNode* __restrict__ nodes, const int32_t* __restrict__ nleaf, uint32_t m,
                                    uint2* __restrict__ cnl) {
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= m) return;
  DNode d = nodes[v];
  cnl[v] = d.left < 0 ? make_uint2(0, 0) : make_uint2((uint32_t)nleaf[d.left], (uint32_t)nleaf[d.right]);
}

__global__ void leaf_count_kernel(const int32_t* __restrict__ left, const int32_t* __restrict__ right, int32_t lo,
                                  int32_t hi, int32_t* __restrict__ nleaf) {
  int32_t v = lo + (int32_t)(blockIdx.x * blockDim.x + threadIdx.x);
  if (v >= hi) return;
  nleaf[v] = left[v] < 0 ? 1 : nleaf[left[v]] + nleaf[right[v]];
}

static unsigned grid_for(uint64_t total, int threads) {
  return (unsigned)std::min<uint64_t>((total + threads - 1) / threads, 152ull * 32);
}

int build_forest(efg_index* idx, uint32_t ntrees) {
  cudaStream_t s = idx->stream;
  Forest& F = idx->forest;
  F.release();
  const uint64_t n = idx->n;
  const uint64_t total = n * ntrees;
  const uint32_t S = idx->bp.S, tns = idx->bp.leaf_size;
  const uint64_t seed = idx->bp.seed;
  const uint64_t cap_nodes = 2 * total + ntrees;  // each split adds two nodes; at most n-1 splits per tree

  EFG_TRY(F.leaves.reserve(total));
  LocalBuf<uint32_t> ids_b(s);
  LocalBuf<int32_t> owner(s);
  LocalBuf<uint64_t> flags(s), pref(s), scan_tmp(s);
  EFG_TRY(ids_b.reserve(total));
  EFG_TRY(owner.reserve(total));
  EFG_TRY(flags.reserve(total));
  EFG_TRY(pref.reserve(total + 1));
  EFG_TRY(scan_tmp.reserve(scan_tmp_elems<uint64_t>(total) + 1));
  EFG_TRY(F.n_start.reserve(cap_nodes));
  EFG_TRY(F.n_end.reserve(cap_nodes));
  EFG_TRY(F.n_tree.reserve(cap_nodes));
  EFG_TRY(F.n_level.reserve(cap_nodes));
  EFG_TRY(F.n_left.reserve(cap_nodes));
  EFG_TRY(F.n_right.reserve(cap_nodes));
  LocalBuf<int32_t> n_dim(s), n_split(s);
  LocalBuf<float> n_val(s);
  EFG_TRY(n_dim.reserve(cap_nodes));
  EFG_TRY(n_split.reserve(cap_nodes));
  EFG_TRY(n_val.reserve(cap_nodes));
  NodeArrays na{F.n_start.p, F.n_end.p, F.n_tree.p, F.n_level.p, F.n_left.p, F.n_right.p, n_dim.p, n_split.p, n_val.p};

  // active lists and per-level scratch (active count <= total)
  uint64_t cap_act = std::max<uint64_t>(total, 2048);
  LocalBuf<int32_t> act(s), next_cand(s);
  LocalBuf<uint32_t> split_flag(s), child_off(s), mids(s), next_flag(s), next_pos(s), tmp32(s);
  EFG_TRY(act.reserve(cap_act));
  EFG_TRY(next_cand.reserve(2 * cap_act));
  EFG_TRY(split_flag.reserve(cap_act));
  EFG_TRY(child_off.reserve(cap_act + 1));
  EFG_TRY(mids.reserve(cap_act));
  EFG_TRY(next_flag.reserve(2 * cap_act));
  EFG_TRY(next_pos.reserve(2 * cap_act + 1));
  EFG_TRY(tmp32.reserve(scan_tmp_elems<uint32_t>(2 * cap_act) + 1));

  ScopedEvents<2> evs;
  cudaEvent_t e0 = evs.e[0], e1 = evs.e[1];
  cudaEventRecord(e0, s);
  perm_init_kernel<<<grid_for(total, 256), 256, 0, s>>>(F.leaves.p, owner.p, n, ntrees, seed);
  roots_init_kernel<<<(ntrees + 255) / 256, 256, 0, s>>>(na, ntrees, n);
  std::vector<int32_t> roots(ntrees);
  for (uint32_t t = 0; t < ntrees; ++t) roots[t] = (int32_t)t;
  EFG_CUDA(cudaMemcpyAsync(act.p, roots.data(), ntrees * 4, cudaMemcpyHostToDevice, s));
  EFG_CUDA(cudaGetLastError());

  uint32_t nactive = ntrees;
  int32_t nnodes = (int32_t)ntrees;
  std::vector<std::pair<int32_t, int32_t>> level_ranges{{0, (int32_t)ntrees}};
  bool phaseA = true;
  int32_t level = 0;
  uint32_t* cur = F.leaves.p;
  uint32_t* other = ids_b.p;
  EFG_TRY(make_bytes(idx));
  const bool bytes = idx->bytes_state == 1;
  const uint32_t blocks128 = (idx->dim + 127) / 128;
  const uint32_t wpn = blocks128 > 4 ? 8 : blocks128 > 2 ? 4 : blocks128;  // warps per node
  const size_t smem = (size_t)(8 / wpn) * idx->dim * sizeof(float);
  if (smem > 48 * 1024)
    EFG_CUDA(cudaFuncSetAttribute(split_stats_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  while (nactive > 0) {
    if (phaseA && nactive >= 1100) phaseA = false;
    int phaseB = phaseA ? 0 : 1;
    const unsigned sgrid = (nactive * wpn + 7) / 8;
    if (bytes)
      split_stats_kernel<<<sgrid, 256, smem, s>>>(idx->bytes.p, idx->ldb, idx->dim, n, cur, na, act.p, nactive, wpn,
                                                  level, phaseB, tns, seed, split_flag.p);
    else
      split_stats_kernel<<<sgrid, 256, smem, s>>>(idx->d_base, idx->ld, idx->dim, n, cur, na, act.p, nactive, wpn,
                                                  level, phaseB, tns, seed, split_flag.p);
    EFG_CUDA(cudaGetLastError());
    EFG_TRY(device_scan<uint32_t>(split_flag.p, nactive, child_off.p, tmp32.p, s));
    classify_kernel<<<grid_for(total, 256), 256, 0, s>>>(idx->d_base, idx->ld, n, ntrees, cur, owner.p, na, level,
                                                         flags.p);
    EFG_CUDA(cudaGetLastError());
    EFG_TRY(device_scan<uint64_t>(flags.p, total, pref.p, scan_tmp.p, s));
    uint32_t nsplit = 0;
    EFG_CUDA(cudaMemcpyAsync(&nsplit, child_off.p + nactive, 4, cudaMemcpyDeviceToHost, s));
    finish_nodes_kernel<<<(nactive + 255) / 256, 256, 0, s>>>(na, n, act.p, nactive, child_off.p, pref.p, nnodes,
                                                              level, phaseB, S, mids.p, next_flag.p, next_cand.p);
    EFG_CUDA(cudaGetLastError());
    scatter_kernel<<<grid_for(total, 256), 256, 0, s>>>(n, ntrees, cur, other, owner.p, na, level, pref.p);
    EFG_CUDA(cudaGetLastError());
    std::swap(cur, other);
    EFG_TRY(device_scan<uint32_t>(next_flag.p, 2ull * nactive, next_pos.p, tmp32.p, s));
    compact_kernel<<<(2 * nactive + 255) / 256, 256, 0, s>>>(next_flag.p, next_pos.p, next_cand.p, 2 * nactive,
                                                             act.p);
    EFG_CUDA(cudaGetLastError());
    uint32_t nnext = 0;
    EFG_CUDA(cudaMemcpyAsync(&nnext, next_pos.p + 2ull * nactive, 4, cudaMemcpyDeviceToHost, s));
    EFG_CUDA(cudaStreamSynchronize(s));
    level_ranges.push_back({nnodes, nnodes + 2 * (int32_t)nsplit});
    nnodes += 2 * (int32_t)nsplit;
    nactive = nnext;
    ++level;
    if ((uint64_t)nnodes + 2ull * nactive > cap_nodes || level > 4096)
      return fail(EFG_ERR_DEVICE_LIMIT, "tree build exceeded its node capacity");
  }
  if (cur != F.leaves.p)
    EFG_CUDA(cudaMemcpyAsync(F.leaves.p, cur, total * 4, cudaMemcpyDeviceToDevice, s));
  EFG_TRY(F.nodes.reserve(nnodes));
  to_dnodes_kernel<<<(nnodes + 255) / 256, 256, 0, s>>>(na, (uint32_t)nnodes, F.nodes.p);
  EFG_TRY(F.nleaf.reserve(nnodes));
  for (size_t l = level_ranges.size(); l-- > 0;) {
    int32_t lo = level_ranges[l].first, hi = level_ranges[l].second;
    if (hi > lo) leaf_count_kernel<<<(hi - lo + 255) / 256, 256, 0, s>>>(na.left, na.right, lo, hi, F.nleaf.p);
  }
  EFG_TRY(F.cnl.reserve(nnodes));
  child_counts_kernel<<<(nnodes + 255) / 256, 256, 0, s>>>(F.nodes.p, F.nleaf.p, (uint32_t)nnodes, F.cnl.p);
  EFG_CUDA(cudaGetLastError());
  // keep dim/val in the DNode array; the SoA start/end/tree/level/left/right stay for the merge
  EFG_TRY(F.d_roots.reserve(ntrees));
  EFG_CUDA(cudaMemcpyAsync(F.d_roots.p, roots.data(), ntrees * 4, cudaMemcpyHostToDevice, s));
  cudaEventRecord(e1, s);
  EFG_CUDA(cudaStreamSynchronize(s));
  float ms = 0;
  cudaEventElapsedTime(&ms, e0, e1);
  idx->bstats.trees_ms = ms;
  F.ntrees = ntrees;
  F.n = n;
  F.nnodes = (uint64_t)nnodes;
  F.roots = roots;
  F.has_soa = true;
  return EFG_OK;
}

int upload_forest(efg_index* idx, const std::vector<HNode>& nodes, const std::vector<int32_t>& roots,
                  const std::vector<uint32_t>& leaves, uint32_t ntrees) {
  Forest& F = idx->forest;
  F.release();
  std::vector<DNode> dn(nodes.size());
  std::vector<int32_t> lvl(nodes.size()), tr(nodes.size(), 0), l(nodes.size()), r(nodes.size());
  std::vector<uint32_t> st(nodes.size()), en(nodes.size());
  for (size_t i = 0; i < nodes.size(); ++i) {
    const HNode& h = nodes[i];
    dn[i].div_dim = h.div_dim;
    dn[i].div_val = h.div_val;
    if (h.left >= 0) {
      dn[i].left = h.left;
      dn[i].right = h.right;
    } else {
      dn[i].left = -(int32_t)h.start - 1;
      dn[i].right = (int32_t)h.end;
    }
    lvl[i] = h.level;
    l[i] = h.left;
    r[i] = h.right;
    st[i] = (uint32_t)h.start;
    en[i] = (uint32_t)h.end;
  }
  for (uint32_t t = 0; t < ntrees; ++t) {  // tree id of every node
    std::vector<int32_t> stack{roots[t]};
    while (!stack.empty()) {
      int32_t v = stack.back();
      stack.pop_back();
      tr[v] = (int32_t)t;
      if (l[v] >= 0) {
        stack.push_back(l[v]);
        stack.push_back(r[v]);
      }
    }
  }
  size_t m = nodes.size();
  std::vector<int32_t> nl(m, 0);
  for (uint32_t t = 0; t < ntrees; ++t) {  // post-order leaf counts
    std::vector<std::pair<int32_t, bool>> stack{{roots[t], false}};
    while (!stack.empty()) {
      auto [v, done] = stack.back();
      stack.pop_back();
      if (l[v] < 0) {
        nl[v] = 1;
      } else if (done) {
        nl[v] = nl[l[v]] + nl[r[v]];
      } else {
        stack.push_back({v, true});
        stack.push_back({l[v], false});
        stack.push_back({r[v], false});
      }
    }
  }
  EFG_TRY(F.nleaf.reserve(m));
  EFG_CUDA(cudaMemcpy(F.nleaf.p, nl.data(), m * 4, cudaMemcpyHostToDevice));
  EFG_TRY(F.nodes.reserve(m));
  EFG_TRY(F.d_roots.reserve(ntrees));
  EFG_TRY(F.leaves.reserve(leaves.size()));
  EFG_TRY(F.n_left.reserve(m));
  EFG_TRY(F.n_right.reserve(m));
  EFG_TRY(F.n_level.reserve(m));
  EFG_TRY(F.n_tree.reserve(m));
  EFG_TRY(F.n_start.reserve(m));
  EFG_TRY(F.n_end.reserve(m));
  EFG_CUDA(cudaMemcpy(F.nodes.p, dn.data(), m * sizeof(DNode), cudaMemcpyHostToDevice));
  EFG_TRY(F.cnl.reserve(m));
  child_counts_kernel<<<(unsigned)((m + 255) / 256), 256>>>(F.nodes.p, F.nleaf.p, (uint32_t)m, F.cnl.p);
  EFG_CUDA(cudaGetLastError());
  EFG_CUDA(cudaStreamSynchronize(0));  // searches run on a non-blocking stream
  EFG_CUDA(cudaMemcpy(F.d_roots.p, roots.data(), ntrees * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(F.leaves.p, leaves.data(), leaves.size() * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(F.n_left.p, l.data(), m * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(F.n_right.p, r.data(), m * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(F.n_level.p, lvl.data(), m * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(F.n_tree.p, tr.data(), m * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(F.n_start.p, st.data(), m * 4, cudaMemcpyHostToDevice));
  EFG_CUDA(cudaMemcpy(F.n_end.p, en.data(), m * 4, cudaMemcpyHostToDevice));
  F.ntrees = ntrees;
  F.n = idx->n;
  F.nnodes = m;
  F.roots = roots;
  F.has_soa = true;
  return EFG_OK;
}

int download_forest(efg_index* idx, std::vector<HNode>& nodes, std::vector<uint32_t>& leaves) {
  Forest& F = idx->forest;
  size_t m = F.nnodes;
  std::vector<DNode> dn(m);
  std::vector<int32_t> l(m), r(m), lvl(m);
  std::vector<uint32_t> st(m), en(m);
  EFG_CUDA(cudaMemcpy(dn.data(), F.nodes.p, m * sizeof(DNode), cudaMemcpyDeviceToHost));
  EFG_CUDA(cudaMemcpy(l.data(), F.n_left.p, m * 4, cudaMemcpyDeviceToHost));
  EFG_CUDA(cudaMemcpy(r.data(), F.n_right.p, m * 4, cudaMemcpyDeviceToHost));
  EFG_CUDA(cudaMemcpy(lvl.data(), F.n_level.p, m * 4, cudaMemcpyDeviceToHost));
  EFG_CUDA(cudaMemcpy(st.data(), F.n_start.p, m * 4, cudaMemcpyDeviceToHost));
  EFG_CUDA(cudaMemcpy(en.data(), F.n_end.p, m * 4, cudaMemcpyDeviceToHost));
  nodes.resize(m);
  for (size_t i = 0; i < m; ++i) {
    nodes[i].div_dim = dn[i].div_dim;
    nodes[i].div_val = dn[i].div_val;
    nodes[i].start = st[i];
    nodes[i].end = en[i];
    nodes[i].left = l[i];
    nodes[i].right = r[i];
    nodes[i].level = lvl[i];
  }
  leaves.resize((size_t)F.ntrees * F.n);
  EFG_CUDA(cudaMemcpy(leaves.data(), F.leaves.p, leaves.size() * 4, cudaMemcpyDeviceToHost));
  return EFG_OK;
}

}  // namespace efg
