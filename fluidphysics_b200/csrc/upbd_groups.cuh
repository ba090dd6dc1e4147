// Solver._recomputeGroups (src/solver.js:488-499) on the GPU, bit for bit.
//
// The reference runs a union-find over the alive constraints in index order:
// ra = find(a), rb = find(b), and when they differ parent[ra] = rb; then
// group[i] = find(i). Its labels are the roots that this exact sequence of
// unions leaves, which depend on the order (a component's root is not its
// smallest index), so a label-propagation pass would not reproduce them.
//
// The scene builder numbers the constraints in lexicographic (a, b) order with
// a < b, so most unions are known without replaying them:
//   - v's first alive constraint, when v is its b end, meets v while v is
//     still alone: a union that makes v the root ("first edge" fe[v], from
//     the smallest alive neighbour p[v] < v). A vertex with no alive smaller
//     neighbour is a seed; following p leads every vertex to its seed, the
//     tree it belongs to.
//   - any other alive constraint inside one tree joins two vertices that are
//     already together (fe of both ends came before it): no union.
//   - only constraints between different trees ("crossing") can unite
//     something else; they are replayed in order over the seeds alone.
// A part's root is the b of its last first edge, unless a join of two parts
// came after that; then it is the root the join's b part had just before the
// join, found the same way one join further down.
//
// An intact or sliced body has a handful of seeds and few crossing
// constraints, so the sequential part all but vanishes: the work is five
// parallel passes and one block's replay of the joins (about 0.3 us each).
// The passes are chains of a few dependent loads over L2-resident data, and
// at this size their six launches are most of the time. Replaying every
// constraint in one warp took 2,806 us on the default body after two cuts
// (93,556 constraints, B200); this takes 31 to 37 us.
#pragma once
#include "upbd_device.cuh"

namespace upbd {

constexpr uint32_t GRP_NONE = 0xffffffffu;
constexpr int GRP_BLOCK = 1024;  // threads of the replay's one block
constexpr int GRP_LANES = 8;     // lanes that look for a vertex's first alive constraint

// Scratch of one call, carved from the density pass's neighbour lists (free
// between substeps): 11 S words and C + C / 32 + 1 more, C <= 13 S, of the
// GLF * NL * N there are.
struct GroupScratch {
  int32_t* p;       // smallest alive neighbour, or the vertex itself (seed)
  uint32_t* fe;     // first edge (constraint index), GRP_NONE for a seed
  int32_t* tree;    // seed of the vertex's tree
  int32_t* par;     // union-find over the seeds
  int32_t* cur;     // join tree: node that stands for the part whose root seed this is
  uint32_t* last;   // join tree, 2 S nodes (seeds, then joins in order): 1 + last first edge, 0 = none
  int32_t* kpar;    // per node: parent or -1
  int32_t* kb;      // per join: node of its b part
  uint32_t* ke;     // per join: its constraint index
  uint32_t* bits;   // crossing constraints, one bit each
  uint32_t* list;   // the same as a list, ascending
};

__host__ inline GroupScratch group_scratch(uint32_t* w, int S, int C) {
  GroupScratch g;
  auto take = [&](size_t n) {
    uint32_t* q = w;
    w += n;
    return q;
  };
  const size_t s = (size_t)S;
  g.p = (int32_t*)take(s);
  g.fe = take(s);
  g.tree = (int32_t*)take(s);
  g.par = (int32_t*)take(s);
  g.cur = (int32_t*)take(s);
  g.last = take(2 * s);
  g.kpar = (int32_t*)take(2 * s);
  g.kb = (int32_t*)take(s);
  g.ke = take(s);
  g.bits = take((size_t)C / 32 + 1);
  g.list = take((size_t)C);
  return g;
}

// First alive constraint of each solid, GRP_LANES lanes a solid (its incident
// constraints come in ascending index, those with a smaller neighbour first).
__global__ void __launch_bounds__(256) k_groups_first(const uint4* __restrict__ cons, const uint32_t* __restrict__ adj,
                                                      int S, int C, GroupScratch g) {
  const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int v = t / GRP_LANES, lane = t % GRP_LANES;
  const unsigned sub = ((1u << GRP_LANES) - 1u) << ((threadIdx.x & 31) / GRP_LANES * GRP_LANES);
  if (v >= S) return;  // whole lane groups
  const uint32_t st = adj[v], en = adj[v + 1];
  const uint32_t* __restrict__ ids = adj + S + 1;
  int32_t p = v;
  uint32_t fe = GRP_NONE;
  for (uint32_t k0 = st; k0 < en; k0 += GRP_LANES) {
    const uint32_t k = k0 + (uint32_t)lane;
    uint32_t c = GRP_NONE;
    uint4 cc = make_uint4(0u, 0u, 0u, 0u);
    if (k < en) {
      c = ids[k];
      if (c < (uint32_t)C) cc = cons[c];
    }
    const bool alive = cc.w != 0u && cc.x < (uint32_t)S && cc.y < (uint32_t)S;
    const unsigned any = __ballot_sync(sub, alive) & sub;
    if (any) {
      const int src = __ffs(any) - 1;
      const uint32_t a = __shfl_sync(sub, cc.x, src), b = __shfl_sync(sub, cc.y, src);
      const uint32_t ci = __shfl_sync(sub, c, src);
      if (b == (uint32_t)v && a < b) {  // else v is the smaller end: a seed
        p = (int32_t)a;
        fe = ci;
      }
      break;
    }
  }
  if (lane == 0) {
    g.p[v] = p;
    g.fe[v] = fe;
    g.par[v] = v;
    g.cur[v] = v;
    g.last[v] = 0u;
    g.last[S + v] = 0u;
    g.kpar[v] = -1;
  }
}

// Seed of each solid's tree: p decreases strictly, so the walk ends (about one
// step per lattice layer).
__global__ void __launch_bounds__(256) k_groups_tree(int S, GroupScratch g) {
  const int v = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (v >= S) return;
  int32_t x = v, q = g.p[x];
  while (q < x) {
    x = q;
    q = g.p[x];
  }
  g.tree[v] = x;
}

// Alive constraints between different trees, the first of each pair of trees
// in a warp's 32 (a later one of the same pair finds them joined).
__global__ void __launch_bounds__(256) k_groups_cross(const uint4* __restrict__ cons, int C, int S, GroupScratch g) {
  const unsigned FULL = 0xffffffffu;
  const int c = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  unsigned long long pair = 0ull;  // no pair: a tree with itself
  if (c < C) {
    const uint4 k = cons[c];
    if (k.w != 0u && k.x < (uint32_t)S && k.y < (uint32_t)S) {
      const uint32_t ta = (uint32_t)g.tree[k.x], tb = (uint32_t)g.tree[k.y];
      if (ta != tb) pair = ((unsigned long long)max(ta, tb) << 32) | min(ta, tb);
    }
  }
  bool cross = pair != 0ull;
  if (__any_sync(FULL, cross)) {
    const unsigned same = __match_any_sync(FULL, pair);
    cross = cross && (int)(threadIdx.x & 31) == __ffs((int)same) - 1;
  }
  const unsigned w = __ballot_sync(FULL, cross);
  if ((threadIdx.x & 31) == 0 && c < C) g.bits[c >> 5] = w;
}

// Root seed of a part. HALVE shortens the path on the way (the replay's block,
// where concurrent writes only ever point nodes at their ancestors).
template <bool HALVE>
__device__ __forceinline__ int32_t grp_find(int32_t* par, int32_t x) {
  int32_t q = par[x];
  while (q != x) {
    if (HALVE) {
      const int32_t r = par[q];
      par[x] = r;
      x = r;
    } else {
      x = q;
    }
    q = par[x];
  }
  return x;
}

// The joins in constraint order, one block.
__global__ void __launch_bounds__(GRP_BLOCK) k_groups_join(const uint4* __restrict__ cons, int C, int S, GroupScratch g) {
  __shared__ uint32_t s_warp[GRP_BLOCK / 32];
  __shared__ uint32_t s_total;
  __shared__ int32_t s_from, s_to;
  const unsigned FULL = 0xffffffffu;
  const int tid = (int)threadIdx.x, lane = tid & 31, wid = tid >> 5;
  // the crossing constraints as an ascending list: each thread a run of words
  const int words = (C + 31) / 32, per = (words + GRP_BLOCK - 1) / GRP_BLOCK;
  const int w0 = tid * per, w1 = min(w0 + per, words);
  uint32_t n = 0;
  for (int w = w0; w < w1; w++) n += (uint32_t)__popc(g.bits[w]);
  uint32_t x = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[wid] = x;
  __syncthreads();
  uint32_t at = x - n;
  {
    const uint32_t mine = s_warp[lane];  // GRP_BLOCK / 32 = 32 warps
    at += __reduce_add_sync(FULL, lane < wid ? mine : 0u);
    if (tid == GRP_BLOCK - 1) s_total = at + n;
  }
  if (n)
    for (int w = w0; w < w1; w++)
      for (uint32_t m = g.bits[w]; m; m &= m - 1u) g.list[at++] = (uint32_t)(w * 32 + __ffs((int)m) - 1);
  __syncthreads();
  const uint32_t total = s_total;
  // replay: all constraints of a batch look up their parts at once; the first
  // one with two different parts is the next join
  uint32_t joins = 0;
  for (uint32_t base = 0; base < total; base += GRP_BLOCK) {
    const bool have = base + (uint32_t)tid < total;
    const uint32_t e = have ? g.list[base + tid] : 0u;
    int32_t ra = 0, rb = 0;
    if (have) {
      const uint4 k = cons[e];
      ra = grp_find<true>(g.par, g.tree[k.x]);
      rb = grp_find<true>(g.par, g.tree[k.y]);
    }
    for (;;) {
      const unsigned diff = __ballot_sync(FULL, have && ra != rb);
      if (lane == 0) s_warp[wid] = diff ? (uint32_t)(wid * 32 + __ffs(diff) - 1) : GRP_NONE;
      __syncthreads();
      const uint32_t first = __reduce_min_sync(FULL, s_warp[lane]);  // GRP_BLOCK / 32 = 32 warps
      if (first == GRP_NONE) break;  // the same on every thread
      if ((uint32_t)tid == first) {  // parent[ra] = rb, and the join's node
        const int32_t na = g.cur[ra], nb = g.cur[rb], node = S + (int32_t)joins;
        g.kpar[na] = node;
        g.kpar[nb] = node;
        g.kpar[node] = -1;
        g.kb[joins] = nb;
        g.ke[joins] = e;
        g.cur[rb] = node;
        g.par[ra] = rb;
        s_from = ra;
        s_to = rb;
      }
      joins++;
      __syncthreads();
      if (ra == s_from) ra = s_to;  // the other ends now rooted there
      if (rb == s_from) rb = s_to;
    }
    __syncthreads();
  }
}

// The part each first edge fell into: from the vertex's seed up the join tree
// to the node that was current at that time. last[node] becomes the last
// first edge of the node's life.
__global__ void __launch_bounds__(256) k_groups_last(int S, GroupScratch g) {
  const unsigned FULL = 0xffffffffu;
  const int v = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const uint32_t f = (v < S) ? g.fe[v] : GRP_NONE;
  const bool have = f != GRP_NONE;
  int32_t node = -1;
  if (have) {
    node = g.tree[v];
    for (int32_t up = g.kpar[node]; up >= 0 && g.ke[up - S] < f; up = g.kpar[node]) node = up;
  }
  // a warp's vertices mostly share one node: one atomic for the warp
  const int32_t top = __reduce_max_sync(FULL, node);
  if (__all_sync(FULL, !have || node == top)) {
    const uint32_t m = __reduce_max_sync(FULL, have ? f + 1u : 0u);
    if ((threadIdx.x & 31) == 0 && m) atomicMax(&g.last[top], m);
  } else if (have) {
    atomicMax(&g.last[node], f + 1u);
  }
}

// group[i]: the part's last first edge made its b end the root; a part whose
// last event was a join has the root its b part had before it.
__global__ void __launch_bounds__(256) k_groups_label(const uint4* __restrict__ cons, int S, GroupScratch g,
                                                      int32_t* __restrict__ group) {
  const int v = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (v >= S) return;
  int32_t node = g.cur[grp_find<false>(g.par, g.tree[v])];
  uint32_t m = g.last[node];
  while (m == 0u && node >= S) {
    node = g.kb[node - S];
    m = g.last[node];
  }
  group[v] = m ? (int32_t)cons[m - 1u].y : node;
}

}  // namespace upbd
