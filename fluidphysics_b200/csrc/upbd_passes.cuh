// Pass bodies of the unified-particle substep (sm_100a). Each body restates
// one or more WGSL passes of the reference (src/gpu/wgsl.js, cited per body)
// and keeps their floating-point operand order; passes that only touch a
// particle's own slot are fused into one body. All of them are FP32 SIMT
// gathers over HBM-resident state: there is no dense contraction on this
// path, so the tensor cores have no role here. The scalar type is `real`
// (upbd_device.cuh): float, or double in the test-only FP64 build that
// re-runs these same bodies as the drift reference.
//
// A body processes one block-sized tile `vb` of one scene (thread index
// vb * blockDim.x + threadIdx.x). The single-scene kernels (upbd_kernels.cuh)
// call it with vb = blockIdx.x; the batched kernels (upbd_batch.cu) call it
// for every tile of every scene from a persistent grid, so one scene's
// arithmetic is the same whichever way it is stepped.
#pragma once
#include "upbd_device.cuh"

namespace upbd {

#define UPBD_VTID (vb * blockDim.x + threadIdx.x)

// --------------------------------------------------- integrate + grid count
// integrate (src/gpu/wgsl.js:121-160) fused with gridCount
// (src/gpu/wgsl.js:173-178). The count keeps each particle's arrival ticket
// and bumps its scan tile's total, so the scan needs no second pass.
__device__ __forceinline__ void count_particle(const SimView& v, double inv_cell, int i, const real4& p) {
  uint32_t key;
  const uint32_t h = cell_of(p.x, p.y, p.z, inv_cell, (uint32_t)v.T - 1u, key);
  v.cell[i] = h;
  if (v.smove) cell_keys(v)[i] = key;
  v.ticket[i] = atomicAdd(&v.counts[h], 1u);
  const int rep = (i >> 5) & (tile_reps(v.num_tiles) - 1);  // a power of two
  atomicAdd(&v.tile_sum[rep * v.num_tiles + (int)(h / SCAN_TILE)], 1u);
}

template <bool INTEGRATE, bool COUNT>
__device__ __forceinline__ void b_integrate_count(const SimView& v, const DevParams* __restrict__ P, uint32_t vb) {
  const int i = UPBD_VTID;
  if (i >= v.N) return;
  uint32_t f = v.flags[i];
  real4 p4 = v.pos[i], vv, pv;
  issued(f);
  issued(p4);
  if (INTEGRATE) {
    vv = v.vel[i];
    pv = v.prev[i];
    issued(vv);
    issued(pv);
  }
  if (!(f & F_ACTIVE)) return;
  if (INTEGRATE) {
    const real h = P->h;
    const real vx = vv.x, vz = vv.z;
    const real vy = vv.y + P->gravity * h;
    const real px = p4.x, py = p4.y, pz = p4.z;
    real nx = px + vx * h, ny = py + vy * h, nz = pz + vz * h;
    real tw = pv.w;
    bool slipped = false;
    if (f & F_GRABBED) {
      const float4 gd = P->grab_delta;
      const real2 dn = v.density[i];
      real tx = pv.w, ty = vv.w, tz = dn.x;
      tx = tx + gd.x; ty = ty + gd.y; tz = tz + gd.z;
      const real ex = nx - tx, ey = ny - ty, ez = nz - tz;
      if (r_sqrt(dot3(ex, ey, ez, ex, ey, ez)) > 1.0f) {
        f &= ~F_GRABBED;
        v.flags[i] = f;
        v.vel[i] = make_real4(vx, vy, vz, 0.f);
        slipped = true;
      } else {
        const real k = P->grab_k * dn.y;
        real cx = (tx - nx) * k, cy = (ty - ny) * k, cz = (tz - nz) * k;
        const real cl = r_sqrt(dot3(cx, cy, cz, cx, cy, cz));
        const real maxC = 0.05f;
        if (cl > maxC) {
          const real g = maxC / cl;
          cx = cx * g; cy = cy * g; cz = cz * g;
        }
        nx = nx + cx; ny = ny + cy; nz = nz + cz;
        tw = tx;
        v.vel[i] = make_real4(vx, vy, vz, ty);
        v.density[i] = make_real2(tz, dn.y);
      }
    } else {
      v.vel[i] = make_real4(vx, vy, vz, vv.w);
    }
    (void)slipped;
    v.prev[i] = make_real4(px, py, pz, tw);
    p4 = make_real4(nx, ny, nz, p4.w);
    v.pos[i] = p4;
    if (i >= v.S) v.mark[i] = 0u;  // contact marks of this substep start clear
  }
  if (COUNT) count_particle(v, P->inv_cell, i, p4);
}

// ------------------------------------------------------------ exclusive scan
// scanBlocks/scanPartials/scanApply (src/gpu/wgsl.js:180-236) as one launch:
// block b scans its own SCAN_TILE counts (SCAN_PER consecutive ones per
// thread), adds the totals of tiles < b (the count's tile counters, all
// replicas) and writes the buckets' rows (all empty: the rank fix-up enters the
// occupied ones' fluid ends, and clears their counts and movement), or in the
// stateless grid build (SCENE false) start[]. The counts and the
// earlier totals are loaded up front so that their latencies overlap, and one
// block barrier publishes both per-warp sums. COUNTS: the counts themselves go
// to counts_out. Four counts a thread: with eight (256 threads a block) the
// launch took 10.7 us on 2^18 buckets, 7.7 now (B200, event-timed, about 4 of
// which are the launch).
constexpr int SCAN_PER = SCAN_TILE / SCAN_THREADS;
static_assert(SCAN_PER == 4, "a thread's counts are one 16-byte row");
template <bool COUNTS = false, bool SCENE = true>
__device__ __forceinline__ void b_scan(const SimView& v, uint32_t vb, uint32_t* __restrict__ counts_out = nullptr) {
  __shared__ uint32_t s_scan[SCAN_THREADS / 32];  // per-warp sums of this tile's counts
  __shared__ uint32_t s_prev[SCAN_THREADS / 32];  // per-warp sums of earlier tiles' totals
  const int tid = threadIdx.x;
  const int lane = tid & 31, wid = tid >> 5;
  const long long t0 = (long long)vb * SCAN_TILE + (long long)tid * SCAN_PER;
  // 16-byte rows when the tile is whole and the arrays allow it (start[] may
  // be a caller's buffer at any 4-byte offset)
  const bool vec = t0 + SCAN_PER <= (long long)v.T &&
                   ((reinterpret_cast<uintptr_t>(v.counts) | reinterpret_cast<uintptr_t>(v.start) |
                     reinterpret_cast<uintptr_t>(counts_out)) & 15u) == 0;
  uint4 c = make_uint4(0u, 0u, 0u, 0u);
  if (vec) {
    c = *reinterpret_cast<const uint4*>(v.counts + t0);
  } else {
    if (t0 < (long long)v.T) c.x = v.counts[t0];
    if (t0 + 1 < (long long)v.T) c.y = v.counts[t0 + 1];
    if (t0 + 2 < (long long)v.T) c.z = v.counts[t0 + 2];
    if (t0 + 3 < (long long)v.T) c.w = v.counts[t0 + 3];
  }
  // earlier tiles: word j holds replica j / num_tiles of tile j mod num_tiles
  // (a power of two, as the bucket count is)
  const int nt = v.num_tiles, words = tile_words(nt);
  uint32_t acc = 0;
#pragma unroll
  for (int k = 0; k < 2048 / SCAN_THREADS; k++) {
    const int j = tid + k * SCAN_THREADS;
    if (j < words && (uint32_t)(j & (nt - 1)) < vb) acc += v.tile_sum[j];
  }
  for (int j = tid + 2048; j < words; j += SCAN_THREADS)  // past 2^22 buckets only
    if ((uint32_t)(j & (nt - 1)) < vb) acc += v.tile_sum[j];
  const uint32_t sum = c.x + c.y + c.z + c.w;
  uint32_t x = sum;  // inclusive scan of the thread sums within the warp
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  acc = __reduce_add_sync(0xffffffffu, acc);
  if (lane == 31) s_scan[wid] = x;
  if (lane == 0) s_prev[wid] = acc;
  __syncthreads();
  uint32_t run = x - sum;
#pragma unroll
  for (int w = 0; w < SCAN_THREADS / 32; w++) {
    run += s_prev[w];
    if (w < wid) run += s_scan[w];
  }
  const uint4 r = make_uint4(run, run + c.x, run + c.x + c.y, run + c.x + c.y + c.z);
  if (vec) {
    if (SCENE) {
      uint4* row = reinterpret_cast<uint4*>(v.brow + t0);
      row[0] = make_uint4(r.x, r.x, r.y, r.y);
      row[1] = make_uint4(r.z, r.z, r.w, r.w);
    } else {
      *reinterpret_cast<uint4*>(v.start + t0) = r;
    }
    if (COUNTS) *reinterpret_cast<uint4*>(counts_out + t0) = c;
  } else {
    const uint32_t cs[4] = {c.x, c.y, c.z, c.w}, rs[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int k = 0; k < SCAN_PER; k++) {
      const long long idx = t0 + k;
      if (idx < v.T) {
        if (SCENE) v.brow[idx] = make_uint2(rs[k], rs[k]);
        else v.start[idx] = rs[k];
        if (COUNTS) counts_out[idx] = cs[k];
      }
    }
  }
  if (vb == (uint32_t)v.num_tiles - 1u && tid == SCAN_THREADS - 1) {
    if (SCENE) v.brow[v.T] = make_uint2(run + sum, run + sum);
    else v.start[v.T] = run + sum;
  }
  if (vb == 0 && tid == 0 && v.bmove) {
    v.scratch[SCR_XMOVE] = 0u;
    v.scratch[SCR_FAR] = 0u;
  }
}

// Scatter by ticket (gridScatter, src/gpu/wgsl.js:238-245, without its
// second atomic), and clear the tile totals for the next count.
// In a scene the particle's cell key goes along, for the rank fix-up. The
// stateless grid build (SCENE false) goes by the buckets its count wrote, and clears every count here, four a thread, so that its
// scratch, which outlives the call, is clear for the next one even where calls
// overlapped (262,139 particles, 2^19 buckets, B200: with the scan storing the
// zeros behind its reads the build took 35.8 us instead of 34.8).
template <bool SCENE = true>
__device__ __forceinline__ void b_scatter(const SimView& v, uint32_t vb) {
  const int i = UPBD_VTID;
  if (i < tile_words(v.num_tiles)) v.tile_sum[i] = 0u;
  if (!SCENE && i < (v.T + 3) / 4) {
    if (4 * i + 3 < v.T) *reinterpret_cast<uint4*>(v.counts + 4 * i) = make_uint4(0u, 0u, 0u, 0u);
    else for (int k = 4 * i; k < v.T; k++) v.counts[k] = 0u;
  }
  if (i >= v.N) return;
  const uint32_t f = SCENE ? v.flags[i] : F_ACTIVE, h = v.cell[i], ticket = v.ticket[i],
                 key = SCENE ? cell_keys(v)[i] : 0u;
  issued(f);
  issued(h);
  issued(ticket);
  issued(key);
  if (SCENE ? !(f & F_ACTIVE) : h == CELL_NONE) return;
  const uint32_t at = (SCENE ? v.brow[h].x : v.start[h]) + ticket;
  if (!UPBD_IDX_OK(v, at, v.N)) return;
  if (SCENE) bucket_pairs(v)[at] = make_uint2((uint32_t)i, key);
  else v.tmp[at] = (uint32_t)i;  // the stateless grid build
}

// Deterministic membership: particle i goes to start[h] + #{j in bucket : j > i},
// i.e. descending index inside a bucket, the order Solver._buildGrid's
// `--cellStart[h]` scatter leaves (src/solver.js:182-183).
//
//
// In a scene it also lays out the density pass's chunks: up to CHUNK fluid
// particles of one bucket and one cell (bucket mates of another cell, found in
// one bucket of seven in a settled pool, would need candidates of their own).
// Inside a bucket the fluid's slots are listed by (cell key, slot) at the
// bucket's places of chunk_places, the first of each chunk with the chunk's
// size (chunk_word). The slot copy of a fluid particle carries
// its slot where the mass would be, for the density pass's lists; the mass goes
// to slot_mass.
template <bool SCENE = true>
__device__ __forceinline__ void b_rankfix(const SimView& v, uint32_t vb) {
  const int i = UPBD_VTID;
  if (i >= v.N) return;
  const uint32_t f = SCENE ? v.flags[i] : F_ACTIVE, h = v.cell[i];
  real4 p = make_real4(0.f, 0.f, 0.f, 0.f);
  if (SCENE) p = v.pos[i];
  issued(f);
  issued(h);
  issued(p);
  if (SCENE ? !(f & F_ACTIVE) : h == CELL_NONE) return;
  const uint32_t s = SCENE ? v.brow[h].x : v.start[h], e = SCENE ? v.brow[h + 1].x : v.start[h + 1];
  if (!UPBD_IDX_OK(v, e, (uint32_t)v.N + 1u)) return;
  uint32_t rank = 0;
  if (!SCENE) {  // the stateless grid build has no bucket-ordered copies
    for (uint32_t k = s; k < e; k++) rank += (v.tmp[k] > (uint32_t)i) ? 1u : 0u;
    if (UPBD_IDX_OK(v, s + rank, v.N)) v.entries[s + rank] = (uint32_t)i;
    return;
  }
  const uint32_t key = cell_keys(v)[i];
  const uint2* __restrict__ pairs = bucket_pairs(v);
  uint32_t solids = 0, before = 0, mates = 0, rank_in = 0;
  for (uint32_t k = s; k < e; k++) {
    const uint2 j = pairs[k];
    const bool ahead = j.x > (uint32_t)i, solid = j.x < (uint32_t)v.S, mate = !solid && j.y == key;
    rank += ahead ? 1u : 0u;
    solids += solid ? 1u : 0u;
    before += (!solid && j.y < key) ? 1u : 0u;
    mates += mate ? 1u : 0u;
    rank_in += (mate && ahead) ? 1u : 0u;
  }
  const uint32_t slot = s + rank;
  if (!UPBD_IDX_OK(v, slot, v.N)) return;
  v.entries[slot] = (uint32_t)i;
  v.slot[i] = slot;
  if (rank == 0u) {
    v.brow[h].y = e - solids;
    v.counts[h] = 0u;  // ready for the next count
    v.bmove[h] = 0u;   // no movement recorded yet this substep
  }
  if (i >= v.S) {
    const uint32_t n = (rank_in % CHUNK == 0u) ? min(CHUNK, mates - rank_in) : 0u;
    const uint32_t place = s + before + rank_in;
    chunk_places(v)[place] = chunk_word(place, slot, n);
    slot_mass(v)[slot] = p.w;
    if (!(r_fabs(p.x) <= FAR && r_fabs(p.y) <= FAR && r_fabs(p.z) <= FAR)) v.scratch[SCR_FAR] = 1u;
    p.w = slot_pack(real(0), slot);
  } else {
    chunk_places(v)[slot] = 0u;  // solids follow the fluid: no chunk starts there
  }
  v.spos[slot] = p;
}

// ------------------------------------------------------------------ fluid
// The fluid-fluid gathers run GLF lanes per particle (see lane_strided); lane 0
// writes. They take the particles by grid slot: the particles of one bucket sit
// in consecutive slots and share their 27 neighbour buckets. A particle's own
// arithmetic does not depend on which group runs it. Groups whose slot holds a
// solid, or lies past the active count, have no work.

// fluidDensity, src/gpu/wgsl.js:254-279. Every grid entry is active (the
// grid is built from the active particles of this substep, before bounds).
//
// A warp takes one chunk (rank fix-up): up to CHUNK fluid particles of one
// cell, GLF lanes each. They share their 27 buckets, so the warp looks them up
// once, a lane a bucket, and copies their fluid to shared memory (four lanes a
// bucket, asynchronous 16-byte copies that bring the slot along); each
// particle's lanes then test their shares there: no cursor, no branch, one
// 16-byte shared load and eight operations a candidate, a bit kept for each
// candidate within the list radius. The bits (one candidate in five) are then
// walked with the square root, the sums and the list entry. The order is
// lane_strided's (candidate c to lane c mod GLF, each lane in sequence), so are
// the sums. A round stages at most STAGE candidates; longer sequences take more
// rounds, and particles whose cell is another one after all (equal keys)
// another turn. A block's warps share out the chunks that start in its window of
// places: 128 for large scenes (two to three chunks a warp in a settled pool,
// so that uneven chunks even out), fewer where that would leave SMs idle.
// Bound by the latency of the shared loads, square roots and shuffles between
// its instructions (58 % of the issue slots of an active SM). On the default
// scene's settled pool (65,536 fluid, 120 candidates and 22 listed each; B200,
// an event pair around an eager launch, as all of the following) a launch takes
// 33.2 us; a walk of each group of GLF lanes with its own cursor, 46 instructions
// a candidate, took 51.4; in the large scene's splash 99.7 against 117.9. With
// half a warp a chunk of 4 everywhere it took a third longer (the set-up is shared
// by half as many), with a warp over 8 consecutive slots of several cells more
// than twice as long.
// Where fluid falls apart in drops of one or two particles a cell, a warp a chunk
// leaves three lanes in four idle and the set-up, some 300 instructions, is
// paid for two particles. There a warp takes two chunks of up to four, a half
// each (W = 16): the large scene's first frames of the fall 147 us a warp a
// chunk, 106 with halves, the default scene's 48.3 and 37.0. A cursor a group
// took 89 and 34 there, in a kernel of 32 registers; within this one, at 48, it
// takes 121 and 45, quarters of a warp 124 (a sequence is 64 long: two rounds),
// lists of slots in shared memory 107 and 38. A launch of its own for such
// windows would cost every other frame 2 to 3 us a substep.
constexpr uint32_t STAGE = 4096 / sizeof(real4);     // 256 candidates a warp and round (FP64: 128)
constexpr size_t STAGE_WARP = STAGE * sizeof(real4);  // dynamic shared bytes per warp
constexpr uint32_t WINDOW_MAX = 128;                  // places of a block's window
// Halves where fewer than one chunk in SPARSE of a window has more than four
// particles. Measured before the look-ups were one row each: at one in two the
// default scene's settled pool took 38.5 us instead of 36.6 and the large scene's
// splash 2069 us a frame instead of 1966; at one in eight and in 32 the fall's
// frames 6 to 15 took 1379 and 1399 us instead of 1324.
constexpr uint32_t SPARSE = 4;

__device__ __forceinline__ void copy_row_async(real4* dst, const real4* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
#pragma unroll
  for (int k = 0; k < (int)sizeof(real4); k += 16)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d + k), "l"((const char*)src + k) : "memory");
}
__device__ __forceinline__ void copy_rows_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Squared distance inside the gathers: the product build's rounding is spelled
// out (the compiler may fuse the x or the y product into the first sum, and
// chooses anew with every change around it), the parity build's operations are
// the reference's. The fluid gathers fuse x, the distance solve y.
__device__ __forceinline__ real dist2(real ex, real ey, real ez) {
#ifdef UPBD_PARITY_BUILD
  return dot3(ex, ey, ez, ex, ey, ez);
#else
  return r_fma(ez, ez, r_fma(ex, ex, ey * ey));
#endif
}
__device__ __forceinline__ real dist2_xy(real ex, real ey, real ez) {
#ifdef UPBD_PARITY_BUILD
  return dot3(ex, ey, ez, ex, ey, ez);
#else
  return r_fma(ez, ez, r_fma(ey, ey, ex * ex));
#endif
}

// bits << 1, plus 1 where d2 is below lim (the parity build: not at or above)
__device__ __forceinline__ uint32_t push_listed(uint32_t bits, real d2, real lim) {
#if defined(UPBD_PARITY_BUILD)
  return (bits << 1) | (d2 >= lim ? 0u : 1u);
#elif defined(UPBD_FP64_BUILD)
  return (bits << 1) | (d2 < lim ? 1u : 0u);
#else
  return __funnelshift_l(__float_as_uint(d2 - lim), bits, 1);  // the sign of the difference (a NaN's is clear)
#endif
}

// threadIdx.x in a register: read once, not again wherever a lane is needed
__device__ __forceinline__ int thread_index() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

// A warp's W-lane parts (W = 32 or 16) each take a chunk of up to W / GLF
// particles; a lane looks up buckets l and, with W = 16, l + 16 of its part's 27.
template <int W>
struct Buckets {
  static constexpr int R = (27 + W - 1) / W;
  uint32_t s0[R], off[R], end[R];  // first slot; the bucket's range of the sequence
};

// One round's copies: copy(row, slot) for candidates q0 .. of the part's
// sequence, ROWS of them a round (CLIP: where there is more than one).
template <int W, uint32_t ROWS, bool CLIP, class Copy>
__device__ __forceinline__ void stage_rows(int L, const Buckets<W>& b, uint32_t q0, Copy&& copy) {
  const unsigned FULL = 0xffffffffu;
  constexpr int LB = W / 8;  // lanes a bucket
  const int l = L & (W - 1);
#pragma unroll
  for (int r = 0; r < 4; r++) {  // buckets 8 r + l / LB, rows l mod LB and every LB-th after it
    const int owner = (8 * r + l / LB) & (W - 1), q = 8 * r / W;
    uint32_t o = __shfl_sync(FULL, b.off[q], owner, W), hi = __shfl_sync(FULL, b.end[q], owner, W);
    const uint32_t sb = __shfl_sync(FULL, b.s0[q], owner, W) - o;
    if (CLIP) {
      o = max(o, q0);
      hi = min(hi, q0 + ROWS);
    }
    uint32_t k = o + (uint32_t)(l & (LB - 1));
    do {
#pragma unroll
      for (int m = 0; m < 2; m++, k += LB)
        if (k < hi) copy(CLIP ? k - q0 : k, sb + k);
    } while (__any_sync(FULL, k < hi));
  }
}

// The chunks that start among the window places from `first` on, listed in
// chunk as (place - first | size << 8); returns how many entries the warps
// share out. Where most chunks hold one or two particles (a fluid that falls
// apart in drops) and there are more of them than warps, an entry is a pair of
// chunks of up to four particles, one to each half of a warp; `halves` is then
// their number, else 0. Every thread of the block calls it.
struct ChunkList {
  uint32_t chunk[WINDOW_MAX + CHUNK], fill[WINDOW_MAX / 32], next;
};
__device__ __forceinline__ uint32_t list_chunks(const SimView& v, ChunkList& s, uint32_t first, uint32_t window,
                                                uint32_t nact, int tid, uint32_t& halves) {
  const int L = tid & 31, wid = tid >> 5;
  const uint32_t place = first + (uint32_t)tid;
  uint32_t word = 0, before = 0, more = 0;
  if ((uint32_t)wid * 32u < window) {
    if ((uint32_t)tid < window && place < nact) word = chunk_word_size(chunk_places(v)[place]);
    const unsigned b = __ballot_sync(0xffffffffu, word != 0u), b4 = __ballot_sync(0xffffffffu, word > CHUNK / 2);
    // chunks, those over four particles, particles
    if (L == 0) s.fill[wid] = (uint32_t)__popc(b) | (uint32_t)__popc(b4) << 8;
    before = (uint32_t)__popc(b & ((1u << L) - 1u));
    more = (uint32_t)__popc(b4 & ((1u << L) - 1u));
  }
  if (tid == 0) s.next = blockDim.x >> 5;
  __syncthreads();
  uint32_t all = 0, mine = 0;
#pragma unroll
  for (int w = 0; w < (int)(WINDOW_MAX / 32); w++)
    if ((uint32_t)w * 32u < window) {
      if (w == wid) mine = all;
      all += s.fill[w];
    }
  const uint32_t chunks = all & 0xffu, big = all >> 8;
  const bool sp = SPARSE * big < chunks && chunks > blockDim.x >> 5;
  halves = sp ? chunks + big : 0u;
  if (word) {
    const uint32_t at = (mine & 0xffu) + before;
    if (!sp) {
      s.chunk[at] = (uint32_t)tid | (word << 8);
    } else {
      const uint32_t a = at + (mine >> 8) + more, h = min(word, CHUNK / 2);
      s.chunk[a] = (uint32_t)tid | (h << 8);
      if (word > h) s.chunk[a + 1] = ((uint32_t)tid + h) | ((word - h) << 8);
    }
  }
  __syncthreads();
  return sp ? (halves + 1) / 2 : chunks;
}
// Entry c's chunk for this lane's part of the warp: the slot of group g's
// particle (0 where it has none) and whether it has one.
template <int W>
__device__ __forceinline__ uint32_t chunk_slot(const SimView& v, const ChunkList& s, uint32_t c, int L, uint32_t first,
                                               uint32_t halves, bool& act) {
  const uint32_t k = (W == 32) ? c : 2 * c + (uint32_t)L / W, g = (uint32_t)(L & (W - 1)) / GLF;
  const uint32_t d = (W == 32 || k < halves) ? s.chunk[k] : 0u;
  act = g < (d >> 8);
  const uint32_t place = first + (d & 0xffu) + g;
  return act ? chunk_word_slot(place, chunk_places(v)[place]) : 0u;
}
// the warp's next chunk after c
__device__ __forceinline__ uint32_t next_chunk(ChunkList& s, uint32_t c, int L) {
  if (L == 0) c = atomicAdd(&s.next, 1u);
  return __shfl_sync(0xffffffffu, c, 0);
}

// Of the part's lanes: those (all four of a group) whose particle lies in the
// cell of the group that starts at lane ll; ca: the lane's cell coordinate (x, y, z, z).
template <int W>
__device__ __forceinline__ unsigned same_cell(double ca, int ll, int lane) {
  const unsigned FULL = 0xffffffffu;
  const bool other = !(ca == __shfl_sync(FULL, ca, ll + lane));
  unsigned turn = ~__ballot_sync(FULL, other);
  turn &= (turn >> 1) & (turn >> 2) & 0x11111111u;  // groups with all three coordinates equal
  return (turn * 15u) | (15u << ll);
}

// inclusive scan over the W lanes of a part
template <int W>
__device__ __forceinline__ uint32_t part_scan(uint32_t x, int L) {
#pragma unroll
  for (int o = 1; o < W; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o, W);
    if ((L & (W - 1)) >= o) x += y;
  }
  return x;
}

// The fluid of the 27 cells around that group's (CellHash::init's buckets);
// each(length, bucket) sees them; none where the part has no work. Returns the
// sequence's length.
template <int W, class Each>
__device__ __forceinline__ uint32_t part_buckets(const SimView& v, double ca, int ll, int L, bool work, Buckets<W>& b,
                                                 Each&& each) {
  const unsigned FULL = 0xffffffffu;
  const int l = L & (W - 1);
  const int axis = (l < 9) ? l / 3 : 2;  // lane j < 9: component j, axis j / 3, cell offset j % 3 - 1
  const double cl = __shfl_sync(FULL, ca, ll + axis);
  const double K = (axis == 0) ? 92837111.0 : ((axis == 1) ? 689287499.0 : 283923481.0);
  const int32_t comp = js_toint32(__dmul_rn(__dadd_rn(cl, (double)(l - 3 * axis - 1)), K));
  const uint32_t mask = (uint32_t)v.T - 1u;
  uint32_t n[Buckets<W>::R];
#pragma unroll
  for (int r = 0; r < Buckets<W>::R; r++) {
    const int k = l + W * r;
    const int ka = k / 9, kb = (k - 9 * ka) / 3, kc = k - 9 * ka - 3 * kb;
    const uint32_t hb = (uint32_t)(__shfl_sync(FULL, comp, ka, W) ^ __shfl_sync(FULL, comp, 3 + kb, W) ^
                                   __shfl_sync(FULL, comp, 6 + kc, W)) & mask;
    b.s0[r] = 0;
    n[r] = 0;
    if (k < 27 && (W == 32 || work)) {
      const uint2 q = bucket_range<0>(v, hb);
      b.s0[r] = q.x;
      n[r] = q.y;
      each(q.y, hb);
    }
  }
  uint32_t total = 0;
#pragma unroll
  for (int r = 0; r < Buckets<W>::R; r++) {
    b.end[r] = total + part_scan<W>(n[r], L);  // in cell order
    b.off[r] = b.end[r] - n[r];
    total = __shfl_sync(FULL, b.end[r], W - 1, W);
  }
  return total;
}
template <int W>
__device__ __forceinline__ uint32_t longest(uint32_t total) {
  return W == 32 ? total : max(total, __shfl_xor_sync(0xffffffffu, total, 16));
}
template <int W>
__device__ __forceinline__ bool parts_left(unsigned rem) {
  return W == 32 ? rem != 0u : __any_sync(0xffffffffu, rem != 0u);
}
// the lane's part
template <int W>
__device__ __forceinline__ unsigned part_lanes(int L) {
  return W == 32 ? 0xffffffffu : ((1u << (W & 31)) - 1u) << (L & ~(W - 1));
}

template <int W>
__device__ __forceinline__ void density_chunks(const SimView& v, const DevParams* __restrict__ P, ChunkList& s_list,
                                               real4* sx, uint32_t first, uint32_t chunks, uint32_t halves, int tid) {
  const unsigned FULL = 0xffffffffu;
  const int L = tid & 31, wid = tid >> 5, lane = L & (GLF - 1);
  constexpr uint32_t ROWS = STAGE * W / 32;
  sx += (L / W) * ROWS;
  const double inv = P->inv_cell;
  const real H = P->fluid_h, H2 = H * H;
  const real HS = H * (1.0f + XSKIN), HS2 = HS * HS;  // list radius (for xsph)
  const uint32_t NS = (uint32_t)v.N;
#ifndef UPBD_PARITY_BUILD
  const real invH = 1.0f / H;
  const bool far = v.scratch[SCR_FAR] != 0u || !(r_fabs(invH) <= 3.0e38f);
#endif
  for (uint32_t c = (uint32_t)wid; c < chunks; c = next_chunk(s_list, c, L)) {
    bool act;
    const uint32_t myslot = chunk_slot<W>(v, s_list, c, L, first, halves, act);
    const real4 pi = act ? v.spos[myslot] : make_real4(0.f, 0.f, 0.f, 0.f);
    const real mass = slot_mass(v)[myslot];
    // lane l's c-th listed candidate goes to row l*NL + c, column myslot
    uint32_t* nbr = list_entry(v.nbr + myslot, lane * NL, NS);
    uint32_t cnt = 0;
    real rho = 0.f, rhoNear = 0.f;
    const double ca = floor(__dmul_rn((double)(lane == 0 ? pi.x : (lane == 1 ? pi.y : pi.z)), inv));
    unsigned rem = __ballot_sync(FULL, act) & part_lanes<W>(L);  // the part's particles whose cell has not had its turn
    do {
      // the first remaining particle and those of its cell
      const bool work = W == 32 || rem != 0u;
      const int ll = work ? __ffs((int)rem) - 1 : L & ~(W - 1);
      const unsigned turn = same_cell<W>(ca, ll, lane) & rem;
      rem &= ~turn;
      Buckets<W> b;
      const uint32_t total = part_buckets<W>(v, ca, ll, L, work, b, [](uint32_t, uint32_t) {});
      const uint32_t most = longest<W>(total);
      for (uint32_t q0 = 0; q0 < most; q0 += ROWS) {
        auto copy = [&](uint32_t k, uint32_t e) {
          if (UPBD_IDX_OK(v, e, NS)) copy_row_async(&sx[k], &v.spos[e]);
          else sx[k] = make_real4(__int_as_float(0x7f800000), 0.f, 0.f, 0.f);  // never listed (reported)
        };
        if (most <= ROWS) stage_rows<W, ROWS, false>(L, b, 0u, copy);
        else stage_rows<W, ROWS, true>(L, b, q0, copy);
        copy_rows_wait();
        __syncwarp();
        const uint32_t len = (W == 32 || q0 < total) ? min(total - q0, ROWS) : 0u;
        const uint32_t mine = (turn >> L & 1u) ? (len + (GLF - 1) - lane) / GLF : 0u;  // this lane's share
        const real4* __restrict__ row = sx + lane;
        for (uint32_t u0 = 0; u0 * GLF < len; u0 += 32, row += 32 * GLF) {
          // up to 32 candidates a lane, the first one's bit on top
          const uint32_t steps = min((len + (GLF - 1)) / GLF - u0, 32u);
          uint32_t bits = 0;
          const real4* __restrict__ r4 = row;
          for (uint32_t u = 0; u < steps; u += 4, r4 += 4 * GLF) {  // reads past the share stay in the warp's rows
#pragma unroll
            for (int k = 0; k < 4; k++) {
              const real4 pj = r4[k * GLF];
              const real d2 = dist2(pj.x - pi.x, pj.y - pi.y, pj.z - pi.z);
              bits = push_listed(bits, d2, HS2);
            }
          }
          bits <<= (32u - ((steps + 3u) & ~3u)) & 31u;
          const uint32_t own = (mine > u0) ? mine - u0 : 0u;  // drop the rows past the share
          if (own < 32u) bits &= ~(0xffffffffu >> own);
          // two listed candidates at a time: their loads and square roots overlap
          while (bits) {
            const int k0 = __clz((int)bits);
            bits &= ~(0x80000000u >> k0);
            const int k1 = bits ? __clz((int)bits) : k0;
            const bool two = bits != 0u;
            bits &= ~(0x80000000u >> k1);
            const real4 p0 = row[k0 * GLF], p1 = row[k1 * GLF];
            const real d0 = dist2(p0.x - pi.x, p0.y - pi.y, p0.z - pi.z);
            const real d1 = dist2(p1.x - pi.x, p1.y - pi.y, p1.z - pi.z);
            const uint32_t e0 = slot_unpack(p0.w), e1 = slot_unpack(p1.w);
            const bool use0 = e0 != myslot, use1 = two && e1 != myslot;
            const bool in0 = d0 < H2, in1 = d1 < H2;
            if (use0) {
              if (cnt < NL) *list_entry(nbr, cnt, NS) = e0 | (in0 ? NBR_IN : 0u);  // for fluidDisp (same positions) and xsph
              cnt++;
            }
            if (use1) {
              if (cnt < NL) *list_entry(nbr, cnt, NS) = e1 | (in1 ? NBR_IN : 0u);
              cnt++;
            }
#ifdef UPBD_PARITY_BUILD
            if (use0 && !(d0 >= H2)) {
              const real q = 1.0f - r_sqrt(d0) / H;
              rho = rho + q * q;
              rhoNear = rhoNear + q * q * q;
            }
            if (use1 && !(d1 >= H2)) {
              const real q = 1.0f - r_sqrt(d1) / H;
              rho = rho + q * q;
              rhoNear = rhoNear + q * q * q;
            }
#else
            const real q0_ = r_fma(-approx_sqrt(d0), invH, real(1.0f)), q1_ = r_fma(-approx_sqrt(d1), invH, real(1.0f));
            const real qq0 = (use0 && in0) ? r_mul(q0_, q0_) : real(0.0f), qq1 = (use1 && in1) ? r_mul(q1_, q1_) : real(0.0f);
            rho = rho + qq0;
            rhoNear = r_fma(qq0, q0_, rhoNear);
            rho = rho + qq1;
            rhoNear = r_fma(qq1, q1_, rhoNear);
#endif
          }
        }
#ifndef UPBD_PARITY_BUILD
        // a candidate at no finite distance is not listed, but leaves the near
        // density NaN: it adds 0 times its q, as every candidate out of range
        // does in exact terms
        if (far)
          for (uint32_t u = 0; u < mine; u++) {
            const real4 pj = sx[lane + u * GLF];
            const real d2 = dist2(pj.x - pi.x, pj.y - pi.y, pj.z - pi.z);
            rhoNear = r_fma(real(0.0f), r_fma(-approx_sqrt(d2), invH, real(1.0f)), rhoNear);
          }
#endif
        __syncwarp();  // the next round rewrites the rows
      }
    } while (parts_left<W>(rem));
    if (act) v.ncount[lane * NS + myslot] = cnt;
    rho = lane_sum<GLF>(rho);
    rhoNear = lane_sum<GLF>(rhoNear);
    if (act && lane == 0) {
      v.density[v.entries[myslot]] = make_real2(rho, rhoNear);
      store_row_pair(&v.drow[2 * (size_t)myslot], pi, make_real4(rho, rhoNear, mass, 0.f));
    }
  }
}

// window <= min(WINDOW_MAX, blockDim), at most 256 threads a block.
__device__ __forceinline__ void b_density(const SimView& v, const DevParams* __restrict__ P, uint32_t window,
                                          uint32_t vb) {
  extern __shared__ __align__(16) unsigned char s_stage[];
  __shared__ ChunkList s_list;
  const int tid = thread_index();
  const uint32_t nact = active_slots(v), first = vb * window;
  if (first >= nact) return;
  uint32_t halves;
  const uint32_t chunks = list_chunks(v, s_list, first, window, nact, tid, halves);
  real4* sx = reinterpret_cast<real4*>(s_stage + (tid >> 5) * STAGE_WARP);
  if (halves) density_chunks<16>(v, P, s_list, sx, first, chunks, halves, tid);
  else density_chunks<32>(v, P, s_list, sx, first, chunks, halves, tid);
}

// Contact marks (mark_fluid_near below) find a fluid particle from the
// solid's side, through the bucket the grid build put it in; the particle's
// own contact walk runs around the cell it is in after its displacement. A
// displacement that carries it into another cell can bring it within contact
// range of a solid two cells from its grid cell, which no mark walk reaches,
// so the pass that applies the fluid's move (from o, the position the grid
// was built from, to p) marks such a particle itself and it walks. Every
// particle that kept its cell and is in range of a solid is in a bucket of
// the 27 around that solid's cell, where the mark walk finds it.
__device__ __forceinline__ void mark_if_cell_changed(const SimView& v, const DevParams* __restrict__ P, int i,
                                                     const real4& o, const real4& p) {
  if (!P->use_mark) return;
  const double inv = P->inv_cell;
  const bool same = floor(__dmul_rn((double)o.x, inv)) == floor(__dmul_rn((double)p.x, inv)) &&
                    floor(__dmul_rn((double)o.y, inv)) == floor(__dmul_rn((double)p.y, inv)) &&
                    floor(__dmul_rn((double)o.z, inv)) == floor(__dmul_rn((double)p.z, inv));
  if (!same) v.mark[i] = 1u;  // also for a coordinate that is not finite
}

// fluidDisp, src/gpu/wgsl.js:281-316, DL threads per slot over the density
// pass's lists (same positions). Thread h of a slot takes lanes h*GLF/DL ..
// (h+1)*GLF/DL - 1: lane l's in-range neighbours (its NBR_IN entries) in its
// walk order, then the next lane's, summed one after another; the DL partials combine by the xor
// butterfly. A thread whose lists overflowed walks the 27 buckets for its
// lanes' shares instead, in the same order. With APPLY it also applies the
// displacement (applyDeltaFluid, src/gpu/wgsl.js:318-323): pos[i] and the own
// sfp slot are written, while every thread reads neighbours from spos, so no
// read sees a moved particle.
template <bool APPLY>
__device__ __forceinline__ void b_disp(const SimView& v, const DevParams* __restrict__ P, uint32_t vb) {
  constexpr int LPT = GLF / DL;  // lanes' lists per thread
  const uint32_t e0 = UPBD_VTID / DL;
  const int h = (int)(threadIdx.x & (DL - 1));
  const real4* __restrict__ rows = v.drow;
  const uint32_t NS = (uint32_t)v.N, eld = min(e0, NS - 1u);
  const uint32_t nact = active_slots(v);
  const uint32_t i = v.entries[eld];
  real4 pi, di;
  load_row_pair(&rows[2 * (size_t)eld], pi, di);
  uint32_t cnt[LPT];
#pragma unroll
  for (int u = 0; u < LPT; u++) cnt[u] = v.ncount[(size_t)(h * LPT + u) * NS + eld];
  issued(nact);
  issued(i);
#pragma unroll
  for (int u = 0; u < LPT; u++) issued(cnt[u]);
  const bool act = e0 < nact && i >= (uint32_t)v.S;
  if (DL > 1) {
    if (!__any_sync(0xffffffffu, act)) return;
  } else if (!act) {
    return;
  }
  const real H = P->fluid_h, H2 = H * H;
  real sx = 0.f, sy = 0.f, sz = 0.f;
  if (act) {
    const real maxPair = 0.05f * H;
    const real k = P->stiffness, kn = P->near_stiffness, rho0 = P->rest_density;
    const real Pi = k * (di.x - rho0);
    const real PNi = kn * di.y;
#ifndef UPBD_PARITY_BUILD
    const real invH = 1.0f / H;
#endif
    auto pair = [&](const real4& pj, const real4& dj) {
      const real ex = pj.x - pi.x, ey = pj.y - pi.y, ez = pj.z - pi.z;
      const real d2 = dot3(ex, ey, ez, ex, ey, ez);
      if (d2 >= H2 || d2 < 1e-12f) return;
#ifdef UPBD_PARITY_BUILD
      const real d = r_sqrt(d2);
      const real q = 1.0f - d / H;
#else
      const real rd = r_rsqrt(d2);  // d2 >= 1e-12 here
      const real d = d2 * rd;
      const real q = 1.0f - d * invH;
#endif
      const real Pj = k * (dj.x - rho0);
      const real PNj = kn * dj.y;
      real D = 0.25f * ((Pi + Pj) * q + (PNi + PNj) * q * q);
      D = clampf(D, -maxPair, maxPair);
#ifdef UPBD_PARITY_BUILD
      const real f = D / d;
#else
      const real f = D * rd;
#endif
      sx = sx - ex * f; sy = sy - ey * f; sz = sz - ez * f;
    };
    const int l0 = h * LPT;
    bool over = false;
#pragma unroll
    for (int u = 0; u < LPT; u++) over = over || cnt[u] > NL;
    if (!over) {
      uint32_t* const nbr = v.nbr + e0;
#pragma unroll
      for (int u = 0; u < LPT; u++) {
        // four entries at a time: their list, position and density loads are
        // in flight together (a lane list holds ~4)
        for (uint32_t c = 0; c < cnt[u]; c += 4) {
          uint32_t e[4];
          real4 pj[4], dj[4];
#pragma unroll
          for (int w = 0; w < 4; w++) {
            // entries beyond H (listed for xsph) and past the count become the
            // own slot, which pair() skips (d2 = 0)
            const uint32_t r = (c + w < cnt[u]) ? __ldg(list_entry(nbr, (uint32_t)(l0 + u) * NL + c + w, NS)) : e0;
            e[w] = (r & NBR_IN) ? (r & ~NBR_IN) : e0;
            if (!UPBD_IDX_OK(v, e[w], NS)) e[w] = e0;  // out of range: the own slot (skipped, reported)
          }
#pragma unroll
          for (int w = 0; w < 4; w++) load_row_pair(&rows[2 * (size_t)e[w]], pj[w], dj[w]);
#pragma unroll
          for (int w = 0; w < 4; w++)
            if (c + w < cnt[u]) pair(pj[w], dj[w]);
        }
      }
    } else {
      // lane l's share of the walk: candidates c = l, l+GLF, ... of the sequence
      CellHash ch;
      ch.init(pi.x, pi.y, pi.z, P->inv_cell);
      const uint32_t mask = (uint32_t)v.T - 1u;
      for (int l = l0; l < l0 + LPT; l++) {
        uint32_t c = 0;
        for (int kk = 0; kk < 27; kk++) {
          const uint32_t hb = ch.bucket_k(kk, mask);
          const uint2 r = bucket_range<0>(v, hb);
          for (uint32_t e = r.x; e < r.x + r.y; e++, c++)
            if ((c & (GLF - 1)) == (uint32_t)l && e != e0) pair(rows[2 * (size_t)e], rows[2 * (size_t)e + 1]);
        }
      }
    }
  }
#pragma unroll
  for (int d = DL / 2; d > 0; d >>= 1) {
    sx = sx + __shfl_xor_sync(0xffffffffu, sx, d);
    sy = sy + __shfl_xor_sync(0xffffffffu, sy, d);
    sz = sz + __shfl_xor_sync(0xffffffffu, sz, d);
  }
  if (!act || h != 0) return;
  const real maxTotal = 0.35f * H;
  const real s2 = dot3(sx, sy, sz, sx, sy, sz);
  if (s2 > maxTotal * maxTotal) {
    const real f = maxTotal / r_sqrt(s2);
    sx = sx * f; sy = sy * f; sz = sz * f;
  }
  if (APPLY) {  // pi is pos[i] (but for its w): the grid build copied it and nothing moved it since
    const real4 p = make_real4(pi.x + sx, pi.y + sy, pi.z + sz, di.z);
    v.pos[i] = p;
    v.sfp[e0] = p;
    mark_if_cell_changed(v, P, (int)i, pi, p);
  } else {
    v.delta[i] = make_real4(sx, sy, sz, 1.0f);
  }
}

// applyDeltaFluid, src/gpu/wgsl.js:318-323 (standalone form)
__device__ __forceinline__ void b_apply_fluid(const SimView& v, const DevParams* __restrict__ P, uint32_t vb) {
  const int i = v.S + (int)UPBD_VTID;
  if (i >= v.N) return;
  if (!(v.flags[i] & F_ACTIVE)) return;
  const real4 o = v.pos[i];
  real4 p = o;
  const real4 d = v.delta[i];
  p.x = p.x + d.x; p.y = p.y + d.y; p.z = p.z + d.z;
  v.pos[i] = p;
  v.sfp[v.slot[i]] = p;
  mark_if_cell_changed(v, P, i, o, p);
}

// ------------------------------------------------------------------ solids
// Marks the fluid particles within contact range of solid i at position p
// (G lanes per solid). The bound is widened by 1e-5 so the set only grows:
// the contacts pass makes the exact test.
// Every lane of the warp calls it (the hash is shared by shuffles); only
// active solids walk.
// FROM_GRID: the fluid's positions are those of the grid build (spos), from
// before its displacement, which moves a particle by at most 0.35 H (the
// displacement pass's clamp): the reach grows by that much (and a relative
// 1e-3, far above the rounding of the positions), so every particle that
// ends within contact range is marked, and the marks need not wait for the
// displacement pass.
template <int G = GL, bool FROM_GRID = false>
__device__ __forceinline__ void mark_fluid_near(const SimView& v, const DevParams* __restrict__ P, real4 p,
                                                bool act, int lane) {
  CellHash ch;
  group_cell_hash<G>(p.x, p.y, p.z, P->inv_cell, ch);
  const real rsum = P->solid_radius + P->fluid_radius;
  const real reach = FROM_GRID ? (rsum + 0.35f * P->fluid_h) * 1.001f : rsum;
  const real lim2 = reach * reach * 1.00001f;
  // without FROM_GRID the fluid has moved by its displacement (sfp)
  const real4* __restrict__ sfp = FROM_GRID ? v.spos : v.sfp;
  uint32_t* __restrict__ mark = v.mark;
  lane_strided<0, G>(v, ch, lane, act, [&](uint32_t e) { return sfp[e]; }, [&](uint32_t e, const real4& pj) {
    const real ex = p.x - pj.x, ey = p.y - pj.y, ez = p.z - pj.z;
    if (ex * ex + ey * ey + ez * ez < lim2) {
      const uint32_t j = v.entries[e];
      if (UPBD_IDX_OK(v, j, v.N)) mark[j] = 1u;
    }
  });
}

// solidSolve, src/gpu/wgsl.js:326-359, GL lanes per solid: lane l takes the
// incident constraints k = st+l, st+l+GL, ... of the static CSR, whose other
// endpoint and pair scale 1/max(deg_i, deg_j) are precomputed (both are fixed
// for the life of the scene); the partials combine like lane_sum.
// U constraints' loads are in flight together. Bound by the latency of its
// loads (offsets -> constraint ids and other ends -> constraint and position):
// with two in flight behind one another's branches a launch took 10.7 us on
// 8,512 solids, with four at once 8.7 (B200, event-timed, about 4 of which are
// the launch). The batch, bound by occupancy, keeps two and 40 registers.
// Threads from solid_pad on (a warp multiple, so the solve's warps are whole)
// apply the fluid displacement when APPLY_FLUID (applyDeltaFluid,
// src/gpu/wgsl.js:318-323): the solve reads solid positions only.
//
// OUT selects what the solve does with solid i's correction:
//   SOLVE_DELTA  writes delta[i] for b_apply_solid (the reference's split).
//   SOLVE_STEP   applies it too (applyDeltaSolid, src/gpu/wgsl.js:361-366) as
//                one phase of the folded solve (below).
//   SOLVE_LAST   the last phase: applies it into pos and the slot copy, then
//                marks the fluid near the final position (b_apply_solid's
//                work).
//   SOLVE_FINAL  as SOLVE_LAST without the marks (b_contact_mark follows).
//
// The folded solve is a sequence of Q >= 2 phases: per iteration the distance
// solve, then the tet solve and the solid contacts where the scene has them,
// each with its apply. Phase q reads the positions phase q - 1 left and writes
// the other of two copies (solid_src, solid_store): pos -> sbuf[0] -> sbuf[1]
// -> sbuf[0] ... -> pos and the slot copy, inactive solids carried over. Every
// phase reads its predecessor's positions only, as the split passes do, with
// the same expressions, so the results are the split passes' bit for bit.
// (One phase alone may not write what it reads: that case stays split.)
// A phase is a launch of a few microseconds of dependent loads, so what
// counts is their number: with tets and contacts 24 a substep of 8 iterations
// instead of 48.
constexpr int SOLVE_DELTA = 0, SOLVE_STEP = 1, SOLVE_LAST = 2, SOLVE_FINAL = 3;
__device__ __forceinline__ const real4* solid_src(const SimView& v, int q) {
  return q == 0 ? v.pos : v.sbuf + (size_t)((q - 1) & 1) * v.S;
}
template <bool LAST>
__device__ __forceinline__ void solid_store(const SimView& v, int q, int i, bool act, const real4& p) {
  if (!LAST) {
    v.sbuf[(size_t)(q & 1) * v.S + i] = p;
  } else if (act) {
    v.pos[i] = p;
    v.spos[v.slot[i]] = p;
  }
}

template <bool APPLY_FLUID, int OUT, int U>
__device__ __forceinline__ void b_solid_solve(const SimView& v, const DevParams* __restrict__ P, int solid_pad, int q,
                                              uint32_t vb) {
  const int t = UPBD_VTID;
  if (t >= solid_pad) {
    const int i = v.S + (t - solid_pad);
    if (APPLY_FLUID && i < v.N && (v.flags[i] & F_ACTIVE)) {
      const real4 o = v.pos[i];
      real4 p = o;
      const real4 d = v.delta[i];
      p.x = p.x + d.x; p.y = p.y + d.y; p.z = p.z + d.z;
      v.pos[i] = p;
      v.sfp[v.slot[i]] = p;
      mark_if_cell_changed(v, P, i, o, p);
    }
    return;
  }
  const int i = t / GL;
  const int lane = threadIdx.x & (GL - 1);
  const real4* __restrict__ pos = (OUT == SOLVE_DELTA) ? v.pos : solid_src(v, q);
  real4 pi = make_real4(0.f, 0.f, 0.f, 0.f);
  uint32_t fl = 0, st = 0, en = 0;
  if (i < v.S) {
    fl = v.flags[i];
    pi = pos[i];
    st = v.adj[i];
    en = v.adj[i + 1];
    issued(fl);
    issued(pi);
    issued(st);
    issued(en);
  }
  const bool act = (fl & F_ACTIVE) != 0u;
  real cx = 0.f, cy = 0.f, cz = 0.f;
  if (act) {
    const real wi = pi.w;
    const real h = P->h;
    const real alpha = P->compliance / (h * h);
    const uint32_t* __restrict__ ids = v.adj + v.S + 1;
    const uint4* __restrict__ cons = v.cons;
    // U constraints at a time: their loads are in flight together (a lane has
    // at most four of an inner solid's 26)
    for (uint32_t k0 = st + lane; k0 < en; k0 += GL * U) {
      uint32_t ci[U], other[U];
      real s[U];
      real4 po[U];
      uint2 rw[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const uint32_t k = min(k0 + (uint32_t)(u * GL), en - 1u);
        ci[u] = __ldg(&ids[k]);
        other[u] = __ldg(&v.adj_other[k]);
        s[u] = __ldg(&v.adj_scale[k]);
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (!UPBD_IDX_OK(v, ci[u], v.C) || !UPBD_IDX_OK(v, other[u], v.S)) {
          rw[u] = make_uint2(0u, 0u);
          po[u] = pi;
          continue;
        }
        po[u] = pos[other[u]];
        rw[u] = *reinterpret_cast<const uint2*>(&cons[ci[u]].z);  // rest bits, alive
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (k0 + (uint32_t)(u * GL) >= en || rw[u].y == 0u) continue;
        const real rest = __uint_as_float(rw[u].x);
        const real ex = pi.x - po[u].x, ey = pi.y - po[u].y, ez = pi.z - po[u].z;
        const real d = r_sqrt(dist2_xy(ex, ey, ez));
        if (d < 1e-9f) continue;
        const real wsum = wi + po[u].w;
        if (wsum == 0.f) continue;
        const real dl = -(d - rest) / (wsum + alpha);
        const real f = dl * wi / d * s[u];
        cx = cx + ex * f; cy = cy + ey * f; cz = cz + ez * f;
      }
    }
  }
  cx = lane_sum(cx);
  cy = lane_sum(cy);
  cz = lane_sum(cz);
  if (OUT == SOLVE_DELTA) {
    if (act && lane == 0) v.delta[i] = make_real4(cx, cy, cz, 1.0f);
    return;
  }
  // applyDeltaSolid on the correction just summed (the delta b_apply_solid reads)
  const real w = P->omega;
  real4 p = pi;
  if (act) {
    p.x = p.x + cx * w; p.y = p.y + cy * w; p.z = p.z + cz * w;
  }
  if (i < v.S && lane == 0) solid_store<OUT != SOLVE_STEP>(v, q, i, act, p);
  if (OUT == SOLVE_LAST && P->use_mark) mark_fluid_near(v, P, act ? p : make_real4(0.f, 0.f, 0.f, 0.f), act, lane);
}

// applyDeltaSolid, src/gpu/wgsl.js:361-366, of a solve of one split
// iteration: GL lanes per solid, which also mark the fluid near its final
// position for the contacts pass; the fluid positions are final by then.
__device__ __forceinline__ void b_apply_solid(const SimView& v, const DevParams* __restrict__ P, uint32_t vb) {
  const int t = UPBD_VTID;
  const int i = t / GL;
  const bool act = i < v.S && (v.flags[i] & F_ACTIVE);
  const real w = P->omega;
  real4 p = make_real4(0.f, 0.f, 0.f, 0.f);
  if (act) {
    p = v.pos[i];
    const real4 d = v.delta[i];
    p.x = p.x + d.x * w; p.y = p.y + d.y * w; p.z = p.z + d.z * w;
  }
  const int lane = threadIdx.x & (GL - 1);
  if (act && lane == 0) {
    v.pos[i] = p;
    v.spos[v.slot[i]] = p;
  }
  if (P->use_mark) mark_fluid_near(v, P, p, act, lane);
}

// Contact marking on its own (when the solve's last position update does not
// carry it), G lanes per solid. Marks are a set, so the lane count is free:
// a whole warp per solid makes the 27 bucket lookups one round.
template <int G = GL, bool FROM_GRID = false>
__device__ __forceinline__ void b_contact_mark(const SimView& v, const DevParams* __restrict__ P, uint32_t vb) {
  if (!P->use_mark) return;
  const int t = UPBD_VTID;
  const int i = t / G;
  const bool act = i < v.S && (v.flags[i] & F_ACTIVE);
  mark_fluid_near<G, FROM_GRID>(v, P, act ? v.pos[i] : make_real4(0.f, 0.f, 0.f, 0.f), act, threadIdx.x & (G - 1));
}

// latticeRest, src/gpu/wgsl.js:373-381
__device__ __forceinline__ real lattice_rest(const SimView& v, real spacing, uint32_t a0, uint32_t b0) {
  uint32_t a = a0, b = b0, D = (uint32_t)v.dim1;
  if (a0 >= (uint32_t)v.N1) { a = a0 - v.N1; b = b0 - v.N1; D = (uint32_t)(v.dim2 > 1 ? v.dim2 : 1); }
  const real ax = (real)(a / (D * D)), ay = (real)((a / D) % D), az = (real)(a % D);
  const real bx = (real)(b / (D * D)), by = (real)((b / D) % D), bz = (real)(b % D);
  const real dx = ax - bx, dy = ay - by, dz = az - bz;
  return spacing * r_sqrt(dx * dx + dy * dy + dz * dz);
}

// solidRsum: the contact distance of two solids, lattice neighbours or not
__device__ __forceinline__ real solid_rsum(const DevParams* __restrict__ P, bool near) {
  const real rsum = 2.0f * P->solid_radius;
  if (near) return mn(rsum, P->spacing * 0.97f);
  return rsum;
}

// collectContacts, src/gpu/wgsl.js:532-560, a warp per solid: the lanes take
// 32 candidates of the solids' part of the 27 buckets at a time, in sequence
// order, and a ballot gives each kept one its place, so the cache holds what
// one invocation of the reference would list (the first C_K kept candidates).
// A candidate's position is its slot copy (the solve writes the copies only at
// its end). The solid's lattice neighbours (at most 26, ascending, one per lane)
// are searched by shuffles: a candidate found there is adjacent, and bonded if
// its constraint is alive. Entries carry CL_NEAR for lattice neighbours, whose
// contact distance differs (solid_rsum), so the iterations need no index
// arithmetic. Bound by the latency of its three or four dependent loads. One
// thread per solid, as a chain of ~70 candidates with a constraint scan for each
// in range, took 710 us a launch on 8,512 solids (B200, event-timed); a warp with
// lattice coordinates by division and 26 shuffles a round 24.9, this 14.8.
__device__ __forceinline__ void b_collect_contacts(const SimView& v, const DevParams* __restrict__ P, uint32_t vb) {
  const unsigned FULL = 0xffffffffu;
  const int i = (int)(UPBD_VTID >> 5), lane = (int)(threadIdx.x & 31);
  if (i >= v.S) return;  // whole warps
  if (!(v.flags[i] & F_ACTIVE)) {
    if (lane == 0) v.ccount[i] = 0u;
    return;
  }
  const real4 pi = v.pos[i];
  CellHash ch;
  group_cell_hash<32>(pi.x, pi.y, pi.z, P->inv_cell, ch);
  const int row = (int)(threadIdx.x >> 5) * (32 / GLF);
  const uint32_t run = walk_tables<1, 32>(v, ch, lane, true, row);
  // the solid's lattice neighbours, one a lane in ascending index, and which of
  // their constraints are alive
  const uint32_t st = v.adj[i], deg = v.adj[i + 1] - st;
  uint32_t neighbour = 0xffffffffu;
  bool tied = false;
  if ((uint32_t)lane < deg) {
    const uint32_t ci = v.adj[v.S + 1 + st + lane];
    neighbour = v.adj_other[st + lane];
    tied = UPBD_IDX_OK(v, ci, v.C) && v.cons[ci].w != 0u;
  }
  const unsigned bonds = __ballot_sync(FULL, tied);
  const real margin = 2.0f * P->solid_radius;
  const real lim_near = solid_rsum(P, true) + margin, lim_far = solid_rsum(P, false) + margin;
  uint32_t cnt = 0, k = 0, next = s_walk_off[row][1], base = s_walk_base[row][0];
  for (uint32_t c0 = 0; c0 < run && cnt < C_K; c0 += 32) {
    const uint32_t c = c0 + (uint32_t)lane;
    uint32_t j = 0xffffffffu;
    real d2 = 0.f;
    if (c < run) {
      while (c >= next) {
        k++;
        next = s_walk_off[row][k + 1];
        base = s_walk_base[row][k];
      }
      const uint32_t e = base + c;
      if (UPBD_IDX_OK(v, e, v.N)) {
        j = v.entries[e];
        const real4 pj = v.spos[e];
        const real ex = pi.x - pj.x, ey = pi.y - pj.y, ez = pi.z - pj.z;
        d2 = dot3(ex, ey, ez, ex, ey, ez);
      }
    }
    const bool other = j != (uint32_t)i && j < (uint32_t)v.S;
    // latticeAdjacent (src/gpu/wgsl.js:409-416) is the 26-neighbourhood, which
    // is what the constraints tie; isBonded (599-607) asks for an alive one.
    // The place of j among the neighbours, five halvings:
    uint32_t at = 0;
#pragma unroll
    for (uint32_t h = 16; h > 0; h >>= 1)
      if (__shfl_sync(FULL, neighbour, (int)(at + h - 1u)) < j) at += h;
    const bool near = __shfl_sync(FULL, neighbour, (int)at) == j && other;
    const real lim = near ? lim_near : lim_far;
    const bool keep = other && !(d2 >= lim * lim) && !(near && (bonds >> at & 1u));
    const unsigned kept = __ballot_sync(FULL, keep);
    const uint32_t place = cnt + (uint32_t)__popc(kept & ((1u << lane) - 1u));
    if (keep && place < C_K) v.clist[(size_t)i * C_K + place] = j | (near ? CL_NEAR : 0u);
    cnt = min(cnt + (uint32_t)__popc(kept), C_K);
  }
  if (lane == 0) v.ccount[i] = cnt;
  __syncwarp();  // the next call may rewrite this warp's tables
}

// Clamp of applySolidContacts (src/gpu/wgsl.js:587-596) on a correction of
// solid position p: the apply of the tet and contact phases.
__device__ __forceinline__ real4 apply_clamped(const DevParams* __restrict__ P, real4 p, real dx, real dy, real dz) {
  const real maxC = 0.5f * P->solid_radius;
  const real m2 = dot3(dx, dy, dz, dx, dy, dz);
  if (m2 > maxC * maxC) {
    const real f = maxC / r_sqrt(m2);
    dx = dx * f; dy = dy * f; dz = dz * f;
  }
  p.x = p.x + dx; p.y = p.y + dy; p.z = p.z + dz;
  return p;
}

// solidContacts + applySolidContacts, src/gpu/wgsl.js:562-596, as a phase of
// the folded solve: GL lanes per solid take the cache's entries side by side,
// then every lane adds the terms up in the cache's order (one fused or one
// rounded multiply-add per term, as the one-thread loop). An uncut lattice
// lists about six entries a solid, so one round.
template <bool LAST>
__device__ __forceinline__ void b_solid_contacts(const SimView& v, const DevParams* __restrict__ P, int q, uint32_t vb) {
  const unsigned FULL = 0xffffffffu;
  const int i = (int)(UPBD_VTID / GL), lane = (int)(threadIdx.x & (GL - 1));
  const real4* __restrict__ pos = solid_src(v, q);
  real4 pi = make_real4(0.f, 0.f, 0.f, 0.f);
  uint32_t fl = 0, n = 0, e = 0;
  if (i < v.S) {
    fl = v.flags[i];
    n = v.ccount[i];
    pi = pos[i];
    e = v.clist[(size_t)i * C_K + lane];  // the first round's entry, should there be one
    issued(fl);
    issued(n);
    issued(pi);
    issued(e);
  }
  const bool act = (fl & F_ACTIVE) != 0u;
  if (!act) n = 0;
  const real wi = pi.w;
  real cx = 0.f, cy = 0.f, cz = 0.f;
  for (uint32_t k0 = 0; __any_sync(FULL, k0 < n); k0 += GL) {
    real ex = 0.f, ey = 0.f, ez = 0.f, f = 0.f;
    bool hit = false;
    if (k0 + (uint32_t)lane < n) {
      if (k0 > 0) e = v.clist[(size_t)i * C_K + k0 + lane];
      const uint32_t j = e & ~CL_NEAR;
      if (UPBD_IDX_OK(v, j, v.S)) {
        const real4 pj = pos[j];
        const real dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
        const real rsum = solid_rsum(P, (e & CL_NEAR) != 0u);
        const real d2 = dot3(dx, dy, dz, dx, dy, dz);
        const real wsum = wi + pj.w;
        hit = !(d2 >= rsum * rsum || d2 < 1e-12f) && wsum != 0.f;
        if (hit) {
          const real d = r_sqrt(d2);
          ex = dx; ey = dy; ez = dz;
          f = (rsum - d) / d * wi / wsum * 0.5f;
        }
      }
    }
    if (!__any_sync(FULL, hit)) continue;
#pragma unroll
    for (int l = 0; l < GL; l++) {
      const real fl = __shfl_sync(FULL, f, l, GL);
      cx = cx + __shfl_sync(FULL, ex, l, GL) * fl;
      cy = cy + __shfl_sync(FULL, ey, l, GL) * fl;
      cz = cz + __shfl_sync(FULL, ez, l, GL) * fl;
    }
  }
  if (i < v.S && lane == 0) solid_store<LAST>(v, q, i, act, act ? apply_clamped(P, pi, cx, cy, cz) : pi);
}

__device__ __forceinline__ void cross3(real ax, real ay, real az, real bx, real by, real bz,
                                       real& x, real& y, real& z) {
  x = ay * bz - az * by;
  y = az * bx - ax * bz;
  z = ax * by - ay * bx;
}

// solveTets, src/gpu/wgsl.js:423-468: corner i's correction from one tet with
// corners q, rest volume V0 and pair scale s
__device__ __forceinline__ void tet_corner(const DevParams* __restrict__ P, const real4* __restrict__ pos, uint32_t i,
                                           const uint4& q, real V0, real s, real& ox, real& oy, real& oz) {
  ox = 0.f; oy = 0.f; oz = 0.f;
  const real4 pa = pos[q.x], pb = pos[q.y], pc = pos[q.z], pd = pos[q.w];
  const real bax = pb.x - pa.x, bay = pb.y - pa.y, baz = pb.z - pa.z;
  const real cax = pc.x - pa.x, cay = pc.y - pa.y, caz = pc.z - pa.z;
  const real dax = pd.x - pa.x, day = pd.y - pa.y, daz = pd.z - pa.z;
  real xx, xy, xz;
  cross3(bax, bay, baz, cax, cay, caz, xx, xy, xz);
  const real V = dot3(xx, xy, xz, dax, day, daz) / 6.0f;
  const real Cv = V - V0;
  real gbx, gby, gbz, gcx, gcy, gcz, gdx, gdy, gdz;
  cross3(cax, cay, caz, dax, day, daz, gbx, gby, gbz);
  gbx = gbx / 6.0f; gby = gby / 6.0f; gbz = gbz / 6.0f;
  cross3(dax, day, daz, bax, bay, baz, gcx, gcy, gcz);
  gcx = gcx / 6.0f; gcy = gcy / 6.0f; gcz = gcz / 6.0f;
  cross3(bax, bay, baz, cax, cay, caz, gdx, gdy, gdz);
  gdx = gdx / 6.0f; gdy = gdy / 6.0f; gdz = gdz / 6.0f;
  const real gax = -((gbx + gcx) + gdx), gay = -((gby + gcy) + gdy), gaz = -((gbz + gcz) + gdz);
  const real w = pa.w;
  const real denom = w * (dot3(gax, gay, gaz, gax, gay, gaz) + dot3(gbx, gby, gbz, gbx, gby, gbz) +
                           dot3(gcx, gcy, gcz, gcx, gcy, gcz) + dot3(gdx, gdy, gdz, gdx, gdy, gdz));
  if (denom < 1e-12f) return;
  const real dl = -Cv / denom;
  real gx = gax, gy = gay, gz = gaz;
  if (i == q.y) { gx = gbx; gy = gby; gz = gbz; }
  else if (i == q.z) { gx = gcx; gy = gcy; gz = gcz; }
  else if (i == q.w) { gx = gdx; gy = gdy; gz = gdz; }
  const real f = w * dl * s;
  real c1x = gx * f, c1y = gy * f, c1z = gz * f;
  const real cl2 = dot3(c1x, c1y, c1z, c1x, c1y, c1z);
  const real lim = 0.5f * P->solid_radius;
  if (cl2 > lim * lim) {
    const real g = lim / r_sqrt(cl2);
    c1x = c1x * g; c1y = c1y * g; c1z = c1z * g;
  }
  ox = c1x; oy = c1y; oz = c1z;
}

// solveTets + its apply, a phase of the folded solve: G lanes per solid
// compute the corrections of its next G tets side by side (corners and pair
// scale in one row per incidence), then every lane adds them up in the CSR's
// order, so the sum is the one-thread loop's. Bound by latency (record ->
// corners -> arithmetic): inner solids have 8 or 32 tets, so one or two rounds
// of 16 lanes; one thread per solid, 32 tets in a chain, took 34 us a launch
// on 8,512 solids (B200, event-timed), 16 lanes take 10.7. One round of 32
// lanes is faster where the launch fits one block an SM (793 solids: 8.5
// against 8.8 us), slower where half its lanes' issue slots are missed (8,512:
// 12.7).
template <bool LAST, int G = GT>
__device__ __forceinline__ void b_solve_tets(const SimView& v, const DevParams* __restrict__ P, int q, uint32_t vb) {
  const unsigned FULL = 0xffffffffu;
  const int i = (int)(UPBD_VTID / G), lane = (int)(threadIdx.x & (G - 1));
  const real4* __restrict__ pos = solid_src(v, q);
  const uint32_t* __restrict__ ids = v.tet_adj + v.S + 1;
  real4 pi = make_real4(0.f, 0.f, 0.f, 0.f);
  uint32_t fl = 0, st = 0, en = 0;
  if (i < v.S) {
    fl = v.flags[i];
    st = v.tet_adj[i];
    en = v.tet_adj[i + 1];
    pi = pos[i];
    issued(fl);
    issued(st);
    issued(en);
    issued(pi);
  }
  const bool act = (fl & F_ACTIVE) != 0u;
  if (!act) en = st;
  real cx = 0.f, cy = 0.f, cz = 0.f;
  for (uint32_t k0 = st; __any_sync(FULL, k0 < en); k0 += G) {
    const uint32_t k = k0 + (uint32_t)lane;
    real ox = 0.f, oy = 0.f, oz = 0.f;
    if (k < en) {
      const uint4 c = __ldg(&v.tet_rec[k]);
      const uint32_t t = __ldg(&ids[k]);
      const real s = __ldg(&v.tet_scale[k]);
      if (UPBD_IDX_OK(v, t, v.NT) && UPBD_IDX_OK(v, c.x, v.S) && UPBD_IDX_OK(v, c.y, v.S) && UPBD_IDX_OK(v, c.z, v.S) &&
          UPBD_IDX_OK(v, c.w, v.S)) {
        const real V0 = v.tet_vol[t];
        if (!(V0 <= 0.f)) tet_corner(P, pos, (uint32_t)i, c, V0, s, ox, oy, oz);
      }
    }
#pragma unroll
    for (int l = 0; l < G; l++) {
      cx = cx + __shfl_sync(FULL, ox, l, G);
      cy = cy + __shfl_sync(FULL, oy, l, G);
      cz = cz + __shfl_sync(FULL, oz, l, G);
    }
  }
  if (i < v.S && lane == 0) solid_store<LAST>(v, q, i, act, act ? apply_clamped(P, pi, cx, cy, cz) : pi);
}

// -------------------------------------------- bond update + contacts
// Threads [0, nb) run bondUpdate (src/gpu/wgsl.js:383-404) on one constraint
// each, threads [nb, nb+nt) run tetUpdate (src/gpu/wgsl.js:472-491), threads
// [nb+nt, nb+nt+nc) run the solid↔fluid coupling gather `contacts`
// (src/gpu/wgsl.js:609-646). All three read positions only; their outputs
// (constraints, tets, delta) are disjoint.
__device__ __forceinline__ void bond_update(const SimView& v, const DevParams* __restrict__ P, int ci) {
  const uint4 c = v.cons[ci];
  if (c.w == 0u) return;
  if (!UPBD_IDX_OK(v, c.x, v.S) || !UPBD_IDX_OK(v, c.y, v.S)) return;
  const real4 pa = v.pos[c.x], pb = v.pos[c.y];
  const real ex = pa.x - pb.x, ey = pa.y - pb.y, ez = pa.z - pb.z;
  const real d = r_sqrt(dot3(ex, ey, ez, ex, ey, ez));
  const real rest = __uint_as_float(c.z);
  const bool tear = (P->tear_mode == 1) ? (d > rest * P->break_strain)
                                        : (d > rest + P->tear_gap * 2.0f * P->solid_radius);
  if (tear) {
    v.cons[ci].w = 0u;
    return;
  }
  const real strain = (d - rest) / rest;
  real nr = rest;
  if (r_fabs(strain) > P->plastic_threshold) nr = rest + (d - rest) * P->plastic_rate;
  if (P->plastic_clamp) {
    const real r0 = lattice_rest(v, P->spacing, c.x, c.y);
    nr = clampf(nr, 0.9f * r0, 1.25f * r0);
  }
  if (nr != rest) v.cons[ci].z = __float_as_uint((float)nr);
}

__device__ __forceinline__ void tet_update(const SimView& v, const DevParams* __restrict__ P, int t) {
  const real V0 = v.tet_vol[t];
  if (V0 <= 0.f) return;
  const real gap = P->tear_gap * 2.0f * P->solid_radius;
  for (int p = 0; p < 3; p++)
    for (int q = p + 1; q < 4; q++) {
      const uint32_t a = v.tet_idx[4 * t + p], b = v.tet_idx[4 * t + q];
      if (!UPBD_IDX_OK(v, a, v.S) || !UPBD_IDX_OK(v, b, v.S)) return;
      const real4 pa = v.pos[a], pb = v.pos[b];
      const real ex = pa.x - pb.x, ey = pa.y - pb.y, ez = pa.z - pb.z;
      const real d = r_sqrt(dot3(ex, ey, ez, ex, ey, ez));
      if (d > lattice_rest(v, P->spacing, a, b) + gap) {
        v.tet_vol[t] = -V0;
        return;
      }
    }
}

// contacts for particle i, lane `lane` of its GL; every lane reaches the
// shuffles. Fluid particles that no solid marked have no contact and skip the
// walk (their correction is zero either way).
__device__ __forceinline__ void contacts_lane(const SimView& v, const DevParams* __restrict__ P, int i, int lane,
                                              int nc) {
  uint32_t fl = 0, mk = 0;
  if (i < nc) {
    fl = v.flags[i];
    mk = v.mark[i];
    issued(fl);
    issued(mk);
  }
  const bool act = (fl & F_ACTIVE) != 0u;
  const bool iSolid = i < v.S;
  const bool walk = act && (iSolid || !P->use_mark || mk != 0u);
  const unsigned FULL = 0xffffffffu;
  if (!__any_sync(FULL, walk)) {  // most fluid warps: nothing near a solid, no hash to compute
    if (act && lane == 0) v.delta[i] = make_real4(0.f, 0.f, 0.f, 0.f);
    return;
  }
  real cx = 0.f, cy = 0.f, cz = 0.f, cnt = 0.f;
  const real4 pi = walk ? v.pos[i] : make_real4(0.f, 0.f, 0.f, 0.f);
  CellHash ch;
  group_cell_hash(pi.x, pi.y, pi.z, P->inv_cell, ch);
  const real wi = pi.w;
  const real rs = P->solid_radius, rf = P->fluid_radius, scale = P->contact_scale;
  // a solid meets the fluid part of each bucket, a fluid particle the solid
  // part (fluid-fluid is DDR's job, solid-solid the contact cache's)
  const real ri = iSolid ? rs : rf;
  const real rsum = ri + (iSolid ? rf : rs);
  const real4* __restrict__ spos = v.spos;
  const real4* __restrict__ sfp = v.sfp;
  auto load_fluid = [&](uint32_t e) { return sfp[e]; };  // after the displacement
  auto load_solid = [&](uint32_t e) { return spos[e]; };  // after the solve
  auto pair = [&](uint32_t, const real4& pj) {
    const real ex = pi.x - pj.x, ey = pi.y - pj.y, ez = pi.z - pj.z;
    const real d2 = dot3(ex, ey, ez, ex, ey, ez);
    if (d2 >= rsum * rsum || d2 < 1e-12f) return;
    const real wsum = wi + pj.w;
    if (wsum == 0.f) return;
#ifdef UPBD_PARITY_BUILD
    const real d = r_sqrt(d2);
    const real f = (rsum - d) / d * wi / wsum * scale;
#else
    const real rd = r_rsqrt(d2);  // d2 >= 1e-12 here
    const real f = (rsum - d2 * rd) * rd * r_fdiv(wi, wsum) * scale;
#endif
    cx = cx + ex * f; cy = cy + ey * f; cz = cz + ez * f;
    cnt = cnt + 1.0f;
  };
  // a warp holds solids or fluid or both (at the S boundary): the two walks
  // are separate calls, each with every lane of the warp
  if (__any_sync(FULL, walk && iSolid)) lane_strided<0>(v, ch, lane, walk && iSolid, load_fluid, pair);
  if (__any_sync(FULL, walk && !iSolid)) lane_strided<1>(v, ch, lane, walk && !iSolid, load_solid, pair);
  cx = lane_sum(cx);
  cy = lane_sum(cy);
  cz = lane_sum(cz);
  cnt = lane_sum(cnt);
  if (act && lane == 0) v.delta[i] = make_real4(cx, cy, cz, cnt);
}

// nb_pad is nb + nt rounded up to a multiple of 32, so the contact threads
// start on a warp boundary and whole warps reach lane_sum's shuffles.
__device__ __forceinline__ void b_bond_contacts(const SimView& v, const DevParams* __restrict__ P,
                                                       int nb, int nt, int nb_pad, int nc, uint32_t vb) {
  // by groups of GL threads: the threads themselves pass 2^31 from 2^28 particles on
  const uint32_t group = vb * (blockDim.x / GL) + threadIdx.x / GL, first = (uint32_t)nb_pad / GL;
  if (group < first) {
    const int k = (int)(group * GL + (threadIdx.x & (GL - 1)));
    if (k < nb)
      bond_update(v, P, k);
    else if (k < nb + nt)
      tet_update(v, P, k - nb);
    return;
  }
  contacts_lane(v, P, (int)(group - first), (int)(threadIdx.x & (GL - 1)), nc);
}

// -------------------------------- apply + bounds + velocity (per particle)
// The movement allowance of xsph's list test (XSKIN above), the same float on
// both sides of the test.
__device__ __forceinline__ real xsph_allowance(const DevParams* __restrict__ P) {
  return XSKIN * P->fluid_h * XMOVE_FRAC;
}

// Records how far fluid particle i (at slot sl) moved since the density pass
// (o: the position that pass saw, which its slot copy holds until the bounds
// pass writes p there): smove gets the distance (+inf when the particle left
// its cell or a coordinate is not finite), its grid bucket's bmove and the
// scene's SCR_XMOVE the largest distance above the recording threshold (the
// latter one atomic per warp).
__device__ __forceinline__ void record_move(const SimView& v, const DevParams* __restrict__ P, int i, uint32_t sl,
                                            const real4& o, const real4& p) {
  const real dx = p.x - o.x, dy = p.y - o.y, dz = p.z - o.z;
  const real INF = __int_as_float(0x7f800000);
  real m = r_sqrt(dot3(dx, dy, dz, dx, dy, dz));
  if (!(m <= 3.0e38f)) m = INF;  // NaN or inf
  const double inv = P->inv_cell;
  const bool same = floor(__dmul_rn((double)o.x, inv)) == floor(__dmul_rn((double)p.x, inv)) &&
                    floor(__dmul_rn((double)o.y, inv)) == floor(__dmul_rn((double)p.y, inv)) &&
                    floor(__dmul_rn((double)o.z, inv)) == floor(__dmul_rn((double)p.z, inv));
  v.smove[sl] = same ? r_to_float_up(m) : __int_as_float(0x7f800000);
  const bool rec = m > XMOVE_REC * xsph_allowance(P);
  if (rec) atomicMax(&v.bmove[v.cell[i]], __float_as_uint(r_to_float_up(m)));
  const unsigned am = __activemask();
  const uint32_t wm = __reduce_max_sync(am, rec ? __float_as_uint(r_to_float_up(m)) : 0u);
  if (wm != 0u && (int)(threadIdx.x & 31) == __ffs(am) - 1) atomicMax(&v.scratch[SCR_XMOVE], wm);
}

// applyDeltaAll (src/gpu/wgsl.js:648-660), bounds (src/gpu/wgsl.js:663-697)
// and velocityUpdate (src/gpu/wgsl.js:700-710): each touches only its own
// particle, so one launch runs all three. stage 1/2/3 stops after the first,
// second or third.
__device__ __forceinline__ void b_apply_bounds_vel(const SimView& v, const DevParams* __restrict__ P,
                                                          int stage, uint32_t vb) {
  const int i = UPBD_VTID;
  if (i >= v.N) return;
  const uint32_t f = v.flags[i], sl = v.slot[i];
  real4 p = v.pos[i];
  const real4 dd = v.delta[i], pv = v.prev[i], ov = v.vel[i];
  issued(f);
  issued(sl);
  issued(p);
  issued(dd);
  issued(pv);
  issued(ov);
  if (!(f & F_ACTIVE)) return;
  const bool iSolid = i < v.S;
  const real r = iSolid ? P->solid_radius : P->fluid_radius;
  const real4 o = iSolid ? p : v.spos[sl];  // a fluid particle's density-pass position, read before any store
  // applyDeltaAll
  {
    real dx = dd.x, dy = dd.y, dz = dd.z;
    const real m2 = dot3(dx, dy, dz, dx, dy, dz);
    if (m2 > r * r) {
      const real g = r / r_sqrt(m2);
      dx = dx * g; dy = dy * g; dz = dz * g;
    }
    p.x = p.x + dx; p.y = p.y + dy; p.z = p.z + dz;
  }
  if (stage < 2) {
    v.pos[i] = p;
    return;
  }
  // bounds
  real px = p.x, py = p.y, pz = p.z;
  if (py < r) {
    py = r;
    const real mu = iSolid ? P->friction_solid : P->friction_fluid;
    px = px - (px - pv.x) * mu;
    pz = pz - (pz - pv.z) * mu;
  }
  if (py < P->wall_h + r) {
    const real lim = r + P->wall_t;
    const real wx = P->wall_x, wz = P->wall_z;
    if (r_fabs(r_fabs(px) - wx) < lim) {
      const real side = signf(px);
      px = (r_fabs(px) < wx) ? side * (wx - lim) : side * (wx + lim);
    }
    if (r_fabs(r_fabs(pz) - wz) < lim) {
      const real side = signf(pz);
      pz = (r_fabs(pz) < wz) ? side * (wz - lim) : side * (wz + lim);
    }
  }
  bool culled = false;
  if (!iSolid) {
    const real cr = P->cull_r;
    if (py < -3.0f || px * px + pz * pz > cr * cr) {
      v.flags[i] = 0u;
      culled = true;
    }
  }
  p.x = px; p.y = py; p.z = pz;
  v.pos[i] = p;
  if (stage < 3) return;
  if (!iSolid) record_move(v, P, i, sl, o, p);
  if (culled) {
    // xsph still reads a culled neighbour's velocity (src/gpu/wgsl.js:761
    // does not test its flag): its slot keeps the unchanged velocity
    store_row_pair(&v.pvrow[2 * (size_t)sl], make_real4(p.x, p.y, p.z, slot_pack(real(0), sl)), ov);
    return;
  }
  // velocityUpdate
  const real h = P->h;
  real vx = (p.x - pv.x) / h, vy = (p.y - pv.y) / h, vz = (p.z - pv.z) / h;
  const real damp = iSolid ? P->damp_solid : P->damp_fluid;
  const real g = mx(0.0f, 1.0f - damp * h);
  vx = vx * g; vy = vy * g; vz = vz * g;
  const real sp2 = dot3(vx, vy, vz, vx, vy, vz);
  const real ms = P->max_speed;
  if (sp2 > ms * ms) {
    const real q = ms / r_sqrt(sp2);
    vx = vx * q; vy = vy * q; vz = vz * q;
  }
  if (!isfinite(vx) || !isfinite(vy) || !isfinite(vz)) atomicOr(&v.scratch[SCR_HEALTH], 1u);
  const real4 nv = make_real4(vx, vy, vz, ov.w);
  v.vel[i] = nv;
  if (!iSolid) store_row_pair(&v.pvrow[2 * (size_t)sl], make_real4(p.x, p.y, p.z, slot_pack(real(0), sl)), nv);  // xsph's neighbours
}

// solidVisc, src/gpu/wgsl.js:717-735, GL lanes per solid: they load its next GL
// neighbours' velocities side by side, then every lane adds the bonded ones up
// in the CSR's order (the one-thread loop's sums). Bound by latency: one thread
// a solid, 26 neighbours in a chain, took 9.7 us a launch on 793 solids, 7.6 now
// (B200, event-timed).
__device__ __forceinline__ void b_solid_visc(const SimView& v, const DevParams* __restrict__ P, uint32_t vb) {
  const unsigned FULL = 0xffffffffu;
  const int i = (int)(UPBD_VTID / GL), lane = (int)(threadIdx.x & (GL - 1)), group = (int)(threadIdx.x & 31) & ~(GL - 1);
  uint32_t fl = 0, st = 0, en = 0;
  real4 vi = make_real4(0.f, 0.f, 0.f, 0.f);
  if (i < v.S) {
    fl = v.flags[i];
    st = v.adj[i];
    en = v.adj[i + 1];
    vi = v.vel[i];
    issued(fl);
    issued(st);
    issued(en);
    issued(vi);
  }
  const bool act = (fl & F_ACTIVE) != 0u;
  if (!act) en = st;
  real sx = 0.f, sy = 0.f, sz = 0.f, m = 0.f;
  for (uint32_t k0 = st; __any_sync(FULL, k0 < en); k0 += GL) {
    const uint32_t k = k0 + (uint32_t)lane;
    bool bonded = false;
    real4 vo = make_real4(0.f, 0.f, 0.f, 0.f);
    if (k < en) {
      const uint32_t ci = v.adj[v.S + 1 + k], other = v.adj_other[k];
      if (UPBD_IDX_OK(v, ci, v.C) && UPBD_IDX_OK(v, other, v.S)) {
        bonded = v.cons[ci].w != 0u;
        vo = v.vel[other];
      }
    }
    const unsigned bonds = __ballot_sync(FULL, bonded) >> group;
#pragma unroll
    for (int l = 0; l < GL; l++) {
      const real x = __shfl_sync(FULL, vo.x, l, GL), y = __shfl_sync(FULL, vo.y, l, GL), z = __shfl_sync(FULL, vo.z, l, GL);
      if (bonds >> l & 1u) {
        sx = sx + x; sy = sy + y; sz = sz + z;
        m = m + 1.0f;
      }
    }
  }
  if (!act || lane != 0) return;
  real vx = vi.x, vy = vi.y, vz = vi.z;
  if (m > 0.f) {
    const real mu = P->solid_viscosity;
    vx = vx + mu * (sx / m - vx);
    vy = vy + mu * (sy / m - vy);
    vz = vz + mu * (sz / m - vz);
  }
  v.delta[i] = make_real4(vx, vy, vz, 0.f);
}

// solidViscApply, src/gpu/wgsl.js:737-742
__device__ __forceinline__ void b_solid_visc_apply(const SimView& v, uint32_t vb) {
  const int i = UPBD_VTID;
  if (i >= v.S) return;
  if (!(v.flags[i] & F_ACTIVE)) return;
  const real4 d = v.delta[i];
  const real w = v.vel[i].w;
  v.vel[i] = make_real4(d.x, d.y, d.z, w);
}

// xsph, src/gpu/wgsl.js:745-771, over the density pass's chunks. The grid still
// holds the particles bounds culled this substep: they are neighbours (the
// reference does not test their flag) but have no pass of their own. Neighbour
// rows (position, velocity) are slot copies, so with APPLY the blended velocity
// goes straight to vel[i] (xsphApply's result, src/gpu/wgsl.js:773-778) and the
// copy pass is not needed; without it the result waits in delta, where the
// reference's xsph pass leaves it.
// A particle that passes the list test (XSKIN) has its lanes read their
// density-pass lists: each lane's listed candidates are a subsequence, in order,
// of its walk share that holds every candidate within H now. For the others the
// warp stages the candidates' positions and velocities around their present
// cell, as the density pass does, and the lanes walk the bits of those within H.
// Either way a lane adds the same terms in the same order (a candidate out of
// range would add +0 to a sum that starts at +0).
// Bound by latency (list entry -> row) where the fluid has settled, by the
// staged walks where it moves. With each group of lanes walking its own buckets
// in a launch of its own beside the list readers, the default scene's settled
// pool took 34.7 us (both forms in one launch; B200, an event pair around an
// eager launch), the large scene's splash 115.4; now 23.3 and 102.3. Position and
// velocity come as one 32-byte row: with two 16-byte rows a tenth longer. Windows
// of small chunks go by half-warps as in the density pass: in the large scene's
// fall 68 us, a warp a chunk 91.
constexpr uint32_t XROWS = STAGE / 2;  // candidates staged a round: positions and velocities in the same bytes
constexpr int XCH = 4;                 // list entries whose loads are in flight together
template <bool APPLY, int W>
__device__ __forceinline__ void xsph_chunks(const SimView& v, const DevParams* __restrict__ P, ChunkList& s_list,
                                            real4* sx, uint32_t first, uint32_t chunks, uint32_t halves, int tid) {
  const unsigned FULL = 0xffffffffu;
  const int L = tid & 31, wid = tid >> 5, lane = L & (GLF - 1);
  constexpr uint32_t ROWS = XROWS * W / 32;
  sx += (L / W) * ROWS;
  real4* __restrict__ sv = sx + XROWS;
  const double inv = P->inv_cell;
  const real H = P->fluid_h, H2 = H * H;
  const real4* __restrict__ rows = v.pvrow;
  const uint32_t NS = (uint32_t)v.N;
  const real allow = xsph_allowance(P), rec = XMOVE_REC * allow;
  const real scene = r_fmax(rec, (real)__uint_as_float(v.scratch[SCR_XMOVE]));
  for (uint32_t c = (uint32_t)wid; c < chunks; c = next_chunk(s_list, c, L)) {
    bool mem;
    const uint32_t myslot = chunk_slot<W>(v, s_list, c, L, first, halves, mem);
    const uint32_t i = v.entries[myslot];
    const real4 pi = rows[2 * (size_t)myslot];
    const real sm = v.smove[myslot];
    uint32_t cnt = v.ncount[(size_t)lane * NS + myslot];
    const bool act = mem && (v.flags[i] & F_ACTIVE);
    // the list test: the particle kept its cell (smove finite), it and every
    // particle of its 27 buckets moved within the allowance, and no lane's list
    // overflowed. The scene's largest recorded movement bounds every bucket's,
    // so when it passes the buckets are not looked at.
    const unsigned full = __ballot_sync(FULL, cnt > NL);
    const bool over = (full >> (L & ~(GLF - 1)) & ((1u << GLF) - 1u)) != 0u;
    bool listed = act && !over && sm + scene <= allow;
    real sx_ = 0.f, sy_ = 0.f, sz_ = 0.f, m = 0.f;
    unsigned rem = __ballot_sync(FULL, act && !listed);
    if (rem) {
      rem &= part_lanes<W>(L);
      const double ca = floor(__dmul_rn((double)(lane == 0 ? pi.x : (lane == 1 ? pi.y : pi.z)), inv));
      do {
        const bool work = W == 32 || rem != 0u;
      const int ll = work ? __ffs((int)rem) - 1 : L & ~(W - 1);
        const unsigned turn = same_cell<W>(ca, ll, lane) & rem;
        rem &= ~turn;
        const bool mine_turn = (turn >> L & 1u) != 0u;
        uint32_t bm = 0;  // the buckets' fluid: a finite distance or +inf
        Buckets<W> b;
        const uint32_t total = part_buckets<W>(v, ca, ll, L, work, b, [&](uint32_t n, uint32_t hb) {
          const uint32_t moved = v.bmove[hb];
          if (n) bm = max(bm, moved);
        });
        const uint32_t most = longest<W>(total);
        if (W == 32) {
          bm = __reduce_max_sync(FULL, bm);
        } else {
#pragma unroll
          for (int o = 1; o < W; o <<= 1) bm = max(bm, __shfl_xor_sync(FULL, bm, o));
        }
        if (mine_turn) listed = !over && sm + r_fmax(rec, (real)__uint_as_float(bm)) <= allow;
        const bool walks = mine_turn && !listed;
        if (!__any_sync(FULL, walks)) continue;
        for (uint32_t q0 = 0; q0 < most; q0 += ROWS) {
          auto copy = [&](uint32_t k, uint32_t e) {
            if (UPBD_IDX_OK(v, e, NS)) {
              copy_row_async(&sx[k], &rows[2 * (size_t)e]);
              copy_row_async(&sv[k], &rows[2 * (size_t)e + 1]);
            } else {
              sx[k] = make_real4(__int_as_float(0x7f800000), 0.f, 0.f, 0.f);  // never in range (reported)
            }
          };
          if (most <= ROWS) stage_rows<W, ROWS, false>(L, b, 0u, copy);
          else stage_rows<W, ROWS, true>(L, b, q0, copy);
          copy_rows_wait();
          __syncwarp();
          const uint32_t len = (W == 32 || q0 < total) ? min(total - q0, ROWS) : 0u;
          const uint32_t own = walks ? (len + (GLF - 1) - lane) / GLF : 0u;  // this lane's share, at most 32
          const uint32_t steps = (len + (GLF - 1)) / GLF;
          uint32_t bits = 0;  // within H, the first candidate's bit on top
          const real4* __restrict__ r4 = sx + lane;
          for (uint32_t u = 0; u < steps; u += 4, r4 += 4 * GLF) {  // reads past the share stay in the warp's rows
#pragma unroll
            for (int k = 0; k < 4; k++) {
              const real4 pj = r4[k * GLF];
              const bool in = slot_unpack(pj.w) != myslot && dist2(pj.x - pi.x, pj.y - pi.y, pj.z - pi.z) < H2;
              bits = (bits << 1) | (in ? 1u : 0u);
            }
          }
          bits <<= (32u - ((steps + 3u) & ~3u)) & 31u;
          if (own < 32u) bits &= ~(0xffffffffu >> own);
          while (bits) {
            const int k = __clz((int)bits);
            bits &= ~(0x80000000u >> k);
            const real4 w = sv[lane + k * GLF];
            sx_ = sx_ + w.x; sy_ = sy_ + w.y; sz_ = sz_ + w.z;
            m = m + 1.0f;
          }
          __syncwarp();  // the next round rewrites the rows
        }
      } while (parts_left<W>(rem));
    }
    if (listed) {
      uint32_t* const nbr = list_entry(v.nbr + myslot, lane * NL, NS);
      for (uint32_t k = 0; k < cnt; k += XCH) {
        uint32_t e[XCH];
        real4 p[XCH], w[XCH];
#pragma unroll
        for (int q = 0; q < XCH; q++) {
          e[q] = (k + q < cnt) ? (__ldg(list_entry(nbr, k + q, NS)) & ~NBR_IN) : myslot;
          if (!UPBD_IDX_OK(v, e[q], NS)) e[q] = myslot;  // out of range: the own slot (skipped, reported)
        }
#pragma unroll
        for (int q = 0; q < XCH; q++) load_row_pair(&rows[2 * (size_t)e[q]], p[q], w[q]);
#pragma unroll
        for (int q = 0; q < XCH; q++) {
          const bool in = e[q] != myslot && dist2(p[q].x - pi.x, p[q].y - pi.y, p[q].z - pi.z) < H2;
          sx_ = sx_ + (in ? w[q].x : 0.f); sy_ = sy_ + (in ? w[q].y : 0.f); sz_ = sz_ + (in ? w[q].z : 0.f);
          m = m + (in ? 1.0f : 0.f);
        }
      }
    }
    sx_ = lane_sum<GLF>(sx_);
    sy_ = lane_sum<GLF>(sy_);
    sz_ = lane_sum<GLF>(sz_);
    m = lane_sum<GLF>(m);
    if (act && lane == 0) {
      const real4 vi = v.vel[i];
      real vx = vi.x, vy = vi.y, vz = vi.z;
      if (m > 0.f) {
        const real mu = P->viscosity;
        vx = vx + mu * (sx_ / m - vx);
        vy = vy + mu * (sy_ / m - vy);
        vz = vz + mu * (sz_ / m - vz);
      }
      if (APPLY)
        v.vel[i] = make_real4(vx, vy, vz, 0.f);
      else
        v.delta[i] = make_real4(vx, vy, vz, m);
    }
  }
}
template <bool APPLY>
__device__ __forceinline__ void b_xsph(const SimView& v, const DevParams* __restrict__ P, uint32_t window, uint32_t vb) {
  extern __shared__ __align__(16) unsigned char s_stage[];
  __shared__ ChunkList s_list;
  const int tid = thread_index();
  const uint32_t nact = active_slots(v), first = vb * window;
  if (first >= nact) return;
  uint32_t halves;
  const uint32_t chunks = list_chunks(v, s_list, first, window, nact, tid, halves);
  real4* sx = reinterpret_cast<real4*>(s_stage + (tid >> 5) * STAGE_WARP);
  if (halves) xsph_chunks<APPLY, 16>(v, P, s_list, sx, first, chunks, halves, tid);
  else xsph_chunks<APPLY, 32>(v, P, s_list, sx, first, chunks, halves, tid);
}

// countActive (src/gpu/wgsl.js:874-879) with a last-block epilogue that
// publishes the count and the health bits to mapped host memory.
__device__ __forceinline__ void b_count_active(const SimView& v, uint32_t vb, uint32_t nblk) {
  const int i = v.S + (int)UPBD_VTID;
  uint32_t a = (i < v.N && (v.flags[i] & F_ACTIVE)) ? 1u : 0u;
  a = __reduce_add_sync(0xffffffffu, a);
  __shared__ uint32_t s_sum;
  if (threadIdx.x == 0) s_sum = 0;
  __syncthreads();
  if ((threadIdx.x & 31) == 0 && a) atomicAdd(&s_sum, a);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_sum) atomicAdd(&v.scratch[SCR_ACTIVE], s_sum);
    __threadfence();
    const uint32_t done = atomicAdd(&v.scratch[SCR_DONE], 1u);
    if (done == nblk - 1u) {
      __threadfence();
      const uint32_t total = atomicExch(&v.scratch[SCR_ACTIVE], 0u);
      v.scratch[SCR_DONE] = 0u;
      volatile uint32_t* hm = v.host_mapped;
      hm[HM_ACTIVE] = total;
      hm[HM_HEALTH] = atomicOr(&v.scratch[SCR_HEALTH], 0u);
    }
  }
}

}  // namespace upbd
