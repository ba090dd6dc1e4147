// Single-scene sm_100a kernels of libupbd: the per-pass wrappers around the
// pass bodies of upbd_passes.cuh, and the tool kernels (emit, wedge cut,
// pick, grab, drain) that run on demand.
#pragma once
#include "upbd_passes.cuh"

namespace upbd {

#define UPBD_TID (blockIdx.x * blockDim.x + threadIdx.x)

// ------------------------------------------------------------------ emit
// emit, src/gpu/wgsl.js:781-801 (hose ring buffer)
__global__ void __launch_bounds__(64) k_emit(SimView v, const DevParams* __restrict__ P) {
  const uint32_t k = UPBD_TID;
  if (k >= P->emit_count) return;
  const int slot = v.S + (int)((P->emit_start + k) % (uint32_t)v.F);
  const float4 E_pos = P->emit_pos, E_dir = P->emit_dir, E_side = P->emit_side, E_up = P->emit_up;
  const real phase = E_dir.w + (real)k * 2.39996f;
  const real spacing = P->fluid_radius * 2.2f;
  const real fk = (real)k * 0.618034f;
  const real rad = spacing * (0.4f + 1.6f * (fk - floorf(fk)));
  const real c = cosf(phase), s = sinf(phase);
  const real along = (real)(k % 8u) * spacing * 0.5f;
  const real offx = E_side.x * (c * rad) + E_up.x * (s * rad) + E_dir.x * along;
  const real offy = E_side.y * (c * rad) + E_up.y * (s * rad) + E_dir.y * along;
  const real offz = E_side.z * (c * rad) + E_up.z * (s * rad) + E_dir.z * along;
  const real px = E_pos.x + offx, py = E_pos.y + offy, pz = E_pos.z + offz;
  const real a = sinf(phase * 12.9898f) * 43758.547f;
  const real b = sinf(phase * 78.233f) * 12543.123f;
  const real d = sinf(phase * 39.425f) * 26781.897f;
  const real jx = ((a - floorf(a)) - 0.5f) * 0.5f;
  const real jy = ((b - floorf(b)) - 0.5f) * 0.5f;
  const real jz = ((d - floorf(d)) - 0.5f) * 0.5f;
  const real speed = E_pos.w;
  const real w = v.pos[slot].w;
  v.pos[slot] = make_real4(px, py, pz, w);
  v.prev[slot] = make_real4(px, py, pz, 0.f);
  v.vel[slot] = make_real4(E_dir.x * speed + jx, E_dir.y * speed + jy, E_dir.z * speed + jz, 0.f);
  v.flags[slot] = F_ACTIVE;
}

// Solver.emitFluid for a batch, src/solver.js:139-149 (ring buffer).
__global__ void k_emit_particles(SimView v, const float* __restrict__ p3,
                                 const float* __restrict__ v3, int n, int start, float inv_mass) {
  const int k = UPBD_TID;
  if (k >= n) return;
  const int slot = v.S + (int)(((long long)start + k) % v.F);
  const real x = p3[3 * k], y = p3[3 * k + 1], z = p3[3 * k + 2];
  v.pos[slot] = make_real4(x, y, z, inv_mass);
  v.prev[slot] = make_real4(x, y, z, 0.f);
  v.vel[slot] = make_real4(v3[3 * k], v3[3 * k + 1], v3[3 * k + 2], 0.f);
  v.flags[slot] = F_ACTIVE;
}

// ------------------------------------------------- single-scene kernels
// One launch per pass over one scene: tile vb = blockIdx.x.
template <bool INTEGRATE, bool COUNT>
__global__ void __launch_bounds__(256) k_integrate_count(SimView v, const DevParams* __restrict__ P) {
  b_integrate_count<INTEGRATE, COUNT>(v, P, blockIdx.x);
}
__global__ void __launch_bounds__(SCAN_THREADS) k_scan(SimView v) { b_scan(v, blockIdx.x); }
// the stateless grid build's forms: the cell size in the arguments, the bucket
// counts written by the scan that reads them. The count alone reads the caller's
// flags: the passes after it go by the buckets it wrote.
__global__ void __launch_bounds__(256) k_grid_count(SimView v, double inv_cell) {
  const int i = UPBD_TID;
  if (i >= v.N) return;
  if (v.flags[i] & F_ACTIVE) count_particle(v, inv_cell, i, v.pos[i]);
  else v.cell[i] = CELL_NONE;
}
template <bool COUNTS>
__global__ void __launch_bounds__(SCAN_THREADS) k_grid_scan(SimView v, uint32_t* counts) {
  b_scan<COUNTS, false>(v, blockIdx.x, counts);
}
__global__ void __launch_bounds__(256) k_grid_scatter(SimView v) { b_scatter<false>(v, blockIdx.x); }
__global__ void __launch_bounds__(256) k_grid_rankfix(SimView v) { b_rankfix<false>(v, blockIdx.x); }
// the first words of n bucket rows
__global__ void __launch_bounds__(256) k_bucket_starts(const uint2* __restrict__ rows, uint32_t* __restrict__ out, int n) {
  const int h = UPBD_TID;
  if (h < n) out[h] = rows[h].x;
}
__global__ void __launch_bounds__(256) k_scatter(SimView v) { b_scatter(v, blockIdx.x); }
__global__ void __launch_bounds__(256) k_rankfix(SimView v) { b_rankfix(v, blockIdx.x); }
// 5 CTAs of 256 per SM: 48 registers (with 6 and 40 a launch took 3 % longer)
__global__ void __launch_bounds__(256, 5) k_density(SimView v, const DevParams* __restrict__ P, uint32_t window) {
  b_density(v, P, window, blockIdx.x);
}
template <bool APPLY>
__global__ void __launch_bounds__(256) k_disp(SimView v, const DevParams* __restrict__ P) {
  b_disp<APPLY>(v, P, blockIdx.x);
}
__global__ void __launch_bounds__(256) k_apply_fluid(SimView v, const DevParams* __restrict__ P) {
  b_apply_fluid(v, P, blockIdx.x);
}
template <bool APPLY_FLUID, int OUT>
__global__ void __launch_bounds__(256) k_solid_solve(SimView v, const DevParams* __restrict__ P, int solid_pad, int q) {
  b_solid_solve<APPLY_FLUID, OUT, 4>(v, P, solid_pad, q, blockIdx.x);
}
__global__ void __launch_bounds__(256) k_apply_solid(SimView v, const DevParams* __restrict__ P) {
  b_apply_solid(v, P, blockIdx.x);
}
template <int G, bool FROM_GRID = false>
__global__ void __launch_bounds__(256) k_contact_mark(SimView v, const DevParams* __restrict__ P) {
  b_contact_mark<G, FROM_GRID>(v, P, blockIdx.x);
}
__global__ void __launch_bounds__(256) k_collect_contacts(SimView v, const DevParams* __restrict__ P) {
  b_collect_contacts(v, P, blockIdx.x);
}
template <bool LAST>
__global__ void __launch_bounds__(256) k_solid_contacts(SimView v, const DevParams* __restrict__ P, int q) {
  b_solid_contacts<LAST>(v, P, q, blockIdx.x);
}
template <bool LAST, int G>
__global__ void __launch_bounds__(256) k_solve_tets(SimView v, const DevParams* __restrict__ P, int q) {
  b_solve_tets<LAST, G>(v, P, q, blockIdx.x);
}
__global__ void __launch_bounds__(256) k_bond_contacts(SimView v, const DevParams* __restrict__ P, int nb, int nt,
                                                       int nb_pad, int nc) {
  b_bond_contacts(v, P, nb, nt, nb_pad, nc, blockIdx.x);
}
__global__ void __launch_bounds__(256) k_apply_bounds_vel(SimView v, const DevParams* __restrict__ P, int stage) {
  b_apply_bounds_vel(v, P, stage, blockIdx.x);
}
__global__ void __launch_bounds__(256) k_solid_visc(SimView v, const DevParams* __restrict__ P) {
  b_solid_visc(v, P, blockIdx.x);
}
__global__ void __launch_bounds__(256) k_solid_visc_apply(SimView v) { b_solid_visc_apply(v, blockIdx.x); }
// 4 CTAs of 256 per SM: four list entries in flight without spills (5 CTAs and
// 48 registers: a seventh longer on the default scene)
template <bool APPLY>
__global__ void __launch_bounds__(256, 4) k_xsph(SimView v, const DevParams* __restrict__ P, uint32_t window) {
  b_xsph<APPLY>(v, P, window, blockIdx.x);
}
__global__ void __launch_bounds__(256) k_count_active(SimView v) { b_count_active(v, blockIdx.x, gridDim.x); }

// ------------------------------------------------------------------ tools
// Wedge cut over the constraint buffer (kernel shape of src/gpu/wgsl.js:804-823)
// with the double-precision arithmetic of Solver.cut, src/solver.js:458-486.
// Every operation is an explicit round-to-nearest intrinsic so no multiply-add
// is fused and the alive flags match the CPU solver bit for bit.
__global__ void __launch_bounds__(256) k_cut(SimView v, const DevParams* __restrict__ P) {
  const int c = UPBD_TID;
  if (c >= v.C) return;
  const uint4 cc = v.cons[c];
  if (cc.w == 0u) return;
  const double ox = P->cut_o[0], oy = P->cut_o[1], oz = P->cut_o[2];
  const double d1x = P->cut_d1[0], d1y = P->cut_d1[1], d1z = P->cut_d1[2];
  const double d2x = P->cut_d2[0], d2y = P->cut_d2[1], d2z = P->cut_d2[2];
  const double nx = __dsub_rn(__dmul_rn(d1y, d2z), __dmul_rn(d1z, d2y));
  const double ny = __dsub_rn(__dmul_rn(d1z, d2x), __dmul_rn(d1x, d2z));
  const double nz = __dsub_rn(__dmul_rn(d1x, d2y), __dmul_rn(d1y, d2x));
  const double nl = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(nx, nx), __dmul_rn(ny, ny)), __dmul_rn(nz, nz)));
  if (nl < 1e-8) return;
  if (!UPBD_IDX_OK(v, cc.x, v.S) || !UPBD_IDX_OK(v, cc.y, v.S)) return;
  const real4 A = v.pos[cc.x], B = v.pos[cc.y];
  const double ax = A.x, ay = A.y, az = A.z, bx = B.x, by = B.y, bz = B.z;
  const double sa = __dadd_rn(__dadd_rn(__dmul_rn(__dsub_rn(ax, ox), nx), __dmul_rn(__dsub_rn(ay, oy), ny)),
                              __dmul_rn(__dsub_rn(az, oz), nz));
  const double sb = __dadd_rn(__dadd_rn(__dmul_rn(__dsub_rn(bx, ox), nx), __dmul_rn(__dsub_rn(by, oy), ny)),
                              __dmul_rn(__dsub_rn(bz, oz), nz));
  if (__dmul_rn(sa, sb) >= 0.0) return;
  const double t = __ddiv_rn(sa, __dsub_rn(sa, sb));
  const double px = __dsub_rn(__dadd_rn(ax, __dmul_rn(__dsub_rn(bx, ax), t)), ox);
  const double py = __dsub_rn(__dadd_rn(ay, __dmul_rn(__dsub_rn(by, ay), t)), oy);
  const double pz = __dsub_rn(__dadd_rn(az, __dmul_rn(__dsub_rn(bz, az), t)), oz);
  const double c1 = __dadd_rn(__dadd_rn(__dmul_rn(__dsub_rn(__dmul_rn(d1y, pz), __dmul_rn(d1z, py)), nx),
                                        __dmul_rn(__dsub_rn(__dmul_rn(d1z, px), __dmul_rn(d1x, pz)), ny)),
                              __dmul_rn(__dsub_rn(__dmul_rn(d1x, py), __dmul_rn(d1y, px)), nz));
  const double c2 = __dadd_rn(__dadd_rn(__dmul_rn(__dsub_rn(__dmul_rn(py, d2z), __dmul_rn(pz, d2y)), nx),
                                        __dmul_rn(__dsub_rn(__dmul_rn(pz, d2x), __dmul_rn(px, d2z)), ny)),
                              __dmul_rn(__dsub_rn(__dmul_rn(px, d2y), __dmul_rn(py, d2x)), nz));
  if (c1 < 0.0 || c2 < 0.0) return;
  v.cons[c].w = 0u;
  atomicAdd(&v.scratch[SCR_CUT], 1u);
}

// cutTets, src/gpu/wgsl.js:494-519 (f32 wedge, as the reference kernel)
__global__ void __launch_bounds__(256) k_cut_tets(SimView v, const DevParams* __restrict__ P) {
  const int t = UPBD_TID;
  if (t >= v.NT) return;
  const real V0 = v.tet_vol[t];
  if (V0 <= 0.f) return;
  const real ox = (real)P->cut_o[0], oy = (real)P->cut_o[1], oz = (real)P->cut_o[2];
  const real ax1 = (real)P->cut_d1[0], ay1 = (real)P->cut_d1[1], az1 = (real)P->cut_d1[2];
  const real ax2 = (real)P->cut_d2[0], ay2 = (real)P->cut_d2[1], az2 = (real)P->cut_d2[2];
  real nx, ny, nz;
  cross3(ax1, ay1, az1, ax2, ay2, az2, nx, ny, nz);
  if (dot3(nx, ny, nz, nx, ny, nz) < 1e-16f) return;
  for (int p = 0; p < 3; p++)
    for (int q = p + 1; q < 4; q++) {
      const uint32_t ta = v.tet_idx[4 * t + p], tb = v.tet_idx[4 * t + q];
      if (!UPBD_IDX_OK(v, ta, v.S) || !UPBD_IDX_OK(v, tb, v.S)) return;
      const real4 A = v.pos[ta];
      const real4 B = v.pos[tb];
      const real pax = A.x - ox, pay = A.y - oy, paz = A.z - oz;
      const real pbx = B.x - ox, pby = B.y - oy, pbz = B.z - oz;
      const real sa = dot3(pax, pay, paz, nx, ny, nz);
      const real sb = dot3(pbx, pby, pbz, nx, ny, nz);
      if (sa * sb >= 0.f) continue;
      const real tt = sa / (sa - sb);
      const real ppx = pax + (pbx - pax) * tt, ppy = pay + (pby - pay) * tt, ppz = paz + (pbz - paz) * tt;
      real cx, cy, cz;
      cross3(ax1, ay1, az1, ppx, ppy, ppz, cx, cy, cz);
      if (dot3(cx, cy, cz, nx, ny, nz) < 0.f) continue;
      cross3(ppx, ppy, ppz, ax2, ay2, az2, cx, cy, cz);
      if (dot3(cx, cy, cz, nx, ny, nz) < 0.f) continue;
      v.tet_vol[t] = -V0;
      return;
    }
}

// Pick: smallest t (Solver.pickSolid, src/solver.js:502-515, in double), the
// lowest index among the particles at it. t >= 0 and never -0, so its IEEE bits
// order like unsigned integers. One launch with the ray in its arguments: each block
// leaves its best (t, index) in parts, the last one to finish reduces those
// into mapped host memory. The call is all latency: with the ray copied to the
// uniform block, a memset, two launches (smallest t, then lowest index) and a
// copy back it took 29.3 us on 8,000 solids (B200, host clock, through the Python
// mirror), this takes 16.2: the host watches the call's number arrive instead of
// waiting for the stream (18.7).
struct PickRay {
  double o[3], d[3], max_perp;
};
struct PickBest {
  unsigned long long t;
  uint32_t i;
};

__device__ __forceinline__ bool pick_t(const SimView& v, const PickRay& ray, int i, double& t) {
  if (!(v.flags[i] & F_ACTIVE)) return false;
  const real4 p = v.pos[i];
  const double mp = ray.max_perp;
  const double dx = ray.d[0], dy = ray.d[1], dz = ray.d[2];
  const double px = __dsub_rn((double)p.x, ray.o[0]), py = __dsub_rn((double)p.y, ray.o[1]),
               pz = __dsub_rn((double)p.z, ray.o[2]);
  t = __dadd_rn(__dadd_rn(__dmul_rn(px, dx), __dmul_rn(py, dy)), __dmul_rn(pz, dz));
  if (!(t >= 0.0)) return false;
  t = __dadd_rn(t, 0.0);  // -0 (a particle at the origin of the ray) becomes +0
  const double qx = __dsub_rn(px, __dmul_rn(dx, t)), qy = __dsub_rn(py, __dmul_rn(dy, t)),
               qz = __dsub_rn(pz, __dmul_rn(dz, t));
  const double q2 = __dadd_rn(__dadd_rn(__dmul_rn(qx, qx), __dmul_rn(qy, qy)), __dmul_rn(qz, qz));
  if (q2 > __dmul_rn(mp, mp)) return false;
  return true;
}

__device__ __forceinline__ void pick_better(PickBest& a, unsigned long long t, uint32_t i) {
  if (t < a.t || (t == a.t && i < a.i)) {
    a.t = t;
    a.i = i;
  }
}

// the block's best in thread 0 (256 threads)
__device__ __forceinline__ PickBest pick_block(PickBest b) {
  __shared__ PickBest s_best[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    pick_better(b, __shfl_down_sync(0xffffffffu, b.t, o), __shfl_down_sync(0xffffffffu, b.i, o));
  __syncthreads();  // an earlier call's reads
  if ((threadIdx.x & 31) == 0) s_best[threadIdx.x >> 5] = b;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < 8; w++) pick_better(b, s_best[w].t, s_best[w].i);
  return b;
}

__global__ void __launch_bounds__(256) k_pick(SimView v, PickRay ray, PickBest* parts, uint32_t call) {
  __shared__ bool s_last;
  PickBest b{~0ull, 0xffffffffu};
  for (long long i = UPBD_TID; i < v.S; i += (long long)gridDim.x * 256) {
    double t;
    if (pick_t(v, ray, (int)i, t)) pick_better(b, (unsigned long long)__double_as_longlong(t), (uint32_t)i);
  }
  b = pick_block(b);
  if (threadIdx.x == 0) {
    parts[blockIdx.x] = b;
    __threadfence();
    s_last = atomicAdd(&v.scratch[SCR_PICK], 1u) == gridDim.x - 1u;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  b = PickBest{~0ull, 0xffffffffu};
  for (uint32_t k = threadIdx.x; k < gridDim.x; k += 256) {
    const volatile PickBest* q = parts + k;
    pick_better(b, q->t, q->i);
  }
  b = pick_block(b);
  if (threadIdx.x == 0) {
    v.scratch[SCR_PICK] = 0u;
    volatile uint32_t* hm = v.host_mapped;
    hm[HM_PICK_T] = (uint32_t)b.t;
    hm[HM_PICK_T + 1] = (uint32_t)(b.t >> 32);
    hm[HM_PICK_I] = b.i;
    __threadfence_system();  // the result, then the word the host waits for
    hm[HM_PICK_CALL] = call;
  }
}

// grabSelect, src/gpu/wgsl.js:843-865
__global__ void __launch_bounds__(256) k_grab_select(SimView v, const DevParams* __restrict__ P) {
  const int i = UPBD_TID;
  if (i >= v.S) return;
  uint32_t f = v.flags[i];
  if (!(f & F_ACTIVE)) return;
  const uint32_t lat = (i >= v.N1) ? 1u : 0u;
  if (P->grab_lattice != 0xffffu && lat != P->grab_lattice) return;
  const float4 c = P->grab_c;
  const real4 p = v.pos[i];
  const real dx = p.x - c.x, dy = p.y - c.y, dz = p.z - c.z;
  const real q2 = dot3(dx, dy, dz, dx, dy, dz) / (c.w * c.w);
  if (q2 < 1.0f) {
    v.flags[i] = f | F_GRABBED;
    const real w = (1.0f - q2) * (1.0f - q2) * 0.95f + 0.05f;
    v.prev[i].w = p.x;
    v.vel[i].w = p.y;
    v.density[i] = make_real2(p.z, w);
  }
}

// Explicit-list grab: spring target given or at the current position.
__global__ void k_grab_indices(SimView v, const uint32_t* __restrict__ idx, const float* __restrict__ w,
                               const float* __restrict__ t3, int n) {
  const int k = UPBD_TID;
  if (k >= n) return;
  const uint32_t i = idx[k];
  if (i >= (uint32_t)v.S) return;
  const uint32_t f = v.flags[i];
  if (!(f & F_ACTIVE)) return;
  const real4 p = v.pos[i];
  const real tx = t3 ? t3[3 * k] : p.x, ty = t3 ? t3[3 * k + 1] : p.y, tz = t3 ? t3[3 * k + 2] : p.z;
  v.flags[i] = f | F_GRABBED;
  v.prev[i].w = tx;
  v.vel[i].w = ty;
  v.density[i] = make_real2(tz, w ? w[k] : 1.0f);
}

// grabRelease, src/gpu/wgsl.js:867-871
__global__ void k_grab_release(SimView v) {
  const int i = UPBD_TID;
  if (i < v.S) v.flags[i] &= ~F_GRABBED;
}

// GpuSim.clearFluid, src/gpu/sim.js:294-297
// the body of every kernel node in upbd_profile_graph_floor's copy of a frame
__global__ void k_empty() {}

__global__ void k_drain(SimView v) {
  const int i = v.S + (int)UPBD_TID;
  if (i < v.N) v.flags[i] = 0u;
}

}  // namespace upbd
