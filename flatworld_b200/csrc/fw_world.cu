// fw_world.cu -- C ABI (include/fwb200.h) and the general ("gather") step of
// the explicit 2D FEM world: any number of scenes, bodies and contact pairs.
//
// Per substep two kernels run on the context stream:
//   k_elements  one thread per triangle: deformation gradient, PK2 stress
//               (elastic / NeoHookean / J2 radial return), the three corner
//               forces -(B^T S)A written to a corner buffer kept in node
//               order (each corner at its place in its node's ascending-
//               element list, so a node reads one contiguous run).  Block 0 first
//               runs the per-step control (scene modes, broad-phase gates,
//               step counters, AABB slot reset).
//   k_nodes     one thread per node: penalty contact (boundary nodes only),
//               the node's corner forces summed in ascending element order,
//               boundary conditions, symplectic Euler, and the per-body AABB of
//               boundary nodes (warp reduction + ordered-int atomics).
// Summing a node's corners in ascending element order after its contact terms
// is exactly the order in which the reference's serial CPU path applies its
// atomic adds (flatworld/mixedcontact.py:1654-1755 then
// flatworld/femspringmanager.py:217-280), so the sum is deterministic and
// identical run to run, with no float atomics.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <map>
#include <mutex>
#include <cstdio>
#include <cstring>
#include <exception>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "../../include/fwb200.h"
#include "fw_device.cuh"
#include "fw_rigid.cuh"
#include "fw_adjoint.cuh"

using fw::ElemMat;
using fw::Pair;
using fw::Rigid;

namespace {

constexpr int kBlock = 256;     // default block size of the gather kernels
constexpr int kMaxBlock = 512;  // launch bound (block sizes are a runtime option)
constexpr int kGraphSteps = 32;
// Nodes of a served scene's cluster patch: latency before throughput, up to a
// point.  128 / 256 / 512: 48 requests of 100 to 4000 nodes 3.44 / 3.13 / 2.92 ms,
// 8 such 1.33 / 1.42 / 1.72, 16 of 100 to 1000 nodes 1.49 / 1.69 / 1.76.
constexpr int kCluServedNodes = 256;
constexpr size_t kCluSharedBytes = 232448 - 64;  // of a CTA on sm_100

// Substeps of a call from which a stream world's scenes are stepped on chip: a
// patch is loaded and written once per call, which costs as much as that many
// substeps gain, and gain less the more patches share an SM.  One call of ragged
// bodies, on chip / stream kernels, us: 109,000 triangles 3 substeps 43 / 53;
// 517,000 4: 99 / 94, 5: 110 / 113; 959,000 5: 175 / 177; 1,732,000 6: 340 / 332,
// 8: 399 / 437; 3,674,000 6: 678 / 622, 8: 801 / 824.  A substep more where the
// scenes' wide clusters (8 CTAs and more: an SM for each) do not run all at once
// and each load is waited for twice: 3 substeps of 16 scenes of 3200 triangles 60
// / 47, 4: 59 / 55; of 8 scenes of 7200 triangles 3: 46 / 44, 4: 47 / 55.
int clu_min_steps(int sms, int64_t triangles, int64_t wide_ctas) {
  return triangles <= (int64_t)sms * 1500 ? (wide_ctas > sms ? 4 : 3) : triangles <= (int64_t)sms * 6500 ? 5 : 8;
}
constexpr int kCluWide = 8;

// ... and of an arena, whose patches are smaller (kCluServedNodes: latency before
// throughput), so that its scenes take more CTAs, and whose launches are put
// together on the host for each call.  One call, on chip / stream kernels, us:
// wide clusters of 1.7 CTAs an SM, 3 substeps 75 / 74, 6: 91 / 104; of 2.6, 6: 117 /
// 111, 8: 133 / 141; of 5.1, 8: 223 / 207, 12: 286 / 298; of 6.9 (scenes of 16,200
// triangles), 12: 423 / 387, 16: 532 / 511, 24: 730 / 756; of 27, 16: 1623 /
// 1622; of 32, 16: 2140 / 1910, 50: 5550 / 5870; 512 scenes of 200 triangles, 4: 87 / 62, 6: 90 / 85, 8: 99 / 106.
int arena_min_steps(int sms, int64_t triangles, int64_t wide_ctas, int64_t scenes) {
  const int wide = wide_ctas > 16 * (int64_t)sms ? 32 : wide_ctas > 4 * (int64_t)sms ? 16 : wide_ctas > 2 * (int64_t)sms ? 7 : 3;
  return std::max({clu_min_steps(sms, triangles, wide_ctas), wide, scenes > 2 * (int64_t)sms ? 6 : 3});
}

// The same for a single scene, whose shorter calls run on the gather kernels,
// two plain launches a substep instead of a cooperative one and the patches'
// loads.  A call and its synchronisation, on chip / gather, us: 2 substeps of
// 2048 triangles 30 / 23, of 131072 35 / 25, of 319200 42 / 31; 3 of 2048 29 / 31,
// 32768 33 / 32, 131072 41 / 33, 409600 53 / 46; 4 of 131072 41 / 43, 409600
// 53 / 58, 655360 72 / 78.  A call and a read of one node: 3 of 32768 37 / 40,
// 131072 42 / 41, 409600 53 / 52.
int grid_min_steps(int sms, int64_t triangles) { return triangles <= (int64_t)sms * 500 ? 3 : 4; }

struct Dev {
  float2* x;
  float2* x_alt;       // stream path: the other position buffer (swapped every substep)
  float2* v;
  float2* x0;
  float2* bcv;
  float2* corner;      // corner forces in node (CSR) order: node i's are corner[csr_off[i] .. csr_end[i])
  int32_t* corner_pos; // 3 per triangle: where corner (e, c) goes in corner[]
  uint32_t* node_word;
  float* mass;
  int32_t* csr_off;   // node i's corners are csr_slot[csr_off[i] .. csr_end[i]), ascending element
  int32_t* csr_end;
  int32_t* csr_slot;
  int32_t* conn;
  float4* jinv;
  ElemMat* emat;
  float2* body_lm;     // stream path: each body's Lame constants (its triangles share them)
  float2* j2par;
  float4* j2state;
  float4* j2_alt;      // stream path: the other J2 state buffer
  float* ndmass;
  int32_t* body_scene;
  int32_t* body_pair_off;
  int32_t* body_pair_cnt;
  Pair* pairs;
  int32_t* pair_active;
  float* heights;
  int8_t* occ;
  ushort4* vox;        // per voxel cell its nearest free cells (k_voxel_table); null: none
  float* scene_dt;
  float* scene_damp;
  int32_t* scene_counter;
  int32_t* scene_active;
  int32_t* scene_mode_req;
  int32_t* scene_mode;
  int32_t* scene_bad;  // set to 1 when a node of the scene gets a non-finite position or velocity
  // stream arenas (fw_step_served_budget): substeps each active scene may
  // still run in this call; a scene whose budget is spent sits the rest out
  // (null: no budgets)
  int32_t* scene_budget;
  // optional second segment: once scene_budget[s] is spent the scene runs
  // scene_budget_next[s] more substeps at scene_dt_next[s] (null: none)
  int32_t* scene_budget_next;
  float* scene_dt_next;
  int32_t* aabb_ring;  // [2][B][4] ordered ints
  int N, E, B, S, P;
  int has_j2;
  // uniform_dt != 0: every scene steps dt_uniform (kernel argument, baked into
  // the captured graph); otherwise scene_dt[] holds one dt per scene.
  int uniform_dt;
  float dt_uniform;
  // chunked launch (arena worlds): only these element / node ranges are stepped
  int use_chunks;
  int n_e_chunks, n_n_chunks;
  const int2* e_chunks;  // (first element, count <= element block size)
  const int2* n_chunks;  // (first node, count <= node block size)
  // FEM-FEM contact (fw_flex.cuh); flex_slot == nullptr when the world has none.
  // Node i (if flex_slot[i] >= 0) receives this substep's contact forces as
  // (work item, force) entries flex_item/flex_force[slot * kFlexListCap ..
  // + flex_cnt[slot]), which node_step adds in work-item order.
  int32_t* flex_slot;
  int32_t* flex_cnt;
  int32_t* flex_item;
  float2* flex_force;
  // FEM-rigid contact (fw_rigid.cuh); rig == nullptr when the world has none.
  // A rigid pair's work item for node i is ritem[pair.n0 + bslot[i]]
  // (bslot: the node's index in its body's boundary node list).
  Rigid* rig;
  float4* ritem;
  int32_t* bslot;
  // The work items are evaluated by the element step's trailing blocks
  // (their inputs are the substep's start state): rwork[it] = (pair, node),
  // rforce[it] = the force the item adds to its node (when ritem[it] is a
  // hit); the node step adds the gated ones in pair order.
  int2* rwork;
  float2* rforce;
  int n_ritems;
  // CFL monitor (cfl_ord == nullptr: off): per scene, the smallest current-
  // shape stable time 0.4 L / c of its triangles since the last read, as the
  // int bits of a non-negative float (int order = float order); body_cfl =
  // 0.4 / sqrt(E / rho) per body (0 for spring domains: not monitored).
  int32_t* cfl_ord;
  float* body_cfl;
  float one = 1.0f;  // fw::Packed2::one
};

}  // namespace


namespace {

// ------------------------------------------------------------------ kernels

// The gate of pair pr of a body whose box of the previous substep is r, in
// substep k of its scene.
__device__ __forceinline__ int gate_of(const Dev& d, const Pair& pr, const int* r, int k) {
  if (pr.kind == fw::PAIR_RIGID) {  // the rigid's current box; plain overlap when the loop skips the BVH
    const Rigid& g = d.rig[pr.table];
    return fw::box_gate(fw::ord2f(r[0]), fw::ord2f(r[1]), fw::ord2f(r[2]), fw::ord2f(r[3]), g.lb[0], g.lb[1], g.ub[0],
                        g.ub[1], pr.n1 ? 1 : k) ? 1 : 0;
  }
  if (pr.gate > 0) {  // a ground of a loop with a moving plane: its entry's current box
    const Rigid& g = d.rig[pr.gate - 1];
    return fw::box_gate(fw::ord2f(r[0]), fw::ord2f(r[1]), fw::ord2f(r[2]), fw::ord2f(r[3]), g.lb[0], g.lb[1], g.ub[0],
                        g.ub[1], k) ? 1 : 0;
  }
  return fw::pair_gate(pr, fw::ord2f(r[0]), fw::ord2f(r[1]), fw::ord2f(r[2]), fw::ord2f(r[3]), k) ? 1 : 0;
}

__device__ void step_control(const Dev& d) {
  const int t = threadIdx.x;
  for (int s = t; s < d.S; s += blockDim.x) {
    const int act = d.scene_active[s];
    const int req = d.scene_mode_req[s];
    d.scene_mode[s] = act ? (req ? fw::MODE_INIT : fw::MODE_STEP) : fw::MODE_FROZEN;
    if (act && req) d.scene_mode_req[s] = 0;
  }
  __syncthreads();
  for (int p = t; p < d.P; p += blockDim.x) {
    const Pair& pr = d.pairs[p];
    const int s = d.body_scene[pr.body];
    if (d.scene_mode[s] != fw::MODE_STEP) continue;
    const int k = d.scene_counter[s];
    d.pair_active[p] = gate_of(d, pr, d.aabb_ring + ((size_t)(k & 1) * d.B + pr.body) * 4, k);
  }
  __syncthreads();
  for (int s = t; s < d.S; s += blockDim.x)
    if (d.scene_mode[s] == fw::MODE_STEP) d.scene_counter[s] += 1;
  __syncthreads();
  for (int b = t; b < d.B; b += blockDim.x) {
    const int s = d.body_scene[b];
    if (d.scene_mode[s] == fw::MODE_FROZEN) continue;
    int* r = d.aabb_ring + ((size_t)(d.scene_counter[s] & 1) * d.B + b) * 4;
    r[0] = fw::f2ord(1e30f);
    r[1] = fw::f2ord(1e30f);
    r[2] = fw::f2ord(-1e30f);
    r[3] = fw::f2ord(-1e30f);
  }
}

// step_control for one scene whose bodies and pairs are the ranges rng (first
// body, bodies, first pair, pairs), by one block: nothing is looked up per body,
// and a few pairs' loads are in flight together.
__device__ void scene_control(const Dev& d, int s, int4 rng) {
  const int t = threadIdx.x, T = blockDim.x;
  const int act = d.scene_active[s], req = d.scene_mode_req[s], k = d.scene_counter[s];
  const int mode = act ? (req ? fw::MODE_INIT : fw::MODE_STEP) : fw::MODE_FROZEN;
  const bool step = mode == fw::MODE_STEP;
  __syncthreads();  // every thread has read them
  if (t == 0) {
    d.scene_mode[s] = mode;
    if (act && req) d.scene_mode_req[s] = 0;
    if (step) d.scene_counter[s] = k + 1;
  }
  if (mode == fw::MODE_FROZEN) return;
  if (step) {
    constexpr int U = 4;
    for (int p0 = rng.z + t; p0 < rng.z + rng.w; p0 += U * T) {
      Pair pr[U];
      int4 box[U];
#pragma unroll
      for (int u = 0; u < U; ++u) pr[u] = d.pairs[min(p0 + u * T, rng.z + rng.w - 1)];
#pragma unroll
      for (int u = 0; u < U; ++u)
        box[u] = *reinterpret_cast<const int4*>(d.aabb_ring + ((size_t)(k & 1) * d.B + pr[u].body) * 4);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (p0 + u * T < rng.z + rng.w) d.pair_active[p0 + u * T] = gate_of(d, pr[u], &box[u].x, k);
    }
  }
  const int k2 = step ? k + 1 : k;
  const int big = fw::f2ord(1e30f), low = fw::f2ord(-1e30f);
  for (int b = rng.x + t; b < rng.x + rng.y; b += T)
    *reinterpret_cast<int4*>(d.aabb_ring + ((size_t)(k2 & 1) * d.B + b) * 4) = make_int4(big, big, low, low);
}

// step_control for a list of scenes (stream arenas: the active scenes of the
// call), one thread per scene: the same four steps for that scene -- mode
// (and budget), its pairs' gates from the box of the previous substep, its
// counter, the reset of its bodies' next box slot -- in the same order.
// Budgets (fw_step_served_budget): a scene runs scene_budget[s] substeps at
// its dt, then scene_budget_next[s] at scene_dt_next[s], then sits out.
// rng[s] = (first body, bodies, first pair, pairs) of scene s.
__global__ void k_control_scenes(Dev d, const int32_t* __restrict__ list, int n, const int4* __restrict__ rng) {
  // the patch step that follows may start now: it gathers positions, which
  // this kernel does not touch, and waits for this kernel before reading what
  // it writes (griddepcontrol.wait)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int s = list[i];
  int act = d.scene_active[s];
  if (act && d.scene_budget) {
    const int left = d.scene_budget[s];
    if (left > 0) {
      d.scene_budget[s] = left - 1;
    } else {
      const int left2 = d.scene_budget_next ? d.scene_budget_next[s] : 0;
      if (left2 > 0) {  // the second segment: switch to its step size once
        if (left == 0) {
          d.scene_dt[s] = d.scene_dt_next[s];
          d.scene_budget[s] = -1;
        }
        d.scene_budget_next[s] = left2 - 1;
      } else {
        act = 0;
      }
    }
  }
  const int req = d.scene_mode_req[s];
  const int mode = act ? (req ? fw::MODE_INIT : fw::MODE_STEP) : fw::MODE_FROZEN;
  d.scene_mode[s] = mode;
  if (act && req) d.scene_mode_req[s] = 0;
  if (mode != fw::MODE_STEP && mode != fw::MODE_INIT) return;
  const int4 r = rng[s];
  if (mode == fw::MODE_STEP) {
    const int k = d.scene_counter[s];
    for (int p = r.z; p < r.z + r.w; ++p) {
      const Pair& pr = d.pairs[p];
      const int* box = d.aabb_ring + ((size_t)(k & 1) * d.B + pr.body) * 4;
      d.pair_active[p] = fw::pair_gate(pr, fw::ord2f(box[0]), fw::ord2f(box[1]), fw::ord2f(box[2]),
                                       fw::ord2f(box[3]), k) ? 1 : 0;
    }
    d.scene_counter[s] = k + 1;
  }
  const int k2 = d.scene_counter[s];
  for (int b = r.x; b < r.x + r.y; ++b) {
    int* box = d.aabb_ring + ((size_t)(k2 & 1) * d.B + b) * 4;
    box[0] = fw::f2ord(1e30f);
    box[1] = fw::f2ord(1e30f);
    box[2] = fw::f2ord(-1e30f);
    box[3] = fw::f2ord(-1e30f);
  }
}

// CFL monitor: the current-shape stable time of one triangle, the reference's
// 0.4 * L_min / sqrt(E / rho) (femdomain.py:24) on the shortest edge of the
// deformed triangle (coef = 0.4 / sqrt(E / rho) of its body).  Every step
// implementation evaluates it with these operations.
__device__ __forceinline__ float cfl_bound(float2 a, float2 b, float2 c, float coef) {
  const float l0 = (a.x - b.x) * (a.x - b.x) + (a.y - b.y) * (a.y - b.y);
  const float l1 = (b.x - c.x) * (b.x - c.x) + (b.y - c.y) * (b.y - c.y);
  const float l2 = (c.x - a.x) * (c.x - a.x) + (c.y - a.y) * (c.y - a.y);
  return sqrtf(fminf(l0, fminf(l1, l2))) * coef;
}

// Minimum over a whole warp (every lane present) of a non-negative float;
// +inf where no lane had a value.
__device__ __forceinline__ int warp_min_bits(float v) {
  return (int)__reduce_min_sync(0xFFFFFFFFu, (unsigned)__float_as_int(v));
}

// Loads that depend only on the triangle index are issued before the scene
// check, so the gather of corner positions does not wait for it.
__device__ __forceinline__ float element_step(const Dev& d, int e) {
  {
    const ElemMat m = d.emat[e];
    const int c0 = d.conn[3 * e], c1 = d.conn[3 * e + 1], c2 = d.conn[3 * e + 2];
    const float4 ji = d.jinv[e];
    const int q0 = d.corner_pos[3 * e], q1 = d.corner_pos[3 * e + 1], q2 = d.corner_pos[3 * e + 2];
    const float2 a = d.x[c0], b = d.x[c1], c = d.x[c2];
    const int s = d.body_scene[fw::elem_body(m.word)];
    if (!d.scene_active[s]) return __int_as_float(0x7f800000);
    if (fw::elem_type(m.word) == fw::MAT_SPRING) {  // _spring_force_kernel, femspringmanager.py:283-312
      const float2 va = d.v[c0], vb = d.v[c1];
      const float xx = a.x - b.x, xy = a.y - b.y;
      const float lnew = sqrtf(xx * xx + xy * xy);
      const float dx = xx / lnew, dy = xy / lnew;
      const float sc = m.lam * (lnew / m.area - 1.0f);  // stiffness x strain; area holds the rest length
      float fx = sc * dx, fy = sc * dy;
      const float vx = va.x - vb.x, vy = va.y - vb.y;
      const float dmp = m.mu * (vx * dx + vy * dy);  // mu holds the damping
      fx = fx + dmp * dx;
      fy = fy + dmp * dy;
      d.corner[q0] = make_float2(-fx, -fy);
      d.corner[q1] = make_float2(fx, fy);
      return __int_as_float(0x7f800000);
    }
    float4 j2 = make_float4(0.f, 0.f, 0.f, 0.f);
    float sy = 0.f, H = 0.f;
    const bool mises = fw::elem_type(m.word) == fw::MAT_MISES;
    if (mises) {
      j2 = d.j2state[e];
      const float2 q = d.j2par[e];
      sy = q.x;
      H = q.y;
    }
    float2 f1, f2, f3;
    fw::element_forces(fw::Scalar2{}, a, b, c, ji, m, sy, H, j2, f1, f2, f3);
    if (mises) d.j2state[e] = j2;
    d.corner[q0] = f1;
    d.corner[q1] = f2;
    d.corner[q2] = f3;
    if (!d.cfl_ord) return __int_as_float(0x7f800000);
    return cfl_bound(a, b, c, d.body_cfl[fw::elem_body(m.word)]);
  }
}

// Warp-shuffle minimum of the lanes' CFL bounds per scene (lanes of one warp
// can hold triangles of different scenes), one atomic per scene and warp.
__device__ __forceinline__ void cfl_reduce(const Dev& d, int e, float dtc) {
  const unsigned mask = __activemask();
  const int s = d.body_scene[fw::elem_body(d.emat[e].word)];
  const unsigned grp = __match_any_sync(mask, s);
  const int m = (int)__reduce_min_sync(grp, (unsigned)__float_as_int(dtc));
  if ((int)(threadIdx.x & 31) == __ffs(grp) - 1 && m < 0x7f800000) atomicMin(d.cfl_ord + s, m);
}

__global__ void __launch_bounds__(kMaxBlock) k_elements(Dev d) {
  const int nb = gridDim.x;
  if (blockIdx.x == 0) step_control(d);
  if (d.use_chunks) {
    for (int c = blockIdx.x; c < d.n_e_chunks; c += nb) {
      const int2 ch = d.e_chunks[c];
      if ((int)threadIdx.x < ch.y) {
        const float dtc = element_step(d, ch.x + threadIdx.x);
        if (d.cfl_ord) cfl_reduce(d, ch.x + threadIdx.x, dtc);
      }
    }
    return;
  }
  const int stride = nb * blockDim.x;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < d.E; e += stride) {
    const float dtc = element_step(d, e);
    if (d.cfl_ord) cfl_reduce(d, e, dtc);
  }
}

}  // namespace

#include "fw_flex.cuh"

namespace {

// Worlds with FEM-rigid contact: block 0 does the step control, blocks [1, eb]
// run the element step, the others evaluate every FEM-rigid work item -- one
// thread per item instead of one thread per boundary node walking all its rigid
// pairs -- from the substep's start state, whatever the gate and the scene's
// mode (the node step and the rigid sums use an item only when its scene steps
// and its pair is gated on).
// rigid_item adds its force to a -0 start, which leaves it exactly as it
// would be added to the node's sum.
__global__ void __launch_bounds__(kMaxBlock) k_elements_rigid(Dev d, int eb) {
  if (blockIdx.x == 0) {
    step_control(d);
    return;
  }
  const int b = blockIdx.x - 1;
  if (b < eb) {
    for (int e = b * blockDim.x + threadIdx.x; e < d.E; e += eb * blockDim.x) {
      const float dtc = element_step(d, e);
      if (d.cfl_ord) cfl_reduce(d, e, dtc);
    }
    return;
  }
  const int stride = (gridDim.x - 1 - eb) * blockDim.x;
  for (int it = (b - eb) * blockDim.x + threadIdx.x; it < d.n_ritems; it += stride) {
    const int2 w = d.rwork[it];
    const Pair& pr = d.pairs[w.x];
    const float dt = d.uniform_dt ? d.dt_uniform : d.scene_dt[d.body_scene[pr.body]];
    float2 f = make_float2(-0.0f, -0.0f);
    d.ritem[it] = fw::rigid_item(d.rig[pr.table], pr.table, pr.penalty, pr.f[0], pr.pad != 0, d.x[w.y], d.v[w.y],
                                 dt, f);
    d.rforce[it] = f;
  }
}

// This substep's FEM-FEM contact forces on one node: their number and the
// first four, loaded with the node's own state.
struct FlexList {
  int slot = -1, n = 0;
  int4 item;
  float4 f01, f23;
  __device__ __forceinline__ void load(const Dev& d, int i) {
    slot = d.flex_slot[i];
    if (slot < 0) return;
    n = min(d.flex_cnt[slot], kFlexListCap);
    if (n == 0) return;
    item = *reinterpret_cast<const int4*>(d.flex_item + slot * kFlexListCap);
    const float4* f = reinterpret_cast<const float4*>(d.flex_force + slot * kFlexListCap);
    f01 = f[0];
    f23 = f[1];
  }
};

// Adds them in work-item order (the reference adds them with atomic_add in
// launch order): the entries' item ids are distinct, so each pass adds the
// entry with the next larger id.  The list is emptied for the next substep.
__device__ __forceinline__ void flex_add(const Dev& d, const FlexList& l, float2& f) {
  if (l.n == 0) return;
  if (l.n <= 4) {
    int4 w = l.item;
    if (l.n < 4) w.w = 0x7FFFFFFF;
    if (l.n < 3) w.z = 0x7FFFFFFF;
    if (l.n < 2) w.y = 0x7FFFFFFF;
    for (int r = 0; r < l.n; ++r) {
      const int m = min(min(w.x, w.y), min(w.z, w.w));
      const float2 c = w.x == m   ? make_float2(l.f01.x, l.f01.y)
                       : w.y == m ? make_float2(l.f01.z, l.f01.w)
                       : w.z == m ? make_float2(l.f23.x, l.f23.y)
                                  : make_float2(l.f23.z, l.f23.w);
      if (w.x == m) w.x = 0x7FFFFFFF;
      if (w.y == m) w.y = 0x7FFFFFFF;
      if (w.z == m) w.z = 0x7FFFFFFF;
      if (w.w == m) w.w = 0x7FFFFFFF;
      f.x += c.x;
      f.y += c.y;
    }
  } else {
    const int* items = d.flex_item + l.slot * kFlexListCap;
    const float2* forces = d.flex_force + l.slot * kFlexListCap;
    int last = -1;
    for (int r = 0; r < l.n; ++r) {
      int pick = 0, best = 0x7FFFFFFF;
      for (int j = 0; j < l.n; ++j) {
        const int w = items[j];
        if (w > last && w < best) {
          best = w;
          pick = j;
        }
      }
      const float2 c = forces[pick];
      f.x += c.x;
      f.y += c.y;
      last = best;
    }
  }
  d.flex_cnt[l.slot] = 0;
}

// The node's own state, its CSR range and its first kNodeCorners corner
// forces are loaded before the scene lookup, so one node waits on few
// dependent loads; the corners are then summed in the same ascending order.
constexpr int kNodeCorners = 6;  // an interior node of a structured triangulation has 6

template <bool FLEX, bool RIGID>
__device__ __forceinline__ void node_step(const Dev& d, int i, bool valid) {
  const uint32_t w = valid ? d.node_word[i] : 0u;
  float2 x = make_float2(0.f, 0.f), v = make_float2(0.f, 0.f), bv0 = make_float2(0.f, 0.f);
  int k0 = 0, k1 = 0;
  float mass = 1.0f;
  if (valid) {
    x = d.x[i];
    v = d.v[i];
    k0 = d.csr_off[i];
    k1 = d.csr_end[i];
    mass = d.mass[i];
    bv0 = d.bcv[i];
  }
  FlexList fl;
  if (FLEX && valid && (w & fw::NODE_BOUNDARY)) fl.load(d, i);
  float2 cq[kNodeCorners];
#pragma unroll
  for (int u = 0; u < kNodeCorners; ++u) cq[u] = k0 + u < k1 ? d.corner[k0 + u] : make_float2(0.f, 0.f);
  const int b = (int)(w >> fw::NODE_BODY_SHIFT);
  const int s = valid ? d.body_scene[b] : 0;
  const int mode = valid ? d.scene_mode[s] : fw::MODE_FROZEN;
  const bool live = mode != fw::MODE_FROZEN;
  bool bnd = false;
  if (live) {
    const float dt = mode == fw::MODE_INIT ? 0.0f : (d.uniform_dt ? d.dt_uniform : d.scene_dt[s]);
    const float damp = mode == fw::MODE_INIT ? 0.0f : d.scene_damp[s];
    float2 f = make_float2(0.f, 0.f);
    bnd = (w & fw::NODE_BOUNDARY) != 0;
    if (bnd && mode == fw::MODE_STEP) {
      const int p0 = d.body_pair_off[b], pn = d.body_pair_cnt[b];
      const int bs = RIGID ? d.bslot[i] : 0;  // this node's slot in its body's boundary list
      bool flex_done = !FLEX || fl.slot < 0;
      // U pairs at a time.  Rigid pairs: the items were evaluated by
      // k_elements_rigid from this same state, and are fetched together (one
      // after the other, the 13 pairs of a slab under 12 rigids were a chain of
      // 39 loads).
      constexpr int U = RIGID ? 4 : 1;
      for (int k0 = 0; k0 < pn; k0 += U) {
        int kind[U], on[U], slot[U];
        float2 rf[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          on[u] = 0;
          if (k0 + u >= pn) continue;
          const Pair& pr = d.pairs[p0 + k0 + u];
          on[u] = d.pair_active[p0 + k0 + u];
          kind[u] = pr.kind;
          slot[u] = pr.n0 + bs;
        }
        if (RIGID) {
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (k0 + u < pn && kind[u] == fw::PAIR_RIGID && on[u]) {
              on[u] = __float_as_int(d.ritem[slot[u]].w) >= 0;
              rf[u] = d.rforce[slot[u]];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (k0 + u >= pn) continue;
          if (FLEX && !flex_done && kind[u] != fw::PAIR_PLANE) {
            flex_add(d, fl, f);  // FEM-FEM contact runs after the planes, before the height fields / voxels
            flex_done = true;
          }
          if (!on[u]) continue;
          float2 cf;
          if (RIGID && kind[u] == fw::PAIR_RIGID)
            cf = rf[u];
          else if (!fw::contact_force(d.pairs[p0 + k0 + u], d.heights, d.occ, d.vox, x, v, dt, cf))
            continue;
          f.x += cf.x;
          f.y += cf.y;
        }
      }
      if (FLEX && !flex_done) flex_add(d, fl, f);
    }
#pragma unroll
    for (int u = 0; u < kNodeCorners; ++u)  // contiguous, ascending element
      if (k0 + u < k1) {
        f.x += cq[u].x;
        f.y += cq[u].y;
      }
    for (int k = k0 + kNodeCorners; k < k1; ++k) {
      const float2 c = d.corner[k];
      f.x += c.x;
      f.y += c.y;
    }
    const int bc = (int)(w & fw::NODE_BC_MASK);
    const float2 bv = (bc & (fw::BC_A | fw::BC_GRAVITY | fw::BC_FORCE | fw::BC_V)) ? bv0 : make_float2(0.f, 0.f);
    fw::integrate(bc, f, mass, bv, dt, damp, x, v);
    d.x[i] = x;
    d.v[i] = v;
    if (!(isfinite(x.x) && isfinite(x.y) && isfinite(v.x) && isfinite(v.y))) d.scene_bad[s] = 1;
  }
  // Per-body AABB of boundary nodes (femspringmanager.py:361-408).
  const unsigned full = 0xFFFFFFFFu;
  const unsigned mb = __ballot_sync(full, bnd);
  if (mb == 0u) return;
  const int leader = __ffs(mb) - 1;
  const int bl = __shfl_sync(full, b, leader);
  const bool uniform = __all_sync(full, !bnd || b == bl);
  const bool okx = bnd && x.x == x.x, oky = bnd && x.y == x.y;  // NaN widens no box
  float lx = okx ? x.x : 1e30f, ly = oky ? x.y : 1e30f;
  float hx = okx ? x.x : -1e30f, hy = oky ? x.y : -1e30f;
  if (uniform) {
    for (int o = 16; o > 0; o >>= 1) {
      lx = fminf(lx, __shfl_xor_sync(full, lx, o));
      ly = fminf(ly, __shfl_xor_sync(full, ly, o));
      hx = fmaxf(hx, __shfl_xor_sync(full, hx, o));
      hy = fmaxf(hy, __shfl_xor_sync(full, hy, o));
    }
    if ((int)(threadIdx.x & 31) == leader) {
      int* r = d.aabb_ring + ((size_t)(d.scene_counter[s] & 1) * d.B + b) * 4;
      atomicMin(r + 0, fw::f2ord(lx));
      atomicMin(r + 1, fw::f2ord(ly));
      atomicMax(r + 2, fw::f2ord(hx));
      atomicMax(r + 3, fw::f2ord(hy));
    }
  } else if (bnd) {
    int* r = d.aabb_ring + ((size_t)(d.scene_counter[s] & 1) * d.B + b) * 4;
    atomicMin(r + 0, fw::f2ord(lx));
    atomicMin(r + 1, fw::f2ord(ly));
    atomicMax(r + 2, fw::f2ord(hx));
    atomicMax(r + 3, fw::f2ord(hy));
  }
}

__global__ void __launch_bounds__(kMaxBlock) k_nodes(Dev d) {
  if (d.use_chunks) {
    for (int c = blockIdx.x; c < d.n_n_chunks; c += gridDim.x) {
      const int2 ch = d.n_chunks[c];
      node_step<false, false>(d, ch.x + (int)threadIdx.x, (int)threadIdx.x < ch.y);
    }
    return;
  }
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  node_step<false, false>(d, i, i < d.N);
}

// k_nodes of worlds with FEM-FEM contact: the node's contact forces from the
// work items join its plane and ground contact forces in launch order.
__global__ void __launch_bounds__(kMaxBlock) k_nodes_flex(Dev d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  node_step<true, false>(d, i, i < d.N);
}

// The rigid side of a substep: one warp per rigid of a stepping scene adds
// its work items' reactions to its accumulators in work-item order (its
// pairs in pair order, each gated pair's items in boundary-node order: lanes
// load 256 records at a time, and every lane adds the hits in ascending lane
// order through shuffles, so the sum is a serial run of the reference's atomic
// adds).  The warp that finishes a scene's last rigid (a per-scene arrival count
// after a fence) counts the substep and, on the substeps of its schedule, runs
// the rigid update (fw_rigid.cuh), a lane per rigid.
struct RigidDev {
  Rigid* rig;
  int n;
  float4* gbox;
  int* gkind;
  int n_ground;
  float4* item;
  int n_items;
  int* rp_off;   // per rigid: its pairs' item ranges rp_rng[rp_off[g] .. rp_off[g + 1])
  int4* rp_rng;  // (first item, item count, pair), pair order
  fw::RigidScene* rs;  // the scenes with rigids
  int n_rs;
  int* done;           // per scene with rigids: warps finished this substep
  const fw::RigidClock* clock;  // per scene
  int* count;                   // per scene: the reference's rigid_update_times
  int* err;
};

// Warp g of the rigid side.
__device__ __forceinline__ void rigid_step(const Dev& d, const RigidDev& r, int g) {
  const unsigned full = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  const float4 none = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
  if (g >= r.n) return;
  Rigid& rg = r.rig[g];
  const int q0 = r.rp_off[g], q1 = r.rp_off[g + 1], k = rg.rs;
  if (d.scene_mode[rg.scene] != fw::MODE_STEP) return;
  float ax = rg.acc[0], ay = rg.acc[1], aw = rg.accw;
  for (int q = q0; q < q1; ++q) {
    const int4 rng = r.rp_rng[q];
    if (!d.pair_active[rng.z]) continue;
    for (int base = 0; base < rng.y; base += 256) {
      float4 rec[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int it = base + 32 * u + lane;
        rec[u] = it < rng.y ? r.item[rng.x + it] : none;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        unsigned m = __ballot_sync(full, __float_as_int(rec[u].w) >= 0);
        while (m) {
          const int l = __ffs(m) - 1;
          m &= m - 1;
          ax = ax + __shfl_sync(full, rec[u].x, l);
          ay = ay + __shfl_sync(full, rec[u].y, l);
          aw = aw + __shfl_sync(full, rec[u].z, l);
        }
      }
    }
  }
  const fw::RigidScene rs = r.rs[k];
  const fw::RigidClock ck = r.clock[rs.scene];
  int last = 0;
  if (lane == 0) {
    rg.acc[0] = ax;
    rg.acc[1] = ay;
    rg.accw = aw;
    __threadfence();
    last = atomicAdd(r.done + k, 1) + 1 == rs.rn;
    __threadfence();
  }
  if (!__shfl_sync(full, last, 0)) return;
  __threadfence();  // every lane reads the other warps' sums
  const int cnt = __ldcg(r.count + rs.scene) + 1;
  __syncwarp();
  if (lane == 0) {
    r.done[k] = 0;
    r.count[rs.scene] = cnt;
  }
  if (ck.every < 1 || cnt % ck.every != 0) return;
  fw::rigid_update(r.rig + rs.r0, rs.rn, r.gbox + rs.g0, r.gkind + rs.g0, rs.gn, ck.dt, ck.damping, r.err, lane);
}

// k_nodes of worlds with FEM-rigid contact (FLEX: FEM-FEM contact as well).
// Blocks [0, rb) are the rigid side, a warp per rigid: the node step reads
// nothing that it writes.
// Bound by the latency of either side's chain.  A slab of 8192 triangles under
// 12 rigids: 20.3 us a substep with the rigid side in a launch of its own (one
// thread updating the rigids one after the other through global memory) and the
// node step walking its pairs one by one, 10.2 us now; 640 triangles under one
// rigid 11.1 and 7.5.
template <bool FLEX>
__global__ void __launch_bounds__(kMaxBlock) k_nodes_rigid(Dev d, RigidDev r, int rb) {
  if ((int)blockIdx.x < rb) {
    rigid_step(d, r, blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
    return;
  }
  const int i = (blockIdx.x - rb) * blockDim.x + threadIdx.x;
  node_step<FLEX, true>(d, i, i < d.N);
}

// Rotation cache and boxes of the rigids at construction
// (precompute_rigid_transforms + updateBBox, explicitloop.py:198-201).
__global__ void k_rigid_init(Rigid* rig, int n) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= n) return;
  fw::rigid_rot(rig[a]);
  if (rig[a].type != fw::RIGID_ANALYTICAL) fw::rigid_aabb(rig[a]);  // an analytical entry starts at getBBox()
}

__global__ void k_log(const float* __restrict__ x, float* __restrict__ y, float* __restrict__ quotient, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  y[i] = fw::fw_log(x[i]);
  if (quotient) quotient[i] = fw::log_quotient(x[i]);
}

// Per cell of the voxel pairs [p0, p0 + gridDim.x) the nearest free cells that
// fw::contact_force looks for (zero for a cell that is not occupied): left + 1,
// right, below + 1, above (0, nx, 0, ny: the grid's edge).  A pair's warps, one
// to a block, take 32 columns each (a lane walks one, 32 loads in flight), one way
// or the other, and then the rows (32 cells at a time, by ballots).  A new scene waits
// for this before its first substep: 128 x 128 cells 9 us, 66 by one block with a
// thread per row and per column, bound by a walk's loads one after the other.
constexpr int kVoxelBlocks = 128;
__global__ void __launch_bounds__(32) k_voxel_table(Dev d, int p0) {
  const Pair pr = d.pairs[p0 + blockIdx.x];
  if (pr.kind != fw::PAIR_VOXEL || pr.pad) return;
  const int nx = pr.n0, ny = pr.n1, lane = threadIdx.x, cols = (ny + 31) / 32;
  const int8_t* g = d.occ + pr.table;
  ushort4* w = d.vox + pr.table;
  for (int unit = blockIdx.y; unit < 2 * cols + nx; unit += gridDim.y) {
    constexpr int U = 32;
    if (unit < cols) {
      const int j = 32 * unit + lane;
      if (j >= ny) continue;
      int near = 0;
      for (int i0 = 0; i0 < nx; i0 += U) {
        int8_t o[U];
#pragma unroll
        for (int u = 0; u < U; ++u) o[u] = __ldg(g + (size_t)min(i0 + u, nx - 1) * ny + j);
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (i0 + u < nx) {
            w[(size_t)(i0 + u) * ny + j].x = o[u] == 1 ? (unsigned short)near : 0;
            if (o[u] == 0) near = i0 + u + 1;
          }
      }
      continue;
    }
    if (unit < 2 * cols) {
      const int j = 32 * (unit - cols) + lane;
      if (j >= ny) continue;
      int near = nx;
      for (int i0 = nx - 1; i0 >= 0; i0 -= U) {
        int8_t o[U];
#pragma unroll
        for (int u = 0; u < U; ++u) o[u] = __ldg(g + (size_t)max(i0 - u, 0) * ny + j);
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (i0 - u >= 0) {
            w[(size_t)(i0 - u) * ny + j].y = o[u] == 1 ? (unsigned short)near : 0;
            if (o[u] == 0) near = i0 - u;
          }
      }
      continue;
    }
    const size_t row = (size_t)(unit - 2 * cols) * ny;
    int near = 0;
    for (int j0 = 0; j0 < ny; j0 += 32) {
      const int j = j0 + lane;
      const int8_t o = j < ny ? __ldg(g + row + j) : (int8_t)1;
      const unsigned free = __ballot_sync(0xFFFFFFFFu, o == 0), before = free & ((1u << lane) - 1u);
      if (j < ny) w[row + j].z = o == 1 ? (unsigned short)(before ? j0 + 32 - __clz(before) : near) : 0;
      if (free) near = j0 + 32 - __clz(free);
    }
    near = ny;
    for (int j0 = (cols - 1) * 32; j0 >= 0; j0 -= 32) {
      const int j = j0 + lane;
      const int8_t o = j < ny ? __ldg(g + row + j) : (int8_t)1;
      const unsigned free = __ballot_sync(0xFFFFFFFFu, o == 0), after = free & ~((2u << lane) - 1u);
      if (j < ny) w[row + j].w = o == 1 ? (unsigned short)(after ? j0 + __ffs(after) - 1 : near) : 0;
      if (free) near = j0 + __ffs(free) - 1;
    }
  }
}

// Reference-shape precompute, _prepare_fem_data_kernel
// (flatworld/femspringmanager.py:113-138), plus the Lame constants of
// getStress2D (materialfunctions.py:12-13), which depend only on E and nu.
__global__ void k_prepare_elements(Dev d, const float* __restrict__ young,
                                   const float* __restrict__ poisson,
                                   const float* __restrict__ rho, int e_lo, int e_hi) {
  const int e = e_lo + blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= e_hi) return;
  if (fw::elem_type(d.emat[e].word) == fw::MAT_SPRING) {  // addSpringDomain (femspringmanager.py:848-861)
    ElemMat m = d.emat[e];
    m.area = rho[e - e_lo];     // rest length
    m.lam = young[e - e_lo];    // spring stiffness
    m.mu = poisson[e - e_lo];   // damping
    d.emat[e] = m;
    d.jinv[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    d.ndmass[e] = 0.0f;         // the nodes carry the domain's mass
    return;
  }
  const int c0 = d.conn[3 * e], c1 = d.conn[3 * e + 1], c2 = d.conn[3 * e + 2];
  const float2 a = d.x0[c0], b = d.x0[c1], c = d.x0[c2];
  const float j00 = a.x - c.x, j01 = b.x - c.x, j10 = a.y - c.y, j11 = b.y - c.y;
  const float det = j00 * j11 - j01 * j10;
  const float area = fabsf(det) * 0.5f;
  float4 ji = make_float4(0.f, 0.f, 0.f, 0.f);
  if (det != 0.0f) {
    const float r = 1.0f / det;
    ji = make_float4(j11 * r, -j01 * r, -j10 * r, j00 * r);
  }
  d.jinv[e] = ji;
  const float E = young[e - e_lo], nu = poisson[e - e_lo];
  ElemMat m = d.emat[e];
  m.area = area;
  m.lam = E * nu / ((1.0f + nu) * (1.0f - 2.0f * nu));
  m.mu = E / (2.0f * (1.0f + nu));
  d.emat[e] = m;
  d.ndmass[e] = area * rho[e - e_lo] / 3.0f;
}

// Lumped mass: each node adds its elements' shares in ascending element order,
// the order of the reference's serial atomic adds.
__global__ void k_prepare_mass(Dev d, int n_lo, int n_hi) {
  const int i = n_lo + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_hi) return;
  float m = 0.0f;
  for (int k = d.csr_off[i]; k < d.csr_end[i]; ++k) m += d.ndmass[d.csr_slot[k] / 3];
  d.mass[i] = m;
}

// Selective mass scaling, _mass_scaling_kernel (femspringmanager.py:139-196):
// a triangle whose critical step 0.4 L_min / sqrt(E / rho) is below dt_target
// gets the density that makes it dt_target, and its three nodes a third of
// the added mass each.  The reference runs it on one thread in element order;
// here k_mass_scale_elems finds each triangle's share and k_mass_scale_nodes
// adds a node's shares in ascending element order (its CSR list), the same
// additions in the same order.
__global__ void k_mass_scale_elems(Dev d, const float* __restrict__ young, const float* __restrict__ rho,
                                   float dt_target, float* __restrict__ dm, int32_t* __restrict__ hit) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= d.E) return;
  if (fw::elem_type(d.emat[e].word) == fw::MAT_SPRING) {  // springs: the node pass
    dm[e] = 0.0f;
    hit[e] = 0;
    return;
  }
  const float2 a = d.x[d.conn[3 * e]], b = d.x[d.conn[3 * e + 1]], c = d.x[d.conn[3 * e + 2]];
  const float e01x = b.x - a.x, e01y = b.y - a.y, e12x = c.x - b.x, e12y = c.y - b.y, e20x = a.x - c.x, e20y = a.y - c.y;
  const float e01 = sqrtf(e01x * e01x + e01y * e01y), e12 = sqrtf(e12x * e12x + e12y * e12y);
  const float e20 = sqrtf(e20x * e20x + e20y * e20y);
  const float m12 = e12 < e20 ? e12 : e20;
  const float L = e01 < m12 ? e01 : m12;
  const float E = young[e], r = rho[e];
  const float ce = sqrtf(E / r);
  const float dt_elem = 0.4f * L / ce;
  int h = 0;
  float add = 0.0f;
  if (dt_elem < dt_target && L > 1e-15f) {
    const float q = dt_target / (0.4f * L);
    const float rho_new = E * q * q;
    add = (rho_new - r) * d.emat[e].area / 3.0f;
    h = 1;
  }
  dm[e] = add;
  hit[e] = h;
}

__global__ void k_mass_scale_nodes(Dev d, const float* __restrict__ dm, const int32_t* __restrict__ hit,
                                   float dt_target) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.N) return;
  float m = d.mass[i];
  for (int k = d.csr_off[i]; k < d.csr_end[i]; ++k) {  // triangles first (the reference's first loop)
    const int e = d.csr_slot[k] / 3;
    if (hit[e]) m = m + dm[e];
  }
  for (int k = d.csr_off[i]; k < d.csr_end[i]; ++k) {  // then springs: at least 4 k dt^2 (its second loop)
    const int e = d.csr_slot[k] / 3;
    const ElemMat em = d.emat[e];
    if (fw::elem_type(em.word) != fw::MAT_SPRING) continue;
    const float m_min = 4.0f * em.lam * dt_target * dt_target;
    if (m < m_min) m = m_min;
  }
  d.mass[i] = m;
}

// Lame constants of elements [e_lo, e_hi) from new Young's moduli (same
// formula as k_prepare_elements).
__global__ void k_set_young(Dev d, const float* __restrict__ young, const float* __restrict__ poisson,
                            int e_lo, int e_hi) {
  const int e = e_lo + blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= e_hi) return;
  const float E = young[e - e_lo], nu = poisson[e];
  ElemMat m = d.emat[e];
  m.lam = E * nu / ((1.0f + nu) * (1.0f - 2.0f * nu));
  m.mu = E / (2.0f * (1.0f + nu));
  d.emat[e] = m;
}

// The adjoint state is accumulated in FP64, so that summing thousands of
// substeps adds no error of its own; the element Jacobian products are FP32
// dual numbers on the recorded FP32 trajectory, i.e. this is the exact
// adjoint of the FP32 forward up to FP32 rounding of those products.
struct Adj {
  double2* xb;   // adjoint of positions
  double2* vb;   // adjoint of velocities
  double2* fb;   // adjoint of the node force of the current substep
  double* Eb;    // d loss / d Young's modulus, per element
  float* young;  // Young's modulus per element
  float2* traj;  // recorded positions of the segment, [K][N]
  float2* trajv;  // recorded velocities of the segment, [K][N] (contact damping terms)
  float4* trajs;  // recorded J2 state of the segment, [K][E] (worlds with J2 triangles)
  double* sb;     // adjoint of the J2 state (eps_p Voigt, eqps), 4 per element
  int32_t* gates;  // recorded broad-phase gates, [K][P]
  float2* io_x;  // FP32 staging of xb / vb / Eb for the C ABI
  float2* io_v;
  float* io_E;
};

// Adjoint of "v' = v + dt f / m; BC override" at every node: from (xb', vb')
// form the force adjoint fb and the velocity adjoint of the previous substep.
// With damping c, v' = v (1 - dt c / m) + dt f / m.
__device__ __forceinline__ void adj_node_prep(const Dev& d, const Adj& a, int i, float dt, float damp) {
  const int bc = (int)(d.node_word[i] & fw::NODE_BC_MASK);
  const double2 xb = a.xb[i], vb = a.vb[i];
  const double h = (double)dt;
  const double2 vt = make_double2(vb.x + h * xb.x, vb.y + h * xb.y);
  const bool vfixed = (bc & (fw::BC_U | fw::BC_V)) != 0;
  const bool fdead = vfixed || (bc & fw::BC_A) != 0;
  const double s = h / (double)d.mass[i];
  const double keep = 1.0 - s * (double)damp;
  a.fb[i] = fdead ? make_double2(0.0, 0.0) : make_double2(s * vt.x, s * vt.y);
  a.vb[i] = vfixed ? make_double2(0.0, 0.0) : make_double2(keep * vt.x, keep * vt.y);
}

__global__ void k_adj_seed(Adj a, int N, int has_x, int has_v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const float2 x = has_x ? a.io_x[i] : make_float2(0.f, 0.f);
  const float2 v = has_v ? a.io_v[i] : make_float2(0.f, 0.f);
  a.xb[i] = make_double2(x.x, x.y);
  a.vb[i] = make_double2(v.x, v.y);
}

__global__ void k_adj_out(Adj a, int N, int E) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) {
    a.io_x[i] = make_float2((float)a.xb[i].x, (float)a.xb[i].y);
    a.io_v[i] = make_float2((float)a.vb[i].x, (float)a.vb[i].y);
  }
  if (i < E) a.io_E[i] = (float)a.Eb[i];
}

__global__ void k_adj_prep(Dev d, Adj a, float dt, float damp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < d.N) adj_node_prep(d, a, i, dt, damp);
}

__global__ void k_adj_elements(Dev d, Adj a, const float2* __restrict__ x, const float4* __restrict__ st) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= d.E) return;
  const ElemMat m = d.emat[e];
  const int c0 = d.conn[3 * e], c1 = d.conn[3 * e + 1], c2 = d.conn[3 * e + 2];
  const double2 b0 = a.fb[c0], b1 = a.fb[c1], b2 = a.fb[c2];
  if (fw::elem_type(m.word) == fw::MAT_MISES) {
    // transpose of the local Jacobian, column by column: 6 positions, 4 state, E
    const float2 p0 = x[c0], p1 = x[c1], p2 = x[c2];
    const float xs[6] = {p0.x, p0.y, p1.x, p1.y, p2.x, p2.y};
    const float4 s4 = st[e];
    const float ss[4] = {s4.x, s4.y, s4.z, s4.w};
    double ob[10] = {b0.x, b0.y, b1.x, b1.y, b2.x, b2.y, 0.0, 0.0, 0.0, 0.0};
    for (int k = 0; k < 4; ++k) ob[6 + k] = a.sb[4 * (size_t)e + k];
    const float young = a.young[e];
    const float2 yp = d.j2par[e];
    float corner[6];
    double snew[4];
    double eb = 0.0;
    for (int col = 0; col < 11; ++col) {
      fw::Dual X[6], S[4], F[6], SN[4];
      for (int r = 0; r < 6; ++r) X[r] = fw::dmk(xs[r], col == r ? 1.f : 0.f);
      for (int k = 0; k < 4; ++k) S[k] = fw::dmk(ss[k], col == 6 + k ? 1.f : 0.f);
      const fw::Dual lam = fw::dmk(m.lam, col == 10 ? m.lam / young : 0.f);
      const fw::Dual mu = fw::dmk(m.mu, col == 10 ? m.mu / young : 0.f);
      fw::element_j2_dual(X, d.jinv[e], lam, mu, yp.x, yp.y, S, m.area, F, SN);
      double dot = 0.0;
      for (int r = 0; r < 6; ++r) dot += ob[r] * (double)F[r].d;
      for (int k = 0; k < 4; ++k) dot += ob[6 + k] * (double)SN[k].d;
      if (col < 6) corner[col] = (float)dot;
      else if (col < 10) snew[col - 6] = dot;
      else eb = dot;
    }
    d.corner[d.corner_pos[3 * e]] = make_float2(corner[0], corner[1]);
    d.corner[d.corner_pos[3 * e + 1]] = make_float2(corner[2], corner[3]);
    d.corner[d.corner_pos[3 * e + 2]] = make_float2(corner[4], corner[5]);
    for (int k = 0; k < 4; ++k) a.sb[4 * (size_t)e + k] = snew[k];
    a.Eb[e] += eb;
    return;
  }
  const float2 w0 = make_float2((float)b0.x, (float)b0.y), w1 = make_float2((float)b1.x, (float)b1.y),
               w2 = make_float2((float)b2.x, (float)b2.y);
  fw::Dual f[6];
  fw::element_forces_jvp(x[c0], x[c1], x[c2], w0, w1, w2, d.jinv[e], fw::elem_type(m.word), m.lam, m.mu,
                         m.area, f);
  d.corner[d.corner_pos[3 * e]] = make_float2(f[0].d, f[1].d);
  d.corner[d.corner_pos[3 * e + 1]] = make_float2(f[2].d, f[3].d);
  d.corner[d.corner_pos[3 * e + 2]] = make_float2(f[4].d, f[5].d);
  const double dot = b0.x * f[0].v + b0.y * f[1].v + b1.x * f[2].v + b1.y * f[3].v + b2.x * f[4].v + b2.y * f[5].v;
  a.Eb[e] += dot / (double)a.young[e];
}

// xb <- xb' + sum of element VJPs + plane-contact VJP; with prep, also the
// force / velocity adjoints of the previous substep (fused, saves a launch).
__global__ void k_adj_nodes(Dev d, Adj a, const float2* __restrict__ x, const float2* __restrict__ v,
                            const int32_t* __restrict__ gates, float dt, float damp, int prep) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.N) return;
  double2 xb = a.xb[i];
  const double2 fb = a.fb[i];
  for (int k = d.csr_off[i]; k < d.csr_end[i]; ++k) {
    const float2 c = d.corner[k];
    xb.x += c.x;
    xb.y += c.y;
  }
  const uint32_t w = d.node_word[i];
  if (w & fw::NODE_BOUNDARY) {
    const int b = (int)(w >> fw::NODE_BODY_SHIFT);
    const float2 xi = x[i], vi = v[i];
    double2 vb = a.vb[i];
    for (int q = 0; q < d.body_pair_cnt[b]; ++q) {
      const int p = d.body_pair_off[b] + q;
      if (!gates[p]) continue;
      fw::contact_vjp(d.pairs[p], d.heights, d.occ, xi, vi, dt, fb, xb, vb);
    }
    a.vb[i] = vb;
  }
  a.xb[i] = xb;
  if (prep) adj_node_prep(d, a, i, dt, damp);
}

// ------------------------------------------------------------------ tangent
// Forward-mode derivative of the same substep along (dx, dv, dE), on the
// recorded FP32 trajectory and gates: df = J(x) dx + f_e dE_e / E_e
// (+ plane contact -k n (n . dx) while the node penetrates), then
// dv' = dv (1 - dt c / m) + dt df / m (zero for fixed / enforced-velocity
// nodes, no df for prescribed-acceleration nodes), dx' = dx + dt dv'.
// Used to check that the adjoint is the exact transpose (dot-product test) and
// for forward-mode gradients.
struct Tan {
  double2* dx;
  double2* dv;
  float* dE;     // perturbation of Young's modulus per element
  float* young;  // Young's modulus per element
  float2* xs;    // positions at the start of the substep
  float2* vs;    // velocities at the start of the substep
  float2* io_x;  // FP32 staging for the C ABI
  float2* io_v;
};

__global__ void k_tan_elements(Dev d, Tan t) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= d.E) return;
  const ElemMat m = d.emat[e];
  const int c0 = d.conn[3 * e], c1 = d.conn[3 * e + 1], c2 = d.conn[3 * e + 2];
  const double2 u0 = t.dx[c0], u1 = t.dx[c1], u2 = t.dx[c2];
  fw::Dual f[6];
  fw::element_forces_jvp(t.xs[c0], t.xs[c1], t.xs[c2], make_float2((float)u0.x, (float)u0.y),
                         make_float2((float)u1.x, (float)u1.y), make_float2((float)u2.x, (float)u2.y), d.jinv[e],
                         fw::elem_type(m.word), m.lam, m.mu, m.area, f);
  const float r = t.dE[e] / t.young[e];
  d.corner[d.corner_pos[3 * e]] = make_float2(f[0].d + f[0].v * r, f[1].d + f[1].v * r);
  d.corner[d.corner_pos[3 * e + 1]] = make_float2(f[2].d + f[2].v * r, f[3].d + f[3].v * r);
  d.corner[d.corner_pos[3 * e + 2]] = make_float2(f[4].d + f[4].v * r, f[5].d + f[5].v * r);
}

__global__ void k_tan_nodes(Dev d, Tan t, float dt, float damp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.N) return;
  const uint32_t w = d.node_word[i];
  const int bc = (int)(w & fw::NODE_BC_MASK);
  const double2 dx = t.dx[i], dv = t.dv[i];
  double fx = 0.0, fy = 0.0;
  if (w & fw::NODE_BOUNDARY) {
    const int b = (int)(w >> fw::NODE_BODY_SHIFT);
    const float2 xi = t.xs[i], vi = t.vs[i];
    for (int q = 0; q < d.body_pair_cnt[b]; ++q) {
      const int p = d.body_pair_off[b] + q;
      if (!d.pair_active[p]) continue;
      fw::contact_jvp(d.pairs[p], d.heights, d.occ, xi, vi, dt, dx, dv, fx, fy);
    }
  }
  for (int k = d.csr_off[i]; k < d.csr_end[i]; ++k) {
    const float2 c = d.corner[k];
    fx += c.x;
    fy += c.y;
  }
  const double h = (double)dt, s = h / (double)d.mass[i], keep = 1.0 - s * (double)damp;
  double2 nv;
  if (bc & (fw::BC_U | fw::BC_V)) nv = make_double2(0.0, 0.0);
  else if (bc & fw::BC_A) nv = make_double2(keep * dv.x, keep * dv.y);
  else nv = make_double2(keep * dv.x + s * fx, keep * dv.y + s * fy);
  t.dv[i] = nv;
  t.dx[i] = make_double2(dx.x + h * nv.x, dx.y + h * nv.y);
}

__global__ void k_tan_seed(Tan t, int N, int has_x, int has_v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const float2 x = has_x ? t.io_x[i] : make_float2(0.f, 0.f);
  const float2 v = has_v ? t.io_v[i] : make_float2(0.f, 0.f);
  t.dx[i] = make_double2(x.x, x.y);
  t.dv[i] = make_double2(v.x, v.y);
}

__global__ void k_tan_out(Tan t, int N) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  t.io_x[i] = make_float2((float)t.dx[i].x, (float)t.dx[i].y);
  t.io_v[i] = make_float2((float)t.dv[i].x, (float)t.dv[i].y);
}

// ------------------------------------------------------------------ energy
// Total energy, reduced in FP64 (the only FP64 step of the library).  Terms
// per node: kinetic 1/2 m |v|^2; external potential -m g.x (gravity BC) or
// -f.x (constant nodal force), following the BC precedence of the update
// (fixed / prescribed-acceleration nodes have none); penalty 1/2 k sd^2 for
// every penetrating boundary node and contact pair of its body (the elastic
// part of the contact force, evaluated at zero velocity; not gated by the
// broad phase).  Per triangle: area x strain energy density --
//   Elastic (St-Venant-Kirchhoff): lambda/2 tr(E)^2 + mu E:E
//   NeoHookean: mu/2 (tr C - 2) - mu ln J + lambda/2 (ln J)^2
//   J2: the St-Venant-Kirchhoff form of the elastic strain E - eps_p
// -- the energies whose E-derivatives are the stresses of the step
// (materialfunctions.py:10-101).  Positions and moduli are the FP32 state,
// every operation after loading them is FP64.
struct EnergyChunk {
  int group;   // output row
  int n0, nn;  // node range
  int e0, ne;  // triangle range
};

__device__ double elem_energy(const Dev& d, int e) {
  const ElemMat m = d.emat[e];
  const int c0 = d.conn[3 * e], c1 = d.conn[3 * e + 1], c2 = d.conn[3 * e + 2];
  const float2 a = d.x[c0], b = d.x[c1], c = d.x[c2];
  if (fw::elem_type(m.word) == fw::MAT_SPRING) {  // k L0 / 2 (l / L0 - 1)^2, whose l-derivative is the spring force
    const double dx = (double)a.x - b.x, dy = (double)a.y - b.y;
    const double st = sqrt(dx * dx + dy * dy) / (double)m.area - 1.0;
    return 0.5 * (double)m.lam * (double)m.area * st * st;
  }
  const float4 ji = d.jinv[e];
  const double j00 = (double)a.x - (double)c.x, j01 = (double)b.x - (double)c.x;
  const double j10 = (double)a.y - (double)c.y, j11 = (double)b.y - (double)c.y;
  const double F00 = j00 * ji.x + j01 * ji.z, F01 = j00 * ji.y + j01 * ji.w;
  const double F10 = j10 * ji.x + j11 * ji.z, F11 = j10 * ji.y + j11 * ji.w;
  const double C00 = F00 * F00 + F10 * F10, C01 = F00 * F01 + F10 * F11, C11 = F01 * F01 + F11 * F11;
  const double lam = m.lam, mu = m.mu;
  const int type = fw::elem_type(m.word);
  double W;
  if (type == fw::MAT_NEOHOOKEAN) {
    const double lj = log(F00 * F11 - F01 * F10);
    W = 0.5 * mu * (C00 + C11 - 2.0) - mu * lj + 0.5 * lam * lj * lj;
  } else {
    double e0 = 0.5 * (C00 - 1.0), e1 = 0.5 * (C11 - 1.0), e2 = 0.5 * C01;
    if (type == fw::MAT_MISES) {
      const float4 ep = d.j2state[e];
      e0 -= ep.x;
      e1 -= ep.y;
      e2 -= ep.z;
    }
    const double tr = e0 + e1;
    W = 0.5 * lam * tr * tr + mu * (e0 * e0 + e1 * e1 + 2.0 * e2 * e2);
  }
  return (double)m.area * W;
}

__device__ void node_energy(const Dev& d, int i, double& ke, double& ext, double& pen) {
  const float2 x = d.x[i], v = d.v[i], bcv = d.bcv[i];
  const double m = d.mass[i];
  ke += 0.5 * m * ((double)v.x * v.x + (double)v.y * v.y);
  const uint32_t w = d.node_word[i];
  const int bc = (int)(w & fw::NODE_BC_MASK);
  if (bc & (fw::BC_U | fw::BC_A)) {
  } else if (bc & fw::BC_GRAVITY) {
    ext -= m * ((double)bcv.x * x.x + (double)bcv.y * x.y);
  } else if (bc & fw::BC_FORCE) {
    ext -= (double)bcv.x * x.x + (double)bcv.y * x.y;
  }
  if (w & fw::NODE_BOUNDARY) {
    const int b = (int)(w >> fw::NODE_BODY_SHIFT);
    for (int q = 0; q < d.body_pair_cnt[b]; ++q) {
      const Pair& pr = d.pairs[d.body_pair_off[b] + q];
      float2 f;
      if (pr.kind == fw::PAIR_RIGID) {  // the normal penalty force of the primitive
        float nx, ny, cx, cy;
        const Rigid& g = d.rig[pr.table];
        const float depth = fw::rigid_detect(g, x.x, x.y, nx, ny, cx, cy) - 1e-4f;
        if (depth < 0.0f) pen += 0.5 * (double)pr.penalty * (double)depth * (double)depth;
        continue;
      }
      if (fw::contact_force(pr, d.heights, d.occ, d.vox, x, make_float2(0.f, 0.f), 0.f, f))
        pen += 0.5 * ((double)f.x * f.x + (double)f.y * f.y) / (double)pr.penalty;
    }
  }
}

constexpr int kEnergyThreads = 256;
// Nodes and triangles of a block.  The FP64 logarithm and divides of a NeoHookean
// triangle set a block's time, so the blocks have to fill the SMs: chunks of
// 8192 left 131072 triangles on 16 of them (92 us a report, 40 with 1024).
constexpr int kEnergyChunk = 1024;

// One block per chunk: fixed-order strided sums, then a fixed tree.
__global__ void __launch_bounds__(kEnergyThreads) k_energy_chunks(Dev d, const EnergyChunk* ch, double4* part) {
  __shared__ double sm[4][kEnergyThreads];
  const EnergyChunk c = ch[blockIdx.x];
  const int t = threadIdx.x;
  double ke = 0.0, st = 0.0, ext = 0.0, pen = 0.0;
  for (int i = t; i < c.nn; i += kEnergyThreads) node_energy(d, c.n0 + i, ke, ext, pen);
  for (int e = t; e < c.ne; e += kEnergyThreads) st += elem_energy(d, c.e0 + e);
  sm[0][t] = ke;
  sm[1][t] = st;
  sm[2][t] = ext;
  sm[3][t] = pen;
  __syncthreads();
  for (int h = kEnergyThreads / 2; h > 0; h >>= 1) {
    if (t < h)
      for (int k = 0; k < 4; ++k) sm[k][t] += sm[k][t + h];
    __syncthreads();
  }
  if (t == 0) part[blockIdx.x] = make_double4(sm[0][0], sm[1][0], sm[2][0], sm[3][0]);
}

// One block per group: strided sums of its chunks' partials, then a fixed tree.
constexpr int kEnergyGroupThreads = 64;
__global__ void __launch_bounds__(kEnergyGroupThreads) k_energy_groups(const int* first, const double4* part, double4* out) {
  __shared__ double4 sm[kEnergyGroupThreads];
  const int g = blockIdx.x, t = threadIdx.x;
  double4 s = make_double4(0.0, 0.0, 0.0, 0.0);
  for (int k = first[g] + t; k < first[g + 1]; k += kEnergyGroupThreads) {
    const double4 p = part[k];
    s = make_double4(s.x + p.x, s.y + p.y, s.z + p.z, s.w + p.w);
  }
  sm[t] = s;
  __syncthreads();
  for (int h = kEnergyGroupThreads / 2; h > 0; h >>= 1) {
    if (t < h) {
      const double4 a = sm[t], b = sm[t + h];
      sm[t] = make_double4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
    }
    __syncthreads();
  }
  if (t == 0) out[g] = sm[0];
}

}  // namespace

#include "fw_resident.cuh"
#include "fw_stream.cuh"
#include "fw_cluster.cuh"

// ------------------------------------------------------------------ context

// Page-locked blocks for reads into pageable memory, one to a context while
// they last (a context without one reads as before), handed back when it goes.
// They are parts of one allocation made for the first context: one costs the
// driver as much as a dozen small reads.
constexpr size_t kHostRead = 128 << 10;         // larger reads go to the caller's memory directly
constexpr size_t kHostBlock = 256 + kHostRead;  // the error flags, then the data
constexpr int kHostBlocks = 16;
std::mutex host_blocks_lock;
unsigned char* host_slab = nullptr;
bool host_tried = false, host_taken[kHostBlocks] = {};

unsigned char* take_host_block() {
  std::lock_guard<std::mutex> hold(host_blocks_lock);
  if (!host_tried) {
    host_tried = true;
    if (cudaHostAlloc((void**)&host_slab, kHostBlock * kHostBlocks, cudaHostAllocPortable) != cudaSuccess) {
      host_slab = nullptr;
      cudaGetLastError();
    }
  }
  for (int k = 0; host_slab && k < kHostBlocks; ++k)
    if (!host_taken[k]) {
      host_taken[k] = true;
      return host_slab + k * kHostBlock;
    }
  return nullptr;
}

void give_host_block(unsigned char* b) {
  if (!b) return;
  std::lock_guard<std::mutex> hold(host_blocks_lock);
  host_taken[(size_t)(b - host_slab) / kHostBlock] = false;
}

// A node's corners (CSR, ascending 3 * triangle + corner) and the rest shape,
// kept where a step may be laid out after fw_finalize.
struct HostLists {
  std::vector<int32_t> off, slot;
  std::vector<float2> x0;
};

struct fw_ctx {
  unsigned char* host = nullptr;  // a page-locked block (kHostBlock), or null
  int device = 0;
  std::string err;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  bool finalized = false;
  int64_t launches = 0;
  // host staging
  int N = 0, E = 0, B = 0, S = 0;
  std::vector<float> h_x, h_v, h_bcv;
  std::vector<int32_t> h_bc;
  std::vector<int32_t> h_conn, h_type;
  std::vector<float> h_E, h_nu, h_rho, h_sy, h_H;
  std::vector<int32_t> h_noff, h_ncnt, h_eoff, h_ecnt, h_scene, h_bnoff, h_bncnt, h_bnodes;
  std::vector<float> h_damp;
  std::vector<Pair> h_pairs;
  std::vector<float> h_heights;
  std::vector<int8_t> h_occ;
  std::vector<float> cur_dt;
  std::vector<int32_t> cur_active;
  Dev d{};
  std::vector<void*> allocs;
  // captured step graphs, keyed by (uniform flag, substeps, dt bits); the
  // adjoint's recompute / reverse graphs, keyed by (kind, substeps, dt bits)
  std::vector<std::pair<uint64_t, cudaGraphExec_t>> graphs;
  std::vector<std::pair<uint64_t, cudaGraphExec_t>> adj_graphs;
  cudaStream_t graph_stream = nullptr;
  int grid_e = 1, grid_n = 1;
  int block_e = kBlock, block_n = kBlock, grid_e_cap = 0, sms = 148;
  // snapshots: device copies of the full step state, one set per slot
  struct Snap {
    float2 *x = nullptr, *v = nullptr;
    float4* j2 = nullptr;
    int32_t *counter = nullptr, *ring = nullptr, *mode_req = nullptr;
    int64_t host_counter = 0;
    bool valid = false;
  };
  std::vector<Snap> snaps;
  // ---- arena (serving): fixed capacity, scenes inserted / removed at run time
  struct FreeList {
    std::map<int64_t, int64_t> free;  // start -> length, coalesced
    void init(int64_t cap) { free.clear(); if (cap > 0) free[0] = cap; }
    bool take(int64_t len, int64_t* off) {
      if (len == 0) { *off = 0; return true; }
      for (auto it = free.begin(); it != free.end(); ++it)
        if (it->second >= len) {
          *off = it->first;
          const int64_t rest = it->second - len, start = it->first + len;
          free.erase(it);
          if (rest) free[start] = rest;
          return true;
        }
      return false;
    }
    void give(int64_t off, int64_t len) {
      if (len == 0) return;
      auto it = free.emplace(off, len).first;
      auto nx = std::next(it);
      if (nx != free.end() && it->first + it->second == nx->first) { it->second += nx->second; free.erase(nx); }
      if (it != free.begin()) {
        auto pv = std::prev(it);
        if (pv->first + pv->second == it->first) { pv->second += it->second; free.erase(it); }
      }
    }
    int64_t total() const { int64_t t = 0; for (auto& f : free) t += f.second; return t; }
  };
  struct ArenaScene {
    bool live = false;
    int64_t n0 = 0, nn = 0, e0 = 0, ne = 0, b0 = 0, nb = 0, p0 = 0, np = 0, h0 = 0, nh = 0, o0 = 0, no = 0;
    // stream arenas: patches, halo nodes, patch triangles, corner-list offsets
    int64_t pp0 = 0, npp = 0, hh0 = 0, nhh = 0, t0 = 0, nt = 0, cp0 = 0, ncp = 0;
    // ... and, where it fits a cluster, its cluster patches and their bytes
    CluLaunch clu{};
    int64_t cq0 = 0, ncq = 0, cb0 = 0, ncb = 0;
  };
  bool arena = false;
  FreeList fl_nodes, fl_elems, fl_bodies, fl_pairs, fl_heights, fl_occ;
  // stream arenas (fw_set_path(FW_PATH_STREAM) before fw_arena_init): the
  // records of each committed scene's patches; owned-node records use the
  // scene's node range and corner lists its 3 x triangle range
  bool a_stream = false;
  FreeList fl_patch, fl_halo, fl_ptri, fl_csrp, fl_cpatch, fl_cblob;
  int64_t st_ptri_cap = 0;  // patch triangles the arena holds
  int64_t occ_cap = 0;      // voxel cells the arena holds
  bool vox_asked = false;   // their table has been asked for
  CluPatch* d_cpatch = nullptr;
  unsigned char* d_cblob = nullptr;
  CluScene* d_cscene = nullptr;  // the scenes of a call, in launch order
  bool clu_size_ok[kCluMaxCtas + 1] = {};  // cluster sizes the device can hold
  bool arena_clu = true;                   // the arena's lists leave out the scenes that are stepped on chip
  size_t clu_cap = 0;
  int32_t* d_plist = nullptr;     // the active scenes' patches (CTA -> patch)
  int32_t* d_budget = nullptr;    // fw_step_served_budget: per-scene substep budgets
  int32_t* d_budget2 = nullptr;   // ... of the second segment
  float* d_dt2 = nullptr;         // ... and its step sizes
  std::vector<int32_t> h_budget, h_budget2;
  std::vector<float> h_dt2;
  unsigned char* d_stage = nullptr;  // device staging buffer of fw_arena_commit_pack
  size_t stage_cap = 0;
  int32_t* d_slist = nullptr;     // the active scenes (k_control_scenes)
  int4* d_srng = nullptr;         // per scene: first body, bodies, first pair, pairs
  std::vector<int32_t> h_slist;
  int st_slist_n = 0;
  std::vector<int32_t> h_plist;
  int st_list_n = 0;
  std::vector<ArenaScene> ascenes;
  std::vector<int> free_scene_ids;
  std::vector<int32_t> a_body_scene;
  bool chunks_dirty = true;
  std::vector<int2> h_echunks, h_nchunks;
  int2 *d_echunks = nullptr, *d_nchunks = nullptr;
  int64_t chunk_cap = 0;
  float *a_young = nullptr, *a_poisson = nullptr, *a_rho = nullptr;
  // differentiable form
  Adj adj{};
  int adj_cap = 0;  // steps per segment the trajectory buffer holds
  Tan tan{};
  // stream path (FW_PATH_STREAM)
  StreamDev sd{};
  int st_P = 0;
  size_t st_smem = 0;
  float2* x_buf0 = nullptr;  // the position buffer allocated first (parity of the swaps)
  int st_ne = 0, st_no = 0;  // patch triangles and owned nodes (record counts)
  int st_nodes = kStreamNodes;  // FW_OPT_STREAM_PATCH: owned nodes per patch = threads per CTA
  int st_minb = 32;             // FW_OPT_STREAM_MINB: CTAs per SM the kernel's registers are budgeted for
  int st_bulk = 0;              // FW_OPT_STREAM_BULK: stage triangle records with one bulk copy
  size_t st_smem_bulk = 0;
  // cluster-resident scenes (fw_cluster.cuh): the launches that step them, by cluster size and patch size; the
  // other scenes' patches and ids (stream worlds)
  struct CluGroup {
    CluLaunch r{};
    int scenes = 0, threads = 0;
    size_t smem = 0;
  };
  int clu_opt = 1;          // FW_OPT_CLUSTER
  bool shape_asked = false;  // a launch shape of the resident or stream step was set explicitly: that step runs
  std::vector<CluGroup> clu;
  std::vector<CluScene> clu_scenes;
  int* d_flags = nullptr;  // the steps' error flags, one word each, read in one copy: enum Flag
  enum Flag { kFlagFlex, kFlagRigid, kFlagStream, kFlagCluster, kFlagResident, kFlags };
  uint64_t short_key = 0;   // the last gather call of two or three substeps (launch_singly)
  bool flags_due = false;   // launches whose waits may give up, since the flags were last found clear
  bool flags_kept = false;  // ... and one of them went into a caller's graph, which may run at any time
  uint32_t clu_epoch = 0;  // grid form: tags used so far
  std::vector<int32_t> rest_scenes;  // stream worlds: scenes too large for a cluster
  int32_t* d_rest_scenes = nullptr;
  int4* d_rest_rng = nullptr;
  int rest_patches = 0;
  CluRun* d_runs = nullptr;  // fw_step_runs: every scene's runs, in the groups' order
  std::vector<int> clu_order;  // the scenes in the groups' order
  int clu_patches = 0;
  int64_t clu_wide = 0;  // CTAs of the scenes' wide clusters (clu_min_steps)
  uint64_t clu_last_key = 0;
  HostLists lists;
  std::vector<cudaStream_t> side_streams;  // the groups after the first run beside it
  std::vector<cudaEvent_t> side_events;
  CluAdj clu_adj{};                // the reverse pass on the grid form's patches (k_cluster_adj); words null: not used
  int clu_adj_threads = 0;
  uint32_t clu_adj_epoch = 0;
  size_t clu_adj_smem = 0;
  bool res_adj = false;            // the reverse pass runs resident (k_res_adj)
  size_t res_adj_smem = 0;
  unsigned long long* fll = nullptr;  // [2][N][4] flag-in-data force adjoints of the reverse pass
  float* d_poisson = nullptr;
  // path selection and the resident (shared-memory) step
  int path_req = FW_PATH_AUTO, patches_req = 0;
  int front_warps = 6;
  int res_threads = 512;     // FW_OPT_RES_THREADS
  int res_sync = 0;          // FW_OPT_RES_SYNC
  int64_t wait_limit = 0;    // FW_OPT_WAIT_LIMIT (0: the built-in limits)
  int withhold_cta = -1;     // FW_OPT_TEST_WITHHOLD
  // fw_energy scratch (plain cudaMalloc, freed in fw_destroy)
  EnergyChunk* d_echunk = nullptr;
  double4* d_epart = nullptr;
  int* d_efirst = nullptr;
  double4* d_eout = nullptr;
  size_t energy_cap = 0, energy_gcap = 0;
  int energy_chunks = 0, energy_groups = 0;
  bool energy_dirty = true;  // the chunks on the device are not those of the present scenes
  bool res_ll = false;       // resident path uses flag-in-data words
  uint32_t res_epoch = 1;    // epoch base of the next resident launch
  int path = FW_PATH_GATHER;
  Res res{};
  size_t res_smem = 0;
  std::string res_reason;
  int64_t host_counter = 0;  // step counter of scene 0 (single-scene worlds)
  // FEM-FEM contact (fw_flex.cuh): staging, then the device state
  std::vector<int2> h_be;                   // boundary edges, global node ids
  std::vector<int32_t> h_be_off, h_be_cnt;  // per body
  struct FlexPair {
    int b1, b2;
    float pen, fric;
    int tied;
  };
  std::vector<FlexPair> h_flex;
  struct FlexSceneHost {
    int skip_bvh = 0;
    std::vector<int32_t> dom_obj, dom_body;
    std::vector<float4> dom_box;
  };
  std::map<int, FlexSceneHost> h_flex_scene;  // scene -> its domains (fw_set_flex_scene)
  std::vector<int> flex_scene_of;              // per FEM-FEM scene (kernel order): the scene
  bool has_flex = false;
  FlexDev fx{};
  size_t flex_pre_smem = 0;  // k_flex_pre: (domains + FEM bodies) boxes
  std::vector<double> flex_clock;  // per FEM-FEM scene: the float64 substep dt (host copy)
  double flex_clock_all = 0.0;     // fw_set_flex_clock before fw_finalize
  double* d_flex_clock = nullptr;
  int32_t* cfl_ord_buf = nullptr;  // CFL monitor (fw_set_cfl_monitor)
  float* cfl_coef_buf = nullptr;
  // spring-mass domains: per body its node mass (0: an FEM body)
  std::vector<float> h_spring_mass;
  bool has_springs = false;
  // rigid primitives (fw_rigid.cuh): staging, then the device state
  std::vector<Rigid> h_rigid;
  std::vector<float4> h_gbox;
  std::vector<int> h_gkind, h_gscene;
  bool rigid_set = false, has_rigid = false;
  RigidDev rd{};
  fw::RigidClock* d_rclock = nullptr;
};

namespace {

int fail(fw_ctx* c, int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  if (c) c->err = buf;
  return code;
}

// On failure the runtime's last-error state is cleared too, so that a later
// launch check of this or another context does not report a stale error.
#define FW_CUDA(ctx, call)                                                                 \
  do {                                                                                     \
    cudaError_t _e = (call);                                                               \
    if (_e != cudaSuccess) {                                                               \
      cudaGetLastError();                                                                  \
      return fail((ctx), _e == cudaErrorMemoryAllocation ? FW_ERR_OOM : FW_ERR_CUDA,       \
                  "%s failed: %s (%s:%d)", #call, cudaGetErrorString(_e), __FILE__, __LINE__); \
    }                                                                                      \
  } while (0)

template <typename T>
int dalloc(fw_ctx* c, T** p, size_t count) {
  size_t bytes = sizeof(T) * (count ? count : 1);
  cudaError_t e = cudaMalloc((void**)p, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(c, FW_ERR_OOM, "cudaMalloc(%zu bytes) failed: %s", bytes, cudaGetErrorString(e));
  }
  c->allocs.push_back((void*)*p);
  return FW_OK;
}

// Device memory that a world gets faster with but does without: false (and a
// null *p) where there is none.
template <typename T>
bool dalloc_spare(fw_ctx* c, T** p, size_t count) {
  const std::string err = c->err;
  if (dalloc(c, p, count) == FW_OK) return true;
  c->err = err;
  *p = nullptr;
  return false;
}

// Gives back what was allocated after the first `mark` allocations.
void dfree_from(fw_ctx* c, size_t mark) {
  cudaStreamSynchronize(c->stream);  // copies into it may be on their way
  for (; c->allocs.size() > mark; c->allocs.pop_back()) cudaFree(c->allocs.back());
}

int alloc_flags(fw_ctx* c) {
  if (c->d_flags) return FW_OK;
  cudaError_t e = cudaMalloc((void**)&c->d_flags, sizeof(int) * fw_ctx::kFlags);
  if (e != cudaSuccess) return fail(c, FW_ERR_OOM, "cudaMalloc of the error flags failed: %s", cudaGetErrorString(e));
  c->allocs.push_back(c->d_flags);
  FW_CUDA(c, cudaMemsetAsync(c->d_flags, 0, sizeof(int) * fw_ctx::kFlags, c->stream));
  return FW_OK;
}

template <typename T>
int upload(fw_ctx* c, T** p, const std::vector<T>& h) {
  int rc = dalloc(c, p, h.size());
  if (rc) return rc;
  if (!h.empty())
    FW_CUDA(c, cudaMemcpyAsync(*p, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice, c->stream));
  return FW_OK;
}

int check_kernel(fw_ctx* c, const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(c, FW_ERR_CUDA, "%s launch failed: %s", what, cudaGetErrorString(e));
  return FW_OK;
}

void set_grids(fw_ctx* c) {
  const int E = c->E > 0 ? c->E : 1, N = c->N > 0 ? c->N : 1;
  const int cap = c->grid_e_cap > 0 ? c->grid_e_cap : c->sms * 8;
  c->grid_e = std::max(1, std::min((E + c->block_e - 1) / c->block_e, cap));
  c->grid_n = std::max(1, (N + c->block_n - 1) / c->block_n);
}

// The FEM-FEM contact of one substep (force: the construction-time hash
// build only): k_flex_pre, then k_flex_contact.  Worlds without rigid bodies
// have the element step in the first and the step control in the second.
void flex_launch(fw_ctx* c, int force) {
  const FlexDev& f = c->fx;
  const int with_step = force || c->has_rigid ? 0 : 1;
  const int cb = with_step ? (c->S + f.n_fs - 1) / f.n_fs : 0;  // blocks of step control per row
  const int eb = with_step ? std::max(1, std::min((c->E + 127) / 128, std::max(c->sms - f.n_fs, (c->E + 2047) / 2048))) : 0;
  k_flex_pre<<<f.n_fs + eb, kFlexScanThreads, c->flex_pre_smem, c->stream>>>(c->d, f, force);
  c->launches += 1;
  if (!force) {
    const int64_t threads = (int64_t)f.n_items * kFlexLanes;
    const int64_t want = (threads + kFlexContactThreads - 1) / kFlexContactThreads;
    const int bx = (int)std::max<int64_t>(1, std::min<int64_t>(want, 8 * c->sms) / f.n_fs);
    k_flex_contact<<<dim3(bx + cb, f.n_fs), kFlexContactThreads, 0, c->stream>>>(c->d, f, cb);
    c->launches += 1;
  }
}

// Kernel launches of one gather-path substep.
int step_launches(const fw_ctx* c) { return c->has_flex ? (c->has_rigid ? 4 : 3) : 2; }

int launch_step(fw_ctx* c) {
  if (c->has_flex) flex_launch(c, 0);
  if (c->has_rigid) {
    // the element step plus one thread per FEM-rigid work item
    const int rb = std::max(1, std::min((c->d.n_ritems + c->block_e - 1) / c->block_e, c->sms * 8));
    k_elements_rigid<<<1 + c->grid_e + rb, c->block_e, 0, c->stream>>>(c->d, c->grid_e);
    const int wb = c->block_n / 32, gb = (c->rd.n + wb - 1) / wb;  // blocks of the rigid side
    if (c->has_flex)
      k_nodes_rigid<true><<<c->grid_n + gb, c->block_n, 0, c->stream>>>(c->d, c->rd, gb);
    else
      k_nodes_rigid<false><<<c->grid_n + gb, c->block_n, 0, c->stream>>>(c->d, c->rd, gb);
  } else if (c->has_flex) {
    k_nodes_flex<<<c->grid_n, c->block_n, 0, c->stream>>>(c->d);
  } else {
    k_elements<<<c->grid_e, c->block_e, 0, c->stream>>>(c->d);
    k_nodes<<<c->grid_n, c->block_n, 0, c->stream>>>(c->d);
  }
  c->launches += c->has_flex && !c->has_rigid ? 1 : 2;
  return check_kernel(c, "step");
}

void drop_graphs(fw_ctx* c) {
  for (auto& g : c->graphs) cudaGraphExecDestroy(g.second);
  c->graphs.clear();
  for (auto& g : c->adj_graphs) cudaGraphExecDestroy(g.second);
  c->adj_graphs.clear();
}

// A graph of the work `body` queues on the context stream, cached under key
// in cache.  A graph holds the world descriptor and buffer addresses it was
// captured with, so caches are dropped when those change.
template <class Body>
int cached_graph(fw_ctx* c, std::vector<std::pair<uint64_t, cudaGraphExec_t>>& cache, uint64_t key, Body body,
                 cudaGraphExec_t* out) {
  if (c->graph_stream != c->stream) {
    drop_graphs(c);
    c->graph_stream = c->stream;
  }
  for (auto& g : cache)
    if (g.first == key) {
      *out = g.second;
      return FW_OK;
    }
  if (cache.size() >= 16) {
    for (auto& g : cache) cudaGraphExecDestroy(g.second);
    cache.clear();
  }
  cudaGraph_t g = nullptr;
  FW_CUDA(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
  body();
  cudaError_t ce = cudaStreamEndCapture(c->stream, &g);
  if (ce != cudaSuccess) return fail(c, FW_ERR_CUDA, "graph capture failed: %s", cudaGetErrorString(ce));
  cudaGraphExec_t exec = nullptr;
  ce = cudaGraphInstantiate(&exec, g, 0);
  cudaGraphDestroy(g);
  if (ce != cudaSuccess) return fail(c, FW_ERR_CUDA, "graph instantiate failed: %s", cudaGetErrorString(ce));
  cache.push_back({key, exec});
  *out = exec;
  return FW_OK;
}

uint32_t float_bits(float v) {
  uint32_t bits;
  memcpy(&bits, &v, sizeof(bits));
  return bits;
}

uint64_t graph_key(const fw_ctx* c, int n) {
  return ((uint64_t)(c->d.uniform_dt ? 1 : 0) << 63) | ((uint64_t)n << 32) |
         (c->d.uniform_dt ? float_bits(c->d.dt_uniform) : 0u);
}

// Two or three substeps at a step size that neither a graph nor the last such
// call has: launched one by one, since making a graph costs more than it gives
// once (a call of 2 with a new step size each time and its synchronisation, 2048
// triangles: 90 us with a graph made for it, 33 without; a repeated one 23).
bool launch_singly(fw_ctx* c, int n) {
  if (n > 3) return false;
  const uint64_t key = graph_key(c, n);
  const bool again = key == c->short_key;
  c->short_key = key;
  if (again) return false;
  if (c->graph_stream == c->stream)
    for (const auto& g : c->graphs)
      if (g.first == key) return false;
  return true;
}

// Graph of n substeps (n <= kGraphSteps) of the gather step.
int get_graph(fw_ctx* c, int n, cudaGraphExec_t* out) {
  const uint64_t key = graph_key(c, n);
  const int64_t before = c->launches;
  const int rc = cached_graph(c, c->graphs, key, [&] {
    for (int k = 0; k < n; ++k) launch_step(c);  // every launch of a substep, FEM-FEM contact included
  }, out);
  c->launches = before;  // counted when the graph is launched
  return rc;
}

int launch_resident(fw_ctx* c, int n);

int rebuild_chunks(fw_ctx* c);

int stream_steps(fw_ctx* c, int n);

int arena_stream_steps(fw_ctx* c, int n);

int launch_cluster(fw_ctx* c, int n, const float2* x_in, float2* x_out, const float4* j2_in, float4* j2_out,
                   const CluRun* runs = nullptr, bool direct = false);
int arena_cluster_steps(fw_ctx* c, int n);

int build_resident(fw_ctx* c, const std::vector<int32_t>& off, const std::vector<int32_t>& slot,
                   const std::vector<float2>& x0, bool has_j2);

int run_steps(fw_ctx* c, int n) {
  int rc = FW_OK;
  if (c->arena && c->a_stream) return arena_stream_steps(c, n);
  if (c->arena && (rc = rebuild_chunks(c))) return rc;
  if (c->path == FW_PATH_RESIDENT && c->d.uniform_dt && (c->clu.empty() || n >= grid_min_steps(c->sms, c->E)))
    return launch_resident(c, n);
  if (c->path == FW_PATH_STREAM) return stream_steps(c, n);
  c->host_counter += n;
  if (n >= kGraphSteps) {
    cudaGraphExec_t g = nullptr;
    rc = get_graph(c, kGraphSteps, &g);
    if (rc) return rc;
    while (n >= kGraphSteps) {
      FW_CUDA(c, cudaGraphLaunch(g, c->stream));
      c->launches += step_launches(c) * kGraphSteps;
      n -= kGraphSteps;
    }
  }
  if (n >= 2 && !launch_singly(c, n)) {  // the remainder as one graph too
    cudaGraphExec_t g = nullptr;
    if ((rc = get_graph(c, n, &g))) return rc;
    FW_CUDA(c, cudaGraphLaunch(g, c->stream));
    c->launches += step_launches(c) * n;
    n = 0;
  }
  for (int k = 0; k < n && rc == FW_OK; ++k) rc = launch_step(c);
  return rc;
}


using StreamKernel = void (*)(Dev, StreamDev, const float2*, float2*, const float4*, float4*);

// The stream kernel of a launch shape (patch size, register budget, staging);
// nullptr for a shape that is not built.
StreamKernel stream_kernel(int nodes, int minb, int bulk) {
  if (nodes == 64 && minb == 32) return bulk ? k_stream<64, 32, true> : k_stream<64, 32, false>;
  if (nodes == 64 && minb == 16) return bulk ? k_stream<64, 16, true> : k_stream<64, 16, false>;
  if (nodes == 128 && minb == 16) return bulk ? k_stream<128, 16, true> : k_stream<128, 16, false>;
  if (nodes == 128 && minb == 8) return bulk ? k_stream<128, 8, true> : k_stream<128, 8, false>;
  // intermediate register budgets (40 and 48 registers), per-thread record loads only
  if (!bulk && nodes == 64 && minb == 24) return k_stream<64, 24, false>;
  if (!bulk && nodes == 64 && minb == 20) return k_stream<64, 20, false>;
  if (!bulk && nodes == 128 && minb == 12) return k_stream<128, 12, false>;
  if (!bulk && nodes == 128 && minb == 10) return k_stream<128, 10, false>;
  return nullptr;
}

// n substeps of the stream path: k_control + k_stream each, alternating the
// position / J2 buffers; graphs of up to kGraphSteps substeps, cached per
// (starting buffer, dt mode, dt, count).
int stream_steps(fw_ctx* c, int n) {
  c->host_counter += n;
  const bool clu = !c->clu.empty() && n >= clu_min_steps(c->sms, c->E, c->clu_wide);
  StreamDev sd = c->sd;
  if (!clu) sd.list = nullptr;
  if (clu) {
    // the scenes that fit on clusters in one go; the rest below, in buffers that end where this leaves the state
    const bool moved = !c->rest_scenes.empty() && (n & 1);
    const int rc = launch_cluster(c, n, c->d.x, moved ? c->d.x_alt : c->d.x, c->d.j2state,
                                  moved ? c->d.j2_alt : c->d.j2state);
    if (rc || c->rest_scenes.empty()) return rc;
  }
  while (n > 0) {
    const int m = std::min(n, kGraphSteps);
    const uint64_t parity = c->d.x == c->x_buf0 ? 0 : 1;
    const uint64_t key = (1ull << 62) | (parity << 61) | ((uint64_t)(c->d.uniform_dt ? 1 : 0) << 60) |
                         ((uint64_t)(clu ? 1 : 0) << 59) | ((uint64_t)m << 32) |
                         (c->d.uniform_dt ? float_bits(c->d.dt_uniform) : 0u);
    cudaGraphExec_t g = nullptr;
    int rc = cached_graph(c, c->graphs, key, [&] {
      float2 *xa = c->d.x, *xb = c->d.x_alt;
      float4 *ja = c->d.j2state, *jb = c->d.j2_alt;
      for (int k = 0; k < m; ++k) {
        const int nr = (int)c->rest_scenes.size();
        if (clu)
          k_control_scenes<<<(nr + 127) / 128, 128, 0, c->stream>>>(c->d, c->d_rest_scenes, nr, c->d_rest_rng);
        else
          k_control<<<1, kMaxBlock, 0, c->stream>>>(c->d);
        // the patch step as a programmatic dependent of the control (see k_stream)
        cudaLaunchAttribute pdl[1];
        pdl[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        pdl[0].val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(clu ? c->rest_patches : c->st_P);
        cfg.blockDim = dim3(c->st_nodes);
        cfg.dynamicSmemBytes = c->st_bulk ? c->st_smem_bulk : c->st_smem;
        cfg.stream = c->stream;
        cfg.attrs = pdl;
        cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, stream_kernel(c->st_nodes, c->st_minb, c->st_bulk), c->d, sd,
                           (const float2*)xa, xb, (const float4*)ja, jb);
        std::swap(xa, xb);
        std::swap(ja, jb);
      }
    }, &g);
    if (rc) return rc;
    FW_CUDA(c, cudaGraphLaunch(g, c->stream));
    c->launches += 2 * m;
    if (m & 1) {
      std::swap(c->d.x, c->d.x_alt);
      std::swap(c->d.j2state, c->d.j2_alt);
    }
    n -= m;
  }
  return check_kernel(c, "stream step");
}

void rcb(const std::vector<float2>& x, std::vector<int>& idx, int lo, int hi, int p0, int np,
         std::vector<int>& part);

// Triangles of one body with different moduli (FemDomain.elementYoung): the
// stream records then keep Lame constants per triangle, not per body.
bool mixed_moduli(const fw_ctx* c) {
  for (size_t b = 0; b < c->h_noff.size(); ++b) {
    const int e0 = c->h_eoff[b];
    for (int e = e0 + 1; e < e0 + c->h_ecnt[b]; ++e)
      if (c->h_E[e] != c->h_E[e0] || c->h_nu[e] != c->h_nu[e0]) return true;
  }
  return false;
}

// (Re)build the patch-ordered records of the stream path from the element and
// node arrays (after finalize, and after a Young's modulus changes).
int stream_records(fw_ctx* c) {
  if (c->st_ne > 0)
    k_stream_elems<<<(c->st_ne + kBlock - 1) / kBlock, kBlock, 0, c->stream>>>(c->d, c->sd.eid, c->sd.conn,
                                                                               c->sd.elem, c->sd.lm, c->st_ne);
  if (c->st_no > 0)
    k_stream_nodes<<<(c->st_no + kBlock - 1) / kBlock, kBlock, 0, c->stream>>>(c->d, c->sd.nodes, c->sd.node,
                                                                               c->st_no);
  c->launches += 2;
  return check_kernel(c, "stream records");
}

// Patches of the stream path (host side, no context state): each body
// [noff[b], +ncnt[b]) of a node set cut into patches of at most patch_nodes
// nodes; per patch the owned nodes, the triangles touching them, the halo
// nodes, local connectivity and the owned nodes' corner lists in ascending
// element order.  Ids in the result are those of the input (conn / off /
// slot); a patch's scene is its first owned node's body's scene.
struct PatchSet {
  std::vector<StreamPatch> patches;
  std::vector<int32_t> rn, rh, re;  // owned nodes, halo nodes, patch triangles
  std::vector<uint2> rc;            // local corners of each patch triangle
  std::vector<uint16_t> rcp, rcs;   // corner-list offsets, corner lists
  int no_max = 1, nh_max = 1, ne_max = 1;
};

int make_patches(int N, int E, const int32_t* conn, const std::vector<int32_t>& off,
                 const std::vector<int32_t>& slot, const std::vector<float2>& x0, const std::vector<int32_t>& noff,
                 const std::vector<int32_t>& ncnt, const std::vector<int32_t>& body_scene, int patch_nodes,
                 PatchSet& out, std::string& why) {
  std::vector<int> part(N, -1), idx;
  int P = 0;
  for (size_t b = 0; b < noff.size(); ++b) {
    const int n0 = noff[b], nn = ncnt[b];
    if (nn <= 0) continue;
    const int np = (nn + patch_nodes - 1) / patch_nodes;
    idx.resize(nn);
    for (int k = 0; k < nn; ++k) idx[k] = n0 + k;
    rcb(x0, idx, 0, nn, P, np, part);
    P += np;
  }
  std::vector<std::vector<int>> owned(P);
  for (int i = 0; i < N; ++i) {
    if (part[i] < 0) {
      why = "stream path: node " + std::to_string(i) + " belongs to no body";
      return FW_ERR_ARG;
    }
    owned[part[i]].push_back(i);
  }
  std::vector<int> node_scene(N, 0), node_body(N, 0);
  for (size_t b = 0; b < noff.size(); ++b)
    for (int k = 0; k < ncnt[b]; ++k) {
      node_scene[noff[b] + k] = body_scene[b];
      node_body[noff[b] + k] = (int)b;
    }
  std::vector<StreamPatch>& patches = out.patches;
  patches.assign(P, StreamPatch{});
  std::vector<int32_t>& rn = out.rn;
  std::vector<int32_t>& rh = out.rh;
  std::vector<int32_t>& re = out.re;
  std::vector<uint2>& rc = out.rc;
  std::vector<uint16_t>& rcs = out.rcs;
  std::vector<int32_t> rcp;
  std::vector<int> loc(N, -1), eloc(E, -1);
  int no_max = 1, nh_max = 1, ne_max = 1;
  for (int p = 0; p < P; ++p) {
    const std::vector<int>& ow = owned[p];
    if ((int)ow.size() > patch_nodes) {
      why = "stream path: patch larger than " + std::to_string(patch_nodes) + " nodes";
      return FW_ERR_ARG;
    }
    std::vector<int> tri;
    for (int n : ow)
      for (int k = off[n]; k < off[n + 1]; ++k) tri.push_back(slot[k] / 3);
    std::sort(tri.begin(), tri.end());
    tri.erase(std::unique(tri.begin(), tri.end()), tri.end());
    std::vector<int> hal;
    for (int e : tri)
      for (int k = 0; k < 3; ++k) {
        const int n = conn[3 * e + k];
        if (part[n] != p) hal.push_back(n);
      }
    std::sort(hal.begin(), hal.end());
    hal.erase(std::unique(hal.begin(), hal.end()), hal.end());
    if (ow.size() + hal.size() >= 65536 || 3 * tri.size() >= 65536) {
      why = "stream path: patch too large for 16-bit local indices";
      return FW_ERR_ARG;
    }
    StreamPatch& sp = patches[p];
    sp.node_off = (int)rn.size();
    sp.no = (int)ow.size();
    sp.halo_off = (int)rh.size();
    sp.nh = (int)hal.size();
    sp.elem_off = (int)re.size();
    sp.ne = (int)tri.size();
    sp.csrp_off = (int)rcp.size();
    sp.csr_off = (int)rcs.size();
    sp.scene = node_scene[ow[0]];
    sp.body = node_body[ow[0]];
    for (int i = 0; i < sp.no; ++i) {
      loc[ow[i]] = i;
      rn.push_back(ow[i]);
    }
    for (int h = 0; h < sp.nh; ++h) {
      loc[hal[h]] = sp.no + h;
      rh.push_back(hal[h]);
    }
    for (int q = 0; q < sp.ne; ++q) {
      const int e = tri[q];
      eloc[e] = q;
      re.push_back(e);
      const uint32_t a = loc[conn[3 * e]], b = loc[conn[3 * e + 1]], cc = loc[conn[3 * e + 2]];
      const uint32_t writer = part[conn[3 * e]] == p ? 1u : 0u;
      rc.push_back(make_uint2(a | (b << 16), cc | (writer << 16)));
    }
    int cnt = 0;
    for (int i = 0; i < sp.no; ++i) {
      rcp.push_back((int32_t)cnt);
      const int n = ow[i];
      for (int k = off[n]; k < off[n + 1]; ++k) {
        rcs.push_back((uint16_t)(3 * eloc[slot[k] / 3] + slot[k] % 3));
        ++cnt;
      }
    }
    rcp.push_back((int32_t)cnt);
    if (cnt >= 65536) {
      why = "stream path: patch corner list too long";
      return FW_ERR_ARG;
    }
    for (int n : ow) loc[n] = -1;
    for (int n : hal) loc[n] = -1;
    for (int e : tri) eloc[e] = -1;
    no_max = std::max(no_max, sp.no);
    nh_max = std::max(nh_max, sp.nh);
    ne_max = std::max(ne_max, sp.ne);
  }
  out.rcp.assign(rcp.begin(), rcp.end());
  out.no_max = no_max;
  out.nh_max = nh_max;
  out.ne_max = ne_max;
  return FW_OK;
}

// Stream path of a finalized world: its patches, device arrays and records.
int build_stream(fw_ctx* c, const std::vector<int32_t>& off, const std::vector<int32_t>& slot,
                 const std::vector<float2>& x0, bool has_j2) {
  const int N = c->N, E = c->E;
  PatchSet ps;
  std::string why;
  if (make_patches(N, E, c->h_conn.data(), off, slot, x0, c->h_noff, c->h_ncnt, c->h_scene, c->st_nodes, ps, why))
    return fail(c, FW_ERR_ARG, "%s", why.c_str());
  const int P = (int)ps.patches.size();
  const std::vector<StreamPatch>& patches = ps.patches;
  const std::vector<int32_t>&rn = ps.rn, &rh = ps.rh, &re = ps.re;
  const std::vector<uint2>& rc = ps.rc;
  const std::vector<uint16_t>& rcs = ps.rcs;
  const int no_max = ps.no_max, nh_max = ps.nh_max, ne_max = ps.ne_max;
  const std::vector<uint16_t>& rcp16 = ps.rcp;
  int r;
  StreamPatch* dp = nullptr;
  int32_t *dn = nullptr, *dh = nullptr, *de = nullptr;
  uint2* dc = nullptr;
  uint16_t *dcp = nullptr, *dcs = nullptr;
  if ((r = upload(c, &dp, patches)) || (r = upload(c, &dn, rn)) || (r = upload(c, &dh, rh)) ||
      (r = upload(c, &de, re)) || (r = upload(c, &dc, rc)) || (r = upload(c, &dcp, rcp16)) ||
      (r = upload(c, &dcs, rcs)) || (r = dalloc(c, &c->d.x_alt, N)) ||
      (r = dalloc(c, &c->d.j2_alt, has_j2 ? E : 1)))
    return r;
  FW_CUDA(c, cudaMemcpyAsync(c->d.x_alt, c->d.x, sizeof(float2) * N, cudaMemcpyDeviceToDevice, c->stream));
  if (has_j2)
    FW_CUDA(c, cudaMemcpyAsync(c->d.j2_alt, c->d.j2state, sizeof(float4) * E, cudaMemcpyDeviceToDevice, c->stream));
  StreamElem* dse = nullptr;
  StreamNode* dsn = nullptr;
  if ((r = dalloc(c, &dse, re.size())) || (r = dalloc(c, &dsn, rn.size()))) return r;
  c->sd = StreamDev{dp, dn, dh, de, dc, dcp, dcs, no_max, nh_max, ne_max, dse, dsn, c->d_flags + fw_ctx::kFlagStream};
  c->st_ne = (int)re.size();
  c->st_no = (int)rn.size();
  if (mixed_moduli(c) && (r = dalloc(c, &c->sd.lm, (size_t)std::max(1, c->st_ne)))) return r;
  if ((r = stream_records(c))) return r;
  c->st_P = P;
  c->st_smem = sizeof(float2) * (size_t)(no_max + nh_max) + sizeof(float2) * 3 * (size_t)ne_max;
  c->st_smem_bulk = stream_rec_offset(no_max, nh_max, ne_max) + sizeof(StreamElem) * (size_t)ne_max;
  c->x_buf0 = c->d.x;
  int optin = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
  if ((long)c->st_smem > optin) return fail(c, FW_ERR_ARG, "stream path: patch needs %zu B of shared memory", c->st_smem);
  if ((long)c->st_smem_bulk > optin) c->st_bulk = 0;  // staging does not fit: plain loads
  for (int minb : {8, 10, 12, 16, 20, 24, 32})
    for (int bulk = 0; bulk < 2; ++bulk)
      if (StreamKernel k = stream_kernel(c->st_nodes, minb, bulk))
        FW_CUDA(c, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - 64));
  return FW_OK;
}

void rcb(const std::vector<float2>& x, std::vector<int>& idx, int lo, int hi, int p0, int np,
         std::vector<int>& part) {
  if (np <= 1 || hi - lo <= 1) {
    for (int k = lo; k < hi; ++k) part[idx[k]] = p0;
    return;
  }
  float mnx = 3e38f, mny = 3e38f, mxx = -3e38f, mxy = -3e38f;
  for (int k = lo; k < hi; ++k) {
    const float2 q = x[idx[k]];
    mnx = std::min(mnx, q.x); mxx = std::max(mxx, q.x);
    mny = std::min(mny, q.y); mxy = std::max(mxy, q.y);
  }
  const int axis = (mxx - mnx) >= (mxy - mny) ? 0 : 1;
  const int k1 = np / 2;
  const int mid = lo + (int)(((int64_t)(hi - lo) * k1) / np);
  std::nth_element(idx.begin() + lo, idx.begin() + mid, idx.begin() + hi, [&](int a, int b) {
    const float va = axis ? x[a].y : x[a].x, vb = axis ? x[b].y : x[b].x;
    return va < vb || (va == vb && a < b);
  });
  rcb(x, idx, lo, mid, p0, k1, part);
  rcb(x, idx, mid, hi, p0 + k1, np - k1, part);
}


// ------------------------------------------------------------------ cluster-resident scenes

// f(k) for k in [0, n) on up to `threads` host threads (this one among them; on
// fewer where no more can be made).  What f throws is thrown here, once all
// threads have ended.
template <class F>
void parallel_for(int n, int threads, F f) {
  std::atomic<int> next{0};
  std::exception_ptr thrown;
  std::mutex lock;
  auto work = [&] {
    try {
      for (int k; (k = next.fetch_add(1)) < n;) f(k);
    } catch (...) {
      std::lock_guard<std::mutex> hold(lock);
      if (!thrown) thrown = std::current_exception();
      next = n;
    }
  };
  std::vector<std::thread> pool;
  try {
    for (int k = 1; k < std::min(n, threads); ++k) pool.emplace_back(work);
  } catch (const std::exception&) {  // the threads there are take the rest
  }
  work();
  for (std::thread& th : pool) th.join();
  if (thrown) std::rethrow_exception(thrown);
}

// Threads for host work on so many nodes: a few thousand nodes are cut faster
// than a thread starts.
int host_threads(int64_t nodes) {
  return (int)std::min<int64_t>({16, std::max(1u, std::thread::hardware_concurrency()), 1 + nodes / 4096});
}

// A C entry's work, with what the C++ library throws as an error code.
template <class F>
int guarded(fw_ctx* c, F f) {
  try {
    return f();
  } catch (const std::bad_alloc&) {
    return fail(c, FW_ERR_OOM, "out of host memory");
  } catch (const std::exception& e) {
    return fail(c, FW_ERR_STATE, "%s", e.what());
  }
}

// One scene's patches for `ctas` CTAs into out / blob (ids relative to the
// scene; byte offsets relative to blob).  Returns false when the scene does not
// fit the encodings.
bool make_cluster_patches(const fw_ctx* c, const CluScene& sc, int nn, const std::vector<int32_t>& off,
                          const std::vector<int32_t>& slot, const std::vector<float2>& x0,
                          const std::vector<uint32_t>& word, int ctas, std::vector<int>& part, int threads,
                          std::vector<CluPatch>& out, std::vector<unsigned char>& blob) {
  const int32_t* conn = c->h_conn.data();
  std::vector<int> idx(nn);
  for (int k = 0; k < nn; ++k) idx[k] = sc.n0 + k;
  rcb(x0, idx, 0, nn, 0, ctas, part);
  struct Part {
    std::vector<int> owned, tri, halo;  // ascending; interior triangles first
    std::vector<unsigned char> blob;
    int n_int = 0;
  };
  std::vector<Part> parts(ctas);
  for (int i = sc.n0; i < sc.n0 + nn; ++i) parts[part[i]].owned.push_back(i);
  parallel_for(ctas, threads, [&](int p) {
    Part& q = parts[p];
    for (int n : q.owned)
      for (int k = off[n]; k < off[n + 1]; ++k) q.tri.push_back(slot[k] / 3);
    std::sort(q.tri.begin(), q.tri.end());
    q.tri.erase(std::unique(q.tri.begin(), q.tri.end()), q.tri.end());
    for (int e : q.tri)
      for (int k = 0; k < 3; ++k)
        if (part[conn[3 * e + k]] != p) q.halo.push_back(conn[3 * e + k]);
    std::sort(q.halo.begin(), q.halo.end());
    q.halo.erase(std::unique(q.halo.begin(), q.halo.end()), q.halo.end());
    q.n_int = (int)(std::stable_partition(q.tri.begin(), q.tri.end(), [&](int e) {
      return part[conn[3 * e]] == p && part[conn[3 * e + 1]] == p && part[conn[3 * e + 2]] == p;
    }) - q.tri.begin());
  });
  // per node the (patch << 24 | halo slot) that read it, as ranges of one list
  std::vector<int32_t> doff(nn + 1, 0);
  for (const Part& q : parts)
    for (int n : q.halo) doff[n - sc.n0 + 1]++;
  for (int i = 0; i < nn; ++i) doff[i + 1] += doff[i];
  std::vector<uint32_t> dest(doff[nn]);
  {
    std::vector<int32_t> fill(doff.begin(), doff.end() - 1);
    for (int p = 0; p < ctas; ++p)
      for (size_t j = 0; j < parts[p].halo.size(); ++j)
        dest[fill[parts[p].halo[j] - sc.n0]++] = ((uint32_t)p << 24) | (uint32_t)j;
  }
  out.assign(ctas, CluPatch{});
  std::atomic<bool> fits{true};
  parallel_for(ctas, threads, [&](int p) {
    Part& pt = parts[p];
    std::vector<int>& ow = pt.owned;
    // boundary nodes, then the others that neighbours read, then the rest, each group ascending
    auto first = std::stable_partition(ow.begin(), ow.end(), [&](int n) { return (word[n] & fw::NODE_BOUNDARY) != 0; });
    std::stable_partition(first, ow.end(), [&](int n) { return doff[n - sc.n0] < doff[n - sc.n0 + 1]; });
    const std::vector<int>&tri = pt.tri, &h = pt.halo;
    CluPatch& q = out[p];
    q.no = (int)ow.size();
    q.nh = (int)h.size();
    q.ne = (int)tri.size();
    q.n_int = pt.n_int;
    q.nbnd = (int)(first - ow.begin());
    q.slot_shift = q.no > 2048 ? 12 : 11;
    if (q.no > 4096 || q.nh >= (int)kCluHalo || q.no + q.nh >= 0x7FFF) {
      fits = false;
      return;
    }
    std::vector<std::pair<int, int>> order(q.no);  // node -> its place here
    for (int i = 0; i < q.no; ++i) order[i] = {ow[i], i};
    std::sort(order.begin(), order.end());
    auto local = [&](int n) {
      if (part[n] == p)
        return (uint32_t)std::lower_bound(order.begin(), order.end(), std::make_pair(n, 0))->second;
      return kCluHalo | (uint32_t)(std::lower_bound(h.begin(), h.end(), n) - h.begin());
    };
    std::vector<int32_t> gid(q.no), hid(q.nh), eid(q.ne);
    std::vector<uint32_t> info(q.no), push, pos(q.ne);
    std::vector<uint2> tr(q.ne);
    for (int i = 0; i < q.no; ++i) {
      const int n = ow[i], body = (int)(word[n] >> fw::NODE_BODY_SHIFT) - sc.body0;
      const int d0 = doff[n - sc.n0], dn = doff[n - sc.n0 + 1] - d0;
      if (dn > 7 || push.size() >= (1u << 15)) {
        fits = false;
        return;
      }
      gid[i] = n - sc.n0;
      info[i] = (word[n] & (fw::NODE_BC_MASK | fw::NODE_BOUNDARY)) | ((uint32_t)body << kCluBodyShift) |
                ((uint32_t)dn << kCluPushCntShift) | ((uint32_t)push.size() << kCluPushOffShift);
      for (int k = 0; k < dn; ++k) push.push_back(dest[d0 + k]);
      q.deg = std::max(q.deg, off[n + 1] - off[n]);
    }
    if (q.deg > (q.slot_shift == 11 ? 30 : 14) || (int64_t)(q.deg + 4) * q.no >= (int64_t)kCluNoSlot) {
      fits = false;
      return;
    }
    for (int j = 0; j < q.nh; ++j) hid[j] = h[j] - sc.n0;
    for (int k = 0; k < q.ne; ++k) {
      const int e = tri[k];
      const int* cn = conn + 3 * e;
      eid[k] = e - sc.e0;
      q.n_j2 += c->h_type[e] == fw::MAT_MISES ? 1 : 0;
      uint32_t sl[3], at[3];
      for (int m = 0; m < 3; ++m) {
        at[m] = local(cn[m]);
        sl[m] = kCluNoSlot;
        if (part[cn[m]] != p) continue;
        const int32_t *b = slot.data() + off[cn[m]], *en = slot.data() + off[cn[m] + 1];
        const int32_t* it = std::lower_bound(b, en, 3 * e + m);  // a node's corners ascend
        sl[m] = (uint32_t)(it - b) << q.slot_shift | at[m];
      }
      tr[k] = make_uint2((at[0] | (part[cn[0]] == p ? 0x8000u : 0u)) | (at[1] << 16), at[2] | (sl[0] << 16));
      pos[k] = sl[1] | (sl[2] << 16);
    }
    q.npush = (int)push.size();
    auto put = [&](const void* src, size_t bytes) {
      const int64_t o = (int64_t)pt.blob.size();
      pt.blob.resize(((size_t)o + bytes + 15) & ~(size_t)15);
      if (bytes) memcpy(pt.blob.data() + o, src, bytes);
      return o;
    };
    q.gid = put(gid.data(), 4 * gid.size());
    q.info = put(info.data(), 4 * info.size());
    q.hid = put(hid.data(), 4 * hid.size());
    q.push = put(push.data(), 4 * push.size());
    q.eid = put(eid.data(), 4 * eid.size());
    q.tri = put(tr.data(), 8 * tr.size());
    q.pos = put(pos.data(), 4 * pos.size());
  });
  if (!fits) return false;
  for (int p = 0; p < ctas; ++p) {
    const int64_t base = (int64_t)blob.size();
    for (int64_t* o : {&out[p].gid, &out[p].info, &out[p].hid, &out[p].push, &out[p].eid, &out[p].tri, &out[p].pos})
      *o += base;
    blob.insert(blob.end(), parts[p].blob.begin(), parts[p].blob.end());
  }
  return true;
}

// The maxima of a patch into a launch's.
void clu_widen(CluLaunch& r, const CluPatch& q) {
  r.no = std::max(r.no, q.no);
  r.nh = std::max(r.nh, q.nh);
  r.ne = std::max(r.ne, q.ne);
  r.deg = std::max(r.deg, q.deg);
  r.npush = std::max(r.npush, q.npush);
  r.nbnd = std::max(r.nbnd, q.nbnd);
  r.has_j2 |= q.n_j2 > 0 ? 1 : 0;
}

size_t clu_smem(CluLaunch r) { return clu_layout(r); }

// Threads of a CTA, control warps included: a control warp for the boxes and
// one per 64 boundary nodes for their contact forces, at most 4; and a thread
// per triangle where that fits a CTA (r.one), else an equal share of them.
// One scene on the whole GPU: two triangles per thread as soon as a thread each
// would leave it less than the 96 registers the substep needs (640 threads).
// 64 substeps of 36,000 to 58,000 nodes, one / two per thread: 2.95 / 2.73,
// 3.13 / 2.88, 3.16 / 2.90, 3.21 / 2.98, 3.30 / 3.08 us per substep; of 32,000
// nodes (576 threads) 2.27 / 2.69.
// Where the scenes fill the GPU (`shared`), two triangles per thread: 384
// bodies of 60 to 400 nodes ran 5.06 / 4.08 / 4.53 / 4.83 us per substep at
// 1 / 2 / 3 / 4, 256 of 100 to 20000 nodes 33.5 / 33.4 / 33.3 / 36.3.
int clu_threads(CluLaunch& r, bool shared) {
  r.ctl = r.np ? std::min(4, 1 + (r.nbnd + 63) / 64) : 1;
  const int most = kCluMaxThreads - 32 * r.ctl, work = std::max(1, std::max(r.ne, r.no));
  int rounds = (work + most - 1) / most;
  if ((shared && r.ne >= 128) || (r.grid && work + 32 * r.ctl > kCluOneThreads)) rounds = std::max(rounds, 2);
  r.one = rounds == 1 ? 1 : 0;
  return (((work + rounds - 1) / rounds + 31) / 32 + r.ctl) * 32;
}

// Does a launch of `ctas`-CTA clusters with this much shared memory fit the device?
bool clu_fits(const CluLaunch& r, int threads, size_t smem) {
  if (r.ctas == 1) return true;
  if (r.grid) {
    int per_sm = 0, sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, clu_kernel(threads, r.one, 1, r.tri_l2), threads, smem);
    cudaGetLastError();
    return e == cudaSuccess && per_sm * sms >= r.ctas;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = r.ctas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(r.ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  const cudaError_t e = cudaOccupancyMaxActiveClusters(&n, clu_kernel(threads, r.one, 0), &cfg);
  cudaGetLastError();
  return e == cudaSuccess && n >= 1;
}

// Streams and events for the groups after the first, which run beside it.
int clu_side_streams(fw_ctx* c) {
  const size_t G = c->clu.size();
  while (c->side_streams.size() + 1 < G) {
    cudaStream_t st = nullptr;
    FW_CUDA(c, cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    c->side_streams.push_back(st);
  }
  while (G > 1 && c->side_events.size() < G) {
    cudaEvent_t ev = nullptr;
    FW_CUDA(c, cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    c->side_events.push_back(ev);
  }
  return FW_OK;
}

// Shared memory a CTA may have, the kernels' attributes, and the cluster sizes
// the device can hold with that much of it.
int clu_prepare(fw_ctx* c, size_t* cap, bool* size_ok) {
  int optin = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
  *cap = (size_t)optin - kCluStatic;
  for (int grid = 0; grid < 2; ++grid)
    for (int one = 0; one < 2; ++one)
      for (int threads : {512, 1024}) {
        CluKernel k = clu_kernel(threads, one, grid);
        if (grid && !one && threads == 1024)
          FW_CUDA(c, cudaFuncSetAttribute(clu_kernel(threads, 0, 1, 1), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*cap));
        FW_CUDA(c, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*cap));
        if (!grid) FW_CUDA(c, cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
      }
  for (int k = 1; size_ok && k <= kCluMaxCtas; k *= 2) {
    CluLaunch r{};
    r.ctas = k;
    size_ok[k] = clu_fits(r, kCluMaxThreads, *cap);
  }
  return FW_OK;
}

// Cut the world's scenes for clusters where they fit, group them into
// launches, and (stream worlds) list what is left.  Leaves c->clu empty when
// nothing fits.
int build_cluster(fw_ctx* c, const std::vector<int32_t>& off, const std::vector<int32_t>& slot,
                  const std::vector<float2>& x0, const std::vector<uint32_t>& word, bool single) {
  if (!c->clu_opt || c->shape_asked) return FW_OK;
  size_t cap = 0;
  bool size_ok[kCluMaxCtas + 1] = {};
  if (int rp = clu_prepare(c, &cap, single ? nullptr : size_ok)) return rp;
  const int S = c->S;
  std::vector<CluScene> scenes(S);
  std::vector<int> nn(S, 0);
  std::vector<char> ok(S, 0);
  {  // bodies, nodes, triangles and pairs of a scene, each one contiguous range
    for (int s = 0; s < S; ++s) scenes[s].body0 = -1;
    for (int b = 0; b < c->B; ++b) {
      CluScene& sc = scenes[c->h_scene[b]];
      if (sc.body0 < 0) {
        sc = CluScene{0, c->h_scene[b], 0, c->h_noff[b], c->h_eoff[b], b, 0, 0, 0};
        ok[sc.scene] = 1;
      }
      const int s = sc.scene;
      const int ne0 = sc.e0;
      if (b != sc.body0 + sc.nb || c->h_noff[b] != sc.n0 + nn[s]) ok[s] = 0;
      if (c->h_eoff[b] < ne0) ok[s] = 0;
      sc.nb += 1;
      nn[s] += c->h_ncnt[b];
    }
    std::vector<int> cnt(c->B, 0);
    for (const Pair& p : c->h_pairs) cnt[p.body]++;
    int at = 0;
    std::vector<int> first(c->B + 1, 0);
    for (int b = 0; b < c->B; ++b) {
      first[b] = at;
      at += cnt[b];
    }
    first[c->B] = at;
    for (int s = 0; s < S; ++s) {
      if (!ok[s]) continue;
      CluScene& sc = scenes[s];
      sc.pair0 = first[sc.body0];
      sc.np = first[sc.body0 + sc.nb] - sc.pair0;
      if (sc.nb > kCluMaxBodies || sc.np > kCluMaxPairs || nn[s] <= 0) ok[s] = 0;
    }
  }
  // triangles of a patch share one material when their body's do
  std::vector<char> scene_tri(S, 0);
  for (int b = 0; b < c->B; ++b) {
    const int s = c->h_scene[b];
    if (scenes[s].nb > 1) scene_tri[s] = 1;
    const int e0 = c->h_eoff[b];
    for (int e = e0 + 1; e < e0 + c->h_ecnt[b] && !scene_tri[s]; ++e)
      if (c->h_E[e] != c->h_E[e0] || c->h_nu[e] != c->h_nu[e0] || c->h_type[e] != c->h_type[e0] ||
          c->h_sy[e] != c->h_sy[e0] || c->h_H[e] != c->h_H[e0])
        scene_tri[s] = 1;
  }
  std::vector<int> part(c->N, 0), n_tri(S, 0);
  for (int b = 0; b < c->B; ++b) n_tri[c->h_scene[b]] += c->h_ecnt[b];
  std::vector<CluPatch> patches;
  std::vector<unsigned char> blob;
  struct Made {
    int s, ctas;
    size_t smem;
    int tri, grid;
  };
  std::vector<Made> made;
  // nodes of a patch: one scene, 128 (64 to 128 run within 3% of each other on
  // meshes of 441 to 8232 nodes, 192 takes a fourth longer); many, an SM's
  // share of all nodes, as far as they fit
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
  const int want_nodes = single ? 128 : std::min(1300, std::max(128, c->N / sms));
  const bool shared = !single && (int64_t)c->E > (int64_t)sms * 900;
  // each scene by itself (disjoint ranges of part), on the host's threads
  struct Cut {
    int ctas = 0;
    size_t smem = 0;
    int kind = 0, tri_l2 = 0;
    std::vector<CluPatch> patches;
    std::vector<unsigned char> blob;
  };
  std::vector<Cut> cuts(S);
  parallel_for(S, host_threads(c->N), [&](int s) {
    if (!ok[s]) return;
    const int most = single ? sms : kCluMaxCtas;
    int ctas = single ? std::min(sms, (nn[s] + want_nodes - 1) / want_nodes) : 1;
    while (!single && ctas < most && (nn[s] + ctas - 1) / ctas > want_nodes) ctas *= 2;
    for (; ctas <= most && ctas <= nn[s]; ctas *= 2) {
      // more nodes than threads and not enough room for positions, node state,
      // corner forces and triangle records: not cut at all
      const int64_t room = (int64_t)ctas * (int64_t)cap, nodes = (int64_t)nn[s] * 32 + (int64_t)n_tri[s] * 24;
      if (nn[s] > ctas * kCluMaxThreads && (single ? nodes : nodes + (int64_t)n_tri[s] * 32) > room) continue;
      Cut& k = cuts[s];
      k.patches.clear();
      k.blob.clear();
      if (!make_cluster_patches(c, scenes[s], nn[s], off, slot, x0, word, ctas, part, S == 1 ? host_threads(nn[s]) : 1, k.patches,
                                k.blob))
        continue;
      CluLaunch r{};
      r.ctas = ctas;
      r.grid = single ? 1 : 0;
      for (const CluPatch& q : k.patches) clu_widen(r, q);
      r.nb = scenes[s].nb;
      r.np = scenes[s].np;
      r.per_tri = scene_tri[s];
      const int threads = clu_threads(r, shared);
      k.smem = clu_smem(r);
      // A mesh whose records do not fit beside its nodes leaves them in L2, read
      // once a substep: us per substep against the gather kernels, 537600
      // triangles 8.0 / 14.6, 655360 9.2 / 17.4, 798000 11.2 / 20.2 (409600,
      // the records still on chip: 5.75 / 12.7).
      if (single && k.smem > cap) {
        r.tri_l2 = 1;
        k.smem = clu_smem(r);
      }
      k.tri_l2 = r.tri_l2;
      if (k.smem > cap || !(single ? clu_fits(r, threads, k.smem) : size_ok[ctas])) continue;
      k.ctas = ctas;
      k.kind = scene_tri[s] * 2 + (r.has_j2 ? 1 : 0);
      break;
    }
  });
  for (int s = 0; s < S; ++s) {
    Cut& k = cuts[s];
    if (!k.ctas) continue;
    const int64_t base = (int64_t)blob.size();
    scenes[s].patch0 = (int)patches.size();
    for (CluPatch& q : k.patches) {
      for (int64_t* o : {&q.gid, &q.info, &q.hid, &q.push, &q.eid, &q.tri, &q.pos}) *o += base;
      patches.push_back(q);
    }
    blob.insert(blob.end(), k.blob.begin(), k.blob.end());
    made.push_back(Made{s, k.ctas, k.smem, k.kind, single ? 1 : 0});
    if (!single && k.ctas >= kCluWide) c->clu_wide += k.ctas;
  }
  if (made.empty()) return FW_OK;
  if (single && made.size() != (size_t)S) return FW_OK;
  int rc;
  int n_halo = 0;
  int n_rec = 0;
  for (CluPatch& q : patches) {
    q.halo0 = n_halo;
    n_halo += q.nh;
    q.tri0 = n_rec;
    n_rec += q.ne;
  }
  CluPatch* dp = nullptr;
  unsigned char* db = nullptr;
  if ((rc = upload(c, &dp, patches)) || (rc = upload(c, &db, blob))) return rc;
  // groups: same cluster size and, for one CTA, the same kind of triangles and
  // similar shared memory (so that small patches share an SM), largest first; a
  // scene joins while the common carve-up fits
  std::stable_sort(made.begin(), made.end(), [](const Made& a, const Made& b) {
    return a.ctas != b.ctas ? a.ctas > b.ctas : (a.ctas == 1 && a.tri != b.tri ? a.tri > b.tri : a.smem > b.smem);
  });
  std::vector<std::vector<CluScene>> lists;
  int group_tri = -1;
  size_t group_smem = 0;
  for (const Made& m : made) {
    const CluScene& sc = scenes[m.s];
    auto widened = [&](CluLaunch r) {
      for (int k = 0; k < m.ctas; ++k) clu_widen(r, patches[sc.patch0 + k]);
      r.nb = std::max(r.nb, sc.nb);
      r.np = std::max(r.np, sc.np);
      r.per_tri |= m.tri >> 1;
      clu_threads(r, shared);
      return r;
    };
    bool join = !c->clu.empty() && c->clu.back().r.ctas == m.ctas && (m.ctas > 1 || (group_tri == m.tri && 2 * m.smem > group_smem));
    if (join && clu_smem(widened(c->clu.back().r)) > cap) join = false;
    if (!join) {
      fw_ctx::CluGroup g;
      g.r.ctas = m.ctas;
      g.r.grid = m.grid;
      g.r.tri_l2 = single ? cuts[m.s].tri_l2 : 0;
      c->clu.push_back(g);
      lists.emplace_back();
      group_tri = m.tri;
      group_smem = m.smem;
    }
    c->clu.back().r = widened(c->clu.back().r);
    lists.back().push_back(sc);
    c->clu_order.push_back(m.s);
    ok[m.s] = 2;
  }
  for (size_t k = 0; k < c->clu.size(); ++k) {
    fw_ctx::CluGroup& g = c->clu[k];
    CluScene* ds = nullptr;
    if ((rc = upload(c, &ds, lists[k]))) return rc;
    g.r.scene = ds;
    g.r.patch = dp;
    g.r.blob = db;
    g.r.err = c->d_flags + fw_ctx::kFlagCluster;
    g.r.withhold_cta = -1;
    g.r.wait_limit = kCluWaitLimit;
    if (g.r.tri_l2) {
      if ((rc = dalloc(c, &g.r.gji, n_rec)) || (rc = dalloc(c, &g.r.grec, n_rec)) || (rc = dalloc(c, &g.r.glm, n_rec)) ||
          (rc = dalloc(c, &g.r.gj2, g.r.has_j2 ? n_rec : 1)))
        return rc;
    }
    if (g.r.grid) {
      g.r.n_halo = n_halo;
      const size_t nbox = 4 * (size_t)kCluBoxRing * g.r.ctas * g.r.nb;
      if ((rc = dalloc(c, &g.r.ghalo, 2 * (size_t)n_halo)) || (rc = dalloc(c, &g.r.gbox, nbox))) return rc;
      FW_CUDA(c, cudaMemsetAsync(g.r.ghalo, 0, sizeof(ulonglong2) * 2 * (size_t)n_halo, c->stream));
      FW_CUDA(c, cudaMemsetAsync(g.r.gbox, 0, sizeof(unsigned long long) * nbox, c->stream));
    }
    g.scenes = (int)lists[k].size();
    g.threads = clu_threads(g.r, shared);
    g.smem = clu_layout(g.r);
  }
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  for (int s = 0; s < S; ++s)
    if (ok[s] != 2) c->rest_scenes.push_back(s);
  if (!c->rest_scenes.empty()) {  // their patches go to the stream kernels
    std::vector<int32_t> plist;
    std::vector<int4> rng(S, make_int4(0, 0, 0, 0));
    for (int s : c->rest_scenes) {  // bodies and pairs as ranges: k_control_scenes needs them contiguous
      const CluScene& sc = scenes[s];
      if (sc.body0 < 0 || ok[s] == 0) {
        c->clu.clear();
        c->rest_scenes.clear();
        return FW_OK;
      }
      rng[s] = make_int4(sc.body0, sc.nb, sc.pair0, sc.np);
    }
    std::vector<StreamPatch> sp(c->st_P);
    FW_CUDA(c, cudaMemcpy(sp.data(), c->sd.patch, sizeof(StreamPatch) * c->st_P, cudaMemcpyDeviceToHost));
    for (int p = 0; p < c->st_P; ++p)
      if (ok[sp[p].scene] != 2) plist.push_back(p);
    int32_t* dl = nullptr;
    if ((rc = upload(c, &dl, plist)) || (rc = upload(c, &c->d_rest_scenes, c->rest_scenes)) ||
        (rc = upload(c, &c->d_rest_rng, rng)))
      return rc;
    c->sd.list = dl;
    c->rest_patches = (int)plist.size();
    FW_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  c->clu_patches = (int)patches.size();
  return clu_side_streams(c);
}

// build_cluster where there is device memory for it; else the path's own
// kernels step every scene.
int try_cluster(fw_ctx* c, const std::vector<int32_t>& off, const std::vector<int32_t>& slot,
                const std::vector<float2>& x0, const std::vector<uint32_t>& word, bool single) {
  const size_t mark = c->allocs.size();
  const std::string err = c->err;
  const int rc = build_cluster(c, off, slot, x0, word, single);
  if (rc != FW_ERR_OOM) return rc;
  dfree_from(c, mark);
  c->err = err;
  c->clu.clear();
  c->clu_order.clear();
  c->rest_scenes.clear();
  c->d_rest_scenes = nullptr;
  c->d_rest_rng = nullptr;
  c->sd.list = nullptr;
  return FW_OK;
}

// The resident patches, laid out when they are first needed (> 0: they do not fit).
int own_resident(fw_ctx* c) {
  if (c->path != FW_PATH_RESIDENT || c->res.err) return FW_OK;
  const int rc = build_resident(c, c->lists.off, c->lists.slot, c->lists.x0, c->d.has_j2 != 0);
  if (rc < 0) return rc;
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  return rc;
}

// Back to the path's own kernels for every scene.
int cluster_off(fw_ctx* c) {
  if (c->clu.empty()) return FW_OK;
  const int rc = own_resident(c);
  if (rc < 0) return rc;
  if (rc > 0) c->path = FW_PATH_GATHER;
  c->clu.clear();
  c->rest_scenes.clear();
  c->sd.list = nullptr;
  drop_graphs(c);
  return FW_OK;
}

// From here on the scenes' triangles carry their own Lame constants.
int cluster_per_tri(fw_ctx* c) {
  int optin = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
  for (fw_ctx::CluGroup& g : c->clu) {
    if (g.r.per_tri) continue;
    drop_graphs(c);  // they hold the carve-up
    g.r.per_tri = 1;
    g.smem = clu_layout(g.r);
    if (g.smem + kCluStatic > (size_t)optin || !clu_fits(g.r, g.threads, g.smem)) return cluster_off(c);
  }
  return FW_OK;
}

// Before a launch whose waits may give up (and raise a flag).
void flags_may_rise(fw_ctx* c) {
  c->flags_due = true;
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(c->stream, &st) != cudaSuccess)
    cudaGetLastError();
  else if (st != cudaStreamCaptureStatusNone)
    c->flags_kept = true;
}

// n substeps of every cluster-resident scene: the groups side by side (forked
// from the context stream and joined to it), reading x_in / j2_in and leaving
// the state in x_out / j2_out.
int launch_cluster(fw_ctx* c, int n, const float2* x_in, float2* x_out, const float4* j2_in, float4* j2_out,
                   const CluRun* runs, bool direct) {
  const size_t G = c->clu.size();
  if (G > 1 && !direct && n < (1 << 26)) {  // fork, launches and join as one graph: about 6 us of host work a group less
    const uint64_t key = (3ull << 62) | ((uint64_t)(runs ? 1 : 0) << 61) | ((uint64_t)(x_in == c->x_buf0 ? 1 : 0) << 60) |
                         ((uint64_t)(x_in == x_out ? 1 : 0) << 59) | ((uint64_t)(c->d.uniform_dt ? 1 : 0) << 58) |
                         ((uint64_t)n << 32) | (c->d.uniform_dt ? float_bits(c->d.dt_uniform) : 0u);
    const bool again = key == c->clu_last_key;
    c->clu_last_key = key;
    if (!again) return launch_cluster(c, n, x_in, x_out, j2_in, j2_out, runs, true);  // a graph pays from the second call on
    cudaGraphExec_t g = nullptr;
    int rc = FW_OK;
    const int64_t before = c->launches;
    const int rg = cached_graph(c, c->graphs, key,
                                [&] { rc = launch_cluster(c, n, x_in, x_out, j2_in, j2_out, runs, true); }, &g);
    c->launches = before;
    if (rg || rc) return rg ? rg : rc;
    FW_CUDA(c, cudaGraphLaunch(g, c->stream));
    c->launches += (int64_t)G;
    return FW_OK;
  }
  flags_may_rise(c);
  if (G > 1) FW_CUDA(c, cudaEventRecord(c->side_events[0], c->stream));
  for (size_t k = 0; k < G; ++k) {
    fw_ctx::CluGroup& g = c->clu[k];
    cudaStream_t st = k == 0 ? c->stream : c->side_streams[k - 1];
    if (k > 0) FW_CUDA(c, cudaStreamWaitEvent(st, c->side_events[0], 0));
    CluLaunch r = g.r;
    r.runs = runs;
    if (runs) runs += g.scenes;
    r.wait_limit = c->wait_limit > 0 ? c->wait_limit : kCluWaitLimit;
    r.withhold_cta = c->withhold_cta;
    if (c->res.rec_x) {
      r.rec_x = c->res.rec_x;
      r.rec_v = c->res.rec_v;
      r.rec_gates = c->res.rec_gates;
      r.rec_stride = c->res.rec_stride;
    }
    cudaLaunchAttribute at[1];
    if (r.grid) {  // every patch on an SM at once; this launch's tags follow the last one's
      at[0].id = cudaLaunchAttributeCooperative;
      at[0].val.cooperative = 1;
      if (c->clu_epoch > 0xF0000000u) {  // about to wrap: clear the words, restart
        FW_CUDA(c, cudaMemsetAsync(r.ghalo, 0, sizeof(ulonglong2) * 2 * (size_t)r.n_halo, st));
        FW_CUDA(c, cudaMemsetAsync(r.gbox, 0, sizeof(unsigned long long) * 4 * kCluBoxRing * (size_t)r.ctas * r.nb, st));
        c->clu_epoch = 0;
      }
      r.ep0 = c->clu_epoch;
      c->clu_epoch += (uint32_t)n + 2u;
    } else {
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = r.ctas;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(g.scenes * r.ctas);
    cfg.blockDim = dim3(g.threads);
    cfg.dynamicSmemBytes = g.smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = r.ctas > 1 ? 1 : 0;
    FW_CUDA(c, cudaLaunchKernelEx(&cfg, clu_kernel(g.threads, r.one, r.grid, r.tri_l2), (const Dev)c->d, (const CluLaunch)r, x_in, x_out, j2_in, j2_out, n));
    c->launches += 1;
    if (k > 0) {
      FW_CUDA(c, cudaEventRecord(c->side_events[k], st));
      FW_CUDA(c, cudaStreamWaitEvent(c->stream, c->side_events[k], 0));
    }
  }
  return check_kernel(c, "cluster step");
}

// Build the patches of the resident path; returns FW_OK, or a positive value
// (with c->res_reason) when the world does not fit and the gather path is used.
int build_resident(fw_ctx* c, const std::vector<int32_t>& off, const std::vector<int32_t>& slot,
                   const std::vector<float2>& x0, bool has_j2) {
  const int N = c->N, E = c->E;
  if (c->S != 1) { c->res_reason = "more than one scene"; return 1; }
  if ((int)c->h_pairs.size() > kResMaxPairs) { c->res_reason = "more than 64 contact pairs"; return 1; }
  int sms = 148, optin = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
  int P = c->patches_req > 0 ? c->patches_req : std::max(1, std::min(sms, (N + 127) / 128));
  if (P > N) P = N;
  if ((int64_t)N * 40 + (int64_t)E * 64 > (int64_t)P * optin) {  // node state, corner forces and triangle records alone
    c->res_reason = "patches of " + std::to_string(N / P) + " nodes do not fit in shared memory";
    return 1;
  }
  std::vector<int> idx(N), part(N, 0);
  for (int i = 0; i < N; ++i) idx[i] = i;
  rcb(x0, idx, 0, N, 0, P, part);
  std::vector<std::vector<int>> owned(P), pel(P);
  for (int i = 0; i < N; ++i) owned[part[i]].push_back(i);
  for (int e = 0; e < E; ++e) {
    int ps[3] = {part[c->h_conn[3 * e]], part[c->h_conn[3 * e + 1]], part[c->h_conn[3 * e + 2]]};
    for (int k = 0; k < 3; ++k) {
      bool dup = false;
      for (int j = 0; j < k; ++j) dup |= ps[j] == ps[k];
      if (!dup) pel[ps[k]].push_back(e);
    }
  }
  std::vector<char> exported(N, 0);
  std::vector<std::vector<int>> halo(P);
  for (int p = 0; p < P; ++p) {
    std::vector<int>& h = halo[p];
    for (int e : pel[p])
      for (int k = 0; k < 3; ++k) {
        const int n = c->h_conn[3 * e + k];
        if (part[n] != p) h.push_back(n);
      }
    std::sort(h.begin(), h.end());
    h.erase(std::unique(h.begin(), h.end()), h.end());
    for (int n : h) exported[n] = 1;
  }
  std::vector<char> body_bnd(N, 0);
  for (size_t k = 0; k < c->h_bnodes.size(); ++k) body_bnd[c->h_bnodes[k]] = 1;
  // group 1 first (read by other patches or on a body boundary), each group ascending
  for (int p = 0; p < P; ++p)
    std::stable_partition(owned[p].begin(), owned[p].end(),
                          [&](int n) { return exported[n] || body_bnd[n]; });
  std::vector<ResPatch> patches(P);
  std::vector<int32_t> rnodes, rhalo, reid, rcsrp;
  std::vector<uint2> rconn;
  std::vector<uint16_t> rcsrs;
  std::vector<int> loc(N, -1), eloc(E, -1);
  int no_max = 0, nh_max = 0, ne_max = 0, ncsr_max = 0;
  for (int p = 0; p < P; ++p) {
    ResPatch& rp = patches[p];
    const std::vector<int>& ow = owned[p];
    const std::vector<int>& h = halo[p];
    rp.node_off = (int)rnodes.size();
    rp.no = (int)ow.size();
    rp.n_g1 = 0;
    for (int n : ow) rp.n_g1 += (exported[n] || body_bnd[n]) ? 1 : 0;
    rp.halo_off = (int)rhalo.size();
    rp.nh = (int)h.size();
    if (rp.no + rp.nh >= 65536) { c->res_reason = "patch with >= 65536 nodes"; return 1; }
    for (int i = 0; i < rp.no; ++i) {
      loc[ow[i]] = i;
      rnodes.push_back(ow[i] | (exported[ow[i]] ? (int32_t)kExported : 0));
    }
    for (int j = 0; j < rp.nh; ++j) {
      loc[h[j]] = rp.no + j;
      rhalo.push_back(h[j]);
    }
    std::vector<int> inter, cut;
    for (int e : pel[p]) {
      const bool in = part[c->h_conn[3 * e]] == p && part[c->h_conn[3 * e + 1]] == p &&
                      part[c->h_conn[3 * e + 2]] == p;
      (in ? inter : cut).push_back(e);
    }
    rp.elem_off = (int)reid.size();
    rp.ne = (int)pel[p].size();
    rp.n_int = (int)inter.size();
    if (3 * rp.ne >= 65536) { c->res_reason = "patch with > 21845 triangles"; return 1; }
    int q = 0;
    for (const std::vector<int>* grp : {&inter, &cut})
      for (int e : *grp) {
        eloc[e] = q++;
        reid.push_back(e);
        const uint32_t a = loc[c->h_conn[3 * e]], b = loc[c->h_conn[3 * e + 1]], cc = loc[c->h_conn[3 * e + 2]];
        const uint32_t writer = part[c->h_conn[3 * e]] == p ? kJ2Writer : 0u;
        rconn.push_back(make_uint2(a | (b << 16), cc | (writer << 16)));
      }
    rp.csr_ptr_off = (int)rcsrp.size();
    rp.csr_off = (int)rcsrs.size();
    int cnt = 0;
    for (int i = 0; i < rp.no; ++i) {
      rcsrp.push_back(cnt);
      const int n = ow[i];
      for (int k = off[n]; k < off[n + 1]; ++k) {
        const int sl = slot[k];
        rcsrs.push_back((uint16_t)(3 * eloc[sl / 3] + sl % 3));
        ++cnt;
      }
    }
    rcsrp.push_back(cnt);
    rp.ncsr = cnt;
    for (int n : ow) loc[n] = -1;
    for (int n : h) loc[n] = -1;
    for (int e : pel[p]) eloc[e] = -1;
    no_max = std::max(no_max, rp.no);
    nh_max = std::max(nh_max, rp.nh);
    ne_max = std::max(ne_max, rp.ne);
    ncsr_max = std::max(ncsr_max, rp.ncsr);
  }
  Res& r = c->res;
  r.P = P;
  r.no_max = no_max;
  r.nh_max = nh_max;
  r.ne_max = ne_max;
  r.ncsr_max = ncsr_max;
  r.has_j2 = has_j2 ? 1 : 0;
  const size_t tab_bytes = c->h_heights.size() * sizeof(float) + c->h_occ.size();
  const bool stage = tab_bytes <= (size_t)kResTableBytes;
  r.tab_h = stage ? (int)c->h_heights.size() : 0;
  r.tab_o = stage ? (int)c->h_occ.size() : 0;
  r.n_bodies = c->B;
  if (c->B > 4096) { c->res_reason = "more than 4096 bodies"; return 1; }
  const size_t smem = res_layout(r, nullptr, nullptr);
  if ((long)smem + 64 > optin) {
    c->res_reason = "patch needs " + std::to_string(smem) + " B of shared memory";
    return 1;
  }
  const bool ll = c->res_sync == 0 && c->B <= kLLMaxBodies;
  ResKernel kern = res_kernel(c->front_warps, ll, c->res_threads);
  // The attribute is per function and process-wide: every context sets it to
  // the device maximum, so a context with small patches cannot lower the limit
  // below what another context launches with.
  cudaFuncAttributes fa{};
  cudaFuncGetAttributes(&fa, kern);
  cudaError_t e1 = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        optin - (int)fa.sharedSizeBytes);
  int per_sm = 0;
  cudaError_t e2 = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, c->res_threads, smem);
  if (e1 != cudaSuccess || e2 != cudaSuccess || per_sm * sms < P) {
    cudaGetLastError();
    c->res_reason = "patches cannot all be resident";
    return 1;
  }
  int rc;
  ResPatch* dpatch = nullptr;
  int32_t *dn = nullptr, *dh = nullptr, *de = nullptr, *dcp = nullptr;
  uint2* dc = nullptr;
  uint16_t* dcs = nullptr;
  if ((rc = upload(c, &dpatch, patches)) || (rc = upload(c, &dn, rnodes)) || (rc = upload(c, &dh, rhalo)) ||
      (rc = upload(c, &de, reid)) || (rc = upload(c, &dc, rconn)) || (rc = upload(c, &dcp, rcsrp)) ||
      (rc = upload(c, &dcs, rcsrs)) || (rc = dalloc(c, &r.xpub, 2 * (size_t)N)) ||
      (rc = dalloc(c, &r.aabb3, 12 * (size_t)c->B)) || (rc = dalloc(c, &r.bar, 1)))
    return rc;
  if (ll) {
    const size_t nbll = 4 * (size_t)kBoxRing * c->B * P;
    if ((rc = dalloc(c, &r.xll, 4 * (size_t)N)) || (rc = dalloc(c, &r.bll, nbll))) return rc;
    FW_CUDA(c, cudaMemsetAsync(r.xll, 0, sizeof(unsigned long long) * 4 * (size_t)N, c->stream));
    FW_CUDA(c, cudaMemsetAsync(r.bll, 0, sizeof(unsigned long long) * nbll, c->stream));
  }
  c->res_ll = ll;
  c->res_epoch = 1;
  r.patch = dpatch;
  r.nodes = dn;
  r.halo = dh;
  r.eid = de;
  r.conn = dc;
  r.csr_ptr = dcp;
  r.csr_slot = dcs;
  r.err = c->d_flags + fw_ctx::kFlagResident;
  c->res_smem = smem;
  return FW_OK;
}

int launch_resident(fw_ctx* c, int n) {
  // keep the arrivals counter (P * steps) far from int overflow
  constexpr int kMaxStepsPerLaunch = 1 << 20;
  while (n > kMaxStepsPerLaunch) {
    int rc = launch_resident(c, kMaxStepsPerLaunch);
    if (rc) return rc;
    n -= kMaxStepsPerLaunch;
  }
  if (n <= 0) return FW_OK;
  if (!c->clu.empty()) {
    c->host_counter += n;
    return launch_cluster(c, n, c->d.x, c->d.x, c->d.j2state, c->d.j2state);
  }
  const int step0 = (int)c->host_counter;
  const bool ll = c->res_ll;
  if (ll && c->res_epoch > 0xF0000000u) {  // epochs about to wrap: clear the words, restart
    FW_CUDA(c, cudaMemsetAsync(c->res.xll, 0, sizeof(unsigned long long) * 4 * (size_t)c->N, c->stream));
    FW_CUDA(c, cudaMemsetAsync(c->res.bll, 0, sizeof(unsigned long long) * 4 * (size_t)kBoxRing * c->B * c->res.P,
                               c->stream));
    c->res_epoch = 1;
  }
  uint32_t ep0 = c->res_epoch;
  c->res_epoch += (uint32_t)n + 1u;
  c->res.wait_limit = c->wait_limit > 0 ? c->wait_limit : (ll ? kPollLimit : kSpinLimit);
  c->res.withhold_cta = c->withhold_cta;
  flags_may_rise(c);
  k_res_prologue<<<1, 256, 0, c->stream>>>(c->d, c->res, step0, ll ? 1 : 0);
  float dt = c->d.dt_uniform, damp = c->h_damp[0];
  void* args[] = {(void*)&c->d, (void*)&c->res, (void*)&step0, (void*)&n, (void*)&dt, (void*)&damp, (void*)&ep0};
  FW_CUDA(c, cudaLaunchCooperativeKernel((const void*)res_kernel(c->front_warps, ll, c->res_threads),
                                         dim3(c->res.P), dim3(c->res_threads), args, c->res_smem, c->stream));
  if (ll)
    k_res_epilogue_ll<<<1, 256, 0, c->stream>>>(c->d, c->res, step0, n);
  else
    k_res_epilogue<<<1, 256, 0, c->stream>>>(c->d, c->res, step0, n);
  c->launches += 3;
  c->host_counter += n;
  return check_kernel(c, "resident step");
}

// The error flags of the work queued so far (waits for it).  The plain gather
// kernels raise none, whatever the world's path: a call on them alone is not
// charged with the flags' copy (7 us of a one-substep call and its
// synchronisation at 409,600 triangles, 26 us without).
bool raises_flags(const fw_ctx* c) {
  return c->has_flex || c->has_rigid || c->path == FW_PATH_STREAM || c->flags_due;
}

int report_flags(fw_ctx* c, const int* flag);

int check_device_error(fw_ctx* c) {
  if (!raises_flags(c)) return FW_OK;
  int local[fw_ctx::kFlags];
  int* flag = c->host ? (int*)c->host : local;
  FW_CUDA(c, cudaMemcpyAsync(flag, c->d_flags, sizeof(local), cudaMemcpyDeviceToHost, c->stream));
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  return report_flags(c, flag);
}

// `bytes` of device memory into pageable host memory with the error flags in
// the same trip; small reads go through the context's page-locked block, so
// that the whole is one wait (the pageable copy and the flags took one each).
int read_pageable(fw_ctx* c, void* dst, const void* src, size_t bytes) {
  const bool flags = raises_flags(c) && c->host, small = c->host && bytes <= kHostRead;
  if (flags)
    FW_CUDA(c, cudaMemcpyAsync(c->host, c->d_flags, sizeof(int) * fw_ctx::kFlags, cudaMemcpyDeviceToHost, c->stream));
  FW_CUDA(c, cudaMemcpyAsync(small ? c->host + 256 : dst, src, bytes, cudaMemcpyDeviceToHost, c->stream));
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  if (small) memcpy(dst, c->host + 256, bytes);
  return flags ? report_flags(c, (const int*)c->host) : check_device_error(c);
}

int report_flags(fw_ctx* c, const int* flag) {
  if (flag[fw_ctx::kFlagFlex] & 1)
    return fail(c, FW_ERR_ARG, "FEM-FEM contact: a node received more than %d contact forces in one substep",
                kFlexListCap);
  if (flag[fw_ctx::kFlagRigid] & 1)
    return fail(c, FW_ERR_UNSUPPORTED,
                "a rigid body came within 0.01 of a ground or of another contact rigid (rigid-rigid and "
                "rigid-ground contact, the reference's constraint solve, are outside this library), or its "
                "state is no longer finite");
  if (flag[fw_ctx::kFlagStream])
    return fail(c, FW_ERR_TIMEOUT, "stream step: a staged copy of triangle records did not complete");
  if (flag[fw_ctx::kFlagCluster]) {
    FW_CUDA(c, cudaMemsetAsync(c->d_flags + fw_ctx::kFlagCluster, 0, sizeof(int), c->stream));
    return fail(c, FW_ERR_TIMEOUT, "cluster step: a CTA gave up waiting for the others");
  }
  if (flag[fw_ctx::kFlagResident]) {
    if (!c->clu.empty() || c->path != FW_PATH_RESIDENT)  // no k_res_prologue clears it
      FW_CUDA(c, cudaMemsetAsync(c->d_flags + fw_ctx::kFlagResident, 0, sizeof(int), c->stream));
    return fail(c, FW_ERR_TIMEOUT, "resident step: a CTA gave up waiting for the others");
  }
  c->flags_due = c->flags_kept;
  return FW_OK;
}


int rebuild_chunks(fw_ctx* c) {
  if (!c->chunks_dirty) return FW_OK;
  c->h_echunks.clear();
  c->h_nchunks.clear();
  for (size_t s = 0; s < c->ascenes.size(); ++s) {
    const fw_ctx::ArenaScene& a = c->ascenes[s];
    if (!a.live || !c->cur_active[s]) continue;
    for (int64_t k = 0; k < a.ne; k += c->block_e)
      c->h_echunks.push_back(make_int2((int)(a.e0 + k), (int)std::min<int64_t>(c->block_e, a.ne - k)));
    for (int64_t k = 0; k < a.nn; k += c->block_n)
      c->h_nchunks.push_back(make_int2((int)(a.n0 + k), (int)std::min<int64_t>(c->block_n, a.nn - k)));
  }
  if ((int64_t)std::max(c->h_echunks.size(), c->h_nchunks.size()) > c->chunk_cap)
    return fail(c, FW_ERR_ARG, "arena: chunk list overflow");
  if (!c->h_echunks.empty())
    FW_CUDA(c, cudaMemcpyAsync(c->d_echunks, c->h_echunks.data(), sizeof(int2) * c->h_echunks.size(),
                               cudaMemcpyHostToDevice, c->stream));
  if (!c->h_nchunks.empty())
    FW_CUDA(c, cudaMemcpyAsync(c->d_nchunks, c->h_nchunks.data(), sizeof(int2) * c->h_nchunks.size(),
                               cudaMemcpyHostToDevice, c->stream));
  // pageable-source copies are staged before cudaMemcpyAsync returns, so the
  // host vectors may change again right away
  c->d.n_e_chunks = (int)c->h_echunks.size();
  c->d.n_n_chunks = (int)c->h_nchunks.size();
  c->grid_e = std::max(1, std::min(c->d.n_e_chunks, c->sms * 8));
  c->grid_n = std::max(1, std::min(c->d.n_n_chunks, c->sms * 8));
  drop_graphs(c);
  c->chunks_dirty = false;
  return FW_OK;
}

int set_scene_dt(fw_ctx* c, const float* dt) {
  bool same = c->cur_dt.size() == (size_t)c->S;
  for (int s = 0; same && s < c->S; ++s) same = memcmp(&c->cur_dt[s], &dt[s], sizeof(float)) == 0;
  if (same) return FW_OK;
  c->cur_dt.assign(dt, dt + c->S);
  FW_CUDA(c, cudaMemcpyAsync(c->d.scene_dt, c->cur_dt.data(), sizeof(float) * c->S,
                             cudaMemcpyHostToDevice, c->stream));
  // the copy reads c->cur_dt; keep it stable until the copy ran
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  return FW_OK;
}

// Relocation of one committed scene's arrays from scene-local to arena ids
// (fw_arena_commit_pack uploads them as packed), and the scene's control
// words (thread 0).
struct ArenaReloc {
  int n0, e0, b0, p0, h0, o0, s;
  int Ns, Es, Bs, Np;
  int32_t* rn;  // stream arenas: the scene's owned-node, halo and triangle id ranges (else null)
  int32_t* rh;
  int32_t* re;
  int Hs, Ts;
  StreamPatch* patch;  // stream arenas: the scene's patch records
  int Ps, hh0, t0, cp0;
  int4* srng;  // stream arenas: per-scene body / pair ranges
  float damp;
  int64_t count;  // max of the counts above and 3 Es
};

__global__ void k_arena_reloc(Dev d, ArenaReloc r) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid == 0) {
    d.scene_damp[r.s] = r.damp;
    d.scene_counter[r.s] = 0;
    d.scene_mode_req[r.s] = 1;  // the zero-dt construction step at the next substep it runs
    d.scene_active[r.s] = 1;
    d.scene_bad[r.s] = 0;
    if (r.srng) r.srng[r.s] = make_int4(r.b0, r.Bs, r.p0, r.Np);
  }
  for (int64_t i = tid; i < r.count; i += stride) {
    if (i < r.Ns) {
      const int64_t g = r.n0 + i;
      d.node_word[g] += (uint32_t)r.b0 << fw::NODE_BODY_SHIFT;
      d.csr_off[g] += 3 * r.e0;
      d.csr_end[g] += 3 * r.e0;
      if (r.rn) r.rn[i] += r.n0;
    }
    if (i < 3 * (int64_t)r.Es) {
      const int64_t q = 3 * (int64_t)r.e0 + i;
      d.csr_slot[q] += 3 * r.e0;
      d.corner_pos[q] += 3 * r.e0;
      d.conn[q] += r.n0;
    }
    if (i < r.Es) d.emat[r.e0 + i].word += r.b0 << 2;
    if (i < r.Bs) {
      d.body_pair_off[r.b0 + i] += r.p0;
      d.body_scene[r.b0 + i] = r.s;
    }
    if (i < r.Np) {
      Pair& pr = d.pairs[r.p0 + i];
      pr.body += r.b0;
      if (pr.kind == fw::PAIR_HEIGHTFIELD) pr.table += r.h0;
      if (pr.kind == fw::PAIR_VOXEL) pr.table += r.o0;
    }
    if (r.rh && i < r.Hs) r.rh[i] += r.n0;
    if (r.re && i < r.Ts) r.re[i] += r.e0;
    if (r.patch && i < r.Ps) {
      StreamPatch& sp = r.patch[i];
      sp.node_off += r.n0;
      sp.halo_off += r.hh0;
      sp.elem_off += r.t0;
      sp.csrp_off += r.cp0;
      sp.csr_off += 3 * r.e0;
      sp.scene = r.s;
      sp.body += r.b0;
    }
  }
}

// Parts of a pack copied from the device staging buffer to their arena
// ranges: part k = stage[off[k] .. +len[k]) -> dst[k] (blockIdx.y = part).
constexpr int kScatterParts = 29;  // the pack's parts and the rest positions again (as the current ones)
struct ArenaScatter {
  unsigned char* dst[kScatterParts];
  uint32_t off[kScatterParts];
  uint32_t len[kScatterParts];
};

__global__ void k_arena_scatter(const unsigned char* __restrict__ stage, ArenaScatter sc) {
  const int k = blockIdx.y;
  const uint32_t len = sc.len[k];
  if (!len) return;
  const unsigned char* src = stage + sc.off[k];
  unsigned char* dst = sc.dst[k];
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (((uintptr_t)dst & 3) == 0 && (len & 3) == 0) {  // the source parts are 16-byte aligned
    const uint32_t* s4 = reinterpret_cast<const uint32_t*>(src);
    uint32_t* d4 = reinterpret_cast<uint32_t*>(dst);
    for (uint32_t i = t; i < len / 4; i += stride) d4[i] = s4[i];
  } else {
    for (uint32_t i = t; i < len; i += stride) dst[i] = src[i];
  }
}

// Shared memory of a stream launch for the given patch maxima.
void stream_smem(int no_max, int nh_max, int ne_max, size_t* plain, size_t* bulk) {
  *plain = sizeof(float2) * (size_t)(no_max + nh_max) + sizeof(float2) * 3 * (size_t)ne_max;
  *bulk = stream_rec_offset(no_max, nh_max, ne_max) + sizeof(StreamElem) * (size_t)ne_max;
}

// Every built stream kernel of a patch size may use the device's opt-in shared memory.
int stream_attrs(fw_ctx* c, int optin) {
  for (int minb : {8, 10, 12, 16, 20, 24, 32})
    for (int bulk = 0; bulk < 2; ++bulk)
      if (StreamKernel k = stream_kernel(c->st_nodes, minb, bulk))
        FW_CUDA(c, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - 64));
  return FW_OK;
}

// n substeps of an arena's active scenes that have cluster patches: each through
// its own runs (its budget at its dt, then the next budget), one launch per
// cluster size.
int arena_cluster_steps(fw_ctx* c, int n) {
  struct Item {
    uint64_t key;  // cluster size, triangles of the largest patch
    int s;
    CluRun run;
  };
  std::vector<Item> items;
  int64_t tris = 0;
  for (size_t s = 0; s < c->ascenes.size(); ++s) {
    const fw_ctx::ArenaScene& a = c->ascenes[s];
    if (!a.live || !c->cur_active[s] || !a.clu.ctas) continue;
    CluRun run{};
    run.n[0] = c->d.scene_budget ? std::max(0, std::min(n, c->h_budget[s])) : n;
    run.dt[0] = c->d.uniform_dt ? c->d.dt_uniform : c->cur_dt[s];
    if (c->d.scene_budget_next) {
      run.n[1] = std::max(0, std::min(n - run.n[0], c->h_budget2[s]));
      run.dt[1] = c->h_dt2[s];
    }
    if (run.n[0] + run.n[1] == 0) continue;
    items.push_back(Item{(uint64_t)a.clu.ctas << 32 | (uint32_t)a.clu.ne, (int)s, run});
    tris += a.ne;
  }
  c->clu.clear();
  if (items.empty()) return FW_OK;
  // the largest scenes first, so that the small ones fill in behind them
  std::sort(items.begin(), items.end(),
            [](const Item& p, const Item& q) { return p.key != q.key ? p.key > q.key : p.s < q.s; });
  const bool shared = tris > (int64_t)c->sms * 900;
  std::vector<CluScene> scenes;
  std::vector<CluRun> runs;
  scenes.reserve(items.size());
  runs.reserve(items.size());
  for (const Item& it : items) {
    const fw_ctx::ArenaScene& a = c->ascenes[it.s];
    // most scenes are no larger than those before them in any respect: nothing to lay out anew
    auto within = [&](const CluLaunch& r) {
      const CluLaunch& b = a.clu;
      return b.no <= r.no && b.nh <= r.nh && b.ne <= r.ne && b.deg <= r.deg && b.npush <= r.npush && b.nbnd <= r.nbnd &&
             b.nb <= r.nb && b.np <= r.np && b.has_j2 <= r.has_j2 && b.per_tri <= r.per_tri;
    };
    auto widened = [&](CluLaunch r) {
      const CluLaunch& b = a.clu;
      r.no = std::max(r.no, b.no); r.nh = std::max(r.nh, b.nh); r.ne = std::max(r.ne, b.ne); r.deg = std::max(r.deg, b.deg);
      r.npush = std::max(r.npush, b.npush); r.nbnd = std::max(r.nbnd, b.nbnd);
      r.nb = std::max(r.nb, b.nb); r.np = std::max(r.np, b.np);
      r.has_j2 |= b.has_j2; r.per_tri |= b.per_tri;
      clu_threads(r, shared);
      return r;
    };
    bool join = !c->clu.empty() && c->clu.back().r.ctas == a.clu.ctas && 4 * a.clu.ne > c->clu.back().r.ne;
    const bool inside = join && within(c->clu.back().r);
    if (join && !inside && clu_smem(widened(c->clu.back().r)) > c->clu_cap) join = false;
    if (!join) {
      fw_ctx::CluGroup g;
      g.r.ctas = a.clu.ctas;
      c->clu.push_back(g);
    }
    fw_ctx::CluGroup& g = c->clu.back();
    if (!inside) g.r = widened(g.r);
    g.scenes += 1;
    scenes.push_back(CluScene{a.cb0, it.s, (int)a.cq0, (int)a.n0, (int)a.e0, (int)a.b0, (int)a.nb, (int)a.p0, (int)a.np});
    runs.push_back(it.run);
  }
  // staged before the calls return
  FW_CUDA(c, cudaMemcpyAsync(c->d_cscene, scenes.data(), sizeof(CluScene) * scenes.size(), cudaMemcpyHostToDevice, c->stream));
  FW_CUDA(c, cudaMemcpyAsync(c->d_runs, runs.data(), sizeof(CluRun) * runs.size(), cudaMemcpyHostToDevice, c->stream));
  const CluScene* at = c->d_cscene;
  for (fw_ctx::CluGroup& g : c->clu) {
    g.r.scene = at;
    at += g.scenes;
    g.r.patch = c->d_cpatch;
    g.r.blob = c->d_cblob;
    g.r.err = c->d_flags + fw_ctx::kFlagCluster;
    g.threads = clu_threads(g.r, shared);
    g.smem = clu_layout(g.r);
  }
  int rc = clu_side_streams(c);
  if (!rc) rc = launch_cluster(c, n, c->d.x, c->d.x, c->d.j2state, c->d.j2state, c->d_runs, true);
  c->clu.clear();
  return rc;
}

// n substeps of a stream arena: k_control + k_stream over the active scenes'
// patches each, then (n odd) the carry back into the first buffers.
int arena_stream_steps(fw_ctx* c, int n) {
  int64_t tris = 0, wide = 0, scenes = 0;
  for (size_t s = 0; n < 32 && s < c->ascenes.size(); ++s)
    if (c->ascenes[s].live && c->cur_active[s]) {
      scenes += 1;
      tris += c->ascenes[s].ne;
      wide += c->ascenes[s].clu.ctas >= kCluWide ? c->ascenes[s].clu.ctas : 0;
    }
  const bool clu = c->clu_opt && c->d_cpatch && n >= arena_min_steps(c->sms, tris, wide, scenes);
  if (clu != c->arena_clu) {  // the lists hold what is not stepped on chip
    c->arena_clu = clu;
    c->chunks_dirty = true;
  }
  if (c->chunks_dirty) {
    c->h_plist.clear();
    c->h_slist.clear();
    for (size_t s2 = 0; s2 < c->ascenes.size(); ++s2) {
      const fw_ctx::ArenaScene& a = c->ascenes[s2];
      if (!a.live || !c->cur_active[s2] || (clu && a.clu.ctas)) continue;
      c->h_slist.push_back((int32_t)s2);
      for (int64_t k = 0; k < a.npp; ++k) c->h_plist.push_back((int32_t)(a.pp0 + k));
    }
    // staged before the calls return
    if (!c->h_plist.empty())
      FW_CUDA(c, cudaMemcpyAsync(c->d_plist, c->h_plist.data(), sizeof(int32_t) * c->h_plist.size(),
                                 cudaMemcpyHostToDevice, c->stream));
    if (!c->h_slist.empty())
      FW_CUDA(c, cudaMemcpyAsync(c->d_slist, c->h_slist.data(), sizeof(int32_t) * c->h_slist.size(),
                                 cudaMemcpyHostToDevice, c->stream));
    c->st_list_n = (int)c->h_plist.size();
    c->st_slist_n = (int)c->h_slist.size();
    c->chunks_dirty = false;
  }
  c->host_counter += n;
  if (n <= 0) return FW_OK;
  if (clu)
    if (int rc = arena_cluster_steps(c, n)) return rc;
  if (c->st_list_n == 0) return FW_OK;
  float2 *xa = c->d.x, *xb = c->d.x_alt;
  float4 *ja = c->d.j2state, *jb = c->d.j2_alt;
  const StreamKernel k = stream_kernel(c->st_nodes, c->st_minb, c->st_bulk);
  const size_t smem = c->st_bulk ? c->st_smem_bulk : c->st_smem;
  const int gs = (c->st_slist_n + 127) / 128;
  // the patch step is a programmatic dependent of the control kernel (its
  // position gather overlaps the control; see k_stream)
  cudaLaunchAttribute pdl[1];
  pdl[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  pdl[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(c->st_list_n);
  cfg.blockDim = dim3(c->st_nodes);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cfg.attrs = pdl;
  cfg.numAttrs = 1;
  for (int j = 0; j < n; ++j) {
    k_control_scenes<<<gs, 128, 0, c->stream>>>(c->d, c->d_slist, c->st_slist_n, c->d_srng);
    FW_CUDA(c, cudaLaunchKernelEx(&cfg, k, c->d, c->sd, (const float2*)xa, xb, (const float4*)ja, jb));
    std::swap(xa, xb);
    std::swap(ja, jb);
  }
  c->launches += 2 * (int64_t)n;
  if (n & 1) {
    k_stream_carry<<<c->st_list_n, c->st_nodes, 0, c->stream>>>(c->sd, xa, xb, ja, jb, c->d.has_j2);
    c->launches += 1;
  }
  return check_kernel(c, "arena stream step");
}

}  // namespace

// Host image of one staged scene with ids local to the scene (fw_arena_pack):
// every array an arena holds per scene, laid out in one host block (page-
// locked when asked for, so that a commit's copies run asynchronously).
struct fw_pack {
  enum Part {
    X0, V0, BCV, WORD, CBEG, CEND, SLOT, CPOS, CONN, EMAT, J2PAR, YOUNG, POISSON, RHO, POFF, PCNT, PAIRS,
    HEIGHTS, OCC, RN, RH, RE, RC, RCP, RCS, PATCH, CPATCH, CBLOB, NPARTS
  };
  int64_t Ns = 0, Es = 0, Bs = 0, Np = 0, Nh = 0, No = 0;
  int64_t Ps = 0, Hs = 0, Ts = 0, CPs = 0;  // stream records (patch_nodes > 0)
  int patch_nodes = 0;
  int no_max = 0, nh_max = 0, ne_max = 0;
  bool mixed = false;  // a body's triangles have different moduli
  CluLaunch clu{};  // cluster size and maxima of its cluster patches (ctas 0: none)
  float damp = 0.f;
  unsigned char* block = nullptr;
  bool pinned = false;
  size_t bytes = 0;  // the block's size (parts 16-byte aligned)
  size_t off[NPARTS] = {}, len[NPARTS] = {};
  int64_t dev_bytes = 0;
  const void* at(Part p) const { return block + off[p]; }
  ~fw_pack() {
    if (pinned) cudaFreeHost(block);
    else free(block);
  }
};

namespace {

// The scene staged on context c (fw_set_nodes / fw_set_elements /
// fw_set_bodies / fw_set_scenes(1, ...) / fw_add_*_pair, ids local to the
// scene) as a pack; the stage is cleared.  Host work only.
int build_pack(fw_ctx* c, int patch_nodes, bool pinned, fw_pack** out) {
  const int64_t Ns = (int64_t)c->h_x.size() / 2, Es = (int64_t)c->h_conn.size() / 3;
  const int Bs = (int)c->h_noff.size();
  if (Ns <= 0 || Es <= 0 || Bs <= 0) return fail(c, FW_ERR_ARG, "fw_arena_pack: nothing staged");
  for (int b = 0; b < Bs; ++b)
    if (c->h_scene[b] != 0) return fail(c, FW_ERR_ARG, "fw_arena_pack: stage exactly one scene (scene 0)");
  if (patch_nodes != 0 && patch_nodes != 64 && patch_nodes != 128)
    return fail(c, FW_ERR_ARG, "fw_arena_pack: patch_nodes must be 0, 64 or 128");
  if (c->has_springs || !c->h_flex.empty() || !c->h_rigid.empty())
    return fail(c, FW_ERR_ARG, "fw_arena_pack: arena scenes hold FEM triangles and ground pairs only");
  std::vector<int32_t> node_body(Ns, -1), elem_body(Es, -1);
  for (int b = 0; b < Bs; ++b) {
    if (c->h_noff[b] < 0 || c->h_noff[b] + (int64_t)c->h_ncnt[b] > Ns || c->h_eoff[b] < 0 ||
        c->h_eoff[b] + (int64_t)c->h_ecnt[b] > Es)
      return fail(c, FW_ERR_ARG, "fw_arena_pack: body %d range out of bounds", b);
    for (int i = c->h_noff[b]; i < c->h_noff[b] + c->h_ncnt[b]; ++i) node_body[i] = b;
    for (int e = c->h_eoff[b]; e < c->h_eoff[b] + c->h_ecnt[b]; ++e) elem_body[e] = b;
  }
  for (int64_t e = 0; e < Es; ++e)
    for (int k = 0; k < 3; ++k) {
      const int n = c->h_conn[3 * e + k];
      if (elem_body[e] < 0 || n < 0 || n >= Ns || node_body[n] != elem_body[e])
        return fail(c, FW_ERR_ARG, "fw_arena_pack: element %lld has a bad node id", (long long)e);
    }
  for (int64_t i = 0; i < Ns; ++i)
    if (node_body[i] < 0) return fail(c, FW_ERR_ARG, "fw_arena_pack: node %lld belongs to no body", (long long)i);
  // node records (body ids local; the commit adds the scene's first body)
  std::vector<uint32_t> word(Ns);
  std::vector<float2> x0(Ns), v0(Ns), bcv(Ns);
  for (int64_t i = 0; i < Ns; ++i) {
    word[i] = (uint32_t)c->h_bc[i] | ((uint32_t)node_body[i] << fw::NODE_BODY_SHIFT);
    x0[i] = make_float2(c->h_x[2 * i], c->h_x[2 * i + 1]);
    v0[i] = make_float2(c->h_v[2 * i], c->h_v[2 * i + 1]);
    bcv[i] = make_float2(c->h_bcv[2 * i], c->h_bcv[2 * i + 1]);
  }
  for (int b = 0; b < Bs; ++b)
    for (int k = 0; k < c->h_bncnt[b]; ++k) word[c->h_bnodes[c->h_bnoff[b] + k]] |= fw::NODE_BOUNDARY;
  // triangles and the corner lists (ascending element per node)
  std::vector<int32_t> conn(c->h_conn.begin(), c->h_conn.end()), cbeg(Ns), cend(Ns), slot(3 * Es), cpos(3 * Es);
  std::vector<ElemMat> emat(Es);
  std::vector<float2> j2par(Es);
  for (int64_t e = 0; e < Es; ++e) {
    emat[e].area = emat[e].lam = emat[e].mu = 0.f;
    emat[e].word = (c->h_type[e] & 3) | (elem_body[e] << 2);
    j2par[e] = make_float2(c->h_sy[e], c->h_H[e]);
  }
  std::vector<int32_t> off(Ns + 1, 0);
  for (int64_t e = 0; e < Es; ++e)
    for (int k = 0; k < 3; ++k) off[conn[3 * e + k] + 1]++;
  for (int64_t i = 0; i < Ns; ++i) off[i + 1] += off[i];
  {
    std::vector<int32_t> fill(off.begin(), off.end() - 1);
    for (int64_t e = 0; e < Es; ++e)
      for (int k = 0; k < 3; ++k) {
        const int32_t at = fill[conn[3 * e + k]]++;
        slot[at] = (int32_t)(3 * e + k);
        cpos[3 * e + k] = at;
      }
    for (int64_t i = 0; i < Ns; ++i) {
      cbeg[i] = off[i];
      cend[i] = off[i + 1];
    }
  }
  // contact pairs grouped by body (stable: staging order within a body)
  std::vector<Pair> pairs = c->h_pairs;
  std::stable_sort(pairs.begin(), pairs.end(), [](const Pair& x, const Pair& y) { return x.body < y.body; });
  std::vector<int32_t> poff(Bs, 0), pcnt(Bs, 0);
  for (const Pair& pr : pairs) {
    if (pr.body < 0 || pr.body >= Bs) return fail(c, FW_ERR_ARG, "fw_arena_pack: pair body out of range");
    pcnt[pr.body]++;
  }
  for (int b = 1; b < Bs; ++b) poff[b] = poff[b - 1] + pcnt[b - 1];
  // cluster patches, beside the stream records below
  CluLaunch clu{};
  std::vector<CluPatch> cpatch;
  std::vector<unsigned char> cblob;
  auto cut_clusters = [&] {
    if (Bs > kCluMaxBodies || pairs.size() > (size_t)kCluMaxPairs) return;
    bool per_tri = Bs > 1;
    int64_t at = 0;
    for (int b = 0; b < Bs; ++b) {  // bodies one after the other
      if (c->h_noff[b] != at) return;
      at += c->h_ncnt[b];
    }
    for (int64_t e = 1; e < Es && !per_tri; ++e)
      per_tri = c->h_E[e] != c->h_E[0] || c->h_nu[e] != c->h_nu[0] || c->h_type[e] != c->h_type[0] ||
                c->h_sy[e] != c->h_sy[0] || c->h_H[e] != c->h_H[0];
    const CluScene sc{0, 0, 0, 0, 0, 0, Bs, 0, (int)pairs.size()};
    std::vector<int> part(Ns, 0);
    int ctas = 1;
    while (ctas < kCluMaxCtas && (Ns + ctas - 1) / ctas > kCluServedNodes) ctas *= 2;
    for (; ctas <= kCluMaxCtas && ctas <= Ns; ctas *= 2) {
      if (Ns > ctas * (int64_t)kCluMaxThreads && Ns * 32 + Es * 56 > ctas * (int64_t)kCluSharedBytes) continue;
      cpatch.clear();
      cblob.clear();
      if (!make_cluster_patches(c, sc, (int)Ns, off, slot, x0, word, ctas, part, 1, cpatch, cblob)) continue;
      CluLaunch r{};
      r.ctas = ctas;
      for (const CluPatch& q : cpatch) clu_widen(r, q);
      r.nb = Bs;
      r.np = (int)pairs.size();
      r.per_tri = per_tri;
      clu_threads(r, true);
      r.one = 0;  // the larger of the two carve-ups: a launch decides by its largest patch
      if (clu_smem(r) > kCluSharedBytes) continue;
      clu = r;
      return;
    }
    cpatch.clear();
    cblob.clear();
  };
  auto cut = [&] {  // without them the stream kernels step the scene
    try {
      cut_clusters();
    } catch (const std::exception&) {
      clu = CluLaunch{};
      cpatch.clear();
      cblob.clear();
    }
  };
  // stream records
  PatchSet ps;
  if (patch_nodes) {
    struct Join {
      std::thread t;
      ~Join() { if (t.joinable()) t.join(); }
    } cutter;
    bool beside = host_threads(4 * Ns) > 1;
    if (beside) {
      try {
        cutter.t = std::thread(cut);
      } catch (const std::exception&) {  // no thread to be had
        beside = false;
      }
    }
    if (!beside) cut();
    std::string why;
    std::vector<int32_t> bscene(Bs, 0);
    if (make_patches((int)Ns, (int)Es, conn.data(), off, slot, x0, c->h_noff, c->h_ncnt, bscene, patch_nodes, ps, why))
      return fail(c, FW_ERR_ARG, "%s", why.c_str());
  }
  fw_pack* pk = new fw_pack();
  pk->clu = clu;
  pk->mixed = mixed_moduli(c);
  pk->Ns = Ns; pk->Es = Es; pk->Bs = Bs; pk->Np = (int64_t)pairs.size();
  pk->Nh = (int64_t)c->h_heights.size(); pk->No = (int64_t)c->h_occ.size();
  pk->damp = c->h_damp.empty() ? 0.f : c->h_damp[0];
  pk->patch_nodes = patch_nodes;
  pk->Ps = (int64_t)ps.patches.size(); pk->Hs = (int64_t)ps.rh.size(); pk->Ts = (int64_t)ps.re.size();
  pk->CPs = (int64_t)ps.rcp.size();
  pk->no_max = ps.no_max; pk->nh_max = ps.nh_max; pk->ne_max = ps.ne_max;
  struct Src { const void* p; size_t bytes; };
  const Src src[fw_pack::NPARTS] = {
      {x0.data(), sizeof(float2) * Ns}, {v0.data(), sizeof(float2) * Ns}, {bcv.data(), sizeof(float2) * Ns},
      {word.data(), sizeof(uint32_t) * Ns}, {cbeg.data(), sizeof(int32_t) * Ns}, {cend.data(), sizeof(int32_t) * Ns},
      {slot.data(), sizeof(int32_t) * 3 * Es}, {cpos.data(), sizeof(int32_t) * 3 * Es},
      {conn.data(), sizeof(int32_t) * 3 * Es}, {emat.data(), sizeof(ElemMat) * Es}, {j2par.data(), sizeof(float2) * Es},
      {c->h_E.data(), sizeof(float) * Es}, {c->h_nu.data(), sizeof(float) * Es}, {c->h_rho.data(), sizeof(float) * Es},
      {poff.data(), sizeof(int32_t) * Bs}, {pcnt.data(), sizeof(int32_t) * Bs}, {pairs.data(), sizeof(Pair) * pairs.size()},
      {c->h_heights.data(), sizeof(float) * c->h_heights.size()}, {c->h_occ.data(), c->h_occ.size()},
      {ps.rn.data(), sizeof(int32_t) * ps.rn.size()}, {ps.rh.data(), sizeof(int32_t) * ps.rh.size()},
      {ps.re.data(), sizeof(int32_t) * ps.re.size()}, {ps.rc.data(), sizeof(uint2) * ps.rc.size()},
      {ps.rcp.data(), sizeof(uint16_t) * ps.rcp.size()}, {ps.rcs.data(), sizeof(uint16_t) * ps.rcs.size()},
      {ps.patches.data(), sizeof(StreamPatch) * ps.patches.size()},
      {cpatch.data(), sizeof(CluPatch) * cpatch.size()}, {cblob.data(), cblob.size()}};
  size_t total = 0;
  for (int k = 0; k < fw_pack::NPARTS; ++k) {
    pk->off[k] = total;
    pk->len[k] = src[k].bytes;
    total += (src[k].bytes + 15) & ~(size_t)15;
  }
  pk->bytes = total;
  if (pinned && cudaHostAlloc((void**)&pk->block, total ? total : 16, cudaHostAllocDefault) == cudaSuccess) {
    pk->pinned = true;
  } else {
    cudaGetLastError();
    pk->block = (unsigned char*)malloc(total ? total : 16);
    if (!pk->block) {
      delete pk;
      return fail(c, FW_ERR_OOM, "fw_arena_pack: host allocation of %zu bytes failed", total);
    }
  }
  for (int k = 0; k < fw_pack::NPARTS; ++k)
    if (src[k].bytes) memcpy(pk->block + pk->off[k], src[k].p, src[k].bytes);
  // device bytes of the scene's ranges
  int64_t dev = 48 * Ns + 136 * Es + 64 * pk->Np + 4 * pk->Nh + pk->No;
  if (patch_nodes)
    dev += (int64_t)sizeof(StreamPatch) * pk->Ps + 4 * pk->Hs + (4 + 8 + (int64_t)sizeof(StreamElem)) * pk->Ts +
           2 * pk->CPs + 6 * Es + (4 + (int64_t)sizeof(StreamNode)) * Ns + (int64_t)cblob.size() +
           (int64_t)(sizeof(CluPatch) * cpatch.size());
  pk->dev_bytes = dev;
  // clear the stage for the next scene
  c->h_x.clear(); c->h_v.clear(); c->h_bc.clear(); c->h_bcv.clear();
  c->h_conn.clear(); c->h_type.clear(); c->h_E.clear(); c->h_nu.clear(); c->h_rho.clear(); c->h_sy.clear(); c->h_H.clear();
  c->h_noff.clear(); c->h_ncnt.clear(); c->h_eoff.clear(); c->h_ecnt.clear(); c->h_scene.clear();
  c->h_bnoff.clear(); c->h_bncnt.clear(); c->h_bnodes.clear(); c->h_pairs.clear(); c->h_heights.clear(); c->h_occ.clear();
  *out = pk;
  return FW_OK;
}

}  // namespace

// ------------------------------------------------------------------ C ABI

extern "C" {

int fw_create(fw_ctx** out, int device) {
  if (!out) return FW_ERR_ARG;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) return FW_ERR_CUDA;
  if (device < 0 || device >= ndev) return FW_ERR_ARG;
  fw_ctx* c = new fw_ctx();
  c->device = device;
  if (cudaSetDevice(device) != cudaSuccess ||
      cudaStreamCreateWithFlags(&c->own_stream, cudaStreamNonBlocking) != cudaSuccess) {
    delete c;
    return FW_ERR_CUDA;
  }
  c->stream = c->own_stream;
  c->host = take_host_block();
  *out = c;
  return FW_OK;
}

int fw_create_stage(fw_ctx** out) {
  if (!out) return FW_ERR_ARG;
  fw_ctx* c = new fw_ctx();
  c->device = -1;  // staging only: no device, no stream
  *out = c;
  return FW_OK;
}

void fw_destroy(fw_ctx* c) {
  if (!c) return;
  if (c->device < 0) {
    delete c;
    return;
  }
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  drop_graphs(c);
  for (void* p : c->allocs) cudaFree(p);
  for (void* p : {(void*)c->d_echunk, (void*)c->d_epart, (void*)c->d_efirst, (void*)c->d_eout})
    if (p) cudaFree(p);
  give_host_block(c->host);  // the stream is idle: nothing writes it any more
  for (cudaStream_t st : c->side_streams) cudaStreamDestroy(st);
  for (cudaEvent_t ev : c->side_events) cudaEventDestroy(ev);
  if (c->own_stream) cudaStreamDestroy(c->own_stream);
  delete c;
}

const char* fw_last_error(const fw_ctx* c) { return c ? c->err.c_str() : "null context"; }

int fw_set_stream(fw_ctx* c, void* stream) {
  if (!c) return FW_ERR_ARG;
  c->stream = stream ? (cudaStream_t)stream : c->own_stream;
  return FW_OK;
}

int fw_set_nodes(fw_ctx* c, int32_t n, const float* coords, const float* vel,
                 const int32_t* bc_bits, const float* bc_values) {
  if (!c) return FW_ERR_ARG;
  if (c->finalized && !c->arena) return fail(c, FW_ERR_STATE, "fw_set_nodes after fw_finalize");
  if (n <= 0 || !coords) return fail(c, FW_ERR_ARG, "fw_set_nodes: need n_nodes > 0 and coords");
  if (!c->arena) c->N = n;
  c->h_x.assign(coords, coords + 2 * (size_t)n);
  c->h_v.assign(2 * (size_t)n, 0.f);
  if (vel) c->h_v.assign(vel, vel + 2 * (size_t)n);
  c->h_bc.assign(n, 0);
  if (bc_bits) c->h_bc.assign(bc_bits, bc_bits + n);
  c->h_bcv.assign(2 * (size_t)n, 0.f);
  if (bc_values) c->h_bcv.assign(bc_values, bc_values + 2 * (size_t)n);
  for (int i = 0; i < n; ++i)
    if (c->h_bc[i] & ~0x1FF) return fail(c, FW_ERR_ARG, "node %d: bc bits 0x%x outside 0x1FF", i, c->h_bc[i]);
  return FW_OK;
}

int fw_set_elements(fw_ctx* c, int32_t n, const int32_t* conn, const int32_t* mat_type,
                    const float* young, const float* poisson, const float* density,
                    const float* yield_stress, const float* hardening) {
  if (!c) return FW_ERR_ARG;
  if (c->finalized && !c->arena) return fail(c, FW_ERR_STATE, "fw_set_elements after fw_finalize");
  if (n <= 0 || !conn || !mat_type || !young || !poisson || !density)
    return fail(c, FW_ERR_ARG, "fw_set_elements: need n_elems > 0 and conn/type/E/nu/rho");
  if (!c->arena) c->E = n;
  c->h_conn.assign(conn, conn + 3 * (size_t)n);
  c->h_type.assign(mat_type, mat_type + n);
  c->h_E.assign(young, young + n);
  c->h_nu.assign(poisson, poisson + n);
  c->h_rho.assign(density, density + n);
  c->h_sy.assign(n, 0.f);
  c->h_H.assign(n, 0.f);
  if (yield_stress) c->h_sy.assign(yield_stress, yield_stress + n);
  if (hardening) c->h_H.assign(hardening, hardening + n);
  for (int e = 0; e < n; ++e) {
    const int t = c->h_type[e];
    if (t != fw::MAT_SPRING && t != fw::MAT_ELASTIC && t != fw::MAT_NEOHOOKEAN && t != fw::MAT_MISES)
      return fail(c, FW_ERR_ARG, "element %d: unknown material type %d", e, t);
    if (t == fw::MAT_SPRING && c->arena)
      return fail(c, FW_ERR_ARG, "element %d: spring-mass domains are not served from an arena", e);
  }
  return FW_OK;
}

int fw_set_bodies(fw_ctx* c, int32_t nb, const int32_t* noff, const int32_t* ncnt,
                  const int32_t* eoff, const int32_t* ecnt, const int32_t* scene,
                  const int32_t* bnoff, const int32_t* bncnt, int32_t n_bnodes,
                  const int32_t* bnodes) {
  if (!c) return FW_ERR_ARG;
  if (c->finalized && !c->arena) return fail(c, FW_ERR_STATE, "fw_set_bodies after fw_finalize");
  if (nb <= 0 || !noff || !ncnt || !eoff || !ecnt || !scene || !bnoff || !bncnt)
    return fail(c, FW_ERR_ARG, "fw_set_bodies: need n_bodies > 0 and all range arrays");
  if (nb >= (1 << 22)) return fail(c, FW_ERR_ARG, "fw_set_bodies: at most 4194303 bodies");
  if (!c->arena) c->B = nb;
  c->h_noff.assign(noff, noff + nb);
  c->h_ncnt.assign(ncnt, ncnt + nb);
  c->h_eoff.assign(eoff, eoff + nb);
  c->h_ecnt.assign(ecnt, ecnt + nb);
  c->h_scene.assign(scene, scene + nb);
  c->h_spring_mass.assign(nb, 0.0f);
  c->h_bnoff.assign(bnoff, bnoff + nb);
  c->h_bncnt.assign(bncnt, bncnt + nb);
  c->h_bnodes.assign(bnodes, bnodes + (n_bnodes > 0 ? n_bnodes : 0));
  return FW_OK;
}

int fw_set_scenes(fw_ctx* c, int32_t ns, const float* damping) {
  if (!c) return FW_ERR_ARG;
  if (c->finalized && !c->arena) return fail(c, FW_ERR_STATE, "fw_set_scenes after fw_finalize");
  if (ns <= 0) return fail(c, FW_ERR_ARG, "fw_set_scenes: need n_scenes > 0");
  if (c->arena && ns != 1) return fail(c, FW_ERR_ARG, "arena: stage one scene at a time");
  if (!c->arena) c->S = ns;
  c->h_damp.assign(ns, 0.f);
  if (damping) c->h_damp.assign(damping, damping + ns);
  return FW_OK;
}

int fw_set_damping(fw_ctx* c, int32_t scene, float damping) {
  if (!c) return FW_ERR_ARG;
  if (!c->finalized || c->arena) return fail(c, FW_ERR_STATE, "fw_set_damping needs a finalized world (not an arena)");
  if (scene < 0 || scene >= c->S) return fail(c, FW_ERR_ARG, "fw_set_damping: scene %d out of range", scene);
  c->h_damp[scene] = damping;
  // pageable source: the copy is staged before the call returns
  FW_CUDA(c, cudaMemcpyAsync(c->d.scene_damp + scene, &c->h_damp[scene], sizeof(float), cudaMemcpyHostToDevice,
                             c->stream));
  return FW_OK;
}

static int add_pair(fw_ctx* c, Pair p, const float* lo, const float* hi) {
  if (!c) return FW_ERR_ARG;
  if (c->finalized && !c->arena) return fail(c, FW_ERR_STATE, "contact pair added after fw_finalize");
  if (!lo || !hi) return fail(c, FW_ERR_ARG, "contact pair: gate box required");
  if (p.body < 0) return fail(c, FW_ERR_ARG, "contact pair: bad body %d", p.body);
  p.glo[0] = lo[0];
  p.glo[1] = lo[1];
  p.ghi[0] = hi[0];
  p.ghi[1] = hi[1];
  c->h_pairs.push_back(p);
  return FW_OK;
}

int fw_add_plane_pair(fw_ctx* c, int32_t body, float penalty, const float* lo, const float* hi,
                      float px, float py, float nx, float ny) {
  Pair p{};
  p.kind = fw::PAIR_PLANE;
  p.body = body;
  p.penalty = penalty;
  p.f[0] = px;
  p.f[1] = py;
  p.f[2] = nx;
  p.f[3] = ny;
  return add_pair(c, p, lo, hi);
}

int fw_add_heightfield_pair(fw_ctx* c, int32_t body, float penalty, const float* lo,
                            const float* hi, int32_t n_samples, const float* heights, float lb_x,
                            float ub_x, int32_t reverse) {
  if (!c) return FW_ERR_ARG;
  if (n_samples < 2 || !heights)
    return fail(c, FW_ERR_ARG, "heightfield pair: need >= 2 samples");
  Pair p{};
  p.kind = fw::PAIR_HEIGHTFIELD;
  p.body = body;
  p.penalty = penalty;
  p.table = (int)c->h_heights.size();
  p.n0 = n_samples;
  p.n1 = reverse ? 1 : 0;
  p.f[0] = lb_x;
  p.f[1] = ub_x;
  c->h_heights.insert(c->h_heights.end(), heights, heights + n_samples);
  return add_pair(c, p, lo, hi);
}

int fw_add_voxel_pair(fw_ctx* c, int32_t body, float penalty, const float* lo, const float* hi,
                      int32_t nx, int32_t ny, const int32_t* occ, float lb_x, float lb_y, float dx,
                      float dz) {
  if (!c) return FW_ERR_ARG;
  if (nx <= 0 || ny <= 0 || !occ) return fail(c, FW_ERR_ARG, "voxel pair: need nx, ny > 0 and occupancy");
  Pair p{};
  p.kind = fw::PAIR_VOXEL;
  p.body = body;
  p.penalty = penalty;
  p.table = (int)c->h_occ.size();
  p.n0 = nx;
  p.n1 = ny;
  p.pad = nx > 0xFFFF || ny > 0xFFFF ? 1 : 0;
  p.f[0] = lb_x;
  p.f[1] = lb_y;
  p.f[2] = dx;
  p.f[3] = dz;
  // 1 = occupied, 0 = free, 2 = any other value (neither test matches it)
  const size_t n = (size_t)nx * ny;
  const size_t base = c->h_occ.size();
  c->h_occ.resize(base + n);
  for (size_t k = 0; k < n; ++k) c->h_occ[base + k] = occ[k] == 1 ? 1 : (occ[k] == 0 ? 0 : 2);
  return add_pair(c, p, lo, hi);
}

int fw_set_boundary_edges(fw_ctx* c, int32_t n_edges, const int32_t* edges, const int32_t* body_off,
                          const int32_t* body_cnt) {
  if (!c || n_edges < 0 || (n_edges && !edges) || !body_off || !body_cnt) return FW_ERR_ARG;
  if (c->finalized || c->arena) return fail(c, FW_ERR_STATE, "fw_set_boundary_edges after fw_finalize / on an arena");
  if (c->B <= 0) return fail(c, FW_ERR_STATE, "fw_set_boundary_edges before fw_set_bodies");
  for (int b = 0; b < c->B; ++b)
    if (body_off[b] < 0 || body_cnt[b] < 0 || (int64_t)body_off[b] + body_cnt[b] > n_edges)
      return fail(c, FW_ERR_ARG, "fw_set_boundary_edges: body %d range outside [0, %d)", b, n_edges);
  c->h_be.resize(n_edges);
  for (int k = 0; k < n_edges; ++k) c->h_be[k] = make_int2(edges[2 * k], edges[2 * k + 1]);
  c->h_be_off.assign(body_off, body_off + c->B);
  c->h_be_cnt.assign(body_cnt, body_cnt + c->B);
  return FW_OK;
}

int fw_set_flex_scene(fw_ctx* c, int32_t scene, int32_t skip_bvh, int32_t n_domains, const int32_t* dom_obj,
                      const int32_t* dom_body, const float* dom_box) {
  if (!c || n_domains < 0 || (n_domains && (!dom_obj || !dom_body || !dom_box))) return FW_ERR_ARG;
  if (c->finalized || c->arena) return fail(c, FW_ERR_STATE, "fw_set_flex_scene after fw_finalize / on an arena");
  if (scene < 0) return fail(c, FW_ERR_ARG, "fw_set_flex_scene: scene %d", scene);
  fw_ctx::FlexSceneHost& h = c->h_flex_scene[scene];
  h.skip_bvh = skip_bvh ? 1 : 0;
  h.dom_obj.assign(dom_obj, dom_obj + n_domains);
  h.dom_body.assign(dom_body, dom_body + n_domains);
  h.dom_box.resize(n_domains);
  for (int g = 0; g < n_domains; ++g)
    h.dom_box[g] = make_float4(dom_box[4 * g], dom_box[4 * g + 1], dom_box[4 * g + 2], dom_box[4 * g + 3]);
  return FW_OK;
}

int fw_add_flex_pair(fw_ctx* c, int32_t body1, int32_t body2, float penalty, float friction) {
  if (!c) return FW_ERR_ARG;
  if (c->finalized || c->arena) return fail(c, FW_ERR_STATE, "fw_add_flex_pair after fw_finalize / on an arena");
  if (body1 < 0 || body2 < 0 || body1 >= c->B || body2 >= c->B || body1 == body2)
    return fail(c, FW_ERR_ARG, "fw_add_flex_pair: bodies %d, %d", body1, body2);
  c->h_flex.push_back(fw_ctx::FlexPair{body1, body2, penalty, friction, 0});
  return FW_OK;
}

int fw_tie_flex_pair(fw_ctx* c, int32_t pair) {
  if (!c) return FW_ERR_ARG;
  if (c->finalized || c->arena) return fail(c, FW_ERR_STATE, "fw_tie_flex_pair after fw_finalize / on an arena");
  if (pair < 0 || pair >= (int)c->h_flex.size()) return fail(c, FW_ERR_ARG, "fw_tie_flex_pair: pair %d", pair);
  c->h_flex[pair].tied = 1;
  return FW_OK;
}

int fw_mass_scaling(fw_ctx* c, float dt_target) {
  if (!c) return FW_ERR_ARG;
  if (!c->finalized || c->arena) return fail(c, FW_ERR_STATE, "fw_mass_scaling needs a finalized world (not an arena)");
  if (!(dt_target > 0.0f)) return fail(c, FW_ERR_ARG, "fw_mass_scaling: dt_target must be > 0");
  if ((int)c->h_E.size() != c->E || (int)c->h_rho.size() != c->E)
    return fail(c, FW_ERR_STATE, "fw_mass_scaling: element materials are no longer staged");
  float *young = nullptr, *rho = nullptr, *dm = nullptr;
  int32_t* hit = nullptr;
  int rc;
  if ((rc = upload(c, &young, c->h_E)) || (rc = upload(c, &rho, c->h_rho)) || (rc = dalloc(c, &dm, c->E)) ||
      (rc = dalloc(c, &hit, c->E)))
    return rc;
  k_mass_scale_elems<<<(c->E + kBlock - 1) / kBlock, kBlock, 0, c->stream>>>(c->d, young, rho, dt_target, dm, hit);
  k_mass_scale_nodes<<<(c->N + kBlock - 1) / kBlock, kBlock, 0, c->stream>>>(c->d, dm, hit, dt_target);
  c->launches += 2;
  if ((rc = check_kernel(c, "mass scaling"))) return rc;
  if (c->path == FW_PATH_STREAM && (rc = stream_records(c))) return rc;  // its node records hold the masses
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  return FW_OK;
}

int fw_read_flex_state(fw_ctx* c, int32_t* item_cache, int32_t n_items, float* grid) {
  if (!c) return FW_ERR_ARG;
  if (!c->has_flex) return fail(c, FW_ERR_STATE, "fw_read_flex_state: the world has no FEM-FEM contact");
  if (n_items != c->fx.n_items) return fail(c, FW_ERR_ARG, "fw_read_flex_state: %d work items, not %d", c->fx.n_items, n_items);
  FlexGrid g{};
  if (item_cache)
    FW_CUDA(c, cudaMemcpyAsync(item_cache, c->fx.item_cache, sizeof(int32_t) * n_items, cudaMemcpyDeviceToHost, c->stream));
  FW_CUDA(c, cudaMemcpyAsync(&g, c->fx.g, sizeof(FlexGrid), cudaMemcpyDeviceToHost, c->stream));  // the first FEM-FEM scene
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  if (grid) {
    int est = g.estimate >= 0 ? g.estimate : g.estimate ^ 0x7FFFFFFF;  // ordered int -> float bits
    float estf;
    memcpy(&estf, &est, sizeof(float));
    const float v[8] = {(float)g.tc, (float)g.cnx, (float)g.cny, g.olx, g.oly, g.gsx, g.gsy, estf};
    memcpy(grid, v, sizeof(v));
  }
  return FW_OK;
}

int fw_set_spring_bodies(fw_ctx* c, int32_t n, const int32_t* bodies, const float* node_mass) {
  if (!c || n < 0 || (n && (!bodies || !node_mass))) return FW_ERR_ARG;
  if (c->finalized || c->arena) return fail(c, FW_ERR_STATE, "fw_set_spring_bodies after fw_finalize / on an arena");
  if ((int)c->h_spring_mass.size() != c->B) return fail(c, FW_ERR_STATE, "fw_set_spring_bodies before fw_set_bodies");
  for (int k = 0; k < n; ++k) {
    if (bodies[k] < 0 || bodies[k] >= c->B) return fail(c, FW_ERR_ARG, "fw_set_spring_bodies: body %d", bodies[k]);
    if (!(node_mass[k] > 0.0f)) return fail(c, FW_ERR_ARG, "fw_set_spring_bodies: node mass must be > 0");
    c->h_spring_mass[bodies[k]] = node_mass[k];
  }
  c->has_springs = n > 0;
  return FW_OK;
}

int fw_set_rigids(fw_ctx* c, int32_t n, const float* params, const int32_t* ints, int32_t n_ground,
                  const float* grounds) {
  if (!c) return FW_ERR_ARG;
  if (c->finalized) return fail(c, FW_ERR_STATE, "fw_set_rigids after fw_finalize");
  if (c->arena) return fail(c, FW_ERR_STATE, "rigid bodies are not part of arena (served) worlds");
  if (n < 0 || n_ground < 0 || (n > 0 && (!params || !ints)) || (n_ground > 0 && !grounds))
    return fail(c, FW_ERR_ARG, "fw_set_rigids: bad sizes or pointers");
  c->h_rigid.assign(n, Rigid{});
  for (int a = 0; a < n; ++a) {
    const float* q = params + 20 * (size_t)a;
    Rigid& g = c->h_rigid[a];
    g.type = ints[4 * a];
    g.bc = ints[4 * a + 1];
    g.in_contact = ints[4 * a + 2];
    g.scene = ints[4 * a + 3];
    if (g.type != fw::RIGID_BALL && g.type != fw::RIGID_BOX && g.type != fw::RIGID_CAPSULE &&
        g.type != fw::RIGID_ANALYTICAL)
      return fail(c, FW_ERR_ARG, "rigid %d: type %d is not a ball, box, capsule or analytical entry", a, g.type);
    g.c[0] = q[0]; g.c[1] = q[1]; g.prim[0] = q[2]; g.prim[1] = q[3];
    g.radius = q[4]; g.quat = q[5]; g.mass = q[6]; g.inertia = q[7];
    g.V[0] = q[8]; g.V[1] = q[9]; g.W = q[10];
    g.bcT[0] = q[11]; g.bcT[1] = q[12]; g.bcG[0] = q[13]; g.bcG[1] = q[14]; g.bcR = q[15];
    g.lb[0] = q[16]; g.lb[1] = q[17]; g.ub[0] = q[18]; g.ub[1] = q[19];  // an analytical entry's first box
  }
  c->h_gbox.resize(n_ground);
  c->h_gkind.resize(n_ground);
  c->h_gscene.resize(n_ground);
  for (int k = 0; k < n_ground; ++k) {
    const float* q = grounds + 6 * (size_t)k;
    if (q[0] != 0.0f && q[0] != 1.0f) return fail(c, FW_ERR_ARG, "ground %d: kind must be 0 (plane) or 1 (box)", k);
    c->h_gkind[k] = (int)q[0];
    c->h_gbox[k] = make_float4(q[1], q[2], q[3], q[4]);
    c->h_gscene[k] = (int)q[5];
  }
  c->rigid_set = true;
  return FW_OK;
}

int fw_add_rigid_pair(fw_ctx* c, int32_t body, int32_t rigid, float penalty, float friction, int32_t skip_bvh,
                      int32_t tied) {
  if (!c) return FW_ERR_ARG;
  if (!c->rigid_set) return fail(c, FW_ERR_STATE, "fw_add_rigid_pair before fw_set_rigids");
  if (rigid < 0 || rigid >= (int)c->h_rigid.size())
    return fail(c, FW_ERR_ARG, "rigid pair: rigid %d outside [0, %d)", rigid, (int)c->h_rigid.size());
  Pair p{};
  p.kind = fw::PAIR_RIGID;
  p.body = body;
  p.penalty = penalty;
  p.table = rigid;
  p.n1 = skip_bvh ? 1 : 0;
  p.pad = tied ? 1 : 0;  // a tied pair (rigid pairs only)
  p.f[0] = friction;
  const float zero[2] = {0.0f, 0.0f};
  return add_pair(c, p, zero, zero);
}

int fw_gate_by_rigid(fw_ctx* c, int32_t entry) {
  if (!c) return FW_ERR_ARG;
  if (c->finalized) return fail(c, FW_ERR_STATE, "fw_gate_by_rigid after fw_finalize");
  if (c->h_pairs.empty() || c->h_pairs.back().kind == fw::PAIR_RIGID)
    return fail(c, FW_ERR_STATE, "fw_gate_by_rigid: the last pair added is not a ground pair");
  if (entry < 0 || entry >= (int)c->h_rigid.size())
    return fail(c, FW_ERR_ARG, "fw_gate_by_rigid: entry %d outside [0, %d)", entry, (int)c->h_rigid.size());
  c->h_pairs.back().gate = entry + 1;
  return FW_OK;
}

int fw_set_rigid_clocks(fw_ctx* c, const int32_t* every, const float* dt, const float* damping) {
  if (!c || !every || !dt || !damping) return FW_ERR_ARG;
  if (!c->has_rigid) return fail(c, FW_ERR_STATE, "fw_set_rigid_clocks: no rigid bodies (or before fw_finalize)");
  std::vector<fw::RigidClock> ck(c->S);
  for (int s = 0; s < c->S; ++s) {
    if (every[s] < 1) return fail(c, FW_ERR_ARG, "fw_set_rigid_clocks: every[%d] must be >= 1", s);
    ck[s] = fw::RigidClock{every[s], dt[s], damping[s], 0};
  }
  FW_CUDA(c, cudaMemcpyAsync(c->d_rclock, ck.data(), sizeof(fw::RigidClock) * ck.size(), cudaMemcpyHostToDevice,
                             c->stream));
  FW_CUDA(c, cudaStreamSynchronize(c->stream));  // ck lives on this stack frame
  return FW_OK;
}

int fw_set_rigid_clock(fw_ctx* c, int32_t every, float dt, float damping) {
  if (!c) return FW_ERR_ARG;
  if (!c->has_rigid) return fail(c, FW_ERR_STATE, "fw_set_rigid_clock: no rigid bodies (or before fw_finalize)");
  const std::vector<int32_t> e(c->S, every);
  const std::vector<float> t(c->S, dt), m(c->S, damping);
  return fw_set_rigid_clocks(c, e.data(), t.data(), m.data());
}

int fw_read_rigids(fw_ctx* c, float* out, int32_t* flags) {
  if (!c || !out) return FW_ERR_ARG;
  if (!c->has_rigid) return fail(c, FW_ERR_STATE, "fw_read_rigids: no rigid bodies (or before fw_finalize)");
  std::vector<Rigid> h(c->rd.n);
  int err = 0;
  FW_CUDA(c, cudaMemcpyAsync(h.data(), c->rd.rig, sizeof(Rigid) * h.size(), cudaMemcpyDeviceToHost, c->stream));
  FW_CUDA(c, cudaMemcpyAsync(&err, c->rd.err, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  for (size_t a = 0; a < h.size(); ++a) {
    const Rigid& g = h[a];
    float* o = out + 12 * a;
    o[0] = g.c[0]; o[1] = g.c[1]; o[2] = g.quat; o[3] = g.V[0]; o[4] = g.V[1]; o[5] = g.W;
    o[6] = g.U[0]; o[7] = g.U[1]; o[8] = g.lb[0]; o[9] = g.lb[1]; o[10] = g.ub[0]; o[11] = g.ub[1];
  }
  if (flags) *flags = err;
  return FW_OK;
}

int fw_set_flex_clock(fw_ctx* c, double dt) {
  if (!c) return FW_ERR_ARG;
  for (double& v : c->flex_clock) v = dt;
  c->flex_clock_all = dt;
  if (c->has_flex)
    FW_CUDA(c, cudaMemcpyAsync(c->d_flex_clock, c->flex_clock.data(), sizeof(double) * c->flex_clock.size(),
                               cudaMemcpyHostToDevice, c->stream));
  return FW_OK;
}

int fw_set_flex_clocks(fw_ctx* c, const double* dt) {
  if (!c || !dt) return FW_ERR_ARG;
  if (!c->has_flex) return fail(c, FW_ERR_STATE, "fw_set_flex_clocks: no FEM-FEM contact (or before fw_finalize)");
  for (size_t k = 0; k < c->flex_clock.size(); ++k) c->flex_clock[k] = dt[c->flex_scene_of[k]];
  FW_CUDA(c, cudaMemcpyAsync(c->d_flex_clock, c->flex_clock.data(), sizeof(double) * c->flex_clock.size(),
                             cudaMemcpyHostToDevice, c->stream));
  return FW_OK;
}

// Device state of the FEM-FEM contact: per scene with ContactFlexFlex pairs,
// its work items in the reference's order (per pair: domain2's boundary nodes
// against domain1's edges, then domain1's against domain2's;
// mixedcontact.py:1876-1924), its spatial hash arrays sized as the reference
// sizes them for that loop (femspringmanager.py:545-548 MAX_BOUNDARY_ELEMENTS;
// spatialmanager.py:520-525: 3^2 pairs per element, 100000 cells), and the
// per-node contribution lists.
int build_flex(fw_ctx* c) {
  const int B = c->B, N = c->N;
  if ((int)c->h_be_off.size() != B) return fail(c, FW_ERR_ARG, "FEM-FEM contact: fw_set_boundary_edges missing");
  const int n_be = (int)c->h_be.size();
  std::vector<int32_t> be_dom(std::max(n_be, 1), 0), be_off(B), be_cnt(B);
  int run = 0;
  for (int b = 0; b < B; ++b) {
    if (c->h_be_off[b] != run) return fail(c, FW_ERR_ARG, "FEM-FEM contact: boundary edges must be stored body by body");
    be_off[b] = c->h_be_off[b];
    be_cnt[b] = c->h_be_cnt[b];
    for (int k = 0; k < be_cnt[b]; ++k) {
      const int2 e = c->h_be[run + k];
      if (e.x < c->h_noff[b] || e.x >= c->h_noff[b] + c->h_ncnt[b] || e.y < c->h_noff[b] ||
          e.y >= c->h_noff[b] + c->h_ncnt[b])
        return fail(c, FW_ERR_ARG, "FEM-FEM contact: boundary edge %d leaves body %d", run + k, b);
      be_dom[run + k] = b;
    }
    run += be_cnt[b];
  }
  if (run != n_be || n_be == 0) return fail(c, FW_ERR_ARG, "FEM-FEM contact: boundary edge counts do not add up");
  // bodies of each scene (contiguous, in body order)
  std::vector<int> s_b0(c->S, -1), s_nb(c->S, 0);
  for (int b = 0; b < B; ++b) {
    const int sc = c->h_scene[b];
    if (s_b0[sc] < 0) s_b0[sc] = b;
    if (s_b0[sc] + s_nb[sc] != b) return fail(c, FW_ERR_ARG, "FEM-FEM contact: a scene's bodies must be contiguous");
    ++s_nb[sc];
  }
  // pairs grouped by scene, creation order kept within a scene
  std::map<int, std::vector<int>> pairs_of;
  for (size_t p = 0; p < c->h_flex.size(); ++p) {
    const fw_ctx::FlexPair& fp = c->h_flex[p];
    if (c->h_scene[fp.b1] != c->h_scene[fp.b2]) return fail(c, FW_ERR_ARG, "FEM-FEM pair %zu joins two scenes", p);
    pairs_of[c->h_scene[fp.b1]].push_back((int)p);
  }
  std::vector<int32_t> item_node, item_target, item_pair;
  std::vector<float> item_pen, item_fric;
  std::vector<int2> pair_body;
  std::vector<int32_t> pair_tied;
  std::vector<int4> segs;  // (first item, count, pair in its scene, target)
  int n_units = 0;
  std::vector<FlexScene> scs;
  std::vector<int32_t> dom_obj, dom_body;
  std::vector<float4> dom_box;
  std::vector<int32_t> slot(N, -1);
  int n_slots = 0, pair_base = 0, max_dom_fem = 1;
  c->flex_scene_of.clear();
  for (auto& kv : pairs_of) {
    const int sc = kv.first;
    auto it = c->h_flex_scene.find(sc);
    if (it == c->h_flex_scene.end()) return fail(c, FW_ERR_ARG, "FEM-FEM contact: fw_set_flex_scene missing for scene %d", sc);
    const fw_ctx::FlexSceneHost& h = it->second;
    FlexScene fsd{};
    fsd.scene = sc;
    fsd.body0 = s_b0[sc];
    fsd.n_fem = s_nb[sc];
    fsd.dom_off = (int)dom_obj.size();
    fsd.n_dom = (int)h.dom_obj.size();
    fsd.skip_bvh = h.skip_bvh;
    for (int g = 0; g < fsd.n_dom; ++g) {
      const int db = h.dom_body[g];
      if (db >= 0 && (db < fsd.body0 || db >= fsd.body0 + fsd.n_fem))
        return fail(c, FW_ERR_ARG, "FEM-FEM contact: scene %d domain %d names body %d of another scene", sc, g, db);
      dom_obj.push_back(h.dom_obj[g]);
      dom_body.push_back(db);
      dom_box.push_back(h.dom_box[g]);
    }
    fsd.pair_off = (int)pair_body.size();
    fsd.n_pairs = (int)kv.second.size();
    fsd.seg_base = (int)segs.size();
    int scene_nodes = 0;
    for (int b = fsd.body0; b < fsd.body0 + fsd.n_fem; ++b) scene_nodes += c->h_ncnt[b];
    fsd.be0 = be_off[fsd.body0];
    fsd.n_be = 0;
    for (int b = fsd.body0; b < fsd.body0 + fsd.n_fem; ++b) fsd.n_be += be_cnt[b];
    const int max_nodes = std::max(scene_nodes + 1024, 2048);
    const int max_elements = std::max(fsd.n_be + 1024, max_nodes);
    fsd.max_pairs = 9 * max_elements;
    fsd.pair_base = pair_base;
    pair_base += fsd.max_pairs;
    fsd.cell_base = (int)scs.size() * kFlexMaxCells;
    for (int lp = 0; lp < fsd.n_pairs; ++lp) {
      const fw_ctx::FlexPair& fp = c->h_flex[kv.second[lp]];
      pair_body.push_back(make_int2(fp.b1, fp.b2));
      pair_tied.push_back(fp.tied);
      (fp.tied ? fsd.n_tied : fsd.n_untied) += c->h_bncnt[fp.b1] + c->h_bncnt[fp.b2];
      for (int side = 0; side < 2; ++side) {
        const int src = side == 0 ? fp.b2 : fp.b1, dst = side == 0 ? fp.b1 : fp.b2;
        segs.push_back(make_int4((int)item_node.size(), c->h_bncnt[src], lp, dst));
        for (int k = 0; k < c->h_bncnt[src]; ++k) {
          const int n = c->h_bnodes[c->h_bnoff[src] + k];
          item_node.push_back(n);
          item_target.push_back(dst);
          item_pair.push_back(fsd.pair_off + lp);
          item_pen.push_back(fp.pen);
          item_fric.push_back(fp.fric);
          if (slot[n] < 0) slot[n] = n_slots++;
        }
      }
    }
    fsd.n_seg = (int)segs.size() - fsd.seg_base;
    fsd.unit_base = n_units;
    for (int k = fsd.seg_base; k < (int)segs.size(); ++k) n_units += (segs[k].y + kFlexUnit - 1) / kFlexUnit;
    for (int k = fsd.be0; k < fsd.be0 + fsd.n_be; ++k)  // edge nodes receive the reactions
      for (int n : {c->h_be[k].x, c->h_be[k].y})
        if (slot[n] < 0) slot[n] = n_slots++;
    max_dom_fem = std::max(max_dom_fem, fsd.n_dom + fsd.n_fem);
    scs.push_back(fsd);
    c->flex_scene_of.push_back(sc);
  }
  const int n_fs = (int)scs.size();
  if (n_fs > 65535)  // the contact launch puts the scenes in gridDim.y
    return fail(c, FW_ERR_ARG, "FEM-FEM contact: %d scenes with FEM-FEM pairs in one world, at most 65535", n_fs);
  const int n_items = (int)item_node.size();
  FlexDev f{};
  f.n_items = n_items;
  f.n_fs = n_fs;
  f.mpd = std::max(powf(100000.0f, 0.5f), 1.0f);
  c->flex_clock.assign(n_fs, c->flex_clock_all);
  if (dom_obj.empty()) {
    dom_obj.push_back(0);
    dom_body.push_back(-1);
    dom_box.push_back(make_float4(0.f, 0.f, 0.f, 0.f));
  }
  std::vector<int32_t> minus1(std::max(n_items, 1), -1);
  int rc;
  int32_t *inode = nullptr, *itgt = nullptr, *ipair = nullptr, *icache = nullptr, *bdom = nullptr, *boff = nullptr,
          *bcnt = nullptr, *dobj = nullptr, *dbody = nullptr, *ecount = nullptr,
          *ebase = nullptr, *ccount = nullptr, *cstart = nullptr, *cend = nullptr, *cursor = nullptr,
          *sorted = nullptr, *dslot = nullptr, *dcnt = nullptr, *ditem = nullptr;
  float *ipen = nullptr, *ifric = nullptr;
  int32_t *ptied = nullptr, *telem = nullptr;
  float *tw0 = nullptr, *tw1 = nullptr, *tgap = nullptr;
  int2 *pbody = nullptr, *dbe = nullptr, *crange = nullptr, *scell = nullptr;
  int4 *srec = nullptr, *dseg = nullptr, *ecell = nullptr, *bcell = nullptr, *dunit = nullptr;
  float4 *dbox = nullptr, *ebox = nullptr;
  float2* dforce = nullptr;
  FlexGrid* grid = nullptr;
  FlexScene* dsc = nullptr;
  const size_t cells = (size_t)n_fs * kFlexMaxCells;
  if ((rc = upload(c, &inode, item_node)) || (rc = upload(c, &itgt, item_target)) || (rc = upload(c, &ipair, item_pair)) ||
      (rc = upload(c, &ipen, item_pen)) || (rc = upload(c, &ifric, item_fric)) || (rc = upload(c, &icache, minus1)) ||
      (rc = upload(c, &pbody, pair_body)) || (rc = upload(c, &dbe, c->h_be)) || (rc = upload(c, &bdom, be_dom)) ||
      (rc = upload(c, &boff, be_off)) || (rc = upload(c, &bcnt, be_cnt)) || (rc = upload(c, &dobj, dom_obj)) ||
      (rc = upload(c, &dbody, dom_body)) || (rc = upload(c, &dbox, dom_box)) || (rc = upload(c, &dsc, scs)) ||
      (rc = dalloc(c, &grid, n_fs)) || (rc = dalloc(c, &ebox, n_be)) || (rc = dalloc(c, &ecount, n_be)) ||
      (rc = dalloc(c, &ebase, n_be)) || (rc = dalloc(c, &ccount, cells)) || (rc = dalloc(c, &cstart, cells)) ||
      (rc = dalloc(c, &cend, cells)) || (rc = dalloc(c, &cursor, cells)) || (rc = dalloc(c, &crange, cells)) ||
      (rc = dalloc(c, &sorted, (size_t)pair_base)) || (rc = dalloc(c, &srec, (size_t)pair_base)) ||
      (rc = dalloc(c, &scell, (size_t)pair_base)) || (rc = dalloc(c, &ecell, n_be)) ||
      (rc = upload(c, &dseg, segs)) || (rc = dalloc(c, &bcell, B)) || (rc = dalloc(c, &dunit, std::max(1, n_units))) ||
      (rc = upload(c, &dslot, slot)) || (rc = dalloc(c, &dcnt, std::max(1, n_slots))) ||
      (rc = dalloc(c, &ditem, std::max(1, n_slots) * kFlexListCap)) ||
      (rc = dalloc(c, &dforce, std::max(1, n_slots) * kFlexListCap)) || (rc = dalloc(c, &c->d_flex_clock, n_fs)) ||
      (rc = upload(c, &ptied, pair_tied)) ||
      (rc = upload(c, &telem, minus1)) || (rc = dalloc(c, &tw0, std::max(n_items, 1))) ||
      (rc = dalloc(c, &tw1, std::max(n_items, 1))) || (rc = dalloc(c, &tgap, std::max(n_items, 1))))
    return rc;
  FW_CUDA(c, cudaMemsetAsync(grid, 0, sizeof(FlexGrid) * n_fs, c->stream));
  FW_CUDA(c, cudaMemcpyAsync(c->d_flex_clock, c->flex_clock.data(), sizeof(double) * n_fs, cudaMemcpyHostToDevice,
                             c->stream));
  FW_CUDA(c, cudaMemsetAsync(dcnt, 0, sizeof(int32_t) * std::max(1, n_slots), c->stream));
  FW_CUDA(c, cudaMemsetAsync(cstart, 0, sizeof(int32_t) * cells, c->stream));
  FW_CUDA(c, cudaMemsetAsync(cend, 0, sizeof(int32_t) * cells, c->stream));
  f.item_node = inode; f.item_target = itgt; f.item_pair = ipair; f.item_pen = ipen; f.item_fric = ifric;
  f.item_cache = icache; f.pair_body = pbody; f.be = dbe; f.be_dom = bdom; f.be_off = boff; f.be_cnt = bcnt;
  f.dom_obj = dobj; f.dom_body = dbody; f.dom_box = dbox; f.g = grid;
  f.ebox = ebox; f.ecount = ecount; f.ebase = ebase; f.cell_count = ccount; f.cell_start = cstart;
  f.cell_end = cend; f.cursor = cursor; f.sorted = sorted; f.crange = crange; f.ecell = ecell;
  f.srec = srec; f.scell = scell;
  f.seg = dseg; f.unit = dunit; f.bcell = bcell;
  f.sc = dsc; f.clock_dt = c->d_flex_clock; f.err = c->d_flags + fw_ctx::kFlagFlex;
  {  // the scenes' bodies and pairs as ranges (the pairs go to the device in body order)
    std::vector<int4> rng(c->S, make_int4(0, 0, 0, 0));
    std::vector<int> cnt(B, 0);
    for (const Pair& p : c->h_pairs) cnt[p.body]++;
    int at = 0;
    for (int b = 0; b < B; ++b) {
      int4& r = rng[c->h_scene[b]];
      if (r.y == 0) r = make_int4(b, 0, at, 0);
      r.y += 1;
      r.w += cnt[b];
      at += cnt[b];
    }
    int4* drng = nullptr;
    if ((rc = upload(c, &drng, rng))) return rc;
    FW_CUDA(c, cudaStreamSynchronize(c->stream));
    f.scene_rng = drng;
  }
  f.pair_tied = ptied; f.tie_elem = telem; f.tie_w0 = tw0; f.tie_w1 = tw1; f.tie_gap = tgap;
  c->flex_pre_smem = sizeof(float4) * (size_t)max_dom_fem;
  int optin = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
  // always the most that the kernel's static arrays leave: the attribute belongs
  // to the function, so one context's figure must not fall below what another
  // context launches with
  cudaFuncAttributes fa{};
  FW_CUDA(c, cudaFuncGetAttributes(&fa, k_flex_pre));
  const size_t most = (size_t)optin - fa.sharedSizeBytes;
  if (c->flex_pre_smem > most)
    return fail(c, FW_ERR_ARG, "FEM-FEM contact: a scene's domains need %zu B of shared memory", c->flex_pre_smem);
  FW_CUDA(c, cudaFuncSetAttribute(k_flex_pre, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
  c->fx = f;
  c->d.flex_slot = dslot;
  c->d.flex_cnt = dcnt;
  c->d.flex_item = ditem;
  c->d.flex_force = dforce;
  c->has_flex = true;
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  return FW_OK;
}

static int finalize(fw_ctx* c) {
  if (c->device < 0) return fail(c, FW_ERR_STATE, "fw_finalize on a staging context (fw_create_stage)");
  if (c->finalized) return fail(c, FW_ERR_STATE, "fw_finalize called twice");
  if (c->N <= 0 || c->E <= 0 || c->B <= 0 || c->S <= 0)
    return fail(c, FW_ERR_STATE, "fw_finalize: nodes, elements, bodies and scenes must be set");
  FW_CUDA(c, cudaSetDevice(c->device));
  const int N = c->N, E = c->E, B = c->B, S = c->S;
  // ---- validation and host-side packing
  std::vector<int32_t> node_body(N, -1), elem_body(E, -1);
  for (int b = 0; b < B; ++b) {
    if (c->h_scene[b] < 0 || c->h_scene[b] >= S) return fail(c, FW_ERR_ARG, "body %d: bad scene", b);
    if (c->h_noff[b] < 0 || c->h_ncnt[b] < 0 || (int64_t)c->h_noff[b] + c->h_ncnt[b] > N)
      return fail(c, FW_ERR_ARG, "body %d: node range outside [0, %d)", b, N);
    if (c->h_eoff[b] < 0 || c->h_ecnt[b] < 0 || (int64_t)c->h_eoff[b] + c->h_ecnt[b] > E)
      return fail(c, FW_ERR_ARG, "body %d: element range outside [0, %d)", b, E);
    for (int i = c->h_noff[b]; i < c->h_noff[b] + c->h_ncnt[b]; ++i) {
      if (node_body[i] >= 0) return fail(c, FW_ERR_ARG, "node %d in two bodies", i);
      node_body[i] = b;
    }
    for (int e = c->h_eoff[b]; e < c->h_eoff[b] + c->h_ecnt[b]; ++e) {
      if (elem_body[e] >= 0) return fail(c, FW_ERR_ARG, "element %d in two bodies", e);
      elem_body[e] = b;
    }
  }
  for (int i = 0; i < N; ++i)
    if (node_body[i] < 0) return fail(c, FW_ERR_ARG, "node %d belongs to no body", i);
  for (int e = 0; e < E; ++e) {
    if (elem_body[e] < 0) return fail(c, FW_ERR_ARG, "element %d belongs to no body", e);
    const bool spring = c->h_type[e] == fw::MAT_SPRING;
    if (spring != (c->h_spring_mass[elem_body[e]] > 0.0f))
      return fail(c, FW_ERR_ARG, "element %d: springs (type 0) belong to spring-mass bodies, triangles to FEM bodies", e);
    for (int k = 0; k < 3; ++k) {
      const int n = c->h_conn[3 * e + k];
      if (spring && k == 2) {
        if (n != -1) return fail(c, FW_ERR_ARG, "spring %d: third node id must be -1", e);
        continue;
      }
      if (n < 0 || n >= N) return fail(c, FW_ERR_ARG, "element %d: node id %d outside [0, %d)", e, n, N);
      if (node_body[n] != elem_body[e])
        return fail(c, FW_ERR_ARG, "element %d references node %d of another body", e, n);
    }
  }
  std::vector<uint32_t> word(N);
  for (int i = 0; i < N; ++i)
    word[i] = (uint32_t)c->h_bc[i] | ((uint32_t)node_body[i] << fw::NODE_BODY_SHIFT);
  for (int b = 0; b < B; ++b) {
    if (c->h_bnoff[b] < 0 || c->h_bncnt[b] < 0 ||
        (size_t)c->h_bnoff[b] + c->h_bncnt[b] > c->h_bnodes.size())
      return fail(c, FW_ERR_ARG, "body %d: boundary-node range out of bounds", b);
    for (int k = 0; k < c->h_bncnt[b]; ++k) {
      const int n = c->h_bnodes[c->h_bnoff[b] + k];
      if (n < 0 || n >= N || node_body[n] != b)
        return fail(c, FW_ERR_ARG, "body %d: boundary node %d not in the body", b, n);
      word[n] |= fw::NODE_BOUNDARY;
    }
  }
  // pairs grouped by body, launch order kept within a body
  std::vector<Pair> pairs = c->h_pairs;
  for (const Pair& p : pairs)
    if (p.body >= B) return fail(c, FW_ERR_ARG, "contact pair: body %d >= %d", p.body, B);
  int n_ritems = 0;  // FEM-rigid work items: per rigid pair (added order) its body's boundary nodes
  for (Pair& p : pairs)
    if (p.kind == fw::PAIR_RIGID) {
      if (p.table < 0 || p.table >= (int)c->h_rigid.size())
        return fail(c, FW_ERR_ARG, "rigid pair: rigid %d outside [0, %d)", p.table, (int)c->h_rigid.size());
      p.n0 = n_ritems;
      n_ritems += c->h_bncnt[p.body];
    }
  c->has_rigid = !c->h_rigid.empty();
  std::stable_sort(pairs.begin(), pairs.end(), [](const Pair& a, const Pair& b) { return a.body < b.body; });
  std::vector<int32_t> poff(B, 0), pcnt(B, 0);
  for (size_t k = 0; k < pairs.size(); ++k) pcnt[pairs[k].body]++;
  for (int b = 1; b < B; ++b) poff[b] = poff[b - 1] + pcnt[b - 1];
  // CSR node -> (element, corner), ascending element
  std::vector<int32_t> off(N + 1, 0), slot(3 * (size_t)E);
  for (int e = 0; e < E; ++e)
    for (int k = 0; k < 3; ++k)
      if (c->h_conn[3 * e + k] >= 0) off[c->h_conn[3 * e + k] + 1]++;
  for (int i = 0; i < N; ++i) off[i + 1] += off[i];
  std::vector<int32_t> cpos(3 * (size_t)E);
  {
    std::vector<int32_t> fill(off.begin(), off.end() - 1);
    for (int e = 0; e < E; ++e)
      for (int k = 0; k < 3; ++k) {
        if (c->h_conn[3 * e + k] < 0) {  // a spring's missing third corner: never written
          cpos[3 * (size_t)e + k] = cpos[3 * (size_t)e + k - 1];
          continue;
        }
        const int32_t at = fill[c->h_conn[3 * e + k]]++;
        slot[at] = 3 * e + k;
        cpos[3 * (size_t)e + k] = at;
      }
  }
  std::vector<ElemMat> emat(E);
  std::vector<float2> j2par(E);
  bool has_j2 = false;
  for (int e = 0; e < E; ++e) {
    emat[e].area = emat[e].lam = emat[e].mu = 0.f;
    emat[e].word = (c->h_type[e] & 3) | (elem_body[e] << 2);
    j2par[e] = make_float2(c->h_sy[e], c->h_H[e]);
    has_j2 |= c->h_type[e] == fw::MAT_MISES;
  }
  // device connectivity: a spring's missing third node repeats its second, so
  // loads that every element issues stay in bounds
  std::vector<int32_t> conn_dev(c->h_conn);
  for (int e = 0; e < E; ++e)
    if (conn_dev[3 * (size_t)e + 2] < 0) conn_dev[3 * (size_t)e + 2] = conn_dev[3 * (size_t)e + 1];
  std::vector<float2> x0(N), bcv(N), v0(N);
  for (int i = 0; i < N; ++i) {
    x0[i] = make_float2(c->h_x[2 * i], c->h_x[2 * i + 1]);
    v0[i] = make_float2(c->h_v[2 * i], c->h_v[2 * i + 1]);
    bcv[i] = make_float2(c->h_bcv[2 * i], c->h_bcv[2 * i + 1]);
  }
  // ---- device buffers
  if (int rf = alloc_flags(c)) return rf;
  Dev& d = c->d;
  d.N = N; d.E = E; d.B = B; d.S = S; d.P = (int)pairs.size(); d.has_j2 = has_j2;
  int rc = 0;
  if ((rc = upload(c, &d.x0, x0)) || (rc = upload(c, &d.x, x0)) || (rc = upload(c, &d.v, v0)) ||
      (rc = upload(c, &d.bcv, bcv)) || (rc = upload(c, &d.node_word, word)) ||
      (rc = dalloc(c, &d.mass, N)) || (rc = upload(c, &d.csr_off, off)) ||
      (rc = upload(c, &d.csr_slot, slot)) || (rc = upload(c, &d.corner_pos, cpos)) ||
      (rc = upload(c, &d.conn, conn_dev)) ||
      (rc = dalloc(c, &d.jinv, E)) || (rc = upload(c, &d.emat, emat)) ||
      (rc = upload(c, &d.j2par, j2par)) || (rc = dalloc(c, &d.j2state, has_j2 ? E : 1)) ||
      (rc = dalloc(c, &d.ndmass, E)) || (rc = dalloc(c, &d.corner, 3 * (size_t)E)) ||
      (rc = upload(c, &d.body_scene, c->h_scene)) || (rc = upload(c, &d.body_pair_off, poff)) ||
      (rc = dalloc(c, &d.body_lm, B)) ||
      (rc = upload(c, &d.body_pair_cnt, pcnt)) || (rc = upload(c, &d.pairs, pairs)) ||
      (rc = dalloc(c, &d.pair_active, pairs.size())) || (rc = upload(c, &d.heights, c->h_heights)) ||
      (rc = upload(c, &d.occ, c->h_occ)) || (rc = dalloc(c, &d.scene_dt, S)) ||
      (rc = upload(c, &d.scene_damp, c->h_damp)) || (rc = dalloc(c, &d.scene_counter, S)) ||
      (rc = dalloc(c, &d.scene_active, S)) || (rc = dalloc(c, &d.scene_mode_req, S)) ||
      (rc = dalloc(c, &d.scene_mode, S)) || (rc = dalloc(c, &d.aabb_ring, 8 * (size_t)B)) ||
      (rc = dalloc(c, &d.scene_bad, S)))
    return rc;
  FW_CUDA(c, cudaMemsetAsync(d.scene_bad, 0, sizeof(int32_t) * S, c->stream));
  FW_CUDA(c, cudaMemsetAsync(d.j2state, 0, sizeof(float4) * (has_j2 ? E : 1), c->stream));
  FW_CUDA(c, cudaMemsetAsync(d.pair_active, 0, sizeof(int32_t) * (pairs.empty() ? 1 : pairs.size()), c->stream));
  FW_CUDA(c, cudaMemsetAsync(d.scene_dt, 0, sizeof(float) * S, c->stream));
  FW_CUDA(c, cudaMemsetAsync(d.scene_counter, 0, sizeof(int32_t) * S, c->stream));
  FW_CUDA(c, cudaMemsetAsync(d.aabb_ring, 0, sizeof(int32_t) * 8 * (size_t)B, c->stream));
  std::vector<int32_t> ones(S, 1);
  c->cur_active = ones;
  FW_CUDA(c, cudaMemcpyAsync(d.scene_active, ones.data(), sizeof(int32_t) * S, cudaMemcpyHostToDevice, c->stream));
  FW_CUDA(c, cudaMemcpyAsync(d.scene_mode_req, ones.data(), sizeof(int32_t) * S, cudaMemcpyHostToDevice, c->stream));
  float *dE = nullptr, *dnu = nullptr, *drho = nullptr;
  if ((rc = upload(c, &dE, c->h_E)) || (rc = upload(c, &dnu, c->h_nu)) || (rc = upload(c, &drho, c->h_rho)))
    return rc;
  d.csr_end = d.csr_off + 1;
  k_prepare_elements<<<(E + kBlock - 1) / kBlock, kBlock, 0, c->stream>>>(d, dE, dnu, drho, 0, E);
  k_prepare_mass<<<(N + kBlock - 1) / kBlock, kBlock, 0, c->stream>>>(d, 0, N);
  c->launches += 2;
  bool table = false;  // of the nearest free voxel cells
  for (const Pair& p : pairs) table |= p.kind == fw::PAIR_VOXEL && !p.pad;
  if (table && dalloc_spare(c, &d.vox, c->h_occ.size())) {  // without it the grids are walked
    k_voxel_table<<<dim3((unsigned)pairs.size(), kVoxelBlocks), 32, 0, c->stream>>>(d, 0);
    c->launches += 1;
  }
  if ((rc = check_kernel(c, "prepare"))) return rc;
  if (c->has_springs) {  // a spring-mass domain's nodes carry its mass (femspringmanager.py:844-845)
    std::vector<float> sm(N);
    FW_CUDA(c, cudaMemcpyAsync(sm.data(), d.mass, sizeof(float) * N, cudaMemcpyDeviceToHost, c->stream));
    FW_CUDA(c, cudaStreamSynchronize(c->stream));
    for (int b = 0; b < B; ++b)
      if (c->h_spring_mass[b] > 0.0f)
        for (int k = 0; k < c->h_ncnt[b]; ++k) sm[c->h_noff[b] + k] = c->h_spring_mass[b];
    FW_CUDA(c, cudaMemcpyAsync(d.mass, sm.data(), sizeof(float) * N, cudaMemcpyHostToDevice, c->stream));
    FW_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, c->device);
  set_grids(c);
  if (c->has_springs && (c->path_req == FW_PATH_RESIDENT || c->path_req == FW_PATH_STREAM))
    return fail(c, FW_ERR_ARG, "spring-mass domains run on the gather path only");
  if (!c->h_flex.empty()) {
    if (c->path_req == FW_PATH_RESIDENT || c->path_req == FW_PATH_STREAM)
      return fail(c, FW_ERR_ARG, "FEM-FEM contact runs on the gather path only");
    if ((rc = build_flex(c))) return rc;
  }
  if (c->has_rigid) {
    if (c->path_req == FW_PATH_RESIDENT || c->path_req == FW_PATH_STREAM)
      return fail(c, FW_ERR_ARG, "FEM-rigid contact runs on the gather path only");
    std::vector<int32_t> bslot(N, 0);
    for (int b = 0; b < B; ++b)
      for (int k = 0; k < c->h_bncnt[b]; ++k) bslot[c->h_bnodes[c->h_bnoff[b] + k]] = k;
    // work item -> (pair, boundary node), for the element step's item blocks
    std::vector<int2> rwork(std::max(1, n_ritems), make_int2(0, 0));
    for (size_t q = 0; q < pairs.size(); ++q)
      if (pairs[q].kind == fw::PAIR_RIGID) {
        const Pair& p = pairs[q];
        for (int k = 0; k < c->h_bncnt[p.body]; ++k)
          rwork[p.n0 + k] = make_int2((int)q, c->h_bnodes[c->h_bnoff[p.body] + k]);
      }
    // per rigid, its pairs' item ranges in pair (= item) order; `pairs` is
    // grouped by body by now, so order the rigid pairs by first item again
    std::vector<Pair> rpairs;
    for (const Pair& p : pairs)
      if (p.kind == fw::PAIR_RIGID) rpairs.push_back(p);
    std::sort(rpairs.begin(), rpairs.end(), [](const Pair& a, const Pair& b) { return a.n0 < b.n0; });
    const int nr = (int)c->h_rigid.size();
    std::vector<int32_t> rp_off(nr + 1, 0);
    for (const Pair& p : rpairs) rp_off[p.table + 1]++;
    for (int g = 0; g < nr; ++g) rp_off[g + 1] += rp_off[g];
    std::vector<int4> rp_rng(std::max(1, rp_off[nr]));
    {
      std::vector<int32_t> fill(rp_off.begin(), rp_off.end() - 1);
      for (const Pair& p : rpairs) rp_rng[fill[p.table]++] = make_int4(p.n0, c->h_bncnt[p.body], c->h_bncnt[p.body] ? rwork[p.n0].x : 0, 0);
    }
    // the scenes with rigids: their rigids and grounds, each a contiguous range
    std::vector<fw::RigidScene> rs;
    for (int a = 0, q = 0; a < nr;) {
      const int sc = c->h_rigid[a].scene;
      if (sc < 0 || sc >= S) return fail(c, FW_ERR_ARG, "rigid %d: scene %d outside [0, %d)", a, sc, S);
      if (!rs.empty() && sc <= rs.back().scene)
        return fail(c, FW_ERR_ARG, "rigids must be grouped by scene in ascending scene order");
      fw::RigidScene e{sc, a, 0, 0, 0, {0, 0, 0}};
      while (a < nr && c->h_rigid[a].scene == sc) c->h_rigid[a].rs = (int)rs.size(), ++a, ++e.rn;
      while (q < (int)c->h_gscene.size() && c->h_gscene[q] < sc) ++q;
      e.g0 = q;
      while (q < (int)c->h_gscene.size() && c->h_gscene[q] == sc) ++q, ++e.gn;
      rs.push_back(e);
    }
    for (size_t k = 1; k < c->h_gscene.size(); ++k)
      if (c->h_gscene[k] < c->h_gscene[k - 1]) return fail(c, FW_ERR_ARG, "grounds must be grouped by scene");
    RigidDev& r = c->rd;
    r.n = (int)c->h_rigid.size();
    r.n_ground = (int)c->h_gbox.size();
    r.n_items = n_ritems;
    r.n_rs = (int)rs.size();
    std::vector<fw::RigidClock> ck(S, fw::RigidClock{1, 0.0f, 0.0f, 0});
    if ((rc = upload(c, &r.rig, c->h_rigid)) || (rc = upload(c, &d.bslot, bslot)) ||
        (rc = upload(c, &d.rwork, rwork)) || (rc = dalloc(c, &d.rforce, (size_t)std::max(1, n_ritems))) ||
        (rc = dalloc(c, &r.item, (size_t)n_ritems)) || (rc = upload(c, &r.gbox, c->h_gbox)) ||
        (rc = upload(c, &r.gkind, c->h_gkind)) || (rc = upload(c, &r.rp_off, rp_off)) ||
        (rc = upload(c, &r.rp_rng, rp_rng)) || (rc = upload(c, &r.rs, rs)) ||
        (rc = upload(c, &c->d_rclock, ck)) || (rc = dalloc(c, &r.count, S)) ||
        (rc = dalloc(c, &r.done, rs.size())))
      return rc;
    FW_CUDA(c, cudaMemsetAsync(r.count, 0, sizeof(int) * S, c->stream));
    FW_CUDA(c, cudaMemsetAsync(r.done, 0, sizeof(int) * rs.size(), c->stream));
    r.err = c->d_flags + fw_ctx::kFlagRigid;
    r.clock = c->d_rclock;
    d.rig = r.rig;
    d.ritem = r.item;
    d.n_ritems = n_ritems;
    k_rigid_init<<<(r.n + 127) / 128, 128, 0, c->stream>>>(r.rig, r.n);
    c->launches += 1;
    if ((rc = check_kernel(c, "rigid init"))) return rc;
    FW_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  // zero-dt construction step (setGlobalAABB -> substep(0, 0))
  if ((rc = launch_step(c))) return rc;
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  if (c->has_flex) {  // the initial FEM spatial hash (explicitloop.py:383-385)
    flex_launch(c, 1);
    if ((rc = check_kernel(c, "FEM-FEM hash"))) return rc;
    FW_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  c->path = FW_PATH_GATHER;
  if (c->has_flex || c->has_springs || c->has_rigid) {
    c->finalized = true;
    return FW_OK;
  }
  if (c->path_req == FW_PATH_STREAM) {
    if ((rc = build_stream(c, off, slot, x0, has_j2))) return rc;
    if ((rc = try_cluster(c, off, slot, x0, word, false))) return rc;
    c->path = FW_PATH_STREAM;
    FW_CUDA(c, cudaStreamSynchronize(c->stream));
  } else if (c->path_req != FW_PATH_GATHER) {
    if (S == 1 && c->patches_req == 0 && (rc = try_cluster(c, off, slot, x0, word, true))) return rc;
    if (!c->clu.empty()) {
      c->path = FW_PATH_RESIDENT;
    } else {
      rc = build_resident(c, off, slot, x0, has_j2);
      if (rc < 0) return rc;
      if (rc == 0) {
        c->path = FW_PATH_RESIDENT;
      } else if (c->path_req == FW_PATH_RESIDENT) {
        return fail(c, FW_ERR_ARG, "resident path requested but unavailable: %s", c->res_reason.c_str());
      }
    }
    FW_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  if (!c->clu.empty() && S == 1) c->lists = HostLists{std::move(off), std::move(slot), std::move(x0)};
  c->finalized = true;
  return FW_OK;
}

int fw_set_path(fw_ctx* c, int32_t path, int32_t patches) {
  if (!c) return FW_ERR_ARG;
  if (c->finalized) return fail(c, FW_ERR_STATE, "fw_set_path after fw_finalize");
  if (path != FW_PATH_AUTO && path != FW_PATH_GATHER && path != FW_PATH_RESIDENT && path != FW_PATH_STREAM)
    return fail(c, FW_ERR_ARG, "fw_set_path: unknown path %d", path);
  if (patches < 0) return fail(c, FW_ERR_ARG, "fw_set_path: patches < 0");
  c->path_req = path;
  c->patches_req = patches;
  return FW_OK;
}

static int shared_optin(fw_ctx* c) {
  int optin = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
  return optin;
}

int fw_finalize(fw_ctx* c) {
  if (!c) return FW_ERR_ARG;
  return guarded(c, [&] { return finalize(c); });
}

int fw_set_option(fw_ctx* c, int32_t option, int32_t value) {
  if (!c) return FW_ERR_ARG;
  switch (option) {
    case FW_OPT_FRONT_WARPS: {
      if (c->finalized) return fail(c, FW_ERR_STATE, "FW_OPT_FRONT_WARPS after fw_finalize");
      bool ok = false;
      if (c->res_threads == 1024)
        for (int v : kFrontChoices1024) ok |= v == value;
      else
        for (int v : kFrontChoices) ok |= v == value;
      if (!ok)
        return fail(c, FW_ERR_ARG, "FW_OPT_FRONT_WARPS must be %s", c->res_threads == 1024 ? "8, 12 or 16 (1024 threads)"
                                                                                          : "2, 4, 6 or 8");
      c->front_warps = value;
      c->shape_asked = true;
      return FW_OK;
    }
    case FW_OPT_RES_THREADS: {
      if (c->finalized) return fail(c, FW_ERR_STATE, "FW_OPT_RES_THREADS after fw_finalize");
      if (value != 512 && value != 1024) return fail(c, FW_ERR_ARG, "FW_OPT_RES_THREADS must be 512 or 1024");
      c->res_threads = value;
      c->shape_asked = true;
      c->front_warps = value == 1024 ? 12 : 6;  // the default split for that size
      return FW_OK;
    }
    case FW_OPT_BLOCK_ELEMS:
    case FW_OPT_BLOCK_NODES: {
      if (value < 32 || value > kMaxBlock || value % 32)
        return fail(c, FW_ERR_ARG, "block size must be a multiple of 32 in [32, %d]", kMaxBlock);
      (option == FW_OPT_BLOCK_ELEMS ? c->block_e : c->block_n) = value;
      set_grids(c);
      drop_graphs(c);
      return FW_OK;
    }
    case FW_OPT_GRID_ELEMS: {
      if (value < 0) return fail(c, FW_ERR_ARG, "FW_OPT_GRID_ELEMS must be >= 0");
      c->grid_e_cap = value;
      set_grids(c);
      drop_graphs(c);
      return FW_OK;
    }
    case FW_OPT_WAIT_LIMIT:
      if (value < 0) return fail(c, FW_ERR_ARG, "FW_OPT_WAIT_LIMIT must be >= 0");
      c->wait_limit = value;
      drop_graphs(c);  // they hold the limit
      return FW_OK;
    case FW_OPT_TEST_WITHHOLD:
      if (value < -1) return fail(c, FW_ERR_ARG, "FW_OPT_TEST_WITHHOLD must be >= -1");
      c->withhold_cta = value;
      drop_graphs(c);
      return FW_OK;
    case FW_OPT_STREAM_PATCH: {
      if (c->finalized) return fail(c, FW_ERR_STATE, "FW_OPT_STREAM_PATCH after fw_finalize");
      if (value != 64 && value != 128) return fail(c, FW_ERR_ARG, "FW_OPT_STREAM_PATCH must be 64 or 128");
      c->st_nodes = value;
      c->st_minb = value == 64 ? 32 : 16;
      c->shape_asked = true;
      return FW_OK;
    }
    case FW_OPT_STREAM_MINB: {
      if (!stream_kernel(c->st_nodes, value, 0))
        return fail(c, FW_ERR_ARG, "FW_OPT_STREAM_MINB: %d-node patches are built for %s CTAs per SM", c->st_nodes,
                    c->st_nodes == 64 ? "16, 20, 24 or 32" : "8, 10, 12 or 16");
      c->st_minb = value;
      if (c->st_bulk && !stream_kernel(c->st_nodes, value, 1)) c->st_bulk = 0;  // loads-only budget
      if (!c->finalized) c->shape_asked = true;
      drop_graphs(c);
      return FW_OK;
    }
    case FW_OPT_STREAM_BULK: {
      if (value != 0 && value != 1) return fail(c, FW_ERR_ARG, "FW_OPT_STREAM_BULK must be 0 or 1");
      if (value && c->finalized && c->path == FW_PATH_STREAM && c->st_smem_bulk + 64 > (size_t)shared_optin(c))
        return fail(c, FW_ERR_ARG, "FW_OPT_STREAM_BULK: the staged records do not fit in shared memory");
      if (value && !stream_kernel(c->st_nodes, c->st_minb, 1))
        return fail(c, FW_ERR_ARG, "FW_OPT_STREAM_BULK: no staged variant at %d CTAs per SM", c->st_minb);
      c->st_bulk = value;
      if (!c->finalized) c->shape_asked = true;
      drop_graphs(c);
      return FW_OK;
    }
    case FW_OPT_RES_SYNC: {
      if (c->finalized) return fail(c, FW_ERR_STATE, "FW_OPT_RES_SYNC after fw_finalize");
      if (value != 0 && value != 1) return fail(c, FW_ERR_ARG, "FW_OPT_RES_SYNC must be 0 or 1");
      c->res_sync = value;
      c->shape_asked = true;
      return FW_OK;
    }
    case FW_OPT_CLUSTER: {
      if (value != 0 && value != 1) return fail(c, FW_ERR_ARG, "FW_OPT_CLUSTER must be 0 or 1");
      if (c->finalized && value) return fail(c, FW_ERR_STATE, "FW_OPT_CLUSTER: clusters are laid out by fw_finalize");
      c->clu_opt = value;
      c->chunks_dirty = true;  // an arena's lists
      return value ? FW_OK : cluster_off(c);
    }
    default:
      return fail(c, FW_ERR_ARG, "fw_set_option: unknown option %d", option);
  }
}

int fw_get_option(const fw_ctx* c, int32_t option, int32_t* value) {
  if (!c || !value) return FW_ERR_ARG;
  switch (option) {
    case FW_OPT_FRONT_WARPS: *value = c->front_warps; return FW_OK;
    case FW_OPT_RES_THREADS: *value = c->res_threads; return FW_OK;
    case FW_OPT_BLOCK_ELEMS: *value = c->block_e; return FW_OK;
    case FW_OPT_BLOCK_NODES: *value = c->block_n; return FW_OK;
    case FW_OPT_STREAM_PATCH: *value = c->st_nodes; return FW_OK;
    case FW_OPT_STREAM_MINB: *value = c->st_minb; return FW_OK;
    case FW_OPT_STREAM_BULK: *value = c->st_bulk; return FW_OK;
    case FW_OPT_RES_SYNC: *value = c->res_sync; return FW_OK;
    case FW_OPT_CLUSTER: *value = c->clu.empty() ? 0 : (c->rest_scenes.empty() ? 1 : 2); return FW_OK;
    default: return FW_ERR_ARG;
  }
}

// A snapshot's arrays, between the context and a slot, in one launch (six copies
// took 38 us a snapshot for 4225 nodes, most of it their launches).
struct StateCopy {
  uint32_t* dst[6];
  const uint32_t* src[6];
  uint32_t words[6];
};

static __global__ void k_copy_state(StateCopy s) {
  const int part = blockIdx.y;
  const uint32_t n = s.words[part], n4 = n / 4;
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  for (uint32_t i = t; i < n4; i += stride) reinterpret_cast<uint4*>(s.dst[part])[i] = reinterpret_cast<const uint4*>(s.src[part])[i];
  for (uint32_t i = 4 * n4 + t; i < n; i += stride) s.dst[part][i] = s.src[part][i];
}

static int copy_state(fw_ctx* c, const fw_ctx::Snap& sn, bool save) {
  // every array is an allocation of its own: 16-byte aligned
  struct Part {
    void *live, *kept;
    size_t bytes;
  } parts[6] = {{c->d.x, sn.x, sizeof(float2) * (size_t)c->N},
                {c->d.v, sn.v, sizeof(float2) * (size_t)c->N},
                {c->d.j2state, sn.j2, sizeof(float4) * (size_t)(c->d.has_j2 ? c->E : 0)},
                {c->d.scene_counter, sn.counter, sizeof(int32_t) * (size_t)c->S},
                {c->d.aabb_ring, sn.ring, sizeof(int32_t) * 8 * (size_t)c->B},
                {c->d.scene_mode_req, sn.mode_req, sizeof(int32_t) * (size_t)c->S}};
  StateCopy s{};
  size_t most = 0;
  for (int k = 0; k < 6; ++k) {
    s.dst[k] = (uint32_t*)(save ? parts[k].kept : parts[k].live);
    s.src[k] = (const uint32_t*)(save ? parts[k].live : parts[k].kept);
    s.words[k] = (uint32_t)(parts[k].bytes / 4);
    most = std::max(most, parts[k].bytes / 16);
  }
  const unsigned gx = (unsigned)std::min<size_t>(std::max<size_t>((most + 255) / 256, 1), 4 * (size_t)c->sms);
  k_copy_state<<<dim3(gx, 6), 256, 0, c->stream>>>(s);
  c->launches += 1;
  return check_kernel(c, "state copy");
}

int fw_snapshot(fw_ctx* c, int32_t slot) {
  if (c && c->has_rigid) return fail(c, FW_ERR_STATE, "snapshots do not hold the rigid bodies' state");
  if (c && c->has_flex)
    return fail(c, FW_ERR_STATE, "snapshots do not hold the FEM-FEM contact state (hash, element caches)");
  if (!c) return FW_ERR_ARG;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_snapshot before fw_finalize");
  if (slot < 0 || slot >= 1024) return fail(c, FW_ERR_ARG, "fw_snapshot: slot outside [0, 1024)");
  if ((int)c->snaps.size() <= slot) c->snaps.resize(slot + 1);
  fw_ctx::Snap& sn = c->snaps[slot];
  const size_t E = c->d.has_j2 ? c->E : 1;
  int rc;
  if (!sn.x) {
    if ((rc = dalloc(c, &sn.x, c->N)) || (rc = dalloc(c, &sn.v, c->N)) || (rc = dalloc(c, &sn.j2, E)) ||
        (rc = dalloc(c, &sn.counter, c->S)) || (rc = dalloc(c, &sn.ring, 8 * (size_t)c->B)) ||
        (rc = dalloc(c, &sn.mode_req, c->S)))
      return rc;
  }
  if ((rc = copy_state(c, sn, true))) return rc;
  sn.host_counter = c->host_counter;
  sn.valid = true;
  return FW_OK;
}

int fw_restore(fw_ctx* c, int32_t slot) {
  if (c && c->has_rigid) return fail(c, FW_ERR_STATE, "snapshots do not hold the rigid bodies' state");
  if (c && c->has_flex)
    return fail(c, FW_ERR_STATE, "snapshots do not hold the FEM-FEM contact state (hash, element caches)");
  if (!c) return FW_ERR_ARG;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_restore before fw_finalize");
  if (slot < 0 || slot >= (int)c->snaps.size() || !c->snaps[slot].valid)
    return fail(c, FW_ERR_ARG, "fw_restore: slot %d holds no snapshot", slot);
  fw_ctx::Snap& sn = c->snaps[slot];
  if (int rc = copy_state(c, sn, false)) return rc;
  c->host_counter = sn.host_counter;
  return FW_OK;
}


int fw_arena_init(fw_ctx* c, int64_t max_nodes, int64_t max_elems, int32_t max_bodies, int32_t max_scenes,
                  int32_t max_pairs, int64_t max_heights, int64_t max_occ) {
  if (!c) return FW_ERR_ARG;
  if (c->device < 0) return fail(c, FW_ERR_STATE, "fw_arena_init on a staging context (fw_create_stage)");
  if (c->finalized) return fail(c, FW_ERR_STATE, "fw_arena_init on a finalized context");
  if (max_nodes <= 0 || max_elems <= 0 || max_bodies <= 0 || max_scenes <= 0 || max_pairs < 0 ||
      max_heights < 0 || max_occ < 0)
    return fail(c, FW_ERR_ARG, "fw_arena_init: capacities must be positive");
  if (max_nodes >= (1ll << 31) / 2 || 3 * max_elems >= (1ll << 31) || max_bodies >= (1 << 22))
    return fail(c, FW_ERR_ARG, "fw_arena_init: capacity beyond 32-bit indexing");
  FW_CUDA(c, cudaSetDevice(c->device));
  const int64_t N = max_nodes, E = max_elems;
  const int B = max_bodies, S = max_scenes + 1;  // scene S-1: the dead scene of free bodies
  Dev& d = c->d;
  d = Dev{};
  d.N = (int)N; d.E = (int)E; d.B = B; d.S = S; d.P = max_pairs; d.has_j2 = 1;
  int rc;
  if ((rc = dalloc(c, &d.x0, N)) || (rc = dalloc(c, &d.x, N)) || (rc = dalloc(c, &d.v, N)) ||
      (rc = dalloc(c, &d.bcv, N)) || (rc = dalloc(c, &d.node_word, N)) || (rc = dalloc(c, &d.mass, N)) ||
      (rc = dalloc(c, &d.csr_off, N)) || (rc = dalloc(c, &d.csr_end, N)) || (rc = dalloc(c, &d.csr_slot, 3 * E)) ||
      (rc = dalloc(c, &d.corner_pos, 3 * E)) ||
      (rc = dalloc(c, &d.conn, 3 * E)) || (rc = dalloc(c, &d.jinv, E)) || (rc = dalloc(c, &d.emat, E)) ||
      (rc = dalloc(c, &d.j2par, E)) || (rc = dalloc(c, &d.j2state, E)) || (rc = dalloc(c, &d.ndmass, E)) ||
      (rc = dalloc(c, &d.corner, 3 * E)) || (rc = dalloc(c, &d.body_scene, B)) ||
      (rc = dalloc(c, &d.body_pair_off, B)) || (rc = dalloc(c, &d.body_pair_cnt, B)) ||
      (rc = dalloc(c, &d.body_lm, B)) ||
      (rc = dalloc(c, &d.pairs, max_pairs)) || (rc = dalloc(c, &d.pair_active, max_pairs)) ||
      (rc = dalloc(c, &d.heights, max_heights)) || (rc = dalloc(c, &d.occ, max_occ)) ||
      (rc = dalloc(c, &d.scene_dt, S)) || (rc = dalloc(c, &d.scene_damp, S)) ||
      (rc = dalloc(c, &d.scene_counter, S)) || (rc = dalloc(c, &d.scene_active, S)) ||
      (rc = dalloc(c, &d.scene_mode_req, S)) || (rc = dalloc(c, &d.scene_mode, S)) ||
      (rc = dalloc(c, &d.aabb_ring, 8 * (size_t)B)) || (rc = dalloc(c, &c->a_young, E)) ||
      (rc = dalloc(c, &c->a_poisson, E)) || (rc = dalloc(c, &c->a_rho, E)) || (rc = dalloc(c, &d.scene_bad, S)))
    return rc;
  FW_CUDA(c, cudaMemsetAsync(d.scene_bad, 0, sizeof(int32_t) * S, c->stream));
  c->stage_cap = (size_t)64 << 20;  // packs up to 64 MB commit in one copy (larger ones part by part)
  if ((rc = dalloc(c, &c->d_stage, c->stage_cap))) return rc;
  c->chunk_cap = E / 32 + N / 32 + 2 * (int64_t)S + 16;
  if ((rc = dalloc(c, &c->d_echunks, c->chunk_cap)) || (rc = dalloc(c, &c->d_nchunks, c->chunk_cap))) return rc;
  std::vector<int32_t> dead(B, S - 1);
  FW_CUDA(c, cudaMemcpyAsync(d.body_scene, dead.data(), sizeof(int32_t) * B, cudaMemcpyHostToDevice, c->stream));
  FW_CUDA(c, cudaMemsetAsync(d.body_pair_cnt, 0, sizeof(int32_t) * B, c->stream));
  FW_CUDA(c, cudaMemsetAsync(d.body_pair_off, 0, sizeof(int32_t) * B, c->stream));
  if (max_pairs) FW_CUDA(c, cudaMemsetAsync(d.pairs, 0, sizeof(Pair) * max_pairs, c->stream));
  FW_CUDA(c, cudaMemsetAsync(d.scene_active, 0, sizeof(int32_t) * S, c->stream));
  FW_CUDA(c, cudaMemsetAsync(d.scene_mode_req, 0, sizeof(int32_t) * S, c->stream));
  FW_CUDA(c, cudaMemsetAsync(d.scene_counter, 0, sizeof(int32_t) * S, c->stream));
  FW_CUDA(c, cudaMemsetAsync(d.scene_dt, 0, sizeof(float) * S, c->stream));
  FW_CUDA(c, cudaMemsetAsync(d.scene_damp, 0, sizeof(float) * S, c->stream));
  FW_CUDA(c, cudaMemsetAsync(d.aabb_ring, 0, sizeof(int32_t) * 8 * (size_t)B, c->stream));
  FW_CUDA(c, cudaMemsetAsync(d.j2state, 0, sizeof(float4) * E, c->stream));
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  d.use_chunks = 1;
  d.e_chunks = c->d_echunks;
  d.n_chunks = c->d_nchunks;
  c->fl_nodes.init(N);
  c->fl_elems.init(E);
  c->fl_bodies.init(B);
  c->fl_pairs.init(max_pairs);
  c->fl_heights.init(max_heights);
  c->fl_occ.init(max_occ);
  c->occ_cap = max_occ;
  c->ascenes.assign(S, fw_ctx::ArenaScene{});
  c->a_body_scene.assign(B, S - 1);
  c->free_scene_ids.clear();
  for (int s2 = S - 2; s2 >= 0; --s2) c->free_scene_ids.push_back(s2);
  c->cur_active.assign(S, 0);
  c->N = (int)N; c->E = (int)E; c->B = B; c->S = S;
  cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, c->device);
  if ((rc = alloc_flags(c))) return rc;
  c->arena = true;
  c->finalized = true;
  c->path = FW_PATH_GATHER;
  c->chunks_dirty = true;
  if (c->path_req == FW_PATH_STREAM) {
    // stream arena: record capacities (patches of a body: at most nodes / patch + 1;
    // patch triangles and halo nodes: at most twice the triangles / nodes, a
    // scene needing more waits like any scene that does not fit)
    const int64_t Pcap = N / c->st_nodes + B + 16, Hcap = 2 * N, Tcap = 2 * E, CPcap = N + Pcap;
    StreamPatch* dp = nullptr;
    int32_t *dn = nullptr, *dh = nullptr, *de = nullptr;
    uint2* dc = nullptr;
    uint16_t *dcp = nullptr, *dcs = nullptr;
    StreamElem* dse = nullptr;
    StreamNode* dsn = nullptr;
    if ((rc = dalloc(c, &dp, Pcap)) || (rc = dalloc(c, &dn, N)) || (rc = dalloc(c, &dh, Hcap)) ||
        (rc = dalloc(c, &de, Tcap)) || (rc = dalloc(c, &dc, Tcap)) || (rc = dalloc(c, &dcp, CPcap)) ||
        (rc = dalloc(c, &dcs, 3 * E)) || (rc = dalloc(c, &dse, Tcap)) || (rc = dalloc(c, &dsn, N)) ||
        (rc = dalloc(c, &c->d_plist, Pcap)) || (rc = dalloc(c, &c->d_budget, S)) ||
        (rc = dalloc(c, &c->d_budget2, S)) || (rc = dalloc(c, &c->d_dt2, S)) ||
        (rc = dalloc(c, &c->d_slist, S)) || (rc = dalloc(c, &c->d_srng, S)) ||
        (rc = dalloc(c, &d.x_alt, N)) ||
        (rc = dalloc(c, &d.j2_alt, E)))
      return rc;
    c->sd = StreamDev{dp, dn, dh, de, dc, dcp, dcs, 1, 1, 1, dse, dsn, c->d_flags + fw_ctx::kFlagStream, c->d_plist};
    c->fl_patch.init(Pcap);
    c->fl_halo.init(Hcap);
    c->fl_ptri.init(Tcap);
    c->st_ptri_cap = Tcap;
    c->fl_csrp.init(CPcap);
    if (c->clu_opt) {
      const int64_t Qcap = N / kCluServedNodes * 2 + 16 * (int64_t)S, Bcap = 24 * N + 32 * E + 256 * Qcap;
      const size_t mark = c->allocs.size();
      if (dalloc_spare(c, &c->d_cblob, Bcap) && dalloc_spare(c, &c->d_cscene, S) && dalloc_spare(c, &c->d_runs, S) &&
          dalloc_spare(c, &c->d_cpatch, Qcap)) {
        if ((rc = clu_prepare(c, &c->clu_cap, c->clu_size_ok))) return rc;
        c->fl_cpatch.init(Qcap);
        c->fl_cblob.init(Bcap);
      } else {  // no room: the stream kernels step every scene
        dfree_from(c, mark);
        c->d_cblob = nullptr;
        c->d_cscene = nullptr;
        c->d_runs = nullptr;
      }
    }
    stream_smem(1, 1, 1, &c->st_smem, &c->st_smem_bulk);
    if ((rc = stream_attrs(c, shared_optin(c)))) return rc;
    c->st_list_n = 0;
    c->x_buf0 = d.x;
    c->a_stream = true;
    c->path = FW_PATH_STREAM;
    FW_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  c->h_x.clear(); c->h_conn.clear(); c->h_pairs.clear(); c->h_heights.clear(); c->h_occ.clear();
  return FW_OK;
}

int fw_arena_pack(fw_ctx* stage, int32_t patch_nodes, int32_t flags, fw_pack** out) {
  if (!stage || !out) return FW_ERR_ARG;
  *out = nullptr;
  if (stage->finalized && !stage->arena)
    return fail(stage, FW_ERR_STATE, "fw_arena_pack: stage on a context that is not finalized, or on an arena");
  return guarded(stage, [&] { return build_pack(stage, patch_nodes, (flags & FW_PACK_PINNED) != 0, out); });
}

int fw_pack_info(const fw_pack* pk, int64_t* info) {
  if (!pk || !info) return FW_ERR_ARG;
  info[0] = pk->dev_bytes; info[1] = pk->Ns; info[2] = pk->Es; info[3] = pk->Bs;
  info[4] = pk->patch_nodes; info[5] = pk->Ps; info[6] = pk->Ts; info[7] = pk->pinned ? 1 : 0;
  return FW_OK;
}

void fw_pack_destroy(fw_pack* pk) { delete pk; }

int fw_arena_commit_pack(fw_ctx* c, const fw_pack* pk, int32_t* scene_out) {
  if (!c || !pk || !scene_out) return FW_ERR_ARG;
  if (!c->arena) return fail(c, FW_ERR_STATE, "fw_arena_commit_pack without fw_arena_init");
  if (c->a_stream && pk->patch_nodes != c->st_nodes)
    return fail(c, FW_ERR_ARG, "fw_arena_commit_pack: the pack is cut into %d-node patches, the arena steps %d-node "
                               "patches", pk->patch_nodes, c->st_nodes);
  if (c->free_scene_ids.empty()) return fail(c, FW_ERR_OOM, "arena: no free scene slot");
  if (c->a_stream && pk->mixed && !c->sd.lm) {
    // the first such scene: Lame constants per triangle from here on, for the resident scenes as well
    float2* lm = nullptr;
    if (int rl = dalloc(c, &lm, (size_t)c->st_ptri_cap)) return rl;
    c->sd.lm = lm;
    for (const fw_ctx::ArenaScene& o : c->ascenes)
      if (o.live && o.nt > 0) {
        k_stream_elems<<<(int)((o.nt + kBlock - 1) / kBlock), kBlock, 0, c->stream>>>(
            c->d, c->sd.eid + o.t0, c->sd.conn + o.t0, c->sd.elem + o.t0, lm + o.t0, (int)o.nt);
        c->launches += 1;
      }
    if (int rk = check_kernel(c, "arena records")) return rk;
  }
  fw_ctx::ArenaScene a;
  a.nn = pk->Ns; a.ne = pk->Es; a.nb = pk->Bs; a.np = pk->Np; a.nh = pk->Nh; a.no = pk->No;
  if (c->a_stream) { a.npp = pk->Ps; a.nhh = pk->Hs; a.nt = pk->Ts; a.ncp = pk->CPs; }
  fw_ctx::FreeList* lists[10] = {&c->fl_nodes, &c->fl_elems, &c->fl_bodies, &c->fl_pairs, &c->fl_heights,
                                 &c->fl_occ, &c->fl_patch, &c->fl_halo, &c->fl_ptri, &c->fl_csrp};
  int64_t* offs[10] = {&a.n0, &a.e0, &a.b0, &a.p0, &a.h0, &a.o0, &a.pp0, &a.hh0, &a.t0, &a.cp0};
  const int64_t lens[10] = {a.nn, a.ne, a.nb, a.np, a.nh, a.no, a.npp, a.nhh, a.nt, a.ncp};
  const int nl = c->a_stream ? 10 : 6;
  for (int k = 0; k < nl; ++k)
    if (!lists[k]->take(lens[k], offs[k])) {
      for (int j = 0; j < k; ++j) lists[j]->give(*offs[j], lens[j]);
      return fail(c, FW_ERR_OOM, "arena: not enough free capacity for this scene");
    }
  // stream arenas: the launch's shared memory covers the largest patch so far
  int no_max = c->sd.no_max, nh_max = c->sd.nh_max, ne_max = c->sd.ne_max;
  size_t smem = c->st_smem, smem_bulk = c->st_smem_bulk;
  if (c->a_stream) {
    no_max = std::max(no_max, pk->no_max);
    nh_max = std::max(nh_max, pk->nh_max);
    ne_max = std::max(ne_max, pk->ne_max);
    stream_smem(no_max, nh_max, ne_max, &smem, &smem_bulk);
    if ((long)smem > shared_optin(c) - 64) {
      for (int j = 0; j < nl; ++j) lists[j]->give(*offs[j], lens[j]);
      return fail(c, FW_ERR_ARG, "arena: a patch of this scene needs %zu B of shared memory", smem);
    }
  }
  // cluster patches, where the device and the arena have room; else the stream kernels step the scene
  a.clu = pk->clu;
  a.ncq = (int64_t)(pk->len[fw_pack::CPATCH] / sizeof(CluPatch));
  a.ncb = (int64_t)pk->len[fw_pack::CBLOB];
  if (!c->d_cpatch || !a.clu.ctas || !c->clu_size_ok[a.clu.ctas] || clu_smem(a.clu) > c->clu_cap) a.clu.ctas = 0;
  if (a.clu.ctas && !c->fl_cpatch.take(a.ncq, &a.cq0)) a.clu.ctas = 0;
  else if (a.clu.ctas && !c->fl_cblob.take(a.ncb, &a.cb0)) {
    c->fl_cpatch.give(a.cq0, a.ncq);
    a.clu.ctas = 0;
  }
  const int s = c->free_scene_ids.back();
  c->free_scene_ids.pop_back();
  a.live = true;
  c->energy_dirty = true;
  // upload (queued on the stream: the steps that follow see the scene, and a
  // pinned pack's copy runs asynchronously): the whole pack in one copy to
  // the device staging buffer, then one kernel puts each part in its range
  Dev& d = c->d;
  const int64_t n0 = a.n0, e0 = a.e0;
  static_assert(kScatterParts == fw_pack::NPARTS + 1, "one scatter slot per pack part, plus the current positions");
  unsigned char* dst[fw_pack::NPARTS] = {};
  auto B = [](const void* p) { return (unsigned char*)const_cast<void*>(p); };
  dst[fw_pack::X0] = B(d.x0 + n0); dst[fw_pack::V0] = B(d.v + n0); dst[fw_pack::BCV] = B(d.bcv + n0);
  dst[fw_pack::WORD] = B(d.node_word + n0); dst[fw_pack::CBEG] = B(d.csr_off + n0); dst[fw_pack::CEND] = B(d.csr_end + n0);
  dst[fw_pack::SLOT] = B(d.csr_slot + 3 * e0); dst[fw_pack::CPOS] = B(d.corner_pos + 3 * e0);
  dst[fw_pack::CONN] = B(d.conn + 3 * e0); dst[fw_pack::EMAT] = B(d.emat + e0); dst[fw_pack::J2PAR] = B(d.j2par + e0);
  dst[fw_pack::YOUNG] = B(c->a_young + e0); dst[fw_pack::POISSON] = B(c->a_poisson + e0);
  dst[fw_pack::RHO] = B(c->a_rho + e0); dst[fw_pack::POFF] = B(d.body_pair_off + a.b0);
  dst[fw_pack::PCNT] = B(d.body_pair_cnt + a.b0); dst[fw_pack::PAIRS] = B(d.pairs + a.p0);
  dst[fw_pack::HEIGHTS] = B(d.heights + a.h0); dst[fw_pack::OCC] = B(d.occ + a.o0);
  if (c->a_stream) {
    dst[fw_pack::RN] = B(c->sd.nodes + n0); dst[fw_pack::RH] = B(c->sd.halo + a.hh0); dst[fw_pack::RE] = B(c->sd.eid + a.t0);
    dst[fw_pack::RC] = B(c->sd.conn + a.t0); dst[fw_pack::RCP] = B(c->sd.csrp + a.cp0);
    dst[fw_pack::RCS] = B(c->sd.csrs + 3 * e0); dst[fw_pack::PATCH] = B(c->sd.patch + a.pp0);
  }
  if (a.clu.ctas) {
    dst[fw_pack::CPATCH] = B(c->d_cpatch + a.cq0);
    dst[fw_pack::CBLOB] = B(c->d_cblob + a.cb0);
  }
  if (pk->bytes <= c->stage_cap) {
    FW_CUDA(c, cudaMemcpyAsync(c->d_stage, pk->block, pk->bytes, cudaMemcpyHostToDevice, c->stream));
    ArenaScatter sc{};
    uint32_t most = 0;
    for (int k = 0; k < fw_pack::NPARTS; ++k) {
      sc.dst[k] = dst[k];
      sc.off[k] = (uint32_t)pk->off[k];
      sc.len[k] = dst[k] ? (uint32_t)pk->len[k] : 0u;
      most = std::max(most, sc.len[k]);
    }
    sc.dst[fw_pack::NPARTS] = B(d.x + n0);  // the current positions start at the rest positions
    sc.off[fw_pack::NPARTS] = (uint32_t)pk->off[fw_pack::X0];
    sc.len[fw_pack::NPARTS] = (uint32_t)pk->len[fw_pack::X0];
    const int gx = (int)std::max<uint32_t>(1u, std::min<uint32_t>((most / 4 + kBlock - 1) / kBlock, 256u));
    k_arena_scatter<<<dim3(gx, kScatterParts), kBlock, 0, c->stream>>>(c->d_stage, sc);
    c->launches += 1;
  } else {  // larger than the staging buffer: one copy per part
    for (int k = 0; k < fw_pack::NPARTS; ++k)
      if (dst[k] && pk->len[k])
        FW_CUDA(c, cudaMemcpyAsync(dst[k], pk->at((fw_pack::Part)k), pk->len[k], cudaMemcpyHostToDevice, c->stream));
    FW_CUDA(c, cudaMemcpyAsync(d.x + n0, pk->at(fw_pack::X0), pk->len[fw_pack::X0], cudaMemcpyHostToDevice, c->stream));
  }
  FW_CUDA(c, cudaMemsetAsync(d.j2state + e0, 0, sizeof(float4) * a.ne, c->stream));
  ArenaReloc r{};
  r.n0 = (int)n0; r.e0 = (int)e0; r.b0 = (int)a.b0; r.p0 = (int)a.p0; r.h0 = (int)a.h0; r.o0 = (int)a.o0; r.s = s;
  r.Ns = (int)a.nn; r.Es = (int)a.ne; r.Bs = (int)a.nb; r.Np = (int)a.np;
  r.damp = pk->damp;
  if (c->a_stream) {
    r.rn = const_cast<int32_t*>(c->sd.nodes) + n0;
    r.rh = const_cast<int32_t*>(c->sd.halo) + a.hh0;
    r.re = const_cast<int32_t*>(c->sd.eid) + a.t0;
    r.Hs = (int)a.nhh;
    r.Ts = (int)a.nt;
    r.patch = const_cast<StreamPatch*>(c->sd.patch) + a.pp0;
    r.Ps = (int)a.npp;
    r.hh0 = (int)a.hh0;
    r.t0 = (int)a.t0;
    r.cp0 = (int)a.cp0;
    r.srng = c->d_srng;
  }
  r.count = std::max<int64_t>({3 * a.ne, a.nn, a.nb, a.np, a.nhh, a.nt, a.npp});
  k_arena_reloc<<<(int)std::min<int64_t>((r.count + kBlock - 1) / kBlock, 8 * c->sms), kBlock, 0, c->stream>>>(d, r);
  const int e_lo = (int)e0, e_hi = (int)(e0 + a.ne), n_lo = (int)n0, n_hi = (int)(n0 + a.nn);
  if (a.np > 0 && a.no > 0) {
    // the arena's first voxel pairs: the cell table, eight times the cells'
    // bytes, which arenas without such pairs do not need (no room for it: the
    // grids are walked)
    if (!c->vox_asked) dalloc_spare(c, &d.vox, (size_t)c->occ_cap);
    c->vox_asked = true;
    if (d.vox) k_voxel_table<<<dim3((unsigned)a.np, kVoxelBlocks), 32, 0, c->stream>>>(d, (int)a.p0);
  }
  k_prepare_elements<<<(int)((a.ne + kBlock - 1) / kBlock), kBlock, 0, c->stream>>>(d, c->a_young + e0, c->a_poisson + e0,
                                                                                  c->a_rho + e0, e_lo, e_hi);
  k_prepare_mass<<<(int)((a.nn + kBlock - 1) / kBlock), kBlock, 0, c->stream>>>(d, n_lo, n_hi);
  c->launches += 3;
  if (c->a_stream) {
    if (a.nt > 0)
      k_stream_elems<<<(int)((a.nt + kBlock - 1) / kBlock), kBlock, 0, c->stream>>>(
          d, c->sd.eid + a.t0, c->sd.conn + a.t0, c->sd.elem + a.t0, c->sd.lm ? c->sd.lm + a.t0 : nullptr, (int)a.nt);
    k_stream_nodes<<<(int)((a.nn + kBlock - 1) / kBlock), kBlock, 0, c->stream>>>(d, c->sd.nodes + n0,
                                                                                  c->sd.node + n0, (int)a.nn);
    c->launches += 2;
    c->sd.no_max = no_max; c->sd.nh_max = nh_max; c->sd.ne_max = ne_max;
    c->st_smem = smem;
    c->st_smem_bulk = smem_bulk;
    if ((long)smem_bulk > shared_optin(c) - 64) c->st_bulk = 0;  // staging no longer fits: plain loads
  }
  int rc;
  if ((rc = check_kernel(c, "arena commit"))) return rc;
  c->ascenes[s] = a;
  for (int64_t b = 0; b < a.nb; ++b) c->a_body_scene[a.b0 + b] = s;
  c->cur_active[s] = 1;
  c->chunks_dirty = true;
  *scene_out = s;
  return FW_OK;
}

int fw_arena_commit(fw_ctx* c, int32_t* scene_out) {
  if (!c || !scene_out) return FW_ERR_ARG;
  if (!c->arena) return fail(c, FW_ERR_STATE, "fw_arena_commit without fw_arena_init");
  fw_pack* pk = nullptr;
  int rc = guarded(c, [&] { return build_pack(c, c->a_stream ? c->st_nodes : 0, false, &pk); });
  if (rc) return rc;
  rc = fw_arena_commit_pack(c, pk, scene_out);
  delete pk;  // pageable: its copies were staged before they returned
  return rc;
}

int fw_arena_remove(fw_ctx* c, int32_t s) {
  if (!c) return FW_ERR_ARG;
  if (!c->arena) return fail(c, FW_ERR_STATE, "fw_arena_remove without fw_arena_init");
  if (s < 0 || s >= c->S - 1 || !c->ascenes[s].live) return fail(c, FW_ERR_ARG, "fw_arena_remove: scene %d is not live", s);
  fw_ctx::ArenaScene& a = c->ascenes[s];
  std::vector<int32_t> dead(a.nb, c->S - 1);
  const int32_t zero = 0;
  FW_CUDA(c, cudaMemcpyAsync(c->d.body_scene + a.b0, dead.data(), sizeof(int32_t) * a.nb, cudaMemcpyHostToDevice, c->stream));
  FW_CUDA(c, cudaMemcpyAsync(c->d.scene_active + s, &zero, sizeof(int32_t), cudaMemcpyHostToDevice, c->stream));
  FW_CUDA(c, cudaMemcpyAsync(c->d.scene_bad + s, &zero, sizeof(int32_t), cudaMemcpyHostToDevice, c->stream));
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  for (int64_t b = 0; b < a.nb; ++b) c->a_body_scene[a.b0 + b] = c->S - 1;
  c->fl_nodes.give(a.n0, a.nn);
  c->fl_elems.give(a.e0, a.ne);
  c->fl_bodies.give(a.b0, a.nb);
  c->fl_pairs.give(a.p0, a.np);
  c->fl_heights.give(a.h0, a.nh);
  c->fl_occ.give(a.o0, a.no);
  if (c->a_stream) {
    c->fl_patch.give(a.pp0, a.npp);
    c->fl_halo.give(a.hh0, a.nhh);
    c->fl_ptri.give(a.t0, a.nt);
    c->fl_csrp.give(a.cp0, a.ncp);
  }
  if (a.clu.ctas) {
    c->fl_cpatch.give(a.cq0, a.ncq);
    c->fl_cblob.give(a.cb0, a.ncb);
  }
  a = fw_ctx::ArenaScene{};
  c->energy_dirty = true;
  c->cur_active[s] = 0;
  c->free_scene_ids.push_back(s);
  c->chunks_dirty = true;
  return FW_OK;
}

int fw_step_served(fw_ctx* c, const float* dt) { return fw_step_served_n(c, dt, 1); }

int fw_step_served_n(fw_ctx* c, const float* dt, int32_t n_steps) {
  if (!c || !dt || n_steps < 0) return FW_ERR_ARG;
  if (n_steps == 0) return FW_OK;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_step_served before fw_finalize / fw_arena_init");
  bool changed = false;
  for (int s = 0; s < c->S; ++s) {
    const int want = (dt[s] > 0.0f && (!c->arena || c->ascenes[s].live)) ? 1 : 0;
    if (want != c->cur_active[s]) {
      c->cur_active[s] = want;
      changed = true;
    }
  }
  if (changed) {
    FW_CUDA(c, cudaMemcpyAsync(c->d.scene_active, c->cur_active.data(), sizeof(int32_t) * c->S,
                               cudaMemcpyHostToDevice, c->stream));
    c->chunks_dirty = true;
  }
  c->cur_dt.assign(dt, dt + c->S);
  FW_CUDA(c, cudaMemcpyAsync(c->d.scene_dt, c->cur_dt.data(), sizeof(float) * c->S, cudaMemcpyHostToDevice,
                             c->stream));
  c->d.uniform_dt = 0;
  if (c->arena && c->a_stream) return arena_stream_steps(c, n_steps);
  int rc;
  if (c->arena && (rc = rebuild_chunks(c))) return rc;
  for (int k = 0; k < n_steps; ++k)
    if ((rc = launch_step(c))) return rc;
  return FW_OK;
}

int fw_step_served_budget(fw_ctx* c, const float* dt, const int32_t* budget, const float* dt_next,
                          const int32_t* budget_next, int32_t n_steps) {
  if (!c || !dt || !budget || n_steps < 0 || (!dt_next) != (!budget_next)) return FW_ERR_ARG;
  if (!c->arena || !c->a_stream)
    return fail(c, FW_ERR_STATE, "fw_step_served_budget needs a stream arena (fw_set_path FW_PATH_STREAM before "
                                 "fw_arena_init)");
  if (n_steps == 0) return FW_OK;
  // staged before the calls return
  c->h_budget.assign(budget, budget + c->S);
  FW_CUDA(c, cudaMemcpyAsync(c->d_budget, c->h_budget.data(), sizeof(int32_t) * c->S, cudaMemcpyHostToDevice,
                             c->stream));
  c->d.scene_budget = c->d_budget;
  if (budget_next) {
    c->h_budget2.assign(budget_next, budget_next + c->S);
    c->h_dt2.assign(dt_next, dt_next + c->S);
    FW_CUDA(c, cudaMemcpyAsync(c->d_budget2, c->h_budget2.data(), sizeof(int32_t) * c->S, cudaMemcpyHostToDevice,
                               c->stream));
    FW_CUDA(c, cudaMemcpyAsync(c->d_dt2, c->h_dt2.data(), sizeof(float) * c->S, cudaMemcpyHostToDevice, c->stream));
    c->d.scene_budget_next = c->d_budget2;
    c->d.scene_dt_next = c->d_dt2;
  }
  const int rc = fw_step_served_n(c, dt, n_steps);
  c->d.scene_budget = nullptr;
  c->d.scene_budget_next = nullptr;
  c->d.scene_dt_next = nullptr;
  return rc;
}

int fw_arena_scene_info(fw_ctx* c, int32_t s, int64_t* info) {
  if (!c || !info) return FW_ERR_ARG;
  if (!c->arena) return fail(c, FW_ERR_STATE, "fw_arena_scene_info without fw_arena_init");
  if (s < 0 || s >= c->S - 1 || !c->ascenes[s].live) return fail(c, FW_ERR_ARG, "scene %d is not live", s);
  const fw_ctx::ArenaScene& a = c->ascenes[s];
  info[0] = a.n0; info[1] = a.nn; info[2] = a.e0; info[3] = a.ne; info[4] = a.b0; info[5] = a.nb;
  info[6] = c->fl_nodes.total(); info[7] = c->fl_elems.total();
  return FW_OK;
}


int fw_set_element_young(fw_ctx* c, int32_t first, int32_t count, const float* young, int32_t on_device) {
  if (!c || !young) return FW_ERR_ARG;
  // (the resident step loads the Lame constants at every launch; the stream path's
  // patch records are rebuilt below)
  if (!c->finalized || c->arena)
    return fail(c, FW_ERR_STATE, "fw_set_element_young needs a finalized world (not an arena)");
  if (first < 0 || count < 0 || (int64_t)first + count > c->E) return fail(c, FW_ERR_ARG, "element range out of bounds");
  if (c->has_springs) return fail(c, FW_ERR_STATE, "fw_set_element_young: the world has spring-mass domains");
  if (count == 0) return FW_OK;
  int rc;
  if (!c->d_poisson && (rc = upload(c, &c->d_poisson, c->h_nu))) return rc;
  if (!c->adj.young && (rc = upload(c, &c->adj.young, c->h_E))) return rc;
  float* dst = c->adj.young + first;
  FW_CUDA(c, cudaMemcpyAsync(dst, young, sizeof(float) * count,
                             on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, c->stream));
  k_set_young<<<(count + kBlock - 1) / kBlock, kBlock, 0, c->stream>>>(c->d, dst, c->d_poisson, first, first + count);
  c->launches += 1;
  if ((rc = check_kernel(c, "set young"))) return rc;
  if ((rc = cluster_per_tri(c))) return rc;
  if (c->path != FW_PATH_STREAM) return FW_OK;
  // a body's triangles may now differ: the stream records take their Lame
  // constants per triangle from here on
  if (!c->sd.lm) {
    if ((rc = dalloc(c, &c->sd.lm, (size_t)std::max(1, c->st_ne)))) return rc;
    drop_graphs(c);
  }
  return stream_records(c);
}

int fw_adj_begin(fw_ctx* c, int32_t max_segment_steps) {
  if (c && (c->has_flex || c->has_springs || c->has_rigid))
    return fail(c, FW_ERR_STATE, "the adjoint covers FEM triangles without FEM-FEM contact");
  if (!c) return FW_ERR_ARG;
  // The forward may run on either path (identical bits); the recompute and the
  // reverse use the gather kernels and data, which every non-arena world has.
  if (!c->finalized || c->arena || c->S != 1 || c->path == FW_PATH_STREAM)
    return fail(c, FW_ERR_STATE, "the adjoint needs a finalized single-scene world on the gather or resident path");
  if (max_segment_steps <= 0) return fail(c, FW_ERR_ARG, "max_segment_steps must be > 0");
  int rc;
  Adj& a = c->adj;
  if (!a.young) {
    if ((rc = upload(c, &a.young, c->h_E))) return rc;
  }
  if (!a.xb) {
    if ((rc = dalloc(c, &a.xb, c->N)) || (rc = dalloc(c, &a.vb, c->N)) || (rc = dalloc(c, &a.fb, c->N)) ||
        (rc = dalloc(c, &a.Eb, c->E)) || (rc = dalloc(c, &a.io_x, c->N)) || (rc = dalloc(c, &a.io_v, c->N)) ||
        (rc = dalloc(c, &a.io_E, c->E)))
      return rc;
  }
  if (c->adj_cap < max_segment_steps) {
    drop_graphs(c);  // graphs hold the old trajectory buffers
    if ((rc = dalloc(c, &a.traj, (size_t)max_segment_steps * c->N)) ||
        (rc = dalloc(c, &a.trajv, (size_t)max_segment_steps * c->N)) ||
        (rc = dalloc(c, &a.trajs, (size_t)max_segment_steps * (c->d.has_j2 ? c->E : 1))) ||
        (rc = dalloc(c, &a.gates, (size_t)max_segment_steps * std::max(1, c->d.P))))
      return rc;
    c->adj_cap = max_segment_steps;
  }
  if (c->d.has_j2 && !a.sb) {
    if ((rc = dalloc(c, &a.sb, 4 * (size_t)c->E))) return rc;
  }
  if (a.sb) FW_CUDA(c, cudaMemsetAsync(a.sb, 0, sizeof(double) * 4 * (size_t)c->E, c->stream));
  // Reverse pass on the grid form's patches where a CTA has a thread per
  // triangle and node (64 x 64 quads: 4.4 / 2.4 us a reverse substep against
  // k_res_adj); larger patches and J2 worlds go on below.
  if (!c->clu.empty() && c->clu[0].r.grid && !c->d.has_j2 && !c->clu_adj.words) {
    CluAdj q{};
    q.r = c->clu[0].r;
    const int threads = (std::max({q.r.ne, q.r.no, q.r.nh}) + 31) / 32 * 32;
    int optin = 0, sms = 148, per_sm = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
    const size_t need = clu_adj_layout(q);
    if (threads <= 768 && need + kCluStatic <= (size_t)optin) {
      CluAdjKernel k = clu_adj_kernel(threads);
      FW_CUDA(c, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)((size_t)optin - kCluStatic)));
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, need) == cudaSuccess &&
          per_sm * sms >= q.r.ctas && dalloc_spare(c, &q.words, 4 * (size_t)q.r.n_halo)) {
        FW_CUDA(c, cudaMemsetAsync(q.words, 0, sizeof(ulonglong2) * 4 * (size_t)q.r.n_halo, c->stream));
        c->clu_adj = q;
        c->clu_adj_threads = threads;
        c->clu_adj_smem = need;
      }
    }
    cudaGetLastError();
  }
  // Resident reverse pass when the world runs resident and the adjoint state
  // fits on chip too (J2 worlds reverse on the gather kernels).
  if (c->path == FW_PATH_RESIDENT && !c->res_adj && !c->d.has_j2 && !c->clu_adj.words) {
    if (!c->clu.empty() && (rc = own_resident(c)) < 0) return rc;
  }
  if (c->path == FW_PATH_RESIDENT && !c->res_adj && !c->d.has_j2 && !c->clu_adj.words && c->res.err) {
    int optin = 0, sms = 148;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
    const size_t need = res_layout(c->res, nullptr, nullptr) + res_adj_layout(c->res, nullptr, nullptr);
    cudaFuncAttributes fa{};
    cudaFuncGetAttributes(&fa, k_res_adj);
    int per_sm = 0;
    if ((long)need + (long)fa.sharedSizeBytes + 64 <= optin &&
        cudaFuncSetAttribute(k_res_adj, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             optin - (int)fa.sharedSizeBytes) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_res_adj, kResThreads, need) == cudaSuccess &&
        per_sm * sms >= c->res.P) {
      if ((rc = dalloc(c, &c->fll, 8 * (size_t)c->N))) return rc;
      FW_CUDA(c, cudaMemsetAsync(c->fll, 0, sizeof(unsigned long long) * 8 * (size_t)c->N, c->stream));
      c->res_adj = true;
      c->res_adj_smem = need;
    }
    cudaGetLastError();
  }
  FW_CUDA(c, cudaMemsetAsync(a.Eb, 0, sizeof(double) * c->E, c->stream));
  FW_CUDA(c, cudaMemsetAsync(a.xb, 0, sizeof(double2) * c->N, c->stream));
  FW_CUDA(c, cudaMemsetAsync(a.vb, 0, sizeof(double2) * c->N, c->stream));
  return FW_OK;
}

int fw_adj_seed(fw_ctx* c, const float* xbar, const float* vbar, int32_t on_device) {
  if (!c) return FW_ERR_ARG;
  if (!c->adj.xb) return fail(c, FW_ERR_STATE, "fw_adj_seed before fw_adj_begin");
  const cudaMemcpyKind k = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
  if (xbar) FW_CUDA(c, cudaMemcpyAsync(c->adj.io_x, xbar, sizeof(float2) * c->N, k, c->stream));
  if (vbar) FW_CUDA(c, cudaMemcpyAsync(c->adj.io_v, vbar, sizeof(float2) * c->N, k, c->stream));
  k_adj_seed<<<(c->N + kBlock - 1) / kBlock, kBlock, 0, c->stream>>>(c->adj, c->N, xbar != nullptr, vbar != nullptr);
  c->launches += 1;
  FW_CUDA(c, cudaMemsetAsync(c->adj.Eb, 0, sizeof(double) * c->E, c->stream));
  if (c->adj.sb) FW_CUDA(c, cudaMemsetAsync(c->adj.sb, 0, sizeof(double) * 4 * (size_t)c->E, c->stream));
  return check_kernel(c, "adjoint seed");
}

int fw_adj_segment(fw_ctx* c, int32_t n_steps, float dt) {
  if (!c) return FW_ERR_ARG;
  if (!c->adj.xb) return fail(c, FW_ERR_STATE, "fw_adj_segment before fw_adj_begin");
  if (n_steps <= 0 || n_steps > c->adj_cap) return fail(c, FW_ERR_ARG, "n_steps outside (0, max_segment_steps]");
  Adj& a = c->adj;
  const int N = c->N, E = c->E, P = std::max(1, c->d.P);
  c->d.uniform_dt = 1;
  c->d.dt_uniform = dt;
  int rc;
  if (c->clu_adj.words && c->clu.empty()) c->clu_adj.words = nullptr;  // the forms' patches were given up (cluster_off)
  if (c->clu_adj.words) {
    // recompute on the grid form, recording positions and gates, then reverse on the same patches
    if (c->d.P > 0) FW_CUDA(c, cudaMemsetAsync(a.gates, 0, sizeof(int32_t) * (size_t)P * n_steps, c->stream));
    c->res.rec_x = a.traj;
    c->res.rec_v = a.trajv;
    c->res.rec_gates = c->d.P > 0 ? a.gates : nullptr;
    c->res.rec_stride = P;
    rc = launch_resident(c, n_steps);
    c->res.rec_x = nullptr;
    c->res.rec_v = nullptr;
    c->res.rec_gates = nullptr;
    if (rc) return rc;
    CluAdj q = c->clu_adj;
    q.r.wait_limit = c->wait_limit > 0 ? c->wait_limit : kCluWaitLimit;
    if (c->clu_adj_epoch > 0xF0000000u) {
      FW_CUDA(c, cudaMemsetAsync(q.words, 0, sizeof(ulonglong2) * 4 * (size_t)q.r.n_halo, c->stream));
      c->clu_adj_epoch = 0;
    }
    flags_may_rise(c);
    q.r.ep0 = c->clu_adj_epoch;
    c->clu_adj_epoch += (uint32_t)n_steps + 1u;
    q.rec_x = a.traj;
    q.rec_v = a.trajv;
    q.rec_gates = a.gates;
    q.gate_stride = P;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(q.r.ctas);
    cfg.blockDim = dim3(c->clu_adj_threads);
    cfg.dynamicSmemBytes = c->clu_adj_smem;
    cfg.stream = c->stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    FW_CUDA(c, cudaLaunchKernelEx(&cfg, clu_adj_kernel(c->clu_adj_threads), (const Dev)c->d, (const CluAdj)q, (const Adj)a,
                                  (int)n_steps, dt, c->h_damp.empty() ? 0.0f : c->h_damp[0]));
    c->launches += 1;
    return check_kernel(c, "adjoint segment");
  }
  if (c->res_adj) {
    // recompute on the resident step, recording positions and gates, then the resident reverse
    if (!c->clu.empty()) FW_CUDA(c, cudaMemsetAsync(a.gates, 0, sizeof(int32_t) * (size_t)P * n_steps, c->stream));
    c->res.rec_x = a.traj;
    c->res.rec_v = a.trajv;
    c->res.rec_gates = a.gates;
    c->res.rec_stride = P;
    rc = launch_resident(c, n_steps);
    c->res.rec_x = nullptr;
    c->res.rec_v = nullptr;
    c->res.rec_gates = nullptr;
    if (rc) return rc;
    if (c->res_epoch > 0xF0000000u) {
      FW_CUDA(c, cudaMemsetAsync(c->fll, 0, sizeof(unsigned long long) * 8 * (size_t)N, c->stream));
      FW_CUDA(c, cudaMemsetAsync(c->res.xll, 0, sizeof(unsigned long long) * 4 * (size_t)N, c->stream));
      FW_CUDA(c, cudaMemsetAsync(c->res.bll, 0, sizeof(unsigned long long) * 4 * (size_t)kBoxRing * c->B * c->res.P,
                                 c->stream));
      c->res_epoch = 1;
    }
    uint32_t ep0 = c->res_epoch;
    c->res_epoch += (uint32_t)n_steps + 1u;
    float damp_f = c->h_damp.empty() ? 0.0f : c->h_damp[0];
    int nn = n_steps, gs = P;
    const float2* tx = a.traj;
    const float2* tv = a.trajv;
    const int* tg = a.gates;
    void* args[] = {(void*)&c->d, (void*)&c->res, (void*)&c->adj, (void*)&tx, (void*)&tv, (void*)&tg, (void*)&gs,
                    (void*)&c->fll, (void*)&nn, (void*)&dt, (void*)&damp_f, (void*)&ep0};
    flags_may_rise(c);
    FW_CUDA(c, cudaLaunchCooperativeKernel((const void*)k_res_adj, dim3(c->res.P), dim3(kResThreads), args,
                                           c->res_adj_smem, c->stream));
    c->launches += 1;
    return check_kernel(c, "resident adjoint segment");
  }
  const uint64_t key_lo = ((uint64_t)n_steps << 32) | float_bits(dt);
  // recompute the segment from the current state, recording positions and gates
  cudaGraphExec_t g_fwd = nullptr;
  rc = cached_graph(c, c->adj_graphs, (1ull << 62) | key_lo, [&] {
    for (int j = 0; j < n_steps; ++j) {
      cudaMemcpyAsync(a.traj + (size_t)j * N, c->d.x, sizeof(float2) * N, cudaMemcpyDeviceToDevice, c->stream);
      cudaMemcpyAsync(a.trajv + (size_t)j * N, c->d.v, sizeof(float2) * N, cudaMemcpyDeviceToDevice, c->stream);
      if (c->d.has_j2)
        cudaMemcpyAsync(a.trajs + (size_t)j * E, c->d.j2state, sizeof(float4) * E, cudaMemcpyDeviceToDevice,
                        c->stream);
      k_elements<<<c->grid_e, c->block_e, 0, c->stream>>>(c->d);
      k_nodes<<<c->grid_n, c->block_n, 0, c->stream>>>(c->d);
      if (c->d.P > 0)
        cudaMemcpyAsync(a.gates + (size_t)j * P, c->d.pair_active, sizeof(int32_t) * c->d.P,
                        cudaMemcpyDeviceToDevice, c->stream);
    }
  }, &g_fwd);
  if (rc) return rc;
  FW_CUDA(c, cudaGraphLaunch(g_fwd, c->stream));
  c->host_counter += n_steps;
  c->launches += 2 * n_steps;
  // (xb, vb) hold the adjoint of the segment's end state; the segment leaves
  // the adjoint of its start state there (the checkpoint it was restored from).
  const int gn = (N + kBlock - 1) / kBlock, ge = (E + kBlock - 1) / kBlock;
  const float damp = c->h_damp.empty() ? 0.0f : c->h_damp[0];
  cudaGraphExec_t g_rev = nullptr;
  rc = cached_graph(c, c->adj_graphs, (2ull << 62) | key_lo, [&] {
    k_adj_prep<<<gn, kBlock, 0, c->stream>>>(c->d, a, dt, damp);  // force / velocity adjoints of the last substep
    for (int j = n_steps - 1; j >= 0; --j) {
      const float2* x = a.traj + (size_t)j * N;
      const float2* v = a.trajv + (size_t)j * N;
      k_adj_elements<<<ge, kBlock, 0, c->stream>>>(c->d, a, x, a.trajs + (c->d.has_j2 ? (size_t)j * E : 0));
      k_adj_nodes<<<gn, kBlock, 0, c->stream>>>(c->d, a, x, v, a.gates + (size_t)j * P, dt, damp, j > 0);
    }
  }, &g_rev);
  if (rc) return rc;
  FW_CUDA(c, cudaGraphLaunch(g_rev, c->stream));
  c->launches += 1 + 2 * n_steps;
  return check_kernel(c, "adjoint segment");
}

int fw_adj_read(fw_ctx* c, float* xbar, float* vbar, float* Ebar, int32_t on_device) {
  if (!c) return FW_ERR_ARG;
  if (!c->adj.xb) return fail(c, FW_ERR_STATE, "fw_adj_read before fw_adj_begin");
  const cudaMemcpyKind k = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
  const int n = std::max(c->N, c->E);
  k_adj_out<<<(n + kBlock - 1) / kBlock, kBlock, 0, c->stream>>>(c->adj, c->N, c->E);
  c->launches += 1;
  if (xbar) FW_CUDA(c, cudaMemcpyAsync(xbar, c->adj.io_x, sizeof(float2) * c->N, k, c->stream));
  if (vbar) FW_CUDA(c, cudaMemcpyAsync(vbar, c->adj.io_v, sizeof(float2) * c->N, k, c->stream));
  if (Ebar) FW_CUDA(c, cudaMemcpyAsync(Ebar, c->adj.io_E, sizeof(float) * c->E, k, c->stream));
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  return FW_OK;
}

int fw_tan_begin(fw_ctx* c, const float* dx0, const float* dv0, const float* dE, int32_t on_device) {
  if (c && (c->has_flex || c->has_springs || c->has_rigid))
    return fail(c, FW_ERR_STATE, "the tangent covers FEM triangles without FEM-FEM contact");
  if (!c) return FW_ERR_ARG;
  if (!c->finalized || c->arena || c->S != 1 || c->path == FW_PATH_STREAM)
    return fail(c, FW_ERR_STATE, "the tangent needs a finalized single-scene world on the gather or resident path");
  if (c->d.has_j2) return fail(c, FW_ERR_ARG, "the tangent covers Elastic and NeoHookean triangles (no J2)");
  Tan& t = c->tan;
  int rc;
  if (!c->adj.young && (rc = upload(c, &c->adj.young, c->h_E))) return rc;
  t.young = c->adj.young;
  if (!t.dx) {
    if ((rc = dalloc(c, &t.dx, c->N)) || (rc = dalloc(c, &t.dv, c->N)) || (rc = dalloc(c, &t.dE, c->E)) ||
        (rc = dalloc(c, &t.xs, c->N)) || (rc = dalloc(c, &t.vs, c->N)) || (rc = dalloc(c, &t.io_x, c->N)) ||
        (rc = dalloc(c, &t.io_v, c->N)))
      return rc;
  }
  const cudaMemcpyKind k = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
  if (dx0) FW_CUDA(c, cudaMemcpyAsync(t.io_x, dx0, sizeof(float2) * c->N, k, c->stream));
  if (dv0) FW_CUDA(c, cudaMemcpyAsync(t.io_v, dv0, sizeof(float2) * c->N, k, c->stream));
  if (dE) FW_CUDA(c, cudaMemcpyAsync(t.dE, dE, sizeof(float) * c->E, k, c->stream));
  else FW_CUDA(c, cudaMemsetAsync(t.dE, 0, sizeof(float) * c->E, c->stream));
  k_tan_seed<<<(c->N + kBlock - 1) / kBlock, kBlock, 0, c->stream>>>(t, c->N, dx0 != nullptr, dv0 != nullptr);
  c->launches += 1;
  return check_kernel(c, "tangent seed");
}

int fw_tan_step(fw_ctx* c, int32_t n_steps, float dt) {
  if (!c) return FW_ERR_ARG;
  if (!c->tan.dx) return fail(c, FW_ERR_STATE, "fw_tan_step before fw_tan_begin");
  if (n_steps < 0) return fail(c, FW_ERR_ARG, "n_steps must be >= 0");
  Tan& t = c->tan;
  c->d.uniform_dt = 1;
  c->d.dt_uniform = dt;
  const float damp = c->h_damp.empty() ? 0.0f : c->h_damp[0];
  const int gn = (c->N + kBlock - 1) / kBlock, ge = (c->E + kBlock - 1) / kBlock;
  int rc;
  for (int j = 0; j < n_steps; ++j) {
    FW_CUDA(c, cudaMemcpyAsync(t.xs, c->d.x, sizeof(float2) * c->N, cudaMemcpyDeviceToDevice, c->stream));
    FW_CUDA(c, cudaMemcpyAsync(t.vs, c->d.v, sizeof(float2) * c->N, cudaMemcpyDeviceToDevice, c->stream));
    if ((rc = launch_step(c))) return rc;  // the substep itself (sets this substep's gates)
    c->host_counter += 1;
    k_tan_elements<<<ge, kBlock, 0, c->stream>>>(c->d, t);
    k_tan_nodes<<<gn, kBlock, 0, c->stream>>>(c->d, t, dt, damp);
    c->launches += 2;
  }
  return check_kernel(c, "tangent step");
}

int fw_tan_read(fw_ctx* c, float* dx, float* dv, int32_t on_device) {
  if (!c) return FW_ERR_ARG;
  if (!c->tan.dx) return fail(c, FW_ERR_STATE, "fw_tan_read before fw_tan_begin");
  const cudaMemcpyKind k = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
  k_tan_out<<<(c->N + kBlock - 1) / kBlock, kBlock, 0, c->stream>>>(c->tan, c->N);
  c->launches += 1;
  if (dx) FW_CUDA(c, cudaMemcpyAsync(dx, c->tan.io_x, sizeof(float2) * c->N, k, c->stream));
  if (dv) FW_CUDA(c, cudaMemcpyAsync(dv, c->tan.io_v, sizeof(float2) * c->N, k, c->stream));
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  return FW_OK;
}

int fw_get_path(const fw_ctx* c, int32_t* path, int32_t* patches) {
  if (!c || !path) return FW_ERR_ARG;
  *path = c->finalized ? c->path : FW_PATH_AUTO;
  if (patches) *patches = !c->clu.empty() && c->rest_scenes.empty() ? c->clu_patches : (c->path == FW_PATH_RESIDENT ? c->res.P : (c->path == FW_PATH_STREAM ? c->st_P : 0));
  return FW_OK;
}

int fw_step(fw_ctx* c, int32_t n_steps, float dt) {
  if (!c) return FW_ERR_ARG;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_step before fw_finalize");
  if (n_steps < 0) return fail(c, FW_ERR_ARG, "fw_step: n_steps < 0");
  c->d.uniform_dt = 1;
  c->d.dt_uniform = dt;
  return run_steps(c, n_steps);
}

int fw_step_scenes(fw_ctx* c, int32_t n_steps, const float* dt) {
  if (!c || !dt) return FW_ERR_ARG;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_step_scenes before fw_finalize");
  if (n_steps < 0) return fail(c, FW_ERR_ARG, "fw_step_scenes: n_steps < 0");
  int rc = set_scene_dt(c, dt);
  if (rc) return rc;
  c->d.uniform_dt = 0;
  return run_steps(c, n_steps);
}

int fw_step_runs(fw_ctx* c, int32_t n_runs, const int32_t* counts, const float* dts) {
  if (!c || !counts || !dts) return FW_ERR_ARG;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_step_runs before fw_finalize");
  if (n_runs < 1 || n_runs > kCluRuns) return fail(c, FW_ERR_ARG, "fw_step_runs: n_runs outside [1, %d]", kCluRuns);
  if (c->path != FW_PATH_STREAM || c->clu.empty() || !c->rest_scenes.empty())
    return fail(c, FW_ERR_STATE, "fw_step_runs: not every scene of the world is stepped on chip (FW_OPT_CLUSTER)");
  std::vector<CluRun> runs(c->S, CluRun{});
  for (int j = 0; j < c->S; ++j)
    for (int k = 0; k < n_runs; ++k) {
      const int s = c->clu_order[j], n = counts[(size_t)s * n_runs + k];
      if (n < 0) return fail(c, FW_ERR_ARG, "fw_step_runs: scene %d: count < 0", s);
      runs[j].n[k] = n;
      runs[j].dt[k] = dts[(size_t)s * n_runs + k];
    }
  int rc;
  if (!c->d_runs && (rc = dalloc(c, &c->d_runs, c->S))) return rc;
  // pageable source: staged before the call returns; on the stream, after the last launch that read the buffer
  FW_CUDA(c, cudaMemcpyAsync(c->d_runs, runs.data(), sizeof(CluRun) * c->S, cudaMemcpyHostToDevice, c->stream));
  return launch_cluster(c, 0, c->d.x, c->d.x, c->d.j2state, c->d.j2state, c->d_runs);
}

int fw_set_active(fw_ctx* c, const int32_t* active) {
  if (!c || !active) return FW_ERR_ARG;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_set_active before fw_finalize");
  c->cur_active.assign(active, active + c->S);
  if (c->arena)  // a scene that is not live stays inactive
    for (int s = 0; s < c->S; ++s)
      if (!c->ascenes[s].live) c->cur_active[s] = 0;
  FW_CUDA(c, cudaMemcpyAsync(c->d.scene_active, c->cur_active.data(), sizeof(int32_t) * c->S,
                             cudaMemcpyHostToDevice, c->stream));
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  c->chunks_dirty = true;
  return FW_OK;
}

int fw_synchronize(fw_ctx* c) {
  if (!c) return FW_ERR_ARG;
  if (c->finalized && raises_flags(c)) return check_device_error(c);  // which waits: one trip
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  return FW_OK;
}

int fw_read_nodes(fw_ctx* c, int32_t field, int32_t first, int32_t count, float* dst, int32_t on_device) {
  if (!c || !dst) return FW_ERR_ARG;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_read_nodes before fw_finalize");
  if (first < 0 || count < 0 || (int64_t)first + count > c->N)
    return fail(c, FW_ERR_ARG, "fw_read_nodes: range [%d, %d) outside [0, %d)", first, first + count, c->N);
  const void* src = nullptr;
  size_t per = 2 * sizeof(float);
  switch (field) {
    case FW_FIELD_X: src = c->d.x + first; break;
    case FW_FIELD_V: src = c->d.v + first; break;
    case FW_FIELD_X0: src = c->d.x0 + first; break;
    case FW_FIELD_MASS: src = c->d.mass + first; per = sizeof(float); break;
    default: return fail(c, FW_ERR_ARG, "fw_read_nodes: unknown field %d", field);
  }
  if (count == 0) return fw_synchronize(c);
  if (!on_device) {
    cudaPointerAttributes at{};
    const bool pinned = cudaPointerGetAttributes(&at, dst) == cudaSuccess && at.type != cudaMemoryTypeUnregistered;
    cudaGetLastError();
    if (!pinned) return read_pageable(c, dst, src, per * count);
  }
  FW_CUDA(c, cudaMemcpyAsync(dst, src, per * count,
                             on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, c->stream));
  if (!raises_flags(c)) {
    FW_CUDA(c, cudaStreamSynchronize(c->stream));
    return FW_OK;
  }
  return check_device_error(c);
}

int fw_write_nodes(fw_ctx* c, int32_t field, int32_t first, int32_t count, const float* src, int32_t on_device) {
  if (!c || !src) return FW_ERR_ARG;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_write_nodes before fw_finalize");
  if (first < 0 || count < 0 || (int64_t)first + count > c->N)
    return fail(c, FW_ERR_ARG, "fw_write_nodes: range [%d, %d) outside [0, %d)", first, first + count, c->N);
  void* dst = nullptr;
  switch (field) {
    case FW_FIELD_X: dst = c->d.x + first; break;
    case FW_FIELD_V: dst = c->d.v + first; break;
    default: return fail(c, FW_ERR_ARG, "fw_write_nodes: field %d is not writable", field);
  }
  FW_CUDA(c, cudaMemcpyAsync(dst, src, 2 * sizeof(float) * count,
                             on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, c->stream));
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  return FW_OK;
}

int fw_read_aabb(fw_ctx* c, float* dst) {
  if (!c || !dst) return FW_ERR_ARG;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_read_aabb before fw_finalize");
  std::vector<int32_t> ring(8 * (size_t)c->B), cnt(c->S);
  FW_CUDA(c, cudaMemcpyAsync(ring.data(), c->d.aabb_ring, sizeof(int32_t) * ring.size(), cudaMemcpyDeviceToHost, c->stream));
  FW_CUDA(c, cudaMemcpyAsync(cnt.data(), c->d.scene_counter, sizeof(int32_t) * c->S, cudaMemcpyDeviceToHost, c->stream));
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  for (int b = 0; b < c->B; ++b) {
    const int sc = c->arena ? c->a_body_scene[b] : c->h_scene[b];
    const int slot = cnt[sc] & 1;
    for (int k = 0; k < 4; ++k) {
      int v = ring[((size_t)slot * c->B + b) * 4 + k];
      v = v >= 0 ? v : v ^ 0x7FFFFFFF;
      memcpy(&dst[4 * b + k], &v, sizeof(float));
    }
  }
  return FW_OK;
}

int fw_read_plastic(fw_ctx* c, float* eps_p, float* eqps) {
  if (!c) return FW_ERR_ARG;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_read_plastic before fw_finalize");
  std::vector<float4> st(c->d.has_j2 ? c->E : 0);
  if (c->d.has_j2) {
    FW_CUDA(c, cudaMemcpyAsync(st.data(), c->d.j2state, sizeof(float4) * c->E, cudaMemcpyDeviceToHost, c->stream));
    FW_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  for (int e = 0; e < c->E; ++e) {
    const float4 s = c->d.has_j2 ? st[e] : make_float4(0.f, 0.f, 0.f, 0.f);
    if (eps_p) {
      eps_p[3 * e] = s.x;
      eps_p[3 * e + 1] = s.y;
      eps_p[3 * e + 2] = s.z;
    }
    if (eqps) eqps[e] = s.w;
  }
  return FW_OK;
}

int fw_read_reference_shape(fw_ctx* c, float* area, float* jinv) {
  if (!c) return FW_ERR_ARG;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_read_reference_shape before fw_finalize");
  std::vector<ElemMat> m(c->E);
  FW_CUDA(c, cudaMemcpyAsync(m.data(), c->d.emat, sizeof(ElemMat) * c->E, cudaMemcpyDeviceToHost, c->stream));
  if (jinv) FW_CUDA(c, cudaMemcpyAsync(jinv, c->d.jinv, sizeof(float4) * c->E, cudaMemcpyDeviceToHost, c->stream));
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  if (area)
    for (int e = 0; e < c->E; ++e) area[e] = m[e].area;
  return FW_OK;
}

int fw_energy(fw_ctx* c, double* out) {
  if (!c || !out) return FW_ERR_ARG;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_energy before fw_finalize");
  // groups: bodies (summed per scene below) or, in an arena, scene slots; laid
  // out once, and again after an arena's scenes changed
  if (c->energy_dirty) {
    struct Range { int n0, nn, e0, ne; };
    std::vector<Range> groups;
    if (c->arena) {
      for (const fw_ctx::ArenaScene& a : c->ascenes)
        groups.push_back(a.live ? Range{(int)a.n0, (int)a.nn, (int)a.e0, (int)a.ne} : Range{0, 0, 0, 0});
    } else {
      for (int b = 0; b < c->B; ++b) groups.push_back(Range{c->h_noff[b], c->h_ncnt[b], c->h_eoff[b], c->h_ecnt[b]});
    }
    const int G = (int)groups.size();
    std::vector<EnergyChunk> chunks;
    std::vector<int> first(G + 1, 0);
    for (int g = 0; g < G; ++g) {
      first[g] = (int)chunks.size();
      const Range& r = groups[g];
      const int n = (std::max(r.nn, r.ne) + kEnergyChunk - 1) / kEnergyChunk;
      for (int k = 0; k < n; ++k) {
        EnergyChunk ch;
        ch.group = g;
        ch.n0 = r.n0 + std::min(r.nn, k * kEnergyChunk);
        ch.nn = std::max(0, std::min(kEnergyChunk, r.nn - k * kEnergyChunk));
        ch.e0 = r.e0 + std::min(r.ne, k * kEnergyChunk);
        ch.ne = std::max(0, std::min(kEnergyChunk, r.ne - k * kEnergyChunk));
        chunks.push_back(ch);
      }
    }
    first[G] = (int)chunks.size();
    const size_t nc = chunks.size();
    if (nc > c->energy_cap || (size_t)G + 1 > c->energy_gcap) {
      for (void* p : {(void*)c->d_echunk, (void*)c->d_epart, (void*)c->d_efirst, (void*)c->d_eout})
        if (p) cudaFree(p);
      c->d_echunk = nullptr;
      c->d_epart = nullptr;
      c->d_efirst = nullptr;
      c->d_eout = nullptr;
      c->energy_cap = c->energy_gcap = 0;
      const size_t cap = std::max(nc, (size_t)64), gcap = std::max((size_t)G + 1, (size_t)64);
      FW_CUDA(c, cudaMalloc((void**)&c->d_echunk, sizeof(EnergyChunk) * cap));
      FW_CUDA(c, cudaMalloc((void**)&c->d_epart, sizeof(double4) * cap));
      FW_CUDA(c, cudaMalloc((void**)&c->d_efirst, sizeof(int) * gcap));
      FW_CUDA(c, cudaMalloc((void**)&c->d_eout, sizeof(double4) * gcap));
      c->energy_cap = cap;
      c->energy_gcap = gcap;
    }
    if (nc)
      FW_CUDA(c, cudaMemcpyAsync(c->d_echunk, chunks.data(), sizeof(EnergyChunk) * nc, cudaMemcpyHostToDevice, c->stream));
    FW_CUDA(c, cudaMemcpyAsync(c->d_efirst, first.data(), sizeof(int) * (G + 1), cudaMemcpyHostToDevice, c->stream));
    c->energy_chunks = (int)nc;
    c->energy_groups = G;
    c->energy_dirty = false;
  }
  const int G = c->energy_groups;
  if (c->energy_chunks > 0)
    k_energy_chunks<<<(unsigned)c->energy_chunks, kEnergyThreads, 0, c->stream>>>(c->d, c->d_echunk, c->d_epart);
  k_energy_groups<<<G, kEnergyGroupThreads, 0, c->stream>>>(c->d_efirst, c->d_epart, c->d_eout);
  c->launches += 2;
  int rc = check_kernel(c, "energy");
  if (rc) return rc;
  std::vector<double4> res(G);
  FW_CUDA(c, cudaMemcpyAsync(res.data(), c->d_eout, sizeof(double4) * G, cudaMemcpyDeviceToHost, c->stream));
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  const int S = c->arena ? (int)c->ascenes.size() : c->S;
  for (int s = 0; s < 4 * S; ++s) out[s] = 0.0;
  for (int g = 0; g < G; ++g) {  // bodies of a scene in ascending order
    const int sc = c->arena ? g : c->h_scene[g];
    out[4 * sc + 0] += res[g].x;
    out[4 * sc + 1] += res[g].y;
    out[4 * sc + 2] += res[g].z;
    out[4 * sc + 3] += res[g].w;
  }
  return FW_OK;
}

int fw_scene_status(fw_ctx* c, int32_t* bad, int32_t async) {
  if (!c || !bad) return FW_ERR_ARG;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_scene_status before fw_finalize");
  FW_CUDA(c, cudaMemcpyAsync(bad, c->d.scene_bad, sizeof(int32_t) * c->S, cudaMemcpyDeviceToHost, c->stream));
  if (!async) FW_CUDA(c, cudaStreamSynchronize(c->stream));
  return FW_OK;
}

int fw_clear_scene_status(fw_ctx* c, int32_t scene) {
  if (!c) return FW_ERR_ARG;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_clear_scene_status before fw_finalize");
  if (scene < -1 || scene >= c->S) return fail(c, FW_ERR_ARG, "scene %d out of range", scene);
  if (scene < 0) FW_CUDA(c, cudaMemsetAsync(c->d.scene_bad, 0, sizeof(int32_t) * c->S, c->stream));
  else FW_CUDA(c, cudaMemsetAsync(c->d.scene_bad + scene, 0, sizeof(int32_t), c->stream));
  return FW_OK;
}

int fw_set_cfl_monitor(fw_ctx* c, const float* coef_per_body) {
  if (!c) return FW_ERR_ARG;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_set_cfl_monitor before fw_finalize");

  int rc;
  drop_graphs(c);  // captured graphs hold the previous monitor pointers
  if (!coef_per_body) {
    c->d.cfl_ord = nullptr;
    return FW_OK;
  }
  if (!c->cfl_ord_buf) {
    if ((rc = dalloc(c, &c->cfl_ord_buf, (size_t)c->S)) || (rc = dalloc(c, &c->cfl_coef_buf, (size_t)c->B)))
      return rc;
  }
  FW_CUDA(c, cudaMemcpyAsync(c->cfl_coef_buf, coef_per_body, sizeof(float) * c->B, cudaMemcpyHostToDevice, c->stream));
  std::vector<int32_t> inf(c->S, 0x7f800000);
  FW_CUDA(c, cudaMemcpyAsync(c->cfl_ord_buf, inf.data(), sizeof(int32_t) * c->S, cudaMemcpyHostToDevice, c->stream));
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  c->d.cfl_ord = c->cfl_ord_buf;
  c->d.body_cfl = c->cfl_coef_buf;
  return FW_OK;
}

int fw_read_cfl(fw_ctx* c, float* out, int32_t reset) {
  if (!c || !out) return FW_ERR_ARG;
  if (!c->d.cfl_ord) return fail(c, FW_ERR_STATE, "fw_read_cfl: the CFL monitor is off");
  std::vector<int32_t> v(c->S);
  FW_CUDA(c, cudaMemcpyAsync(v.data(), c->d.cfl_ord, sizeof(int32_t) * c->S, cudaMemcpyDeviceToHost, c->stream));
  if (reset) {
    std::vector<int32_t> inf(c->S, 0x7f800000);
    FW_CUDA(c, cudaMemcpyAsync(c->d.cfl_ord, inf.data(), sizeof(int32_t) * c->S, cudaMemcpyHostToDevice, c->stream));
  }
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  for (int s = 0; s < c->S; ++s) {
    float f;
    std::memcpy(&f, &v[s], sizeof(float));
    out[s] = f;
  }
  return FW_OK;
}

int fw_read_counters(fw_ctx* c, int64_t* counters) {
  if (!c || !counters) return FW_ERR_ARG;
  if (!c->finalized) return fail(c, FW_ERR_STATE, "fw_read_counters before fw_finalize");
  std::vector<int32_t> cnt(c->S);
  FW_CUDA(c, cudaMemcpyAsync(cnt.data(), c->d.scene_counter, sizeof(int32_t) * c->S, cudaMemcpyDeviceToHost, c->stream));
  FW_CUDA(c, cudaStreamSynchronize(c->stream));
  for (int s = 0; s < c->S; ++s) counters[s] = cnt[s];
  return FW_OK;
}

int64_t fw_launch_count(const fw_ctx* c) { return c ? c->launches : 0; }

int fw_log_f32(const float* x, float* log_x, float* quotient, int64_t n, void* stream) {
  if (!x || !log_x || n < 0 || n > (1ll << 31)) return FW_ERR_ARG;
  if (n == 0) return FW_OK;
  k_log<<<(unsigned)((n + kBlock - 1) / kBlock), kBlock, 0, (cudaStream_t)stream>>>(x, log_x, quotient, n);
  return cudaGetLastError() == cudaSuccess ? FW_OK : FW_ERR_CUDA;
}

const char* fw_build_info(void) {
  return "libfwb200: sm_100a, -fmad=false, IEEE div/sqrt; gather step + shared-memory-resident step";
}

}  // extern "C"
