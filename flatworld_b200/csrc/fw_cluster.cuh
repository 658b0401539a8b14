// fw_cluster.cuh -- scenes that stay on chip for a whole fw_step call.
//
// A scene is cut into patches, one per CTA, whose nodes and triangles stay in
// shared memory and registers through all substeps of a call.  Two forms of
// one kernel:
//  - cluster (scenes that fit the shared memory of a thread-block cluster, up to
//    16 SMs): one launch steps any number of scenes, each on its own cluster
//    with its own step size.  Positions cross CTAs through distributed shared
//    memory, so a substep needs no global memory.
//  - grid (one larger scene): a cooperative launch with a patch per SM;
//    positions cross through L2.
// Either way a CTA writes an updated position straight into the halo slot of
// each CTA that reads it, as two 64-bit words (substep tag << 32 | value bits),
// and the thread that evaluates a cut triangle polls those words itself: no
// fence, no counter, no grid-wide wait and no launch per substep.  (st.async
// with a byte count on the neighbour's mbarrier was measured first: the sends
// of one warp of nodes took about 2000 cycles, the counts being serialised.)
//
// What bounds it: with few warps on an SM, the number of instructions on the
// chain halo -> cut triangles -> node update -> neighbours' halo (about five
// cycles each: fixed latencies, instruction fetch), two CTA barriers and one
// shared-memory hop; with many scenes, instruction issue.  So the chain holds
// only what it must: the contact forces of the boundary nodes and the body
// boxes, which depend on a substep's start state alone, belong to the CTA's
// last warps ("control warps") and run beside the triangles, and where a patch
// has a thread per triangle and node (ONE), their static data and the node
// state live in registers.
//
// Broad-phase gates without waiting for anyone: a node that lies inside a
// pair's gate box proves the gate on, since the body's box contains the node
// (on the 10%-growth substeps too: growth only enlarges both boxes), and a
// pair that gives a node no force changes nothing, gate on or off.  Only a
// node that would get a force from outside the gate box needs the scene's
// boxes: every CTA keeps its partial boxes of the last substeps in a ring of
// tagged words (in its shared memory; grid form: in global memory), and the
// warp in need reads the others'.
// Once every kCluBoxSync substeps each CTA waits until all have reached it,
// which bounds how far CTAs drift apart, so no slot of the ring is rewritten
// before its last reader.  (Exchanging all boxes every substep took 1800 of a
// substep's 4100 cycles on a 2048-triangle mesh.)
//
// Layout of a CTA's shared memory (one carve-up per launch, sized by the
// largest patch of the launch, so that a slot has the same offset in every CTA
// of a cluster):
//   x      owned positions; the boundary nodes first, then the other nodes that
//          neighbours read
//   halo   (cluster form) the neighbours' positions as tagged words, two copies
//          (parity of the substep)
//   f      corner forces in node order: corner k (ascending element) of node i
//          at f[i * fs + k], so a node's sum needs no index list and reads two
//          corners per 16-byte load; fs is 2 mod 4, which keeps those loads
//          free of bank conflicts; slots past a node's last corner stay zero,
//          and adding +0 leaves the sum's bits alone (it starts at +0)
//   cf, bv, bb  boundary nodes: contact force, velocity, body
//   jinv, rec   (not ONE) 32 bytes per triangle: Dm^-1, area, local corners,
//          corner slots
//   lm, j2      (not ONE) per triangle only where needed: Lame constants (unless
//          the patch's triangles share them), J2 state and parameters
//   vm, bcv     (not ONE) velocity, 1/mass and flag word of a node; its BC value
//          (times its mass where the update multiplies by it)
// Triangles that touch only owned nodes come first; they are evaluated while
// the neighbours' positions are on their way, and only the warps that hold cut
// triangles wait for them.
//
// Why two halo copies suffice: halo membership is
// symmetric (a cut triangle is held by each patch that touches it), so a
// neighbour sends positions k + 1 only after it has received this CTA's
// positions k, and positions k + 2 only after it has received this CTA's
// k + 1, which this CTA sends after its wait for k.
//
// The arithmetic and its order are those of the gather step: the results are
// the same bits.
#pragma once

namespace {

constexpr int kCluMaxCtas = 16;
constexpr int kCluOneThreads = 640;  // grid form: most threads with a thread per triangle (clu_threads)
constexpr int kCluMaxBodies = 8;   // per scene
constexpr int kCluMaxPairs = 32;   // per scene
constexpr int kCluMaxThreads = 1024;
constexpr long long kCluWaitLimit = 1ll << 22;
constexpr uint32_t kCluNoSlot = 0xFFFFu;
constexpr int kCluBoxSync = 16;
constexpr int kCluBoxRing = 2 * kCluBoxSync;
constexpr size_t kCluStatic = 64;  // at least the kernel's static shared memory

// Flag word of an owned node: BC bits 0-8 and NODE_BOUNDARY as in node_word;
// the body's index in its scene; the node's entries in the push list.
constexpr int kCluBodyShift = 10;      // 4 bits
constexpr int kCluPushCntShift = 14;   // 3 bits
constexpr int kCluPushOffShift = 17;   // 15 bits

// A patch's static description in HBM (16-byte aligned parts, ids relative to
// the scene's first node / triangle).
struct CluPatch {
  int no, nh, ne, n_int;  // owned and halo nodes, triangles, interior triangles
  int npush, deg, n_j2, nbnd;  // nbnd: boundary nodes (the first ones)
  int halo0, tri0;             // grid form: its first halo slot in CluLaunch::ghalo, its first triangle record in gji and grec
  int slot_shift, pad;         // corner slots in the blob: corner << slot_shift | node
  int64_t gid, info, hid, push, eid, tri, pos;  // byte offsets into the blob
};

// The substeps of one scene in a call: n[0] at dt[0], then n[1] at dt[1], ...
constexpr int kCluRuns = 4;
struct CluRun {
  int n[kCluRuns];
  float dt[kCluRuns];
};

struct CluScene {
  int64_t blob0;  // arenas: its patches' byte offsets count from here
  int scene;
  int patch0;     // its patches: patch[patch0 .. + cluster size)
  int n0, e0;     // its first node and triangle
  int body0, nb;  // its bodies
  int pair0, np;  // its contact pairs
};

// Byte offsets of the parts of a CTA's dynamic shared memory.
struct CluAt {
  int x;      // owned positions
  int halo;   // [2][nh] neighbours' positions (tag << 32 | x bits, tag << 32 | y bits)
  int f;      // [no][fs] corner forces
  int cf, bv, bb;  // boundary nodes: contact force, velocity, body
  int jinv, rec;
  int lm;     // per triangle (lam, mu, word)
  int j2, j2p;
  int vm;     // velocity, 1 / mass, flag word
  int bcv;    // BC value, times the mass for gravity and prescribed accelerations
  int push;   // (CTA << 24 | halo slot) of the owned nodes' readers
  int pairs, gate;
  int bst;    // body -> its boundary nodes [bst[b], bst[b + 1])
  int box;    // cluster form: [kCluBoxRing][nb][4] this CTA's partial boxes (tag << 32 | ordered int)
};

// One launch: scenes with the same cluster size.
struct CluLaunch {
  CluAt at;
  const CluScene* scene;
  const CluPatch* patch;
  const unsigned char* blob;
  int ctas;                      // CTAs per scene
  int grid;                      // the grid form
  int no, nh, ne, deg, npush, nbnd;  // maxima over the launch's patches
  int one;                       // a thread per triangle and per node (k_cluster's ONE)
  int ctl;                       // control warps
  int fs;                        // corner slots of a node
  int nb, np;                    // maxima over its scenes
  int has_j2, per_tri;           // J2 state / Lame constants per triangle
  int* err;                      // != 0: a wait gave up
  long long wait_limit;
  int withhold_cta;              // test hook: this CTA sends nothing after its first substep (-1: none)
  float2* rec_x;                 // adjoint recompute (one scene): state at the start of each substep
  float2* rec_v;
  int* rec_gates;                // 1 where a pair gave a force (a pair that gave none has no adjoint either)
  int rec_stride;
  const CluRun* runs;            // per scene of the launch (null: nsteps substeps of the scene's dt)
  // grid form
  ulonglong2* ghalo;             // [2][n_halo]
  unsigned long long* gbox;      // [kCluBoxRing][ctas][nb][4]
  int n_halo;
  // ... of patches whose triangle records do not fit beside the nodes: records
  // in global memory (L2), in patch order, read once a substep
  float4* gji;
  uint4* grec;
  float4* glm;                   // lam, mu, word (per_tri)
  float4* gj2;
  int tri_l2;
  uint32_t ep0;                  // tags of this launch count up from here
};

// The carve-up (host): byte offsets of r.at from the launch's maxima; returns
// the byte count.  The offsets travel as 32-bit kernel arguments: pointers
// derived in the kernel from the maxima were rebuilt by long address chains in
// every phase of a substep.
inline size_t clu_layout(CluLaunch& r) {
  size_t o = 0;
  auto take = [&](int& at, size_t bytes) {
    at = (int)o;
    o += (bytes + 15) & ~(size_t)15;
  };
  take(r.at.x, sizeof(float2) * (size_t)r.no);
  take(r.at.halo, r.grid ? 0 : sizeof(ulonglong2) * 2 * (size_t)r.nh);
  r.fs = (r.deg + 1) / 4 * 4 + 2;  // >= deg, 2 mod 4
  take(r.at.f, sizeof(float2) * (size_t)r.fs * r.no);
  const size_t nb = r.np ? r.nbnd : 0, ne = r.one || r.tri_l2 ? 0 : r.ne, no = r.one ? 0 : r.no;
  take(r.at.cf, sizeof(float2) * nb);
  take(r.at.bv, sizeof(float2) * nb);
  take(r.at.bb, sizeof(int) * (size_t)r.nbnd);
  take(r.at.jinv, sizeof(float4) * ne);
  take(r.at.rec, sizeof(uint4) * ne);
  take(r.at.lm, r.per_tri ? sizeof(float4) * ne : 0);
  take(r.at.j2, r.has_j2 ? sizeof(float4) * ne : 0);
  take(r.at.j2p, r.has_j2 && r.per_tri ? sizeof(float2) * ne : 0);
  take(r.at.vm, sizeof(float4) * no);
  take(r.at.bcv, sizeof(float2) * no);
  take(r.at.push, sizeof(uint32_t) * (size_t)r.npush);
  take(r.at.pairs, sizeof(Pair) * (size_t)r.np);
  take(r.at.gate, sizeof(int) * (size_t)r.np);
  take(r.at.bst, sizeof(int) * (size_t)(r.nb + 1));
  take(r.at.box, r.grid ? 0 : sizeof(unsigned long long) * 4 * kCluBoxRing * (size_t)r.nb);
  return o;
}

extern __shared__ __align__(16) unsigned char clu_mem[];

// The parts of a CTA's shared memory.
struct CluSmem {
  const CluAt& at;
  template <class T>
  __device__ __forceinline__ T* part(int off) const { return reinterpret_cast<T*>(clu_mem + off); }
  __device__ __forceinline__ float2* x() const { return part<float2>(at.x); }
  __device__ __forceinline__ ulonglong2* halo() const { return part<ulonglong2>(at.halo); }
  __device__ __forceinline__ float2* f() const { return part<float2>(at.f); }
  __device__ __forceinline__ float2* cf() const { return part<float2>(at.cf); }
  __device__ __forceinline__ float2* bv() const { return part<float2>(at.bv); }
  __device__ __forceinline__ int* bb() const { return part<int>(at.bb); }
  __device__ __forceinline__ float4* jinv() const { return part<float4>(at.jinv); }
  __device__ __forceinline__ uint4* rec() const { return part<uint4>(at.rec); }
  __device__ __forceinline__ float4* lm() const { return part<float4>(at.lm); }
  __device__ __forceinline__ float4* j2() const { return part<float4>(at.j2); }
  __device__ __forceinline__ float2* j2p() const { return part<float2>(at.j2p); }
  __device__ __forceinline__ float4* vm() const { return part<float4>(at.vm); }
  __device__ __forceinline__ float2* bcv() const { return part<float2>(at.bcv); }
  __device__ __forceinline__ uint32_t* push() const { return part<uint32_t>(at.push); }
  __device__ __forceinline__ Pair* pairs() const { return part<Pair>(at.pairs); }
  __device__ __forceinline__ int* gate() const { return part<int>(at.gate); }
  __device__ __forceinline__ int* bst() const { return part<int>(at.bst); }
  __device__ __forceinline__ unsigned long long* box() const { return part<unsigned long long>(at.box); }
};

__device__ __forceinline__ uint32_t clu_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t clu_map(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void clu_sync() {
  asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}
// Tagged words: 64-bit relaxed accesses, each single-copy atomic.
template <bool GRID>
__device__ __forceinline__ void clu_send(const CluLaunch& r, uint32_t to, int copy, uint32_t tag, float2 v) {
  const unsigned long long wx = ll_pack(tag, __float_as_uint(v.x)), wy = ll_pack(tag, __float_as_uint(v.y));
  if (GRID)
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(r.ghalo + (size_t)copy * r.n_halo + (to - 1u)), "l"(wx),
                 "l"(wy)
                 : "memory");
  else
    asm volatile("st.relaxed.cluster.shared::cluster.v2.u64 [%0], {%1, %2};" ::"r"(to + 16u * (uint32_t)(copy * r.nh)),
                 "l"(wx), "l"(wy)
                 : "memory");
}
template <bool GRID>
__device__ __forceinline__ ulonglong2 clu_peek(const CluLaunch& r, const CluSmem& s, int halo0, int copy, int j) {
  ulonglong2 v;
  if (GRID)
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                 : "=l"(v.x), "=l"(v.y)
                 : "l"(r.ghalo + (size_t)copy * r.n_halo + halo0 + j)
                 : "memory");
  else
    asm volatile("ld.relaxed.cluster.shared::cta.v2.u64 {%0, %1}, [%2];"
                 : "=l"(v.x), "=l"(v.y)
                 : "r"(smem_addr(s.halo() + copy * r.nh + j))
                 : "memory");
  return v;
}
// Component comp of CTA c's partial box of body b in ring slot `slot`.
template <bool GRID>
__device__ __forceinline__ unsigned long long clu_peek_box(const CluLaunch& r, const CluSmem& s, int c, int slot, int b,
                                                           int comp) {
  unsigned long long v;
  if (GRID) {
    v = ll_load(r.gbox + (((size_t)slot * r.ctas + c) * r.nb + b) * 4 + comp);
  } else {
    uint32_t at = smem_addr(s.box() + ((size_t)slot * r.nb + b) * 4 + comp);
    if (r.ctas > 1) at = clu_map(at, (uint32_t)c);
    asm volatile("ld.relaxed.cluster.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(at) : "memory");
  }
  return v;
}
// One more poll of a wait: false when it gives up.
__device__ __forceinline__ bool clu_again(long long& it, long long limit, int* err, int* abort) {
  if (++it <= limit && ((it & 1023) != 0 || *(volatile const int*)err == 0)) return true;
  atomicExch(err, 1);
  *abort = 1;
  return false;
}

// Blob encodings, independent of a launch's maxima: a local corner is the owned
// node, or kCluHalo + the halo node; a corner slot is
// corner << CluPatch::slot_shift | node (11 bits of node leave 31 corners, 12 leave 15).
constexpr uint32_t kCluHalo = 0x4000u;
__device__ __forceinline__ uint32_t clu_index(uint32_t c, int no) { return c & kCluHalo ? (c & 0x3FFFu) + no : c; }
__device__ __forceinline__ uint32_t clu_slot(uint32_t p, int fs, int shift) {
  return p == kCluNoSlot ? p : (p & ((1u << shift) - 1u)) * fs + (p >> shift);
}

// A triangle's static data (and J2 state).
struct CluTri {
  float4 ji;
  uint4 rec;  // area, corners, corner slots
  float lam, mu, sy, H;
  int word;
  float4 j2;
};

__device__ __forceinline__ uint4 clu_rec(const CluLaunch& r, uint2 c, uint32_t p, float area, int shift) {
  const uint32_t i0 = clu_index(c.x & 0x7FFFu, r.no) | (c.x & 0x8000u), i1 = clu_index(c.x >> 16, r.no);
  return make_uint4(__float_as_uint(area), i0 | (i1 << 16),
                    clu_index(c.y & 0xFFFFu, r.no) | (clu_slot(c.y >> 16, r.fs, shift) << 16),
                    clu_slot(p & 0xFFFFu, r.fs, shift) | (clu_slot(p >> 16, r.fs, shift) << 16));
}

// Corner forces of one triangle in substep k (the halo's tag); returns its
// current-shape CFL bound when body_cfl is given, else +inf.
template <bool GRID>
__device__ __forceinline__ float clu_element(const fw::Packed2& p2, const CluLaunch& r, const CluSmem& s, CluTri& m, bool cut, int halo0, int k,
                                             uint32_t tag, int* abort, const float* body_cfl) {
  const uint4 c = m.rec;
  const int i0 = c.y & 0x7FFFu, i1 = c.y >> 16, i2 = c.z & 0xFFFFu;
  float2 a, b, cc;
  if (!cut) {
    a = s.x()[i0];
    b = s.x()[i1];
    cc = s.x()[i2];
  } else {  // poll the halo corners together
    const int copy = k & 1, no = r.no;
    const bool h0 = i0 >= no, h1 = i1 >= no, h2 = i2 >= no;
    for (long long it = 0;;) {
      const unsigned long long done = ll_pack(tag, 0u);
      ulonglong2 w0 = make_ulonglong2(done, done), w1 = w0, w2 = w0;
      if (h0) w0 = clu_peek<GRID>(r, s, halo0, copy, i0 - no);
      if (h1) w1 = clu_peek<GRID>(r, s, halo0, copy, i1 - no);
      if (h2) w2 = clu_peek<GRID>(r, s, halo0, copy, i2 - no);
      const bool here = ll_has(w0.x, tag) && ll_has(w0.y, tag) && ll_has(w1.x, tag) && ll_has(w1.y, tag) &&
                        ll_has(w2.x, tag) && ll_has(w2.y, tag);
      a = make_float2(__uint_as_float((uint32_t)w0.x), __uint_as_float((uint32_t)w0.y));
      b = make_float2(__uint_as_float((uint32_t)w1.x), __uint_as_float((uint32_t)w1.y));
      cc = make_float2(__uint_as_float((uint32_t)w2.x), __uint_as_float((uint32_t)w2.y));
      if (here || !clu_again(it, r.wait_limit, r.err, abort)) break;
    }
    if (!h0) a = s.x()[i0];
    if (!h1) b = s.x()[i1];
    if (!h2) cc = s.x()[i2];
  }
  ElemMat em;
  em.area = __uint_as_float(c.x);
  em.lam = m.lam;
  em.mu = m.mu;
  em.word = m.word;
  float2 f1, f2, f3;
  fw::element_forces(p2, a, b, cc, m.ji, em, m.sy, m.H, m.j2, f1, f2, f3);
  const uint32_t o0 = c.z >> 16, o1 = c.w & 0xFFFFu, o2 = c.w >> 16;
  if (o0 != kCluNoSlot) s.f()[o0] = f1;
  if (o1 != kCluNoSlot) s.f()[o1] = f2;
  if (o2 != kCluNoSlot) s.f()[o2] = f3;
  return body_cfl ? cfl_bound(a, b, cc, body_cfl[fw::elem_body(m.word)]) : __int_as_float(0x7f800000);
}

// An owned node's state and static data.
struct CluNode {
  float2 x, v, b;
  float im;
  uint32_t w;
  uint32_t to;  // its first reader's slot (0: none; the rest are in the push list)
};

// fw::integrate_im with the BC value already multiplied by the mass where the
// update multiplies by it.
__device__ __forceinline__ void clu_integrate(const fw::Packed2& p, int bc, float2 f, float im, float2 b, float dt,
                                              float damping, float2& x, float2& v) {
  if (bc & fw::BC_U) {
    f = make_float2(0.0f, 0.0f);
  } else if (bc & fw::BC_A) {
    f = b;
  } else if (bc & (fw::BC_GRAVITY | fw::BC_FORCE)) {
    f = p.add(f, b);
  }
  const float2 h = fw::dup2(dt);
  const float2 acc =
      p.add(p.mul(p.add(p.mul(fw::dup2(-damping), v), f), fw::dup2(im)), make_float2(0.0f, 0.0f));  // (f - c v) / m
  v = p.add(p.mul(acc, h), v);
  if (bc & fw::BC_V) {
    v = b;
  } else if (bc & fw::BC_U) {
    v = make_float2(0.0f, 0.0f);
  }
  x = p.add(p.mul(v, h), x);
}

__device__ __forceinline__ int clu_box_identity(int comp) { return comp < 2 ? fw::f2ord(1e30f) : fw::f2ord(-1e30f); }

// This CTA's partial boxes at the start of substep k into the ring, by one
// warp; `bodies` has a bit for each body with a boundary node here.
template <bool GRID>
__device__ __forceinline__ void clu_publish(const CluLaunch& r, const CluSmem& s, int rank, int nb, uint32_t bodies, int k,
                                            int lane) {
  const unsigned full = 0xFFFFFFFFu;
  const int big = fw::f2ord(1e30f), low = fw::f2ord(-1e30f), comp = lane & 3;
  int v = comp < 2 ? big : low;  // lane 4 b + comp: that component of body b
  for (uint32_t m = bodies; m; m &= m - 1) {
    const int b = __ffs(m) - 1, hi = s.bst()[b + 1];
    int lx = big, ly = big, hx = low, hy = low;
    for (int i = s.bst()[b] + lane; i < hi; i += 32) {
      const float2 x = s.x()[i];
      const int ox = fw::f2ord(x.x), oy = fw::f2ord(x.y);
      if (x.x == x.x) {  // NaN widens no box
        lx = min(lx, ox);
        hx = max(hx, ox);
      }
      if (x.y == x.y) {
        ly = min(ly, oy);
        hy = max(hy, oy);
      }
    }
    lx = __reduce_min_sync(full, lx);
    ly = __reduce_min_sync(full, ly);
    hx = __reduce_max_sync(full, hx);
    hy = __reduce_max_sync(full, hy);
    if (lane >> 2 == b) v = comp == 0 ? lx : (comp == 1 ? ly : (comp == 2 ? hx : hy));
  }
  if (lane < 4 * nb) {
    const unsigned long long w = ll_pack(r.ep0 + (uint32_t)k + 1u, (uint32_t)v);
    const int slot = k % kCluBoxRing;
    if (GRID)
      ll_store(r.gbox + ((size_t)slot * r.ctas + rank) * r.nb * 4 + lane, w);
    else
      asm volatile("st.relaxed.cluster.shared::cta.u64 [%0], %1;" ::"r"(smem_addr(s.box() + (size_t)slot * r.nb * 4 + lane)),
                   "l"(w)
                   : "memory");
  }
}

// Body b's box at the start of substep k, from every CTA's ring, by one warp.
template <bool GRID>
__device__ __noinline__ int4 clu_box(const CluLaunch& r, const CluSmem& s, int b, int k, int* abort) {
  const unsigned full = 0xFFFFFFFFu;
  int v[4];
  for (int comp = 0; comp < 4; ++comp) v[comp] = clu_box_identity(comp);
  for (int c = threadIdx.x & 31; c < r.ctas; c += 32)
    for (int comp = 0; comp < 4; ++comp) {
      const uint32_t tag = r.ep0 + (uint32_t)k + 1u;
      unsigned long long u = clu_peek_box<GRID>(r, s, c, k % kCluBoxRing, b, comp);
      for (long long it = 0; !ll_has(u, tag) && clu_again(it, r.wait_limit, r.err, abort);)
        u = clu_peek_box<GRID>(r, s, c, k % kCluBoxRing, b, comp);
      const int o = (int)(uint32_t)u;
      v[comp] = comp < 2 ? min(v[comp], o) : max(v[comp], o);
    }
  return make_int4(__reduce_min_sync(full, v[0]), __reduce_min_sync(full, v[1]), __reduce_max_sync(full, v[2]),
                   __reduce_max_sync(full, v[3]));
}

__device__ __forceinline__ bool clu_gate(const Pair& pr, int4 bb, int g) {
  return fw::pair_gate(pr, fw::ord2f(bb.x), fw::ord2f(bb.y), fw::ord2f(bb.z), fw::ord2f(bb.w), g);
}

// Steps every scene of the launch through nsteps substeps: the j-th group of
// r.ctas CTAs holds scene r.scene[j].  Positions and J2 state are read from x_in / j2_in and
// written to x_out / j2_out (the same buffers, or a stream world's pair).
template <int MAXT, bool ONE, bool GRID, bool L2TRI = false>
__global__ void __launch_bounds__(MAXT, 1)
k_cluster(const __grid_constant__ Dev d, const __grid_constant__ CluLaunch r, const float2* x_in, float2* x_out,
          const float4* j2_in, float4* j2_out, int n_all) {
  __shared__ int s_abort, s_cfl;
  const CluSmem s{r.at};
  const fw::Packed2 p2{d.one};
  const int t = threadIdx.x, C = r.ctas;
  const int T = blockDim.x - 32 * r.ctl;  // threads with triangles and nodes
  const int rank = GRID ? (int)blockIdx.x : (C > 1 ? (int)clu_rank() : 0);
  const CluScene sc = r.scene[GRID ? 0 : blockIdx.x / C];
  const CluPatch& Pg = r.patch[sc.patch0 + rank];
  const int S = sc.scene, no = Pg.no, ne = Pg.ne, nbnd = Pg.nbnd, first_cut = Pg.n_int,
            halo0 = Pg.halo0, tri0 = Pg.tri0;
  const unsigned char* blob = r.blob + sc.blob0;
  const int32_t* gid = reinterpret_cast<const int32_t*>(blob + Pg.gid);
  const int32_t* eid = reinterpret_cast<const int32_t*>(blob + Pg.eid);
  const uint2* tri = reinterpret_cast<const uint2*>(blob + Pg.tri);
  const CluRun* runs = r.runs ? r.runs + (GRID ? 0 : blockIdx.x / C) : nullptr;
  int nsteps = n_all;
  if (runs) {
    nsteps = 0;
    for (int j = 0; j < kCluRuns; ++j) nsteps += runs->n[j];
  }
  if (!d.scene_active[S] || nsteps <= 0) {  // every CTA of the scene leaves: the state stays (or moves over)
    if (x_in != x_out) {
      for (int i = t; i < no; i += blockDim.x) x_out[sc.n0 + gid[i]] = x_in[sc.n0 + gid[i]];
      if (d.has_j2)
        for (int q = t; q < ne; q += blockDim.x)
          if (tri[q].x & 0x8000u) j2_out[sc.e0 + eid[q]] = j2_in[sc.e0 + eid[q]];
    }
    return;
  }
  const bool control = t >= T;
  const int counter0 = d.scene_counter[S];
  const int lane = t & 31;
  // ---- load the patch
  if (t == 0) {
    s_abort = 0;
    s_cfl = 0x7f800000;
  }
  const uint32_t* pos = reinterpret_cast<const uint32_t*>(blob + Pg.pos);
  const uint32_t* info = reinterpret_cast<const uint32_t*>(blob + Pg.info);
  // a patch's triangles share one material unless the launch keeps it per triangle
  CluTri tr{};
  if (ne > 0) {
    const int e = sc.e0 + eid[0];
    const ElemMat m = d.emat[e];
    tr.lam = m.lam;
    tr.mu = m.mu;
    tr.word = m.word;
    if (fw::elem_type(m.word) == fw::MAT_MISES) {
      tr.sy = d.j2par[e].x;
      tr.H = d.j2par[e].y;
    }
  }
  if (ONE) {
    if (!control && t < ne) {
      const int e = sc.e0 + eid[t];
      const ElemMat m = d.emat[e];
      tr.ji = d.jinv[e];
      tr.rec = clu_rec(r, tri[t], pos[t], m.area, Pg.slot_shift);
      tr.lam = m.lam;
      tr.mu = m.mu;
      tr.word = m.word;
      if (fw::elem_type(m.word) == fw::MAT_MISES) {
        tr.j2 = j2_in[e];
        tr.sy = d.j2par[e].x;
        tr.H = d.j2par[e].y;
      }
    }
  } else {
    // several triangles' loads in flight per thread: a patch's load is two
    // dependent trips to memory, whatever its size
    constexpr int U = 3;
    const int W = blockDim.x;
    for (int q0 = t; q0 < ne; q0 += U * W) {
      int e[U];
      ElemMat m[U];
      float4 ji[U], j2[U];
      uint2 c[U];
      uint32_t ps[U];
#pragma unroll
      for (int u = 0; u < U; ++u) e[u] = q0 + u * W < ne ? sc.e0 + eid[q0 + u * W] : -1;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (e[u] >= 0) {
          m[u] = d.emat[e[u]];
          ji[u] = d.jinv[e[u]];
          c[u] = tri[q0 + u * W];
          ps[u] = pos[q0 + u * W];
          if (r.has_j2) j2[u] = j2_in[e[u]];
        }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (e[u] >= 0) {
          const int q = q0 + u * W;
          const uint4 rec = clu_rec(r, c[u], ps[u], m[u].area, Pg.slot_shift);
          const float4 lm = make_float4(m[u].lam, m[u].mu, __int_as_float(m[u].word), 0.f);
          if (L2TRI) {
            r.gji[tri0 + q] = ji[u];
            r.grec[tri0 + q] = rec;
            if (r.per_tri) r.glm[tri0 + q] = lm;
            if (r.has_j2) r.gj2[tri0 + q] = j2[u];
            continue;
          }
          s.jinv()[q] = ji[u];
          s.rec()[q] = rec;
          if (r.per_tri) s.lm()[q] = lm;
          if (r.has_j2) {
            s.j2()[q] = j2[u];
            if (r.per_tri) s.j2p()[q] = d.j2par[e[u]];
          }
        }
    }
  }
  CluNode nd{};
  if (!control)
    for (int i = t; i < no; i += T) {
      const int g = sc.n0 + gid[i];
      const float m = d.mass[g];
      nd.x = x_in[g];
      nd.v = d.v[g];
      nd.w = info[i];
      nd.im = 1.0f / m;
      nd.b = d.bcv[g];
      if (!(nd.w & fw::BC_V) && (nd.w & (fw::BC_A | fw::BC_GRAVITY))) nd.b = make_float2(m * nd.b.x, m * nd.b.y);
      s.x()[i] = nd.x;
      if (i < nbnd) {
        const int body = (int)(nd.w >> kCluBodyShift) & 15;
        const int before = i > 0 ? (int)(info[i - 1] >> kCluBodyShift) & 15 : -1;
        for (int b = before + 1; b <= body; ++b) s.bst()[b] = i;
        if (i == nbnd - 1)
          for (int b = body + 1; b <= sc.nb; ++b) s.bst()[b] = nbnd;
        s.bb()[i] = body;
        if (sc.np > 0) s.bv()[i] = nd.v;
      }
      if (r.rec_x) {
        r.rec_x[g] = nd.x;
        r.rec_v[g] = nd.v;
      }
      if (ONE) break;
      s.vm()[i] = make_float4(nd.v.x, nd.v.y, nd.im, __uint_as_float(nd.w));
      s.bcv()[i] = nd.b;
    }
  {
    const int nh = Pg.nh, npush = Pg.npush;
    const int32_t* hid = reinterpret_cast<const int32_t*>(blob + Pg.hid);
    const uint32_t* push = reinterpret_cast<const uint32_t*>(blob + Pg.push);
    const int W = blockDim.x;
    if (!GRID) {
      for (int i = t; i < nh; i += W) {  // substep 0's halo; the other copy holds no tag that is waited for
        const float2 x = x_in[sc.n0 + hid[i]];
        s.halo()[i] = make_ulonglong2(ll_pack(1u, __float_as_uint(x.x)), ll_pack(1u, __float_as_uint(x.y)));
        s.halo()[r.nh + i] = make_ulonglong2(0ull, 0ull);
      }
      for (int i = t; i < 4 * kCluBoxRing * r.nb; i += W) s.box()[i] = 0ull;
    }
    // a send's target: the reader's slot in its shared memory (the first copy), or in ghalo (+ 1)
    for (int i = t; i < npush; i += W) {
      const uint32_t to = push[i] >> 24, j = push[i] & 0xFFFFFFu;
      s.push()[i] = GRID ? (uint32_t)r.patch[sc.patch0 + to].halo0 + j + 1u : clu_map(smem_addr(s.halo() + j), to);
    }
    for (int i = t; i < r.fs * r.no; i += W) s.f()[i] = make_float2(0.f, 0.f);
    for (int i = t; i < sc.np; i += W) {
      const Pair pr = d.pairs[sc.pair0 + i];
      s.pairs()[i] = pr;
      // gates at the start of the call: the boxes of the previous call's last
      // substep (a node's position may have been set since)
      s.gate()[i] = clu_gate(pr, __ldcg(reinterpret_cast<const int4*>(
                                     d.aabb_ring + ((size_t)(counter0 & 1) * d.B + pr.body) * 4)), counter0) ? 1 : 0;
    }
    if (nbnd == 0)
      for (int b = t; b <= sc.nb; b += W) s.bst()[b] = 0;
  }
  float dt = runs ? runs->dt[0] : (d.uniform_dt ? d.dt_uniform : d.scene_dt[S]);
  int run = 0, run_end = runs ? runs->n[0] : nsteps;  // dt holds for substeps [.., run_end)
  const float damp = d.scene_damp[S];
  // a scene just committed to an arena: its first substep is the zero-dt
  // construction step (no contact, no damping, not counted)
  const int init = d.scene_mode_req[S] ? 1 : 0;
  const float* bcfl = d.cfl_ord ? d.body_cfl : nullptr;
  float cfl = __int_as_float(0x7f800000);
  bool bad = false;
  __syncthreads();
  if (ONE && !control && t < no && ((nd.w >> kCluPushCntShift) & 7u)) nd.to = s.push()[nd.w >> kCluPushOffShift];
  if (GRID) {  // substep 0's halo is sent like the others': no CTA reads what another may already write back
    if (!control)
      for (int i = t; i < no; i += T) {
        const uint32_t w = info[i];
        for (uint32_t j = 0; j < ((w >> kCluPushCntShift) & 7u); ++j)
          clu_send<GRID>(r, s.push()[(w >> kCluPushOffShift) + j], 0, r.ep0 + 1u, s.x()[i]);
      }
  } else if (C > 1) {
    clu_sync();  // every CTA's words are initialised, and its halo is read
  }
  // the bodies with boundary nodes here, and the pairs of the first to the last of them
  uint32_t bodies = 0;
  int p_lo = 0, p_hi = 0;
  if (control && nbnd > 0) {
    for (int b = 0; b < sc.nb; ++b) bodies |= s.bst()[b] < s.bst()[b + 1] ? 1u << b : 0u;
    p_lo = d.body_pair_off[sc.body0 + s.bb()[0]] - sc.pair0;
    const int last = sc.body0 + s.bb()[nbnd - 1];
    p_hi = d.body_pair_off[last] + d.body_pair_cnt[last] - sc.pair0;
  }
  if (control) {
    // ---- control warps: the boxes and the contact forces of the substep's start state
    const int ct = t - T, CT = 32 * r.ctl;
    const int g0 = counter0 - init;
    for (int k = 0; k < nsteps; ++k) {
      while (k == run_end) {
        dt = runs->dt[++run];
        run_end += runs->n[run];
      }
      if (sc.np > 0) {
        const int g = g0 + k;
        if (ct < 32) {  // the first one keeps the boxes
          if (!(k == 1 && (int)blockIdx.x == r.withhold_cta)) clu_publish<GRID>(r, s, rank, sc.nb, bodies, k, lane);
          if (k % kCluBoxSync == 0 && k > 0 && C > 1)  // everyone has come this far
            for (int c = lane; c < C; c += 32)
              for (long long it = 0; !ll_has(clu_peek_box<GRID>(r, s, c, k % kCluBoxRing, 0, 0), r.ep0 + (uint32_t)k + 1u) &&
                                     clu_again(it, r.wait_limit, r.err, &s_abort);) {
              }
        }
        // the others' contact forces (a single control warp does both)
        const int first = r.ctl > 1 ? (ct & ~31) - 32 : 0, step = r.ctl > 1 ? CT - 32 : 32;
        for (int i0 = first; i0 >= 0 && i0 < nbnd; i0 += step) {
          const int i = i0 + lane;
          const bool valid = i < nbnd;
          const float2 x = valid ? s.x()[i] : make_float2(0.f, 0.f), v = valid ? s.bv()[i] : make_float2(0.f, 0.f);
          const int body = valid ? s.bb()[i] : -1;
          float2 f = make_float2(0.f, 0.f);
          for (int p = p_lo; p < p_hi; ++p) {
            const Pair& pr = s.pairs()[p];
            float2 cf;
            const bool hit = pr.body - sc.body0 == body && k >= init && fw::contact_force(pr, d.heights, d.occ, d.vox, x, v, dt, cf);
            bool on = k == 0 ? s.gate()[p] != 0
                             : x.x >= pr.glo[0] && x.x <= pr.ghi[0] && x.y >= pr.glo[1] && x.y <= pr.ghi[1];
            if (k > 0 && __any_sync(0xFFFFFFFFu, hit && !on))  // a force from outside the gate box: the gate itself
              on |= clu_gate(pr, clu_box<GRID>(r, s, pr.body - sc.body0, k, &s_abort), g);
            if (hit && on) {
              f.x += cf.x;
              f.y += cf.y;
              if (r.rec_gates) r.rec_gates[(size_t)k * r.rec_stride + p] = 1;  // zero before the launch
            }
          }
          if (valid) s.cf()[i] = f;
        }
      }
      __syncthreads();  // A
      if (s_abort) break;
      __syncthreads();  // B
    }
  } else {
    for (int k = 0; k < nsteps; ++k) {
      while (k == run_end) {
        dt = runs->dt[++run];
        run_end += runs->n[run];
      }
      // ---- corner forces: interior triangles, then the cut ones as the halo arrives
      if (ONE) {
        const bool cut = first_cut <= (t | 31);  // the warp holds cut triangles
        if (t < ne) cfl = fminf(cfl, clu_element<GRID>(p2, r, s, tr, cut, halo0, k, r.ep0 + (uint32_t)k + 1u, &s_abort, bcfl));
      } else if (L2TRI) {
        // each record is fetched from L2 while the one before it is evaluated
        float4 nx_ji{};
        uint4 nx_rec{};
        if (t < ne) {
          nx_ji = __ldcg(&r.gji[tri0 + t]);
          nx_rec = __ldcg(&r.grec[tri0 + t]);
        }
        for (int q = t; q < ne; q += T) {
          tr.ji = nx_ji;
          tr.rec = nx_rec;
          if (q + T < ne) {
            nx_ji = __ldcg(&r.gji[tri0 + q + T]);
            nx_rec = __ldcg(&r.grec[tri0 + q + T]);
          }
          if (r.per_tri) {
            const float4 l = __ldcg(&r.glm[tri0 + q]);
            tr.lam = l.x;
            tr.mu = l.y;
            tr.word = __float_as_int(l.z);
          }
          const bool mises = fw::elem_type(tr.word) == fw::MAT_MISES;
          if (mises) {
            tr.j2 = __ldcg(&r.gj2[tri0 + q]);
            if (r.per_tri) {
              const float2 jp = d.j2par[sc.e0 + eid[q]];
              tr.sy = jp.x;
              tr.H = jp.y;
            }
          }
          cfl = fminf(cfl, clu_element<GRID>(p2, r, s, tr, first_cut <= (q | 31), halo0, k, r.ep0 + (uint32_t)k + 1u, &s_abort, bcfl));
          if (mises) __stcg(&r.gj2[tri0 + q], tr.j2);
        }
      } else {
        for (int q = t; q < ne; q += T) {
          const bool cut = first_cut <= (q | 31);
          tr.rec = s.rec()[q];
          tr.ji = s.jinv()[q];
          if (r.per_tri) {
            const float4 l = s.lm()[q];
            tr.lam = l.x;
            tr.mu = l.y;
            tr.word = __float_as_int(l.z);
          }
          const bool mises = fw::elem_type(tr.word) == fw::MAT_MISES;
          if (mises) {
            tr.j2 = s.j2()[q];
            if (r.per_tri) {
              const float2 jp = s.j2p()[q];
              tr.sy = jp.x;
              tr.H = jp.y;
            }
          }
          cfl = fminf(cfl, clu_element<GRID>(p2, r, s, tr, cut, halo0, k, r.ep0 + (uint32_t)k + 1u, &s_abort, bcfl));
          if (mises) s.j2()[q] = tr.j2;
        }
      }
      __syncthreads();  // A: every corner and contact force of substep k
      if (s_abort) break;
      // ---- nodes; the ones neighbours read leave as soon as they are computed
      const bool send = k + 1 < nsteps && !(k == 0 && (int)blockIdx.x == r.withhold_cta);
      const int copy = (k + 1) & 1;
      const uint32_t tag = r.ep0 + (uint32_t)k + 2u;
      for (int i = t; i < no; i += T) {
        if (!ONE) {
          const float4 vm = s.vm()[i];
          nd.x = s.x()[i];
          nd.v = make_float2(vm.x, vm.y);
          nd.im = vm.z;
          nd.w = __float_as_uint(vm.w);
          nd.b = s.bcv()[i];
        }
        float2 f = make_float2(0.f, 0.f);
        if (i < nbnd && sc.np > 0) f = s.cf()[i];
        const float4* c = reinterpret_cast<const float4*>(s.f() + i * r.fs);
        {
          float4 cq[3];
#pragma unroll
          for (int w = 0; w < 3; ++w) cq[w] = 2 * w < r.fs ? c[w] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int w = 0; w < 3; ++w) {
            f = p2.add(f, make_float2(cq[w].x, cq[w].y));
            f = p2.add(f, make_float2(cq[w].z, cq[w].w));
          }
        }
        for (int w = 3; 2 * w < r.fs; ++w) {
          const float4 cq = c[w];
          f = p2.add(f, make_float2(cq.x, cq.y));
          f = p2.add(f, make_float2(cq.z, cq.w));
        }
        clu_integrate(p2, (int)(nd.w & fw::NODE_BC_MASK), f, nd.im, nd.b, k < init ? 0.0f : dt, k < init ? 0.0f : damp, nd.x,
                      nd.v);
        if (!ONE) nd.to = (nd.w >> kCluPushCntShift) & 7u ? s.push()[nd.w >> kCluPushOffShift] : 0u;
        if (nd.to && send) {
          clu_send<GRID>(r, nd.to, copy, tag, nd.x);
          const uint32_t n = (nd.w >> kCluPushCntShift) & 7u;
          if (n > 1)
            for (uint32_t j = 1; j < n; ++j) clu_send<GRID>(r, s.push()[(nd.w >> kCluPushOffShift) + j], copy, tag, nd.x);
        }
        s.x()[i] = nd.x;
        if (i < nbnd && sc.np > 0) s.bv()[i] = nd.v;
        if (!ONE) s.vm()[i] = make_float4(nd.v.x, nd.v.y, nd.im, __uint_as_float(nd.w));
        bad |= !(isfinite(nd.x.x) && isfinite(nd.x.y) && isfinite(nd.v.x) && isfinite(nd.v.y));
        if (r.rec_x && k + 1 < nsteps) {
          const size_t at = (size_t)(k + 1) * d.N + sc.n0 + gid[i];
          r.rec_x[at] = nd.x;
          r.rec_v[at] = nd.v;
        }
        if (ONE) break;
      }
      __syncthreads();  // B: every position of substep k + 1's start
    }
  }
  __syncthreads();
  // ---- write the state back
  const bool ok = s_abort == 0;
  if (ok && control && t - T < 32) {  // the scene's boxes and counter, by its first CTA
    clu_publish<GRID>(r, s, rank, sc.nb, bodies, nsteps, lane);
    __syncwarp();
    if (rank == 0) {
      const int after = counter0 + nsteps - init;
      for (int b = 0; b < sc.nb; ++b) {
        const int4 bb = clu_box<GRID>(r, s, b, nsteps, &s_abort);
        if (lane == 0) *reinterpret_cast<int4*>(d.aabb_ring + ((size_t)(after & 1) * d.B + sc.body0 + b) * 4) = bb;
      }
      if (lane == 0) {
        d.scene_counter[S] = after;
        if (init) d.scene_mode_req[S] = 0;
      }
    }
  }
  if (bad) d.scene_bad[S] = 1;
  if (d.cfl_ord) {
    const int m = warp_min_bits(cfl);
    if (lane == 0 && m < 0x7f800000) atomicMin(&s_cfl, m);
    __syncthreads();
    if (t == 0 && s_cfl < 0x7f800000) atomicMin(d.cfl_ord + S, s_cfl);
  }
  if (!control) {
    for (int i = t; i < no; i += T) {
      const int g = sc.n0 + gid[i];
      x_out[g] = s.x()[i];
      if (ONE) {
        d.v[g] = nd.v;
        break;
      }
      const float4 vm = s.vm()[i];
      d.v[g] = make_float2(vm.x, vm.y);
    }
    if (r.has_j2)
      for (int q = t; q < ne; q += T)
        if (tri[q].x & 0x8000u) {
          const int e = sc.e0 + eid[q];
          const int word = d.emat[e].word;
          if (fw::elem_type(word) == fw::MAT_MISES) j2_out[e] = ONE ? tr.j2 : (L2TRI ? __ldcg(&r.gj2[tri0 + q]) : s.j2()[q]);
        }
  }
  if (!GRID && C > 1) {
    clu_sync();  // no CTA leaves while another may still write into its shared memory
    if (!ok) __nanosleep(20000);  // what was sent to a CTA that gave up has landed by then
  }
}

// ------------------------------------------------------------------ adjoint
// Reverse pass of one recorded segment on the grid form's patches, a thread per
// triangle and per node: the adjoint state of a node (FP64) and the static data
// and dL/dE of a triangle stay in registers, the force adjoints that neighbours
// read are pushed into their halo slots (four tagged words each), and the
// positions of the next substep are fetched while this one's triangles are
// evaluated.  The arithmetic and its order are those of k_adj_prep /
// k_adj_elements / k_adj_nodes.  Bound, like the forward step, by the latency of
// one substep's chain.
struct CluAdj {
  CluLaunch r;  // patches, err, wait limit, tags
  int x, fb, f, push, pairs;  // byte offsets in shared memory: positions (owned, halo), force adjoints, corner slots
  ulonglong2* words;          // [2][n_halo][2] force adjoints
  const float2* rec_x;
  const float2* rec_v;
  const int* rec_gates;
  int gate_stride;
};

inline size_t clu_adj_layout(CluAdj& q) {
  size_t o = 0;
  auto take = [&](int& at, size_t bytes) {
    at = (int)o;
    o += (bytes + 15) & ~(size_t)15;
  };
  const CluLaunch& r = q.r;
  take(q.x, sizeof(float2) * (size_t)(r.no + r.nh));
  take(q.fb, sizeof(double2) * (size_t)r.no);
  take(q.f, sizeof(float2) * (size_t)r.fs * r.no);
  take(q.push, sizeof(uint32_t) * (size_t)r.npush);
  take(q.pairs, sizeof(Pair) * (size_t)r.np);
  return o;
}

template <int MAXT>
__global__ void __launch_bounds__(MAXT, 1)
k_cluster_adj(const __grid_constant__ Dev d, const __grid_constant__ CluAdj q, const __grid_constant__ Adj a, int nsteps,
              float dt, float damp) {
  __shared__ int s_abort;
  const CluLaunch& r = q.r;
  const int t = threadIdx.x, T = blockDim.x, N = d.N;
  const CluScene sc = r.scene[0];
  const CluPatch& P = r.patch[sc.patch0 + blockIdx.x];
  const int no = P.no, nh = P.nh, ne = P.ne, nbnd = P.nbnd;
  float2* xs = reinterpret_cast<float2*>(clu_mem + q.x);
  double2* fbs = reinterpret_cast<double2*>(clu_mem + q.fb);
  float2* fs = reinterpret_cast<float2*>(clu_mem + q.f);
  uint32_t* push = reinterpret_cast<uint32_t*>(clu_mem + q.push);
  Pair* pairs = reinterpret_cast<Pair*>(clu_mem + q.pairs);
  // ---- load
  if (t == 0) s_abort = 0;
  const bool tri = t < ne, node = t < no, halo = t < nh;
  CluTri m{};
  double Eb = 0.0;
  float young = 1.f;
  int eg = 0;
  if (tri) {
    eg = sc.e0 + reinterpret_cast<const int32_t*>(r.blob + P.eid)[t];
    const ElemMat em = d.emat[eg];
    m.ji = d.jinv[eg];
    m.rec = clu_rec(r, reinterpret_cast<const uint2*>(r.blob + P.tri)[t], reinterpret_cast<const uint32_t*>(r.blob + P.pos)[t],
                    em.area, P.slot_shift);
    m.lam = em.lam;
    m.mu = em.mu;
    m.word = em.word;
    young = a.young[eg];
    if (m.rec.y & 0x8000u) Eb = a.Eb[eg];
  }
  const bool cut = P.n_int <= (t | 31);
  double2 xb = make_double2(0.0, 0.0), vb = xb, fb = xb;
  double step = 0.0, keep = 0.0;
  uint32_t w = 0;
  int gn = 0, gh = 0;
  const double h = (double)dt;
  if (node) {
    gn = sc.n0 + reinterpret_cast<const int32_t*>(r.blob + P.gid)[t];
    w = reinterpret_cast<const uint32_t*>(r.blob + P.info)[t];
    xb = a.xb[gn];
    vb = a.vb[gn];
    step = h / (double)d.mass[gn];
    keep = 1.0 - step * (double)damp;
  }
  if (halo) gh = sc.n0 + reinterpret_cast<const int32_t*>(r.blob + P.hid)[t];
  for (int i = t; i < P.npush; i += T) {
    const uint32_t to = reinterpret_cast<const uint32_t*>(r.blob + P.push)[i];
    push[i] = (uint32_t)r.patch[sc.patch0 + (to >> 24)].halo0 + (to & 0xFFFFFFu);
  }
  for (int i = t; i < r.fs * r.no; i += T) fs[i] = make_float2(0.f, 0.f);
  for (int i = t; i < sc.np; i += T) pairs[i] = d.pairs[sc.pair0 + i];
  const int bc = (int)(w & fw::NODE_BC_MASK);
  const bool vfixed = (bc & (fw::BC_U | fw::BC_V)) != 0, fdead = vfixed || (bc & fw::BC_A) != 0;
  int p_lo = 0, p_hi = 0;  // the pairs of a boundary node's body
  if (t < nbnd) {
    const int b = sc.body0 + ((int)(w >> kCluBodyShift) & 15);
    p_lo = d.body_pair_off[b] - sc.pair0;
    p_hi = p_lo + d.body_pair_cnt[b];
  }
  auto prep = [&] {  // the adjoints of the node force and of the previous velocity
    const double2 vt = make_double2(vb.x + h * xb.x, vb.y + h * xb.y);
    fb = fdead ? make_double2(0.0, 0.0) : make_double2(step * vt.x, step * vt.y);
    vb = vfixed ? make_double2(0.0, 0.0) : make_double2(keep * vt.x, keep * vt.y);
  };
  prep();
  size_t row = (size_t)(nsteps - 1) * N;
  float2 xn = node ? q.rec_x[row + gn] : make_float2(0.f, 0.f), xh = halo ? q.rec_x[row + gh] : make_float2(0.f, 0.f);
  __syncthreads();
  for (int rr = 0; rr < nsteps; ++rr) {
    const int j = nsteps - 1 - rr;
    const uint32_t tag = r.ep0 + (uint32_t)rr + 1u;
    ulonglong2* copy = q.words + (size_t)(rr & 1) * r.n_halo * 2;
    const float2 xi = xn;
    if (node) {
      const uint32_t n_to = (w >> kCluPushCntShift) & 7u;
      for (uint32_t k = 0; k < n_to; ++k) {
        ulonglong2* to = copy + 2 * (size_t)push[(w >> kCluPushOffShift) + k];
        asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(to), "l"(ll_pack(tag, lo32(fb.x))),
                     "l"(ll_pack(tag, hi32(fb.x)))
                     : "memory");
        asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(to + 1), "l"(ll_pack(tag, lo32(fb.y))),
                     "l"(ll_pack(tag, hi32(fb.y)))
                     : "memory");
      }
      fbs[t] = fb;
      xs[t] = xn;
    }
    if (halo) xs[r.no + t] = xh;
    __syncthreads();  // positions and force adjoints of substep j
    float2 vi = make_float2(0.f, 0.f);
    if (t < nbnd && p_hi > p_lo) vi = q.rec_v[row + gn];
    if (j > 0) {  // the next substep's positions, on their way meanwhile
      const size_t up = row - N;
      if (node) xn = q.rec_x[up + gn];
      if (halo) xh = q.rec_x[up + gh];
    }
    if (tri) {
      const uint4 c = m.rec;
      const int i0 = c.y & 0x7FFFu, i1 = c.y >> 16, i2 = c.z & 0xFFFFu;
      double2 b0, b1, b2;
      if (cut) {  // poll the halo corners together
        const bool h0 = i0 >= r.no, h1 = i1 >= r.no, h2 = i2 >= r.no;
        const ulonglong2* base = copy + 2 * ((ptrdiff_t)P.halo0 - r.no);
        for (long long it = 0;;) {
          const unsigned long long done = ll_pack(tag, 0u);
          ulonglong2 u[6];
#pragma unroll
          for (int k = 0; k < 6; ++k) {
            const bool hk = k < 2 ? h0 : (k < 4 ? h1 : h2);
            const int ik = k < 2 ? i0 : (k < 4 ? i1 : i2);
            u[k] = make_ulonglong2(done, done);
            if (hk)
              asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                           : "=l"(u[k].x), "=l"(u[k].y)
                           : "l"(base + 2 * (ptrdiff_t)ik + (k & 1))
                           : "memory");
          }
          bool here = true;
#pragma unroll
          for (int k = 0; k < 6; ++k) here = here && ll_has(u[k].x, tag) && ll_has(u[k].y, tag);
          b0 = make_double2(join64((uint32_t)u[0].x, (uint32_t)u[0].y), join64((uint32_t)u[1].x, (uint32_t)u[1].y));
          b1 = make_double2(join64((uint32_t)u[2].x, (uint32_t)u[2].y), join64((uint32_t)u[3].x, (uint32_t)u[3].y));
          b2 = make_double2(join64((uint32_t)u[4].x, (uint32_t)u[4].y), join64((uint32_t)u[5].x, (uint32_t)u[5].y));
          if (here || !clu_again(it, r.wait_limit, r.err, &s_abort)) break;
        }
        if (!h0) b0 = fbs[i0];
        if (!h1) b1 = fbs[i1];
        if (!h2) b2 = fbs[i2];
      } else {
        b0 = fbs[i0];
        b1 = fbs[i1];
        b2 = fbs[i2];
      }
      fw::Dual f[6];
      fw::element_forces_jvp(xs[i0], xs[i1], xs[i2], make_float2((float)b0.x, (float)b0.y), make_float2((float)b1.x, (float)b1.y),
                             make_float2((float)b2.x, (float)b2.y), m.ji, fw::elem_type(m.word), m.lam, m.mu,
                             __uint_as_float(c.x), f);
      const uint32_t o0 = c.z >> 16, o1 = c.w & 0xFFFFu, o2 = c.w >> 16;
      if (o0 != kCluNoSlot) fs[o0] = make_float2(f[0].d, f[1].d);
      if (o1 != kCluNoSlot) fs[o1] = make_float2(f[2].d, f[3].d);
      if (o2 != kCluNoSlot) fs[o2] = make_float2(f[4].d, f[5].d);
      if (c.y & 0x8000u) {
        const double dot = b0.x * f[0].v + b0.y * f[1].v + b1.x * f[2].v + b1.y * f[3].v + b2.x * f[4].v + b2.y * f[5].v;
        Eb += dot / (double)young;
      }
    }
    __syncthreads();  // every corner's share of substep j
    if (s_abort) break;
    if (node) {
      const float4* c = reinterpret_cast<const float4*>(fs + t * r.fs);
      for (int k = 0; 2 * k < r.fs; ++k) {
        const float4 cq = c[k];
        xb.x += cq.x;
        xb.y += cq.y;
        xb.x += cq.z;
        xb.y += cq.w;
      }
      for (int p = p_lo; p < p_hi; ++p)
        if (q.rec_gates[(size_t)j * q.gate_stride + p]) fw::contact_vjp(pairs[p], d.heights, d.occ, xi, vi, dt, fb, xb, vb);
      if (j > 0) prep();
    }
    row -= N;
  }
  if (node) {
    a.xb[gn] = xb;
    a.vb[gn] = vb;
  }
  if (tri && (m.rec.y & 0x8000u)) a.Eb[eg] = Eb;
}

using CluAdjKernel = void (*)(const Dev, const CluAdj, const Adj, int, float, float);
inline CluAdjKernel clu_adj_kernel(int threads) { return threads <= 512 ? k_cluster_adj<512> : k_cluster_adj<768>; }

using CluKernel = void (*)(const Dev, const CluLaunch, const float2*, float2*, const float4*, float4*, int);
inline CluKernel clu_kernel(int threads, int one, int grid, int tri_l2 = 0) {
  if (grid) {
    if (tri_l2) return k_cluster<1024, false, true, true>;
    if (one) return threads <= 512 ? k_cluster<512, true, true> : k_cluster<kCluOneThreads, true, true>;
    return threads <= 640 ? k_cluster<640, false, true> : k_cluster<1024, false, true>;
  }
  if (one) return threads <= 512 ? k_cluster<512, true, false> : k_cluster<1024, true, false>;
  return k_cluster<1024, false, false>;
}

}  // namespace
