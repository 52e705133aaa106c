// trace.cuh -- closest-hit scene queries, sampling and photon lookups.
//
// intersect_scene() returns the closest hit over the mesh instances and the
// surfel cloud, the FirstHit mode of intersectScene
// (Pale/Renderer/Kernels/IntersectionKernels.h:954-1097).  The surfel part
// walks the LBVH with a short stack of (node, entry distance) pairs; the
// first `top_nodes` nodes are read from a shared-memory copy staged by the
// calling kernel.
#pragma once

#include "common.cuh"

namespace pale {

struct Hit {
  int inst;        // -1 miss; mesh instance index; == mesh.instances for a surfel
  uint32_t prim;   // triangle id or surfel index (BVH order)
  float t;         // world-space distance along the ray
  float alpha;     // alpha_geom of a surfel hit (0 for meshes)
  V3 pos;          // world hit position
};

struct TraceCounters {
  uint32_t nodes;
  uint32_t tests;
};

// safeInvDir (KernelHelpers.h:140-148).
__device__ __forceinline__ V3 safe_inv(V3 d) {
  return v3(fabsf(d.x) < 1e-6f ? 1e30f : 1.f / d.x, fabsf(d.y) < 1e-6f ? 1e30f : 1.f / d.y,
            fabsf(d.z) < 1e-6f ? 1e30f : 1.f / d.z);
}

// slabIntersectAABB (KernelHelpers.h:150-214): returns the entry distance
// or +inf on a miss.
__device__ __forceinline__ float slab_entry(V3 o, V3 inv, float lx, float ly, float lz, float hx, float hy,
                                            float hz, float limit) {
  float t0x = (lx - o.x) * inv.x, t1x = (hx - o.x) * inv.x;
  float t0y = (ly - o.y) * inv.y, t1y = (hy - o.y) * inv.y;
  float t0z = (lz - o.z) * inv.z, t1z = (hz - o.z) * inv.z;
  float tmin = fmaxf(fmaxf(fminf(t0x, t1x), fminf(t0y, t1y)), fminf(t0z, t1z));
  float tmax = fminf(fminf(fmaxf(t0x, t1x), fmaxf(t0y, t1y)), fmaxf(t0z, t1z));
  if (tmin > tmax || tmax < 0.0f || tmin > limit) return __int_as_float(0x7f800000);
  return tmin;
}

// A box is entered when the slab test hit it (finite entry) no farther
// than the current closest hit.  The finiteness check matters while `best`
// is still +inf: a miss (+inf) must not compare as "<= best".
__device__ __forceinline__ bool entered(float e, float best) { return e < 3.402823466e+38f && e <= best; }

// intersectTriangle (KernelHelpers.h:248-277).
__device__ __forceinline__ bool tri_hit(V3 o, V3 d, V3 v0, V3 v1, V3 v2, float tmin, float& t_out) {
  V3 e1 = v1 - v0, e2 = v2 - v0;
  V3 h = cross(d, e2);
  float a = dot(e1, h);
  if (fabsf(a) < 1.0e-4f) return false;
  float f = 1.0f / a;
  V3 s = o - v0;
  float u = f * dot(s, h);
  if (u < 0.0f || u > 1.0f) return false;
  V3 q = cross(s, e1);
  float v = f * dot(d, q);
  if (v < 0.0f || u + v > 1.0f) return false;
  float t = f * dot(e2, q);
  if (t <= tmin) return false;
  t_out = t;
  return true;
}

// intersectSurfel + opacityBeta (KernelHelpers.h:506-669) on the
// precomputed surfel arrays.
__device__ __forceinline__ bool surfel_hit(const SurfelView& sf, uint32_t i, V3 o, V3 d, float tmin, float tmax,
                                           float& t_out, V3& x_out, float& a_out) {
  const float4 n4 = __ldg(&sf.n[i]);
  const float4 pe = __ldg(&sf.pe[i]);
  V3 n = xyz(n4);
  float nd = dot(n, d);
  if (fabsf(nd) < 1e-6f) return false;
  V3 p = xyz(pe);
  float th = dot(n, p - o) / nd;
  if (th <= tmin || th >= tmax) return false;
  const float4 u4 = __ldg(&sf.u[i]);
  const float4 v4 = __ldg(&sf.v[i]);
  V3 x = o + scale(d, th);
  V3 r = x - p;
  float u = dot(xyz(u4), r) / u4.w;
  float v = dot(xyz(v4), r) / v4.w;
  float r2 = u * u + v * v;
  if (r2 >= 1.0f) return false;
  a_out = powf(1.0f - r2, pe.w);
  t_out = th;
  x_out = x;
  return true;
}

// The hit point and alpha_geom of surfel i at distance th along (o, d):
// the operations of surfel_hit after its distance test, so the values are
// the ones it computed for that hit.
__device__ __forceinline__ void surfel_eval(const SurfelView& sf, uint32_t i, V3 o, V3 d, float th, V3& x_out,
                                            float& a_out) {
  const float4 pe = __ldg(&sf.pe[i]);
  const float4 u4 = __ldg(&sf.u[i]);
  const float4 v4 = __ldg(&sf.v[i]);
  V3 x = o + scale(d, th);
  V3 r = x - xyz(pe);
  float u = dot(xyz(u4), r) / u4.w;
  float v = dot(xyz(v4), r) / v4.w;
  float r2 = u * u + v * v;
  a_out = powf(1.0f - r2, pe.w);
  x_out = x;
}

#if PALE_HALF_NODES
// Two floats in a 64-bit register, for the packed multiply-add.
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long half2_to_float2(uint32_t v) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v));
  return pack2(f.x, f.y);
}

// A ray as the node test wants it: 1/d and -o/d by planes (x, y) and (z,
// z), and the byte permutations that pick the near and far planes by the
// signs of the direction.
struct NodeRay {
  unsigned long long inv_xy, inv_zz, no_xy, no_zz;
  uint32_t near_xy, near_z;
  __device__ __forceinline__ void set(V3 o, V3 inv) {
    inv_xy = pack2(inv.x, inv.y);
    inv_zz = pack2(inv.z, inv.z);
    no_xy = pack2(-(o.x * inv.x), -(o.y * inv.y));
    no_zz = pack2(-(o.z * inv.z), -(o.z * inv.z));
    near_xy = (inv.x < 0.0f ? 0x54u : 0x10u) | (inv.y < 0.0f ? 0x7600u : 0x3200u);
    near_z = inv.z < 0.0f ? 0x7654u : 0x3210u;
  }
};

// The slab tests of a node's two child boxes: e0, e1 the entry distances,
// and whether a box is entered no farther than `best` (slab_entry and
// entered(): in front of the origin, not past the current closest hit).  A
// plane's distance is one multiply-add, plane / d - o / d: against (plane -
// o) / d its rounding moves the plane by up to 2^-24 |o|, which the boxes'
// padding covers (half_nodes): a surfel's own excess, 1e-4 of its scale, is
// less than that for a small surfel a few units from the origin.
__device__ __forceinline__ void node_test(const NodeRay& r, const BvhNodeH& nd, float best, float& e0, float& e1,
                                          bool& h0, bool& h1) {
  const uint4 &q0 = nd.q0, &q1 = nd.q1;
  const uint32_t far_xy = r.near_xy ^ 0x4444u, far_z = r.near_z ^ 0x4444u;
  const float2 n0 = unpack2(fma2(half2_to_float2(__byte_perm(q0.x, q0.y, r.near_xy)), r.inv_xy, r.no_xy));
  const float2 f0 = unpack2(fma2(half2_to_float2(__byte_perm(q0.x, q0.y, far_xy)), r.inv_xy, r.no_xy));
  const float2 n1 = unpack2(fma2(half2_to_float2(__byte_perm(q0.z, q0.w, r.near_xy)), r.inv_xy, r.no_xy));
  const float2 f1 = unpack2(fma2(half2_to_float2(__byte_perm(q0.z, q0.w, far_xy)), r.inv_xy, r.no_xy));
  const float2 nz = unpack2(fma2(half2_to_float2(__byte_perm(q1.x, q1.y, r.near_z)), r.inv_zz, r.no_zz));
  const float2 fz = unpack2(fma2(half2_to_float2(__byte_perm(q1.x, q1.y, far_z)), r.inv_zz, r.no_zz));
  e0 = fmaxf(fmaxf(n0.x, n0.y), nz.x);
  e1 = fmaxf(fmaxf(n1.x, n1.y), nz.y);
  const float x0 = fminf(fminf(fminf(f0.x, f0.y), fz.x), best), x1 = fminf(fminf(fminf(f1.x, f1.y), fz.y), best);
  h0 = fmaxf(e0, 0.0f) <= x0;
  h1 = fmaxf(e1, 0.0f) <= x1;
}

__device__ __forceinline__ uint2 child_words(const BvhNodeH& nd) { return make_uint2(nd.q1.z, nd.q1.w); }
__device__ __forceinline__ BvhNodeH fetch_node(const BvhNodeH* nd) {
  BvhNodeH h;
  h.q0 = __ldg(&nd->q0);
  h.q1 = __ldg(&nd->q1);
  return h;
}
#else
struct NodeRay {
  V3 o, inv;
  __device__ __forceinline__ void set(V3 o_, V3 inv_) {
    o = o_;
    inv = inv_;
  }
};

__device__ __forceinline__ void node_test(const NodeRay& r, const BvhNode& nd, float best, float& e0, float& e1,
                                          bool& h0, bool& h1) {
  const float4 &a = nd.a, &b = nd.b, &c = nd.c;
  e0 = slab_entry(r.o, r.inv, a.x, a.y, a.z, a.w, b.x, b.y, best);
  e1 = slab_entry(r.o, r.inv, b.z, b.w, c.x, c.y, c.z, c.w, best);
  h0 = entered(e0, best);
  h1 = entered(e1, best);
}

__device__ __forceinline__ uint2 child_words(const BvhNode& nd) { return make_uint2(nd.d.x, nd.d.y); }
__device__ __forceinline__ BvhNode fetch_node(const BvhNode* nd) {
  BvhNode n;
  n.a = __ldg(&nd->a);
  n.b = __ldg(&nd->b);
  n.c = __ldg(&nd->c);
  n.d = __ldg(&nd->d);
  return n;
}
#endif

__device__ __forceinline__ TravNode load_node(const SceneView& S, const TravNode* __restrict__ smem_top,
                                              uint32_t idx) {
  return idx < S.top_nodes ? smem_top[idx] : fetch_node(S.nodes + idx);
}

// The traversal stack of one thread: its first PALE_SMEM_STACK entries in
// shared memory after the staged top nodes (entry k of thread t at
// [k * blockDim.x + t], so a warp's accesses hit distinct banks), the rest
// in a local array.  Traversal kernels size their dynamic shared memory for
// it (top_smem).  The local part alone would be 512 B per thread, more than
// L1 holds for four resident blocks, so pops would wait on L2.
struct TravStack {
#if PALE_SMEM_STACK > 0
  uint2* sm;
#endif
  uint32_t node[kStackDepth - PALE_SMEM_STACK];
  float t[kStackDepth - PALE_SMEM_STACK];
  __device__ __forceinline__ TravStack(const TravNode* smem_top, uint32_t top_nodes) {
#if PALE_SMEM_STACK > 0
    sm = reinterpret_cast<uint2*>(const_cast<TravNode*>(smem_top) + top_nodes) + threadIdx.x;
#else
    (void)smem_top;
    (void)top_nodes;
#endif
  }
  __device__ __forceinline__ void push(int sp, uint32_t n, float tt) {
#if PALE_SMEM_STACK > 0
    if (sp < PALE_SMEM_STACK) {
      sm[(size_t)sp * blockDim.x] = make_uint2(n, __float_as_uint(tt));
      return;
    }
#endif
    node[sp - PALE_SMEM_STACK] = n;
    t[sp - PALE_SMEM_STACK] = tt;
  }
  __device__ __forceinline__ void get(int sp, uint32_t& n, float& tt) const {
#if PALE_SMEM_STACK > 0
    if (sp < PALE_SMEM_STACK) {
      const uint2 e = sm[(size_t)sp * blockDim.x];
      n = e.x;
      tt = __uint_as_float(e.y);
      return;
    }
#endif
    n = node[sp - PALE_SMEM_STACK];
    tt = t[sp - PALE_SMEM_STACK];
  }
};

// One walk over the surfel LBVH, one step() at a time, so that a persistent
// kernel can hand a lane a new ray between steps.  A walk's position is a
// child word with its entry distance: an inner node (a step loads it, tests
// its two child boxes, continues with the nearer child hit and pushes the
// farther) or a leaf (a step tests its surfels).  Leaves go through the same
// near-to-far order and stack as inner nodes, so that a warp can run the
// steps of its lanes that stand at leaves together, apart from the inner
// visits (at_leaf()): the surfel test and the node visit are long and
// different code, and a lane that tested its leaf inside the node visit
// kept the other lanes of its warp waiting.  `Leaf` is the walk's leaf
// test (a closest hit, or the K closest hits).
template <class Leaf>
struct WalkBase {
  V3 o, d;
  NodeRay ray;
  float tmin;
  uint32_t node, visit;
  int sp;
  __device__ __forceinline__ void start(V3 o_, V3 d_, float tmin_) {
    o = o_;
    d = d_;
    ray.set(o_, safe_inv(d_));
    tmin = tmin_;
    node = 0;        // the root, an inner node
    visit = 0;
    sp = 0;
  }
  __device__ __forceinline__ bool at_leaf() const { return (node & kLeafFlag) != 0u; }
  // the next position from the stack whose box the ray can still enter
  __device__ __forceinline__ bool pop(const TravStack& stk, float best) {
    while (sp > 0) {
      --sp;
      uint32_t sn;
      float st_t;
      stk.get(sp, sn, st_t);
      if (st_t <= best) {
        node = sn;
        return true;
      }
    }
    return false;
  }
  __device__ __forceinline__ bool step(const SceneView& S, const TravNode* __restrict__ smem_top, TravStack& stk,
                                       TraceCounters& ctr, RunState* st) {
    Leaf& self = *static_cast<Leaf*>(this);
    if (at_leaf()) {
      // (its box was entered within `best`, which only this test changes)
      const uint32_t f0 = node & 0x0FFFFFFFu, cnt = ((node >> 28) & 7u) + 1u;
      if (f0 + cnt > S.sf.count) {
        flag_error(st, kErrBounds);
      } else {
        for (uint32_t j = 0; j < cnt; ++j) {
          ctr.tests++;
          self.test(S.sf, f0 + j);
        }
      }
      return pop(stk, self.best);
    }
    // an acyclic tree visits each node at most once
    const uint32_t visit_cap = 2u * S.node_count + 64u;
    if (node >= S.node_count || visit > visit_cap) {
      flag_error(st, kErrBounds);
      return false;
    }
    ++visit;
    const TravNode nd = load_node(S, smem_top, node);
    const uint2 w = child_words(nd);
    ctr.nodes++;
    float e0, e1;
    bool h0, h1;
    node_test(ray, nd, self.best, e0, e1, h0, h1);
    h0 = h0 && w.x != kEmptyChild;
    h1 = h1 && w.y != kEmptyChild;
    if (h0 && h1) {
      const bool first0 = e0 <= e1;
      if (sp < kStackDepth) {
        stk.push(sp, first0 ? w.y : w.x, first0 ? e1 : e0);
        ++sp;
      } else {
        flag_error(st, kErrStackOverflow);
      }
      node = first0 ? w.x : w.y;
      return true;
    }
    if (h0 || h1) {
      node = h0 ? w.x : w.y;
      return true;
    }
    return pop(stk, self.best);
  }
};

// Closest surfel with t in (tmin, limit): after start(), step() returns
// true while the walk goes on; `hit`, `prim` and `best` then hold the
// closest surfel.
struct ClosestWalk : WalkBase<ClosestWalk> {
  float best;
  uint32_t prim;
  bool hit;
  __device__ __forceinline__ void init(V3 o_, V3 d_, float tmin_, float limit) {
    start(o_, d_, tmin_);
    best = limit;
    prim = 0;
    hit = false;
  }
  __device__ __forceinline__ void test(const SurfelView& sf, uint32_t i) {
    float th, aa;
    V3 xx;
    // only the distance and the surfel stay live in the walk; the hit point
    // and alpha of the closest are evaluated after it
    if (surfel_hit(sf, i, o, d, tmin, best, th, xx, aa)) {
      best = th;
      hit = true;
      prim = i;
    }
  }
};

// Closest surfel with t in (tmin, limit) along (o, d) (the surfel cloud's
// transform is the identity, so this is intersectBLASPointCloudFirstHit,
// IntersectionKernels.h:585-675, where tmin is rayEpsilon = 1e-5).  Returns
// false on a miss.
__device__ __forceinline__ bool surfel_closest(const SceneView& S, const TravNode* __restrict__ smem_top, V3 o, V3 d,
                                               float tmin, float limit, uint32_t& prim, float& t, V3& x,
                                               float& alpha, TraceCounters& ctr, RunState* st) {
  if (S.node_count == 0) return false;
  TravStack stk(smem_top, S.top_nodes);
  ClosestWalk w;
  w.init(o, d, tmin, limit);
  while (w.step(S, smem_top, stk, ctr, st)) {
  }
  if (w.hit) {
    prim = w.prim;
    t = w.best;
    surfel_eval(S.sf, w.prim, o, d, w.best, x, alpha);
  }
  return w.hit;
}

// The K closest surfels with t in (tmin, limit) along (o, d), in increasing
// t (ties keep the surfel found first), with the culling distance of the
// K-th hit found so far.  After init(), step() returns true while the walk
// goes on; `count` (<= K) and t_out/prim_out then hold the hits in order.
template <int K>
struct KHitWalk : WalkBase<KHitWalk<K>> {
  float best;   // t_out[K - 1] once K hits are held
  uint32_t count;
  float t_out[K];
  uint32_t prim_out[K];
  __device__ __forceinline__ void init(V3 o_, V3 d_, float tmin_, float limit) {
    this->start(o_, d_, tmin_);
    best = limit;
    count = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      t_out[k] = limit;
      prim_out[k] = 0;
    }
  }
  __device__ __forceinline__ void test(const SurfelView& sf, uint32_t i) {
    float th, aa;
    V3 xx;
    if (surfel_hit(sf, i, this->o, this->d, this->tmin, best, th, xx, aa)) {
      // insert into the sorted list (static indices: stays in registers)
      uint32_t pj = i;
#pragma unroll
      for (int q = 0; q < K; ++q) {
        if (th < t_out[q]) {
          const float tt = t_out[q];
          const uint32_t pp = prim_out[q];
          t_out[q] = th;
          prim_out[q] = pj;
          th = tt;
          pj = pp;
        }
      }
      count = count < (uint32_t)K ? count + 1 : count;
      if (count == (uint32_t)K) best = t_out[K - 1];
    }
  }
};

// The same walk with its sorted hit list in shared memory instead of
// registers (entry q of a thread at hits[q * blockDim.x], (t, surfel)
// pairs), which frees the registers of the list for one more resident
// block; the list is read only when a surfel is hit.
template <int K>
struct KHitWalkS : WalkBase<KHitWalkS<K>> {
  float best;   // the K-th distance once K hits are held
  uint32_t count;
  uint2* hits;  // this thread's first entry
  __device__ __forceinline__ void bind(uint2* h) { hits = h; }
  __device__ __forceinline__ void init(V3 o_, V3 d_, float tmin_, float limit) {
    this->start(o_, d_, tmin_);
    best = limit;
    count = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) hits[(size_t)k * blockDim.x] = make_uint2(__float_as_uint(limit), 0u);
  }
  __device__ __forceinline__ void test(const SurfelView& sf, uint32_t i) {
    float th, aa;
    V3 xx;
    if (surfel_hit(sf, i, this->o, this->d, this->tmin, best, th, xx, aa)) {
      uint32_t pj = i;
#pragma unroll
      for (int q = 0; q < K; ++q) {
        const uint2 e = hits[(size_t)q * blockDim.x];
        const float tq = __uint_as_float(e.x);
        if (th < tq) {
          hits[(size_t)q * blockDim.x] = make_uint2(__float_as_uint(th), pj);
          th = tq;
          pj = e.y;
        }
      }
      count = count < (uint32_t)K ? count + 1 : count;
      if (count == (uint32_t)K) best = __uint_as_float(hits[(size_t)(K - 1) * blockDim.x].x);
    }
  }
  __device__ __forceinline__ uint32_t prim(int k) const { return hits[(size_t)k * blockDim.x].y; }
};

// One step of a persistent walk loop for the lanes of a warp: the lanes
// whose walk stands at a leaf step together once at least `batch` of them
// (or all of the walking lanes) do, the other times the lanes at inner nodes
// step, kBurst nodes at a time.  Returns for this lane whether its walk
// goes on (a lane that sat out the step keeps walking).  Every lane of the
// warp calls it.
template <int kBurst, class W>
__device__ __forceinline__ bool warp_step(W& w, bool walking, int batch, const SceneView& S,
                                          const TravNode* __restrict__ smem_top, TravStack& stk, TraceCounters& ctr,
                                          RunState* st) {
  const bool lf = walking && w.at_leaf();
  const unsigned ml = __ballot_sync(0xffffffffu, lf);
  const unsigned ma = __ballot_sync(0xffffffffu, walking);
  const bool leaf_phase = ml != 0u && (ml == ma || __popc(ml) >= batch);
  if (walking && lf == leaf_phase) {
    bool on = w.step(S, smem_top, stk, ctr, st);
#pragma unroll
    for (int k = 1; k < kBurst; ++k)
      if (!leaf_phase && on && !w.at_leaf()) on = w.step(S, smem_top, stk, ctr, st);
    return on;
  }
  return walking;
}

// The lanes of a warp that walk when `n` rays are shared by `warps` warps:
// all of them, or, when the rays would not fill every warp, as many as give
// each warp its share (a warp's lanes wait for one another at every step, so
// few rays are walked faster spread over idle warps than packed into one).
constexpr uint32_t kMinWalkLanes = 4;
__device__ __forceinline__ uint32_t walk_lanes(uint32_t n, uint32_t warps) {
  const uint32_t share = (n + warps - 1u) / warps;
  return share >= 32u ? 32u : (share < kMinWalkLanes ? kMinWalkLanes : share);
}

// A 4x4 instance matrix (16 floats, 64 B aligned) in four 16-byte loads.
__device__ __forceinline__ void load_matrix(const float* M, float (&m)[16]) {
  const float4* m4 = reinterpret_cast<const float4*>(M);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const float4 v = __ldg(&m4[r]);
    m[4 * r] = v.x;
    m[4 * r + 1] = v.y;
    m[4 * r + 2] = v.z;
    m[4 * r + 3] = v.w;
  }
}

// The closest mesh hit, in object space per instance (intersectBLASMesh,
// IntersectionKernels.h:37-105); `best` is the world distance of the hit
// (+inf on a miss).  The boxes of up to 32 instances are tested first, then
// each lane goes through the instances its own ray enters, in their order
// and while their box is no farther than its closest hit: a ray enters one
// or two of a room's walls, but the rays of a warp all of them, and testing
// each instance as its box is met made the warp run every instance's
// transform and triangles.
__device__ __forceinline__ Hit intersect_meshes(const SceneView& S, V3 o, V3 d, V3 invw, float& best) {
  Hit h;
  h.inst = -1;
  h.prim = 0;
  h.t = 3.402823466e+38f;
  h.alpha = 0.f;
  h.pos = v3(0.f, 0.f, 0.f);
  best = __int_as_float(0x7f800000);
  const MeshView& M = S.mesh;
  auto enters = [&](uint32_t i) {
    const float4 lo = __ldg(&M.box[2 * i]), hi = __ldg(&M.box[2 * i + 1]);
    return entered(slab_entry(o, invw, lo.x, lo.y, lo.z, hi.x, hi.y, hi.z, best), best);
  };
  for (uint32_t base = 0; base < M.instances; base += 32) {
    const uint32_t n = M.instances - base < 32u ? M.instances - base : 32u;
    uint32_t mask = 0;
    for (uint32_t k = 0; k < n; ++k) mask |= enters(base + k) ? 1u << k : 0u;
    const float before = best;
    for (; mask; mask &= mask - 1u) {
      const uint32_t i = base + (__ffs(mask) - 1);
      if (best < before && !enters(i)) continue;
      float w2o[16];
      load_matrix(M.w2o + 16 * i, w2o);
      V3 oo = xform_point(w2o, o);
      V3 dd = xform_dir(w2o, d);
      uint2 rg = __ldg(&M.tri_range[i]);
      float bt = __int_as_float(0x7f800000);
      bool any = false;
      uint32_t bprim = 0;
      for (uint32_t k = 0; k < rg.y; ++k) {
        const float4* tv = M.tri + 3 * (rg.x + k);
        float t;
        if (tri_hit(oo, dd, xyz(__ldg(&tv[0])), xyz(__ldg(&tv[1])), xyz(__ldg(&tv[2])), 1e-4f, t) && t < bt &&
            t > 0.0f) {
          bt = t;
          any = true;
          bprim = rg.x + k;
        }
      }
      if (!any) continue;
      float o2w[16];
      load_matrix(M.o2w + 16 * i, o2w);
      V3 hw = xform_point(o2w, oo + scale(dd, bt));
      float tw = dot(hw - o, d);
      if (tw > 0.0f && tw < best) {
        best = tw;
        h.inst = (int)i;
        h.t = tw;
        h.pos = hw;
        h.prim = bprim;
        h.alpha = 0.0f;
      }
    }
  }
  return h;
}

// intersectScene, FirstHit mode: mesh instances, then the surfel cloud;
// the closest world-space distance wins (:1060-1081).
__device__ __forceinline__ Hit intersect_scene(const SceneView& S, const TravNode* __restrict__ smem_top, V3 o, V3 d,
                                               TraceCounters& ctr, RunState* st) {
  float best;
  const V3 invw = safe_inv(d);
  Hit h = intersect_meshes(S, o, d, invw, best);
  if (S.has_pc &&
      entered(slab_entry(o, invw, S.pc_lo.x, S.pc_lo.y, S.pc_lo.z, S.pc_hi.x, S.pc_hi.y, S.pc_hi.z, best), best)) {
    V3 dd = normalize(d);
    // prune with the mesh hit plus a relative margin: a surfel beyond the
    // margin cannot have a smaller world distance than the mesh hit
    float limit = best < 3.0e38f ? best * 1.00001f + 1e-6f : __int_as_float(0x7f800000);
    uint32_t prim;
    float t, a;
    V3 x;
    if (surfel_closest(S, smem_top, o, dd, 1e-5f, limit, prim, t, x, a, ctr, st)) {
      float tw = dot(x - o, d);
      if (tw > 0.0f && tw < best) {
        best = tw;
        h.inst = (int)S.mesh.instances;
        h.t = tw;
        h.pos = x;
        h.prim = prim;
        h.alpha = a;
      }
    }
  }
  return h;
}

// intersectScene, Transmit mode (:1066-1090): the closest mesh hit, and the
// surfel cloud's transmissivity T over the whole ray
// (intersectBLASPointCloudTransmit, :837-948): the successive closest
// surfels from the same origin, t in (tMin, inf) with tMin = t_hit + 1e-4
// after each hit (the reference rejects t <= tMin after intersectSurfel's
// t > 1e-5, and tMin >= 1e-5), T *= 1 - opacity * alpha_geom, stopping once
// T <= 0.001.  The cloud is skipped (T = 1) when its box starts beyond the
// mesh hit, as the instance loop culls it.  `max_hits` bounds the walk (the
// kernel flags kErrLayerCap when it is reached).
__device__ __forceinline__ Hit intersect_scene_transmit(const SceneView& S, const TravNode* __restrict__ smem_top,
                                                        V3 o, V3 d, float& T, uint32_t max_hits,
                                                        TraceCounters& ctr, RunState* st) {
  float best;
  const V3 invw = safe_inv(d);
  Hit h = intersect_meshes(S, o, d, invw, best);
  T = 1.0f;
  if (S.has_pc &&
      entered(slab_entry(o, invw, S.pc_lo.x, S.pc_lo.y, S.pc_lo.z, S.pc_hi.x, S.pc_hi.y, S.pc_hi.z, best), best)) {
    const V3 dd = normalize(d);
    float tmin = 1e-5f;
    uint32_t k = 0;
    for (; k < max_hits; ++k) {
      uint32_t prim;
      float t, a;
      V3 x;
      if (!surfel_closest(S, smem_top, o, dd, tmin, __int_as_float(0x7f800000), prim, t, x, a, ctr, st)) break;
      const float alpha_eff = __ldg(&S.sf.n[prim]).w * a;
      T *= 1.0f - alpha_eff;
      tmin = t + 1e-4f;
      if (T <= 0.001f) break;
    }
    if (k == max_hits) flag_error(st, kErrLayerCap);
  }
  return h;
}

// buildIntersectionNormal (KernelHelpers.h:480-503).
__device__ __forceinline__ V3 hit_normal(const SceneView& S, const Hit& h) {
  if (h.inst < (int)S.mesh.instances) {
    // the world-space copy holds xform_point(o2w, v) of the triangle's vertices
    const uint32_t k = h.prim - __ldg(&S.mesh.tri_range[h.inst]).x;
    const float4* tv = S.mesh.wtri + 3 * (__ldg(&S.mesh.wtri_range[h.inst]).x + k);
    const V3 p0 = xyz(__ldg(&tv[0])), p1 = xyz(__ldg(&tv[1])), p2 = xyz(__ldg(&tv[2]));
    return normalize(cross(p1 - p0, p2 - p0));
  }
  return xyz(__ldg(&S.sf.cn[h.prim]));
}

// ------------------------------------------------------------- sampling
// sampleCosineHemisphere, rng-first overload (KernelHelpers.h:317-337).
__device__ __forceinline__ void sample_cosine(Rng& r, V3 n, V3& out, float& pdf) {
  float u1 = r.next_float(), u2 = r.next_float();
  float z = sqrtf(1.f - u1);
  float rr = sqrtf(1 - (z * z));
  float phi = 2.f * kPi * u2;
  float x = rr * cosf(phi), y = rr * sinf(phi);
  V3 up = fabsf(n.z) < .999f ? v3(0, 0, 1) : v3(1, 0, 0);
  V3 tang = normalize(cross(up, n));
  V3 bit = cross(n, tang);
  out = normalize(scale(tang, x) + scale(bit, y) + scale(n, z));
  pdf = fmaxf(0.f, dot(out, n)) / kPi;
}

// sampleUniformHemisphereAroundNormal with the Frisvad basis
// (KernelHelpers.h:541-611).
__device__ __forceinline__ void sample_uniform_hemi(Rng& r, V3 normal, V3& out, float& pdf) {
  V3 n = normalize(normal);
  float u1 = r.next_float(), u2 = r.next_float();
  float z = u1;
  float phi = 2.0f * kPi * u2;
  float rr = sqrtf(fmaxf(0.0f, 1.0f - z * z));
  float x = rr * cosf(phi), y = rr * sinf(phi);
  float sign = copysignf(1.0f, n.z);
  float a = -1.0f / (sign + n.z);
  float b = n.x * n.y * a;
  V3 T = v3(1.0f + sign * n.x * n.x * a, sign * b, -sign * n.x);
  V3 B = v3(b, sign + n.y * n.y * a, -n.y);
  out = normalize(scale(T, x) + scale(B, y) + scale(n, z));
  pdf = 1.0f / (2.0f * kPi);
}

// applyRussianRoulette (KernelHelpers.h:1612-1657).
__device__ __forceinline__ bool russian_roulette(Rng& r, uint32_t bounce, V3& thr, uint32_t start) {
  if (bounce < start) return true;
  if (!isfinite(thr.x) || !isfinite(thr.y) || !isfinite(thr.z)) return false;
  float lum = 0.2126f * thr.x + 0.7152f * thr.y + 0.0722f * thr.z;
  float p = clampf(lum, 0.0f, 0.99f);
  if (r.next_float() > p) return false;
  float c = 1.0f / p;
  c = fminf(c, 10.0f);
  thr = scale(thr, c);
  return true;
}

// sampleMeshAreaLight (KernelHelpers.h:340-449).
__device__ __forceinline__ bool sample_light(const SceneView& S, Rng& r, V3& pos, V3& nrm, V3& dir, V3& power) {
  const LightView& L = S.lights;
  if (L.count == 0) return false;
  float ul = r.next_float();
  uint32_t li = (uint32_t)(ul * (float)L.count);
  if (li > L.count - 1u) li = L.count - 1u;
  uint4 rec = __ldg(&L.rec[li]);
  float area = __ldg(&L.area[li]);
  if (rec.z == 0u || area <= 0.0f) return false;
  float ut = r.next_float();
  uint32_t lo = 0, hi = rec.z - 1u;
  while (lo < hi) {
    uint32_t mid = (lo + hi) >> 1u;
    if (ut <= __ldg(&L.cdf[rec.y + mid])) hi = mid;
    else lo = mid + 1u;
  }
  uint32_t tri = __ldg(&L.tri[rec.y + lo]);
  const float4* tv = S.mesh.tri + 3 * tri;
  V3 p0 = xyz(__ldg(&tv[0])), p1 = xyz(__ldg(&tv[1])), p2 = xyz(__ldg(&tv[2]));
  float u1 = r.next_float(), u2 = r.next_float();
  float su1 = sqrtf(u1);
  float b0 = 1.0f - su1, b1 = su1 * (1.0f - u2), b2 = su1 * u2;
  V3 xo = scale(p0, b0) + scale(p1, b1) + scale(p2, b2);
  float o2w[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) o2w[k] = __ldg(&S.mesh.o2w[16 * rec.x + k]);
  V3 w0 = xform_point(o2w, p0), w1 = xform_point(o2w, p1), w2 = xform_point(o2w, p2);
  V3 e0 = w1 - w0, e1 = w2 - w0;
  V3 nw = v3(e0.y * e1.z - e0.z * e1.y, e0.z * e1.x - e0.x * e1.z, e0.x * e1.y - e0.y * e1.x);
  float nl = sqrtf(dot(nw, nw));
  if (nl <= 0.0f) return false;
  nw = divs(nw, nl);
  float pdf;
  sample_cosine(r, nw, dir, pdf);
  pos = xform_point(o2w, xo);
  nrm = nw;
  float4 col = __ldg(&L.col[li]);
  power = scale(xyz(col), col.w);
  return true;
}

// --------------------------------------------------------------- photons
// worldToCellClamped / linearCellIndex (KernelHelpers.h:900-987).
__device__ __forceinline__ void world_to_cell(const GridView& G, V3 p, int c[3]) {
  V3 l = p - G.origin;
  float f[3] = {l.x / G.cell.x, l.y / G.cell.y, l.z / G.cell.z};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    int v = (int)floorf(f[a]);
    v = v < 0 ? 0 : v;
    v = v > G.res[a] - 1 ? G.res[a] - 1 : v;
    c[a] = v;
  }
}

// Per-launch constants of the lookups: 1 / (pi r^2), 1 / cell, and the
// T / D factor of the photon store (0 when nothing was deposited, so an
// empty map gives zero irradiance).
struct GatherConst {
  float inv_area;
  float inv_cx;
  float scale;
  uint32_t total_ph;   // photons in the sorted grid
};

__device__ __forceinline__ GatherConst gather_const(const GridView& G) {
  GatherConst c;
  const float r = G.radius, r2 = r * r;
  c.inv_area = 1.0f / (kPi * r2);
  c.inv_cx = 1.0f / G.cell.x;
  const uint32_t T = *G.attempts;
  const uint32_t D = (uint64_t)T < G.capacity ? T : (uint32_t)G.capacity;
  c.scale = D == 0u ? 0.0f : (float)T / (float)D;
  c.total_ph = __ldg(&G.cell_off[G.cells]);
  return c;
}

// The cell window [c0, c1] of a whole warp's lookup at x: lanes 0-5 each do
// one coordinate of world_to_cell(x - (r, r, r)) and world_to_cell(x + (r, r,
// r)), the same operations.
__device__ __forceinline__ void window_corners(const GridView& G, V3 x, int (&c0)[3], int (&c1)[3]) {
  const int lane = threadIdx.x & 31;
  const float r = G.radius;
  int wc = 0;
  if (lane < 6) {
    const int a = lane % 3;
    const float xa = a == 0 ? x.x : (a == 1 ? x.y : x.z);
    const float oa = a == 0 ? G.origin.x : (a == 1 ? G.origin.y : G.origin.z);
    const float ca = a == 0 ? G.cell.x : (a == 1 ? G.cell.y : G.cell.z);
    const float p = lane < 3 ? xa - r : xa + r;
    int v = (int)floorf((p - oa) / ca);
    v = v < 0 ? 0 : v;
    v = v > G.res[a] - 1 ? G.res[a] - 1 : v;
    wc = v;
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    c0[a] = __shfl_sync(0xffffffffu, wc, a);
    c1[a] = __shfl_sync(0xffffffffu, wc, 3 + a);
  }
}

// Row k of the window: its first photon j0 and its length (0 past the rows,
// or when every photon of the row is too far).
__device__ __forceinline__ void clip_row(const GridView& G, const GatherConst& GC, V3 x, const int (&c0)[3],
                                         const int (&c1)[3], int rows, int ny, float inv_ny, int k, uint32_t& j0,
                                         uint32_t& len) {
  const float r2 = G.radius * G.radius;
  const float inv_cx = GC.inv_cx;
  const uint32_t total_ph = GC.total_ph;
  if (k < rows) {
    const int kz = (int)(((float)k + 0.5f) * inv_ny);
    const int cz = c0[2] + kz, cy = c0[1] + (k - kz * ny);
    const uint32_t row = (uint32_t)((cz * G.res[1] + cy) * G.res[0]);
    // Clip the row to the sphere of radius r around x.  A photon binned
    // to cell c lies in [c, c + 1] cells from the origin up to rounding
    // (1% of a cell covers it), except in the edge cells, which also hold
    // the clamped photons from beyond the grid.  Every photon left out
    // lies farther than r * 1.001 from x, so the reference's loop rejects
    // it; the photons kept are summed in the same order.
    const float reach2 = r2 * 1.002f;
    float dy = 0.f, dz = 0.f;
    if (cy > 0) dy = fmaxf(dy, (G.origin.y + (float)cy * G.cell.y - 0.01f * G.cell.y) - x.y);
    if (cy < G.res[1] - 1) dy = fmaxf(dy, x.y - (G.origin.y + (float)(cy + 1) * G.cell.y + 0.01f * G.cell.y));
    if (cz > 0) dz = fmaxf(dz, (G.origin.z + (float)cz * G.cell.z - 0.01f * G.cell.z) - x.z);
    if (cz < G.res[2] - 1) dz = fmaxf(dz, x.z - (G.origin.z + (float)(cz + 1) * G.cell.z + 0.01f * G.cell.z));
    const float rho2 = dy * dy + dz * dz;
    if (rho2 <= reach2) {
      // (an approximate square root is enough: the 1.001 factor covers it)
      const float q = fmaxf(reach2 - rho2, 1e-30f);
      const float w = q * rsqrtf(q) * 1.001f + 0.01f * G.cell.x;
      // (a reciprocal is enough here: the 1% margin covers its rounding)
      int lo = (int)floorf(((x.x - w) - G.origin.x) * inv_cx);
      int hi = (int)floorf(((x.x + w) - G.origin.x) * inv_cx);
      lo = lo > c0[0] ? lo : c0[0];
      hi = hi < c1[0] ? hi : c1[0];
      if (lo <= hi) {
        uint32_t a = __ldg(&G.cell_off[row + lo]);
        uint32_t b = __ldg(&G.cell_off[row + hi + 1]);
        b = b < total_ph ? b : total_ph;
        a = a < b ? a : b;
        j0 = a;
        len = b - a;
      }
    }
  }
}

// Rounds of a row in flight (2 and 4 measured 36.4 and 35.5 ms, 7.9 and 7.1 ms
// over dense photons).
constexpr int kHeavyUnroll = 4;
// gatherDiffuseIrradianceAtPoint (KernelHelpers.h:990-1037), done by a
// whole warp for one query (x, n), which every lane passes.  Photons are
// stored sorted by cell with ascending deposit index inside a cell, and the
// cells of one grid row (fixed y, z) are contiguous, so each row of the
// query window is one contiguous photon range and walking the rows in
// (z, y) order visits the photons in the reference's cell-by-cell order.
// Photon v of that sequence (numbered anew after every 32 rows) is lane v
// mod 32's: every lane adds the power of its photons that pass the radius
// and cosine tests into its own running sum, and the 32 sums are added at
// the end by a butterfly of shuffles: the same terms as the reference's
// one-photon-at-a-time loop, summed in another order (the result differs
// from it by float rounding, about 1e-7 relative; a photon within a rounding
// error of the radius can fall on either side).  Row after row, a round of
// 32 photons is its three loads and about 15 instructions; a row's last
// round is partly filled, which long rows do not feel.
// Returns the irradiance in every lane and adds the photons scanned to
// `count`.
__device__ __forceinline__ V3 gather_irradiance_rows(const GridView& G, const GatherConst& GC, V3 x, V3 n,
                                                     uint32_t& count) {
  const int lane = threadIdx.x & 31;
  const float r2 = G.radius * G.radius;
  const float invArea = GC.inv_area;
  int c0[3], c1[3];
  window_corners(G, x, c0, c1);
  const int ny = c1[1] - c0[1] + 1;
  const int rows = (c1[2] - c0[2] + 1) * ny;
  const float inv_ny = __fdividef(1.0f, (float)ny);
  float ax = 0.f, ay = 0.f, az = 0.f;
  for (int rb = 0; rb < rows; rb += 32) {
    uint32_t j0 = 0, len = 0;
    clip_row(G, GC, x, c0, c1, rows, ny, inv_ny, rb + lane, j0, len);
    uint32_t ex = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, ex, o);
      if (lane >= o) ex += y;
    }
    count += __shfl_sync(0xffffffffu, ex, 31);
    ex -= len;
    // per row: its end, and the photon whose turn is lane 0's
    const uint32_t end = j0 + len, turn = j0 - ex;
    for (unsigned nm = __ballot_sync(0xffffffffu, len > 0); nm; nm &= nm - 1u) {
      const int k = __ffs(nm) - 1;
      const uint32_t rj0 = __shfl_sync(0xffffffffu, j0, k), rend = __shfl_sync(0xffffffffu, end, k);
      const uint32_t rturn = __shfl_sync(0xffffffffu, turn, k);
#pragma unroll kHeavyUnroll
      for (uint32_t j = rj0 + ((lane + rturn - rj0) & 31u); j < rend; j += 32) {
        const float4 pa = __ldg(&G.pa[j]), pb = __ldg(&G.pb[j]);
        const float pc = __ldg(&G.pc[j]);
        const float dx = pa.x - x.x, dy = pa.y - x.y, dz = pa.z - x.z;
        const float d2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx));
        const float cosine = -__fmaf_rn(n.z, pb.z, __fmaf_rn(n.y, pb.y, n.x * pb.x));
        if (d2 <= r2 && !(cosine < 0.0f)) {
          ax = __fmaf_rn(pa.w, invArea, ax);
          ay = __fmaf_rn(pb.w, invArea, ay);
          az = __fmaf_rn(pc, invArea, az);
        }
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ax += __shfl_xor_sync(0xffffffffu, ax, o);
    ay += __shfl_xor_sync(0xffffffffu, ay, o);
    az += __shfl_xor_sync(0xffffffffu, az, o);
  }
  const float s = GC.scale;
  return v3(ax * s, ay * s, az * s);
}

// The lookup of gather_irradiance_rows for a query of any length by a whole
// warp: the rows are concatenated (a warp scan of their lengths) and each
// round the 32 lanes take 32 consecutive photons of that sequence, loaded
// one round ahead of their tests and sum; the same photons in the same
// lanes, so the result is that function's, bit for bit.  `terms` is this
// warp's 32 float4 of shared memory (the row compaction).  For queries
// without neighbours of like length beside them (the adjoint's events).
__device__ __forceinline__ V3 gather_irradiance_warp(const GridView& G, const GatherConst& GC, V3 x, V3 n,
                                                     float4* terms, uint32_t& count) {
  const int lane = threadIdx.x & 31;
  const float r = G.radius, r2 = r * r;
  const float invArea = GC.inv_area;
  int c0[3], c1[3];
  window_corners(G, x, c0, c1);
  const int ny = c1[1] - c0[1] + 1;
  const int rows = (c1[2] - c0[2] + 1) * ny;
  // row k of the window is (z, y) = (k / ny, k % ny); (k + 1/2) / ny is at
  // least 1/(2 ny) from an integer, far beyond float rounding
  const float inv_ny = __fdividef(1.0f, (float)ny);
  float ax = 0.f, ay = 0.f, az = 0.f;   // this lane's sums of the accepted terms
  uint32_t scanned = 0;
  for (int rb = 0; rb < rows; rb += 32) {
    // this lane's row: first photon and length
    const int k = rb + lane;
    uint32_t j0 = 0, len = 0;
    clip_row(G, GC, x, c0, c1, rows, ny, inv_ny, k, j0, len);
    uint32_t incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const uint32_t excl = incl - len;
    const uint32_t seq = __shfl_sync(0xffffffffu, incl, 31);
    scanned += seq;
    // the non-empty rows, compacted into lanes 0..nne-1 in row order (their
    // starts are then strictly increasing); staged through the terms buffer
    const unsigned nm = __ballot_sync(0xffffffffu, len > 0);
    const int nne = __popc(nm);
    uint32_t* cw = reinterpret_cast<uint32_t*>(terms);
    if (len > 0) {
      const int o = __popc(nm & ((1u << lane) - 1u));
      cw[o] = j0;
      cw[32 + o] = excl;
    }
    __syncwarp();
    const uint32_t cj0 = lane < nne ? cw[lane] : 0u;
    const uint32_t cex = lane < nne ? cw[32 + lane] : 0xFFFFFFFFu;
    __syncwarp();
    // The photon of sequence index base + lane: its three records at once
    // (one memory round trip per round).
    auto fetch = [&](uint32_t base, float4& pa, float4& pb, float& pc) {
      const uint32_t v = base + lane;
      // row holding sequence index v: the non-empty rows starting at or
      // before v are those starting before this round plus those starting
      // in the round at lanes <= this one (one bit per row start)
      const bool starts_here = lane < nne && cex >= base && cex - base < 32u;
      const uint32_t smask = __reduce_or_sync(0xffffffffu, starts_here ? (1u << (cex - base)) : 0u);
      const uint32_t before = __popc(__ballot_sync(0xffffffffu, lane < nne && cex < base));
      const int ord = (int)before + __popc(smask & (0xFFFFFFFFu >> (31 - lane))) - 1;
      const uint32_t rj0 = __shfl_sync(0xffffffffu, cj0, ord & 31);
      const uint32_t rex = __shfl_sync(0xffffffffu, cex, ord & 31);
      if (v < seq) {
        const uint32_t j = rj0 + (v - rex);
        pa = __ldg(&G.pa[j]);
        pb = __ldg(&G.pb[j]);
        pc = __ldg(&G.pc[j]);
      }
    };
    float4 pa = make_float4(0.f, 0.f, 0.f, 0.f), pb = pa;
    float pc = 0.f;
    if (seq > 0) fetch(0, pa, pb, pc);
    for (uint32_t base = 0; base < seq; base += 32) {
      float4 na = make_float4(0.f, 0.f, 0.f, 0.f), nb = na;
      float nc = 0.f;
      if (base + 32 < seq) fetch(base + 32, na, nb, nc);
      const uint32_t v = base + lane;
      if (v < seq) {
        const float dx = pa.x - x.x, dy = pa.y - x.y, dz = pa.z - x.z;
        const float d2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx));
        const float cosine = -__fmaf_rn(n.z, pb.z, __fmaf_rn(n.y, pb.y, n.x * pb.x));
        if (d2 <= r2 && !(cosine < 0.0f)) {
          ax = __fmaf_rn(pa.w, invArea, ax);
          ay = __fmaf_rn(pb.w, invArea, ay);
          az = __fmaf_rn(pc, invArea, az);
        }
      }
      pa = na;
      pb = nb;
      pc = nc;
    }
  }
  count += scanned;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ax += __shfl_xor_sync(0xffffffffu, ax, o);
    ay += __shfl_xor_sync(0xffffffffu, ay, o);
    az += __shfl_xor_sync(0xffffffffu, az, o);
  }
  const float s = GC.scale;
  return v3(ax * s, ay * s, az * s);
}

// Whether any photon can lie in the window of a lookup at x (false: its
// irradiance is zero).  The window starts at cell c0; the bit of c0 covers
// kLitCells cells from there in every axis.
__device__ __forceinline__ bool window_lit(const GridView& G, V3 x) {
  const float r = G.radius;
  int c0[3], c1[3];
  world_to_cell(G, v3(x.x - r, x.y - r, x.z - r), c0);
  world_to_cell(G, v3(x.x + r, x.y + r, x.z + r), c1);
  // a window that rounding made wider is looked at in full
  if (c1[0] - c0[0] >= kLitCells || c1[1] - c0[1] >= kLitCells || c1[2] - c0[2] >= kLitCells) return true;
  const size_t row = (size_t)c0[2] * G.res[1] + c0[1];
  return (__ldg(&G.lit[row * G.lit_row + ((uint32_t)c0[0] >> 5)]) >> (c0[0] & 31)) & 1u;
}

// The lookup of gather_irradiance_rows by kLanes lanes of a warp, 32 /
// kLanes queries at a time: every lane passes its group's query (a group
// without one passes valid = false) and gets its irradiance.  The photons of
// a query, concatenated over its clipped rows, are numbered as there, and
// photon v goes into partial sum v mod 32: lane p holds the kSlots partial
// sums p, p + kLanes, ... in registers, and the sums are added as the
// butterfly over 32 lanes adds them (the levels above kLanes inside the
// lane, the others by shuffles), so the result is that function's, bit for
// bit.  What it saves is the per-query work, most of a short lookup's
// instructions: window corners, row clipping, scan and butterfly run for
// 32 / kLanes queries at once, and a lane finds a photon's row by counting,
// in a word of bits, the rows that start up to it (the rows' first photons
// stand in shared memory), so that short rows leave no lane idle: on lookups
// of up to 256 photons about 190 warp instructions a lookup against 380 by a
// whole warp.  The photon numbers of neighbouring queries are neighbours when
// the queries are grouped by cell.  A query of more than
// kLookupHeavy photons is not done (heavy; its result is undefined): there
// the photons' own work counts, which a whole warp shares better.
// (128, 256 and 512: 74.3, 68.6 and 66.1 ms of camera lookups on 200k surfels,
// 8 views; 18.8, 17.4 and 17.1 ms on three scenes; 1.51, 1.35 and 1.47 ms on
// six small views)
#ifndef PALE_LOOKUP_HEAVY
#define PALE_LOOKUP_HEAVY 256
#endif
constexpr uint32_t kLookupHeavy = PALE_LOOKUP_HEAVY;
static_assert(PALE_LOOKUP_HEAVY >= 32 && PALE_LOOKUP_HEAVY % 32 == 0 && PALE_LOOKUP_HEAVY < 4095,
              "PALE_LOOKUP_HEAVY: whole words of 32 photons, below the row length that counts as heavy");

// Shared memory of a group's lookup: per non-empty row its first photon less
// its place in the sequence; a bit per photon of the sequence, set where a
// row starts; squared distances to the window's y rows and z slabs.
struct LaneLookup {
  uint32_t row[32];
  uint32_t starts[kLookupHeavy / 32];
  float sq[16];
};

template <int kLanes>
__device__ __forceinline__ V3 gather_irradiance_lanes(const GridView& G, const GatherConst& GC, V3 x, V3 n,
                                                      bool valid, LaneLookup& sm, uint32_t& count, bool& heavy) {
  constexpr int kSlots = 32 / kLanes;   // partial sums per lane, and rows per lane of 32
  const int p = threadIdx.x & (kLanes - 1);
  const float r = G.radius, r2 = r * r;
  const float invArea = GC.inv_area;
  // window corners (the operations of world_to_cell(x -+ (r, r, r)))
  int wc[(6 + kLanes - 1) / kLanes];
#pragma unroll
  for (int t = 0; t < (6 + kLanes - 1) / kLanes; ++t) {
    const int i = p + t * kLanes, a = i % 3;
    const float xa = a == 0 ? x.x : (a == 1 ? x.y : x.z);
    const float oa = a == 0 ? G.origin.x : (a == 1 ? G.origin.y : G.origin.z);
    const float ca = a == 0 ? G.cell.x : (a == 1 ? G.cell.y : G.cell.z);
    const int ra = a == 0 ? G.res[0] : (a == 1 ? G.res[1] : G.res[2]);
    const float q = i < 3 ? xa - r : xa + r;
    int v = (int)floorf((q - oa) / ca);
    v = v < 0 ? 0 : v;
    wc[t] = v > ra - 1 ? ra - 1 : v;
  }
  int c0[3], c1[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    c0[a] = __shfl_sync(0xffffffffu, wc[a / kLanes], a % kLanes, kLanes);
    c1[a] = __shfl_sync(0xffffffffu, wc[(3 + a) / kLanes], (3 + a) % kLanes, kLanes);
  }
  const int ny = c1[1] - c0[1] + 1, nz = c1[2] - c0[2] + 1;
  const int rows = valid ? nz * ny : 0;
  const float inv_ny = __fdividef(1.0f, (float)ny);
  const float inv_cx = GC.inv_cx;
  const uint32_t total_ph = GC.total_ph;
  const float reach2 = r2 * 1.002f;
  // squared distances of x to the window's y rows (0..7) and z slabs (8..15);
  // a window that rounding made wider than 8 cells has its photons within r
  // in the first 8 (there a cell is finer than the positions)
#pragma unroll
  for (int t = 0; t < 16 / kLanes; ++t) {
    const int i = p + t * kLanes;
    const bool isz = i >= 8;
    const int c = isz ? c0[2] + (i - 8) : c0[1] + i;
    const float o = isz ? G.origin.z : G.origin.y, ce = isz ? G.cell.z : G.cell.y, xa = isz ? x.z : x.y;
    const int ra = isz ? G.res[2] : G.res[1];
    float dd = 0.f;
    if (c > 0) dd = fmaxf(dd, (o + (float)c * ce - 0.01f * ce) - xa);
    if (c < ra - 1) dd = fmaxf(dd, xa - (o + (float)(c + 1) * ce + 0.01f * ce));
    sm.sq[i] = dd * dd;
  }
  __syncwarp();
  float ax[kSlots], ay[kSlots], az[kSlots];
#pragma unroll
  for (int s = 0; s < kSlots; ++s) ax[s] = ay[s] = az[s] = 0.f;
  uint32_t scanned = 0;
  heavy = false;
  for (int rb = 0; __any_sync(0xffffffffu, rb < rows); rb += 32) {
    // this lane's kSlots consecutive rows: first photon and length, clipped
    // to the sphere (as clip_row)
    uint32_t j0[kSlots], len[kSlots], tot = 0;
#pragma unroll
    for (int t = 0; t < kSlots; ++t) {
      const int k = rb + p * kSlots + t;
      j0[t] = len[t] = 0;
      if (k < rows) {
        const int kz = (int)(((float)k + 0.5f) * inv_ny);
        const int ky = k - kz * ny;
        const float rho2 = sm.sq[ky & 7] + sm.sq[8 + (kz & 7)];
        if (rho2 <= reach2) {
          const float q = fmaxf(reach2 - rho2, 1e-30f);
          const float w = q * rsqrtf(q) * 1.001f + 0.01f * G.cell.x;
          int lo = (int)floorf(((x.x - w) - G.origin.x) * inv_cx);
          int hi = (int)floorf(((x.x + w) - G.origin.x) * inv_cx);
          lo = lo > c0[0] ? lo : c0[0];
          hi = hi < c1[0] ? hi : c1[0];
          if (lo <= hi) {
            const uint32_t row = (uint32_t)(((c0[2] + kz) * G.res[1] + (c0[1] + ky)) * G.res[0]);
            uint32_t a = __ldg(&G.cell_off[row + lo]);
            uint32_t b = __ldg(&G.cell_off[row + hi + 1]);
            b = b < total_ph ? b : total_ph;
            a = a < b ? a : b;
            j0[t] = a;
            len[t] = b - a;
          }
        }
      }
    }
    // places in the sequence (lengths in the low half, non-empty rows in the
    // high half; a lane's length stops at 4095, which is heavy already)
    uint32_t ne = 0;
#pragma unroll
    for (int t = 0; t < kSlots; ++t) {
      tot += len[t] < 4095u ? len[t] : 4095u;
      ne += len[t] != 0u ? 1u : 0u;
    }
    const uint32_t own = (tot < 4095u ? tot : 4095u) | (ne << 16);
    uint32_t ex = own;
#pragma unroll
    for (int o = 1; o < kLanes; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, ex, o, kLanes);
      if (p >= o) ex += y;
    }
    uint32_t seq = __shfl_sync(0xffffffffu, ex, kLanes - 1, kLanes) & 0xFFFFu;
    ex -= own;
    if (seq > kLookupHeavy) heavy = true;
    if (heavy) seq = 0;
    scanned += seq;
    const uint32_t most = __reduce_max_sync(0xffffffffu, seq);
    if (most == 0u) continue;
#pragma unroll
    for (uint32_t w = 0; w < kLookupHeavy / 32; w += kLanes)
      if (w + p < kLookupHeavy / 32) sm.starts[w + p] = 0u;
    __syncwarp();
    {
      uint32_t v = ex & 0xFFFFu, k = ex >> 16;
#pragma unroll
      for (int t = 0; t < kSlots; ++t) {
        if (len[t] != 0u && v < seq) {
          sm.row[k] = j0[t] - v;
          atomicOr(&sm.starts[v >> 5], 1u << (v & 31u));
          ++k;
          v += len[t];
        }
      }
    }
    __syncwarp();
    uint32_t before = 0xFFFFFFFFu;   // rows that start before the block, less one
    for (uint32_t b = 0; b < most; b += 32) {
      const uint32_t starts = sm.starts[b >> 5];
      constexpr int kAhead = kSlots < 4 ? kSlots : 4;   // photons loaded at once
#pragma unroll
      for (int s0 = 0; s0 < kSlots; s0 += kAhead) {
        if (b + s0 * kLanes >= most) break;
        float4 pa[kAhead];
        uint32_t j[kAhead];
#pragma unroll
        for (int s = 0; s < kAhead; ++s) {
          const int l = (s0 + s) * kLanes + p;
          const uint32_t v = b + l;
          pa[s] = make_float4(__int_as_float(0x7f800000), 0.f, 0.f, 0.f);   // fails the radius test
          j[s] = 0;
          if (v < seq) {
            j[s] = v + sm.row[before + __popc(starts & (0xFFFFFFFFu >> (31 - l)))];
            pa[s] = __ldg(&G.pa[j[s]]);
          }
        }
#pragma unroll
        for (int s = 0; s < kAhead; ++s) {
          const float dx = pa[s].x - x.x, dy = pa[s].y - x.y, dz = pa[s].z - x.z;
          const float d2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx));
          if (d2 <= r2) {
            const float4 pb = __ldg(&G.pb[j[s]]);
            const float pc = __ldg(&G.pc[j[s]]);
            const float cosine = -__fmaf_rn(n.z, pb.z, __fmaf_rn(n.y, pb.y, n.x * pb.x));
            if (!(cosine < 0.0f)) {
              ax[s0 + s] = __fmaf_rn(pa[s].w, invArea, ax[s0 + s]);
              ay[s0 + s] = __fmaf_rn(pb.w, invArea, ay[s0 + s]);
              az[s0 + s] = __fmaf_rn(pc, invArea, az[s0 + s]);
            }
          }
        }
      }
      before += __popc(starts);
    }
    __syncwarp();
  }
  count += scanned;
#pragma unroll
  for (int o = kSlots / 2; o > 0; o >>= 1) {
#pragma unroll
    for (int s = 0; s < o; ++s) {
      ax[s] += ax[s + o];
      ay[s] += ay[s + o];
      az[s] += az[s + o];
    }
  }
#pragma unroll
  for (int o = kLanes / 2; o > 0; o >>= 1) {
    ax[0] += __shfl_xor_sync(0xffffffffu, ax[0], o);
    ay[0] += __shfl_xor_sync(0xffffffffu, ay[0], o);
    az[0] += __shfl_xor_sync(0xffffffffu, az[0], o);
  }
  const float s = GC.scale;
  return v3(ax[0] * s, ay[0] * s, az[0] * s);
}

// Lanes per short lookup: 4, 8 and 16 measured 67.1, 68.6 and 75.6 ms of camera
// lookups on 200k surfels, 8 views; 16.6, 17.4 and 18.0 ms on three scenes;
// 1.44, 1.35 and 1.31 ms on six small views.
#ifndef PALE_LOOKUP_LANES
#define PALE_LOOKUP_LANES 8
#endif
constexpr int kLookupLanes = PALE_LOOKUP_LANES;
static_assert(kLookupLanes == 4 || kLookupLanes == 8 || kLookupLanes == 16,
              "PALE_LOOKUP_LANES: 4, 8 or 16 lanes (the 16 squared distances are split over them)");

}  // namespace pale
