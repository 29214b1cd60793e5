// Software two-level BVH traversal: closest hit and any hit.
//
// Replaces the hardware ray queries of the reference wavefront
// (nativeTraceSurface, ordinarylight/shaders/wavefront_intersect.comp:96-235;
// nativeOccluded in ordinarylight/shaders/transport_v1/lighting.glsl).
// * TLAS and BLAS nodes share one node pool; a TLAS leaf is one instance.
//   Traversal reads the BVH4 form of the pool (BvhNode4: up to four
//   descendants of a BVH2 node in one 128-byte line, collapsed at the least
//   surface-area cost, with up to two triangles a leaf), so each dependent fetch descends about two levels of the
//   binary hierarchy.  A ray picks each axis's near and far box planes once
//   from its direction's signs, so the slab test needs no per-axis min/max.
//   Entering an instance transforms the ray to object space (t is preserved
//   because the direction is not renormalised) and pushes a marker that
//   restores the world ray when the instance's subtree is exhausted; the
//   world ray and its derived terms are kept meanwhile in OLC_RAY_SAVE shared
//   words per thread instead of being recomputed.
// * The traversal stack lives in shared memory (STACK entries per thread,
//   entry k of thread t at k * blockDim.x + t, so a warp's pushes hit 32
//   distinct banks), followed by the per-thread shared words in the same
//   column layout; a launch gives (STACK + OLC_RAY_SAVE) * blockDim.x words.
//   What a ray needs only at instance transitions or at its end (the world
//   ray, the closest hit's barycentrics) lives there rather than in
//   registers, which keeps eight blocks of 128 threads resident per SM.
//   Deeper entries spill to a bounded local array.  A push beyond both is
//   counted as a traversal error instead of writing out of bounds.
// * Triangles use the watertight test of Woop, Benthin and Wald (JCGT 2013):
//   the edge functions are evaluated without FMA contraction so that an edge
//   shared by two triangles gets exactly negated values, with a double
//   precision re-evaluation when an edge function is exactly zero.
// * Closest-hit ties (equal t) resolve to the lowest packed triangle index,
//   the rule of ReferencePathTracer._intersect (strict "<" over triangles in
//   packed order, ordinarylight/renderers/reference/path_tracer.py:159-175),
//   which also makes the result independent of traversal order.
#pragma once

#include "olc_common.cuh"

#define OLC_SPILL 96
// Shared words per thread beyond the stack: the world ray's derived terms
// (0-6), restored on leaving an instance; the world ray's origin (7-9) and
// direction (10-12); the closest hit's barycentrics (13-14).
#define OLC_RAY_SAVE 15
#define OLC_SAVE_ORIGIN 7
#define OLC_SAVE_DIR 10
#define OLC_SAVE_UV 13
#define OLC_NO_INSTANCE 0xffffffffu
#define OLC_MARKER 0x7fffffff
#define OLC_TRAVERSAL_BUDGET (1u << 22)
// Lanes that hold a leaf before a warp tests leaves, in queues long enough for
// it (kLeafWaitRays).  Lanes part, so a step has 7 to 9 of 32 active, and a
// leaf's code (a triangle test, or an instance's matrix and ray setup) ran for
// one or two of them at a time.  A waiting lane loses a step or two but keeps
// its order, so nothing is tested that was not before, and the wait is no step
// of its budget.  0 -> 6 lanes: 1080p instanced frame 6.22 -> 6.17 ms, terrain
// 10.61 -> 10.34 ms, textured 2.22 -> 2.20 ms; 4, 8 and 12 lanes: 6.50, 6.50
// and 6.55 ms where 6 gave 6.48, terrain 11.25, 11.19 and 11.22 where 6 gave
// 11.19.  (Stepping the whole warp together, with rays replaced as soon as 8
// to 20 lanes idle, was 2-5 % slower: lanes that part hide each other's loads.)
#define OLC_LEAF_LANES 6

struct TraceRay {
  float3 o;            // origin permuted by the shear permutation: (o[kx], o[ky], o[kz])
  float3 inv, noinv;   // reciprocal direction; -origin * reciprocal
  int kp;              // shear permutation kx | ky << 2 | kz << 4
  float sx, sy, sz;
  int nx, ny, nz;      // float4 index of each axis's near plane in a BvhNode4 (its far plane is index ^ 1)
};

OLC_D float3 permuted(float3 v, int kp) { return f3(get(v, kp & 3), get(v, (kp >> 2) & 3), get(v, kp >> 4)); }

// a / b, given r = 1 / b rounded to nearest: one residual correction of a * r
// rounds it to nearest (Markstein, IBM Journal of Research and Development
// 34(1), 1990) where nothing over- or underflows.
OLC_D float quotient(float a, float b, float r) {
  const float q = __fmul_rn(a, r);
  return __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
}

// One reciprocal per axis; the shear terms share the largest axis's (three
// divisions a ray instead of six: this runs at every ray's start and instance
// entry, with few lanes).  1080p instanced frame 6.38 -> 6.37 ms, textured
// 2.349 -> 2.340 ms.
OLC_D void setup_ray(TraceRay& r, float3 o, float3 d) {
  float dx = fabsf(d.x) < 1e-20f ? copysignf(1e-20f, d.x) : d.x;
  float dy = fabsf(d.y) < 1e-20f ? copysignf(1e-20f, d.y) : d.y;
  float dz = fabsf(d.z) < 1e-20f ? copysignf(1e-20f, d.z) : d.z;
  r.inv = f3(1.0f / dx, 1.0f / dy, 1.0f / dz);
  r.noinv = f3(-(o.x * r.inv.x), -(o.y * r.inv.y), -(o.z * r.inv.z));
  r.nx = r.inv.x < 0.0f ? 1 : 0;
  r.ny = r.inv.y < 0.0f ? 3 : 2;
  r.nz = r.inv.z < 0.0f ? 5 : 4;
  float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
  int kz = (ax > ay) ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
  int kx = kz + 1 == 3 ? 0 : kz + 1;
  int ky = kx + 1 == 3 ? 0 : kx + 1;
  float dkz = get(d, kz);
  if (dkz < 0.0f) { int t = kx; kx = ky; ky = t; }
  r.kp = kx | (ky << 2) | (kz << 4);
  r.o = permuted(o, r.kp);
  r.sz = get(r.inv, kz);
  r.sx = quotient(get(d, kx), dkz, r.sz);
  r.sy = quotient(get(d, ky), dkz, r.sz);
  // an infinite or tiny direction, whose reciprocal or residual is out of range
  if (!(fabsf(dkz) > 1e-18f && fabsf(dkz) < 1e18f)) {
    r.sz = 1.0f / dkz;
    r.sx = get(d, kx) / dkz;
    r.sy = get(d, ky) / dkz;
  }
}

// Watertight ray/triangle test on the slot's float4 triple `tv` (one float4
// per axis: that coordinate of the three vertices), so the shear permutation
// picks which float4 is read instead of selecting components.  Returns true
// with t, b1 (weight of v1), b2 (weight of v2) when the ray hits with
// t_min < t <= t_max.
OLC_D bool intersect_triangle(const TraceRay& r, const float4* tv, float t_min, float t_max, float& t_out, float& b1,
                              float& b2) {
  const float4 px = __ldg(tv + (r.kp & 3)), py = __ldg(tv + ((r.kp >> 2) & 3)), pz = __ldg(tv + (r.kp >> 4));
  float Akz = pz.x - r.o.z, Bkz = pz.y - r.o.z, Ckz = pz.z - r.o.z;
  float Ax = __fmaf_rn(-r.sx, Akz, px.x - r.o.x);
  float Ay = __fmaf_rn(-r.sy, Akz, py.x - r.o.y);
  float Bx = __fmaf_rn(-r.sx, Bkz, px.y - r.o.x);
  float By = __fmaf_rn(-r.sy, Bkz, py.y - r.o.y);
  float Cx = __fmaf_rn(-r.sx, Ckz, px.z - r.o.x);
  float Cy = __fmaf_rn(-r.sy, Ckz, py.z - r.o.y);
  float U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
  float V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
  float W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
  if (U == 0.0f || V == 0.0f || W == 0.0f) {
    double CxBy = (double)Cx * (double)By, CyBx = (double)Cy * (double)Bx;
    U = (float)(CxBy - CyBx);
    double AxCy = (double)Ax * (double)Cy, AyCx = (double)Ay * (double)Cx;
    V = (float)(AxCy - AyCx);
    double BxAy = (double)Bx * (double)Ay, ByAx = (double)By * (double)Ax;
    W = (float)(BxAy - ByAx);
  }
  if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
  float det = U + V + W;
  if (det == 0.0f) return false;
  float Az = r.sz * Akz, Bz = r.sz * Bkz, Cz = r.sz * Ckz;
  float T = U * Az + V * Bz + W * Cz;
  float t = __fdiv_rn(T, det);
  if (!(t > t_min) || !(t <= t_max)) return false;
  float rcp = 1.0f / det;
  t_out = t;
  b1 = V * rcp;
  b2 = W * rcp;
  return true;
}

// Save / restore the terms setup_ray derives from the world ray (o, d): the
// reciprocals, the shear permutation and constants; restoring also reads back
// the world origin and multiplies the slab offsets again.  `w` is this thread's column (stride threads).
OLC_D void save_ray(float* w, int stride, const TraceRay& r) {
  w[0 * stride] = r.inv.x; w[1 * stride] = r.inv.y; w[2 * stride] = r.inv.z;
  w[3 * stride] = r.sx; w[4 * stride] = r.sy; w[5 * stride] = r.sz;
  w[6 * stride] = __int_as_float(r.kp | (r.nx << 6) | (r.ny << 9) | (r.nz << 12));
}
OLC_D float3 saved3(const float* w, int stride, int first) {
  return f3(w[first * stride], w[(first + 1) * stride], w[(first + 2) * stride]);
}
OLC_D void restore_ray(const float* w, int stride, TraceRay& r) {
  const int k = __float_as_int(w[6 * stride]);
  r.kp = k & 63;
  r.nx = (k >> 6) & 7; r.ny = (k >> 9) & 7; r.nz = (k >> 12) & 7;
  const float3 o = saved3(w, stride, OLC_SAVE_ORIGIN);
  r.o = permuted(o, r.kp);
  r.inv = saved3(w, stride, 0);
  r.noinv = f3(-(o.x * r.inv.x), -(o.y * r.inv.y), -(o.z * r.inv.z));
  r.sx = w[3 * stride]; r.sy = w[4 * stride]; r.sz = w[5 * stride];
}

// Traversal stack of one thread: STACK words of its shared-memory column
// (addressed by their shared-window byte address, so a push is one store and
// one add), then a bounded local array.
template <int STACK>
struct TraversalStack {
  uint32_t base, top;  // byte address of entry 0 and of the next free entry
  uint32_t stride;     // bytes between entries
  uint32_t limit;      // address past the last shared entry
  int* spill;          // local overflow: OLC_SPILL entries, then their count (valid while top == limit)

  OLC_D void init(int* smem, int tid, int threads, int* spill_area) {
    base = (uint32_t)__cvta_generic_to_shared(smem + tid);
    stride = 4u * (uint32_t)threads;
    limit = base + (uint32_t)STACK * stride;
    top = base;
    spill = spill_area;
  }
  OLC_D bool empty() const { return top == base; }
  // Whether three more entries fit the shared words with one to spare.
  OLC_D bool roomy() const { return top + 3u * stride < limit; }
  OLC_D void push_shared(int v, bool want) {
    if (want) {
      asm volatile("st.shared.b32 [%0], %1;" ::"r"(top), "r"(v));
      top += stride;
    }
  }
  OLC_D bool push(int v, uint32_t& err) {
    if (top != limit) {
      push_shared(v, true);
      if (top == limit) spill[OLC_SPILL] = 0;
      return true;
    }
    const int n = spill[OLC_SPILL];
    if (n < OLC_SPILL) {
      spill[n] = v;
      spill[OLC_SPILL] = n + 1;
      return true;
    }
    err = 1u;
    return false;
  }
  OLC_D int pop() {
    if (top == limit) {
      const int n = spill[OLC_SPILL];
      if (n > 0) {
        spill[OLC_SPILL] = n - 1;
        return spill[n - 1];
      }
    }
    top -= stride;
    int v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(top));
    return v;
  }
};

OLC_D void load_instance_w2o(const InstanceRec* inst, uint32_t i, Affine& w2o, uint32_t& root) {
  const float4* p = reinterpret_cast<const float4*>(inst + i);
  w2o.r0 = __ldg(p + 0);
  w2o.r1 = __ldg(p + 1);
  w2o.r2 = __ldg(p + 2);
  root = __ldg(&inst[i].blas_root);
}

// Packed triangle index (Scene.triangles order) of triangle slot `slot` hit
// through instance `inst`: the closest-hit tie-break key.  Record 0, the
// identity instance of baked world-space triangles, has offset 0.
OLC_D uint32_t packed_index(const SceneView& s, uint32_t inst, uint32_t slot) {
  return __ldg(&s.instances[inst].prim_offset) + __ldg(s.tri_index + slot);
}

// Three-input float max / min (one instruction on sm_100).
OLC_D float fmax3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
OLC_D float fmin3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Distances to one axis's planes of two children: two fused multiply-adds in
// one instruction (each rounded as the scalar one).
OLC_D float2 plane2(float a, float b, float inv, float noinv) {
  float2 r;
  asm("{\n\t.reg .b64 p, q, c, d;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %4};\n\tmov.b64 c, {%5, %5};\n\t"
      "fma.rn.f32x2 d, p, q, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a), "f"(b), "f"(inv), "f"(noinv));
  return r;
}

// Slab test of one child box (Kay and Kajiya) on its near and far planes
// (chosen per ray by the direction's signs, so no min/max per axis), with the
// conservative far bound of robust traversal (Ize 2013): a few ulps of slack
// so rounding in the slab test never culls a box the ray touches.  Unused
// slots hold an inverted box (lo +inf, hi -inf), whose near distance is +inf
// and far distance -inf for every ray.
OLC_D bool slabs(float nx, float fx, float ny, float fy, float nz, float fz, float t_min, float t_max, float& near_t) {
  const float n = fmax3(nx, ny, fmaxf(nz, t_min));
  const float f = fmin3(fx, fy, fminf(fz, t_max));
  near_t = n;
  return n <= f * 1.0000004f;
}
// Bound: latency of the dependent node loads and the instructions issued per
// step (issue slots 60 % busy, 8-23 lanes active; a closest-hit ray makes 12-20
// node visits and 1-2 triangle tests).  The step is kept short: two planes per
// multiply-add instruction (plane2), the nearest child by a minimum instead of
// a sorting network, pushes of one store and one add with one bounds check per
// node, triangle vertices stored by axis, and no world ray restored for a ray
// that ends with its instance.  1080p instanced frame: trace_closest 4.05 ->
// 3.86 ms, trace_shadow 2.16 -> 2.06 ms, the frame's GPU time 6.50 -> 6.28 ms.
//
// Resumable traversal of the two-level structure.  ANY_HIT stops at the
// first hit in (t_min, t_max).  advance() runs at most `iterations` loop
// iterations (node visits, leaf tests, instance transitions) and returns true
// once the ray is finished, so a persistent kernel can refill lanes whose rays
// finished while the other lanes of the warp are still traversing.
//
// Register state is kept to what every iteration reads: the current ray, the
// closest t with its slot and instance, the node, the instance being walked
// (OLC_NO_INSTANCE in the TLAS) and the stack pointer.  The world ray and the
// closest hit's barycentrics live in the thread's shared words, and the
// packed tie-break index is looked up only when two hits have equal t.
template <int STACK, bool ANY_HIT>
struct Traversal {
  TraceRay ray;
  float t_min;
  float hit_t;
  uint32_t hit_slot;   // triangle slot (BVH order) of the closest hit so far
  uint32_t hit_inst;   // its instance; OLC_NO_INSTANCE while nothing was hit
  int node;
  uint32_t cur_inst;   // instance whose BLAS is being walked, or OLC_NO_INSTANCE
  uint32_t budget;
  float* save;         // this thread's column of OLC_RAY_SAVE shared words
  int stride;          // words between entries of the column
  TraversalStack<STACK> st;

  OLC_D bool found() const { return hit_inst != OLC_NO_INSTANCE; }
  OLC_D float hit_u() const { return save[OLC_SAVE_UV * stride]; }
  OLC_D float hit_v() const { return save[(OLC_SAVE_UV + 1) * stride]; }

  OLC_D void init(int* smem_base, int* spill_area) {
    st.init(smem_base, threadIdx.x, blockDim.x, spill_area);
    stride = blockDim.x;
    save = reinterpret_cast<float*>(smem_base + STACK * blockDim.x) + threadIdx.x;
  }

  OLC_D void begin(float3 o, float3 d, float tmin, float tmax, uint32_t tlas_root) {
    st.top = st.base;
    const int w = stride;
    save[(OLC_SAVE_ORIGIN + 0) * w] = o.x;
    save[(OLC_SAVE_ORIGIN + 1) * w] = o.y;
    save[(OLC_SAVE_ORIGIN + 2) * w] = o.z;
    save[(OLC_SAVE_DIR + 0) * w] = d.x;
    save[(OLC_SAVE_DIR + 1) * w] = d.y;
    save[(OLC_SAVE_DIR + 2) * w] = d.z;
    t_min = tmin;
    setup_ray(ray, o, d);
    save_ray(save, w, ray);   // the world ray's terms, restored on leaving an instance
    hit_t = tmax;
    hit_inst = OLC_NO_INSTANCE;
    hit_slot = 0;
    cur_inst = OLC_NO_INSTANCE;
    node = (int)tlas_root;
    // A well-formed tree is acyclic and finite; the budget only guarantees
    // the loop ends (and reports an error) should the structure be corrupt.
    budget = OLC_TRAVERSAL_BUDGET;
  }

  // A triangle hit at t (<= hit_t) through instance `inst`: keep it if it is
  // nearer, or equally near with a lower packed index.  Returns true when the
  // ray is finished (any hit).
  OLC_D bool offer(const SceneView& s, uint32_t inst, uint32_t slot, float t, float b1, float b2) {
    if (ANY_HIT) {
      hit_t = t;
      hit_inst = inst;
      hit_slot = slot;
      return true;
    }
    if (hit_inst == OLC_NO_INSTANCE || t < hit_t ||
        packed_index(s, inst, slot) < packed_index(s, hit_inst, hit_slot)) {
      hit_t = t;
      hit_inst = inst;
      hit_slot = slot;
      save[OLC_SAVE_UV * stride] = b1;
      save[(OLC_SAVE_UV + 1) * stride] = b2;
    }
    return false;
  }

  template <bool WAIT>
  OLC_D bool advance(const SceneView& s, int iterations, uint32_t& err) {
    // The budget is charged per call, not per iteration (a call may charge
    // more than it uses; the bound only has to end a corrupt walk).
    const uint32_t steps = min((uint32_t)iterations, budget);
    budget -= steps;
    for (uint32_t it = 0; it < steps; ++it) {
      // `node` is never the instance marker here: a marker is only popped,
      // and the pop below steps past it.
      if (WAIT) {
        // leaves wait until OLC_LEAF_LANES lanes of those walking together
        // hold one, or none of them has anything else to do
        const uint32_t group = __activemask();
        const uint32_t leaves = __ballot_sync(group, node < 0);
        if (node < 0 && leaves != group && __popc(leaves) < OLC_LEAF_LANES) {
          ++budget;   // waiting is no step of the ray; some other lane of the group takes one
          continue;
        }
      }
      int next = OLC_MARKER;   // nothing to enter: take the next node from the stack
      if (node >= 0) {
        // BVH4 node: test the four child boxes, descend into the nearest
        // hit child (closest hit) or the first (any hit) and push the others
        // in slot order: three or more of a node's boxes are hit at one node
        // in twenty, and the order of the rest changes nothing but time.
        const float4* p = reinterpret_cast<const float4*>(s.wide + node);
        const float4 nx = __ldg(p + ray.nx), fx = __ldg(p + (ray.nx ^ 1));
        const float4 ny = __ldg(p + ray.ny), fy = __ldg(p + (ray.ny ^ 1));
        const float4 nz = __ldg(p + ray.nz), fz = __ldg(p + (ray.nz ^ 1));
        const int4 ch = __ldg(reinterpret_cast<const int4*>(p + 6));
        float n0, n1, n2, n3;
        const float2 nx0 = plane2(nx.x, nx.y, ray.inv.x, ray.noinv.x), nx1 = plane2(nx.z, nx.w, ray.inv.x, ray.noinv.x);
        const float2 fx0 = plane2(fx.x, fx.y, ray.inv.x, ray.noinv.x), fx1 = plane2(fx.z, fx.w, ray.inv.x, ray.noinv.x);
        const float2 ny0 = plane2(ny.x, ny.y, ray.inv.y, ray.noinv.y), ny1 = plane2(ny.z, ny.w, ray.inv.y, ray.noinv.y);
        const float2 fy0 = plane2(fy.x, fy.y, ray.inv.y, ray.noinv.y), fy1 = plane2(fy.z, fy.w, ray.inv.y, ray.noinv.y);
        const float2 nz0 = plane2(nz.x, nz.y, ray.inv.z, ray.noinv.z), nz1 = plane2(nz.z, nz.w, ray.inv.z, ray.noinv.z);
        const float2 fz0 = plane2(fz.x, fz.y, ray.inv.z, ray.noinv.z), fz1 = plane2(fz.z, fz.w, ray.inv.z, ray.noinv.z);
        const bool h0 = slabs(nx0.x, fx0.x, ny0.x, fy0.x, nz0.x, fz0.x, t_min, hit_t, n0);
        const bool h1 = slabs(nx0.y, fx0.y, ny0.y, fy0.y, nz0.y, fz0.y, t_min, hit_t, n1);
        const bool h2 = slabs(nx1.x, fx1.x, ny1.x, fy1.x, nz1.x, fz1.x, t_min, hit_t, n2);
        const bool h3 = slabs(nx1.y, fx1.y, ny1.y, fy1.y, nz1.y, fz1.y, t_min, hit_t, n3);
        if (h0 || h1 || h2 || h3) {
          // the child entered: the nearest by a minimum over the hit ones
          // (instead of a sorting network over all four)
          bool e0 = h0, e1 = h1, e2 = h2;
          if (!ANY_HIT) {
            const float k = fminf(fminf(h0 ? n0 : CUDART_INF_F, h1 ? n1 : CUDART_INF_F),
                                  fminf(h2 ? n2 : CUDART_INF_F, h3 ? n3 : CUDART_INF_F));
            e0 = h0 && n0 == k;
            e1 = h1 && n1 == k;
            e2 = h2 && n2 == k;
          }
          next = e0 ? ch.x : e1 ? ch.y : e2 ? ch.z : ch.w;
          // the hit children but the one entered
          const bool p0 = h0 && !e0, p1 = h1 && (e0 || !e1), p2 = h2 && (e0 || e1 || !e2), p3 = h3 && (e0 || e1 || e2);
          if (st.roomy()) {
            st.push_shared(ch.w, p3);
            st.push_shared(ch.z, p2);
            st.push_shared(ch.y, p1);
            if (!ANY_HIT) st.push_shared(ch.x, p0);
          } else {
            if (p3) st.push(ch.w, err);
            if (p2) st.push(ch.z, err);
            if (p1) st.push(ch.y, err);
            if (p0) st.push(ch.x, err);
          }
        }
      } else {
        const uint32_t first = olc_leaf_first(node);
        const uint32_t kind = olc_leaf_count(node);
        const bool tlas = cur_inst == OLC_NO_INSTANCE;
        if (tlas && kind != OLC_TLAS_LEAF_TRIANGLE) {
          // instance leaf (TLAS leaves hold one instance)
          Affine w2o;
          uint32_t root;
          load_instance_w2o(s.instances, first, w2o, root);
          if (st.push(OLC_MARKER, err)) {
            setup_ray(ray, xform_point(w2o, saved3(save, stride, OLC_SAVE_ORIGIN)),
                      xform_vector(w2o, saved3(save, stride, OLC_SAVE_DIR)));
            cur_inst = first;
            next = (int)root;
          }
        } else {
          // a BLAS leaf's triangles, or one baked world-space triangle that
          // the TLAS references directly
          const uint32_t inst = tlas ? OLC_IDENTITY_INSTANCE : cur_inst;
          const uint32_t count = tlas ? 1u : kind;
          for (uint32_t k = 0; k < count; ++k) {
            const uint32_t slot = first + k;
            float t, b1, b2;
            if (intersect_triangle(ray, s.tri_verts + 3ull * slot, t_min, hit_t, t, b1, b2) &&
                offer(s, inst, slot, t, b1, b2))
              return true;
          }
        }
      }
      if (next == OLC_MARKER) {
        if (st.empty()) return true;
        next = st.pop();
        if (next == OLC_MARKER) {
          if (st.empty()) return true;   // no ray left to restore the world terms for
          cur_inst = OLC_NO_INSTANCE;
          restore_ray(save, stride, ray);
          next = st.pop();
        }
      }
      node = next;
    }
    if (budget == 0u) {
      err = 1u;
      return true;
    }
    return false;
  }
};
