// hs_stream.cuh -- one frame of one strand, streaming form.
//
// Same frame as strand_frame (hs_step.cuh), bit for bit, arranged for small
// code: the strand's state lives on chip and every pass over the strand is
// one runtime loop over its points. With one constraint iteration per
// substep (the DFTL default) a substep is a single pass in which iteration
// i loads point i+1, runs chain link i, and finishes point i-1 (push-out,
// velocity, store): only the chain link is on the loop-carried path, so the
// rest fills its latency. More iterations (reference mode: 8) run a predict
// pass then one pass per iteration.
//
// Slots: X[i] holds point i's position (reference mode) or its segment
// s_i = p_i - p_{i-1} (DFTL mode, the segment form of hs_step.cuh), V[i]
// its velocity, or within a substep its displacement D_i. The rest length
// rides in the w of one of them. Any point count up to
// HS_MAX_POINTS_PER_STRAND.
#pragma once

#include "hs_step.cuh"

namespace hs {

// Velocity slots in shared memory, [point][thread] float4, so a warp
// touches 512 contiguous bytes per access (no bank conflicts, no padding).
// The other store, in tensor memory, is VTmem (hs_tmem.cuh).
// kPrefetch: the single pass reads a velocity one point ahead of its use
// (issue, then complete), which hides the shared-memory latency.
struct VShared {
  static constexpr bool kShared = true;
  static constexpr bool kPrefetch = true;
  using Pending = float4;
  float4* p;
  int B;
  __device__ __forceinline__ float4 load(int i) const { return p[i * B]; }
  __device__ __forceinline__ void store(int i, float4 v) const { p[i * B] = v; }
  __device__ __forceinline__ void fence() const {}
  __device__ __forceinline__ Pending issue(int i) const { return p[i * B]; }
  __device__ __forceinline__ float4 complete(Pending t) const { return t; }
};

// Position (or segment) slots. XShared4: float4 [point][thread] with the
// rest length in w. XShared3: the compact form beside tensor-memory
// velocities, float2 (x, y) and float z arrays [point][thread], 12 bytes a
// point; the rest length then travels in the w of the point's velocity
// slot (kRestInV).
struct XShared4 {
  static constexpr bool kRestInV = false;
  float4* p;
  int B;
  __device__ __forceinline__ float4 load(int i) const { return p[i * B]; }
  __device__ __forceinline__ void store(int i, float4 v) const { p[i * B] = v; }
};
struct XShared3 {
  static constexpr bool kRestInV = true;
  float2* xy;
  float* z;
  int B;
  __device__ __forceinline__ float4 load(int i) const {
    const float2 a = xy[i * B];
    return make_float4(a.x, a.y, z[i * B], 0.0f);
  }
  __device__ __forceinline__ void store(int i, float4 v) const {
    xy[i * B] = make_float2(v.x, v.y);
    z[i * B] = v.z;
  }
};
// An X slot's load with its rest length in w, wherever it is kept.
template <typename XS>
__device__ __forceinline__ float4 with_rest(float4 x, float4 v) {
  if constexpr (XS::kRestInV) return make_float4(x.x, x.y, x.z, v.w);
  else return x;
}
// The rest length of point i alone.
template <typename XS, typename VS>
__device__ __forceinline__ float rest_of(const XS& X, const VS& V, int i) {
  if constexpr (XS::kRestInV) return V.load_w(i);
  else return X.load(i).w;
}
// The w a velocity slot stores: the rest length where it lives there.
template <typename XS>
__device__ __forceinline__ float vel_w(float rest) {
  if constexpr (XS::kRestInV) return rest;
  else return 0.0f;
}

// Reference mode: up to M of a strand's reachable spheres sit in registers;
// the rest are read from shared memory. kCachedSpheres is the width of the
// batched kernels' cache; the plain step also has an 8-wide one
// (strand_frame_stream). The DFTL passes have a filter (SphereFilter).
constexpr int kCachedSpheres = 4;

template <int M>
struct SphereCache {
  float cx[M], cy[M], cz[M], r[M], r2[M];
  float2 ncx[M / 2], ncy[M / 2], ncz[M / 2];  // negated centres, in pairs
  int ncached;      // spheres cached (this lane's)
  uint32_t rest;    // reachable spheres beyond the cached ones, in index order
};

template <int M>
__device__ __forceinline__ SphereCache<M> cache_spheres(const SphereSet& S, uint32_t reach) {
  SphereCache<M> C;
  C.ncached = 0;
#pragma unroll
  for (int q = 0; q < M; ++q) {
    C.cx[q] = C.cy[q] = C.cz[q] = C.r[q] = 0.0f;
    C.r2[q] = -1.0f;
    if (reach) {
      const int k = __ffs(reach) - 1;
      reach &= reach - 1u;
      const float4 c = S.c[k];
      C.cx[q] = c.x;
      C.cy[q] = c.y;
      C.cz[q] = c.z;
      C.r[q] = c.w;
      C.r2[q] = S.r2[k];
      C.ncached = q + 1;
    }
  }
  C.rest = reach;
#pragma unroll
  for (int q = 0; q < M / 2; ++q) {
    C.ncx[q] = make_float2(-C.cx[2 * q], -C.cx[2 * q + 1]);
    C.ncy[q] = make_float2(-C.cy[2 * q], -C.cy[2 * q + 1]);
    C.ncz[q] = make_float2(-C.cz[2 * q], -C.cz[2 * q + 1]);
  }
  return C;
}

// CollideSphere(+1, c, r, p) (cs_simulation.glsl:129-139) of one sphere. VEL:
// the point's velocity is reflected too (a substep's last iteration).
template <bool VEL>
__device__ __forceinline__ void push_out(V3 cc, float r, float r2, V3& p, V3& v) {
  const V3 pt = sub(p, cc);
  const float dp = dot(pt, pt);
  if (dp < r2) {
    const V3 nn = dp > 0.0f ? mul(pt, inversesqrt(dp)) : v3(0.0f, 1.0f, 0.0f);
    p = add(cc, mul(r, nn));
    if (VEL) v = reflect(v, nn);  // :137
  }
}

// Collision of one point, split so the cheap part can be scheduled with
// other work: tests() checks the cached spheres branch-free; only if one
// of them is hit (or the warp reaches spheres beyond the cache) does
// push_all() run the exact in-order push-out. With no hit the in-order
// result is the untouched point, so both paths agree.
// NC is the number of cache slots tested; unused slots have r2 = -1 and
// never hit, so NC may exceed the number of spheres cached.
template <int NC, int M>
__device__ __forceinline__ bool tests(const SphereCache<M>& C, V3 p) {
  static_assert(NC <= M, "tests reach past the cache");
  bool hit = C.rest != 0u;
  // Two spheres per packed operation: p - c as p + (-c), then the dot
  // product in the contract's order, lane by lane. The packed forms keep
  // the scalar contract's bits here because no packed product feeds a
  // packed add: the compiler fuses __fadd2_rn(a, __fmul2_rn(b, c)) into
  // one packed fma (one rounding), even with -fmad=false, which the
  // contract's separate multiply and add would not match.
  const float2 px = make_float2(p.x, p.x), py = make_float2(p.y, p.y), pz = make_float2(p.z, p.z);
#pragma unroll
  for (int q = 0; q < NC / 2; ++q) {
    const float2 dx = __fadd2_rn(px, C.ncx[q]);
    const float2 dy = __fadd2_rn(py, C.ncy[q]);
    const float2 dz = __fadd2_rn(pz, C.ncz[q]);
    const float2 d2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
    hit |= (d2.x < C.r2[2 * q]) | (d2.y < C.r2[2 * q + 1]);
  }
  return hit;
}

// The exact in-order push-out (rare), kept inline: an out-of-line call
// would take the addresses of the callers' per-lane arrays and move them
// to local memory.
template <bool VEL, int NC, int M>
__device__ __forceinline__ void push_all(const SphereCache<M>& C, const SphereSet& S, V3& p, V3& v) {
#pragma unroll
  for (int q = 0; q < M; ++q)
    if (q < C.ncached) push_out<VEL>(v3(C.cx[q], C.cy[q], C.cz[q]), C.r[q], C.r2[q], p, v);
  for (uint32_t more = C.rest; more; more &= more - 1u) {
    const int k = __ffs(more) - 1;
    const float4 c = S.c[k];
    push_out<VEL>(v3(c.x, c.y, c.z), c.w, S.r2[k], p, v);
  }
}

template <bool VEL, int NC, int M>
__device__ __forceinline__ void collide_fast(const SphereCache<M>& C, const SphereSet& S, V3& p, V3& v) {
  if (tests<NC>(C, p)) push_all<VEL, NC>(C, S, p, v);
}

// Per-strand constants of a frame.
struct StrandConsts {
  V3 F;            // force per unit mass
  V3 h2F;          // h^2 F (DFTL: the force's part of a substep's displacement)
  float h, h2, inv_h, damping, neg_damping, lscale;
};

// ---- reference mode: world coordinates (cs_simulation.glsl) -----------

// Chain link (DistanceConstraint, :109-117): point p follows `prev`.
__device__ __forceinline__ V3 link(const StrandConsts& K, V3 prev, V3 p, float rest, V3& nprev, V3& corr) {
  const V3 d = sub(p, prev);
  const float d2 = dot(d, d);
  const V3 nd = d2 > 0.0f ? mul(d, inversesqrt(d2)) : nprev;
  nprev = nd;
  const V3 pc = add(prev, mul(__fmul_rn(K.lscale, rest), nd));
  corr = sub(pc, p);
  return pc;
}

// Finishes point j after its chain link: velocity (the next point's
// correction damped, the tip its own, :116-121), push-out with reflection
// (:129-153), store.
template <int NC, typename XS, typename VS, int M>
__device__ __forceinline__ void finish_point_ref(const StrandConsts& K, const SphereCache<M>& C, const SphereSet& S,
                                                 V3 q, bool hit, V3 corr_next, float rest, bool tip, V3 corr_own,
                                                 const XS& X, const VS& V, int j) {
  V3 v = tip ? corr_own : mul(corr_next, K.damping);
  if (hit) push_all<true, NC>(C, S, q, v);
  X.store(j, f4(q, rest));
  V.store(j, f4(v, vel_w<XS>(rest)));
}

__device__ __forceinline__ V3 predict(const StrandConsts& K, float4 x, float4 v) {
  return fmas(K.h2, K.F, fmas(K.h, xyz(v), xyz(x)));  // :179-183
}

// One substep with one constraint iteration, as a single software-pipelined
// pass. The loop body predicts point i+1, runs chain link i and tests point
// i-1 against the spheres in one branch-free block (three independent
// streams of work for the scheduler), then finishes point i-1.
template <int NC, typename XS, typename VS, int M>
__device__ __forceinline__ void substep_single_pass_ref(const StrandConsts& K, const SphereCache<M>& C,
                                                        const SphereSet& S, int n, V3 p0, const XS& X, const VS& V) {
  V3 nprev = v3(0.0f, -1.0f, 0.0f);
  // Link 1.
  const float4 v1 = V.load(1);
  const float4 x1 = with_rest<XS>(X.load(1), v1);
  V3 corr_prev;
  V3 prev = link(K, p0, predict(K, x1, v1), x1.w, nprev, corr_prev);
  float rest_prev = x1.w;
  if (n >= 3) {
    const float4 v2 = V.load(2);
    float4 xc = with_rest<XS>(X.load(2), v2);
    V3 p_cur = predict(K, xc, v2);
    typename VS::Pending pend{};
    if constexpr (VS::kPrefetch) {
      if (n > 3) pend = V.issue(3);
    }
    // Unrolled by two so the carried values change registers instead of
    // being copied each iteration.
#pragma unroll 2
    for (int i = 2; i < n - 1; ++i) {
      const float4 xr = X.load(i + 1);
      float4 vn;
      if constexpr (VS::kPrefetch) {
        vn = V.complete(pend);
        if (i + 2 < n) pend = V.issue(i + 2);
      } else {
        vn = V.load(i + 1);
      }
      const float4 xn = with_rest<XS>(xr, vn);
      const V3 p_next = predict(K, xn, vn);
      V3 corr;
      const V3 pc = link(K, prev, p_cur, xc.w, nprev, corr);
      const bool hit = tests<NC>(C, prev);
      finish_point_ref<NC>(K, C, S, prev, hit, corr, rest_prev, false, corr_prev, X, V, i - 1);
      prev = pc;
      corr_prev = corr;
      rest_prev = xc.w;
      xc = xn;
      p_cur = p_next;
    }
    // Link n-1 and point n-2.
    V3 corr;
    const V3 pc = link(K, prev, p_cur, xc.w, nprev, corr);
    const bool hit = tests<NC>(C, prev);
    finish_point_ref<NC>(K, C, S, prev, hit, corr, rest_prev, false, corr_prev, X, V, n - 2);
    prev = pc;
    corr_prev = corr;
    rest_prev = xc.w;
  }
  // The tip keeps its own correction (:116).
  const bool hit = tests<NC>(C, prev);
  finish_point_ref<NC>(K, C, S, prev, hit, v3(0.0f, 0.0f, 0.0f), rest_prev, true, corr_prev, X, V, n - 1);
}

// One constraint iteration that leaves no velocities: each iteration sets
// them all, so only a substep's last one does. 60,000 strands x 16, 8
// iterations, 4 spheres: 31.2 -> 26.1 us a frame, 100,003 x 12 41.0 -> 34.7.
template <int NC, typename XS, typename VS, int M>
__device__ __forceinline__ void positions_pass_ref(const StrandConsts& K, const SphereCache<M>& C, const SphereSet& S,
                                                   int n, V3 p0, const XS& X, const VS& V) {
  V3 prev = p0, nprev = v3(0.0f, -1.0f, 0.0f), unused = p0;
  float4 next = X.load(1);
  if constexpr (XS::kRestInV) next.w = V.load_w(1);
  for (int i = 1; i < n; ++i) {
    const float4 x = next;
    if (i + 1 < n) {
      next = X.load(i + 1);
      if constexpr (XS::kRestInV) next.w = V.load_w(i + 1);
    }
    prev = link(K, prev, xyz(x), x.w, nprev, unused);
    V3 q = prev;
    collide_fast<false, NC>(C, S, q, unused);
    X.store(i, f4(q, x.w));
  }
}

// One substep with several constraint iterations (reference mode: 8): a
// predict pass, then one pass per iteration.
template <int NC, typename XS, typename VS, int M>
__device__ __forceinline__ void substep_multi_pass_ref(const StrandConsts& K, const SphereCache<M>& C,
                                                       const SphereSet& S, int n, int iterations, V3 p0, const XS& X,
                                                       const VS& V) {
  for (int i = 1; i < n; ++i) {
    const float4 vi = V.load(i);
    const float4 xi = with_rest<XS>(X.load(i), vi);
    X.store(i, f4(fmas(K.h2, K.F, fmas(K.h, xyz(vi), xyz(xi))), xi.w));
  }
  V.fence();
  for (int it = 1; it < iterations; ++it) positions_pass_ref<NC>(K, C, S, n, p0, X, V);
  V3 prev = p0;
  V3 nprev = v3(0.0f, -1.0f, 0.0f);
  V3 corr_prev = v3(0.0f, 0.0f, 0.0f);
  float rest_prev = 0.0f;
  for (int i = 1; i <= n; ++i) {
    V3 corr = v3(0.0f, 0.0f, 0.0f);
    float rest_i = 0.0f;
    V3 pc = prev;
    if (i < n) {
      float4 pi4 = X.load(i);
      if constexpr (XS::kRestInV) pi4.w = V.load(i).w;
      const V3 pi = xyz(pi4);
      rest_i = pi4.w;
      const V3 d = sub(pi, prev);
      const float d2 = dot(d, d);
      const V3 nd = d2 > 0.0f ? mul(d, inversesqrt(d2)) : nprev;
      nprev = nd;
      pc = add(prev, mul(__fmul_rn(K.lscale, rest_i), nd));
      corr = sub(pc, pi);
    }
    if (i >= 2) {
      const bool tip = i == n;
      V3 q = prev;
      V3 v = tip ? corr_prev : mul(corr, K.damping);
      collide_fast<true, NC>(C, S, q, v);
      V.store(i - 1, f4(v, vel_w<XS>(rest_prev)));
      X.store(i - 1, f4(q, rest_prev));
    }
    prev = pc;
    corr_prev = corr;
    rest_prev = rest_i;
  }
  V.fence();
}

// ---- DFTL mode: segment form (see hs_step.cuh) ---------------------------

// Within a frame the velocity slots of the DFTL passes carry u = h v (the
// frame's load scales by h, its store by 1/h: frame_velocity): a substep's
// displacement from prediction is D = u + h^2 F, and a finished point's
// slot takes fma(-damping, e, D) as it is, where v would need a multiply
// by 1/h at every point-substep.
__device__ __forceinline__ V3 disp(const StrandConsts& K, float4 u) { return add(xyz(u), K.h2F); }
__device__ __forceinline__ V3 vel_of(const StrandConsts&, V3 x) { return x; }
// A velocity slot at a frame's start (LOAD: h v) or end (u / h), where the
// slots carry u (SCALE: the DFTL passes; w kept).
template <bool SCALE, bool LOAD>
__device__ __forceinline__ float4 frame_velocity(const FrameConst& fc, float4 v) {
  if constexpr (!SCALE) {
    return v;
  } else {
    const float f = LOAD ? fc.h : fc.inv_h;
    return make_float4(__fmul_rn(f, v.x), __fmul_rn(f, v.y), __fmul_rn(f, v.z), v.w);
  }
}

// Chain link in the segment form: d is the point's offset from its leader
// (already moved), s' = (L * inversesqrt(d.d)) d, e = s' - d.
// FAST: the hardware reciprocal square root (the FAST contract).
template <bool FAST = false>
__device__ __forceinline__ void link_seg(const StrandConsts& K, V3 d, float rest, V3& sn, V3& e) {
  const float d2 = dot(d, d);
  const float sc = __fmul_rn(__fmul_rn(K.lscale, rest), FAST ? rsqrt_fast(d2) : inversesqrt(d2));
  sn = mul(sc, d);
  e = sub(sn, d);
}

// ---- spheres of the DFTL passes ------------------------------------------
//
// A point is first tested against a conservative filter, and only a flagged
// one runs the exact in-order push-out (push_seg). The filter holds, of the
// spheres the strand can reach, up to NF as (-2c, |c|^2 - r^2 - margin): a
// point p inside sphere k has dot(-2c, p) + (|c|^2 - r^2 - margin) <=
// -|p|^2. That is three fused multiply-adds a sphere, where the exact test
// takes six operations and a comparison, and its slots 2-3 and 4-7 are
// skipped by warps whose strands reach no more than two or four spheres
// (two thirds of the 64-groom workload's warps reach at most two). More than
// NF spheres: the last slot is a ball around the rest, which flags points it
// need not. Measured against exact tests of four cached spheres, which sent
// every point of a strand with more to the push-out, and the set-up below
// done with IEEE divisions and square roots in two loops over the spheres:
// 64-groom frame 938 -> 773 us, 262,144 x 32 groom 284 -> 242 us (EXACT),
// 251 -> 218 us (FAST).
//
// The margin. With u = 2^-24, the exact test dot(p - c, p - c) < fl(r^2)
// in FP32 implies |p - c|^2 < r^2 (1 + 8u); the rounding of the filter's
// sums (three terms each) is below 9u ((|p| + |c|)^2 + r^2): together less
// than 17u = 1.02e-6 times that, and the margin is 1.25e-6 times it (at
// 4e-6 the points resting near a surface were flagged, and more warps took
// the push-out). |p| is bounded by the ball the strand stays in during the
// frame (near_spheres, its margins included).
template <int NF>
struct SphereFilter {
  float cx[NF], cy[NF], cz[NF], k[NF];
  uint32_t reach;  // the strand's reachable spheres
  bool many;       // a strand of the warp reaches more than two
  bool most;       // more than four
};

// Square root to a few ulp, for distances that are compared with a margin
// of 1e-3.
__device__ __forceinline__ float sqrt_near(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The ball a strand stays in during the frame: the root's path about its
// midpoint, and the links' total length R beyond it.
struct StrandBall {
  V3 mid;
  float half_path, radius;
  __device__ __forceinline__ StrandBall(V3 x0, V3 target, float R) {
    const float dx = target.x - x0.x, dy = target.y - x0.y, dz = target.z - x0.z;
    mid = v3(0.5f * (x0.x + target.x), 0.5f * (x0.y + target.y), 0.5f * (x0.z + target.z));
    half_path = 0.5f * sqrt_near(dx * dx + dy * dy + dz * dz);
    radius = R + half_path;
  }
  // The largest |p| of a point in it, with near_spheres' margins.
  __device__ __forceinline__ float far() const {
    return (sqrt_near(mid.x * mid.x + mid.y * mid.y + mid.z * mid.z) + radius) * 1.002f + 1.0e-3f;
  }
};

// near_spheres (hs_step.cuh) of one strand, and the smallest summed link
// length at which a point of it may touch a sphere: the distance from `mid`
// to the sphere's surface less the root's half path, with the same margins.
// A point whose links from the root sum to less cannot be inside any sphere
// this frame.
struct SphereReach {
  uint32_t near;
  float threshold;
};
__device__ __forceinline__ SphereReach sphere_reach(const SphereSet& S, const StrandBall& b) {
  const float mag = fmaxf(fmaxf(fabsf(b.mid.x), fabsf(b.mid.y)), fmaxf(fabsf(b.mid.z), b.radius)) + 1.0f;
  const float slack = mag * 1.0e-4f;
  SphereReach o{0u, 3.0e38f};
#pragma unroll 2
  for (int k = 0; k < S.n; ++k) {
    const float4 c = S.c[k];
    const float dx = c.x - b.mid.x, dy = c.y - b.mid.y, dz = c.z - b.mid.z;
    const float d2 = dx * dx + dy * dy + dz * dz;
    const float reach = (c.w + b.radius) * 1.001f + slack;
    if (d2 < reach * reach) o.near |= 1u << k;
    o.threshold = fminf(o.threshold, (sqrt_near(d2) - slack) * 0.999f - c.w - b.half_path);
  }
  return o;
}

// far: the largest |p| of the strand's points during the frame. Every lane
// of the warp calls it. Slots that no strand of the warp fills are left out
// (flagged does not read them).
template <int NF>
__device__ __forceinline__ SphereFilter<NF> filter_spheres(const SphereSet& S, uint32_t reach, float far) {
  SphereFilter<NF> F;
  F.reach = reach;
  F.many = __any_sync(0xffffffffu, __popc(reach) > 2);
  F.most = NF > 4 && __any_sync(0xffffffffu, __popc(reach) > 4);
#pragma unroll
  for (int q = 0; q < NF; ++q) {
    float cx = 0.0f, cy = 0.0f, cz = 0.0f, kk = __int_as_float(0x7f800000);  // no sphere: never flagged
    if ((q < 2 || (q < 4 ? F.many : F.most)) && reach) {
      const int i = __ffs(reach) - 1;
      const uint32_t more = reach & (reach - 1u);
      const float4 c = S.c[i];
      cx = c.x;
      cy = c.y;
      cz = c.z;
      float r2 = S.r2[i];
      if (q == NF - 1 && more) {
        // A ball around the remaining spheres, centred about their mean.
        float cnt = 1.0f;
        for (uint32_t m = more; m; m &= m - 1u) {
          const float4 d = S.c[__ffs(m) - 1];
          cx += d.x;
          cy += d.y;
          cz += d.z;
          cnt += 1.0f;
        }
        cnt = __fdividef(1.0f, cnt);
        cx *= cnt;
        cy *= cnt;
        cz *= cnt;
        float rr = 0.0f;
        for (uint32_t m = reach; m; m &= m - 1u) {
          const float4 d = S.c[__ffs(m) - 1];
          const float dx = d.x - cx, dy = d.y - cy, dz = d.z - cz;
          rr = fmaxf(rr, sqrt_near(dx * dx + dy * dy + dz * dz) + d.w);
        }
        rr = rr * 1.0001f + 1.0e-5f * (fabsf(cx) + fabsf(cy) + fabsf(cz));
        r2 = rr * rr;
      }
      reach = more;
      const float c2 = cx * cx + cy * cy + cz * cz;
      const float big = far + sqrt_near(c2) * 1.0001f;
      const float size = big * big + r2;
      // Coordinates too large for the sums: every point is flagged.
      kk = size < 1.0e30f ? (c2 - r2) - (1.25e-6f * size + 1.0e-30f) : __int_as_float(0xff800000);
    }
    F.cx[q] = -2.0f * cx;
    F.cy[q] = -2.0f * cy;
    F.cz[q] = -2.0f * cz;
    F.k[q] = kk;
  }
  return F;
}

template <int NF>
__device__ __forceinline__ float filter_value(const SphereFilter<NF>& F, int q, V3 w) {
  return __fmaf_rn(F.cx[q], w.x, __fmaf_rn(F.cy[q], w.y, __fmaf_rn(F.cz[q], w.z, F.k[q])));
}

// Whether a point may be inside a sphere. (Overflow: an infinite |p|^2 flags
// nothing a finite slot did not, and such a point is in no sphere.)
template <int NF>
__device__ __forceinline__ bool flagged(const SphereFilter<NF>& F, V3 w) {
  float m = fminf(filter_value(F, 0, w), filter_value(F, 1, w));
  if (F.many) {
#pragma unroll
    for (int q = 2; q < 4; ++q) m = fminf(m, filter_value(F, q, w));
    if (NF > 4 && F.most) {
#pragma unroll
      for (int q = 4; q < NF; ++q) m = fminf(m, filter_value(F, q, w));
    }
  }
  return m <= -dot(w, w);
}

// Spheres of a groom up to which its strands reach few of them, and the
// push-out goes through all of those (measured at 7 and 16: push_seg).
constexpr int kFewSpheres = 8;

// The exact in-order push-out (push_out) of point j at its chain position w,
// against the strand's reachable spheres in index order, read from shared
// memory. A push by g moves D_j and s_j by +g and the next segment by -g
// (none at the tip).
//
// A strand in contact waits for this path at every point-substep, so it has
// no branch around the push: with one, a frame of 50,021 x 23 strands among
// 7 spheres takes 50.6 instead of 49.6 us. PICK, for grooms among many
// spheres: warps whose strands reach more than two go through the spheres
// the point is flagged for alone, and after a push also through the later
// ones that overlap the pushing sphere (the point, on its surface, can be in
// no other). 262,144 x 32 strands among 16 spheres: 241 -> 231 us a frame
// (EXACT), 215 -> 211 us (FAST); the code is larger, which costs the
// batched kernel more than it saves (64 grooms: 782 -> 824 us) and grooms
// among few spheres (the 7 above: 49.6 -> 52.1 us). BRANCH: past the spheres
// that the point is not inside, where it goes through many.
template <bool PICK, bool FAST, bool BRANCH = false, int NF>
__device__ __forceinline__ void push_seg(const SphereFilter<NF>& F, const SphereSet& S, V3 w, V3& D, V3& s, V3& s_next,
                                         bool tip) {
  uint32_t todo = F.reach;
  if (PICK && F.many) {
    const float w2 = dot(w, w);
    uint32_t left = F.reach;
    todo = 0u;
#pragma unroll
    for (int q = 0; q < NF; ++q) {
      if (q < 4 || F.most) {
        const uint32_t low = q == NF - 1 ? left : left & (0u - left);
        if (filter_value(F, q, w) <= -w2) todo |= low;
        left ^= low;
      }
    }
  }
  V3 p = w;
  bool pushed = false;
  while (todo) {
    const int k = __ffs(todo) - 1;
    todo &= todo - 1u;
    const float4 c = S.c[k];
    const V3 cc = v3(c.x, c.y, c.z);
    const V3 d = sub(p, cc);
    const float d2 = dot(d, d);
    const bool hit = d2 < S.r2[k];
    if (BRANCH && !hit) continue;
    const V3 u = mul(d, FAST ? rsqrt_fast(d2) : inversesqrt(d2));
    const bool off = d2 > 0.0f;  // not at the centre
    const V3 q = add(cc, mul(c.w, v3(off ? u.x : 0.0f, off ? u.y : 1.0f, off ? u.z : 0.0f)));
    p = v3(hit ? q.x : p.x, hit ? q.y : p.y, hit ? q.z : p.z);
    pushed |= hit;
    if (PICK) todo |= hit ? S.adj[k] & F.reach & (0xfffffffeu << k) : 0u;
  }
  if (pushed) {
    const V3 g = sub(p, w);
    D = add(D, g);
    s = add(s, g);
    if (!tip) s_next = sub(s_next, g);
  }
}

// Iteration i of the single pass (2 <= i <= n - 2): uses point i's loads
// (a_cur = s_i + D_i, dp_cur, rest_cur), loads point i + 1, runs link i,
// finishes point i - 1, testing it against the spheres if TEST and
// i - 1 >= jmin.
template <bool TEST, bool PICK, bool FAST, typename XS, typename VS, int NF>
struct SegPass {
  const StrandConsts& K;
  const SphereFilter<NF>& F;
  const SphereSet& S;
  const XS& X;
  const VS& V;
  int n, jmin;
  V3 D_prev, w_prev, s_prev, a_cur, dp_cur;
  float rest_prev, rest_cur;
  typename VS::Pending pend;
  __device__ __forceinline__ void step(int i) {
    const float4 xr = X.load(i + 1);
    float4 vn;
    if constexpr (VS::kPrefetch) {
      vn = V.complete(pend);
      if (i + 2 < n) pend = V.issue(i + 2);
    }
    else vn = V.load(i + 1);
    V3 sn, e;
    link_seg<FAST>(K, sub(a_cur, D_prev), rest_cur, sn, e);
    const V3 D_i = add(dp_cur, e);
    const V3 w_i = add(w_prev, sn);
    if (TEST && i - 1 >= jmin && flagged(F, w_prev)) push_seg<PICK, FAST>(F, S, w_prev, D_prev, s_prev, sn, false);
    const float4 xn = with_rest<XS>(xr, vn);
    const V3 dp_next = disp(K, vn);
    const V3 a_next = add(xyz(xn), dp_next);
    X.store(i - 1, f4(s_prev, rest_prev));
    V.store(i - 1, f4(vel_of(K, fmas(K.neg_damping, e, D_prev)), vel_w<XS>(rest_prev)));
    s_prev = sn;
    D_prev = D_i;
    w_prev = w_i;
    rest_prev = rest_cur;
    a_cur = a_next;
    dp_cur = dp_next;
    rest_cur = xn.w;
  }
};

// One substep with one constraint iteration, one pass. Iteration i loads
// point i+1 (its segment plus displacement, independent of the chain),
// runs link i (d = (s_i + D_i) - D_{i-1}, the loop-carried path), and
// finishes point i-1: tests at its chain position, push-out, Eq. 9
// velocity v = fma(-damping, e_i, D_{i-1}) / h, stores. Points below jmin
// cannot reach a sphere this frame (strand_frame_stream) and skip the
// tests. Measured code shapes (the hot loop must stay in the instruction
// cache): SPLIT, a loop without tests up to jmin then one with them, else
// one loop with the jmin check.
template <bool SPLIT, bool PICK, bool FAST, typename XS, typename VS, int NF>
__device__ __forceinline__ void substep_single_pass_seg(const StrandConsts& K, const SphereFilter<NF>& F,
                                                        const SphereSet& S, int n, int jmin, V3 D0, V3 R,
                                                        const XS& X, const VS& V) {
  constexpr bool kSplit = SPLIT;
  // Link 1.
  const float4 v1 = V.load(1);
  const float4 x1 = with_rest<XS>(X.load(1), v1);
  const V3 dp1 = disp(K, v1);
  V3 sn, e;
  link_seg<FAST>(K, sub(add(xyz(x1), dp1), D0), x1.w, sn, e);
  V3 D_prev = add(dp1, e);
  V3 w_prev = add(R, sn);
  V3 s_prev = sn;
  float rest_prev = x1.w;
  if (n >= 3) {
    const float4 v2 = V.load(2);
    const float4 x2 = with_rest<XS>(X.load(2), v2);
    const V3 dp2 = disp(K, v2);
    SegPass<!kSplit, PICK, FAST, XS, VS, NF> A{K,      F,      S,      X,      V,   n, jmin, D_prev, w_prev, s_prev, add(xyz(x2), dp2),
                                     dp2, rest_prev, x2.w, {}};
    if constexpr (VS::kPrefetch) {
      if (n > 3) A.pend = V.issue(3);
    }
    int i = 2;
    if constexpr (kSplit) {
      // Iterations finishing points below jmin: no tests.
      const int ia = min(max(jmin + 1, 2), n - 1);
      // Unrolled by two so the carried values change registers instead of
      // being copied each iteration.
#pragma unroll 2
      for (; i < ia; ++i) A.step(i);
    }
    SegPass<true, PICK, FAST, XS, VS, NF> B{K,        F,        S,           X,          V,     n, jmin, A.D_prev, A.w_prev, A.s_prev,
                                  A.a_cur, A.dp_cur, A.rest_prev, A.rest_cur, A.pend};
#pragma unroll 2
    for (; i < n - 1; ++i) B.step(i);
    // Link n-1 and point n-2.
    link_seg<FAST>(K, sub(B.a_cur, B.D_prev), B.rest_cur, sn, e);
    const V3 D_i = add(B.dp_cur, e);
    const V3 w_i = add(B.w_prev, sn);
    D_prev = B.D_prev;
    s_prev = B.s_prev;
    if (n - 2 >= jmin && flagged(F, B.w_prev)) push_seg<PICK, FAST>(F, S, B.w_prev, D_prev, s_prev, sn, false);
    X.store(n - 2, f4(s_prev, B.rest_prev));
    V.store(n - 2, f4(vel_of(K, fmas(K.neg_damping, e, D_prev)), vel_w<XS>(B.rest_prev)));
    s_prev = sn;
    D_prev = D_i;
    w_prev = w_i;
    rest_prev = B.rest_cur;
  }
  // The tip: no next correction, v = D / h.
  if (n - 1 >= jmin && flagged(F, w_prev)) push_seg<PICK, FAST>(F, S, w_prev, D_prev, s_prev, sn, true);
  X.store(n - 1, f4(s_prev, rest_prev));
  V.store(n - 1, f4(vel_of(K, D_prev), vel_w<XS>(rest_prev)));
}

// One substep with several constraint iterations: a predict pass (the
// velocity slots take D_i), then one pass per iteration. The first
// iteration's link is d = (s_i + D_i) - D_{i-1} (as in the single pass),
// later ones d = s_i - e_{i-1} (e: that iteration's correction of the
// leader); the last pass forms the velocities.
template <bool PICK, bool FAST, typename XS, typename VS, int NF>
__device__ __forceinline__ void substep_multi_pass_seg(const StrandConsts& K, const SphereFilter<NF>& F,
                                                       const SphereSet& S, int n, int jmin, int iterations, V3 D0,
                                                       V3 R, const XS& X, const VS& V) {
  for (int i = 1; i < n; ++i) {
    const float4 v = V.load(i);
    V.store(i, f4(disp(K, v), v.w));
  }
  V.fence();
  const V3 zero = v3(0.0f, 0.0f, 0.0f);
  for (int it = 0; it < iterations; ++it) {
    const bool last = it + 1 == iterations;
    V3 D_prev = D0, e_prev = zero, w_prev = R, s_prev = zero;
    float rest_prev = 0.0f;
    for (int i = 1; i <= n; ++i) {
      V3 sn = zero, e = zero, D_i = zero, w_i = zero;
      float rest_i = 0.0f;
      if (i < n) {
        const float4 vd = V.load(i);
        const float4 x = with_rest<XS>(X.load(i), vd);
        rest_i = x.w;
        const V3 d = it == 0 ? sub(add(xyz(x), xyz(vd)), D_prev) : sub(xyz(x), e_prev);
        link_seg<FAST>(K, d, rest_i, sn, e);
        D_i = add(xyz(vd), e);
        w_i = add(w_prev, sn);
      }
      if (i >= 2) {
        const bool tip = i == n;
        V3 Dj = D_prev, sj = s_prev;
        if (i - 1 >= jmin && flagged(F, w_prev)) push_seg<PICK, FAST>(F, S, w_prev, Dj, sj, sn, tip);
        const V3 out = last ? vel_of(K, tip ? Dj : fmas(K.neg_damping, e, Dj)) : Dj;
        X.store(i - 1, f4(sj, rest_prev));
        V.store(i - 1, f4(out, vel_w<XS>(rest_prev)));
      }
      D_prev = D_i;
      e_prev = e;
      w_prev = w_i;
      s_prev = sn;
      rest_prev = rest_i;
    }
    V.fence();
  }
}

// The root over a frame: pinned, or linear from x0 to its target.
struct RootPath {
  V3 x0, target;
  int substeps;
  bool moving;
  // Offset from the frame's start at the end of substep k: rel_k = alpha_k
  // delta, delta itself at the last substep.
  __device__ __forceinline__ V3 rel(int k) const {
    if (!moving || k < 0) return v3(0.0f, 0.0f, 0.0f);
    const V3 delta = sub(target, x0);
    if (k + 1 == substeps) return delta;
    return mul(__fdiv_rn(static_cast<float>(k + 1), static_cast<float>(substeps)), delta);
  }
  // Position at the end of substep k (rel: rel(k)).
  __device__ __forceinline__ V3 at(int k, V3 rel) const {
    if (!moving) return x0;
    return k + 1 == substeps ? target : add(x0, rel);
  }
};

// ---- several substeps at once --------------------------------------------

// Two-wide form of a strand's sphere filter.
template <int NF>
struct SphereFilter2 {
  F2 cx[NF], cy[NF], cz[NF], k[NF];
  uint32_t reach;
  bool many, most;
  explicit __device__ __forceinline__ SphereFilter2(const SphereFilter<NF>& F)
      : reach(F.reach), many(F.many), most(F.most) {
#pragma unroll
    for (int q = 0; q < NF; ++q) {
      cx[q] = f2(F.cx[q], F.cx[q]);
      cy[q] = f2(F.cy[q], F.cy[q]);
      cz[q] = f2(F.cz[q], F.cz[q]);
      k[q] = f2(F.k[q], F.k[q]);
    }
  }
  __device__ __forceinline__ F2 value(int q, V3x2 w) const {
    return fma2(cx[q], w.x, fma2(cy[q], w.y, fma2(cz[q], w.z, k[q])));
  }
  // Whether one of the two points may be inside a sphere.
  __device__ __forceinline__ bool flagged(V3x2 w) const {
    const F2 w2 = dot2(w, w);
    F2 v = value(0, w), u = value(1, w);
    float ma = fminf(lo(v), lo(u)), mb = fminf(hi(v), hi(u));
    if (many) {
#pragma unroll
      for (int q = 2; q < 4; ++q) {
        v = value(q, w);
        ma = fminf(ma, lo(v));
        mb = fminf(mb, hi(v));
      }
      if (NF > 4 && most) {
#pragma unroll
        for (int q = 4; q < NF; ++q) {
          v = value(q, w);
          ma = fminf(ma, lo(v));
          mb = fminf(mb, hi(v));
        }
      }
    }
    return ma <= -lo(w2) || mb <= -hi(w2);
  }
};

// Points a strand needs for W substeps at once: the first stage's loads of a
// sweep stay behind the last one's stores of the one before.
template <int W>
constexpr int kWaveMinPoints = 4 * W;

// Two stages of the pipeline as the halves of pairs (the earlier substep in
// the low halves): the point to link next (its segment plus displacement a,
// displacement d, rest length) and the one linked last (displacement D,
// chain position w, segment s, rest length).
struct WaveStages {
  V3x2 a, d, D, w, s;
  float next_a, next_b, last_a, last_b;
};
struct WaveLinked {
  V3x2 s, e, D, w;
};

// Substeps k0 + W r .. k0 + W r + W - 1, r = 0 .. sweeps - 1 (W = 2 P), each
// W of them one sweep over the points, as the stages of a pipeline: stage k
// takes the points stage k - 1 has finished from registers, so the slots are
// read and written once every W substeps, and two stages are the halves of
// two-wide FP32 instructions (F2). The arithmetic of a point and substep is
// SegPass::step's, operation for operation.
//
// It is for strands whose warps wait on their chain links: where a warp or
// two a scheduler run (33 to 64 points, tensor memory's limit), or less
// than a wave of warps. The steps between sweeps and the moves between the
// halves cost what the shared loads and stores save in instructions, so
// that with 16 busy warps an SM the single pass is faster (64 grooms: 1,150
// against 880 us).
//
// Step i of a sweep links point i - 2k
// in stage k and finishes point i - 2k - 1. The sweeps follow each other
// without a gap: while the last stages end a sweep, the first ones are at
// the first points of the next. The 2 W + 1 steps where a stage starts or
// ends run in `edge` (t = i - (n - 1), which are i = 0, 1, .. of the next
// sweep), the others in `step`. Slot 0 holds the root meanwhile (X: where it
// starts, V: its target).
template <int P, bool FAST, typename XS, typename VS, int NF>
struct WavePass {
  static constexpr int W = 2 * P;
  const StrandConsts& K;
  const FrameConst& fc;
  const SphereFilter2<NF>& F;
  const SphereSet& S;
  const XS& X;
  const VS& V;
  int n, jmin, k0;
  F2 neg0;
  WaveStages st[P];

  __device__ __forceinline__ WaveLinked link(const WaveStages& q) const {
    WaveLinked l;
    const V3x2 d = sub2(q.a, q.D);
    const F2 d2 = dot2(d, d);
    const F2 rs = FAST ? rsqrt_fast2(d2) : inversesqrt2(d2);
    const F2 sc = f2(__fmul_rn(__fmul_rn(K.lscale, q.next_a), lo(rs)), __fmul_rn(__fmul_rn(K.lscale, q.next_b), hi(rs)));
    l.s = mul2_kept(sc, d, neg0);
    l.e = sub2(l.s, d);
    l.D = add2(q.d, l.e);
    l.w = add2(q.w, l.s);
    return l;
  }
  // The in-order push-out (push_seg) of both stages' points linked last.
  // `ta`, `tb`: whether the stage's point is tested.
  __device__ __forceinline__ void push(bool ta, bool tb, WaveStages& st, V3x2& s_next) const {
    V3x2 p = st.w;
    bool pa = false, pb = false;
    for (uint32_t m = F.reach; m; m &= m - 1u) {
      const int k = __ffs(m) - 1;
      const float4 c = S.c[k];
      const float r2 = S.r2[k];
      const V3x2 cc = V3x2{f2(c.x, c.x), f2(c.y, c.y), f2(c.z, c.z)};
      const V3x2 d = sub2(p, cc);
      const F2 dp = dot2(d, d);
      const bool ha = ta && lo(dp) < r2, hb = tb && hi(dp) < r2;
      if (ha || hb) {
        const V3x2 u = mul2_kept(FAST ? rsqrt_fast2(dp) : inversesqrt2(dp), d, neg0);
        const bool oa = lo(dp) > 0.0f, ob = hi(dp) > 0.0f;  // not at the centre
        const V3x2 nn = V3x2{f2(oa ? lo(u.x) : 0.0f, ob ? hi(u.x) : 0.0f), f2(oa ? lo(u.y) : 1.0f, ob ? hi(u.y) : 1.0f),
                             f2(oa ? lo(u.z) : 0.0f, ob ? hi(u.z) : 0.0f)};
        const V3x2 q = add2(cc, mul2_kept(f2(c.w, c.w), nn, neg0));
        p = V3x2{f2(ha ? lo(q.x) : lo(p.x), hb ? hi(q.x) : hi(p.x)), f2(ha ? lo(q.y) : lo(p.y), hb ? hi(q.y) : hi(p.y)),
                 f2(ha ? lo(q.z) : lo(p.z), hb ? hi(q.z) : hi(p.z))};
        pa |= ha;
        pb |= hb;
      }
    }
    if (pa | pb) {
      const V3x2 g = sub2(p, st.w);
      shift(pa, pb, g.x, st.D.x, st.s.x, s_next.x);
      shift(pa, pb, g.y, st.D.y, st.s.y, s_next.y);
      shift(pa, pb, g.z, st.D.z, st.s.z, s_next.z);
    }
  }
  // A push by g: D and s by +g, the next segment by -g (at the tip there is
  // none, and s_next is not used).
  static __device__ __forceinline__ void shift(bool pa, bool pb, F2 g, F2& D, F2& s, F2& s_next) {
    const F2 Dn = add2(D, g), sn = add2(s, g), nn = sub2(s_next, g);
    D = f2(pa ? lo(Dn) : lo(D), pb ? hi(Dn) : hi(D));
    s = f2(pa ? lo(sn) : lo(s), pb ? hi(sn) : hi(s));
    s_next = f2(pa ? lo(nn) : lo(s_next), pb ? hi(nn) : hi(s_next));
  }
  __device__ __forceinline__ void store(int i, V3 s, V3 u, float rest) const {
    X.store(i, f4(s, rest));
    V.store(i, f4(u, vel_w<XS>(rest)));
  }
  // The velocity slot of a finished point: fma(-damping, e, D).
  __device__ __forceinline__ V3 carry(V3 e, V3 D) const {
    return V3{__fmaf_rn(K.neg_damping, e.x, D.x), __fmaf_rn(K.neg_damping, e.y, D.y),
              __fmaf_rn(K.neg_damping, e.z, D.z)};
  }
  // One component of the points to link next: the pair's first stage takes
  // (segment xs, u = vs), its second what the first finished (s, ua).
  static __device__ __forceinline__ void next(F2& a, F2& d, float xs, float vs, float s, float ua, float f) {
    const float da = __fadd_rn(vs, f), db = __fadd_rn(ua, f);
    d = f2(da, db);
    a = f2(__fadd_rn(xs, da), __fadd_rn(s, db));
  }
  __device__ __forceinline__ void advance(WaveStages& q, const WaveLinked& l, V3 x, V3 u, float rest, V3 ua) const {
    next(q.a.x, q.d.x, x.x, u.x, lo(q.s.x), ua.x, K.h2F.x);
    next(q.a.y, q.d.y, x.y, u.y, lo(q.s.y), ua.y, K.h2F.y);
    next(q.a.z, q.d.z, x.z, u.z, lo(q.s.z), ua.z, K.h2F.z);
    q.last_b = q.next_b;
    q.next_b = q.last_a;
    q.last_a = q.next_a;
    q.next_a = rest;
    q.s = l.s;
    q.D = l.D;
    q.w = l.w;
  }
  // Step i, 2 W <= i <= n - 2.
  __device__ __forceinline__ void step(int i) {
    const float4 vn = V.load(i + 1);
    const float4 xn = with_rest<XS>(X.load(i + 1), vn);
    WaveLinked l[P];
#pragma unroll
    for (int q = 0; q < P; ++q) l[q] = link(st[q]);
    if (i - 1 >= jmin) {
#pragma unroll
      for (int q = 0; q < P; ++q)
        if (F.flagged(st[q].w)) push(true, true, st[q], l[q].s);
    }
    store(i - (2 * W - 1), hi(st[P - 1].s), carry(hi(l[P - 1].e), hi(st[P - 1].D)), st[P - 1].last_b);
#pragma unroll
    for (int q = P - 1; q >= 0; --q) {
      const V3 ua = carry(lo(l[q].e), lo(st[q].D));
      if (q == 0) {
        advance(st[0], l[0], xyz(xn), xyz(vn), xn.w, ua);
      } else {
        const WaveStages& o = st[q > 0 ? q - 1 : 0];
        advance(st[q], l[q], hi(o.s), carry(hi(l[q > 0 ? q - 1 : 0].e), hi(o.D)), o.last_b, ua);
      }
    }
  }
  // Whether stage k tests the point it finishes in step t, and finishes one.
  __device__ __forceinline__ bool tested(int tk, bool more, bool before) const {
    return tk < 2 ? before && n - 2 + tk >= jmin : more && tk > 2 && tk - 2 >= jmin;
  }
  // Step t of the 2 W + 1 between sweeps r - 1 and r: stage k finishes its
  // tip at t = 2 k + 1 and starts at t = 2 k + 2.
  __device__ __forceinline__ void edge(int t, int r, int sweeps) {
    const bool more = r < sweeps, before = r > 0;
    if (t == 1) V.fence();  // points up to n - 2 W of sweep r - 1
    float4 vn = make_float4(0.0f, 0.0f, 0.0f, 0.0f), xn = vn;
    if (t >= 1 && more) {
      vn = V.load(t);
      xn = with_rest<XS>(X.load(t), vn);
    }
    if (more && t >= 2 && t % 2 == 0) {  // a stage starts: its leader is the root
      const RootPath path{xyz(X.load(0)), xyz(V.load(0)), fc.substeps, fc.root_mode != HS_ROOT_PINNED};
      const int ks = t / 2 - 1, k = k0 + W * r + ks;
      const V3 rel = path.rel(k), D0 = sub(rel, path.rel(k - 1)), R = path.at(k, rel);
#pragma unroll
      for (int q = 0; q < P; ++q) {
        if (ks == 2 * q) {
          st[q].D = v3x2(D0, hi(st[q].D));
          st[q].w = v3x2(R, hi(st[q].w));
        }
        if (ks == 2 * q + 1) {
          st[q].D = v3x2(lo(st[q].D), D0);
          st[q].w = v3x2(lo(st[q].w), R);
        }
      }
    }
    WaveLinked l[P];
    V3 ua[P], ub[P];
#pragma unroll
    for (int q = 0; q < P; ++q) {
      l[q] = link(st[q]);
      const int ta = t - 4 * q, tb = ta - 2;  // the two stages' own steps
      const bool testa = tested(ta, more, before), testb = tested(tb, more, before);
      if ((testa || testb) && F.flagged(st[q].w)) push(testa, testb, st[q], l[q].s);
      ua[q] = ta == 1 ? lo(st[q].D) : carry(lo(l[q].e), lo(st[q].D));  // a tip has no next correction
      ub[q] = tb == 1 ? hi(st[q].D) : carry(hi(l[q].e), hi(st[q].D));
    }
    if (before && t < 2 * W) store(n - 2 * W + t, hi(st[P - 1].s), ub[P - 1], st[P - 1].last_b);
#pragma unroll
    for (int q = P - 1; q >= 0; --q) {
      if (q == 0) {
        advance(st[0], l[0], xyz(xn), xyz(vn), xn.w, ua[0]);
      } else {
        const WaveStages& o = st[q > 0 ? q - 1 : 0];
        advance(st[q], l[q], hi(o.s), ub[q > 0 ? q - 1 : 0], o.last_b, ua[q]);
      }
    }
    if (t == 2 * W) V.fence();  // the last points of sweep r - 1
  }
  __device__ __forceinline__ void run(int sweeps) {
    const F2 z = f2(0.0f, 0.0f);
    const V3x2 z3{z, z, z};
#pragma unroll
    for (int q = 0; q < P; ++q) st[q] = WaveStages{z3, z3, z3, z3, z3, 0.0f, 0.0f, 0.0f, 0.0f};
    for (int r = 0; r <= sweeps; ++r) {
      const int last = r < sweeps ? 2 * W : 2 * W - 1;
#pragma unroll 1
      for (int t = r == 0 ? 1 : 0; t <= last; ++t) edge(t, r, sweeps);
      if (r < sweeps) {
#pragma unroll 2
        for (int i = 2 * W; i < n - 1; ++i) step(i);
      }
    }
    V.fence();
  }
};

// Substeps 0 .. k - 1 in sweeps of 2 P, then of 2; returns k. The others
// (an odd last one, short strands) go one at a time (substeps_seg).
template <int P, bool FAST, typename XS, typename VS, int NF>
__device__ __forceinline__ int wave_substeps(const FrameConst& fc, const StrandConsts& K, const SphereFilter<NF>& F1,
                                             const SphereSet& S, int n, int jmin, int pairs, const XS& X, const VS& V) {
  const SphereFilter2<NF> F(F1);
  int k = 0;
  if (P > 1 && pairs >= P && n >= kWaveMinPoints<2 * P> && fc.substeps >= 2 * P) {
    WavePass<P, FAST, XS, VS, NF> pass{K, fc, F, S, X, V, n, jmin, 0, negative_zero()};
    pass.run(fc.substeps / (2 * P));
    k = fc.substeps / (2 * P) * (2 * P);
  }
  if (n >= kWaveMinPoints<2> && fc.substeps - k >= 2) {
    WavePass<1, FAST, XS, VS, NF> pass{K, fc, F, S, X, V, n, jmin, k, negative_zero()};
    pass.run((fc.substeps - k) / 2);
    k += (fc.substeps - k) / 2 * 2;
  }
  return k;
}

// ---- the frame ------------------------------------------------------------

// Per-strand constants of a frame: force per unit mass, gravity
// (CalculateForces, :70-77) plus the wind with its per-strand jitter. The
// jitter hashes the caller's strand index (the library stores strands in
// its own order).
__device__ __forceinline__ StrandConsts strand_consts(const FrameConst& fc, const GroomView& g, uint32_t s,
                                                      bool active) {
  StrandConsts K;
  const float u = hash_u01(fc.wind_key, g.strand_base + (active ? g.order[s] : s));
  const float j = __fadd_rn(1.0f, __fmul_rn(fc.wind_jitter, __fsub_rn(1.0f, __fmul_rn(2.0f, u))));
  K.F = v3(__fmaf_rn(j, fc.wx, fc.Gx), __fmaf_rn(j, fc.wy, fc.Gy), __fmaf_rn(j, fc.wz, fc.Gz));
  K.h = fc.h;
  K.h2 = fc.h2;
  K.h2F = mul(fc.h2, K.F);
  K.inv_h = fc.inv_h;
  K.damping = fc.damping;
  K.neg_damping = -fc.damping;
  K.lscale = fc.length_scale;
  return K;
}

// The root's position at the end of the frame: the rest root moved by the
// groom's transform (RIGID) or skinned by its bones (SKINNED), the
// caller's target (EXPLICIT), else where it starts.
__device__ __forceinline__ V3 root_target(const FrameConst& fc, const GroomView& g, uint32_t s, bool active,
                                          V3 x0_start) {
  V3 target = x0_start;
  if (active) {
    if (fc.root_mode == HS_ROOT_RIGID) {
      const float4 r = g.root_rest[s];
      target = v3(__fmaf_rn(fc.m[8], r.z, __fmaf_rn(fc.m[4], r.y, __fmaf_rn(fc.m[0], r.x, fc.m[12]))),
                  __fmaf_rn(fc.m[9], r.z, __fmaf_rn(fc.m[5], r.y, __fmaf_rn(fc.m[1], r.x, fc.m[13]))),
                  __fmaf_rn(fc.m[10], r.z, __fmaf_rn(fc.m[6], r.y, __fmaf_rn(fc.m[2], r.x, fc.m[14]))));
    } else if (fc.root_mode == HS_ROOT_EXPLICIT) {
      const float4 t = g.root_target[s];
      target = v3(t.x, t.y, t.z);
    } else if (fc.root_mode == HS_ROOT_SKINNED) {
      const float4 r = g.root_rest[s];
      target = skin_point(fc, v3(r.x, r.y, r.z), g.skin[s]);
    }
  }
  return target;
}

template <int NC, typename XS, typename VS, int M>
__device__ __forceinline__ void substeps_ref(const FrameConst& fc, const StrandConsts& K, const SphereCache<M>& C,
                                             const SphereSet& S, int n, V3 x0_start, V3 target, float rest0,
                                             const XS& X, const VS& V) {
  const bool moving = fc.root_mode != HS_ROOT_PINNED;
  const V3 root_delta = sub(target, x0_start);
  V3 root = x0_start;  // root position at the start of the substep
  for (int k = 0; k < fc.substeps; ++k) {
    // Root (:184-193): kinematic, linear to its target, on it at the end.
    V3 p0 = root;
    if (moving) {
      const float alpha = __fdiv_rn(static_cast<float>(k + 1), static_cast<float>(fc.substeps));
      p0 = (k + 1 == fc.substeps) ? target : fmas(alpha, root_delta, x0_start);
    }
    const V3 v0 = sub(p0, root);  // :192
    root = p0;
    X.store(0, f4(p0, rest0));
    V.store(0, f4(v0, vel_w<XS>(rest0)));
    if (n >= 2) {
      if (fc.iterations == 1) substep_single_pass_ref<NC>(K, C, S, n, p0, X, V);
      else substep_multi_pass_ref<NC>(K, C, S, n, fc.iterations, p0, X, V);
    }
    V.fence();
  }
}

// Substeps k0 .. substeps - 1, one at a time.
template <bool SPLIT, bool PICK, bool FAST, typename XS, typename VS, int NF>
__device__ __forceinline__ void substeps_seg(const FrameConst& fc, const StrandConsts& K, const SphereFilter<NF>& F,
                                             const SphereSet& S, int n, int jmin, int k0, const RootPath& path,
                                             const XS& X, const VS& V) {
  V3 rel_prev = path.rel(k0 - 1);
  for (int k = k0; k < fc.substeps; ++k) {
    const V3 rel = path.rel(k), D0 = sub(rel, rel_prev), R = path.at(k, rel);
    rel_prev = rel;
    if (n >= 2) {
      if (fc.iterations == 1) substep_single_pass_seg<SPLIT, PICK, FAST>(K, F, S, n, jmin, D0, R, X, V);
      else substep_multi_pass_seg<PICK, FAST>(K, F, S, n, jmin, fc.iterations, D0, R, X, V);
    }
    V.fence();
  }
}

// One frame of strand s. X: the position/segment slots (XShared4 or
// XShared3, this thread's column of the block's shared [point][thread]
// arrays); V: the velocity slots (VShared, or VTmem: whose loads and stores
// are warp-collective, so every lane runs every pass, active or not).
// M (reference mode): sphere-cache width. With M = 8 a warp that reaches
// more than kCachedSpheres spheres tests 8 cached ones instead of running
// the exact push-out at every point; the others keep the 4-wide tests.
// SPLIT: the DFTL pass shape (substep_single_pass_seg). One code shape per
// kernel keeps the instruction cache warm: the batched kernels run one
// loop; the plain step splits it.
// PICK: the push-out's form (push_seg). P: pairs of substeps at once
// (WavePass; 0: one substep at a time). NF: slots of the sphere filter.
// EACH: grooms of fewer pairs share the kernel (FrameConst::pairs); those of
// none test 8 slots, whatever NF.
template <bool REF, typename XS, typename VS, int M = kCachedSpheres, bool SPLIT = false, bool PICK = false,
          bool FAST = false, int P = 0, int NF = 8, bool EACH = false>
__device__ __forceinline__ void strand_frame_stream(const FrameConst& fc, const SphereSet& S, const GroomView& g,
                                                    uint32_t s, bool active, const XS& X, const VS& V) {
  const int n = static_cast<int>(g.npoints);
  float R = 0.0f;  // total link length, for culling
  float rest0 = 0.0f;
  V3 x0_start = v3(0.0f, 0.0f, 0.0f);
  V3 last = x0_start;  // previous point (DFTL: segments are differences)
  // The strand comes in kLoadBatch points at a time: all their HBM loads
  // are issued before the first on-chip store (a TMEM store is a compiler
  // barrier, which would otherwise leave one load in flight per thread).
  constexpr int kLoadBatch = 8;
  for (int i0 = 0; i0 < n; i0 += kLoadBatch) {
    float4 p[kLoadBatch], v[kLoadBatch];
#pragma unroll
    for (int k = 0; k < kLoadBatch; ++k) {
      p[k] = v[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (active && i0 + k < n) {
        p[k] = g.pos[static_cast<size_t>(i0 + k) * g.stride + s];
        v[k] = g.vel[static_cast<size_t>(i0 + k) * g.stride + s];
      }
    }
#pragma unroll
    for (int k = 0; k < kLoadBatch; ++k) {
      const int i = i0 + k;
      if (i < n) {  // uniform over the warp (TMEM stores are warp-collective)
        float4 xs = p[k];
        if (i == 0) {
          x0_start = xyz(p[k]);
          rest0 = p[k].w;
        }
        if (!REF) {
          xs = f4(i == 0 ? v3(0.0f, 0.0f, 0.0f) : sub(xyz(p[k]), last), p[k].w);
          last = xyz(p[k]);
        }
        X.store(i, xs);
        const float4 vk = frame_velocity<!REF, true>(fc, v[k]);
        V.store(i, make_float4(vk.x, vk.y, vk.z, XS::kRestInV ? p[k].w : v[k].w));
        if (i > 0) R += fabsf(fc.length_scale * p[k].w);
      }
    }
  }
  V.fence();

  const StrandConsts K = strand_consts(fc, g, s, active);
  V3 target = root_target(fc, g, s, active, x0_start);

  // Spheres each strand can touch during the frame (see hs_step.cuh), and
  // the warp's first point that can touch one: point j stays within R_j (its
  // links' lengths summed from the root) of the root, so it cannot reach
  // sphere k before R_j covers the distance from the root's path to k's
  // surface (same margins as near_spheres). A sphere reached only through
  // an overlap is entered by a point another sphere pushed first.
  if constexpr (REF) {
    uint32_t reach = 0u;
    if (S.n > 0) {
      const V3 root_delta = sub(target, x0_start);
      const V3 mid = v3(0.5f * (x0_start.x + target.x), 0.5f * (x0_start.y + target.y), 0.5f * (x0_start.z + target.z));
      const float half_path = 0.5f * sqrtf(root_delta.x * root_delta.x + root_delta.y * root_delta.y +
                                           root_delta.z * root_delta.z);
      reach = active ? overlap_closure(S, near_spheres(S, mid, R + half_path)) : 0u;
    }
    const SphereCache<M> C = cache_spheres<M>(S, reach);
    // All tested slots are tested whether filled or not (empty ones never
    // hit). The width is chosen per warp.
    const int warp_cached = __reduce_max_sync(0xffffffffu, C.ncached);
    if (M > kCachedSpheres && warp_cached > kCachedSpheres)
      substeps_ref<M>(fc, K, C, S, n, x0_start, target, rest0, X, V);
    else
      substeps_ref<kCachedSpheres>(fc, K, C, S, n, x0_start, target, rest0, X, V);
  } else {
    uint32_t reach = 0u;
    int jmin = n;
    float far = 0.0f;
    if (S.n > 0) {
      const StrandBall ball(x0_start, target, R);
      const SphereReach q = sphere_reach(S, ball);
      reach = active ? overlap_closure(S, q.near) : 0u;
      far = ball.far();
      if (__any_sync(0xffffffffu, reach)) {
        float Rj = 0.0f;
        int jl = n;
        for (int i = 1; i < n; ++i) {  // the same sum as R, point by point
          Rj += fabsf(fc.length_scale * rest_of(X, V, i));
          if (jl == n && Rj >= q.threshold) jl = i;
        }
        jmin = __reduce_min_sync(0xffffffffu, active ? jl : n);
      }
    }
    const bool moves = fc.root_mode != HS_ROOT_PINNED;
    if (EACH && NF != 8 && fc.pairs == 0) {
      substeps_seg<SPLIT, PICK, FAST>(fc, K, filter_spheres<8>(S, reach, far), S, n, jmin, 0,
                                      RootPath{x0_start, target, fc.substeps, moves}, X, V);
    } else {
      const SphereFilter<NF> F = filter_spheres<NF>(S, reach, far);
      int k0 = 0;  // substeps done in pairs
      if constexpr (P > 0) {
        if (!EACH || fc.pairs > 0) {
          // The root's path waits in slot 0.
          X.store(0, f4(x0_start, rest0));
          V.store(0, f4(target, rest0));
          k0 = wave_substeps<P, FAST>(fc, K, F, S, n, jmin, EACH ? fc.pairs : P, X, V);
          V.fence();
          const float4 v0 = V.load(0);
          x0_start = xyz(X.load(0));
          target = xyz(v0);
          rest0 = v0.w;
        }
      }
      substeps_seg<SPLIT, PICK, FAST>(fc, K, F, S, n, jmin, k0, RootPath{x0_start, target, fc.substeps, moves}, X, V);
    }
    const RootPath path{x0_start, target, fc.substeps, moves};
    const V3 D0 = sub(path.rel(fc.substeps - 1), path.rel(fc.substeps - 2));
    X.store(0, f4(v3(0.0f, 0.0f, 0.0f), rest0));
    V.store(0, f4(vel_of(K, D0), vel_w<XS>(rest0)));
    V.fence();
  }

  // Store: reference mode holds positions; DFTL mode rebuilds them from the
  // final root and the segments.
  const bool moving = fc.root_mode != HS_ROOT_PINNED;
  V3 w = moving ? target : x0_start;
  TileStats ts;
  ts.init();
  for (int i = 0; i < n; ++i) {
    const float4 vs = V.load(i);
    if (active) {
      float4 x = with_rest<XS>(X.load(i), vs);
      const float4 v = frame_velocity<!REF, false>(fc, vs);
      if (!REF) {
        if (i > 0) w = add(w, xyz(x));
        x = f4(w, x.w);
      }
      g.pos[static_cast<size_t>(i) * g.stride + s] = x;
      g.vel[static_cast<size_t>(i) * g.stride + s] = make_float4(v.x, v.y, v.z, 0.0f);
      ts.add(x, v);
    }
  }
  ts.store(g.stats, s / 32u, (g.nstrands + 31u) / 32u, static_cast<int>(threadIdx.x % 32u));
}

// Register form of a DFTL frame (short strands): the segments in
// registers, the velocity slots (then displacements) in registers or
// shared rows (VStore, hs_step.cuh). The passes of substep_multi_pass_seg,
// unrolled over CAP; with one iteration they compute what
// substep_single_pass_seg does, operation for operation.
// MANY (more than kFewSpheres spheres): the push-out branches past spheres
// the point is not inside. Registers are for four filter slots, so a strand
// that reaches more sends most points through all of them: 50,021 x 8 among
// 32 spheres, 8 substeps, EXACT, 47.8 -> 40.1 us, x 4 22.6 -> 18.6; among 12
// 21.4 -> 20.6. (Eight slots and flagged spheres only take 36.4 there, but 43
// against 37 us for 120,000 x 8 among 24.)
template <int CAP, bool VSMEM, bool FAST, bool MANY>
__device__ __forceinline__ void strand_frame_regs_dftl(const FrameConst& fc, const SphereSet& S, const GroomView& g,
                                                       uint32_t s, bool active, float4* vs_rows, int thread) {
  const int n = static_cast<int>(g.npoints);
  const V3 zero = v3(0.0f, 0.0f, 0.0f);
  V3 Sg[CAP];
  VStore<CAP, VSMEM> vs;
  vs.bind(vs_rows, thread);
  float R = 0.0f, rest0 = 0.0f;
  V3 x0_start = zero, last = zero;
#pragma unroll
  for (int i = 0; i < CAP; ++i) {
    Sg[i] = zero;
    if (i < n) {
      float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f), v = p;
      if (active) {
        p = g.pos[static_cast<size_t>(i) * g.stride + s];
        v = g.vel[static_cast<size_t>(i) * g.stride + s];
      }
      if (i == 0) {
        x0_start = xyz(p);
        rest0 = p.w;
      } else {
        Sg[i] = sub(xyz(p), last);
        R += fabsf(fc.length_scale * p.w);
      }
      last = xyz(p);
      const float4 vin = frame_velocity<true, true>(fc, v);
      vs.set(i, make_float4(vin.x, vin.y, vin.z, p.w));
    }
  }

  const StrandConsts K = strand_consts(fc, g, s, active);
  const V3 target = root_target(fc, g, s, active, x0_start);
  const bool moving = fc.root_mode != HS_ROOT_PINNED;
  uint32_t reach = 0u;
  float far = 0.0f;
  if (S.n > 0) {
    const StrandBall ball(x0_start, target, R);
    reach = active ? overlap_closure(S, near_spheres(S, ball.mid, ball.radius)) : 0u;  // per lane
    far = ball.far();
  }
  const SphereFilter<4> F = filter_spheres<4>(S, reach, far);

  const V3 delta = sub(target, x0_start);
  V3 rel_prev = zero, D0 = zero;
  for (int k = 0; k < fc.substeps; ++k) {
    V3 rel = zero, Rk = x0_start;
    if (moving) {
      const bool lastk = k + 1 == fc.substeps;
      const float alpha = __fdiv_rn(static_cast<float>(k + 1), static_cast<float>(fc.substeps));
      rel = lastk ? delta : mul(alpha, delta);
      Rk = lastk ? target : add(x0_start, rel);
    }
    D0 = sub(rel, rel_prev);
    rel_prev = rel;
#pragma unroll
    for (int i = 1; i < CAP; ++i) {
      if (i < n) {
        const float4 sl = vs.get(i);
        vs.set(i, f4(disp(K, sl), sl.w));
      }
    }
    for (int it = 0; it < fc.iterations; ++it) {
      const bool last_it = it + 1 == fc.iterations;
      V3 D_prev = D0, e_prev = zero, w_prev = Rk, s_prev = zero;
      float rest_prev = 0.0f;
#pragma unroll
      for (int i = 1; i <= CAP; ++i) {
        if (i <= n) {
          V3 sn = zero, e = zero, D_i = zero, w_i = zero;
          float rest_i = 0.0f;
          if (i < CAP && i < n) {
            const float4 sl = vs.get(i);
            rest_i = sl.w;
            const V3 d = it == 0 ? sub(add(Sg[i], xyz(sl)), D_prev) : sub(Sg[i], e_prev);
            link_seg<FAST>(K, d, rest_i, sn, e);
            D_i = add(xyz(sl), e);
            w_i = add(w_prev, sn);
          }
          if (i >= 2) {
            const bool tip = i == n;
            V3 Dj = D_prev, sj = s_prev;
            if (flagged(F, w_prev)) push_seg<false, FAST, MANY>(F, S, w_prev, Dj, sj, sn, tip);
            const V3 out = last_it ? vel_of(K, tip ? Dj : fmas(K.neg_damping, e, Dj)) : Dj;
            Sg[i - 1] = sj;
            vs.set(i - 1, f4(out, rest_prev));
          }
          D_prev = D_i;
          e_prev = e;
          w_prev = w_i;
          s_prev = sn;
          rest_prev = rest_i;
        }
      }
    }
  }
  vs.set(0, f4(vel_of(K, D0), rest0));

  TileStats ts;
  ts.init();
  if (active) {
    V3 w = moving ? target : x0_start;
#pragma unroll
    for (int i = 0; i < CAP; ++i) {
      if (i < n) {
        const float4 v = frame_velocity<true, false>(fc, vs.get(i));
        if (i > 0) w = add(w, Sg[i]);
        const float4 x = f4(w, v.w);
        g.pos[static_cast<size_t>(i) * g.stride + s] = x;
        g.vel[static_cast<size_t>(i) * g.stride + s] = make_float4(v.x, v.y, v.z, 0.0f);
        ts.add(x, v);
      }
    }
  }
  ts.store(g.stats, s / 32u, (g.nstrands + 31u) / 32u, static_cast<int>(threadIdx.x % 32u));
}

}  // namespace hs
