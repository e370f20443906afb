// Four-wide ordered traversal (device): the hits of trace_ray, in fewer and fuller warp steps.
//
// Why it finds the same hits. The reference's traversal (intersect.rs:172-263) visits the leaves of
// the binary hierarchy in an order fixed by the ray alone (at every interior node the child with the
// strictly smaller entry distance first, else the right one), and visits a leaf exactly when the
// leaf's own box passes the slab test with the closest distance held at its turn: the boxes above it
// contain it, every slab operation is a monotone rounding of one plane, so an ancestor's box passes
// whenever the leaf's does, and the closest distance only shrinks. A wide node therefore tests the
// four grandchildren of an interior node at once, leaves out the two boxes between (their entry
// distances, needed for the order, are the minima over their children's planes), and a stacked
// child is re-tested against the closest distance when it is popped.
//
// Along an axis with d = 0 a plane's product is NaN when the origin lies on the plane, else +-inf, and a
// NaN falls out of every maximum and minimum over the axes: on a face is inside. For the box in
// between, a product of NaN among its children's near planes says that its own near plane is the
// origin's (NaN) or before it (-inf); either leaves the entry distance to the other axes, so the
// minimum over the children keeps the NaN (min_keep_nan). One axis must have a finite 1/d, or all
// three could be NaN: rays without one, and non-finite ones, are left to trace_ray. With all
// axis-parallel rays left to it, 1,048,576 rays straight down took 583 us on 2,051 primitives, 349 on
// the mixed scene, 1,190 in the room and 452 on the terrain (one thread per ray over the pairs: 418,
// 251, 875 and 361); now 240, 173, 669 and 297.
//
// Cost model and choices (per 38 M-ray mixed-scene frame, 40 M-ray room frame and 31 M-ray terrain
// frame; trace launches; binary while-while loop: 11.5, 40.2 and 8.6 ms at 8.2, 6.8 and 13.6 of 32
// lanes per instruction). The traversal is bound by instruction issue and, in the room, by the L1
// data stage (89% busy), which serves a warp's scattered 16-byte loads at about 2.5 lanes a clock:
//   - wide nodes and packed FP32 (add/mul.f32x2) halve the instructions per ray; the near and far
//     planes are picked by address (sign of the direction) instead of by 12 selects per node;
//   - a node is one 128-byte line whose quads are swizzled by the node index: without it the lanes'
//     loads of one quad collide in the same banks (12.0 -> 11.5 and 34.9 -> 31.9 ms);
//   - a leaf's primitives are tested two at a time (LeafPair);
//   - the caller's loop alternates node and leaf phases by warp vote instead of waiting for every
//     lane to reach a leaf, and refills lanes whose ray is done;
//   - the direction is kept in shared memory between leaf steps: 64 registers, 8 blocks per SM.
// Together 9.2, 24.9 and 7.7 ms (13.9, 16.9 and 19.0 lanes per instruction).
#ifndef TOASTER_B200_TRAVERSE_WIDE_CUH
#define TOASTER_B200_TRAVERSE_WIDE_CUH

#include "traverse.cuh"

namespace tcb {

using f32x2 = unsigned long long;  // two FP32 values of one packed operation

__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// a - b with one rounding, written as b * -1 + a. The assembler contracts mul.rn.f32x2 feeding
// add.rn.f32x2 into one fused operation, which would lose the product's rounding; this form it
// keeps (the bit-exact hit tests would show a change). Sums of products below are therefore all
// differences, with one factor's sign flipped beforehand.
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(b), "l"(0xBF800000BF800000ull), "l"(a));
  return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

__device__ __forceinline__ float min_keep_nan(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

struct WideRay {
  f32x2 nox, noy, noz;  // (-o, -o)
  f32x2 ix, iy, iz;     // (1/d, 1/d)
  uint32_t ax, ay, az;  // byte offset of the near planes' quad (the far planes' is ^ 16)
};

// Rays the wide traversal takes: finite, no 1/d zero or NaN, and not every 1/d infinite.
__device__ __forceinline__ bool wide_takes(const RayQ& r) {
  const float low = fminf(fminf(fabsf(r.ix), fabsf(r.iy)), fabsf(r.iz));
  const float far = (fabsf(r.ox) + fabsf(r.oy)) + fabsf(r.oz);  // NaN or inf when one is
  const float any = (fabsf(r.ix) + fabsf(r.iy)) + fabsf(r.iz);  // NaN when one is
  return low > 0.0f && low < CUDART_INF_F && far < CUDART_INF_F && any == any;
}

__device__ __forceinline__ WideRay make_wide_ray(const RayQ& r) {
  WideRay w;
  w.nox = pack2(-r.ox, -r.ox);
  w.noy = pack2(-r.oy, -r.oy);
  w.noz = pack2(-r.oz, -r.oz);
  w.ix = pack2(r.ix, r.ix);
  w.iy = pack2(r.iy, r.iy);
  w.iz = pack2(r.iz, r.iz);
  w.ax = r.sx ? 16u : 0u;
  w.ay = r.sy ? 48u : 32u;
  w.az = r.sz ? 80u : 64u;
  return w;
}

// The ray's direction as the leaf step reads it, in this thread's words of a shared array (three
// rows of kStride): x, -y, -z.
template <int kStride>
__device__ __forceinline__ void store_direction(float* dir, const RayQ& r) {
  dir[0] = r.dx;
  dir[kStride] = -r.dy;
  dir[2 * kStride] = -r.dz;
}

struct WideTraversal {
  uint32_t cur;   // wide node, kLeafBit | leaf pair, or kNoNode when the traversal is over
  int sp;
  float closest;
  uint32_t rec;   // accepted primitive record, kNoNode while there is none
  __device__ __forceinline__ bool at_node() const { return (cur & kLeafBit) == 0u; }
  __device__ __forceinline__ bool at_leaf() const { return (cur & kLeafBit) != 0u && cur != kNoNode; }
  __device__ __forceinline__ bool live() const { return cur != kNoNode; }
};

__device__ __forceinline__ void wide_start(WideTraversal& T, const ChildRec& root, const RayQ& r, float tmin,
                                           float tmax) {
  T.closest = tmax;
  T.rec = kNoNode;
  T.sp = 0;
  float entry, tn;
  T.cur = box_test(root.min_x, root.min_y, root.min_z, root.max_x, root.max_y, root.max_z, r, tmin, tmax, entry, tn)
              ? root.link
              : kNoNode;
}

// Next stacked child whose entry is still within the closest distance.
__device__ __forceinline__ void wide_pop(WideTraversal& T, const uint2* st) {
  uint32_t cur = kNoNode;
  while (T.sp > 0) {
    --T.sp;
    const uint2 e = st[T.sp];
    if (__uint_as_float(e.y) <= T.closest) {
      cur = e.x;
      break;
    }
  }
  T.cur = cur;
}

// Tests the four boxes of wide node T.cur, goes to the first one hit and stacks the others.
__device__ __forceinline__ void wide_node_step(WideTraversal& T, const WideRay& r, float tmin,
                                               const WideNode* __restrict__ nodes, uint2* st) {
  const char* base = reinterpret_cast<const char*>(nodes);
  const uint32_t off = (T.cur << 7) | ((T.cur & 7u) << 4);
  auto quad = [&](uint32_t o) { return __ldg(reinterpret_cast<const ulonglong2*>(base + o)); };
  const uint32_t ox = off ^ r.ax, oy = off ^ r.ay, oz = off ^ r.az;
  const ulonglong2 qnx = quad(ox), qny = quad(oy), qnz = quad(oz);
  const ulonglong2 qfx = quad(ox ^ 16u), qfy = quad(oy ^ 16u), qfz = quad(oz ^ 16u);
  const uint4 link = __ldg(reinterpret_cast<const uint4*>(base + (off ^ 96u)));
  auto slab = [](f32x2 plane, f32x2 no, f32x2 inv) { return unpack2(mul2(add2(plane, no), inv)); };
  const float2 nx01 = slab(qnx.x, r.nox, r.ix), nx23 = slab(qnx.y, r.nox, r.ix);
  const float2 ny01 = slab(qny.x, r.noy, r.iy), ny23 = slab(qny.y, r.noy, r.iy);
  const float2 nz01 = slab(qnz.x, r.noz, r.iz), nz23 = slab(qnz.y, r.noz, r.iz);
  const float2 fx01 = slab(qfx.x, r.nox, r.ix), fx23 = slab(qfx.y, r.nox, r.ix);
  const float2 fy01 = slab(qfy.x, r.noy, r.iy), fy23 = slab(qfy.y, r.noy, r.iy);
  const float2 fz01 = slab(qfz.x, r.noz, r.iz), fz23 = slab(qfz.y, r.noz, r.iz);
  const float e0 = max3(nx01.x, ny01.x, nz01.x), e1 = max3(nx01.y, ny01.y, nz01.y);
  const float e2 = max3(nx23.x, ny23.x, nz23.x), e3 = max3(nx23.y, ny23.y, nz23.y);
  const float t0 = fmaxf(e0, tmin), t1 = fmaxf(e1, tmin), t2 = fmaxf(e2, tmin), t3 = fmaxf(e3, tmin);
  const bool h0 = fminf(min3(fx01.x, fy01.x, fz01.x), T.closest) >= t0;
  const bool h1 = fminf(min3(fx01.y, fy01.y, fz01.y), T.closest) >= t1;
  const bool h2 = fminf(min3(fx23.x, fy23.x, fz23.x), T.closest) >= t2;
  const bool h3 = fminf(min3(fx23.y, fy23.y, fz23.y), T.closest) >= t3;
  // Entry distances of the two boxes in between.
  const float ea = max3(min_keep_nan(nx01.x, nx01.y), min_keep_nan(ny01.x, ny01.y), min_keep_nan(nz01.x, nz01.y));
  const float eb = max3(min_keep_nan(nx23.x, nx23.y), min_keep_nan(ny23.x, ny23.y), min_keep_nan(nz23.x, nz23.y));
  const bool a_first = ea < eb;
  // First and second hit child of each half in traversal order, then the halves in theirs.
  const bool take0 = h0 && (e0 < e1 || !h1), take2 = h2 && (e2 < e3 || !h3);
  const uint32_t fa = take0 ? link.x : link.y, sa = take0 ? link.y : link.x;
  const float fa_t = take0 ? t0 : t1, sa_t = take0 ? t1 : t0;
  const uint32_t fb = take2 ? link.z : link.w, sb = take2 ? link.w : link.z;
  const float fb_t = take2 ? t2 : t3, sb_t = take2 ? t3 : t2;
  const bool hit_a = h0 || h1, hit_b = h2 || h3, both_a = h0 && h1, both_b = h2 && h3;
  int sp = T.sp;
  if (a_first ? both_b : both_a) st[sp++] = make_uint2(a_first ? sb : sa, __float_as_uint(a_first ? sb_t : sa_t));
  if (hit_a && hit_b) st[sp++] = make_uint2(a_first ? fb : fa, __float_as_uint(a_first ? fb_t : fa_t));
  if (a_first ? both_a : both_b) st[sp++] = make_uint2(a_first ? sa : sb, __float_as_uint(a_first ? sa_t : sb_t));
  T.sp = sp;
  if (hit_a || hit_b) T.cur = hit_a && (a_first || !hit_b) ? fa : fb;
  else wide_pop(T, st);
}

// One 32-byte sector in one load.
struct Sector {
  f32x2 a, b, c, d;
};
__device__ __forceinline__ Sector load_sector(const void* p) {
  Sector s;
  asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(s.a), "=l"(s.b), "=l"(s.c), "=l"(s.d) : "l"(p));
  return s;
}

// Tests the two primitives of leaf pair T.cur in leaf order, then goes to the leaf's next pair or the
// next stacked child. A slot's distance does not depend on the closest distance, so both are
// computed at once and accepted in order (`t <= closest`, as the reference does).
template <int kStride>
__device__ __forceinline__ void wide_leaf_step(WideTraversal& T, const WideRay& r, const float* dir, float tmin,
                                               bool any_hit, const LeafPair* __restrict__ leaves, const uint2* st) {
  const char* p = reinterpret_cast<const char*>(leaves + (T.cur & ~kLeafBit));
  const Sector q0 = load_sector(p), q1 = load_sector(p + 32);
  const ulonglong2 q2 = __ldg(reinterpret_cast<const ulonglong2*>(p + 64));
  const float dx1 = dir[0], ndy1 = dir[kStride], ndz1 = dir[2 * kStride];
  const f32x2 dx = pack2(dx1, dx1), ndy = pack2(ndy1, ndy1), ndz = pack2(ndz1, ndz1);
  const uint32_t first = uint32_t(q2.y), flags = uint32_t(q2.y >> 32);
  const f32x2 e1x = q0.d, e1y = q1.a, e1z = q1.b, e2x = q1.c, ne2y = q1.d, ne2z = q2.x;
  // Moller-Trumbore (intersect.rs:87-120) with the reference's roundings; n marks a flipped sign.
  const f32x2 px = sub2(mul2(ndy, ne2z), mul2(ne2y, ndz));
  const f32x2 npy = sub2(mul2(ndz, e2x), mul2(ne2z, dx));
  const f32x2 npz = sub2(mul2(dx, ne2y), mul2(e2x, ndy));
  const float2 det = unpack2(sub2(sub2(mul2(e1x, px), mul2(e1y, npy)), mul2(e1z, npz)));
  const f32x2 inv = pack2(__frcp_rn(det.x), __frcp_rn(det.y));
  const f32x2 sx = sub2(q0.a, r.nox), sy = sub2(q0.b, r.noy), sz = sub2(q0.c, r.noz);  // o - v0
  const f32x2 u2 = mul2(sub2(sub2(mul2(sx, px), mul2(sy, npy)), mul2(sz, npz)), inv);
  const f32x2 qx = sub2(mul2(sy, e1z), mul2(e1y, sz));
  const f32x2 qy = sub2(mul2(sz, e1x), mul2(e1z, sx));
  const f32x2 qz = sub2(mul2(sx, e1y), mul2(e1x, sy));
  const f32x2 v2 = mul2(sub2(sub2(mul2(dx, qx), mul2(ndy, qy)), mul2(ndz, qz)), inv);
  const f32x2 t2 = mul2(sub2(sub2(mul2(e2x, qx), mul2(ne2y, qy)), mul2(ne2z, qz)), inv);
  const float2 u = unpack2(u2), v = unpack2(v2), t = unpack2(t2);
  bool ok0 = !(fabsf(det.x) < 1e-8f) & (u.x >= 0.0f) & (u.x <= 1.0f) & !(v.x < 0.0f) &
             !(__fadd_rn(u.x, v.x) > 1.0f) & !(t.x < tmin);
  bool ok1 = !(fabsf(det.y) < 1e-8f) & (u.y >= 0.0f) & (u.y <= 1.0f) & !(v.y < 0.0f) &
             !(__fadd_rn(u.y, v.y) > 1.0f) & !(t.y < tmin);
  float t0 = t.x, t1 = t.y;
  if (flags & (kPairSphere0 | kPairSphere1)) {
    // Spheres (intersect.rs:28-50): both slots up to the discriminant, then the roots of the slots
    // that can be hit, one slot per round (a lane seldom has two). The far root is taken exactly
    // when the near one lies before tmin: behind a near root beyond `closest` the far one is too.
    const float a = __fadd_rn(__fadd_rn(__fmul_rn(dx1, dx1), __fmul_rn(ndy1, ndy1)), __fmul_rn(ndz1, ndz1));
    const f32x2 hb2 = sub2(sub2(mul2(sx, dx), mul2(sy, ndy)), mul2(sz, ndz));
    const float2 xx = unpack2(mul2(sx, sx)), yy = unpack2(mul2(sy, sy)), zz = unpack2(mul2(sz, sz));
    const float2 rr = unpack2(e1y);
    const f32x2 c = pack2(__fsub_rn(__fadd_rn(__fadd_rn(xx.x, yy.x), zz.x), rr.x),
                          __fsub_rn(__fadd_rn(__fadd_rn(xx.y, yy.y), zz.y), rr.y));
    const float2 disc = unpack2(sub2(mul2(hb2, hb2), mul2(pack2(a, a), c))), hb = unpack2(hb2);
    uint32_t todo = 0u;
    if (flags & kPairSphere0) {
      ok0 = !(disc.x < 0.0f);
      todo = ok0 ? 1u : 0u;
    }
    if (flags & kPairSphere1) {
      ok1 = !(disc.y < 0.0f);
      todo |= ok1 ? 2u : 0u;
    }
    while (todo) {
      const bool second = (todo & 1u) == 0u;
      todo = second ? 0u : todo & 2u;
      const float h = second ? hb.y : hb.x;
      const float root = __fsqrt_rn(second ? disc.y : disc.x);
      float ts = __fdiv_rn(__fsub_rn(-h, root), a);
      if (ts < tmin) ts = __fdiv_rn(__fadd_rn(-h, root), a);
      const bool ok = !(ts < tmin);
      if (second) {
        t1 = ts;
        ok1 = ok;
      } else {
        t0 = ts;
        ok0 = ok;
      }
    }
  }
  ok0 = ok0 & !(t0 > T.closest);
  T.closest = ok0 ? t0 : T.closest;
  T.rec = ok0 ? first : T.rec;
  ok1 = ok1 & !(t1 > T.closest);
  T.closest = ok1 ? t1 : T.closest;
  T.rec = ok1 ? first + 1u : T.rec;
  if ((ok0 | ok1) & any_hit) T.cur = kNoNode;
  else if (flags & kPairLast) wide_pop(T, st);
  else T.cur += 1u;
}

// One round of a warp's traversals (every lane calls it): node steps while more than `keep` lanes
// stand at a node, then leaf steps while more than kLeafRest lanes stand at a leaf. Lanes at a leaf
// wait for the node phase to end and the other way round, so the thresholds trade fuller steps
// against waiting: keep 8 / 10 / 12 / 16 took 9.72 / 9.80 / 9.91 / 10.28 ms on the mixed scene and
// 26.4 / 26.1 / 26.1 / 26.8 ms in the room, kLeafRest 0 / 4 / 6 / 8 10.66 / 9.80 / 9.63 / 9.60 ms.
constexpr int kNodeKeep = 10;
constexpr int kLeafRest = 6;
template <int kStride>
__device__ __forceinline__ void wide_round(WideTraversal& T, const WideRay& r, const float* dir, float tmin,
                                           bool any_hit, const WideNode* __restrict__ nodes,
                                           const LeafPair* __restrict__ leaves, uint2* st, int keep) {
  unsigned m;
#pragma unroll 1
  do {
    if (T.at_node()) wide_node_step(T, r, tmin, nodes, st);
    m = __ballot_sync(0xffffffffu, T.at_node());
  } while (__popc(m) > keep);
#pragma unroll 1
  do {
    if (T.at_leaf()) wide_leaf_step<kStride>(T, r, dir, tmin, any_hit, leaves, st);
    m = __ballot_sync(0xffffffffu, T.at_leaf());
  } while (__popc(m) > kLeafRest);
}

// The same ray through trace_ray, for the few rays the wide traversal does not take (kept out of line:
// inlined, its registers would count against every caller).
__device__ __noinline__ bool trace_pairs(const PairNode* pairs, const PrimRecord* prims, const ChildRec* root,
                                         const RayQ& q, float tmin, float tmax, bool any_hit, TraceResult& tr) {
  uint32_t visits = 0;
  return trace_ray(pairs, prims, *root, q, tmin, tmax, any_hit, tr, visits);
}

// Begins a ray of the wide traversal, or traces it whole when the wide traversal does not take it.
__device__ __forceinline__ void wide_begin(WideTraversal& T, const PairNode* pairs, const PrimRecord* prims,
                                           const ChildRec* root_dev, const ChildRec& root, const RayQ& q, float tmin,
                                           float tmax, bool any_hit) {
  wide_start(T, root, q, tmin, tmax);
  if (!wide_takes(q)) {
    TraceResult tr;
    T.cur = kNoNode;
    if (trace_pairs(pairs, prims, root_dev, q, tmin, tmax, any_hit, tr)) {
      T.closest = tr.t;
      T.rec = tr.rec;
    }
  }
}

}  // namespace tcb

#endif
