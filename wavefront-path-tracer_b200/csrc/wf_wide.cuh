// Traversal of the compressed 8-wide BVHs (WideNode, wf_device.cuh): closest
// hit and any hit as resumable per-lane state machines, used by every kernel
// that traces rays but camera rays and frame guides, whose warps visit the
// same BVH2 nodes together, and the ray batches of shallow scenes (ray_route).
//
// The node layout and the test of eight quantised child boxes against a
// ray-order hit mask follow Ylitie, Karras and Laine, "Efficient Incoherent
// Ray Traversal on GPUs Through Compressed Wide BVHs" (HPG 2017).  Traversal
// is bound by dependent node fetches and by the divergence of a warp's
// lanes; an 8-wide node takes the place of about three BVH2 levels, so a ray
// makes a third of the fetches and loop turns.
//
// Same results as the reference's BVH2 traversal (traceRay / isOccluded,
// device_traversal.cuh:1035-1184; trace_closest_binary and trace_any_binary
// here).  A candidate is a primitive whose own test and whose boxes' slab
// tests pass, the closest distance left aside.  The slab test's operations
// are monotone in the box planes, so the boxes of one BVH2 pass exactly when
// the leaf's does: exact_leaf_box and exact_triangle_box check it, in the
// BVH2's arithmetic, for the TLAS leaf and for the triangle.  The BVH2 also
// culls by "entry < closestT", in its own visit order.  Its answer is the
// closest candidate whatever the order when the entries of that candidate's
// boxes (the TLAS leaf's, of the world ray, and the triangle's, of the local
// one) lie before the distance of every other candidate.  The lane sees every
// candidate up to kNear past the closest one and notes whether that holds for
// certain (lane_near); a ray for which it may not is traced once more by
// trace_closest_binary.  Rays through a shared edge of two triangles and hits
// of coincident triangles are the usual cases.  Any-hit queries do not depend
// on the order.
//
// Nodes are culled here only where no candidate below them can be the
// closest.  A candidate's computed distance may lie before its own box, by
// the rounding of its test, so the entry that culls is that of a box grown by
// the errors below (WideRay::margin); the boxes' own tests are not widened.
//   * A triangle's distance is that of a triangle moved by a few roundings of
//     the vector from the ray's origin to it (some 24 u / sin of its sharpest
//     corner at most, u = 2^-24): 2^-15 of the distance to the farthest
//     corner of the BVH's box, which leaves room for corners down to 3
//     degrees.
//     Not covered: a ray within about a degree of the triangle's plane that
//     meets it within rounding of the edge of its box, in front of a surface
//     closer than that error; such a ray may keep that surface's hit where
//     the BVH2's order finds the triangle's.
//   * An instance's distance is found in its own frame.  Its world box is off
//     by the roundings of the ray's transform, 8 u |L| |W| (local to world,
//     world to local) times the distance, and of the translation and the box
//     itself: WideBvh::reach and ::base, from the scene's instances.
//   * A sphere's discriminant cancels: its distance is that of a sphere whose
//     squared radius is off by 12 u of its squared distance.  Up to 295 radii
//     away that is less than 2^-13 of the distance on the radius (reach);
//     beyond, box and sphere together are 2^-6 of the distance
//     (WideBvh::slack).
// The margin is one value per ray and BVH.  It costs the 1080p mesh 1.5 % (60.3
// -> 61.2 ms), 3,000,001 ray queries 3.8 % (3.16 -> 3.28 ms); following the
// distance to each node it cost 2.6 and 4.7 %.
//
// Conservative boxes.  With S = 2^15 cell inv and O' = (p - o) inv - S a
// plane q lies at fma(1 + q 2^-15, S, O'), and 1 + q 2^-15 is q's byte put
// into the second byte of 1.0f.  Rounding moves it by less than
// 2^-8 cells + 2^-21 of the distance against the BVH2's own slab value; the
// builder leaves 1/64 cell on either side and the test 2^-15 of the distance
// (kSlack).  1 / d is held to 2^88: the spare of the smallest cell (1e-9)
// times that (4.8e15) still reaches past any distance a direction of at least
// 1e-6 covers (3.5e15).  The bounds on origin (1e9), direction (1e-6 to 1e6)
// and scene coordinates (kWideMaxCoordinate) keep every product finite: cells
// are at most 2^23, S at most 2^126.  Rays outside them take the BVH2s.
#pragma once

#include "wf_traverse.cuh"

namespace wf {

// Entries of the node groups on the way: at most one per level of the TLAS
// and one per level of the BLAS (each at most kMaxBvhDepth = 60 deep), and
// the TLAS leaves left when an instance is entered.
constexpr int kLaneStack = 128;
constexpr float kSlack = kWideSlack;
constexpr float kNear = 1.0f + 1.0f / 131072.0f;

// The ray of the current BVH as the node test wants it.
struct WideRay {
    V3 o, d;
    V3 inv;         // 1 / d, at most kInverseMax in size
    uint32_t oct4;  // per byte: bit a set when inv's component a is positive
    float margin;   // how far outside its box a primitive's distance may lie
};
constexpr float kInverseMax = 3.0948500982134507e26f;  // 2^88

WF_DEV float held_inverse(float d) {
    return copysignf(fminf(fabsf(1.0f / d), kInverseMax), d);
}

// False for rays the wide test's bounds do not cover (NaN too: fmaxf drops a
// NaN operand, the sum does not).
WF_DEV bool ray_covered(V3 o, V3 d) {
    float m = fmaxf(fabsf(d.x), fmaxf(fabsf(d.y), fabsf(d.z)));
    float far = fmaxf(fabsf(o.x), fmaxf(fabsf(o.y), fabsf(o.z)));
    return m >= 1.0e-6f && m <= 1.0e6f && far <= kWideMaxCoordinate && (o.x + o.y + o.z) + (d.x + d.y + d.z) < 1.0e11f;
}

WF_DEV void wide_ray(WideRay& r, V3 o, V3 d) {
    r.o = o;
    r.d = d;
    r.inv = V3{held_inverse(d.x), held_inverse(d.y), held_inverse(d.z)};
    uint32_t oct = (r.inv.x > 0.0f ? 1u : 0u) | (r.inv.y > 0.0f ? 2u : 0u) | (r.inv.z > 0.0f ? 4u : 0u);
    r.oct4 = oct * 0x01010101u;
}

// The BVH2's inverse direction: 1 / d itself (infinite for a zero component).
WF_DEV V3 exact_inverse(const WideRay& r) {
    V3 inv = r.inv;
    if (fmaxf(fabsf(inv.x), fmaxf(fabsf(inv.y), fabsf(inv.z))) >= kInverseMax) inv = inverse_direction(r.d);
    return inv;
}

// One byte of `w` as 1 + byte 2^-15.
template <int kByte>
WF_DEV float plane(uint32_t w) {
    return __uint_as_float(__byte_perm(w, 0x3f800000u, 0x7604u | (kByte << 4)));
}

struct WideSlabs {
    float sx, sy, sz, ox, oy, oz, cull;
    float nx, ny, nz;  // ox, oy, oz for the near planes, moved out by the margin
};

// WideRay::margin in a BVH with root box lo, hi.
WF_DEV float cull_margin(V3 o, V3 lo, V3 hi, float reach, float base) {
    float x = fmaxf(fabsf(lo.x - o.x), fabsf(hi.x - o.x)), y = fmaxf(fabsf(lo.y - o.y), fabsf(hi.y - o.y)),
          z = fmaxf(fabsf(lo.z - o.z), fabsf(hi.z - o.z));
    return __fmaf_rn(fmaxf(x, fmaxf(y, z)), reach, base);
}
WF_DEV float cull_margin(V3 o, const Box& b, float reach, float base) {
    return cull_margin(o, V3{b.lo[0], b.lo[1], b.lo[2]}, V3{b.hi[0], b.hi[1], b.hi[2]}, reach, base);
}

template <int kByte>
WF_DEV bool wide_child(const WideSlabs& b, uint32_t nx, uint32_t ny, uint32_t nz, uint32_t fx, uint32_t fy,
                       uint32_t fz) {
    float tx0 = __fmaf_rn(plane<kByte>(nx), b.sx, b.nx), tx1 = __fmaf_rn(plane<kByte>(fx), b.sx, b.ox);
    float ty0 = __fmaf_rn(plane<kByte>(ny), b.sy, b.ny), ty1 = __fmaf_rn(plane<kByte>(fy), b.sy, b.oy);
    float tz0 = __fmaf_rn(plane<kByte>(nz), b.sz, b.nz), tz1 = __fmaf_rn(plane<kByte>(fz), b.sz, b.oz);
    float entry = fmaxf(fmaxf(tx0, ty0), fmaxf(tz0, 0.0f));
    float exit = fminf(fminf(fminf(tx1, ty1), tz1) * kSlack, b.cull);
    return entry <= exit;
}

// Tests the children of wide node `index`: the internal hits (in visit
// order: highest bit first) with the internal mask into `group`, the leaf
// hits into `leaves`.  Children whose entry is past `cull` are left out; for
// a closest hit it is the entry of their boxes grown by the ray's margin.
template <bool kAny>
WF_DEV void wide_node(const WideNode* nodes, uint32_t index, const WideRay& r, float cull, uint2& group,
                      uint2& leaves) {
    const uint4* n = reinterpret_cast<const uint4*>(nodes + index);
    uint4 a = __ldg(n), b = __ldg(n + 1), c0 = __ldg(n + 2), c1 = __ldg(n + 3), c2 = __ldg(n + 4);
    WideSlabs s;
    s.sx = __uint_as_float((a.w & 0xffu) << 23) * r.inv.x;
    s.sy = __uint_as_float((a.w & 0xff00u) << 15) * r.inv.y;
    s.sz = __uint_as_float((a.w & 0xff0000u) << 7) * r.inv.z;
    s.ox = __fmaf_rn(__uint_as_float(a.x) - r.o.x, r.inv.x, -s.sx);
    s.oy = __fmaf_rn(__uint_as_float(a.y) - r.o.y, r.inv.y, -s.sy);
    s.oz = __fmaf_rn(__uint_as_float(a.z) - r.o.z, r.inv.z, -s.sz);
    s.nx = kAny ? s.ox : s.ox - fabsf(r.margin * r.inv.x);
    s.ny = kAny ? s.oy : s.oy - fabsf(r.margin * r.inv.y);
    s.nz = kAny ? s.oz : s.oz - fabsf(r.margin * r.inv.z);
    s.cull = cull;
    bool px = r.oct4 & 1u, py = r.oct4 & 2u, pz = r.oct4 & 4u;
    uint32_t hits = 0;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        uint32_t meta = half ? b.w : b.z;
        uint32_t lx = half ? c0.y : c0.x, ly = half ? c0.w : c0.z, lz = half ? c1.y : c1.x;
        uint32_t hx = half ? c1.w : c1.z, hy = half ? c2.y : c2.x, hz = half ? c2.w : c2.z;
        uint32_t nx = px ? lx : hx, fx = px ? hx : lx;
        uint32_t ny = py ? ly : hy, fy = py ? hy : ly;
        uint32_t nz = pz ? lz : hz, fz = pz ? hz : lz;
        // bit position of each child: an internal child's slot bits are
        // exchanged by the ray's octant, a leaf child's entry stays (its
        // internal flag, bits 3 and 4 both set, is out of a leaf's range)
        uint32_t inner = (meta & (meta << 1) & 0x10101010u) >> 4;
        uint32_t position = (meta ^ (r.oct4 & (inner * 7u))) & 0x1f1f1f1fu;
        uint32_t bits = meta >> 5 & 0x07070707u;
        if (wide_child<0>(s, nx, ny, nz, fx, fy, fz)) hits |= (bits & 7u) << (position & 31u);
        if (wide_child<1>(s, nx, ny, nz, fx, fy, fz)) hits |= (bits >> 8 & 7u) << (position >> 8 & 31u);
        if (wide_child<2>(s, nx, ny, nz, fx, fy, fz)) hits |= (bits >> 16 & 7u) << (position >> 16 & 31u);
        if (wide_child<3>(s, nx, ny, nz, fx, fy, fz)) hits |= (bits >> 24 & 7u) << (position >> 24);
    }
    group = make_uint2(b.x, (hits & 0xff000000u) | a.w >> 24);
    leaves = make_uint2(b.y, hits & 0x00ffffffu);
}

// Takes the next child of a node group (its highest hit bit) and returns its
// node index.
WF_DEV uint32_t wide_next(uint2& group, uint32_t oct4) {
    uint32_t bit = 31u - uint32_t(__clz(int(group.y)));
    group.y &= ~(1u << bit);
    uint32_t slot = (bit - 24u) ^ (oct4 & 7u);
    return group.x + uint32_t(__popc(group.y & 0xffu & ((1u << slot) - 1u)));
}

// The triangle test on precomputed edges (intersect_triangle, wf_traverse.cuh).
WF_DEV bool intersect_edges(V3 o, V3 d, V3 v0, V3 e1, V3 e2, float& t, float& u, float& v) {
    V3 p = cross(d, e2);
    float det = dot(e1, p);
    float scale = fabsf(e1.x) * (fabsf(d.y * e2.z) + fabsf(d.z * e2.y)) +
                  fabsf(e1.y) * (fabsf(d.z * e2.x) + fabsf(d.x * e2.z)) +
                  fabsf(e1.z) * (fabsf(d.x * e2.y) + fabsf(d.y * e2.x));
    if (!isfinite(det) || fabsf(det) <= 8.0f * FLT_EPSILON * scale) return false;
    float inv = 1.0f / det;
    V3 ov = o - v0;
    u = dot(ov, p) * inv;
    if (u < 0.0f || u > 1.0f) return false;
    V3 q = cross(ov, e1);
    v = dot(d, q) * inv;
    if (v < 0.0f || u + v > 1.0f) return false;
    t = dot(e2, q) * inv;
    return t > kRayMinDistance;
}

// Whether the BVH2's own box of a triangle (its vertices' bounds) passes its
// slab test; `entry` is the box's entry distance.
WF_DEV bool exact_triangle_box(const DeviceScene& s, uint32_t ti, const WideRay& r, float closest_t, float& entry) {
    TriVerts t = load_triangle(s, ti);
    return slab(r.o, exact_inverse(r), fminf(fminf(t.v0.x, t.v1.x), t.v2.x), fmaxf(fmaxf(t.v0.x, t.v1.x), t.v2.x),
                fminf(fminf(t.v0.y, t.v1.y), t.v2.y), fmaxf(fmaxf(t.v0.y, t.v1.y), t.v2.y),
                fminf(fminf(t.v0.z, t.v1.z), t.v2.z), fmaxf(fmaxf(t.v0.z, t.v1.z), t.v2.z), closest_t, entry);
}
WF_DEV bool exact_leaf_box(float4 lo, float4 hi, const WideRay& r, float closest_t, float& entry) {
    return slab(r.o, exact_inverse(r), lo.x, hi.x, lo.y, hi.y, lo.z, hi.z, closest_t, entry);
}
// Whether a box with entry distance `entry`, grown by the ray's margin, starts
// past `cull` for certain (the margin moves no axis further than this).
WF_DEV bool box_past(float entry, const WideRay& r, float cull) {
    return entry > __fmaf_rn(r.margin, fmaxf(fabsf(r.inv.x), fmaxf(fabsf(r.inv.y), fabsf(r.inv.z))), cull);
}

// (By value: a lane's fields whose address is taken would live in memory.)
// The linear triangle lists (static triangles, and a direct list without a
// BVH), out of line: most scenes have neither, and their loops would cost
// the traversal registers (Tally::kLinearLists compiles them out).
template <typename Tally>
WF_CALL TraceState scan_closest(const DeviceScene& s, uint32_t first, uint32_t count, V3 o, V3 d, TraceState h,
                                Tally& tally) {
    for (uint32_t i = 0; i < count; ++i) {
        uint32_t ti = first + i;
        tally.triangle();
        TriVerts tri = load_triangle(s, ti);
        float t, u, v;
        if (!intersect_triangle(o, d, tri.v0, tri.v1, tri.v2, t, u, v) || t >= h.t) continue;
        if (alpha_rejects<Tally>(s, tri.material, ti, u, v)) continue;
        h.t = t;
        h.u = u;
        h.v = v;
        h.prim = make_prim(kHitTriangle, ti);
        h.inst = kInvalid;
    }
    return h;
}
template <typename Tally>
WF_CALL bool scan_any(const DeviceScene& s, uint32_t first, uint32_t count, V3 o, V3 d, float t_max, Tally& tally) {
    for (uint32_t i = 0; i < count; ++i) {
        tally.triangle();
        TriVerts tri = load_triangle(s, first + i);
        float t, u, v;
        if (intersect_triangle(o, d, tri.v0, tri.v1, tri.v2, t, u, v) && t < t_max &&
            !alpha_rejects<Tally>(s, tri.material, first + i, u, v))
            return true;
    }
    return false;
}
// Direct instances scan their mesh in original order (no BVH).
template <typename Tally>
WF_CALL TraceState direct_instances_closest(const DeviceScene& s, V3 o, V3 d, TraceState h, Tally& tally) {
    for (uint32_t i = 0; i < s.direct_instance_count; ++i)
        instance_closest(s, s.direct_instances[i], o, d, h, false, tally);
    return h;
}
template <typename Tally>
WF_CALL bool direct_instances_any(const DeviceScene& s, V3 o, V3 d, float t_max, Tally& tally) {
    for (uint32_t i = 0; i < s.direct_instance_count; ++i)
        if (instance_any(s, s.direct_instances[i], o, d, t_max, false, tally)) return true;
    return false;
}

// -------------------------------------------------------------- the lane
// One ray's traversal, a node or a leaf entry at a time.  The loop's live
// state is what bounds the kernels' occupancy (64 registers, 8 CTAs of 128
// per SM, without spills in the loop), so only what every step reads is in
// the struct's scalars: the hit record goes to the Sink as it is found, the
// world ray waits in memory while the lane is inside an instance, and the
// instance and its material are looked up when a hit needs them.
// kAny lanes (occlusion) keep t at the ray's length and stop at a hit.
struct Lane {
    WideRay r;      // ray of the current BVH (instance-local inside a BLAS)
    float t;        // closest hit so far; the ray's length (kAny)
    uint2 group;    // current node group: child base, hits << 24 | internal mask
    uint2 leaves;   // leaf entries to test: base, mask
    uint32_t state; // stage and the flags below
    uint32_t leaf;  // TLAS leaf entry of the current BLAS
    int size;       // stack entries
    float4 world[3];  // world ray: (o, inv.x) (d, inv.y) (inv.z, oct4, margin, entry of the TLAS leaf)
    uint2 stack[kLaneStack];
};
enum : uint32_t {
    kStageTlas = 0, kStageBlas = 1, kStageDirect = 2, kStageDone = 3, kStageMask = 3,
    kTie = 4,   // another candidate or the closest one's entry leaves the order a say
    kRedo = 8,  // the BVH2s must decide whatever comes
    kHit = 16,  // kAny: occluded
    kLate = 32  // the closest candidate's entry is past its distance
};

WF_DEV bool lane_done(const Lane& L) { return (L.state & kStageMask) == kStageDone; }
WF_DEV void lane_stage(Lane& L, uint32_t stage) { L.state = (L.state & ~kStageMask) | stage; }

// Where a closest hit's record goes: a local TraceState (one ray per call),
// or a queue entry's record in memory (the wavefront kernels).
struct StateSink {
    TraceState h;
    WF_DEV void hit(float t, float u, float v, uint32_t prim, uint32_t inst) {
        h.t = t;
        h.u = u;
        h.v = v;
        h.prim = prim;
        h.inst = inst;
    }
};
struct QueueSink {
    float4* hit_a;  // t, u, v, primitive
    uint32_t* hit_inst;
    uint32_t i;
    WF_DEV void hit(float t, float u, float v, uint32_t prim, uint32_t inst) {
        hit_a[i] = make_float4(t, u, v, __uint_as_float(prim));
        hit_inst[i] = inst;
    }
};
struct NoSink {
    WF_DEV void hit(float, float, float, uint32_t, uint32_t) {}
};

// The distance that a box's own test compares with: the ray's length, or none
// (lane_near weighs a closest hit's).
template <bool kAny>
WF_DEV float box_limit(const Lane& L) {
    return kAny ? L.t : 1.0e30f;
}

// A closest-hit candidate at distance t <= L.t * kNear whose boxes start at
// `entry`: returns whether it is the closest one so far.  A new closest one
// is certain when it and its entry lie before the former closest, and so
// before every other, and the entry within the reach of what is seen; it stays
// so until another turns up at its distance, or (kLate) maybe before its
// entry.
WF_DEV bool lane_near(Lane& L, float t, float entry) {
    if (t >= L.t) {
        if ((L.state & kLate) || t == L.t) L.state |= kTie;
        return false;
    }
    L.state &= ~(kTie | kLate);
    if (entry > t) L.state |= kLate;
    if (fmaxf(t, entry) >= L.t || entry > t * kNear) L.state |= kTie;
    L.t = t;
    return true;
}

// Starts the TLAS or the direct list's BVH (each the only tree over its kind
// of leaf entries, so a tree of one leaf has entry 0).
WF_DEV void lane_root(Lane& L, const BvhRef& tree) {
    if (tree.root >= 0) {
        L.group = make_uint2(tree.wide, 0x80000000u);  // no internal mask: wide_next returns the base
        L.leaves = make_uint2(0u, 0u);
    } else {  // one leaf, whose box is the root box that was just tested
        L.group = make_uint2(0u, 0u);
        L.leaves = make_uint2(0u, 1u);
    }
}

WF_DEV void lane_occluded(Lane& L) { L.state |= kHit | kStageDone; }

WF_DEV void lane_save_world(Lane& L) {
    L.world[0] = make_float4(L.r.o.x, L.r.o.y, L.r.o.z, L.r.inv.x);
    L.world[1] = make_float4(L.r.d.x, L.r.d.y, L.r.d.z, L.r.inv.y);
    L.world[2] = make_float4(L.r.inv.z, __uint_as_float(L.r.oct4), L.r.margin, 0.0f);
}
WF_DEV void lane_restore_world(Lane& L) {
    float4 a = L.world[0], b = L.world[1], c = L.world[2];
    L.r.o = f4xyz(a);
    L.r.d = f4xyz(b);
    L.r.inv = V3{a.w, b.w, c.x};
    L.r.oct4 = __float_as_uint(c.y);
    L.r.margin = c.z;
}

// A triangle of the current BVH hit at distance t.
template <bool kAny, typename Tally, typename Sink>
WF_DEV void lane_candidate(Lane& L, const DeviceScene& s, Sink& sink, uint32_t ti, uint32_t material, float t, float u,
                           float v) {
    bool blas = (L.state & kStageMask) == kStageBlas;
    if (s.any_alpha_reject) {
        if (blas) {
            uint32_t over = __float_as_uint(__ldg(&s.wide.leaves[L.leaf].root_lo.w));
            if (over != kInvalid) material = over;
        }
        if (alpha_rejects<Tally>(s, material, ti, u, v)) return;
    }
    float entry;
    if (!exact_triangle_box(s, ti, L.r, box_limit<kAny>(L), entry)) return;
    if (kAny) {
        lane_occluded(L);
        return;
    }
    if (blas) entry = fmaxf(entry, L.world[2].w);
    if (!lane_near(L, t, entry)) return;
    uint32_t inst = blas ? __float_as_uint(__ldg(&s.wide.leaves[L.leaf].lo.w)) : kInvalid;
    sink.hit(t, u, v, make_prim(blas ? kHitMesh : kHitTriangle, ti), inst);
}

// Direct triangle list (last stage of traceRay / isOccluded): the lane
// traverses its BVH; a list without one is scanned by lane_finish.
template <bool kAny>
WF_DEV void lane_begin_direct(Lane& L, const DeviceScene& s) {
    lane_stage(L, kStageDone);
    if (s.direct_count == 0 || s.direct_bvh.root == kNoRoot) return;
    float near_t;
    if (!slab_box(L.r.o, exact_inverse(L.r), s.direct_bvh.box, box_limit<kAny>(L), near_t)) return;
    if (!kAny) L.r.margin = cull_margin(L.r.o, s.direct_bvh.box, kWideReach, 0.0f);
    lane_stage(L, kStageDirect);
    lane_root(L, s.direct_bvh);
}

// Starts a ray: the linear stages of traceRay / isOccluded, then the TLAS
// root.  t_max: a kAny ray's length.  Rays and scenes that the wide test does
// not cover go to the BVH2s before the linear stages, which those repeat.
template <bool kAny, typename Tally, typename Sink>
WF_DEV void lane_begin(Lane& L, const DeviceScene& s, Sink& sink, V3 o, V3 d, float t_max, Tally& tally) {
    L.state = kStageDone;
    L.t = t_max;
    L.size = 0;
    L.world[0] = make_float4(o.x, o.y, o.z, 0.0f);
    L.world[1] = make_float4(d.x, d.y, d.z, 0.0f);
    if (!s.wide.usable || !ray_covered(o, d)) {
        L.state |= kRedo;
        return;
    }
    if (kAny) {
        for (uint32_t i = 0; i < s.direct_sphere_count; ++i) {
            float t;
            tally.sphere();
            if (intersect_sphere(o, d, __ldg(&s.spheres[s.direct_spheres[i]]), t) && t < t_max) L.state |= kHit;
        }
        if constexpr (Tally::kLinearLists) {
            if (s.direct_instance_count && direct_instances_any(s, o, d, t_max, tally)) L.state |= kHit;
            if (s.static_count && scan_any(s, s.static_first, s.static_count, o, d, t_max, tally)) L.state |= kHit;
        }
        if (L.state & kHit) return;
    } else {
        TraceState h;
        trace_state_init(h, 1e30f);
        for (uint32_t i = 0; i < s.direct_sphere_count; ++i) sphere_closest(s, s.direct_spheres[i], o, d, h, tally);
        if constexpr (Tally::kLinearLists) {
            if (s.direct_instance_count) h = direct_instances_closest(s, o, d, h, tally);
            if (s.static_count) h = scan_closest(s, s.static_first, s.static_count, o, d, h, tally);
        }
        L.t = h.t;
        sink.hit(h.t, h.u, h.v, h.prim, h.inst);
    }
    wide_ray(L.r, o, d);
    // (the TLAS's; lane_begin_direct has its own BVH's)
    if (!kAny) L.r.margin = cull_margin(o, s.tlas.box, s.wide.reach, s.wide.base);
    if (s.tlas.root != kNoRoot) {
        lane_save_world(L);
        float near_t;
        if (slab_box(o, exact_inverse(L.r), s.tlas.box, box_limit<kAny>(L), near_t)) {
            lane_stage(L, kStageTlas);
            lane_root(L, s.tlas);
            return;
        }
    }
    lane_begin_direct<kAny>(L, s);
}

// Pops the next group; at the mark below a BLAS's groups the lane is back in
// the TLAS, at the bottom the BVH is finished (TLAS -> direct -> done).
template <bool kAny>
WF_DEV void lane_pop(Lane& L, const DeviceScene& s) {
    if (L.size == 0) {
        if ((L.state & kStageMask) == kStageTlas) lane_begin_direct<kAny>(L, s);
        else lane_stage(L, kStageDone);
        return;
    }
    uint2 e = L.stack[--L.size];
    if (e.y == 0) {
        lane_stage(L, kStageTlas);
        lane_restore_world(L);
        if (L.size == 0) return;
        e = L.stack[--L.size];
    }
    if (e.y & 0xff000000u) L.group = e; else L.leaves = e;
}

// One TLAS leaf: a sphere test, or entry into an instance's BLAS.
template <bool kAny, typename Tally, typename Sink>
WF_DEV void lane_tlas_leaf(Lane& L, const DeviceScene& s, Sink& sink, uint32_t entry, Tally& tally) {
    const float4* rec = reinterpret_cast<const float4*>(s.wide.leaves + entry);
    float4 lo = __ldg(rec + 3), hi = __ldg(rec + 4), x = __ldg(rec);
    uint32_t word = __float_as_uint(lo.w);
    float near_t;
    if (!exact_leaf_box(lo, hi, L.r, box_limit<kAny>(L), near_t)) return;
    if (word & 0x80000000u) {
        float t;
        tally.sphere();
        if (!intersect_sphere(L.r.o, L.r.d, x, t)) return;
        if (kAny) {
            if (t < L.t) lane_occluded(L);
            return;
        }
        // (equal distances among spheres go by their index: a tie too)
        if (t <= L.t * kNear && lane_near(L, t, near_t))
            sink.hit(t, 0.0f, 0.0f, make_prim(kHitSphere, word & 0x7fffffffu), kInvalid);
        return;
    }
    if (!kAny && box_past(near_t, L.r, L.t * kSlack)) return;
    tally.instance();
    Instance in;
    in.w2l_x = x;
    in.w2l_y = __ldg(rec + 1);
    in.w2l_z = __ldg(rec + 2);
    float4 root_lo = __ldg(rec + 5), root_hi = __ldg(rec + 6);
    uint32_t root = __float_as_uint(hi.w);
    if (root == kNoWide) {  // a mesh without a BVH: the BVH2 path scans it
        L.state |= kRedo;
        return;
    }
    wide_ray(L.r, to_local_vector(in, L.r.o - instance_translation(in)), to_local_vector(in, L.r.d));
    bool covered = ray_covered(L.r.o, L.r.d);
    if (!kAny) L.r.margin = cull_margin(L.r.o, f4xyz(root_lo), f4xyz(root_hi), kWideReach, 0.0f);
    float local_t;
    if (!covered || !exact_leaf_box(root_lo, root_hi, L.r, box_limit<kAny>(L), local_t) ||
        (!kAny && box_past(local_t, L.r, L.t * kSlack))) {
        if (!covered) L.state |= kRedo;  // a scale the wide test's bounds do not cover
        lane_restore_world(L);
        return;
    }
    if (!kAny) L.world[2].w = near_t;
    // what is left of this TLAS node waits below the BLAS's groups, under a mark
    if (L.group.y & 0xff000000u) L.stack[L.size++] = L.group;
    if (L.leaves.y) L.stack[L.size++] = L.leaves;
    L.stack[L.size++] = make_uint2(0u, 0u);
    L.leaf = entry;
    lane_stage(L, kStageBlas);
    L.group = make_uint2(root, 0x80000000u);
    L.leaves = make_uint2(0u, 0u);
}

// Pops a group if there is none left, and visits a node; leaf entries that
// it leaves wait for lane_triangle / lane_tlas_leaf.
template <bool kAny, typename Tally>
WF_DEV void lane_node(Lane& L, const DeviceScene& s, Tally& tally) {
    if (!L.leaves.y && !(L.group.y & 0xff000000u)) lane_pop<kAny>(L, s);
    if (!L.leaves.y && (L.group.y & 0xff000000u)) {
        uint2 rest = L.group;
        uint32_t node = wide_next(rest, L.r.oct4);
        if (rest.y & 0xff000000u) L.stack[L.size++] = rest;
        tally.node();
        float slack = !kAny && (L.state & kStageMask) == kStageTlas ? s.wide.slack : kSlack;
        wide_node<kAny>(s.wide.nodes, node, L.r, L.t * slack, L.group, L.leaves);
    }
}

// Takes the next leaf entry (leaves.y != 0).
WF_DEV uint32_t lane_entry(Lane& L) {
    uint32_t k = uint32_t(__ffs(int(L.leaves.y))) - 1u;
    L.leaves.y &= L.leaves.y - 1u;
    return L.leaves.x + k;
}
WF_DEV bool lane_in_tlas(const Lane& L) { return (L.state & kStageMask) == kStageTlas; }

// The next leaf entry of a triangle BVH.
template <bool kAny, typename Tally, typename Sink>
WF_DEV void lane_triangle(Lane& L, const DeviceScene& s, Sink& sink, Tally& tally) {
    const float4* rec = reinterpret_cast<const float4*>(s.wide.triangles + lane_entry(L));
    float4 v0 = __ldg(rec), e1 = __ldg(rec + 1), e2 = __ldg(rec + 2);
    tally.triangle();
    float t, u, v;
    if (intersect_edges(L.r.o, L.r.d, f4xyz(v0), f4xyz(e1), f4xyz(e2), t, u, v) &&
        (kAny ? t < L.t : t <= L.t * kNear))
        lane_candidate<kAny, Tally>(L, s, sink, __float_as_uint(v0.w), __float_as_uint(e1.w), t, u, v);
}

// One step of one ray: a node, then one leaf entry if there is any.  (Leaf
// entries that wait until 4, 8 or 12 lanes of the warp hold one cost more
// than they save: 1080p mesh +0 / +2 / +10 %, sphere field +4 / +7 / +12 %.)
template <bool kAny, typename Tally, typename Sink>
WF_DEV void lane_step(Lane& L, const DeviceScene& s, Sink& sink, Tally& tally) {
    lane_node<kAny>(L, s, tally);
    if (!L.leaves.y) return;
    if (lane_in_tlas(L))
        lane_tlas_leaf<kAny>(L, s, sink, lane_entry(L), tally);
    else
        lane_triangle<kAny>(L, s, sink, tally);
}

// Whether the finished ray's answer could depend on the visit order, or it
// met something the wide test does not cover: trace_closest_binary /
// trace_any_binary decide it.  The kernels that refill their lanes do that
// after their loop: a call inside it would cost the loop some 20 registers
// of spills.
WF_DEV bool lane_doubt(const Lane& L) { return (L.state & (kTie | kRedo)) && !(L.state & kHit); }

// Called once when the lane is done: the linear scan of a direct list
// without a BVH.
template <bool kAny, typename Tally, typename Sink>
WF_DEV void lane_finish(Lane& L, const DeviceScene& s, Sink& sink, Tally& tally) {
    if constexpr (Tally::kLinearLists) {
        if (s.direct_count == 0 || s.direct_bvh.root != kNoRoot || (L.state & (kTie | kRedo | kHit))) return;
        V3 o = f4xyz(L.world[0]), d = f4xyz(L.world[1]);
        if (kAny) {
            if (scan_any(s, s.direct_first, s.direct_count, o, d, L.t, tally)) L.state |= kHit;
            return;
        }
        TraceState h;
        trace_state_init(h, L.t);
        h = scan_closest(s, s.direct_first, s.direct_count, o, d, h, tally);
        if (h.t < L.t) sink.hit(h.t, h.u, h.v, h.prim, h.inst);
    }
}

// ------------------------------------------------- one ray to its end
// (Without a warp vote: keeping the lanes together by one at every step costs
// the inverse step 3 %, 9.00 against 8.70 ms, and small ray batches 2-4 %.)
template <bool kAny, typename Tally, typename Sink>
WF_DEV bool lane_run(Lane& L, const DeviceScene& s, Sink& sink, V3 o, V3 d, float t_max, Tally& tally) {
    lane_begin<kAny>(L, s, sink, o, d, t_max, tally);
    while (!lane_done(L)) lane_step<kAny>(L, s, sink, tally);
    lane_finish<kAny>(L, s, sink, tally);
    if (!lane_doubt(L)) return (L.state & kHit) != 0;
    V3 wo = f4xyz(L.world[0]), wd = f4xyz(L.world[1]);
    if (kAny) return trace_any_binary(s, wo, wd, t_max, tally);
    TraceState h = trace_closest_binary(s, wo, wd, tally);
    sink.hit(h.t, h.u, h.v, h.prim, h.inst);
    return false;
}

// traceRay, device_traversal.cuh:1115-1150.
template <typename Tally>
WF_DEV TraceState trace_closest(const DeviceScene& s, V3 o, V3 d, Tally& tally) {
    Lane L;
    StateSink sink;
    lane_run<false>(L, s, sink, o, d, 1e30f, tally);
    return sink.h;
}

// isOccluded, device_traversal.cuh:1035-1113.
template <typename Tally>
WF_DEV bool trace_any(const DeviceScene& s, V3 o, V3 d, float t_max, Tally& tally) {
    Lane L;
    NoSink sink;
    return lane_run<true>(L, s, sink, o, d, t_max, tally);
}

// The same out of line, for kernels that do much else between rays: the
// traversal loop gets the registers to itself and the caller's state is
// saved once per ray instead of being spilled inside the loop.
template <typename Tally>
WF_CALL TraceState trace_closest_call(const DeviceScene& s, V3 o, V3 d, Tally& tally) {
    return trace_closest(s, o, d, tally);
}
template <typename Tally>
WF_CALL bool trace_any_call(const DeviceScene& s, V3 o, V3 d, float t_max, Tally& tally) {
    return trace_any(s, o, d, t_max, tally);
}

}  // namespace wf
