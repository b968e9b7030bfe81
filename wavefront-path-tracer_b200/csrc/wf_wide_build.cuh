// How a wide node is made from the BVH2 nodes below it (host and device code:
// the kernels of wf_wide_build.cu, and a host build of the same functions in
// the tests).
#pragma once

#include <cmath>
#include <cstring>

#include "wf_device.cuh"

namespace wf {

constexpr int kWide = 8;
// Triangles of the largest leaf child: 2 (the format holds 3).  Against 1 and
// 3 the Cornell box renders 9 % and 0 % faster, the 1080p mesh 0.6 % and
// 0.5 %, the sphere field 0 % and 1 %.  TLAS leaves stay single: an instance
// entry costs far more than a box test.
constexpr int kLeafTriangles = 2;
// A work item is the BVH2 ref a wide node stands for.
constexpr uint32_t kTlasItem = 0x40000000u;  // flag: the node belongs to the TLAS
constexpr uint32_t kLeafItem = 0x80000000u;  // flag: the ref is ~leaf (a tree of one leaf)

struct Child {
    int ref;
    float lo[3], hi[3];
};

WF_HDI float child_area(const Child& c) {
    float x = c.hi[0] - c.lo[0], y = c.hi[1] - c.lo[1], z = c.hi[2] - c.lo[2];
    return x * y + y * z + z * x;
}

WF_HDI void load_pair(const BvhNode* nodes, int ref, Child& l, Child& r) {
    const BvhNode n = nodes[ref];
    l.ref = n.child.x;
    l.lo[0] = n.lxy.x; l.hi[0] = n.lxy.y; l.lo[1] = n.lxy.z; l.hi[1] = n.lxy.w; l.lo[2] = n.lrz.x; l.hi[2] = n.lrz.y;
    r.ref = n.child.y;
    r.lo[0] = n.rxy.x; r.hi[0] = n.rxy.y; r.lo[1] = n.rxy.z; r.hi[1] = n.rxy.w; r.lo[2] = n.lrz.z; r.hi[2] = n.lrz.w;
}

// Leaves below `ref`, up to kLeafTriangles, written to `out` in the BVH2's
// depth-first order; returns kLeafTriangles + 1 when there are more.
WF_HDI int small_leaves(const BvhNode* nodes, int ref, int out[kLeafTriangles]) {
    int stack[kLeafTriangles + 1], size = 0, count = 0;
    stack[size++] = ref;
    while (size > 0) {
        int r = stack[--size];
        if (r < 0) {
            if (count == kLeafTriangles) return kLeafTriangles + 1;
            out[count++] = ~r;
        } else {
            // every entry on the stack holds at least one more leaf
            if (size + count + 2 > kLeafTriangles) return kLeafTriangles + 1;
            stack[size++] = nodes[r].child.y;
            stack[size++] = nodes[r].child.x;
        }
    }
    return count;
}

// The children of the wide node over BVH2 ref `ref` by slot (count[slot] = 0
// empty, -1 internal, else leaf entries).  The slots order the children
// along the eight octant directions: slot bit a is set for children on the
// positive side of axis a, assigned greedily by the largest projection.
struct Collapsed {
    Child child[kWide];
    int count[kWide];
    int leaf[kWide][kLeafTriangles];
    int internal, leaves;
};

// `root`: the tree's root box, read for a tree of one leaf only.
WF_HDI void collapse(const BvhNode* nodes, uint32_t item, const BvhRef* root, Collapsed& out) {
    bool tlas = (item & kTlasItem) != 0;
    int ref = (item & kLeafItem) ? ~int(item & 0x3fffffffu) : int(item & 0x3fffffffu);
    Child c[kWide];
    int n;
    if (ref < 0) {  // a tree of one leaf: its root box
        c[0].ref = ref;
        for (int a = 0; a < 3; ++a) {
            c[0].lo[a] = root->box.lo[a];
            c[0].hi[a] = root->box.hi[a];
        }
        n = 1;
    } else {
        load_pair(nodes, ref, c[0], c[1]);
        n = 2;
    }
    while (n < kWide) {
        int best = -1;
        float best_area = -1.0f;
        for (int k = 0; k < n; ++k)
            if (c[k].ref >= 0 && child_area(c[k]) > best_area) {
                best_area = child_area(c[k]);
                best = k;
            }
        if (best < 0) break;
        Child l, r;
        load_pair(nodes, c[best].ref, l, r);
        c[best] = l;
        c[n++] = r;
    }
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int k = 0; k < n; ++k)
        for (int a = 0; a < 3; ++a) {
            lo[a] = fminf(lo[a], c[k].lo[a]);
            hi[a] = fmaxf(hi[a], c[k].hi[a]);
        }
    for (int slot = 0; slot < kWide; ++slot) out.count[slot] = 0;
    unsigned free_slots = 0xffu, left = (1u << n) - 1u;
    for (int round = 0; round < n; ++round) {
        int bk = -1, bs = -1;
        float best = -INFINITY;
        for (int k = 0; k < n; ++k) {
            if (!(left >> k & 1u)) continue;
            float d[3];
            for (int a = 0; a < 3; ++a) d[a] = (c[k].lo[a] + c[k].hi[a]) - (lo[a] + hi[a]);
            for (int slot = 0; slot < kWide; ++slot) {
                if (!(free_slots >> slot & 1u)) continue;
                float v = (slot & 1 ? d[0] : -d[0]) + (slot & 2 ? d[1] : -d[1]) + (slot & 4 ? d[2] : -d[2]);
                if (bk < 0 || v > best) {
                    best = v;
                    bk = k;
                    bs = slot;
                }
            }
        }
        left &= ~(1u << bk);
        free_slots &= ~(1u << bs);
        out.child[bs] = c[bk];
        int entries[kLeafTriangles];
        int m = 1;
        if (c[bk].ref < 0) {
            out.leaf[bs][0] = ~c[bk].ref;
        } else {
            m = tlas ? kLeafTriangles + 1 : small_leaves(nodes, c[bk].ref, entries);
            if (m <= kLeafTriangles)
                for (int k = 0; k < m; ++k) out.leaf[bs][k] = entries[k];
        }
        out.count[bs] = m <= kLeafTriangles ? m : -1;
    }
    out.internal = out.leaves = 0;
    for (int slot = 0; slot < kWide; ++slot) {
        if (out.count[slot] < 0) ++out.internal;
        else out.leaves += out.count[slot];
    }
}

// Numbers the children of the wide node that `item` stands for: the first
// entries of its internal children (appended to `items`) and of its leaves.
// add(k, n) adds n to counter k and returns what it held: [0] nodes, [1]
// triangles, [2] TLAS leaves.  `fits`: whether its boxes are in the range of
// the ray test.
template <typename Add>
WF_HDI uint2 number_children(const BvhNode* nodes, uint32_t item, const BvhRef* root, uint32_t* items, Add add,
                             bool& fits) {
    bool tlas = (item & kTlasItem) != 0;
    Collapsed c;
    collapse(nodes, item, root, c);
    uint32_t base = c.internal ? add(0, uint32_t(c.internal)) : 0u;
    uint32_t leaf_base = c.leaves ? add(tlas ? 2 : 1, uint32_t(c.leaves)) : 0u;
    fits = true;
    uint32_t next = base;
    for (int slot = 0; slot < kWide; ++slot) {
        if (c.count[slot] == 0) continue;
        for (int a = 0; a < 3; ++a)
            fits = fits && fabsf(c.child[slot].lo[a]) <= kWideMaxCoordinate &&
                   fabsf(c.child[slot].hi[a]) <= kWideMaxCoordinate;
        if (c.count[slot] < 0) items[next++] = uint32_t(c.child[slot].ref) | (tlas ? kTlasItem : 0u);
    }
    return make_uint2(base, leaf_base);
}

// The first items: the roots of the trees.
WF_HDI uint32_t root_item(const BvhRef& tree, bool tlas) {
    return (tree.root < 0 ? (kLeafItem | uint32_t(~tree.root)) : uint32_t(tree.root)) | (tlas ? kTlasItem : 0u);
}

// Grid of one axis: cells of 2^e with 252 of them at least as long as the
// node, no finer than the rounding of its coordinates, 2^-20 of its longest
// side or 1e-9 (the ray test's bounds, wf_wide.cuh); the origin lies one
// cell below the node.
WF_HDI void axis_grid(float lo, float hi, float longest, float& origin, int& exponent) {
    float cell = fmaxf((hi - lo) * (1.0f / 252.0f), fmaxf(fabsf(lo), fabsf(hi)) * 2.384185791015625e-7f);
    cell = fmaxf(cell, fmaxf(longest * 9.5367431640625e-7f, 1.0e-9f));
    int e;
    float m = frexpf(cell, &e);  // cell = m 2^e, m in [0.5, 1)
    if (m == 0.5f) --e;
    // the byte that holds e + 142; boxes past the range make the scene unusable anyway
    exponent = e < -141 ? -141 : (e > 112 ? 112 : e);
    e = exponent;
    float step = ldexpf(1.0f, e);
    origin = lo - step;  // rounded down
    if (double(origin) > double(lo) - double(step)) origin = nextafterf(origin, -INFINITY);
}

// Planes with 1/64 cell to spare on either side (the ray test's rounding).
WF_HDI uint32_t plane_lo(float v, float origin, int exponent) {
    double q = floor(ldexp(double(v) - double(origin), -exponent) - 1.0 / 64.0);
    return uint32_t(fmin(fmax(q, 0.0), 255.0));
}
WF_HDI uint32_t plane_hi(float v, float origin, int exponent) {
    double q = ceil(ldexp(double(v) - double(origin), -exponent) + 1.0 / 64.0);
    return uint32_t(fmin(fmax(q, 0.0), 255.0));
}

WF_HDI float bits_to_float(uint32_t u) {
    float f;
    memcpy(&f, &u, 4);
    return f;
}

// The node's record; its leaf entries go to `triangles` or (TLAS) `leaves`
// from leaf_base on.
WF_HDI WideNode wide_record(const DeviceScene& s, const Collapsed& c, bool tlas, uint32_t child_base,
                            uint32_t leaf_base, WideTriangle* triangles, WideLeaf* leaves) {
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int slot = 0; slot < kWide; ++slot) {
        if (c.count[slot] == 0) continue;
        for (int a = 0; a < 3; ++a) {
            lo[a] = fminf(lo[a], c.child[slot].lo[a]);
            hi[a] = fmaxf(hi[a], c.child[slot].hi[a]);
        }
    }
    float longest = fmaxf(hi[0] - lo[0], fmaxf(hi[1] - lo[1], hi[2] - lo[2]));
    float origin[3];
    int exponent[3];
    for (int a = 0; a < 3; ++a) axis_grid(lo[a], hi[a], longest, origin[a], exponent[a]);
    WideNode n;
    n.px = origin[0];
    n.py = origin[1];
    n.pz = origin[2];
    n.scale = 0;
    for (int a = 0; a < 3; ++a) n.scale |= uint32_t(exponent[a] + 15 + 127) << (8 * a);
    n.child_base = child_base;
    n.leaf_base = leaf_base;
    n.meta[0] = n.meta[1] = 0;
    for (int k = 0; k < 12; ++k) n.planes[k] = 0;
    uint32_t entry = 0;
    for (int slot = 0; slot < kWide; ++slot) {
        int m = c.count[slot];
        if (m == 0) continue;
        const Child& ch = c.child[slot];
        uint32_t meta;
        if (m < 0) {
            n.scale |= 1u << (24 + slot);
            meta = 0x20u | uint32_t(24 + slot);
        } else {
            meta = ((1u << m) - 1u) << 5 | entry;
        }
        int w = slot >> 2, shift = 8 * (slot & 3);
        n.meta[w] |= meta << shift;
        for (int a = 0; a < 3; ++a) {
            n.planes[2 * a + w] |= plane_lo(ch.lo[a], origin[a], exponent[a]) << shift;
            n.planes[6 + 2 * a + w] |= plane_hi(ch.hi[a], origin[a], exponent[a]) << shift;
        }
        for (int k = 0; k < m; ++k, ++entry) {
            if (tlas) {
                uint32_t word = s.tlas_leaves[c.leaf[slot][k]];
                WideLeaf leaf;
                memset(&leaf, 0, sizeof(leaf));
                leaf.lo = make_float4(ch.lo[0], ch.lo[1], ch.lo[2], bits_to_float(word));
                leaf.hi = make_float4(ch.hi[0], ch.hi[1], ch.hi[2], bits_to_float(kNoWide));
                if (word & 0x80000000u) {
                    leaf.x = s.spheres[word & 0x7fffffffu];
                } else {
                    const Instance& in = s.instances[word];
                    const Blas& b = s.blases[in.blas];
                    leaf.x = in.w2l_x;
                    leaf.y = in.w2l_y;
                    leaf.z = in.w2l_z;
                    leaf.hi.w = bits_to_float(b.bvh.root == kNoRoot ? kNoWide : b.bvh.wide);
                    leaf.root_lo = make_float4(b.bvh.box.lo[0], b.bvh.box.lo[1], b.bvh.box.lo[2],
                                               bits_to_float(in.material_override));
                    leaf.root_hi = make_float4(b.bvh.box.hi[0], b.bvh.box.hi[1], b.bvh.box.hi[2], 0.0f);
                }
                leaves[n.leaf_base + entry] = leaf;
            } else {
                uint32_t ti = uint32_t(c.leaf[slot][k]);
                float4 a = s.triangles[3 * size_t(ti)], b = s.triangles[3 * size_t(ti) + 1],
                       d = s.triangles[3 * size_t(ti) + 2];
                WideTriangle t;
                t.v0 = make_float4(a.x, a.y, a.z, bits_to_float(ti));
                t.e1 = make_float4(b.x - a.x, b.y - a.y, b.z - a.z, b.w);
                t.e2 = make_float4(d.x - a.x, d.y - a.y, d.z - a.z, 0.0f);
                triangles[n.leaf_base + entry] = t;
            }
        }
    }
    return n;
}

}  // namespace wf
