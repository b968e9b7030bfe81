// Host build of the wide BVH's construction and traversal (wf_wide_build.cuh,
// wf_wide.cuh) for tests/test_wide_bvh.py: every ray of a batch is traced by
// the wide traversal and by the BVH2 traversal of the same scene.
#include "host_shims.h"

#include "wf_internal.h"
#include "wf_bvh_gpu.h"
#include "wf_wide.cuh"
#include "wf_wide_build.cuh"

namespace wf {
bool build_binary_bvh_gpu(const BvhBox*, uint32_t, std::vector<BvhBinaryNode>&, int, char*, size_t, int) {
    return false;
}
}  // namespace wf

using namespace wf;

namespace {
struct Built {
    HostScene h;
    DeviceScene v{};
    std::vector<WideNode> nodes;
    std::vector<WideTriangle> triangles;
    std::vector<WideLeaf> leaves;
};

void build_wide(Built& b) {
    std::vector<BvhRef> trees;
    auto number = [&](BvhRef& r) {
        if (r.root == kNoRoot) return;
        r.wide = uint32_t(trees.size());
        trees.push_back(r);
    };
    for (Blas& x : b.h.blases) number(x.bvh);
    number(b.h.direct_bvh);
    number(b.h.tlas);
    // as build_wide_bvh: one node at a time, with room for every BVH2 node
    uint32_t counters[3] = {uint32_t(trees.size()), 0, 0};
    std::vector<uint32_t> items(b.h.nodes.size() + trees.size());
    for (uint32_t i = 0; i < trees.size(); ++i) items[i] = root_item(trees[i], i == b.h.tlas.wide);
    bool usable = b.h.margins.usable != 0;
    std::vector<uint2> bases;
    for (uint32_t i = 0; i < counters[0]; ++i) {
        bool fits;
        bases.push_back(number_children(
            b.h.nodes.data(), items[i], trees.data() + i, items.data(),
            [&](int k, uint32_t n) { uint32_t old = counters[k]; counters[k] += n; return old; }, fits));
        usable = usable && fits;
    }
    items.resize(counters[0]);
    DeviceScene& v = b.v;
    v.triangles = b.h.triangles.data();
    v.nodes = b.h.nodes.data();
    v.blases = b.h.blases.data();
    v.instances = b.h.instances.data();
    v.mesh_linear = b.h.mesh_linear.data();
    v.tlas_leaves = b.h.tlas_leaves.data();
    v.spheres = b.h.spheres.data();
    v.direct_spheres = b.h.direct_spheres.data();
    v.direct_instances = b.h.direct_instances.data();
    v.materials = b.h.materials.data();
    v.material_textures = b.h.material_textures.empty() ? nullptr : b.h.material_textures.data();
    v.texels = b.h.texels.data();
    v.textures = b.h.textures.data();
    v.tri_attr = b.h.tri_attr.empty() ? nullptr : b.h.tri_attr.data();
    v.texture_count = uint32_t(b.h.textures.size());
    v.tlas = b.h.tlas;
    v.direct_bvh = b.h.direct_bvh;
    v.static_first = b.h.static_first;
    v.static_count = b.h.static_count;
    v.direct_first = b.h.direct_first;
    v.direct_count = b.h.direct_count;
    v.direct_sphere_count = uint32_t(b.h.direct_spheres.size());
    v.direct_instance_count = uint32_t(b.h.direct_instances.size());
    v.any_alpha_reject = b.h.any_alpha_reject ? 1u : 0u;
    v.wide = b.h.margins;
    b.triangles.resize(counters[1]);
    b.leaves.resize(counters[2]);
    for (uint32_t i = 0; i < items.size(); ++i) {
        Collapsed c;
        collapse(v.nodes, items[i], trees.data() + i, c);
        b.nodes.push_back(wide_record(v, c, (items[i] & kTlasItem) != 0, bases[i].x, bases[i].y, b.triangles.data(),
                                      b.leaves.data()));
    }
    v.wide.nodes = b.nodes.data();
    v.wide.triangles = b.triangles.data();
    v.wide.leaves = b.leaves.data();
    v.wide.usable = usable ? 1u : 0u;
}
}  // namespace

// counts: [0] closest hits that differ, [1] occlusion answers that differ,
// [2] rays, [3] wide nodes, [4] wide node visits, [5] BVH2 node visits,
// [6] usable, [7] rays that the BVH2s decided, [8] hits, [9] and [10]
// primitive and instance tests of the wide and the BVH2 closest hits
extern "C" int wide_check(const wf_scene_desc* desc, const wf_ray* rays, const float* limits, uint32_t count,
                          uint64_t* counts) {
    Built b;
    if (wf_status e = build_host_scene(desc, b.h)) return int(e);
    build_wide(b);
    for (int k = 0; k < 11; ++k) counts[k] = 0;
    counts[2] = count;
    counts[3] = b.nodes.size();
    counts[6] = b.v.wide.usable;
    for (uint32_t i = 0; i < count; ++i) {
        V3 o{rays[i].origin[0], rays[i].origin[1], rays[i].origin[2]};
        V3 d{rays[i].direction[0], rays[i].direction[1], rays[i].direction[2]};
        CountTally steps, wide, wide_any, binary, unused;
        TraceState x, y;
        Lane lane;
        StateSink sink;
        lane_begin<false>(lane, b.v, sink, o, d, 1e30f, steps);
        while (!lane_done(lane)) lane_step<false>(lane, b.v, sink, steps);
        if (lane_doubt(lane)) ++counts[7];
        x = trace_closest(b.v, o, d, wide);
        y = trace_closest_binary(b.v, o, d, binary);
        // u and v mean something for triangles only, the instance for meshes
        uint32_t kind = hit_kind(y.prim);
        bool triangle = kind == kHitMesh || kind == kHitTriangle;
        if (x.prim != y.prim || std::memcmp(&x.t, &y.t, triangle ? 12 : 4) != 0 ||
            (kind == kHitMesh && x.inst != y.inst))
            ++counts[0];
        if (kind != kHitMiss) ++counts[8];
        bool p = trace_any(b.v, o, d, limits[i], wide_any), q = trace_any_binary(b.v, o, d, limits[i], unused);
        if (p != q) ++counts[1];
        counts[4] += wide.nodes;
        counts[5] += binary.nodes;
        counts[9] += wide.triangles + wide.spheres + wide.instances;
        counts[10] += binary.triangles + binary.spheres + binary.instances;
    }
    return 0;
}
