// Collapses the scene's BVH2s into compressed 8-wide nodes on the GPU.
//
// One thread per wide node, level by level: a wide node starts with the two
// children of its BVH2 node and opens its largest internal child (by box
// area) until it has eight; what is left of at most kLeafTriangles triangles
// becomes a leaf child.  The first pass numbers the nodes (each node's
// internal children are contiguous) and counts the leaf entries, the second
// writes the nodes, the triangles in leaf order and the TLAS leaf records, so
// no array is larger than it has to be.  Bound by the random reads of the
// BVH2 nodes (64 B each, read twice per pass at most).
#include "wf_wide_bvh.h"
#include "wf_renderer.h"
#include "wf_wide_build.cuh"

#include <algorithm>
#include <cmath>

namespace wf {
namespace {

// counters: [0] nodes, [1] triangles, [2] TLAS leaves, [3] boxes out of range
__global__ void k_wide_number(const BvhNode* nodes, const BvhRef* roots, uint32_t begin, uint32_t end,
                              uint32_t* items, uint2* bases, uint32_t* counters) {
    uint32_t i = begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= end) return;
    bool fits;
    bases[i] = number_children(
        nodes, items[i], roots + i, items, [&](int k, uint32_t n) { return atomicAdd(&counters[k], n); }, fits);
    if (!fits) counters[3] = 1u;
}

__global__ void k_wide_emit(DeviceScene s, const BvhRef* roots, uint32_t count, const uint32_t* items,
                            const uint2* bases, WideNode* out, WideTriangle* triangles, WideLeaf* leaves) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    Collapsed c;
    collapse(s.nodes, items[i], roots + i, c);
    out[i] = wide_record(s, c, (items[i] & kTlasItem) != 0, bases[i].x, bases[i].y, triangles, leaves);
}

}  // namespace

cudaError_t build_wide_bvh(DeviceScene& view, const std::vector<BvhRef>& roots, uint32_t node_count,
                           uint32_t tlas_root, std::vector<void*>& allocations, uint64_t& bytes) {
    if (roots.empty()) return cudaSuccess;
    uint32_t root_count = uint32_t(roots.size());
    const size_t kept = allocations.size();
    const uint64_t kept_bytes = bytes;
    // Wide nodes other than the roots stand for distinct internal BVH2 nodes.
    size_t capacity = size_t(node_count) + root_count;
    // one allocation: counters, bases, items, root refs (each part's alignment
    // divides the size of those before it)
    static_assert(sizeof(BvhRef) % sizeof(uint32_t) == 0 && alignof(BvhRef) == sizeof(uint32_t), "packed after words");
    char* scratch = nullptr;
    // A small scene keeps it: a stream-ordered allocation takes 0.8 ms, a large
    // part of such a scene's creation, and cudaFree waits for other streams.
    const size_t scratch_bytes =
        16 + capacity * (sizeof(uint2) + sizeof(uint32_t)) + root_count * sizeof(BvhRef);
    const bool keep_scratch = scratch_bytes <= (size_t(1) << 20);
    cudaError_t e;
    if (keep_scratch) {
        e = device_alloc(reinterpret_cast<void**>(&scratch), scratch_bytes);
        if (e == cudaSuccess) {
            allocations.push_back(scratch);
            bytes += scratch_bytes;
        }
    } else {
        e = device_alloc_async(reinterpret_cast<void**>(&scratch), scratch_bytes, cudaStreamLegacy);
    }
    uint32_t* counters = reinterpret_cast<uint32_t*>(scratch);
    uint2* bases = reinterpret_cast<uint2*>(scratch + 16);
    uint32_t* items = reinterpret_cast<uint32_t*>(bases + capacity);
    BvhRef* root_refs = reinterpret_cast<BvhRef*>(items + capacity);
    uint32_t host[4] = {root_count, 0, 0, 0};
    if (e == cudaSuccess) {
        std::vector<uint32_t> first(root_count);
        for (uint32_t i = 0; i < root_count; ++i) first[i] = root_item(roots[i], i == tlas_root);
        e = cudaMemcpy(items, first.data(), root_count * sizeof(uint32_t), cudaMemcpyHostToDevice);
    }
    if (e == cudaSuccess) e = cudaMemcpy(counters, host, sizeof(host), cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(root_refs, roots.data(), root_count * sizeof(BvhRef), cudaMemcpyHostToDevice);
    uint32_t begin = 0;
    while (e == cudaSuccess && begin < host[0]) {  // one level of all trees at a time
        uint32_t end = host[0];
        k_wide_number<<<(end - begin + 127) / 128, 128>>>(view.nodes, root_refs, begin, end, items, bases, counters);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpy(host, counters, sizeof(host), cudaMemcpyDeviceToHost);
        begin = end;
    }
    WideNode* nodes = nullptr;
    WideTriangle* triangles = nullptr;
    WideLeaf* leaves = nullptr;
    auto keep = [&](auto** p, size_t count) {
        if (e != cudaSuccess) return;
        size_t n = sizeof(**p) * std::max<size_t>(count, 1);
        e = device_alloc(reinterpret_cast<void**>(p), n);
        if (e != cudaSuccess) return;
        allocations.push_back(*p);
        bytes += n;
    };
    keep(&nodes, host[0]);
    keep(&triangles, host[1]);
    keep(&leaves, host[2]);
    if (e == cudaSuccess) {
        k_wide_emit<<<(host[0] + 127) / 128, 128>>>(view, root_refs, host[0], items, bases, nodes, triangles, leaves);
        e = cudaGetLastError();
    }
    // the legacy stream alone: renders on other streams go on
    if (scratch && !keep_scratch) cudaFreeAsync(scratch, cudaStreamLegacy);
    cudaError_t waited = cudaStreamSynchronize(cudaStreamLegacy);
    if (e == cudaSuccess) e = waited;
    if (e != cudaSuccess) {
        for (size_t i = kept; i < allocations.size(); ++i) cudaFree(allocations[i]);
        allocations.resize(kept);
        bytes = kept_bytes;
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            view.wide.usable = 0u;
            return cudaSuccess;
        }
    } else {
        view.wide.nodes = nodes;
        view.wide.triangles = triangles;
        view.wide.leaves = leaves;
        if (host[3]) view.wide.usable = 0u;
    }
    return e;
}

}  // namespace wf
