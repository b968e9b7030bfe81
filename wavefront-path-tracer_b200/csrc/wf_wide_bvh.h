// Wide BVH of a device scene (built on the GPU from its BVH2s at creation).
#pragma once

#include "wf_internal.h"

namespace wf {

// Collapses every BVH2 of the scene (BLASes, TLAS, direct list), whose nodes,
// triangles, instances and BLAS records are already on the device, into
// 8-wide compressed nodes and completes view.wide (HostScene::margins).  Tree i (roots[i], with its
// root box) gets wide node i as its root; tree `tlas_root` is the TLAS
// (kNoWide: none).  `node_count` is the number of BVH2 nodes.  The arrays go
// to `allocations` and their size is added to `bytes`.  Without the memory for
// them the scene keeps its BVH2s alone (view.wide.usable = 0).  Runs on the legacy
// stream and waits for it.
cudaError_t build_wide_bvh(DeviceScene& view, const std::vector<BvhRef>& roots, uint32_t node_count,
                           uint32_t tlas_root, std::vector<void*>& allocations, uint64_t& bytes);

}  // namespace wf
