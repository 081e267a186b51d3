// Device build of the reference's binary SAH BVH (code/Bvh/Bvh.cpp:122-325):
// same nodes, bit for bit, and the same triangle order as `build_bvh`.
#pragma once

#include <cuda_runtime.h>

#include <functional>

#include "../../include/pcr_cuda.h"

namespace pcr {

// put(d_verts) uploads the n triangles as v0 v1 v2 (9 floats each), ordered on
// `st`; take(d_nodes, count, d_order) receives the nodes in depth-first preorder
// and, per leaf position, the input index of its triangle, on the device,
// ordered on `st` and valid until it returns.  Synchronous; the workspace
// (about 360 bytes per triangle) comes from `pool` (null: the device's default
// pool).
void device_build_bvh(int device, cudaStream_t st, cudaMemPool_t pool, int n, const std::function<void(float*)>& put,
                      const std::function<void(const pcr_bvh_node*, int, const int*)>& take);

}  // namespace pcr
