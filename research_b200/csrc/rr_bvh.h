// rr_bvh.h — host BVH builder interface (host-only header).
#pragma once

#include <cstdint>
#include <vector>
#include <vector_types.h>

namespace rr {
struct BvhBuild {
    std::vector<float4> nodes;     // 4 float4 per node (layout in rr_trace.cuh)
    std::vector<float4> nodes4;    // the same tree collapsed 4-wide: 8 float4 per node (layout in rr_trace.cuh)
    // Both trees again with their boxes on a grid over the scene (layout in
    // rr_trace.cuh); empty where that grid does not serve the scene.
    std::vector<uint4> qnodes;     // binary: 2 uint4 per node
    std::vector<uint4> qnodes4;    // 4-wide: 4 uint4 per node
    float qbase[3] = {0, 0, 0};    // grid plane q of axis a lies at qbase[a] + (128 + q / 256) * qscale[a]
    float qscale[3] = {0, 0, 0};
    std::vector<uint32_t> order;   // leaf order -> flattened triangle id
    uint32_t max_depth = 0;
};
// tri_world: 9 floats per triangle (v0, v1, v2 in world space).
BvhBuild build_bvh(const std::vector<float>& tri_world, int threads);
} // namespace rr
