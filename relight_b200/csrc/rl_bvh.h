// BVH construction for the B200 traversal kernels.
#pragma once

#include <cmath>
#include <cstdint>
#include <vector>

#ifdef __CUDACC__
#define RL_BOTH __host__ __device__
#else
#define RL_BOTH
#endif

namespace rl {

// A child box's centre and half-extent along one axis, as the nodes hold them.
// The half-extent covers the box after the centre's rounding, and grows by
// 2^-21 of both: the slab test's rounding of (centre - origin) / direction is
// below that share of the box's size and place.  A box that is not finite is
// met by every ray.
RL_BOTH inline void box_centre_half(float lo, float hi, float* centre, float* half) {
    float c = 0.5f * lo + 0.5f * hi;
    float h = hi - c > c - lo ? hi - c : c - lo;
    h += (h + fabsf(c)) * (1.0f / (1 << 21));
    if (!(h <= 1e38f)) {
        c = 0.0f;
        h = 3e38f;
    }
    *centre = c;
    *half = h;
}

struct BvhBuild {
    std::vector<float> nodes;  // 16 floats per node (four float4: centres and half-extents, see rl_device.cuh)
    std::vector<float> tris;   // 12 floats per triangle in leaf order (three float4)
    std::vector<float> nodes4; // 32 floats per 4-wide node (eight float4, see rl_device.cuh)
    int64_t nodes4_count = 0;
    std::vector<uint32_t> nodes8;  // 20 words per compressed 8-wide node (five uint4, see rl_device.cuh)
    std::vector<float> tris8;      // triangle records in 8-wide node order (12 floats each)
    int64_t nodes8_count = 0;
    int64_t leaves = 0;
    int depth = 0;
    double sah = 0.0;
};

// Binned-SAH build over `ntris` triangles given as three vertex ids into
// `pos` ([nverts][3]); triangle ids are the global ids (position in `tris`).
// wide8: also emit the compressed 8-wide tree (nodes8 / tris8).
bool build_bvh_sah(const float* pos, int nverts, const int32_t* tris, int ntris, BvhBuild& out, const char** err,
                   bool wide8 = false);

}  // namespace rl
