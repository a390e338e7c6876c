// rt_bvh.h - host build of the compressed 8-wide BVH.
#pragma once

#include <string>
#include <vector>

#include "rt_device.cuh"
#include "rt_internal.h"

namespace rth {

struct BuiltBvh {
    std::vector<rtd::CwNode> nodes;  // node 0 is the root
    std::vector<int> order;          // triangle slot -> original triangle index
    int depth;                       // number of wide levels
};

// tv: ntri * 9 floats (three vertices per triangle).  Host build, validated.
bool build_cwbvh(const float* tv, int64_t ntri, BuiltBvh& out, std::string& err);
// The same rules built on the current device (rt_bvh_gpu.cu); tv is host memory.
bool build_cwbvh_gpu(const float* tv, int64_t ntri, BuiltBvh& out, std::string& err, cudaStream_t st);
// Checks a wide BVH against its triangles: every index a traversal can form is
// in range, the triangle order is a permutation and every quantised child box
// contains what it stands for.
bool validate_cwbvh(const BuiltBvh& bvh, const float* tv, int64_t ntri, std::string& err);

// A wide BVH built on the current device and left there.  The nodes lie level
// by level: level l is nodes [level_begin[l], level_begin[l + 1]).
struct DeviceBvh {
    rti::DevBuf nodes, order;
    std::vector<int> level_begin;  // depth + 1 entries
    int num_nodes = 0, depth = 0;
};
bool build_cwbvh_device(const float* d_tv, int64_t ntri, DeviceBvh& out, std::string& err, cudaStream_t st);
// The checks of validate_cwbvh on a device build; false: the check itself failed (err).
bool check_cwbvh_device(const DeviceBvh& bvh, const float* d_tv, int64_t ntri, bool& valid, std::string& err,
                        cudaStream_t st);
// The triangle records (SceneView::tri_v, tri_a) in leaf order; device arrays.
void launch_pack_triangles(const int* order, int n, const float* tv, const float* tn, const float* tuv,
                           const int* tri_mesh, const int* mesh_key, float4* out_v, float4* out_a, cudaStream_t st);
// The environment's sampling cache (env_sampling_cache) on the device: d_rgba
// and d_cache hold w * h float4; `sum` is env_luminance_sum of the same image.
float env_luminance_sum(const float* rgba, int width, int height);
cudaError_t env_sampling_cache_device(const float4* d_rgba, int w, int h, float sum, float4* d_cache, cudaStream_t st);

// Host tables shared with the device (rt_tables.cpp).
void kulla_conty_tables(float* bsdf_avg, float* albedo_avg);
void env_sampling_cache(const float* rgba, int width, int height, float* cache);

}  // namespace rth
