// rt_scene_gpu.cu - what a scene's upload computes on the device besides the
// acceleration structure itself: the checks of a device-built wide BVH, the
// triangle records and the environment's sampling cache.
//
// This file is compiled with the host's arithmetic (build.py): denormals kept,
// divisions correctly rounded, nothing contracted.
#include <cuda_runtime.h>

#include <string>

#include "rt_bvh.h"

namespace rts {

// ------------------------------------------------------------------ validation
// The checks of validate_cwbvh (rt_bvh.cpp) on the device build, whose nodes
// lie level by level: every index a traversal can form is in range, every node
// but the root has one parent, the order is a permutation, and every quantised
// child box contains what it stands for.  `bad` becomes non-zero otherwise.
struct Bounds {
    float lo[3], hi[3];
};

__global__ void k_check_order(const int* __restrict__ order, int n, unsigned* __restrict__ seen, int* __restrict__ bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int t = order[i];
    if (t < 0 || t >= n || (atomicOr(seen + (t >> 5), 1u << (t & 31)) >> (t & 31)) & 1u) *bad = 1;
}

// Nodes [begin, end) of one level, whose children are nodes [end, next_end):
// deeper levels first, so that a child's bounds are there.
__global__ void k_check_level(const rtd::CwNode* __restrict__ nodes, int begin, int end, int next_end,
                              const int* __restrict__ order, const float* __restrict__ tv, int n,
                              Bounds* __restrict__ bounds, int* __restrict__ parents, int* __restrict__ bad) {
    const int i = begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= end) return;
    const rtd::CwNode nd = nodes[i];
    const float p[3] = {nd.px, nd.py, nd.pz};
    const int e[3] = {int(nd.ex) - 127, int(nd.ey) - 127, int(nd.ez) - 127};
    Bounds own;
    for (int a = 0; a < 3; a++) {
        own.lo[a] = INFINITY;
        own.hi[a] = -INFINITY;
    }
    bool ok = true;
    int rank = 0;
    for (int s = 0; s < 8; s++) {
        const bool inner = (nd.imask >> s) & 1u;
        if (nd.meta[s] == 0) {
            ok = ok && !inner;
            continue;
        }
        double lo[3], hi[3];
        for (int a = 0; a < 3; a++) {
            lo[a] = double(p[a]) + ldexp(double(nd.q[a][2 * s]), e[a]);
            hi[a] = double(p[a]) + ldexp(double(nd.q[a][2 * s + 1]), e[a]);
        }
        auto take = [&](float x, float y, float z) {
            const float v[3] = {x, y, z};
            for (int a = 0; a < 3; a++) {
                if (double(v[a]) < lo[a] || double(v[a]) > hi[a]) ok = false;
                own.lo[a] = fminf(own.lo[a], v[a]);
                own.hi[a] = fmaxf(own.hi[a], v[a]);
            }
        };
        if (inner) {
            const uint64_t c = uint64_t(nd.child_base) + uint64_t(rank++);
            if (c < uint64_t(end) || c >= uint64_t(next_end) || nd.meta[s] != uint8_t((1u << 5) | uint32_t(24 + s))) {
                ok = false;
                continue;
            }
            atomicAdd(parents + c, 1);
            const Bounds b = bounds[c];
            take(b.lo[0], b.lo[1], b.lo[2]);
            take(b.hi[0], b.hi[1], b.hi[2]);
        } else {
            const uint32_t unary = nd.meta[s] >> 5, off = nd.meta[s] & 31u;
            const int cnt = unary == 1 ? 1 : unary == 3 ? 2 : unary == 7 ? 3 : 0;
            if (cnt == 0 || off + uint32_t(cnt) > 24 || uint64_t(nd.tri_base) + off + uint32_t(cnt) > uint64_t(n)) {
                ok = false;
                continue;
            }
            for (int k = 0; k < cnt; k++) {
                const int t = order[nd.tri_base + off + k];
                if (t < 0 || t >= n) {
                    ok = false;
                    continue;
                }
                const float* v = tv + size_t(t) * 9;
                for (int c = 0; c < 3; c++) take(v[3 * c], v[3 * c + 1], v[3 * c + 2]);
            }
        }
    }
    bounds[i] = own;
    if (!ok) *bad = 1;
}

__global__ void k_check_parents(const int* __restrict__ parents, int n, int* __restrict__ bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > 0 && i < n && parents[i] != 1) *bad = 1;
}

// ------------------------------------------------------------------ triangle records
// The traversal and shading records of every triangle in leaf order
// (SceneView::tri_v, tri_a) from the scene's arrays: per triangle nine
// position and nine normal floats, six texture coordinates, the mesh; per mesh
// the shade bucket.  Without normals (null) the face normal of
// rt_scene_add_mesh (Scene.cpp:150-158), without texture coordinates its
// defaults (Scene.cpp:160-165).  A gather bound by HBM (0.2 ms for 2.59M
// triangles).
__global__ void __launch_bounds__(256) k_pack_triangles(const int* __restrict__ order, int n,
                                                        const float* __restrict__ tv, const float* __restrict__ tn,
                                                        const float* __restrict__ tuv, const int* __restrict__ tri_mesh,
                                                        const int* __restrict__ mesh_key, float4* __restrict__ out_v,
                                                        float4* __restrict__ out_a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int o = order[i];
    const float* p = tv + size_t(o) * 9;
    float m[9], uv[6] = {0.f, 0.f, 1.f, 0.f, 0.f, 1.f};
    if (tn) {
        for (int k = 0; k < 9; k++) m[k] = tn[size_t(o) * 9 + k];
    } else {
        const rtd::v3 v0 = rtd::ld3(p), v1 = rtd::ld3(p + 3), v2 = rtd::ld3(p + 6);
        const rtd::v3 f = normalize(cross(normalize(v1 - v0), normalize(v2 - v0)));
        for (int k = 0; k < 3; k++) m[3 * k] = f.x, m[3 * k + 1] = f.y, m[3 * k + 2] = f.z;
    }
    if (tuv)
        for (int k = 0; k < 6; k++) uv[k] = tuv[size_t(o) * 6 + k];
    const int mesh = tri_mesh[o];
    float4* v = out_v + size_t(i) * 3;
    float4* a = out_a + size_t(i) * 4;
    v[0] = make_float4(p[0], p[1], p[2], __int_as_float(o));
    v[1] = make_float4(p[3], p[4], p[5], __int_as_float(mesh_key[mesh]));
    v[2] = make_float4(p[6], p[7], p[8], 0.0f);
    a[0] = make_float4(m[0], m[1], m[2], uv[0]);
    a[1] = make_float4(m[3], m[4], m[5], uv[1]);
    a[2] = make_float4(m[6], m[7], m[8], uv[2]);
    a[3] = make_float4(uv[3], uv[4], uv[5], __int_as_float(mesh));
}

// ------------------------------------------------------------------ environment
// HdrTexture::CalculateHdrCache (core/src/Scene.cpp:217-313), bit for bit the
// table of env_sampling_cache in rt_tables.cpp.  Every sum keeps the host's
// order: the luminance sum comes from the host, a column's marginal and
// conditional sums run down the column in one thread.  The table's two binary
// searches per texel were 0.15 of the 0.2 s that a host thread took for a
// 2048 x 1024 image.
__global__ void __launch_bounds__(256) k_env_pdf(const float4* __restrict__ rgba, size_t n, float sum,
                                                 float* __restrict__ pdf) {
    const size_t q = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const float4 p = rgba[q];
    const float lum = 0.299f * p.x + 0.587f * p.y + 0.114f * p.z;
    pdf[q] = lum / sum;
}

// Column x: its sum over y, then the running sum of pdf / column sum.
__global__ void __launch_bounds__(32) k_env_columns(const float* __restrict__ pdf, int w, int h,
                                                    float* __restrict__ col, float* __restrict__ cdf_row) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= w) return;
    float sum = 0.0f;
#pragma unroll 16
    for (int y = 0; y < h; y++) sum += pdf[size_t(y) * w + x];
    col[x] = sum;
    float run = 0.0f;
#pragma unroll 16
    for (int y = 0; y < h; y++) {
        const float c = pdf[size_t(y) * w + x] / sum;
        run = y == 0 ? c : run + c;
        cdf_row[size_t(y) * w + x] = run;
    }
}

// Running sum of the column sums, in place, in one thread (the order counts).
__global__ void k_env_marginal(float* __restrict__ col, int w) {
    float run = col[0];
#pragma unroll 16
    for (int x = 1; x < w; x++) {
        run = col[x] + run;
        col[x] = run;
    }
}

// The first of n values (`stride` apart) not below v, by the bisection of
// std::lower_bound (which decides what columns of zero luminance, whose sums
// are not numbers, give).
RT_D int first_not_below(const float* __restrict__ a, int n, size_t stride, float v) {
    int first = 0;
    while (n > 0) {
        const int half = n >> 1, mid = first + half;
        if (__ldg(a + size_t(mid) * stride) < v) {
            first = mid + 1;
            n -= half + 1;
        } else {
            n = half;
        }
    }
    return first;
}

__global__ void __launch_bounds__(256) k_env_table(const float* __restrict__ pdf, const float* __restrict__ cdf_col,
                                                   const float* __restrict__ cdf_row, int w, int h,
                                                   float4* __restrict__ cache) {
    const size_t q = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (q >= size_t(w) * h) return;
    const int x = int(q % size_t(w)), y = int(q / size_t(w));
    const int cx = min(first_not_below(cdf_col, w, 1, float(y) / float(h)), w - 1);
    const int cy = first_not_below(cdf_row + cx, h, size_t(w), float(x) / float(w));
    cache[q] = make_float4(float(cx) / float(w), float(cy) / float(h), pdf[q], 0.0f);
}

}  // namespace rts

namespace rth {

namespace {
struct Arena {  // scratch arrays handed out of one allocation
    rti::DevBuf buf;
    size_t bytes = 0;
    size_t take(size_t n) {
        const size_t at = bytes;
        bytes += (n + 255) / 256 * 256;
        return at;
    }
    template <class T>
    T* at(size_t off) const {
        return reinterpret_cast<T*>(static_cast<char*>(buf.ptr) + off);
    }
};
}  // namespace

#define SG_CUDA(call)                                                      \
    do {                                                                   \
        cudaError_t e_ = (call);                                           \
        if (e_ != cudaSuccess) {                                           \
            err = std::string("GPU BVH check: ") + cudaGetErrorString(e_); \
            return false;                                                  \
        }                                                                  \
    } while (0)

bool check_cwbvh_device(const DeviceBvh& b, const float* d_tv, int64_t ntri, bool& valid, std::string& err,
                        cudaStream_t st) {
    using namespace rts;
    valid = true;
    if (ntri <= 0) return true;
    const int n = int(ntri), nn = b.num_nodes;
    Arena ar;
    const size_t o_bounds = ar.take(size_t(nn) * sizeof(Bounds));
    const size_t o_parents = ar.take(size_t(nn) * 4), o_seen = ar.take((size_t(n) + 31) / 32 * 4), o_bad = ar.take(4);
    SG_CUDA(ar.buf.alloc(ar.bytes));
    SG_CUDA(cudaMemsetAsync(ar.at<char>(o_parents), 0, ar.bytes - o_parents, st));
    int* bad = ar.at<int>(o_bad);
    k_check_order<<<(n + 255) / 256, 256, 0, st>>>(b.order.as<int>(), n, ar.at<unsigned>(o_seen), bad);
    for (int l = b.depth - 1; l >= 0; l--) {
        const int begin = b.level_begin[size_t(l)], end = b.level_begin[size_t(l) + 1];
        const int next = l + 1 < b.depth ? b.level_begin[size_t(l) + 2] : end;
        k_check_level<<<(end - begin + 127) / 128, 128, 0, st>>>(b.nodes.as<rtd::CwNode>(), begin, end, next,
                                                                 b.order.as<int>(), d_tv, n, ar.at<Bounds>(o_bounds),
                                                                 ar.at<int>(o_parents), bad);
    }
    k_check_parents<<<(nn + 255) / 256, 256, 0, st>>>(ar.at<int>(o_parents), nn, bad);
    SG_CUDA(cudaGetLastError());
    int h = 0;
    SG_CUDA(cudaMemcpyAsync(&h, bad, 4, cudaMemcpyDeviceToHost, st));
    SG_CUDA(cudaStreamSynchronize(st));
    valid = h == 0;
    return true;
}

void launch_pack_triangles(const int* order, int n, const float* tv, const float* tn, const float* tuv,
                           const int* tri_mesh, const int* mesh_key, float4* out_v, float4* out_a, cudaStream_t st) {
    if (n <= 0) return;
    rts::k_pack_triangles<<<(n + 255) / 256, 256, 0, st>>>(order, n, tv, tn, tuv, tri_mesh, mesh_key, out_v, out_a);
}

cudaError_t env_sampling_cache_device(const float4* d_rgba, int w, int h, float sum, float4* d_cache, cudaStream_t st) {
    if (w <= 0 || h <= 0) return cudaSuccess;
    const size_t n = size_t(w) * h;
    rti::DevBuf buf;
    if (cudaError_t e = buf.alloc((2 * n + size_t(w)) * sizeof(float))) return e;
    float *pdf = buf.as<float>(), *cdf_row = pdf + n, *col = cdf_row + n;
    const unsigned blocks = unsigned((n + 255) / 256);
    rts::k_env_pdf<<<blocks, 256, 0, st>>>(d_rgba, n, sum, pdf);
    rts::k_env_columns<<<(w + 31) / 32, 32, 0, st>>>(pdf, w, h, col, cdf_row);
    rts::k_env_marginal<<<1, 1, 0, st>>>(col, w);
    rts::k_env_table<<<blocks, 256, 0, st>>>(pdf, col, cdf_row, w, h, d_cache);
    if (cudaError_t e = cudaGetLastError()) return e;
    return cudaStreamSynchronize(st);  // before the scratch goes
}

}  // namespace rth
