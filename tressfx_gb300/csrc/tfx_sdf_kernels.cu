// Signed-distance-field kernels of the plain path (src/Shaders/TressFXSDFCollision.hlsl) and the
// collision-mesh bone skinning kernel (src/Shaders/TressFXBoneSkinning.hlsl:57-94).
//
// The SDF grid is uint32[X*Y*Z] holding FloatFlip3-encoded distances while it is built (atomicMin
// over the encoding = min |d|, ties to the positive value) and plain floats after Finalize.
// atomicMin is order independent, and the distance arithmetic below is the reference's in the
// same order with no FMA contraction, so the finished grid matches the oracle bit for bit.
#include <algorithm>
#include <atomic>

#include "tfx_launch.cuh"
#include "tfx_sdf_math.cuh"

namespace tfx {

// --------------------------------------------------------------------------------------------
__device__ __forceinline__ TriJob plain_job(uint32_t* sdf, const SdfGrid& g, const float4* mesh,
                                            const uint32_t* idx, int t) {
    const float3 x0 = xyz(mesh[2 * (size_t)idx[3 * (size_t)t + 0]]);
    const float3 x1 = xyz(mesh[2 * (size_t)idx[3 * (size_t)t + 1]]);
    const float3 x2 = xyz(mesh[2 * (size_t)idx[3 * (size_t)t + 2]]);
    return tri_job(g, sdf, x0, x1, x2);
}

// InitializeSignedDistanceField, :301-312 (vectorised: 4 cells per 16 B store), with the job of every
// triangle beside it when there is a job array.
__global__ void __launch_bounds__(256) k_sdf_initialize(uint32_t* __restrict__ sdf, long long cells, SdfGrid g,
                                                        const float4* mesh, const uint32_t* idx,
                                                        int ntri, TriJob* __restrict__ jobs) {
    after_previous();
    const uint32_t v = float_flip3(1e10f);
    const long long n4 = cells >> 2;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long me = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    for (long long t = me; t < ntri; t += stride) jobs[t] = plain_job(sdf, g, mesh, idx, (int)t);
    uint4* s4 = reinterpret_cast<uint4*>(sdf);
    for (long long i = me; i < n4; i += stride) s4[i] = make_uint4(v, v, v, v);
    for (long long i = (n4 << 2) + me; i < cells; i += stride) sdf[i] = v;
}

// ConstructSignedDistanceField, :329-397, over the jobs made beforehand.
__global__ void __launch_bounds__(128, kConstructBlocksPerSM) k_sdf_construct_jobs(const TriJob* jobs, int ntri) {
    after_previous();
    extern __shared__ __align__(16) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const SdfWarpArea area = sdf_warp_area(smem, warp, kSdfJobsAhead);
    sdf_construct_jobs_warp(area, jobs, ntri, blockIdx.x * 4 + warp, gridDim.x * 4, lane);
}

// ConstructSignedDistanceField, :329-397.  Each warp takes chunks of `per` (<= 32) consecutive
// triangles (sdf_construct_chunk_warp: lane k makes the job of the chunk's k-th triangle), then
// runs the triangles' cell loops in turn; the warps stride over the chunks.
__global__ void __launch_bounds__(128) k_sdf_construct(uint32_t* __restrict__ sdf, SdfGrid g,
                                                       const float4* mesh,
                                                       const uint32_t* idx, int ntri, int per, bool all) {
    after_previous();
    extern __shared__ __align__(16) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    SdfWarpArea area = sdf_warp_area(smem, warp, per);
    const int warpsTotal = gridDim.x * (blockDim.x >> 5);
    const int chunks = (ntri + per - 1) / per;
    for (int k = blockIdx.x * (blockDim.x >> 5) + warp; k < chunks; k += warpsTotal) {
        const int first = k * per;
        sdf_construct_chunk_warp(area, first, min(per, ntri - first), lane, all, [&](int t) {
            return plain_job(sdf, g, mesh, idx, t);
        });
    }
}

// FinalizeSignedDistanceField, :400-412 (vectorised)
__global__ void __launch_bounds__(256) k_sdf_finalize(uint32_t* __restrict__ sdf, long long cells) {
    after_previous();
    const long long n4 = cells >> 2;
    const long long stride = (long long)gridDim.x * blockDim.x;
    uint4* s4 = reinterpret_cast<uint4*>(sdf);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += stride) {
        uint4 u = s4[i];
        s4[i] = make_uint4(ifloat_flip3(u.x), ifloat_flip3(u.y), ifloat_flip3(u.z), ifloat_flip3(u.w));
    }
    for (long long i = (n4 << 2) + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < cells; i += stride)
        sdf[i] = ifloat_flip3(sdf[i]);
}

// CollideHairVerticesWithSdf_forward, :531-595.  One thread per hair vertex (guides and follows).
//
// Bound by the gathers and the warps that hide them: 128 threads and ten blocks an SM (48 registers, five
// words spilled) measured better than 256 threads at 62 registers (a dispatched 6,007 x 64 frame 50.4
// against 53.0 us, a 2,240 x 32 character 53.4 against 54.1), eight blocks (51.5, 53.7) and twelve (51.4, 54.9).
constexpr int kCollideThreads = 128;
__global__ void __launch_bounds__(kCollideThreads, 10) k_sdf_collide(const float* sdf, SdfGrid g, float margin,
                                                     float4* __restrict__ pos, float4* __restrict__ prev,
                                                     int n, long long vtot) {
    after_previous();
    const long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (v >= vtot) return;
    const int local = v >> 32 ? (int)(v % n) : (int)((uint32_t)v % (uint32_t)n);
    if (local == 0 || local == 1) return;
    const float4 hv = pos[v];
    float3 proj;
    if (sdf_collide_point(sdf, g, margin, xyz(hv), proj)) {
        pos[v] = with_xyz(hv, proj);
        const float4 pv = prev[v];
        prev[v] = with_xyz(pv, proj);
    }
}

// BoneSkinning, src/Shaders/TressFXBoneSkinning.hlsl:57-94.  One thread per mesh vertex.
// in/out: {float4 position, float4 normal}; skin: {float4 boneIndex, float4 boneWeight}.
// CollideHairVerticesWithSdf (TressFXSDFCollision.hlsl:599-715), the mixed-difference variant: one
// thread per vertex (roots included), one 8-corner fetch, the gradient by forward or backward
// differences within the same cell (h = 0.1 * cellSize added to the cell-normalised coordinates,
// as the shader writes it).
__global__ void __launch_bounds__(256) k_sdf_collide_mixed(const float* sdf, SdfGrid g, float margin,
                                                           float4* __restrict__ pos, float4* __restrict__ prev,
                                                           int64_t vtot) {
    after_previous();
    const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (v >= vtot) return;
    const float4 hv = pos[v];
    const float3 p = xyz(hv);
    const int3 gc = sdf_coords(g, p);
    if (!(0 <= gc.x && gc.x < g.nx - 2) || !(0 <= gc.y && gc.y < g.ny - 2) || !(0 <= gc.z && gc.z < g.nz - 2)) return;
    const long long X = 1, Y = g.nx, Z = (long long)g.ny * g.nx;
    const long long base = Z * gc.z + Y * gc.y + gc.x;
    const long long off[8] = {0, X, Y, Y + X, Z, Z + X, Z + Y, Z + Y + X};
    float d[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        d[j] = sdf[base + off[j]];
        if (d[j] == 1e10f) return;
    }
    auto tri = [&](float x, float y, float z) {
        const float b0 = lerp_ref(lerp_ref(d[0], d[1], x), lerp_ref(d[2], d[3], x), y);
        const float b1 = lerp_ref(lerp_ref(d[4], d[5], x), lerp_ref(d[6], d[7], x), y);
        return lerp_ref(b0, b1, z);
    };
    const float3 cp = sdf_cell_pos(g, gc.x, gc.y, gc.z);
    const float3 ip = divs(sub(p, cp), g.cell);
    const float dist = tri(ip.x, ip.y, ip.z);
    const float h = 0.1f * g.cell;
    const float3 dir = mk3((ip.x + h < 1.0f) ? 1.0f : -1.0f, (ip.y + h < 1.0f) ? 1.0f : -1.0f, (ip.z + h < 1.0f) ? 1.0f : -1.0f);
    const float3 nd = mk3(tri(ip.x + h * dir.x, ip.y, ip.z), tri(ip.x, ip.y + h * dir.y, ip.z), tri(ip.x, ip.y, ip.z + h * dir.z));
    const float3 grad = mk3((dir.x * (nd.x - dist)) / h, (dir.y * (nd.y - dist)) / h, (dir.z * (nd.z - dist)) / h);
    const float3 nrm = normalize(grad);
    if (dist < margin) {
        const float3 proj = add(p, mul(nrm, margin - dist));
        pos[v] = with_xyz(hv, proj);
        prev[v] = with_xyz(prev[v], proj);
    }
}

__global__ void __launch_bounds__(256) k_mesh_skin(float4* __restrict__ out, const float4* in,
                                                   const float4* skin, const float4* bones,
                                                   int nverts) {
    after_previous();
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nverts) return;
    const float4 p = in[2 * v], nr = in[2 * v + 1];
    float m[4][4];
    blend_bones(bones, skin[2 * v], skin[2 * v + 1], m);
    out[2 * v] = with_xyz(p, xform_row(xyz(p), 1.0f, m));
    out[2 * v + 1] = with_xyz(nr, xform_row(xyz(nr), 0.0f, m));
}

// A frame's inputs from page-locked host memory, read by the kernel itself: `quads` 16-byte words.  Between two
// kernels a copy by the copy engine costs 7 us, this 2.
__global__ void __launch_bounds__(128) k_upload(const uint4* src, uint4* __restrict__ dst, int quads) {
    after_previous();
    let_next_in();
    for (int i = blockIdx.x * 128 + threadIdx.x; i < quads; i += gridDim.x * 128) {
        uint4 v;
        asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(src + i));
        dst[i] = v;
    }
}

// --------------------------------------------------------------------------------------------
int sm_count() {
    constexpr int kMaxDevices = 64;
    static std::atomic<int> cache[kMaxDevices];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 1;
    int v = cache[dev].load(std::memory_order_relaxed);
    if (v <= 0) {
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) return 1;
        cache[dev].store(v, std::memory_order_relaxed);
    }
    return v;
}

static inline unsigned grid_for(long long work, int threads, unsigned cap) {
    long long b = (work + threads - 1) / threads;
    if (b < 1) b = 1;
    return (unsigned)(b > cap ? cap : b);
}

size_t sdf_job_bytes() { return sizeof(TriJob); }
bool sdf_takes_jobs(int64_t tris) { return sdf_fills_device(tris, sm_count()); }

cudaError_t launch_upload(void* dst, const void* pinned, size_t bytes, cudaStream_t s) {
    const int quads = (int)(bytes / 16);
    if (quads <= 0) return cudaSuccess;
    return launch_after(k_upload, grid_for(quads, 128, sm_count() * 4), 128, 0, s, static_cast<const uint4*>(pinned),
                        static_cast<uint4*>(dst), quads);
}

cudaError_t launch_sdf_initialize(uint32_t* sdf, int64_t cells, cudaStream_t s, const SdfGrid* g, const float4* mesh,
                                  const uint32_t* idx, int ntri, TriJob* jobs) {
    if (cells <= 0) return cudaSuccess;
    const int n = jobs ? ntri : 0;
    const long long work = std::max<long long>((cells + 3) / 4, n);
    return launch_after(k_sdf_initialize, grid_for(work, 256, sm_count() * 16), 256, 0, s, sdf, cells, g ? *g : SdfGrid{}, mesh,
                        idx, n, jobs);
}

cudaError_t launch_sdf_jobs(TriJob* jobs, uint32_t* sdf, const SdfGrid& g, const float4* mesh, const uint32_t* idx, int ntri,
                            cudaStream_t s) {
    if (ntri <= 0) return cudaSuccess;
    return launch_after(k_sdf_initialize, grid_for(ntri, 256, sm_count() * 16), 256, 0, s, sdf, 0, g, mesh, idx, ntri, jobs);
}

cudaError_t launch_sdf_construct_jobs(const TriJob* jobs, int ntri, cudaStream_t s) {
    if (ntri <= 0) return cudaSuccess;
    const unsigned blocks = (unsigned)std::min<long long>(((long long)ntri + 3) / 4, (long long)sm_count() * kConstructBlocksPerSM);
    return launch_after(k_sdf_construct_jobs, blocks, 128, sdf_construct_smem(4, kSdfJobsAhead), s, jobs, ntri);
}

cudaError_t launch_sdf_construct(uint32_t* sdf, const SdfGrid& g, const float4* mesh, const uint32_t* idx, int ntri,
                                 cudaStream_t s) {
    if (ntri <= 0) return cudaSuccess;
    const int per = sdf_construct_chunk(ntri, sm_count());
    const long long chunks = ((long long)ntri + per - 1) / per;
    const unsigned blocks = (unsigned)std::min<long long>((chunks + 3) / 4, (long long)sm_count() * 64);
    return launch_after(k_sdf_construct, blocks, 128, sdf_construct_smem(4, per), s, sdf, g, mesh, idx, ntri, per,
                        !sdf_fills_device(ntri, sm_count()));
}

cudaError_t launch_sdf_finalize(uint32_t* sdf, int64_t cells, cudaStream_t s) {
    if (cells <= 0) return cudaSuccess;
    return launch_after(k_sdf_finalize, grid_for((cells + 3) / 4, 256, sm_count() * 16), 256, 0, s, sdf, cells);
}

cudaError_t launch_sdf_collide(const uint32_t* sdf, const SdfGrid& g, float margin, float4* pos, float4* prev, int n,
                               int64_t vtot, cudaStream_t s) {
    if (vtot <= 0) return cudaSuccess;
    return launch_after(k_sdf_collide, (unsigned)((vtot + kCollideThreads - 1) / kCollideThreads), kCollideThreads, 0, s, reinterpret_cast<const float*>(sdf), g, margin,
                        pos, prev, n, vtot);
}

cudaError_t launch_sdf_collide_mixed(const uint32_t* sdf, const SdfGrid& g, float margin, float4* pos, float4* prev,
                                     int64_t vtot, cudaStream_t s) {
    if (vtot <= 0) return cudaSuccess;
    return launch_after(k_sdf_collide_mixed, (unsigned)((vtot + 255) / 256), 256, 0, s, reinterpret_cast<const float*>(sdf), g,
                        margin, pos, prev, vtot);
}

cudaError_t launch_mesh_skin(float4* out, const float4* in, const float4* skin, const float4* bones, int nverts,
                             cudaStream_t s) {
    if (nverts <= 0) return cudaSuccess;
    return launch_after(k_mesh_skin, (nverts + 255) / 256, 256, 0, s, out, in, skin, bones, nverts);
}

}  // namespace tfx
