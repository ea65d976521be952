// Kernels of the learned collision proxy (tfx_neural.cuh): inference, training (fused forward +
// backward, weight gradients, Adam) and training-sample generation from grid SDFs.
//
// mma.sync m16n8k16 (bf16 x bf16 -> f32) fragment layouts used throughout, with g = lane / 4 and
// i = lane % 4:  A (16 x 16, row-major) regs {row g, cols 2i..2i+1}, {row g+8, same}, {row g,
// cols 2i+8..}, {row g+8, cols 2i+8..};  B (16 x 8) regs {rows 2i..2i+1, col g}, {rows 2i+8.., col g};
// C (16 x 8, f32) {row g, cols 2i, 2i+1}, {row g+8, cols 2i, 2i+1}.  The C fragments of n-tiles 2k and
// 2k+1 are exactly the A fragment of k-tile k of the next layer, so activations never leave registers.
#include <algorithm>
#include <type_traits>

#include "tfx_launch.cuh"
#include "tfx_neural.cuh"
#include "tfx_sdf_math.cuh"

namespace tfx {
namespace nsdf {

namespace {

__constant__ float c_freq[NFREQ] = {
    1.0f, 1.2599210498948732f, 1.5874010519681994f, 2.0f, 2.5198420997897464f, 3.174802103936399f,
    4.0f, 5.039684199579493f, 6.349604207872798f, 8.0f, 10.079368399158986f, 12.699208415745595f,
    16.0f, 20.158736798317972f, 25.39841683149119f, 32.0f};   // 2^(k/3)

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The network is an approximation.  Its activation, SiLU(z) = z * sigmoid(z) = 0.5 z (1 + tanh(z / 2)),
// is evaluated on bf16 pairs with the hardware tanh: one MUFU operation per two activations, and
// the result is directly the next layer's bf16 A-fragment register.
__device__ __forceinline__ uint32_t silu2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(0.5f * a, 0.5f * b);
    uint32_t t;
    asm("tanh.approx.bf16x2 %0, %1;" : "=r"(t) : "r"(*reinterpret_cast<uint32_t*>(&h)));
    const __nv_bfloat162 r = __hfma2(h, *reinterpret_cast<__nv_bfloat162*>(&t), h);
    return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ float silu_grad(float z) {
    const float s = __fdividef(1.0f, 1.0f + __expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

// sin(pi x), cos(pi x): x reduced exactly to [-1, 1] (x - 2 * rint(x / 2) is exact in binary floating
// point), then the hardware sine / cosine of pi * x'.
__device__ __forceinline__ void sincospi_fast(float x, float* s, float* c) {
    const float r = x - 2.0f * rintf(0.5f * x);
    const float a = 3.14159265358979f * r;
    *s = __sinf(a);
    *c = __cosf(a);
}

__device__ __forceinline__ uint32_t hash32(uint32_t x) {   // lowbias32 (C. Wellons)
    x ^= x >> 16; x *= 0x7feb352dU; x ^= x >> 15; x *= 0x846ca68bU; x ^= x >> 16;
    return x;
}
__device__ __forceinline__ float u01(uint32_t h) { return (float)(h >> 8) * (1.0f / 16777216.0f); }

// A fragment of k-tile kt from a 16-row bf16 tile in shared memory (row stride rs elements).
__device__ __forceinline__ void load_a(const __nv_bfloat16* T, int rs, int kt, int lane, uint32_t (&a)[4]) {
    const int g = lane >> 2, i = lane & 3;
    const __nv_bfloat16* r0 = T + g * rs + kt * 16 + 2 * i;
    const __nv_bfloat16* r1 = r0 + 8 * rs;
    a[0] = *reinterpret_cast<const uint32_t*>(r0);
    a[1] = *reinterpret_cast<const uint32_t*>(r1);
    a[2] = *reinterpret_cast<const uint32_t*>(r0 + 8);
    a[3] = *reinterpret_cast<const uint32_t*>(r1 + 8);
}
// B fragment (n-tile nt, k-tile kt) of a weight block stored with n as the row (row stride rs).
__device__ __forceinline__ void load_b(const __nv_bfloat16* W, int rs, int nt, int kt, int lane, uint32_t& b0,
                                       uint32_t& b1) {
    const int g = lane >> 2, i = lane & 3;
    const __nv_bfloat16* r = W + (nt * 8 + g) * rs + kt * 16 + 2 * i;
    b0 = *reinterpret_cast<const uint32_t*>(r);
    b1 = *reinterpret_cast<const uint32_t*>(r + 8);
}
// B fragments of n-tiles nt and nt+1 (k-tile kt) with one ldmatrix.x4: lanes 8m..8m+7 address the rows
// of 8x8 matrix m = (n-tile nt + m/2, k half m%2); rows are 16-byte aligned (row strides 144 / 240 B)
// and the eight rows of a matrix fall in distinct bank quads.
__device__ __forceinline__ void load_b2(const __nv_bfloat16* W, int rs, int nt, int kt, int lane, uint32_t (&b)[4]) {
    const int m = lane >> 3, r = lane & 7;
    const __nv_bfloat16* row = W + ((nt + (m >> 1)) * 8 + r) * rs + kt * 16 + (m & 1) * 8;
    const uint32_t addr = (uint32_t)__cvta_generic_to_shared(row);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
                 : "r"(addr));
}
// C fragments (8 n-tiles) initialised with a bias vector.
__device__ __forceinline__ void init_bias(float (&C)[8][4], const float* b, int lane) {
    const int i = lane & 3;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        const float b0 = b[nt * 8 + 2 * i], b1 = b[nt * 8 + 2 * i + 1];
        C[nt][0] = b0; C[nt][1] = b1; C[nt][2] = b0; C[nt][3] = b1;
    }
}
// A fragments of the next layer from C, through SiLU.
__device__ __forceinline__ void c_to_a(const float (&C)[8][4], uint32_t (&A)[4][4]) {
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
        A[kt][0] = silu2(C[2 * kt][0], C[2 * kt][1]);
        A[kt][1] = silu2(C[2 * kt][2], C[2 * kt][3]);
        A[kt][2] = silu2(C[2 * kt + 1][0], C[2 * kt + 1][1]);
        A[kt][3] = silu2(C[2 * kt + 1][2], C[2 * kt + 1][3]);
    }
}
// Features of one point into row s of the tile: the lane pair (2s, 2s+1) splits the work.
__device__ __forceinline__ void write_features(__nv_bfloat16* F, int s, int half, float ux, float uy, float uz, float p0,
                                               float p1, float p2, bool valid) {
    __nv_bfloat16* row = F + s * RS1;
    const float u[3] = {ux, uy, uz};
    if (half == 0) {
        row[0] = __float2bfloat16(valid ? ux : 0.f);
        row[1] = __float2bfloat16(valid ? uy : 0.f);
        row[2] = __float2bfloat16(valid ? uz : 0.f);
        row[3] = __float2bfloat16(valid ? p0 : 0.f);
        row[4] = __float2bfloat16(valid ? p1 : 0.f);
        row[5] = __float2bfloat16(valid ? p2 : 0.f);
    }
    // f_{k+3} = 2 f_k: the three base frequencies of this half (k0, k0+1, k0+2) by the hardware sine /
    // cosine, every later one by the double-angle formulas sin 2a = 2 sin a cos a, cos 2a = 1 - 2 sin^2 a
    const int k0 = half * (NFREQ / 2);
#pragma unroll
    for (int b = 0; b < 3; ++b) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            float sn = 0.f, cs = 0.f;
            if (valid) sincospi_fast(c_freq[k0 + b] * u[d], &sn, &cs);
#pragma unroll
            for (int k = k0 + b; k < k0 + NFREQ / 2; k += 3) {
                *reinterpret_cast<__nv_bfloat162*>(row + 6 + 6 * k + 2 * d) = __floats2bfloat162_rn(sn, cs);
                const float s2 = 2.0f * sn * cs, c2 = 1.0f - 2.0f * sn * sn;
                sn = s2; cs = c2;
            }
        }
    }
    if (half == 1)
#pragma unroll
        for (int f = NFEAT; f < KIN; ++f) row[f] = __float2bfloat16(0.f);
}

// Stores a C-fragment tile (rows = 16 samples, ntiles x 8 columns) as sample-pair-interleaved bf16:
// 32-bit word (pair p, column c) holds (row 2p, row 2p+1) of column c at base[p * F + c].
__device__ __forceinline__ void store_pairs(const float (&C)[8][4], int ntiles, uint32_t* base, int F, int lane) {
    const int g = lane >> 2, i = lane & 3;
    const bool even = (g & 1) == 0;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        if (nt >= ntiles) break;
        const float v00 = C[nt][0], v01 = C[nt][1], v10 = C[nt][2], v11 = C[nt][3];
        const float x0 = __shfl_xor_sync(0xffffffffu, even ? v01 : v00, 4);
        const float x1 = __shfl_xor_sync(0xffffffffu, even ? v11 : v10, 4);
        const int c0 = nt * 8 + 2 * i;
        if (even) {
            base[(g >> 1) * F + c0] = pack_bf16(v00, x0);
            base[((g + 8) >> 1) * F + c0] = pack_bf16(v10, x1);
        } else {
            base[(g >> 1) * F + c0 + 1] = pack_bf16(x0, v01);
            base[((g + 8) >> 1) * F + c0 + 1] = pack_bf16(x1, v11);
        }
    }
}

// Inference forward pass of a 32-point tile (two m-tiles sharing every weight fragment): rows
// g, g+8 of tile 0 and g, g+8 of tile 1 come back in y[0..3] (valid in lanes with lane % 4 == 0).
__device__ __forceinline__ void mlp_forward32(const __nv_bfloat16* sW, const float* sB, const __nv_bfloat16* F, int lane,
                                              float (&y)[4]) {
    float C[2][8][4];
    init_bias(C[0], sB, lane);
    init_bias(C[1], sB, lane);
#pragma unroll 1
    for (int kt = 0; kt < KIN / 16; ++kt) {
        uint32_t a0[4], a1[4];
        load_a(F, RS1, kt, lane, a0);
        load_a(F + 16 * RS1, RS1, kt, lane, a1);
#pragma unroll
        for (int nt = 0; nt < 8; nt += 2) {
            uint32_t b[4];
            load_b2(sW + OFF_WT1, RS1, nt, kt, lane, b);
            mma16816(C[0][nt], a0[0], a0[1], a0[2], a0[3], b[0], b[1]);
            mma16816(C[1][nt], a1[0], a1[1], a1[2], a1[3], b[0], b[1]);
            mma16816(C[0][nt + 1], a0[0], a0[1], a0[2], a0[3], b[2], b[3]);
            mma16816(C[1][nt + 1], a1[0], a1[1], a1[2], a1[3], b[2], b[3]);
        }
    }
    const int woff[3] = {OFF_WT2, OFF_WT3, OFF_WT4};
#pragma unroll 1
    for (int l = 0; l < 3; ++l) {
        uint32_t A0[4][4], A1[4][4];
        c_to_a(C[0], A0);
        c_to_a(C[1], A1);
        init_bias(C[0], sB + (l + 1) * HID, lane);
        init_bias(C[1], sB + (l + 1) * HID, lane);
        const __nv_bfloat16* W = sW + woff[l];
#pragma unroll
        for (int kt = 0; kt < 4; ++kt)
#pragma unroll
            for (int nt = 0; nt < 8; nt += 2) {
                uint32_t b[4];
                load_b2(W, RSH, nt, kt, lane, b);
                mma16816(C[0][nt], A0[kt][0], A0[kt][1], A0[kt][2], A0[kt][3], b[0], b[1]);
                mma16816(C[1][nt], A1[kt][0], A1[kt][1], A1[kt][2], A1[kt][3], b[0], b[1]);
                mma16816(C[0][nt + 1], A0[kt][0], A0[kt][1], A0[kt][2], A0[kt][3], b[2], b[3]);
                mma16816(C[1][nt + 1], A1[kt][0], A1[kt][1], A1[kt][2], A1[kt][3], b[2], b[3]);
            }
    }
    uint32_t A0[4][4], A1[4][4];
    c_to_a(C[0], A0);
    c_to_a(C[1], A1);
    float C5[2][4];
    {
        const int i = lane & 3;
        const float b0 = sB[4 * HID + 2 * i], b1 = sB[4 * HID + 2 * i + 1];
#pragma unroll
        for (int t = 0; t < 2; ++t) { C5[t][0] = b0; C5[t][1] = b1; C5[t][2] = b0; C5[t][3] = b1; }
    }
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
        uint32_t b0, b1;
        load_b(sW + OFF_WT5, RSH, 0, kt, lane, b0, b1);
        mma16816(C5[0], A0[kt][0], A0[kt][1], A0[kt][2], A0[kt][3], b0, b1);
        mma16816(C5[1], A1[kt][0], A1[kt][1], A1[kt][2], A1[kt][3], b0, b1);
    }
    y[0] = C5[0][0]; y[1] = C5[0][2]; y[2] = C5[1][0]; y[3] = C5[1][2];
}

template <int WORDS>
__device__ __forceinline__ void stage_weights(uint4* dst, const __nv_bfloat16* wbf, float* sB, const float* bias) {
    const uint4* src = reinterpret_cast<const uint4*>(wbf);
    for (int k = threadIdx.x; k < WORDS; k += blockDim.x) dst[k] = src[k];
    for (int k = threadIdx.x; k < NBIAS; k += blockDim.x) sB[k] = bias[k];
}

constexpr int FWD_U4 = WBF_FWD * 2 / 16;
constexpr int ALL_U4 = WBF_ALL * 2 / 16;
static_assert(WBF_FWD * 2 % 16 == 0 && WBF_ALL * 2 % 16 == 0, "weight blocks are copied as uint4");
constexpr int TILE_BYTES = 16 * RS1 * 2;
constexpr int QUERY_WARPS = 4;
constexpr size_t QUERY_SMEM = (size_t)WBF_FWD * 2 + NBIAS * 4 + QUERY_WARPS * 2 * TILE_BYTES;
// training: a block carries TRAIN_TILES tiles of 16 samples, four warps to a tile
constexpr int TRAIN_TILES = 4;
constexpr int TRAIN_THREADS = TRAIN_TILES * 128;
constexpr int ACT_BYTES = 16 * RSH * 2;   // a tile's activations or gradients of one layer
constexpr size_t TRAIN_SMEM = (size_t)WBF_ALL * 2 + NBIAS * 4 + TRAIN_TILES * (TILE_BYTES + 2 * ACT_BYTES + 2 * 16 * 4);

// ------------------------------------------------------------------------------------------ query
template <bool SAMPLES>
__global__ void __launch_bounds__(QUERY_WARPS * 32) k_nsdf_query(const __nv_bfloat16* __restrict__ wbf,
                                                                 const float* __restrict__ bias, Frame fr,
                                                                 const float4* __restrict__ pts,
                                                                 const Sample* __restrict__ samples, int count, Pose pose,
                                                                 float* __restrict__ out) {
    extern __shared__ uint4 smem_q[];
    __nv_bfloat16* sW = reinterpret_cast<__nv_bfloat16*>(smem_q);
    float* sB = reinterpret_cast<float*>(sW + WBF_FWD);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __nv_bfloat16* sF = reinterpret_cast<__nv_bfloat16*>(sB + NBIAS) + warp * 32 * RS1;
    stage_weights<FWD_U4>(smem_q, wbf, sB, bias);
    __syncthreads();
    const int g = lane >> 2, i = lane & 3;
    const int nw = gridDim.x * QUERY_WARPS;
    for (int tile = blockIdx.x * QUERY_WARPS + warp; tile * 32 < count; tile += nw) {
        const int idx = tile * 32 + lane;
        const bool valid = idx < count;
        float px = 0.f, py = 0.f, pz = 0.f, a0 = pose.a0, a1 = pose.a1, a2 = pose.a2;
        if (valid) {
            if constexpr (SAMPLES) {
                const Sample S = samples[idx];
                px = S.x; py = S.y; pz = S.z; a0 = S.p0; a1 = S.p1; a2 = S.p2;
            } else {
                const float4 P = pts[idx];
                px = P.x; py = P.y; pz = P.z;
            }
        }
        const float ux = (px - fr.cx) * fr.ihx, uy = (py - fr.cy) * fr.ihy, uz = (pz - fr.cz) * fr.ihz;
        write_features(sF, lane, 0, ux, uy, uz, a0 * fr.poseScale, a1 * fr.poseScale, a2 * fr.poseScale, valid);
        write_features(sF, lane, 1, ux, uy, uz, a0 * fr.poseScale, a1 * fr.poseScale, a2 * fr.poseScale, valid);
        __syncwarp();
        float y[4];
        mlp_forward32(sW, sB, sF, lane, y);
        __syncwarp();
        if (i == 0) {
            const float sc = SAMPLES ? 1.0f : fr.cell;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int row = tile * 32 + (r >> 1) * 16 + g + 8 * (r & 1);
                if (row < count) out[row] = y[r] * sc;
            }
        }
    }
}

// ------------------------------------------------------------------------------------------ training
__device__ __forceinline__ void copy_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// One minibatch: forward with saved activations, loss, backward to every layer's pre-activation
// gradient.  Activations and gradients go to `acts` in the pair layout for k_nsdf_wgrad:
//   H0 [B/2][KIN], H1..H4 [B/2][64], dZ1..dZ4 [B/2][64], dZ5 [B/2][8]   (32-bit words).
//
// Four warps carry a tile of 16 samples, each a quarter of every layer's 64 columns (two n-tiles of the
// MMA): a minibatch has only batch / 16 tiles (512 at 8,192 samples), so one warp per tile left four warps
// on an SM and its time was one warp's chain through the ten layers.  A layer's activations pass between
// the warps through shared memory (bf16, two buffers by turns), its pre-activations stay in registers for
// the backward pass.  Bound: that chain and the barrier per layer (8,192 samples, ncu: 23.4 -> 11.9 us).
__device__ __forceinline__ void tile_sync(int tile) { asm volatile("bar.sync %0, 128;" ::"r"(tile + 1) : "memory"); }

// Two n-tiles' words (bf16 pairs of columns c0, c0 + 1; [nt][0] row g, [nt][1] row g + 8) into the tile's
// shared buffer, and as sample pairs into global memory: words of (row 2p, row 2p + 1), column c.
__device__ __forceinline__ void store_act(const uint32_t (&w)[2][2], __nv_bfloat16* T, uint32_t* out, int wq, int lane) {
    const int g = lane >> 2, i = lane & 3;
    const bool even = (g & 1) == 0;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int c0 = (2 * wq + q) * 8 + 2 * i;
        if (T) {
            *reinterpret_cast<uint32_t*>(T + g * RSH + c0) = w[q][0];
            *reinterpret_cast<uint32_t*>(T + (g + 8) * RSH + c0) = w[q][1];
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t mine = w[q][r], other = __shfl_xor_sync(0xffffffffu, mine, 4);
            out[((g + 8 * r) >> 1) * HID + c0 + (even ? 0 : 1)] =
                even ? __byte_perm(mine, other, 0x5410) : __byte_perm(other, mine, 0x7632);
        }
    }
}

// C += the tile's 16 x 64 operand in T times the two n-tiles of a 64-wide layer's weights ([n][k], stride RSH).
__device__ __forceinline__ void layer_quarter(float (&C)[2][4], const __nv_bfloat16* T, const __nv_bfloat16* W, int wq, int lane) {
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
        uint32_t a[4], b[4];
        load_a(T, RSH, kt, lane, a);
        load_b2(W, RSH, 2 * wq, kt, lane, b);
        mma16816(C[0], a[0], a[1], a[2], a[3], b[0], b[1]);
        mma16816(C[1], a[0], a[1], a[2], a[3], b[2], b[3]);
    }
}
__device__ __forceinline__ void bias_quarter(float (&C)[2][4], const float* b, int wq, int lane) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const float2 v = *reinterpret_cast<const float2*>(b + (2 * wq + q) * 8 + 2 * (lane & 3));
        C[q][0] = v.x; C[q][1] = v.y; C[q][2] = v.x; C[q][3] = v.y;
    }
}

__global__ void __launch_bounds__(TRAIN_THREADS, 1) k_nsdf_train(const __nv_bfloat16* wbf,
                                                                 const float* bias, Frame fr,
                                                                 const Sample* __restrict__ pool, long long poolSize,
                                                                 int batch, uint32_t seed, uint32_t* __restrict__ acts,
                                                                 float* __restrict__ lossSum) {
    extern __shared__ uint4 smem_t[];
    __nv_bfloat16* sW = reinterpret_cast<__nv_bfloat16*>(smem_t);
    float* sB = reinterpret_cast<float*>(sW + WBF_ALL);
    const int tg = threadIdx.x >> 7, wq = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31, tid = threadIdx.x & 127;
    unsigned char* area = reinterpret_cast<unsigned char*>(sB + NBIAS) + (size_t)tg * (TILE_BYTES + 2 * ACT_BYTES + 2 * 16 * 4);
    __nv_bfloat16* sF = reinterpret_cast<__nv_bfloat16*>(area);
    __nv_bfloat16* act[2] = {reinterpret_cast<__nv_bfloat16*>(area + TILE_BYTES), reinterpret_cast<__nv_bfloat16*>(area + TILE_BYTES + ACT_BYTES)};
    float* sT = reinterpret_cast<float*>(area + TILE_BYTES + 2 * ACT_BYTES);   // targets, then weights
    const long long B2 = batch / 2;
    uint32_t* H0 = acts;
    uint32_t* H1 = H0 + B2 * KIN;          // H1..H4, then dZ1..dZ4, then dZ5
    uint32_t* dZ1 = H1 + 4 * B2 * HID;
    uint32_t* dZ5 = dZ1 + 4 * B2 * HID;
    const int g = lane >> 2, i = lane & 3;
    const int s = tid >> 3, part = tid & 7;   // the thread's sample and its eighth of the features
    auto features = [&](int tile) {   // as write_features, a sample's 18 recurrences over eight threads
        const uint32_t h = hash32(seed ^ hash32((uint32_t)(tile * 16 + s) * 2654435761u));
        const Sample S = pool[(long long)(((unsigned long long)h * (unsigned long long)poolSize) >> 32)];
        const float u[3] = {(S.x - fr.cx) * fr.ihx, (S.y - fr.cy) * fr.ihy, (S.z - fr.cz) * fr.ihz};
        __nv_bfloat16* row = sF + s * RS1;
        if (part == 0) {
            const float f[6] = {u[0], u[1], u[2], S.p0 * fr.poseScale, S.p1 * fr.poseScale, S.p2 * fr.poseScale};
#pragma unroll
            for (int k = 0; k < 6; ++k) row[k] = __float2bfloat16(f[k]);
            sT[s] = S.target;
            sT[16 + s] = S.weight;
        } else if (part == 1) {
#pragma unroll
            for (int f = NFEAT; f < KIN; ++f) row[f] = __float2bfloat16(0.f);
        }
        for (int c = part; c < 18; c += 8) {
            const int k0 = c >= 9 ? NFREQ / 2 : 0, b = (c % 9) / 3, d = c % 3;
            float sn, cs;
            sincospi_fast(c_freq[k0 + b] * (d == 0 ? u[0] : d == 1 ? u[1] : u[2]), &sn, &cs);
            for (int k = k0 + b; k < k0 + NFREQ / 2; k += 3) {
                *reinterpret_cast<__nv_bfloat162*>(row + 6 + 6 * k + 2 * d) = __floats2bfloat162_rn(sn, cs);
                const float s2 = 2.0f * sn * cs, c2 = 1.0f - 2.0f * sn * sn;
                sn = s2; cs = c2;
            }
        }
    };
    float lossAcc = 0.f;
    int tile = blockIdx.x * TRAIN_TILES + tg;
    // the first tile's features need only the samples, which the launch before this one does not write
    if (tile * 16 < batch) features(tile);
    after_previous();
    let_next_in();
    for (int k = threadIdx.x; k < ALL_U4; k += TRAIN_THREADS) copy_async16(smem_t + k, reinterpret_cast<const uint4*>(wbf) + k);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int k = threadIdx.x; k < NBIAS; k += TRAIN_THREADS) sB[k] = bias[k];
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (bool first = true; tile * 16 < batch; tile += gridDim.x * TRAIN_TILES, first = false) {
        if (!first) {
            features(tile);
            tile_sync(tg);
        }
        {   // H0 in the pair layout
            uint32_t* h0 = H0 + (long long)tile * 8 * KIN;
            for (int w = tid; w < 8 * KIN; w += 128) {
                const int p = w / KIN, f = w - p * KIN;
                __nv_bfloat162 v;
                v.x = sF[(2 * p) * RS1 + f];
                v.y = sF[(2 * p + 1) * RS1 + f];
                h0[w] = *reinterpret_cast<uint32_t*>(&v);
            }
        }
        float C[2][4], z[4][8];
        uint32_t w[2][2];
        bias_quarter(C, sB, wq, lane);
#pragma unroll
        for (int kt = 0; kt < KIN / 16; ++kt) {
            uint32_t a[4], b[4];
            load_a(sF, RS1, kt, lane, a);
            load_b2(sW + OFF_WT1, RS1, 2 * wq, kt, lane, b);
            mma16816(C[0], a[0], a[1], a[2], a[3], b[0], b[1]);
            mma16816(C[1], a[0], a[1], a[2], a[3], b[2], b[3]);
        }
        const int wt[3] = {OFF_WT2, OFF_WT3, OFF_WT4}, wn[3] = {OFF_WN2, OFF_WN3, OFF_WN4};
#pragma unroll
        for (int l = 0; l < 4; ++l) {   // C = pre-activations of layer l + 1
#pragma unroll
            for (int q = 0; q < 2; ++q) {
#pragma unroll
                for (int e = 0; e < 4; ++e) z[l][4 * q + e] = C[q][e];
                w[q][0] = silu2(C[q][0], C[q][1]);
                w[q][1] = silu2(C[q][2], C[q][3]);
            }
            store_act(w, act[l & 1], H1 + l * B2 * HID + (long long)tile * 8 * HID, wq, lane);
            tile_sync(tg);
            if (l < 3) {
                bias_quarter(C, sB + (l + 1) * HID, wq, lane);
                layer_quarter(C, act[l & 1], sW + wt[l], wq, lane);
            }
        }
        // the output, by every warp: rows g and g + 8 in the lanes with i = 0
        float C5[4];
        {
            const float2 v = *reinterpret_cast<const float2*>(sB + 4 * HID + 2 * i);
            C5[0] = v.x; C5[1] = v.y; C5[2] = v.x; C5[3] = v.y;
        }
#pragma unroll
        for (int kt = 0; kt < 4; ++kt) {
            uint32_t a[4], b0, b1;
            load_a(act[1], RSH, kt, lane, a);
            load_b(sW + OFF_WT5, RSH, 0, kt, lane, b0, b1);
            mma16816(C5, a[0], a[1], a[2], a[3], b0, b1);
        }
        const float y0 = __shfl_sync(0xffffffffu, C5[0], lane & ~3), y1 = __shfl_sync(0xffffffffu, C5[2], lane & ~3);
        const float e0 = y0 - sT[g], e1 = y1 - sT[g + 8], w0 = sT[16 + g], w1 = sT[16 + g + 8];
        const float inv = 1.0f / (float)batch;
        const float dy0 = 2.0f * w0 * e0 * inv, dy1 = 2.0f * w1 * e1 * inv;
        if (wq == 0) {
            if (i == 0) lossAcc += w0 * e0 * e0 + w1 * e1 * e1;
            float D5[8][4] = {};
            if (i == 0) { D5[0][0] = dy0; D5[0][2] = dy1; }   // column 0 only
            store_pairs(D5, 1, dZ5 + (long long)tile * 8 * OUTN, OUTN, lane);
        }
        // dH4 = dy * W5[:, 0], then through SiLU
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int n0 = (2 * wq + q) * 8 + 2 * i;
            const float w50 = __bfloat162float(sW[OFF_WT5 + n0]), w51 = __bfloat162float(sW[OFF_WT5 + n0 + 1]);
            C[q][0] = dy0 * w50 * silu_grad(z[3][4 * q + 0]);
            C[q][1] = dy0 * w51 * silu_grad(z[3][4 * q + 1]);
            C[q][2] = dy1 * w50 * silu_grad(z[3][4 * q + 2]);
            C[q][3] = dy1 * w51 * silu_grad(z[3][4 * q + 3]);
        }
#pragma unroll
        for (int l = 3; l >= 0; --l) {   // C = dZ of layer l + 1; produce dZ of layer l
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                w[q][0] = pack_bf16(C[q][0], C[q][1]);
                w[q][1] = pack_bf16(C[q][2], C[q][3]);
            }
            // act[1] was last read for the output, act[0] before the barrier of layer 4
            __nv_bfloat16* T = act[(l & 1) ^ 1];
            store_act(w, l > 0 ? T : nullptr, dZ1 + l * B2 * HID + (long long)tile * 8 * HID, wq, lane);
            if (l == 0) break;
            tile_sync(tg);
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int e = 0; e < 4; ++e) C[q][e] = 0.f;
            layer_quarter(C, T, sW + wn[l - 1], wq, lane);
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int e = 0; e < 4; ++e) C[q][e] *= silu_grad(z[l - 1][4 * q + e]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lossAcc += __shfl_xor_sync(0xffffffffu, lossAcc, o);
    if (wq == 0 && lane == 0) atomicAdd(lossSum, lossAcc);
}

// Weight and bias gradients, all five layers in one launch: dW_l = H_{l-1}^T dZ_l, db_l = 1^T dZ_l.  A
// block owns one layer for a part of the batch (512 samples; `rounds` of them in batches beyond 32,768): it
// brings both operands into shared memory whole (16-byte copies in four groups; rows padded by eight
// words, which keeps the fragment reads free of bank conflicts), its warps multiply 16-row tiles -- layer
// 1 has seven of 64 columns, layers 2 to 4 four of which two warps take 32 columns each, layer 5 four of
// eight; the bias is one more row of ones -- and it writes its sums to the part's own copy of the gradient,
// which k_nsdf_adam adds up: the sums do not depend on the order of the blocks.  The tensor cores cut an
// accumulator off where FP32 addition rounds, so the length of a chain of MMAs shows in the result: 512
// samples a chain is the length the gradient has always had, and a shorter one (128 samples, 64 parts, 10
// us) left training off by more than two runs of the atomic form differ.
// Bound: the latency of the copies and the chain.  8,192 samples (ncu): one warp per 16-row tile and 512
// samples, added with atomics, took 42 us, this form 11; a whole step of 8,192 samples took 19.4 us with it when 64 parts of
// 128 samples took 20.1.
constexpr int WG_SAMPLES = 512;
constexpr int WG_PAIRS = WG_SAMPLES / 2;
constexpr int WG_THREADS = 256;
constexpr int WG_PAD = 8;
constexpr size_t WG_SMEM = sizeof(uint32_t) * WG_PAIRS * (KIN + WG_PAD + HID + WG_PAD);
constexpr int WG_GROUPS = 4;    // copy groups of a part
constexpr int WG_CHUNK = 512;   // batches are a multiple of this

__global__ void __launch_bounds__(WG_THREADS) k_nsdf_wgrad(const uint32_t* acts, int batch, int rounds,
                                                           float* __restrict__ parts) {
    extern __shared__ uint4 smem_w[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int layer = blockIdx.x % 5 + 1, part = blockIdx.x / 5;
    const int chunks = batch / WG_SAMPLES, chunk0 = part * rounds, chunk1 = min(chunk0 + rounds, chunks);
    float* grads = parts + (size_t)part * NPARAM;
    const long long B2 = batch / 2;
    const uint32_t* H1 = acts + B2 * KIN;
    const uint32_t* dZ1 = H1 + 4 * B2 * HID;
    const int fin = layer == 1 ? KIN : HID, fout = layer == 5 ? OUTN : HID;
    const uint32_t* Hp = layer == 1 ? acts : H1 + (layer - 2) * B2 * HID;
    const uint32_t* dZ = dZ1 + (layer - 1) * B2 * HID;
    const int pW = layer == 1 ? P_W1 : layer == 2 ? P_W2 : layer == 3 ? P_W3 : layer == 4 ? P_W4 : P_W5;
    const int pB = layer == 1 ? P_B1 : layer == 2 ? P_B2 : layer == 3 ? P_B3 : layer == 4 ? P_B4 : P_B5;
    const int sa = fin + WG_PAD, sb = fout + WG_PAD;
    uint32_t* A = reinterpret_cast<uint32_t*>(smem_w);
    uint32_t* B = A + WG_PAIRS * sa;
    const int g = lane >> 2, i = lane & 3;
    after_previous();
    let_next_in();
    constexpr int GP = WG_PAIRS / WG_GROUPS;
    auto bring = [&](int chunk) {
        const uint32_t* a = Hp + (long long)chunk * WG_PAIRS * fin;
        const uint32_t* b = dZ + (long long)chunk * WG_PAIRS * fout;
        for (int q = 0; q < WG_GROUPS; ++q) {
            for (int k = threadIdx.x; k < GP * fin / 4; k += WG_THREADS) {
                const int r = q * GP + k / (fin / 4), c = 4 * (k % (fin / 4));
                copy_async16(A + r * sa + c, a + r * fin + c);
            }
            for (int k = threadIdx.x; k < GP * fout / 4; k += WG_THREADS) {
                const int r = q * GP + k / (fout / 4), c = 4 * (k % (fout / 4));
                copy_async16(B + r * sb + c, b + r * fout + c);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    };
    auto landed = [&](int q) {   // groups 0 .. q are in shared memory
        if (q == 0) asm volatile("cp.async.wait_group 3;" ::: "memory");
        else if (q == 1) asm volatile("cp.async.wait_group 2;" ::: "memory");
        else if (q == 2) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
    };
    // every warp of the block goes through the same rounds; `rows`: it has a tile (mt, columns n0..);
    // `ones`: it has the bias of its columns
    auto tile = [&](bool rows, bool ones, int mt, int n0, auto ntiles) {
        constexpr int NT = decltype(ntiles)::value;
        float S[2][NT][4];   // [0] the tile's, [1] the bias's
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int q = 0; q < 4; ++q) S[0][nt][q] = S[1][nt][q] = 0.f;
        const uint32_t one = g == 0 ? pack_bf16(1.0f, 1.0f) : 0u;
        for (int chunk = chunk0; chunk < chunk1; ++chunk) {
            if (chunk > chunk0) __syncthreads();   // the last round's reads come before its copies
            bring(chunk);
            float C[2][NT][4];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int q = 0; q < 4; ++q) C[0][nt][q] = C[1][nt][q] = 0.f;
            for (int q = 0; q < WG_GROUPS; ++q) {
                landed(q);
#pragma unroll
                for (int k = 0; k < GP / 8; ++k) {
                    const int row = q * GP + 8 * k + i;   // sample pairs of k rows 2i.. and 2i+8..
                    const uint32_t* a = A + row * sa + mt * 16 + g;
                    const uint32_t* b = B + row * sb + n0 + g;
                    if (rows)
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt)
                            mma16816(C[0][nt], a[0], a[8], a[4 * sa], a[4 * sa + 8], b[nt * 8], b[4 * sb + nt * 8]);
                    if (ones)
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt) mma16816(C[1][nt], one, 0u, one, 0u, b[nt * 8], b[4 * sb + nt * 8]);
                }
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int q = 0; q < 4; ++q) { S[0][nt][q] += C[0][nt][q]; S[1][nt][q] += C[1][nt][q]; }
        }
        if (rows) {
            float* out = grads + pW + (mt * 16 + g) * fout + n0 + 2 * i;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                *reinterpret_cast<float2*>(out + nt * 8) = make_float2(S[0][nt][0], S[0][nt][1]);
                *reinterpret_cast<float2*>(out + 8 * fout + nt * 8) = make_float2(S[0][nt][2], S[0][nt][3]);
            }
        }
        if (ones && g == 0)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                grads[pB + n0 + nt * 8 + 2 * i] = S[1][nt][0];
                grads[pB + n0 + nt * 8 + 2 * i + 1] = S[1][nt][1];
            }
    };
    if (layer == 1) tile(warp < KIN / 16, warp == KIN / 16, warp, 0, std::integral_constant<int, 8>{});
    else if (layer < 5) tile(true, warp < 2, warp >> 1, (warp & 1) * 32, std::integral_constant<int, 4>{});
    else tile(warp < 4, warp == 4, warp, 0, std::integral_constant<int, 1>{});
}

// Parameter p's places in the bf16 weight block / bias vector.
__device__ __forceinline__ void publish(int p, float w, __nv_bfloat16* wbf, float* bias) {
    const __nv_bfloat16 b = __float2bfloat16(w);
    if (p < P_B1) {
        const int in = p / HID, out = p % HID;
        wbf[OFF_WT1 + out * RS1 + in] = b;
    } else if (p < P_W2) {
        bias[p - P_B1] = w;
    } else if (p < P_B4 + HID) {
        const int l = (p - P_W2) / (HID * HID + HID);           // 0..2 for W2..W4 (+ biases)
        const int r = (p - P_W2) - l * (HID * HID + HID);
        if (r < HID * HID) {
            const int in = r / HID, out = r % HID;
            const int wt = l == 0 ? OFF_WT2 : (l == 1 ? OFF_WT3 : OFF_WT4);
            const int wn = l == 0 ? OFF_WN2 : (l == 1 ? OFF_WN3 : OFF_WN4);
            wbf[wt + out * RSH + in] = b;
            wbf[wn + in * RSH + out] = b;
        } else {
            bias[(l + 1) * HID + (r - HID * HID)] = w;
        }
    } else if (p < P_B5) {
        const int in = (p - P_W5) / OUTN, out = (p - P_W5) % OUTN;
        wbf[OFF_WT5 + out * RSH + in] = b;
    } else {
        bias[4 * HID + (p - P_B5)] = w;
    }
}

// The bf16 / bias copies of the fp32 master parameters, which the kernels read.
__global__ void k_nsdf_publish(const float* __restrict__ params, __nv_bfloat16* __restrict__ wbf, float* __restrict__ bias) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < NPARAM) publish(p, params[p], wbf, bias);
}

// A sum that carries its rounding error along (D. E. Knuth, The Art of Computer Programming 2, 4.2.2, theorem B:
// the error of a floating-point addition is itself a float).  The value is the exact sum rounded once, but for the
// rounding of the errors' own sum, 2^-24 of it.
struct CarrySum {
    float sum = 0.f, rest = 0.f;
    __device__ __forceinline__ void add(float x, float r = 0.f) {
        const float s = sum + x, b = s - sum;
        rest += ((sum - (s - b)) + (x - b)) + r;
        sum = s;
    }
    __device__ __forceinline__ void add(const CarrySum& x) { add(x.sum, x.rest); }
    __device__ __forceinline__ float value() const { return sum + rest; }
};

// The gradient as the sum of its `nparts` parts, Adam (Kingma & Ba 2015) on the fp32 master parameters, then
// their copies.  Eight lanes share four consecutive parameters: each adds an eighth of the parts, every other
// lane updates one parameter.  The parts were once added by atomics in the order in which blocks ended, and
// every order rounds differently: training follows such a difference (a weight at a bf16 boundary flips, and the
// gradients part by 1e-5 to 1e-3 within 64 steps).  The exact sum is the middle of what the orders give:
// after 40 steps of 4,608 samples its gradients are at 6e-8 from a run with atomics in the median, where two such
// runs are at 2e-5 (and a fixed tree of FP32 additions was at 1e-5).  It costs 0.3 us of a step's 19.8 (8,192
// samples).
constexpr int ADAM_THREADS = 256;
static_assert(NPARAM % 4 == 0, "parameters are summed four at a time");
__global__ void __launch_bounds__(ADAM_THREADS) k_nsdf_adam(float* __restrict__ params, const float* parts, int nparts,
                                                            float* __restrict__ grads, float* __restrict__ m, float* __restrict__ v,
                                                            int step, float lr, __nv_bfloat16* __restrict__ wbf,
                                                            float* __restrict__ bias) {
    const int t = blockIdx.x * ADAM_THREADS + threadIdx.x;
    const int quad = t >> 3, lane8 = t & 7;
    const bool mine = quad < NPARAM / 4, update = mine && (lane8 & 1) == 0;
    const int p = 4 * quad + (lane8 >> 1);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float corr1 = 1.0f - powf(b1, (float)step), corr2 = 1.0f - powf(b2, (float)step);
    after_previous();
    let_next_in();
    // behind the wait: the step before wrote these, and only the wait makes its writes visible here
    const float m0 = update ? m[p] : 0.f, v0 = update ? v[p] : 0.f, w0 = update ? params[p] : 0.f;
    CarrySum gr[4];
    if (mine) {
        const float4* src = reinterpret_cast<const float4*>(parts) + quad;
#pragma unroll 8
        for (int c = lane8; c < nparts; c += 8) {
            const float4 x = src[(size_t)c * (NPARAM / 4)];
            gr[0].add(x.x); gr[1].add(x.y); gr[2].add(x.z); gr[3].add(x.w);
        }
    }
    // the eight lanes' sums: a lane gives away two of its four parameters, then one of two, then adds its neighbour's
    auto from = [](const CarrySum& x, int o) {
        return CarrySum{__shfl_xor_sync(0xffffffffu, x.sum, o), __shfl_xor_sync(0xffffffffu, x.rest, o)};
    };
    const bool upper = lane8 & 4, odd = lane8 & 2;
    CarrySum pair[2] = {upper ? gr[2] : gr[0], upper ? gr[3] : gr[1]};
    pair[0].add(from(upper ? gr[0] : gr[2], 4));
    pair[1].add(from(upper ? gr[1] : gr[3], 4));
    CarrySum all = odd ? pair[1] : pair[0];
    all.add(from(odd ? pair[0] : pair[1], 2));
    all.add(from(all, 1));
    if (!update) return;
    const float g = all.value();
    grads[p] = g;
    const float mm = b1 * m0 + (1.0f - b1) * g;
    const float vv = b2 * v0 + (1.0f - b2) * g * g;
    m[p] = mm; v[p] = vv;
    const float mh = mm / corr1, vh = vv / corr2;
    float w = w0 - lr * mh / (sqrtf(vh) + eps);
    // the padding rows of the first layer and the unused output columns stay zero
    const bool pad = (p < P_B1 && p / HID >= NFEAT) || (p >= P_W5 && p < P_B5 && (p - P_W5) % OUTN != 0) || (p >= P_B5 && p != P_B5);
    if (pad) w = 0.f;
    params[p] = w;
    publish(p, w, wbf, bias);
}

// Uniform fan-in initialisation (He-style bound for SiLU), zero biases and padding.
__global__ void k_nsdf_init(float* __restrict__ params, uint32_t seed) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= NPARAM) return;
    float w = 0.f;
    int fanIn = 0;
    if (p < P_B1) fanIn = p / HID < NFEAT ? NFEAT : 0;
    else if (p >= P_W2 && p < P_B4 + HID && ((p - P_W2) % (HID * HID + HID)) < HID * HID) fanIn = HID;
    else if (p >= P_W5 && p < P_B5 && (p - P_W5) % OUTN == 0) fanIn = HID;
    if (fanIn > 0) w = (2.0f * u01(hash32(seed ^ hash32((uint32_t)p))) - 1.0f) * sqrtf(6.0f / (float)fanIn);
    params[p] = w;
}

// ------------------------------------------------------------------------------------------ samples
__global__ void k_nsdf_sample(const float4* __restrict__ mesh, int nverts, const float* __restrict__ grid, SdfGrid g,
                              float band, float sigma, float3 sc, float sr, Pose pose, int count, uint32_t seed,
                              Sample* __restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count) return;
    uint32_t h = hash32(seed ^ hash32((uint32_t)t * 0x9E3779B9u));
    auto next = [&]() { h = hash32(h + 0x6D2B79F5u); return u01(h); };
    float3 p;
    if (next() < 0.75f) {   // near the surface: a mesh vertex, moved along its normal and sideways
        const int v = min(nverts - 1, (int)(next() * (float)nverts));
        const float4 pos = mesh[2 * v], nrm = mesh[2 * v + 1];
        const float u1 = fmaxf(next(), 1e-7f), u2 = next(), u3 = fmaxf(next(), 1e-7f), u4 = next();
        const float r1 = sqrtf(-2.0f * __logf(u1)), r2 = sqrtf(-2.0f * __logf(u3));
        const float n0 = r1 * __cosf(6.2831853f * u2), n1 = r1 * __sinf(6.2831853f * u2), n2 = r2 * __cosf(6.2831853f * u4);
        const float along = n0 * sigma;
        p = mk3(pos.x + nrm.x * along + n1 * 0.5f * sigma, pos.y + nrm.y * along + n2 * 0.5f * sigma,
                pos.z + nrm.z * along + (n1 - n2) * 0.35f * sigma);
    } else {                // anywhere in the grid box
        p = mk3(g.ox + next() * g.nx * g.cell, g.oy + next() * g.ny * g.cell, g.oz + next() * g.nz * g.cell);
    }
    const float d = sdf_lookup(grid, g, p);
    Sample S;
    S.x = p.x; S.y = p.y; S.z = p.z;
    S.p0 = pose.a0; S.p1 = pose.a1; S.p2 = pose.a2;
    if (d == 1e10f) {
        const float dx = p.x - sc.x, dy = p.y - sc.y, dz = p.z - sc.z;
        const bool outside = dx * dx + dy * dy + dz * dz > sr * sr;
        S.target = band;
        S.weight = outside ? 1.0f : 0.0f;
    } else {
        S.target = fminf(fmaxf(d / g.cell, -band), band);
        S.weight = 1.0f;
    }
    out[t] = S;
}

}  // namespace

// A training step's scratch: the minibatch's activations and gradients in the pair layout, then the parts
// of the weight gradient (at most TRAIN_PARTS, one per 512 samples or more).
constexpr int TRAIN_PARTS = 64;
static size_t acts_words(int batch) { return (size_t)batch / 2 * (KIN + 8 * HID + OUTN); }
size_t train_scratch_bytes(int batch) { return 4 * acts_words(batch) + sizeof(float) * (size_t)NPARAM * TRAIN_PARTS; }

cudaError_t launch_query(const __nv_bfloat16* wbf, const float* bias, const Frame& fr, const float4* points, int count,
                         Pose pose, float* out, cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(k_nsdf_query<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)QUERY_SMEM);
    if (e != cudaSuccess) return e;
    const int tiles = (count + 31) / 32;
    const int blocks = std::min((tiles + QUERY_WARPS - 1) / QUERY_WARPS, sm_count() * 8);
    k_nsdf_query<false><<<blocks, QUERY_WARPS * 32, QUERY_SMEM, s>>>(wbf, bias, fr, points, nullptr, count, pose, out);
    return cudaGetLastError();
}

cudaError_t launch_query_samples(const __nv_bfloat16* wbf, const float* bias, const Frame& fr, const Sample* samples,
                                 int count, float* out, cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(k_nsdf_query<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)QUERY_SMEM);
    if (e != cudaSuccess) return e;
    const int tiles = (count + 31) / 32;
    const int blocks = std::min((tiles + QUERY_WARPS - 1) / QUERY_WARPS, sm_count() * 8);
    k_nsdf_query<true><<<blocks, QUERY_WARPS * 32, QUERY_SMEM, s>>>(wbf, bias, fr, nullptr, samples, count, Pose{0, 0, 0},
                                                                    out);
    return cudaGetLastError();
}

cudaError_t launch_train_step(const TrainStep& t, cudaStream_t s) {
    if (t.batch <= 0 || t.batch % WG_CHUNK != 0 || t.poolSize <= 0) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(k_nsdf_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TRAIN_SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_nsdf_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WG_SMEM);
    if (e != cudaSuccess) return e;
    uint32_t* acts = static_cast<uint32_t*>(t.scratch);
    float* parts = reinterpret_cast<float*>(acts + acts_words(t.batch));
    const int blocks = std::min(t.batch / (16 * TRAIN_TILES), sm_count());
    if (t.first) {
        k_nsdf_train<<<blocks, TRAIN_THREADS, TRAIN_SMEM, s>>>(t.wbf, t.bias, t.fr, t.pool, t.poolSize, t.batch, t.seed, acts, t.lossSum);
        e = cudaGetLastError();
    } else {
        e = launch_after(k_nsdf_train, blocks, TRAIN_THREADS, TRAIN_SMEM, s, t.wbf, t.bias, t.fr, t.pool, t.poolSize, t.batch,
                         t.seed, acts, t.lossSum);
    }
    if (e != cudaSuccess) return e;
    const int chunks = t.batch / WG_SAMPLES, rounds = (chunks + TRAIN_PARTS - 1) / TRAIN_PARTS, nparts = (chunks + rounds - 1) / rounds;
    e = launch_after(k_nsdf_wgrad, (unsigned)nparts * 5, WG_THREADS, WG_SMEM, s, acts, t.batch, rounds, parts);
    if (e != cudaSuccess) return e;
    return launch_after(k_nsdf_adam, (NPARAM / 4 * 8 + ADAM_THREADS - 1) / ADAM_THREADS, ADAM_THREADS, 0, s, t.params, parts, nparts,
                        t.grads, t.m, t.v, t.step, t.lr, t.wbf, t.bias);
}

cudaError_t launch_publish(const float* params, __nv_bfloat16* wbf, float* bias, cudaStream_t s) {
    k_nsdf_publish<<<(NPARAM + 255) / 256, 256, 0, s>>>(params, wbf, bias);
    return cudaGetLastError();
}

cudaError_t launch_init_params(float* params, uint32_t seed, __nv_bfloat16* wbf, float* bias, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(wbf, 0, sizeof(__nv_bfloat16) * WBF_ALL, s);
    if (e != cudaSuccess) return e;
    k_nsdf_init<<<(NPARAM + 255) / 256, 256, 0, s>>>(params, seed);
    return launch_publish(params, wbf, bias, s);
}

cudaError_t launch_sample(const float4* mesh, int nverts, const float* grid, const SdfGrid& g, float band, float sigma,
                          float3 sphereCentre, float sphereRadius, Pose pose, int count, uint32_t seed, Sample* out,
                          cudaStream_t s) {
    if (count <= 0 || nverts <= 0) return cudaSuccess;
    k_nsdf_sample<<<(count + 255) / 256, 256, 0, s>>>(mesh, nverts, grid, g, band, sigma, sphereCentre, sphereRadius, pose,
                                                      count, seed, out);
    return cudaGetLastError();
}

}  // namespace nsdf
}  // namespace tfx

// ================================================================================================
// collision with the proxy
namespace tfx {
namespace nsdf {
namespace {

__device__ __forceinline__ void mark_block(uint32_t* marks, const SdfGrid& g, int3 c) {
    for (int dz = 0; dz < 3; ++dz)
        for (int dy = 0; dy < 3; ++dy)
            for (int dx = 0; dx < 3; ++dx) {
                const int x = c.x + dx, y = c.y + dy, z = c.z + dz;
                if (x < 0 || y < 0 || z < 0 || x >= g.nx || y >= g.ny || z >= g.nz) continue;
                const long long cell = ((long long)z * g.ny + y) * g.nx + x;
                atomicOr(marks + (cell >> 5), 1u << (cell & 31));
            }
}

__global__ void __launch_bounds__(QUERY_WARPS * 32) k_nsdf_classify(CollideArgs a) {
    extern __shared__ uint4 smem_c[];
    __nv_bfloat16* sW = reinterpret_cast<__nv_bfloat16*>(smem_c);
    float* sB = reinterpret_cast<float*>(sW + WBF_FWD);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __nv_bfloat16* sF = reinterpret_cast<__nv_bfloat16*>(sB + NBIAS) + warp * 32 * RS1;
    stage_weights<FWD_U4>(smem_c, a.wbf, sB, a.bias);
    __syncthreads();
    const Frame fr = a.fr;
    const int g = lane >> 2, i = lane & 3;
    const long long nw = (long long)gridDim.x * QUERY_WARPS;
    const float limit = a.margin / fr.cell + a.slackCells;   // band: network distance below margin + slack
    for (long long tile = (long long)blockIdx.x * QUERY_WARPS + warp; tile * 32 < a.vtot; tile += nw) {
        const long long v = tile * 32 + lane;
        const bool valid = v < a.vtot;
        const float4 P = valid ? a.pos[v] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float ux = (P.x - fr.cx) * fr.ihx, uy = (P.y - fr.cy) * fr.ihy, uz = (P.z - fr.cz) * fr.ihz;
        const float p0 = a.pose.a0 * fr.poseScale, p1 = a.pose.a1 * fr.poseScale, p2 = a.pose.a2 * fr.poseScale;
        write_features(sF, lane, 0, ux, uy, uz, p0, p1, p2, valid);
        write_features(sF, lane, 1, ux, uy, uz, p0, p1, p2, valid);
        __syncwarp();
        float y[4];
        mlp_forward32(sW, sB, sF, lane, y);
        __syncwarp();
        if (i == 0) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const long long vr = tile * 32 + (r >> 1) * 16 + g + 8 * (r & 1);
                if (vr >= a.vtot || (int)(vr % a.n) < 2 || !(y[r] < limit)) continue;
                a.bandList[atomicAdd(a.bandCount, 1)] = (int)vr;
                const float4 pv = a.pos[vr];
                mark_block(a.marks, a.grid, sdf_coords(a.grid, mk3(pv.x, pv.y, pv.z)));
            }
        }
    }
}

// Words of the per-cell marks (the coarse map of 4x4x4-cell blocks follows them).
__host__ __device__ __forceinline__ long long mark_words(long long cells) { return (cells + 31) / 32; }
__host__ __device__ __forceinline__ int coarse_dim(int n) { return (n + 3) >> 2; }

// The words' initial value, and the coarse map: the block of every marked cell.
__global__ void __launch_bounds__(256) k_gated_init(uint32_t* __restrict__ w, const uint32_t* __restrict__ marks,
                                                    uint32_t* __restrict__ coarse, SdfGrid g, const int* __restrict__ count) {
    if (*count == 0) return;
    const uint32_t v = float_flip3(1e10f);
    const long long cells = (long long)g.nx * g.ny * g.nz;
    const int cbx = coarse_dim(g.nx), cby = coarse_dim(g.ny);
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < cells; c += (long long)gridDim.x * blockDim.x) {
        w[c] = v;
        if ((__ldg(marks + (c >> 5)) >> (c & 31)) & 1u) {
            const long long nxy = (long long)g.nx * g.ny;
            const int z = (int)(c / nxy);
            const long long r = c - (long long)z * nxy;
            const int y = (int)(r / g.nx), x = (int)(r - (long long)y * g.nx);
            const int b = ((z >> 2) * cby + (y >> 2)) * cbx + (x >> 2);
            atomicOr(coarse + (b >> 5), 1u << (b & 31));
        }
    }
}

// ConstructSignedDistanceField (TressFXSDFCollision.hlsl:329-397) restricted to marked cells: every
// (triangle, cell) pair of a marked cell is evaluated, so each marked cell gets its exact value.  A
// warp takes a triangle, its lanes test the 4x4x4-cell blocks the reference's cell box overlaps, and a
// triangle whose box holds no marked cell is left at once (it contributes to no marked cell).  Box
// coordinates use the float reciprocal only below 2^22 cells, where it gives the integer quotient
// (as in the full construct).
__global__ void __launch_bounds__(256) k_gated_construct(CollideArgs a) {
    if (*a.bandCount == 0) return;
    const SdfGrid g = a.grid;
    const int lane = threadIdx.x & 31;
    const int warpsTotal = gridDim.x * (blockDim.x >> 5);
    const long long cells = (long long)g.nx * g.ny * g.nz;
    const uint32_t* coarse = a.marks + mark_words(cells);
    const int cbx = coarse_dim(g.nx), cby = coarse_dim(g.ny);
    for (int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < a.ntri; t += warpsTotal) {
        const float3 x0 = xyz(__ldg(a.mesh + 2 * (size_t)__ldg(a.indices + 3 * t + 0)));
        const float3 x1 = xyz(__ldg(a.mesh + 2 * (size_t)__ldg(a.indices + 3 * t + 1)));
        const float3 x2 = xyz(__ldg(a.mesh + 2 * (size_t)__ldg(a.indices + 3 * t + 2)));
        int3 lo, hi;
        tri_cell_box(g, x0, x1, x2, lo, hi);
        const int bx0 = lo.x >> 2, by0 = lo.y >> 2, bz0 = lo.z >> 2;
        const int nbx = (hi.x >> 2) - bx0 + 1, nby = (hi.y >> 2) - by0 + 1, nbz = (hi.z >> 2) - bz0 + 1;
        const int nb = nbx * nby * nbz;
        bool any = false;
        for (int k = lane; k < nb && !any; k += 32) {
            const int kz = k / (nbx * nby), kr = k - kz * nbx * nby, ky = kr / nbx, kx = kr - ky * nbx;
            const int b = ((bz0 + kz) * cby + (by0 + ky)) * cbx + (bx0 + kx);
            any = (__ldg(coarse + (b >> 5)) >> (b & 31)) & 1u;
        }
        if (!__any_sync(0xffffffffu, any)) continue;
        const int nx = hi.x - lo.x + 1, ny = hi.y - lo.y + 1, nz = hi.z - lo.z + 1;
        const int nxy = nx * ny, vol = nxy * nz;
        const bool floatIdx = vol < (1 << 22);
        const float inxy = 1.0f / (float)nxy, inx = 1.0f / (float)nx;
        const TriPre P = tri_pre(x0, x1, x2);
        for (int c = lane; c < vol; c += 32) {
            int cz, r, cy;
            if (floatIdx) {
                cz = (int)(((float)c + 0.5f) * inxy);
                r = c - cz * nxy;
                cy = (int)(((float)r + 0.5f) * inx);
            } else {
                cz = c / nxy;
                r = c - cz * nxy;
                cy = r / nx;
            }
            const int x = lo.x + (r - cy * nx), y = lo.y + cy, z = lo.z + cz;
            const long long cell = ((long long)z * g.ny + y) * g.nx + x;
            if (!((__ldg(a.marks + (cell >> 5)) >> (cell & 31)) & 1u)) continue;
            atomicMin(a.words + cell, float_flip3(signed_dist_pre(sdf_cell_pos(g, x, y, z), P)));
        }
    }
}

__global__ void __launch_bounds__(256) k_gated_finalize(uint32_t* __restrict__ w, long long cells, const int* __restrict__ count) {
    if (*count == 0) return;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < cells; c += (long long)gridDim.x * blockDim.x)
        w[c] = ifloat_flip3(w[c]);
}

__global__ void __launch_bounds__(256) k_band_collide(CollideArgs a) {
    const int cnt = *a.bandCount;
    const float* sdf = reinterpret_cast<const float*>(a.words);
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < cnt; k += gridDim.x * blockDim.x) {
        const int v = a.bandList[k];
        const float4 p = a.pos[v];
        float3 proj;
        if (sdf_collide_point<ReadOnlyLoad>(sdf, a.grid, a.margin, xyz(p), proj)) {
            a.pos[v] = with_xyz(p, proj);
            a.prev[v] = with_xyz(a.prev[v], proj);
        }
    }
}

}  // namespace

cudaError_t launch_collide(const CollideArgs& a, cudaStream_t s) {
    if (a.vtot <= 0) return cudaSuccess;
    const long long cells = (long long)a.grid.nx * a.grid.ny * a.grid.nz;
    cudaError_t e = cudaMemsetAsync(a.bandCount, 0, sizeof(int), s);
    const long long coarseBits = (long long)coarse_dim(a.grid.nx) * coarse_dim(a.grid.ny) * coarse_dim(a.grid.nz);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(a.marks, 0, sizeof(uint32_t) * (size_t)(mark_words(cells) + (coarseBits + 31) / 32), s);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_nsdf_classify, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)QUERY_SMEM);
    if (e != cudaSuccess) return e;
    if (a.wtc) {   // the network on the tcgen05 path
        TcArgs t{};
        t.wtc = a.wtc; t.fr = a.fr; t.pose = a.pose; t.pts = a.pos; t.err = a.err;
        t.vtot = a.vtot; t.n = a.n; t.margin = a.margin; t.slackCells = a.slackCells; t.grid = a.grid;
        t.bandList = a.bandList; t.bandCount = a.bandCount; t.marks = a.marks;
        e = launch_classify_tc(t, s);
        if (e != cudaSuccess) return e;
    } else {
        const long long tiles = (a.vtot + 31) / 32;
        const int blocks = (int)std::min<long long>((tiles + QUERY_WARPS - 1) / QUERY_WARPS, sm_count() * 8);
        k_nsdf_classify<<<blocks, QUERY_WARPS * 32, QUERY_SMEM, s>>>(a);
    }
    const unsigned gc = (unsigned)std::min<long long>((cells + 255) / 256, (long long)sm_count() * 16);
    k_gated_init<<<gc, 256, 0, s>>>(a.words, a.marks, a.marks + mark_words(cells), a.grid, a.bandCount);
    if (a.ntri > 0) k_gated_construct<<<(unsigned)std::min(( a.ntri + 7) / 8, sm_count() * 32), 256, 0, s>>>(a);
    k_gated_finalize<<<gc, 256, 0, s>>>(a.words, cells, a.bandCount);
    k_band_collide<<<sm_count() * 4, 256, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace nsdf
}  // namespace tfx
