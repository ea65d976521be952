// Device-side SDF helpers shared by the plain SDF kernels and the batched (tiled) build / fused
// collide: FloatFlip3 encoding, grid coordinates, signed point-triangle distance and the
// trilinear lookup of src/Shaders/TressFXSDFCollision.hlsl, evaluated in the reference's order.
#pragma once
#include "tfx_cell_queue.cuh"
#include "tfx_device_math.cuh"
#include "tfx_internal.h"

namespace tfx {

// FloatFlip3 / IFloatFlip3, TressFXSDFCollision.hlsl:92-100
__device__ __forceinline__ uint32_t float_flip3(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u << 1) | (u >> 31);
}
__device__ __forceinline__ uint32_t ifloat_flip3(uint32_t u) { return (u >> 1) | (u << 31); }

// True when p certainly fails the lookup's bounds test 0 <= ftoi((p - origin) / cell) < dims - 2 on
// some axis, decided without the division.  d = p - origin is the reference's own first operation;
// d <= -2 cell (exact product) gives a quotient <= -2, and d >= RN(dims * cell) >= dims * cell *
// (1 - 2^-24) gives a quotient that truncates to dims - 1 or more (division is monotonic, dims is far
// below 2^22).  Infinite d goes the same way as the reference (its quotient saturates); NaN and the
// points near the range's faces take the exact path.
__device__ __forceinline__ bool sdf_surely_outside(const SdfGrid& g, float3 p) {
    const float dx = p.x - g.ox, dy = p.y - g.oy, dz = p.z - g.oz;
    const float lo = -2.0f * g.cell;
    return dx <= lo || dy <= lo || dz <= lo || dx >= (float)g.nx * g.cell || dy >= (float)g.ny * g.cell ||
           dz >= (float)g.nz * g.cell;
}

// GetSdfCoordinates, :103-113
__device__ __forceinline__ int3 sdf_coords(const SdfGrid& g, float3 p) {
    const float sx = (p.x - g.ox) / g.cell, sy = (p.y - g.oy) / g.cell, sz = (p.z - g.oz) / g.cell;
    return make_int3(ftoi(sx), ftoi(sy), ftoi(sz));
}
// GetSdfCellPosition, :115-121
__device__ __forceinline__ float3 sdf_cell_pos(const SdfGrid& g, int x, int y, int z) {
    const float3 c = mk3((float)x * g.cell, (float)y * g.cell, (float)z * g.cell);
    return add(c, mk3(g.ox, g.oy, g.oz));
}

// SignedDistancePointToTriangle (:163-215) and DistancePointToEdge (:147-159) split in two: the
// triangle-only terms, computed once per triangle, and signed_dist_pre(p, T), the per-cell part.
// Every term is the shader's expression on the same inputs in the same order, so the distance is
// bit-identical to evaluating the two functions per cell.
struct TriPre {
    float3 x0, x1, x2;
    float3 x02n, x12n;   // normalised edge frame
    float l0, l1, l2;
    float3 nTri;
    float3 e01, e12, e02; // x1-x0, x2-x1, x2-x0 (the x10 of the three edge calls)
    float d01, d12, d02;  // dot(x10, x10) of the three edge calls
};

__device__ __forceinline__ TriPre tri_pre(float3 x0, float3 x1, float3 x2) {
    TriPre T;
    T.x0 = x0; T.x1 = x1; T.x2 = x2;
    float3 x02 = sub(x0, x2);
    T.l0 = length(x02) + 1e-30f;
    T.x02n = divs(x02, T.l0);
    float3 x12 = sub(x1, x2);
    T.l1 = dot(x12, T.x02n);
    x12 = sub(x12, mul(T.l1, T.x02n));
    T.l2 = length(x12) + 1e-30f;
    T.x12n = divs(x12, T.l2);
    T.nTri = cross(sub(x1, x0), sub(x2, x0));
    T.e01 = sub(x1, x0); T.d01 = dot(T.e01, T.e01);
    T.e12 = sub(x2, x1); T.d12 = dot(T.e12, T.e12);
    T.e02 = sub(x2, x0); T.d02 = dot(T.e02, T.e02);
    return T;
}

// Squared DistancePointToEdge(p, a, b) with x10 = b - a and dot(x10, x10) precomputed: the value
// whose sqrtf the reference takes.
__device__ __forceinline__ float edge_dist2_pre(float3 p, float3 a, float3 b, float3 x10, float dd) {
    float t = dot(sub(b, p), x10) / dd;
    t = fmaxf(0.0f, fminf(t, 1.0f));
    const float3 q = sub(p, add(mul(t, a), mul(1.0f - t, b)));
    return dot(q, q);
}

// SignedDistancePointToTriangle with one square root: the reference takes sqrtf of the face
// distance, or of each edge distance and then the minimum; sqrtf is correctly rounded and so
// monotone, hence min(sqrtf(u), sqrtf(v)) == sqrtf(min(u, v)) and the result is the same float.
__device__ __forceinline__ float signed_dist_pre(float3 p, const TriPre& T) {
    const float3 px2 = sub(p, T.x2);
    const float b = dot(T.x12n, px2) / T.l2;
    const float a = (dot(T.x02n, px2) - T.l1 * b) / T.l0;
    const float c = (1.0f - a) - b;
    const float tol = 1e-8f;
    float d2;
    if (a >= -tol && b >= -tol && c >= -tol) {
        const float3 nn = sub(p, add(add(mul(a, T.x0), mul(b, T.x1)), mul(c, T.x2)));
        d2 = dot(nn, nn);
    } else {
        const float u01 = edge_dist2_pre(p, T.x0, T.x1, T.e01, T.d01);
        const float u12 = edge_dist2_pre(p, T.x1, T.x2, T.e12, T.d12);
        const float u02 = edge_dist2_pre(p, T.x0, T.x2, T.e02, T.d02);
        d2 = fminf(fminf(u01, u12), u02);
    }
    float d = sqrtf(d2);
    d = (dot(sub(p, T.x0), T.nTri) < 0.0f) ? -d : d;
    return d;
}

// The cell box ConstructSignedDistanceField visits for a triangle (:351-363): AABB +- one cell,
// grid coordinates -+ GRID_MARGIN, clamped to the grid.
__device__ __forceinline__ void tri_cell_box(const SdfGrid& g, float3 t0, float3 t1, float3 t2, int3& lo, int3& hi) {
    const float3 m = mk3(g.cell, g.cell, g.cell);
    const float3 aabbMin = sub(vmin(t0, vmin(t1, t2)), m);
    const float3 aabbMax = add(vmax(t0, vmax(t1, t2)), m);
    lo = sdf_coords(g, aabbMin);
    hi = sdf_coords(g, aabbMax);
    lo.x = max(0, min(lo.x - 1, g.nx - 1)); lo.y = max(0, min(lo.y - 1, g.ny - 1)); lo.z = max(0, min(lo.z - 1, g.nz - 1));
    hi.x = max(0, min(hi.x + 1, g.nx - 1)); hi.y = max(0, min(hi.y + 1, g.ny - 1)); hi.z = max(0, min(hi.z + 1, g.nz - 1));
}

// What ConstructSignedDistanceField (:329-397) computes once per triangle: its invariants, the
// reference's cell box, the grid that box indexes, and the terms of a lower bound on the triangle's
// distance at the box's cells (sdf_construct_job_warp).  A thread makes a job; a warp runs its cell loop
// with the job in shared memory.  Every value is the shader's expression on the same inputs, so making it
// once per triangle instead of once per cell changes no result.  64 words: the first 20 are what the
// loop keeps in registers, the rest what an evaluated cell reads.
struct alignas(16) TriJob {
    float hx, hy, hz, h0;           // distance along the unit normal: h0 at the box's corner, the steps per cell
    float bx, by, bz, cell;         // corner of the box less the centroid; cell size
    float R, slack, inxy, inx;      // radius around the centroid; absolute slack of the bound; 1 / nxy, 1 / nx
    float nx, nxy, plane, gnx;      // cells of a box row and slice, of a grid slice and row
    int vol, narrow;                // cells of the box; see below
    uint32_t* first;                // the word of the box's first cell
    float ox, oy, oz;               // the grid's origin
    float lox, loy, loz;            // the box's first cell
    float rl0, rl2, r01, r12, r02;  // reciprocals of the five divisors of the distance
    int ranged;                     // the divisors and the box are in div_by's range
    float3 x0, x1, x2, x02n, x12n, nTri, e01, e12;   // as in TriPre
    float l0, l1, l2, d01, d12, d02;
    float pad[2];
};
static_assert(sizeof(TriJob) == 256, "a triangle job is 64 words");
// narrow: the box has fewer than 2^20 cells, and it and its offsets in the grid count exactly in floats.
// Otherwise nx, nxy, plane (rows per grid slice), gnx and lox, loy, loz hold the integers' bits.

__device__ __forceinline__ TriPre job_pre(const TriJob& J) {
    TriPre T;
    T.x0 = J.x0; T.x1 = J.x1; T.x2 = J.x2; T.x02n = J.x02n; T.x12n = J.x12n; T.nTri = J.nTri;
    T.l0 = J.l0; T.l1 = J.l1; T.l2 = J.l2;
    T.e01 = J.e01; T.e12 = J.e12; T.e02 = sub(J.x2, J.x0);
    T.d01 = J.d01; T.d12 = J.d12; T.d02 = J.d02;
    return T;
}

__device__ __forceinline__ TriJob tri_job(const SdfGrid& g, uint32_t* words, float3 x0, float3 x1, float3 x2) {
    TriJob J;
    int3 lo, hi;
    tri_cell_box(g, x0, x1, x2, lo, hi);
    const TriPre P = tri_pre(x0, x1, x2);
    J.x0 = x0; J.x1 = x1; J.x2 = x2; J.x02n = P.x02n; J.x12n = P.x12n; J.nTri = P.nTri; J.e01 = P.e01; J.e12 = P.e12;
    J.l0 = P.l0; J.l1 = P.l1; J.l2 = P.l2; J.d01 = P.d01; J.d12 = P.d12; J.d02 = P.d02;
    J.ox = g.ox; J.oy = g.oy; J.oz = g.oz; J.cell = g.cell;
    const int nx = hi.x - lo.x + 1, ny = hi.y - lo.y + 1, nz = hi.z - lo.z + 1, nxy = nx * ny;
    J.vol = nxy * nz;
    const long long plane = (long long)g.ny * g.nx;
    J.first = words + (plane * lo.z + ((long long)lo.y * g.nx + lo.x));
    const int bound = 1 << 23;
    J.narrow = J.vol < (1 << 20) && plane * nz < bound && g.nx < bound && g.ny < bound && g.nz < bound;
    J.inxy = 1.0f / (float)nxy;
    J.inx = 1.0f / (float)nx;
    if (J.narrow) {
        J.nx = (float)nx; J.nxy = (float)nxy; J.plane = (float)plane; J.gnx = (float)g.nx;
        J.lox = (float)lo.x; J.loy = (float)lo.y; J.loz = (float)lo.z;
    } else {
        J.nx = __int_as_float(nx); J.nxy = __int_as_float(nxy); J.plane = __int_as_float(g.ny); J.gnx = __int_as_float(g.nx);
        J.lox = __int_as_float(lo.x); J.loy = __int_as_float(lo.y); J.loz = __int_as_float(lo.z);
    }
    // the bound's terms: c the centroid, m a unit normal (zero for a degenerate triangle, which leaves
    // the sphere bound), R = max |x_i - c|, w = max |<x_i - c, m>|
    const float3 c = mul(add(add(x0, x1), x2), 1.0f / 3.0f);
    const float3 a0 = sub(x0, c), a1 = sub(x1, c), a2 = sub(x2, c);
    const float R = sqrtf(fmaxf(fmaxf(dot(a0, a0), dot(a1, a1)), dot(a2, a2)));
    const float nn = dot(P.nTri, P.nTri);
    float3 m = mk3(0.0f, 0.0f, 0.0f);
    if (nn > 1e-30f && nn < 1e30f) m = mul(P.nTri, rsqrtf(nn));
    const float w = fmaxf(fmaxf(fabsf(dot(a0, m)), fabsf(dot(a1, m))), fabsf(dot(a2, m)));
    const float far = fmaxf(fmaxf(fabsf(x0.x) + fabsf(x0.y) + fabsf(x0.z), fabsf(x1.x) + fabsf(x1.y) + fabsf(x1.z)),
                            fabsf(x2.x) + fabsf(x2.y) + fabsf(x2.z)) + (fabsf(g.ox) + fabsf(g.oy) + fabsf(g.oz));
    const float3 b = sub(sdf_cell_pos(g, lo.x, lo.y, lo.z), c);
    J.bx = b.x; J.by = b.y; J.bz = b.z;
    J.hx = m.x * g.cell; J.hy = m.y * g.cell; J.hz = m.z * g.cell;
    J.h0 = dot(b, m);
    J.R = R;
    const float reach = fabsf(b.x) + fabsf(b.y) + fabsf(b.z) + g.cell * ((float)nx + (float)ny + (float)nz);
    J.slack = 0x1p-17f * (((far + reach) + R) + w) + (w + 2e-7f * R);
    auto fits = [](float v) { return v >= kDivisorMin && v <= kDivisorMax; };
    J.ranged = fits(P.l0) && fits(P.l2) && fits(P.d01) && fits(P.d12) && fits(P.d02) && reach + R < 0x1p30f;
    J.rl0 = 1.0f / P.l0; J.rl2 = 1.0f / P.l2;
    J.r01 = 1.0f / P.d01; J.r12 = 1.0f / P.d12; J.r02 = 1.0f / P.d02;
    J.pad[0] = J.pad[1] = 0.0f;
    return J;
}

// Squared DistancePointToEdge(p, a, b) for num = dot(b - p, b - a) and its quotient by dot(b - a, b - a).
__device__ __forceinline__ float edge_dist2_at(float3 p, float3 a, float3 b, float t) {
    t = fmaxf(0.0f, fminf(t, 1.0f));
    const float3 q = sub(p, add(mul(t, a), mul(1.0f - t, b)));
    return dot(q, q);
}

// A key of a numerator that is below kNumKey exactly where the numerator is below div_by's range and not zero (twice
// the bits less one, which makes a zero of either sign the largest).
__device__ __forceinline__ uint32_t num_key(float a) { return 2u * __float_as_uint(a) - 1u; }
constexpr uint32_t kNumKey = 2u * 0x21800000u - 1u;   // kDivMin's

// SignedDistancePointToTriangle of the job's triangle, the bits of signed_dist_pre: the five divisions are
// by the triangle's own invariants, so they take a multiplication and two fused multiply-adds with the
// job's reciprocals, and the square root the ranged form; a pair with a numerator below div_by's range or a
// squared distance outside sqrt_ranged's takes signed_dist_pre.  A numerator of exactly zero, which whole planes
// of cells have around an axis-aligned mesh, is fine: its quotient may come out as the other zero, which no
// comparison, clamp or square tells apart.  (Sent to signed_dist_pre as well, zeros made a box of 48 triangles in
// 128^3 take 192 us, 82 without; before the short forms it was 151.)  Above the range only `na` can lie (a
// needle: l1 b), and only a quotient beyond the floats would differ: `a` is then NaN where the operator gives an
// infinity, and either takes the edges.  dot(x2 - p, e) is -dot(p - x2, e): negation is exact and rounding
// symmetric.
__device__ __forceinline__ float signed_dist_job(float3 p, const TriJob& J) {
    const float3 x2 = J.x2, px2 = sub(p, x2);
    const float nb = dot(J.x12n, px2);
    const float b = div_by(nb, J.l2, J.rl2);
    const float na = dot(J.x02n, px2) - J.l1 * b;
    const float a = div_by(na, J.l0, J.rl0);
    const float c = (1.0f - a) - b;
    const float tol = 1e-8f;
    const float3 x0 = J.x0, x1 = J.x1;
    uint32_t least = min(num_key(na), num_key(nb));
    float d2;
    if (a >= -tol && b >= -tol && c >= -tol) {
        const float3 nn = sub(p, add(add(mul(a, x0), mul(b, x1)), mul(c, x2)));
        d2 = dot(nn, nn);
    } else {
        const float n01 = dot(sub(x1, p), J.e01), n12 = -dot(px2, J.e12), n02 = -dot(px2, sub(x2, x0));
        least = min(least, num_key(n01));
        least = min(least, num_key(n12));
        least = min(least, num_key(n02));
        const float u01 = edge_dist2_at(p, x0, x1, div_by(n01, J.d01, J.r01));
        const float u12 = edge_dist2_at(p, x1, x2, div_by(n12, J.d12, J.r12));
        const float u02 = edge_dist2_at(p, x0, x2, div_by(n02, J.d02, J.r02));
        d2 = fminf(fminf(u01, u12), u02);
    }
    if (!J.ranged || least < kNumKey || !sqrt_in_range(d2)) return signed_dist_pre(p, job_pre(J));
    const float d = sqrt_ranged(d2);
    return (dot(sub(p, x0), J.nTri) < 0.0f) ? -d : d;
}

__device__ __forceinline__ float sqrt_approx_ftz(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// The cell's word as it stands in L2 (other warps lower it meanwhile; any value read is one it has had).
__device__ __forceinline__ uint32_t load_word(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// Box coordinates of cell c of a narrow box, as floats: with i the rounded reciprocal of m,
// c i + (i / 2 - 1 / 2) is within (c / m) 2^-23 + 2^-25 of (c + 0.5) / m - 0.5, which lies at least 0.5 / m
// from the half integers, so rounding it (by adding and taking away 1.5 * 2^23) gives the quotient while
// c < 2^20; the remainders are exact.
struct BoxIndex {
    float nx, nxy, inx, inxy, kx, kxy;
};
__device__ __forceinline__ BoxIndex box_index(float nx, float nxy, float inx, float inxy) {
    return BoxIndex{nx, nxy, inx, inxy, 0.5f * inx - 0.5f, 0.5f * inxy - 0.5f};
}
__device__ __forceinline__ float3 box_cell(const BoxIndex& B, float c) {
    constexpr float magic = 12582912.0f;
    const float z = __fadd_rn(__fadd_rn(__fmaf_rn(c, B.inxy, B.kxy), magic), -magic);
    const float r = __fmaf_rn(-z, B.nxy, c);
    const float y = __fadd_rn(__fadd_rn(__fmaf_rn(r, B.inx, B.kx), magic), -magic);
    return mk3(__fmaf_rn(-y, B.nx, r), y, z);
}

// The cell loop of one job by one warp.  The lanes run over the box and keep the cells whose word the
// triangle may still lower; the kept cells are collected in `queue` (the warp's own 64 entries) and
// evaluated 32 at a time, with the reference's distance and atomicMin on the FloatFlip3 word.
//
// A cell is left out only when its computed distance is provably larger in magnitude than its current
// word: FloatFlip3 orders words by |d| first and words only fall, so the pair cannot be the minimum,
// whatever else runs at the same time.  The proof is the one of the tiled construct: both branches of
// SignedDistancePointToTriangle return the distance to a point of the triangle up to rounding, so
// |d| >= (dist(p, T) - delta)(1 - 5 eps), delta <= 15 eps max|x_i| + 6e-8 R, and for any centre c and
// unit m, dist >= sqrt(h^2 + (u - R)+^2) - w with h = <p - c, m>, u the length of the rest.  Here h and
// p - c come from the box's corner and the cell's steps (fma), which differ from the rounded cell
// position by a few eps of |x_i|, of the grid's origin and of the box's size; u^2 = |p - c|^2 - h^2
// carries a few eps of |p - c|^2, which moves the bound by a few eps of |h| + u, and |h| + u is at most
// sqrt(2) times the bound plus R.  All are well inside the slack: 2^-17 of max|x_i| + |origin| + box + R + w
// and 2^-15 of the word itself.  A NaN keeps the cell.
//
// A box that is not narrow has every cell evaluated, and so has every box of a launch too small to fill the device
// (`all`): there a triangle's time is its one warp's chain, which the tests lengthen, and few words are low enough
// to decide one.  A 12-triangle box in 64^3: 106 us with the tests, 75 without (115 before there were any); 816
// triangles in 128^3: 52 and 43 (55); 3,474 in 64^3: 17.5 and 16.2 (25).
//
// Bound: issue, and the latency of a step's chain (26 warps per SM).  About 50 instructions test 32 cells,
// about 230 evaluate 32; of the 200 cells of a box 35 are evaluated, in 1.6 steps of 6.6.  50,040
// triangles on a 128^3 grid: 42 M warp instructions and 58 us (ncu), where evaluating every cell took
// 96 M and 97 us.  Each step loads its words one step ahead (61 us without).
__device__ __forceinline__ void sdf_construct_job_warp(const TriJob& J, uint2* queue, int lane, bool all) {
    const int vol = J.vol;
    uint32_t* const first = J.first;
    if (!J.narrow) {
        const int nx = __float_as_int(J.nx), nxy = __float_as_int(J.nxy), gnx = __float_as_int(J.gnx), gny = __float_as_int(J.plane);
        const int lox = __float_as_int(J.lox), loy = __float_as_int(J.loy), loz = __float_as_int(J.loz);
        SdfGrid g;
        g.ox = J.ox; g.oy = J.oy; g.oz = J.oz; g.cell = J.cell;
        for (int c = lane; c < vol; c += 32) {
            const int z = c / nxy, r = c - z * nxy, y = r / nx, x = r - y * nx;
            const float d = signed_dist_job(sdf_cell_pos(g, lox + x, loy + y, loz + z), J);
            atomicMin(first + (((long long)gny * z + y) * gnx + x), float_flip3(d));
        }
        __syncwarp();
        return;
    }
    const BoxIndex B = box_index(J.nx, J.nxy, J.inx, J.inxy);
    const float cell = J.cell, R = J.R, slack = J.slack, plane = J.plane, gnx = J.gnx;
    const float bx = J.bx, by = J.by, bz = J.bz, hx = J.hx, hy = J.hy, hz = J.hz, h0 = J.h0;
    auto word_at = [&](float3 b) { return first + (int)__fmaf_rn(b.z, plane, __fmaf_rn(b.y, gnx, b.x)); };
    // A cell is queued with the word its test read: a distance that is not below it changes nothing (words
    // only fall), and the atomic that would say so is left out.  Atomics are 4 % of the construct: 185 -> 178 us
    // at 199,656 triangles in 128^3, 66.0 -> 63.7 at 50,040, 37.4 -> 35.4 at 25,700 in 64 x 96 x 56.
    auto evaluate = [&](float c, uint32_t seen) {   // the invariants are read from shared memory: they are not kept across the tests
        const float3 b = box_cell(B, c);
        // GetSdfCellPosition of cell lo + b
        const float3 p = add(mk3((J.lox + b.x) * cell, (J.loy + b.y) * cell, (J.loz + b.z) * cell), mk3(J.ox, J.oy, J.oz));
        const uint32_t w = float_flip3(signed_dist_job(p, J));
        if (w < seen) atomicMin(word_at(b), w);
    };
    if (all) {
        for (int c = lane; c < vol; c += 32) evaluate((float)c, 0xffffffffu);
        __syncwarp();
        return;
    }
    CellQueue<DeviceWarp, uint2*> kept{queue, lane};
    float fc = (float)lane;
    float3 nextCell = box_cell(B, fc);   // each step's word is loaded a step ahead
    uint32_t nextWord = 0u;
    if (lane < vol) nextWord = load_word(word_at(nextCell));
    for (int left = vol - lane; left > -lane; left -= 32, fc += 32.0f) {
        const float3 b = nextCell;
        const uint32_t word = nextWord;
        nextCell = box_cell(B, fc + 32.0f);
        if (left > 32) nextWord = load_word(word_at(nextCell));
        const float dx = __fmaf_rn(b.x, cell, bx), dy = __fmaf_rn(b.y, cell, by), dz = __fmaf_rn(b.z, cell, bz);
        const float h = __fmaf_rn(b.x, hx, __fmaf_rn(b.y, hy, __fmaf_rn(b.z, hz, h0)));
        const float hh = __fmul_rn(h, h);
        const float rr = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
        const float u = sqrt_approx_ftz(fmaxf(rr - hh, 0.0f));
        const float over = fmaxf(u - R, 0.0f);
        const float lb2 = __fmaf_rn(over, over, hh);
        const float cur = __uint_as_float(word >> 1);   // magnitude of the word
        const float thr = __fmaf_rn(cur, 1.0f + 0x1p-15f, slack);
        const bool keep = left > 0 && !(lb2 > __fmul_rn(thr, thr));
        kept.add(keep, make_uint2(__float_as_uint(fc), word));
        if (kept.full()) {
            const uint2 e = kept.take();
            evaluate(__uint_as_float(e.x), e.y);
        }
    }
    uint2 e;
    if (kept.last(e)) evaluate(__uint_as_float(e.x), e.y);
    __syncwarp();
}

// Four-warp construct blocks per SM the kernels over a job array are compiled for (72 registers): 7 measured
// faster than 6 and 8.
constexpr int kConstructBlocksPerSM = 7;

// A construct warp's part of its block's shared memory: the jobs of one chunk and the queue of the cells
// to evaluate.
struct SdfWarpArea {
    TriJob* jobs;
    uint2* queue;
};
constexpr int kSdfQueueBytes = 64 * 8;
constexpr int kSdfJobsAhead = 2;   // jobs a warp holds when they come from a job array: the current and the next
__device__ __forceinline__ SdfWarpArea sdf_warp_area(unsigned char* smem, int warp, int per) {
    unsigned char* p = smem + (size_t)warp * (kSdfQueueBytes + (size_t)per * sizeof(TriJob));
    return SdfWarpArea{reinterpret_cast<TriJob*>(p + kSdfQueueBytes), reinterpret_cast<uint2*>(p)};
}
inline size_t sdf_construct_smem(int warps, int per) { return (size_t)warps * (kSdfQueueBytes + (size_t)per * sizeof(TriJob)); }

// Triangles per warp chunk for a launch over `tris` triangles without a job array: one chunk per resident
// warp (about 24 per SM), at most 16 triangles.
inline int sdf_construct_chunk(long long tris, int sms) {
    const long long per = tris / ((long long)sms * 24);
    return (int)(per < 1 ? 1 : per > 16 ? 16 : per);
}
// Whether a launch over `tris` triangles fills the device: a triangle for every resident warp.  From there on the
// construct reads its jobs from an array, where it has one, and tests the cells; below, its warps make their own
// and evaluate every cell (sdf_construct_job_warp).  Around the line the two ways to the jobs are equal: a plain
// rebuild in 64^3 of 2,500 / 3,600 / 4,500 / 6,000 / 9,000 triangles takes 13.8 / 14.0 / 13.9 / 14.2 / 16.2 us
// with the array, 14.2 / 14.2 / 14.4 / 16.1 / 17.0 with each warp making its own; a batched frame of 2,240 x 32
// strands around it 21.3 / 22.3 / 22.7 / 23.9 / 26.0 and 21.4 / 22.8 / 22.9 / 25.0 / 26.9.  Well above it, the
// array is ahead where the strand kernels fill the device (200,000 x 16 and 50,000 triangles: 251 against 283 us)
// and behind where a frame is little else than its mesh (2,240 x 32 and 25,800: 40.3 against 37.2).
inline bool sdf_fills_device(long long tris, int sms) { return tris >= (long long)sms * 24; }

// One warp's chunk of `count` (<= the area's jobs) consecutive triangles starting at `first`: lane k makes
// the job of triangle first + k with make(t), then the warp runs the cell loops; the chunk ends with the
// warp synchronised, so the area can take the next chunk.
template <class MakeJob>
__device__ __forceinline__ void sdf_construct_chunk_warp(const SdfWarpArea& area, int first, int count, int lane, bool all,
                                                         MakeJob make) {
    if (lane < count) area.jobs[lane] = make(first + lane);
    __syncwarp();
    for (int j = 0; j < count; ++j) sdf_construct_job_warp(area.jobs[j], area.queue, lane, all);
    __syncwarp();
}

// The construct over an array of jobs made beforehand (a thread per triangle: beside the words' initialisation on
// the plain path, in a launch of its own in a batch): the launch's warps stride over the triangles, each bringing its next job into shared
// memory while it runs the current one.  Triangles are taken 16 apart, the starting points in
// bit-reversed order, so that the first ones already give every part of the mesh a word near its result
// and the later ones find most of their cells decided.
constexpr int kJobSpreadLog = 4;
struct SdfJobOrder {
    int total, rows, row, phase;
    __device__ __forceinline__ SdfJobOrder(int n, int start)
        : total(n), rows((n + (1 << kJobSpreadLog) - 1) >> kJobSpreadLog), row(start), phase(0) {
        settle();
    }
    __device__ __forceinline__ void settle() {
        while (row >= rows) { row -= rows; ++phase; }
    }
    __device__ __forceinline__ int triangle() const {
        return (row << kJobSpreadLog) + (int)(__brev((unsigned)phase) >> (32 - kJobSpreadLog));
    }
    // this or the next step that has a triangle: its index, or -1 at the end
    __device__ __forceinline__ int find(int warps) {
        for (; phase < (1 << kJobSpreadLog); step(warps))
            if (triangle() < total) return triangle();
        return -1;
    }
    __device__ __forceinline__ void step(int warps) { row += warps; settle(); }
};

// A block's jobs on their way to the job array: a thread's job is 256 bytes, so written by the thread itself
// each of its 16-byte stores would touch a line of its own.
constexpr int kJobThreads = 128;
struct JobStage {
    uint4 part[kJobThreads][sizeof(TriJob) / 16 + 1];   // a row and 16 bytes: free of bank conflicts
    __device__ __forceinline__ void put(int t, const TriJob& J) {
        const uint4* p = reinterpret_cast<const uint4*>(&J);
#pragma unroll
        for (int k = 0; k < (int)(sizeof(TriJob) / 16); ++k) part[t][k] = p[k];
    }
    // by all threads of the block
    __device__ __forceinline__ void write(TriJob* __restrict__ jobs, int count) {
        constexpr int P = sizeof(TriJob) / 16;
        __syncthreads();
        for (int i = threadIdx.x; i < count * P; i += kJobThreads) reinterpret_cast<uint4*>(jobs)[i] = part[i / P][i % P];
    }
};

__device__ __forceinline__ void sdf_job_prefetch(TriJob* dst, const TriJob* src, int lane) {
    if (lane < (int)(sizeof(TriJob) / 16)) {
        const uint32_t d = (uint32_t)__cvta_generic_to_shared(reinterpret_cast<char*>(dst) + 16 * lane);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(reinterpret_cast<const char*>(src) + 16 * lane)
                     : "memory");
    }
}
__device__ __forceinline__ void sdf_construct_jobs_warp(const SdfWarpArea& area, const TriJob* jobs, int total,
                                                        int warp, int warps, int lane) {
    SdfJobOrder order(total, warp);
    int tri = order.find(warps);
    if (tri < 0) return;
    sdf_job_prefetch(area.jobs, jobs + tri, lane);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int cur = 0; tri >= 0; cur ^= 1) {
        order.step(warps);
        tri = order.find(warps);
        if (tri >= 0) sdf_job_prefetch(area.jobs + (cur ^ 1), jobs + tri, lane);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        sdf_construct_job_warp(area.jobs[cur], area.queue, lane, false);   // ends with the warp synchronised
    }
}

// GetSignedDistance + TrilinearInterpolate, :414-527.  The grid is what the launch before may have written: plain
// loads (tfx_launch.cuh).
__device__ __forceinline__ float lerp_ref(float a, float b, float t) { return a * (1.0f - t) + b * t; }

__device__ __forceinline__ float sdf_lookup(const float* sdf, const SdfGrid& g, float3 p) {
    if (sdf_surely_outside(g, p)) return 1e10f;
    const int3 gc = sdf_coords(g, p);
    if (!(0 <= gc.x && gc.x < g.nx - 2) || !(0 <= gc.y && gc.y < g.ny - 2) || !(0 <= gc.z && gc.z < g.nz - 2))
        return 1e10f;
    const long long X = 1, Y = g.nx, Z = (long long)g.ny * g.nx;
    const long long base = Z * gc.z + Y * gc.y + gc.x;
    float d[8];
    d[0] = sdf[base];
    d[1] = sdf[base + X];
    d[2] = sdf[base + Y];
    d[3] = sdf[base + Y + X];
    d[4] = sdf[base + Z];
    d[5] = sdf[base + Z + X];
    d[6] = sdf[base + Z + Y];
    d[7] = sdf[base + Z + Y + X];
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if (d[j] == 1e10f) return 1e10f;
    const float3 cp = sdf_cell_pos(g, gc.x, gc.y, gc.z);
    const float3 ip = divs(sub(p, cp), g.cell);
    const float b0 = lerp_ref(lerp_ref(d[0], d[1], ip.x), lerp_ref(d[2], d[3], ip.x), ip.y);
    const float b1 = lerp_ref(lerp_ref(d[4], d[5], ip.x), lerp_ref(d[6], d[7], ip.x), ip.y);
    return lerp_ref(b0, b1, ip.z);
}

// CollideHairVerticesWithSdf_forward for one vertex (j >= 2): returns true and the projected
// position when the vertex is pushed out (then Pos.xyz and Prev.xyz both take it).
// In the shader's own form: the lookup at p and three more, 0.1 cells along each axis.
static __device__ __noinline__ bool sdf_collide_general(const float* sdf, SdfGrid g, float margin, float3 p, float3* proj) {
    const float distance = sdf_lookup(sdf, g, p);
    if (distance > margin) return false;
    const float h = 0.1f * g.cell;
    const float fx = sdf_lookup(sdf, g, add(p, mul(mk3(1.0f, 0.0f, 0.0f), h)));
    const float fy = sdf_lookup(sdf, g, add(p, mul(mk3(0.0f, 1.0f, 0.0f), h)));
    const float fz = sdf_lookup(sdf, g, add(p, mul(mk3(0.0f, 0.0f, 1.0f), h)));
    const float3 grad = mk3((fx - distance) / h, (fy - distance) / h, (fz - distance) / h);
    const float3 nrm = normalize(grad);
    if (distance < margin) {
        *proj = add(p, mul(nrm, margin - distance));
        return true;
    }
    return false;
}

// The grid's two divisors, the cell size and the gradient's step, with their reciprocals for the short
// exact division, made once per thread; `ranged` is false where the short form's ranges do not hold.
struct SdfSteps {
    float rcell, h, rh;
    bool ranged;
};
__device__ __forceinline__ SdfSteps sdf_steps(const SdfGrid& g, float margin) {
    SdfSteps s;
    s.h = 0.1f * g.cell;
    s.rcell = 1.0f / g.cell;
    s.rh = 1.0f / s.h;
    s.ranged = g.cell >= 16.0f * kDivisorMin && g.cell <= kDivisorMax && fabsf(g.ox) <= 0x1p90f && fabsf(g.oy) <= 0x1p90f &&
               fabsf(g.oz) <= 0x1p90f && margin < 1e10f && (long long)g.nx * g.ny * g.nz < (1ll << 31);
    return s;
}
// At least kDivKey for the numerators div_by is exact for: zero, and magnitudes from kDivMin on.
__device__ __forceinline__ uint32_t div_key(float a) { return (__float_as_uint(a) & 0x7fffffffu) - 1u; }
constexpr uint32_t kDivKey = 0x21800000u - 1u;   // kDivMin's bits, less one
__device__ __forceinline__ bool div_keys(float a, float b, float c) { return min(min(div_key(a), div_key(b)), div_key(c)) >= kDivKey; }

// The same result from the corners of one cell.  Along each axis the probe lies in p's cell (nine of
// ten) or in the next: its lookup shares the other two axes' fractions with p's, and takes p's corners or
// their far half and four new ones.  So a vertex reads 8 corners and, for a probe that leaves the cell,
// 4 more, in place of 32, does 7 + 4 + 2 interpolations for the gradient in place of 21, and 8 divisions, in
// their short form, in place of 27.  corners(base, d) gives the 8 corners of the cell at index base.
constexpr int kCollideMiss = 0, kCollideHit = 1, kCollideGeneral = 2;
template <class Corners>
__device__ __forceinline__ int sdf_collide_shared(const float* sdf, const SdfGrid& g, const SdfSteps& st, float margin,
                                                 float3 p, float3& proj, const Corners& cell) {
    if (!st.ranged) return kCollideGeneral;
    if (sdf_surely_outside(g, p)) return kCollideMiss;
    // a numerator below the short form's range gives a quotient below 1 by either form
    auto coord = [&](float d) { return ftoi(div_by(d, g.cell, st.rcell)); };
    const int x = coord(p.x - g.ox), y = coord(p.y - g.oy), z = coord(p.z - g.oz);
    if (!(0 <= x && x < g.nx - 2) || !(0 <= y && y < g.ny - 2) || !(0 <= z && z < g.nz - 2)) return kCollideMiss;
    const int Y = g.nx, Z = g.ny * g.nx;
    const int base = Z * z + Y * y + x;
    float d[8];
    cell.corners(base, d);
    bool far = false;
#pragma unroll
    for (int j = 0; j < 8; ++j) far |= d[j] == 1e10f;
    if (far) return kCollideMiss;
    const float3 cp = sdf_cell_pos(g, x, y, z);
    const float3 a = sub(p, cp);
    const float3 ip = mk3(div_by(a.x, g.cell, st.rcell), div_by(a.y, g.cell, st.rcell), div_by(a.z, g.cell, st.rcell));
    const float x00 = lerp_ref(d[0], d[1], ip.x), x10 = lerp_ref(d[2], d[3], ip.x);
    const float x01 = lerp_ref(d[4], d[5], ip.x), x11 = lerp_ref(d[6], d[7], ip.x);
    const float b0 = lerp_ref(x00, x10, ip.y), b1 = lerp_ref(x01, x11, ip.y);
    const float distance = lerp_ref(b0, b1, ip.z);
    if (!div_keys(a.x, a.y, a.z)) return kCollideGeneral;
    if (!(distance < margin)) return kCollideMiss;

    const float qx = p.x + st.h, qy = p.y + st.h, qz = p.z + st.h;
    const int px = coord(qx - g.ox), py = coord(qy - g.oy), pz = coord(qz - g.oz);
    const bool mx = px != x, my = py != y, mz = pz != z;
    const bool ox = px >= g.nx - 2, oy = py >= g.ny - 2, oz = pz >= g.nz - 2;   // past the grid: the lookup's 1e10
    float4 e = make_float4(0.f, 0.f, 0.f, 0.f), f = e, k = e;
    if (mx && !ox) e = cell.beyond_x(base);
    if (my && !oy) f = cell.beyond_y(base);
    if (mz && !oz) k = cell.beyond_z(base);
    const float ax = qx - ((float)px * g.cell + g.ox), ay = qy - ((float)py * g.cell + g.oy), az = qz - ((float)pz * g.cell + g.oz);
    const float tx = div_by(ax, g.cell, st.rcell), ty = div_by(ay, g.cell, st.rcell), tz = div_by(az, g.cell, st.rcell);
    float fx = lerp_ref(lerp_ref(lerp_ref(mx ? d[1] : d[0], mx ? e.x : d[1], tx), lerp_ref(mx ? d[3] : d[2], mx ? e.y : d[3], tx), ip.y),
                        lerp_ref(lerp_ref(mx ? d[5] : d[4], mx ? e.z : d[5], tx), lerp_ref(mx ? d[7] : d[6], mx ? e.w : d[7], tx), ip.y),
                        ip.z);
    if (ox || e.x == 1e10f || e.y == 1e10f || e.z == 1e10f || e.w == 1e10f) fx = 1e10f;
    float fy = lerp_ref(lerp_ref(my ? x10 : x00, my ? lerp_ref(f.x, f.y, ip.x) : x10, ty),
                        lerp_ref(my ? x11 : x01, my ? lerp_ref(f.z, f.w, ip.x) : x11, ty), ip.z);
    if (oy || f.x == 1e10f || f.y == 1e10f || f.z == 1e10f || f.w == 1e10f) fy = 1e10f;
    float fz = lerp_ref(mz ? b1 : b0, mz ? lerp_ref(lerp_ref(k.x, k.y, ip.x), lerp_ref(k.z, k.w, ip.x), ip.y) : b1, tz);
    if (oz || k.x == 1e10f || k.y == 1e10f || k.z == 1e10f || k.w == 1e10f) fz = 1e10f;
    const float gx = fx - distance, gy = fy - distance, gz = fz - distance;
    // the shader adds 0 to the other two coordinates of a probe, which changes a zero's sign; a difference
    // of zeros has a sign too; a step that spans more than a cell (a cell near p's rounding) shares nothing
    const bool shared = (unsigned)(px - x) <= 1u && (unsigned)(py - y) <= 1u && (unsigned)(pz - z) <= 1u && p.x != 0.0f &&
                        p.y != 0.0f && p.z != 0.0f && distance != 0.0f && div_keys(ax, ay, az) && div_keys(gx, gy, gz) &&
                        fmaxf(fmaxf(fabsf(gx), fabsf(gy)), fabsf(gz)) <= kDivMax;
    if (!shared) return kCollideGeneral;
    const float3 nrm = normalize(mk3(div_by(gx, st.h, st.rh), div_by(gy, st.h, st.rh), div_by(gz, st.h, st.rh)));
    proj = add(p, mul(nrm, margin - distance));
    return kCollideHit;
}

template <class Corners>
__device__ __forceinline__ bool sdf_collide_cell(const float* sdf, const SdfGrid& g, const SdfSteps& st, float margin,
                                                 float3 p, float3& proj, const Corners& cell) {
    const int r = sdf_collide_shared(sdf, g, st, margin, p, proj, cell);
    if (r != kCollideGeneral) return r == kCollideHit;
    float3 q;
    if (!sdf_collide_general(sdf, g, margin, p, &q)) return false;
    proj = q;
    return true;
}

// How a kernel reads the finished grid.  PlainLoad anywhere; ReadOnlyLoad only in a kernel launched plainly, which
// starts when the launches that write the grid have ended (tfx_launch.cuh).
struct PlainLoad {
    __device__ __forceinline__ float operator()(const float* p) const { return *p; }
};
struct ReadOnlyLoad {
    __device__ __forceinline__ float operator()(const float* p) const { return __ldg(p); }
};

// The corners of cell `base` straight from the grid: its own 8, and the 4 that the next cell along an axis adds.
template <class Load = PlainLoad>
struct GridCorners {
    const float* sdf;
    int Y, Z;
    __device__ __forceinline__ GridCorners(const float* s, const SdfGrid& g) : sdf(s), Y(g.nx), Z(g.ny * g.nx) {}
    __device__ __forceinline__ float4 four(const float* w, int a, int b, int c, int d) const {
        const Load load;
        return make_float4(load(w + a), load(w + b), load(w + c), load(w + d));
    }
    __device__ __forceinline__ void corners(int base, float (&d)[8]) const {
        const float *w00 = sdf + base, *w10 = w00 + Y, *w01 = w00 + Z, *w11 = w01 + Y;
        const Load load;
        d[0] = load(w00);
        d[1] = load(w00 + 1);
        d[2] = load(w10);
        d[3] = load(w10 + 1);
        d[4] = load(w01);
        d[5] = load(w01 + 1);
        d[6] = load(w11);
        d[7] = load(w11 + 1);
    }
    __device__ __forceinline__ float4 beyond_x(int base) const { return four(sdf + base + 2, 0, Y, Z, Z + Y); }
    __device__ __forceinline__ float4 beyond_y(int base) const { return four(sdf + base + 2 * Y, 0, 1, Z, Z + 1); }
    __device__ __forceinline__ float4 beyond_z(int base) const { return four(sdf + base + 2 * Z, 0, 1, Y, Y + 1); }
};

template <class Load = PlainLoad>
__device__ __forceinline__ bool sdf_collide_point(const float* sdf, const SdfGrid& g, float margin, float3 p, float3& proj) {
    return sdf_collide_cell(sdf, g, sdf_steps(g, margin), margin, p, proj, GridCorners<Load>(sdf, g));
}

}  // namespace tfx
