// Signed distance of a branched vessel on a voxel grid: the field of vessel.k_sdf (vessel.py:178-207), evaluated on
// the GPU in float32 in the same order of operations, so that build_lattice sees the reference's field.
//
// Per voxel p = origin + (i, j, k) dx: for each branch, the minimum over its segments of the round-cone distance
// |p - (a + t ab)| - r(t) (t = the clamped projection of p on the segment, r interpolated linearly), cut by the flat
// caps near its open ends (a half-space max within 2.5 cap radii); branches are joined by the polynomial smooth
// minimum with blend radius `blend`. Negative inside the lumen. C order (k fastest); a block works a brick of voxels, two
// a thread, with the segments that can be nearest there.
#include "cs_common.cuh"

namespace cs {
namespace {

struct SdfArgs {
    float origin[3];
    float dx;
    const float* pts;        // (n_pts, 3) centreline points, branches back to back
    const float* rad;        // (n_pts,) radius at each point
    const int32_t* br_start; // (nbranch,) first point of each branch
    const int32_t* br_count; // (nbranch,) points of each branch
    const float* cap_p;      // (2 nbranch, 3) cap centres (start, end of each branch)
    const float* cap_n;      // (2 nbranch, 3) outward cap normals
    const float* cap_r;      // (2 nbranch,) cap radius, 0 = no cap
    float blend;
    int nbranch;
    int64_t nx, ny, nz;
    float* out;
};

__device__ __forceinline__ float smin(float a, float b, float k) {
    // vessel.py:178-181
    const float h = fminf(fmaxf(0.5f + 0.5f * (b - a) / k, 0.0f), 1.0f);
    return b + (a - b) * h - k * h * (1.0f - h);
}

// Bricks of 8 x 8 x 8 voxels, one block of 256 threads each, two voxels a thread. Evaluating every segment at every
// voxel is bound by instruction issue (about 45 per segment, the division and the square root among them; 320 segments
// on a vessel of two branches), so a block first drops the segments that cannot be the nearest anywhere in its brick
// (86 stay on average) and a thread then skips those of the rest that cannot beat the distance it already has. Only
// evaluations whose result the minimum would discard are left out, so the field is the same bit for bit. 6.8 M voxels:
// 4.35 ms for the field with every segment at every voxel, 0.86 now (0.94 with a voxel a thread); still issue-bound
// (89 %), two thirds of it in the loop over the list. Testing a warp's voxels together, or the exact distance without
// its division and root before the exact one, left the time as it was.
//
// Bounds, for a segment k with axis distance D_k(c) from the brick's centre c, brick half-diagonal h, and the radii
// r0, r1 at its ends: anywhere in the brick |p - q| - r lies in [D_k(c) - h - max(r0, r1), D_k(c) + h - min(r0, r1)]
// (a distance to a segment changes by at most the way walked). A segment whose lower end lies above the least upper
// end U of all segments of its branch is never the minimum. For a voxel p and a segment of half-length l and midpoint
// m, |p - q| >= |p - m| - l. Each bound carries a margin of 1e-5 of the lengths that enter it (the coordinates and the
// grid's origin, the distance, the segment's own length and radii), over a hundred times the rounding of its own
// evaluation and of the distances it is compared with. A segment shorter than 1e-6 is projected on by a bounded divisor,
// which can put the point taken for the nearest anywhere on it: 1e-6 more. A comparison with NaN keeps the segment.
constexpr int BX = 8, BY = 8, BZ = 8, SDF_PER = 2;       // voxels a thread, BY / SDF_PER apart along y
constexpr int SDF_THREADS = BX * BY * BZ / SDF_PER;
constexpr float SDF_MARGIN = 1.0e-5f, SDF_TINY = 1.0e-6f;

// Axis distance of point c from segment k of the packed centrelines; margin: of the bounds made from it.
__device__ __forceinline__ float axis_distance(const SdfArgs& s, int k, float cx, float cy, float cz, float size, float r0,
                                                float r1, float& margin) {
    const float ax = __ldg(s.pts + 3 * k), ay = __ldg(s.pts + 3 * k + 1), az = __ldg(s.pts + 3 * k + 2);
    const float bx = __ldg(s.pts + 3 * k + 3) - ax, by = __ldg(s.pts + 3 * k + 4) - ay, bz = __ldg(s.pts + 3 * k + 5) - az;
    const float qx = cx - ax, qy = cy - ay, qz = cz - az;
    const float t = fminf(fmaxf((qx * bx + qy * by + qz * bz) / fmaxf(bx * bx + by * by + bz * bz, 1.0e-12f), 0.0f), 1.0f);
    const float ex = qx - bx * t, ey = qy - by * t, ez = qz - bz * t;
    const float dk = sqrtf(ex * ex + ey * ey + ez * ez);
    margin = SDF_MARGIN * (size + dk + fabsf(bx) + fabsf(by) + fabsf(bz) + fmaxf(fabsf(r0), fabsf(r1))) + SDF_TINY;
    return dk;
}

// vessel.py:195-199: distance of p to the round cone from a along b with radius r0 + dr t.
__device__ __forceinline__ float cone_distance(float px, float py, float pz, float ax, float ay, float az, float bx,
                                               float by, float bz, float r0, float dr) {
    const float qx = px - ax, qy = py - ay, qz = pz - az;
    const float t = fminf(fmaxf((qx * bx + qy * by + qz * bz) / fmaxf(bx * bx + by * by + bz * bz, 1.0e-12f), 0.0f), 1.0f);
    const float r = r0 + dr * t;
    const float ex = px - (ax + bx * t), ey = py - (ay + by * t), ez = pz - (az + bz * t);
    return sqrtf(ex * ex + ey * ey + ez * ez) - r;
}

// IDX: int32_t when there are fewer than 2^31 bricks (a 64-bit division takes some 70 instructions).
template <class IDX>
__global__ void __launch_bounds__(SDF_THREADS) k_sdf(const SdfArgs s, const IDX nby, const IDX nbz,
                                                     const int64_t bricks) {
    __shared__ float4 s_seg[2][SDF_THREADS];   // start and r0; direction and r1 - r0
    __shared__ float4 s_mid[SDF_THREADS];      // midpoint; half-length + larger radius + margin
    __shared__ float s_u[SDF_THREADS / 32];
    __shared__ int s_cnt[SDF_THREADS / 32 + 1], s_best;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int64_t br = blockIdx.x; br < bricks; br += gridDim.x) {
        const IDX row = IDX(br) / nbz, slab = row / nby;
        const IDX z0 = (IDX(br) - row * nbz) * BZ, y0 = (row - slab * nby) * BY, x0 = slab * BX;
        constexpr int HY = BY / SDF_PER;
        const IDX l = z0 + tid % BZ, j = y0 + (tid / BZ) % HY, i = x0 + tid / (BZ * HY);
        const float px = s.origin[0] + float(i) * s.dx;
        float py[SDF_PER], d[SDF_PER];
#pragma unroll
        for (int v = 0; v < SDF_PER; ++v) {
            py[v] = s.origin[1] + float(j + v * HY) * s.dx;
            d[v] = 1.0e9f;
        }
        const float pz = s.origin[2] + float(l) * s.dx;
        const float cx = s.origin[0] + (float(x0) + 0.5f * float(BX - 1)) * s.dx;
        const float cy = s.origin[1] + (float(y0) + 0.5f * float(BY - 1)) * s.dx;
        const float cz = s.origin[2] + (float(z0) + 0.5f * float(BZ - 1)) * s.dx;
        const float h = 0.5f * s.dx * sqrtf(float((BX - 1) * (BX - 1) + (BY - 1) * (BY - 1) + (BZ - 1) * (BZ - 1)));
        const float size = fabsf(cx) + fabsf(cy) + fabsf(cz) + 4.0f * h + fabsf(s.origin[0]) + fabsf(s.origin[1]) +
                           fabsf(s.origin[2]);          // of the coordinates in the brick and the sums that gave them
        for (int b = 0; b < s.nbranch; ++b) {
            const int s0 = __ldg(s.br_start + b), last = s0 + __ldg(s.br_count + b) - 1;
            // least upper bound over the branch's segments, and the segment that has it
            float u_own = 3.0e38f, dk = 0.0f, r0 = 0.0f, r1 = 0.0f, margin = 0.0f;
            int k_own = -1;
            for (int k = s0 + tid; k < last; k += SDF_THREADS) {
                r0 = __ldg(s.rad + k);
                r1 = __ldg(s.rad + k + 1);
                dk = axis_distance(s, k, cx, cy, cz, size, r0, r1, margin);
                const float up = dk + h - fminf(r0, r1) + margin;
                if (up < u_own) {
                    u_own = up;
                    k_own = k;
                }
            }
            float u = u_own;
            for (int o = 16; o > 0; o >>= 1) u = fminf(u, __shfl_xor_sync(0xffffffffu, u, o));
            if (lane == 0) s_u[warp] = u;
            if (tid == 0) s_best = -1;
            __syncthreads();
            for (int w = 0; w < SDF_THREADS / 32; ++w) u = fminf(u, s_u[w]);
            if (k_own >= 0 && u_own == u) s_best = k_own;      // of several, any
            __syncthreads();
            // the brick's nearest segment first: most of the others then fall to the test of their midpoint
            float db[SDF_PER];
#pragma unroll
            for (int v = 0; v < SDF_PER; ++v) db[v] = 1.0e9f;
            if (s_best >= 0) {
                const int k = s_best;
                const float ax = __ldg(s.pts + 3 * k), ay = __ldg(s.pts + 3 * k + 1), az = __ldg(s.pts + 3 * k + 2);
                const float ra = __ldg(s.rad + k);
                const float bx = __ldg(s.pts + 3 * k + 3) - ax, by = __ldg(s.pts + 3 * k + 4) - ay,
                            bz = __ldg(s.pts + 3 * k + 5) - az, dr = __ldg(s.rad + k + 1) - ra;
#pragma unroll
                for (int v = 0; v < SDF_PER; ++v)
                    db[v] = fminf(db[v], cone_distance(px, py[v], pz, ax, ay, az, bx, by, bz, ra, dr));
            }
            for (int k0 = s0; k0 < last; k0 += SDF_THREADS) {
                // the segments of this chunk that may be the nearest, kept in their order in shared memory
                const int k = k0 + tid;
                bool keep = false;
                if (k < last) {
                    if (last - s0 > SDF_THREADS) {         // of a single chunk the first pass left them in registers
                        r0 = __ldg(s.rad + k);
                        r1 = __ldg(s.rad + k + 1);
                        dk = axis_distance(s, k, cx, cy, cz, size, r0, r1, margin);
                    }
                    keep = !(dk - h - fmaxf(r0, r1) - margin > u);
                }
                const unsigned mask = __ballot_sync(0xffffffffu, keep);
                if (lane == 0) s_cnt[warp] = __popc(mask);
                __syncthreads();
                if (tid == 0) {
                    int run = 0;
                    for (int w = 0; w < SDF_THREADS / 32; ++w) {
                        const int c = s_cnt[w];
                        s_cnt[w] = run;
                        run += c;
                    }
                    s_cnt[SDF_THREADS / 32] = run;
                }
                __syncthreads();
                if (keep) {
                    const int o = s_cnt[warp] + __popc(mask & ((1u << lane) - 1u));
                    const float ax = __ldg(s.pts + 3 * k), ay = __ldg(s.pts + 3 * k + 1), az = __ldg(s.pts + 3 * k + 2);
                    const float bx = __ldg(s.pts + 3 * k + 3) - ax, by = __ldg(s.pts + 3 * k + 4) - ay,
                                bz = __ldg(s.pts + 3 * k + 5) - az;
                    const float b2 = bx * bx + by * by + bz * bz, half = 0.5f * sqrtf(b2);
                    s_seg[0][o] = make_float4(ax, ay, az, r0);
                    s_seg[1][o] = make_float4(bx, by, bz, r1 - r0);
                    s_mid[o] = make_float4(ax + 0.5f * bx, ay + 0.5f * by, az + 0.5f * bz,
                                           half + fmaxf(r0, r1) + margin);
                }
                __syncthreads();
                const int cnt = s_cnt[SDF_THREADS / 32];
                for (int c = 0; c < cnt; ++c) {
                    const float4 m = s_mid[c];
                    const float gx = px - m.x, gz = pz - m.z, gxz = gx * gx + gz * gz;
#pragma unroll
                    for (int v = 0; v < SDF_PER; ++v) {
                        // |p - m| - reach >= db: the distance below cannot be smaller than db
                        const float gy = py[v] - m.y, far = (db[v] + m.w) * (1.0f + SDF_MARGIN);
                        if (far < 0.0f || gxz + gy * gy > far * far) continue;
                        const float4 a = s_seg[0][c], e = s_seg[1][c];
                        db[v] = fminf(db[v], cone_distance(px, py[v], pz, a.x, a.y, a.z, e.x, e.y, e.z, a.w, e.w));
                    }
                }
                __syncthreads();                    // the list is rewritten by the next chunk or branch
            }
#pragma unroll
            for (int v = 0; v < SDF_PER; ++v) {
                for (int e = 0; e < 2; ++e) {
                    const int cc = b * 2 + e;
                    const float cr = __ldg(s.cap_r + cc);
                    if (cr > 0.0f) {
                        const float qx = px - __ldg(s.cap_p + 3 * cc), qy = py[v] - __ldg(s.cap_p + 3 * cc + 1),
                                    qz = pz - __ldg(s.cap_p + 3 * cc + 2);
                        if (sqrtf(qx * qx + qy * qy + qz * qz) < 2.5f * cr)
                            db[v] = fmaxf(db[v], qx * __ldg(s.cap_n + 3 * cc) + qy * __ldg(s.cap_n + 3 * cc + 1) +
                                                     qz * __ldg(s.cap_n + 3 * cc + 2));
                    }
                }
                d[v] = smin(d[v], db[v], s.blend);
            }
            __syncthreads();                        // s_u is rewritten by the next branch
        }
#pragma unroll
        for (int v = 0; v < SDF_PER; ++v) {
            const IDX jv = j + v * HY;
            if (i < s.nx && jv < s.ny && l < s.nz) s.out[(int64_t(i) * s.ny + jv) * s.nz + l] = d[v];
        }
    }
}

}  // namespace
}  // namespace cs

using namespace cs;

extern "C" int cs_sdf_vessel(const float* pts, const float* rad, const int32_t* br_start, const int32_t* br_count,
                             int32_t nbranch, const float* cap_p, const float* cap_n, const float* cap_r, float blend,
                             const float* origin, float dx, int64_t nx, int64_t ny, int64_t nz, float* out,
                             void* stream) {
    if (nx < 0 || ny < 0 || nz < 0 || nbranch < 0 || !origin || !(dx > 0.0f) || !(blend > 0.0f))
        return fail(CS_ERR_ARG, "cs_sdf_vessel: grid %lld x %lld x %lld, %d branches, dx %g, blend %g", (long long)nx,
                    (long long)ny, (long long)nz, nbranch, double(dx), double(blend));
    const int64_t total = nx * ny * nz;
    if (total == 0) return CS_OK;
    if (!out || (nbranch > 0 && (!pts || !rad || !br_start || !br_count || !cap_p || !cap_n || !cap_r)))
        return fail(CS_ERR_ARG, "cs_sdf_vessel: null buffer");
    SdfArgs a{{origin[0], origin[1], origin[2]}, dx, pts, rad, br_start, br_count, cap_p, cap_n, cap_r, blend,
              nbranch, nx, ny, nz, out};
    const int64_t nbx = ceil_div(nx, BX), nby = ceil_div(ny, BY), nbz = ceil_div(nz, BZ);
    const int64_t bricks = nbx * nby * nbz;
    const unsigned grid = unsigned(std::min<int64_t>(bricks, 148 * 64));
    if (bricks < (int64_t(1) << 28) && std::max(nx, std::max(ny, nz)) < (int64_t(1) << 30))
        k_sdf<int32_t><<<grid, SDF_THREADS, 0, as_stream(stream)>>>(a, int32_t(nby), int32_t(nbz), bricks);
    else
        k_sdf<int64_t><<<grid, SDF_THREADS, 0, as_stream(stream)>>>(a, nby, nbz, bricks);
    CS_CHECK_LAUNCH("k_sdf");
    return CS_OK;
}
