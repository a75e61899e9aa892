// Wall shear stress from a velocity field: the per-vertex weighted fit of wss.shear (wss.py:50-57) on the GPU.
//
// For vertex v with inward unit normal n_v and its K fit coefficients c_vj over lumen cells idx_vj (from the
// host-side fit, wss.weights), tau_v = scale * sum_j c_vj (u_j - (u_j . n_v) n_v): the tangential velocity of the
// nearby cells, weighted so that the sum is the slope a of u_t(d) = a d + b d^2 at the wall. scale = mu * 1e3
// turns (m/s)/mm into Pa. FP64 accumulation as the reference's NumPy sum.
//
// The projection is linear, so the weighted velocity S = sum_j c_vj u_j is summed first and projected once. WSS_LANES
// lanes share a vertex: they read its K coefficients and indices side by side (one thread per vertex read them K words
// apart) and add their parts by shuffles. Bound by the gathers of the cells' velocities.
#include "cs_common.cuh"

namespace cs {
namespace {

constexpr int WSS_LANES = 16;
constexpr int WSS_THREADS = 256;

__global__ void __launch_bounds__(WSS_THREADS) k_wss_shear(const float* __restrict__ U, const int32_t* __restrict__ idx,
                                                           const float* __restrict__ c, const float* __restrict__ nrm,
                                                           int64_t n_vert, int K, int64_t n_cells, double scale,
                                                           float* __restrict__ tau) {
    const int64_t v = (blockIdx.x * int64_t(WSS_THREADS) + threadIdx.x) / WSS_LANES;
    const int lane = threadIdx.x % WSS_LANES;
    double sx = 0.0, sy = 0.0, sz = 0.0;
    if (v < n_vert) {
#pragma unroll 3
        for (int j = lane; j < K; j += WSS_LANES) {
            const float w = __ldg(c + v * K + j);
            const int32_t cell = __ldg(idx + v * K + j);
            if (w == 0.0f || cell < 0 || cell >= n_cells) continue;
            const float* u = U + 3 * int64_t(cell);
            sx += double(w) * double(__ldg(u));
            sy += double(w) * double(__ldg(u + 1));
            sz += double(w) * double(__ldg(u + 2));
        }
    }
    for (int o = WSS_LANES / 2; o > 0; o >>= 1) {
        sx += __shfl_xor_sync(0xffffffffu, sx, o);
        sy += __shfl_xor_sync(0xffffffffu, sy, o);
        sz += __shfl_xor_sync(0xffffffffu, sz, o);
    }
    if (v < n_vert && lane < 3) {
        const double nx = nrm[3 * v], ny = nrm[3 * v + 1], nz = nrm[3 * v + 2];
        const double sn = sx * nx + sy * ny + sz * nz;
        const double s = lane == 0 ? sx - sn * nx : (lane == 1 ? sy - sn * ny : sz - sn * nz);
        tau[3 * v + lane] = float(scale * s);
    }
}

}  // namespace
}  // namespace cs

using namespace cs;

extern "C" int cs_wss_shear(const float* U, int64_t n_cells, const int32_t* idx, const float* c, const float* normals,
                            int64_t n_vert, int32_t K, double scale, float* tau, void* stream) {
    if (n_vert < 0 || n_cells < 0 || K < 1 || K > 1024)
        return fail(CS_ERR_ARG, "cs_wss_shear: %lld vertices, %lld cells, K %d", (long long)n_vert,
                    (long long)n_cells, K);
    if (n_vert == 0) return CS_OK;
    if (!U || !idx || !c || !normals || !tau) return fail(CS_ERR_ARG, "cs_wss_shear: null buffer");
    k_wss_shear<<<unsigned(ceil_div(n_vert * WSS_LANES, WSS_THREADS)), WSS_THREADS, 0, as_stream(stream)>>>(
        U, idx, c, normals, n_vert, K, n_cells, scale, tau);
    CS_CHECK_LAUNCH("k_wss_shear");
    return CS_OK;
}
