// Sparse lattice / neighbour-table builder on the GPU: the tables of lbm.build_lattice (lbm.py:264-330), bit-exact.
//
// Phase 1 (cs_lattice_count): tiles of 4096 grid cells count phi < 0, one block scans the tile counts, and each
// tile ranks its fluid cells in C order (warp ballots) into a dense rank grid (scratch), so node ids equal the
// reference's np.argwhere order (lbm.py:274-278).
// Phase 2 (cs_lattice_fill): coords from the rank grid; for every (link i, node n) the pull source x - c_i with
// periodic wrap (lbm.py:288-293); missing links are matched against the openings (inlets first, then outlets, first
// hit wins: lbm.py:294-306) and wall links get q = -phi_x / (phi_s - phi_x), clipped to [1e-3, 1], non-finite -> 0.5
// (lbm.py:307-316); the inlet profile of every cell with an inlet link comes from the LAST inlet (lbm.py:322-328).
// Floating-point steps use explicitly rounded intrinsics in the order NumPy evaluates them on the host that wrote
// the reference's tables: products and sums are separate roundings, and a row dot product `rel @ nrm` is
// fma(z, n2, fma(x, n0, y * n1)) (the BLAS gemv kernel) except when the batch holds a single row, where NumPy's
// plain dot gives fma(z, n2, fma(y, n1, x * n0)).
#include "cs_common.cuh"

namespace cs {
namespace {

constexpr int TILE_THREADS = 256;
constexpr int TILE_ROUNDS = 16;
constexpr int64_t TILE = TILE_THREADS * TILE_ROUNDS;
constexpr int MAX_OPENINGS = 32;
constexpr uint32_t INLET_CELL = 1u;      // in a node's first profile word, between pass B and the profile itself

__constant__ int8_t k_c[3][Q] = {
    {0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, -1, 1},
    {0, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, -1, 1, 1, -1},
    {0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1, 1, -1, -1, 1, 1, -1, 1, -1}};

struct ScratchLayout {
    int64_t n_tiles;
    size_t off_rank, off_tile, off_misc, total;
};

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

ScratchLayout layout(int64_t nx, int64_t ny, int64_t nz) {
    ScratchLayout s;
    int64_t m = nx * ny * nz;
    s.n_tiles = ceil_div(m, TILE);
    s.off_rank = 0;
    s.off_tile = align256(size_t(m) * sizeof(int32_t));
    s.off_misc = s.off_tile + align256(size_t(s.n_tiles + 1) * sizeof(int64_t));
    s.total = s.off_misc + align256(64 * sizeof(int64_t));  // misc: [0] n_fluid, [1..27] misses, [28] inlet cells
    return s;
}

__global__ void k_tile_count(const float* __restrict__ phi, int64_t m, int64_t* __restrict__ tile_cnt) {
    __shared__ int warp_sum[TILE_THREADS / 32];
    int64_t base = int64_t(blockIdx.x) * TILE;
    int cnt = 0;
    for (int r = 0; r < TILE_ROUNDS; ++r) {
        int64_t c = base + int64_t(r) * TILE_THREADS + threadIdx.x;
        if (c < m && phi[c] < 0.0f) ++cnt;
    }
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t t = 0;
        for (int w = 0; w < TILE_THREADS / 32; ++w) t += warp_sum[w];
        tile_cnt[blockIdx.x] = t;
    }
}

// Exclusive scan of the tile counts by one block (tile_cnt[n_tiles] receives the total).
__global__ void __launch_bounds__(1024) k_tile_scan(int64_t* __restrict__ tile_cnt, int64_t n_tiles, int64_t* __restrict__ n_fluid) {
    block_exclusive_scan(tile_cnt, n_tiles);
    if (threadIdx.x == 0) *n_fluid = tile_cnt[n_tiles];
}

// Each warp ranks TILE_ROUNDS consecutive groups of 32 cells: all its loads are issued before the first ballot, and
// the block meets once (a barrier per group of 256 cells took 16 us on a grid of 2.8 M cells, this takes 5).
__global__ void k_tile_rank(const float* __restrict__ phi, int64_t m, const int64_t* __restrict__ tile_off,
                            int32_t* __restrict__ rank) {
    __shared__ int warp_cnt[TILE_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t base = int64_t(blockIdx.x) * TILE + int64_t(warp) * (32 * TILE_ROUNDS) + lane;
    float v[TILE_ROUNDS];
#pragma unroll
    for (int r = 0; r < TILE_ROUNDS; ++r) v[r] = base + 32 * r < m ? phi[base + 32 * r] : 0.0f;
    unsigned mask[TILE_ROUNDS];
    int total = 0;
#pragma unroll
    for (int r = 0; r < TILE_ROUNDS; ++r) {
        mask[r] = __ballot_sync(0xffffffffu, v[r] < 0.0f);
        total += __popc(mask[r]);
    }
    if (lane == 0) warp_cnt[warp] = total;
    __syncthreads();
    int64_t before = tile_off[blockIdx.x];
    for (int w = 0; w < warp; ++w) before += warp_cnt[w];
#pragma unroll
    for (int r = 0; r < TILE_ROUNDS; ++r) {
        if (base + 32 * r < m)
            rank[base + 32 * r] = (mask[r] >> lane) & 1u ? int32_t(before + __popc(mask[r] & ((1u << lane) - 1u))) : -1;
        before += __popc(mask[r]);
    }
}

// IDX: int32_t when the grid has fewer than 2^31 cells (a 64-bit division is a subroutine of some 70 instructions).
template <class IDX>
__global__ void k_coords(const int32_t* __restrict__ rank, int64_t nx, int64_t ny, int64_t nz,
                         int32_t* __restrict__ coords) {
    const int64_t m = nx * ny * nz;
    for (int64_t c = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; c < m; c += int64_t(gridDim.x) * blockDim.x) {
        const int32_t r = rank[c];
        if (r >= 0) {
            const IDX row = IDX(c) / IDX(nz), k = IDX(c) - row * IDX(nz);
            const IDX i = row / IDX(ny), j = row - i * IDX(ny);
            coords[3 * int64_t(r)] = int32_t(i);
            coords[3 * int64_t(r) + 1] = int32_t(j);
            coords[3 * int64_t(r) + 2] = int32_t(k);
        }
    }
}

struct OpeningSet {
    int n;                       // openings in claim order (inlets, then outlets)
    int last_inlet;              // index of the last inlet, -1 if none
    int code[MAX_OPENINGS];      // INLET or OUTLET0 - k
    double c[MAX_OPENINGS][3];
    double nrm[MAX_OPENINGS][3];
    double lim[MAX_OPENINGS];    // radius + slack * dx
    double radius[MAX_OPENINGS];
};

struct Grid {
    int64_t dims[3];
    int periodic;
    double origin[3];
    double dx;
};

// Coordinate v - c of one axis (c = -1, 0, 1), wrapped when the axis is periodic; -1 when it leaves the grid.
template <class IDX>
__device__ __forceinline__ IDX shifted(IDX v, int c, IDX dim, bool periodic) {
    IDX x = v - IDX(c);
    if (periodic) x = x < 0 ? x + dim : (x >= dim ? x - dim : x);
    return x >= 0 && x < dim ? x : IDX(-1);
}

// Cell of node (x, y, z)'s pull source along link i, or -1 outside the grid.
template <class IDX>
__device__ __forceinline__ IDX source_cell(const Grid& g, IDX x, IDX y, IDX z, int cx, int cy, int cz, IDX out[3]) {
    out[0] = shifted(x, cx, IDX(g.dims[0]), g.periodic & 1);
    out[1] = shifted(y, cy, IDX(g.dims[1]), (g.periodic >> 1) & 1);
    out[2] = shifted(z, cz, IDX(g.dims[2]), (g.periodic >> 2) & 1);
    if (out[0] < 0 || out[1] < 0 || out[2] < 0) return IDX(-1);
    return (out[0] * IDX(g.dims[1]) + out[1]) * IDX(g.dims[2]) + out[2];
}

// Pass A: pull sources; the missing links of each node as a mask of directions in miss_mask[3 n]; missing links per
// direction (len(miss) at lbm.py:294). One thread per node finds all 27 sources, so its coordinates are read once and
// the 27 reads of the rank grid hit the lines its neighbours read; bound by the 216 bytes a node writes. One thread
// per link instead, with its 64-bit divisions, took 905 us on 839 k nodes.
template <class IDX>
__global__ void __launch_bounds__(256) k_links_src(Grid g, const int32_t* __restrict__ coords,
                                                   const int32_t* __restrict__ rank, int64_t n_fl,
                                                   int32_t* __restrict__ nbr, float* __restrict__ q,
                                                   uint32_t* __restrict__ miss_mask, int64_t* __restrict__ misses) {
    __shared__ int miss_blk[Q];
    if (threadIdx.x < Q) miss_blk[threadIdx.x] = 0;
    __syncthreads();
    const int64_t n = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    uint32_t mask = 0;
    if (n < n_fl) {
        const IDX x = coords[3 * n], y = coords[3 * n + 1], z = coords[3 * n + 2];
        int32_t src[Q];
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            IDX cell[3];
            const IDX c = source_cell<IDX>(g, x, y, z, Lat::cx(i), Lat::cy(i), Lat::cz(i), cell);
            src[i] = c >= 0 ? __ldg(rank + c) : -1;
        }
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            if (src[i] < 0) mask |= 1u << i;
            nbr[int64_t(i) * n_fl + n] = src[i] < 0 ? CS_WALL : src[i];
            q[int64_t(i) * n_fl + n] = 0.5f;
        }
        miss_mask[3 * n] = mask;
    }
    if (__any_sync(0xffffffffu, mask != 0)) {
        const int lane = threadIdx.x & 31;
        int cnt = 0;
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            const unsigned b = __ballot_sync(0xffffffffu, (mask >> i) & 1u);
            if (lane == i) cnt = __popc(b);
        }
        if (cnt) atomicAdd(&miss_blk[lane], cnt);
    }
    __syncthreads();
    if (threadIdx.x < Q && miss_blk[threadIdx.x])
        atomicAdd((unsigned long long*)&misses[threadIdx.x], (unsigned long long)miss_blk[threadIdx.x]);
}

__device__ inline double row_dot(double x, double y, double z, const double* nv, bool single_row) {
    if (single_row) return __fma_rn(z, nv[2], __fma_rn(y, nv[1], __dmul_rn(x, nv[0])));
    return __fma_rn(z, nv[2], __fma_rn(x, nv[0], __dmul_rn(y, nv[1])));
}

// Axial coordinate of point p along the opening, and what its distance from the axis needs (lbm.py:301-303).
__device__ inline double axial(const double p[3], const double* c, const double* nv, bool single_row, double r[3]) {
    for (int a = 0; a < 3; ++a) r[a] = __dsub_rn(p[a], c[a]);
    return row_dot(r[0], r[1], r[2], nv, single_row);
}

__device__ inline double lateral(const double r[3], double ax, const double* nv) {
    const double v0 = __dsub_rn(r[0], __dmul_rn(ax, nv[0]));
    const double v1 = __dsub_rn(r[1], __dmul_rn(ax, nv[1]));
    const double v2 = __dsub_rn(r[2], __dmul_rn(ax, nv[2]));
    return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(v0, v0), __dmul_rn(v1, v1)), __dmul_rn(v2, v2)));
}

constexpr int C_THREADS = 256;
constexpr int C_NODES = 512;

// Pass B: classify missing links, wall q, link counts. A block lists the missing links of its window of nodes in shared
// memory (one node in ten has any, then some seven) and gives each link a thread, so that whole warps work: a thread
// per link of every node took 309 us on 839 k nodes, four threads per boundary node 154 (7.6 of 32 lanes at work), this
// 41. It also clears the inlet profile, whose first word per node brought the mask, and marks there the cells with
// an inlet link.
template <class IDX>
__global__ void __launch_bounds__(C_THREADS) k_links_classify(Grid g, OpeningSet os, const float* __restrict__ phi,
                                                              const int32_t* __restrict__ coords, int64_t n_fl,
                                                              const int64_t* __restrict__ misses,
                                                              int32_t* __restrict__ nbr, float* __restrict__ q,
                                                              float* __restrict__ uin, int64_t* __restrict__ counts,
                                                              int n_outlets, int64_t* __restrict__ n_inlet_cells) {
    __shared__ uint16_t s_link[C_NODES * Q];           // node in the window * 32 + direction
    __shared__ uint8_t s_inlet[C_NODES], s_single[Q];
    __shared__ int s_n, s_cells, s_cnt[2 + MAX_OPENINGS];
    const int lane = threadIdx.x & 31;
    const int64_t base = int64_t(blockIdx.x) * C_NODES;
    if (threadIdx.x == 0) s_n = s_cells = 0;
    if (threadIdx.x < Q) s_single[threadIdx.x] = misses[threadIdx.x] == 1;
    for (int k = threadIdx.x; k < 2 + MAX_OPENINGS; k += C_THREADS) s_cnt[k] = 0;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < C_NODES / C_THREADS; ++r) {
        const int k = r * C_THREADS + threadIdx.x;
        uint32_t m = base + k < n_fl ? reinterpret_cast<const uint32_t*>(uin)[3 * (base + k)] : 0u;
        s_inlet[k] = 0;
        if (!__any_sync(0xffffffffu, m != 0)) continue;
        const int own = __popc(m);
        int upto = own;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        int at = 0;
        if (lane == 31) at = atomicAdd(&s_n, upto);
        at = __shfl_sync(0xffffffffu, at, 31) + upto - own;
        for (; m; m &= m - 1) s_link[at++] = uint16_t(k * 32 + __ffs(m) - 1);
    }
    __syncthreads();
    const int64_t words = 3 * (min(n_fl - base, int64_t(C_NODES)));
    for (int k = threadIdx.x; k < words; k += C_THREADS) uin[3 * base + k] = 0.0f;
    const int links = s_n;
    int wall = 0, inlet = 0;
    for (int w = threadIdx.x; w < links; w += C_THREADS) {
        const int e = s_link[w] >> 5, i = s_link[w] & 31;
        const int64_t n = base + e;
        const IDX at[3] = {IDX(coords[3 * n]), IDX(coords[3 * n + 1]), IDX(coords[3 * n + 2])};
        const int c3[3] = {k_c[0][i], k_c[1][i], k_c[2][i]};
        IDX cell[3];
        const IDX m = source_cell<IDX>(g, at[0], at[1], at[2], c3[0], c3[1], c3[2], cell);
        const float px = phi[(at[0] * IDX(g.dims[1]) + at[1]) * IDX(g.dims[2]) + at[2]];
        const float ps = m >= 0 ? phi[m] : __int_as_float(0x7fc00000);       // NaN outside the grid
        // the source's position, wrapped on the periodic axes only
        double p[3];
        for (int a = 0; a < 3; ++a) {
            const IDX v = cell[a] >= 0 ? cell[a] : at[a] - IDX(c3[a]);
            p[a] = __dadd_rn(g.origin[a], __dmul_rn(double(v), g.dx));
        }
        const bool single = s_single[i] != 0;
        int32_t code = CS_WALL;
        for (int o = 0; o < os.n; ++o) {
            double r[3];
            const double ax = axial(p, os.c[o], os.nrm[o], single, r);
            if (ax >= -1e-6 && lateral(r, ax, os.nrm[o]) < os.lim[o]) {
                code = os.code[o];
                break;
            }
        }
        const int64_t t = int64_t(i) * n_fl + n;
        if (code == CS_WALL) {
            const float qq = __fdiv_rn(-px, __fsub_rn(ps, px));
            q[t] = isfinite(qq) ? fminf(fmaxf(qq, 0.001f), 1.0f) : 0.5f;
            ++wall;
        } else {
            nbr[t] = code;
            if (code == CS_INLET) {
                s_inlet[e] = 1;
                ++inlet;
            } else {
                atomicAdd(&s_cnt[2 + (CS_OUTLET0 - code)], 1);
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        wall += __shfl_down_sync(0xffffffffu, wall, o);
        inlet += __shfl_down_sync(0xffffffffu, inlet, o);
    }
    if (lane == 0) {
        if (wall) atomicAdd(&s_cnt[0], wall);
        if (inlet) atomicAdd(&s_cnt[1], inlet);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < C_NODES; e += C_THREADS)
        if (s_inlet[e]) {
            reinterpret_cast<uint32_t*>(uin)[3 * (base + e)] = INLET_CELL;
            atomicAdd(&s_cells, 1);
        }
    __syncthreads();
    if (threadIdx.x == 0 && s_cells) atomicAdd((unsigned long long*)n_inlet_cells, (unsigned long long)s_cells);
    for (int k = threadIdx.x; k < 2 + n_outlets; k += C_THREADS)
        if (s_cnt[k]) atomicAdd((unsigned long long*)&counts[k], (unsigned long long)s_cnt[k]);
}

// Inlet profile of the marked cells, from the last inlet (lbm.py:322-328).
__global__ void k_inlet_profile(Grid g, OpeningSet os, const int32_t* __restrict__ coords, int64_t n_fl,
                                const int64_t* __restrict__ n_inlet_cells, float* __restrict__ uin) {
    const int64_t n = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (n < n_fl && reinterpret_cast<const uint32_t*>(uin)[3 * n] == INLET_CELL) {
        const int o = os.last_inlet;
        double p[3], r[3];
        for (int a = 0; a < 3; ++a) p[a] = __dadd_rn(g.origin[a], __dmul_rn(double(coords[3 * n + a]), g.dx));
        const double ax = axial(p, os.c[o], os.nrm[o], *n_inlet_cells == 1, r);
        const double rr = __ddiv_rn(lateral(r, ax, os.nrm[o]), os.radius[o]);
        double prof = __dmul_rn(2.0, __dsub_rn(1.0, __dmul_rn(rr, rr)));
        prof = prof < 0.0 ? 0.0 : prof;  // np.clip(., 0, None): NaN stays NaN
        for (int a = 0; a < 3; ++a) uin[3 * n + a] = __double2float_rn(__dmul_rn(-prof, os.nrm[o][a]));
    }
}

template <class IDX>
int fill_tables(const Grid& g, const OpeningSet& os, const float* phi, const int32_t* rank, int64_t* misc, int64_t n_fluid,
                int n_out, int32_t* nbr, float* q, float* uin, int32_t* coords, int64_t* counts, cudaStream_t st) {
    const int64_t m = g.dims[0] * g.dims[1] * g.dims[2];
    CS_CUDA(cudaMemsetAsync(misc + 1, 0, 28 * sizeof(int64_t), st));
    k_coords<IDX><<<unsigned(std::min<int64_t>(ceil_div(m, 256), 148 * 64)), 256, 0, st>>>(rank, g.dims[0], g.dims[1],
                                                                                         g.dims[2], coords);
    CS_CHECK_LAUNCH("k_coords");
    k_links_src<IDX><<<unsigned(ceil_div(n_fluid, 256)), 256, 0, st>>>(g, coords, rank, n_fluid, nbr, q,
                                                                     reinterpret_cast<uint32_t*>(uin), misc + 1);
    CS_CHECK_LAUNCH("k_links_src");
    k_links_classify<IDX><<<unsigned(ceil_div(n_fluid, C_NODES)), C_THREADS, 0, st>>>(
        g, os, phi, coords, n_fluid, misc + 1, nbr, q, uin, counts, n_out, misc + 28);
    CS_CHECK_LAUNCH("k_links_classify");
    if (os.last_inlet >= 0) {
        k_inlet_profile<<<unsigned(ceil_div(n_fluid, 256)), 256, 0, st>>>(g, os, coords, n_fluid, misc + 28, uin);
        CS_CHECK_LAUNCH("k_inlet_profile");
    }
    return CS_OK;
}

}  // namespace
}  // namespace cs

using namespace cs;

extern "C" size_t cs_lattice_scratch_bytes(int64_t nx, int64_t ny, int64_t nz) {
    if (nx < 0 || ny < 0 || nz < 0) return 0;
    return layout(nx, ny, nz).total;
}

extern "C" int cs_lattice_count(const float* phi, int64_t nx, int64_t ny, int64_t nz, void* scratch,
                                int64_t* n_fluid, void* stream) {
    if (nx < 0 || ny < 0 || nz < 0 || !n_fluid) return fail(CS_ERR_ARG, "cs_lattice_count: bad grid or output");
    int64_t m = nx * ny * nz;
    if (m > 0 && (!phi || !scratch)) return fail(CS_ERR_ARG, "cs_lattice_count: null phi or scratch");
    if (m > (int64_t(1) << 40)) return fail(CS_ERR_SIZE, "cs_lattice_count: grid of %lld cells", (long long)m);
    ScratchLayout L = layout(nx, ny, nz);
    cudaStream_t st = as_stream(stream);
    char* s = static_cast<char*>(scratch);
    int64_t* tile = reinterpret_cast<int64_t*>(s + L.off_tile);
    int64_t* misc = reinterpret_cast<int64_t*>(s + L.off_misc);
    CS_CUDA(cudaMemsetAsync(misc, 0, 64 * sizeof(int64_t), st));
    if (m > 0) {
        k_tile_count<<<unsigned(L.n_tiles), TILE_THREADS, 0, st>>>(phi, m, tile);
        CS_CHECK_LAUNCH("k_tile_count");
        k_tile_scan<<<1, 1024, 0, st>>>(tile, L.n_tiles, misc);
        CS_CHECK_LAUNCH("k_tile_scan");
        k_tile_rank<<<unsigned(L.n_tiles), TILE_THREADS, 0, st>>>(phi, m, tile,
                                                                    reinterpret_cast<int32_t*>(s + L.off_rank));
        CS_CHECK_LAUNCH("k_tile_rank");
    }
    int64_t nf = 0;
    CS_CUDA(cudaMemcpyAsync(&nf, misc, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    CS_CUDA(cudaStreamSynchronize(st));
    if (nf >= (int64_t(1) << 30))
        return fail(CS_ERR_SIZE, "cs_lattice_count: %lld fluid nodes (node ids are int32 < 2^30)", (long long)nf);
    *n_fluid = nf;
    return CS_OK;
}

extern "C" int cs_lattice_fill(const float* phi, int64_t nx, int64_t ny, int64_t nz, const double* origin,
                               double dx, const cs_opening* openings, int32_t n_openings, int32_t periodic_mask,
                               double opening_slack, void* scratch, int64_t n_fluid, int32_t* nbr, float* q,
                               float* uin, int32_t* coords, int64_t* counts, void* stream) {
    if (nx < 0 || ny < 0 || nz < 0 || n_fluid < 0 || !origin) return fail(CS_ERR_ARG, "cs_lattice_fill: bad arguments");
    if (n_openings < 0 || n_openings > MAX_OPENINGS)
        return fail(CS_ERR_SIZE, "cs_lattice_fill: %d openings (at most %d)", n_openings, MAX_OPENINGS);
    if (n_openings > 0 && !openings) return fail(CS_ERR_ARG, "cs_lattice_fill: null openings");
    if (!counts) return fail(CS_ERR_ARG, "cs_lattice_fill: null counts");
    OpeningSet os{};
    int n_out = 0;
    os.last_inlet = -1;
    for (int pass = 0; pass < 2; ++pass) {          // inlets first, then outlets (lbm.py:298)
        for (int k = 0; k < n_openings; ++k) {
            const cs_opening& o = openings[k];
            if (o.kind != 0 && o.kind != 1) return fail(CS_ERR_ARG, "cs_lattice_fill: opening %d kind %d", k, o.kind);
            if (o.kind != pass) continue;
            int idx = os.n++;
            os.code[idx] = pass == 0 ? CS_INLET : CS_OUTLET0 - n_out++;
            if (pass == 0) os.last_inlet = idx;
            for (int a = 0; a < 3; ++a) {
                os.c[idx][a] = o.centre[a];
                os.nrm[idx][a] = o.normal[a];
            }
            os.lim[idx] = o.radius + opening_slack * dx;
            os.radius[idx] = o.radius;
        }
    }
    cudaStream_t st = as_stream(stream);
    CS_CUDA(cudaMemsetAsync(counts, 0, size_t(2 + n_out) * sizeof(int64_t), st));
    if (n_fluid == 0) return CS_OK;
    if (!phi || !scratch || !nbr || !q || !uin || !coords) return fail(CS_ERR_ARG, "cs_lattice_fill: null buffer");
    ScratchLayout L = layout(nx, ny, nz);
    char* s = static_cast<char*>(scratch);
    const int32_t* rank = reinterpret_cast<const int32_t*>(s + L.off_rank);
    int64_t* misc = reinterpret_cast<int64_t*>(s + L.off_misc);
    const Grid g{{nx, ny, nz}, periodic_mask & 7, {origin[0], origin[1], origin[2]}, dx};
    return nx * ny * nz < (int64_t(1) << 31)
               ? fill_tables<int32_t>(g, os, phi, rank, misc, n_fluid, n_out, nbr, q, uin, coords, counts, st)
               : fill_tables<int64_t>(g, os, phi, rank, misc, n_fluid, n_out, nbr, q, uin, coords, counts, st);
}

// ---- sponge (lbm.py:398-416) --------------------------------------------------------------------------------------
// Per-cell relaxation near the openings, in the reference's float64 order of operations and rounding: tau_cell = max
// over the chosen openings of tau + (tau_max - tau) * smoothstep(clip(1 - depth / length, 0, 1)) where the cell is
// within 1.5 radii of the opening's axis, depth = -axial / dx; om = float32(1 / tau_cell). The reference's cell
// positions come from np.argwhere, a column-major (N, 3) array, and NumPy's `rel @ nrm` on it evaluates, on the host
// that wrote the fixtures, fma(x, n0, y * n1) + z * n2 for all rows but the last N mod 4, and fma(z, n2, fma(y, n1,
// x * n0)) for those (the column-major BLAS kernel's blocks of four rows and its remainder).
namespace cs {
namespace {

struct SpongeSet {
    int n;
    double c[MAX_OPENINGS][3];
    double nrm[MAX_OPENINGS][3];
    double reach[MAX_OPENINGS];   // 1.5 radius
};

__global__ void k_sponge(const int32_t* __restrict__ coords, int64_t n, double o0, double o1, double o2, double dx,
                         SpongeSet ss, double tau, double length, double tau_max, float* __restrict__ om,
                         double* __restrict__ tau_out) {
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= n) return;
    const double origin[3] = {o0, o1, o2};
    double p[3];
    for (int a = 0; a < 3; ++a) p[a] = __dadd_rn(origin[a], __dmul_rn(double(coords[3 * k + a]), dx));
    const bool tail = k >= n - n % 4;
    double out = tau;
    for (int j = 0; j < ss.n; ++j) {
        const double* nv = ss.nrm[j];
        const double r0 = __dsub_rn(p[0], ss.c[j][0]), r1 = __dsub_rn(p[1], ss.c[j][1]);
        const double r2 = __dsub_rn(p[2], ss.c[j][2]);
        const double ax = tail ? __fma_rn(r2, nv[2], __fma_rn(r1, nv[1], __dmul_rn(r0, nv[0])))
                               : __dadd_rn(__fma_rn(r0, nv[0], __dmul_rn(r1, nv[1])), __dmul_rn(r2, nv[2]));
        const double v0 = __dsub_rn(r0, __dmul_rn(ax, nv[0]));
        const double v1 = __dsub_rn(r1, __dmul_rn(ax, nv[1]));
        const double v2 = __dsub_rn(r2, __dmul_rn(ax, nv[2]));
        const double lat = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(v0, v0), __dmul_rn(v1, v1)), __dmul_rn(v2, v2)));
        const double depth = __ddiv_rn(-ax, dx);
        double w = __dsub_rn(1.0, __ddiv_rn(depth, length));
        w = w < 0.0 ? 0.0 : (w > 1.0 ? 1.0 : w);
        w = __dmul_rn(__dmul_rn(w, w), __dsub_rn(3.0, __dmul_rn(2.0, w)));
        const double v = lat < ss.reach[j] ? __dadd_rn(tau, __dmul_rn(__dsub_rn(tau_max, tau), w)) : tau;
        out = v > out ? v : out;
    }
    om[k] = __double2float_rn(__ddiv_rn(1.0, out));
    if (tau_out) tau_out[k] = out;
}

}  // namespace
}  // namespace cs

extern "C" int cs_sponge_om(const int32_t* coords, int64_t n, const double* origin, double dx,
                            const cs_opening* openings, int32_t n_openings, int32_t kinds_mask, double tau,
                            double length, double tau_max, float* om, double* tau_out, void* stream) {
    if (n < 0 || !origin || !(dx > 0.0) || !(length > 0.0) || (kinds_mask & ~3))
        return fail(CS_ERR_ARG, "cs_sponge_om: bad arguments");
    if (n_openings < 0 || n_openings > MAX_OPENINGS)
        return fail(CS_ERR_SIZE, "cs_sponge_om: %d openings (at most %d)", n_openings, MAX_OPENINGS);
    if (n_openings > 0 && !openings) return fail(CS_ERR_ARG, "cs_sponge_om: null openings");
    SpongeSet ss{};
    for (int k = 0; k < n_openings; ++k) {
        const cs_opening& o = openings[k];
        if (o.kind != 0 && o.kind != 1) return fail(CS_ERR_ARG, "cs_sponge_om: opening %d kind %d", k, o.kind);
        if (!(kinds_mask & (1 << o.kind))) continue;
        const int j = ss.n++;
        for (int a = 0; a < 3; ++a) {
            ss.c[j][a] = o.centre[a];
            ss.nrm[j][a] = o.normal[a];
        }
        ss.reach[j] = 1.5 * o.radius;             // one IEEE product, as NumPy
    }
    if (n == 0) return CS_OK;
    if (!coords || !om) return fail(CS_ERR_ARG, "cs_sponge_om: null buffer");
    k_sponge<<<unsigned(ceil_div(n, 256)), 256, 0, as_stream(stream)>>>(coords, n, origin[0], origin[1], origin[2], dx,
                                                                      ss, tau, length, tau_max, om, tau_out);
    CS_CHECK_LAUNCH("k_sponge");
    return CS_OK;
}
