// Sparse D3Q27 step on the GPU: lbm.k_clock + lbm.k_step (lbm.py:90-257) and, for the artery solver,
// simulate.k_flux + simulate.k_bc (simulate.py:65-82).
//
// One step = two or three kernels on one stream, each launched programmatically so that its blocks start under the last
// one's (all with one division of the SM's memory: set_carveout):
//  1. k_boundary — the wall / inlet / outlet link list (lbm.py:163-181). One thread per ghost slot (a boundary link of
//     one direction); it evaluates what the reference's pull produces for that link — Bouzidi interpolation (q < 0.5
//     with the second node, q >= 0.5 with the node's own population), half-way bounce-back, the velocity inlet with the
//     drive, the pressure outlet with p_out and the previous velocity — and stores it in the ghost slot
//     f_in[i * fstride + n + g] of the step's input buffer.
//  2. k_bulk (k_bulk_dense: the regularised step without body force in blocks of <= 128 threads, 8 or 9 per SM) — one
//     thread per fluid node, C-ordered nodes, link-major populations (the reference's SoA layout).
//     Every link is a plain pull f_in[i * fstride + links[i * n + node]] (a fluid source or a ghost slot), so the 27
//     loads carry no branch and issue back to back; for each link the warp's 32 sources are mostly consecutive,
//     so each load and store moves whole 128-byte lines. Links come in pairs (i, opp(i)) with c_opp = -c_i: the
//     pull accumulates dr, j and Pi = sum c c^T f from each pair's sum and difference, and the collision output is
//     w_i (A + E_i +- O_i) with E even and O odd in c, so each pair's terms are evaluated once. By the D3Q27
//     isotropy sum_i w_i c c^T feq2_i = dr/3 I + u u^T, the regularised projection P = sum c c^T (f - feq2)
//     (lbm.py:219-223) is Pi - dr/3 I - u u^T; no population is kept in registers. Galilean correction
//     (lbm.py:192-204) from the six axis neighbours' previous velocity (a ghost slot gives the wall's q or marks an
//     opening); cells with an inlet link (om < 0) get the inlet equilibrium (lbm.py:205-216); TRT (lbm.py:241-255)
//     keeps the populations.
//     Its first block is the clock (lbm.py:94-102): it stores this step's drive, advances tick[1 - a] = tick[a] + 1 and
//     evaluates the next step's drive.
//  3. k_bc (only with the resistance coupling) — one block: p_out[0] = drive, p_out[k] relaxed towards R_k Q_k - pref
//     in FP64, Qlast = Q, Q = 0 (simulate.py:76-82). The slab flux Q_k = sum u . w itself is reduced in the
//     bulk kernel in FP64 by the blocks that hold flux cells (simulate.py:65-69).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "cs_common.cuh"

#include <vector>

namespace cs {
namespace {

constexpr int MAX_BLOCK = 256;
constexpr int MIN_BLOCKS = 4;   // 4 x 256 threads per SM (64 registers): occupancy hides the pulls' latency
constexpr int MAX_OPEN = 8;
constexpr int B_THREADS = 256;
constexpr float PI_F = 3.14159265358979323846f;

__constant__ int k_cx[Q] = {0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, -1, 1};
__constant__ int k_cy[Q] = {0, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, -1, 1, 1, -1};
__constant__ int k_cz[Q] = {0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1, 1, -1, -1, 1, 1, -1, 1, -1};

// A descriptor with its layout, as the kernels take it.
struct StepArgs : cs_step_desc {
    float* drive2;
    int64_t fstride, vstride;
    StepArgs() = default;
    StepArgs(const cs_step_desc& d, const cs_step_layout* l) : cs_step_desc(d) {
        drive2 = l ? l->drive2 : nullptr;
        fstride = l && l->fstride ? l->fstride : d.npad;
        vstride = l && l->vstride ? l->vstride : d.n;
    }
    // where the drive of the step that reads buffer a stands (two pointers to choose from by a: the batched FP32 kernels
    // without a loop spill, 57.2 us against 54.4 a step for four vessels of 100-400 k nodes)
    __device__ __forceinline__ float* drive_slot(int a) const { return drive2 ? drive2 + a : drive; }
};

__device__ __forceinline__ float weight_rt(int i) {
    return i == 0 ? 8.0f / 27.0f : (i < 7 ? 2.0f / 27.0f : (i < 19 ? 1.0f / 54.0f : 1.0f / 216.0f));
}

// 1024 / w_i of the 16-bit formats for a link known at run time, without a division at run time.
__device__ __forceinline__ float scale_rt(int i) {
    constexpr float s0 = 1024.0f / wgt(0), s1 = 1024.0f / wgt(1), s7 = 1024.0f / wgt(7), s19 = 1024.0f / wgt(19);
    return i == 0 ? s0 : (i < 7 ? s1 : (i < 19 ? s7 : s19));
}

// ---- the step's chain of kernels ----------------------------------------------------------------------------------
// Programmatic dependent launch (sm_90+): a kernel launched with the programmatic-serialization attribute may start
// while the previous kernel of the stream is still running; it reads only static tables until
// grid_dependency_wait(), which returns once that kernel has completed and its writes are visible. A kernel calls
// launch_dependents() once the next kernel may be scheduled beside it. Both are no-ops for an ordinary launch.
struct Waited {
    uint32_t token;
};
__device__ __forceinline__ Waited grid_dependency_wait() {
    Waited w;
    asm volatile("griddepcontrol.wait;\n\tmov.u32 %0, 0;" : "=r"(w.token)::"memory");
    return w;
}
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" :::); }

// What a kernel of the step writes (populations, velocities, drive, pressures) is read by ordinary loads after the wait:
// a kernel begins under the one that writes it, and read-only loads (ld.global.nc, __ldg) are neither tied to the wait
// nor meant for memory written while the kernel runs. Tables written before the call take __ldg. The loads take what the
// wait returns, so that the compiler keeps them behind it and orders them among themselves as it likes. (Volatile, in the
// order written, the 1.49 M-node artery took 2 % longer in FP16; through plain pointers, whose space the compiler does not
// know, all steps 1.5-2.5 %.) FIRST: a population that its reader will not need again, out of the caches first.
template <bool FIRST = false>
__device__ __forceinline__ float ld_step(Waited w, const float* p) {
    float v;
    if constexpr (FIRST) asm("ld.global.L1::evict_first.f32 %0, [%1];" : "=f"(v) : "l"(p), "r"(w.token));
    else asm("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p), "r"(w.token));
    return v;
}
__device__ __forceinline__ int32_t ld_step(Waited w, const int32_t* p) {
    int32_t v;
    asm("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(p), "r"(w.token));
    return v;
}
template <bool FIRST>
__device__ __forceinline__ unsigned short ld_step16(Waited w, const void* p) {
    unsigned short v;
    if constexpr (FIRST) asm("ld.global.L1::evict_first.u16 %0, [%1];" : "=h"(v) : "l"(p), "r"(w.token));
    else asm("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p), "r"(w.token));
    return v;
}

// ---- population storage -----------------------------------------------------------------------------------------
// 32-bit element offsets: 27 * fstride < 2^31 is checked on the host. FIRST: see k_bulk_dense.
template <int ST> struct Pop;

template <> struct Pop<CS_STORE_F32> {
    template <bool FIRST = false>
    static __device__ __forceinline__ float ld(Waited t, const void* b, uint32_t idx, float) {
        return ld_step<FIRST>(t, static_cast<const float*>(b) + idx);
    }
    static __device__ __forceinline__ void st(void* b, uint32_t idx, float, float v) { static_cast<float*>(b)[idx] = v; }
    static __device__ __forceinline__ void st_link(void* b, uint32_t idx, int, float v) { static_cast<float*>(b)[idx] = v; }
};

// 16-bit formats store (f - w_i) * 1024 / w_i: all links share one range, well inside FP16's normal numbers, so the
// relative rounding error is the format's 2^-11 (FP16) or 2^-8 (BF16) on every link. w is the link's weight.
template <> struct Pop<CS_STORE_F16> {
    template <bool FIRST = false>
    static __device__ __forceinline__ float ld(Waited t, const void* b, uint32_t idx, float w) {
        return __half2float(__ushort_as_half(ld_step16<FIRST>(t, static_cast<const __half*>(b) + idx))) *
               (w * (1.0f / 1024.0f));
    }
    static __device__ __forceinline__ void st(void* b, uint32_t idx, float w, float v) {
        static_cast<__half*>(b)[idx] = __float2half_rn(v * (1024.0f / w));
    }
    // a value already in the stored scale, (f - w) 1024 / w
    static __device__ __forceinline__ void st_scaled(void* b, uint32_t idx, float g) {
        static_cast<__half*>(b)[idx] = __float2half_rn(g);
    }
    // a value of link i, known at run time
    static __device__ __forceinline__ void st_link(void* b, uint32_t idx, int i, float v) {
        static_cast<__half*>(b)[idx] = __float2half_rn(v * scale_rt(i));
    }
};

template <> struct Pop<CS_STORE_BF16> {
    template <bool FIRST = false>
    static __device__ __forceinline__ float ld(Waited t, const void* b, uint32_t idx, float w) {
        return __bfloat162float(__ushort_as_bfloat16(ld_step16<FIRST>(t, static_cast<const __nv_bfloat16*>(b) + idx))) *
               (w * (1.0f / 1024.0f));
    }
    static __device__ __forceinline__ void st(void* b, uint32_t idx, float w, float v) {
        static_cast<__nv_bfloat16*>(b)[idx] = __float2bfloat16_rn(v * (1024.0f / w));
    }
    static __device__ __forceinline__ void st_scaled(void* b, uint32_t idx, float g) {
        static_cast<__nv_bfloat16*>(b)[idx] = __float2bfloat16_rn(g);
    }
    // a value of link i, known at run time
    static __device__ __forceinline__ void st_link(void* b, uint32_t idx, int i, float v) {
        static_cast<__nv_bfloat16*>(b)[idx] = __float2bfloat16_rn(v * scale_rt(i));
    }
};

// ---- helpers ------------------------------------------------------------------------------------------------------
// drive(t) (lbm.py:95-100, float32) by a whole warp, each lane one term's sine or cosine: a thread alone waits for its
// coefficients from memory one harmonic after the other (4 us for three).
__device__ __forceinline__ float drive_value_warp(const StepArgs& d, int t) {
    const int lane = threadIdx.x & 31;
    const float ph = 2.0f * PI_F * float(t % d.period) / float(d.period);
    float v = d.coef[0];
    for (int k0 = 1; k0 <= d.nh; k0 += 16) {
        const int k = k0 + (lane >> 1);
        float c = 0.0f, f = 0.0f;
        if (k <= d.nh) {
            c = d.coef[2 * k - 1 + (lane & 1)];
            f = lane & 1 ? sinf(float(k) * ph) : cosf(float(k) * ph);
        }
        for (int j = 0; j < 16 && k0 + j <= d.nh; ++j) {
            const float cc = __shfl_sync(0xffffffffu, c, 2 * j), cs_ = __shfl_sync(0xffffffffu, c, 2 * j + 1);
            const float fc = __shfl_sync(0xffffffffu, f, 2 * j), fs = __shfl_sync(0xffffffffu, f, 2 * j + 1);
            v += __fmaf_rn(cs_, fs, cc * fc);       // as the compiler contracts the sum in one thread
        }
    }
    if (t < d.ramp) v *= 0.5f - 0.5f * cosf(PI_F * float(t) / float(d.ramp));
    return v;
}

// Non-uniform central difference (lbm.py:105-126) of one velocity component: gm / gp are the values loaded through
// the links that pull from x - e_a (sm) and x + e_a (sp) — the neighbour's previous velocity component for a fluid
// source, the ghost slot's gq for a boundary link (q >= 0: wall at distance max(q, 0.1) with u = 0; -1: an opening,
// u = u0 at distance 1). Two fluid neighbours (the common case) give the central difference (v2 - v1) / 2.
__device__ __forceinline__ float ddx_g(int32_t sm, int32_t sp, float gm, float gp, float u0, int32_t n_nodes) {
    if (sm < n_nodes && sp < n_nodes) return 0.5f * (gp - gm);
    float h1 = 1.0f, v1 = u0, h2 = 1.0f, v2 = u0;
    if (sm < n_nodes) {
        v1 = gm;
    } else if (gm >= 0.0f) {
        h1 = fmaxf(gm, 0.1f);
        v1 = 0.0f;
    }
    if (sp < n_nodes) {
        v2 = gp;
    } else if (gp >= 0.0f) {
        h2 = fmaxf(gp, 0.1f);
        v2 = 0.0f;
    }
    return (h1 * h1 * (v2 - u0) + h2 * h2 * (u0 - v1)) / (h1 * h2 * (h1 + h2));
}

// Address of what the difference along link k (1..6) reads for velocity component c: the neighbour's component, or
// the ghost slot's q.
__device__ __forceinline__ const float* grad_src(const StepArgs& d, const float* vin, int k, int c, int32_t s) {
    return s < d.n ? vin + int64_t(c) * d.vstride + s : d.gq + int64_t(k) * d.gmax + (s - d.n);
}

// Third-order equilibrium term of link I (lbm.py:129-137) from the velocity monomials; odd in c.
struct Cubic {
    float xxy, xxz, xyy, yyz, xzz, yzz, xyz;
    __device__ __forceinline__ explicit Cubic(float x, float y, float z)
        : xxy(x * x * y), xxz(x * x * z), xyy(x * y * y), yyz(y * y * z), xzz(x * z * z), yzz(y * z * z),
          xyz(x * y * z) {}
    template <int I>
    __device__ __forceinline__ float h3() const {
        constexpr float t = 1.0f / 3.0f;
        constexpr int x = Lat::cx(I), y = Lat::cy(I), z = Lat::cz(I);
        constexpr float ax = float(x * x) - t, ay = float(y * y) - t, az = float(z * z) - t;
        float s = 0.0f;
        if (y) s += ax * float(y) * xxy;
        if (z) s += ax * float(z) * xxz;
        if (x) s += ay * float(x) * xyy;
        if (z) s += ay * float(z) * yyz;
        if (x) s += az * float(x) * xzz;
        if (y) s += az * float(y) * yzz;
        if (x && y && z) s += float(2 * x * y * z) * xyz;   // 27 x y z u_x u_y u_z = 13.5 * (2 x y z) u_x u_y u_z
        return 13.5f * s;
    }
};

template <int I, int N_>
struct Unroll {
    template <class F>
    static __device__ __forceinline__ void run(F&& f) {
        f(std::integral_constant<int, I>{});
        Unroll<I + 1, N_>::run(f);
    }
};
template <int N_>
struct Unroll<N_, N_> {
    template <class F>
    static __device__ __forceinline__ void run(F&&) {}
};

// Moment sums from pulled values; a pair (I, opp(I)) enters through its sum s and difference dd.
struct Moments {
    float dr = 0.f, jx = 0.f, jy = 0.f, jz = 0.f;
    float pxx = 0.f, pyy = 0.f, pzz = 0.f, pxy = 0.f, pxz = 0.f, pyz = 0.f;
    template <int I>
    __device__ __forceinline__ void add_pair(float v, float vo) {
        constexpr int x = Lat::cx(I), y = Lat::cy(I), z = Lat::cz(I);
        const float s = v + vo, dd = v - vo;
        dr += s;
        if (x) jx += x * dd;
        if (y) jy += y * dd;
        if (z) jz += z * dd;
        if (x) pxx += s;
        if (y) pyy += s;
        if (z) pzz += s;
        if (x && y) pxy += (x * y) * s;
        if (x && z) pxz += (x * z) * s;
        if (y && z) pyz += (y * z) * s;
    }
};

// c^T M c for link I with M given by its diagonal and twice its off-diagonal entries.
template <int I>
__device__ __forceinline__ float quad(float mxx, float myy, float mzz, float mxy2, float mxz2, float myz2) {
    constexpr int x = Lat::cx(I), y = Lat::cy(I), z = Lat::cz(I);
    float s = 0.0f;
    if (x) s += mxx;
    if (y) s += myy;
    if (z) s += mzz;
    if (x && y) s += float(x * y) * mxy2;
    if (x && z) s += float(x * z) * mxz2;
    if (y && z) s += float(y * z) * myz2;
    return s;
}

template <int I>
__device__ __forceinline__ float cdot(float ax, float ay, float az) {
    constexpr int x = Lat::cx(I), y = Lat::cy(I), z = Lat::cz(I);
    float s = 0.0f;
    if (x) s += float(x) * ax;
    if (y) s += float(y) * ay;
    if (z) s += float(z) * az;
    return s;
}

// The links the grouped sums below name by index: axis 1, 3, 5 (+x, +y, +z); edges 7 (1,1,0), 9 (1,-1,0), 11 (1,0,1),
// 13 (1,0,-1), 15 (0,1,1), 17 (0,1,-1); corners 19 (1,1,1), 21 (1,1,-1), 23 (1,-1,1), 25 (-1,1,1); each with its
// opposite at index + 1.
constexpr bool pair_is(int i, int x, int y, int z) {
    return Lat::cx(i) == x && Lat::cy(i) == y && Lat::cz(i) == z && Lat::opp(i) == i + 1;
}
static_assert(pair_is(1, 1, 0, 0) && pair_is(3, 0, 1, 0) && pair_is(5, 0, 0, 1), "axis links");
static_assert(pair_is(7, 1, 1, 0) && pair_is(9, 1, -1, 0) && pair_is(11, 1, 0, 1) && pair_is(13, 1, 0, -1) &&
                  pair_is(15, 0, 1, 1) && pair_is(17, 0, 1, -1), "edge links");
static_assert(pair_is(19, 1, 1, 1) && pair_is(21, 1, 1, -1) && pair_is(23, 1, -1, 1) && pair_is(25, -1, 1, 1),
              "corner links");

// Moments of the 27 pulled values (dr = sum f, j = sum c f, Pi = sum c c^T f): each pair (I, opp I) enters through
// its sum s and difference d, and the terms several moments share are added once — the three edge planes, and the
// four corner pairs through a butterfly (their sums give the trace and the three off-diagonals of Pi, their
// differences the corner parts of j). 81 additions instead of 111 for the link-by-link sums.
__device__ __forceinline__ void moments27(const float (&f)[Q], Moments& m) {
    float sp[Q / 2 + 1], dp[Q / 2 + 1];
#pragma unroll
    for (int k = 0; k < 13; ++k) {
        sp[k] = f[1 + 2 * k] + f[2 + 2 * k];
        dp[k] = f[1 + 2 * k] - f[2 + 2 * k];
    }
    // pair k holds links 1 + 2k and 2 + 2k: k = 0, 1, 2 axis; 3 .. 8 edges; 9 .. 12 corners
    const float exy = sp[3] + sp[4], exz = sp[5] + sp[6], eyz = sp[7] + sp[8];
    const float ca = sp[9] + sp[10], cb = sp[9] - sp[10], cc = sp[11] + sp[12], ce = sp[11] - sp[12];
    const float sc = ca + cc;
    m.dr = f[0] + sp[0] + sp[1] + sp[2] + exy + exz + eyz + sc;
    m.pxx = sp[0] + exy + exz + sc;
    m.pyy = sp[1] + exy + eyz + sc;
    m.pzz = sp[2] + exz + eyz + sc;
    m.pxy = (sp[3] - sp[4]) + (ca - cc);
    m.pxz = (sp[5] - sp[6]) + (cb + ce);
    m.pyz = (sp[7] - sp[8]) + (cb - ce);
    const float dpp = dp[9] + dp[10], dpr = dp[9] - dp[10], dpt = dp[11] + dp[12], dpv = dp[11] - dp[12];
    m.jx = dp[0] + dp[3] + dp[4] + dp[5] + dp[6] + (dpp + dpv);
    m.jy = dp[1] + dp[3] - dp[4] + dp[7] + dp[8] + (dpp - dpv);
    m.jz = dp[2] + dp[5] - dp[6] + dp[7] - dp[8] + (dpr + dpt);
}

// One pair's outputs: FP32 stores w (A + e +- o); the 16-bit formats store (f - w) 1024 / w = 1024 (A + e +- o),
// for which A, e and o arrive already multiplied by 1024 (no per-link weight or scale left to apply).
template <int ST, int I>
__device__ __forceinline__ void store_pair(void* fout, uint32_t NP, int32_t n, float A, float e, float o) {
    constexpr int O = Lat::opp(I);
    if constexpr (ST == CS_STORE_F32) {
        constexpr float w = wgt(I);
        const float wb = w * (A + e);
        Pop<ST>::st(fout, uint32_t(I) * NP + uint32_t(n), w, fmaf(w, o, wb));
        Pop<ST>::st(fout, uint32_t(O) * NP + uint32_t(n), w, fmaf(-w, o, wb));
    } else {
        const float b = A + e;
        Pop<ST>::st_scaled(fout, uint32_t(I) * NP + uint32_t(n), b + o);
        Pop<ST>::st_scaled(fout, uint32_t(O) * NP + uint32_t(n), b - o);
    }
}

// Regularised collision output without a body force (lbm.py:129-137, 230-240): f_I = w_I (A + e_I + o_I) and
// f_opp = w_I (A + e_I - o_I), with e_I = c_I^T M c_I for M = 4.5 u u^T + 4.5 (1 - om) P' (given as its diagonal
// and twice its off-diagonal: m*) and o_I = 3 c_I . u + h3_I (the third-order term, with the Galilean model). Axis,
// edge and corner links differ only in signs, so the 13 pairs' e and o come from shared partial sums.
template <int ST, bool GAL>
__device__ __forceinline__ void store_regularised(void* fout, uint32_t NP, int32_t n, float A, float ux, float uy,
                                                  float uz, float mxx, float myy, float mzz, float mxy2,
                                                  float mxz2, float myz2) {
    // SC: the stored scale (1024 for the 16-bit formats, applied to A, M and the constants; exact in binary)
    constexpr float SC = ST == CS_STORE_F32 ? 1.0f : 1024.0f;
    if constexpr (ST == CS_STORE_F32) {
        Pop<ST>::st(fout, uint32_t(n), wgt(0), wgt(0) * A);
    } else {
        A *= SC;
        mxx *= SC;
        myy *= SC;
        mzz *= SC;
        mxy2 *= SC;
        mxz2 *= SC;
        myz2 *= SC;
        Pop<ST>::st_scaled(fout, uint32_t(n), A);
    }
    // third-order terms from the velocity monomials: axis links -4.5 (sum of two), edges 9 (..) - 4.5 (..),
    // corners 9 (+-A1 +-A2 +-A3) +- 27 xyz
    float h1 = 0.f, h3 = 0.f, h5 = 0.f, h7 = 0.f, h9 = 0.f, h11 = 0.f, h13 = 0.f, h15 = 0.f, h17 = 0.f;
    float h19 = 0.f, h21 = 0.f, h23 = 0.f, h25 = 0.f;
    if (GAL) {
        const float x2 = ux * ux, y2 = uy * uy, z2 = uz * uz;
        const float xxy = x2 * uy, xxz = x2 * uz, xyy = ux * y2, yyz = y2 * uz, xzz = ux * z2, yzz = uy * z2;
        const float xyz = ux * uy * uz;
        const float a1 = xxy + yzz, a2 = xxz + yyz, a3 = xyy + xzz;
        h1 = (-4.5f * SC) * a3;
        h3 = (-4.5f * SC) * a1;
        h5 = (-4.5f * SC) * a2;
        h7 = (9.0f * SC) * (xyy + xxy) - (4.5f * SC) * (xzz + yzz);
        h9 = (9.0f * SC) * (xyy - xxy) - (4.5f * SC) * (xzz - yzz);
        h11 = (9.0f * SC) * (xzz + xxz) - (4.5f * SC) * (xyy + yyz);
        h13 = (9.0f * SC) * (xzz - xxz) - (4.5f * SC) * (xyy - yyz);
        h15 = (9.0f * SC) * (yzz + yyz) - (4.5f * SC) * (xxy + xxz);
        h17 = (9.0f * SC) * (yzz - yyz) - (4.5f * SC) * (xxy - xxz);
        const float b1 = (9.0f * SC) * a1, b2 = (9.0f * SC) * a2, b3 = (9.0f * SC) * a3, bx = (27.0f * SC) * xyz;
        const float p_ = b1 + b3, q_ = b2 + bx, m_ = b3 - b1, n_ = b2 - bx;
        h19 = p_ + q_;
        h21 = p_ - q_;
        h23 = m_ + n_;
        h25 = n_ - m_;
    }
    // axis
    store_pair<ST, 1>(fout, NP, n, A, mxx, (3.0f * SC) * ux + h1);
    store_pair<ST, 3>(fout, NP, n, A, myy, (3.0f * SC) * uy + h3);
    store_pair<ST, 5>(fout, NP, n, A, mzz, (3.0f * SC) * uz + h5);
    // edges, plane by plane
    const float sxy = mxx + myy, sxz = mxx + mzz, syz = myy + mzz;
    const float u7 = ux + uy, u9 = ux - uy;
    store_pair<ST, 7>(fout, NP, n, A, sxy + mxy2, (3.0f * SC) * u7 + h7);
    store_pair<ST, 9>(fout, NP, n, A, sxy - mxy2, (3.0f * SC) * u9 + h9);
    store_pair<ST, 11>(fout, NP, n, A, sxz + mxz2, (3.0f * SC) * (ux + uz) + h11);
    store_pair<ST, 13>(fout, NP, n, A, sxz - mxz2, (3.0f * SC) * (ux - uz) + h13);
    store_pair<ST, 15>(fout, NP, n, A, syz + myz2, (3.0f * SC) * (uy + uz) + h15);
    store_pair<ST, 17>(fout, NP, n, A, syz - myz2, (3.0f * SC) * (uy - uz) + h17);
    // corners
    const float tr = sxy + mzz, ca = tr + mxy2, cb = tr - mxy2, cg = mxz2 + myz2, cd = mxz2 - myz2;
    store_pair<ST, 19>(fout, NP, n, A, ca + cg, (3.0f * SC) * (u7 + uz) + h19);
    store_pair<ST, 21>(fout, NP, n, A, ca - cg, (3.0f * SC) * (u7 - uz) + h21);
    store_pair<ST, 23>(fout, NP, n, A, cb + cd, (3.0f * SC) * (u9 + uz) + h23);
    store_pair<ST, 25>(fout, NP, n, A, cb - cd, (3.0f * SC) * (uz - u9) + h25);
}

// ---- 1. boundary-link kernel and clock ----------------------------------------------------------------------------
// The clock. A step reads its drive, drive2[a], from memory: evaluating it (coefficients from memory, a sine and a
// cosine per harmonic) took about 4 us on the step's critical path, in the boundary kernel that everything waits for.
// The bulk kernel of the step before evaluates it beside its nodes. Before the first step of a call there is none: its
// boundary kernel (START) evaluates the drive, each warp with an inlet link for itself and one for everybody, and k_clock
// where there are no boundary links. (A k_clock of its own before every call was a third launch of calls of one step:
// 41.4 us against 37.7 without. Evaluated by every warp, before its populations are asked for, it made a single step from a
// cold L2 2 us longer on the 347 k-node pipe and 5 us on the 1.57 M-node artery.) A caller without a drive2 has no place for
// the next step's drive, and every step begins like the first.
__device__ __forceinline__ void advance_clock(const StepArgs& d, const int a) {
    const int t = d.tick[a];
    if (d.drive2) {
        const float next = drive_value_warp(d, t + 1);
        if ((threadIdx.x & 31) == 0) {
            *d.drive = d.drive2[a];
            d.drive2[1 - a] = next;
        }
    }
    if ((threadIdx.x & 31) == 0) d.tick[1 - a] = t + 1;
}

// The first kernel of a call, this or the START boundary kernel, reads nothing and releases nothing before its wait: what
// the stream did before the call (a caller's kernel that wrote the tables or the relaxation rates) is then complete, and
// every later kernel of the call may read them before its own wait.
__global__ void __launch_bounds__(32) k_clock(const StepArgs d, const int a) {
    grid_dependency_wait();
    launch_dependents();
    const float v = drive_value_warp(d, d.tick[a]);
    if (threadIdx.x == 0) *d.drive_slot(a) = v;
}

// Without nodes there is no bulk kernel to advance the clock.
__global__ void __launch_bounds__(32) k_clock_only(const StepArgs d, const int a) { advance_clock(d, a); }

// Block (bx, by) of a lattice's boundary-link grid: by = direction, bx = chunk of its ghost slots. Pure latency: the
// slot's table words (static, read before the previous kernel has ended), its two populations, the ghost's write. Both
// populations are addressed without a branch, so their loads are in flight together. START: the first kernel of a call;
// publish: this block leaves the drive for the other kernels of the step.
template <int ST, bool START>
__device__ __forceinline__ void boundary_body(const StepArgs& d, const int a, const int bx, const int by,
                                              const bool publish) {
    const int i = by;
    const int32_t g = bx * B_THREADS + int(threadIdx.x);
    const uint32_t slot = uint32_t(i) * uint32_t(d.gmax) + uint32_t(g);       // < 27 npad < 2^31
    const bool live = g < d.gmax;
    Waited t;
    int32_t node, info;
    float q;
    if constexpr (START) {
        t = grid_dependency_wait();
        launch_dependents();
        node = live ? ld_step(t, d.gnode + slot) : -1;
        info = live ? ld_step(t, d.ginfo + slot) : 0;
        q = live ? ld_step(t, d.gq + slot) : 0.0f;
    } else {
        node = live ? __ldg(d.gnode + slot) : -1;
        info = live ? __ldg(d.ginfo + slot) : 0;
        q = live ? __ldg(d.gq + slot) : 0.0f;
    }
    const int io = Lat::opp(i);
    const uint32_t NP = uint32_t(d.fstride), own = uint32_t(io) * NP + uint32_t(node);
    // Bouzidi's second population: the wall's second node (q < 0.5) or the node's own along i
    const bool second = info >= 0 && q < 0.5f;
    const uint32_t other = second ? uint32_t(io) * NP + uint32_t(info) : uint32_t(i) * NP + uint32_t(node);
    const float w = weight_rt(i);                                             // the opposite's weight too
    const void* fin = d.f[a];
    float fo = 0.0f, f2 = 0.0f, dv = 0.0f;
    if constexpr (START) {
        if (node >= 0) {
            fo = Pop<ST>::ld(t, fin, own, w);
            f2 = Pop<ST>::ld(t, fin, other, w);
        }
        asm volatile("" ::"f"(fo), "f"(f2));                // in flight before the drive is evaluated
        const bool first = publish && threadIdx.x < 32;
        if (__any_sync(0xffffffffu, first || (node >= 0 && info == CS_INLET))) {
            dv = drive_value_warp(d, d.tick[a]);
            if (first && threadIdx.x == 0) *d.drive_slot(a) = dv;
        }
        if (node < 0) return;                               // padding slot of a direction with fewer links
    } else {
        t = grid_dependency_wait();
        launch_dependents();                                // the bulk kernel may start its static loads
        if (node < 0) return;
        fo = Pop<ST>::ld(t, fin, own, w);
        if (info >= CS_WALL) f2 = Pop<ST>::ld(t, fin, other, w);
    }
    float v;
    if (info >= CS_WALL) {
        // lbm.py:163-173: interpolated bounce-back, or half-way bounce-back without Bouzidi
        v = fo;
        if (d.bouzidi) {
            if (q < 0.5f) {
                if (second) v = 2.0f * q * fo + (1.0f - 2.0f * q) * f2;
            } else {
                v = fo / (2.0f * q) + (2.0f * q - 1.0f) / (2.0f * q) * f2;
            }
        }
    } else {
        const float cx = float(k_cx[i]), cy = float(k_cy[i]), cz = float(k_cz[i]);
        if (info == CS_INLET) {
            // lbm.py:174-177: bounce-back with the prescribed velocity
            const float* u = d.uin + 3 * int64_t(node);
            if constexpr (!START) dv = ld_step(t, d.drive_slot(a));
            const float cu = cx * (__ldg(u) * dv) + cy * (__ldg(u + 1) * dv) + cz * (__ldg(u + 2) * dv);
            v = fo + 6.0f * w * cu;
        } else {
            // lbm.py:178-181: anti-bounce-back with the outlet's pressure and the previous velocity
            const float* vin = d.vel[a];
            const float e0 = ld_step(t, vin + node), e1 = ld_step(t, vin + d.vstride + node),
                        e2 = ld_step(t, vin + 2 * d.vstride + node);
            const float pk = ld_step(t, d.p_out + (CS_OUTLET0 - info));
            const float cu = cx * e0 + cy * e1 + cz * e2;
            // (rounded as spelled out, so that the result does not hang on the compiler's choice of what to fuse)
            const float usq = __fmaf_rn(e2, e2, __fmaf_rn(e0, e0, e1 * e1));
            const float eq = __fmaf_rn(-1.5f, usq, __fmaf_rn(4.5f * cu, cu, 3.0f * pk));
            v = __fmaf_rn(2.0f * w, eq, -fo);
        }
    }
    Pop<ST>::st_link(d.f[a], uint32_t(i) * NP + uint32_t(d.n) + uint32_t(g), i, v);
}

// Direction of block b of the unpadded boundary grid: the largest i with gblock[i] <= b.
__device__ __forceinline__ int grid_direction(const int32_t* gblock, int b) {
    int lo = 0, hi = Q - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (gblock[mid] <= b) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Work item `item` of a lattice's boundary-link grid: a 256-slot chunk of one direction (unpadded grid when gblock
// is set, else ceil(gmax / 256) chunks per direction).
template <int ST, bool START>
__device__ __forceinline__ void boundary_item(const StepArgs& d, const int a, const int item) {
    if (d.gblock[Q] > 0) {
        const int i = grid_direction(d.gblock, item);
        boundary_body<ST, START>(d, a, item - d.gblock[i], i, item == 0);
    } else {
        const int nbx = int(max(int64_t(1), ceil_div(d.gmax, B_THREADS)));
        boundary_body<ST, START>(d, a, item % nbx, item / nbx, item == 0);
    }
}

__host__ __device__ __forceinline__ int boundary_items(const cs_step_desc& d) {
    if (d.gblock[Q] > 0) return d.gblock[Q];
    const int64_t nbx = d.gmax > 0 ? (d.gmax + B_THREADS - 1) / B_THREADS : 1;
    return int(Q * nbx);
}

template <int ST, bool START>
__global__ void __launch_bounds__(B_THREADS) k_boundary(const StepArgs d, const int a) {
    boundary_item<ST, START>(d, a, blockIdx.x);
}

// ---- 2. bulk kernel -----------------------------------------------------------------------------------------------
// Writes the 27 outputs w_i (A + E_i + O_i) of a pair-symmetric collision: E(I) even and O(I) odd in c, so link I
// and its opposite share both (the rest link is w_0 A).
template <int ST, class EvenOdd>
__device__ __forceinline__ void store_pairs(void* fout, uint32_t NP, int32_t n, float A, EvenOdd&& eo) {
    Pop<ST>::st(fout, uint32_t(n), wgt(0), wgt(0) * A);
    Unroll<0, 13>::run([&](auto pc) {
        constexpr int I = 1 + 2 * decltype(pc)::value;
        constexpr int O = Lat::opp(I);
        float e, o;
        eo(std::integral_constant<int, I>{}, e, o);
        const float base = A + e;
        Pop<ST>::st(fout, uint32_t(I) * NP + uint32_t(n), wgt(I), wgt(I) * (base + o));
        Pop<ST>::st(fout, uint32_t(O) * NP + uint32_t(n), wgt(O), wgt(O) * (base - o));
    });
}

// EARLY: the drive is loaded with everything else; otherwise, without a body force, by the inlet cells that need it. (Late,
// the batched kernels spill less, a sweep of six FP16 vessels 90.5 -> 87.8 us a step; the single kernel of the 1.49 M-node
// FP16 artery takes 69.5 us instead of 67.8.)
template <int ST, int MODEL, bool GAL, bool FORCE, bool FIRST, bool EARLY>
__device__ __forceinline__ void node_update(const StepArgs& d, int a, int32_t n, float& ux_o, float& uy_o,
                                            float& uz_o) {
    const int32_t N = int32_t(d.n), NV = int32_t(d.vstride);
    const uint32_t NP = uint32_t(d.fstride);
    const void* fin = d.f[a];
    void* fout = d.f[1 - a];
    const float* vin = d.vel[a];
    float* vout = d.vel[1 - a];
    // connectivity and omega are static: load them while the boundary kernel may still be running
    int32_t lk[Q];
    const int32_t code = __ldg(d.lcode + n);
    if (code >= 0) {
        // one 112-byte row, shared by the warp's nodes of a segment: seven 128-bit loads
        const int4* sd = reinterpret_cast<const int4*>(d.segdelta + int64_t(code) * CS_SEG_STRIDE);
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            const int4 v = __ldg(sd + k);
            lk[4 * k] = n + v.x;
            if (4 * k + 1 < Q) lk[4 * k + 1] = n + v.y;
            if (4 * k + 2 < Q) lk[4 * k + 2] = n + v.z;
            if (4 * k + 3 < Q) lk[4 * k + 3] = n + v.w;
        }
    } else {
        const int32_t* ir = d.irr + (-1 - code);
#pragma unroll
        for (int i = 0; i < Q; ++i) lk[i] = __ldg(ir + int64_t(i) * d.n_irr);
    }
    const float om_signed = __ldg(d.om + n);
    const Waited waited = grid_dependency_wait();
    const float dv = EARLY || FORCE ? ld_step(waited, d.drive_slot(a)) : 0.0f;
    const float upx = ld_step(waited, vin + n), upy = ld_step(waited, vin + NV + n),
                upz = ld_step(waited, vin + 2 * NV + n);

    // six loads for the Galilean differences, issued with the pull
    float g[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (GAL) {
#pragma unroll
        for (int k = 0; k < 6; ++k) g[k] = ld_step(waited, grad_src(d, vin, 1 + k, k / 2, lk[1 + k]));
    }

    // the 27 pulls (TRT and the body-force path use the populations themselves after the moments)
    Moments m;
    float fk[Q];
    Unroll<0, Q>::run([&](auto ic) {
        constexpr int I = decltype(ic)::value;
        fk[I] = Pop<ST>::template ld<FIRST>(waited, fin, uint32_t(I) * NP + uint32_t(lk[I]), wgt(I));
    });
    moments27(fk, m);

    const bool inlet_cell = om_signed < 0.0f;
    const float om = fabsf(om_signed);
    // without a body force (FORCE false) every force term folds away at compile time
    const float Fx = FORCE ? d.force[0] * dv : 0.0f, Fy = FORCE ? d.force[1] * dv : 0.0f;
    const float Fz = FORCE ? d.force[2] * dv : 0.0f;
    const float ux = m.jx + Fx * 0.5f, uy = m.jy + Fy * 0.5f, uz = m.jz + Fz * 0.5f;
    const float usq = ux * ux + uy * uy + uz * uz;
    const float uF = ux * Fx + uy * Fy + uz * Fz;
    float t3 = 0.0f, edx = 0.0f, edy = 0.0f, edz = 0.0f;
    if (GAL) {
        t3 = 1.0f;
        const float tp3 = 3.0f * __frcp_rn(om);
        edx = tp3 * ux * ux * ddx_g(lk[1], lk[2], g[0], g[1], upx, N);
        edy = tp3 * uy * uy * ddx_g(lk[3], lk[4], g[2], g[3], upy, N);
        edz = tp3 * uz * uz * ddx_g(lk[5], lk[6], g[4], g[5], upz, N);
    }
    const float dr = m.dr;

    if (inlet_cell) {
        // lbm.py:205-216: equilibrium at the prescribed velocity
        const float* u = d.uin + 3 * int64_t(n);
        const float di = EARLY || FORCE ? dv : ld_step(waited, d.drive_slot(a));
        const float tx = __ldg(u) * di, ty = __ldg(u + 1) * di, tz = __ldg(u + 2) * di;
        const float tsq = tx * tx + ty * ty + tz * tz;
        const Cubic cu3(tx, ty, tz);
        store_pairs<ST>(fout, NP, n, dr - 1.5f * tsq, [&](auto ic, float& e, float& o) {
            constexpr int I = decltype(ic)::value;
            const float cu = cdot<I>(tx, ty, tz);
            e = 4.5f * cu * cu;
            o = 3.0f * cu + t3 * cu3.template h3<I>();
        });
        vout[n] = tx;
        vout[NV + n] = ty;
        vout[2 * NV + n] = tz;
        d.rho[n] = dr;
        ux_o = tx;
        uy_o = ty;
        uz_o = tz;
        return;
    }

    const Cubic cu3(ux, uy, uz);
    if constexpr (MODEL == CS_MODEL_REGULARISED) {
        float pxx, pyy, pzz, pxy, pxz, pyz;
        if constexpr (FORCE) {
            // with a body force, P link by link as the reference sums it (lbm.py:220-223): a slowly forced steady
            // state (Poiseuille at tau ~ 0.505, forces ~1e-7) keeps the FP32 rounding of this order
            pxx = pyy = pzz = pxy = pxz = pyz = 0.0f;
            Unroll<0, Q>::run([&](auto ic) {
                constexpr int I = decltype(ic)::value;
                constexpr int x = Lat::cx(I), y = Lat::cy(I), z = Lat::cz(I);
                const float cu = cdot<I>(ux, uy, uz);
                const float sv = fk[I] - wgt(I) * (dr + 3.0f * cu + 4.5f * cu * cu - 1.5f * usq);
                if (x) pxx += sv;
                if (y) pyy += sv;
                if (z) pzz += sv;
                if (x && y) pxy += float(x * y) * sv;
                if (x && z) pxz += float(x * z) * sv;
                if (y && z) pyz += float(y * z) * sv;
            });
        } else {
            const float d3 = dr * (1.0f / 3.0f);
            pxx = m.pxx - d3 - ux * ux, pyy = m.pyy - d3 - uy * uy, pzz = m.pzz - d3 - uz * uz;
            pxy = m.pxy - ux * uy, pxz = m.pxz - ux * uz, pyz = m.pyz - uy * uz;
        }
        if (d.sigma < 1.0f) {
            // hybrid regularisation (lbm.py:224-229): G[a][b] = du_b/dx_a from the previous step's velocity
            float gr[3][3];
            const float u0[3] = {upx, upy, upz};
#pragma unroll
            for (int ax = 0; ax < 3; ++ax) {
                const int km = 1 + 2 * ax, kp = 2 + 2 * ax;
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    gr[ax][c] = ddx_g(lk[km], lk[kp], ld_step(waited, grad_src(d, vin, km, c, lk[km])),
                                      ld_step(waited, grad_src(d, vin, kp, c, lk[kp])), u0[c], N);
            }
            const float sg = d.sigma, k = (1.0f - sg) / (3.0f * om);
            pxx = sg * pxx - k * (2.0f * gr[0][0]);
            pyy = sg * pyy - k * (2.0f * gr[1][1]);
            pzz = sg * pzz - k * (2.0f * gr[2][2]);
            pxy = sg * pxy - k * (gr[0][1] + gr[1][0]);
            pxz = sg * pxz - k * (gr[0][2] + gr[2][0]);
            pyz = sg * pyz - k * (gr[1][2] + gr[2][1]);
        }
        pxx -= edx;
        pyy -= edy;
        pzz -= edz;
        const float trp = (pxx + pyy + pzz) * (1.0f / 3.0f);
        const float k_ne = 1.0f - om, k_src = 1.0f - 0.5f * om;
        if constexpr (FORCE) {
            // f_out = feq + (1 - om) fneq + (1 - om/2) src per link in the reference's order (lbm.py:232-240)
            const float w0 = wgt(0);
            Pop<ST>::st(fout, uint32_t(n), w0, w0 * (dr - 1.5f * usq) + k_ne * (w0 * (4.5f * (0.0f - trp))) +
                                                   k_src * (w0 * (-3.0f * uF)));
            Unroll<0, 13>::run([&](auto pc) {
                constexpr int I = 1 + 2 * decltype(pc)::value;
                constexpr int O = Lat::opp(I);
                const float cu = cdot<I>(ux, uy, uz), cF = cdot<I>(Fx, Fy, Fz);
                const float cpc = quad<I>(pxx, pyy, pzz, 2.0f * pxy, 2.0f * pxz, 2.0f * pyz);
                const float h = t3 * cu3.template h3<I>();
                const float w = wgt(I);
                const float feq_i = w * (dr + 3.0f * cu + 4.5f * cu * cu - 1.5f * usq + h);
                const float feq_o = w * (dr - 3.0f * cu + 4.5f * cu * cu - 1.5f * usq - h);
                const float fneq_i = w * (4.5f * (cpc - trp) - 1.5f * cF);
                const float fneq_o = w * (4.5f * (cpc - trp) + 1.5f * cF);
                const float src_i = w * (3.0f * cF + 9.0f * cu * cF - 3.0f * uF);
                const float src_o = w * (-3.0f * cF + 9.0f * cu * cF - 3.0f * uF);
                Pop<ST>::st(fout, uint32_t(I) * NP + uint32_t(n), w, feq_i + k_ne * fneq_i + k_src * src_i);
                Pop<ST>::st(fout, uint32_t(O) * NP + uint32_t(n), w, feq_o + k_ne * fneq_o + k_src * src_o);
            });
            vout[n] = ux;
            vout[NV + n] = uy;
            vout[2 * NV + n] = uz;
            d.rho[n] = dr;
            ux_o = ux;
            uy_o = uy;
            uz_o = uz;
            return;
        }
        // without a force: f_out = feq + (1 - om) fneq + (1 - om/2) src (lbm.py:236-240) regrouped as
        // w (A + E +- O), each pair's terms evaluated once
        const float A = dr - 1.5f * usq - 4.5f * k_ne * trp;
        const float s = 4.5f * k_ne;
        const float hx = 4.5f * ux, hy = 4.5f * uy;
        store_regularised<ST, GAL>(fout, NP, n, A, ux, uy, uz, fmaf(hx, ux, s * pxx), fmaf(hy, uy, s * pyy),
                                   fmaf(4.5f * uz, uz, s * pzz), fmaf(2.0f * hx, uy, 2.0f * s * pxy),
                                   fmaf(2.0f * hx, uz, 2.0f * s * pxz), fmaf(2.0f * hy, uz, 2.0f * s * pyz));
    } else {
        // TRT + Guo forcing (lbm.py:241-255)
        const float om_m = 1.0f / (0.5f + d.magic / (1.0f / om - 0.5f));
        const float ddx_ = -(1.0f - om) * edx, ddy_ = -(1.0f - om) * edy, ddz_ = -(1.0f - om) * edz;
        const float trd = (ddx_ + ddy_ + ddz_) / 3.0f;
        // FP32: a pair's links differ only in the sign of what is odd in c, so the half sum and the half difference of the two
        // are relaxed apart and added at the end; without a body force its terms are zero and left out (75 k-node pipe 8.3
        // -> 7.0 us a step, 222 k nodes with a force 16.6 -> 13.0). Rounded as spelled out: left to the compiler's
        // contraction, with the equilibria rounded before the difference, the velocity's error against 64 bits was 1.03 of
        // the link-by-link sums' (rms over 48 runs), so it is 0.95 (density 1.00). The 16-bit formats keep the link-by-link
        // sums: another rounding in 32 bits would move stored values by a unit of the 16-bit format.
        if constexpr (ST == CS_STORE_F32) {
            const float ke = 1.0f - 0.5f * om, ko = 1.0f - 0.5f * om_m;
            const float rest = __fmaf_rn(-1.5f, usq, dr);
            {
                float v = __fmaf_rn(-om, __fmaf_rn(-wgt(0), rest, fk[0]), fk[0]);
                if constexpr (FORCE) v += ke * (wgt(0) * (-3.0f * uF));
                Pop<ST>::st(fout, uint32_t(n), wgt(0), __fmaf_rn(wgt(0) * 4.5f, 0.0f - trd, v));
            }
            Unroll<0, 13>::run([&](auto pc) {
                constexpr int I = 1 + 2 * decltype(pc)::value;
                constexpr int O = Lat::opp(I);
                constexpr int x = Lat::cx(I), y = Lat::cy(I), z = Lat::cz(I);
                const float cv = float(x) * ux + float(y) * uy + float(z) * uz;
                const float pd = float(x * x) * ddx_ + float(y * y) * ddy_ + float(z * z) * ddz_ - trd;
                const float hs = 0.5f * (fk[I] + fk[O]), hd = 0.5f * (fk[I] - fk[O]);
                const float even = __fmaf_rn(-wgt(I), __fmaf_rn(4.5f * cv, cv, rest), hs);
                const float odd = __fmaf_rn(-wgt(I), __fmaf_rn(3.0f, cv, t3 * cu3.template h3<I>()), hd);
                float pe = __fmaf_rn(wgt(I) * 4.5f, pd, __fmaf_rn(-om, even, hs)), mo = __fmaf_rn(-om_m, odd, hd);
                if constexpr (FORCE) {
                    const float cF = float(x) * Fx + float(y) * Fy + float(z) * Fz;
                    pe = __fmaf_rn(ke, wgt(I) * __fmaf_rn(9.0f * cv, cF, -3.0f * uF), pe);
                    mo = __fmaf_rn(ko, wgt(I) * 3.0f * cF, mo);
                }
                const float vi = pe + mo, vo = pe - mo;
                Pop<ST>::st(fout, uint32_t(I) * NP + uint32_t(n), wgt(I), vi);
                Pop<ST>::st(fout, uint32_t(O) * NP + uint32_t(n), wgt(I), vo);
            });
        } else {
            Unroll<0, Q>::run([&](auto ic) {
                constexpr int I = decltype(ic)::value;
                constexpr int jo = Lat::opp(I);
                constexpr int x = Lat::cx(I), y = Lat::cy(I), z = Lat::cz(I);
                const float cv = float(x) * ux + float(y) * uy + float(z) * uz;
                const float cF = float(x) * Fx + float(y) * Fy + float(z) * Fz;
                const float eqp = wgt(I) * (dr + 4.5f * cv * cv - 1.5f * usq);
                const float eqm = wgt(I) * (3.0f * cv + t3 * cu3.template h3<I>());
                const float psi = wgt(I) * 4.5f * (float(x * x) * ddx_ + float(y * y) * ddy_ + float(z * z) * ddz_ - trd);
                const float fp = 0.5f * (fk[I] + fk[jo]);
                const float fm = 0.5f * (fk[I] - fk[jo]);
                const float sp = wgt(I) * (9.0f * cv * cF - 3.0f * uF);
                const float smv = wgt(I) * 3.0f * cF;
                Pop<ST>::st(fout, uint32_t(I) * NP + uint32_t(n), wgt(I),
                            fk[I] - om * (fp - eqp) - om_m * (fm - eqm) + (1.0f - 0.5f * om) * sp +
                                (1.0f - 0.5f * om_m) * smv + psi);
            });
        }
    }
    vout[n] = ux;
    vout[NV + n] = uy;
    vout[2 * NV + n] = uz;
    d.rho[n] = dr;
    ux_o = ux;
    uy_o = uy;
    uz_o = uz;
}

// Block bx of a lattice's bulk grid (nodes bx * blockDim .. + blockDim - 1). Called by every thread of the block.
// OPEN: the lattice may have open ends (n_open > 0); compiled apart for the kernels that lose by carrying their reduction
// (cylinder 5.14 us a step against 5.07; batches of a block an item 59.4 against 55.4 on four FP32 vessels of 100-400 k
// nodes, 97.3 against 92.0 on six FP16 ones). clock: this block also advances the clock.
template <int ST, int MODEL, bool GAL, bool FORCE, bool OPEN, bool FIRST = false, bool EARLY = false>
__device__ __forceinline__ void bulk_body(const StepArgs& d, const int a, const int bx, const bool clock) {
    const int32_t n0 = int32_t(bx) * int32_t(blockDim.x);
    const int32_t n = n0 + int32_t(threadIdx.x);
    // read after the update: bring the line in meanwhile, at the cost of no register
    if (OPEN && d.n_open > 0) asm volatile("prefetch.global.L1 [%0];" ::"l"(d.flux_block + bx));
    float ux = 0.f, uy = 0.f, uz = 0.f;
    if (n < d.n) node_update<ST, MODEL, GAL, FORCE, FIRST, EARLY>(d, a, n, ux, uy, uz);
    grid_dependency_wait();      // (threads without a node) the flux accumulators were reset by the last step
    launch_dependents();
    if (clock && threadIdx.x < 32) advance_clock(d, a);

    if (OPEN && d.n_open > 0) {
        // slab flux Q_k = sum u . w over this block's flux entries (simulate.py:65-69), FP64, in a fixed order: each
        // thread sums its entries, warps reduce by shuffles, the warps' sums are added in order; the block's partial
        // sums go to its own row of q_part, which k_bc adds up in a fixed order too (no atomics: bit-reproducible).
        // In an order along the vessel nearly every block holds a few entries (7 of 128 nodes on a 190 k-node
        // artery), so only the warps and open ends that have any take part.
        const int e0 = __ldg(d.flux_block + bx), e1 = __ldg(d.flux_block + bx + 1);
        if (e1 > e0) {
            __shared__ float s_u[3][MAX_BLOCK];
            s_u[0][threadIdx.x] = ux;
            s_u[1][threadIdx.x] = uy;
            s_u[2][threadIdx.x] = uz;
            __syncthreads();
            __shared__ double s_w[MAX_BLOCK / 32][MAX_OPEN];
            const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
            const int busy = min(int(blockDim.x) / 32, (e1 - e0 + 31) / 32);
            if (warp < busy) {
                double acc[MAX_OPEN];
#pragma unroll
                for (int k = 0; k < MAX_OPEN; ++k) acc[k] = 0.0;
                for (int e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
                    const int loc = __ldg(d.flux_idx + e) - n0;
                    if (loc < 0 || loc >= int(blockDim.x)) continue;  // partition built for another block size
                    const float* w = d.flux_w + 3 * int64_t(e);
                    const double v = double(s_u[0][loc]) * double(__ldg(w)) + double(s_u[1][loc]) * double(__ldg(w + 1)) +
                                     double(s_u[2][loc]) * double(__ldg(w + 2));
                    const int slot = __ldg(d.flux_slot + e);
#pragma unroll
                    for (int k = 0; k < MAX_OPEN; ++k) acc[k] += slot == k ? v : 0.0;
                }
#pragma unroll
                for (int k = 0; k < MAX_OPEN; ++k) {
                    if (k >= d.n_open) break;
                    double x = acc[k];
                    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
                    if (lane == 0) s_w[warp][k] = x;
                }
            }
            __syncthreads();
            if (threadIdx.x < d.n_open) {
                double t = 0.0;
                for (int w = 0; w < busy; ++w) t += s_w[w][threadIdx.x];
                d.q_part[int64_t(bx) * MAX_OPEN + threadIdx.x] = t;
            }
        }
    }
}

// A block of a single lattice's grid; the first is the clock, beside the node blocks.
template <int ST, int MODEL, bool GAL, bool FORCE, bool OPEN, bool FIRST = false>
__device__ __forceinline__ void bulk_block(const StepArgs& d, const int a) {
    if (blockIdx.x == 0) {
        grid_dependency_wait();
        if (threadIdx.x < 32) advance_clock(d, a);
        launch_dependents();
        return;
    }
    bulk_body<ST, MODEL, GAL, FORCE, OPEN, FIRST, true>(d, a, int(blockIdx.x) - 1, false);
}

template <int ST, int MODEL, bool GAL, bool FORCE, bool OPEN>
__global__ void __launch_bounds__(MAX_BLOCK, MIN_BLOCKS) k_bulk(const StepArgs d, const int a) {
    bulk_block<ST, MODEL, GAL, FORCE, OPEN>(d, a);
}

// The regularised step without a body force (every open vessel) in blocks of at most 128 threads, compiled for as many
// of them per SM as hide the pulls' latency best: 8 at 64 registers in FP32 (artery 79.6 us a step against 80.5 for 9 at
// 56, 190 k-node artery 9.9 against 10.6), 9 at 56 in the 16-bit formats (67.4 against 67.6). One build with and without
// open ends: the FP32 one without their reduction spills 8 bytes (this one none), 18.2 us a step on the pipe against 17.9.
//
// FIRST: a step reads a population once, writes it to the other buffer, and a step later that copy is what is read. While
// both buffers fit the L2, lines that have been read should go before lines just written. Loads marked evict-first take
// the 347 k-node FP32 pipe (75 MB) from 20.4 to 18.1 us a step, 522 k nodes (113 MB) from 29.4 to 27.2, 678 k nodes in FP16
// (73 MB) from 31.7 to 27.5. The qualifier names the L1; that the gain is the L2's shows in DRAM reads (pipe: 12.8 MB a
// step without it, 1.3 with it) and in that an L2 policy does the same (18.0 us; L1::no_allocate 17.9). Past the L2 they
// lose the sectors that neighbouring warps share: 678 k nodes in FP32 (146 MB) 36.4 to 37.5, the artery (322 MB) 79.6 to
// 86.1. So the line is the L2's size, of one lattice: several that run at once share it, which costs the concurrent
// schedules 1-2 % on two streams and 3-6 % on four (four FP32 vessels of 300-340 k nodes 73.7 to 78.3 us a step), while one
// after the other they gain as above (68.9 to 62.2).
constexpr int DENSE_BLOCK = 128;
constexpr int dense_blocks(int st) { return st == CS_STORE_F32 ? 8 : 9; }

template <int ST, bool GAL, bool FIRST>
__global__ void __launch_bounds__(DENSE_BLOCK, dense_blocks(ST)) k_bulk_dense(const StepArgs d, const int a) {
    bulk_block<ST, CS_MODEL_REGULARISED, GAL, false, true, FIRST>(d, a);
}

// ---- 3. outlet resistances ----------------------------------------------------------------------------------------
constexpr int BC_THREADS = 512;

// simulate.py:76-82 in FP64 (one block of BC_THREADS threads); the drive of this step was stored by the bulk kernel's
// clock block. Q_k = the flux blocks' partial sums: a thread adds its rows (all open ends of a row lie side by side), warps
// reduce by shuffles and the warps' sums are added in order (the same order at every step and run). The kernel is pure
// latency on the path from one step to the next: launched programmatically, it reads fb_list before the bulk kernel has
// ended and lets the next boundary kernel become resident while it works. A tree over all threads per open end and an
// ordinary launch took 8.3 us on 1487 rows, a quarter of a step of 190 k nodes.
__device__ __forceinline__ void bc_body(const StepArgs& d) {
    __shared__ double s_w[BC_THREADS / 32][MAX_OPEN];
    constexpr int AHEAD = 4;
    launch_dependents();
    int32_t row[AHEAD];
#pragma unroll
    for (int r = 0; r < AHEAD; ++r) {
        const int j = threadIdx.x + r * BC_THREADS;
        row[r] = j < d.n_fb ? __ldg(d.fb_list + j) : -1;
    }
    double acc[MAX_OPEN];
#pragma unroll
    for (int k = 0; k < MAX_OPEN; ++k) acc[k] = 0.0;
    grid_dependency_wait();
#pragma unroll
    for (int k = 0; k < MAX_OPEN; ++k) {
        if (k >= d.n_open) break;
        double v[AHEAD];
#pragma unroll
        for (int r = 0; r < AHEAD; ++r) v[r] = row[r] >= 0 ? d.q_part[int64_t(row[r]) * MAX_OPEN + k] : 0.0;
#pragma unroll
        for (int r = 0; r < AHEAD; ++r) acc[k] += v[r];
    }
    for (int j = threadIdx.x + AHEAD * BC_THREADS; j < d.n_fb; j += BC_THREADS) {
        const double* q = d.q_part + int64_t(__ldg(d.fb_list + j)) * MAX_OPEN;
#pragma unroll
        for (int k = 0; k < MAX_OPEN; ++k)
            if (k < d.n_open) acc[k] += q[k];
    }
#pragma unroll
    for (int k = 0; k < MAX_OPEN; ++k) {
        if (k >= d.n_open) break;
        double x = acc[k];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5][k] = x;
    }
    __syncthreads();
    const int k = threadIdx.x;
    if (k >= d.n_open) return;
    double qk = 0.0;
#pragma unroll
    for (int w = 0; w < BC_THREADS / 32; ++w) qk += s_w[w][k];
    d.q_last[k] = qk;
    double pk;
    if (k == 0) {
        const float dv = *d.drive;
        d.p_out[0] = dv;
        pk = double(dv);
    } else {
        pk = d.p_out64[k] + d.alpha * (double(d.r_out[k]) * qk - d.pref - d.p_out64[k]);
        d.p_out[k] = float(pk);
    }
    d.p_out64[k] = pk;
    if (d.beat_acc) {
        // running sums for the beat means of the open ends' pressure and flow (one thread per open end)
        d.beat_acc[k] += pk;
        d.beat_acc[d.n_open + k] += qk;
        if (k == 0) d.beat_acc[2 * d.n_open] += 1.0;
    }
}

__global__ void __launch_bounds__(BC_THREADS) k_bc(const StepArgs d, const int) { bc_body(d); }

using StepFn = void (*)(const StepArgs, const int);

template <int ST, bool GAL, bool OPEN>
StepFn pick_collision(int model, bool force, int block, bool first) {
    if (model != CS_MODEL_REGULARISED)
        return force ? k_bulk<ST, CS_MODEL_TRT, GAL, true, OPEN> : k_bulk<ST, CS_MODEL_TRT, GAL, false, OPEN>;
    if (force) return k_bulk<ST, CS_MODEL_REGULARISED, GAL, true, OPEN>;
    if (block <= DENSE_BLOCK) return first ? k_bulk_dense<ST, GAL, true> : k_bulk_dense<ST, GAL, false>;
    return k_bulk<ST, CS_MODEL_REGULARISED, GAL, false, OPEN>;
}

// L2 bytes of the current device (0 if it cannot be asked: no kernel then assumes that anything fits).
int64_t l2_bytes() {
    int dev = 0, bytes = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&bytes, cudaDevAttrL2CacheSize, dev) != cudaSuccess) return 0;
    return bytes;
}

template <int ST>
StepFn pick_model(const StepArgs& d) {
    const bool force = d.force[0] != 0.0f || d.force[1] != 0.0f || d.force[2] != 0.0f;
    const int block = d.block ? d.block : MAX_BLOCK;
    const bool first = 2 * int64_t(Q) * d.fstride * (ST == CS_STORE_F32 ? 4 : 2) <= l2_bytes();
    if (d.n_open > 0)
        return d.gal ? pick_collision<ST, true, true>(d.model, force, block, first)
                     : pick_collision<ST, false, true>(d.model, force, block, first);
    return d.gal ? pick_collision<ST, true, false>(d.model, force, block, first)
                 : pick_collision<ST, false, false>(d.model, force, block, first);
}

StepFn pick_bulk(const StepArgs& d) {
    switch (d.storage) {
        case CS_STORE_F16: return pick_model<CS_STORE_F16>(d);
        case CS_STORE_BF16: return pick_model<CS_STORE_BF16>(d);
        default: return pick_model<CS_STORE_F32>(d);
    }
}

StepFn pick_boundary(const StepArgs& d, bool start) {
    switch (d.storage) {
        case CS_STORE_F16: return start ? k_boundary<CS_STORE_F16, true> : k_boundary<CS_STORE_F16, false>;
        case CS_STORE_BF16: return start ? k_boundary<CS_STORE_BF16, true> : k_boundary<CS_STORE_BF16, false>;
        default: return start ? k_boundary<CS_STORE_F32, true> : k_boundary<CS_STORE_F32, false>;
    }
}

int validate(const cs_step_desc* d, const cs_step_layout* layout) {
    if (!d) return fail(CS_ERR_ARG, "cs_step: null descriptor");
    if (d->n < 0 || d->n >= (int64_t(1) << 30)) return fail(CS_ERR_SIZE, "cs_step: n = %lld", (long long)d->n);
    if (d->gmax < 0 || d->npad != d->n + d->gmax || int64_t(Q) * d->npad >= (int64_t(1) << 31))
        return fail(CS_ERR_SIZE, "cs_step: npad %lld must be n + gmax with 27 * npad < 2^31", (long long)d->npad);
    const int64_t fstride = layout && layout->fstride ? layout->fstride : d->npad;
    const int64_t vstride = layout && layout->vstride ? layout->vstride : d->n;
    if (fstride < d->npad || fstride > INT32_MAX / Q || vstride < d->n || vstride > INT32_MAX / 3)
        return fail(CS_ERR_SIZE, "cs_step: row strides %lld (npad %lld; 27 rows below 2^31) and %lld (n %lld)",
                    (long long)fstride, (long long)d->npad, (long long)vstride, (long long)d->n);
    if (d->gblock[0] != 0) return fail(CS_ERR_ARG, "cs_step: gblock[0] = %d", d->gblock[0]);
    for (int i = 0; i < Q; ++i) {
        const int64_t w = int64_t(d->gblock[i + 1]) - d->gblock[i];
        if (w < 0 || w * B_THREADS > std::max<int64_t>(d->gmax, 0) + B_THREADS - 1)
            return fail(CS_ERR_ARG, "cs_step: gblock[%d..%d] = %d..%d for gmax %lld", i, i + 1, d->gblock[i],
                        d->gblock[i + 1], (long long)d->gmax);
    }
    if (d->storage < 0 || d->storage > 2) return fail(CS_ERR_ARG, "cs_step: storage %d", d->storage);
    if (d->model != CS_MODEL_TRT && d->model != CS_MODEL_REGULARISED) return fail(CS_ERR_ARG, "cs_step: model %d", d->model);
    if (d->block != 0 && (d->block < 32 || d->block > MAX_BLOCK || d->block % 32))
        return fail(CS_ERR_ARG, "cs_step: block %d (32..%d, multiple of 32)", d->block, MAX_BLOCK);
    if (d->period < 1 || d->nh < 0 || d->ramp < 0) return fail(CS_ERR_ARG, "cs_step: period %d nh %d ramp %d", d->period, d->nh, d->ramp);
    if (!d->tick || !d->drive || !d->coef || !d->p_out || d->n_out < 1)
        return fail(CS_ERR_ARG, "cs_step: null clock / outlet state");
    if (d->n > 0 && (!d->f[0] || !d->f[1] || !d->vel[0] || !d->vel[1] || !d->rho || !d->lcode || !d->uin || !d->om))
        return fail(CS_ERR_ARG, "cs_step: null lattice buffer");
    if (d->gmax > 0 && (!d->gnode || !d->ginfo || !d->gq)) return fail(CS_ERR_ARG, "cs_step: null ghost table");
    if (d->n_open < 0 || d->n_open > MAX_OPEN || d->n_open > d->n_out)
        return fail(CS_ERR_ARG, "cs_step: n_open %d (at most %d and at most n_out %d)", d->n_open, MAX_OPEN, d->n_out);
    if (d->n_open > 0 && (!d->flux_block || !d->q_part || !d->q_last || !d->p_out64 || !d->r_out ||
                          d->n_fb < 0 || (d->n_fb > 0 && !d->fb_list) ||
                          (d->n_flux > 0 && (!d->flux_idx || !d->flux_w || !d->flux_slot))))
        return fail(CS_ERR_ARG, "cs_step: null flux buffer");
    return CS_OK;
}

// One division of the SM's memory between L1 and shared memory for every kernel of a single lattice's step. By default the driver picks
// it by each kernel's own shared memory (none in the boundary kernel, 9 blocks x 4.6 KB in the bulk kernel), and an SM
// that changes it between two kernels drains first: the next kernel's blocks then do not start under the last one's
// (20 k-node cylinder 9.6 us a step, with one division 5.0; tilted pipe of 75 k nodes 12.6 and 8.4). 28 % is the 64 KB
// that nine blocks of the bulk kernel need; half of it leaves room for seven (artery 88.6 against 86.5 us). The batched
// kernels keep the driver's choice: persistent grids that start under one another took 68.9 us a step against 54.1 on four
// FP32 vessels of 100-400 k nodes, 71.0 against 60.0 on five of 150-250 k, and grids of a block an item the same.
constexpr int CARVEOUT = 28;

int set_carveout(const void* fn) {
    struct Set {
        int dev;
        const void* fn;
    };
    static std::mutex m;
    static Set done[512];               // what has been set; past that the attribute is set again at each call
    static int n = 0;
    int dev = 0;
    CS_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(m);
    for (int k = 0; k < n; ++k)
        if (done[k].dev == dev && done[k].fn == fn) return CS_OK;
    CS_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, CARVEOUT));
    if (n < 512) done[n++] = Set{dev, fn};
    return CS_OK;
}

// Launch with programmatic stream serialization, so the kernel's static prologue overlaps the previous kernel.
int launch_pdl(StepFn fn, dim3 grid, dim3 block, cudaStream_t st, const StepArgs& d, int a) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, fn, d, a);
    if (e != cudaSuccess) return fail(CS_ERR_CUDA, "launch of a step kernel failed: %s", cudaGetErrorString(e));
    return CS_OK;
}

int launch_steps(const StepArgs& args, int a, int steps, cudaStream_t st) {
    const StepArgs* d = &args;
    const int block = d->block ? d->block : MAX_BLOCK;
    const unsigned grid = unsigned(d->n > 0 ? ceil_div(d->n, block) : 0);
    const dim3 bgrid(unsigned(boundary_items(*d)));
    StepFn bulk = pick_bulk(*d);
    StepFn bound = pick_boundary(*d, false), bound_start = pick_boundary(*d, true);
    for (StepFn fn : {bulk, bound, bound_start, StepFn(k_bc), StepFn(k_clock)}) {
        const int rc = set_carveout(reinterpret_cast<const void*>(fn));
        if (rc != CS_OK) return rc;
    }
    for (int s = 0; s < steps; ++s) {
        const bool start = s == 0 || !d->drive2;
        int rc = CS_OK;
        if (grid == 0) {
            k_clock<<<1, 32, 0, st>>>(*d, a);
            k_clock_only<<<1, 32, 0, st>>>(*d, a);
            CS_CHECK_LAUNCH("k_clock_only");
        } else {
            if (d->gmax > 0) rc = launch_pdl(start ? bound_start : bound, bgrid, dim3(B_THREADS), st, *d, a);
            else if (start) rc = launch_pdl(k_clock, dim3(1), dim3(32), st, *d, a);
            if (rc != CS_OK) return rc;
            rc = launch_pdl(bulk, dim3(grid + 1), dim3(block), st, *d, a);
            if (rc != CS_OK) return rc;
        }
        if (d->n_open > 0) {
            rc = launch_pdl(k_bc, dim3(1), dim3(BC_THREADS), st, *d, a);
            if (rc != CS_OK) return rc;
        }
        a = 1 - a;
    }
    return CS_OK;
}

__global__ void k_flux_blocks(const int32_t* __restrict__ idx, int64_t n_flux, int block, int32_t* __restrict__ out,
                              int64_t n_blocks) {
    const int64_t b = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (b > n_blocks) return;
    const int64_t key = b * block;
    int64_t lo = 0, hi = n_flux;  // first entry with idx >= key
    while (lo < hi) {
        const int64_t mid = (lo + hi) / 2;
        if (int64_t(idx[mid]) < key) lo = mid + 1; else hi = mid;
    }
    out[b] = int32_t(lo);
}

}  // namespace
}  // namespace cs

using namespace cs;

extern "C" int cs_flux_blocks(const int32_t* flux_idx, int64_t n_flux, int64_t n, int32_t block, int32_t* out,
                              void* stream) {
    if (n < 0 || n_flux < 0 || block < 32 || block > MAX_BLOCK || !out || (n_flux > 0 && !flux_idx))
        return fail(CS_ERR_ARG, "cs_flux_blocks: bad arguments");
    const int64_t nb = n > 0 ? ceil_div(n, block) : 1;
    k_flux_blocks<<<unsigned(ceil_div(nb + 1, 256)), 256, 0, as_stream(stream)>>>(flux_idx, n_flux, block, out, nb);
    CS_CHECK_LAUNCH("k_flux_blocks");
    return CS_OK;
}

extern "C" int cs_step_ex(const cs_step_desc* d, const cs_step_layout* layout, int32_t a, int32_t steps, void* stream) {
    int rc = validate(d, layout);
    if (rc != CS_OK) return rc;
    if ((a != 0 && a != 1) || steps < 0) return fail(CS_ERR_ARG, "cs_step: a %d steps %d", a, steps);
    return launch_steps(StepArgs(*d, layout), a, steps, as_stream(stream));
}

extern "C" int cs_step(const cs_step_desc* d, int32_t a, int32_t steps, void* stream) {
    return cs_step_ex(d, nullptr, a, steps, stream);
}

namespace {
struct Graph {
    cudaGraphExec_t exec;
};
}  // namespace

extern "C" int cs_graph_capture_ex(const cs_step_desc* d, const cs_step_layout* layout, int32_t a, int32_t steps,
                                   void* stream, void** graph) {
    int rc = validate(d, layout);
    if (rc != CS_OK) return rc;
    if ((a != 0 && a != 1) || steps < 1 || !graph) return fail(CS_ERR_ARG, "cs_graph_capture: a %d steps %d", a, steps);
    cudaStream_t st = as_stream(stream);
    if (st == nullptr) return fail(CS_ERR_ARG, "cs_graph_capture: the legacy default stream cannot be captured");
    CS_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    rc = launch_steps(StepArgs(*d, layout), a, steps, st);
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(st, &g);
    if (rc != CS_OK) {
        if (g) cudaGraphDestroy(g);
        return rc;
    }
    if (e != cudaSuccess) return fail(CS_ERR_CUDA, "cudaStreamEndCapture: %s", cudaGetErrorString(e));
    cudaGraphExec_t ex = nullptr;
    e = cudaGraphInstantiate(&ex, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return fail(CS_ERR_CUDA, "cudaGraphInstantiate: %s", cudaGetErrorString(e));
    *graph = new Graph{ex};
    return CS_OK;
}

extern "C" int cs_graph_capture(const cs_step_desc* d, int32_t a, int32_t steps, void* stream, void** graph) {
    return cs_graph_capture_ex(d, nullptr, a, steps, stream, graph);
}

extern "C" int cs_graph_launch(void* graph, void* stream) {
    if (!graph) return fail(CS_ERR_ARG, "cs_graph_launch: null graph");
    CS_CUDA(cudaGraphLaunch(static_cast<Graph*>(graph)->exec, as_stream(stream)));
    return CS_OK;
}

extern "C" int cs_graph_destroy(void* graph) {
    if (!graph) return CS_OK;
    Graph* g = static_cast<Graph*>(graph);
    cudaError_t e = cudaGraphExecDestroy(g->exec);
    delete g;
    if (e != cudaSuccess) return fail(CS_ERR_CUDA, "cudaGraphExecDestroy: %s", cudaGetErrorString(e));
    return CS_OK;
}

extern "C" int cs_step_check(const cs_step_desc* d) { return validate(d, nullptr); }

// ---- batched step -------------------------------------------------------------------------------------------------
// The instances' descriptors travel in the kernels' parameter space (constant bank), CS_BATCH_GROUP instances per
// launch: every block reads the descriptor of the instance it works on there, as the single-lattice kernels read
// theirs, instead of staging it in shared memory (which costs registers and spills in the collision).
namespace cs {
namespace {

struct BatchGroup {
    int32_t n_inst, bulk_items, bnd_items, pad_;
    int32_t* counter;
    int32_t bulk_prefix[CS_BATCH_GROUP + 1];
    int32_t bnd_prefix[CS_BATCH_GROUP + 1];
    int32_t parity[CS_BATCH_GROUP];
    StepArgs d[CS_BATCH_GROUP];
};
static_assert(sizeof(BatchGroup) < 32000, "batched kernel parameters exceed the 32 KB limit");

// Largest i in [0, n) with prefix[i] <= item.
__device__ __forceinline__ int find_instance(const int32_t* prefix, int n, int item) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (prefix[mid] <= item) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// A persistent block's share of the boundary work list: a contiguous range of items.
struct ItemRange {
    int lo, hi;
    __device__ ItemRange(int items) {
        const int per = items / int(gridDim.x), rem = items % int(gridDim.x), bx = int(blockIdx.x);
        lo = bx * per + min(bx, rem);
        hi = lo + per + (bx < rem ? 1 : 0);
    }
};

// Instance of each item for a block walking its items in increasing order.
struct InstanceCursor {
    const int32_t* prefix;
    int n, inst = -1, first = 0, end = 0;
    __device__ InstanceCursor(const int32_t* prefix_, int n_) : prefix(prefix_), n(n_) {}
    __device__ __forceinline__ int next(int item) {
        if (item >= end) {
            inst = inst < 0 ? find_instance(prefix, n, item) : inst + 1;
            while (prefix[inst + 1] <= item) ++inst;
            first = prefix[inst];
            end = prefix[inst + 1];
        }
        return item - first;
    }
};

template <int ST, bool START>
__global__ void __launch_bounds__(B_THREADS) k_boundary_batch(const __grid_constant__ BatchGroup g, const int a) {
    const ItemRange r(g.bnd_items);
    InstanceCursor cur(g.bnd_prefix, g.n_inst);
    for (int item = r.lo; item < r.hi; ++item) {
        const int local = cur.next(item);
        boundary_item<ST, START>(g.d[cur.inst], a ^ g.parity[cur.inst], local);
    }
    // the previous bulk kernel has finished (boundary_body waited for it) and the next one takes no item before
    // this kernel ends: reset its work counter
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        grid_dependency_wait();
        *g.counter = 0;
    }
}

// Bulk items are handed out dynamically: block x starts with item x, then takes the next unclaimed item from a
// counter (reset by the boundary kernel each step), so that blocks finishing cheap items (few boundary rows) take
// more of them. The claim for the following item is issued at the start of the current one and lands while it
// runs. Which block updates which item does not change any result (each item writes its own nodes and its own row
// of flux partial sums).
template <int ST, int MODEL, bool GAL, bool FORCE, bool OPEN>
__global__ void __launch_bounds__(MAX_BLOCK, MIN_BLOCKS) k_bulk_batch(const __grid_constant__ BatchGroup g,
                                                                      const int a) {
    __shared__ int s_item[2];
    InstanceCursor cur(g.bulk_prefix, g.n_inst);
    int item = blockIdx.x, buf = 0;
    bool first = true;
    while (item < g.bulk_items) {
        const int local = cur.next(item);
        int claim = 0;
        if (!first && threadIdx.x == 0) claim = atomicAdd(g.counter, 1);
        bulk_body<ST, MODEL, GAL, FORCE, OPEN>(g.d[cur.inst], a ^ g.parity[cur.inst], local, local == 0);
        if (first && threadIdx.x == 0) claim = atomicAdd(g.counter, 1);   // after the wait inside bulk_body
        first = false;
        if (threadIdx.x == 0) s_item[buf] = int(gridDim.x) + claim;
        __syncthreads();                        // also: the flux partial sums reuse shared memory
        item = s_item[buf];
        buf ^= 1;
    }
}

// One block per bulk item, no loop and no claims (grid_bulk = 0): the regularised step without body force in blocks
// of at most 128 threads, compiled for 9 blocks per SM in every format (FP32 too: 55.4 us a step against 57.6 for 8 on four
// vessels of 100-400 k nodes), which the persistent loop's state does not leave registers for (at 56 it spills and loses
// 9 %). The block finds its instance by a binary search over the item prefix in the parameters.
template <int ST, bool GAL, bool OPEN>
__global__ void __launch_bounds__(DENSE_BLOCK, 9) k_bulk_batch_dense(const __grid_constant__ BatchGroup g,
                                                                                  const int a) {
    const int item = int(blockIdx.x);
    const int inst = find_instance(g.bulk_prefix, g.n_inst, item);
    const int local = item - g.bulk_prefix[inst];
    bulk_body<ST, CS_MODEL_REGULARISED, GAL, false, OPEN>(g.d[inst], a ^ g.parity[inst], local, local == 0);
}

// The instances without nodes, whose clock no bulk block advances.
__global__ void __launch_bounds__(32) k_clock_empty_batch(const __grid_constant__ BatchGroup g, const int a) {
    if (g.d[blockIdx.x].n == 0) advance_clock(g.d[blockIdx.x], a ^ g.parity[blockIdx.x]);
}

__global__ void __launch_bounds__(BC_THREADS) k_bc_batch(const __grid_constant__ BatchGroup g, const int) {
    const StepArgs& d = g.d[blockIdx.x];
    if (d.n_open > 0) {
        bc_body(d);
    } else {
        grid_dependency_wait();     // the next boundary kernel waits for this one, and through it for the bulk kernel
    }
}

using BatchFn = void (*)(const BatchGroup, const int);

template <int ST, bool GAL, bool OPEN>
BatchFn pick_batch_collision(int model, bool force, bool dense) {
    if (model != CS_MODEL_REGULARISED)
        return force ? k_bulk_batch<ST, CS_MODEL_TRT, GAL, true, OPEN> : k_bulk_batch<ST, CS_MODEL_TRT, GAL, false, OPEN>;
    if (force) return k_bulk_batch<ST, CS_MODEL_REGULARISED, GAL, true, OPEN>;
    return dense ? k_bulk_batch_dense<ST, GAL, OPEN> : k_bulk_batch<ST, CS_MODEL_REGULARISED, GAL, false, OPEN>;
}

template <int ST>
BatchFn pick_batch_model(const cs_batch_desc& b, bool dense) {
    const bool force = b.force != 0;
    if (b.any_open)
        return b.gal ? pick_batch_collision<ST, true, true>(b.model, force, dense)
                     : pick_batch_collision<ST, false, true>(b.model, force, dense);
    return b.gal ? pick_batch_collision<ST, true, false>(b.model, force, dense)
                 : pick_batch_collision<ST, false, false>(b.model, force, dense);
}

// Also for instances without boundary links: their items are empty, but the first step's evaluate their drive.
BatchFn pick_batch_boundary(int storage, bool start) {
    switch (storage) {
        case CS_STORE_F16: return start ? k_boundary_batch<CS_STORE_F16, true> : k_boundary_batch<CS_STORE_F16, false>;
        case CS_STORE_BF16: return start ? k_boundary_batch<CS_STORE_BF16, true> : k_boundary_batch<CS_STORE_BF16, false>;
        default: return start ? k_boundary_batch<CS_STORE_F32, true> : k_boundary_batch<CS_STORE_F32, false>;
    }
}

int validate_batch(const cs_batch_desc* b, const cs_step_layout* layouts) {
    if (!b) return fail(CS_ERR_ARG, "cs_batch_step: null descriptor");
    if (b->n_inst < 1 || !b->descs || !b->parity || !b->counter)
        return fail(CS_ERR_ARG, "cs_batch_step: %d instances or null tables", b->n_inst);
    if (b->storage < 0 || b->storage > 2 || (b->model != CS_MODEL_TRT && b->model != CS_MODEL_REGULARISED))
        return fail(CS_ERR_ARG, "cs_batch_step: storage %d model %d", b->storage, b->model);
    if (b->block < 32 || b->block > MAX_BLOCK || b->block % 32)
        return fail(CS_ERR_ARG, "cs_batch_step: block %d (32..%d, multiple of 32)", b->block, MAX_BLOCK);
    if (b->grid_bulk < 0 || b->grid_bnd < 0)
        return fail(CS_ERR_ARG, "cs_batch_step: grid sizes %d / %d", b->grid_bulk, b->grid_bnd);
    int64_t items = 0;
    for (int i = 0; i < b->n_inst; ++i) {
        const cs_step_desc& d = b->descs[i];
        const int rc = validate(&d, layouts ? layouts + i : nullptr);
        if (rc != CS_OK) return rc;
        if (d.storage != b->storage || d.model != b->model || d.gal != b->gal || d.block != b->block)
            return fail(CS_ERR_ARG, "cs_batch_step: instance %d differs from the batch in storage, model, Galilean "
                                    "setting or block size", i);
        if ((d.force[0] != 0.f || d.force[1] != 0.f || d.force[2] != 0.f) && !b->force)
            return fail(CS_ERR_ARG, "cs_batch_step: instance %d has a body force but the batch has force = 0", i);
        if (d.n_open > 0 && !b->any_open)
            return fail(CS_ERR_ARG, "cs_batch_step: instance %d has open ends but the batch has any_open = 0", i);
        if (b->parity[i] != 0 && b->parity[i] != 1)
            return fail(CS_ERR_ARG, "cs_batch_step: parity[%d] = %d", i, b->parity[i]);
        items += ceil_div(d.n, int64_t(b->block)) + boundary_items(d);
    }
    if (items > INT32_MAX - int64_t(MAX_BLOCK) * 2048)
        return fail(CS_ERR_SIZE, "cs_batch_step: %lld work items", (long long)items);
    return CS_OK;
}

// The launch groups of a batch: CS_BATCH_GROUP instances each, work items counted per instance.
std::vector<BatchGroup> make_groups(const cs_batch_desc* b, const cs_step_layout* layouts) {
    std::vector<BatchGroup> gs;
    for (int i0 = 0; i0 < b->n_inst; i0 += CS_BATCH_GROUP) {
        BatchGroup g;
        std::memset(&g, 0, sizeof(g));
        g.n_inst = std::min(CS_BATCH_GROUP, b->n_inst - i0);
        g.counter = b->counter + i0 / CS_BATCH_GROUP;
        int64_t bulk = 0, bnd = 0;
        for (int k = 0; k < g.n_inst; ++k) {
            const StepArgs d(b->descs[i0 + k], layouts ? layouts + i0 + k : nullptr);
            g.d[k] = d;
            g.parity[k] = b->parity[i0 + k];
            g.bulk_prefix[k] = int32_t(bulk);
            g.bnd_prefix[k] = int32_t(bnd);
            bulk += ceil_div(d.n, int64_t(b->block));
            bnd += boundary_items(d);
        }
        g.bulk_prefix[g.n_inst] = int32_t(bulk);
        g.bnd_prefix[g.n_inst] = int32_t(bnd);
        g.bulk_items = int32_t(bulk);
        g.bnd_items = int32_t(bnd);
        gs.push_back(g);
    }
    return gs;
}

int launch_batch_pdl(BatchFn fn, unsigned grid, unsigned block, cudaStream_t st, const BatchGroup& g, int a) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, fn, g, a);
    if (e != cudaSuccess) return fail(CS_ERR_CUDA, "launch of a batched step kernel failed: %s", cudaGetErrorString(e));
    return CS_OK;
}

int launch_batch(const cs_batch_desc* b, const cs_step_layout* layouts, int a, int steps, cudaStream_t st) {
    const std::vector<BatchGroup> gs = make_groups(b, layouts);
    const bool dense = b->grid_bulk == 0 && b->block <= DENSE_BLOCK;     // one block per item: k_bulk_batch_dense
    BatchFn bulk = b->storage == CS_STORE_F16    ? pick_batch_model<CS_STORE_F16>(*b, dense)
                   : b->storage == CS_STORE_BF16 ? pick_batch_model<CS_STORE_BF16>(*b, dense)
                                                 : pick_batch_model<CS_STORE_F32>(*b, dense);
    BatchFn bound = pick_batch_boundary(b->storage, false), bound_start = pick_batch_boundary(b->storage, true);
    bool empty = false, every = !layouts;           // every: some instance has no place for the next step's drive
    for (int i = 0; i < b->n_inst; ++i) {
        empty = empty || b->descs[i].n == 0;
        every = every || !layouts[i].drive2;
    }
    for (int s = 0; s < steps; ++s) {
        for (const BatchGroup& g : gs) {
            const unsigned gb = unsigned(b->grid_bnd > 0 ? std::min(b->grid_bnd, g.bnd_items) : g.bnd_items);
            const int rc = launch_batch_pdl(s == 0 || every ? bound_start : bound, gb, B_THREADS, st, g, a);
            if (rc != CS_OK) return rc;
        }
        if (empty)
            for (const BatchGroup& g : gs) {
                k_clock_empty_batch<<<unsigned(g.n_inst), 32, 0, st>>>(g, a);
                CS_CHECK_LAUNCH("k_clock_empty_batch");
            }
        for (const BatchGroup& g : gs) {
            const unsigned gk = unsigned(b->grid_bulk > 0 ? std::min(b->grid_bulk, g.bulk_items) : g.bulk_items);
            if (gk == 0) continue;
            const int rc = launch_batch_pdl(bulk, gk, unsigned(b->block), st, g, a);
            if (rc != CS_OK) return rc;
        }
        if (b->any_open) {
            for (const BatchGroup& g : gs) {
                const int rc = launch_batch_pdl(k_bc_batch, unsigned(g.n_inst), BC_THREADS, st, g, a);
                if (rc != CS_OK) return rc;
            }
        }
        a = 1 - a;
    }
    return CS_OK;
}

}  // namespace
}  // namespace cs

extern "C" int cs_batch_step_ex(const cs_batch_desc* b, const cs_step_layout* layouts, int32_t a, int32_t steps,
                                void* stream) {
    int rc = validate_batch(b, layouts);
    if (rc != CS_OK) return rc;
    if ((a != 0 && a != 1) || steps < 0) return fail(CS_ERR_ARG, "cs_batch_step: a %d steps %d", a, steps);
    return launch_batch(b, layouts, a, steps, as_stream(stream));
}

extern "C" int cs_batch_step(const cs_batch_desc* b, int32_t a, int32_t steps, void* stream) {
    return cs_batch_step_ex(b, nullptr, a, steps, stream);
}

extern "C" int cs_batch_graph_capture_ex(const cs_batch_desc* b, const cs_step_layout* layouts, int32_t a, int32_t steps,
                                         void* stream, void** graph) {
    int rc = validate_batch(b, layouts);
    if (rc != CS_OK) return rc;
    if ((a != 0 && a != 1) || steps < 1 || !graph)
        return fail(CS_ERR_ARG, "cs_batch_graph_capture: a %d steps %d", a, steps);
    cudaStream_t st = as_stream(stream);
    if (st == nullptr) return fail(CS_ERR_ARG, "cs_batch_graph_capture: the legacy default stream cannot be captured");
    CS_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    rc = launch_batch(b, layouts, a, steps, st);
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(st, &g);
    if (rc != CS_OK) {
        if (g) cudaGraphDestroy(g);
        return rc;
    }
    if (e != cudaSuccess) return fail(CS_ERR_CUDA, "cudaStreamEndCapture: %s", cudaGetErrorString(e));
    cudaGraphExec_t ex = nullptr;
    e = cudaGraphInstantiate(&ex, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return fail(CS_ERR_CUDA, "cudaGraphInstantiate: %s", cudaGetErrorString(e));
    *graph = new Graph{ex};
    return CS_OK;
}

extern "C" int cs_batch_graph_capture(const cs_batch_desc* b, int32_t a, int32_t steps, void* stream, void** graph) {
    return cs_batch_graph_capture_ex(b, nullptr, a, steps, stream, graph);
}
