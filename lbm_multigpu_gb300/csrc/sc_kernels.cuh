/*
 * sc_kernels.cuh -- the stream-collide kernels, templated on the storage
 * format S and on the population layout LAY (Level::blocked: structure of
 * arrays, or blocks of 32 nodes).  sc_instance.cu is compiled once per format
 * and layout, so that the sets build in parallel.
 *
 * k_stream_collide is the hot kernel: one thread per lattice node, a warp
 * spans 32 consecutive x of one row, so every population load and store of a
 * warp touches one aligned run of 32 elements (x-shifted pulls straddle two
 * runs, the neighbour warp's part is then an L2 hit).  It fuses, per node and
 * per step, what the reference spreads over update_inn/update_top/update_bot
 * (LR7:1127-1628):
 *   pull streaming (LR7:1445-1491) with the z halo planes replaced by a
 *   periodic index wrap inside one domain,
 *   full-way bounce-back (LR7:1493-1526), or half-way bounce-back through
 *   per-node link masks,
 *   inlet/outlet rebuilds (LR7:1531-1561), the moving lid,
 *   MRT/BGK collision with Smagorinsky (LR7:583-711, DI3:599-832),
 *   running statistics (LR7:1567-1584),
 *   the coarse-moment export for the refinement (LR7:1590-1605).
 * The momentum exchange on the body (LR7:1607-1626) is summed by a separate
 * kernel, k_force_list, from the same populations.
 */
#pragma once

#include <algorithm>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "d3q19.cuh"
#include "lbm_kernels.cuh"
#include "sgs_infer.cuh"

namespace lbm {

/* ---- storage formats: FP32, FP64, and FP16/BF16 holding f - off with FP32
 * math; off is the equilibrium at the level's reference velocity (Level::off),
 * so the stored numbers are small deviations and keep their relative precision.
 * ld / st convert between stored values and populations; ldr / str / st2 move
 * stored values as they are (st2: two adjacent elements with one store). */
template <class S> struct Fmt;
template <> struct Fmt<float> {
    using T = float;
    static __device__ __forceinline__ float ldr(const float* p) { return __ldg(p); }
    static __device__ __forceinline__ void str(float* p, float v) { *p = v; }
    static __device__ __forceinline__ void st2(float* p, float a, float b) {
        *reinterpret_cast<float2*>(p) = make_float2(a, b);
    }
    static __device__ __forceinline__ float ld(const float* p, float) { return __ldg(p); }
    static __device__ __forceinline__ void st(float* p, float v, float) { *p = v; }
};
template <> struct Fmt<double> {
    using T = double;
    static __device__ __forceinline__ double ldr(const double* p) { return __ldg(p); }
    static __device__ __forceinline__ void str(double* p, double v) { *p = v; }
    static __device__ __forceinline__ void st2(double* p, double a, double b) {
        *reinterpret_cast<double2*>(p) = make_double2(a, b);
    }
    static __device__ __forceinline__ double ld(const double* p, float) { return __ldg(p); }
    static __device__ __forceinline__ void st(double* p, double v, float) { *p = v; }
};
template <> struct Fmt<__half> {
    using T = float;
    static __device__ __forceinline__ float ldr(const __half* p) { return __half2float(__ldg(p)); }
    static __device__ __forceinline__ void str(__half* p, float v) { *p = __float2half_rn(v); }
    static __device__ __forceinline__ void st2(__half* p, float a, float b) {
        *reinterpret_cast<__half2*>(p) = __floats2half2_rn(a, b);
    }
    static __device__ __forceinline__ float ld(const __half* p, float off) { return ldr(p) + off; }
    static __device__ __forceinline__ void st(__half* p, float v, float off) { str(p, v - off); }
};
template <> struct Fmt<__nv_bfloat16> {
    using T = float;
    static __device__ __forceinline__ float ldr(const __nv_bfloat16* p) { return __bfloat162float(__ldg(p)); }
    static __device__ __forceinline__ void str(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }
    static __device__ __forceinline__ void st2(__nv_bfloat16* p, float a, float b) {
        *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b);
    }
    static __device__ __forceinline__ float ld(const __nv_bfloat16* p, float off) { return ldr(p) + off; }
    static __device__ __forceinline__ void st(__nv_bfloat16* p, float v, float off) { str(p, v - off); }
};

/* Per-node addressing of the populations in the two layouts (Level):
 *   0 structure-of-arrays: q qstride + z plane + y pitch + x, each pull the
 *     sum of a population, a z, a y and an x term;
 *   1 blocked: a node's populations sit at compile-time offsets from its
 *     block position, pair_qoff(q) + 2 (x % 32) (population 0 at x % 32),
 *     and a neighbour's at a signed offset of a few elements in x and of
 *     19 pitch / 19 plane in y / z.  The pull of population q is then one
 *     base pointer plus the sum of at most three per-thread offsets plus an
 *     immediate, and the stores of a node one base pointer plus immediates.
 * pull(f, q): the population q arriving from x - c_q; own(f, q): this
 * node's population q; at(f, q, cn): population q of node cn (the
 * neighbours of the inlet / outlet rebuilds). */
template <int LAY> struct NodeIdx;
template <> struct NodeIdx<0> {
    unsigned zb[3], yb[3], xs[3], qs, self;
    __device__ __forceinline__ NodeIdx(const Level& L, unsigned xm, unsigned x, unsigned xp, unsigned ym, unsigned y,
                                       unsigned yp, unsigned zm, unsigned z, unsigned zp) {
        const unsigned plane = unsigned(L.plane), pitch = unsigned(L.pitch);
        zb[0] = zm * plane, zb[1] = z * plane, zb[2] = zp * plane;
        yb[0] = ym * pitch, yb[1] = y * pitch, yb[2] = yp * pitch;
        xs[0] = xm, xs[1] = x, xs[2] = xp;
        qs = unsigned(L.qstride);
        self = zb[1] + yb[1] + x;
    }
    template <class P> __device__ __forceinline__ P* pull(P* f, int q) const {
        return f + (unsigned(q) * qs + zb[1 - cz(q)] + yb[1 - cy(q)] + xs[1 - cx(q)]);
    }
    template <class P> __device__ __forceinline__ P* own(P* f, int q) const { return f + (unsigned(q) * qs + self); }
    template <class P> __device__ __forceinline__ P* at(P* f, int q, unsigned cn) const {
        return f + (unsigned(q) * qs + cn);
    }
};
template <> struct NodeIdx<1> {
    unsigned base, lane;
    int dx[3], dy[3], dz[3]; /* element offsets to the x-1 / x / x+1 (y, z) neighbours' pair slots */
    __device__ __forceinline__ NodeIdx(const Level& L, unsigned xm, unsigned x, unsigned xp, unsigned ym, unsigned y,
                                       unsigned yp, unsigned zm, unsigned z, unsigned zp) {
        const int ry = int(L.pitch) * 19, rz = int(L.plane) * 19;
        lane = x & 31u;
        const unsigned xq = (x >> 5) * BLOCK_ELEMS + 2u * lane;
        base = z * unsigned(rz) + y * unsigned(ry) + xq;
        dx[0] = int((xm >> 5) * BLOCK_ELEMS + 2u * (xm & 31u)) - int(xq);
        dx[1] = 0;
        dx[2] = int((xp >> 5) * BLOCK_ELEMS + 2u * (xp & 31u)) - int(xq);
        dy[0] = (int(ym) - int(y)) * ry, dy[1] = 0, dy[2] = (int(yp) - int(y)) * ry;
        dz[0] = (int(zm) - int(z)) * rz, dz[1] = 0, dz[2] = (int(zp) - int(z)) * rz;
    }
    /* the neighbour part is summed in 32 bits (the element index stays below
     * 2^31) and widened once; the population's constant offset is added to
     * the 64-bit pointer, where it becomes the load's immediate */
    template <class P> __device__ __forceinline__ P* pull(P* f, int q) const {
        if (q == 0) return f + (base - lane);
        return (f + (base + unsigned(dz[1 - cz(q)] + dy[1 - cy(q)] + dx[1 - cx(q)]))) + pair_qoff(q);
    }
    template <class P> __device__ __forceinline__ P* own(P* f, int q) const {
        return q == 0 ? f + (base - lane) : (f + base) + pair_qoff(q);
    }
    template <class P> __device__ __forceinline__ P* at(P* f, int q, unsigned cn) const {
        return f + ((cn >> 5) * BLOCK_ELEMS + pair_qoff(q) + (q == 0 ? 1u : 2u) * (cn & 31u));
    }
};

/* the 19 values g of this node into buffer f: raw stored values (RAW) or
 * populations with the format's offsets removed; the blocked layout writes
 * each opposite pair with one store */
template <class S, int LAY, bool RAW, class IDX>
__device__ __forceinline__ void store19(const Level& L, S* __restrict__ f, const IDX& n,
                                        const typename Fmt<S>::T g[19]) {
    using F = Fmt<S>;
    if constexpr (LAY == 1) {
        F::str(n.own(f, 0), RAW ? g[0] : g[0] - L.off[0]);
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const int q1 = pair_first(k), q2 = opp(q1);
            F::st2(n.own(f, q1), RAW ? g[q1] : g[q1] - L.off[q1], RAW ? g[q2] : g[q2] - L.off[q2]);
        }
    } else {
#pragma unroll
        for (int q = 0; q < 19; ++q) {
            if (RAW) F::str(n.own(f, q), g[q]);
            else F::st(n.own(f, q), g[q], L.off[q]);
        }
    }
}

/* FEAT: compile-time features, chosen at launch from the configuration and
 * the node types present, so a channel kernel carries no lid code (whose
 * 19-entry temporaries would otherwise set every variant's register count) */
constexpr int FEAT_HALFWAY = 1, FEAT_LID = 2, FEAT_CLAMP = 4, FEAT_XBC = 8;
/* LR7's MRT model (which takes no body force): the projected collision only,
 * on the stored deviations of FP16 / BF16 (collide_mrt_dev; the other models
 * convert those to populations and back) and on populations
 * (collide_mrt_pop): FP64, whose bound is the FP64 pipe (1.05 M nodes: 0.54 ms
 * through collide_mrt, 0.30 ms so), and FP32 (48 registers instead of 56:
 * level on the 512 x 128 x 128 channel, which HBM bounds, 21.88 -> 21.74 ms
 * for 100 steps; where a step is two or three waves of blocks the latency
 * counts: 4 % on a ragged channel of 0.7 M nodes, 2 % on a refined one) */
constexpr int FEAT_DEVMRT = 16;
/* the relaxation time of each node from the learned closure's last refresh
 * (StepParams::nu) instead of the LES setting */
constexpr int FEAT_NUBUF = 32;

/* FP16 / BF16 nodes collide their stored deviations (no offsets on the way
 * in and out) */
#ifndef LBM_SC_DEV
#define LBM_SC_DEV 1
#endif
/* resident blocks per SM the register allocation must allow (0: no bound)
 * for the FP16 / BF16 deviation kernels without lid or alternate
 * boundaries: 10 blocks of 128 threads, 48 registers, no spills (measured
 * 3 % faster than 9 blocks at 55 registers on the 512 x 128 x 128 channel) */
#ifndef LBM_SC_MINB
#define LBM_SC_MINB 10
#endif

/* the step index of the launch; a load for launches replayed from a graph,
 * so it is read only where it is needed */
__device__ __forceinline__ int sc_time(const StepParams& p) { return p.t + (p.step_dev ? *p.step_dev : 0); }

/* vel_av / vel_fluc (LR7:1018-1058) of node c with the velocity (u, v) after
 * the collision: running mean, then variance about it */
__device__ __forceinline__ void sc_stats(const StepParams& p, float* __restrict__ stats, unsigned qs, unsigned c,
                                         float u, float v) {
    const int t = sc_time(p);
    if (t < p.start_av) return;
    float* au = stats;
    float* av = stats + qs;
    const float w = p.stats_weight;
    if (t < p.start_fluc) {
        const float nn = float(t - p.start_av);
        au[c] = (au[c] * nn + u * w) / (nn + w);
        av[c] = (av[c] * nn + v * w) / (nn + w);
    } else {
        float* fu = stats + 2 * (size_t)qs;
        float* fv = stats + 3 * (size_t)qs;
        const float nn = float(t - p.start_fluc);
        const float du = (u - au[c]) * (u - au[c]);
        const float dv = (v - av[c]) * (v - av[c]);
        fu[c] = (fu[c] * nn + du * w) / (nn + w);
        fv[c] = (fv[c] * nn + dv * w) / (nn + w);
    }
}

/* whether the refinement's band fill writes this node */
__device__ __forceinline__ bool sc_in_band(const Level& L, const StepParams& p, int x, int y, int z) {
    const int b = p.band;
    return b && (x < b || x >= L.nx - b || y < b || y >= L.ny - b || (p.band_z && (z < b || z >= L.nz - b)));
}

/* the collision, statistics, store and moment export of a non-solid node;
 * f holds populations, or for DEV their stored deviations.  With DEVMRT on
 * populations an inlet's or outlet's rebuild (bc, uin; FLUID otherwise) is
 * part of the collision: it only replaces the density or the momentum, which
 * the projected collision has by then, and f is its neighbour's as stored */
template <class S, int LAY, bool DEVMRT, bool NUBUF>
__device__ __forceinline__ void sc_collide_store(const Level& L, const StepParams& p, S* __restrict__ fB,
                                                 float* __restrict__ stats, const NodeIdx<LAY>& n,
                                                 typename Fmt<S>::T f[19], unsigned c, const int x, const int y,
                                                 const int z, const int bc, const typename Fmt<S>::T uin) {
    using T = typename Fmt<S>::T;
    constexpr bool DEV = LBM_SC_DEV && sizeof(S) == 2;
    const unsigned qs = unsigned(L.qstride);
    /* the learned closure's eddy viscosity of this node from its last
     * refresh, or the configured relaxation */
    const float om = NUBUF ? 1.f / (p.tau0 + 3.f * p.nu[c]) : p.omega;
    const bool les = !NUBUF && p.les != 0;
    if constexpr (DEVMRT) {
        if constexpr (DEV)
            collide_mrt_dev<T>(f, T(om), les, T(p.tau0), T(p.smag_k), T(L.u_ref));
        else if constexpr (sizeof(T) == 8)
            collide_mrt_pop<T>(f, T(om), les, p.tau0_d, p.smag_k_d, bc, T(p.rho_out), uin);
        else
            collide_mrt_pop<T>(f, T(om), les, p.tau0, p.smag_k, bc, T(p.rho_out), uin);
    } else {
        T dp = T(p.dpdy_dev ? *p.dpdy_dev : p.dpdy);
        if (y > p.dyn_y1) dp = T(0);
        if (DEV) {
#pragma unroll
            for (int q = 0; q < 19; ++q) f[q] += L.off[q];
        }
        collide_other<T>(p.model, f, T(om), les, T(p.cs), dp);
        if (DEV) {
#pragma unroll
            for (int q = 0; q < 19; ++q) f[q] -= L.off[q];
        }
    }
    if (p.extras) {
        if (p.stats_on) {
            T u = 0, v = 0;
#pragma unroll
            for (int q = 0; q < 19; ++q) {
                const T g = DEV ? f[q] + L.off[q] : f[q];
                if (cx(q)) u += T(cx(q)) * g;
                if (cy(q)) v += T(cy(q)) * g;
            }
            sc_stats(p, stats, qs, c, float(u), float(v));
        }
        if (sc_in_band(L, p, x, y, z)) return;
    }
    store19<S, LAY, DEV>(L, fB, n, f);
}

/* moments for the coarse->fine interpolation (LR7:1590-1605): post-collision
 * for fluid nodes, the pulled values at bounce-back nodes */
template <class S>
__device__ __forceinline__ void sc_export(const Level& L, const StepParams& p, float* __restrict__ mom_export,
                                          const typename Fmt<S>::T f[19], const int x, const int y, const int z) {
    constexpr bool DEV = LBM_SC_DEV && sizeof(S) == 2;
    const int ex = x - p.exp_x0, ey = y - p.exp_y0;
    if (ex >= 0 && ex < p.exp_nx && ey >= 0 && ey < p.exp_ny) {
        float ff[19], mom[9];
#pragma unroll
        for (int q = 0; q < 19; ++q) ff[q] = DEV ? float(f[q]) + L.off[q] : float(f[q]);
        physical_moments<float>(ff, mom);
        const unsigned ne = unsigned(p.exp_nx * p.exp_ny * L.nz);
        const unsigned ce = (unsigned(z) * p.exp_ny + ey) * p.exp_nx + ex;
#pragma unroll
        for (int i = 0; i < 9; ++i) mom_export[i * ne + ce] = mom[i];
    }
}

/* one node of the step: its addressing, mask byte and coordinates */
template <int LAY> struct ScNode {
    NodeIdx<LAY> n;
    unsigned c;
    int mbyte, type, x, y, z;
};

template <int FEAT, int LAY>
__device__ __forceinline__ ScNode<LAY> sc_setup(const Level& L, const uint8_t* __restrict__ mask, const int x,
                                                const int y, const int z) {
    /* 32-bit element offsets: a level holds fewer than 2^31 elements per
     * buffer (checked at allocation) */
    const unsigned plane = unsigned(L.plane), pitch = unsigned(L.pitch);
    const unsigned c = z * plane + y * pitch + x;
    const int mbyte = mask[c];
    /* periodic neighbours; only boundary nodes, whose pulled values the
     * reference discards or bounces, ever wrap in x or y */
    constexpr bool cl = (FEAT & FEAT_CLAMP) != 0;
    const unsigned xm = (x == 0) ? (cl ? 0 : L.nx - 1) : x - 1;
    const unsigned xp = (x == L.nx - 1) ? (cl ? x : 0) : x + 1;
    const unsigned ym = (y == 0) ? (cl ? 0 : L.ny - 1) : y - 1;
    const unsigned yp = (y == L.ny - 1) ? (cl ? y : 0) : y + 1;
    const unsigned zm = (z == 0) ? (cl ? 0 : L.nz - 1) : z - 1;
    const unsigned zp = (z == L.nz - 1) ? (cl ? z : 0) : z + 1;
    return ScNode<LAY>{NodeIdx<LAY>(L, xm, unsigned(x), xp, ym, unsigned(y), yp, zm, unsigned(z), zp), c, mbyte,
                       mbyte & TYPE_MASK, x, y, z};
}

/* the 19 pulls of a node: populations, or for DEV their stored deviations */
template <class S>
__device__ __forceinline__ constexpr bool sc_dev() { return LBM_SC_DEV && sizeof(S) == 2; }
template <class S, int LAY>
__device__ __forceinline__ void sc_load(const Level& L, const S* __restrict__ fA, const ScNode<LAY>& nd,
                                        typename Fmt<S>::T f[19]) {
    using F = Fmt<S>;
    using T = typename F::T;
#pragma unroll
    for (int q = 0; q < 19; ++q)
        f[q] = sc_dev<S>() ? T(F::ldr(nd.n.pull(fA, q))) : F::ld(nd.n.pull(fA, q), L.off[q]);
}

/* the rest of the node update once its pulls are in f.
 * FP16 / BF16 storage (DEV): the node works on the stored deviations
 * h = f - off and LR7's MRT collides them in that form (collide_mrt_dev),
 * so no population is offset on its way in or out; boundary rebuilds, the
 * lid, the alternate boundaries, the other collision models, the
 * statistics and the moment export see populations f = h + off. */
template <class S, int FEAT, int LAY>
__device__ __forceinline__ void sc_finish(const Level& L, const StepParams& p, const S* __restrict__ fA,
                                          S* __restrict__ fB, float* __restrict__ stats,
                                          float* __restrict__ mom_export, const uint32_t* __restrict__ links,
                                          const ScNode<LAY>& nd, typename Fmt<S>::T f[19]) {
    using F = Fmt<S>;
    using T = typename F::T;
    constexpr bool DEV = sc_dev<S>();
    constexpr bool HALFWAY = (FEAT & FEAT_HALFWAY) != 0;
    const NodeIdx<LAY>& n = nd.n;
    const unsigned c = nd.c, pitch = unsigned(L.pitch);
    const int mbyte = nd.mbyte, type = nd.type, x = nd.x, y = nd.y, z = nd.z;
    /* the neighbours of the inlet / outlet rebuilds (wrapped as the pulls) */
    constexpr bool cl = (FEAT & FEAT_CLAMP) != 0;
    const unsigned xm = (x == 0) ? (cl ? 0 : L.nx - 1) : x - 1;
    const unsigned xp = (x == L.nx - 1) ? (cl ? x : 0) : x + 1;
    const unsigned ym = (y == 0) ? (cl ? 0 : L.ny - 1) : y - 1;
    const unsigned yp = (y == L.ny - 1) ? (cl ? y : 0) : y + 1;
    if (HALFWAY && (mbyte & NEAR_SOLID)) {
        /* a population that would come from a solid node is the node's own
         * post-collision population of the opposite direction, reflected
         * half-way to the solid; links has bit q set for those q */
        const uint32_t lk = links[c];
#pragma unroll
        for (int q = 1; q < 19; ++q)
            if (lk & (1u << q))
                f[q] = DEV ? F::ldr(n.own(fA, opp(q))) + (L.off[opp(q)] - L.off[q])
                           : F::ld(n.own(fA, opp(q)), L.off[opp(q)]);
    }

    if (type == WALL || type == BODY) {
        /* full-way bounce-back (LR7:1493-1526); the momentum exchange of BODY
         * nodes is summed by k_force_list from the same fA */
        T g[19];
#pragma unroll
        for (int q = 0; q < 19; ++q) g[q] = DEV ? f[opp(q)] + (L.off[opp(q)] - L.off[q]) : f[opp(q)];
        store19<S, LAY, DEV>(L, fB, n, g);
        if (p.exp_nx > 0) sc_export<S>(L, p, mom_export, f, x, y, z);
        return;
    } else {
        int bc = FLUID;
        T uin = T(p.u_in);
        if (type >= WEST_INLET && type <= NORTH_OUTLET) {
            /* rebuild from the neighbour's stored post-collision state */
            const unsigned cn = type == WEST_INLET ? c - x + xp : type == EAST_OUTLET ? c - x + xm
                              : type == SOUTH_INLET ? c + (yp - y) * pitch : c + (ym - y) * pitch;
#pragma unroll
            for (int q = 0; q < 19; ++q) f[q] = F::ld(n.at(fA, q, cn), L.off[q]);
            if (p.noise_amp != 0.f) {
                const uint32_t cell = uint32_t((z * L.ny + y) * L.nx + x);
                const float xi = philox_uniform(p.noise_seed, cell, uint32_t(sc_time(p)));
                uin = uin + T(p.u_in) * T(p.noise_amp) * (T(2) * T(xi) - T(1));
            }
            if constexpr (!DEV && (FEAT & FEAT_DEVMRT) != 0) {
                bc = type;
            } else {
                extrap<T>(type, f, T(p.rho_out), uin);
                if (DEV) {
#pragma unroll
                    for (int q = 0; q < 19; ++q) f[q] -= L.off[q];
                }
            }
        } else if (((FEAT & FEAT_LID) && type == LID) || ((FEAT & FEAT_XBC) && type >= DIR_WEST)) {
            if (DEV) {
#pragma unroll
                for (int q = 0; q < 19; ++q) f[q] += L.off[q];
            }
            if ((FEAT & FEAT_LID) && type == LID) {
                lid<T>(f, p.lid_face, T(p.lid_u[0]), T(p.lid_u[1]), T(p.lid_u[2]), p.lid_quirk != 0);
            } else if (FEAT & FEAT_XBC) {
                alt_boundary<T>(type, f, x, y, z, L.nx, L.ny, L.nz, T(p.u_in), sc_time(p));
            }
            if (DEV) {
#pragma unroll
                for (int q = 0; q < 19; ++q) f[q] -= L.off[q];
            }
        }
        sc_collide_store<S, LAY, (FEAT & FEAT_DEVMRT) != 0, (FEAT & FEAT_NUBUF) != 0>(L, p, fB, stats, n, f, c,
                                                                                      x, y, z, bc, uin);
    }
    if (p.exp_nx > 0) sc_export<S>(L, p, mom_export, f, x, y, z);
}


/* the node update of one node (x, y, z) inside the level */
template <class S, int FEAT, int LAY>
__device__ __forceinline__ void sc_node(const Level& L, const StepParams& p, const S* __restrict__ fA,
                                        S* __restrict__ fB, const uint8_t* __restrict__ mask,
                                        float* __restrict__ stats, float* __restrict__ mom_export,
                                        const uint32_t* __restrict__ links, const int x, const int y, const int z) {
    const ScNode<LAY> nd = sc_setup<FEAT, LAY>(L, mask, x, y, z);
    typename Fmt<S>::T f[19];
    sc_load<S, LAY>(L, fA, nd, f);
    sc_finish<S, FEAT, LAY>(L, p, fA, fB, stats, mom_export, links, nd, f);
}

template <class S, int FEAT> __host__ __device__ constexpr int sc_min_blocks() {
    return sizeof(S) == 2 && (FEAT & FEAT_DEVMRT) && !(FEAT & (FEAT_LID | FEAT_XBC)) ? LBM_SC_MINB : 0;
}

template <class S, int FEAT, int LAY>
__global__ void __launch_bounds__(SC_BX* SC_BY, sc_min_blocks<S, FEAT>()) k_stream_collide(const Level L, const StepParams p,
                                                                  const S* __restrict__ fA, S* __restrict__ fB,
                                                                  const uint8_t* __restrict__ mask,
                                                                  float* __restrict__ stats,
                                                                  float* __restrict__ mom_export,
                                                                  const uint32_t* __restrict__ links) {
    pdl_wait();
    const int x = blockIdx.x * SC_BX + threadIdx.x;
    const int y = blockIdx.y * SC_BY + threadIdx.y;
    if (x >= L.nx || y >= L.ny) return;
    sc_node<S, FEAT, LAY>(L, p, fA, fB, mask, stats, mom_export, links, x, y, int(blockIdx.z));
}

/* The stream-collide step with the learned subgrid closure in place of the
 * Smagorinsky model: the node update of k_stream_collide (pull, half-way or
 * full-way bounce-back, inlet/outlet rebuild with inlet noise, running
 * statistics; no lid, no clamped edges, no refinement export), with the
 * eddy viscosity of every node from the MLP evaluated on the tensor cores
 * for the whole 32 x 4 tile at once.  Persistent blocks walk the tiles so
 * that each block stages the weights and allocates its TMEM once per launch.
 * MRT collision (LR7:583-711) at tau_eff = tau0 + 3 nu_t; FP32 arithmetic.
 *
 * What bounds it is the L1 cache: the pair-interleaved layout brings every
 * sector of a row twice to an SM (q and its opposite are pulled by different
 * rows) unless L1 still holds it, and a block's operands take 27 KB of the
 * array that L1 shares with shared memory.  So the launch asks for exactly the
 * shared memory of its resident blocks (5: 140 of 228 KB).  512 x 128 x 128,
 * FP32, 40 steps and a read-back: 16.4 ms, with all of the array as shared
 * memory 21.4 ms.  Five blocks per SM also leave 96 registers a thread and so
 * no spills; 7 blocks (72 registers) take 16.3 ms there, but 4.56 instead of
 * 4.00 ms for 50 steps of 211 x 90 x 70 nodes (FP16 / BF16: 4.60 and 4.00 ms;
 * 4 blocks 4.37, 6 blocks 4.04).  Copying the next tile's pulls into shared
 * memory with cp.async cost more L1 than it hid. */
constexpr int MLP_BY = 4; /* tile 32 x 4: one M = 128 MMA per layer */
constexpr int MLP_ROWS = SC_BX * MLP_BY;
constexpr int MLP_BLOCKS = 5;

/* the 19 values g of node c into buffer f, as store19 */
template <int LAY> struct CellIdx {
    unsigned c, qs;
    template <class P> __device__ __forceinline__ P* own(P* f, int q) const {
        if (LAY == 0) return f + (unsigned(q) * qs + c);
        return q == 0 ? f + ((c >> 5) * BLOCK_ELEMS + (c & 31u))
                      : (f + ((c >> 5) * BLOCK_ELEMS + 2u * (c & 31u))) + pair_qoff(q);
    }
};

template <class S, bool HALFWAY, int LAY>
__global__ void __launch_bounds__(MLP_ROWS, MLP_BLOCKS)
    k_stream_collide_mlp(const Level L, const StepParams p, const S* __restrict__ fA, S* __restrict__ fB,
                         const uint8_t* __restrict__ mask, float* __restrict__ stats,
                         const uint32_t* __restrict__ links, const unsigned char* __restrict__ blob,
                         int* __restrict__ err) {
    using F = Fmt<S>;
    extern __shared__ __align__(128) unsigned char dsm[];
#if defined(__CUDA_ARCH__)
    sgs::InferSmem<MLP_ROWS>& sm = *reinterpret_cast<sgs::InferSmem<MLP_ROWS>*>(dsm);
    sgs::infer_setup<MLP_ROWS>(sm, blob);
    const unsigned qs = unsigned(L.qstride);
    const unsigned plane = unsigned(L.plane), pitch = unsigned(L.pitch);
    const int tiles_x = L.pitch / SC_BX, tiles_y = (L.ny + MLP_BY - 1) / MLP_BY;
    const int ntiles = tiles_x * tiles_y * L.nz;
    const float tau0 = 1.f / p.omega, inv_t0 = p.omega;
    /* tile g = (tz tiles_y + ty) tiles_x + tx, advanced by the grid without
     * dividing again */
    struct Tile {
        int x, y, z;
    };
    auto tile_of = [&](int g) {
        const int r = g / tiles_x;
        return Tile{g - r * tiles_x, r % tiles_y, r / tiles_y};
    };
    const Tile hop = tile_of(int(gridDim.x));
    auto next_of = [&](Tile t) {
        t.x += hop.x, t.y += hop.y, t.z += hop.z;
        if (t.x >= tiles_x) t.x -= tiles_x, ++t.y;
        if (t.y >= tiles_y) t.y -= tiles_y, ++t.z;
        return t;
    };
    /* this thread's node in a tile; its mask byte, or -1 outside the domain */
    auto cell_of = [&](const Tile& t, int& x, int& y) {
        x = t.x * SC_BX + int(threadIdx.x), y = t.y * MLP_BY + int(threadIdx.y);
        return unsigned(t.z) * plane + unsigned(y) * pitch + unsigned(x);
    };
    auto mask_of = [&](const Tile& t) {
        int x, y;
        const unsigned c = cell_of(t, x, y);
        return x < L.nx && y < L.ny ? int(mask[c]) : -1;
    };
    Tile t = tile_of(int(blockIdx.x));
    int mbyte = int(blockIdx.x) < ntiles ? mask_of(t) : -1;
    for (int g = blockIdx.x; g < ntiles; g += gridDim.x) {
        /* the next tile's mask is on its way during this tile's work */
        const Tile tn = next_of(t);
        const int mnext = g + int(gridDim.x) < ntiles ? mask_of(tn) : -1;
        const bool live = mbyte >= 0;
        const int type = live ? mbyte & TYPE_MASK : int(FLUID);
        int x, y;
        const CellIdx<LAY> n{cell_of(t, x, y), qs};
        float f[19];
        if (live) {
            const int z = t.z;
            const unsigned xm = (x == 0) ? L.nx - 1 : x - 1, xp = (x == L.nx - 1) ? 0 : x + 1;
            const unsigned ym = (y == 0) ? L.ny - 1 : y - 1, yp = (y == L.ny - 1) ? 0 : y + 1;
            const unsigned zm = (z == 0) ? L.nz - 1 : z - 1, zp = (z == L.nz - 1) ? 0 : z + 1;
            const NodeIdx<LAY> ni(L, xm, unsigned(x), xp, ym, unsigned(y), yp, zm, unsigned(z), zp);
            if (type >= WEST_INLET && type <= NORTH_OUTLET) {
                /* rebuild from the neighbour's stored post-collision state */
                const unsigned cn = type == WEST_INLET ? n.c - x + xp : type == EAST_OUTLET ? n.c - x + xm
                                  : type == SOUTH_INLET ? n.c + (yp - y) * pitch : n.c + (ym - y) * pitch;
#pragma unroll
                for (int q = 0; q < 19; ++q) f[q] = F::ld(ni.at(fA, q, cn), L.off[q]);
                float uin = p.u_in;
                if (p.noise_amp != 0.f) {
                    const uint32_t cell = uint32_t((z * L.ny + y) * L.nx + x);
                    const float xi = philox_uniform(p.noise_seed, cell, uint32_t(sc_time(p)));
                    uin = uin + p.u_in * p.noise_amp * (2.f * xi - 1.f);
                }
                extrap<float>(type, f, p.rho_out, uin);
            } else {
#pragma unroll
                for (int q = 0; q < 19; ++q) f[q] = F::ld(ni.pull(fA, q), L.off[q]);
                if (HALFWAY && (mbyte & NEAR_SOLID)) {
                    const uint32_t lk = links[n.c];
#pragma unroll
                    for (int q = 1; q < 19; ++q)
                        if (lk & (1u << q)) f[q] = F::ld(ni.own(fA, opp(q)), L.off[opp(q)]);
                }
            }
        } else {
#pragma unroll
            for (int q = 0; q < 19; ++q) f[q] = wq(q);
        }
        /* bounce-back nodes are done before the closure, so that only the
         * moments stay live across its tensor-core round trips */
        const bool solid = live && (type == WALL || type == BODY);
        if (solid) {
            float gb[19];
#pragma unroll
            for (int q = 0; q < 19; ++q) gb[q] = f[opp(q)];
            store19<S, LAY, false>(L, fB, n, gb);
        }
        /* the closure for the whole tile; the collision's moments give
         * Pi_neq (the projected MRT collision on full populations) */
        const MrtDev<float> mo = mrt_dev_moments<float>(f, 0.f);
        float p6[6], xf[sgs::NIN];
        mrt_dev_pi(mo, p6);
        const float sc = -1.5f / mo.rho;
#pragma unroll
        for (int k = 0; k < 6; ++k) p6[k] *= sc;
        sgs::features_fast(p6, tau0, inv_t0, xf);
        /* across the tensor-core round trips only rho, j and the five
         * stresses stay live; the products are formed again afterwards */
        float keep[10] = {mo.rho, mo.jx, mo.jy, mo.jz, mo.n9, mo.n11, mo.n13, mo.n14, mo.n15,
                          sgs::strain_gain(xf, inv_t0)};
        const float o = sgs::infer_nu<MLP_ROWS>(sm, xf, err);
        if (o < 0.f) break; /* a tensor-core wait ran out (block-uniform) */
        t = tn;
        mbyte = mnext;
        if (!live || solid) continue;
#pragma unroll
        for (int k = 0; k < 10; ++k) asm volatile("" : "+f"(keep[k]));
        const float nu = o * keep[9];
        if (p.nu) p.nu[n.c] = nu;
        MrtDev<float> mr;
        mr.rho = keep[0], mr.jx = keep[1], mr.jy = keep[2], mr.jz = keep[3], mr.n9 = keep[4], mr.n11 = keep[5];
        mr.n13 = keep[6], mr.n14 = keep[7], mr.n15 = keep[8], mr.n1 = 0.f;
        mrt_dev_complete(mr, 0.f);
        mrt_dev_relax(f, mr, 1.f / (tau0 + 3.f * nu));
        if (p.stats_on) {
            float u = 0, v = 0;
#pragma unroll
            for (int q = 0; q < 19; ++q) {
                if (cx(q)) u += float(cx(q)) * f[q];
                if (cy(q)) v += float(cy(q)) * f[q];
            }
            sc_stats(p, stats, qs, n.c, u, v);
        }
        store19<S, LAY, false>(L, fB, n, f);
    }
    sgs::infer_teardown<MLP_ROWS>(sm);
#endif
}

/* whether launch_sc_t has a kernel of these features */
template <class S> inline bool sc_feat_built(int feat) {
    if (feat & FEAT_NUBUF) return sizeof(S) <= 4 && !(feat & (FEAT_LID | FEAT_CLAMP | FEAT_XBC));
    return feat >= 0 && feat < 32;
}

/* the stream-collide launch of one storage format and layout */
template <class S, int LAY>
inline cudaError_t launch_sc_t(const Level& L, const StepParams& p, const void* fA, void* fB, const uint8_t* mask,
                               float* stats, float* mom_export, cudaStream_t s, const uint32_t* links) {
    const dim3 block(SC_BX, SC_BY), grid(L.pitch / SC_BX, (L.ny + SC_BY - 1) / SC_BY, L.nz);
    const int feat = (p.halfway ? FEAT_HALFWAY : 0) | (p.has_lid ? FEAT_LID : 0) | (p.pull_clamp ? FEAT_CLAMP : 0) |
                     (p.has_xbc ? FEAT_XBC : 0) | (p.model == MRT ? FEAT_DEVMRT : 0) |
                     (p.nu_reuse ? FEAT_NUBUF : 0);
    if (!sc_feat_built<S>(feat)) return cudaErrorInvalidValue;
#define LBM_SC(FT)                                                                                            \
    case FT:                                                                                                  \
        return launch_pdl_if(p.early, k_stream_collide<S, FT, LAY>, grid, block, 0, s, L, p, (const S*)fA, (S*)fB, \
                             mask, stats, mom_export, links);
    switch (feat) {
        /* every combination of half-way, lid, clamp and alternate boundaries,
         * without and with the projected MRT */
        LBM_SC(0) LBM_SC(1) LBM_SC(2) LBM_SC(3) LBM_SC(4) LBM_SC(5) LBM_SC(6) LBM_SC(7)
        LBM_SC(8) LBM_SC(9) LBM_SC(10) LBM_SC(11) LBM_SC(12) LBM_SC(13) LBM_SC(14) LBM_SC(15)
        LBM_SC(16) LBM_SC(17) LBM_SC(18) LBM_SC(19) LBM_SC(20) LBM_SC(21) LBM_SC(22) LBM_SC(23)
        LBM_SC(24) LBM_SC(25) LBM_SC(26) LBM_SC(27) LBM_SC(28) LBM_SC(29) LBM_SC(30) LBM_SC(31)
        default:
            /* the steps between refreshes of the learned closure (channels:
             * no lid, no alternate boundaries, no clamped pulls; not FP64) */
            if constexpr (sizeof(S) <= 4) {
                switch (feat) { LBM_SC(32) LBM_SC(33) LBM_SC(48) LBM_SC(49) default: break; }
            }
    }
#undef LBM_SC
    return cudaErrorInvalidValue;
}

template <class S, bool HW, int LAY>
static cudaError_t sc_mlp_t(const Level& L, const StepParams& p, const void* fA, void* fB, const uint8_t* mask,
                            float* stats, const uint32_t* links, const void* blob, int* err, cudaStream_t s) {
    const size_t smem = sgs::infer_dyn_smem<MLP_ROWS>();
    static sgs::DeviceGrids grids;
    int grid = 0;
    const cudaError_t attr = grids.get(
        [smem](int* g) {
            return sgs::infer_resident(k_stream_collide_mlp<S, HW, LAY>, MLP_ROWS, smem, sgs::tmem_cols<MLP_ROWS>(),
                                       MLP_BLOCKS, g);
        },
        &grid);
    if (attr != cudaSuccess) return attr;
    const int ntiles = (L.pitch / SC_BX) * ((L.ny + MLP_BY - 1) / MLP_BY) * L.nz;
    k_stream_collide_mlp<S, HW, LAY><<<grid < ntiles ? grid : ntiles, dim3(SC_BX, MLP_BY), smem, s>>>(
        L, p, (const S*)fA, (S*)fB, mask, stats, links, (const unsigned char*)blob, err);
    return cudaGetLastError();
}

/* the closure's stream-collide launch of one storage format and layout */
template <class S, int LAY>
inline cudaError_t launch_sc_mlp_t(const Level& L, const StepParams& p, const void* fA, void* fB, const uint8_t* mask,
                                   float* stats, const uint32_t* links, const void* blob, int* err, cudaStream_t s) {
    return p.halfway ? sc_mlp_t<S, true, LAY>(L, p, fA, fB, mask, stats, links, blob, err, s)
                     : sc_mlp_t<S, false, LAY>(L, p, fA, fB, mask, stats, links, blob, err, s);
}

/* the instances, one storage format and layout per translation unit
 * (sc_instance.cu, compiled once for each), so that they build in parallel */
#define LBM_SC_INSTANCES(X) X(f32, 0) X(f16, 0) X(bf16, 0) X(f64, 0) X(f32, 1) X(f16, 1) X(bf16, 1)
#define LBM_SC_DECLARE(NAME, LAY)                                                                                  \
    cudaError_t launch_sc_##NAME##_##LAY(const Level& L, const StepParams& p, const void* fA, void* fB,           \
                                         const uint8_t* mask, float* stats, float* mom_export, cudaStream_t s,    \
                                         const uint32_t* links);                                                  \
    cudaError_t launch_sc_mlp_##NAME##_##LAY(const Level& L, const StepParams& p, const void* fA, void* fB,       \
                                             const uint8_t* mask, float* stats, const uint32_t* links,            \
                                             const void* blob, int* err, cudaStream_t s);
LBM_SC_INSTANCES(LBM_SC_DECLARE)
#undef LBM_SC_DECLARE

}  // namespace lbm
