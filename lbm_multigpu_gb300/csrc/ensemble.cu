/* Ensemble kernels: many periodic D3Q19 boxes of uneven sizes advanced
 * together by one launch per step.
 *
 * Every member is a compact SoA level f[q][z][y][pitch] (pitch = n rounded up
 * to 32) inside one A and one B buffer; a block of 32 x TY threads updates a
 * 32 x TY tile of one z plane of one member (TY 4 or 8, 4 with the closure).  The launch is persistent: a
 * grid sized by the autotuner walks the global tile list, so the per-member
 * work is balanced across the SMs whatever the mix of sizes, and a CUDA graph
 * of several steps replays the whole sequence with one host call.
 *
 * The collision is the LR7 MRT (LRTurbTest/LRMultiGPU7.cu:583-711) with
 *   SGS_NONE   molecular viscosity only (the 2x-resolution "truth" runs),
 *   SGS_SMAG   the constant-Cs Smagorinsky model of LR7:683-685,
 *   SGS_MLP    the learned closure: Pi_neq -> features -> tensor-core MLP ->
 *              nu_t -> tau_eff = tau0 + 3 nu_t.
 * Also: the random-phase turbulence initialisation, velocity and energy
 * read-outs, and the 2x2x2 box filter that turns fine members into training
 * samples for the closure.
 */
#include <cuda_runtime.h>

#include "d3q19.cuh"
#include "ensemble.cuh"
#include "lbm_kernels.cuh"
#include "sgs_infer.cuh"

namespace lbm {
namespace ens {

__device__ __forceinline__ int find_member(const Table& T, int g) {
    int m = 0;
    while (m + 1 < T.count && g >= T.m[m + 1].tile0) ++m;
    return m;
}

/* Bound by HBM and by the warps in flight: lanes outside the box go through the
 * collision too (on the rest state), which takes 48 registers (56 with four
 * rows and no model); left out of it by a `continue`, the kernel took 56 to 64
 * and a step longer: 16 boxes of 26 M nodes 606 -> 624 us with Smagorinsky,
 * 604 -> 612 us without, eight boxes of 7 M 169.0 -> 173.4, 167.6 -> 169.8.
 * Dependent launches: 2 M nodes 60.9 -> 60.5 us, 0.3 M 11.0 -> 10.8. */
template <int TY, int SGS>
__global__ void __launch_bounds__(32 * TY) k_ens_step(const Table T, const float* __restrict__ fA,
                                                      float* __restrict__ fB, float cs) {
    pdl_wait();
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int g = blockIdx.x; g < T.ntiles; g += gridDim.x) {
        const int mi = find_member(T, g);
        const Member& M = T.m[mi];
        const int local = g - M.tile0;
        const int per_z = M.tiles_x * M.tiles_y;
        const int z = local / per_z, r = local - z * per_z;
        const int y = (r / M.tiles_x) * TY + ty, x = (r % M.tiles_x) * 32 + tx;
        const int n = M.n;
        const bool live = x < n && y < n;
        const unsigned pitch = unsigned(M.pitch), plane = unsigned(n) * pitch, qs = plane * unsigned(n);
        const float* a = fA + M.off;
        float* b = fB + M.off;
        float f[19];
        unsigned c = 0;
        if (live) {
            c = unsigned(z) * plane + unsigned(y) * pitch + unsigned(x);
            const unsigned xs[3] = {unsigned(x == 0 ? n - 1 : x - 1), unsigned(x), unsigned(x == n - 1 ? 0 : x + 1)};
            const unsigned yb[3] = {(y == 0 ? n - 1 : y - 1) * pitch, y * pitch, (y == n - 1 ? 0 : y + 1) * pitch};
            const unsigned zb[3] = {(z == 0 ? n - 1 : z - 1) * plane, z * plane, (z == n - 1 ? 0 : z + 1) * plane};
#pragma unroll
            for (int q = 0; q < 19; ++q) f[q] = __ldg(a + q * qs + zb[1 - cz(q)] + yb[1 - cy(q)] + xs[1 - cx(q)]);
        } else {
#pragma unroll
            for (int q = 0; q < 19; ++q) f[q] = wq(q);
        }
        collide_mrt<MRT>(f, M.omega, SGS == SGS_SMAG, cs, 0.f);
        if (live) {
#pragma unroll
            for (int q = 0; q < 19; ++q) b[q * qs + c] = f[q];
        }
    }
}

/* The step with the learned closure, as k_stream_collide_mlp: tiles of 32 x 4
 * (one M = 128 MMA per layer) and persistent blocks; the populations stay in
 * registers across the tensor-core round trips.  Eight boxes of sides 32 to 80
 * (1.8 M nodes): about 100 us with 5 blocks per SM and just their shared
 * memory taken from L1 (one block of 256 rows per SM, what the occupancy API
 * made of kernels with TMEM: 188 us).  The features are rounded to BF16, so
 * the order of operations that leads to them is part of the result: the
 * projected collision (87 us) moves the fields of 50 steps by 1e-5. */
constexpr int MLP_TY = 4, MLP_ROWS = 32 * MLP_TY, MLP_BLOCKS = 5;
__global__ void __launch_bounds__(MLP_ROWS, MLP_BLOCKS) k_ens_step_mlp(const Table T, const float* __restrict__ fA,
                                                                       float* __restrict__ fB,
                                                                       const unsigned char* __restrict__ blob,
                                                                       int* __restrict__ err) {
    extern __shared__ __align__(128) unsigned char dsm[];
#if defined(__CUDA_ARCH__)
    sgs::InferSmem<MLP_ROWS>& sm = *reinterpret_cast<sgs::InferSmem<MLP_ROWS>*>(dsm);
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    sgs::infer_setup<MLP_ROWS>(sm, blob);
    for (int g = blockIdx.x; g < T.ntiles; g += gridDim.x) {
        const Member& M = T.m[find_member(T, g)];
        const int local = g - M.tile0, per_z = M.tiles_x * M.tiles_y;
        const int z = local / per_z, r = local - z * per_z;
        const int y = (r / M.tiles_x) * MLP_TY + ty, x = (r % M.tiles_x) * 32 + tx;
        const int n = M.n;
        const bool live = x < n && y < n;
        const unsigned pitch = unsigned(M.pitch), plane = unsigned(n) * pitch, qs = plane * unsigned(n);
        const unsigned c = unsigned(z) * plane + unsigned(y) * pitch + unsigned(x);
        float f[19];
        if (live) {
            const float* a = fA + M.off;
            const unsigned xs[3] = {unsigned(x == 0 ? n - 1 : x - 1), unsigned(x), unsigned(x == n - 1 ? 0 : x + 1)};
            const unsigned yb[3] = {(y == 0 ? n - 1 : y - 1) * pitch, y * pitch, (y == n - 1 ? 0 : y + 1) * pitch};
            const unsigned zb[3] = {(z == 0 ? n - 1 : z - 1) * plane, z * plane, (z == n - 1 ? 0 : z + 1) * plane};
#pragma unroll
            for (int q = 0; q < 19; ++q) f[q] = __ldg(a + q * qs + zb[1 - cz(q)] + yb[1 - cy(q)] + xs[1 - cx(q)]);
        } else {
#pragma unroll
            for (int q = 0; q < 19; ++q) f[q] = wq(q);
        }
        float rho, p6[6], xf[sgs::NIN];
        pi_neq<float>(f, rho, p6);
        const float sc = -1.5f / rho;
#pragma unroll
        for (int k = 0; k < 6; ++k) p6[k] *= sc;
        sgs::features_fast(p6, M.tau0, M.omega, xf); /* omega = 1 / tau0 */
        const float gain = sgs::strain_gain(xf, M.omega);
        const float o = sgs::infer_nu<MLP_ROWS>(sm, xf, err);
        if (o < 0.f) break; /* a tensor-core wait ran out (block-uniform) */
        if (!live) continue;
        collide_mrt<MRT>(f, 1.f / (M.tau0 + 3.f * o * gain), false, 0.f, 0.f);
        float* b = fB + M.off + c;
#pragma unroll
        for (int q = 0; q < 19; ++q) b[q * qs] = f[q];
    }
    sgs::infer_teardown<MLP_ROWS>(sm);
#endif
}

/* random-phase solenoidal field: u = sum_m a_m e_m cos(2 pi k_m.x / n + phi_m),
 * the equilibrium at rho = 1 and u into the first buffer (a step overwrites
 * the whole of the second before anything reads it).
 *
 * Bound by the FP64 pipe (2 operations per clock and SM on this chip), so the
 * sum is factored by the x wavenumber: a block takes rows of one z plane and
 *   1. adds, per row and kx, the amplitudes (A + iB) e^{i 2 pi (ky y + kz z)/n}
 *      of its modes (sorted by kx) into a complex Z[kx], one thread per (row,
 *      kx) with the rows in adjacent lanes, so that a warp's lanes share their
 *      mode list;
 *   2. forms u(x) = sum_kx Re Z cos - Im Z sin, and u(n - x) from the same two
 *      sums (C - S, C + S).
 * The angles are multiples of 2 pi / n: one table of n cosines and sines per
 * block, no cosine per node and mode.  About 3 (kmax + 1) + 12 modes / n FP64
 * operations per node instead of a cosine and 3 products for every mode:
 * eight boxes of sides 48 to 128 (7.1 M nodes, some 300 modes each) took
 * 143 ms that way. */
constexpr int INIT_THREADS = 256;
__global__ void __launch_bounds__(INIT_THREADS) k_ens_init(const Table T, const KMode* __restrict__ modes,
                                                           float* __restrict__ fA, int mi, int rows) {
    extern __shared__ double ism[];
    const Member& M = T.m[mi];
    const int n = M.n, nk = M.kmax + 1;
    double2* tab = reinterpret_cast<double2*>(ism); /* cos, sin of 2 pi i / n */
    double* Z = ism + 2 * n;                        /* [kx][6][rows]: Re x y z, Im x y z */
    const int z = blockIdx.y, y0 = blockIdx.x * rows;
    for (int i = threadIdx.x; i < n; i += INIT_THREADS) {
        double sn, cs;
        sincospi(2.0 * i / n, &sn, &cs);
        tab[i] = make_double2(cs, sn);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nk * rows; i += INIT_THREADS) {
        const int kx = i / rows, r = i - kx * rows, y = min(y0 + r, n - 1);
        double re[3] = {0, 0, 0}, im[3] = {0, 0, 0};
        /* the member's modes of this kx: [lower bound, upper bound) of the sorted list */
        int lo = M.mode0, hi = M.mode0 + M.nmodes;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (modes[mid].k[0] < kx) lo = mid + 1;
            else hi = mid;
        }
        for (int m = lo; m < M.mode0 + M.nmodes && modes[m].k[0] == kx; ++m) {
            int ph = int(((long long)modes[m].k[1] * y + (long long)modes[m].k[2] * z) % n);
            if (ph < 0) ph += n;
            const double2 w = tab[ph];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double a = modes[m].re[k], b = modes[m].im[k];
                re[k] += a * w.x - b * w.y;
                im[k] += a * w.y + b * w.x;
            }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            Z[(6 * kx + k) * rows + r] = re[k];
            Z[(6 * kx + 3 + k) * rows + r] = im[k];
        }
    }
    __syncthreads();
    const unsigned pitch = unsigned(M.pitch), plane = unsigned(n) * pitch, qs = plane * unsigned(n);
    const int half = n / 2 + 1;
    for (int i = threadIdx.x; i < rows * half; i += INIT_THREADS) {
        const int r = i / half, x = i - r * half, y = y0 + r;
        if (y >= n) break;
        double C[3] = {0, 0, 0}, S[3] = {0, 0, 0};
        int ph = 0;
        for (int kx = 0; kx < nk; ++kx) {
            const double2 w = tab[ph];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                C[k] += Z[(6 * kx + k) * rows + r] * w.x;
                S[k] += Z[(6 * kx + 3 + k) * rows + r] * w.y;
            }
            ph += x;
            if (ph >= n) ph -= n;
        }
        for (int side = 0; side < 2; ++side) {
            const int xx = side ? n - x : x;
            if (side && (x == 0 || xx == x)) break;
            const double sg = side ? 1.0 : -1.0;
            const float ux = float(C[0] + sg * S[0]), uy = float(C[1] + sg * S[1]), uz = float(C[2] + sg * S[2]);
            const float usq = ux * ux + uy * uy + uz * uz;
            const unsigned c = unsigned(z) * plane + unsigned(y) * pitch + unsigned(xx);
#pragma unroll
            for (int q = 0; q < 19; ++q) {
                const float cu = float(cx(q)) * ux + float(cy(q)) * uy + float(cz(q)) * uz;
                fA[M.off + q * qs + c] = wq(q) * (1.f + 3.f * cu + 4.5f * cu * cu - 1.5f * usq);
            }
        }
    }
}

/* equilibrium at rho = 1 and the given velocity field (compact, per member
 * at Member::uoff) */
__global__ void k_ens_init_from(const Table T, const float* __restrict__ u, float* __restrict__ fA,
                                float* __restrict__ fB) {
    const int g = blockIdx.x;
    if (g >= T.ntiles) return;
    const int mi = find_member(T, g);
    const Member& M = T.m[mi];
    const int local = g - M.tile0, per_z = M.tiles_x * M.tiles_y;
    const int z = local / per_z, r = local - z * per_z;
    const int y = (r / M.tiles_x) * T.ty + (threadIdx.x >> 5), x = (r % M.tiles_x) * 32 + (threadIdx.x & 31);
    const int n = M.n;
    if (x >= n || y >= n) return;
    const size_t o = M.uoff + (size_t(z) * n + y) * n + x, nn = size_t(n) * n * n;
    const float ux = u[o], uy = u[o + nn], uz = u[o + 2 * nn];
    const unsigned pitch = unsigned(M.pitch), plane = unsigned(n) * pitch, qs = plane * unsigned(n);
    const unsigned c = unsigned(z) * plane + unsigned(y) * pitch + unsigned(x);
    const float usq = ux * ux + uy * uy + uz * uz;
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        const float cu = float(cx(q)) * ux + float(cy(q)) * uy + float(cz(q)) * uz;
        const float fe = wq(q) * (1.f + 3.f * cu + 4.5f * cu * cu - 1.5f * usq);
        fA[M.off + q * qs + c] = fe;
        fB[M.off + q * qs + c] = fe;
    }
}

/* density and momentum of the node whose population 0 is at f */
__device__ __forceinline__ void node_moments(const float* __restrict__ f, unsigned qs, float& rho, float j[3]) {
    rho = j[0] = j[1] = j[2] = 0;
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        const float v = f[q * qs];
        rho += v;
        if (cx(q)) j[0] += float(cx(q)) * v;
        if (cy(q)) j[1] += float(cy(q)) * v;
        if (cz(q)) j[2] += float(cz(q)) * v;
    }
}

/* velocity j / rho of every member into the compact buffer at Member::uoff */
__global__ void k_ens_velocity(const Table T, const float* __restrict__ f, float* __restrict__ u) {
    const int g = blockIdx.x;
    if (g >= T.ntiles) return;
    const int mi = find_member(T, g);
    const Member& M = T.m[mi];
    const int local = g - M.tile0, per_z = M.tiles_x * M.tiles_y;
    const int z = local / per_z, r = local - z * per_z;
    const int y = (r / M.tiles_x) * T.ty + (threadIdx.x >> 5), x = (r % M.tiles_x) * 32 + (threadIdx.x & 31);
    const int n = M.n;
    if (x >= n || y >= n) return;
    const unsigned pitch = unsigned(M.pitch), plane = unsigned(n) * pitch, qs = plane * unsigned(n);
    const unsigned c = unsigned(z) * plane + unsigned(y) * pitch + unsigned(x);
    float rho, j[3];
    node_moments(f + M.off + c, qs, rho, j);
    const size_t o = M.uoff + (size_t(z) * n + y) * n + x, nn = size_t(n) * n * n;
    u[o] = j[0] / rho;
    u[o + nn] = j[1] / rho;
    u[o + 2 * nn] = j[2] / rho;
}

/* per-member kinetic energy 1/2 <|u|^2> over the nodes, FP64, from the
 * populations (u = j / rho in FP32, as k_ens_velocity): ENERGY_BLOCKS block
 * partials per member, one warp per row, summed by k_ens_energy_final in a
 * fixed order.  Bound by the one read of the populations */
__global__ void __launch_bounds__(256) k_ens_energy(const Table T, const float* __restrict__ f,
                                                    double* __restrict__ part) {
    const Member& M = T.m[blockIdx.y];
    const int n = M.n, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned pitch = unsigned(M.pitch), qs = unsigned(n) * unsigned(n) * pitch;
    double s = 0;
    for (int row = blockIdx.x * 8 + warp; row < n * n; row += ENERGY_BLOCKS * 8)
        for (int x = lane; x < n; x += 32) {
            float rho, j[3];
            node_moments(f + M.off + unsigned(row) * pitch + x, qs, rho, j);
            const double a = j[0] / rho, b = j[1] / rho, c = j[2] / rho;
            s += a * a + b * b + c * c;
        }
    __shared__ double red[8];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) red[warp] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0;
        for (int w = 0; w < 8; ++w) v += red[w];
        part[blockIdx.y * ENERGY_BLOCKS + blockIdx.x] = v;
    }
}
__global__ void __launch_bounds__(32) k_ens_energy_final(const Table T, const double* __restrict__ part,
                                                         double* __restrict__ out) {
    const int mi = blockIdx.x, n = T.m[mi].n;
    double s = 0;
    for (int i = threadIdx.x; i < ENERGY_BLOCKS; i += 32) s += part[mi * ENERGY_BLOCKS + i];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) out[mi] = 0.5 * s / (double(n) * n * n);
}

/* 2x2x2 box filter of one fine member's velocity (compact [3][n][n][n]) onto
 * the coarse grid: ubar[3][nc^3], uu[6][nc^3] (xx, yy, zz, xy, xz, yz) */
__global__ void k_box_filter(const float* __restrict__ u, int n, double* __restrict__ ubar, double* __restrict__ uu) {
    const int nc = n / 2;
    const size_t cn = size_t(nc) * nc * nc, fn = size_t(n) * n * n;
    const size_t o = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (o >= cn) return;
    const int x = int(o % nc), y = int((o / nc) % nc), z = int(o / (size_t(nc) * nc));
    double s[3] = {0, 0, 0}, p[6] = {0, 0, 0, 0, 0, 0};
    for (int c = 0; c < 8; ++c) {
        const size_t i = (size_t(2 * z + (c >> 2)) * n + 2 * y + ((c >> 1) & 1)) * n + 2 * x + (c & 1);
        const double a = u[i], b = u[fn + i], d = u[2 * fn + i];
        s[0] += a, s[1] += b, s[2] += d;
        p[0] += a * a, p[1] += b * b, p[2] += d * d, p[3] += a * b, p[4] += a * d, p[5] += b * d;
    }
    for (int k = 0; k < 3; ++k) ubar[k * cn + o] = s[k] / 8;
    for (int k = 0; k < 6; ++k) uu[k * cn + o] = p[k] / 8;
}

/* training samples of the filtered member, pass 1 per coarse cell: the
 * filtered strain S (central differences, periodic) and the two
 * contractions of the least-squares eddy viscosity, tau^d : S and S : S,
 * with tau = uu - ubar ubar the filtered subgrid stress */
__global__ void k_sgs_contract(const double* __restrict__ ubar, const double* __restrict__ uu, int nc,
                               double* __restrict__ s8) {
    const size_t cn = size_t(nc) * nc * nc;
    const size_t o = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (o >= cn) return;
    const int x = int(o % nc), y = int((o / nc) % nc), z = int(o / (size_t(nc) * nc));
    auto at = [&](int k, int xx, int yy, int zz) {
        xx = (xx + nc) % nc, yy = (yy + nc) % nc, zz = (zz + nc) % nc;
        return ubar[k * cn + (size_t(zz) * nc + yy) * nc + xx];
    };
    double g[3][3];
    for (int k = 0; k < 3; ++k) {
        g[k][0] = 0.5 * (at(k, x + 1, y, z) - at(k, x - 1, y, z));
        g[k][1] = 0.5 * (at(k, x, y + 1, z) - at(k, x, y - 1, z));
        g[k][2] = 0.5 * (at(k, x, y, z + 1) - at(k, x, y, z - 1));
    }
    const double S[6] = {g[0][0], g[1][1], g[2][2], 0.5 * (g[0][1] + g[1][0]), 0.5 * (g[0][2] + g[2][0]),
                         0.5 * (g[1][2] + g[2][1])};
    const double u0 = ubar[o], u1 = ubar[cn + o], u2 = ubar[2 * cn + o];
    double tau[6] = {uu[o] - u0 * u0,          uu[cn + o] - u1 * u1,     uu[2 * cn + o] - u2 * u2,
                     uu[3 * cn + o] - u0 * u1, uu[4 * cn + o] - u0 * u2, uu[5 * cn + o] - u1 * u2};
    const double tr = (tau[0] + tau[1] + tau[2]) / 3;
    for (int k = 0; k < 3; ++k) tau[k] -= tr;
    double ts = 0, ss = 0;
    for (int k = 0; k < 6; ++k) {
        const double w = k < 3 ? 1 : 2;
        ts += w * tau[k] * S[k];
        ss += w * S[k] * S[k];
    }
    for (int k = 0; k < 6; ++k) s8[k * cn + o] = S[k];
    s8[6 * cn + o] = ts;
    s8[7 * cn + o] = ss;
}

/* pass 2: nu = max(0, -<tau^d:S> / (2 <S:S>)) with <> the 3x3x3 box average
 * (periodic), the features of p = (tau0 + 3 nu) S, and the target nu */
__global__ void k_sgs_targets(const double* __restrict__ s8, int nc, double tau0, float* __restrict__ X,
                              float* __restrict__ T) {
    const size_t cn = size_t(nc) * nc * nc;
    const size_t o = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (o >= cn) return;
    const int x = int(o % nc), y = int((o / nc) % nc), z = int(o / (size_t(nc) * nc));
    double ts = 0, ss = 0;
    for (int dz = -1; dz <= 1; ++dz)
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx) {
                const size_t i = (size_t((z + dz + nc) % nc) * nc + (y + dy + nc) % nc) * nc + (x + dx + nc) % nc;
                ts += s8[6 * cn + i];
                ss += s8[7 * cn + i];
            }
    double nu = ss > 1e-30 ? -ts / (2 * ss) : 0;
    if (nu < 0) nu = 0;
    double p[6], xf[sgs::NIN];
    for (int k = 0; k < 6; ++k) p[k] = (tau0 + 3 * nu) * s8[k * cn + o];
    sgs::features<double>(p, tau0, xf);
    for (int k = 0; k < sgs::NIN; ++k) X[o * sgs::NIN + k] = float(xf[k]);
    T[o] = float(nu);
}

__global__ void k_d2f(const double* __restrict__ a, float* __restrict__ b, size_t n) {
    const size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (i < n) b[i] = float(a[i]);
}

}  // namespace ens

/* ---- launchers */
static size_t mlp_step_smem() { return sgs::infer_dyn_smem<ens::MLP_ROWS>(); }

cudaError_t launch_ens_step(const ens::Table& T, const float* fA, float* fB, int model, const void* blob, float cs,
                            int* err, int grid, cudaStream_t s) {
    if (model == ens::SGS_MLP) {
        if (T.ty != ens::MLP_TY) return cudaErrorInvalidValue;
        const size_t smem = mlp_step_smem();
        cudaError_t e = cudaFuncSetAttribute(ens::k_ens_step_mlp, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e != cudaSuccess) return e;
        TmemLane lane(s);
        if (lane.status() != cudaSuccess) return lane.status();
        ens::k_ens_step_mlp<<<grid, ens::MLP_ROWS, smem, lane.stream()>>>(T, fA, fB, (const unsigned char*)blob, err);
        return cudaGetLastError();
    }
    if (T.ty == 4 && model == ens::SGS_NONE) return launch_pdl(ens::k_ens_step<4, ens::SGS_NONE>, grid, 128, s, T, fA, fB, cs);
    if (T.ty == 4) return launch_pdl(ens::k_ens_step<4, ens::SGS_SMAG>, grid, 128, s, T, fA, fB, cs);
    if (T.ty == 8 && model == ens::SGS_NONE) return launch_pdl(ens::k_ens_step<8, ens::SGS_NONE>, grid, 256, s, T, fA, fB, cs);
    if (T.ty == 8) return launch_pdl(ens::k_ens_step<8, ens::SGS_SMAG>, grid, 256, s, T, fA, fB, cs);
    return cudaErrorInvalidValue;
}

int ens_step_resident(int ty, int model) {
    int nb = 0, dev = 0, sms = 0;
    cudaError_t e = cudaSuccess;
    if (model == ens::SGS_MLP) {
        e = sgs::infer_resident(ens::k_ens_step_mlp, ens::MLP_ROWS, mlp_step_smem(), sgs::tmem_cols<ens::MLP_ROWS>(),
                                ens::MLP_BLOCKS, &nb);
        if (e == cudaSuccess) return nb;
        nb = 0;
    } else if (ty == 4 && model == ens::SGS_NONE) {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, ens::k_ens_step<4, ens::SGS_NONE>, 128, 0);
    } else if (ty == 4) {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, ens::k_ens_step<4, ens::SGS_SMAG>, 128, 0);
    } else if (model == ens::SGS_NONE) {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, ens::k_ens_step<8, ens::SGS_NONE>, 256, 0);
    } else {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, ens::k_ens_step<8, ens::SGS_SMAG>, 256, 0);
    }
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
        sms = 152;
    return sms * (e != cudaSuccess || nb < 1 ? 1 : nb);
}

cudaError_t launch_ens_init(const ens::Table& T, const ens::KMode* modes, float* fA, cudaStream_t s) {
    /* rows of a block: as many as 64 KB hold, so that three blocks share an
     * SM (32 at kmax 16; one row always fits: n <= 1024, kmax <= 512) */
    constexpr size_t BUDGET = 64 * 1024;
    cudaError_t e = cudaFuncSetAttribute(ens::k_ens_init, cudaFuncAttributeMaxDynamicSharedMemorySize, int(BUDGET));
    if (e != cudaSuccess) return e;
    for (int m = 0; m < T.count; ++m) {
        const ens::Member& M = T.m[m];
        const size_t table = size_t(M.n) * 2 * sizeof(double), row = size_t(M.kmax + 1) * 6 * sizeof(double);
        int rows = 32;
        while (rows > 1 && table + rows * row > BUDGET) rows /= 2;
        ens::k_ens_init<<<dim3((M.n + rows - 1) / rows, M.n), ens::INIT_THREADS, table + rows * row, s>>>(T, modes, fA,
                                                                                                    m, rows);
    }
    return cudaGetLastError();
}
cudaError_t launch_ens_init_from(const ens::Table& T, const float* u, float* fA, float* fB, cudaStream_t s) {
    ens::k_ens_init_from<<<T.ntiles, 32 * T.ty, 0, s>>>(T, u, fA, fB);
    return cudaGetLastError();
}
cudaError_t launch_ens_velocity(const ens::Table& T, const float* f, float* u, cudaStream_t s) {
    ens::k_ens_velocity<<<T.ntiles, 32 * T.ty, 0, s>>>(T, f, u);
    return cudaGetLastError();
}
cudaError_t launch_ens_energy(const ens::Table& T, const float* f, double* part, double* out, cudaStream_t s) {
    ens::k_ens_energy<<<dim3(ens::ENERGY_BLOCKS, T.count), 256, 0, s>>>(T, f, part);
    ens::k_ens_energy_final<<<T.count, 32, 0, s>>>(T, part, out);
    return cudaGetLastError();
}
cudaError_t launch_box_filter(const float* u, int n, double* ubar, double* uu, cudaStream_t s) {
    const size_t cn = size_t(n / 2) * (n / 2) * (n / 2);
    ens::k_box_filter<<<unsigned((cn + 255) / 256), 256, 0, s>>>(u, n, ubar, uu);
    return cudaGetLastError();
}
cudaError_t launch_d2f(const double* a, float* b, size_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    ens::k_d2f<<<unsigned((n + 255) / 256), 256, 0, s>>>(a, b, n);
    return cudaGetLastError();
}
cudaError_t launch_sgs_targets(const double* ubar, const double* uu, int nc, double tau0, double* s8, float* X,
                               float* T, cudaStream_t s) {
    const size_t cn = size_t(nc) * nc * nc;
    const unsigned nb = unsigned((cn + 255) / 256);
    ens::k_sgs_contract<<<nb, 256, 0, s>>>(ubar, uu, nc, s8);
    ens::k_sgs_targets<<<nb, 256, 0, s>>>(s8, nc, tau0, X, T);
    return cudaGetLastError();
}

}  // namespace lbm
