/* Training and evaluation kernels of the learned subgrid closure, and the
 * self-check of the tensor-core path.
 *
 * k_mlp_grad fuses forward, loss and backward for tiles of 64 samples, FP32
 * on the CUDA cores (the master weights, activations and sums are FP32; the
 * tensor core's formats are narrower).  Every product of a tile is a small
 * GEMM of 128 threads out of shared memory, each thread keeping a register
 * tile of 8 units x 4 samples, or 8 x 4 weights, so that a 16-byte
 * shared-memory read feeds about 11 multiply-adds (activations are stored
 * [unit][sample], weights in both orders).  Two blocks share an SM, so
 * that one computes while the other waits at a barrier.  Bound by the FP32
 * pipe and the issue slots (61 % and 73 % of their rates in the forward half);
 * packed pairs (fma.rn.f32x2) have the same FP32 rate on this chip and, with
 * the activations interleaved for them, measured slower (0.73 against 0.66 ms
 * for a million samples).  Each block writes its partial gradient; k_mlp_adam sums
 * the partials in a fixed order (so runs are reproducible) and applies one
 * Adam step.  Loss: mean squared error of o / NU_SCALE, o the network's
 * coefficient (the eddy viscosity is o * strain_gain in the collision).
 */
#include <cstdint>
#include <cuda_bf16.h>

#include "lbm_kernels.cuh"
#include "sgs_infer.cuh"
#include "sgs_mlp.cuh"
#include "tc_sm103.cuh"

namespace lbm {
namespace sgs {

constexpr int GT = 64;         /* samples per tile */
constexpr int GTH = 128;       /* threads per block */
constexpr int LS = GT + 4;     /* row stride of the activations [unit][sample]: rows 4 banks apart */
constexpr int LW = NH + 4;     /* row stride of the weights, likewise */

__device__ __forceinline__ float softplus(float y) { return y > 20.f ? y : log1pf(expf(y)); }
__device__ __forceinline__ float sigmoid(float y) { return 1.f / (1.f + expf(-y)); }

struct FwdSmem {
    float w1t[NIN * LW], w2t[NH * LW]; /* [in][out] */
    float x[NIN * LS], h1[NH * LS];
    float yp[8 * GT]; /* the output's sum, by half-warp */
    float b2[NH], w3[NH];
    float b3;
};
struct GradSmem : FwdSmem {
    alignas(16) float w2[NH * LW];              /* [out][in] */
    alignas(16) float d2[NH * LS], d1[NH * LS]; /* dL/dz2, dL/dz1 */
    alignas(16) float dy[GT];
    float red[GTH / 32][2];
};

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
/* this thread's tile in the GEMMs over units x samples: units u0 .. u0 + 7
 * (the same for a half-warp) of samples q0 .. q0 + 3 */
__device__ __forceinline__ int unit0() { return 8 * (threadIdx.x >> 4); }
__device__ __forceinline__ int sample0() { return 4 * (threadIdx.x & 15); }

__device__ __forceinline__ void fwd_weights(FwdSmem& s, const float* __restrict__ params) {
    const int t = threadIdx.x;
    for (int i = t; i < NH * NIN; i += GTH) s.w1t[(i % NIN) * LW + i / NIN] = params[OFF_W1 + i];
    for (int i = t; i < NH * NH; i += GTH) s.w2t[(i % NH) * LW + i / NH] = params[OFF_W2 + i];
    if (t < NH) {
        s.b2[t] = params[OFF_B2 + t];
        s.w3[t] = params[OFF_W3 + t];
    }
    if (t == 0) s.b3 = params[OFF_B3];
}

/* z[8][4] += sum over K of w[k][u0 + .] a[k][q0 + .] */
template <int K> __device__ __forceinline__ void gemm8x4(const float* w, const float* a, float z[8][4]) {
    const float* wp = w + unit0();
    const float* ap = a + sample0();
#pragma unroll 8
    for (int k = 0; k < K; ++k) {
        const float4 wa = ld4(wp + k * LW), wb = ld4(wp + k * LW + 4), v = ld4(ap + k * LS);
        const float wr[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            z[j][0] = fmaf(wr[j], v.x, z[j][0]);
            z[j][1] = fmaf(wr[j], v.y, z[j][1]);
            z[j][2] = fmaf(wr[j], v.z, z[j][2]);
            z[j][3] = fmaf(wr[j], v.w, z[j][3]);
        }
    }
}

/* the features of the tile's samples (thread t takes half t % 2 of sample
 * t / 2, row si of X; negative: none) into x; vec: X is 16-byte aligned
 * (every row then is) */
__device__ __forceinline__ void fwd_load(FwdSmem& s, const float* __restrict__ X, long long si, bool vec) {
    const int q = threadIdx.x >> 1, k0 = (threadIdx.x & 1) * 8;
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = 0.f;
    if (si >= 0) {
        const float* src = X + si * NIN + k0;
        if (vec) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(src)), b = __ldg(reinterpret_cast<const float4*>(src) + 1);
            v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = __ldg(src + k);
        }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) s.x[(k0 + k) * LS + q] = v[k];
}

/* both hidden layers of the tile in x: h1 in shared memory, h2 of this
 * thread's 8 units x 4 samples in registers; returns the pre-activation of
 * the output of sample threadIdx.x (threads 0 .. GT - 1) */
__device__ __forceinline__ float fwd_tile(FwdSmem& s, float h2[8][4]) {
    const int u0 = unit0(), q0 = sample0();
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) h2[j][i] = 0.f;
    gemm8x4<NIN>(s.w1t, s.x, h2);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const bool one = u0 + j == HC; /* the constant unit */
        *reinterpret_cast<float4*>(s.h1 + (u0 + j) * LS + q0) =
            make_float4(one ? 1.f : fmaxf(h2[j][0], 0.f), one ? 1.f : fmaxf(h2[j][1], 0.f),
                        one ? 1.f : fmaxf(h2[j][2], 0.f), one ? 1.f : fmaxf(h2[j][3], 0.f));
#pragma unroll
        for (int i = 0; i < 4; ++i) h2[j][i] = s.b2[u0 + j];
    }
    __syncthreads();
    gemm8x4<NH>(s.w2t, s.h1, h2);
    float y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            h2[j][i] = fmaxf(h2[j][i], 0.f);
            y[i] = fmaf(s.w3[u0 + j], h2[j][i], y[i]);
        }
    *reinterpret_cast<float4*>(s.yp + (threadIdx.x >> 4) * GT + q0) = make_float4(y[0], y[1], y[2], y[3]);
    __syncthreads();
    float z = s.b3;
    if (threadIdx.x < GT)
#pragma unroll
        for (int k = 0; k < 8; ++k) z += s.yp[k * GT + threadIdx.x];
    return z;
}

__device__ __forceinline__ float dot4(const float4& a, const float4& b, float c) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, c))));
}

/* a register tile of a weight gradient, sum over the tile's samples of
 * d[row] a[column]: rows r0 + RS m (m < R), columns c0 + CS n (n < C), added
 * to g.  A tile's products are summed on their own first: shorter chains of
 * rounding than one running sum */
template <int R, int RS, int C, int CS>
__device__ __forceinline__ void outer_tile(const float* d, int r0, const float* a, int c0, float g[R][C]) {
    float c[R][C] = {};
#pragma unroll 2
    for (int q = 0; q < GT; q += 4) {
        float4 v[C];
#pragma unroll
        for (int n = 0; n < C; ++n) v[n] = ld4(a + (c0 + CS * n) * LS + q);
#pragma unroll
        for (int m = 0; m < R; ++m) {
            const float4 e = ld4(d + (r0 + RS * m) * LS + q);
#pragma unroll
            for (int n = 0; n < C; ++n) c[m][n] = dot4(e, v[n], c[m][n]);
        }
    }
#pragma unroll
    for (int m = 0; m < R; ++m)
#pragma unroll
        for (int n = 0; n < C; ++n) g[m][n] += c[m][n];
}
template <int R, int RS, int C, int CS>
__device__ __forceinline__ void outer_store(float* out, int ld, int r0, int c0, const float g[R][C]) {
#pragma unroll
    for (int m = 0; m < R; ++m)
#pragma unroll
        for (int n = 0; n < C; ++n) out[(r0 + RS * m) * ld + c0 + CS * n] = g[m][n];
}

/* grad_part[block][NPARAM + 1]: the block's gradient sum and loss sum over
 * its samples (idx[i] selects sample i of the batch, or i itself when idx is
 * null); the loss is scaled by 1/n_total.  Measured (GB300): 1,000,003
 * samples 0.66 ms (one sample per thread with scalar shared-memory reads:
 * 2.85 ms; the FP32 peak: 0.39 ms), a batch of 16,384 24 us (69 us). */
__global__ void __launch_bounds__(GTH, 2) k_mlp_grad(const float* __restrict__ params, const float* __restrict__ X,
                                                     const float* __restrict__ T, const int* __restrict__ idx, int n,
                                                     float inv_n, float* __restrict__ grad_part, int vec) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    GradSmem& s = *reinterpret_cast<GradSmem*>(smem_raw);
    pdl_wait();
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    const int u0 = unit0(), q0 = sample0();
    fwd_weights(s, params);
    for (int i = t; i < NH * NH; i += GTH) s.w2[(i / NH) * LW + i % NH] = params[OFF_W2 + i];
    /* register tiles of the weight gradients (a warp reads 4 x 8 adjacent
     * rows, which lie in different banks) */
    const int r2 = (w >> 1) * 4 + (lane >> 3), c2 = (w & 1) * 8 + (lane & 7);
    const int r1 = w * 4 + (lane >> 3), c1 = lane & 7;
    float g2[8][4] = {}, g1[4][2] = {};
    float gw3[8] = {}, gb2[8] = {}, gl = 0.f, gd3 = 0.f;

    for (long long base = (long long)blockIdx.x * GT; base < n; base += (long long)gridDim.x * GT) {
        const long long q = base + (t >> 1);
        fwd_load(s, X, q < n ? (idx ? idx[q] : q) : -1, vec);
        float h2[8][4];
        const float y = fwd_tile(s, h2);
        if (t < GT) {
            const long long i = base + t;
            float dy = 0.f;
            if (i < n) {
                const float err = softplus(y) - T[idx ? idx[i] : i] * (1.f / NU_SCALE);
                gl += err * err * inv_n;
                dy = 2.f * err * inv_n * sigmoid(y);
            }
            s.dy[t] = dy;
            gd3 += dy;
        }
        __syncthreads();
        /* dz2 = dy w3 relu'(z2); slopes are factors, so that a dy that is not a
         * number reaches every weight */
        const float4 dy = ld4(s.dy + q0);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float w3 = s.w3[u0 + j];
            const float4 d = make_float4(dy.x * (h2[j][0] > 0.f ? w3 : 0.f), dy.y * (h2[j][1] > 0.f ? w3 : 0.f),
                                         dy.z * (h2[j][2] > 0.f ? w3 : 0.f), dy.w * (h2[j][3] > 0.f ? w3 : 0.f));
            *reinterpret_cast<float4*>(s.d2 + (u0 + j) * LS + q0) = d;
            gb2[j] += (d.x + d.y) + (d.z + d.w);
            gw3[j] += (dy.x * h2[j][0] + dy.y * h2[j][1]) + (dy.z * h2[j][2] + dy.w * h2[j][3]);
        }
        __syncthreads();
        /* dz1 = (W2^T dz2) relu'(z1) */
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) h2[j][i] = 0.f;
        gemm8x4<NH>(s.w2, s.d2, h2);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float4 h = ld4(s.h1 + (u0 + j) * LS + q0);
            const bool on = u0 + j != HC;
            *reinterpret_cast<float4*>(s.d1 + (u0 + j) * LS + q0) =
                make_float4(h2[j][0] * (on && h.x > 0.f ? 1.f : 0.f), h2[j][1] * (on && h.y > 0.f ? 1.f : 0.f),
                            h2[j][2] * (on && h.z > 0.f ? 1.f : 0.f), h2[j][3] * (on && h.w > 0.f ? 1.f : 0.f));
        }
        outer_tile<8, 8, 4, 16>(s.d2, r2, s.h1, c2, g2); /* dW2 = dz2 h1^T */
        __syncthreads();
        outer_tile<4, 16, 2, 8>(s.d1, r1, s.x, c1, g1); /* dW1 = dz1 x^T */
        __syncthreads();
    }
    float* out = grad_part + size_t(blockIdx.x) * (NPARAM + 1);
    outer_store<8, 8, 4, 16>(out + OFF_W2, NH, r2, c2, g2);
    outer_store<4, 16, 2, 8>(out + OFF_W1, NIN, r1, c1, g1);
    /* the sums over samples: the 16 lanes of a half-warp (loss and db3: the
     * warp), then for loss and db3 the warps */
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (o < 16) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                gb2[j] += __shfl_xor_sync(0xffffffffu, gb2[j], o);
                gw3[j] += __shfl_xor_sync(0xffffffffu, gw3[j], o);
            }
        }
        gl += __shfl_xor_sync(0xffffffffu, gl, o);
        gd3 += __shfl_xor_sync(0xffffffffu, gd3, o);
    }
    if (q0 == 0) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            out[OFF_B2 + u0 + j] = gb2[j];
            out[OFF_W3 + u0 + j] = gw3[j];
        }
    }
    if (lane == 0) {
        s.red[w][0] = gl;
        s.red[w][1] = gd3;
    }
    __syncthreads();
    if (t == 0) {
        float l = 0.f, d = 0.f;
        for (int k = 0; k < GT / 32; ++k) {
            l += s.red[k][0];
            d += s.red[k][1];
        }
        out[NPARAM] = l;
        out[OFF_B3] = d;
    }
}
/* sum the block partials in a fixed order (16 warps take every 16th, then
 * the 16 sums in turn; a warp reads 32 adjacent parameters); optionally one
 * Adam step */
constexpr int ADAM_WARPS = 16;
__global__ void __launch_bounds__(32 * ADAM_WARPS) k_mlp_adam(const float* __restrict__ grad_part, int nblocks,
                                                              float* __restrict__ params, float* __restrict__ m,
                                                              float* __restrict__ v, float* __restrict__ grad_out,
                                                              float* __restrict__ loss_out, float lr, float b1,
                                                              float b2, float eps, int step) {
    __shared__ float part[ADAM_WARPS][32];
    pdl_wait();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p = blockIdx.x * 32 + lane;
    float g = 0.f;
    if (p <= NPARAM)
#pragma unroll 8
        for (int b = w; b < nblocks; b += ADAM_WARPS) g += grad_part[size_t(b) * (NPARAM + 1) + p];
    part[w][lane] = g;
    __syncthreads();
    if (w > 0 || p > NPARAM) return;
    for (int k = 1; k < ADAM_WARPS; ++k) g += part[k][lane];
    if (p == NPARAM) {
        if (loss_out) *loss_out = g;
        return;
    }
    if (grad_out) grad_out[p] = g;
    if (step > 0) {
        const float mm = b1 * m[p] + (1.f - b1) * g;
        const float vv = b2 * v[p] + (1.f - b2) * g * g;
        m[p] = mm;
        v[p] = vv;
        const float mh = mm / (1.f - powf(b1, float(step)));
        const float vh = vv / (1.f - powf(b2, float(step)));
        params[p] -= lr * mh / (sqrtf(vh) + eps);
    }
}

/* the coefficient of n samples (FP32, CUDA cores): the forward half of
 * k_mlp_grad.  Measured at 1,000,003 samples: 0.21 ms (one sample per
 * thread, its hidden layer in local memory: 372 us) */
__global__ void __launch_bounds__(GTH) k_mlp_predict(const float* __restrict__ params, const float* __restrict__ X,
                                                     int n, float* __restrict__ nu, int vec) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FwdSmem& s = *reinterpret_cast<FwdSmem*>(smem_raw);
    fwd_weights(s, params);
    for (long long base = (long long)blockIdx.x * GT; base < n; base += (long long)gridDim.x * GT) {
        const long long q = base + (threadIdx.x >> 1);
        fwd_load(s, X, q < n ? q : -1, vec);
        float h2[8][4];
        const float y = fwd_tile(s, h2);
        if (threadIdx.x < GT && base + threadIdx.x < n) nu[base + threadIdx.x] = NU_SCALE * softplus(y);
        /* the next tile's x is not read before the barrier in fwd_tile, and
         * this tile's was last read before it; yp is rewritten two barriers on */
    }
}

/* ---- the mini-batch shuffle: Fisher-Yates, for i = n - 1 .. 1 swap elements
 * i and H[i] = r_i mod (i + 1), r_i the i-th draw of splitmix64 (a counter
 * generator: any draw by itself), with the result of the sequential loop.
 *
 * Swaps of disjoint elements commute, so a swap may go ahead once no earlier
 * one (a larger i) that touches its elements is still due.  In a round every
 * swap still due enters its i at both of its elements (atomicMax) and goes
 * ahead if it finds itself at both (Shun, Gu, Blelloch, Fineman and Gibbons,
 * "Sequential random permutation, list contraction and tree contraction are
 * highly parallel", SODA 2015: O(log n) rounds).  A round's entries carry its
 * number above the i, so that R need not be cleared.  SHUFFLE_ROUNDS rounds run
 * over the whole chip, each on the list of swaps the one before left; a
 * single block finishes the few after them.  On the host (one division and
 * two random accesses per element, then a copy to the device) 262,144
 * elements took 1.1 ms, here 0.1 ms */
constexpr int SHUFFLE_ROUNDS = 24;
using U64 = unsigned long long;

__device__ __forceinline__ GridWalk my_walk() { return grid_walk(blockIdx.x, gridDim.x, threadIdx.x, blockDim.x); }

__global__ void k_shuffle_draw(int* __restrict__ H, int n, U64 state) {
    for (GridWalk w = my_walk(); w.at < unsigned(n); w.at += w.step) {
        const int i = int(w.at);
        U64 z = state + U64(n - i) * 0x9E3779B97F4A7C15ull;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        if (i > 0) H[i] = int((z ^ (z >> 31)) % (U64(i) + 1));
    }
}

__device__ __forceinline__ void shuffle_enter(const int* __restrict__ H, U64* __restrict__ R, int i, U64 round) {
    atomicMax(R + i, round << 32 | U64(i));
    atomicMax(R + H[i], round << 32 | U64(i));
}
/* the swap of i, if it is its turn */
__device__ __forceinline__ bool shuffle_swap(const int* __restrict__ H, const U64* __restrict__ R, int* perm, int i,
                                             U64 round) {
    const int h = H[i];
    const U64 v = round << 32 | U64(i);
    if (__ldcg(R + i) != v || __ldcg(R + h) != v) return false;
    const int a = __ldcg(perm + i);
    perm[i] = __ldcg(perm + h);
    perm[h] = a;
    return true;
}

/* the swaps due in a round: list[0 .. *count), or all of 1 .. n - 1 */
__global__ void k_shuffle_enter(const int* __restrict__ H, U64* __restrict__ R, const int* __restrict__ list,
                                const int* __restrict__ count, int n, U64 round) {
    pdl_wait();
    const int m = list ? __ldcg(count) : n - 1;
    for (GridWalk w = my_walk(); w.at < unsigned(m); w.at += w.step)
        shuffle_enter(H, R, list ? __ldcg(list + w.at) : int(w.at) + 1, round);
}
__global__ void k_shuffle_swap(const int* __restrict__ H, const U64* __restrict__ R, int* perm,
                               const int* __restrict__ list, const int* __restrict__ count, int n, U64 round,
                               int* __restrict__ left, int* __restrict__ left_count) {
    pdl_wait();
    const int m = list ? __ldcg(count) : n - 1;
    for (GridWalk w = my_walk(); w.at < unsigned(m); w.at += w.step) {
        const int i = list ? __ldcg(list + w.at) : int(w.at) + 1;
        const bool due = !shuffle_swap(H, R, perm, i, round);
        const unsigned who = __activemask(), ask = __ballot_sync(who, due);
        if (!due) continue;
        const int lane = threadIdx.x & 31, first = __ffs(ask) - 1;
        int base = 0;
        if (lane == first) base = atomicAdd(left_count, __popc(ask));
        base = __shfl_sync(ask, base, first);
        left[base + __popc(ask & ((1u << lane) - 1u))] = i;
    }
}
/* the rounds after SHUFFLE_ROUNDS, one block; every round does at least the
 * swap of the largest i, so it ends after at most as many as swaps are left */
__global__ void __launch_bounds__(1024) k_shuffle_rest(const int* __restrict__ H, U64* __restrict__ R, int* perm,
                                                       int* list, int* other, const int* __restrict__ count, U64 round) {
    pdl_wait();
    __shared__ int left;
    int m = __ldcg(count);
    for (; m > 0; ++round) {
        for (long long j = threadIdx.x; j < m; j += blockDim.x) shuffle_enter(H, R, __ldcg(list + j), round);
        if (threadIdx.x == 0) left = 0;
        __threadfence();
        __syncthreads();
        for (long long j = threadIdx.x; j < m; j += blockDim.x) {
            const int i = __ldcg(list + j);
            if (!shuffle_swap(H, R, perm, i, round)) other[atomicAdd(&left, 1)] = i;
        }
        __threadfence();
        __syncthreads();
        m = left;
        __syncthreads();
        int* const t = list;
        list = other;
        other = t;
    }
}
__global__ void k_iota(int* p, int n) {
    for (GridWalk w = my_walk(); w.at < unsigned(n); w.at += w.step) p[w.at] = int(w.at);
}

/* ---- tensor-core self-check: D[128][64] = A[128][K] B[64][K]^T, K = 16 * kc */
__global__ void __launch_bounds__(128) k_tc_selftest(const __nv_bfloat16* __restrict__ A,
                                                     const __nv_bfloat16* __restrict__ B, int kc,
                                                     float* __restrict__ D, int* __restrict__ err) {
    __shared__ __align__(1024) unsigned char sa[128 * 64 * 2];
    __shared__ __align__(1024) unsigned char sb[64 * 64 * 2];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tslot;
    const int t = threadIdx.x, warp = t >> 5;
    const int K = 16 * kc;
    const uint32_t lbo = 128, sbo = uint32_t(K / 8) * 128;
    /* operands into the core-matrix layout, 16 bytes (8 bf16) at a time */
    for (int k8 = 0; k8 < K / 8; ++k8) {
        *reinterpret_cast<uint4*>(sa + tc::core_off(t, k8 * 8, lbo, sbo)) =
            *reinterpret_cast<const uint4*>(A + size_t(t) * K + k8 * 8);
        if (t < 64)
            *reinterpret_cast<uint4*>(sb + tc::core_off(t, k8 * 8, lbo, sbo)) =
                *reinterpret_cast<const uint4*>(B + size_t(t) * K + k8 * 8);
    }
#if defined(__CUDA_ARCH__)
    if (t == 0) tc::mbar_init(&mbar, 1);
    if (warp == 0) tc::tmem_alloc(&tslot, 64);
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tm = tslot;
    if (t == 0) {
        const uint32_t id = tc::idesc_bf16_f32(128, 64);
        for (int c = 0; c < kc; ++c)
            tc::mma_bf16(tm, tc::sdesc(tc::smem_u32(sa) + c * 2 * lbo, lbo, sbo),
                         tc::sdesc(tc::smem_u32(sb) + c * 2 * lbo, lbo, sbo), id, c > 0);
        tc::mma_commit(&mbar);
    }
    const bool ok = __syncthreads_and(tc::mbar_wait(&mbar, 0, 1u << 22));
    tc::fence_after_sync();
    if (ok) {
        uint32_t r[64];
        const uint32_t ta = tm + (uint32_t(warp * 32) << 16);
#pragma unroll
        for (int c = 0; c < 4; ++c) tc::tmem_ld16(ta + 16 * c, r + 16 * c);
        tc::tmem_wait_ld();
        tc::tmem_fence_regs<64>(r);
#pragma unroll
        for (int c = 0; c < 64; ++c) D[size_t(t) * 64 + c] = __uint_as_float(r[c]);
    } else if (t == 0) {
        atomicExch(err, 1);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tm, 64);
#endif
}

/* nu_t of n samples through the tensor-core inference path (the one the
 * collide kernels use): persistent blocks of 128 rows */
__global__ void __launch_bounds__(128) k_mlp_predict_tc(const unsigned char* __restrict__ blob,
                                                        const float* __restrict__ X, int n, float* __restrict__ nu,
                                                        int* __restrict__ err) {
    extern __shared__ __align__(128) unsigned char dsm[];
#if defined(__CUDA_ARCH__)
    InferSmem<128>& s = *reinterpret_cast<InferSmem<128>*>(dsm);
    infer_setup<128>(s, blob);
    /* the block's tiles: the same number of passes for all of its threads */
    for (GridWalk w = grid_walk(blockIdx.x, gridDim.x, 0, 128); w.at < unsigned(n); w.at += w.step) {
        const long long i = w.at + threadIdx.x;
        float x[NIN];
#pragma unroll
        for (int k = 0; k < NIN; ++k) x[k] = i < n ? X[i * NIN + k] : 0.f;
        const float v = infer_nu<128>(s, x, err);
        if (v < 0.f) break; /* a tensor-core wait ran out (block-uniform) */
        if (i < n) nu[i] = v;
    }
    infer_teardown<128>(s);
#endif
}

}  // namespace sgs

/* ---- launchers */
/* two blocks (98 KB of shared memory) per SM of a 152-SM GB300 */
int mlp_grad_blocks(int n) {
    const long long b = ((long long)n + sgs::GT - 1) / sgs::GT;
    return b < 1 ? 1 : (b > 152 * 2 ? 152 * 2 : int(b));
}

static int vec16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

cudaError_t launch_mlp_grad(const float* params, const float* X, const float* T, const int* idx, int n,
                            float* grad_part, int nblocks, cudaStream_t s) {
    const size_t sm = sizeof(sgs::GradSmem);
    cudaError_t e = cudaFuncSetAttribute(sgs::k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm));
    if (e != cudaSuccess) return e;
    const float inv_n = 1.f / float(n > 0 ? n : 1);
    return launch_pdl_if(true, sgs::k_mlp_grad, nblocks, sgs::GTH, sm, s, params, X, T, idx, n, inv_n, grad_part,
                         vec16(X));
}

cudaError_t launch_mlp_adam(const float* grad_part, int nblocks, float* params, float* m, float* v, float* grad_out,
                            float* loss_out, float lr, int step, cudaStream_t s) {
    const int n = sgs::NPARAM + 1;
    return launch_pdl(sgs::k_mlp_adam, (n + 31) / 32, 32 * sgs::ADAM_WARPS, s, grad_part, nblocks, params, m, v,
                      grad_out, loss_out, lr, 0.9f, 0.999f, 1e-8f, step);
}

cudaError_t launch_mlp_predict(const float* params, const float* X, int n, float* nu, cudaStream_t s) {
    const size_t sm = sizeof(sgs::FwdSmem);
    cudaError_t e = cudaFuncSetAttribute(sgs::k_mlp_predict, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm));
    if (e != cudaSuccess) return e;
    /* 4 resident blocks (46 KB) per SM */
    const long long tiles = ((long long)n + sgs::GT - 1) / sgs::GT;
    const int b = tiles < 1 ? 1 : tiles > 152 * 4 ? 152 * 4 : int(tiles);
    sgs::k_mlp_predict<<<b, sgs::GTH, sm, s>>>(params, X, n, nu, vec16(X));
    return cudaGetLastError();
}

size_t shuffle_scratch_bytes(int n) {
    return size_t(n) * (sizeof(sgs::U64) + 3 * sizeof(int)) + (sgs::SHUFFLE_ROUNDS + 1) * sizeof(int);
}

cudaError_t launch_shuffle(int* perm, int n, unsigned long long state, int epoch, void* scratch, cudaStream_t s) {
    using sgs::U64;
    const int wide = sgs::groups_of(n, 256, 152 * 8);
    U64* R = static_cast<U64*>(scratch);
    int* H = reinterpret_cast<int*>(R + n);
    int *list = H + n, *other = list + n, *count = other + n;
    cudaError_t e = cudaMemsetAsync(count, 0, (sgs::SHUFFLE_ROUNDS + 1) * sizeof(int), s);
    if (epoch == 0) sgs::k_iota<<<wide, 256, 0, s>>>(perm, n);
    /* round numbers have 32 bits: 2^20 for each of 2^12 epochs (some 2.7 ln n
     * are needed), then R is cleared */
    const int era = epoch & 4095;
    if (era == 0 && e == cudaSuccess) e = cudaMemsetAsync(R, 0, size_t(n) * sizeof(U64), s);
    if (e != cudaSuccess) return e;
    sgs::k_shuffle_draw<<<wide, 256, 0, s>>>(H, n, state);
    U64 round = (U64(era) << 20) + 1;
    const int* from = nullptr;
    for (int r = 0; r < sgs::SHUFFLE_ROUNDS && e == cudaSuccess; ++r, ++round) {
        e = launch_pdl(sgs::k_shuffle_enter, wide, 256, s, H, R, from, count + r, n, round);
        if (e == cudaSuccess)
            e = launch_pdl(sgs::k_shuffle_swap, wide, 256, s, H, R, perm, from, count + r, n, round, list, count + r + 1);
        from = list;
        int* const t = list;
        list = other;
        other = t;
    }
    /* `other` is the list that the last round wrote */
    if (e == cudaSuccess)
        e = launch_pdl(sgs::k_shuffle_rest, 1, 1024, s, H, R, perm, other, list, count + sgs::SHUFFLE_ROUNDS, round);
    return e;
}

cudaError_t launch_mlp_predict_tc(const void* blob, const float* X, int n, float* nu, int* err, cudaStream_t s) {
    const int b = sgs::groups_of(n, 128, 152 * 4);
    const size_t smem = sgs::infer_dyn_smem<128>();
    const cudaError_t attr = cudaFuncSetAttribute(sgs::k_mlp_predict_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (attr != cudaSuccess) return attr;
    TmemLane lane(s);
    if (lane.status() != cudaSuccess) return lane.status();
    sgs::k_mlp_predict_tc<<<b, 128, smem, lane.stream()>>>((const unsigned char*)blob, X, n, nu, err);
    return cudaGetLastError();
}

cudaError_t launch_tc_selftest(const void* A, const void* B, int kc, float* D, int* err, cudaStream_t s) {
    if (kc < 1 || kc > 4) return cudaErrorInvalidValue;
    TmemLane lane(s);
    if (lane.status() != cudaSuccess) return lane.status();
    sgs::k_tc_selftest<<<1, 128, 0, lane.stream()>>>((const __nv_bfloat16*)A, (const __nv_bfloat16*)B, kc, D, err);
    return cudaGetLastError();
}

}  // namespace lbm
