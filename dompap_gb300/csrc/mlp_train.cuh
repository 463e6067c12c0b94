// mlp_train.cuh — training and batch evaluation of the pair surrogate
// (statically compiled; included by dompap_gpu.cu after mlp_common.cuh).
//
// Parameters (fp32 masters, flat, DP_MLP_NPARAM): w1[64], b1[64],
// W2[64][64] (row = output unit), b2[64], W3[2][64], b3[2]. The forward pass
// uses bf16-rounded W2 (the tensor-core operand; quantisation-aware
// training) and fp32 biases; w1 and W3 feed float32 FMAs and stay fp32 unless
// DP_MLP_SCALAR_BF16 is 1. Loss per sample: (y0 - t0)^2 + wf (y1 - t1)^2,
// averaged over the batch.
#pragma once

#ifndef DP_MLP_SCALAR_BF16
#define DP_MLP_SCALAR_BF16 0
#endif

#define DP_MLP_NPARAM (64 + 64 + 64 * 64 + 64 + 2 * 64 + 2)
#define DP_MLP_OFF_W1 0
#define DP_MLP_OFF_B1 64
#define DP_MLP_OFF_W2 128
#define DP_MLP_OFF_B2 (128 + 4096)
#define DP_MLP_OFF_W3 (128 + 4096 + 64)
#define DP_MLP_OFF_B3 (128 + 4096 + 64 + 128)

__device__ __forceinline__ float dp_round_bf16(float v) {
    const uint32_t p = dp_pack_bf16(v, 0.0f);
    return dp_bf16_lo_as_float(p);
}

// masters + normalisation -> the device struct used by every forward pass
__global__ void k_mlp_pack(const float* __restrict__ p, const float* __restrict__ norm, dp_mlp_dev* m,
                           uint32_t* __restrict__ w2t) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < 64) {
        const float w1 = p[DP_MLP_OFF_W1 + t], w30 = p[DP_MLP_OFF_W3 + t], w31 = p[DP_MLP_OFF_W3 + 64 + t];
        m->w1[t] = DP_MLP_SCALAR_BF16 ? dp_round_bf16(w1) : w1;
        m->b1[t] = p[DP_MLP_OFF_B1 + t];
        m->b2[t] = p[DP_MLP_OFF_B2 + t];
        m->w3[0][t] = DP_MLP_SCALAR_BF16 ? dp_round_bf16(w30) : w30;
        m->w3[1][t] = DP_MLP_SCALAR_BF16 ? dp_round_bf16(w31) : w31;
    }
    if (t < 2) m->b3[t] = p[DP_MLP_OFF_B3 + t];
    if (t == 0) {
        m->x_mean = norm[0];
        m->x_inv_scale = norm[1];
        m->u_scale = norm[2];
        m->f_scale = norm[3];
    }
    // B fragments of W2: [kt][nt][lane][2]; B[k][n] = W2[n][k]
    if (t < 4 * 8 * 32) {
        const int lane = t & 31, nt = (t >> 5) & 7, kt = t >> 8;
        const int n = nt * 8 + (lane >> 2), k = kt * 16 + 2 * (lane & 3);
        const float* w = p + DP_MLP_OFF_W2 + n * 64;
        m->w2frag[t * 2 + 0] = dp_pack_bf16(w[k], w[k + 1]);
        m->w2frag[t * 2 + 1] = dp_pack_bf16(w[k + 8], w[k + 9]);
        // and of its transpose (backward product dz2 W2): B[n][k] = W2[n][k]
        const float* wt = p + DP_MLP_OFF_W2 + k * 64 + n;
        w2t[t * 2 + 0] = dp_pack_bf16(wt[0], wt[64]);
        w2t[t * 2 + 1] = dp_pack_bf16(wt[8 * 64], wt[9 * 64]);
    }
}

// y (n x 2) for inputs s (n); 8 warps per block, 16 samples per warp tile.
template <bool ACCURATE>
__global__ void __launch_bounds__(256) k_mlp_eval(const float* __restrict__ s, long long n, const dp_mlp_dev* mdev,
                                                   float* __restrict__ y) {
    __shared__ dp_mlp_dev m;
    dp_mlp_load(&m, mdev);
    __syncthreads();
    const int lane = threadIdx.x & 31, g = lane >> 2;
    const long long tiles = (n + 15) / 16;
    for (long long tile = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); tile < tiles; tile += (long long)gridDim.x * 8) {
        const long long r0 = tile * 16 + g, r1 = r0 + 8;
        const float sg = r0 < n ? s[r0] : m.x_mean;
        const float sg8 = r1 < n ? s[r1] : m.x_mean;
        float out[2][2];
        dp_mlp_tile<ACCURATE>(m, sg, sg8, out);
        if ((lane & 3) == 0) {
            if (r0 < n) {
                y[2 * r0] = out[0][0];
                y[2 * r0 + 1] = out[0][1];
            }
            if (r1 < n) {
                y[2 * r1] = out[1][0];
                y[2 * r1 + 1] = out[1][1];
            }
        }
    }
}

// Gradient of the batch loss: forward on tensor cores (as inference), the
// backward GEMMs dW2 = dZ2^T H1 and dH1 = dZ2 W2 as bf16 mma.sync with fp32
// accumulation. Every sum across 16-row tiles and CTAs is taken in 64-bit fixed
// point (integer adds are exact, so the result does not depend on their order
// and training is reproducible for a seed): in registers for dW2, one slot per
// warp in shared memory for the rest, then one atomic per CTA and parameter
// into gradfx[]. Samples: drawn in the kernel (draw != 0) or s[b], b < batch.
//
// Bound by latency (one wave of CTAs, a chain of small products per tile; the
// tensor pipe idles), so what counts is the length of that chain and of the
// step. A CTA takes 128 rows, a warp a 16-row tile of the forward pass and of
// dH1, whose operands come straight from the accumulator registers (the C
// layout of one product is the A layout of the next). dW2 is split over the
// warps by output tile instead: each owns a 16 x 32 piece of it for all 128
// rows (operands by ldmatrix.trans), so no two warps add to the same element.
// Sums over the rows of a tile halve the values with each exchange (14
// shuffles per quantity and not 48) in the same tree. Batch 16,384, a
// step of a 64-step call: 62 us before (64-bit shared-memory atomics per tile,
// seven launches a step), 18 us now (two launches, k_mlp_grad and k_mlp_update,
// and the conversions of dp_fx), every weight bit for bit as before.
struct MlpTrainArgs {
    const float* s;
    const float2* t;
    long long batch;
    const dp_mlp_dev* mdev;
    const uint32_t* w2t;               // B fragments of W2 transposed (bf16)
    unsigned long long* gradfx;        // DP_MLP_NPARAM, fixed point 2^DP_MLP_GRAD_FX_BITS
    unsigned long long* lossfx;        // sum of per-sample losses, fixed point 2^DP_MLP_LOSS_FX_BITS
    float wf;
    float inv_batch;
    int draw;                          // 1: sample b is s[i], i drawn from (seed, step, b)
    unsigned long long n;              // size of the training set
    unsigned long long seed;
    long long step;
};

#define DP_MLP_GRAD_FX_BITS 36
#define DP_MLP_LOSS_FX_BITS 32

// v as a two's-complement fixed-point integer 2^BITS v, rounded to nearest even
// (saturating; a gradient beyond 2^(63-BITS) means the training has diverged
// anyway). A conversion to 64 bits runs on this GPU's float64 pipe at 1/64 rate;
// with 141 of them a group of rows that pipe was busy in 51 % of the active cycles
// (35 % of the kernel's time). A float below 2^31 converts in 32 bits, a larger
// one is an integer and only shifted: the same integer for every float. 64 steps
// of batch 16,384, the whole call: 1,390 us before, 1,150 us now.
template <int BITS>
__device__ __forceinline__ unsigned long long dp_fx(float v) {
    const float x = v * (float)(1ull << BITS);
    if (fabsf(x) <= 2147483520.0f) return (unsigned long long)(long long)__float2int_rn(x);
    const uint32_t b = __float_as_uint(x);
    const int e = (int)((b >> 23) & 0xFFu) - 150;  // x = m 2^e, e >= 8
    if (e > 39) return (unsigned long long)__float2ll_rn(x);  // out of range, infinite, not a number
    const unsigned long long m = (unsigned long long)((b & 0x7FFFFFu) | 0x800000u) << e;
    return (b >> 31) ? 0ull - m : m;
}

// Programmatic dependent launch: the next kernel's blocks may be placed now;
// and: wait until every kernel this one depends on has finished.
__device__ __forceinline__ void dp_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void dp_grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Minibatch sample b of one training step (Philox).
__device__ __forceinline__ long long dp_mlp_draw(long long b, unsigned long long n, unsigned long long seed,
                                                 long long step) {
    const uint4 r = dp_philox4x32_10(make_uint4((uint32_t)b, (uint32_t)step, (uint32_t)(step >> 32), 0x6d6c7031u),
                                     make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)));
    const unsigned long long v = ((unsigned long long)r.x << 32) | r.y;
    return (long long)(v % n);
}

// Four 8 x 8 bf16 matrices from shared memory, each transposed.
__device__ __forceinline__ void dp_ldmatrix4_trans(uint32_t* r, const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

// Sum over the 8 row groups (lanes with equal lane & 3) of the 16 values
// v[2 nt + e] a lane holds; afterwards v[0], v[1] are the sums of e = 0, 1 for
// nt = dp_mlp_owned_nt(lane). The additions pair up as in a butterfly over
// 4, 8, 16.
__device__ __forceinline__ void dp_mlp_group_sums(float* v, int lane) {
#pragma unroll
    for (int half = 8, o = 4; half >= 2; half >>= 1, o <<= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int t = 0; t < half; ++t) {
            const float send = up ? v[t] : v[t + half];
            const float keep = up ? v[t + half] : v[t];
            v[t] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
}
__device__ __forceinline__ int dp_mlp_owned_nt(int lane) {
    return ((lane >> 2) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 4) & 1);
}

#define DP_MLP_ROWS 128  // rows of one CTA: 8 warps x 16
#define DP_MLP_LD 72     // padded row of the staged dz2 and h1 (bf16): ldmatrix rows fall into distinct banks
// per-warp fixed-point sums: gw1[64], gb1[64], gb2[64], gw3[2][64], gb3[2], loss
#define DP_MLP_SUMS (5 * 64 + 3)

struct MlpGradShared {
    dp_mlp_dev m;
    uint32_t w2t[4 * 8 * 32 * 2];
    __nv_bfloat16 dz[DP_MLP_ROWS * DP_MLP_LD];
    __nv_bfloat16 h1[DP_MLP_ROWS * DP_MLP_LD];
    unsigned long long sums[8][DP_MLP_SUMS + 1];
};
// dynamic shared memory of k_mlp_grad (bytes)
#define DP_MLP_GRAD_SMEM ((int)sizeof(MlpGradShared))

template <bool ACCURATE>
__global__ void __launch_bounds__(256, 1) k_mlp_grad(MlpTrainArgs a) {
    extern __shared__ __align__(16) unsigned char dp_grad_smem[];
    MlpGradShared& S = *(MlpGradShared*)dp_grad_smem;
    constexpr int GB = DP_MLP_GRAD_FX_BITS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = 2 * (lane & 3);
    dp_launch_dependents();
    const long long groups = (a.batch + DP_MLP_ROWS - 1) / DP_MLP_ROWS;
    unsigned long long sw2[4][4];  // dW2, rows 16 (warp / 2) + g (+ 8), columns 32 (warp & 1) + 8 q + c (+ 1)
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) sw2[q][e] = 0ull;
    // this lane's pieces of gw1, gb1, gb2, gw3[0], gw3[1]: two columns each
    unsigned long long sv[5][2];
#pragma unroll
    for (int q = 0; q < 5; ++q) sv[q][0] = sv[q][1] = 0ull;
    unsigned long long sb3[2] = {0ull, 0ull}, sloss = 0ull;
    bool loaded = false;
    for (long long group = blockIdx.x; group < groups; group += gridDim.x) {
        const long long b0 = group * DP_MLP_ROWS + warp * 16 + g, b1 = b0 + 8;
        const bool v0 = b0 < a.batch, v1 = b1 < a.batch;
        const long long i0 = !v0 ? 0 : (a.draw ? dp_mlp_draw(b0, a.n, a.seed, a.step) : b0);
        const long long i1 = !v1 ? 0 : (a.draw ? dp_mlp_draw(b1, a.n, a.seed, a.step) : b1);
        const float in0 = a.s[i0], in1 = a.s[i1];
        const float2 t0 = v0 ? a.t[i0] : make_float2(0.f, 0.f), t1 = v1 ? a.t[i1] : make_float2(0.f, 0.f);
        if (!loaded) {  // the samples do not depend on the step before; the network does
            dp_grid_wait();
            dp_mlp_load(&S.m, a.mdev);
            for (int t = threadIdx.x; t < 4 * 8 * 32 * 2; t += blockDim.x) S.w2t[t] = a.w2t[t];
            loaded = true;
        }
        __syncthreads();  // the network is there; the last group's dz2, h1 have been read
        const dp_mlp_dev& m = S.m;
        const float sg = v0 ? in0 : m.x_mean, sg8 = v1 ? in1 : m.x_mean;
        const float xg = (sg - m.x_mean) * m.x_inv_scale, xg8 = (sg8 - m.x_mean) * m.x_inv_scale;
        __nv_bfloat16* rows_dz = S.dz + (warp * 16 + g) * DP_MLP_LD + c;
        __nv_bfloat16* rows_h1 = S.h1 + (warp * 16 + g) * DP_MLP_LD + c;
        // layer 1; h1[nt] at columns nt * 8 + c + e, rows g (e) and g + 8 (2 + e)
        float h1[8][4];
        uint32_t ahi[4][4], alo[4][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const int col = nt * 8 + c;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                h1[nt][e] = dp_mlp_act<ACCURATE>(fmaf(m.w1[col + e], xg, m.b1[col + e]));
                h1[nt][2 + e] = dp_mlp_act<ACCURATE>(fmaf(m.w1[col + e], xg8, m.b1[col + e]));
            }
            const int kt = nt >> 1, half = 2 * (nt & 1);
            dp_split2(h1[nt][0], h1[nt][1], ahi[kt][half], alo[kt][half]);
            dp_split2(h1[nt][2], h1[nt][3], ahi[kt][half + 1], alo[kt][half + 1]);
            *(uint32_t*)(rows_h1 + nt * 8) = ahi[kt][half];
            *(uint32_t*)(rows_h1 + 8 * DP_MLP_LD + nt * 8) = ahi[kt][half + 1];
        }
        float h2[8][4];
        dp_mlp_layer2(m, ahi, alo, h2);
        float p00 = 0.f, p01 = 0.f, p10 = 0.f, p11 = 0.f;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) h2[nt][e] = dp_mlp_act<ACCURATE>(h2[nt][e]);
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int col = nt * 8 + c + e;
                p00 = fmaf(h2[nt][e], m.w3[0][col], p00);
                p01 = fmaf(h2[nt][e], m.w3[1][col], p01);
                p10 = fmaf(h2[nt][2 + e], m.w3[0][col], p10);
                p11 = fmaf(h2[nt][2 + e], m.w3[1][col], p11);
            }
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
            p00 += __shfl_xor_sync(0xffffffffu, p00, o);
            p01 += __shfl_xor_sync(0xffffffffu, p01, o);
            p10 += __shfl_xor_sync(0xffffffffu, p10, o);
            p11 += __shfl_xor_sync(0xffffffffu, p11, o);
        }
        const float e00 = v0 ? p00 + m.b3[0] - t0.x : 0.f, e01 = v0 ? p01 + m.b3[1] - t0.y : 0.f;
        const float e10 = v1 ? p10 + m.b3[0] - t1.x : 0.f, e11 = v1 ? p11 + m.b3[1] - t1.y : 0.f;
        if ((lane & 3) == 0)
            sloss += dp_fx<DP_MLP_LOSS_FX_BITS>(e00 * e00 + a.wf * e01 * e01 + e10 * e10 + a.wf * e11 * e11);
        // dL/dy (mean over the batch)
        const float d00 = 2.f * e00 * a.inv_batch, d01 = 2.f * a.wf * e01 * a.inv_batch;
        const float d10 = 2.f * e10 * a.inv_batch, d11 = 2.f * a.wf * e11 * a.inv_batch;
        // gb3: sum over the 16 rows (one quad lane per group contributes)
        float sb30 = (lane & 3) == 0 ? d00 + d10 : 0.f, sb31 = (lane & 3) == 0 ? d01 + d11 : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sb30 += __shfl_xor_sync(0xffffffffu, sb30, o);
            sb31 += __shfl_xor_sync(0xffffffffu, sb31, o);
        }
        sb3[0] += dp_fx<GB>(sb30);
        sb3[1] += dp_fx<GB>(sb31);
        // dz2 = (dy0 w3[0] + dy1 w3[1]) * act'(z2); gw3, gb2
        float dz[8][4], t16[16];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int col = nt * 8 + c + e;
                const float hg = h2[nt][e], hg8 = h2[nt][2 + e];
                dz[nt][e] = (d00 * m.w3[0][col] + d01 * m.w3[1][col]) * (1.f - hg * hg);
                dz[nt][2 + e] = (d10 * m.w3[0][col] + d11 * m.w3[1][col]) * (1.f - hg8 * hg8);
            }
        }
        auto add = [&](int which) {
            dp_mlp_group_sums(t16, lane);
            sv[which][0] += dp_fx<GB>(t16[0]);
            sv[which][1] += dp_fx<GB>(t16[1]);
        };
#pragma unroll
        for (int t = 0; t < 16; ++t) t16[t] = d00 * h2[t >> 1][t & 1] + d10 * h2[t >> 1][2 + (t & 1)];
        add(3);
#pragma unroll
        for (int t = 0; t < 16; ++t) t16[t] = d01 * h2[t >> 1][t & 1] + d11 * h2[t >> 1][2 + (t & 1)];
        add(4);
#pragma unroll
        for (int t = 0; t < 16; ++t) t16[t] = dz[t >> 1][t & 1] + dz[t >> 1][2 + (t & 1)];
        add(2);
        // dz2 in bf16: the A fragments of dH1, and staged for dW2
        uint32_t az[4][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const int kt = nt >> 1, half = 2 * (nt & 1);
            az[kt][half] = dp_pack_bf16(dz[nt][0], dz[nt][1]);
            az[kt][half + 1] = dp_pack_bf16(dz[nt][2], dz[nt][3]);
            *(uint32_t*)(rows_dz + nt * 8) = az[kt][half];
            *(uint32_t*)(rows_dz + 8 * DP_MLP_LD + nt * 8) = az[kt][half + 1];
        }
        __syncthreads();
        // dW2[n][k] += sum_rows dz2[row][n] h1[row][k]: this warp's piece, one 16-row tile per mma
        {
            const int n0 = (warp >> 1) * 16, k0 = (warp & 1) * 32;
            const int row = lane & 7, mat = lane >> 3;
#pragma unroll 2
            for (int r = 0; r < DP_MLP_ROWS / 16; ++r) {
                uint32_t af[4], bf[4];
                // A: matrices (rows r, n), (r, n + 8), (r + 8, n), (r + 8, n + 8) transposed
                dp_ldmatrix4_trans(af, S.dz + (r * 16 + row + (mat >> 1) * 8) * DP_MLP_LD + n0 + (mat & 1) * 8);
#pragma unroll
                for (int q = 0; q < 4; q += 2) {
                    // B: (r, k), (r + 8, k), (r, k + 8), (r + 8, k + 8) transposed
                    dp_ldmatrix4_trans(bf, S.h1 + (r * 16 + row + (mat & 1) * 8) * DP_MLP_LD + k0 + q * 8 +
                                               (mat >> 1) * 8);
                    float acc0[4] = {0.f, 0.f, 0.f, 0.f}, acc1[4] = {0.f, 0.f, 0.f, 0.f};
                    dp_mma_bf16(acc0, af, bf[0], bf[1]);
                    dp_mma_bf16(acc1, af, bf[2], bf[3]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        sw2[q][e] += dp_fx<GB>(acc0[e]);
                        sw2[q + 1][e] += dp_fx<GB>(acc1[e]);
                    }
                }
            }
        }
        // dh1[row][k] = sum_n dz2[row][n] W2[n][k], then dz1 = dh1 act'(h1) (in dz)
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            float dh[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int kt = 0; kt < 4; ++kt) {
                const uint2 bb = *(const uint2*)(S.w2t + ((kt * 8 + nt) * 32 + lane) * 2);
                dp_mma_bf16(dh, az[kt], bb.x, bb.y);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float hg = h1[nt][e], hg8 = h1[nt][2 + e];
                dz[nt][e] = v0 ? dh[e] * (1.f - hg * hg) : 0.f;
                dz[nt][2 + e] = v1 ? dh[2 + e] * (1.f - hg8 * hg8) : 0.f;
            }
        }
#pragma unroll
        for (int t = 0; t < 16; ++t) t16[t] = dz[t >> 1][t & 1] * xg + dz[t >> 1][2 + (t & 1)] * xg8;
        add(0);
#pragma unroll
        for (int t = 0; t < 16; ++t) t16[t] = dz[t >> 1][t & 1] + dz[t >> 1][2 + (t & 1)];
        add(1);
    }
    // per-warp sums -> shared memory -> one atomic per parameter
    unsigned long long* mine = S.sums[warp];
    {
        const int col = dp_mlp_owned_nt(lane) * 8 + c;
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            mine[q * 64 + col] = sv[q][0];
            mine[q * 64 + col + 1] = sv[q][1];
        }
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) sloss += __shfl_xor_sync(0xffffffffu, sloss, o);
        if (lane == 0) {
            mine[320] = sb3[0];
            mine[321] = sb3[1];
            mine[322] = sloss;
        }
    }
    unsigned long long* G = a.gradfx;
    {
        unsigned long long* w = G + DP_MLP_OFF_W2 + ((warp >> 1) * 16 + g) * 64 + (warp & 1) * 32 + c;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            atomicAdd(w + q * 8, sw2[q][0]);
            atomicAdd(w + q * 8 + 1, sw2[q][1]);
            atomicAdd(w + 8 * 64 + q * 8, sw2[q][2]);
            atomicAdd(w + 8 * 64 + q * 8 + 1, sw2[q][3]);
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < DP_MLP_SUMS; t += blockDim.x) {
        unsigned long long v = 0ull;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += S.sums[w][t];
        unsigned long long* to = t < 64    ? G + DP_MLP_OFF_W1 + t
                                 : t < 128 ? G + DP_MLP_OFF_B1 + (t - 64)
                                 : t < 192 ? G + DP_MLP_OFF_B2 + (t - 128)
                                 : t < 320 ? G + DP_MLP_OFF_W3 + (t - 192)
                                 : t < 322 ? G + DP_MLP_OFF_B3 + (t - 320)
                                           : a.lossfx;
        atomicAdd(to, v);
    }
}

__device__ __forceinline__ float dp_mlp_grad_of(unsigned long long fx) {
    return (float)((double)(long long)fx * (1.0 / (double)(1ull << DP_MLP_GRAD_FX_BITS)));
}
__device__ __forceinline__ float dp_mlp_loss_of(unsigned long long fx) {
    return (float)((double)(long long)fx * (1.0 / (double)(1ull << DP_MLP_LOSS_FX_BITS)));
}

// Fixed-point sums -> float gradient and loss.
__global__ void k_mlp_grad_finish(const unsigned long long* __restrict__ gradfx,
                                  const unsigned long long* __restrict__ lossfx, float* grad, float* loss) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < DP_MLP_NPARAM) grad[t] = dp_mlp_grad_of(gradfx[t]);
    if (t == 0) *loss = dp_mlp_loss_of(*lossfx);
}

// The rest of a training step in one launch: the gradient from its fixed-point
// sums (cleared for the next step), Adam (Kingma & Ba 2015) on the fp32
// masters, and the new weights packed for the forward and backward passes. A
// thread owns the parameters one packed word needs: a 2 x 2 block of W2 (its
// rows give the fragments of W2, its columns those of the transpose), or one
// parameter of the other arrays; nothing passes between threads. Latency-bound
// (4418 parameters): one launch and not four (finish, Adam, pack, loss copy).
struct MlpUpdateArgs {
    float *p, *mo, *ve;
    unsigned long long *gradfx, *lossfx;
    dp_mlp_dev* m;
    uint32_t* w2t;
    float* loss;  // this step's loss
    float lr, b1, b2, eps, c1, c2;
};

__device__ __forceinline__ float dp_mlp_adam(const MlpUpdateArgs& a, int t) {
    const float gr = dp_mlp_grad_of(a.gradfx[t]);
    a.gradfx[t] = 0ull;
    // written out, so that every inlined copy rounds alike
    const float m1 = fmaf(1.f - a.b1, gr, a.b1 * a.mo[t]);
    const float v1 = fmaf((1.f - a.b2) * gr, gr, a.b2 * a.ve[t]);
    a.mo[t] = m1;
    a.ve[t] = v1;
    const float w = a.p[t] - a.lr * (m1 * a.c1) / (sqrtf(v1 * a.c2) + a.eps);
    a.p[t] = w;
    return w;
}

constexpr int kMlpUpdateThreads = 1024 + 64 * 5 + 2 + 1;

__global__ void __launch_bounds__(64) k_mlp_update(MlpUpdateArgs a) {
    dp_launch_dependents();
    dp_grid_wait();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < 1024) {
        const int n = (t >> 5) * 2, k = (t & 31) * 2;
        float w[2][2];
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int e = 0; e < 2; ++e) w[r][e] = dp_mlp_adam(a, DP_MLP_OFF_W2 + (n + r) * 64 + k + e);
        // fragment [kt][nt][lane][reg]: row = nt * 8 + lane / 4, column = kt * 16 + 8 reg + 2 (lane & 3) (+ 1)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int f = (((k >> 4) * 8 + ((n + r) >> 3)) * 32 + ((n + r) & 7) * 4 + ((k & 7) >> 1)) * 2 + ((k >> 3) & 1);
            a.m->w2frag[f] = dp_pack_bf16(w[r][0], w[r][1]);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int f = (((n >> 4) * 8 + ((k + e) >> 3)) * 32 + ((k + e) & 7) * 4 + ((n & 7) >> 1)) * 2 + ((n >> 3) & 1);
            a.w2t[f] = dp_pack_bf16(w[0][e], w[1][e]);
        }
        return;
    }
    const int u = t - 1024;
    if (u < 64) {
        const float w = dp_mlp_adam(a, DP_MLP_OFF_W1 + u);
        a.m->w1[u] = DP_MLP_SCALAR_BF16 ? dp_round_bf16(w) : w;
    } else if (u < 128) {
        a.m->b1[u - 64] = dp_mlp_adam(a, DP_MLP_OFF_B1 + u - 64);
    } else if (u < 192) {
        a.m->b2[u - 128] = dp_mlp_adam(a, DP_MLP_OFF_B2 + u - 128);
    } else if (u < 320) {
        const float w = dp_mlp_adam(a, DP_MLP_OFF_W3 + u - 192);
        a.m->w3[(u - 192) >> 6][(u - 192) & 63] = DP_MLP_SCALAR_BF16 ? dp_round_bf16(w) : w;
    } else if (u < 322) {
        a.m->b3[u - 320] = dp_mlp_adam(a, DP_MLP_OFF_B3 + u - 320);
    } else if (u == 322) {
        *a.loss = dp_mlp_loss_of(*a.lossfx);
        *a.lossfx = 0ull;
    }
}
