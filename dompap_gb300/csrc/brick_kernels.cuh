// brick_kernels.cuh — the pair kernels of large systems, one CTA per brick of
// cells (compiled by NVRTC after pair_kernels.cuh).
//
// A brick is a block of 2^b cells that follow one another in Morton order, so
// its particles hold consecutive slots; every partner its particles can list
// lies in its region, the brick and the cells around it. A CTA first copies
// the region's fixed-point positions into shared memory, and the lists hold
// 16-bit indices into that copy. With lists of slots every listed neighbour is
// a gather from 32 different cache lines, which L1 serves one line at a time
// (~30 cycles a warp): that bounded the pair loop of a liquid, at about five
// times its arithmetic. From shared memory the same gather takes the ~10 cycles
// of its bank conflicts, the region costs one coalesced copy (about eight
// entries a particle in a liquid), and the list is half as long in bytes
// (k_brick_build writes it; chunks of 8 entries, one 16-byte load each).
//
// LANES lanes (1 or 4) share a particle; the forces of LANES > 1 go through shared memory so that the integrator, whose float64
// work would cost a warp the same for 8 active lanes as for 32, runs dense.
// The step kernel of 500,000 LJ particles: 220 us on lists of slots, 104 here.
// Float32 only: the double-float pair terms cost a warp ~50 cycles a pair, which
// hides the gathers, and twice the region (both words of the fixed point)
// leaves too few warps for them: 371 us against 335 with lists of slots
// (256,000-particle mixture).
#if DP_REAL_IS_FLOAT && !DP_MLP && DP_DIM <= 3 && DP_PMODE != 2

struct dp_brick {
    int first, count, entries;
    const uint4* at;  // region: shadows; .w (3-D) or .z (2-D) is the type
    const int32_t* slots;
};

extern __shared__ __align__(16) uint4 dp_brick_smem[];

__device__ __forceinline__ dp_brick dp_brick_load(const dp_pair_args& a) {
    constexpr int D = DP_DIM;
    dp_brick b;
    const int4 info = a.brick_info[blockIdx.x];
    b.first = info.x;
    b.count = info.y;
    b.entries = info.z;
    b.slots = a.brick_slots + (long long)blockIdx.x * a.brick_cap;
    b.at = dp_brick_smem;
#pragma unroll 4
    for (int t = threadIdx.x; t < b.entries; t += blockDim.x) {
        const int j = __ldg(b.slots + t);
        uint32_t u[4] = {0u, 0u, 0u, 0u};
        dp_shadow_unpack<D>(__ldg((const shadow_t*)a.shadow + j), u);
#if DP_PMODE == 1
        u[D] = (uint32_t)__ldg(a.types + j);
#endif
        dp_brick_smem[t] = make_uint4(u[0], u[1], u[2], u[3]);
    }
    __syncthreads();
    return b;
}

__device__ __forceinline__ int dp_brick_entry(const uint4& chunk, int e) {
    const uint32_t w = e < 2 ? chunk.x : (e < 4 ? chunk.y : (e < 6 ? chunk.z : chunk.w));
    return (int)((w >> (16 * (e & 1))) & 0xFFFFu);
}

// The pair sum of slot i: every entry of its list (LANES 1), or the entries lane,
// lane + 4, ... (LANES 4: two of each chunk, which the four lanes load as one).
template <int ACC, int LANES>
__device__ __forceinline__ double dp_brick_sum(const dp_pair_args& a, const dp_brick& b, int i, double* f, int lane) {
    constexpr int D = DP_DIM;
    const long long n = a.n;
    uint32_t ui[D];
    int ti = 0;
#if DP_PMODE == 1
    ti = a.types[i];
#endif
    dp_pair_acc A;
    const int c = a.cnt[i];
    const int chunks = (c + 7) >> 3;
    const uint4* __restrict__ list = a.brick_list + i;
    dp_shadow_unpack<D>(((const shadow_t*)a.shadow)[i], ui);
    // One pass: the pair terms are as cheap as a second gather (programs with a
    // costly force have no brick kernels).
    auto entry = [&](int id, bool listed) {
        const uint4 h = b.at[id];
        const uint32_t uj[4] = {h.x, h.y, h.z, h.w};
        float df[D];
        const float q = dp_shadow_q<D>(ui, uj, a.unit, df);
        // the virial is an upper-triangle sum over slots (symmetric parameters)
        if (listed && q <= a.cut2f && !(ACC == DP_ACC_VIRIAL && __ldg(b.slots + id) <= i))
            dp_pair_eval<ACC>(a, i, 0, ti, (int)uj[D], q, df, A);
    };
    // two chunks in flight ahead of the one being evaluated
    const uint4 none = make_uint4(0u, 0u, 0u, 0u);
    uint4 next = chunks > 0 ? __ldg(list) : none;
    uint4 after = chunks > 1 ? __ldg(list + n) : none;
    for (int ch = 0; ch < chunks; ++ch) {
        const uint4 cur = next;
        next = after;
        list += n;
        after = ch + 2 < chunks ? __ldg(list + n) : none;
        const int m = c - 8 * ch;
        if (LANES == 1) {
#pragma unroll
            for (int e = 0; e < 8; ++e) entry(dp_brick_entry(cur, e), e < m);
        } else {
            const uint32_t w0 = (lane & 2) ? cur.y : cur.x, w1 = (lane & 2) ? cur.w : cur.z;
            const int shift = 16 * (lane & 1);
            entry((int)((w0 >> shift) & 0xFFFFu), lane < m);
            entry((int)((w1 >> shift) & 0xFFFFu), lane + 4 < m);
        }
    }
    return A.template finish<ACC>(f);
}

// Calls body(slot, f) once for every particle of the brick, from consecutive
// threads, with its force; every thread of the CTA takes part.
template <int LANES, typename Body>
__device__ __forceinline__ void dp_brick_forces(const dp_pair_args& a, const dp_brick& b, Body body) {
    constexpr int D = DP_DIM;
    if (LANES == 1) {
        for (int p = threadIdx.x; p < b.count; p += blockDim.x) {
            double f[D];
            dp_brick_sum<DP_ACC_FORCE, 1>(a, b, b.first + p, f, 0);
            body(b.first + p, f);
        }
        return;
    }
    __shared__ double s_f[D][256 / LANES];
    const int per = blockDim.x / LANES;
    const int mine = threadIdx.x / LANES, lane = threadIdx.x % LANES;
    for (int base = 0; base < b.count; base += per) {
        double f[D];
#pragma unroll
        for (int k = 0; k < D; ++k) f[k] = 0.0;
        const bool active = base + mine < b.count;
        if (active) dp_brick_sum<DP_ACC_FORCE, LANES>(a, b, b.first + base + mine, f, lane);
#pragma unroll
        for (int off = LANES / 2; off > 0; off >>= 1) {
#pragma unroll
            for (int k = 0; k < D; ++k) f[k] += __shfl_down_sync(0xffffffffu, f[k], off, LANES);
        }
        if (active && lane == 0) {
#pragma unroll
            for (int k = 0; k < D; ++k) s_f[k][mine] = f[k];
        }
        __syncthreads();
        const int p = base + (int)threadIdx.x;
        if ((int)threadIdx.x < per && p < b.count) {
#pragma unroll
            for (int k = 0; k < D; ++k) f[k] = s_f[k][threadIdx.x];
            body(b.first + p, f);
        }
        __syncthreads();
    }
}

template <int LANES>
__device__ __forceinline__ void dp_step_bricks(const dp_pair_args& a, const dp_int_args& g) {
    if (dp_step_idle(g)) return;
    const dp_brick b = dp_brick_load(a);
    bool old = false, bad = false;
    dp_brick_forces<LANES>(a, b, [&](int i, const double* f) {
#pragma unroll
        for (int k = 0; k < DP_DIM; ++k) bad = bad || !dp_isfinite_bits(f[k]);
        old = dp_integrate_dispatch<DP_DIM, false>(g, i, f, bad) || old;
    });
    dp_step_flags(g, old, bad);
    dp_step_end(g, old);
}

#define DP_BRICK_BOUNDS __launch_bounds__(256, DP_BRICK_BLOCKS)
extern "C" __global__ void DP_BRICK_BOUNDS dp_step_brick1(dp_pair_args a, dp_int_args b) { dp_step_bricks<1>(a, b); }
extern "C" __global__ void DP_BRICK_BOUNDS dp_step_brick4(dp_pair_args a, dp_int_args b) { dp_step_bricks<4>(a, b); }

extern "C" __global__ void __launch_bounds__(256) dp_forces_brick(dp_pair_args a) {
    const dp_brick b = dp_brick_load(a);
    bool bad = false;
    dp_brick_forces<4>(a, b, [&](int i, const double* f) {
#pragma unroll
        for (int k = 0; k < DP_DIM; ++k) {
            a.out[k * a.n + i] = f[k];
            bad = bad || !dp_isfinite_bits(f[k]);
        }
    });
    if (bad) atomicExch(&a.status->nonfinite, 1);
}

// Per-brick partial sums of the energy or the virial.
template <int ACC>
__device__ __forceinline__ void dp_brick_partial(const dp_pair_args& a) {
    __shared__ double smem[32];
    const dp_brick b = dp_brick_load(a);
    double v = 0.0;
    for (int t = threadIdx.x; t < 4 * b.count; t += blockDim.x)
        v += dp_brick_sum<ACC, 4>(a, b, b.first + (t >> 2), nullptr, t & 3);
    v = dp_block_sum(v, smem);
    if (threadIdx.x == 0) a.partial[blockIdx.x] = v;
}

extern "C" __global__ void __launch_bounds__(256) dp_energy_brick(dp_pair_args a) { dp_brick_partial<DP_ACC_ENERGY>(a); }
extern "C" __global__ void __launch_bounds__(256) dp_virial_brick(dp_pair_args a) { dp_brick_partial<DP_ACC_VIRIAL>(a); }

extern "C" __global__ void __launch_bounds__(256) dp_laplacian_brick(dp_pair_args a) {
    const dp_brick b = dp_brick_load(a);
    for (int t = threadIdx.x; t < ((4 * b.count + 31) & ~31); t += blockDim.x) {
        const bool active = t < 4 * b.count;
        double v = active ? dp_brick_sum<DP_ACC_LAPLACE, 4>(a, b, b.first + (t >> 2), nullptr, t & 3) : 0.0;
        v += __shfl_down_sync(0xffffffffu, v, 2, 4);
        v += __shfl_down_sync(0xffffffffu, v, 1, 4);
        if (active && (t & 3) == 0) a.out[b.first + (t >> 2)] = v;
    }
}
#endif
