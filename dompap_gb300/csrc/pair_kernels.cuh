// pair_kernels.cuh — pair force / energy / virial / Laplacian kernels.
//
// This file is compiled at run time by NVRTC for sm_103a, once per
// (dimension, pair potential, sigma/epsilon mode, precision). The host
// prepends the DP_* configuration macros, dp_common.cuh and the device
// functions generated from the SymPy pair potential:
//
//   template <typename R> __device__ R dp_pair_u(R s, R inv_s);   // u(s) - u(r_cut)
//   template <typename R> __device__ R dp_pair_f(R s, R inv_s);   // -du/ds
//   template <typename R> __device__ R dp_pair_c(R s, R inv_s);   // d2u/ds2
//
// Semantics follow dompap's neighbour-list kernels:
//   force      dompap/potential.py:163-188  F_n = sum_m eps f(r/sigma) d/r
//   energy     dompap/potential.py:69-100   U = 1/2 sum_n sum_m eps u(r/sigma)
//   virial     dompap/potential.py:253-279  W = 1/D sum_{n<m} eps(n,m) f(r/sigma(n,m)) r (pairs m > n of each list)
//   laplacian  dompap/potential.py:327-364  sum_m eps c(r/sigma) - (D-1) eps f(r/sigma)/r
// with s = r / sigma and every term 0 where s > r_cut (dompap/potential.py:61-65).
// There is no 1/sigma chain-rule factor, exactly as in the reference.
//
// Layout in HBM: positions are SoA float64 pos[k*N + i]; entry k of slot i's
// neighbour list is nl[k nl_k + i nl_i] (column-major, or a row per slot where a
// warp shares a particle) with per-particle counts cnt[i]; the
// fixed-point shadow is one 8- or 16-byte vector per particle.
//
// Configuration macros (set by the host):
//   DP_DIM          spatial dimension (2, 3 or 4)
//   DP_REAL         pair arithmetic type: double (FP64 mode) or float (FP32 mode)
//   DP_PMODE        0 constant sigma/epsilon, 1 per-type table, 2 dense (N, N) matrix
//   DP_SIGMA_ONE    1 when sigma is the constant 1 (the division is skipped)
//   DP_EPS_ONE      1 when epsilon is the constant 1
//   DP_FF           1 in the float64-parity mode: pair arithmetic in double-float
//                   (dp_ff.cuh) on the exact 64-bit fixed-point displacement; the
//                   cut decision within float rounding of r_cut and positions not
//                   yet wrapped into the box take the float64 path
//   DP_LISTS_BLOCKS, DP_WARP_SUMS, DP_QUAD_SUMS
//                   kernels for sizes that the program may leave out (0): the step that
//                   keeps its own lists (else its CTAs per SM), sums with 32 and with 4
//                   lanes per particle
#ifndef DP_FF
#define DP_FF 0
#endif
#ifndef DP_LISTS_BLOCKS
#define DP_LISTS_BLOCKS 4
#endif
#ifndef DP_WARP_SUMS
#define DP_WARP_SUMS 1
#endif
#ifndef DP_QUAD_SUMS
#define DP_QUAD_SUMS 1
#endif

#ifndef DP_DIM
#error "DP_DIM must be defined"
#endif

// struct dp_pair_args is defined in dp_common.cuh (shared with the host).

typedef DP_REAL real_t;
typedef typename dp_shadow_t<DP_DIM>::type shadow_t;

// sigma, 1/sigma and epsilon of the pair of slots i and j, of types ti and tj.
__device__ __forceinline__ void dp_pair_params(const dp_pair_args& a, long long i, int ti, int j, int tj, double& sig,
                                               double& isig, double& eps) {
#if DP_PMODE == 0
    sig = a.sigma;
    isig = a.inv_sigma;
    eps = a.epsilon;
#elif DP_PMODE == 1
    sig = __ldg(a.sig_tab + ti * a.ntypes + tj);
    isig = __ldg(a.isig_tab + ti * a.ntypes + tj);
    eps = __ldg(a.eps_tab + ti * a.ntypes + tj);
#else
    // the dense (N, N) tables are indexed by particle id; with `upper` by
    // (min, max) of the two ids, as dompap's Newton's-third-law double loop
    // (dompap/potential.py:191-214) evaluates every pair once with
    // sigma(n, m), epsilon(n, m), n < m
    long long pi = __ldg(a.order + i), pj = __ldg(a.order + j);
    if (a.upper && pi > pj) {
        const long long t = pi;
        pi = pj;
        pj = t;
    }
    sig = __ldg(a.sig_tab + pi * a.n + pj);
    isig = 1.0 / sig;
    eps = __ldg(a.eps_tab + pi * a.n + pj);
#endif
}

// What one kernel accumulates for a pair; selected at compile time.
// DP_ACC_ENERGY_UPPER: the energy over the partners m of n with m > n (ids).
enum { DP_ACC_FORCE = 0, DP_ACC_ENERGY = 1, DP_ACC_VIRIAL = 2, DP_ACC_LAPLACE = 3, DP_ACC_ENERGY_UPPER = 4 };

// The pair sum of particle (slot) i takes m > n in particle ids: the virial
// (dompap/potential.py:265-278) and the double-loop energies (:103-160).
// Per-type and constant parameters are symmetric, so any one orientation of
// each pair gives the same total and slots are compared; the dense tables may
// not be, so the ids are.
__device__ __forceinline__ bool dp_upper_skip(const dp_pair_args& a, long long i, int j) {
#if DP_PMODE == 2
    return __ldg(a.order + j) <= __ldg(a.order + i);
#else
    return j <= i;
#endif
}

// What a particle (or a lane of its group) has summed over its pairs.
struct dp_pair_acc {
    real_t v[DP_DIM];  // force: float32, or the float64 path of the parity mode
    double s;          // energy, virial or Laplacian
#if DP_FF
    dpff fv[DP_DIM];   // compensated sums (dpff_accumulate)
    dpff fs;
    bool used64;
#endif
    __device__ __forceinline__ dp_pair_acc() : s(0.0) {
#pragma unroll
        for (int k = 0; k < DP_DIM; ++k) v[k] = real_t(0);
#if DP_FF
        used64 = false;
#endif
    }
    // The scalar sum and, for DP_ACC_FORCE, the force vector.
    template <int ACC>
    __device__ __forceinline__ double finish(double* f) const {
#if DP_FF
        // double-float -> float64 by moving bits (one float64 add per value)
        if (ACC == DP_ACC_FORCE) {
#pragma unroll
            for (int k = 0; k < DP_DIM; ++k)
                f[k] = used64 ? (double)v[k] + dpff_to_double(fv[k]) : dpff_to_double(fv[k]);
        }
        return used64 ? s + dpff_to_double(fs) : dpff_to_double(fs);
#else
        if (ACC == DP_ACC_FORCE) {
#pragma unroll
            for (int k = 0; k < DP_DIM; ++k) f[k] = (double)v[k];
        }
        return s;
#endif
    }
};

// dp_pair_g (f(s)/s as a function of s^2: a double-float reciprocal and no
// square root) where the potential has it, for the forces (the virial would
// lose a bit: its sum cancels). With it and dpff_from_fixed a Lennard-Jones pair takes
// about half the instructions: the mixture of 256,000 (skin 0.5) went from 434
// to 388 us a step.
#if defined(DP_PAIR_EVEN) && DP_FF
#define DP_USES_G(ACC) ((ACC) == DP_ACC_FORCE)
#else
#define DP_USES_G(ACC) false
#endif
#ifndef DP_PAIR_EVEN
template <typename R>
__device__ __forceinline__ R dp_pair_g(R, R) {
    return R(0);
}
#endif

#if DP_REAL_IS_FLOAT
// 1/sqrt of a squared distance, without rsqrtf's scaling of subnormals: a pair
// as close as 1e-19 overflows its force anyway.
__device__ __forceinline__ float dp_rsqrt_normal(float q) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(q));
    return y;
}

// One pair in float32 on the fixed-point displacement df with q = |df|^2.
// (dp_pair_g would save the square root's multiplication here but needs a
// second comparison near the cut, where both forms have to decide alike: no
// gain, 1.7 % slower on 500,000 LJ particles.)
template <int ACC>
__device__ __forceinline__ void dp_pair_eval(const dp_pair_args& a, long long i, int j, int ti, int tj, float q,
                                             const float* df, dp_pair_acc& A) {
    constexpr int D = DP_DIM;
#if DP_PMODE == 0
    const float sig = a.f32_const[0], isig = a.f32_const[1], e = a.f32_const[2];
#elif DP_PMODE == 1
    const float4 par = __ldg(a.f32_tab + ti * a.ntypes + tj);
    const float sig = par.x, isig = par.y, e = par.z;
#else
    double sig64, isig64, eps64;
    dp_pair_params(a, i, ti, j, tj, sig64, isig64, eps64);
    const float sig = (float)sig64, isig = (float)isig64, e = (float)eps64;
#endif
    const float rinv = dp_rsqrt_normal(q);
    const float r = q * rinv;
#if DP_SIGMA_ONE
    const float s = r, sinv = rinv;
#else
    const float s = r * isig, sinv = rinv * sig;
#endif
    if (s > a.rcut_f) return;
    if (ACC == DP_ACC_FORCE) {
#if DP_EPS_ONE
        const float sf = dp_pair_f<float>(s, sinv);
#else
        const float sf = e * dp_pair_f<float>(s, sinv);
#endif
        const float g = sf * rinv;
#pragma unroll
        for (int k = 0; k < D; ++k) A.v[k] = fmaf(g, df[k], A.v[k]);
    } else if (ACC == DP_ACC_ENERGY || ACC == DP_ACC_ENERGY_UPPER) {
        A.s += (double)(e * dp_pair_u<float>(s, sinv));
    } else if (ACC == DP_ACC_VIRIAL) {
        A.s += (double)(e * dp_pair_f<float>(s, sinv) * r);
    } else {
        A.s += (double)(e * dp_pair_c<float>(s, sinv) + (float)(D - 1) * (-e * dp_pair_f<float>(s, sinv)) * rinv);
    }
}
#endif

#if DP_FF
// One pair in double-float on the exact 64-bit fixed-point displacement.
// False: the pair needs the float64 path (its scaled distance lies within float
// rounding of r_cut, or is zero).
template <int ACC>
__device__ __forceinline__ bool dp_pair_eval_ff(const dp_pair_args& a, long long i, int j, int ti, int tj,
                                                const unsigned long long* Xi, const unsigned long long* Xj,
                                                dp_pair_acc& A) {
    constexpr int D = DP_DIM;
    dpff d[D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
        const dpff U(a.unit64_hi[k] * 4294967296.0f, a.unit64_lo[k] * 4294967296.0f);
        d[k] = dpff_from_fixed((long long)(Xi[k] - Xj[k]), U, a.unit64_hi[k] * 256.0f);
    }
    dpff q = dpff_sqr_unnormalised(d[0]);
#pragma unroll
    for (int k = 1; k < D; ++k) dpff_accumulate(q, dpff_sqr_unnormalised(d[k]));
    q = dpff_quick_two_sum(q.hi, q.lo);
#if DP_PMODE == 0
    const float* c = a.ff_const;
    const dpff sig(c[0], c[1]), isig(c[2], c[3]), eps(c[4], c[5]), isig2(c[6], c[7]), eps_isig(c[8], c[9]);
#elif DP_PMODE == 1
    const float2* tri = a.ff_tab + DP_FF_PARAMS * (ti * a.ntypes + tj);
    auto par = [&](int t) {
        const float2 v = __ldg(tri + t);
        return dpff(v.x, v.y);
    };
    const dpff sig = par(0), isig = par(1), eps = par(2);
    const dpff isig2 = par(3), eps_isig = par(4);
#else
    double sig64, isig64, eps64;
    dp_pair_params(a, i, ti, j, tj, sig64, isig64, eps64);
    const dpff sig(sig64), isig(isig64), eps(eps64);
    const dpff isig2 = isig * isig, eps_isig = eps * isig;
#endif
    if (DP_USES_G(ACC)) {
#if DP_SIGMA_ONE
        const dpff s2 = q;
#else
        const dpff s2 = q * isig2;
#endif
        if (a.rcut_finite && fabsf(s2.hi - a.rcut2_f) <= 2e-5f * a.rcut2_f) return false;
        if (!(s2.hi > 0.0f)) return false;
        if (s2.hi > a.rcut2_f) return true;
        const dpff g = dp_pair_g<dpff>(s2, dpff_rcp(s2));
#if DP_SIGMA_ONE && DP_EPS_ONE
        const dpff h = g;
#else
        const dpff h = eps_isig * g;
#endif
#pragma unroll
        for (int k = 0; k < D; ++k) dpff_accumulate_prod(A.fv[k], h, d[k]);
        return true;
    }
    const dpff rinv = dpff_rsqrt(q);
    const dpff r = q * rinv;
#if DP_SIGMA_ONE
    const dpff s = r, sinv = rinv;
#else
    const dpff s = r * isig, sinv = rinv * sig;
#endif
    if (a.rcut_finite && fabsf(s.hi - a.rcut_f) <= 1e-5f * a.rcut_f) return false;
    if (s.hi > a.rcut_f) return true;
    if (ACC == DP_ACC_FORCE) {
#if DP_EPS_ONE
        const dpff g = dp_pair_f<dpff>(s, sinv) * rinv;
#else
        const dpff g = eps * dp_pair_f<dpff>(s, sinv) * rinv;
#endif
#pragma unroll
        for (int k = 0; k < D; ++k) dpff_accumulate_prod(A.fv[k], g, d[k]);
    } else if (ACC == DP_ACC_ENERGY || ACC == DP_ACC_ENERGY_UPPER) {
        dpff_accumulate(A.fs, eps * dp_pair_u<dpff>(s, sinv));
    } else if (ACC == DP_ACC_VIRIAL) {
        dpff_accumulate(A.fs, eps * dp_pair_f<dpff>(s, sinv) * r);
    } else {
        const dpff sf = eps * dp_pair_f<dpff>(s, sinv);
        dpff_accumulate(A.fs, eps * dp_pair_c<dpff>(s, sinv) - dpff(D - 1) * sf * rinv);
    }
    return true;
}
#endif

#if !DP_REAL_IS_FLOAT
// One pair in float64 on the positions of slots i and j. d and r^2 follow the
// reference exactly; 1/r comes from one reciprocal square root (no divisions),
// and where s lies within a few ulp of r_cut, r = sqrt(r^2) and s = r / sigma
// are recomputed with IEEE operations so the cut decision is the reference's.
template <int ACC>
__device__ __forceinline__ void dp_pair_eval_f64(const dp_pair_args& a, long long i, int j, int ti, int tj,
                                                 dp_pair_acc& A) {
    constexpr int D = DP_DIM;
    const long long n = a.n;
#if DP_FF
    A.used64 = true;
#endif
    double sig, isig, eps;
    dp_pair_params(a, i, ti, j, tj, sig, isig, eps);
    double d[D];
#pragma unroll
    for (int k = 0; k < D; ++k) d[k] = dp_min_image(a.pos[k * n + i] - a.pos[k * n + j], a.box[k]);
    const double q = dp_sqsum_exact<D>(d);
    const double rinv = rsqrt(q);
    double r = q * rinv;
#if DP_SIGMA_ONE
    double s = r;
    const double sinv = rinv;
#else
    double s = r * isig;
    const double sinv = rinv * sig;
#endif
    if (fabs(s - a.rcut) <= 1e-14 * a.rcut) {
        r = sqrt(q);
#if DP_SIGMA_ONE
        s = r;
#else
        s = r / sig;
#endif
    }
    if (s > a.rcut) return;
    if (ACC == DP_ACC_FORCE) {
#if DP_EPS_ONE
        const double sf = dp_pair_f<double>(s, sinv);
#else
        const double sf = eps * dp_pair_f<double>(s, sinv);
#endif
        const double g = sf * rinv;
#pragma unroll
        for (int k = 0; k < D; ++k) A.v[k] = fma(g, d[k], A.v[k]);
    } else if (ACC == DP_ACC_ENERGY || ACC == DP_ACC_ENERGY_UPPER) {
        A.s += eps * dp_pair_u<double>(s, sinv);
    } else if (ACC == DP_ACC_VIRIAL) {
        A.s += eps * dp_pair_f<double>(s, sinv) * r;
    } else {
        const double sf = eps * dp_pair_f<double>(s, sinv);
        A.s += eps * dp_pair_c<double>(s, sinv) + (double)(D - 1) * (-sf) * rinv;
    }
}
#endif

// A load of what the step before wrote, or this one (its list). LIVE: this kernel's blocks were placed while
// that step still ran (dp_step_lists), so the value was not read-only for the whole
// of the kernel's life and a read-only load may not be used, nor one that the
// compiler could move across the wait.
template <bool LIVE, typename T>
__device__ __forceinline__ T dp_fetch(const T* p) {
    return LIVE ? *p : __ldg(p);
}

// Window of the two-pass loop: one thread per particle evaluates 64 listed
// neighbours at a time (mixture of 256,000, 150 listed: 320 / 298 / 307 us a
// step with 32 / 64 / 128; 108,000 LJ, 95 listed: 91 / 87 / 84; lists of a
// dozen: equal; 10 us more each with the displacement in its present form).
#define DP_WINDOW 64

// Per-particle neighbour loop. Returns the scalar sum (energy / virial /
// Laplacian) and, for DP_ACC_FORCE, the force vector in f[].
//
// Float64-parity mode (DP_FF): a pair is evaluated in double-float on the
// exact 64-bit fixed-point displacement, with no float64 instruction in the
// loop (this GPU runs float64 at 1/64 of the float32 rate). Pairs whose
// scaled distance lies within float rounding of r_cut, and every pair while
// some position is far outside the box, take the float64 path of the
// reference instead (its min-image displacement, cut decision and pair
// terms).
//
// LANES > 1 (the fused step for small systems): LANES consecutive lanes share
// particle i, lane `lane` of them taking list entries lane, lane + LANES, ...;
// each returns its partial sums (the caller adds them across the group).
// ALL: no list, every other particle is a candidate partner (dompap's
// double-loop and vectorised force and energy methods,
// dompap/potential.py:103-160,191-250,298-324); lane `lane` takes slots
// lane, lane + LANES, ...  listed: the row's length if the caller knows it.
template <int ACC, int LANES = 1, bool ALL = false, bool LIVE = false>
__device__ __forceinline__ double dp_particle_sum(const dp_pair_args& a, long long i, double* f, int lane = 0,
                                                  int listed = -1) {
    constexpr int D = DP_DIM;
    const long long n = a.n;
    const shadow_t* sh = (const shadow_t*)a.shadow;
    uint32_t ui[D];
    int ti = 0;
#if DP_PMODE == 1
    ti = a.types[i];
#endif
    dp_pair_acc A;
#if DP_FF
    typedef typename dp_fixed64_t<D>::type fx_t;
    const fx_t* p64 = (const fx_t*)a.pos64;
    const bool ff_ok = a.status->far == 0;  // single-shift image == nearest image
    unsigned long long Xi[D];
    if (ff_ok) dp_fixed64_unpack<D>(p64[i], Xi);
#endif
    dp_shadow_unpack<D>(sh[i], ui);
    // Two passes over windows of up to DP_WINDOW listed neighbours. Pass 1 runs
    // the float32 pre-filter on the shadows and keeps a bit per neighbour that
    // may lie within r_cut * sigma_max; pass 2 evaluates the pair terms of
    // the kept ones only, in list order. A warp then runs the pair arithmetic
    // as often as its busiest lane has kept neighbours, not once per listed
    // one, and the wider the window the closer the busiest lane is to the
    // average (in a liquid about 73 % of the lanes are busy with 32, 79 % with 64).
    const int c_all = ALL ? (int)n : (listed >= 0 ? listed : a.cnt[i]);
    const int c = LANES > 1 ? (c_all > lane ? (c_all - lane + LANES - 1) / LANES : 0) : c_all;
    // (through the read-only path unless dp_step_lists has just written the row: with plain
    // loads the forces of 1,000,000 2-D LJ particles took 113 us in float32, 76 so)
    const int32_t* row = ALL ? nullptr : a.nl + i * a.nl_i + (LANES > 1 ? lane * a.nl_k : 0LL);
    const long long entry_stride = LANES * a.nl_k;
    constexpr int W = LANES > 1 ? 1 : DP_WINDOW / 32;  // words of a window
    for (int base = 0; base < c; base += 32 * W) {
        uint32_t kept[W];
#pragma unroll
        for (int q = 0; q < W; ++q) {
            const int first = base + 32 * q, w = min(32, c - first);
            kept[q] = 0u;
#pragma unroll 4
            for (int t = 0; t < w; ++t) {
                const int j = ALL ? (first + t) * LANES + lane : dp_fetch<LIVE>(row + (first + t) * entry_stride);
                if (ALL && j == i) continue;
                // the virial and the double-loop energy are upper-triangle sums
                // over n < m with sigma(n, m), epsilon(n, m)
                if ((ACC == DP_ACC_VIRIAL || ACC == DP_ACC_ENERGY_UPPER) && dp_upper_skip(a, i, j)) continue;
                uint32_t uj[D];
                dp_shadow_unpack<D>(dp_fetch<LIVE>(sh + j), uj);
                float df[D];
                if (dp_shadow_q<D>(ui, uj, a.unit, df) <= a.cut2f) kept[q] |= 1u << t;
            }
        }
        int first = base;
        while (true) {
            if (W > 1) {
                // the next word with a bit; each lane on its own
#pragma unroll
                for (int q = 1; q < W; ++q) {
                    if (kept[0] == 0u) {
                        first += 32;
#pragma unroll
                        for (int p = 0; p + 1 < W; ++p) kept[p] = kept[p + 1];
                        kept[W - 1] = 0u;
                    }
                }
            }
            if (kept[0] == 0u) break;
            const int t = __ffs(kept[0]) - 1;
            kept[0] &= kept[0] - 1;
            const int j = ALL ? (first + t) * LANES + lane : dp_fetch<LIVE>(row + (first + t) * entry_stride);
            int tj = 0;
#if DP_PMODE == 1
            tj = __ldg(a.types + j);
#endif
#if DP_REAL_IS_FLOAT
            uint32_t uj[D];
            dp_shadow_unpack<D>(dp_fetch<LIVE>(sh + j), uj);
            float df[D];
            const float qf = dp_shadow_q<D>(ui, uj, a.unit, df);
            dp_pair_eval<ACC>(a, i, j, ti, tj, qf, df, A);
#else
#if DP_FF
            if (ff_ok) {
                unsigned long long Xj[D];
                dp_fixed64_unpack<D>(p64[j], Xj);
                if (dp_pair_eval_ff<ACC>(a, i, j, ti, tj, Xi, Xj, A)) continue;
            }
#endif
            dp_pair_eval_f64<ACC>(a, i, j, ti, tj, A);
#endif
        }
    }
    return A.template finish<ACC>(f);
}

// F (SoA float64) for every particle. One thread per particle; the
// double-float loop is limited to 64 registers (four 256-thread CTAs per SM).
#if DP_FF
#define DP_FORCES_BOUNDS __launch_bounds__(256, 4)
#else
#define DP_FORCES_BOUNDS __launch_bounds__(256)
#endif
extern "C" __global__ void DP_FORCES_BOUNDS dp_forces(dp_pair_args a) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    double f[DP_DIM];
    dp_particle_sum<DP_ACC_FORCE>(a, i, f);
    bool finite = true;
#pragma unroll
    for (int k = 0; k < DP_DIM; ++k) {
        a.out[k * a.n + i] = f[k];
        finite = finite && dp_isfinite_bits(f[k]);
    }
    if (!finite) atomicExch(&a.status->nonfinite, 1);
}

#if !DP_MLP
// One MD step of particle i in one kernel: its pair forces from this step's
// positions (as dp_forces), then its integration, wrap, fixed-point forms and
// skin test (dp_integrate_one) into the second set of position buffers, which
// no thread of this launch reads. The float64 integrator work runs on the
// float64 pipe beside the pair arithmetic of other warps, and the forces
// never go through memory. `far` must have been cleared by the host-side
// step sequence when the previous step wrapped every position.
#ifndef DP_STEP_MIN_BLOCKS
#define DP_STEP_MIN_BLOCKS 0
#endif

// End of a fused step in a graph. Each CTA adds 1 and, in the upper word, 1
// if one of its particles moved beyond skin/2, to one 64-bit counter; the
// CTA that brings the count to the grid size is the last one: every other CTA
// has finished (and read the status words), so it does the step's DP_END_*
// work. No fence is needed: whether a rebuild is due comes from the counter
// itself. Called by every thread of the CTA with its own `old`.
__device__ __forceinline__ void dp_step_end(const dp_int_args& b, bool old) {
    if (b.end_flags == 0) return;  // uniform: launches outside graphs
    const int cta_old = __syncthreads_or(old ? 1 : 0);
    if (threadIdx.x != 0) return;
    const unsigned long long mine = 1ull | ((unsigned long long)(cta_old != 0) << 32);
    const unsigned long long prev = atomicAdd(&b.st->ticket, mine);
    if ((unsigned)(prev & 0xffffffffull) != gridDim.x - 1) return;
    b.st->ticket = 0ull;
    const bool rebuild = ((prev + mine) >> 32) != 0;
    if (b.end_flags & DP_END_OWN_LISTS) {
        // every other CTA has read need_rebuild and far, and finished
        if (b.st->need_rebuild) {
            b.st->rebuilds += 1;
            b.st->ref_far = b.st->far;
        }
        b.st->need_rebuild = rebuild ? 1 : 0;
    }
    if (b.end_flags & DP_END_GROUP) {
        b.st->need_rebuild = rebuild ? 1 : 0;
        b.st->left -= 1;
        b.st->step += 1;
        b.st->parity ^= 1;
    }
    if (b.end_flags & DP_END_CLEAR_FAR) b.st->far = 0;
}

// A grouped step that has nothing to do (uniform over the grid).
__device__ __forceinline__ bool dp_step_idle(const dp_int_args& b) {
    return (b.end_flags & DP_END_GROUP) && (b.st->need_rebuild || b.st->left <= 0);
}

// Moved beyond skin/2: outside graphs and in graphs with a rebuild node per step
// the flag is set at once, otherwise dp_step_end sets it.
__device__ __forceinline__ void dp_step_flags(const dp_int_args& b, bool old, bool bad) {
    const bool any_old = __any_sync(0xffffffffu, old);
    const bool any_bad = __any_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0) {
        if (any_old && !(b.end_flags & (DP_END_OWN_LISTS | DP_END_GROUP))) atomicExch(&b.st->need_rebuild, 1);
        if (any_bad) atomicExch(&b.st->nonfinite, 1);
    }
}
#if DP_STEP_MIN_BLOCKS > 0
#define DP_STEP_BOUNDS __launch_bounds__(256, DP_STEP_MIN_BLOCKS)
#else
#define DP_STEP_BOUNDS __launch_bounds__(256)
#endif
extern "C" __global__ void DP_STEP_BOUNDS dp_step(dp_pair_args a, dp_int_args b) {
    if (dp_step_idle(b)) return;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    bool old = false, bad = false;
    if (i < a.n) {
        double f[DP_DIM];
        dp_particle_sum<DP_ACC_FORCE>(a, i, f);
#pragma unroll
        for (int k = 0; k < DP_DIM; ++k) bad = bad || !dp_isfinite_bits(f[k]);
        old = dp_integrate_dispatch<DP_DIM, DP_FF != 0>(b, i, f, bad);
    }
    dp_step_flags(b, old, bad);
    dp_step_end(b, old);
}

// The list of particle i (one warp): every other particle within the cutoff by
// the test of k_nl_build_allpairs, in ascending order, one row of the list.
// Returns its length (the capacity at most; the status records a longer one).
__device__ __forceinline__ int dp_build_row(const dp_pair_args& a, const dp_list_args& l, long long i, int lane,
                                            bool far) {
    constexpr int D = DP_DIM;
    const long long n = a.n;
    const shadow_t* sh = (const shadow_t*)a.shadow;
    const shadow_t shi = sh[i];
    uint32_t ui[D];
    dp_shadow_unpack<D>(shi, ui);
    int32_t* row = l.nl + i * l.kcap;
    int found = 0;
#pragma unroll 2
    for (int base = 0; base < (int)n; base += 32) {
        const int j = base + lane;
        bool in = false;
        if (j < (int)n && j != (int)i) {
            uint32_t uj[D];
            dp_shadow_unpack<D>(dp_fetch<true>(sh + j), uj);
            float df[D];
            const float q = dp_shadow_q<D>(ui, uj, a.unit, df);
            in = q <= l.hi2;
            if (in && (far || !(q < l.lo2))) {
                double d[D];
#pragma unroll
                for (int k = 0; k < D; ++k) d[k] = dp_min_image(a.pos[k * n + i] - a.pos[k * n + j], a.box[k]);
                in = sqrt(dp_sqsum_exact<D>(d)) < l.cutoff;
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        const int at = found + __popc(m & ((1u << lane) - 1u));
        if (in && at < l.kcap) row[at] = j;
        found += __popc(m);
    }
    const int kept = min(found, l.kcap);
    if (lane == 0) {
        l.cnt[i] = kept;
        ((shadow_t*)l.shadow_ref)[i] = shi;
        atomicMax(&a.status->max_neighbors, found);
    }
    if (lane < D) l.pos_ref[lane * n + i] = a.pos[lane * n + i];
    __syncwarp();
    return kept;
}

// The fused step for small systems: LANES lanes per particle. The lanes
// split the particle's list (dp_particle_sum<..., LANES>), their partial
// forces are added across the group in a fixed order, and the group's first
// lane integrates. Below a few tens of thousands of particles this spreads the
// pair loops over LANES times more threads than dp_step, whose one thread per
// particle leaves most SMs idle.
template <int LANES, bool ALL = false, bool LIVE = false>
__device__ __forceinline__ void dp_step_split(const dp_pair_args& a, const dp_int_args& b, const dp_list_args* own) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long i = t / LANES;
    const int lane = (int)(t % LANES);
    bool old = false, bad = false;
    const bool active = i < a.n;  // uniform across the group, not the warp
    double f[DP_DIM];
#pragma unroll
    for (int k = 0; k < DP_DIM; ++k) f[k] = 0.0;
    int listed = -1, ref_far = -1;
    if (own && a.status->need_rebuild) {  // uniform over the grid: dp_step_end writes it
        ref_far = a.status->far != 0;
        if (active) listed = dp_build_row(a, *own, i, lane, ref_far != 0);
    }
    if (active) dp_particle_sum<DP_ACC_FORCE, LANES, ALL, LIVE>(a, i, f, lane, listed);
    // every lane of the warp takes part in the shuffles (groups past the
    // last particle add zeros)
#pragma unroll
    for (int off = LANES / 2; off > 0; off >>= 1) {
#pragma unroll
        for (int k = 0; k < DP_DIM; ++k) f[k] += __shfl_down_sync(0xffffffffu, f[k], off, LANES);
    }
    if (active && lane == 0) {
#pragma unroll
        for (int k = 0; k < DP_DIM; ++k) bad = bad || !dp_isfinite_bits(f[k]);
        old = dp_integrate_dispatch<DP_DIM, DP_FF != 0>(b, i, f, bad, ref_far);
    }
    dp_step_flags(b, old, bad);
    dp_step_end(b, old);
}

extern "C" __global__ void DP_STEP_BOUNDS dp_step_warp(dp_pair_args a, dp_int_args b) {
    if (dp_step_idle(b)) return;
    dp_step_split<32>(a, b, nullptr);
}
extern "C" __global__ void DP_STEP_BOUNDS dp_step_quad(dp_pair_args a, dp_int_args b) {
    if (dp_step_idle(b)) return;
    dp_step_split<4>(a, b, nullptr);
}

// One warp per particle, which also rebuilds the particle's list when the step
// before asked for it (and reads need_rebuild, which no CTA writes before all
// have read it). A row depends on this step's positions alone, so the rebuild
// needs no kernel of its own and the graph of steps no conditional nodes; the
// next step is placed while this one drains (programmatic dependent launch).
// All pairs are tested, 32 a round: 500 particles take ~5 us, 8,192
// 136 us, once in ~14 steps. Bound by the latency of its chain (gathers, pair
// terms, the sum over the warp, the float64 integrator) and by instruction
// fetch. LJ, float64, a step of a run before and now: 500 particles 23.2 -> 11.9
// us, 2,048 15.6, 4,000 60 -> 22.9, 8,112 41.
#if DP_LISTS_BLOCKS > 0
extern "C" __global__ void __launch_bounds__(256, DP_LISTS_BLOCKS) dp_step_lists(dp_pair_args a, dp_int_args b, dp_list_args l) {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    dp_step_split<32, false, true>(a, b, &l);
}
#endif

// ---------------------------------------------------------------------------
// No neighbour list: dompap's double-loop and vectorised methods
// (dompap/potential.py:103-160 energy, :191-250 and :298-324 forces). One
// warp per particle; lane l takes the slots l, l + 32, ... (every other
// particle is a candidate, tested with the same pre-filter and pair arithmetic
// as the list kernels), and the partial sums are added across the warp in a
// fixed order.
extern "C" __global__ void DP_STEP_BOUNDS dp_step_all(dp_pair_args a, dp_int_args b) {
    dp_step_split<32, true>(a, b, nullptr);
}

extern "C" __global__ void __launch_bounds__(256) dp_forces_all(dp_pair_args a) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long i = t >> 5;
    const int lane = (int)(t & 31);
    const bool active = i < a.n;  // uniform across the warp
    double f[DP_DIM];
#pragma unroll
    for (int k = 0; k < DP_DIM; ++k) f[k] = 0.0;
    if (active) dp_particle_sum<DP_ACC_FORCE, 32, true>(a, i, f, lane);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
        for (int k = 0; k < DP_DIM; ++k) f[k] += __shfl_down_sync(0xffffffffu, f[k], off);
    }
    if (!active || lane != 0) return;
    bool finite = true;
#pragma unroll
    for (int k = 0; k < DP_DIM; ++k) {
        a.out[k * a.n + i] = f[k];
        finite = finite && dp_isfinite_bits(f[k]);
    }
    if (!finite) atomicExch(&a.status->nonfinite, 1);
}

// U = sum over n < m of eps u(r / sigma) (no halving), per-block partials.
extern "C" __global__ void __launch_bounds__(256) dp_energy_all(dp_pair_args a) {
    __shared__ double smem[32];
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long i = t >> 5;
    double v = 0.0;
    if (i < a.n) v = dp_particle_sum<DP_ACC_ENERGY_UPPER, 32, true>(a, i, nullptr, (int)(t & 31));
    v = dp_block_sum(v, smem);
    if (threadIdx.x == 0) a.partial[blockIdx.x] = v;
}
#endif

// The same sums with LANES lanes per particle (32 up to 8,192 particles, 4 up to
// 65,536): one thread per particle leaves most SMs idle there.
// Forces of LJ particles in float64, before and now: 500 49 -> 8.3 us, 4,000 53 ->
// 16.4.
template <int LANES>
__device__ __forceinline__ void dp_forces_split(const dp_pair_args& a) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long i = t / LANES;
    const int lane = (int)(t % LANES);
    const bool active = i < a.n;
    double f[DP_DIM];
#pragma unroll
    for (int k = 0; k < DP_DIM; ++k) f[k] = 0.0;
    if (active) dp_particle_sum<DP_ACC_FORCE, LANES>(a, i, f, lane);
#pragma unroll
    for (int off = LANES / 2; off > 0; off >>= 1) {
#pragma unroll
        for (int k = 0; k < DP_DIM; ++k) f[k] += __shfl_down_sync(0xffffffffu, f[k], off, LANES);
    }
    if (!active || lane != 0) return;
    bool finite = true;
#pragma unroll
    for (int k = 0; k < DP_DIM; ++k) {
        a.out[k * a.n + i] = f[k];
        finite = finite && dp_isfinite_bits(f[k]);
    }
    if (!finite) atomicExch(&a.status->nonfinite, 1);
}

template <int ACC, int LANES>
__device__ __forceinline__ void dp_scalar_split(const dp_pair_args& a) {
    __shared__ double smem[32];
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long i = t / LANES;
    double v = 0.0;
    if (i < a.n) v = dp_particle_sum<ACC, LANES>(a, i, nullptr, (int)(t % LANES));
    v = dp_block_sum(v, smem);
    if (threadIdx.x == 0) a.partial[blockIdx.x] = v;
}

template <int LANES>
__device__ __forceinline__ void dp_laplacian_split(const dp_pair_args& a) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long i = t / LANES;
    double v = 0.0;
    if (i < a.n) v = dp_particle_sum<DP_ACC_LAPLACE, LANES>(a, i, nullptr, (int)(t % LANES));
#pragma unroll
    for (int off = LANES / 2; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off, LANES);
    if (i < a.n && t % LANES == 0) a.out[i] = v;
}

#if !DP_MLP
#define DP_SPLIT_KERNELS(NAME, LANES)                                                                              \
    extern "C" __global__ void DP_FORCES_BOUNDS dp_forces_##NAME(dp_pair_args a) { dp_forces_split<LANES>(a); }     \
    extern "C" __global__ void DP_FORCES_BOUNDS dp_energy_##NAME(dp_pair_args a) {                                  \
        dp_scalar_split<DP_ACC_ENERGY, LANES>(a);                                                                   \
    }                                                                                                               \
    extern "C" __global__ void DP_FORCES_BOUNDS dp_virial_##NAME(dp_pair_args a) {                                  \
        dp_scalar_split<DP_ACC_VIRIAL, LANES>(a);                                                                   \
    }                                                                                                               \
    extern "C" __global__ void DP_FORCES_BOUNDS dp_laplacian_##NAME(dp_pair_args a) { dp_laplacian_split<LANES>(a); }
#if DP_WARP_SUMS
DP_SPLIT_KERNELS(warp, 32)
#endif
#if DP_QUAD_SUMS
DP_SPLIT_KERNELS(quad, 4)
#endif
#endif

// Per-block partial sums of a scalar pair quantity (energy or virial); the
// host-side reduction kernel adds the partials in a fixed order.
template <int ACC>
__device__ __forceinline__ void dp_scalar_partial(const dp_pair_args& a) {
    __shared__ double smem[32];
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double v = 0.0;
    if (i < a.n) v = dp_particle_sum<ACC>(a, i, nullptr);
    v = dp_block_sum(v, smem);
    if (threadIdx.x == 0) a.partial[blockIdx.x] = v;
}

extern "C" __global__ void __launch_bounds__(256) dp_energy(dp_pair_args a) { dp_scalar_partial<DP_ACC_ENERGY>(a); }

extern "C" __global__ void __launch_bounds__(256) dp_virial(dp_pair_args a) { dp_scalar_partial<DP_ACC_VIRIAL>(a); }

// Per-particle Laplacian of the potential energy (float64 out[i]).
extern "C" __global__ void __launch_bounds__(256) dp_laplacian(dp_pair_args a) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    a.out[i] = dp_particle_sum<DP_ACC_LAPLACE>(a, i, nullptr);
}

// u_cut, f_cut, c_cut of the compiled potential at scaled distances s[i]
// (the reference's pair_potential / pair_force / pair_curvature callables).
extern "C" __global__ void dp_eval_pair(const double* s_in, double* u, double* f, double* c, long long n,
                                        double rcut) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double s = s_in[i];
    if (s > rcut) {
        u[i] = 0.0;
        f[i] = 0.0;
        c[i] = 0.0;
        return;
    }
    const real_t sr = (real_t)s, sinv = real_t(1) / sr;
    u[i] = (double)dp_pair_u<real_t>(sr, sinv);
    f[i] = (double)dp_pair_f<real_t>(sr, sinv);
    c[i] = (double)dp_pair_c<real_t>(sr, sinv);
}

#if DP_MLP
// ---------------------------------------------------------------------------
// Pair surrogate path: the generated dp_pair_* functions hold the cheap
// terms of the potential (in float32), the network of mlp_common.cuh the
// costly ones; sigma = epsilon = 1 in this mode. Each unique pair inside
// r_cut is evaluated once (Newton's third law): a warp owns 32 particles, and
// before each round every lane advances along its particle's neighbour list
// to the next partner it owns (dp_owns_pair) inside r_cut, so a round's 32 network rows are
// all real pairs (two 16-row tensor-core tiles); each row's result goes back
// to the lane owning the pair, which adds
//   f/r = f_cheap(r)/r + (f r)_nn / r^2,   u = u_cheap(r) + u_nn.
// Forces: +F to i in registers, -F to j as a 64-bit fixed-point atomic add
// (integer sums are exact, so the result does not depend on the order of the
// atomics; 2^-32 resolution); dp_mlp_forces_finish converts the sums to float64.
#define DP_MLP_FX_LIMIT 1073741824.0f  // 2^30: larger contributions are flagged

// round(v 2^32) for |v| <= 2^30 from the float's bits (integer shifts, no
// 64-bit conversion instruction); halves round away from zero.
__device__ __forceinline__ long long dp_f2fx32(float v) {
    const uint32_t b = __float_as_uint(v);
    const int e = (int)((b >> 23) & 0xFFu) - 127;  // v = 1.m 2^e
    if (e < -33) return 0;                          // |v 2^32| < 1/2 (zeros and subnormals too)
    const long long m = (long long)((b & 0x7FFFFFu) | 0x800000u);
    const int sh = e + 9;                           // v 2^32 = m 2^(e + 32 - 23)
    const long long r = sh >= 0 ? (m << sh) : ((m + (1LL << (-sh - 1))) >> (-sh));
    return (b >> 31) ? -r : r;
}

__device__ __forceinline__ void dp_mlp_fx_add(unsigned long long* p, float v, bool& bad) {
    bad = bad || !(fabsf(v) < DP_MLP_FX_LIMIT);
    const float c = fminf(fmaxf(v, -DP_MLP_FX_LIMIT), DP_MLP_FX_LIMIT);
    atomicAdd(p, (unsigned long long)dp_f2fx32(c));
}

//
// a.mlp_split lanes share a particle (each takes every mlp_split-th entry of its
// list): a warp holds 32 / mlp_split particles, so that a small system still fills
// the GPU and its longest list takes that many fewer rounds. The rounds are
// bound by latency: 4,000 particles take 39 us with 8 lanes, 203 with one.
template <int ACC>
__device__ __forceinline__ void dp_mlp_pass(const dp_pair_args& a, const dp_mlp_dev* mg, unsigned long long* fx) {
    constexpr int D = DP_DIM;
    __shared__ dp_mlp_dev m;
    __shared__ double red[32];
    dp_mlp_load(&m, mg);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2;
    const long long n = a.n;
    const int split = a.mlp_split;  // 1, 2, 4 or 8
    const long long i = (((long long)blockIdx.x * (blockDim.x >> 5) + warp) * 32 + lane) / split;
    const bool active = i < n;
    const shadow_t* __restrict__ sh = (const shadow_t*)a.shadow;
    uint32_t ui[D];
    if (active) dp_shadow_unpack<D>(sh[i], ui);
    const int c = active ? a.cnt[i] : 0;
    const float rc2 = (float)(a.rcut * a.rcut);
    float f[D];
#pragma unroll
    for (int k = 0; k < D; ++k) f[k] = 0.0f;
    double acc = 0.0;
    bool bad = false;
    int kk = lane % split;
    while (true) {
        // this lane's next unique pair inside r_cut
        bool valid = false;
        int j = 0;
        float q = m.x_mean, df[D];
        while (kk < c && !valid) {
            j = __ldg(a.nl + (long long)kk * n + i);
            kk += split;
            if (!dp_owns_pair(i, j)) continue;
            uint32_t uj[D];
            dp_shadow_unpack<D>(__ldg(sh + j), uj);
            const float qq = dp_shadow_q<D>(ui, uj, a.unit, df);
            if (qq <= rc2) {
                valid = true;
                q = qq;
            }
        }
        if (!__any_sync(0xffffffffu, valid)) break;
        float nn_u = 0.f, nn_f = 0.f;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const float sg = __shfl_sync(0xffffffffu, q, 16 * t + g);
            const float sg8 = __shfl_sync(0xffffffffu, q, 16 * t + g + 8);
            float y[2][2];
            dp_mlp_tile<false>(m, sg, sg8, y);
            const int o = lane - 16 * t;       // row of this lane's own pair in tile t
            const int src = 4 * (o & 7);        // quad holding that row
            const float r0u = __shfl_sync(0xffffffffu, y[0][0], src), r0f = __shfl_sync(0xffffffffu, y[0][1], src);
            const float r1u = __shfl_sync(0xffffffffu, y[1][0], src), r1f = __shfl_sync(0xffffffffu, y[1][1], src);
            if (o >= 0 && o < 16) {
                nn_u = (o < 8) ? r0u : r1u;
                nn_f = (o < 8) ? r0f : r1f;
            }
        }
        if (valid) {
            const float rinv = rsqrtf(q);
            const float r = q * rinv;
            const float fr = dp_pair_f<float>(r, rinv) * rinv + nn_f * m.f_scale * (rinv * rinv);
            if (ACC == DP_ACC_FORCE) {
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    const float fk = fr * df[k];
                    f[k] += fk;
                    dp_mlp_fx_add(fx + (long long)k * n + j, -fk, bad);
                }
            } else if (ACC == DP_ACC_ENERGY) {
                // the host halves the full-list sum: a unique pair counts twice
                acc += 2.0 * (double)(dp_pair_u<float>(r, rinv) + nn_u * m.u_scale);
            } else {
                acc += (double)(fr * q);
            }
        }
    }
    if (ACC == DP_ACC_FORCE) {
        for (int o = 1; o < split; o <<= 1) {
#pragma unroll
            for (int k = 0; k < D; ++k) f[k] += __shfl_xor_sync(0xffffffffu, f[k], o);
        }
        if (active && lane % split == 0) {
#pragma unroll
            for (int k = 0; k < D; ++k) dp_mlp_fx_add(fx + (long long)k * n + i, f[k], bad);
        }
        if (__any_sync(0xffffffffu, bad) && lane == 0) atomicExch(&a.status->nonfinite, 1);
    } else {
        const double v = dp_block_sum(acc, red);
        if (threadIdx.x == 0) a.partial[blockIdx.x] = v;
    }
}

extern "C" __global__ void __launch_bounds__(256, 2) dp_forces_mlp(dp_pair_args a, const dp_mlp_dev* mlp,
                                                                unsigned long long* fx) {
    dp_mlp_pass<DP_ACC_FORCE>(a, mlp, fx);
}
extern "C" __global__ void __launch_bounds__(256, 2) dp_energy_mlp(dp_pair_args a, const dp_mlp_dev* mlp,
                                                                unsigned long long* fx) {
    dp_mlp_pass<DP_ACC_ENERGY>(a, mlp, fx);
}
extern "C" __global__ void __launch_bounds__(256, 2) dp_virial_mlp(dp_pair_args a, const dp_mlp_dev* mlp,
                                                                unsigned long long* fx) {
    dp_mlp_pass<DP_ACC_VIRIAL>(a, mlp, fx);
}

// ---------------------------------------------------------------------------
// The same pass on the fifth-generation tensor cores (dp_umma.cuh): a CTA of
// 128 threads owns 128 particles; per round every thread takes its next unique
// pair inside r_cut and writes that pair's layer-1 activations (bf16 high part
// and remainder) as one row of the 128 x 64 A operand in shared memory; one
// thread issues the 4 K-steps x 2 parts of tcgen05.mma against W2 (bf16, in
// shared memory) into a 128-lane x 64-column fp32 TMEM accumulator; each thread
// then reads its own row back (tcgen05.ld) and finishes layers 2 and 3 for its
// pair, with no exchange between threads.
#define DP_TC_WAIT_LIMIT (1 << 22)

template <int ACC>
__device__ __forceinline__ void dp_mlp_pass_tc(const dp_pair_args& a, const dp_mlp_dev* mg, unsigned long long* fx) {
    constexpr int D = DP_DIM;
    constexpr int ROWS = 128;
    __shared__ __align__(128) unsigned char sA_hi[ROWS * 64 * 2];
    __shared__ __align__(128) unsigned char sA_lo[ROWS * 64 * 2];
    __shared__ __align__(128) unsigned char sB[64 * 64 * 2];
    __shared__ float s_w1[64], s_b1[64], s_b2[64], s_w30[64], s_w31[64], s_misc[6];
    __shared__ __align__(8) uint64_t s_mbar;
    __shared__ uint32_t s_tmem;
    __shared__ double red[32];
    const int tid = threadIdx.x, warp = tid >> 5;
    // network: scalars, and W2 from its packed B fragments into the canonical layout
    if (tid < 64) {
        s_w1[tid] = mg->w1[tid];
        s_b1[tid] = mg->b1[tid];
        s_b2[tid] = mg->b2[tid];
        s_w30[tid] = mg->w3[0][tid];
        s_w31[tid] = mg->w3[1][tid];
    }
    if (tid == 0) {
        s_misc[0] = mg->b3[0];
        s_misc[1] = mg->b3[1];
        s_misc[2] = mg->x_mean;
        s_misc[3] = mg->x_inv_scale;
        s_misc[4] = mg->u_scale;
        s_misc[5] = mg->f_scale;
        dp_mbar_init(&s_mbar, 1);
    }
    for (int t = tid; t < 4 * 8 * 32; t += ROWS) {
        const int lane = t & 31, nt = (t >> 5) & 7, kt = t >> 8;
        const int nrow = nt * 8 + (lane >> 2), k = kt * 16 + 2 * (lane & 3);
        *(uint32_t*)(sB + dp_umma_offset(nrow, k, 64)) = mg->w2frag[t * 2 + 0];
        *(uint32_t*)(sB + dp_umma_offset(nrow, k + 8, 64)) = mg->w2frag[t * 2 + 1];
    }
    if (warp == 0) dp_tmem_alloc(&s_tmem, 64);
    dp_async_smem_fence();
    dp_tc_fence_before();
    __syncthreads();
    dp_tc_fence_after();
    const uint32_t tmem = s_tmem;
    const uint32_t idesc = dp_umma_idesc_bf16<ROWS, 64>();
    const float x_mean = s_misc[2], x_inv = s_misc[3], u_scale = s_misc[4], f_scale = s_misc[5];

    const long long n = a.n;
    const long long i = (long long)blockIdx.x * ROWS + tid;
    const bool active = i < n;
    const shadow_t* __restrict__ sh = (const shadow_t*)a.shadow;
    uint32_t ui[D];
    if (active) dp_shadow_unpack<D>(sh[i], ui);
    const int c = active ? a.cnt[i] : 0;
    const float rc2 = (float)(a.rcut * a.rcut);
    float f[D];
#pragma unroll
    for (int k = 0; k < D; ++k) f[k] = 0.0f;
    double acc = 0.0;
    bool bad = false, timed_out = false;
    uint32_t phase = 0;
    int kk = 0;
    // this thread's next unique pair inside r_cut (the search of round r + 1
    // runs while the tensor core computes round r)
    bool nvalid = false;
    int nj = 0;
    float nq = x_mean;
    auto search = [&]() {
        nvalid = false;
        nq = x_mean;
        while (kk < c && !nvalid) {
            const int jj = __ldg(a.nl + (long long)kk * n + i);
            ++kk;
            if (!dp_owns_pair(i, jj)) continue;
            uint32_t uj[D];
            dp_shadow_unpack<D>(__ldg(sh + jj), uj);
            float dd[D];
            const float qq = dp_shadow_q<D>(ui, uj, a.unit, dd);
            if (qq <= rc2) {
                nvalid = true;
                nj = jj;
                nq = qq;
            }
        }
    };
    search();
    while (true) {
        const bool valid = nvalid;
        const int j = nj;
        const float q = nq;
        // previous round's TMEM reads are complete in every thread past this barrier
        dp_tc_fence_before();
        if (!__syncthreads_or(valid)) break;
        dp_tc_fence_after();
        // layer 1 into row tid of the A operand
        const float x = (q - x_mean) * x_inv;
#pragma unroll
        for (int g8 = 0; g8 < 8; ++g8) {
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int k = g8 * 8 + 2 * e;
                dp_split2(dp_mlp_act<false>(fmaf(s_w1[k], x, s_b1[k])),
                          dp_mlp_act<false>(fmaf(s_w1[k + 1], x, s_b1[k + 1])), hi[e], lo[e]);
            }
            const int o = dp_umma_offset(tid, g8 * 8, ROWS);
            *(uint4*)(sA_hi + o) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *(uint4*)(sA_lo + o) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
        dp_async_smem_fence();
        dp_tc_fence_before();
        __syncthreads();
        dp_tc_fence_after();
        if (tid == 0) {
            const uint32_t a_hi = dp_smem_addr(sA_hi), a_lo = dp_smem_addr(sA_lo), b = dp_smem_addr(sB);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                const uint64_t bd = dp_umma_desc(b + ks * (64 * 32));
                dp_umma_bf16(tmem, dp_umma_desc(a_lo + ks * (ROWS * 32)), bd, idesc, ks > 0 ? 1u : 0u);
                dp_umma_bf16(tmem, dp_umma_desc(a_hi + ks * (ROWS * 32)), bd, idesc, 1u);
            }
            dp_umma_commit(&s_mbar);
        }
        search();  // next round's pair, overlapping the MMAs
        const bool ok = dp_mbar_wait(&s_mbar, phase, DP_TC_WAIT_LIMIT);
        phase ^= 1u;
        if (__syncthreads_or(!ok)) {
            timed_out = true;
            break;
        }
        dp_tc_fence_after();
        // layers 2 and 3 for this thread's pair: two halves of 32 columns
        float y0 = s_misc[0], y1 = s_misc[1];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float z[32];
            dp_tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(half * 32), z);
#pragma unroll
            for (int cc = 0; cc < 32; ++cc) {
                const int col = half * 32 + cc;
                const float h = dp_mlp_act<false>(z[cc] + s_b2[col]);
                y0 = fmaf(h, s_w30[col], y0);
                y1 = fmaf(h, s_w31[col], y1);
            }
        }
        if (valid) {
            const float rinv = rsqrtf(q);
            const float r = q * rinv;
            const float fr = dp_pair_f<float>(r, rinv) * rinv + y1 * f_scale * (rinv * rinv);
            if (ACC == DP_ACC_FORCE) {
                // the displacement again from the partner's shadow (cached), not kept across the round
                uint32_t uj[D];
                dp_shadow_unpack<D>(__ldg(sh + j), uj);
                float df[D];
                dp_shadow_q<D>(ui, uj, a.unit, df);
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    const float fk = fr * df[k];
                    f[k] += fk;
                    dp_mlp_fx_add(fx + (long long)k * n + j, -fk, bad);
                }
            } else if (ACC == DP_ACC_ENERGY) {
                acc += 2.0 * (double)(dp_pair_u<float>(r, rinv) + y0 * u_scale);
            } else {
                acc += (double)(fr * q);
            }
        }
    }
    if (timed_out) {
        // the MMAs of the abandoned round may still be in flight: wait (bounded) before freeing TMEM
        dp_mbar_wait(&s_mbar, phase ^ 1u, DP_TC_WAIT_LIMIT);
        if (tid == 0) atomicExch(&a.status->device_error, 1);
    }
    dp_tc_fence_before();
    __syncthreads();
    if (warp == 0) dp_tmem_dealloc(tmem, 64);
    if (ACC == DP_ACC_FORCE) {
        if (active) {
#pragma unroll
            for (int k = 0; k < D; ++k) dp_mlp_fx_add(fx + (long long)k * n + i, f[k], bad);
        }
        if (bad) atomicExch(&a.status->nonfinite, 1);
    } else {
        const double v = dp_block_sum(acc, red);
        if (threadIdx.x == 0) a.partial[blockIdx.x] = v;
    }
}

extern "C" __global__ void __launch_bounds__(128, 5) dp_forces_mlp_tc(dp_pair_args a, const dp_mlp_dev* mlp,
                                                                      unsigned long long* fx) {
    dp_mlp_pass_tc<DP_ACC_FORCE>(a, mlp, fx);
}
extern "C" __global__ void __launch_bounds__(128, 5) dp_energy_mlp_tc(dp_pair_args a, const dp_mlp_dev* mlp,
                                                                      unsigned long long* fx) {
    dp_mlp_pass_tc<DP_ACC_ENERGY>(a, mlp, fx);
}
extern "C" __global__ void __launch_bounds__(128, 5) dp_virial_mlp_tc(dp_pair_args a, const dp_mlp_dev* mlp,
                                                                      unsigned long long* fx) {
    dp_mlp_pass_tc<DP_ACC_VIRIAL>(a, mlp, fx);
}

// Fixed-point force sums -> float64 forces (SoA), and clear the sums.
extern "C" __global__ void __launch_bounds__(256) dp_mlp_forces_finish(dp_pair_args a, unsigned long long* fx) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.n * DP_DIM) return;
    a.out[t] = (double)(long long)fx[t] * (1.0 / 4294967296.0);
    fx[t] = 0ull;
}
#endif
