// dompap_gpu.cu — GB300 (sm_103a) implementation of the C ABI in
// include/dompap_gpu.h: device state, the statically compiled kernels (cell
// list, Verlet list, integrators, reductions, layout transposes) and the NVRTC
// pipeline that compiles the SymPy-generated pair potential together with
// pair_kernels.cuh.
//
// Design (one process, one GPU, one stream per handle):
//  * particle state lives in HBM as SoA float64 pos/vel/beta/force[k*N + i]
//    plus int32 images; a fixed-point copy of the positions (uint32 per axis,
//    packed in one 8/16-byte vector per particle) feeds the pair pre-filter;
//  * lists hold slots, column-major nl[k*N + i] with counts cnt[i] (in rows for
//    systems of at most a warp per particle), or 16-bit region indices for the
//    brick kernels;
//  * run(steps) launches CUDA graphs of fused steps: groups of steps with one
//    conditional rebuild each in a loop on the device, or, for small systems,
//    steps that rebuild their own lists. After each chunk the host reads the
//    status word; on a list or region overflow it grows the capacity. Grouped
//    steps have stopped at that build and go on from it; other chunks are
//    replayed from their start state.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <nvrtc.h>

#include <dlfcn.h>
#include <sys/stat.h>
#include <unistd.h>

#include <algorithm>
#include <cctype>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <cstdlib>
#include <map>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "dompap_gpu.h"
#include "dp_common.cuh"
#include "dp_integrate.cuh"
#include "dp_umma.cuh"
#include "dp_embedded.h"
#include "mlp_common.cuh"
#include "mlp_train.cuh"  // dp_src_common[], dp_src_pair[] (generated at build time)

// ===========================================================================
// errors
// ===========================================================================
static thread_local std::string g_err;

static int fail(int code, const std::string& msg) {
    g_err = msg;
    return code;
}

#define CK(call)                                                                                     \
    do {                                                                                             \
        cudaError_t e_ = (call);                                                                     \
        if (e_ != cudaSuccess) return fail(DP_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

#define RET(call)              \
    do {                       \
        int rc_ = (call);      \
        if (rc_ != DP_OK) return rc_; \
    } while (0)

static inline unsigned grid_for(long long n, int block) {
    long long g = (n + block - 1) / block;
    return (unsigned)std::max<long long>(1, g);
}

// ===========================================================================
// static kernels
// ===========================================================================
namespace {

constexpr int kBlock = 256;

// Host layout (particle id major, (n, dim)) <-> device SoA in slot order:
// element (id, k) lives at k * n + slot_of[id] (slot_of null: slot = id). The
// host side is read or written contiguously (it may be page-locked host memory
// read over the host link); the scattered side is device memory.
template <typename T>
__global__ void k_host_to_slots(const T* __restrict__ in, T* __restrict__ out, const int32_t* __restrict__ slot_of,
                                long long n, int dim) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * dim) return;
    const long long i = t / dim;
    const int k = (int)(t - i * dim);
    out[k * n + (slot_of ? slot_of[i] : i)] = in[t];
}

template <typename T>
__global__ void k_slots_to_host(const T* __restrict__ in, T* __restrict__ out, const int32_t* __restrict__ slot_of,
                                long long n, int dim) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * dim) return;
    const long long i = t / dim;
    const int k = (int)(t - i * dim);
    out[t] = in[k * n + (slot_of ? slot_of[i] : i)];
}

struct ShadowArgs {
    const double* pos;
    void* shadow;
    void* pos64;
    dp_dev_status* st;
    long long n;
    double scale64[DP_MAX_DIM];
    int shift64[DP_MAX_DIM];
    double box[DP_MAX_DIM];
};

// 64-bit fixed point of one coordinate, wrapped into [0, L) first when needed.
__device__ __forceinline__ unsigned long long fixed64_wrapped(double x, double L, double scale64) {
    if (!(x >= 0.0 && x < L)) x -= floor(x / L) * L;
    return dp_fixed64_of(x * scale64);
}

// Fixed-point forms of all positions (the 64-bit X of the position wrapped
// into the box, the shadow its upper word, as the integrators write them);
// flags coordinates outside [-L/4, 5L/4), for which the single-shift image is
// not the nearest one. One float64 product per coordinate in the box: its
// bit pattern is the in-box test.
template <int D>
__global__ void k_shadow(ShadowArgs a) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    uint32_t u[D];
    unsigned long long X[D];
    bool far = false;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        const double x = a.pos[k * a.n + i];
        double p = x * a.scale64[k];
        const long long pb = __double_as_longlong(p);
        if (!(pb >= 0 && pb < 0x43F0000000000000LL)) {  // p outside [0, 2^64): wrap a copy
            far = far || !(x >= -0.25 * a.box[k] && x < 1.25 * a.box[k]);
            const double w = x - floor(x / a.box[k]) * a.box[k];
            p = (w >= 0.0 && w < a.box[k]) ? w * a.scale64[k] : 0.0;
        }
        X[k] = dp_fixed64_of(p);
        u[k] = (uint32_t)(X[k] >> 32);
        X[k] <<= a.shift64[k];
    }
    ((typename dp_shadow_t<D>::type*)a.shadow)[i] = dp_shadow_pack<D>(u);
    ((typename dp_fixed64_t<D>::type*)a.pos64)[i] = dp_fixed64_pack<D>(X);
    if (far) atomicExch(&a.st->far, 1);
}

// --------------------------- skin test ------------------------------------
// neighbor_list_is_old (dompap/neighbor_list.py:183-201): rebuild when some
// particle's min-image displacement^2 since the last build exceeds (skin/2)^2.
// The displacement since the last build is read from the fixed-point shadows
// in float32; only when it lies within the error bound of (skin/2)^2 is it
// recomputed in float64 exactly as the reference does.
struct SkinArgs {
    const double* pos;
    const double* pos_ref;
    const void* shadow;
    const void* shadow_ref;
    dp_dev_status* st;
    long long n;
    double box[DP_MAX_DIM];
    float unit[DP_MAX_DIM];
    double thr;    // (0.5 * skin)^2
    float thr_lo;  // below: certainly not old
    float thr_hi;  // above: certainly old
};

template <int D>
__global__ void k_skin_check(SkinArgs a) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    bool old = false;
    if (i < a.n) {
        typedef typename dp_shadow_t<D>::type sh_t;
        uint32_t u[D];
        dp_shadow_unpack<D>(((const sh_t*)a.shadow)[i], u);
        double x[D];
#pragma unroll
        for (int k = 0; k < D; ++k) x[k] = a.pos[k * a.n + i];
        old = dp_skin_old<D>(a.shadow_ref, a.pos_ref, a.n, a.unit, a.box, a.thr, a.thr_lo, a.thr_hi, i, u, x,
                             a.st->far != 0 || a.st->ref_far != 0);
    }
    if (__any_sync(0xffffffffu, old) && (threadIdx.x & 31) == 0) atomicExch(&a.st->need_rebuild, 1);
}

// --------------------------- cell binning ---------------------------------
// The cell list of dompap/neighbor_list.py:42-180 as a counting sort. Cells
// are at least `cutoff` wide plus an absolute margin for the rounding of the
// fixed-point shadows (nc = floor(L / w) per axis, >= 3), so every pair
// closer than the cutoff lies in the 3^D stencil of its cell; the reference
// uses cells of width `cutoff` with nc = ceil(L / cutoff) and misses pairs
// when L / cutoff is not an integer. A particle's cell comes from its shadow
// in integer arithmetic, c_k = (u_k nc_k) >> 32, i.e. from its periodic image
// in [0, L). Cells are keyed in Morton (Z) order of their coordinates
// (row-major when the padded Morton range would be too large), counted,
// prefix-summed into contiguous slot ranges, and each particle is given a
// slot in its cell's range, ties ordered by particle id, so that the order is
// a function of the positions alone. The per-particle state then moves into
// that order (k_permute): the partners a step gathers lie close together in
// memory, and each cell of the Verlet build is one contiguous range.
struct BinArgs {
    const void* shadow;    // shadows of the current slots
    const void* shadow_alt;  // the same while the second set of position buffers is current
    const int32_t* order;  // particle id of each current slot
    int32_t* key;          // [n] cell key of each current slot
    int32_t* rank;         // [n] arrival rank within its cell (atomic)
    int32_t* bin_cnt;      // [nbins] particles per cell key
    int32_t* bin_start;    // [nbins + 1] first slot of each cell key
    int32_t* bin_part;     // [ceil(nbins / kScanTile)] scan partial sums
    int32_t* src_of;       // [n] current slot of the particle that new slot t receives
    dp_dev_status* st;
    long long n;
    long long nbins;
    int nc[DP_MAX_DIM];
    int morton;            // 1: Morton keys on the power-of-two padded grid
};

constexpr int kScanThreads = 1024;
constexpr int kScanPer = 4;
constexpr int kScanTile = kScanThreads * kScanPer;

// Bit interleaving for Morton keys: bit b of x moves to bit D b.
template <int D>
__device__ __forceinline__ uint32_t dp_spread_bits(uint32_t x);
template <>
__device__ __forceinline__ uint32_t dp_spread_bits<2>(uint32_t x) {
    x &= 0xFFFFu;
    x = (x | (x << 8)) & 0x00FF00FFu;
    x = (x | (x << 4)) & 0x0F0F0F0Fu;
    x = (x | (x << 2)) & 0x33333333u;
    return (x | (x << 1)) & 0x55555555u;
}
template <>
__device__ __forceinline__ uint32_t dp_spread_bits<3>(uint32_t x) {
    x &= 0x3FFu;
    x = (x | (x << 16)) & 0x030000FFu;
    x = (x | (x << 8)) & 0x0300F00Fu;
    x = (x | (x << 4)) & 0x030C30C3u;
    return (x | (x << 2)) & 0x09249249u;
}
template <>
__device__ __forceinline__ uint32_t dp_spread_bits<4>(uint32_t x) {
    x &= 0xFFu;
    x = (x | (x << 12)) & 0x000F000Fu;
    x = (x | (x << 6)) & 0x03030303u;
    return (x | (x << 3)) & 0x11111111u;
}

// Cell coordinates of a shadow (fixed-point position in [0, 2^32) per axis).
template <int D>
__device__ __forceinline__ void shadow_cell(const uint32_t* u, const int* nc, int* c) {
#pragma unroll
    for (int k = 0; k < D; ++k) c[k] = (int)(((unsigned long long)u[k] * (unsigned)nc[k]) >> 32);
}

template <int D>
__device__ __forceinline__ int cell_key(const int* c, const int* nc, int morton) {
    if (morton) {
        uint32_t key = 0;
#pragma unroll
        for (int k = 0; k < D; ++k) key |= dp_spread_bits<D>((uint32_t)c[k]) << (D - 1 - k);
        return (int)key;
    }
    int l = c[0];
#pragma unroll
    for (int k = 1; k < D; ++k) l = l * nc[k] + c[k];
    return l;
}

__global__ void k_bin_clear(BinArgs a) {
    if (!a.st->need_rebuild) return;
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < a.nbins;
         c += (long long)gridDim.x * blockDim.x)
        a.bin_cnt[c] = 0;
}

template <int D>
__global__ void k_bin_count(BinArgs a) {
    if (!a.st->need_rebuild) return;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    typedef typename dp_shadow_t<D>::type sh_t;
    uint32_t u[D];
    dp_shadow_unpack<D>(((const sh_t*)(a.st->parity ? a.shadow_alt : a.shadow))[i], u);
    int c[D];
    shadow_cell<D>(u, a.nc, c);
    const int key = cell_key<D>(c, a.nc, a.morton);
    a.key[i] = key;
    a.rank[i] = atomicAdd(a.bin_cnt + key, 1);
}

// Exclusive scan of one value per thread over a block of kScanThreads.
__device__ __forceinline__ int block_exclusive_scan(int v, int* smem, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) smem[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = lane < nwarps ? smem[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        smem[lane] = w;
    }
    __syncthreads();
    const int before = warp ? smem[warp - 1] : 0;
    *total = smem[nwarps - 1];
    __syncthreads();
    return before + x - v;
}

// Scan of the cell counts: per-tile sums, a one-block scan of those, then
// each tile's exclusive scan plus its offset (bin_start[nbins] = n).
__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(BinArgs a) {
    if (!a.st->need_rebuild) return;
    __shared__ int smem[32];
    const long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanPer;
    int v = 0;
#pragma unroll
    for (int t = 0; t < kScanPer; ++t)
        if (base + t < a.nbins) v += a.bin_cnt[base + t];
    int total = 0;
    block_exclusive_scan(v, smem, &total);
    if (threadIdx.x == 0) a.bin_part[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_top(BinArgs a, int parts) {
    if (!a.st->need_rebuild) return;
    __shared__ int smem[32];
    const int per = (parts + kScanThreads - 1) / kScanThreads;
    const int b = threadIdx.x * per;
    int v = 0;
    for (int t = 0; t < per; ++t)
        if (b + t < parts) v += a.bin_part[b + t];
    int total = 0;
    int run = block_exclusive_scan(v, smem, &total);
    for (int t = 0; t < per; ++t)
        if (b + t < parts) {
            const int x = a.bin_part[b + t];
            a.bin_part[b + t] = run;
            run += x;
        }
}

__global__ void __launch_bounds__(kScanThreads) k_scan_down(BinArgs a) {
    if (!a.st->need_rebuild) return;
    __shared__ int smem[32];
    const long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanPer;
    int c[kScanPer];
    int v = 0;
#pragma unroll
    for (int t = 0; t < kScanPer; ++t) {
        c[t] = base + t < a.nbins ? a.bin_cnt[base + t] : 0;
        v += c[t];
    }
    int total = 0;
    int run = a.bin_part[blockIdx.x] + block_exclusive_scan(v, smem, &total);
#pragma unroll
    for (int t = 0; t < kScanPer; ++t)
        if (base + t < a.nbins) {
            a.bin_start[base + t] = run;
            run += c[t];
        }
    if (blockIdx.x == 0 && threadIdx.x == 0) a.bin_start[a.nbins] = (int)a.n;
}

__global__ void k_bin_scatter(BinArgs a) {
    if (!a.st->need_rebuild) return;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    a.src_of[a.bin_start[a.key[i]] + a.rank[i]] = (int32_t)i;
}

// Each cell's range ordered by particle id (the atomic ranks are not
// deterministic; the result is): four lanes a cell, each entry's place the
// number of smaller ids in its cell. Ids and slots of up to kSortCell entries lie
// in shared memory, those of a longer cell in `key` and `rank`, which have done
// their work by now. (Insertion waits for every step before the next: with one
// thread a cell of 25 entries 46 us at 21,000 particles, longer than the rest of
// the binning together; cells of 109, in 4-D, 1.5 to 2.2 ms at 262,144.)
constexpr int kSortLanes = 4;
constexpr int kSortCell = 48;

__global__ void __launch_bounds__(kBlock) k_bin_sort(BinArgs a) {
    if (!a.st->need_rebuild) return;
    __shared__ int32_t slot[kBlock / kSortLanes][kSortCell], id[kBlock / kSortLanes][kSortCell];
    const int q = threadIdx.x / kSortLanes, l = threadIdx.x % kSortLanes;
    const long long b = (long long)blockIdx.x * (kBlock / kSortLanes) + q;
    const bool cell = b < a.nbins;
    const int lo = cell ? a.bin_start[b] : 0, m = cell ? a.bin_start[b + 1] - lo : 0;
    const bool fits = m <= kSortCell;
    for (int t = l; t < m; t += kSortLanes) {
        const int32_t v = a.src_of[lo + t];
        if (fits) {
            slot[q][t] = v;
            id[q][t] = a.order[v];
        } else {
            a.key[lo + t] = a.order[v];
        }
    }
    __syncwarp();
    if (fits) {
        for (int t = l; t < m; t += kSortLanes) {
            const int32_t mine = id[q][t];
            int place = 0;
            for (int u = 0; u < m; ++u) place += id[q][u] < mine;
            a.src_of[lo + place] = slot[q][t];
        }
    } else {
        for (int t = l; t < m; t += kSortLanes) {
            const int32_t mine = a.key[lo + t];
            int place = 0;
#pragma unroll 4
            for (int u = 0; u < m; ++u) place += a.key[lo + u] < mine;
            a.rank[lo + place] = a.src_of[lo + t];
        }
    }
    __syncwarp();
    if (!fits)
        for (int t = l; t < m; t += kSortLanes) a.src_of[lo + t] = a.rank[lo + t];
}

// --------------------------- permutation of the state ----------------------
// Arrays that move with their particle: element `esize` bytes, `comps`
// components at a stride of n elements (SoA), or one vector per particle.
struct PermArray {
    void* data;     // the state array
    void* scratch;  // same shape, receives the permuted copy
    int esize;      // 1, 4, 8, 16 or 32
    int comps;
    int alt;        // scratch is the second set of position buffers, the source while that is current
};

constexpr int kMaxPermArrays = 12;

struct PermArgs {
    PermArray arr[kMaxPermArrays];
    int count;
    const int32_t* src_of;  // new slot t <- current slot src_of[t] (null: copy back)
    const int32_t* order;   // particle id of each current slot
    int32_t* slot_of;       // [n] slot of each particle id (updated)
    dp_dev_status* st;
    long long n;
};

// Copy the components of one particle's entry: every load is issued before
// the first store (independent loads in flight), element type by size.
template <typename T>
__device__ __forceinline__ void copy_comps(const void* src, void* dst, long long from, long long to, long long n,
                                           int comps) {
    T v[DP_MAX_DIM];
#pragma unroll
    for (int k = 0; k < DP_MAX_DIM; ++k)
        if (k < comps) v[k] = ((const T*)src)[k * n + from];
#pragma unroll
    for (int k = 0; k < DP_MAX_DIM; ++k)
        if (k < comps) ((T*)dst)[k * n + to] = v[k];
}

__device__ __forceinline__ void copy_entry(const PermArray& a, const void* src, void* dst, long long from,
                                           long long to, long long n) {
    switch (a.esize) {
        case 1: copy_comps<uint8_t>(src, dst, from, to, n, a.comps); break;
        case 4: copy_comps<uint32_t>(src, dst, from, to, n, a.comps); break;
        case 8: copy_comps<uint2>(src, dst, from, to, n, a.comps); break;
        case 16: copy_comps<uint4>(src, dst, from, to, n, 1); break;
        default: {  // 32 bytes: two 16-byte halves
            const uint4 lo = ((const uint4*)src)[2 * from], hi = ((const uint4*)src)[2 * from + 1];
            ((uint4*)dst)[2 * to] = lo;
            ((uint4*)dst)[2 * to + 1] = hi;
        }
    }
}

// Gather every state array into cell order (into the scratch arrays) and
// record the new slot of each particle id. One array per blockIdx.y, so the
// arrays are copied side by side rather than one after another per thread.
__global__ void k_permute(PermArgs p) {
    if (!p.st->need_rebuild) return;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= p.n) return;
    const long long o = p.src_of[t];
    const PermArray a = p.arr[blockIdx.y];
    if (a.alt && p.st->parity)
        copy_entry(a, a.scratch, a.data, o, t, p.n);
    else
        copy_entry(a, a.data, a.scratch, o, t, p.n);
    if (blockIdx.y == 0) p.slot_of[p.order[o]] = (int32_t)t;
}

// The permuted copies back into the state arrays (the kernels captured after
// a rebuild read the state at fixed addresses).
__global__ void k_permute_back(PermArgs p) {
    if (!p.st->need_rebuild) return;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= p.n) return;
    const PermArray a = p.arr[blockIdx.y];
    if (a.alt && p.st->parity) return;  // already there
    copy_entry(a, a.scratch, a.data, t, t, p.n);
}

__global__ void k_iota(int32_t* a, int32_t* b, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    a[i] = (int32_t)i;
    b[i] = (int32_t)i;
}

// slot_of from order (after a restore of the backed-up order).
__global__ void k_invert_order(const int32_t* order, int32_t* slot_of, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    slot_of[order[i]] = (int32_t)i;
}

// --------------------------- Verlet list ----------------------------------
// get_neighbor_list_double_loop (dompap/neighbor_list.py:7-39): m is a
// neighbour of n when sqrt(sum d^2) < cutoff with the single-shift minimum
// image, tested in float64 without FMA (bit-identical pair set).
struct NlArgs {
    const double* pos;
    double* pos_ref;
    const void* shadow;
    void* shadow_ref;
    int32_t* nl;
    int32_t* cnt;
    const int32_t* bin_start;  // cell ranges of the cell build
    const int32_t* src_of;     // slot of each entry of the ranges (null: the entries are the slots)
    dp_dev_status* st;
    long long n;
    long long nl_k, nl_i;      // k_nl_build_rows: entry k of slot i at nl[k nl_k + i nl_i] (else column-major)
    int kcap;
    int morton;
    int nc[DP_MAX_DIM];
    double box[DP_MAX_DIM];
    float unit[DP_MAX_DIM];
    double cutoff;
    float lo2;  // float32 r^2 below this: certainly inside the cutoff
    float hi2;  // float32 r^2 above this: certainly outside
    int half;   // 1: only the partners particle i owns (dp_owns_pair; the surrogate mode uses each pair once)
};

template <int D>
__global__ void __launch_bounds__(kBlock) k_nl_build_cells(NlArgs a) {
    if (!a.st->need_rebuild) return;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    typedef typename dp_shadow_t<D>::type sh_t;
    const sh_t* sh = (const sh_t*)a.shadow;
    const bool far = a.st->far != 0;
    const long long n = a.n;
    double xi[D];
#pragma unroll
    for (int k = 0; k < D; ++k) xi[k] = a.pos[k * n + i];
    const sh_t shi = sh[i];
    uint32_t ui[D];
    dp_shadow_unpack<D>(shi, ui);
    int ci[D];
    shadow_cell<D>(ui, a.nc, ci);
    // each axis' share of the key for the cells at offsets -1, 0, +1 (periodic);
    // a stencil cell's key is the sum of one share per axis (Morton: disjoint
    // bits; row-major: coordinate times the axis stride)
    int part[D][3];
    {
        int stride = 1;
#pragma unroll
        for (int k = D - 1; k >= 0; --k) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                int c = ci[k] + d - 1;
                if (c < 0) c += a.nc[k];
                if (c >= a.nc[k]) c -= a.nc[k];
                part[k][d] = a.morton ? (int)(dp_spread_bits<D>((uint32_t)c) << (D - 1 - k)) : c * stride;
            }
            stride *= a.nc[k];
        }
    }
    int count = 0;
    int stencil = 1;
#pragma unroll
    for (int k = 0; k < D; ++k) stencil *= 3;
    for (int s = 0; s < stencil; ++s) {
        int key = 0;
        int rem = s;
#pragma unroll
        for (int k = D - 1; k >= 0; --k) {
            const int d = rem % 3;
            rem /= 3;
            key += d == 0 ? part[k][0] : (d == 1 ? part[k][1] : part[k][2]);
        }
        const int lo = __ldg(a.bin_start + key), hi = __ldg(a.bin_start + key + 1);
        for (int t = lo; t < hi; ++t) {
            const int j = a.src_of ? __ldg(a.src_of + t) : t;
            if (a.half ? !dp_owns_pair(i, j) : j == i) continue;
            // float32 pre-test on the fixed-point displacement (nearest image,
            // never longer than the single-shift one); float64 only near the cutoff
            uint32_t uj[D];
            dp_shadow_unpack<D>(__ldg(sh + j), uj);
            float df[D];
            const float qf = dp_shadow_q<D>(ui, uj, a.unit, df);
            if (qf > a.hi2) continue;
            bool inside = qf < a.lo2 && !far;
            if (!inside) {
                double d[D];
#pragma unroll
                for (int k = 0; k < D; ++k) d[k] = dp_min_image(xi[k] - a.pos[k * n + j], a.box[k]);
                inside = sqrt(dp_sqsum_exact<D>(d)) < a.cutoff;
            }
            if (inside) {
                if (count < a.kcap) a.nl[(long long)count * n + i] = j;
                ++count;
            }
        }
    }
    a.cnt[i] = min(count, a.kcap);
    atomicMax(&a.st->max_neighbors, count);
#pragma unroll
    for (int k = 0; k < D; ++k) a.pos_ref[k * n + i] = xi[k];
    ((sh_t*)a.shadow_ref)[i] = shi;
}

// The same list built brick by brick (a brick: 2^b cells that follow one
// another in Morton order, i.e. consecutive slots). A CTA gathers the brick's
// region - the particles within the cutoff of the brick's box - into shared
// memory and tests every entry against every particle of the brick.
//
// Tested one pair a lane that is bound by instruction issue (~15 a pair, and
// a region holds ~15 times the listed partners), so the distances come from
// the tensor cores: |x_i - x_j|^2 = |x_i|^2 + |x_j|^2 - 2 x_i x_j is a product of
// two 16-vectors (each coordinate as fp16 high and low part, the two squares
// likewise), one mma.m16n8k16 gives it for 16 particles x 8 entries minus the
// cutoff's square, and the sign bits go into the list masks by one funnel shift
// each. The product's error is at most kBrickErr of the largest coordinate
// squared (coordinates relative to the brick's centre in units of half the
// cutoff); a lane that saw a value within that and the float bracket of the cutoff re-tests
// its candidates as k_nl_build_cells does, so the pair set stays exact.
// OUT32: column-major lists of slots (k_nl_build_cells' format, also half
// lists); otherwise 16-bit region indices in chunks of 8 for the brick kernels
// (brick_kernels.cuh), the last chunk filled up with index 0. A whole rebuild (binning, permutation, lists),
// before (k_nl_build_cells, cells sorted by one thread each) and now: 500,000 LJ
// particles 824 -> 519 us, 108,000 315 -> 183, 20,672 244 -> 91, the mixture of
// 256,000 718 -> 397.
struct BrickArgs {
    const int4* base;  // first cell of each brick
    int4* info;        // (first slot, particles, region entries, 0)
    int32_t* slots;    // [bricks][cap] slots of the region entries
    uint4* list;
    int cap;           // region entries per brick
    int cells;         // region cells per brick
    int keys;          // cells per brick (2^b)
    int ext[DP_MAX_DIM];    // region cells per axis (brick + 2)
    float unit[DP_MAX_DIM]; // fixed point to half cutoffs
    float cut;              // the squared cutoff in those units: 4 and the margins
    float alarm;            // a value this close to the cut does not decide
};

constexpr int kBrickThreads = 256;    // at most; 8 warps of 16 particles
// Error of the product per axis and largest coordinate squared: 6 2^-22 for
// what the fp16 parts of the coordinates drop, 2 2^-22 for the squares', 16 2^-22
// for the additions of 16 terms up to twice it in size; twice that.
constexpr float kBrickErr = 1.2e-5f;

__device__ __forceinline__ uint32_t dp_half2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ float dp_half_round(float x) {
    float r;
    asm("{ .reg .f16 h; cvt.rn.f16.f32 h, %1; cvt.f32.f16 %0, h; }" : "=f"(r) : "f"(x));
    return r;
}

// The 16 factors of a position x: per axis (hi, hi, lo) against (-2 hi, -2 lo,
// -2 hi), then |x|^2 (hi, lo) against (1, 1) and (1, 1) against |x|^2, as words of
// two; LEFT: the particle's side.
template <int D, bool LEFT>
__device__ __forceinline__ void dp_brick_factors(const float* x, uint32_t* w) {
    float v[16];
#pragma unroll
    for (int k = 0; k < 12; ++k) v[k] = 0.0f;
    float n2 = 0.0f;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        const float hi = dp_half_round(x[k]), lo = x[k] - hi;
        v[3 * k] = LEFT ? hi : -2.0f * hi;
        v[3 * k + 1] = LEFT ? hi : -2.0f * lo;
        v[3 * k + 2] = LEFT ? lo : -2.0f * hi;
        n2 = fmaf(x[k], x[k], n2);
    }
    const float nh = dp_half_round(n2), nl = n2 - nh;
    v[12] = LEFT ? nh : 1.0f;
    v[13] = LEFT ? nl : 1.0f;
    v[14] = LEFT ? 1.0f : nh;
    v[15] = LEFT ? 1.0f : nl;
#pragma unroll
    for (int k = 0; k < 8; ++k) w[k] = dp_half2(v[2 * k], v[2 * k + 1]);
}

__device__ __forceinline__ void dp_mma_f16(float* d, const uint32_t* a, uint2 b, float c) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y), "f"(c));
}

// Squared float distance from a fixed-point position to a box (centre and half
// sides in fixed point) in the periodic system.
template <int D>
__device__ __forceinline__ float dp_box_q(const uint32_t* u, const uint32_t* centre, const uint32_t* half,
                                          const float* unit) {
    float q = 0.0f;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        const int d = (int)(u[k] - centre[k]);
        const uint32_t m = d < 0 ? 0u - (uint32_t)d : (uint32_t)d;
        const float x = (m > half[k] ? __uint2float_rn(m - half[k]) : 0.0f) * unit[k];
        q = fmaf(x, x, q);
    }
    return q;
}

template <int D, bool OUT32>
__global__ void __launch_bounds__(kBrickThreads, 3) k_brick_build(NlArgs a, BrickArgs b) {
    if (!a.st->need_rebuild) return;
    extern __shared__ __align__(16) unsigned char brick_smem[];
    __shared__ int scan[32];
    typedef typename dp_shadow_t<D>::type sh_t;
    uint2* frag = (uint2*)brick_smem;                // [cap + 8][4] entries' factors: words c and c + 4 side by side
    int* rslot = (int*)(frag + 4 * (b.cap + 8));     // [cap] slots
    int* off = rslot + b.cap;                        // [cells + 1] candidates before each cell
    int* start = off + b.cells + 1;                  // [cells] first slot
    uint16_t* entry_of = (uint16_t*)(start + b.cells);  // [cap] region entry of each particle of the brick
    const sh_t* __restrict__ sh = (const sh_t*)a.shadow;
    const long long n = a.n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int4 base4 = b.base[blockIdx.x];
    const int base[4] = {base4.x, base4.y, base4.z, base4.w};
    const int key0 = cell_key<D>(base, a.nc, 1);
    const int first = a.bin_start[key0], count = a.bin_start[key0 + b.keys] - first;
    if (count == 0) {  // uniform
        if (threadIdx.x == 0) b.info[blockIdx.x] = make_int4(first, 0, 0, 0);
        return;
    }
    // region cells: counts, then their exclusive scan (consecutive cells per thread)
    const int per = (b.cells + (int)blockDim.x - 1) / (int)blockDim.x;
    int sum = 0;
    for (int q = 0; q < per; ++q) {
        const int r = (int)threadIdx.x * per + q;
        if (r >= b.cells) break;
        int rem = r, c[4];
#pragma unroll
        for (int k = D - 1; k >= 0; --k) {
            int x = base[k] + rem % b.ext[k] - 1;
            rem /= b.ext[k];
            if (x < 0) x += a.nc[k];
            if (x >= a.nc[k]) x -= a.nc[k];
            c[k] = x;
        }
        const int key = cell_key<D>(c, a.nc, 1);
        const int lo = __ldg(a.bin_start + key), m = __ldg(a.bin_start + key + 1) - lo;
        start[r] = lo;
        off[r] = m;
        sum += m;
    }
    int total = 0;
    int run = block_exclusive_scan(sum, scan, &total);
    for (int q = 0; q < per; ++q) {
        const int r = (int)threadIdx.x * per + q;
        if (r >= b.cells) break;
        const int m = off[r];
        off[r] = run;
        run += m;
    }
    if (threadIdx.x == 0) off[b.cells] = total;
    __syncthreads();
    // the brick's box in fixed point (a unit wider than its cells on each side)
    uint32_t box_c[D], box_h[D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
        const unsigned long long dim = (unsigned long long)(b.ext[k] - 2), nck = (unsigned long long)a.nc[k];
        box_c[k] = (uint32_t)(((2ull * (unsigned)base[k] + dim) << 31) / nck);
        box_h[k] = (uint32_t)min(((dim << 31) / nck) + 2ull, 0x7FFFFFFFull);
    }
    // entries: the candidates within reach of the box, in order
    int entries = 0;
    for (int t0 = 0; t0 < total; t0 += blockDim.x) {
        const int t = t0 + (int)threadIdx.x;
        bool keep = false;
        int j = 0;
        uint32_t u[4] = {0u, 0u, 0u, 0u};
        if (t < total) {
            int cell = 0, hi = b.cells;  // off[cell] <= t < off[hi]
            while (hi - cell > 1) {
                const int mid = (cell + hi) >> 1;
                if (off[mid] <= t) cell = mid; else hi = mid;
            }
            j = start[cell] + t - off[cell];
            dp_shadow_unpack<D>(__ldg(sh + j), u);
            keep = dp_box_q<D>(u, box_c, box_h, a.unit) <= a.hi2;
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) scan[warp] = __popc(m);
        __syncthreads();
        int before = entries, all = 0;
        for (int w = 0; w < warps; ++w) {
            const int c = scan[w];
            if (w < warp) before += c;
            all += c;
        }
        const int at = before + __popc(m & ((1u << lane) - 1u));
        if (keep && at < b.cap) {
            float x[D];
#pragma unroll
            for (int k = 0; k < D; ++k) x[k] = (float)(int)(u[k] - box_c[k]) * b.unit[k];
            uint32_t w[8];
            dp_brick_factors<D, false>(x, w);
#pragma unroll
            for (int c = 0; c < 4; ++c) frag[4 * at + c] = make_uint2(w[c], w[c + 4]);
            rslot[at] = j;
            if (!OUT32) b.slots[(long long)blockIdx.x * b.cap + at] = j;
            if (j >= first && j < first + min(count, b.cap)) entry_of[j - first] = (uint16_t)at;
        }
        entries += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        b.info[blockIdx.x] = make_int4(first, count, min(entries, b.cap), 0);
        if (entries > b.cap) atomicMax(&a.st->cell_overflow, entries);
    }
    if (entries > b.cap) {  // uniform; no list: the host makes room and has it built again before it counts
        for (int p = threadIdx.x; p < count; p += blockDim.x) a.cnt[first + p] = 0;
        return;
    }
    const bool far = a.st->far != 0;
    const int g = lane >> 2, c = lane & 3;
    const float cut = -b.cut;
    int best = 0;
    for (int p0 = warp * 16; p0 < count; p0 += warps * 16) {
        // rows g and g + 8 of this warp's 16 particles
        int row[2], self[2], found[2] = {0, 0};
        uint32_t am[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int p = p0 + g + 8 * h;
            const bool active = p < count;
            row[h] = active ? first + p : -1;
            self[h] = active ? entry_of[p] : -1;
            uint32_t u[D], w[8];
            dp_shadow_unpack<D>(sh[active ? first + p : first], u);
            float x[D];
#pragma unroll
            for (int k = 0; k < D; ++k) x[k] = (float)(int)(u[k] - box_c[k]) * b.unit[k];
            dp_brick_factors<D, true>(x, w);
            // an idle row: |x|^2 beyond everything
            if (!active) {
#pragma unroll
                for (int k = 0; k < 6; ++k) w[k] = 0u;
                w[6] = dp_half2(60000.0f, 0.0f);
            }
            am[h] = c == 0 ? w[0] : (c == 1 ? w[1] : (c == 2 ? w[2] : w[3]));
            am[2 + h] = c == 0 ? w[4] : (c == 1 ? w[5] : (c == 2 ? w[6] : w[7]));
        }
        for (int t0 = 0; t0 < entries; t0 += 128) {
            const int len = min(128, entries - t0), tiles = (len + 7) >> 3;
            uint32_t mask[2] = {0u, 0u};
            float nearest = 1e30f;
            const uint2* fr = frag + 4 * (t0 + g) + c;
#pragma unroll 4
            for (int t = 0; t < tiles; ++t) {
                float d[4];
                dp_mma_f16(d, am, fr[32 * t], cut);
                mask[0] = __funnelshift_l(__float_as_uint(d[0]), mask[0], 1);
                mask[0] = __funnelshift_l(__float_as_uint(d[1]), mask[0], 1);
                mask[1] = __funnelshift_l(__float_as_uint(d[2]), mask[1], 1);
                mask[1] = __funnelshift_l(__float_as_uint(d[3]), mask[1], 1);
                nearest = fminf(fminf(nearest, fminf(fabsf(d[0]), fabsf(d[1]))), fminf(fabsf(d[2]), fabsf(d[3])));
            }
            // bit 31 - s: entry t0 + 8 (s / 2) + 2 c + s % 2
            const int valid = 2 * (len >> 3) + min(max((len & 7) - 2 * c, 0), 2);
            const uint32_t live = valid > 0 ? 0xFFFFFFFFu << (32 - valid) : 0u;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t m = (mask[h] << (32 - 2 * tiles)) & live;
                const int rel = self[h] - t0;  // not its own partner
                if (rel >= 0 && rel < 128 && ((rel & 7) >> 1) == c) m &= ~(0x80000000u >> (2 * (rel >> 3) + (rel & 1)));
                const int i = row[h];
                if (i >= 0 && (far || nearest <= b.alarm || (OUT32 && a.half))) {
                    // the reference's test of each candidate, as in k_nl_build_cells
                    uint32_t ui[D];
                    dp_shadow_unpack<D>(sh[i], ui);
                    for (uint32_t rest = m; rest;) {
                        const int s = __clz(rest);
                        const uint32_t bit = 0x80000000u >> s;
                        rest &= ~bit;
                        const int j = rslot[t0 + 8 * (s >> 1) + 2 * c + (s & 1)];
                        bool in = !(OUT32 && a.half) || dp_owns_pair(i, j);
                        if (in && (far || nearest <= b.alarm)) {
                            uint32_t uj[D];
                            dp_shadow_unpack<D>(__ldg(sh + j), uj);
                            float df[D];
                            const float qf = dp_shadow_q<D>(ui, uj, a.unit, df);
                            in = qf <= a.hi2;
                            if (in && (far || !(qf < a.lo2))) {
                                double d[D];
#pragma unroll
                                for (int k = 0; k < D; ++k)
                                    d[k] = dp_min_image(a.pos[k * n + i] - a.pos[k * n + j], a.box[k]);
                                in = sqrt(dp_sqsum_exact<D>(d)) < a.cutoff;
                            }
                        }
                        if (!in) m &= ~bit;
                    }
                }
                // lane c takes the 32 entries from t0 + 32 c, so that the row is in
                // the order of the region (the order of k_nl_build_cells: the
                // same float32 sums): byte c of each lane's word holds its two
                // columns of the lane's four tiles
                {
                    uint32_t mixed = 0u;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        uint32_t x = (__shfl_sync(0xffffffffu, m, q, 4) >> (24 - 8 * c)) & 0xFFu;
                        x = (x | (x << 12)) & 0x000F000Fu;
                        x = (x | (x << 6)) & 0x03030303u;
                        mixed |= x << (6 - 2 * q);
                    }
                    m = mixed;
                }
                const int mine = __popc(m);
                int upto = mine;
#pragma unroll
                for (int o = 1; o < 4; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, upto, o, 4);
                    if (c >= o) upto += y;
                }
                const int at = found[h] + upto - mine;
                found[h] += __shfl_sync(0xffffffffu, upto, 3, 4);
                int left = min(mine, a.kcap - at);
                if (OUT32) {
                    int32_t* to = a.nl + at * n + i;
                    for (; left > 0; --left, to += n) {
                        const int s = __clz(m);
                        m &= ~(0x80000000u >> s);
                        *to = rslot[t0 + 32 * c + s];
                    }
                } else {
                    uint16_t* to = (uint16_t*)b.list + (((long long)(at >> 3) * n + i) * 8 + (at & 7));
                    for (int e = at; left > 0; --left) {
                        const int s = __clz(m);
                        m &= ~(0x80000000u >> s);
                        *to = (uint16_t)(t0 + 32 * c + s);
                        ++e;
                        to += (e & 7) ? 1 : 8 * n - 7;
                    }
                }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = row[h];
            if (i < 0) continue;
            best = max(best, found[h]);
            const int kept = min(found[h], a.kcap);
            if (!OUT32) {  // the last chunk, filled up with index 0
                for (int at = kept + c; at < ((kept + 7) & ~7); at += 4)
                    ((uint16_t*)b.list)[((long long)(at >> 3) * n + i) * 8 + (at & 7)] = (uint16_t)0;
            }
            if (c == 0) {
                a.cnt[i] = kept;
                ((sh_t*)a.shadow_ref)[i] = sh[i];
            }
            if (c < D) a.pos_ref[c * n + i] = a.pos[c * n + i];
        }
    }
    best = __reduce_max_sync(0xffffffffu, best);
    if (lane == 0 && best > 0) atomicMax(&a.st->max_neighbors, best);
}

// Brick lists as column-major lists of slots (for the export).
__global__ void k_brick_expand(const int4* __restrict__ info, const int32_t* __restrict__ slots, int cap,
                               const uint16_t* __restrict__ list, const int32_t* __restrict__ cnt, int32_t* out,
                               long long n) {
    const int4 b = info[blockIdx.x];
    const int32_t* __restrict__ mine = slots + (long long)blockIdx.x * cap;
    for (int p = threadIdx.x; p < b.y; p += blockDim.x) {
        const long long i = b.x + p;
        const int c = cnt[i];
        for (int k = 0; k < c; ++k) out[(long long)k * n + i] = mine[list[((long long)(k >> 3) * n + i) * 8 + (k & 7)]];
    }
}

// All-pairs build for boxes with fewer than 3 cells per axis; rows come out in
// ascending index order, exactly the reference's double loop. As in the cell
// build, the float32 shadow test decides every pair outside its error bracket
// and float64 (the reference's test) only the rest.
template <int D>
__global__ void __launch_bounds__(kBlock) k_nl_build_allpairs(NlArgs a) {
    if (!a.st->need_rebuild) return;
    typedef typename dp_shadow_t<D>::type sh_t;
    __shared__ double tile[D][kBlock];
    __shared__ sh_t tsh[kBlock];
    const long long n = a.n;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = i < n;
    const bool far = a.st->far != 0;
    const sh_t* sh = (const sh_t*)a.shadow;
    double xi[D];
#pragma unroll
    for (int k = 0; k < D; ++k) xi[k] = active ? a.pos[k * n + i] : 0.0;
    uint32_t ui[D];
    dp_shadow_unpack<D>(active ? sh[i] : sh_t{}, ui);
    int count = 0;
    for (long long base = 0; base < n; base += kBlock) {
        const long long jl = base + threadIdx.x;
#pragma unroll
        for (int k = 0; k < D; ++k) tile[k][threadIdx.x] = (jl < n) ? a.pos[k * n + jl] : 0.0;
        tsh[threadIdx.x] = (jl < n) ? sh[jl] : sh_t{};
        __syncthreads();
        if (active) {
            const int lim = (int)min((long long)kBlock, n - base);
            for (int t = 0; t < lim; ++t) {
                const long long j = base + t;
                if (a.half ? !dp_owns_pair(i, j) : j == i) continue;
                uint32_t uj[D];
                dp_shadow_unpack<D>(tsh[t], uj);
                float df[D];
                const float qf = dp_shadow_q<D>(ui, uj, a.unit, df);
                if (qf > a.hi2) continue;
                bool inside = qf < a.lo2 && !far;
                if (!inside) {
                    double d[D];
#pragma unroll
                    for (int k = 0; k < D; ++k) d[k] = dp_min_image(xi[k] - tile[k][t], a.box[k]);
                    inside = sqrt(dp_sqsum_exact<D>(d)) < a.cutoff;
                }
                if (inside) {
                    if (count < a.kcap) a.nl[(long long)count * n + i] = (int32_t)j;
                    ++count;
                }
            }
        }
        __syncthreads();
    }
    if (!active) return;
    a.cnt[i] = min(count, a.kcap);
    atomicMax(&a.st->max_neighbors, count);
#pragma unroll
    for (int k = 0; k < D; ++k) a.pos_ref[k * n + i] = xi[k];
    ((sh_t*)a.shadow_ref)[i] = sh[i];
}

// Lists of small systems (a warp per particle; full or half, in rows or
// columns): every other particle tested, 32 at a time, with the same decisions,
// in ascending order. No cells, and the slots keep their order. A rebuild of 500
// LJ particles 82 -> 15 us, of 4,000 434 -> 43 (one thread per particle before).
template <int D>
__global__ void __launch_bounds__(kBlock) k_nl_build_rows(NlArgs a) {
    if (!a.st->need_rebuild) return;
    typedef typename dp_shadow_t<D>::type sh_t;
    const long long n = a.n;
    const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= n) return;  // uniform across the warp
    const bool far = a.st->far != 0;
    const sh_t* __restrict__ sh = (const sh_t*)a.shadow;
    const sh_t shi = sh[i];
    uint32_t ui[D];
    dp_shadow_unpack<D>(shi, ui);
    int32_t* row = a.nl + i * a.nl_i;
    int found = 0;
#pragma unroll 2
    for (int base = 0; base < (int)n; base += 32) {
        const int j = base + lane;
        bool in = false;
        if (j < (int)n && (a.half ? dp_owns_pair(i, j) : j != (int)i)) {
            uint32_t uj[D];
            dp_shadow_unpack<D>(__ldg(sh + j), uj);
            float df[D];
            const float q = dp_shadow_q<D>(ui, uj, a.unit, df);
            in = q <= a.hi2;
            if (in && (far || !(q < a.lo2))) {
                double d[D];
#pragma unroll
                for (int k = 0; k < D; ++k) d[k] = dp_min_image(a.pos[k * n + i] - a.pos[k * n + j], a.box[k]);
                in = sqrt(dp_sqsum_exact<D>(d)) < a.cutoff;
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        const int at = found + __popc(m & ((1u << lane) - 1u));
        if (in && at < a.kcap) row[at * a.nl_k] = j;
        found += __popc(m);
    }
    if (lane == 0) {
        a.cnt[i] = min(found, a.kcap);
        ((sh_t*)a.shadow_ref)[i] = shi;
        atomicMax(&a.st->max_neighbors, found);
    }
    if (lane < D) a.pos_ref[lane * n + i] = a.pos[lane * n + i];
}

// Self-test of the bounded device-side waits, without a GPU fault: one CTA
// allocates tensor memory as the surrogate pass does, waits on an mbarrier
// that nothing arrives at, gives up after `limit` tries, frees the tensor
// memory and records device_error (the host then reports DP_ERR_TIMEOUT).
__global__ void __launch_bounds__(128) k_selftest_bounded_wait(dp_dev_status* st, int limit) {
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t s_tmem;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) dp_mbar_init(&mbar, 1);
    if (warp == 0) dp_tmem_alloc(&s_tmem, 64);
    dp_tc_fence_before();
    __syncthreads();
    dp_tc_fence_after();
    const bool arrived = dp_mbar_wait(&mbar, 0u, limit);
    if (!arrived && threadIdx.x == 0) atomicExch(&st->device_error, 1);
    dp_tc_fence_before();
    __syncthreads();
    if (warp == 0) dp_tmem_dealloc(s_tmem, 64);
}

// kcap, region: room of a row and of a brick's region. Grouped steps stop at a build
// that did not fit (its lists are cut short or empty): the steps before it stand,
// and the host makes room and goes on from there.
__global__ void k_rebuild_done(dp_dev_status* st, int kcap, int region) {
    if (st->need_rebuild) {
        if (st->max_neighbors > kcap || st->cell_overflow > region) st->left = 0;
        st->need_rebuild = 0;
        st->rebuilds += 1;
        st->ref_far = st->far;  // the list's reference positions are the current ones
        st->parity = 0;         // and the permutation left them in the first set
    }
}

__global__ void k_set_rebuild(dp_dev_status* st) { st->need_rebuild = 1; }

// Condition of the graph's rebuild node: the sequence runs only when some
// particle moved more than skin/2 (or a rebuild was requested).
__global__ void k_rebuild_cond(dp_dev_status* st, cudaGraphConditionalHandle h) {
    cudaGraphSetConditional(h, st->need_rebuild ? 1u : 0u);
}


// Grouped steps (build_group): the words a launch starts from and leaves, the
// condition of a group's rebuild node, and whether another group follows. A
// group makes at least one step, so `steps` + 1 groups are enough; one more means
// that the steps do not count themselves.
__global__ void k_group_start(dp_dev_status* st, int steps) {
    st->left = steps;
    st->parity = 0;
    st->groups = 0;
}
__global__ void k_group_begin(dp_dev_status* st, cudaGraphConditionalHandle h) {
    st->groups += 1;
    cudaGraphSetConditional(h, st->need_rebuild ? 1u : 0u);
}
__global__ void k_group_end(dp_dev_status* st, cudaGraphConditionalHandle h, int most) {
    const bool more = st->left > 0;
    if (more && st->groups >= most) st->device_error = 1;
    cudaGraphSetConditional(h, more && st->groups < most ? 1u : 0u);
}

// End of a graph of steps; clear_far: its last (fused) step wrapped every position.
__global__ void k_advance_step(dp_dev_status* st, long long steps, int clear_far) {
    st->step += steps;
    if (clear_far) st->far = 0;
}

// The list of slots (entry k of slot r at k nl_k + r nl_i) -> row-major (N, kout) by particle
// id, entries as particle ids, each row sorted ascending and -1 padded
// (dompap's neighbor_list layout).
__global__ void k_nl_export(const int32_t* __restrict__ nl, const int32_t* __restrict__ cnt, int32_t* out,
                            const int32_t* __restrict__ order, const int32_t* __restrict__ slot_of, long long n,
                            long long nl_k, long long nl_i, int kout) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long r = slot_of[i];
    const int c = cnt[r];
    int32_t* row = out + i * kout;
    int m = 0;  // entries kept so far (<= kout), the kout smallest in ascending order
    for (int k = 0; k < c; ++k) {
        const int32_t v = order[nl[k * nl_k + r * nl_i]];
        int u;
        if (m < kout) {
            u = m - 1;
            ++m;
        } else if (v < row[kout - 1]) {
            u = kout - 2;
        } else {
            continue;
        }
        while (u >= 0 && row[u] > v) {
            row[u + 1] = row[u];
            --u;
        }
        row[u + 1] = v;
    }
    for (int k = m; k < kout; ++k) row[k] = -1;
}

// A half list (each pair in the row of the particle that owns it,
// dp_owns_pair) closed into the full one: row i gets its own entries and i
// from every row j that holds it. The distance test is
// symmetric (the min-image displacement of j - i is the negated one of i - j
// and the sum of squares is the same), so the closure is the list a full
// build at the same reference positions makes. Count pass, then scatter into
// an unsorted column-major list that k_nl_export sorts.
__global__ void k_nl_half_count(const int32_t* __restrict__ nl, const int32_t* __restrict__ cnt, int32_t* fcnt,
                                int32_t* fmax, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int c = cnt[i];
    for (int k = 0; k < c; ++k) atomicAdd(fcnt + nl[(long long)k * n + i], 1);
    const int mine = atomicAdd(fcnt + i, c) + c;
    atomicMax(fmax, mine);
}

__global__ void k_nl_half_scatter(const int32_t* __restrict__ nl, const int32_t* __restrict__ cnt, int32_t* fill,
                                  int32_t* full, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int c = cnt[i];
    for (int k = 0; k < c; ++k) {
        const int32_t j = nl[(long long)k * n + i];
        full[(long long)atomicAdd(fill + i, 1) * n + i] = j;
        full[(long long)atomicAdd(fill + j, 1) * n + j] = (int32_t)i;
    }
}

// --------------------------- integrators ----------------------------------
// Mass handling: MASSMODE 0 one mass for all particles (coefficients as
// arguments), 1 per-particle class index into a coefficient table, 2
// per-particle masses (coefficients computed in the kernel).
// The per-particle step is dp_integrate_one (dp_integrate.cuh). This kernel
// integrates in place after a separate force kernel (the surrogate mode, and
// the timing of the integrator alone); the other modes fuse it into the pair
// kernel.
template <int D, int MASSMODE, bool NVE, bool WRITE64>
__global__ void __launch_bounds__(kBlock) k_integrate(dp_int_args a) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.x == 0 && threadIdx.x == 0) a.st->far = 0;  // every position is wrapped below
    bool old = false, bad = false;
    if (i < a.n) {
        double F[D];
#pragma unroll
        for (int k = 0; k < D; ++k) F[k] = a.force[k * a.n + i];
        old = dp_integrate_one<D, MASSMODE, NVE, WRITE64>(a, i, F, bad, -1);
    }
    const bool any_old = __any_sync(0xffffffffu, old);
    const bool any_bad = __any_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0) {
        if (any_old) atomicExch(&a.st->need_rebuild, 1);
        if (any_bad) atomicExch(&a.st->nonfinite, 1);
    }
}

// sum_n m_n |v_n|^2, per-block partials.
template <int D, int MASSMODE>
__global__ void __launch_bounds__(kBlock) k_sum_mv2(dp_int_args a, const double* class_mass, double* partial) {
    __shared__ double smem[32];
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double v = 0.0;
    if (i < a.n) {
        double m;
        if (MASSMODE == 0) m = class_mass[0];
        else if (MASSMODE == 1) m = class_mass[a.mclass[i]];
        else m = a.mass[i];
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            const double vk = a.vel[k * a.n + i];
            s += vk * vk;
        }
        v = m * s;
    }
    v = dp_block_sum(v, smem);
    if (threadIdx.x == 0) partial[blockIdx.x] = v;
}

// Fixed-order sum of per-block partials (one block): deterministic totals.
__global__ void __launch_bounds__(1024) k_reduce(const double* __restrict__ partial, long long m, double* out) {
    __shared__ double smem[32];
    double v = 0.0;
    for (long long t = threadIdx.x; t < m; t += blockDim.x) v += partial[t];
    v = dp_block_sum(v, smem);
    if (threadIdx.x == 0) out[0] = v;
}

template <int D>
__global__ void k_normals(unsigned long long seed, long long step, double* out, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float z[4];
    dp_normals4(seed, (unsigned long long)step, (uint32_t)i, z);
#pragma unroll
    for (int k = 0; k < D; ++k) out[i * D + k] = (double)z[k];
}

// wrap_into_box on demand (dompap/positions.py:90-98), with the shadow update.
template <int D>
__global__ void k_wrap(dp_int_args a) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.x == 0 && threadIdx.x == 0) a.st->far = 0;
    if (i >= a.n) return;
    uint32_t u[D];
    unsigned long long X[D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
        const long long o = k * a.n + i;
        int32_t im = a.img[o];
        const int32_t im0 = im;
        const double x = dp_wrap_axis(a.pos[o], a.box[k], im);
        a.pos_out[o] = x;
        if (im != im0) a.img[o] = im;
        X[k] = fixed64_wrapped(x, a.box[k], a.scale64[k]);
        u[k] = (uint32_t)(X[k] >> 32);
        X[k] <<= a.shift64[k];
    }
    ((typename dp_shadow_t<D>::type*)a.shadow_out)[i] = dp_shadow_pack<D>(u);
    ((typename dp_fixed64_t<D>::type*)a.pos64_out)[i] = dp_fixed64_pack<D>(X);
}

// Pair-distance histogram for g(r) (dompap/positions.py:58-87): all ordered
// pairs (i in A, j in B, self pairs included), np.round minimum image,
// np.histogram bins (half-open, the last one closed). The distance comes from
// the fixed-point shadow in float32; a pair within the float error of a bin
// edge is recomputed in float64 exactly as NumPy does.
//
// Bounds: the conversions and the reciprocal square root (4 per pair on a
// 16-per-clock unit) and the histogram's shared-memory atomics; the N^2 / 2
// pairs come from shared memory (broadcast), HBM is idle. A CTA takes work items of
// 256 particles i (one per thread) x kRdfChunk particles j; where A and B are
// the same set, only items and pairs with j >= i, counted twice (the distance
// is symmetric bit by bit). The bin comes from a table over uniform cells of r
// (about one compare per pair whatever the edges; a binary search per pair
// costs eight dependent ones). Near an edge - the bracket is the float
// error itself, 1e-6 r, not 1e-5 r - the pair goes to its warp's queue in
// shared memory, and 32 queued pairs take the float64 path together: float64
// runs at 1/64 rate here, and a lane alone in that path holds up its warp for
// as long as a full one. 27,436 particles, 200 bins, whole call: 28.9 ms before
// (a flat loop over p = i n + j with a 64-bit division, no symmetry, binary
// search, float64 in divergent lanes), 1.2 ms now.
constexpr int kRdfChunk = 64;    // particles j of one work item
constexpr int kRdfQueue = 64;    // queued near-edge pairs per warp (a round adds at most 32)
constexpr int kRdfItems = 65536; // items between flushes: 65536 * 256 * 64 * 2 < 2^32 counts per bin

// Small systems (at most one work item per SM): a call is its launches and one
// thread's chain of partners, so the types are compared in the kernel and not
// selected before it, and an item has a quarter of the partners. 500 particles,
// 200 bins: all pairs 73 -> 59 us a call, two calls with types 171 -> 137;
// 1,372: 74 -> 60, 175 -> 139. At 2,048 with the longer items 79 -> 84 (all
// pairs: the comparison is in the loop), hence a form of its own; from there on
// the selected lists are as fast or faster (4,000: 199 against 215).
constexpr int kRdfSmallItems = 152;
constexpr int kRdfSmallChunk = 16;

struct RdfArgs {
    const int32_t* types;     // of the small form, which compares them (null: every particle)
    int type_a, type_b;       // negative: every type
    const double* pos;
    const void* shadow;
    const double* edges;
    const int32_t* idx_a;     // slots of the particles i, j (null: every slot)
    const int32_t* idx_b;
    const int32_t* selected;  // their numbers, [2], [1] where A and B are the same set (null: n)
    unsigned long long* counts;
    long long n;
    int nbins;
    int cells;      // uniform cells of the bin table
    int copies;     // histograms per CTA (lanes spread over them: fewer equal addresses per warp)
    int symmetric;  // A and B are the same set
    float abs_tol;  // error of a shadow distance from the fixed point's resolution
    double box[DP_MAX_DIM];
    float unit[DP_MAX_DIM];
};

// Slots of the particles of type a (blockIdx.y = 0) and b (1), in no particular
// order (the histogram does not depend on it). One launch for both, and none
// for b where it is the same set: on a small system the call is its launches.
__global__ void k_rdf_select(const int32_t* __restrict__ types, long long n, int type_a, int type_b, int32_t* idx,
                             int32_t* count) {
    const int type = blockIdx.y ? type_b : type_a;
    idx += blockIdx.y * n;
    count += blockIdx.y;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool take = i < n && (type < 0 || types[i] == type);
    const unsigned m = __ballot_sync(0xffffffffu, take);
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (lane == 0 && m) base = atomicAdd(count, __popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (take) idx[base + __popc(m & ((1u << lane) - 1u))] = (int32_t)i;
}

// np.histogram's bin of r, -1 outside.
__device__ __forceinline__ int rdf_bin(double r, const double* e, int nb) {
    if (!(r >= e[0]) || !(r <= e[nb])) return -1;
    if (r == e[nb]) return nb - 1;
    int lo = 0, hi = nb;  // e[lo] <= r < e[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (r >= e[mid]) lo = mid; else hi = mid;
    }
    return lo;
}

// The float64 distance and bin of queue entries (all lanes of a warp).
template <int D>
__device__ __forceinline__ void rdf_exact(const RdfArgs& a, const double* edges, int2 pair, bool mine, bool twice,
                                          unsigned int* hist) {
    if (!mine) return;
    double q = 0.0;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        const double L = a.box[k];
        double d = a.pos[k * a.n + pair.x] - a.pos[k * a.n + pair.y];
        d -= L * rint(d / L);
        q = (k == 0) ? __dmul_rn(d, d) : __dadd_rn(q, __dmul_rn(d, d));
    }
    const int b = rdf_bin(sqrt(q), edges, a.nbins);
    if (b >= 0) atomicAdd(hist + b, twice ? 2u : 1u);
}

template <int D, bool SMALL>
__global__ void __launch_bounds__(kBlock) k_rdf(RdfArgs a) {
    constexpr int kChunk = SMALL ? kRdfSmallChunk : kRdfChunk;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    typedef typename dp_shadow_t<D>::type sh_t;
    __shared__ sh_t tile[kChunk];
    __shared__ int32_t tslot[kChunk];
    __shared__ bool tmine[SMALL ? kChunk : 1];
    __shared__ int2 queue[kBlock / 32][kRdfQueue];
    double* edges = (double*)smem_raw;                          // [nbins + 1]
    float* ef = (float*)(edges + a.nbins + 1);                  // [nbins + 1]
    unsigned int* hist = (unsigned int*)(ef + a.nbins + 1);     // [copies][nbins]
    uint16_t* table = (uint16_t*)(hist + a.copies * a.nbins);   // [cells]
    const int nb = a.nbins;
    for (int t = threadIdx.x; t <= nb; t += kBlock) {
        edges[t] = a.edges[t];
        ef[t] = (float)a.edges[t];
    }
    for (int t = threadIdx.x; t < a.copies * nb; t += kBlock) hist[t] = 0u;
    __syncthreads();
    const float r0 = fmaxf(ef[0], 0.0f), r1 = ef[nb];
    const float cell_w = (r1 - r0) / (float)a.cells;
    const float inv_w = cell_w > 0.0f ? 1.0f / cell_w : 0.0f;
    // table[c]: the last bin whose lower edge is not above cell c's start
    for (int c = threadIdx.x; c < a.cells; c += kBlock) {
        const float r = r0 + cell_w * ((float)c - 0.01f);
        int lo = 0, hi = nb;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (r >= ef[mid]) lo = mid; else hi = mid;
        }
        table[c] = (uint16_t)lo;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int* my_hist = hist + (lane % a.copies) * nb;
    const sh_t* __restrict__ sh = (const sh_t*)a.shadow;
    const int na = a.selected ? a.selected[0] : (int)a.n, nbp = a.symmetric ? na : (a.selected ? a.selected[1] : (int)a.n);
    const long long rows = (na + kBlock - 1) / kBlock, chunks = (nbp + kChunk - 1) / kChunk;
    const float rmax = r1 * (1.0f + 2e-6f) + 2.0f * a.abs_tol;
    const float qmax = rmax * rmax * (1.0f + 1e-6f);
    int queued = 0;  // entries in this warp's queue (uniform)
    long long since = 0;
    auto flush = [&]() {
        __syncthreads();
        for (int t = threadIdx.x; t < nb; t += kBlock) {
            unsigned long long c = 0;
            for (int k = 0; k < a.copies; ++k) {
                c += hist[k * nb + t];
                hist[k * nb + t] = 0u;
            }
            if (c) atomicAdd(a.counts + t, c);
        }
        __syncthreads();
    };
    for (long long w = blockIdx.x; w < rows * chunks; w += gridDim.x) {
        const long long row = w / chunks, chunk = w - row * chunks;
        // symmetric: only pairs with j >= i
        if (a.symmetric && (chunk + 1) * kChunk <= row * kBlock) continue;
        if (++since == kRdfItems) {
            flush();
            since = 1;
        }
        const int j0 = (int)(chunk * kChunk), jn = min(kChunk, nbp - j0);
        __syncthreads();
        if ((int)threadIdx.x < jn) {
            const int slot = a.idx_b ? a.idx_b[j0 + threadIdx.x] : j0 + (int)threadIdx.x;
            tslot[threadIdx.x] = slot;
            tile[threadIdx.x] = sh[slot];
            if (SMALL) tmine[threadIdx.x] = !a.types || a.type_b < 0 || a.types[slot] == a.type_b;
        }
        __syncthreads();
        const int i = (int)(row * kBlock) + threadIdx.x;
        const int si = i < na ? (a.idx_a ? a.idx_a[i] : i) : 0;
        const bool active = i < na && (!SMALL || !a.types || a.type_a < 0 || a.types[si] == a.type_a);
        uint32_t ui[D];
        dp_shadow_unpack<D>(sh[si], ui);
        for (int t = 0; t < jn; ++t) {
            uint32_t uj[D];
            dp_shadow_unpack<D>(tile[t], uj);
            float df[D];
            const float q = dp_shadow_q<D>(ui, uj, a.unit, df);
            const int j = j0 + t;
            bool near = false;
            if (active && q <= qmax && (!a.symmetric || j >= i) && (!SMALL || tmine[t])) {
                const float r = q > 0.0f ? q * rsqrtf(q) : 0.0f;
                const float tol = fmaf(1e-6f, r, a.abs_tol);
                int b = table[max(0, min((int)((r - r0) * inv_w), a.cells - 1))];
                while (b + 1 < nb && r >= ef[b + 1]) ++b;
                const float below = r - ef[b], above = ef[b + 1] - r;
                near = fabsf(below) <= tol || fabsf(above) <= tol;
                if (!near && below > 0.0f && above > 0.0f) atomicAdd(my_hist + b, a.symmetric && j != i ? 2u : 1u);
            }
            const unsigned m = __ballot_sync(0xffffffffu, near);
            if (m) {
                if (near) queue[warp][queued + __popc(m & ((1u << lane) - 1u))] = make_int2(si, tslot[t]);
                queued += __popc(m);
                if (queued >= 32) {
                    __syncwarp();
                    queued -= 32;
                    const int2 p = queue[warp][queued + lane];
                    rdf_exact<D>(a, edges, p, true, a.symmetric && p.x != p.y, my_hist);
                    __syncwarp();
                }
            }
        }
    }
    __syncwarp();
    if (lane < queued) {
        const int2 p = queue[warp][lane];
        rdf_exact<D>(a, edges, p, true, a.symmetric && p.x != p.y, my_hist);
    }
    flush();
}

}  // namespace

// ===========================================================================
// allocation-free kinetic sum (see dp_sum_mv2_noalloc in dompap_gpu.h)
// ===========================================================================
// Scratch for the per-block partial sums, one double per block of kBlock
// particles: 16384 blocks = 128 KiB, i.e. at most 4,194,304 particles per
// call. It lives in every GPU that loads this library until the process
// exits. Every call shares it and overwrites exactly the partials it reads,
// so nothing carries over between calls; calls that overlap on the GPU (two
// streams at once) race on it.
#define DP_NOALLOC_MAX_BLOCKS 16384
static __device__ __align__(256) double g_noalloc_partial[DP_NOALLOC_MAX_BLOCKS];

namespace {
__global__ void __launch_bounds__(kBlock) k_mv2_rowmajor(const double* __restrict__ vel,
                                                          const double* __restrict__ mass, long long n, int dim,
                                                          double* __restrict__ partial) {
    __shared__ double smem[32];
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double v = 0.0;
    if (i < n) {
        double s = 0.0;
        for (int k = 0; k < dim; ++k) {
            const double vk = vel[i * dim + k];
            s += vk * vk;
        }
        v = mass[i] * s;
    }
    v = dp_block_sum(v, smem);
    if (threadIdx.x == 0) partial[blockIdx.x] = v;
}
}  // namespace

// Device address of g_noalloc_partial, looked up once per device (host code
// cannot use the symbol itself: on the host it only names a stand-in). The
// cached address belongs to the device's primary context; cudaDeviceReset
// ends that context, and the header tells callers not to call again after it.
static std::mutex g_noalloc_mutex;
static double* g_noalloc_addr[64] = {nullptr};

// ===========================================================================
// NVRTC pair-kernel libraries
// ===========================================================================
struct PairLib {
    cudaLibrary_t lib = nullptr;
    cudaKernel_t forces = nullptr, energy = nullptr, virial = nullptr, laplacian = nullptr, eval = nullptr;
    cudaKernel_t step = nullptr;  // fused forces + integrate (not in the surrogate program)
    cudaKernel_t step_warp = nullptr;  // the same, one warp per particle (small systems)
    cudaKernel_t step_quad = nullptr;  // the same, four lanes per particle
    cudaKernel_t step_lists = nullptr;  // one warp per particle, which rebuilds its own list
    // sums with 32 (0) or 4 (1) lanes per particle: forces, energy, virial, Laplacian
    cudaKernel_t split[2][4] = {{nullptr, nullptr, nullptr, nullptr}, {nullptr, nullptr, nullptr, nullptr}};
    // no neighbour list (dompap's double-loop methods): fused step, forces, energy
    cudaKernel_t step_all = nullptr, forces_all = nullptr, energy_all = nullptr;
    // bricks of cells (not in 4-D, with dense parameters, costly potentials or in the surrogate
    // program): fused step with 1 or 4 lanes per particle, forces, scalars
    cudaKernel_t step_brick[2] = {nullptr, nullptr};
    cudaKernel_t forces_brick = nullptr, energy_brick = nullptr, virial_brick = nullptr, laplacian_brick = nullptr;
    cudaKernel_t batch[4] = {nullptr, nullptr, nullptr, nullptr};  // 128, 256, 512, 1024 threads
    cudaKernel_t forces_mlp = nullptr, energy_mlp = nullptr, virial_mlp = nullptr, mlp_finish = nullptr;
    cudaKernel_t forces_mlp_tc = nullptr, energy_mlp_tc = nullptr, virial_mlp_tc = nullptr;  // tcgen05
};

static std::mutex g_lib_mutex;
static std::unordered_map<std::string, PairLib> g_libs;

// --------------------------- on-disk cubin cache ------------------------
// A pair program takes seconds to compile; its CUBIN is kept on disk under a
// key of the program text and the NVRTC version, in DOMPAP_NVRTC_CACHE (empty
// or "0": off) or else in _build/nvrtc_cache beside the library. A file holds
// the program text it was compiled from and is used only when that text
// matches exactly; unreadable or foreign files are ignored and rewritten.
static std::string cubin_cache_dir(bool explicit_only) {
    if (const char* env = std::getenv("DOMPAP_NVRTC_CACHE")) {
        if (!*env || std::strcmp(env, "0") == 0) return "";
        return env;
    }
    if (explicit_only) return "";
    Dl_info info;
    if (dladdr((void*)&cubin_cache_dir, &info) && info.dli_fname) {
        const std::string lib = info.dli_fname;
        const size_t k = lib.rfind('/');
        if (k != std::string::npos) return lib.substr(0, k) + "/_build/nvrtc_cache";
    }
    return "";
}

static std::string cubin_cache_path(const std::string& dir, const std::string& src) {
    uint64_t h = 1469598103934665603ull;  // FNV-1a
    auto mix = [&h](const void* data, size_t len) {
        const unsigned char* b = (const unsigned char*)data;
        for (size_t i = 0; i < len; ++i) {
            h ^= b[i];
            h *= 1099511628211ull;
        }
    };
    mix(src.data(), src.size());
    int major = 0, minor = 0;
    nvrtcVersion(&major, &minor);
    mix(&major, sizeof(major));
    mix(&minor, sizeof(minor));
    char name[64];
    snprintf(name, sizeof(name), "/%016llx.dpcubin", (unsigned long long)h);
    return dir + name;
}

static const char kCacheMagic[8] = {'D', 'P', 'C', 'U', 'B', 'I', 'N', '1'};

static bool cubin_cache_read(const std::string& path, const std::string& src, std::vector<char>* cubin) {
    FILE* f = std::fopen(path.c_str(), "rb");
    if (!f) return false;
    bool ok = false;
    char magic[8];
    uint64_t src_len = 0, bin_len = 0;
    if (std::fread(magic, 1, 8, f) == 8 && std::memcmp(magic, kCacheMagic, 8) == 0 &&
        std::fread(&src_len, sizeof(src_len), 1, f) == 1 && src_len == src.size()) {
        std::string text(src_len, '\0');
        if (std::fread(&text[0], 1, src_len, f) == src_len && text == src &&
            std::fread(&bin_len, sizeof(bin_len), 1, f) == 1 && bin_len > 0 && bin_len < (1ull << 30)) {
            cubin->resize(bin_len);
            ok = std::fread(cubin->data(), 1, bin_len, f) == bin_len;
        }
    }
    std::fclose(f);
    return ok;
}

static void cubin_cache_write(const std::string& dir, const std::string& path, const std::string& src,
                              const std::vector<char>& cubin) {
    // create the directory and its parent (the library's _build) if needed
    const size_t k = dir.rfind('/');
    if (k != std::string::npos && k > 0) mkdir(dir.substr(0, k).c_str(), 0755);
    mkdir(dir.c_str(), 0755);
    const std::string tmp = path + ".tmp" + std::to_string((long long)getpid());
    FILE* f = std::fopen(tmp.c_str(), "wb");
    if (!f) return;
    const uint64_t src_len = src.size(), bin_len = cubin.size();
    bool ok = std::fwrite(kCacheMagic, 1, 8, f) == 8 && std::fwrite(&src_len, sizeof(src_len), 1, f) == 1 &&
              std::fwrite(src.data(), 1, src_len, f) == src_len && std::fwrite(&bin_len, sizeof(bin_len), 1, f) == 1 &&
              std::fwrite(cubin.data(), 1, bin_len, f) == bin_len;
    ok = (std::fclose(f) == 0) && ok;
    if (ok)
        std::rename(tmp.c_str(), path.c_str());  // atomic: readers see a whole file or none
    else
        std::remove(tmp.c_str());
}

// NVRTC: program text -> sm_103a CUBIN (host only; no GPU needed).
// resource_log (optional): compile with the assembler's verbose report
// (registers, spill bytes, shared memory per kernel) and return that log.
static int nvrtc_compile(const std::string& src, std::vector<char>* cubin, std::string* resource_log);

// cache: use the on-disk cubin cache (explicit_only: only when
// DOMPAP_NVRTC_CACHE names a directory).
static int nvrtc_cubin(const std::string& src, std::vector<char>* cubin, std::string* resource_log = nullptr,
                       bool cache = false, bool explicit_only = false) {
    const std::string dir = cache && !resource_log ? cubin_cache_dir(explicit_only) : std::string();
    if (!dir.empty()) {
        const std::string path = cubin_cache_path(dir, src);
        if (cubin_cache_read(path, src, cubin)) return DP_OK;
        RET(nvrtc_compile(src, cubin, nullptr));
        cubin_cache_write(dir, path, src, *cubin);
        return DP_OK;
    }
    return nvrtc_compile(src, cubin, resource_log);
}

static int nvrtc_compile(const std::string& src, std::vector<char>* cubin, std::string* resource_log) {
    nvrtcProgram prog;
    nvrtcResult r = nvrtcCreateProgram(&prog, src.c_str(), "dompap_pair.cu", 0, nullptr, nullptr);
    if (r != NVRTC_SUCCESS) return fail(DP_ERR_NVRTC, std::string("nvrtcCreateProgram: ") + nvrtcGetErrorString(r));
    const char* opts[] = {"--gpu-architecture=sm_103a", "-std=c++17", "-lineinfo", "--fmad=true",
                          "-DDP_NVRTC=1", "--ptxas-options=-v"};
    const int nopt = (int)(sizeof(opts) / sizeof(opts[0])) - (resource_log ? 0 : 1);
    r = nvrtcCompileProgram(prog, nopt, opts);
    if (r != NVRTC_SUCCESS) {
        size_t log_size = 0;
        nvrtcGetProgramLogSize(prog, &log_size);
        std::string log(log_size, '\0');
        if (log_size) nvrtcGetProgramLog(prog, &log[0]);
        nvrtcDestroyProgram(&prog);
        return fail(DP_ERR_NVRTC, std::string("NVRTC compile of the pair potential failed: ") + log);
    }
    if (resource_log) {
        size_t log_size = 0;
        nvrtcGetProgramLogSize(prog, &log_size);
        resource_log->assign(log_size, '\0');
        if (log_size) nvrtcGetProgramLog(prog, &(*resource_log)[0]);
    }
    size_t cubin_size = 0;
    nvrtcGetCUBINSize(prog, &cubin_size);
    cubin->resize(cubin_size);
    nvrtcGetCUBIN(prog, cubin->data());
    nvrtcDestroyProgram(&prog);
    return DP_OK;
}

static int compile_pair_lib(const std::string& src, PairLib* out) {
    std::lock_guard<std::mutex> lock(g_lib_mutex);
    auto it = g_libs.find(src);
    if (it != g_libs.end()) {
        *out = it->second;
        return DP_OK;
    }
    std::vector<char> cubin;
    RET(nvrtc_cubin(src, &cubin, nullptr, true));
    PairLib pl;
    CK(cudaLibraryLoadData(&pl.lib, cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0));
    CK(cudaLibraryGetKernel(&pl.forces, pl.lib, "dp_forces"));
    CK(cudaLibraryGetKernel(&pl.energy, pl.lib, "dp_energy"));
    CK(cudaLibraryGetKernel(&pl.virial, pl.lib, "dp_virial"));
    CK(cudaLibraryGetKernel(&pl.laplacian, pl.lib, "dp_laplacian"));
    CK(cudaLibraryGetKernel(&pl.eval, pl.lib, "dp_eval_pair"));
    if (src.find("#define DP_MLP 1") == std::string::npos) {
        CK(cudaLibraryGetKernel(&pl.step, pl.lib, "dp_step"));
        CK(cudaLibraryGetKernel(&pl.step_warp, pl.lib, "dp_step_warp"));
        CK(cudaLibraryGetKernel(&pl.step_quad, pl.lib, "dp_step_quad"));
        if (src.find("#define DP_LISTS_BLOCKS 0\n") == std::string::npos)
            CK(cudaLibraryGetKernel(&pl.step_lists, pl.lib, "dp_step_lists"));
        const char* quantity[4] = {"dp_forces_", "dp_energy_", "dp_virial_", "dp_laplacian_"};
        const char* lanes[2] = {"warp", "quad"};
        for (int w = 0; w < 2; ++w) {
            if (src.find(w == 0 ? "#define DP_WARP_SUMS 0\n" : "#define DP_QUAD_SUMS 0\n") != std::string::npos) continue;
            for (int q = 0; q < 4; ++q)
                CK(cudaLibraryGetKernel(&pl.split[w][q], pl.lib, (std::string(quantity[q]) + lanes[w]).c_str()));
        }
        CK(cudaLibraryGetKernel(&pl.step_all, pl.lib, "dp_step_all"));
        CK(cudaLibraryGetKernel(&pl.forces_all, pl.lib, "dp_forces_all"));
        CK(cudaLibraryGetKernel(&pl.energy_all, pl.lib, "dp_energy_all"));
    }
    if (src.find("#define DP_MLP 1") != std::string::npos) {
        CK(cudaLibraryGetKernel(&pl.forces_mlp, pl.lib, "dp_forces_mlp"));
        CK(cudaLibraryGetKernel(&pl.mlp_finish, pl.lib, "dp_mlp_forces_finish"));
        CK(cudaLibraryGetKernel(&pl.forces_mlp_tc, pl.lib, "dp_forces_mlp_tc"));
        CK(cudaLibraryGetKernel(&pl.energy_mlp_tc, pl.lib, "dp_energy_mlp_tc"));
        CK(cudaLibraryGetKernel(&pl.virial_mlp_tc, pl.lib, "dp_virial_mlp_tc"));
        CK(cudaLibraryGetKernel(&pl.energy_mlp, pl.lib, "dp_energy_mlp"));
        CK(cudaLibraryGetKernel(&pl.virial_mlp, pl.lib, "dp_virial_mlp"));
    }
    if (src.find("#define DP_BRICKS 1") != std::string::npos) {
        CK(cudaLibraryGetKernel(&pl.step_brick[0], pl.lib, "dp_step_brick1"));
        CK(cudaLibraryGetKernel(&pl.step_brick[1], pl.lib, "dp_step_brick4"));
        CK(cudaLibraryGetKernel(&pl.forces_brick, pl.lib, "dp_forces_brick"));
        CK(cudaLibraryGetKernel(&pl.energy_brick, pl.lib, "dp_energy_brick"));
        CK(cudaLibraryGetKernel(&pl.virial_brick, pl.lib, "dp_virial_brick"));
        CK(cudaLibraryGetKernel(&pl.laplacian_brick, pl.lib, "dp_laplacian_brick"));
    }
    if (src.find("dp_batch_steps_128") != std::string::npos) {
        CK(cudaLibraryGetKernel(&pl.batch[0], pl.lib, "dp_batch_steps_128"));
        CK(cudaLibraryGetKernel(&pl.batch[1], pl.lib, "dp_batch_steps_256"));
        CK(cudaLibraryGetKernel(&pl.batch[2], pl.lib, "dp_batch_steps_512"));
        CK(cudaLibraryGetKernel(&pl.batch[3], pl.lib, "dp_batch_steps_1024"));
    }
    g_libs.emplace(src, pl);
    *out = pl;
    return DP_OK;
}

// ===========================================================================
// handle
// ===========================================================================
struct GraphEntry {
    long long steps;
    int kind;
    unsigned long long version;
    cudaGraphExec_t exec;
    long long launches;          // launched every time the graph runs
    long long rebuild_launches;  // launched per executed rebuild node (0: gated kernels, counted above)
    bool fused = false;          // dp_step graph: each step moves the positions to the other buffer set
    const double* pos_key = nullptr;  // current position buffer when the graph was captured
};

struct dp_sim {
    int dim = 3;
    long long n = 0;
    int precision = DP_PREC_FP64;
    cudaStream_t stream = nullptr;
    cudaStream_t cstream = nullptr;  // captures the groups of steps
    cudaStream_t bstream = nullptr;  // captures the bodies of conditional rebuild nodes
    bool conditional_graphs = true;  // cleared if the CUDA driver rejects conditional nodes
    bool fused_step = true;          // run() uses dp_step (DOMPAP_FUSED_STEP=0: separate kernels)
    // up to warp_step_max particles the fused step runs one warp per particle
    // (dp_step_warp), up to quad_step_max four lanes per particle
    // (dp_step_quad); DOMPAP_WARP_STEP / DOMPAP_QUAD_STEP set them (0: never)
    long long warp_step_max = 8192;
    long long quad_step_max = 65536;
    // launch shape set by the autotuner (dp_set_step_launch): lanes per
    // particle of the fused step (0: the size thresholds above) and resident
    // CTAs per SM it is compiled for (0: the measured default per mode)
    int step_lanes = 0;
    int step_blocks = 0;
    // force and energy methods (dompap's method strings): DP_METHOD_LIST or
    // the all-pairs kernels (DP_METHOD_ALLPAIRS; DP_METHOD_ALLPAIRS_NEWTON for
    // forces: parameters of each pair by (min, max) id). Not in the surrogate
    // mode, whose kernels are list kernels.
    int force_method = DP_METHOD_LIST;
    int energy_method = DP_METHOD_LIST;
    // surrogate pass: 0 = tcgen05 from 65,536 particles (the 128-particle CTAs
    // fill the GPU; on par with mma.sync there), mma.sync below; 1 = tcgen05;
    // 2 = mma.sync (DOMPAP_MLP_TENSOR=tcgen05 | mma)
    int mlp_tensor = 0;
    // neighbour lists hold only the partners a particle owns (dp_owns_pair)
    // in the surrogate mode (its kernels use each pair once); an export
    // builds a full one for the moment
    int nl_kind = 0;              // kind of the list currently built (list_kind)
    // bricks of cells (k_brick_build): the region's capacity starts at the
    // expected number and grows with overflows; bricks_off: some region does
    // not fit (a system of very uneven density): lists by k_nl_build_cells
    bool bricks = false, bricks_off = false;
    int brick_bits = 0, brick_cells = 0, brick_cap = 0, nbricks = 0, brick_lanes = 1, brick_threads = 256;
    int brick_ext[DP_MAX_DIM] = {1, 1, 1, 1};
    int4 *brick_base = nullptr, *brick_info = nullptr;
    int32_t* brick_slots = nullptr;
    int bricks_alloc = 0;              // bricks the first two have room for
    long long brick_slots_alloc = 0;   // entries of brick_slots
    bool brick_pairs = false;  // the float32 pair kernels run on the bricks
    // second set of position buffers: a fused step reads pos/shadow/pos64 and
    // writes these, then the two sets change roles
    double* pos_alt = nullptr;
    void* shadow_alt = nullptr;
    void* pos64_alt = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;

    double *pos = nullptr, *vel = nullptr, *beta = nullptr, *force = nullptr, *pos_ref = nullptr;
    int32_t* img = nullptr;
    void* shadow = nullptr;
    void* shadow_ref = nullptr;
    void* pos64 = nullptr;
    int shift64[DP_MAX_DIM] = {0, 0, 0, 0};  // the 64-bit fixed point is kept modulo L / 2^shift64 (update_shift64)
    size_t shadow_bytes = 0;
    double *bk_pos = nullptr, *bk_vel = nullptr, *bk_beta = nullptr;
    int32_t* bk_img = nullptr;

    // masses
    int mass_mode = 0;
    std::vector<double> class_mass{1.0};
    uint8_t* mclass = nullptr;
    double* mcoef = nullptr;      // [nclass][5]
    float2* mcoef_f = nullptr;    // [nclass]: float32 b/(2m), sqrt(2 alpha T dt)
    double* class_mass_dev = nullptr;
    double* mass = nullptr;       // per particle (mode 2)

    int32_t* types = nullptr;
    bool have_types = false;
    int min_type = 0, max_type = 0;
    double box[DP_MAX_DIM] = {0, 0, 0, 0};
    bool have_box = false;

    // potential
    bool have_pot = false;
    std::string pot_src;
    double r_cut = 1.0;
    PairLib lib;
    bool lib_valid = false;

    // pair surrogate (DP_PREC_MLP)
    const dp_mlp_dev* mlp_dev = nullptr;
    unsigned long long* mlp_fx = nullptr;  // surrogate mode: fixed-point force sums (zero between launches)

    // pair parameters
    int pmode = DP_PAIR_CONST;
    int ntypes = 1;
    double sigma = 1.0, epsilon = 1.0, sig_max = 1.0;
    double *sig_tab = nullptr, *eps_tab = nullptr, *isig_tab = nullptr;
    float2* ff_tab = nullptr;  // DP_FF_PARAMS double-floats per type pair (pair_consts)
    float4* f32_tab = nullptr; // sigma, 1/sigma, epsilon per type pair

    // neighbour list
    double skin = 1.0;
    int kcap = 512;
    int method = DP_NL_CELL;
    bool use_cells = false;
    double cutoff = 0.0;
    int nc[DP_MAX_DIM] = {0, 0, 0, 0};
    long long ncell = 0;
    int32_t *nl = nullptr, *cnt = nullptr;
    long long nl_alloc = 0;
    // cell binning (counting sort): cell keys, Morton or row-major
    bool morton = false;
    long long nbins = 0, bins_alloc = 0;
    int32_t *bin_cnt = nullptr, *bin_start = nullptr, *bin_part = nullptr;
    int32_t *bin_key = nullptr, *bin_rank = nullptr, *src_of = nullptr;
    // slots: after each cell-list rebuild the per-particle state is stored in
    // cell order; order[slot] = particle id, slot_of[id] = slot
    bool reorder = true;  // DOMPAP_REORDER=0: the state keeps its order, the build reads through src_of
    int32_t *order = nullptr, *slot_of = nullptr;
    // scratch of the permutation (vel, beta, img, order, types, mass classes, masses)
    double *sc_vel = nullptr, *sc_beta = nullptr, *sc_mass = nullptr;
    int32_t *sc_img = nullptr, *sc_order = nullptr, *sc_types = nullptr;
    uint8_t* sc_mclass = nullptr;
    // backup of the permutation-dependent arrays for an overflow replay
    int32_t *bk_order = nullptr, *bk_types = nullptr;
    uint8_t* bk_mclass = nullptr;
    double* bk_mass = nullptr;
    bool nl_config_dirty = true;
    bool nl_built = false;
    bool nl_checked = false;  // the list is known to be valid for the current positions

    // integrator
    double dt = 0.01, temperature = 1.0, tau = 0.1;
    unsigned long long seed = 0;

    dp_dev_status* dstat = nullptr;
    dp_dev_status* hstat = nullptr;  // pinned
    double* partial = nullptr;
    long long partial_alloc = 0;
    double* dsum = nullptr;
    double* hsum = nullptr;  // pinned
    // g(r): edges and counts of up to rdf_bins bins; slots of the selected types
    void* rdf_buf = nullptr;
    int rdf_bins = 0;
    int32_t* rdf_sel = nullptr;

    unsigned long long version = 1;
    std::vector<GraphEntry> graphs;
    long long launches_last = 0;
};

// ---------------------------------------------------------------------------
static void free_graphs(dp_sim* s) {
    for (auto& g : s->graphs) cudaGraphExecDestroy(g.exec);
    s->graphs.clear();
}

static int dalloc(void** p, size_t bytes) {
    if (*p) {
        cudaFree(*p);
        *p = nullptr;
    }
    if (bytes == 0) return DP_OK;
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();  // not a later launch's
        return fail(DP_ERR_CUDA, std::string("cudaMalloc(") + std::to_string(bytes) + "): " + cudaGetErrorString(e));
    }
    return DP_OK;
}

template <typename T>
static int dalloc_t(T** p, size_t count) {
    return dalloc((void**)p, count * sizeof(T));
}

// A buffer of at least `need` entries; one that could not be had has room for none.
template <typename T, typename Count>
static int dgrow_t(T** p, Count need, Count* have) {
    if (need <= *have) return DP_OK;
    *have = 0;
    RET(dalloc_t(p, (size_t)need));
    *have = need;
    return DP_OK;
}

static int ensure_partial(dp_sim* s, long long blocks) {
    if (blocks <= s->partial_alloc) return DP_OK;
    RET(dgrow_t(&s->partial, blocks, &s->partial_alloc));
    s->version++;
    return DP_OK;
}

static void fill_scale(const dp_sim* s, double* scale, float* unit) {
    for (int k = 0; k < DP_MAX_DIM; ++k) {
        const double L = (k < s->dim) ? s->box[k] : 1.0;
        if (scale) scale[k] = 4294967296.0 / L;
        if (unit) unit[k] = (float)(L / 4294967296.0);
    }
}

// Largest fixed-point unit L / 2^32 over the axes times sqrt(D): the absolute
// error bound (with a factor 4 margin) of a float32 distance from the shadows.
static double shadow_abs_error(const dp_sim* s) {
    double lmax = 0.0;
    for (int k = 0; k < s->dim; ++k) lmax = std::max(lmax, s->box[k]);
    return 4.0 * lmax / 4294967296.0 * std::sqrt((double)s->dim);
}

// float32 squared-distance thresholds bracketing a float64 distance `r`:
// below lo the distance is certainly < r, above hi certainly > r.
static void bracket(const dp_sim* s, double r, float* lo2, float* hi2) {
    const double e = shadow_abs_error(s);
    const double lo = (r - e) * (1.0 - 1e-5);
    const double hi = (r + e) * (1.0 + 1e-5);
    *lo2 = lo > 0.0 ? (float)(lo * lo) * (1.0f - 1e-6f) : -1.0f;
    *hi2 = std::isfinite(hi) ? (float)(hi * hi) * (1.0f + 1e-6f) : INFINITY;
}

// After every write of positions or box from outside a step.
static int launch_shadow(dp_sim* s) {
    s->nl_checked = false;
    ShadowArgs a{};
    a.pos = s->pos;
    a.shadow = s->shadow;
    a.pos64 = s->pos64;
    a.st = s->dstat;
    a.n = s->n;
    for (int k = 0; k < DP_MAX_DIM; ++k) a.scale64[k] = 18446744073709551616.0 / ((k < s->dim) ? s->box[k] : 1.0);
    memcpy(a.shift64, s->shift64, sizeof(a.shift64));
    for (int k = 0; k < DP_MAX_DIM; ++k) a.box[k] = (k < s->dim) ? s->box[k] : 1.0;
    CK(cudaMemsetAsync(&s->dstat->far, 0, sizeof(int32_t), s->stream));
    const unsigned g = grid_for(s->n, kBlock);
    switch (s->dim) {
        case 2: k_shadow<2><<<g, kBlock, 0, s->stream>>>(a); break;
        case 3: k_shadow<3><<<g, kBlock, 0, s->stream>>>(a); break;
        default: k_shadow<4><<<g, kBlock, 0, s->stream>>>(a); break;
    }
    CK(cudaGetLastError());
    return DP_OK;
}

// --------------------------- mass classes ---------------------------------
static int upload_mass_coefficients(dp_sim* s) {
    const int nclass = (int)s->class_mass.size();
    std::vector<double> coef((size_t)nclass * 5);
    for (int c = 0; c < nclass; ++c) {
        const double m = s->class_mass[c];
        const double alpha = m / s->tau;
        const double beta_variance = 2 * alpha * s->temperature * s->dt;
        const double numerator = 1.0 - alpha * s->dt / 2.0 / m;
        const double denominator = 1.0 + alpha * s->dt / 2.0 / m;
        const double a = numerator / denominator;
        const double b = 1 / denominator;
        coef[c * 5 + 0] = a;
        coef[c * 5 + 1] = b * s->dt / m;
        coef[c * 5 + 2] = b / 2 / m;
        coef[c * 5 + 3] = std::sqrt(beta_variance);
        coef[c * 5 + 4] = s->dt / m;
    }
    RET(dalloc_t(&s->mcoef, coef.size()));
    CK(cudaMemcpy(s->mcoef, coef.data(), coef.size() * sizeof(double), cudaMemcpyHostToDevice));
    std::vector<float2> coef_f((size_t)nclass);
    for (int c = 0; c < nclass; ++c) coef_f[c] = make_float2((float)coef[c * 5 + 2], (float)coef[c * 5 + 3]);
    RET(dalloc_t(&s->mcoef_f, coef_f.size()));
    CK(cudaMemcpy(s->mcoef_f, coef_f.data(), coef_f.size() * sizeof(float2), cudaMemcpyHostToDevice));
    RET(dalloc_t(&s->class_mass_dev, (size_t)nclass));
    CK(cudaMemcpy(s->class_mass_dev, s->class_mass.data(), nclass * sizeof(double), cudaMemcpyHostToDevice));
    s->version++;
    return DP_OK;
}

// --------------------------- neighbour-list configuration -----------------
// The list's buffers could not be had: nothing may use them before they are.
static void no_list(dp_sim* s) {
    s->nl_built = false;
    s->nl_config_dirty = true;
}

// Room for kcap entries per particle: 4 bytes each, or 2 in 16-byte chunks
// (brick lists), whichever is more.
static int ensure_list(dp_sim* s) {
    const long long need = (long long)std::max(s->kcap, ((s->kcap + 7) & ~7) / 2) * s->n;
    const int rc = dgrow_t(&s->nl, need, &s->nl_alloc);
    if (rc != DP_OK) no_list(s);
    return rc;
}

// Largest region: 117 KB in k_brick_build, 48 KB in the pair kernels.
constexpr int kBrickMaxCap = 3072;

static int alloc_brick_slots(dp_sim* s, int cap) {
    // (grown, never shrunk: a box that is scaled step by step keeps its buffers)
    const int rc = dgrow_t(&s->brick_slots, (long long)s->nbricks * cap, &s->brick_slots_alloc);
    if (rc != DP_OK) {
        no_list(s);
        return rc;
    }
    s->brick_cap = cap;
    s->version++;
    return DP_OK;
}

// Bytes of shared memory of k_brick_build.
static size_t brick_build_smem(const dp_sim* s) {
    return (size_t)(s->brick_cap + 8) * 32 + (size_t)s->brick_cap * (4 + 2) + (size_t)(2 * s->brick_cells + 1) * 4;
}

// Bricks: blocks of 2^b cells in Morton order. The block grows while it holds
// at most 224 particles (a CTA's worth; the region then costs the fewest copies a
// particle), leaves two CTAs for every SM, and its region fits in
// shared memory several times over.
static int configure_bricks(dp_sim* s) {
    // Brick by brick from ~100 candidates a particle (its 3^D cells): below, one
    // thread per particle is as fast or faster (1,048,576 harmonic spheres, 48
    // candidates: 419 us a rebuild against 503; 490,000 in 2-D, 13: 133 against
    // 174; 130,321 in 4-D, 208: 218 against 160; 108,000 LJ, 680: 262 against 184).
    const double per_cell = s->use_cells ? (double)s->n / (double)s->ncell : 0.0;
    s->bricks = s->use_cells && s->morton && s->reorder && !s->bricks_off &&
                per_cell * std::pow(3.0, s->dim) >= 100.0;
    s->brick_pairs = false;
    if (!s->bricks) return DP_OK;
    int bits[DP_MAX_DIM] = {0, 0, 0, 0};
    auto ext_of = [&](const int* bb, int* ext) {
        long long cells = 1;
        for (int k = 0; k < DP_MAX_DIM; ++k) {
            ext[k] = k < s->dim ? (1 << bb[k]) + 2 : 1;
            cells *= ext[k];
        }
        return cells;
    };
    int b = 0;
    for (;; ++b) {
        int next[DP_MAX_DIM], ext[DP_MAX_DIM];
        memcpy(next, bits, sizeof(next));
        const int axis = s->dim - 1 - b % s->dim;  // the Morton key's lowest bit is the last axis'
        next[axis] += 1;
        const double particles = per_cell * (double)(2LL << b);
        const long long cells = ext_of(next, ext);
        if (particles > 224.0 || (double)s->n / particles < 304.0 || cells > 4096 || cells * per_cell > 2000.0 ||
            (1 << next[axis]) + 2 > s->nc[axis])  // a region spans less than the box
            break;
        memcpy(bits, next, sizeof(bits));
    }
    s->brick_bits = b;
    s->brick_cells = (int)ext_of(bits, s->brick_ext);
    std::vector<int4> base;
    int at[DP_MAX_DIM] = {0, 0, 0, 0};
    for (at[0] = 0; at[0] < s->nc[0]; at[0] += 1 << bits[0])
        for (at[1] = 0; at[1] < s->nc[1]; at[1] += 1 << bits[1])
            for (at[2] = 0; at[2] < s->nc[2]; at[2] += 1 << bits[2])
                for (at[3] = 0; at[3] < s->nc[3]; at[3] += 1 << bits[3])
                    base.push_back(make_int4(at[0], at[1], at[2], at[3]));
    s->nbricks = (int)base.size();
    if (s->nbricks > s->bricks_alloc) {
        s->bricks_alloc = 0;
        RET(dalloc_t(&s->brick_base, base.size()));
        RET(dalloc_t(&s->brick_info, base.size()));
        s->bricks_alloc = s->nbricks;
    }
    CK(cudaMemcpyAsync(s->brick_base, base.data(), base.size() * sizeof(int4), cudaMemcpyHostToDevice, s->stream));
    // the box of the brick's cells and everything within the cutoff of it (all of
    // the cells around it at most), with the spread of a random arrangement
    double side[DP_MAX_DIM], volume = 1.0;
    for (int k = 0; k < s->dim; ++k) {
        side[k] = s->box[k] / s->nc[k] * (1 << bits[k]);
        volume *= s->box[k];
    }
    const double c = s->cutoff, pi = 3.141592653589793;
    double region;
    if (s->dim == 2)
        region = side[0] * side[1] + 2 * (side[0] + side[1]) * c + pi * c * c;
    else if (s->dim == 3)
        region = side[0] * side[1] * side[2] + 2 * (side[0] * side[1] + side[1] * side[2] + side[0] * side[2]) * c +
                 pi * (side[0] + side[1] + side[2]) * c * c + 4.0 / 3.0 * pi * c * c * c;
    else
        region = 1e300;
    const double entries = std::min(per_cell * s->brick_cells, (double)s->n / volume * region);
    const double room = entries + 3.0 * std::sqrt(entries) + 32.0;
    if (!(room <= kBrickMaxCap)) {
        s->bricks = false;
        return DP_OK;
    }
    RET(alloc_brick_slots(s, (int)room & ~31));
    const double mean = per_cell * (double)(1LL << b);
    // The float32 pair kernels run on bricks where a particle lists 32 or more
    // (with a dozen listed, the region's copy costs more than the gathers it
    // saves: 101 against 78 us a step for 1,048,576 harmonic spheres), above the
    // sizes of dp_step_warp. Lanes per particle: those of dp_step_quad and dp_step,
    // so that the float32 sums are the same (LJ us a step with 1 / 4: 9,464 particles
    // 18.5 / 12.4; 42,592 20.5 / 22.6; 78,732 26.7 / 38.8).
    const double sphere = s->dim == 2 ? pi * c * c : 4.0 / 3.0 * pi * c * c * c;
    s->brick_pairs = s->dim <= 3 && s->n > s->warp_step_max && (double)s->n / volume * sphere >= 32.0;
    s->brick_lanes = s->n <= s->quad_step_max ? 4 : 1;
    s->brick_threads = std::max(64, std::min(256, ((int)(1.2 * mean * s->brick_lanes) + 31) & ~31));
    return DP_OK;
}

// Pre-filter threshold: a pair is skipped only when its float32 distance,
// whose error is < 1e-6 relative plus a few L / 2^32, certainly exceeds
// r_cut * sigma_max.
static float prefilter_cut2(const dp_sim* s) {
    double lmax = 0.0;
    for (int k = 0; k < s->dim; ++k) lmax = std::max(lmax, s->box[k]);
    const double reach = s->r_cut * s->sig_max;
    if (!std::isfinite(reach)) return INFINITY;
    const double rr = reach * (1.0 + 1e-5) + 8.0 * lmax / 4294967296.0 * std::sqrt((double)s->dim) + 1e-30;
    return (float)(rr * rr * (1.0 + 1e-6));
}

// A pair that passes the pre-filter is closer than `most` on every axis, so its
// displacement is known from the positions modulo L / 2^shift64 > 4 most, and
// their 64 bits hold that many more behind the point of the double-float
// arithmetic (dpff_from_fixed; shifting the differences instead cost the
// 256,000-particle mixture 2.5 %).
static int update_shift64(dp_sim* s) {
    const double cut = std::sqrt((double)prefilter_cut2(s));
    int shift[DP_MAX_DIM] = {0, 0, 0, 0};
    for (int k = 0; k < s->dim; ++k) {
        const double most = 1.001 * cut + 16.0 * s->box[k] / 4294967296.0;
        while (shift[k] < 16 && most * (double)(8LL << shift[k]) < s->box[k]) ++shift[k];
    }
    if (memcmp(shift, s->shift64, sizeof(shift)) == 0) return DP_OK;
    memcpy(s->shift64, shift, sizeof(shift));
    s->version++;
    return launch_shadow(s);
}

static int configure_nl(dp_sim* s) {
    if (!s->nl_config_dirty) return DP_OK;
    if (!s->have_box) return fail(DP_ERR_ARG, "box not set");
    const double reach = s->sig_max * s->r_cut;
    s->cutoff = reach + s->skin;  // dompap/Simulation.py:353-356
    bool cells = s->method == DP_NL_CELL && std::isfinite(s->cutoff) && s->cutoff > 0;
    long long ncell = 1;
    int pmax = 1;  // power of two covering the largest cell count
    for (int k = 0; k < s->dim && cells; ++k) {
        // cells strictly wider than the cutoff plus the shadow's rounding
        // (a few L / 2^32): a pair closer than the cutoff is never more than
        // one cell apart when the cells come from the shadows
        const double w = s->cutoff * (1.0 + 1e-10) + 8.0 * s->box[k] / 4294967296.0;
        const double ncd = std::floor(s->box[k] / w);
        if (!(ncd >= 3.0) || ncd > 65536.0) {
            cells = false;
            break;
        }
        s->nc[k] = (int)ncd;
        ncell *= s->nc[k];
        while (pmax < s->nc[k]) pmax <<= 1;
        if (ncell > (1LL << 30)) cells = false;
    }
    s->use_cells = cells;
    if (!cells) {
        for (int k = 0; k < DP_MAX_DIM; ++k) s->nc[k] = 0;
        s->ncell = 0;
        s->nbins = 0;
    } else {
        for (int k = s->dim; k < DP_MAX_DIM; ++k) s->nc[k] = 1;
        s->ncell = ncell;
        // Morton keys on the padded grid while it stays within 2^26 keys and
        // the bit interleaving's width (16 bits per axis in 2-D, 10 in 3-D, 8 in 4-D)
        long long padded = 1;
        for (int k = 0; k < s->dim; ++k) padded *= pmax;
        const int bits_per_axis = s->dim == 2 ? 16 : (s->dim == 3 ? 10 : 8);
        s->morton = padded <= (1LL << 26) && pmax <= (1 << bits_per_axis);
        s->nbins = s->morton ? padded : ncell;
        if (s->nbins > s->bins_alloc) {
            s->bins_alloc = 0;
            RET(dalloc_t(&s->bin_cnt, (size_t)s->nbins));
            RET(dalloc_t(&s->bin_start, (size_t)s->nbins + 1));
            RET(dalloc_t(&s->bin_part, (size_t)((s->nbins + kScanTile - 1) / kScanTile)));
            s->bins_alloc = s->nbins;
        }
        if (!s->bk_order) {  // the last of them
            const size_t n = (size_t)s->n, nd = n * s->dim;
            RET(dalloc_t(&s->bin_key, n));
            RET(dalloc_t(&s->bin_rank, n));
            RET(dalloc_t(&s->src_of, n));
            RET(dalloc_t(&s->sc_vel, nd));
            RET(dalloc_t(&s->sc_beta, nd));
            RET(dalloc_t(&s->sc_img, nd));
            RET(dalloc_t(&s->sc_order, n));
            RET(dalloc_t(&s->bk_order, n));
        }
    }
    RET(update_shift64(s));
    s->bricks_off = false;
    RET(configure_bricks(s));
    RET(ensure_list(s));
    s->nl_config_dirty = false;
    s->nl_built = false;
    s->version++;
    return DP_OK;
}

// Scratch and backup arrays of the optional per-particle arrays (types, mass
// classes, masses), allocated once those exist.
static int ensure_perm_extras(dp_sim* s) {
    const size_t n = (size_t)s->n;
    if (s->types && !s->bk_types) {
        RET(dalloc_t(&s->sc_types, n));
        RET(dalloc_t(&s->bk_types, n));
    }
    if (s->mclass && !s->bk_mclass) {
        RET(dalloc_t(&s->sc_mclass, n));
        RET(dalloc_t(&s->bk_mclass, n));
    }
    if (s->mass && !s->bk_mass) {
        RET(dalloc_t(&s->sc_mass, n));
        RET(dalloc_t(&s->bk_mass, n));
    }
    return DP_OK;
}

// The state arrays that move with their particle, with their scratch: the
// positions use the second position set (free during a rebuild: a fused step
// writes it after the rebuild, the separate integrator does not use it).
static void fill_perm_args(const dp_sim* s, PermArgs& p) {
    memset(&p, 0, sizeof(p));
    const int sh = s->dim == 2 ? 8 : 16;
    const int p64 = s->dim == 2 ? 16 : 32;
    auto add = [&](void* data, void* scratch, int esize, int comps, int alt = 0) {
        if (data && scratch) p.arr[p.count++] = PermArray{data, scratch, esize, comps, alt};
    };
    add(s->pos, s->pos_alt, 8, s->dim, 1);
    add(s->shadow, s->shadow_alt, sh, 1, 1);
    add(s->pos64, s->pos64_alt, p64, 1, 1);
    add(s->vel, s->sc_vel, 8, s->dim);
    add(s->beta, s->sc_beta, 8, s->dim);
    add(s->img, s->sc_img, 4, s->dim);
    add(s->order, s->sc_order, 4, 1);
    add(s->types, s->sc_types, 4, 1);
    add(s->mclass, s->sc_mclass, 1, 1);
    add(s->mass, s->sc_mass, 8, 1);
    p.src_of = s->src_of;
    p.order = s->order;
    p.slot_of = s->slot_of;
    p.st = s->dstat;
    p.n = s->n;
}

// The gated rebuild sequence (no effect unless need_rebuild is set).
// What the lists hold: slots, column-major, every partner or only the owned ones
// (dp_owns_pair; the surrogate mode uses each pair once); slots in rows, where a
// warp shares a particle; or region indices for the brick kernels.
enum { kListFull = 0, kListHalf = 1, kListBrick = 2, kListRows = 3 };
static int list_kind(const dp_sim* s) {
    if (s->precision == DP_PREC_MLP) return kListHalf;
    if (s->bricks && s->brick_pairs && s->step_lanes != 32 && s->lib.forces_brick) return kListBrick;
    // float32 sums follow the order of the list: cell lists keep theirs
    return s->n <= s->warp_step_max && !(s->precision == DP_PREC_FP32 && s->use_cells) ? kListRows : kListFull;
}

template <int D>
static int launch_brick_build(dp_sim* s, const NlArgs& na) {
    BrickArgs b{};
    b.base = s->brick_base;
    b.info = s->brick_info;
    b.slots = s->brick_slots;
    b.list = (uint4*)s->nl;
    b.cap = s->brick_cap;
    b.cells = s->brick_cells;
    b.keys = 1 << s->brick_bits;
    double largest = 0.0;  // a region's coordinate in half cutoffs
    for (int k = 0; k < DP_MAX_DIM; ++k) {
        b.ext[k] = s->brick_ext[k];
        if (k >= s->dim) continue;
        b.unit[k] = (float)(s->box[k] / 4294967296.0 * 2.0 / s->cutoff);
        largest = std::max(largest, s->box[k] / s->nc[k] * (b.ext[k] - 2) / s->cutoff + 2.0);
    }
    // everything the float bracket calls possibly inside is a candidate, and one
    // farther than `alarm` below the cut is inside for certain
    const double err = kBrickErr * s->dim * largest * largest, scale = 4.0 / (s->cutoff * s->cutoff);
    b.cut = (float)(((double)na.hi2 * scale + err) * (1.0 + 1e-6));
    b.alarm = (float)((2.0 * err + ((double)na.hi2 - (double)na.lo2) * scale) * (1.0 + 1e-3) + 1e-6 * b.cut);
    const size_t smem = brick_build_smem(s);
    // a warp per 16 particles of an average brick
    const int threads = 32 * std::max(2, std::min(kBrickThreads / 32, (int)((double)s->n / s->nbricks / 16.0 + 1.0)));
    void (*k)(NlArgs, BrickArgs) = list_kind(s) != kListBrick ? k_brick_build<D, true> : k_brick_build<D, false>;
    CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k<<<s->nbricks, threads, smem, s->stream>>>(na, b);
    CK(cudaGetLastError());
    return DP_OK;
}

static int launch_rebuild(dp_sim* s, long long* launches) {
    const unsigned gp = grid_for(s->n, kBlock);
    NlArgs na{};
    na.half = list_kind(s) == kListHalf ? 1 : 0;
    na.pos = s->pos;
    na.pos_ref = s->pos_ref;
    na.shadow = s->shadow;
    na.shadow_ref = s->shadow_ref;
    na.nl = s->nl;
    na.cnt = s->cnt;
    na.st = s->dstat;
    na.n = s->n;
    na.nl_k = list_kind(s) == kListRows ? 1 : s->n;
    na.nl_i = list_kind(s) == kListRows ? s->kcap : 1;
    na.kcap = s->kcap;
    na.cutoff = s->cutoff;
    bracket(s, s->cutoff, &na.lo2, &na.hi2);
    fill_scale(s, nullptr, na.unit);
    for (int k = 0; k < DP_MAX_DIM; ++k) na.box[k] = (k < s->dim) ? s->box[k] : 1.0;
    long long nl_launches = 0;
    if (s->n <= s->warp_step_max && list_kind(s) != kListFull) {
        const unsigned gr = grid_for(s->n * 32, kBlock);
        switch (s->dim) {
            case 2: k_nl_build_rows<2><<<gr, kBlock, 0, s->stream>>>(na); break;
            case 3: k_nl_build_rows<3><<<gr, kBlock, 0, s->stream>>>(na); break;
            default: k_nl_build_rows<4><<<gr, kBlock, 0, s->stream>>>(na); break;
        }
        nl_launches = 1;
    } else if (s->use_cells) {
        // counting sort of the slots by cell key
        BinArgs ba{};
        ba.shadow = s->shadow;
        ba.shadow_alt = s->shadow_alt;
        ba.order = s->order;
        ba.key = s->bin_key;
        ba.rank = s->bin_rank;
        ba.bin_cnt = s->bin_cnt;
        ba.bin_start = s->bin_start;
        ba.bin_part = s->bin_part;
        ba.src_of = s->src_of;
        ba.st = s->dstat;
        ba.n = s->n;
        ba.nbins = s->nbins;
        ba.morton = s->morton ? 1 : 0;
        for (int k = 0; k < DP_MAX_DIM; ++k) ba.nc[k] = s->nc[k];
        const int parts = (int)((s->nbins + kScanTile - 1) / kScanTile);
        k_bin_clear<<<(unsigned)std::min<long long>(grid_for(s->nbins, kBlock), 8192), kBlock, 0, s->stream>>>(ba);
        switch (s->dim) {
            case 2: k_bin_count<2><<<gp, kBlock, 0, s->stream>>>(ba); break;
            case 3: k_bin_count<3><<<gp, kBlock, 0, s->stream>>>(ba); break;
            default: k_bin_count<4><<<gp, kBlock, 0, s->stream>>>(ba); break;
        }
        k_scan_reduce<<<parts, kScanThreads, 0, s->stream>>>(ba);
        k_scan_top<<<1, kScanThreads, 0, s->stream>>>(ba, parts);
        k_scan_down<<<parts, kScanThreads, 0, s->stream>>>(ba);
        k_bin_scatter<<<gp, kBlock, 0, s->stream>>>(ba);
        k_bin_sort<<<grid_for(s->nbins, kBlock / kSortLanes), kBlock, 0, s->stream>>>(ba);
        nl_launches = 7;
        if (s->reorder) {
            // the state into cell order: slot t <- slot src_of[t]
            PermArgs pa;
            fill_perm_args(s, pa);
            const dim3 gpa(gp, (unsigned)pa.count);
            k_permute<<<gpa, kBlock, 0, s->stream>>>(pa);
            k_permute_back<<<gpa, kBlock, 0, s->stream>>>(pa);
            nl_launches += 2;
        }
        na.bin_start = s->bin_start;
        na.src_of = s->reorder ? nullptr : s->src_of;
        na.morton = ba.morton;
        for (int k = 0; k < DP_MAX_DIM; ++k) na.nc[k] = s->nc[k];
        if (s->bricks)
            switch (s->dim) {
                case 2: RET(launch_brick_build<2>(s, na)); break;
                case 3: RET(launch_brick_build<3>(s, na)); break;
                default: RET(launch_brick_build<4>(s, na)); break;
            }
        else switch (s->dim) {
            case 2: k_nl_build_cells<2><<<gp, kBlock, 0, s->stream>>>(na); break;
            case 3: k_nl_build_cells<3><<<gp, kBlock, 0, s->stream>>>(na); break;
            default: k_nl_build_cells<4><<<gp, kBlock, 0, s->stream>>>(na); break;
        }
        nl_launches += 1;
    } else {
        switch (s->dim) {
            case 2: k_nl_build_allpairs<2><<<gp, kBlock, 0, s->stream>>>(na); break;
            case 3: k_nl_build_allpairs<3><<<gp, kBlock, 0, s->stream>>>(na); break;
            default: k_nl_build_allpairs<4><<<gp, kBlock, 0, s->stream>>>(na); break;
        }
        nl_launches = 1;
    }
    k_rebuild_done<<<1, 1, 0, s->stream>>>(s->dstat, s->kcap, s->bricks ? s->brick_cap : 0x7FFFFFFF);
    CK(cudaGetLastError());
    if (launches) *launches += nl_launches + 1;
    return DP_OK;
}

// The pair kernels' constants of one (sigma, epsilon): sigma, 1/sigma,
// epsilon, 1/sigma^2, epsilon/sigma (DP_FF_PARAMS), as double-floats in the
// parity mode and as float32 otherwise.
static void pair_consts(double sigma, double epsilon, double* c) {
    c[0] = sigma;
    c[1] = 1.0 / sigma;
    c[2] = epsilon;
    c[3] = 1.0 / (sigma * sigma);
    c[4] = epsilon / sigma;
}
static float2 split_ff(double v) { return make_float2((float)v, (float)(v - (double)(float)v)); }
static float4 pair_consts_f32(const double* c) {
    return make_float4((float)c[0], (float)c[1], (float)c[2], 0.0f);
}

static void fill_pair_args(const dp_sim* s, dp_pair_args& a, double* out) {
    memset(&a, 0, sizeof(a));
    a.pos = s->pos;
    a.shadow = s->shadow;
    a.nl = s->nl;
    a.cnt = s->cnt;
    a.types = s->types;
    a.sig_tab = s->sig_tab;
    a.eps_tab = s->eps_tab;
    a.isig_tab = s->isig_tab;
    a.ff_tab = s->ff_tab;
    a.f32_tab = s->f32_tab;
    a.pos64 = s->pos64;
    a.order = s->order;
    a.nl_k = list_kind(s) == kListRows ? 1 : s->n;
    a.nl_i = list_kind(s) == kListRows ? s->kcap : 1;
    a.brick_info = s->brick_info;
    a.brick_slots = s->brick_slots;
    a.brick_list = (const uint4*)s->nl;
    a.brick_cap = s->brick_cap;
    a.out = out;
    a.partial = s->partial;
    a.status = s->dstat;
    a.n = s->n;
    a.ntypes = s->ntypes;
    for (int k = 0; k < DP_MAX_DIM; ++k) a.box[k] = (k < s->dim) ? s->box[k] : 1.0;
    fill_scale(s, nullptr, a.unit);
    for (int k = 0; k < DP_MAX_DIM; ++k) {
        const double u64 = ((k < s->dim) ? s->box[k] : 1.0) / 18446744073709551616.0 / (double)(1LL << s->shift64[k]);
        a.unit64_hi[k] = (float)u64;
        a.unit64_lo[k] = (float)(u64 - (double)(float)u64);
    }
    a.sigma = s->sigma;
    a.inv_sigma = 1.0 / s->sigma;
    a.epsilon = s->epsilon;
    a.rcut = s->r_cut;
    a.rcut_f = (float)s->r_cut;
    a.rcut_finite = std::isfinite(s->r_cut) ? 1 : 0;
    a.rcut2_f = (float)(s->r_cut * s->r_cut);
    {
        double c[DP_FF_PARAMS];
        pair_consts(s->sigma, s->epsilon, c);
        for (int t = 0; t < DP_FF_PARAMS; ++t) {
            const float2 v = split_ff(c[t]);
            a.ff_const[2 * t] = v.x;
            a.ff_const[2 * t + 1] = v.y;
        }
        const float4 f = pair_consts_f32(c);
        a.f32_const[0] = f.x;
        a.f32_const[1] = f.y;
        a.f32_const[2] = f.z;
        a.f32_const[3] = f.w;
    }
    a.cut2f = prefilter_cut2(s);
}

static bool use_mlp_tcgen05(const dp_sim* s) {
    return s->mlp_tensor == 1 || (s->mlp_tensor == 0 && s->n >= 65536);
}

// Lanes per particle of the mma.sync pass: up to 8, until its warps fill the GPU
// (two 256-thread CTAs on each of 152 SMs).
static int mlp_split(const dp_sim* s) {
    int split = 1;
    while (split < 8 && s->n * split < 152LL * 2 * 256) split *= 2;
    return split;
}

// Fixed-point force sums of the surrogate pass (allocated outside any graph
// capture: run() calls this before capturing).
static int ensure_mlp_fx(dp_sim* s) {
    if (s->mlp_fx) return DP_OK;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    CK(cudaStreamIsCapturing(s->stream, &cs));
    if (cs != cudaStreamCaptureStatusNone) return fail(DP_ERR_CUDA, "surrogate force sums not allocated before capture");
    RET(dalloc_t(&s->mlp_fx, (size_t)s->n * s->dim));
    CK(cudaMemsetAsync(s->mlp_fx, 0, (size_t)s->n * s->dim * sizeof(unsigned long long), s->stream));
    return DP_OK;
}

// Lanes per particle of the force, energy, virial and Laplacian sums over lists
// of slots (not the surrogate program's): the thresholds of the fused step.
static int sum_lanes(const dp_sim* s) {
    if (s->precision == DP_PREC_MLP) return mlp_split(s);
    return s->n <= s->warp_step_max ? 32 : (s->n <= s->quad_step_max ? 4 : 1);
}

// A brick kernel: one CTA per brick, its region in dynamic shared memory.
static size_t brick_smem(const dp_sim* s) { return (size_t)s->brick_cap * 16; }
static int launch_brick(dp_sim* s, cudaKernel_t k, int threads, void** args) {
    int dev = 0;
    CK(cudaGetDevice(&dev));
    const size_t smem = brick_smem(s);
    CK(cudaKernelSetAttributeForDevice(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem, dev));
    CK(cudaLaunchKernel((const void*)k, dim3(s->nbricks), dim3(threads), args, smem, s->stream));
    return DP_OK;
}

static int launch_pair(dp_sim* s, cudaKernel_t k, double* out, long long* launches) {
    dp_pair_args a;
    fill_pair_args(s, a, out);
    if (s->precision == DP_PREC_MLP) {
        cudaKernel_t km = nullptr;
        if (k == s->lib.forces) km = s->lib.forces_mlp;
        else if (k == s->lib.energy) km = s->lib.energy_mlp;
        else if (k == s->lib.virial) km = s->lib.virial_mlp;
        if (!km) return fail(DP_ERR_ARG, "this quantity is not available with the pair surrogate");
        const dp_mlp_dev* mp = s->mlp_dev;
        unsigned long long* fx = nullptr;
        if (km == s->lib.forces_mlp) {
            RET(ensure_mlp_fx(s));
            fx = s->mlp_fx;
        }
        void* args[] = {&a, &mp, &fx};
        if (use_mlp_tcgen05(s)) {
            // the tcgen05 pass: 128 particles (rows of the tensor-core tile) per CTA
            cudaKernel_t kt = km == s->lib.forces_mlp ? s->lib.forces_mlp_tc
                            : (km == s->lib.energy_mlp ? s->lib.energy_mlp_tc : s->lib.virial_mlp_tc);
            CK(cudaLaunchKernel((const void*)kt, dim3(grid_for(s->n, 128)), dim3(128), args, 0, s->stream));
        } else {
            a.mlp_split = mlp_split(s);
            CK(cudaLaunchKernel((const void*)km, dim3(grid_for(s->n * a.mlp_split, kBlock)), dim3(kBlock), args, 0,
                                s->stream));
        }
        if (fx) {
            void* fargs[] = {&a, &fx};
            CK(cudaLaunchKernel((const void*)s->lib.mlp_finish, dim3(grid_for(s->n * s->dim, kBlock)), dim3(kBlock),
                                fargs, 0, s->stream));
            if (launches) *launches += 1;
        }
    } else if (k == s->lib.forces && s->force_method != DP_METHOD_LIST && s->lib.forces_all) {
        a.upper = s->force_method == DP_METHOD_ALLPAIRS_NEWTON ? 1 : 0;
        void* args[] = {&a};
        CK(cudaLaunchKernel((const void*)s->lib.forces_all, dim3(grid_for(s->n * 32, kBlock)), dim3(kBlock), args, 0,
                            s->stream));
    } else if (k == s->lib.energy && s->energy_method != DP_METHOD_LIST && s->lib.energy_all) {
        void* args[] = {&a};
        CK(cudaLaunchKernel((const void*)s->lib.energy_all, dim3(grid_for(s->n * 32, kBlock)), dim3(kBlock), args, 0,
                            s->stream));
    } else if (list_kind(s) == kListBrick) {
        void* args[] = {&a};
        cudaKernel_t kb = k == s->lib.forces ? s->lib.forces_brick
                        : k == s->lib.energy ? s->lib.energy_brick
                        : k == s->lib.virial ? s->lib.virial_brick : s->lib.laplacian_brick;
        RET(launch_brick(s, kb, kBlock, args));
    } else {
        void* args[] = {&a};
        const int lanes = sum_lanes(s);
        if (lanes > 1)
            k = s->lib.split[lanes == 32 ? 0 : 1][k == s->lib.forces ? 0 : (k == s->lib.energy ? 1 : (k == s->lib.virial ? 2 : 3))];
        CK(cudaLaunchKernel((const void*)k, dim3(grid_for(s->n * lanes, kBlock)), dim3(kBlock), args, 0, s->stream));
    }
    if (launches) *launches += 1;
    return DP_OK;
}

// Integrator arguments; the outputs default to the current buffers (in place).
static void fill_int_args(const dp_sim* s, dp_int_args& a, long long step_offset, int kind = DP_INT_GJF) {
    memset(&a, 0, sizeof(a));
    a.pos = s->pos;
    a.pos_out = s->pos;
    a.vel = s->vel;
    a.beta = s->beta;
    a.force = s->force;
    a.img = s->img;
    a.shadow_out = s->shadow;
    a.pos64_out = s->pos64;
    a.pos_ref = s->pos_ref;
    a.shadow_ref = s->shadow_ref;
    a.mclass = s->mclass;
    a.mcoef = s->mcoef;
    a.mcoef_f = s->mcoef_f;
    a.mass = s->mass;
    a.order = s->order;
    a.st = s->dstat;
    a.n = s->n;
    for (int k = 0; k < DP_MAX_DIM; ++k) a.box[k] = (k < s->dim) ? s->box[k] : 1.0;
    fill_scale(s, nullptr, a.unit);
    for (int k = 0; k < DP_MAX_DIM; ++k) a.scale64[k] = 18446744073709551616.0 / ((k < s->dim) ? s->box[k] : 1.0);
    memcpy(a.shift64, s->shift64, sizeof(a.shift64));
    a.thr = (0.5 * s->skin) * (0.5 * s->skin);
    bracket(s, 0.5 * s->skin, &a.thr_lo, &a.thr_hi);
    a.dt = s->dt;
    {
        const double m = s->class_mass[0];
        const double alpha = m / s->tau;
        const double beta_variance = 2 * alpha * s->temperature * s->dt;
        const double numerator = 1.0 - alpha * s->dt / 2.0 / m;
        const double denominator = 1.0 + alpha * s->dt / 2.0 / m;
        const double aa = numerator / denominator;
        const double b = 1 / denominator;
        a.coef[0] = aa;
        a.coef[1] = b * s->dt / m;
        a.coef[2] = b / 2 / m;
        a.coef[3] = std::sqrt(beta_variance);
        a.coef[4] = s->dt / m;
        a.coef_f[0] = (float)a.coef[2];
        a.coef_f[1] = (float)a.coef[3];
    }
    a.temperature = s->temperature;
    a.tau = s->tau;
    a.seed = s->seed;
    a.step_offset = step_offset;
    a.massmode = s->mass_mode;
    a.nve = kind == DP_INT_NVE ? 1 : 0;
}

template <int D, bool NVE, bool W64>
static void launch_integrate_dw(dp_sim* s, const dp_int_args& a) {
    const unsigned g = grid_for(s->n, kBlock);
    switch (s->mass_mode) {
        case 0: k_integrate<D, 0, NVE, W64><<<g, kBlock, 0, s->stream>>>(a); break;
        case 1: k_integrate<D, 1, NVE, W64><<<g, kBlock, 0, s->stream>>>(a); break;
        default: k_integrate<D, 2, NVE, W64><<<g, kBlock, 0, s->stream>>>(a); break;
    }
}

// The 64-bit fixed point is only read by the float64-parity pair kernels.
template <int D, bool NVE>
static void launch_integrate_d(dp_sim* s, const dp_int_args& a) {
    if (s->precision == DP_PREC_FP64)
        launch_integrate_dw<D, NVE, true>(s, a);
    else
        launch_integrate_dw<D, NVE, false>(s, a);
}

static int launch_integrate(dp_sim* s, int kind, long long step_offset, long long* launches) {
    dp_int_args a;
    fill_int_args(s, a, step_offset, kind);
    const bool nve = kind == DP_INT_NVE;
    switch (s->dim) {
        case 2: nve ? launch_integrate_d<2, true>(s, a) : launch_integrate_d<2, false>(s, a); break;
        case 3: nve ? launch_integrate_d<3, true>(s, a) : launch_integrate_d<3, false>(s, a); break;
        default: nve ? launch_integrate_d<4, true>(s, a) : launch_integrate_d<4, false>(s, a); break;
    }
    CK(cudaGetLastError());
    if (launches) *launches += 1;
    return DP_OK;
}

static int launch_skin_check(dp_sim* s) {
    SkinArgs a{};
    a.pos = s->pos;
    a.pos_ref = s->pos_ref;
    a.shadow = s->shadow;
    a.shadow_ref = s->shadow_ref;
    a.st = s->dstat;
    a.n = s->n;
    for (int k = 0; k < DP_MAX_DIM; ++k) a.box[k] = (k < s->dim) ? s->box[k] : 1.0;
    fill_scale(s, nullptr, a.unit);
    a.thr = (0.5 * s->skin) * (0.5 * s->skin);
    bracket(s, 0.5 * s->skin, &a.thr_lo, &a.thr_hi);
    const unsigned g = grid_for(s->n, kBlock);
    switch (s->dim) {
        case 2: k_skin_check<2><<<g, kBlock, 0, s->stream>>>(a); break;
        case 3: k_skin_check<3><<<g, kBlock, 0, s->stream>>>(a); break;
        default: k_skin_check<4><<<g, kBlock, 0, s->stream>>>(a); break;
    }
    CK(cudaGetLastError());
    return DP_OK;
}

static int read_status(dp_sim* s) {
    CK(cudaMemcpyAsync(s->hstat, s->dstat, sizeof(dp_dev_status), cudaMemcpyDeviceToHost, s->stream));
    CK(cudaStreamSynchronize(s->stream));
    return DP_OK;
}

// A bounded device-side wait gave up (the tensor-core surrogate pass): the
// launch's results are invalid; report it and clear the flag.
static int write_status(dp_sim* s);
static int check_device_error(dp_sim* s) {
    if (!s->hstat->device_error) return DP_OK;
    s->hstat->device_error = 0;
    RET(write_status(s));
    return fail(DP_ERR_TIMEOUT, "a bounded device-side wait gave up (tensor-core surrogate pass); the launch's "
                                "results are discarded");
}

// Without a wait: hstat must not change before the next read_status.
static int send_status(dp_sim* s) {
    CK(cudaMemcpyAsync(s->dstat, s->hstat, sizeof(dp_dev_status), cudaMemcpyHostToDevice, s->stream));
    return DP_OK;
}

static int write_status(dp_sim* s) {
    RET(send_status(s));
    CK(cudaStreamSynchronize(s->stream));
    return DP_OK;
}

static int require_ready(dp_sim* s) {
    if (!s) return fail(DP_ERR_ARG, "null handle");
    if (!s->have_box) return fail(DP_ERR_ARG, "box not set");
    if (!s->have_pot || !s->lib_valid) return fail(DP_ERR_NOPOT, "no pair potential set");
    return DP_OK;
}

// Grow capacities after an overflow reported in hstat; returns 1 if grown.
static int grow_after_overflow(dp_sim* s, bool* grown) {
    *grown = false;
    if (s->hstat->max_neighbors > s->kcap) {
        const int want = ((int)(s->hstat->max_neighbors * 1.25) + 32 + 31) & ~31;
        s->kcap = want;
        RET(ensure_list(s));
        *grown = true;
    }
    if (s->bricks && s->hstat->cell_overflow > s->brick_cap) {
        // a denser region than expected
        const int want = ((int)(s->hstat->cell_overflow * 1.2) + 32 + 31) & ~31;
        if (want > kBrickMaxCap) {
            // the lists become lists of slots (list_kind), the pair kernels theirs
            s->bricks_off = true;
            s->bricks = s->brick_pairs = false;
            s->version++;
        } else {
            RET(alloc_brick_slots(s, want));
        }
        *grown = true;
    }
    if (*grown) {
        s->version++;
        s->hstat->max_neighbors = 0;
        s->hstat->cell_overflow = 0;
        s->nl_kind = list_kind(s);  // the caller rebuilds
    }
    return DP_OK;
}

// Rebuild now if needed (check) or unconditionally; handles overflow growth.
// Two waits on the GPU when a rebuild is due and one when none is; none where
// nothing has moved since the last check (nl_checked: cleared by everything that
// writes positions or the box). hstat is current afterwards either way.
static int update_nl(dp_sim* s, bool check, int* rebuilt) {
    RET(configure_nl(s));
    if (rebuilt) *rebuilt = 0;
    const bool usable = s->nl_built && s->nl_kind == list_kind(s);
    if (check && usable && s->nl_checked) return DP_OK;
    if (s->use_cells) RET(ensure_perm_extras(s));
    if (check && usable) RET(launch_skin_check(s));
    RET(read_status(s));
    const long long before = s->hstat->rebuilds;
    bool due = !check || !usable || s->hstat->need_rebuild != 0;
    for (int attempt = 0; due && attempt < 8; ++attempt) {
        s->hstat->need_rebuild = 1;
        s->hstat->max_neighbors = 0;
        s->hstat->cell_overflow = 0;
        RET(send_status(s));
        RET(launch_rebuild(s, nullptr));
        RET(read_status(s));
        RET(grow_after_overflow(s, &due));
    }
    s->nl_built = true;
    s->nl_checked = true;
    s->nl_kind = list_kind(s);
    if (rebuilt) *rebuilt = (s->hstat->rebuilds != before) ? 1 : 0;
    return DP_OK;
}

// --------------------------- graphs ---------------------------------------
// The rebuild sequence as an IF node of the graph being captured on
// s->stream: a one-thread kernel sets the condition from need_rebuild, and the
// body (captured on s->cstream) runs the cell and list kernels, so steps
// without a rebuild launch none of them.
// Or a group's: k_group_begin has set the condition (h).
static int capture_conditional_rebuild(dp_sim* s, cudaGraph_t graph, cudaGraphConditionalHandle h, bool set_cond,
                                       long long* launches, long long* body_launches) {
    if (set_cond) {
        k_rebuild_cond<<<1, 1, 0, s->stream>>>(s->dstat, h);
        CK(cudaGetLastError());
        *launches += 1;
    }
    cudaStreamCaptureStatus cs;
    const cudaGraphNode_t* deps = nullptr;
    size_t nd = 0;
    CK(cudaStreamGetCaptureInfo(s->stream, &cs, nullptr, nullptr, &deps, nullptr, &nd));
    cudaGraphNodeParams p = {cudaGraphNodeTypeConditional};
    p.conditional.handle = h;
    p.conditional.type = cudaGraphCondTypeIf;
    p.conditional.size = 1;
    cudaGraphNode_t node;
    CK(cudaGraphAddNode(&node, graph, deps, nullptr, nd, &p));
    CK(cudaStreamUpdateCaptureDependencies(s->stream, &node, nullptr, 1, cudaStreamSetCaptureDependencies));
    cudaStream_t inner = s->bstream;
    CK(cudaStreamBeginCaptureToGraph(inner, p.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                     cudaStreamCaptureModeThreadLocal));
    std::swap(s->stream, inner);
    long long body = 0;
    const int rc = launch_rebuild(s, &body);
    std::swap(s->stream, inner);
    cudaGraph_t out = nullptr;
    const cudaError_t e = cudaStreamEndCapture(inner, &out);
    RET(rc);
    if (e != cudaSuccess) return fail(DP_ERR_CUDA, std::string("conditional body capture: ") + cudaGetErrorString(e));
    *body_launches = body;
    return DP_OK;
}

static bool use_fused_step(const dp_sim* s) {
    return s->fused_step && s->precision != DP_PREC_MLP && s->lib.step != nullptr;
}

// run() without a neighbour list: the all-pairs fused step
static bool use_allpairs_step(const dp_sim* s) {
    return use_fused_step(s) && s->force_method != DP_METHOD_LIST && s->lib.step_all != nullptr;
}

static int step_lanes(const dp_sim* s) {
    return s->step_lanes ? s->step_lanes : (s->n <= s->warp_step_max ? 32 : (s->n <= s->quad_step_max ? 4 : 1));
}

// The fused steps rebuild their own lists (dp_step_lists): no rebuild kernels in
// the graph of steps.
static bool use_own_lists(const dp_sim* s) {
    return use_fused_step(s) && !use_allpairs_step(s) && list_kind(s) == kListRows && step_lanes(s) == 32;
}

// The two position buffer sets change roles (host pointers only).
static void swap_position_buffers(dp_sim* s) {
    std::swap(s->pos, s->pos_alt);
    std::swap(s->shadow, s->shadow_alt);
    std::swap(s->pos64, s->pos64_alt);
}

// Fused step: forces from the current buffers, integration into the others.
// end_flags: DP_END_* work of the kernel's last CTA (graphs only).
static int launch_step(dp_sim* s, int kind, long long step_offset, long long* launches, int end_flags = 0) {
    dp_pair_args pa;
    fill_pair_args(s, pa, nullptr);
    dp_int_args ia;
    fill_int_args(s, ia, step_offset, kind);
    ia.end_flags = end_flags;
    ia.force = nullptr;
    ia.pos_out = s->pos_alt;
    ia.shadow_out = s->shadow_alt;
    ia.pos64_out = s->pos64_alt;
    void* args[] = {&pa, &ia};
    if (use_allpairs_step(s)) {
        pa.upper = s->force_method == DP_METHOD_ALLPAIRS_NEWTON ? 1 : 0;
        CK(cudaLaunchKernel((const void*)s->lib.step_all, dim3(grid_for(s->n * 32, kBlock)), dim3(kBlock), args, 0,
                            s->stream));
        if (launches) *launches += 1;
        return DP_OK;
    }
    if (list_kind(s) == kListBrick) {
        const int lanes = s->step_lanes ? s->step_lanes : s->brick_lanes;
        RET(launch_brick(s, s->lib.step_brick[lanes == 1 ? 0 : 1], s->brick_threads, args));
        if (launches) *launches += 1;
        return DP_OK;
    }
    const int lanes = step_lanes(s);
    if (end_flags & DP_END_OWN_LISTS) {
        dp_list_args l{};
        l.nl = s->nl;
        l.cnt = s->cnt;
        l.pos_ref = s->pos_ref;
        l.shadow_ref = s->shadow_ref;
        l.cutoff = s->cutoff;
        bracket(s, s->cutoff, &l.lo2, &l.hi2);
        l.kcap = s->kcap;
        // CTAs for every SM before warps for every CTA
        const int warps = (int)std::max<long long>(1, std::min<long long>(8, s->n / 152));
        void* largs[] = {&pa, &ia, &l};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid_for(s->n, warps));
        cfg.blockDim = dim3(32 * warps);
        cfg.stream = s->stream;
        cudaLaunchAttribute attr = {};
        attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr.val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        CK(cudaLaunchKernelExC(&cfg, (const void*)s->lib.step_lists, largs));
    } else if (lanes == 32 && s->lib.step_warp) {
        // small system: one warp per particle (32 n threads)
        CK(cudaLaunchKernel((const void*)s->lib.step_warp, dim3(grid_for(s->n * 32, kBlock)), dim3(kBlock), args, 0,
                            s->stream));
    } else if (lanes == 4 && s->lib.step_quad) {
        CK(cudaLaunchKernel((const void*)s->lib.step_quad, dim3(grid_for(s->n * 4, kBlock)), dim3(kBlock), args, 0,
                            s->stream));
    } else {
        CK(cudaLaunchKernel((const void*)s->lib.step, dim3(grid_for(s->n, kBlock)), dim3(kBlock), args, 0,
                            s->stream));
    }
    if (launches) *launches += 1;
    return DP_OK;
}

// One chunk of steps into the graph being captured on s->stream; with
// `conditional` the rebuild sequence goes into IF nodes, otherwise the gated
// kernels are launched every step. A fused chunk swaps the host's position
// pointers once per captured step (the caller undoes that until the graph
// has run).
static int record_steps(dp_sim* s, long long steps, int kind, cudaGraph_t graph, bool conditional, bool fused,
                        long long* launches, long long* rebuild_launches) {
    *rebuild_launches = 0;
    const bool own_lists = use_own_lists(s);
    const bool no_list = use_allpairs_step(s) || own_lists;
    for (long long t = 0; t < steps; ++t) {
        // after a fused step every position is wrapped and `far` is clear (the
        // step's last CTA clears it); the non-fused kernels clear it in
        // k_integrate, before the next step's list check and pair loop
        if (no_list) {
            // no list to keep (the step reads every particle's position), or the
            // step keeps it
        } else if (conditional) {
            cudaGraphConditionalHandle h;  // one per node
            CK(cudaGraphConditionalHandleCreate(&h, graph, 0, 0));
            RET(capture_conditional_rebuild(s, graph, h, true, launches, rebuild_launches));
        } else {
            RET(launch_rebuild(s, launches));
        }
        if (fused) {
            RET(launch_step(s, kind, t, launches, DP_END_CLEAR_FAR | (own_lists ? DP_END_OWN_LISTS : 0)));
            swap_position_buffers(s);
        } else {
            RET(launch_pair(s, s->lib.forces, s->force, launches));
            RET(launch_integrate(s, kind, t, launches));
        }
    }
    k_advance_step<<<1, 1, 0, s->stream>>>(s->dstat, steps, fused && steps > 0 ? 1 : 0);
    CK(cudaGetLastError());
    *launches += 1;
    return DP_OK;
}

// Grouped steps: cell lists (the small systems that keep their own lists aside).
constexpr int kGroupSteps = 12;  // even: a group that is not interrupted leaves the first position set current

static bool use_groups(const dp_sim* s) {
    const int kind = list_kind(s);
    return s->conditional_graphs && s->cstream && s->bstream && use_fused_step(s) && !use_allpairs_step(s) &&
           !use_own_lists(s) && s->use_cells && s->reorder &&
           (kind == kListFull || kind == kListBrick);
}

// Any number of steps as one WHILE node whose body is a group: an IF node with
// the rebuild, then kGroupSteps steps that do nothing once a rebuild is due or no
// step is left. A conditional node per step cost ~5 us a step, and the
// device runtime in the step's own program, to set the next step's condition,
// ~6 more; a rebuild now wastes the rest of its group, ~2 us a step. The
// rebuild's permutation always leaves the positions in the first buffer set,
// so that an interrupted group starts the next one with its buffers in place.
// LJ with float32 forces, 20,672 particles: 28.3 -> 22.7 us a step; 4-D harmonic,
// 130,321: 36.0 -> 30.0; groups of 4 / 8 / 12 / 16 steps: 24.4 / 24.0 / 22.7 / 23.2.
static int build_group(dp_sim* s, int kind, int most, GraphEntry* g) {
    cudaGraph_t graph = nullptr;
    CK(cudaGraphCreate(&graph, 0));
    const double* pos_key = s->pos;
    long long launches = 0, rebuild_launches = 0;
    auto record = [&]() -> int {
        cudaGraphConditionalHandle again;
        CK(cudaGraphConditionalHandleCreate(&again, graph, 1, cudaGraphCondAssignDefault));
        cudaGraphNodeParams p = {cudaGraphNodeTypeConditional};
        p.conditional.handle = again;
        p.conditional.type = cudaGraphCondTypeWhile;
        p.conditional.size = 1;
        cudaGraphNode_t node;
        CK(cudaGraphAddNode(&node, graph, nullptr, nullptr, 0, &p));
        cudaGraph_t body = p.conditional.phGraph_out[0];
        CK(cudaStreamBeginCaptureToGraph(s->cstream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
        std::swap(s->stream, s->cstream);
        auto group = [&]() -> int {
            cudaGraphConditionalHandle rebuild;
            CK(cudaGraphConditionalHandleCreate(&rebuild, body, 0, 0));
            k_group_begin<<<1, 1, 0, s->stream>>>(s->dstat, rebuild);
            CK(cudaGetLastError());
            RET(capture_conditional_rebuild(s, body, rebuild, false, &launches, &rebuild_launches));
            for (int t = 0; t < kGroupSteps; ++t) {
                RET(launch_step(s, kind, 0, &launches, DP_END_CLEAR_FAR | DP_END_GROUP));
                swap_position_buffers(s);
            }
            k_group_end<<<1, 1, 0, s->stream>>>(s->dstat, again, most);
            CK(cudaGetLastError());
            launches += 2;
            return DP_OK;
        };
        const int rc = group();
        while (s->pos != pos_key) swap_position_buffers(s);
        std::swap(s->stream, s->cstream);
        cudaGraph_t out = nullptr;
        const cudaError_t e = cudaStreamEndCapture(s->cstream, &out);
        RET(rc);
        CK(e);
        return DP_OK;
    };
    int rc = record();
    if (rc == DP_OK) {
        const cudaError_t e = cudaGraphInstantiate(&g->exec, graph, 0);
        if (e != cudaSuccess) rc = fail(DP_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
    }
    if (rc != DP_OK) cudaGetLastError();
    cudaGraphDestroy(graph);
    RET(rc);
    g->steps = -1;
    g->kind = kind;
    g->version = s->version;
    g->launches = launches;  // per group
    g->rebuild_launches = rebuild_launches;
    g->fused = true;
    g->pos_key = pos_key;
    return DP_OK;
}

// Capture a chunk graph (conditional rebuild nodes when the CUDA driver takes
// them) and instantiate it.
static int build_graph(dp_sim* s, long long steps, int kind, bool conditional, GraphEntry* g) {
    cudaGraph_t graph = nullptr;
    CK(cudaGraphCreate(&graph, 0));
    cudaError_t e = cudaStreamBeginCaptureToGraph(s->stream, graph, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) {
        cudaGraphDestroy(graph);
        return fail(DP_ERR_CUDA, std::string("cudaStreamBeginCaptureToGraph: ") + cudaGetErrorString(e));
    }
    long long launches = 0, rebuild_launches = 0;
    const bool fused = use_fused_step(s);
    const double* pos_key = s->pos;
    const int rc = record_steps(s, steps, kind, graph, conditional, fused, &launches, &rebuild_launches);
    // the graph has not run yet: put the position pointers back
    while (s->pos != pos_key) swap_position_buffers(s);
    cudaGraph_t captured = nullptr;
    e = cudaStreamEndCapture(s->stream, &captured);
    if (rc != DP_OK || e != cudaSuccess) {
        cudaGraphDestroy(graph);
        cudaGetLastError();
        return rc != DP_OK ? rc : fail(DP_ERR_CUDA, std::string("cudaStreamEndCapture: ") + cudaGetErrorString(e));
    }
    g->steps = steps;
    g->kind = kind;
    g->version = s->version;
    g->launches = launches;
    g->rebuild_launches = rebuild_launches;
    g->fused = fused;
    g->pos_key = pos_key;
    e = cudaGraphInstantiate(&g->exec, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(DP_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
    }
    return DP_OK;
}

// Steps between status reads (and state backups), at most.
constexpr int kMaxChunk = 1024;

// The graph of `steps` steps; -1: the grouped steps, for any number.
static int get_graph(dp_sim* s, long long steps, int kind, GraphEntry** out) {
    for (auto& g : s->graphs) {
        if (g.steps == steps && g.kind == kind && g.version == s->version && g.pos_key == s->pos &&
            g.fused == use_fused_step(s)) {
            *out = &g;
            return DP_OK;
        }
    }
    // drop stale graphs
    for (auto it = s->graphs.begin(); it != s->graphs.end();) {
        if (it->version != s->version) {
            cudaGraphExecDestroy(it->exec);
            it = s->graphs.erase(it);
        } else {
            ++it;
        }
    }
    GraphEntry g;
    int rc = DP_ERR_CUDA;
    if (s->conditional_graphs && s->cstream && s->bstream) {
        rc = steps < 0 ? build_group(s, kind, kMaxChunk + 2, &g) : build_graph(s, steps, kind, true, &g);
        // a driver without conditional nodes: the gated kernels from now on
        if (rc != DP_OK) s->conditional_graphs = false;
    }
    if (rc != DP_OK && steps < 0) return rc;  // the caller takes chunks of steps
    if (rc != DP_OK) RET(build_graph(s, steps, kind, false, &g));
    s->graphs.push_back(g);
    *out = &s->graphs.back();
    return DP_OK;
}

// The state a chunk of steps starts from, for its replay after a list
// overflow. A rebuild inside the chunk may reorder the slots, so the slot
// order and the per-particle parameters it moves are saved with the state.
static int backup_state(dp_sim* s) {
    const size_t n = (size_t)s->n, bd = n * s->dim * sizeof(double), bi = n * s->dim * sizeof(int32_t);
    CK(cudaMemcpyAsync(s->bk_pos, s->pos, bd, cudaMemcpyDeviceToDevice, s->stream));
    CK(cudaMemcpyAsync(s->bk_vel, s->vel, bd, cudaMemcpyDeviceToDevice, s->stream));
    CK(cudaMemcpyAsync(s->bk_beta, s->beta, bd, cudaMemcpyDeviceToDevice, s->stream));
    CK(cudaMemcpyAsync(s->bk_img, s->img, bi, cudaMemcpyDeviceToDevice, s->stream));
    if (s->bk_order) CK(cudaMemcpyAsync(s->bk_order, s->order, n * 4, cudaMemcpyDeviceToDevice, s->stream));
    if (s->bk_types && s->types) CK(cudaMemcpyAsync(s->bk_types, s->types, n * 4, cudaMemcpyDeviceToDevice, s->stream));
    if (s->bk_mclass && s->mclass) CK(cudaMemcpyAsync(s->bk_mclass, s->mclass, n, cudaMemcpyDeviceToDevice, s->stream));
    if (s->bk_mass && s->mass) CK(cudaMemcpyAsync(s->bk_mass, s->mass, n * 8, cudaMemcpyDeviceToDevice, s->stream));
    return DP_OK;
}

static int restore_state(dp_sim* s) {
    const size_t n = (size_t)s->n, bd = n * s->dim * sizeof(double), bi = n * s->dim * sizeof(int32_t);
    CK(cudaMemcpyAsync(s->pos, s->bk_pos, bd, cudaMemcpyDeviceToDevice, s->stream));
    CK(cudaMemcpyAsync(s->vel, s->bk_vel, bd, cudaMemcpyDeviceToDevice, s->stream));
    CK(cudaMemcpyAsync(s->beta, s->bk_beta, bd, cudaMemcpyDeviceToDevice, s->stream));
    CK(cudaMemcpyAsync(s->img, s->bk_img, bi, cudaMemcpyDeviceToDevice, s->stream));
    if (s->bk_order) {
        CK(cudaMemcpyAsync(s->order, s->bk_order, n * 4, cudaMemcpyDeviceToDevice, s->stream));
        k_invert_order<<<grid_for(s->n, kBlock), kBlock, 0, s->stream>>>(s->order, s->slot_of, s->n);
        CK(cudaGetLastError());
    }
    if (s->bk_types && s->types) CK(cudaMemcpyAsync(s->types, s->bk_types, n * 4, cudaMemcpyDeviceToDevice, s->stream));
    if (s->bk_mclass && s->mclass) CK(cudaMemcpyAsync(s->mclass, s->bk_mclass, n, cudaMemcpyDeviceToDevice, s->stream));
    if (s->bk_mass && s->mass) CK(cudaMemcpyAsync(s->mass, s->bk_mass, n * 8, cudaMemcpyDeviceToDevice, s->stream));
    return launch_shadow(s);
}

static long long chunk_steps(const dp_sim* s) {
    long long c = (4LL << 20) / std::max<long long>(1, s->n);
    c = std::max<long long>(32, std::min<long long>(kMaxChunk, c));
    return c;
}

// Capture and instantiate, before any step runs, every graph a run of `steps`
// steps will launch: the groups, or the chunk lengths, each keyed by the position
// buffer set that is current when it starts (a fused chunk of odd length
// leaves the other set current). A timed run then measures launches only.
static int prepare_one(dp_sim* s, long long c, int kind, bool other_set) {
    if (other_set) swap_position_buffers(s);
    GraphEntry* g = nullptr;
    const int rc = get_graph(s, c, kind, &g);
    if (other_set) swap_position_buffers(s);
    return rc;
}

static int prepare_graphs(dp_sim* s, long long steps, int kind) {
    if (steps <= 0) return DP_OK;
    const long long chunk = chunk_steps(s);
    if (use_groups(s)) {
        // a single step runs without a graph; a chunk may leave either buffer set
        // current, so that the next can start from either
        if (steps == 1) return DP_OK;
        if (prepare_one(s, -1, kind, false) == DP_OK) return steps > chunk ? prepare_one(s, -1, kind, true) : DP_OK;
        // no conditional nodes (conditional_graphs is cleared now): chunks
    }
    const bool odd = use_fused_step(s) && (chunk & 1);  // each full chunk flips the sets
    const long long full = steps / chunk, rem = steps % chunk;
    if (full >= 1) RET(prepare_one(s, chunk, kind, false));
    if (full >= 2 && odd) RET(prepare_one(s, chunk, kind, true));
    if (rem > 0) RET(prepare_one(s, rem, kind, odd && (full & 1)));
    return DP_OK;
}

// After steps (hstat is current): what they ran into.
static int check_run_status(dp_sim* s) {
    RET(check_device_error(s));
    if (!s->hstat->nonfinite) return DP_OK;
    s->hstat->nonfinite = 0;
    RET(write_status(s));
    return fail(DP_ERR_NONFINITE, "a force or position became NaN/Inf during run()");
}

static int run_impl(dp_sim* s, long long steps, int kind, float* ms) {
    RET(require_ready(s));
    if (kind != DP_INT_GJF && kind != DP_INT_NVE) return fail(DP_ERR_ARG, "unknown integrator kind");
    if (steps < 0) return fail(DP_ERR_ARG, "steps must be >= 0");
    // make the list current (the reference checks it at the start of every step)
    RET(update_nl(s, true, nullptr));
    if (steps > 0) s->nl_checked = false;
    RET(ensure_partial(s, grid_for(s->n, kBlock)));
    if (s->precision == DP_PREC_MLP) RET(ensure_mlp_fx(s));
    s->launches_last = 0;
    RET(prepare_graphs(s, steps, kind));
    if (ms) CK(cudaEventRecord(s->ev0, s->stream));
    const long long chunk = chunk_steps(s);
    long long done = 0;
    int retries = 0;  // attempts since the last step that stands
    while (done < steps) {
        const long long c = std::min(chunk, steps - done);
        const long long step0 = s->hstat->step;  // hstat is current: every path here ends in read_status
        const long long rebuilds0 = s->hstat->rebuilds;
        // one step on a list that is valid (hstat is current): no rebuild can be due
        // before it, so it needs no graph
        if (c == 1 && use_groups(s) && !s->hstat->need_rebuild) {
            RET(launch_step(s, kind, 0, &s->launches_last, DP_END_CLEAR_FAR));
            k_advance_step<<<1, 1, 0, s->stream>>>(s->dstat, 1, 1);
            CK(cudaGetLastError());
            swap_position_buffers(s);
            s->launches_last += 1;
            done += 1;
            RET(read_status(s));
            RET(check_run_status(s));
            continue;
        }
        GraphEntry* g = nullptr;
        const bool groups = use_groups(s);
        // a chunk needs the backup only if a list build inside it can
        // overflow: at a later step, or at its first step when a rebuild is
        // pending (hstat is current here); grouped steps stop there
        const bool backed_up = !groups && !use_allpairs_step(s) && (c > 1 || s->hstat->need_rebuild != 0);
        if (backed_up) RET(backup_state(s));
        RET(get_graph(s, groups ? -1 : c, kind, &g));
        if (groups) {
            k_group_start<<<1, 1, 0, s->stream>>>(s->dstat, (int)c);
            CK(cudaGetLastError());
        }
        CK(cudaGraphLaunch(g->exec, s->stream));
        RET(read_status(s));
        // an odd number of fused steps leaves the positions in the other buffer set
        // (grouped steps: since the last rebuild)
        if (groups ? s->hstat->parity != 0 : (g->fused && (c & 1))) swap_position_buffers(s);
        if (groups && s->hstat->parity) {
            s->hstat->parity = 0;
            k_group_start<<<1, 1, 0, s->stream>>>(s->dstat, 0);
            CK(cudaGetLastError());
        }
        // a region without room leaves its brick's lists empty, and unless the steps
        // stopped there, what the chunk went on to do does not count: not even a
        // force that became infinite, or the longest row
        const bool void_chunk = !groups && s->bricks && s->hstat->cell_overflow > s->brick_cap;
        if (void_chunk) {
            s->hstat->nonfinite = 0;
            s->hstat->max_neighbors = 0;
        }
        RET(check_run_status(s));
        bool grown = false;
        RET(grow_after_overflow(s, &grown));
        if (grown) {
            const long long before = groups ? s->hstat->step - step0 : 0;  // steps that stand
            if (!groups && !backed_up) return fail(DP_ERR_OVERFLOW, "neighbour list overflow without a pending build");
            retries = before > 0 ? 0 : retries + 1;
            if (retries > 8) return fail(DP_ERR_OVERFLOW, "neighbour list keeps overflowing");
            if (!groups) {
                RET(restore_state(s));
                s->hstat->step = step0;
            }
            s->hstat->need_rebuild = 1;
            RET(write_status(s));
            if (groups)
                s->launches_last += 1 + s->hstat->groups * g->launches +
                                    (s->hstat->rebuilds - rebuilds0) * g->rebuild_launches;
            done += before;
            continue;  // the build again, and the steps from there (or all of the chunk)
        }
        s->launches_last += (groups ? 1 + s->hstat->groups * g->launches : g->launches) +
                            (s->hstat->rebuilds - rebuilds0) * g->rebuild_launches;
        done += c;
        retries = 0;
    }
    if (ms) {
        CK(cudaEventRecord(s->ev1, s->stream));
        CK(cudaEventSynchronize(s->ev1));
        CK(cudaEventElapsedTime(ms, s->ev0, s->ev1));
    }
    return DP_OK;
}

// ===========================================================================
// C ABI
// ===========================================================================
extern "C" {

const char* dp_last_error(void) { return g_err.c_str(); }

int dp_version(void) { return 100; }

int dp_create(int dim, int64_t n, int precision, dp_sim** out) {
    if (!out) return fail(DP_ERR_ARG, "out is null");
    *out = nullptr;
    if (dim < 2 || dim > 4) return fail(DP_ERR_ARG, "dimension must be 2, 3 or 4");
    if (n < 1 || n > 2147483647LL) return fail(DP_ERR_ARG, "number of particles must be in [1, 2^31)");
    if (precision != DP_PREC_FP64 && precision != DP_PREC_FP32) return fail(DP_ERR_ARG, "unknown precision");
    dp_sim* s = new dp_sim();
    s->dim = dim;
    s->n = n;
    s->precision = precision;
    // DOMPAP_CONDITIONAL_GRAPHS=0 selects the gated rebuild kernels (profilers
    // that do not follow conditional graph nodes see every launch then)
    if (const char* env = std::getenv("DOMPAP_CONDITIONAL_GRAPHS")) s->conditional_graphs = std::atoi(env) != 0;
    if (const char* env = std::getenv("DOMPAP_FUSED_STEP")) s->fused_step = std::atoi(env) != 0;
    if (const char* env = std::getenv("DOMPAP_WARP_STEP")) s->warp_step_max = std::atoll(env);
    if (const char* env = std::getenv("DOMPAP_QUAD_STEP")) s->quad_step_max = std::atoll(env);
    if (const char* env = std::getenv("DOMPAP_REORDER")) s->reorder = std::atoi(env) != 0;
    if (const char* env = std::getenv("DOMPAP_MLP_TENSOR"))
        s->mlp_tensor = std::strcmp(env, "tcgen05") == 0 ? 1 : (std::strcmp(env, "mma") == 0 ? 2 : 0);
    int rc = DP_OK;
    auto cleanup = [&]() {
        dp_destroy(s);
        return rc;
    };
    if (cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaStreamCreateWithFlags(&s->cstream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaStreamCreateWithFlags(&s->bstream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&s->ev0) != cudaSuccess || cudaEventCreate(&s->ev1) != cudaSuccess) {
        rc = fail(DP_ERR_CUDA, std::string("stream/event creation: ") + cudaGetErrorString(cudaGetLastError()));
        return cleanup();
    }
    const size_t nd = (size_t)n * dim;
    if ((rc = dalloc_t(&s->pos, nd)) || (rc = dalloc_t(&s->vel, nd)) || (rc = dalloc_t(&s->beta, nd)) ||
        (rc = dalloc_t(&s->force, nd)) || (rc = dalloc_t(&s->pos_ref, nd)) || (rc = dalloc_t(&s->img, nd)) ||
        (rc = dalloc_t(&s->bk_pos, nd)) || (rc = dalloc_t(&s->bk_vel, nd)) || (rc = dalloc_t(&s->bk_beta, nd)) ||
        (rc = dalloc_t(&s->bk_img, nd)) || (rc = dalloc_t(&s->cnt, (size_t)n)) ||
        (rc = dalloc_t(&s->order, (size_t)n)) || (rc = dalloc_t(&s->slot_of, (size_t)n)))
        return cleanup();
    k_iota<<<grid_for(n, kBlock), kBlock, 0, s->stream>>>(s->order, s->slot_of, n);  // slot = particle id
    s->shadow_bytes = (size_t)n * (dim == 2 ? 8 : 16);
    if ((rc = dalloc(&s->shadow, s->shadow_bytes)) || (rc = dalloc(&s->shadow_ref, s->shadow_bytes)) ||
        (rc = dalloc(&s->pos64, (size_t)n * (dim == 2 ? 16 : 32))) || (rc = dalloc_t(&s->pos_alt, nd)) ||
        (rc = dalloc(&s->shadow_alt, s->shadow_bytes)) || (rc = dalloc(&s->pos64_alt, (size_t)n * (dim == 2 ? 16 : 32))))
        return cleanup();
    if (cudaMemset(s->shadow, 0, s->shadow_bytes) != cudaSuccess ||
        cudaMemset(s->shadow_ref, 0, s->shadow_bytes) != cudaSuccess) {
        rc = fail(DP_ERR_CUDA, "cudaMemset failed");
        return cleanup();
    }
    if (cudaMemset(s->pos, 0, nd * 8) != cudaSuccess || cudaMemset(s->vel, 0, nd * 8) != cudaSuccess ||
        cudaMemset(s->beta, 0, nd * 8) != cudaSuccess || cudaMemset(s->force, 0, nd * 8) != cudaSuccess ||
        cudaMemset(s->pos_ref, 0, nd * 8) != cudaSuccess || cudaMemset(s->img, 0, nd * 4) != cudaSuccess ||
        cudaMemset(s->cnt, 0, (size_t)n * 4) != cudaSuccess) {
        rc = fail(DP_ERR_CUDA, "cudaMemset failed");
        return cleanup();
    }
    if (cudaMalloc(&s->dstat, sizeof(dp_dev_status)) != cudaSuccess ||
        cudaMallocHost(&s->hstat, sizeof(dp_dev_status)) != cudaSuccess ||
        cudaMalloc(&s->dsum, sizeof(double)) != cudaSuccess || cudaMallocHost(&s->hsum, sizeof(double)) != cudaSuccess) {
        rc = fail(DP_ERR_CUDA, "status allocation failed");
        return cleanup();
    }
    memset(s->hstat, 0, sizeof(dp_dev_status));
    if (cudaMemcpy(s->dstat, s->hstat, sizeof(dp_dev_status), cudaMemcpyHostToDevice) != cudaSuccess) {
        rc = fail(DP_ERR_CUDA, "status init failed");
        return cleanup();
    }
    if ((rc = upload_mass_coefficients(s))) return cleanup();
    *out = s;
    return DP_OK;
}

int dp_destroy(dp_sim* s) {
    if (!s) return DP_OK;
    if (s->stream) cudaStreamSynchronize(s->stream);
    free_graphs(s);
    void* bufs[] = {s->pos, s->vel, s->beta, s->force, s->pos_ref, s->img, s->shadow, s->shadow_ref, s->pos64,
                    s->pos_alt, s->shadow_alt, s->pos64_alt, s->mlp_fx,
                    s->ff_tab, s->f32_tab, s->bk_pos,
                    s->bk_vel, s->bk_beta, s->bk_img, s->mclass, s->mcoef, s->mcoef_f, s->class_mass_dev, s->mass, s->types,
                    s->sig_tab, s->eps_tab, s->isig_tab, s->nl, s->cnt, s->bin_cnt, s->bin_start, s->bin_part,
                    s->bin_key, s->bin_rank, s->src_of, s->order, s->slot_of, s->sc_vel, s->sc_beta, s->sc_mass,
                    s->sc_img, s->sc_order, s->sc_types, s->sc_mclass, s->bk_order, s->bk_types, s->bk_mclass,
                    s->bk_mass, s->dstat,
                    s->partial, s->dsum, s->rdf_buf, s->rdf_sel, s->brick_base, s->brick_info, s->brick_slots};
    for (void* b : bufs)
        if (b) cudaFree(b);
    if (s->hstat) cudaFreeHost(s->hstat);
    if (s->hsum) cudaFreeHost(s->hsum);
    if (s->ev0) cudaEventDestroy(s->ev0);
    if (s->ev1) cudaEventDestroy(s->ev1);
    if (s->stream) cudaStreamDestroy(s->stream);
    if (s->cstream) cudaStreamDestroy(s->cstream);
    if (s->bstream) cudaStreamDestroy(s->bstream);
    delete s;
    return DP_OK;
}

static int rebuild_pair_lib(dp_sim* s);

int dp_set_precision(dp_sim* s, int precision) {
    if (!s) return fail(DP_ERR_ARG, "null handle");
    if (precision != DP_PREC_FP64 && precision != DP_PREC_FP32 && precision != DP_PREC_MLP)
        return fail(DP_ERR_ARG, "unknown precision");
    if (precision == DP_PREC_MLP && !s->mlp_dev) return fail(DP_ERR_ARG, "no pair surrogate attached (dp_set_mlp)");
    if (precision == DP_PREC_MLP && s->pmode != DP_PAIR_CONST)
        return fail(DP_ERR_ARG, "the pair surrogate needs constant sigma = epsilon = 1");
    if (precision == DP_PREC_FP64 && s->have_box) RET(launch_shadow(s));  // refresh the 64-bit fixed point
    if (precision == s->precision) return DP_OK;
    s->precision = precision;
    if (s->have_pot) RET(rebuild_pair_lib(s));
    return DP_OK;
}

// --------------------------- state ----------------------------------------
// The device's view of a page-locked host array (cudaHostAlloc / registered),
// or nullptr for pageable memory. The transposing kernels then read or write
// the host array directly over the host link: one pass, no staging copy.
static const void* mapped_view(const void* host) {
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, host) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return attr.type == cudaMemoryTypeHost ? attr.devicePointer : nullptr;
}

// host (n, comps) in particle-id order -> device SoA in slot order; the
// caller synchronises (the host array must not change before that).
static int upload_f64_async(dp_sim* s, const double* host, double* dev_soa, int comps) {
    if (!host) return fail(DP_ERR_ARG, "null array");
    const unsigned g = grid_for(s->n * comps, kBlock);
    if (const double* view = (const double*)mapped_view(host)) {
        k_host_to_slots<double><<<g, kBlock, 0, s->stream>>>(view, dev_soa, s->slot_of, s->n, comps);
    } else {
        // stage through the backup buffer to transpose on the device
        CK(cudaMemcpyAsync(s->bk_pos, host, (size_t)s->n * comps * sizeof(double), cudaMemcpyHostToDevice,
                           s->stream));
        k_host_to_slots<double><<<g, kBlock, 0, s->stream>>>(s->bk_pos, dev_soa, s->slot_of, s->n, comps);
    }
    CK(cudaGetLastError());
    return DP_OK;
}

static int upload_aos_f64_async(dp_sim* s, const double* host, double* dev_soa) {
    return upload_f64_async(s, host, dev_soa, s->dim);
}

static int upload_aos_f64(dp_sim* s, const double* host, double* dev_soa) {
    RET(upload_aos_f64_async(s, host, dev_soa));
    CK(cudaStreamSynchronize(s->stream));
    return DP_OK;
}

// device SoA in slot order -> host (n, comps) in particle-id order; the
// caller synchronises before reading it.
static int download_f64_async(dp_sim* s, const double* dev_soa, double* host, int comps) {
    if (!host) return fail(DP_ERR_ARG, "null array");
    const unsigned g = grid_for(s->n * comps, kBlock);
    if (double* view = (double*)mapped_view(host)) {
        k_slots_to_host<double><<<g, kBlock, 0, s->stream>>>(dev_soa, view, s->slot_of, s->n, comps);
        CK(cudaGetLastError());
    } else {
        k_slots_to_host<double><<<g, kBlock, 0, s->stream>>>(dev_soa, s->bk_vel, s->slot_of, s->n, comps);
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(host, s->bk_vel, (size_t)s->n * comps * sizeof(double), cudaMemcpyDeviceToHost,
                           s->stream));
    }
    return DP_OK;
}

static int download_aos_f64_async(dp_sim* s, const double* dev_soa, double* host) {
    return download_f64_async(s, dev_soa, host, s->dim);
}

static int download_aos_f64(dp_sim* s, const double* dev_soa, double* host) {
    RET(download_aos_f64_async(s, dev_soa, host));
    CK(cudaStreamSynchronize(s->stream));
    return DP_OK;
}

// host int32 (n, comps) in id order -> device SoA in slot order, staged
// through bk_img (n * dim int32, comps <= dim).
static int upload_i32(dp_sim* s, const int32_t* host, int32_t* dev_soa, int comps) {
    const size_t bytes = (size_t)s->n * comps * sizeof(int32_t);
    CK(cudaMemcpyAsync(s->bk_img, host, bytes, cudaMemcpyHostToDevice, s->stream));
    k_host_to_slots<int32_t><<<grid_for(s->n * comps, kBlock), kBlock, 0, s->stream>>>(s->bk_img, dev_soa, s->slot_of,
                                                                                         s->n, comps);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(s->stream));
    return DP_OK;
}

int dp_set_positions(dp_sim* s, const double* p) {
    if (!s) return fail(DP_ERR_ARG, "null handle");
    s->nl_checked = false;
    RET(upload_aos_f64_async(s, p, s->pos));
    if (s->have_box) RET(launch_shadow(s));
    CK(cudaStreamSynchronize(s->stream));
    return DP_OK;
}
int dp_get_positions(dp_sim* s, double* p) {
    if (!s) return fail(DP_ERR_ARG, "null handle");
    return download_aos_f64(s, s->pos, p);
}
int dp_get_reference_positions(dp_sim* s, double* p) {
    if (!s) return fail(DP_ERR_ARG, "null handle");
    return download_aos_f64(s, s->pos_ref, p);
}
int dp_set_velocities(dp_sim* s, const double* v) {
    if (!s) return fail(DP_ERR_ARG, "null handle");
    return upload_aos_f64(s, v, s->vel);
}
int dp_get_velocities(dp_sim* s, double* v) {
    if (!s) return fail(DP_ERR_ARG, "null handle");
    return download_aos_f64(s, s->vel, v);
}
int dp_set_betas(dp_sim* s, const double* b) {
    if (!s) return fail(DP_ERR_ARG, "null handle");
    return upload_aos_f64(s, b, s->beta);
}
int dp_get_betas(dp_sim* s, double* b) {
    if (!s) return fail(DP_ERR_ARG, "null handle");
    return download_aos_f64(s, s->beta, b);
}
int dp_set_images(dp_sim* s, const int32_t* im) {
    if (!s || !im) return fail(DP_ERR_ARG, "null argument");
    return upload_i32(s, im, s->img, s->dim);
}
int dp_get_images(dp_sim* s, int32_t* im) {
    if (!s || !im) return fail(DP_ERR_ARG, "null argument");
    const size_t bytes = (size_t)s->n * s->dim * sizeof(int32_t);
    k_slots_to_host<int32_t><<<grid_for(s->n * s->dim, kBlock), kBlock, 0, s->stream>>>(s->img, s->bk_img,
                                                                                         s->slot_of, s->n, s->dim);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(im, s->bk_img, bytes, cudaMemcpyDeviceToHost, s->stream));
    CK(cudaStreamSynchronize(s->stream));
    return DP_OK;
}

int dp_set_masses(dp_sim* s, const double* m) {
    if (!s || !m) return fail(DP_ERR_ARG, "null argument");
    std::map<double, int> classes;
    for (long long i = 0; i < s->n && classes.size() <= 256; ++i) classes.emplace(m[i], 0);
    if (classes.size() == 1) {
        s->mass_mode = 0;
        s->class_mass.assign(1, m[0]);
    } else if (classes.size() <= 256) {
        s->mass_mode = 1;
        s->class_mass.clear();
        int c = 0;
        for (auto& kv : classes) {
            kv.second = c++;
            s->class_mass.push_back(kv.first);
        }
        std::vector<uint8_t> cls((size_t)s->n);
        for (long long i = 0; i < s->n; ++i) cls[i] = (uint8_t)classes[m[i]];
        if (!s->mclass) RET(dalloc_t(&s->mclass, (size_t)s->n));
        // by particle id into the slot order (staged through bk_img)
        CK(cudaMemcpyAsync(s->bk_img, cls.data(), (size_t)s->n, cudaMemcpyHostToDevice, s->stream));
        k_host_to_slots<uint8_t><<<grid_for(s->n, kBlock), kBlock, 0, s->stream>>>(
            (const uint8_t*)s->bk_img, s->mclass, s->slot_of, s->n, 1);
        CK(cudaGetLastError());
        CK(cudaStreamSynchronize(s->stream));
    } else {
        s->mass_mode = 2;
        s->class_mass.assign(1, m[0]);
        if (!s->mass) RET(dalloc_t(&s->mass, (size_t)s->n));
        RET(upload_f64_async(s, m, s->mass, 1));
        CK(cudaStreamSynchronize(s->stream));
    }
    if (s->mass_mode == 2) {
        // the reduction kernels read per-particle masses
        RET(dalloc_t(&s->class_mass_dev, 1));
        CK(cudaMemcpy(s->class_mass_dev, s->class_mass.data(), sizeof(double), cudaMemcpyHostToDevice));
    }
    return upload_mass_coefficients(s);
}

int dp_set_types(dp_sim* s, const int32_t* t) {
    if (!s || !t) return fail(DP_ERR_ARG, "null argument");
    int lo = t[0], hi = t[0];
    for (long long i = 1; i < s->n; ++i) {
        lo = std::min(lo, (int)t[i]);
        hi = std::max(hi, (int)t[i]);
    }
    if (lo < 0) return fail(DP_ERR_ARG, "particle types must be >= 0");
    if (s->pmode == DP_PAIR_TYPES && hi >= s->ntypes)
        return fail(DP_ERR_ARG, "a particle type exceeds the per-type parameter table");
    s->min_type = lo;
    s->max_type = hi;
    if (!s->types) RET(dalloc_t(&s->types, (size_t)s->n));
    RET(upload_i32(s, t, s->types, 1));
    s->have_types = true;
    s->version++;
    return DP_OK;
}

int dp_set_box(dp_sim* s, const double* box) {
    if (!s || !box) return fail(DP_ERR_ARG, "null argument");
    for (int k = 0; k < s->dim; ++k) {
        if (!(box[k] > 0.0) || !std::isfinite(box[k])) return fail(DP_ERR_ARG, "box sides must be positive and finite");
        s->box[k] = box[k];
    }
    s->have_box = true;
    s->nl_config_dirty = true;
    s->version++;
    return launch_shadow(s);
}

// --------------------------- potential ------------------------------------
static std::string hexd(double v) {
    if (std::isinf(v)) return v > 0 ? "(1.0/0.0)" : "(-1.0/0.0)";
    char buf[64];
    snprintf(buf, sizeof(buf), "%a", v);
    return buf;
}

// What a warp pays for the force of a generated potential, by the calls and
// divisions in dp_pair_f: 1 for those of a few instructions (exp, log, sqrt, a
// division), 2 for the hyperbolic ones and cbrt, 4 for those with long or
// branching code (sin, cos, pow, erf and anything else).
static int pair_cost(const std::string& src) {
    size_t at = src.find("dp_pair_f(");
    at = at == std::string::npos ? at : src.find('{', at);
    if (at == std::string::npos) return 0;
    static const char* const free_of_charge[] = {"R", "dp_k", "dp_ipow", "fabs", "fmin", "fmax", "floor", "ceil", "const",
                                                 "return", "if"};
    static const char* const cheap[] = {"exp", "exp2", "expm1", "log", "log2", "log1p", "sqrt", "rsqrt"};
    static const char* const fair[] = {"tanh", "sinh", "cosh", "cbrt"};
    auto in = [](const std::string& name, const char* const* list, size_t m) {
        for (size_t k = 0; k < m; ++k)
            if (name == list[k]) return true;
        return false;
    };
    int cost = 0, depth = 0;
    for (; at < src.size(); ++at) {
        const char ch = src[at];
        if (ch == '{') ++depth;
        if (ch == '}' && --depth == 0) break;
        if (ch == '/') cost += 1;
        if (!std::isalpha((unsigned char)ch) && ch != '_') {
            // a number: none of its letters is a name
            if (std::isdigit((unsigned char)ch))
                while (at + 1 < src.size() && (std::isalnum((unsigned char)src[at + 1]) || src[at + 1] == '.')) ++at;
            continue;
        }
        size_t end = at;
        while (end < src.size() && (std::isalnum((unsigned char)src[end]) || src[end] == '_')) ++end;
        const std::string name = src.substr(at, end - at);
        at = end - 1;
        if (end >= src.size() || src[end] != '(') continue;  // (the templates' names end in '>')
        if (in(name, free_of_charge, sizeof(free_of_charge) / sizeof(char*))) continue;
        cost += in(name, cheap, sizeof(cheap) / sizeof(char*)) ? 1 : (in(name, fair, sizeof(fair) / sizeof(char*)) ? 2 : 4);
    }
    return cost;
}

// The program has the brick kernels: not for costly potentials. The one pass of
// the brick loop evaluates the force for every listed entry of a warp with a pair
// inside the cut (two in three listed ones, in eight copies of its code); the two passes over
// lists of slots only for kept ones, in one copy. us a step, 108,000 / 1,048,576
// particles, bricks against slots: LJ 73 / 373 against 91 / 591, three exp (3) 91 /
// 566 against 99 / 654, pow (4) 119 / 629 against 109 / 714, two pow (8) 145 against
// 121, LJ + exp (cos + sin) (9) 131 / 852 against 119 / 777, the costly test potential
// with eight more such terms 956 / 6,053 against 318 / 2,476. (Two passes on the bricks
// lost to slots everywhere: 459 / 2,692 on the last, 98 / 619 on LJ.)
constexpr int kCostlyPair = 6;

static bool brick_program(int dim, int precision, int pmode, const std::string& pot_src) {
    return dim <= 3 && precision == DP_PREC_FP32 && pmode != DP_PAIR_DENSE && pair_cost(pot_src) < kCostlyPair;
}

// The generated functions of a costly potential as calls: in float32 their code,
// once in every kernel that evaluates pairs and eight times in an unrolled loop, outgrows the
// registers of the loop around it and the instruction caches. us a step, inlined
// and called, costly test potential with 0 / 1 / 8 / 16 more terms, 1,048,576
// particles: 656 / 851 / 2,294 / 4,746 and 620 / 795 / 1,980 / 4,271; 512
// replicas of 2,048, 0 / 4 / 8 more: 1,981 / 4,351 / 17,390 and 841 / 1,959 / 3,311.
// (Cheap ones stay inline: 512 replicas of a Gaussian on LJ 489 against 500.)
static std::string called_pair_functions(std::string src) {
    const std::string was = "__forceinline__ R dp_pair_", now = "__noinline__ R dp_pair_";
    for (size_t at = 0; (at = src.find(was, at)) != std::string::npos; at += now.size()) src.replace(at, was.size(), now);
    return src;
}

// The kernels a program has besides those of any size, and the CTAs per SM that the
// steps are compiled for (0: without that kernel). A program with all of them takes
// NVRTC twice as long as the part a system of one size uses (Lennard-Jones 3.9 s against
// 1.9, the costly test potential with 32 more terms 42.7 against 9).
struct ProgramParts {
    int step_blocks = 6, brick_blocks = 4, lists_blocks = 4;
    bool warp_sums = true, quad_sums = true;
};

static std::string pair_program(int dim, int precision, int pmode, bool sig_one, bool eps_one,
                                const std::string& pot_src, bool with_batch, const ProgramParts& parts) {
    std::string src;
    src += "#define DP_LISTS_BLOCKS " + std::to_string(parts.lists_blocks) + "\n";
    src += std::string("#define DP_WARP_SUMS ") + (parts.warp_sums ? "1" : "0") + "\n";
    src += std::string("#define DP_QUAD_SUMS ") + (parts.quad_sums ? "1" : "0") + "\n";
    src += "#define DP_DIM " + std::to_string(dim) + "\n";
    if (precision == DP_PREC_MLP) src += "#define DP_MLP 1\n";
    if (precision == DP_PREC_FP64) src += "#define DP_FF 1\n";
    if (precision == DP_PREC_FP32 || precision == DP_PREC_MLP) {
        src += "#define DP_REAL float\n#define DP_REAL_IS_FLOAT 1\n";
    } else {
        src += "#define DP_REAL double\n#define DP_REAL_IS_FLOAT 0\n";
    }
    src += "#define DP_PMODE " + std::to_string(pmode) + "\n";
    src += std::string("#define DP_SIGMA_ONE ") + (sig_one ? "1" : "0") + "\n";
    src += std::string("#define DP_EPS_ONE ") + (eps_one ? "1" : "0") + "\n";
    // resident 256-thread CTAs per SM the fused step kernel is compiled for
    // (register cap 65536 / (256 n)); DOMPAP_STEP_MIN_BLOCKS overrides
    int step_blocks = parts.step_blocks;
    if (const char* env = std::getenv("DOMPAP_STEP_MIN_BLOCKS")) step_blocks = std::atoi(env);
    src += "#define DP_STEP_MIN_BLOCKS " + std::to_string(std::max(0, std::min(8, step_blocks))) + "\n";
    src += dp_src_common;
    src += dp_src_integrate;
    if (precision == DP_PREC_MLP) src += dp_src_mlp;
    if (precision == DP_PREC_MLP) src += dp_src_umma;
    if (precision == DP_PREC_FP64) src += dp_src_ff;
    src += "\n// ---- generated pair potential ----\n";
    src += precision == DP_PREC_FP32 && pair_cost(pot_src) >= kCostlyPair ? called_pair_functions(pot_src) : pot_src;
    src += "\n// ---- pair kernels ----\n";
    src += dp_src_pair;
    if (parts.brick_blocks > 0 && brick_program(dim, precision, pmode, pot_src)) {
        src += "\n#define DP_BRICKS 1\n#define DP_BRICK_BLOCKS " + std::to_string(parts.brick_blocks) + "\n";
        src += dp_src_brick;
    }
    if (with_batch) {
        src += "\n// ---- batched replicas ----\n";
        src += dp_src_batch;
    }
    return src;
}

// Resident 256-thread CTAs per SM the fused step kernel is compiled for
// (measured on GB300 against 4, 5, 6, 7 and 8): 4 (64 registers) for the
// double-float pair loop in 3 and 4 dimensions, whose pair terms spill under
// a tighter cap (1M LJ particles: 0.99 ms per step against 1.10 with 6; 1M
// harmonic: 3 % faster) and for per-type or per-pair tables (~600 bytes of
// spills under 40 registers; the Wahnstrom mixture ran 17 % slower with 6);
// 6 (40 registers) for the float32 pair loop and in 2 dimensions, where the
// occupancy is worth more (7-8 % faster than with 4), up to costs where it is the
// pair terms' registers that count (the costly test potential with 1 / 8 more terms:
// 6 CTAs 795 / 2,099, 4 CTAs 858 / 1,980).
constexpr int kStepCost = 40;
static int step_blocks_for(int dim, int precision, int pmode, int cost) {
    if (pmode != DP_PAIR_CONST || (precision == DP_PREC_FP32 && cost >= kStepCost)) return 4;
    return precision == DP_PREC_FP64 && dim >= 3 ? 4 : 6;
}

// The same for the brick step: 6 (40 registers, some spills) where a system has
// CTAs for them, 4 below (500,000 LJ particles: 104 us a step against 115;
// 108,000: 30.8 against 28.8).
static int brick_blocks_for(long long n) { return n >= 200000 ? 6 : 4; }

// And for the step that keeps its own lists: 2 (no spills) where its warps do
// not fill the GPU, 4 above (2,048 LJ particles: 15.6 us a step against 20.1;
// 4,000: 28.3 against 22.9).
static int lists_blocks_for(long long n) { return n < 3072 ? 2 : 4; }

static int rebuild_pair_lib(dp_sim* s) {
    const bool sig_one = s->pmode == DP_PAIR_CONST && s->sigma == 1.0;
    const bool eps_one = s->pmode == DP_PAIR_CONST && s->epsilon == 1.0;
    // by the sizes at which sum_lanes, list_kind and step_lanes choose them
    const bool small = s->n <= s->warp_step_max;
    ProgramParts parts;
    parts.step_blocks = s->step_blocks ? s->step_blocks
                                       : step_blocks_for(s->dim, s->precision, s->pmode, pair_cost(s->pot_src));
    parts.brick_blocks = small ? 0 : (s->step_blocks ? s->step_blocks : brick_blocks_for(s->n));
    parts.lists_blocks = !small ? 0 : (s->step_blocks ? s->step_blocks : lists_blocks_for(s->n));
    parts.warp_sums = small;
    parts.quad_sums = !small && s->n <= s->quad_step_max;
    const std::string src =
        pair_program(s->dim, s->precision, s->pmode, sig_one, eps_one, s->pot_src, false, parts);
    PairLib pl;
    RET(compile_pair_lib(src, &pl));
    s->lib = pl;
    s->lib_valid = true;
    s->version++;
    return DP_OK;
}

int dp_set_pair_methods(dp_sim* s, int force_method, int energy_method) {
    if (!s) return fail(DP_ERR_ARG, "null handle");
    if (force_method < DP_METHOD_LIST || force_method > DP_METHOD_ALLPAIRS_NEWTON)
        return fail(DP_ERR_ARG, "unknown force method");
    if (energy_method != DP_METHOD_LIST && energy_method != DP_METHOD_ALLPAIRS)
        return fail(DP_ERR_ARG, "unknown energy method");
    if (force_method != s->force_method || energy_method != s->energy_method) {
        s->force_method = force_method;
        s->energy_method = energy_method;
        s->version++;
    }
    return DP_OK;
}

int dp_set_step_launch(dp_sim* s, int lanes, int blocks_per_sm) {
    if (!s) return fail(DP_ERR_ARG, "null handle");
    if (lanes != 0 && lanes != 1 && lanes != 4 && lanes != 32) return fail(DP_ERR_ARG, "lanes must be 0, 1, 4 or 32");
    if (blocks_per_sm < 0 || blocks_per_sm > 8) return fail(DP_ERR_ARG, "blocks_per_sm must be in [0, 8]");
    if (lanes != s->step_lanes) {
        s->step_lanes = lanes;
        s->version++;
    }
    if (blocks_per_sm != s->step_blocks) {
        s->step_blocks = blocks_per_sm;
        if (s->have_pot) RET(rebuild_pair_lib(s));
    }
    return DP_OK;
}

int dp_get_step_launch(dp_sim* s, int* lanes, int* blocks_per_sm) {
    if (!s || !lanes || !blocks_per_sm) return fail(DP_ERR_ARG, "null argument");
    const bool brick = list_kind(s) == kListBrick;
    *lanes = s->step_lanes ? s->step_lanes
             : brick       ? s->brick_lanes
                           : step_lanes(s);
    *blocks_per_sm = s->step_blocks ? s->step_blocks
                     : brick        ? brick_blocks_for(s->n)
                                    : step_blocks_for(s->dim, s->precision, s->pmode, pair_cost(s->pot_src));
    return DP_OK;
}

int dp_set_potential(dp_sim* s, const char* device_source, double r_cut) {
    if (!s || !device_source) return fail(DP_ERR_ARG, "null argument");
    if (!(r_cut > 0.0)) return fail(DP_ERR_ARG, "r_cut must be positive");
    s->pot_src = device_source;
    s->r_cut = r_cut;
    s->have_pot = true;
    s->lib_valid = false;
    RET(rebuild_pair_lib(s));
    s->nl_config_dirty = true;
    return DP_OK;
}

int dp_set_pair_params(dp_sim* s, int mode, int ntypes, const double* sigma, const double* epsilon) {
    if (!s || !sigma || !epsilon) return fail(DP_ERR_ARG, "null argument");
    double smax = 0.0;
    if (mode == DP_PAIR_CONST) {
        s->sigma = sigma[0];
        s->epsilon = epsilon[0];
        smax = sigma[0];
        s->ntypes = 1;
    } else if (mode == DP_PAIR_TYPES) {
        if (ntypes < 1 || ntypes > 4096) return fail(DP_ERR_ARG, "ntypes must be in [1, 4096]");
        if (!s->have_types) return fail(DP_ERR_ARG, "per-type parameters need particle types (dp_set_types)");
        if (s->max_type >= ntypes) return fail(DP_ERR_ARG, "a particle type exceeds the per-type parameter table");
        const size_t m = (size_t)ntypes * ntypes;
        for (size_t t = 0; t < m; ++t) smax = std::max(smax, sigma[t]);
        std::vector<double> inv(m);
        for (size_t t = 0; t < m; ++t) inv[t] = 1.0 / sigma[t];
        RET(dalloc_t(&s->sig_tab, m));
        RET(dalloc_t(&s->eps_tab, m));
        RET(dalloc_t(&s->isig_tab, m));
        CK(cudaMemcpy(s->sig_tab, sigma, m * sizeof(double), cudaMemcpyHostToDevice));
        CK(cudaMemcpy(s->eps_tab, epsilon, m * sizeof(double), cudaMemcpyHostToDevice));
        CK(cudaMemcpy(s->isig_tab, inv.data(), m * sizeof(double), cudaMemcpyHostToDevice));
        std::vector<float2> ff(DP_FF_PARAMS * m);
        std::vector<float4> f32(m);
        for (size_t t = 0; t < m; ++t) {
            double c[DP_FF_PARAMS];
            pair_consts(sigma[t], epsilon[t], c);
            for (int q = 0; q < DP_FF_PARAMS; ++q) ff[DP_FF_PARAMS * t + q] = split_ff(c[q]);
            f32[t] = pair_consts_f32(c);
        }
        RET(dalloc_t(&s->ff_tab, ff.size()));
        CK(cudaMemcpy(s->ff_tab, ff.data(), ff.size() * sizeof(float2), cudaMemcpyHostToDevice));
        RET(dalloc_t(&s->f32_tab, f32.size()));
        CK(cudaMemcpy(s->f32_tab, f32.data(), f32.size() * sizeof(float4), cudaMemcpyHostToDevice));
        s->ntypes = ntypes;
    } else if (mode == DP_PAIR_DENSE) {
        const size_t m = (size_t)s->n * s->n;
        for (size_t t = 0; t < m; ++t) smax = std::max(smax, sigma[t]);
        RET(dalloc_t(&s->sig_tab, m));
        RET(dalloc_t(&s->eps_tab, m));
        CK(cudaMemcpy(s->sig_tab, sigma, m * sizeof(double), cudaMemcpyHostToDevice));
        CK(cudaMemcpy(s->eps_tab, epsilon, m * sizeof(double), cudaMemcpyHostToDevice));
        s->ntypes = 1;
    } else {
        return fail(DP_ERR_ARG, "unknown pair-parameter mode");
    }
    if (!(smax > 0.0)) return fail(DP_ERR_ARG, "the largest sigma must be positive");
    s->pmode = mode;
    s->sig_max = smax;  // largest sigma (dompap/Simulation.py:346-351)
    s->nl_config_dirty = true;
    s->version++;
    if (s->have_pot) RET(rebuild_pair_lib(s));
    return DP_OK;
}

int dp_set_neighbor_list(dp_sim* s, double skin, int max_neighbors, int method) {
    if (!s) return fail(DP_ERR_ARG, "null handle");
    if (!(skin >= 0.0)) return fail(DP_ERR_ARG, "skin must be >= 0");
    if (max_neighbors < 1) return fail(DP_ERR_ARG, "max_number_of_neighbors must be >= 1");
    if (method != DP_NL_CELL && method != DP_NL_ALLPAIRS) return fail(DP_ERR_ARG, "unknown neighbour-list method");
    s->skin = skin;
    s->kcap = max_neighbors;
    s->method = method;
    s->nl_config_dirty = true;
    s->version++;
    return DP_OK;
}

int dp_update_neighbor_list(dp_sim* s, int check, int* rebuilt) {
    RET(require_ready(s));
    return update_nl(s, check != 0, rebuilt);
}

int dp_get_neighbor_list(dp_sim* s, int32_t* out, int kmax, int32_t* max_count) {
    RET(require_ready(s));
    if (!out || kmax < 1) return fail(DP_ERR_ARG, "bad output");
    RET(update_nl(s, true, nullptr));
    const unsigned g = grid_for(s->n, kBlock);
    const int32_t* rows = s->nl;
    const int32_t* counts = s->cnt;
    int32_t* full = nullptr;  // half and brick lists: the full list of slots, unsorted, column-major
    int32_t* fcnt = nullptr;  // its counts (n) and their maximum
    int32_t fmax = s->hstat->max_neighbors;
    cudaError_t e = cudaSuccess;
    if (s->nl_kind == kListBrick) {
        if (dalloc_t(&full, (size_t)s->n * std::max(fmax, 1)) != DP_OK) e = cudaErrorMemoryAllocation;
        if (e == cudaSuccess) {
            k_brick_expand<<<s->nbricks, kBlock, 0, s->stream>>>(s->brick_info, s->brick_slots, s->brick_cap,
                                                                (const uint16_t*)s->nl, s->cnt, full, s->n);
            e = cudaGetLastError();
        }
        rows = full;
    } else if (s->nl_kind == kListHalf) {
        // the reference's list is the full one (every partner of every particle)
        RET(dalloc_t(&fcnt, (size_t)s->n + 1));
        e = cudaMemsetAsync(fcnt, 0, ((size_t)s->n + 1) * sizeof(int32_t), s->stream);
        if (e == cudaSuccess) {
            k_nl_half_count<<<g, kBlock, 0, s->stream>>>(s->nl, s->cnt, fcnt, fcnt + s->n, s->n);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(&fmax, fcnt + s->n, sizeof(int32_t), cudaMemcpyDeviceToHost, s->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
        if (e == cudaSuccess && dalloc_t(&full, (size_t)s->n * std::max(fmax, 1)) != DP_OK)
            e = cudaErrorMemoryAllocation;
        if (e == cudaSuccess) e = cudaMemsetAsync(fcnt, 0, (size_t)s->n * sizeof(int32_t), s->stream);
        if (e == cudaSuccess) {
            k_nl_half_scatter<<<g, kBlock, 0, s->stream>>>(s->nl, s->cnt, fcnt, full, s->n);
            e = cudaGetLastError();
        }
        rows = full;
        counts = fcnt;
    }
    int32_t* dout = nullptr;
    if (e == cudaSuccess && dalloc_t(&dout, (size_t)s->n * kmax) != DP_OK) e = cudaErrorMemoryAllocation;
    if (e == cudaSuccess) {
        const bool by_rows = s->nl_kind == kListRows;
        k_nl_export<<<g, kBlock, 0, s->stream>>>(rows, counts, dout, s->order, s->slot_of, s->n,
                                                by_rows ? 1 : s->n, by_rows ? s->kcap : 1, kmax);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(out, dout, (size_t)s->n * kmax * sizeof(int32_t), cudaMemcpyDeviceToHost, s->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
    cudaFree(dout);
    cudaFree(full);
    cudaFree(fcnt);
    if (e != cudaSuccess) return fail(DP_ERR_CUDA, std::string("neighbour-list export: ") + cudaGetErrorString(e));
    if (max_count) *max_count = fmax;
    return DP_OK;
}

int dp_set_integrator(dp_sim* s, double time_step, double temperature, double damping_time, uint64_t seed) {
    if (!s) return fail(DP_ERR_ARG, "null handle");
    s->dt = time_step;
    s->temperature = temperature;
    s->tau = damping_time;
    s->seed = seed;
    s->version++;
    return upload_mass_coefficients(s);
}

int dp_run(dp_sim* s, int64_t steps, int kind) { return run_impl(s, steps, kind, nullptr); }

int dp_selftest_bounded_wait(dp_sim* s, int32_t limit) {
    if (!s) return fail(DP_ERR_ARG, "null handle");
    if (limit < 1 || limit > (1 << 20)) return fail(DP_ERR_ARG, "limit must be in [1, 2^20]");
    k_selftest_bounded_wait<<<1, 128, 0, s->stream>>>(s->dstat, limit);
    CK(cudaGetLastError());
    RET(read_status(s));
    return check_device_error(s);
}

int dp_run_timed(dp_sim* s, int64_t steps, int kind, float* ms) {
    if (!ms) return fail(DP_ERR_ARG, "ms is null");
    return run_impl(s, steps, kind, ms);
}

int dp_run_host(dp_sim* s, const double* positions, const double* velocities, const double* betas, int64_t steps,
                int kind, double* positions_out, double* velocities_out, double* betas_out) {
    RET(require_ready(s));
    // uploads, run and downloads are ordered on the stream; the host waits
    // inside run() (its status reads) and once after the downloads
    if (positions) {
        RET(upload_aos_f64_async(s, positions, s->pos));
        RET(launch_shadow(s));
    }
    if (velocities) RET(upload_aos_f64_async(s, velocities, s->vel));
    if (betas) RET(upload_aos_f64_async(s, betas, s->beta));
    RET(run_impl(s, steps, kind, nullptr));
    if (positions_out) RET(download_aos_f64_async(s, s->pos, positions_out));
    if (velocities_out) RET(download_aos_f64_async(s, s->vel, velocities_out));
    if (betas_out) RET(download_aos_f64_async(s, s->beta, betas_out));
    CK(cudaStreamSynchronize(s->stream));
    return DP_OK;
}

// --------------------------- observables ----------------------------------
int dp_forces(dp_sim* s, double* forces) {
    RET(require_ready(s));
    RET(update_nl(s, true, nullptr));
    if (!forces) return fail(DP_ERR_ARG, "null array");
    RET(launch_pair(s, s->lib.forces, s->force, nullptr));
    if (s->precision == DP_PREC_MLP) {  // results of a wait that gave up are not handed over
        RET(read_status(s));
        RET(check_device_error(s));
    }
    RET(download_aos_f64_async(s, s->force, forces));
    RET(read_status(s));
    if (s->hstat->nonfinite) {
        s->hstat->nonfinite = 0;
        RET(write_status(s));
    }
    return DP_OK;
}

static int scalar_pair(dp_sim* s, cudaKernel_t k, double* out) {
    RET(require_ready(s));
    if (!out) return fail(DP_ERR_ARG, "null output");
    RET(update_nl(s, true, nullptr));
    // one partial sum per block of the kernel launch_pair uses
    const bool tc = s->precision == DP_PREC_MLP && use_mlp_tcgen05(s);
    const bool all = k == s->lib.energy && s->energy_method != DP_METHOD_LIST && s->lib.energy_all;
    const long long blocks = all ? grid_for(s->n * 32, kBlock)
                                 : (list_kind(s) == kListBrick ? s->nbricks
                                                                : grid_for(tc ? s->n : s->n * sum_lanes(s), tc ? 128 : kBlock));
    RET(ensure_partial(s, blocks));
    RET(launch_pair(s, k, nullptr, nullptr));
    k_reduce<<<1, 1024, 0, s->stream>>>(s->partial, blocks, s->dsum);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(s->hsum, s->dsum, sizeof(double), cudaMemcpyDeviceToHost, s->stream));
    CK(cudaStreamSynchronize(s->stream));
    *out = *s->hsum;
    if (tc) {
        RET(read_status(s));
        RET(check_device_error(s));
    }
    return DP_OK;
}

int dp_potential_energy(dp_sim* s, double* energy) {
    double e = 0.0;
    RET(scalar_pair(s, s ? s->lib.energy : nullptr, &e));
    // the list kernel sums every pair twice (dompap/potential.py:69-100 halves
    // it); the double-loop kernel sums each pair once (:103-160)
    const bool all = s->energy_method != DP_METHOD_LIST && s->lib.energy_all;
    *energy = all ? e : e / 2;
    return DP_OK;
}

int dp_virial(dp_sim* s, double* virial) {
    double w = 0.0;
    RET(scalar_pair(s, s ? s->lib.virial : nullptr, &w));
    *virial = w / s->dim;
    return DP_OK;
}

int dp_laplacian(dp_sim* s, double* lap) {
    RET(require_ready(s));
    if (!lap) return fail(DP_ERR_ARG, "null output");
    RET(update_nl(s, true, nullptr));
    RET(launch_pair(s, s->lib.laplacian, s->bk_beta, nullptr));
    RET(download_f64_async(s, s->bk_beta, lap, 1));
    CK(cudaStreamSynchronize(s->stream));
    return DP_OK;
}

int dp_sum_mv2(dp_sim* s, double* out) {
    if (!s || !out) return fail(DP_ERR_ARG, "null argument");
    const long long blocks = grid_for(s->n, kBlock);
    RET(ensure_partial(s, blocks));
    dp_int_args a;
    fill_int_args(s, a, 0);
    const unsigned g = (unsigned)blocks;
#define DP_MV2(D)                                                                                               \
    switch (s->mass_mode) {                                                                                     \
        case 0: k_sum_mv2<D, 0><<<g, kBlock, 0, s->stream>>>(a, s->class_mass_dev, s->partial); break;          \
        case 1: k_sum_mv2<D, 1><<<g, kBlock, 0, s->stream>>>(a, s->class_mass_dev, s->partial); break;          \
        default: k_sum_mv2<D, 2><<<g, kBlock, 0, s->stream>>>(a, s->class_mass_dev, s->partial); break;         \
    }
    switch (s->dim) {
        case 2: DP_MV2(2); break;
        case 3: DP_MV2(3); break;
        default: DP_MV2(4); break;
    }
#undef DP_MV2
    k_reduce<<<1, 1024, 0, s->stream>>>(s->partial, blocks, s->dsum);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(s->hsum, s->dsum, sizeof(double), cudaMemcpyDeviceToHost, s->stream));
    CK(cudaStreamSynchronize(s->stream));
    *out = *s->hsum;
    return DP_OK;
}

int dp_eval_potential(dp_sim* s, const double* sv, int64_t n, double* u, double* f, double* c) {
    if (!s || !sv || !u || !f || !c) return fail(DP_ERR_ARG, "null argument");
    if (!s->have_pot || !s->lib_valid) return fail(DP_ERR_NOPOT, "no pair potential set");
    if (n <= 0) return DP_OK;
    double* buf = nullptr;
    RET(dalloc_t(&buf, (size_t)n * 4));
    const size_t b = (size_t)n * sizeof(double);
    cudaError_t e = cudaMemcpyAsync(buf, sv, b, cudaMemcpyHostToDevice, s->stream);
    double* du = buf + n;
    double* df = buf + 2 * n;
    double* dc = buf + 3 * n;
    long long nn = n;
    double rc = s->r_cut;
    void* args[] = {&buf, &du, &df, &dc, &nn, &rc};
    if (e == cudaSuccess)
        e = cudaLaunchKernel((const void*)s->lib.eval, dim3(grid_for(n, kBlock)), dim3(kBlock), args, 0, s->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(u, du, b, cudaMemcpyDeviceToHost, s->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(f, df, b, cudaMemcpyDeviceToHost, s->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(c, dc, b, cudaMemcpyDeviceToHost, s->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
    cudaFree(buf);
    if (e != cudaSuccess) return fail(DP_ERR_CUDA, std::string("dp_eval_potential: ") + cudaGetErrorString(e));
    return DP_OK;
}

int dp_get_normals(dp_sim* s, int64_t step, double* out) {
    if (!s || !out) return fail(DP_ERR_ARG, "null argument");
    const unsigned g = grid_for(s->n, kBlock);
    switch (s->dim) {
        case 2: k_normals<2><<<g, kBlock, 0, s->stream>>>(s->seed, step, s->bk_vel, s->n); break;
        case 3: k_normals<3><<<g, kBlock, 0, s->stream>>>(s->seed, step, s->bk_vel, s->n); break;
        default: k_normals<4><<<g, kBlock, 0, s->stream>>>(s->seed, step, s->bk_vel, s->n); break;
    }
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(out, s->bk_vel, (size_t)s->n * s->dim * sizeof(double), cudaMemcpyDeviceToHost, s->stream));
    CK(cudaStreamSynchronize(s->stream));
    return DP_OK;
}

int dp_get_stats(dp_sim* s, dp_stats* st) {
    if (!s || !st) return fail(DP_ERR_ARG, "null argument");
    RET(read_status(s));
    memset(st, 0, sizeof(*st));
    st->steps = s->hstat->step;
    st->rebuilds = s->hstat->rebuilds;
    st->max_neighbors = s->hstat->max_neighbors;
    st->neighbor_capacity = s->kcap;
    for (int k = 0; k < 4; ++k) st->cells[k] = s->use_cells ? s->nc[k] : 0;
    st->cell_capacity = 0;  // cells are contiguous slot ranges: no capacity
    st->method_used = s->use_cells ? DP_NL_CELL : DP_NL_ALLPAIRS;
    st->nl_cutoff = s->cutoff;
    st->conditional_graphs = s->conditional_graphs && !use_own_lists(s) ? 1 : 0;
    return DP_OK;
}

int dp_time_kernel(dp_sim* s, int which, int reps, float* ms) {
    RET(require_ready(s));
    if (!ms || reps < 1) return fail(DP_ERR_ARG, "bad arguments");
    RET(update_nl(s, true, nullptr));
    RET(ensure_partial(s, grid_for(s->n, kBlock)));
    auto once = [&]() -> int {
        switch (which) {
            case DP_KERNEL_FORCES: return launch_pair(s, s->lib.forces, s->force, nullptr);
            case DP_KERNEL_GJF: return launch_integrate(s, DP_INT_GJF, 0, nullptr);
            case DP_KERNEL_NVE: return launch_integrate(s, DP_INT_NVE, 0, nullptr);
            case DP_KERNEL_REBUILD:
                k_set_rebuild<<<1, 1, 0, s->stream>>>(s->dstat);
                return launch_rebuild(s, nullptr);
            case DP_KERNEL_SKIN: return launch_skin_check(s);
            case DP_KERNEL_STEP:
                if (!use_fused_step(s)) return fail(DP_ERR_ARG, "no fused step kernel in this mode");
                // as run() launches it (`far` stays as it is: the positions are not advanced)
                return launch_step(s, DP_INT_GJF, 0, nullptr, use_own_lists(s) ? DP_END_OWN_LISTS : 0);
            default: return fail(DP_ERR_ARG, "unknown kernel");
        }
    };
    const bool moves = which == DP_KERNEL_GJF || which == DP_KERNEL_NVE || which == DP_KERNEL_STEP;
    s->nl_checked = false;
    if (moves) RET(backup_state(s));
    RET(once());  // warm-up
    CK(cudaEventRecord(s->ev0, s->stream));
    for (int r = 0; r < reps; ++r) RET(once());
    CK(cudaEventRecord(s->ev1, s->stream));
    CK(cudaEventSynchronize(s->ev1));
    float t = 0.0f;
    CK(cudaEventElapsedTime(&t, s->ev0, s->ev1));
    *ms = t / reps;
    // the integrator kernels moved the particles: put the state back and
    // leave a consistent list behind
    if (moves) RET(restore_state(s));
    RET(read_status(s));
    s->hstat->need_rebuild = 1;
    RET(write_status(s));
    RET(update_nl(s, true, nullptr));
    return DP_OK;
}


int dp_wrap(dp_sim* s) {
    if (!s) return fail(DP_ERR_ARG, "null handle");
    if (!s->have_box) return fail(DP_ERR_ARG, "box not set");
    dp_int_args a;
    fill_int_args(s, a, 0);
    s->nl_checked = false;
    const unsigned g = grid_for(s->n, kBlock);
    switch (s->dim) {
        case 2: k_wrap<2><<<g, kBlock, 0, s->stream>>>(a); break;
        case 3: k_wrap<3><<<g, kBlock, 0, s->stream>>>(a); break;
        default: k_wrap<4><<<g, kBlock, 0, s->stream>>>(a); break;
    }
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(s->stream));
    return DP_OK;
}

int dp_rdf_counts(dp_sim* s, int type_a, int type_b, const double* edges, int nbins, uint64_t* counts) {
    if (!s || !edges || !counts) return fail(DP_ERR_ARG, "null argument");
    if (!s->have_box) return fail(DP_ERR_ARG, "box not set");
    if (nbins < 1 || nbins > 8192) return fail(DP_ERR_ARG, "nbins must be in [1, 8192]");
    if ((type_a >= 0 || type_b >= 0) && !s->have_types) return fail(DP_ERR_ARG, "particle types not set");
    for (int b = 0; b < nbins; ++b)
        if (!(edges[b] <= edges[b + 1])) return fail(DP_ERR_ARG, "r_bins array must be sorted in ascending order.");
    // edges, the selections' lengths and counts in one buffer of the handle,
    // grown as needed: the last two are cleared together
    if (nbins > s->rdf_bins) {
        s->rdf_bins = 0;
        RET(dalloc(&s->rdf_buf, (size_t)(nbins + 1) * sizeof(double) + (size_t)(nbins + 1) * sizeof(unsigned long long)));
        s->rdf_bins = nbins;
    }
    RdfArgs a{};
    double* dedges = (double*)s->rdf_buf;
    a.pos = s->pos;
    a.shadow = s->shadow;
    a.edges = dedges;
    unsigned long long* lengths = (unsigned long long*)(dedges + s->rdf_bins + 1);
    a.counts = lengths + 1;
    a.n = s->n;
    a.nbins = nbins;
    // two cells per bin: most need no second compare; at most 4096, so that the
    // largest histogram (8192 bins) still fits in shared memory
    a.cells = std::min(2 * nbins, 4096);
    a.copies = nbins <= 512 ? 8 : (nbins <= 2048 ? 2 : 1);
    a.symmetric = type_a < 0 ? type_b < 0 : type_a == type_b;
    double lmax = 0.0;
    for (int k = 0; k < DP_MAX_DIM; ++k) a.box[k] = (k < s->dim) ? s->box[k] : 1.0;
    for (int k = 0; k < s->dim; ++k) lmax = std::max(lmax, s->box[k]);
    fill_scale(s, nullptr, a.unit);
    a.abs_tol = (float)(4.0 * lmax / 4294967296.0 * std::sqrt((double)s->dim) + 1e-30);
    const unsigned gn = grid_for(s->n, kBlock);
    const bool small = (long long)gn * ((s->n + kRdfChunk - 1) / kRdfChunk) <= kRdfSmallItems;
    CK(cudaMemcpyAsync(dedges, edges, (nbins + 1) * sizeof(double), cudaMemcpyHostToDevice, s->stream));
    CK(cudaMemsetAsync(lengths, 0, (nbins + 1) * sizeof(unsigned long long), s->stream));
    if ((type_a >= 0 || type_b >= 0) && small) {
        a.types = s->types;
        a.type_a = type_a;
        a.type_b = type_b;
    } else if (type_a >= 0 || type_b >= 0) {
        // the two selections in one buffer of the handle
        if (!s->rdf_sel) RET(dalloc_t(&s->rdf_sel, 2 * (size_t)s->n));
        int32_t* len = (int32_t*)lengths;
        k_rdf_select<<<dim3(gn, a.symmetric ? 1 : 2), kBlock, 0, s->stream>>>(s->types, s->n, type_a, type_b,
                                                                             s->rdf_sel, len);
        CK(cudaGetLastError());
        a.idx_a = s->rdf_sel;
        a.idx_b = a.symmetric ? s->rdf_sel : s->rdf_sel + s->n;
        a.selected = len;
    }
    const size_t smem = (size_t)(nbins + 1) * (sizeof(double) + sizeof(float)) +
                        (size_t)a.copies * nbins * sizeof(unsigned int) + (size_t)a.cells * sizeof(uint16_t);
    const int chunk = small ? kRdfSmallChunk : kRdfChunk;
    const long long items = (long long)gn * ((s->n + chunk - 1) / chunk);
    const unsigned g = (unsigned)std::min<long long>(items, 152LL * 8);
    auto launch = [&](auto kernel) -> cudaError_t {
        if (smem > 32 * 1024) {
            const cudaError_t e =
                cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
        }
        kernel<<<g, kBlock, smem, s->stream>>>(a);
        return cudaGetLastError();
    };
    if (small)
        CK(s->dim == 2 ? launch(k_rdf<2, true>) : (s->dim == 3 ? launch(k_rdf<3, true>) : launch(k_rdf<4, true>)));
    else
        CK(s->dim == 2 ? launch(k_rdf<2, false>) : (s->dim == 3 ? launch(k_rdf<3, false>) : launch(k_rdf<4, false>)));
    CK(cudaMemcpyAsync(counts, a.counts, nbins * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s->stream));
    CK(cudaStreamSynchronize(s->stream));
    return DP_OK;
}

int dp_sum_mv2_noalloc(const double* velocities, const double* masses, int64_t n, int dim, double* out,
                       void* stream) {
    if (!velocities || !masses || !out) return fail(DP_ERR_ARG, "null device pointer");
    if (dim < 1 || dim > DP_MAX_DIM) return fail(DP_ERR_ARG, "dimension must be in [1, 4]");
    if (n < 1) return fail(DP_ERR_ARG, "number of particles must be >= 1");
    const long long blocks = (n - 1) / kBlock + 1;  // n >= 1: no overflow near INT64_MAX
    if (blocks > DP_NOALLOC_MAX_BLOCKS)
        return fail(DP_ERR_ARG, "dp_sum_mv2_noalloc: " + std::to_string(n) + " particles exceed its fixed scratch (at most " +
                                    std::to_string((long long)DP_NOALLOC_MAX_BLOCKS * kBlock) + ")");
    int dev = -1;
    CK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(DP_ERR_ARG, "device ordinal out of range");
    double* partial = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        if (!g_noalloc_addr[dev]) {
            void* p = nullptr;
            const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_partial);
            if (e != cudaSuccess || !p)
                return fail(DP_ERR_CUDA, std::string("cudaGetSymbolAddress(g_noalloc_partial): ") + cudaGetErrorString(e));
            g_noalloc_addr[dev] = (double*)p;
        }
        partial = g_noalloc_addr[dev];
    }
    cudaStream_t st = (cudaStream_t)stream;
    k_mv2_rowmajor<<<(unsigned)blocks, kBlock, 0, st>>>(velocities, masses, n, dim, partial);
    k_reduce<<<1, 1024, 0, st>>>(partial, blocks, out);
    CK(cudaGetLastError());
    return DP_OK;
}

int64_t dp_kernel_launches(dp_sim* s) { return s ? s->launches_last : 0; }

}  // extern "C"

// ===========================================================================
// batched replicas (many independent small systems, one persistent kernel)
// ===========================================================================
namespace {

// Fixed-point shadow of every particle of every replica (each with its box).
__global__ void k_batch_shadow(const double* pos, void* shadow, const int32_t* rep_of, const double* box, int dim,
                               long long ntot) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ntot) return;
    const int r = rep_of[i];
    uint32_t u[DP_MAX_DIM] = {0, 0, 0, 0};
    for (int k = 0; k < dim; ++k) u[k] = dp_fixed(pos[k * ntot + i], 4294967296.0 / box[r * DP_MAX_DIM + k]);
    if (dim == 2)
        ((uint2*)shadow)[i] = make_uint2(u[0], u[1]);
    else
        ((uint4*)shadow)[i] = make_uint4(u[0], u[1], u[2], u[3]);
}

}  // namespace

struct BatchGraph {
    long long steps;
    int sample_every, nve, record;
    unsigned long long version;
    cudaGraphExec_t exec;
};

struct dp_batch {
    int dim = 3;
    int n_rep = 0;
    long long ntot = 0;
    cudaStream_t stream = nullptr, stream2 = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr, fork = nullptr, join = nullptr;
    double *pos = nullptr, *vel = nullptr, *beta = nullptr, *stage = nullptr;
    int32_t *img = nullptr, *rep_of = nullptr, *order = nullptr, *ncell = nullptr, *queue = nullptr;
    void* shadow = nullptr;
    long long* offset = nullptr;
    double *box = nullptr, *coef = nullptr, *obs = nullptr;
    float* force_out = nullptr;
    dp_dev_status* dstat = nullptr;
    dp_dev_status* hstat = nullptr;
    // Verlet lists (skin < 0: cell stencil every step); skin 0.45 was the
    // fastest of 0.2 - 0.8 for LJ replicas at T 0.7 - 2.0, dt 0.005
    double skin = 0.45;
    int kmax_req = 0;  // 0: from the densest replica
    int kmax = 0;      // capacity of the allocated lists
    uint16_t* nlist = nullptr;
    int32_t* ncnt = nullptr;
    void* shadow_ref = nullptr;
    unsigned long long* list_stats = nullptr;
    int32_t* list_gen = nullptr;  // per replica: the generation its list was built for
    std::vector<long long> h_offset;
    std::vector<double> h_box, h_temp;
    std::vector<int> h_ncell, h_order;
    bool have_state = false, have_pot = false;
    std::string pot_src;
    double r_cut = 2.5;
    PairLib lib;
    double dt = 0.005, tau = 0.1, mass = 1.0;
    unsigned long long seed = 0;
    int split_n = 1024, threads_small = 256, threads_large = 1024;
    unsigned long long version = 1;
    std::vector<BatchGraph> graphs;
};

static int batch_kernel_index(int threads) {
    switch (threads) {
        case 128: return 0;
        case 256: return 1;
        case 512: return 2;
        case 1024: return 3;
        default: return -1;
    }
}

static int batch_upload_coef(dp_batch* b) {
    std::vector<double> coef((size_t)b->n_rep * 5);
    const double m = b->mass;
    for (int r = 0; r < b->n_rep; ++r) {
        const double T = b->h_temp.empty() ? 1.0 : b->h_temp[r];
        const double alpha = m / b->tau;  // dompap/integrator.py:29-36
        const double beta_variance = 2 * alpha * T * b->dt;
        const double numerator = 1.0 - alpha * b->dt / 2.0 / m;
        const double denominator = 1.0 + alpha * b->dt / 2.0 / m;
        const double bb = 1 / denominator;
        coef[r * 5 + 0] = numerator / denominator;
        coef[r * 5 + 1] = bb * b->dt / m;
        coef[r * 5 + 2] = bb / 2 / m;
        coef[r * 5 + 3] = std::sqrt(beta_variance);
        coef[r * 5 + 4] = b->dt / m;
    }
    CK(cudaMemcpy(b->coef, coef.data(), coef.size() * sizeof(double), cudaMemcpyHostToDevice));
    b->version++;
    return DP_OK;
}

// Cells for the replica's binning, with the cutoff c = r_cut + skin (lists)
// or r_cut (no lists). With lists (binning only for builds) c/2 wide with a
// 5^D stencil where every axis has at least 5 of them (stored negated): fewer
// candidates per build; otherwise, and without lists (binning every step,
// where the loop over many sparse cells costs more), c wide with a 3^D stencil
// (at least 3 per axis); else all pairs inside the replica.
static int batch_configure_cells(dp_batch* b) {
    b->h_ncell.assign((size_t)b->n_rep * DP_MAX_DIM, 0);
    const double width = b->r_cut + std::max(0.0, b->skin);
    const int first_reach = b->skin >= 0.0 ? 2 : 1;
    for (int r = 0; r < b->n_rep; ++r) {
        for (int reach = first_reach; reach >= 1; --reach) {
            bool ok = true;
            int nc[DP_MAX_DIM] = {0, 0, 0, 0};
            for (int k = 0; k < b->dim; ++k) {
                nc[k] = (int)std::floor(b->h_box[r * DP_MAX_DIM + k] * reach / (width * (1.0 + 1e-6)));
                ok = ok && nc[k] >= 2 * reach + 1;
            }
            long long cells = 1;
            for (int k = 0; k < b->dim; ++k) cells *= std::max(nc[k], 1);
            if (!ok || cells > 32768) continue;
            for (int k = 0; k < b->dim; ++k) b->h_ncell[r * DP_MAX_DIM + k] = reach == 2 ? -nc[k] : nc[k];
            break;
        }
    }
    CK(cudaMemcpy(b->ncell, b->h_ncell.data(), b->h_ncell.size() * sizeof(int32_t), cudaMemcpyHostToDevice));
    b->version++;
    return DP_OK;
}

// Replicas sorted by size (largest first) and split into a small and a large
// bucket, each run by its own persistent launch.
struct BatchBucket {
    int first, count, threads, max_n, max_cells;
};

static void batch_buckets(const dp_batch* b, BatchBucket* out, int* nb) {
    *nb = 0;
    int large = 0;
    while (large < b->n_rep) {
        const int r = b->h_order[large];
        if (b->h_offset[r + 1] - b->h_offset[r] <= b->split_n) break;
        ++large;
    }
    auto fill = [&](int first, int count, int threads) {
        BatchBucket bk{first, count, threads, 0, 1};
        for (int q = first; q < first + count; ++q) {
            const int r = b->h_order[q];
            bk.max_n = std::max(bk.max_n, (int)(b->h_offset[r + 1] - b->h_offset[r]));
            int cells = 1;
            for (int k = 0; k < b->dim; ++k) cells *= std::max(std::abs(b->h_ncell[r * DP_MAX_DIM + k]), 1);
            bk.max_cells = std::max(bk.max_cells, cells);
        }
        out[(*nb)++] = bk;
    };
    if (large > 0) fill(0, large, b->threads_large);
    if (large < b->n_rep) fill(large, b->n_rep - large, b->threads_small);
}

static size_t batch_smem(int dim, int max_n, int max_cells) {
    const size_t sh = (dim == 2 ? 8 : 16);
    return (size_t)max_n * sh + (size_t)((max_n + 7) & ~7) * 2 + (size_t)(2 * max_cells + 1) * 4;
}

static int batch_record(dp_batch* b, long long steps, int sample_every, int nve, int record) {
    BatchBucket bk[2];
    int nb = 0;
    batch_buckets(b, bk, &nb);
    CK(cudaMemsetAsync(b->queue, 0, 2 * sizeof(int32_t), b->stream));
    int dev = 0;
    CK(cudaGetDevice(&dev));
    int sms = 0;
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (nb == 2) {
        CK(cudaEventRecord(b->fork, b->stream));
        CK(cudaStreamWaitEvent(b->stream2, b->fork, 0));
    }
    for (int q = 0; q < nb; ++q) {
        const BatchBucket& k = bk[q];
        const int ki = batch_kernel_index(k.threads);
        if (ki < 0) return fail(DP_ERR_ARG, "threads per replica must be 128, 256, 512 or 1024");
        if (k.max_n > 65535) return fail(DP_ERR_ARG, "a replica has more than 65535 particles");
        const size_t smem = batch_smem(b->dim, k.max_n, k.max_cells);
        if (smem > 227 * 1024)
            return fail(DP_ERR_ARG, "a replica does not fit in shared memory (" + std::to_string(smem) + " bytes)");
        CK(cudaKernelSetAttributeForDevice(b->lib.batch[ki], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem,
                                           dev));
        dp_batch_args a;
        memset(&a, 0, sizeof(a));
        a.pos = b->pos;
        a.vel = b->vel;
        a.beta = b->beta;
        a.img = b->img;
        a.shadow = b->shadow;
        a.offset = b->offset;
        a.order = b->order + k.first;
        a.box = b->box;
        a.coef = b->coef;
        a.ncell = b->ncell;
        a.obs = b->obs;
        a.force_out = record ? b->force_out : nullptr;
        a.queue = b->queue + q;
        a.st = b->dstat;
        a.ntot = b->ntot;
        a.n_rep = k.count;
        a.steps = (int)steps;
        a.sample_every = sample_every;
        a.max_n = k.max_n;
        a.max_cells = k.max_cells;
        a.nve = nve;
        a.dt = b->dt;
        a.rc2 = (float)(b->r_cut * b->r_cut);
        a.seed = b->seed;
        if (b->skin >= 0.0 && b->nlist) {
            const double rl = b->r_cut + b->skin;
            a.nlist = b->nlist;
            a.ncnt = b->ncnt;
            a.shadow_ref = b->shadow_ref;
            a.list_stats = b->list_stats;
            a.list_gen = b->list_gen;
            a.gen = (int)(b->version & 0x3FFFFFFF);  // a graph is captured per version
            a.kmax = b->kmax;
            // conservative in float32: the list reaches a little past r_cut + skin
            // and a build comes a little before skin/2
            a.rl2 = (float)(rl * rl * (1.0 + 1e-5));
            a.skin_thr2 = (float)(0.25 * b->skin * b->skin * (1.0 - 1e-5));
        }
        const int per_sm = std::max(1, std::min(2048 / k.threads, (int)((228 * 1024) / (smem + 1024))));
        const unsigned grid = (unsigned)std::max(1, std::min(k.count, sms * per_sm));
        void* args[] = {&a};
        cudaStream_t st = (q == 0) ? b->stream : b->stream2;
        CK(cudaLaunchKernel((const void*)b->lib.batch[ki], dim3(grid), dim3(k.threads), args, smem, st));
    }
    if (nb == 2) {
        CK(cudaEventRecord(b->join, b->stream2));
        CK(cudaStreamWaitEvent(b->stream, b->join, 0));
    }
    k_advance_step<<<1, 1, 0, b->stream>>>(b->dstat, steps, 0);
    CK(cudaGetLastError());
    return DP_OK;
}

extern "C" {

int dp_batch_create(int dim, int n_rep, const int32_t* counts, dp_batch** out) {
    if (!out || !counts) return fail(DP_ERR_ARG, "null argument");
    *out = nullptr;
    if (dim < 2 || dim > 4) return fail(DP_ERR_ARG, "dimension must be 2, 3 or 4");
    if (n_rep < 1) return fail(DP_ERR_ARG, "need at least one replica");
    dp_batch* b = new dp_batch();
    b->dim = dim;
    b->n_rep = n_rep;
    b->h_offset.assign((size_t)n_rep + 1, 0);
    for (int r = 0; r < n_rep; ++r) {
        if (counts[r] < 2 || counts[r] > 65535) {
            delete b;
            return fail(DP_ERR_ARG, "replica sizes must be in [2, 65535]");
        }
        b->h_offset[r + 1] = b->h_offset[r] + counts[r];
    }
    b->ntot = b->h_offset[n_rep];
    b->h_order.resize(n_rep);
    for (int r = 0; r < n_rep; ++r) b->h_order[r] = r;
    std::stable_sort(b->h_order.begin(), b->h_order.end(), [&](int x, int y) { return counts[x] > counts[y]; });
    int rc = DP_OK;
    auto cleanup = [&]() {
        dp_batch_destroy(b);
        return rc;
    };
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaStreamCreateWithFlags(&b->stream2, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&b->ev0) != cudaSuccess || cudaEventCreate(&b->ev1) != cudaSuccess ||
        cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&b->join, cudaEventDisableTiming) != cudaSuccess) {
        rc = fail(DP_ERR_CUDA, "stream/event creation failed");
        return cleanup();
    }
    const size_t nd = (size_t)b->ntot * dim;
    if ((rc = dalloc_t(&b->pos, nd)) || (rc = dalloc_t(&b->vel, nd)) || (rc = dalloc_t(&b->beta, nd)) ||
        (rc = dalloc_t(&b->stage, nd)) || (rc = dalloc_t(&b->img, nd)) || (rc = dalloc_t(&b->rep_of, b->ntot)) ||
        (rc = dalloc_t(&b->order, (size_t)n_rep)) || (rc = dalloc_t(&b->ncell, (size_t)n_rep * DP_MAX_DIM)) ||
        (rc = dalloc_t(&b->queue, 2)) || (rc = dalloc_t(&b->offset, (size_t)n_rep + 1)) ||
        (rc = dalloc_t(&b->box, (size_t)n_rep * DP_MAX_DIM)) || (rc = dalloc_t(&b->coef, (size_t)n_rep * 5)) ||
        (rc = dalloc_t(&b->obs, (size_t)n_rep * 4)) || (rc = dalloc(&b->shadow, (size_t)b->ntot * (dim == 2 ? 8 : 16))))
        return cleanup();
    if (cudaMalloc(&b->dstat, sizeof(dp_dev_status)) != cudaSuccess ||
        cudaMallocHost(&b->hstat, sizeof(dp_dev_status)) != cudaSuccess) {
        rc = fail(DP_ERR_CUDA, "status allocation failed");
        return cleanup();
    }
    memset(b->hstat, 0, sizeof(dp_dev_status));
    std::vector<int32_t> rep_of((size_t)b->ntot);
    for (int r = 0; r < n_rep; ++r)
        for (long long i = b->h_offset[r]; i < b->h_offset[r + 1]; ++i) rep_of[i] = r;
    if (cudaMemcpy(b->dstat, b->hstat, sizeof(dp_dev_status), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(b->rep_of, rep_of.data(), rep_of.size() * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(b->offset, b->h_offset.data(), b->h_offset.size() * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(b->order, b->h_order.data(), (size_t)n_rep * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(b->obs, 0, (size_t)n_rep * 4 * 8) != cudaSuccess || cudaMemset(b->img, 0, nd * 4) != cudaSuccess ||
        cudaMemset(b->beta, 0, nd * 8) != cudaSuccess) {
        rc = fail(DP_ERR_CUDA, "batch initialisation failed");
        return cleanup();
    }
    *out = b;
    return DP_OK;
}

int dp_batch_destroy(dp_batch* b) {
    if (!b) return DP_OK;
    if (b->stream) cudaStreamSynchronize(b->stream);
    if (b->stream2) cudaStreamSynchronize(b->stream2);
    for (auto& g : b->graphs) cudaGraphExecDestroy(g.exec);
    void* bufs[] = {b->pos, b->vel, b->beta, b->stage, b->img, b->rep_of, b->order, b->ncell, b->queue, b->shadow,
                    b->offset, b->box, b->coef, b->obs, b->force_out, b->dstat, b->nlist, b->ncnt, b->shadow_ref,
                    b->list_stats, b->list_gen};
    for (void* p : bufs)
        if (p) cudaFree(p);
    if (b->hstat) cudaFreeHost(b->hstat);
    cudaEvent_t evs[] = {b->ev0, b->ev1, b->fork, b->join};
    for (cudaEvent_t e : evs)
        if (e) cudaEventDestroy(e);
    if (b->stream) cudaStreamDestroy(b->stream);
    if (b->stream2) cudaStreamDestroy(b->stream2);
    delete b;
    return DP_OK;
}

int dp_batch_set_state(dp_batch* b, const double* positions, const double* velocities, const double* boxes,
                       const double* temperatures) {
    if (!b || !positions || !velocities || !boxes || !temperatures) return fail(DP_ERR_ARG, "null argument");
    b->h_box.assign((size_t)b->n_rep * DP_MAX_DIM, 1.0);
    b->h_temp.assign(temperatures, temperatures + b->n_rep);
    for (int r = 0; r < b->n_rep; ++r)
        for (int k = 0; k < b->dim; ++k) {
            const double L = boxes[r * b->dim + k];
            if (!(L > 0.0) || !std::isfinite(L)) return fail(DP_ERR_ARG, "box sides must be positive");
            b->h_box[r * DP_MAX_DIM + k] = L;
        }
    const size_t bytes = (size_t)b->ntot * b->dim * sizeof(double);
    CK(cudaMemcpy(b->box, b->h_box.data(), b->h_box.size() * 8, cudaMemcpyHostToDevice));
    const unsigned g = grid_for(b->ntot * b->dim, kBlock);
    CK(cudaMemcpyAsync(b->stage, positions, bytes, cudaMemcpyHostToDevice, b->stream));
    k_host_to_slots<double><<<g, kBlock, 0, b->stream>>>(b->stage, b->pos, nullptr, b->ntot, b->dim);
    CK(cudaMemcpyAsync(b->stage, velocities, bytes, cudaMemcpyHostToDevice, b->stream));
    k_host_to_slots<double><<<g, kBlock, 0, b->stream>>>(b->stage, b->vel, nullptr, b->ntot, b->dim);
    k_batch_shadow<<<grid_for(b->ntot, kBlock), kBlock, 0, b->stream>>>(b->pos, b->shadow, b->rep_of, b->box, b->dim,
                                                                        b->ntot);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(b->stream));
    b->have_state = true;
    if (b->have_pot) RET(batch_configure_cells(b));
    return batch_upload_coef(b);
}

int dp_batch_get_state(dp_batch* b, double* positions, double* velocities, int32_t* images) {
    if (!b) return fail(DP_ERR_ARG, "null handle");
    const size_t bytes = (size_t)b->ntot * b->dim * sizeof(double);
    const unsigned g = grid_for(b->ntot * b->dim, kBlock);
    if (positions) {
        k_slots_to_host<double><<<g, kBlock, 0, b->stream>>>(b->pos, b->stage, nullptr, b->ntot, b->dim);
        CK(cudaMemcpyAsync(positions, b->stage, bytes, cudaMemcpyDeviceToHost, b->stream));
        CK(cudaStreamSynchronize(b->stream));
    }
    if (velocities) {
        k_slots_to_host<double><<<g, kBlock, 0, b->stream>>>(b->vel, b->stage, nullptr, b->ntot, b->dim);
        CK(cudaMemcpyAsync(velocities, b->stage, bytes, cudaMemcpyDeviceToHost, b->stream));
        CK(cudaStreamSynchronize(b->stream));
    }
    if (images) {
        int32_t* st = (int32_t*)b->stage;
        k_slots_to_host<int32_t><<<g, kBlock, 0, b->stream>>>(b->img, st, nullptr, b->ntot, b->dim);
        CK(cudaMemcpyAsync(images, st, (size_t)b->ntot * b->dim * 4, cudaMemcpyDeviceToHost, b->stream));
        CK(cudaStreamSynchronize(b->stream));
    }
    CK(cudaGetLastError());
    return DP_OK;
}

int dp_batch_set_potential(dp_batch* b, const char* device_source, double r_cut) {
    if (!b || !device_source) return fail(DP_ERR_ARG, "null argument");
    if (!(r_cut > 0.0) || !std::isfinite(r_cut)) return fail(DP_ERR_ARG, "r_cut must be positive and finite");
    ProgramParts parts;
    parts.brick_blocks = parts.lists_blocks = 0;
    parts.warp_sums = parts.quad_sums = false;
    const std::string src = pair_program(b->dim, DP_PREC_FP32, DP_PAIR_CONST, true, true, device_source, true, parts);
    PairLib pl;
    RET(compile_pair_lib(src, &pl));
    if (!pl.batch[0]) return fail(DP_ERR_NVRTC, "batch kernels missing from the compiled program");
    b->lib = pl;
    b->pot_src = device_source;
    b->r_cut = r_cut;
    b->have_pot = true;
    b->version++;
    if (b->have_state) RET(batch_configure_cells(b));
    return DP_OK;
}

int dp_batch_set_integrator(dp_batch* b, double time_step, double damping_time, double mass, uint64_t seed) {
    if (!b) return fail(DP_ERR_ARG, "null handle");
    if (!(mass > 0.0)) return fail(DP_ERR_ARG, "mass must be positive");
    b->dt = time_step;
    b->tau = damping_time;
    b->mass = mass;
    b->seed = seed;
    return batch_upload_coef(b);
}

int dp_batch_set_launch(dp_batch* b, int split_n, int threads_small, int threads_large) {
    if (!b) return fail(DP_ERR_ARG, "null handle");
    if (batch_kernel_index(threads_small) < 0 || batch_kernel_index(threads_large) < 0)
        return fail(DP_ERR_ARG, "threads per replica must be 128, 256, 512 or 1024");
    b->split_n = std::max(0, split_n);
    b->threads_small = threads_small;
    b->threads_large = threads_large;
    b->version++;
    return DP_OK;
}

// List capacity: 1.3 x the pair count of the densest replica's list sphere +
// 16, or the requested one; a multiple of 8 (the lists are stored in 8-entry
// chunks of 16 bytes).
static int batch_list_capacity(const dp_batch* b) {
    if (b->kmax_req > 0) return std::min((b->kmax_req + 7) & ~7, 65528);
    const double rl = b->r_cut + std::max(0.0, b->skin);
    const double pi = 3.141592653589793;
    const double sphere = b->dim == 2 ? pi * rl * rl : (b->dim == 3 ? 4.0 / 3.0 * pi * rl * rl * rl : 0.5 * pi * pi * rl * rl * rl * rl);
    double rho = 0.0;
    for (int r = 0; r < b->n_rep; ++r) {
        double vol = 1.0;
        for (int k = 0; k < b->dim; ++k) vol *= b->h_box[r * DP_MAX_DIM + k];
        rho = std::max(rho, (double)(b->h_offset[r + 1] - b->h_offset[r]) / vol);
    }
    const long long k = ((long long)std::ceil(1.3 * sphere * rho) + 16 + 7) & ~7LL;
    return (int)std::min<long long>(std::max<long long>(k, 8), 65528);
}

static int batch_ensure_lists(dp_batch* b) {
    if (b->skin < 0.0) return DP_OK;
    const int k = batch_list_capacity(b);
    if (b->nlist && k == b->kmax) return DP_OK;
    if (b->nlist) cudaFree(b->nlist);
    b->nlist = nullptr;
    RET(dalloc_t(&b->nlist, (size_t)b->ntot * (size_t)k));
    if (!b->ncnt) RET(dalloc_t(&b->ncnt, (size_t)b->ntot));
    if (!b->shadow_ref) RET(dalloc(&b->shadow_ref, (size_t)b->ntot * (b->dim == 2 ? 8 : 16)));
    if (!b->list_stats) {
        RET(dalloc_t(&b->list_stats, 2));
        CK(cudaMemset(b->list_stats, 0, 2 * sizeof(unsigned long long)));
    }
    if (!b->list_gen) {
        RET(dalloc_t(&b->list_gen, (size_t)b->n_rep));
        CK(cudaMemset(b->list_gen, 0xFF, (size_t)b->n_rep * sizeof(int32_t)));  // -1: never built
    }
    b->kmax = k;
    b->version++;
    return DP_OK;
}

int dp_batch_run(dp_batch* b, int64_t steps, int sample_every, int nve, int record_forces, float* ms) {
    if (!b) return fail(DP_ERR_ARG, "null handle");
    if (!b->have_state || !b->have_pot) return fail(DP_ERR_NOPOT, "batch state or potential not set");
    if (steps < 0 || steps > (1LL << 30)) return fail(DP_ERR_ARG, "bad step count");
    if (steps == 0) return DP_OK;
    if (record_forces && !b->force_out) RET(dalloc_t(&b->force_out, (size_t)b->ntot * b->dim));
    RET(batch_ensure_lists(b));
    BatchGraph* g = nullptr;
    for (auto& x : b->graphs)
        if (x.steps == steps && x.sample_every == sample_every && x.nve == nve && x.record == record_forces &&
            x.version == b->version)
            g = &x;
    if (!g) {
        for (auto& x : b->graphs) cudaGraphExecDestroy(x.exec);
        b->graphs.clear();
        cudaGraph_t graph;
        CK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
        const int rc = batch_record(b, steps, sample_every, nve, record_forces);
        const cudaError_t e = cudaStreamEndCapture(b->stream, &graph);
        if (rc != DP_OK) return rc;
        if (e != cudaSuccess) return fail(DP_ERR_CUDA, std::string("capture: ") + cudaGetErrorString(e));
        BatchGraph bg{steps, sample_every, nve, record_forces, b->version, nullptr};
        const cudaError_t ei = cudaGraphInstantiate(&bg.exec, graph, 0);
        cudaGraphDestroy(graph);
        if (ei != cudaSuccess) return fail(DP_ERR_CUDA, std::string("instantiate: ") + cudaGetErrorString(ei));
        b->graphs.push_back(bg);
        g = &b->graphs.back();
    }
    if (ms) CK(cudaEventRecord(b->ev0, b->stream));
    CK(cudaGraphLaunch(g->exec, b->stream));
    if (ms) CK(cudaEventRecord(b->ev1, b->stream));
    CK(cudaMemcpyAsync(b->hstat, b->dstat, sizeof(dp_dev_status), cudaMemcpyDeviceToHost, b->stream));
    CK(cudaStreamSynchronize(b->stream));
    if (ms) CK(cudaEventElapsedTime(ms, b->ev0, b->ev1));
    if (b->hstat->nonfinite) {
        b->hstat->nonfinite = 0;
        CK(cudaMemcpy(b->dstat, b->hstat, sizeof(dp_dev_status), cudaMemcpyHostToDevice));
        return fail(DP_ERR_NONFINITE, "a position became NaN/Inf in a replica");
    }
    return DP_OK;
}

static int nvrtc_check_impl(int dim, int precision, int pair_mode, int with_batch, const char* device_source,
                            int64_t* cubin_bytes, std::string* resource_log) {
    if (!device_source) return fail(DP_ERR_ARG, "null source");
    if (dim < 2 || dim > 4) return fail(DP_ERR_ARG, "dimension must be 2, 3 or 4");
    if (precision != DP_PREC_FP64 && precision != DP_PREC_FP32 && precision != DP_PREC_MLP)
        return fail(DP_ERR_ARG, "unknown precision");
    if (pair_mode < DP_PAIR_CONST || pair_mode > DP_PAIR_DENSE) return fail(DP_ERR_ARG, "unknown pair mode");
    const bool one = pair_mode == DP_PAIR_CONST;
    ProgramParts parts;  // all of them
    parts.step_blocks = step_blocks_for(dim, precision, pair_mode, pair_cost(device_source));
    if (with_batch) parts.brick_blocks = 0;
    const std::string src = pair_program(dim, precision, pair_mode, one, one, device_source, with_batch != 0, parts);
    std::vector<char> cubin;
    RET(nvrtc_cubin(src, &cubin, resource_log, true, true));
    if (cubin_bytes) *cubin_bytes = (int64_t)cubin.size();
    return DP_OK;
}

int dp_nvrtc_check(int dim, int precision, int pair_mode, int with_batch, const char* device_source,
                   int64_t* cubin_bytes) {
    return nvrtc_check_impl(dim, precision, pair_mode, with_batch, device_source, cubin_bytes, nullptr);
}

int dp_nvrtc_resources(int dim, int precision, int pair_mode, int with_batch, const char* device_source, char* log,
                       int64_t log_capacity, int64_t* log_bytes) {
    if (!log || log_capacity < 1) return fail(DP_ERR_ARG, "bad log buffer");
    std::string text;
    RET(nvrtc_check_impl(dim, precision, pair_mode, with_batch, device_source, nullptr, &text));
    const size_t len = strnlen(text.c_str(), text.size());
    const size_t k = std::min(len, (size_t)(log_capacity - 1));
    memcpy(log, text.data(), k);
    log[k] = '\0';
    if (log_bytes) *log_bytes = (int64_t)len;
    return DP_OK;
}

int dp_batch_set_neighbor_list(dp_batch* b, double skin, int kmax) {
    if (!b) return fail(DP_ERR_ARG, "null handle");
    if (!std::isfinite(skin)) return fail(DP_ERR_ARG, "skin must be finite");
    if (kmax < 0 || kmax > 65535) return fail(DP_ERR_ARG, "kmax must be in [0, 65535]");
    b->skin = skin < 0.0 ? -1.0 : skin;
    b->kmax_req = kmax;
    b->version++;
    if (b->have_state && b->have_pot) RET(batch_configure_cells(b));
    return DP_OK;
}

int dp_batch_list_stats(dp_batch* b, int64_t* builds, int64_t* overflowed, int32_t* kmax) {
    if (!b) return fail(DP_ERR_ARG, "null handle");
    unsigned long long h[2] = {0, 0};
    if (b->list_stats) CK(cudaMemcpy(h, b->list_stats, sizeof(h), cudaMemcpyDeviceToHost));
    if (builds) *builds = (int64_t)h[0];
    if (overflowed) *overflowed = (int64_t)h[1];
    if (kmax) *kmax = b->skin < 0.0 ? 0 : b->kmax;
    return DP_OK;
}

int dp_batch_observables(dp_batch* b, double* out, int reset) {
    if (!b || !out) return fail(DP_ERR_ARG, "null argument");
    CK(cudaMemcpy(out, b->obs, (size_t)b->n_rep * 4 * sizeof(double), cudaMemcpyDeviceToHost));
    if (reset) CK(cudaMemset(b->obs, 0, (size_t)b->n_rep * 4 * sizeof(double)));
    return DP_OK;
}

int dp_batch_last_forces(dp_batch* b, double* forces) {
    if (!b || !forces) return fail(DP_ERR_ARG, "null argument");
    if (!b->force_out) return fail(DP_ERR_ARG, "no step was run with record_forces");
    std::vector<float> f((size_t)b->ntot * b->dim);
    CK(cudaMemcpy(f.data(), b->force_out, f.size() * sizeof(float), cudaMemcpyDeviceToHost));
    for (long long i = 0; i < b->ntot; ++i)
        for (int k = 0; k < b->dim; ++k) forces[i * b->dim + k] = (double)f[(size_t)k * b->ntot + i];
    return DP_OK;
}

}  // extern "C"

// ===========================================================================
// pair surrogate network (training, evaluation)
// ===========================================================================
struct dp_mlp {
    float *master = nullptr, *mo = nullptr, *ve = nullptr, *grad = nullptr, *norm = nullptr, *loss = nullptr;
    unsigned long long* gradfx = nullptr;  // DP_MLP_NPARAM + 1 (the loss last)
    dp_mlp_dev* dev = nullptr;
    uint32_t* w2t = nullptr;  // bf16 fragments of W2 transposed (backward pass)
    float* s = nullptr;
    float2* t = nullptr;
    long long n = 0;
    float* losses = nullptr;
    long long losses_cap = 0;
    long long step = 0;
    cudaStream_t stream = nullptr;
};

static int mlp_pack(dp_mlp* m) {
    k_mlp_pack<<<4, 256, 0, m->stream>>>(m->master, m->norm, m->dev, m->w2t);
    CK(cudaGetLastError());
    return DP_OK;
}

// Launch with programmatic dependent launch: the kernel's blocks may be placed
// while the one before it on the stream still runs; both kernels of a training
// step wait (griddepcontrol.wait) before they touch anything it writes.
template <typename Args>
static cudaError_t mlp_launch(void (*kernel)(Args), unsigned grid, unsigned block, size_t smem, cudaStream_t stream,
                              const Args& args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args);
}

static MlpTrainArgs mlp_grad_args(const dp_mlp* m, const float* s, const float2* t, long long batch, float wf) {
    MlpTrainArgs a;
    memset(&a, 0, sizeof(a));
    a.s = s;
    a.t = t;
    a.batch = batch;
    a.mdev = m->dev;
    a.w2t = m->w2t;
    a.gradfx = m->gradfx;
    a.lossfx = m->gradfx + DP_MLP_NPARAM;
    a.wf = wf;
    a.inv_batch = 1.0f / (float)batch;
    return a;
}

// Adds the batch's gradient and loss to gradfx (which the caller has cleared).
static int mlp_grad_launch(dp_mlp* m, const MlpTrainArgs& a, bool accurate) {
    const long long groups = (a.batch + DP_MLP_ROWS - 1) / DP_MLP_ROWS;
    const unsigned grid = (unsigned)std::max<long long>(1, std::min<long long>(groups, 152LL * 4));
    CK(mlp_launch(accurate ? k_mlp_grad<true> : k_mlp_grad<false>, grid, 256, DP_MLP_GRAD_SMEM, m->stream, a));
    return DP_OK;
}

extern "C" {

int dp_mlp_create(dp_mlp** out) {
    if (!out) return fail(DP_ERR_ARG, "null argument");
    *out = nullptr;
    dp_mlp* m = new dp_mlp();
    int rc = DP_OK;
    if ((rc = dalloc_t(&m->master, DP_MLP_NPARAM)) || (rc = dalloc_t(&m->mo, DP_MLP_NPARAM)) ||
        (rc = dalloc_t(&m->ve, DP_MLP_NPARAM)) || (rc = dalloc_t(&m->grad, DP_MLP_NPARAM)) ||
        (rc = dalloc_t(&m->norm, 4)) || (rc = dalloc_t(&m->loss, 1)) || (rc = dalloc_t(&m->dev, 1)) ||
        (rc = dalloc_t(&m->gradfx, DP_MLP_NPARAM + 1)) || (rc = dalloc_t(&m->w2t, 4 * 8 * 32 * 2))) {
        dp_mlp_destroy(m);
        return rc;
    }
    if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess) {
        dp_mlp_destroy(m);
        return fail(DP_ERR_CUDA, "stream creation failed");
    }
    cudaError_t e = cudaFuncSetAttribute(k_mlp_grad<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, DP_MLP_GRAD_SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_mlp_grad<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, DP_MLP_GRAD_SMEM);
    if (e != cudaSuccess) {
        dp_mlp_destroy(m);
        return fail(DP_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
    }
    *out = m;
    return DP_OK;
}

int dp_mlp_destroy(dp_mlp* m) {
    if (!m) return DP_OK;
    if (m->stream) cudaStreamSynchronize(m->stream);
    void* bufs[] = {m->master, m->mo, m->ve, m->grad, m->norm, m->loss, m->dev, m->s, m->t, m->losses,
                    m->gradfx, m->w2t};
    for (void* p : bufs)
        if (p) cudaFree(p);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return DP_OK;
}

int dp_mlp_param_count(void) { return DP_MLP_NPARAM; }

int dp_set_mlp(dp_sim* s, dp_mlp* m) {
    if (!s) return fail(DP_ERR_ARG, "null handle");
    if (!m && s->precision == DP_PREC_MLP) return fail(DP_ERR_ARG, "switch precision before detaching the surrogate");
    s->mlp_dev = m ? m->dev : nullptr;
    s->version++;
    return DP_OK;
}

int dp_mlp_set_params(dp_mlp* m, const float* params, const float* norm) {
    if (!m || !params || !norm) return fail(DP_ERR_ARG, "null argument");
    CK(cudaMemcpyAsync(m->master, params, DP_MLP_NPARAM * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    CK(cudaMemcpyAsync(m->norm, norm, 4 * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    CK(cudaMemsetAsync(m->mo, 0, DP_MLP_NPARAM * sizeof(float), m->stream));
    CK(cudaMemsetAsync(m->ve, 0, DP_MLP_NPARAM * sizeof(float), m->stream));
    m->step = 0;
    RET(mlp_pack(m));
    CK(cudaStreamSynchronize(m->stream));
    return DP_OK;
}

int dp_mlp_get_params(dp_mlp* m, float* params) {
    if (!m || !params) return fail(DP_ERR_ARG, "null argument");
    CK(cudaMemcpyAsync(params, m->master, DP_MLP_NPARAM * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    CK(cudaStreamSynchronize(m->stream));
    return DP_OK;
}

int dp_mlp_set_data(dp_mlp* m, const float* s, const float* targets, int64_t n) {
    if (!m || !s || !targets || n < 1) return fail(DP_ERR_ARG, "bad training data");
    RET(dalloc_t(&m->s, (size_t)n));
    RET(dalloc_t(&m->t, (size_t)n));
    CK(cudaMemcpy(m->s, s, (size_t)n * sizeof(float), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(m->t, targets, (size_t)n * 2 * sizeof(float), cudaMemcpyHostToDevice));
    m->n = n;
    return DP_OK;
}

int dp_mlp_train(dp_mlp* m, int64_t steps, int batch, float lr0, float lr1, float wf, uint64_t seed, int accurate,
                 float* losses) {
    if (!m || !m->s) return fail(DP_ERR_ARG, "no training data");
    if (steps < 1 || batch < 16) return fail(DP_ERR_ARG, "bad steps / batch");
    RET(dgrow_t(&m->losses, (long long)steps, &m->losses_cap));
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    MlpTrainArgs ga = mlp_grad_args(m, m->s, m->t, batch, wf);
    ga.draw = 1;
    ga.n = (unsigned long long)m->n;
    ga.seed = seed;
    MlpUpdateArgs ua = {m->master, m->mo, m->ve, ga.gradfx, ga.lossfx, m->dev, m->w2t, m->losses, 0.f, b1, b2, eps,
                        0.f, 0.f};
    // cleared once: k_mlp_update leaves the sums at zero
    CK(cudaMemsetAsync(m->gradfx, 0, (DP_MLP_NPARAM + 1) * sizeof(unsigned long long), m->stream));
    for (long long k = 0; k < steps; ++k) {
        // cosine decay from lr0 to lr1
        const double frac = steps > 1 ? (double)k / (double)(steps - 1) : 1.0;
        ua.lr = (float)(lr1 + 0.5 * (lr0 - lr1) * (1.0 + std::cos(3.141592653589793 * frac)));
        ga.step = m->step;
        RET(mlp_grad_launch(m, ga, accurate != 0));
        ++m->step;
        ua.c1 = 1.0f / (1.0f - std::pow(b1, (float)m->step));
        ua.c2 = 1.0f / (1.0f - std::pow(b2, (float)m->step));
        ua.loss = m->losses + k;
        CK(mlp_launch(k_mlp_update, (kMlpUpdateThreads + 63) / 64, 64, 0, m->stream, ua));
    }
    CK(cudaGetLastError());
    if (losses) CK(cudaMemcpyAsync(losses, m->losses, (size_t)steps * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    CK(cudaStreamSynchronize(m->stream));
    return DP_OK;
}

int dp_mlp_eval(dp_mlp* m, const float* s, int64_t n, float* y, int accurate) {
    if (!m || !s || !y || n < 1) return fail(DP_ERR_ARG, "bad arguments");
    float* buf = nullptr;
    RET(dalloc_t(&buf, (size_t)n * 3));
    cudaError_t e = cudaMemcpyAsync(buf, s, (size_t)n * sizeof(float), cudaMemcpyHostToDevice, m->stream);
    const unsigned grid = (unsigned)std::max<long long>(1, std::min<long long>(((n + 15) / 16 + 7) / 8, 152LL * 8));
    if (e == cudaSuccess) {
        if (accurate)
            k_mlp_eval<true><<<grid, 256, 0, m->stream>>>(buf, n, m->dev, buf + n);
        else
            k_mlp_eval<false><<<grid, 256, 0, m->stream>>>(buf, n, m->dev, buf + n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(y, buf + n, (size_t)n * 2 * sizeof(float), cudaMemcpyDeviceToHost, m->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    cudaFree(buf);
    if (e != cudaSuccess) return fail(DP_ERR_CUDA, std::string("dp_mlp_eval: ") + cudaGetErrorString(e));
    return DP_OK;
}

int dp_mlp_gradients(dp_mlp* m, const float* s, const float* targets, int64_t n, float wf, int accurate, float* grad,
                     float* loss) {
    if (!m || !s || !targets || !grad || n < 1) return fail(DP_ERR_ARG, "bad arguments");
    // targets are read as float2: start them on an 8-byte boundary
    const long long toff = (n + 1) & ~1LL;
    float* buf = nullptr;
    RET(dalloc_t(&buf, (size_t)(toff + 2 * n)));
    cudaError_t e = cudaMemcpyAsync(buf, s, (size_t)n * sizeof(float), cudaMemcpyHostToDevice, m->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(buf + toff, targets, (size_t)n * 2 * sizeof(float), cudaMemcpyHostToDevice, m->stream);
    int rc = DP_OK;
    if (e == cudaSuccess)
        e = cudaMemsetAsync(m->gradfx, 0, (DP_MLP_NPARAM + 1) * sizeof(unsigned long long), m->stream);
    if (e == cudaSuccess)
        rc = mlp_grad_launch(m, mlp_grad_args(m, buf, (const float2*)(buf + toff), n, wf), accurate != 0);
    if (e == cudaSuccess && rc == DP_OK) {
        k_mlp_grad_finish<<<grid_for(DP_MLP_NPARAM, kBlock), kBlock, 0, m->stream>>>(
            m->gradfx, m->gradfx + DP_MLP_NPARAM, m->grad, m->loss);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && rc == DP_OK)
        e = cudaMemcpyAsync(grad, m->grad, DP_MLP_NPARAM * sizeof(float), cudaMemcpyDeviceToHost, m->stream);
    float l = 0.f;
    if (e == cudaSuccess && rc == DP_OK) e = cudaMemcpyAsync(&l, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    cudaFree(buf);
    if (rc != DP_OK) return rc;
    if (e != cudaSuccess) return fail(DP_ERR_CUDA, std::string("dp_mlp_gradients: ") + cudaGetErrorString(e));
    if (loss) *loss = l / (float)n;
    return DP_OK;
}

}  // extern "C"
