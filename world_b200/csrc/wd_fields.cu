// wd_fields.cu -- node-centred CIC deposit of mass and momentum.
//
// Weights and layout follow reference src/density_grid_kernel.cu:25-83 (node-centred
// spacing (hi-lo)/(size-1), indices clamped, zero-mass grains skipped, channel-major
// [m, m vx, m vy, m vz], node = (ix*ny + iy)*nz + iz). The reference accumulates with
// float atomicAdd, so its field changes with thread timing. Here every contribution
// (the same float product the reference adds) is converted to a 64-bit fixed-point
// integer with a power-of-two scale chosen per channel from a bound on the channel's
// total, and accumulated with integer atomics: integer addition is associative, so
// the field is bit-identical run to run and is the correctly rounded sum up to the
// 2^-62-relative quantum. Because every part adds the same integers, it may group them as
// it likes; the accumulators are node-major (the four channels of a node share one
// 32-byte sector) and k_deposit's lanes are laid over corners and channels (see there).
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "wd_kernels.h"

namespace wd {

namespace {

// reference src/density_grid_kernel.cu:25-40
__device__ __forceinline__ void axis_weights(float x, float lo, float hi, int size, int& i0,
                                             int& i1, float& w0, float& w1) {
    if (size <= 1) {
        i0 = 0; i1 = 0; w0 = 1.f; w1 = 0.f;
        return;
    }
    const float h = (hi - lo) / static_cast<float>(size - 1);
    const float u = (x - lo) / h;
    const float base = floorf(u);
    const float frac = u - base;
    const int b = __float2int_rz(base);
    i0 = min(size - 1, max(0, b));
    i1 = min(size - 1, max(0, static_cast<int>(static_cast<unsigned>(b) + 1u)));
    w0 = 1.f - frac;
    w1 = frac;
}

struct DepositGeom {
    float lo[3], hi[3];
    int size[3];
};

// Where a deposit's grains come from: the simulation's slots (pos, vel with the mass in w),
// slots of a batch (their scene's grid, scale and nodes), or the caller's AoS6 states.
struct FromSlots {
    const float4* pos;
    const float4* vel;
    DepositGeom g;
    __device__ __forceinline__ float4 momentum(int s) const { return vel[s]; }   // vx vy vz m
    __device__ __forceinline__ float3 place(int s) const {
        const float4 p = pos[s];
        return make_float3(p.x, p.y, p.z);
    }
    __device__ __forceinline__ int scene(int) const { return 0; }
    __device__ __forceinline__ int count(int, int n) const { return n; }
    __device__ __forceinline__ DepositGeom geom(int) const { return g; }
    __device__ __forceinline__ int first_node(int) const { return 0; }
};
struct FromScenes {
    const float4* pos;
    const float4* vel;
    SceneTab T;
    __device__ __forceinline__ float4 momentum(int s) const { return vel[s]; }
    __device__ __forceinline__ float3 place(int s) const {
        const float4 p = pos[s];
        return make_float3(p.x, p.y, p.z);
    }
    __device__ __forceinline__ int scene(int s) const { return T.scene[s]; }
    __device__ __forceinline__ int count(int sc, int) const { return T.params[sc].n; }
    __device__ __forceinline__ DepositGeom geom(int sc) const {
        const DevParams& Q = T.params[sc];
        DepositGeom g;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            g.lo[a] = Q.lo[a];
            g.hi[a] = Q.hi[a];
            g.size[a] = Q.dgrid[a];
        }
        return g;
    }
    __device__ __forceinline__ int first_node(int sc) const { return T.params[sc].node_base; }
};
struct FromAos {
    const float* state;
    const float* mass;
    DepositGeom g;
    __device__ __forceinline__ float4 momentum(int s) const {
        const float* q = state + 6 * static_cast<int64_t>(s);
        return make_float4(q[3], q[4], q[5], mass[s]);
    }
    __device__ __forceinline__ float3 place(int s) const {
        const float* q = state + 6 * static_cast<int64_t>(s);
        return make_float3(q[0], q[1], q[2]);
    }
    __device__ __forceinline__ int scene(int) const { return 0; }
    __device__ __forceinline__ int count(int, int n) const { return n; }
    __device__ __forceinline__ DepositGeom geom(int) const { return g; }
    __device__ __forceinline__ int first_node(int) const { return 0; }
};

// Channel bounds: max |m| and max |m v_a| over grains, per scene (float bits; max of
// non-negative floats is order-independent). A grid of at most kBoundBlocks blocks: the
// maxima meet at four words per scene, and an atomic per warp of 10^6 grains on each took
// 84 us where one per block takes 7. Slots of a scene are consecutive, so a thread's
// grains change scene rarely; it hands its maxima over when they do.
constexpr int kBoundBlocks = 4 * 148;

template <class Src>
__global__ void __launch_bounds__(kBlock)
k_deposit_bounds(int n, Src src, uint32_t* __restrict__ bounds) {
    __shared__ uint32_t block_max[4];
    __shared__ int block_scene;
    const int per = (n + gridDim.x - 1) / gridDim.x;          // consecutive grains per block
    const int first = blockIdx.x * per, last = min(n, first + per);
    if (threadIdx.x < 4) block_max[threadIdx.x] = 0u;
    if (threadIdx.x == 0) block_scene = first < last ? src.scene(first) : 0;
    __syncthreads();
    uint32_t b[4] = {0u, 0u, 0u, 0u};
    int held = block_scene;
    auto hand_over = [&]() {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (b[c]) atomicMax(&bounds[4 * held + c], b[c]);
            b[c] = 0u;
        }
    };
    for (int s = first + static_cast<int>(threadIdx.x); s < last; s += blockDim.x) {
        const int sc = src.scene(s);
        if (sc != held) {
            hand_over();
            held = sc;
        }
        const float4 v = src.momentum(s);
        const float m = v.w;
        if (m != 0.f) {
            b[0] = max(b[0], __float_as_uint(fabsf(m)));
            b[1] = max(b[1], __float_as_uint(fabsf(m * v.x)));
            b[2] = max(b[2], __float_as_uint(fabsf(m * v.y)));
            b[3] = max(b[3], __float_as_uint(fabsf(m * v.z)));
        }
    }
    if (held != block_scene) hand_over();
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const uint32_t x = __reduce_max_sync(0xffffffffu, b[c]);
        if ((threadIdx.x & 31) == 0 && x) atomicMax(&block_max[c], x);
    }
    __syncthreads();
    if (threadIdx.x < 4 && block_max[threadIdx.x])
        atomicMax(&bounds[4 * block_scene + threadIdx.x], block_max[threadIdx.x]);
}

// Exponent k of the scale 2^k = 2^(62-e) with n * bound < 2^e, so that every partial sum
// stays below 2^62 (bound * n is a normal double, whose exponent field gives e).
__device__ __forceinline__ int scale_exponent(int n, uint32_t bound_bits) {
    const double b = static_cast<double>(__uint_as_float(bound_bits)) * static_cast<double>(n);
    if (!(b > 0.0) || !isfinite(b)) return 0;
    return 62 - (((__double2hiint(b) >> 20) & 0x7ff) - 1022);
}
__device__ __forceinline__ float exp2_float(int k) { return __int_as_float((k + 127) << 23); }   // |k| < 127
__device__ __forceinline__ double exp2_double(int k) { return __hiloint2double((k + 1023) << 20, 0); }

// One warp per kDepositGroup consecutive grains, 32 at a time. Each lane works out one
// grain's 32 contributions (8 corners, 4 channels) as integers and leaves them and the 8
// node indices in shared memory; then lane l takes corner l / 4, channel l % 4 of every
// grain in turn and adds up while its node stays the same, so that a node change costs one
// atomic per lane. The lanes of a node's channels, and of the two nodes adjacent in z, fall
// in one or two sectors of the node-major accumulators: 8 sector updates a grain where
// channel planes took 32, and fewer where consecutive grains share nodes.
// A contribution is float(m w) times a power of two, converted to int64: exact but for the
// conversion's own rounding, as the double product was (where the scaled value is too small
// for a normal float it rounds to zero in both). The power goes in two factors, since
// 2^k, k up to 211, need not be a float.
// Bound by the accumulators' sector updates. 1,000,003 grains onto 128^3 nodes in lattice
// order (no two neighbours on a node, the worst case): 77 us, with channel planes and a
// shuffle scan per corner 151; the finish 14 instead of 37, the bounds 8 instead of 84.
constexpr int kDepositWarps = 4;
constexpr int kDepositGroup = 128;

template <class Src>
__global__ void __launch_bounds__(32 * kDepositWarps)
k_deposit(int n, Src src, const uint32_t* __restrict__ bounds, unsigned long long* __restrict__ acc) {
    __shared__ long long val[kDepositWarps][32][33];
    __shared__ int node[kDepositWarps][32][9];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t first = (static_cast<int64_t>(blockIdx.x) * kDepositWarps + w) * kDepositGroup;
    const int corner = lane >> 2, channel = lane & 3;
    long long sum = 0;
    int cur = -1;
    for (int64_t base = first; base < min(first + kDepositGroup, static_cast<int64_t>(n)); base += 32) {
        const int s = static_cast<int>(base) + lane;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (s < n) v = src.momentum(s);
        const float m = v.w;
        if (m != 0.f) {
            const int sc = src.scene(s);
            const DepositGeom g = src.geom(sc);
            const int cnt = src.count(sc, n);
            const float3 x = src.place(s);
            float lo_f[4], hi_f[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int k = scale_exponent(cnt, bounds[4 * sc + c]);
                const int k1 = min(k, 126);
                lo_f[c] = exp2_float(k1);
                hi_f[c] = exp2_float(k - k1);
            }
            int ix[2], iy[2], iz[2];
            float wx[2], wy[2], wz[2];
            axis_weights(x.x, g.lo[0], g.hi[0], g.size[0], ix[0], ix[1], wx[0], wx[1]);
            axis_weights(x.y, g.lo[1], g.hi[1], g.size[1], iy[0], iy[1], wy[0], wy[1]);
            axis_weights(x.z, g.lo[2], g.hi[2], g.size[2], iz[0], iz[1], wz[0], wz[1]);
            const float part[4] = {m, m * v.x, m * v.y, m * v.z};
            const int nodes0 = src.first_node(sc);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int cx = k >> 2, cy = (k >> 1) & 1, cz = k & 1;
                const float wt = wx[cx] * wy[cy] * wz[cz];
                node[w][lane][k] = nodes0 + (ix[cx] * g.size[1] + iy[cy]) * g.size[2] + iz[cz];
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    val[w][lane][4 * k + c] =
                        wt != 0.f ? __float2ll_rn(((part[c] * wt) * lo_f[c]) * hi_f[c]) : 0ll;
            }
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) node[w][lane][k] = -1;
        }
        __syncwarp();
#pragma unroll 4
        for (int q = 0; q < 32; ++q) {
            const int nd = node[w][q][corner];
            if (nd < 0) continue;                     // no mass: the whole warp skips it
            if (nd != cur) {
                if (sum != 0)
                    atomicAdd(&acc[4 * static_cast<int64_t>(cur) + channel],
                              static_cast<unsigned long long>(sum));
                sum = 0;
                cur = nd;
            }
            sum += val[w][q][lane];
        }
        __syncwarp();
    }
    if (sum != 0)
        atomicAdd(&acc[4 * static_cast<int64_t>(cur) + channel], static_cast<unsigned long long>(sum));
}

// Node-major integers to the channel-major field, one node per thread.
__device__ __forceinline__ void finish_node(const unsigned long long* __restrict__ acc, int64_t at,
                                            int64_t nodes, int cnt, const uint32_t* __restrict__ bounds,
                                            float* __restrict__ out) {
    const ulonglong2* a = reinterpret_cast<const ulonglong2*>(acc + 4 * at);
    const ulonglong2 p = a[0], q = a[1];
    const unsigned long long v[4] = {p.x, p.y, q.x, q.y};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        // a NaN or infinite mass or momentum makes its whole channel NaN (the bound is the
        // largest |value| by its bits, so it is not finite exactly when some value is not)
        const bool fine = __uint_as_float(bounds[c]) <= FLT_MAX;
        const double inv = exp2_double(-scale_exponent(cnt, bounds[c]));
        out[c * nodes] = fine ? static_cast<float>(static_cast<double>(static_cast<long long>(v[c])) * inv)
                              : __uint_as_float(0x7fc00000u);
    }
}

__global__ void __launch_bounds__(kBlock)
k_deposit_finish(int n, int nodes, const uint32_t* __restrict__ bounds,
                 const unsigned long long* __restrict__ acc, float* __restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < nodes) finish_node(acc, t, nodes, n, bounds, out + t);
}

// Batched scenes: one field per scene, laid out scene after scene
// ([scene][4][nodes of that scene]), each with its own scale.
__global__ void __launch_bounds__(kBlock)
k_deposit_finish_batch(const DevParams* __restrict__ params, int scenes, int total,
                       const uint32_t* __restrict__ bounds,
                       const unsigned long long* __restrict__ acc, float* __restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    int lo = 0, hi = scenes;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (params[mid].node_base <= t) lo = mid; else hi = mid;
    }
    const DevParams& Q = params[lo];
    const int64_t nodes = static_cast<int64_t>(Q.dgrid[0]) * Q.dgrid[1] * Q.dgrid[2];
    finish_node(acc, t, nodes, Q.n, bounds + 4 * lo,
                out + 4 * static_cast<int64_t>(Q.node_base) + (t - Q.node_base));
}

template <class Src>
void launch_sums(int n, const Src& src, uint32_t* bounds, unsigned long long* acc, cudaStream_t st) {
    if (n <= 0) return;
    k_deposit_bounds<<<std::min(blocks_for(n), kBoundBlocks), kBlock, 0, st>>>(n, src, bounds);
    constexpr int per = kDepositWarps * kDepositGroup;
    k_deposit<<<(n - 1) / per + 1, 32 * kDepositWarps, 0, st>>>(n, src, bounds, acc);
}

}  // namespace

void launch_deposit(int n, const float4* pos, const float4* vel, const float* lo,
                    const float* hi, const int* dgrid, uint32_t* bounds,
                    unsigned long long* acc, float* out, cudaStream_t st) {
    DepositGeom g;
    for (int a = 0; a < 3; ++a) {
        g.lo[a] = lo[a];
        g.hi[a] = hi[a];
        g.size[a] = dgrid[a];
    }
    const int64_t nodes = static_cast<int64_t>(dgrid[0]) * dgrid[1] * dgrid[2];
    cudaMemsetAsync(bounds, 0, 4 * sizeof(uint32_t), st);
    cudaMemsetAsync(acc, 0, 4 * nodes * sizeof(unsigned long long), st);
    launch_sums(n, FromSlots{pos, vel, g}, bounds, acc, st);
    k_deposit_finish<<<blocks_for(nodes), kBlock, 0, st>>>(n, static_cast<int>(nodes), bounds, acc, out);
}

void launch_deposit_batch(int n, const float4* pos, const float4* vel, SceneTab T, int scenes,
                          int64_t total_nodes, uint32_t* bounds, unsigned long long* acc,
                          float* out, cudaStream_t st) {
    cudaMemsetAsync(bounds, 0, 4 * sizeof(uint32_t) * static_cast<size_t>(scenes), st);
    cudaMemsetAsync(acc, 0, 4 * total_nodes * sizeof(unsigned long long), st);
    launch_sums(n, FromScenes{pos, vel, T}, bounds, acc, st);
    k_deposit_finish_batch<<<blocks_for(total_nodes), kBlock, 0, st>>>(
        T.params, scenes, static_cast<int>(total_nodes), bounds, acc, out);
}

}  // namespace wd

// ---------------------------------------------------------------------------------
// Allocation-free variant of the deposit for callers that cannot call cudaMalloc
// (device memory owned by another framework's allocator, or a loop that must not
// allocate). Inputs are the caller's own device arrays in the reference's AoS
// layout; the scratch is the static array below, one per device, never freed.
// ---------------------------------------------------------------------------------
#include <string>

#include "../../include/world_b200.h"
#include "wd_config.h"

namespace {

constexpr long long kNoAllocNodes = WD_NOALLOC_MAX_NODES;
// 4 channels of 64-bit accumulators, then 2 words holding the four 32-bit bounds.
static __device__ __align__(256) unsigned long long g_deposit_scratch[4 * kNoAllocNodes + 2];


// Device address of the scratch array in the current device's context. Looked up on
// every call (a host-side table lookup, no allocation and no device work), so the
// address stays right after a cudaDeviceReset or when another context is made current.
cudaError_t scratch_for_current_device(unsigned long long** out) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_deposit_scratch);
    if (e != cudaSuccess) return e;
    *out = static_cast<unsigned long long*>(p);
    return cudaSuccess;
}

}  // namespace

extern "C" int wd_deposit_grid_noalloc(const float* d_state, const float* d_mass, int64_t n,
                                       const float* lo3, const float* hi3, const int32_t* size3,
                                       float* d_grid, void* stream_v) {
    if (!lo3 || !hi3 || !size3 || !d_grid || (n > 0 && (!d_state || !d_mass))) {
        wd::set_last_error("wd_deposit_grid_noalloc: NULL argument");
        return WD_ERR_INVALID;
    }
    if (n < 0 || n > (int64_t{1} << 30)) {
        wd::set_last_error("wd_deposit_grid_noalloc: grain count must be in [0, 2^30]");
        return WD_ERR_INVALID;
    }
    for (int a = 0; a < 3; ++a) {
        if (size3[a] < 1) {
            wd::set_last_error("wd_deposit_grid_noalloc: grid sizes must be >= 1");
            return WD_ERR_INVALID;
        }
    }
    const int64_t nodes = static_cast<int64_t>(size3[0]) * size3[1] * size3[2];
    if (nodes > kNoAllocNodes) {
        wd::set_last_error("wd_deposit_grid_noalloc: grid of " + std::to_string(nodes) +
                           " nodes exceeds the fixed scratch of " +
                           std::to_string(kNoAllocNodes) + " nodes (64^3)");
        return WD_ERR_CAPACITY;
    }
    unsigned long long* scratch = nullptr;
    cudaError_t e = scratch_for_current_device(&scratch);
    if (e != cudaSuccess) {
        wd::set_last_error(std::string("wd_deposit_grid_noalloc: cudaGetSymbolAddress: ") +
                           cudaGetErrorString(e));
        return WD_ERR_CUDA;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream_v);
    unsigned long long* acc = scratch;
    uint32_t* bounds = reinterpret_cast<uint32_t*>(scratch + 4 * kNoAllocNodes);
    wd::DepositGeom g;
    for (int a = 0; a < 3; ++a) {
        g.lo[a] = lo3[a];
        g.hi[a] = hi3[a];
        g.size[a] = size3[a];
    }
    // the array keeps the previous call's sums: clear what this call reads
    e = cudaMemsetAsync(bounds, 0, 4 * sizeof(uint32_t), st);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(acc, 0, static_cast<size_t>(4 * nodes) * sizeof(unsigned long long), st);
    if (e == cudaSuccess && n > 0) {
        // the same contributions and scale as the simulation's own deposit
        wd::launch_sums(static_cast<int>(n), wd::FromAos{d_state, d_mass, g}, bounds, acc, st);
    }
    if (e == cudaSuccess) {
        wd::k_deposit_finish<<<wd::blocks_for(nodes), wd::kBlock, 0, st>>>(
            static_cast<int>(n), static_cast<int>(nodes), bounds, acc, d_grid);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        wd::set_last_error(std::string("wd_deposit_grid_noalloc: ") + cudaGetErrorString(e));
        return WD_ERR_CUDA;
    }
    return WD_OK;
}
