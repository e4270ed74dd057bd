// wd_adjoint.cu -- reverse pass of the semi-implicit Euler step, and of the CIC deposit.
//
// Step t maps (x, v, springs) to (x', v', springs'): F from the contacts, then
// v' = v + dt F / m and x' = x + dt v' (src/semi_implicit_euler_kernel.cu:4-16). Given
// the adjoints (lx', lv', lxi') of step t's outputs, k_adj_step returns those of its
// inputs and adds the step's share of dL/d(mu, ln e, k_n):
//   lvt = lv' + dt lx',  lF = dt / m lvt,
//   lx = lx' + sum over contacts J_x^T [lF-side; lxi-side],  lv = lvt + sum J_v^T [...].
// A pair force and its new spring are odd in (d, v_rel, xi) with d = x_i - x_j, and the
// two grains keep mirrored copies of the spring, so grain i alone can apply the pair's
// whole contribution to its own adjoints: with respect to d and v_rel the weights are
// (lF_i - lF_j, lxi'_ij - lxi'_ji); with respect to i's stored spring and the parameters
// they are (lF_i, lxi'_ij). Every grain gathers; nothing is scattered.
//
// The contact set, clamp, slip and viscous-cap branches are those of the forward step
// (wd_adjoint.cuh evaluates the laws with the forward's own float operations).
#include "wd_adjoint.cuh"
#include "wd_kernels.h"

namespace wd {
namespace {

__device__ __forceinline__ float3 f3(float4 a) { return make_float3(a.x, a.y, a.z); }

template <class S>
__device__ __forceinline__ Theta<S> make_theta(const DevParams& P, int kt_from_kn, int seed_block) {
    Theta<S> th;
    th.mu = lift<S>(P.mu);
    th.L = lift<S>(P.ln_e);
    th.k = lift<S>(P.k_n);
    if (seed_block) {
        th.mu = dseed<3>(P.mu, 0);
        th.L = dseed<3>(P.ln_e, 1);
        th.k = dseed<3>(P.k_n, 2);
    }
    th.kt = kt_from_kn ? lift<S>(2.f / 7.f) * th.k : lift<S>(P.k_t);
    return th;
}

// Row search: index of partner in a spring row, -1 if absent (first match, as the
// forward's lookup).
__device__ __forceinline__ int row_find(const float4* row, int count, int partner) {
    for (int k = 0; k < count; ++k)
        if (__float_as_int(row[k].w) == partner) return k;
    return -1;
}

// Weighted sums of one Jacobian block: out[c] += sum_o J_f[o][c] wf[o] + J_xi[o][c] wxi[o].
__device__ __forceinline__ void vjp_add(const ContactOut<Dual<3>>& o, float3 wf, float3 wx,
                                        float out[3]) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
        out[c] += o.f[0].d[c] * wf.x + o.f[1].d[c] * wf.y + o.f[2].d[c] * wf.z +
                  o.xi[0].d[c] * wx.x + o.xi[1].d[c] * wx.y + o.xi[2].d[c] * wx.z;
}

using D3 = Dual<3>;

template <bool HIST>
__device__ __forceinline__ void wall_blocks(const DevParams& P, const AdjArgs& A, float3 x,
                                            float3 v, float3 xi, float ri, float mi, int a,
                                            bool upper, float3 wf, float3 wx, float ax[3],
                                            float av[3], float axi[3], double th[3]) {
    const float xv[3] = {x.x, x.y, x.z}, vv[3] = {v.x, v.y, v.z}, sv[3] = {xi.x, xi.y, xi.z};
    const Theta<D3> th0 = make_theta<D3>(P, A.kt_from_kn, 0);
    for (int blk = 0; blk < 4; ++blk) {
        D3 xd[3], vd[3], sd[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            xd[c] = dseed<3>(xv[c], blk == 0 ? c : -1);
            vd[c] = dseed<3>(vv[c], blk == 1 ? c : -1);
            sd[c] = dseed<3>(sv[c], blk == 2 ? c : -1);
        }
        const Theta<D3> tt = blk == 3 ? make_theta<D3>(P, A.kt_from_kn, 1) : th0;
        ContactOut<D3> o;
        wall_t<D3, HIST>(P, tt, xd, vd, sd, ri, mi, a, upper, o);
        if (blk == 0) vjp_add(o, wf, wx, ax);
        else if (blk == 1) vjp_add(o, wf, wx, av);
        else if (blk == 2) vjp_add(o, wf, wx, axi);
        else {
            float t[3] = {0.f, 0.f, 0.f};
            vjp_add(o, wf, wx, t);
#pragma unroll
            for (int c = 0; c < 3; ++c) th[c] += t[c];
        }
    }
}

// lvt = lv' + dt lx' and lF = dt / m lvt of one grain of mass m.
__device__ __forceinline__ float3 force_adjoint(float dt, float m, float4 x, float4 v, float3* lvt) {
    const float3 t = make_float3(fmaf(dt, x.x, v.x), fmaf(dt, x.y, v.y), fmaf(dt, x.z, v.z));
    if (lvt) *lvt = t;
    const float g = m != 0.f ? dt / m : 0.f;
    return make_float3(g * t.x, g * t.y, g * t.z);
}

// One step back. A warp's contacts are numbered grain by grain and taken 32 at a time: first
// a lane each looks one up (geometry, springs, adjoints of both grains), then four lanes
// each evaluate one, a block of three inputs per lane (position, velocity, stored spring,
// parameters), 8 contacts at a time; last, each grain's lane adds its own in order. (A lane
// that evaluates its grain's contacts alone runs the four long passes once per contact of
// the busiest of its 32 grains.) Every entry of the input's spring rows is written: zero, or
// the contact's. Bound by the latency of the dual arithmetic's chains.
constexpr int kAdjBlock = 128;

struct AdjWarp {
    float geo[9][32];        // d, v_rel, stored spring
    float w[12][32];         // relative and own weights: force, spring, each
    float rj[32], mj[32];
    int k_in[32];            // the stored spring's place in the owner's row, or -1
    int queue[32];           // owner lane << 8 | contact
    float out[32][13];
    float ri[32], mi[32], lf[3][32];
    int id[32], rows[32], walls[32];
};

template <bool HIST>
__global__ void __launch_bounds__(kAdjBlock)
k_adj_step(DevParams P, AdjArgs A) {
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ AdjWarp warps[kAdjBlock / 32];
    AdjWarp& W = warps[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int s = blockIdx.x * kAdjBlock + static_cast<int>(threadIdx.x);
    const int s0 = s - lane;                 // the warp's first slot
    const bool live = s < P.n;
    float4 pi = make_float4(0.f, 0.f, 0.f, 0.f), vi = pi, lx = pi;
    float3 lvt = make_float3(0.f, 0.f, 0.f), lf_i = lvt;
    int id = 0, in_count = 0, nc = 0, out_count = 0;
    float ax[3] = {0.f, 0.f, 0.f}, av[3] = {0.f, 0.f, 0.f};
    double th[3] = {0.0, 0.0, 0.0};
    if (live) {
        pi = A.pos[s];
        vi = A.vel[s];
        id = A.ids[s];
        nc = A.ccnt[s];
        lx = A.lx[id];
        lf_i = force_adjoint(P.dt, vi.w, lx, A.lv[id], &lvt);
        const float4* in_row = HIST ? A.hist_in + static_cast<int64_t>(id) * kHistCap : nullptr;
        if (HIST) {
            in_count = A.hcnt_in[s];
            for (int k = 0; k < in_count; ++k)
                A.lxi_out[static_cast<int64_t>(id) * kHistCap + k] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        // walls, in the forward's order: axis 0 lower, upper, axis 1, axis 2
        const float p3[3] = {pi.x, pi.y, pi.z};
        for (int a = 0; a < 3; ++a) {
            for (int up = 0; up < 2; ++up) {
                const float dl = up ? (P.wall_hi[a] - p3[a]) - pi.w : (p3[a] - P.wall_lo[a]) - pi.w;
                if (!(dl < 0.f)) continue;
                const int partner = up ? -2 - 2 * a : -1 - 2 * a;
                float3 xi = make_float3(0.f, 0.f, 0.f), lxi_own = xi;
                int k_in = -1;
                if (HIST) {
                    k_in = row_find(in_row, in_count, partner);
                    if (k_in >= 0) xi = f3(in_row[k_in]);
                    if (out_count < kHistCap)
                        lxi_own = f3(A.lxi[static_cast<int64_t>(id) * kHistCap + out_count]);
                    ++out_count;
                }
                float axi[3] = {0.f, 0.f, 0.f};
                wall_blocks<HIST>(P, A, f3(pi), f3(vi), xi, pi.w, vi.w, a, up != 0, lf_i, lxi_own, ax, av, axi, th);
                if (HIST && k_in >= 0)
                    A.lxi_out[static_cast<int64_t>(id) * kHistCap + k_in] =
                        make_float4(axi[0], axi[1], axi[2], 0.f);
            }
        }
    }
    W.ri[lane] = pi.w;
    W.mi[lane] = vi.w;
    W.lf[0][lane] = lf_i.x;
    W.lf[1][lane] = lf_i.y;
    W.lf[2][lane] = lf_i.z;
    W.id[lane] = id;
    W.rows[lane] = in_count;
    W.walls[lane] = out_count;
    int upto = nc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kAll, upto, o);
        if (lane >= o) upto += y;
    }
    const int off = upto - nc;
    const int total = __shfl_sync(kAll, upto, 31);
    for (int base = 0; base < total; base += 32) {
        const int cnt = min(32, total - base);
        for (int q = max(off, base); q < min(upto, base + 32); ++q) W.queue[q - base] = (lane << 8) | (q - off);
        __syncwarp();
        if (lane < cnt) {
            const int o = W.queue[lane] >> 8, e = W.queue[lane] & 255, so = s0 + o;
            const int j = A.clist[static_cast<int64_t>(e) * P.n + so];
            const float4 po = A.pos[so], vo = A.vel[so], pj = A.pos[j], vj = A.vel[j];
            float3 d;
            pair_norm_sq(po, pj, d);
            const int jd = A.ids[j], io = W.id[o];
            const float3 lf_j = force_adjoint(P.dt, vj.w, A.lx[jd], A.lv[jd], nullptr);
            float3 xi = make_float3(0.f, 0.f, 0.f), lxi_ij = xi, lxi_ji = xi;
            int k_in = -1;
            if (HIST) {
                const float4* row = A.hist_in + static_cast<int64_t>(io) * kHistCap;
                k_in = row_find(row, W.rows[o], jd);
                if (k_in >= 0) xi = f3(row[k_in]);
                const int at = W.walls[o] + e;
                if (at < kHistCap) lxi_ij = f3(A.lxi[static_cast<int64_t>(io) * kHistCap + at]);
                const int kj = row_find(A.hist_next + static_cast<int64_t>(jd) * kHistCap, A.hcnt_next[jd], io);
                if (kj >= 0) lxi_ji = f3(A.lxi[static_cast<int64_t>(jd) * kHistCap + kj]);
            }
            const float geo[9] = {d.x, d.y, d.z, vo.x - vj.x, vo.y - vj.y, vo.z - vj.z, xi.x, xi.y, xi.z};
            const float own[3] = {W.lf[0][o], W.lf[1][o], W.lf[2][o]};
            const float w[12] = {own[0] - lf_j.x, own[1] - lf_j.y, own[2] - lf_j.z,
                                 lxi_ij.x - lxi_ji.x, lxi_ij.y - lxi_ji.y, lxi_ij.z - lxi_ji.z,
                                 own[0], own[1], own[2], lxi_ij.x, lxi_ij.y, lxi_ij.z};
#pragma unroll
            for (int k = 0; k < 9; ++k) W.geo[k][lane] = geo[k];
#pragma unroll
            for (int k = 0; k < 12; ++k) W.w[k][lane] = w[k];
            W.rj[lane] = pj.w;
            W.mj[lane] = vj.w;
            W.k_in[lane] = k_in;
        }
        __syncwarp();
        const int blk = lane & 3;
        for (int c = lane >> 2; c < cnt; c += 8) {
            const int o = W.queue[c] >> 8;
            D3 dd[3], vd[3], xd[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                dd[k] = dseed<3>(W.geo[k][c], blk == 0 ? k : -1);
                vd[k] = dseed<3>(W.geo[3 + k][c], blk == 1 ? k : -1);
                xd[k] = dseed<3>(W.geo[6 + k][c], blk == 2 ? k : -1);
            }
            const Theta<D3> tt = make_theta<D3>(P, A.kt_from_kn, blk == 3);
            ContactOut<D3> r;
            pair_t<D3, HIST>(P, tt, dd, vd, xd, W.ri[o], W.rj[c], W.mi[o], W.mj[c], r);
            const int u = blk < 2 ? 0 : 6;     // relative weights for d and v_rel, own for the rest
            float t[3] = {0.f, 0.f, 0.f};
            vjp_add(r, make_float3(W.w[u][c], W.w[u + 1][c], W.w[u + 2][c]),
                    make_float3(W.w[u + 3][c], W.w[u + 4][c], W.w[u + 5][c]), t);
#pragma unroll
            for (int k = 0; k < 3; ++k) W.out[c][3 * blk + k] = t[k];
            if (HIST && blk == 2 && W.k_in[c] >= 0)
                A.lxi_out[static_cast<int64_t>(W.id[o]) * kHistCap + W.k_in[c]] =
                    make_float4(t[0], t[1], t[2], 0.f);
        }
        __syncwarp();
        for (int q = max(off, base); q < min(upto, base + 32); ++q) {
            const float* r = W.out[q - base];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                ax[k] += r[k];
                av[k] += r[3 + k];
                th[k] += r[9 + k];
            }
        }
        __syncwarp();                        // the records are free again
    }
    if (!live) return;
    A.lx_out[id] = make_float4(lx.x + ax[0], lx.y + ax[1], lx.z + ax[2], 0.f);
    A.lv_out[id] = make_float4(lvt.x + av[0], lvt.y + av[1], lvt.z + av[2], 0.f);
#pragma unroll
    for (int c = 0; c < 3; ++c) A.theta[static_cast<int64_t>(c) * P.n + id] += th[c];
}

// Counts of a spring snapshot by grain id (snapshots keep them by sorted slot).
__global__ void __launch_bounds__(kBlock)
k_counts_by_id(int n, const int* __restrict__ ids, const int* __restrict__ cnt_slot,
               int* __restrict__ cnt_id) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n) cnt_id[ids[s]] = cnt_slot[s];
}

// reference src/density_grid_kernel.cu:25-40 with d(frac)/dx = 1/h.
__device__ __forceinline__ void axis_weights_d(float x, float lo, float hi, int size, int& i0,
                                               int& i1, float& w0, float& w1, float& dw) {
    if (size <= 1) {
        i0 = 0; i1 = 0; w0 = 1.f; w1 = 0.f; dw = 0.f;
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
    dw = 1.f / h;
}

// Adjoint of the CIC deposit at the current state: for node weights w(x) and
// contributions m w, m v_a w, gx = sum_corners dw/dx (m G0 + m v.G_mom), gv_a = sum w m G_a.
__global__ void __launch_bounds__(kBlock)
k_deposit_vjp(int n, const float4* __restrict__ pos, const float4* __restrict__ vel,
              const int* __restrict__ ids, float lo0, float lo1, float lo2, float hi0, float hi1,
              float hi2, int sx, int sy, int sz, const float* __restrict__ g,
              float4* __restrict__ gx, float4* __restrict__ gv) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const float4 x = pos[s], v = vel[s];
    const int id = ids[s];
    const float m = v.w;
    float ax[3] = {0.f, 0.f, 0.f}, av[3] = {0.f, 0.f, 0.f};
    if (m != 0.f) {
        int ix[2], iy[2], iz[2];
        float wx[2], wy[2], wz[2], dx, dy, dz;
        axis_weights_d(x.x, lo0, hi0, sx, ix[0], ix[1], wx[0], wx[1], dx);
        axis_weights_d(x.y, lo1, hi1, sy, iy[0], iy[1], wy[0], wy[1], dy);
        axis_weights_d(x.z, lo2, hi2, sz, iz[0], iz[1], wz[0], wz[1], dz);
        const float sgn[2] = {-1.f, 1.f};
        const int64_t nodes = static_cast<int64_t>(sx) * sy * sz;
        for (int cx = 0; cx < 2; ++cx)
            for (int cy = 0; cy < 2; ++cy)
                for (int cz = 0; cz < 2; ++cz) {
                    const int64_t node = (static_cast<int64_t>(ix[cx]) * sy + iy[cy]) * sz + iz[cz];
                    const float g0 = g[node], g1 = g[nodes + node], g2 = g[2 * nodes + node],
                                g3 = g[3 * nodes + node];
                    const float w = wx[cx] * wy[cy] * wz[cz];
                    const float val = m * (g0 + v.x * g1 + v.y * g2 + v.z * g3);
                    ax[0] += sgn[cx] * dx * wy[cy] * wz[cz] * val;
                    ax[1] += sgn[cy] * dy * wx[cx] * wz[cz] * val;
                    ax[2] += sgn[cz] * dz * wx[cx] * wy[cy] * val;
                    av[0] += w * m * g1;
                    av[1] += w * m * g2;
                    av[2] += w * m * g3;
                }
    }
    gx[id] = make_float4(ax[0], ax[1], ax[2], 0.f);
    gv[id] = make_float4(av[0], av[1], av[2], 0.f);
}

}  // namespace

void launch_adj_step(const DevParams& P, const AdjArgs& a, cudaStream_t st) {
    const int nb = blocks_for(P.n, kAdjBlock);
    if (P.history) k_adj_step<true><<<nb, kAdjBlock, 0, st>>>(P, a);
    else k_adj_step<false><<<nb, kAdjBlock, 0, st>>>(P, a);
}

void launch_counts_by_id(int n, const int* ids, const int* cnt_slot, int* cnt_id, cudaStream_t st) {
    k_counts_by_id<<<blocks_for(n), kBlock, 0, st>>>(n, ids, cnt_slot, cnt_id);
}

void launch_deposit_vjp(int n, const float4* pos, const float4* vel, const int* ids,
                        const float* lo, const float* hi, const int* size, const float* g,
                        float4* gx, float4* gv, cudaStream_t st) {
    k_deposit_vjp<<<blocks_for(n), kBlock, 0, st>>>(n, pos, vel, ids, lo[0], lo[1], lo[2], hi[0],
                                                    hi[1], hi[2], size[0], size[1], size[2], g,
                                                    gx, gv);
}

}  // namespace wd

namespace wd {
namespace {

__global__ void __launch_bounds__(kBlock)
k_aos3_to_f4(int n, const float* __restrict__ a, float4* __restrict__ o) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    o[i] = a ? make_float4(a[3 * static_cast<int64_t>(i)], a[3 * static_cast<int64_t>(i) + 1],
                           a[3 * static_cast<int64_t>(i) + 2], 0.f)
             : make_float4(0.f, 0.f, 0.f, 0.f);
}

__global__ void __launch_bounds__(kBlock)
k_f4_to_aos3(int n, const float4* __restrict__ a, float* __restrict__ o) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 v = a[i];
    o[3 * static_cast<int64_t>(i)] = v.x;
    o[3 * static_cast<int64_t>(i) + 1] = v.y;
    o[3 * static_cast<int64_t>(i) + 2] = v.z;
}

}  // namespace

void launch_aos3_to_f4(int n, const float* a, float4* o, cudaStream_t st) {
    k_aos3_to_f4<<<blocks_for(n), kBlock, 0, st>>>(n, a, o);
}

void launch_f4_to_aos3(int n, const float4* a, float* o, cudaStream_t st) {
    k_f4_to_aos3<<<blocks_for(n), kBlock, 0, st>>>(n, a, o);
}

}  // namespace wd
