// wd_contact.cu -- fused contact force + integrator, and the FP64 energy reduction.
//
// Grains in (cell, id) order. A grain's candidates lie in the 9 neighbor columns of its
// cell; the three z-cells of each column are consecutive runs of the sorted arrays, so the
// candidates of a column are one contiguous slot range read straight from the sorted SoA
// (float4 position+radius, float4 velocity+mass). Each grain's force is summed by its own
// thread: no force atomics and a fixed summation order (stencil order, ids ascending
// inside a cell), hence bit-reproducible steps.
//
// Physics per contact: reference src/compute_rhs_kernel.cu:81-212 (gravity, six
// walls, clamped linear spring, normal dashpot from restitution, Coulomb-capped
// friction), generalised to per-grain radius and mass, with the tangential spring
// and its per-pair history as an option. The integrator runs in the epilogue:
// semi-implicit Euler (src/semi_implicit_euler_kernel.cu:4-16) or one backward
// Euler / Picard update from the step-start snapshot
// (src/backward_euler_picard_kernel.cu:4-17).
#include "wd_kernels.h"

namespace wd {

namespace {

__device__ __forceinline__ bool skipped(const Skip& s) {
    return s.prev_res != nullptr && s.tol > 0.f && __uint_as_float(*s.prev_res) < s.tol;
}

// Force kernel of a searched step. A warp finds the contacts of its 32 / LPG grains, in the
// canonical order, and its lanes then evaluate those contacts together, one each; every
// grain adds its own contacts' terms in order. (A lane that walks its grain's cells and
// evaluates each contact on the way holds its 31 neighbours up: 2.2 thousand warp
// instructions per 32 packed grains, about a third of the lanes active.)
//
// LPG lanes search for one grain: with one lane, row by row through the nine rows of three
// z cells; with more, the rows' slot ranges go to shared memory and the lanes walk the
// candidates as one sequence, LPG apart and four each at a time. A grain with more contacts
// than its buffer holds takes them all on its own lane.
// Bound by load latency and issue; see launch_force for the lanes and what they measured.
constexpr int kForceBlock = 128;
constexpr int kForceHits = 16;              // LPG 1; more lanes share the same buffer

template <int LPG>
struct ForceWarp {
    static constexpr int kGrains = 32 / LPG;
    static constexpr int kCap = LPG == 1 ? kForceHits : 32;
    float4 term[32][2];                     // (nrm, fp), (t, cvn)
    int hit[kCap][kGrains];                 // contacts' slots
    int2 rows[LPG > 1 ? 9 : 1][kGrains];
    unsigned short queue[32];               // owner lane << 8 | contact
};

// Contacts of a grain beyond its buffer: the walk again, each contact as it comes.
template <bool HIST>
__device__ __forceinline__ void force_walk(const DevParams& P, const ForceArgs& A, int s, float4 pi,
                                           float3 vel, float mi, int cx, int cy, int cz, float3& f,
                                           HistRow& h) {
    const float cut = contact_cutoff_sq(pi.w, P.rmax);
    for (int dx = -1; dx <= 1; ++dx) {
        const int nx = cx + dx;
        if (nx < 0 || nx >= P.grid[0]) continue;
        int lo[3], hi[3];
        row_ranges(P, A.table, nx, cy, cz, lo, hi);
        for (int t = 0; t < 3; ++t) {
            for (int j = lo[t]; j < hi[t]; ++j) {
                const float4 pj = __ldg(&A.pos[j]);
                float3 d;
                const float ns = pair_norm_sq(pi, pj, d);
                if (ns > cut || j == s) continue;
                const float norm = sqrtf(ns);
                const float dist = pair_dist(norm, pi.w, pj.w);
                if (!(dist < 0.f)) continue;
                const float4 vj = __ldg(&A.vel[j]);
                const int partner = HIST ? __ldg(&A.ids[j]) : 0;
                pair_force<HIST>(P, d, norm, dist, vel, mi, vj, partner, f, h, A.counters);
            }
        }
    }
}

// REC: also note down the contacts, for the reverse pass.
template <bool HIST, bool PICARD, bool BATCH, bool REC, int LPG>
__global__ void __launch_bounds__(kForceBlock, 8)
k_force(DevParams P0, ForceArgs A, Skip skip) {
    if (skipped(skip)) return;
    using Warp = ForceWarp<LPG>;
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ Warp warps[kForceBlock / 32];
    Warp& W = warps[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, sub = lane % LPG, g = lane / LPG;
    const int s = (blockIdx.x * kForceBlock + static_cast<int>(threadIdx.x)) / LPG;
    const int s0 = (blockIdx.x * kForceBlock + static_cast<int>(threadIdx.x) - lane) / LPG;
    const bool live = s < P0.n;
    uint32_t res_bits = 0u;
    int scene = 0, id = 0;
    float4 pi = make_float4(0.f, 0.f, 0.f, 0.f), vi = pi;
    if (live) {
        scene = BATCH ? A.scene[s] : 0;
        pi = A.pos[s];
        vi = A.vel[s];
        id = A.ids[s];
    }
    const DevParams& P = BATCH ? A.scene_params[scene] : P0;
    const bool frozen = BATCH && live && P.frozen;
    const bool search = live && !frozen, work = search && sub == 0;
    const float3 vel = make_float3(vi.x, vi.y, vi.z);
    const float ri = pi.w, mi = vi.w;
    float3 f = make_float3(0.f, 0.f, 0.f);
    HistRow h;
    h.out_count = 0;
    if (work) {
        if (HIST) {
            h.in = A.hist_in + static_cast<int64_t>(id) * kHistCap;
            h.in_count = A.hcnt_in[s];
            h.out = A.hist_out + static_cast<int64_t>(id) * kHistCap;
            if (REC) A.rec_hcnt[id] = h.in_count;
        }
        wall_forces<HIST>(P, make_float3(pi.x, pi.y, pi.z), vel, ri, mi, f, h, A.counters);
    }
    const int out_walls = HIST ? h.out_count : 0;

    // the contacts, in order
    int cx = 0, cy = 0, cz = 0;
    if (search) cell_coords(P, pi.x, pi.y, pi.z, cx, cy, cz);
    int found = 0;
    auto touches = [&](int j, float4 pj) {
        float3 d;
        const float ns = pair_norm_sq(pi, pj, d);
        return maybe_contact(ns, ri, pj.w) && j != s && pair_dist(sqrtf(ns), ri, pj.w) < 0.f;
    };
    if (LPG == 1) {
        auto visit = [&](int j, float4 pj) {
            if (!touches(j, pj)) return;
            if (found < Warp::kCap) W.hit[found][g] = j;
            if (REC && found < kAdjContacts) A.rec_list[static_cast<int64_t>(found) * P0.n + s] = j;
            ++found;
        };
        for (int dx = -1; dx <= 1; ++dx) {
            const int nx = cx + dx;
            if (!search || nx < 0 || nx >= P.grid[0]) continue;
            int lo[3], hi[3];
            row_ranges(P, A.table, nx, cy, cz, lo, hi);
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                int j = lo[t];
                // an empty row has lo = INT_MAX, hi = 0: the difference does not overflow
                for (; hi[t] - j > 1; j += 2) {
                    const float4 p0 = __ldg(&A.pos[j]), p1 = __ldg(&A.pos[j + 1]);
                    visit(j, p0);
                    visit(j + 1, p1);
                }
                if (j < hi[t]) visit(j, __ldg(&A.pos[j]));
            }
        }
    } else {
        for (int q = sub; q < 9; q += LPG) {
            const int nx = cx + q / 3 - 1, ny = cy + q % 3 - 1;
            int lo = 0, hi = 0;
            if (search && nx >= 0 && nx < P.grid[0] && ny >= 0 && ny < P.grid[1])
                column_range(P, A.table, nx, ny, cz, lo, hi);
            W.rows[q][g] = lo < hi ? make_int2(lo, hi) : make_int2(0, 0);
        }
        __syncwarp();
        int r = -1, j = sub, hi = 0;
        for (;;) {
            int jj[4];
            float4 pp[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                while (j >= hi && r < 9) {
                    const int over = j - hi;      // how far into the next row
                    if (++r < 9) {
                        const int2 q = W.rows[r][g];
                        j = q.x + over;
                        hi = q.y;
                    }
                }
                jj[u] = r < 9 ? j : -1;
                j += LPG;
            }
            if (!__any_sync(kAll, jj[0] >= 0)) break;
#pragma unroll
            for (int u = 0; u < 4; ++u) pp[u] = jj[u] >= 0 ? __ldg(&A.pos[jj[u]]) : pi;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool hit = jj[u] >= 0 && touches(jj[u], pp[u]);
                // the group's lanes hold consecutive candidates
                const unsigned mine = (__ballot_sync(kAll, hit) >> (lane - sub)) & (kAll >> (32 - LPG));
                const int at = found + __popc(mine & ((1u << sub) - 1u));
                found += __popc(mine);
                if (hit && at < Warp::kCap) W.hit[at][g] = jj[u];
                if (REC && hit && at < kAdjContacts) A.rec_list[static_cast<int64_t>(at) * P0.n + s] = jj[u];
            }
        }
        __syncwarp();
    }
    if (REC && work) {
        A.rec_cnt[s] = min(found, kAdjContacts);
        if (found > kAdjContacts) atomicAdd(A.rec_over, 1ull);
    }
    if (found > Warp::kCap) {
        if (work) force_walk<HIST>(P, A, s, pi, vel, mi, cx, cy, cz, f, h);
        found = 0;
    }
    if (__any_sync(kAll, found > 0)) {
        // number the warp's contacts, grain by grain
        int upto = sub == 0 ? found : 0;
#pragma unroll
        for (int o = LPG; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kAll, upto, o);
            if (lane >= o) upto += y;
        }
        if (LPG > 1) upto = __shfl_sync(kAll, upto, lane - sub);
        const int off = upto - found;
        const int total = __shfl_sync(kAll, upto, 31);
        int at = off;
        for (int base = 0; base < total; base += 32) {
            if (sub == 0)
                for (; at < min(upto, base + 32); ++at)
                    W.queue[at - base] = static_cast<unsigned short>((lane << 8) | (at - off));
            __syncwarp();
            const bool active = base + lane < total;
            const int q = active ? W.queue[lane] : 0;
            const int o = q >> 8, e = q & 255;
            const int first = HIST ? __shfl_sync(kAll, out_walls, o) : 0;
            if (active) {
                const int go = o / LPG, so = s0 + go;
                const DevParams& Q = BATCH ? A.scene_params[__ldg(&A.scene[so])] : P0;
                const int j = W.hit[e][go];
                const float4 po = __ldg(&A.pos[so]), vo = __ldg(&A.vel[so]);
                const float4 pj = __ldg(&A.pos[j]), vj = __ldg(&A.vel[j]);
                float3 xi = make_float3(0.f, 0.f, 0.f);
                int io = 0, jd = 0;
                if (HIST) {
                    io = __ldg(&A.ids[so]);
                    jd = __ldg(&A.ids[j]);
                    const int row = __ldg(&A.hcnt_in[so]);
                    if (row > 0) {
                        // rows keep the visiting order, so a lasting contact is about where
                        // it was
                        HistRow k;
                        k.in = A.hist_in + static_cast<int64_t>(io) * kHistCap;
                        k.in_count = row;
                        k.cursor = min(first + e, row - 1);
                        xi = find_spring(k, jd);
                    }
                }
                float3 d;
                const float ns = pair_norm_sq(po, pj, d);
                const float norm = sqrtf(ns);
                const float dist = pair_dist(norm, po.w, pj.w);
                const PairTerms t = pair_terms<HIST>(Q, d, norm, dist, make_float3(vo.x, vo.y, vo.z),
                                                     vo.w, vj, xi);
                W.term[lane][0] = make_float4(t.nrm.x, t.nrm.y, t.nrm.z, t.fp);
                W.term[lane][1] = make_float4(t.t.x, t.t.y, t.t.z, t.cvn);
                if (HIST && first + e < kHistCap)
                    A.hist_out[static_cast<int64_t>(io) * kHistCap + first + e] =
                        make_float4(xi.x, xi.y, xi.z, __int_as_float(jd));
            }
            __syncwarp();
            if (sub == 0) {
                for (int k = max(off - base, 0); k < min(upto - base, 32); ++k) {
                    const float4 a = W.term[k][0], b = W.term[k][1];
                    PairTerms u;
                    u.nrm = make_float3(a.x, a.y, a.z);
                    u.fp = a.w;
                    u.t = make_float3(b.x, b.y, b.z);
                    u.cvn = b.w;
                    pair_accumulate<HIST>(f, u);
                }
            }
            __syncwarp();               // the queue and the terms are free again
        }
        if (HIST && work && found > 0) {
            h.out_count = min(out_walls + found, kHistCap);
            if (out_walls + found > kHistCap)
                atomicAdd(&A.counters[kCntHistOverflow],
                          static_cast<unsigned long long>(out_walls + found - kHistCap));
        }
    }
    if (work) {
        // read again (from L1) rather than held in registers meanwhile
        const float4 x = A.pos[s], v = A.vel[s];
        if (HIST) A.hcnt_out[s] = h.out_count;
        const float3 a = make_float3(f.x / v.w, f.y / v.w, f.z / v.w);
        float3 v1, x1;
        if (!PICARD) {
            v1 = make_float3(fmaf(P.dt, a.x, v.x), fmaf(P.dt, a.y, v.y), fmaf(P.dt, a.z, v.z));
            x1 = make_float3(fmaf(P.dt, v1.x, x.x), fmaf(P.dt, v1.y, x.y), fmaf(P.dt, v1.z, x.z));
        } else {
            const float4 xn = A.npos[s], vn = A.nvel[s];
            v1 = make_float3(fmaf(P.dt, a.x, vn.x), fmaf(P.dt, a.y, vn.y), fmaf(P.dt, a.z, vn.z));
            x1 = make_float3(fmaf(P.dt, v1.x, xn.x), fmaf(P.dt, v1.y, xn.y), fmaf(P.dt, v1.z, xn.z));
            res_bits = max(res_bits, __float_as_uint(fabsf(x1.x - x.x)));
            res_bits = max(res_bits, __float_as_uint(fabsf(x1.y - x.y)));
            res_bits = max(res_bits, __float_as_uint(fabsf(x1.z - x.z)));
        }
        A.pos_out[s] = make_float4(x1.x, x1.y, x1.z, x.w);
        A.vel_out[s] = make_float4(v1.x, v1.y, v1.z, v.w);
        A.ids_out[s] = A.ids[s];
        if (BATCH) A.scene_out[s] = scene;
        A.acc_out[s] = make_float4(a.x, a.y, a.z, 0.f);
    } else if (frozen && sub == 0) {
        // a stopped scene (a diverged rollout): state copied through unchanged
        A.pos_out[s] = pi;
        A.vel_out[s] = vi;
        A.ids_out[s] = id;
        A.scene_out[s] = scene;
        A.acc_out[s] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (HIST) A.hcnt_out[s] = 0;
    }
    if (PICARD) {
        // max of non-negative float bits (NaN above +inf, so it is kept)
        res_bits = __reduce_max_sync(kAll, res_bits);
        if (lane == 0 && res_bits != 0u) atomicMax(A.res_slot, res_bits);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            *A.picard_used = A.iter + 1;
            A.counters[kCntPicardIters] += 1ull;
        }
    }
}

// Deterministic block sum of doubles (fixed tree for a fixed launch shape).
__device__ __forceinline__ double block_sum(double v) {
    __shared__ double ws[kBlock / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) ws[warp] = v;
    __syncthreads();
    double t = 0.0;
    if (warp == 0) {
        t = lane < kBlock / 32 ? ws[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    }
    __syncthreads();
    return t;  // valid in thread 0
}

// reference src/energy_kernel.cu:30-80: kinetic + gravity + wall and pair elastic
// energy (pairs counted from the lower grain id), plus the tangential spring energy
// 1/2 k_t |xi|^2 of stored contacts in history mode. Terms in FP32 as the
// reference, the grain's sum in FP64, written per sorted position for the segmented
// reduction below.
template <bool HIST>
__device__ __forceinline__ double energy_of(const DevParams& P, int s, const float4* __restrict__ pos,
                                            const float4* __restrict__ vel, const int* __restrict__ ids,
                                            const int2* __restrict__ table,
                                            const float4* __restrict__ hist,
                                            const int* __restrict__ hcnt, const int* __restrict__ src) {
    double e = 0.0;
    const float4 pi = pos[s], vi = vel[s];
    const int id = ids[s];
    const float m = vi.w, ri = pi.w;
    const float F = P.max_force, k = P.k_n, cd = P.clamp_overlap;
    float ss = vi.x * vi.x;
    ss = fmaf(vi.y, vi.y, ss);
    ss = fmaf(vi.z, vi.z, ss);
    e += static_cast<double>(0.5f * m * ss);
    e += static_cast<double>((m * P.gravity) * (pi.z - P.wall_lo[2]));
    const float p3[3] = {pi.x, pi.y, pi.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        e += static_cast<double>(contact_energy(ri - (p3[a] - P.wall_lo[a]), cd, F, k));
        e += static_cast<double>(contact_energy(ri - (P.wall_hi[a] - p3[a]), cd, F, k));
    }
    int cx, cy, cz;
    cell_coords(P, pi.x, pi.y, pi.z, cx, cy, cz);
    // a column's nine table entries in one go, candidates two at a time; the partner's id
    // only for the few pairs that overlap (1,000,003 grains 84 us; with the id of every
    // candidate read before its position 114)
    auto visit = [&](int j, float4 pj) {
        float3 d;
        const float ns = pair_norm_sq(pi, pj, d);
        if (!maybe_contact(ns, ri, pj.w) || j == s || ids[j] <= id) return;
        e += static_cast<double>(contact_energy((ri + pj.w) - sqrtf(ns), cd, F, k));
    };
    for (int dx = -1; dx <= 1; ++dx) {
        const int nx = cx + dx;
        if (nx < 0 || nx >= P.grid[0]) continue;
        int lo[3], hi[3];
        row_ranges(P, table, nx, cy, cz, lo, hi);
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            int j = lo[t];
            // an empty row has lo = INT_MAX, hi = 0: the difference does not overflow
            for (; hi[t] - j > 1; j += 2) {
                const float4 p0 = __ldg(&pos[j]), p1 = __ldg(&pos[j + 1]);
                visit(j, p0);
                visit(j + 1, p1);
            }
            if (j < hi[t]) visit(j, __ldg(&pos[j]));
        }
    }
    if (HIST) {
        const int c = hcnt[src[s]];
        for (int q = 0; q < c; ++q) {
            const float4 x = hist[static_cast<int64_t>(id) * kHistCap + q];
            const int partner = __float_as_int(x.w);
            if (partner >= 0 && partner <= id) continue;
            float xs = x.x * x.x;
            xs = fmaf(x.y, x.y, xs);
            xs = fmaf(x.z, x.z, xs);
            e += static_cast<double>(0.5f * P.k_t * xs);
        }
    }
    return e;
}

// CHUNK: a single scene's chunks are this kernel's blocks, so each block leaves its chunk's
// sum (the tree of k_segment_chunks) instead of its grains' values.
template <bool HIST, bool BATCH, bool CHUNK>
__global__ void __launch_bounds__(kBlock, 5)
k_energy(DevParams P0, SceneTab T, const float4* __restrict__ pos, const float4* __restrict__ vel,
         const int* __restrict__ ids, const int2* __restrict__ table,
         const float4* __restrict__ hist, const int* __restrict__ hcnt,
         const int* __restrict__ src, double* __restrict__ out) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (CHUNK) {
        const double t = block_sum(s < P0.n ? energy_of<HIST>(P0, s, pos, vel, ids, table, hist, hcnt, src) : 0.0);
        if (threadIdx.x == 0) out[blockIdx.x] = t;
    } else if (s < P0.n) {
        out[s] = energy_of<HIST>(scene_params<BATCH>(P0, T, s), s, pos, vel, ids, table, hist, hcnt, src);
    }
}

// Segmented sums, step 1: one block per 256-grain chunk of a scene's segment (chunks
// are aligned to the segment start, so a scene reduces the same way alone or in a
// batch). comps values per grain, value c of grain i at v[c * comp_step + i * grain_step].
__global__ void __launch_bounds__(kBlock)
k_segment_chunks(const double* __restrict__ v, int64_t comp_step, int grain_step, int comps, const int* __restrict__ seg,
                 const int* __restrict__ chunk_base, int scenes, double* __restrict__ partials,
                 int total_chunks) {
    const int b = blockIdx.x;
    int lo = 0, hi = scenes;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (chunk_base[mid] <= b) lo = mid; else hi = mid;
    }
    const int sc = lo;
    const int first = seg[sc] + (b - chunk_base[sc]) * kBlock;
    const int i = first + static_cast<int>(threadIdx.x);
    for (int c = 0; c < comps; ++c) {
        const double x =
            i < seg[sc + 1] ? v[c * comp_step + static_cast<int64_t>(i) * grain_step] : 0.0;
        const double t = block_sum(x);
        if (threadIdx.x == 0) partials[static_cast<int64_t>(c) * total_chunks + b] = t;
    }
}

// Segmented sums, step 2: one block per scene and component sums its chunk partials in a
// fixed order, eight loads in flight (one block alone waits for each: 11 us for the 3,907
// partials of 1,000,003 grains, and that three times over for the momentum).
__global__ void __launch_bounds__(kBlock)
k_segment_finish(const double* __restrict__ partials, const int* __restrict__ chunk_base,
                 int comps, int total_chunks, double* __restrict__ out) {
    const int sc = blockIdx.x, c = blockIdx.y;
    const int c0 = chunk_base[sc], c1 = chunk_base[sc + 1];
    const double* v = partials + static_cast<int64_t>(c) * total_chunks;
    double x = 0.0;
    int i = c0 + static_cast<int>(threadIdx.x);
    for (; i + 7 * kBlock < c1; i += 8 * kBlock) {
        double a[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) a[u] = __ldg(&v[i + u * kBlock]);
#pragma unroll
        for (int u = 0; u < 8; ++u) x += a[u];
    }
    for (; i < c1; i += kBlock) x += __ldg(&v[i]);
    const double t = block_sum(x);
    if (threadIdx.x == 0) out[sc * comps + c] = t;
}

// Momentum terms by grain id, so that the sums do not depend on the order of the slots
// (which a step on lists leaves as the last build made it).
__global__ void __launch_bounds__(kBlock)
k_momentum(int n, const float4* __restrict__ vel, const int* __restrict__ ids,
           double* __restrict__ out) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const float4 v = vel[s];
    const double m = v.w;
    // one whole 32-byte sector per grain
    double2* o = reinterpret_cast<double2*>(out + 4 * static_cast<int64_t>(ids[s]));
    o[0] = make_double2(m * v.x, m * v.y);
    o[1] = make_double2(m * v.z, 0.0);
}

// reference src/particle_dynamics.cu:328-344: sqrt(ax^2 + ay^2 + az^2), unfused.
__global__ void __launch_bounds__(kBlock)
k_max_accel(int n, const float4* __restrict__ acc, unsigned long long* __restrict__ counters) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t b = 0u;
    if (s < n) {
        const float4 a = acc[s];
        float sq = 0.f;
        sq = sq + a.x * a.x;
        sq = sq + a.y * a.y;
        sq = sq + a.z * a.z;
        b = __float_as_uint(sqrtf(sq));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
    if ((threadIdx.x & 31) == 0 && b)
        atomicMax(reinterpret_cast<unsigned int*>(&counters[kCntMaxAccel]), b);
}

// reference src/particle_dynamics.cu:311-325: finite and inside the domain box.
template <bool BATCH>
__global__ void __launch_bounds__(kBlock)
k_stability(DevParams P0, SceneTab T, const float4* __restrict__ pos,
            unsigned long long* __restrict__ counters, int* __restrict__ scene_unstable) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= P0.n) return;
    const DevParams& P = scene_params<BATCH>(P0, T, s);
    const float4 p = pos[s];
    const float q[3] = {p.x, p.y, p.z};
    bool bad = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) bad |= !isfinite(q[a]) || q[a] < P.lo[a] || q[a] > P.hi[a];
    if (bad) {
        atomicOr(&counters[kCntUnstable], 1ull);
        if (BATCH && scene_unstable) scene_unstable[T.scene[s]] = 1;
    }
}

}  // namespace

template <int LPG>
static void launch_force_lanes(const DevParams& P, const ForceArgs& a, bool picard, Skip skip, cudaStream_t st) {
    const int nb = blocks_for(P.n, kForceBlock / LPG);
    const bool batch = a.scene_params != nullptr;
#define WD_FORCE(H, PI, B, R) k_force<H, PI, B, R, LPG><<<nb, kForceBlock, 0, st>>>(P, a, skip)
    if (a.rec_list) {
        if (P.history) WD_FORCE(true, false, false, true); else WD_FORCE(false, false, false, true);
    } else if (P.history) {
        if (picard) { if (batch) WD_FORCE(true, true, true, false); else WD_FORCE(true, true, false, false); }
        else { if (batch) WD_FORCE(true, false, true, false); else WD_FORCE(true, false, false, false); }
    } else {
        if (picard) { if (batch) WD_FORCE(false, true, true, false); else WD_FORCE(false, true, false, false); }
        else { if (batch) WD_FORCE(false, false, true, false); else WD_FORCE(false, false, false, false); }
    }
#undef WD_FORCE
}

void launch_force(const DevParams& P, const ForceArgs& a, bool picard, Skip skip, cudaStream_t st) {
    // Lanes per grain: as many as the chip has room for. Searched step of packed grains with
    // springs, 32 / 8 / 1 lanes: 3,000 grains 34.6 / 35.3 / 40.8 us, 5,000 31.5 / 29.4 / 34.8,
    // 16,000 51.8 / 39.7 / 43.7, 32,000 69 / 46.7 / 43.4, 10^6 1285 / 518 / 186; a lane alone
    // that evaluated contacts on its walk took 82, 70, 85, 96 and 411. The default cube (30
    // grains a cell, 800 candidates each), ten steps: 361 / 443 / 793, and 1095.
    if (P.n < 4096) launch_force_lanes<32>(P, a, picard, skip, st);
    else if (P.n < 24576) launch_force_lanes<8>(P, a, picard, skip, st);
    else launch_force_lanes<1>(P, a, picard, skip, st);
}

int reduction_blocks(int n) { return blocks_for(n > 0 ? n : 1); }

void launch_segment_sums(const double* values, int n, int comps, const Segments& g,
                         double* partials, double* out, cudaStream_t st, int grain_step) {
    k_segment_chunks<<<g.total_chunks, kBlock, 0, st>>>(values, grain_step > 1 ? 1 : n, grain_step,
                                                        comps, g.seg, g.chunk_base, g.scenes,
                                                        partials, g.total_chunks);
    k_segment_finish<<<dim3(g.scenes, comps), kBlock, 0, st>>>(partials, g.chunk_base, comps, g.total_chunks, out);
}

void launch_energy(const DevParams& P, SceneTab T, const float4* pos, const float4* vel,
                   const int* ids, const int2* table, const float4* hist, const int* hcnt,
                   const int* src, const Segments& g, double* per_grain, double* partials,
                   double* out, cudaStream_t st) {
    const int nb = reduction_blocks(P.n);
    const bool batch = T.params != nullptr, chunk = g.scenes == 1 && per_grain == nullptr;
    double* to = chunk ? partials : per_grain;
#define WD_ENERGY(H, B, C) k_energy<H, B, C><<<nb, kBlock, 0, st>>>(P, T, pos, vel, ids, table, hist, hcnt, src, to)
    if (P.history) {
        if (batch) WD_ENERGY(true, true, false);
        else if (chunk) WD_ENERGY(true, false, true);
        else WD_ENERGY(true, false, false);
    } else {
        if (batch) WD_ENERGY(false, true, false);
        else if (chunk) WD_ENERGY(false, false, true);
        else WD_ENERGY(false, false, false);
    }
#undef WD_ENERGY
    if (chunk)
        k_segment_finish<<<1, kBlock, 0, st>>>(partials, g.chunk_base, 1, g.total_chunks, out);
    else
        launch_segment_sums(per_grain, P.n, 1, g, partials, out, st);
}

void launch_momentum(int n, const float4* vel, const int* ids, const Segments& g,
                     double* per_grain, double* partials, double* out3, cudaStream_t st) {
    k_momentum<<<reduction_blocks(n), kBlock, 0, st>>>(n, vel, ids, per_grain);
    launch_segment_sums(per_grain, n, 3, g, partials, out3, st, 4);
}

void launch_max_accel(int n, const float4* acc, unsigned long long* counters,
                      cudaStream_t st) {
    k_max_accel<<<blocks_for(n), kBlock, 0, st>>>(n, acc, counters);
}

void launch_stability(const DevParams& P, SceneTab T, const float4* pos,
                      unsigned long long* counters, int* scene_unstable, cudaStream_t st) {
    if (T.params)
        k_stability<true><<<blocks_for(P.n), kBlock, 0, st>>>(P, T, pos, counters, scene_unstable);
    else
        k_stability<false><<<blocks_for(P.n), kBlock, 0, st>>>(P, T, pos, counters, nullptr);
}

}  // namespace wd
