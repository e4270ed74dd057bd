// wd_lists.cu -- Verlet neighbor lists for the semi-implicit Euler and the backward
// Euler / Picard steps.
//
// The reference searches the grid every step (src/particle_dynamics.cu:264-281). With
// simulation.neighbor_skin = s > 0 the search runs only when needed: a build sorts the
// grains as the search does, and lists, for every grain, the grains whose centres are
// closer than r_i + r_j + s, in the contact kernel's canonical visiting order (stencil
// cell, then grain id). Until some grain has moved 0.49 s from where the build saw it
// (kListValid), every contact of every step is in the lists (a pair not listed is still
// >= r_i + r_j + 0.02 s apart), so the step computes the same contact set as the
// searched step.
//
// The results are bit-identical to the searched step because forces are accumulated
// in the same order: the kernel checks that the contacts it meets arrive in canonical
// order for the current positions ((stencil offset of the partner's current cell,
// partner id) non-decreasing); a grain for which a cell crossing broke that order
// re-sorts its contacts before accumulating them.
//
// Between builds the state stays in one order and ping-pongs between two buffers; a
// build gathers it into the new order, lists the neighbors, and copies it back.
//
// Picard iterates every force evaluation of a step on the same lists. Builds start at
// 0.30 skin instead of 0.49, and each iteration checks that its input iterate is still
// within 0.49 skin of the build; if one is not, or if a list overflowed, the step is redone
// from its start state with the per-iteration search, so the results stay those of the
// searched step.
#include <algorithm>
#include <type_traits>

#include "wd_kernels.h"

namespace wd {
namespace {

__device__ __forceinline__ bool skipped(const Skip& s) {
    return s.prev_res != nullptr && s.tol > 0.f && __uint_as_float(*s.prev_res) < s.tol;
}

// One thread: decide whether this step builds (the decision word, kLcDecision) and
// switch the build's conditional node where the graph holds one. The decision needs a bound B on max |x - x_build| of the current state:
// the exact maximum when the last contact kernel measured it (it then read the build
// positions), otherwise the previous bound plus the largest displacement of the last
// step (triangle inequality), so that most steps read no build positions. The measured
// squares carry float rounding of a few ulps, covered by the factor 1 + 2^-16. The
// next kernel measures exactly when B is within two last-step displacements of the
// threshold, so a build is triggered by the bound only when the exact value is close.
// A NaN or infinite displacement makes B infinite: the step builds.
// One thread. The fused form runs in the last block of a contact kernel whose other blocks
// updated these words with atomics: all of them are read from L2, at once, before anything is
// decided (read one after another as they were needed, they held every step up by five round
// trips: 12.3 against 11.1 us a step for 32768 grains).
// pend: non-null for the library's own lists under neighbor_skin 0, whose searched steps
// count a (cell, search) incident whenever a cell holds more than particles_per_cell grains.
// A build counts them of the state it sorts into pend; they are due when the next step
// starts from that state, here at its end (`step`). Between builds there are none unless the
// build found a cell that could fill up (kLcCrowded): then every step builds, and
// kCntAutoCrowded tells the host to search instead.
__device__ bool list_decide_core(uint32_t* ctrl, float thr, int always_exact,
                                 unsigned long long* counters, unsigned long long* pend,
                                 bool at_step, int left) {
    static_assert(kLcDisp == 0 && kLcOverflow == 1 && kLcForce == 2 && kLcStep == 6 &&
                      kLcExact == 7 && kLcBound == 8 && kLcCrowded == 12, "read as vectors");
    const uint4 w0 = __ldcg(reinterpret_cast<const uint4*>(ctrl));
    const uint4 w1 = __ldcg(reinterpret_cast<const uint4*>(ctrl + 4));
    const double bound = __ldcg(reinterpret_cast<const double*>(ctrl + kLcBound));
    const bool crowded = pend != nullptr && __ldcg(ctrl + kLcCrowded) != 0u;
    const unsigned long long overflow = pend != nullptr && at_step ? __ldcg(pend + kCntGridOverflow) : 0ull;
    const double grow = 1.0 + 1.0 / 65536.0;
    const double step = sqrt(static_cast<double>(__uint_as_float(w1.z))) * grow;
    const double disp = sqrt(static_cast<double>(__uint_as_float(w0.x))) * grow;
    double b = w1.w != 0u ? disp : bound + step;
    bool build = w0.z != 0u || w0.y != 0u || !(b < thr);
    if (pend != nullptr) {
        if (at_step) {
            build |= crowded;
            if (overflow) atomicAdd(&counters[kCntGridOverflow], overflow);
            atomicAdd(&counters[kCntAutoSteps], 1ull);
            if (build) atomicAdd(&counters[kCntAutoBuilds], 1ull);
            if (crowded) counters[kCntAutoCrowded] = 1ull;
        }
        if (build) {
            pend[kCntGridOverflow] = 0ull;
            ctrl[kLcCrowded] = 0u;
        }
    }
    ctrl[kLcDecision] = build ? __float_as_uint(1.f) : 0u;
    // in a chain of steps (left: with this one), the rest waits for the build
    ctrl[kLcPending] = build && left > 0 ? 1u : 0u;
    ctrl[kLcLeft] = build && left > 0 ? static_cast<uint32_t>(left - 1) : 0u;
    if (build) {
        b = 0.0;
        ctrl[kLcOverflow] = 0u;
        ctrl[kLcForce] = 0u;
        if (pend == nullptr) atomicAdd(&counters[kCntListBuilds], 1ull);
    }
    *reinterpret_cast<double*>(ctrl + kLcBound) = b;
    ctrl[kLcDisp] = 0u;
    ctrl[kLcStep] = 0u;
    const bool exact = always_exact || (!build && !(b + 2.0 * step < thr));
    ctrl[kLcExact] = exact ? 1u : 0u;
    if (exact && pend == nullptr) atomicAdd(&counters[kCntListExact], 1ull);
    return build;
}

__global__ void k_list_decide(uint32_t* __restrict__ ctrl, float thr, int always_exact,
                              unsigned long long* __restrict__ counters,
                              unsigned long long* __restrict__ pend, int use_cond,
                              cudaGraphConditionalHandle cond) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const bool build = list_decide_core(ctrl, thr, always_exact, counters, pend, false, 0);
    if (always_exact) counters[kCntHistBefore] = counters[kCntHistOverflow];  // a Picard step begins
    if (use_cond) cudaGraphSetConditional(cond, build ? 1u : 0u);
}

// Cells that a grain at p can be in while it stays within half a skin of p (the lists hold
// up to 0.49 skin; the rest covers the rounding of p -+ r and of the displacement bound).
template <typename Visit>
__device__ __forceinline__ void reachable_cells(const DevParams& P, float4 p, Visit visit) {
    const float r = 0.5f * P.skin;
    int a0, a1, b0, b1, c0, c1;
    cell_coords(P, p.x - r, p.y - r, p.z - r, a0, b0, c0);
    cell_coords(P, p.x + r, p.y + r, p.z + r, a1, b1, c1);
    for (int x = a0; x <= a1; ++x)
        for (int y = b0; y <= b1; ++y)
            for (int z = c0; z <= c1; ++z) visit(P.cell_base + flat_cell(P, x, y, z));
}

__global__ void __launch_bounds__(kBlock)
k_cell_clear(DevParams P, const float4* __restrict__ xbuild, uint32_t* __restrict__ load, Skip skip) {
    if (skipped(skip)) return;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < P.n) reachable_cells(P, xbuild[s], [&](uint32_t c) { load[c] = 0u; });
}

// One atomic per reachable cell: 1.3 a grain at this skin, spread over the grid (about 8 us
// for 2^20 grains, of a build of about 300).
__global__ void __launch_bounds__(kBlock)
k_cell_load(DevParams P, const float4* __restrict__ pos, uint32_t* __restrict__ load,
            uint32_t* __restrict__ ctrl, Skip skip) {
    if (skipped(skip)) return;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= P.n) return;
    bool over = false;
    reachable_cells(P, pos[s], [&](uint32_t c) {
        over |= static_cast<int64_t>(atomicAdd(&load[c], 1u)) >= static_cast<int64_t>(P.ppc);
    });
    if (over) atomicOr(&ctrl[kLcCrowded], 1u);
}

// The decision fused into the tail of a semi-implicit Euler list kernel: the last block
// to finish (every block's displacement atomics done) decides whether the lists are
// rebuilt before the next step: it switches the build's conditional node where the step
// graph holds one, or leaves the decision word to the kernel that launches the build's
// graphs from the device (wd_launch.cu). All threads
// of every block call it, with their displacement maxima. The block's maxima meet in shared
// memory first (one atomic a block and word instead of one a warp: 4736 at one address), and
// thread 0's fence orders its atomics before its ticket.
__device__ __forceinline__ void list_tail_decide(const ListArgs& A, bool exact, uint32_t disp_bits,
                                                 uint32_t step_bits) {
    __shared__ uint32_t top[kBlock / 32][2];
    disp_bits = exact ? __reduce_max_sync(0xffffffffu, disp_bits) : 0u;
    step_bits = __reduce_max_sync(0xffffffffu, step_bits);
    if ((threadIdx.x & 31) == 0) {
        top[threadIdx.x >> 5][0] = disp_bits;
        top[threadIdx.x >> 5][1] = step_bits;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < static_cast<int>(blockDim.x) / 32; ++w) {
            disp_bits = max(disp_bits, top[w][0]);
            step_bits = max(step_bits, top[w][1]);
        }
        if (disp_bits != 0u) atomicMax(&A.list_ctrl[kLcDisp], disp_bits);
        if (step_bits != 0u) atomicMax(&A.list_ctrl[kLcStep], step_bits);
        __threadfence();
        const unsigned ticket = atomicAdd(A.tail_count, 1u);
        if (ticket == gridDim.x - 1) {
            __threadfence();
            const bool build =
                list_decide_core(A.list_ctrl, A.thr, 0, A.counters, A.pend, true, A.left);
            *A.tail_count = 0u;
            if (A.use_cond) cudaGraphSetConditional(A.cond, build ? 1u : 0u);
        }
    }
}

// A step of a chain whose predecessor decided a build: it runs after the build instead, from
// the graph that the build launches for the steps left over.
__device__ __forceinline__ bool list_step_waits(const ListArgs& A) {
    return A.left > 0 && A.list_ctrl[kLcPending] != 0u;
}

// Grains in cells two apart along an axis are more than a cell width apart, so the 27
// stencil cells hold every contact; but when 2 r_max + skin exceeds a cell width, a pair
// two cells apart can be closer than r_i + r_j + skin and meet before the next build.
// A build then walks the outer shell of the 5 x 5 x 5 block too, cell by cell where its
// box lies within the grain's reach r_i + r_max + skin (only grains near a face of their
// cell, so few). Each shell cell is visited in the pass of the first axis along which
// it lies two cells away; its grains follow the stencil's in the list.
template <typename Visit>
__device__ __forceinline__ void list_far_shell(const DevParams& P, const int2* __restrict__ table,
                                               const float4* __restrict__ pos, float4 pi,
                                               int cx, int cy, int cz, Visit& visit) {
    const float reach_max = (pi.w + P.rmax) + P.skin;
    // the grain's offset in its cell per axis (the fast path's t minus the index) and the
    // cell mapping's rounding margin, in cells
    const float f0 = ((pi.x - P.lo[0]) * P.inv_len[0]) * static_cast<float>(P.grid[0]) -
                     static_cast<float>(cx);
    const float f1 = ((pi.y - P.lo[1]) * P.inv_len[1]) * static_cast<float>(P.grid[1]) -
                     static_cast<float>(cy);
    const float f2 = ((pi.z - P.lo[2]) * P.inv_len[2]) * static_cast<float>(P.grid[2]) -
                     static_cast<float>(cz);
    // distance from the grain to the box of cell c + o along axis a, shortened by the
    // margin (a NaN offset gives 0: every cell in reach)
    auto gap = [&](int a, int o) {
        const float f = a == 0 ? f0 : (a == 1 ? f1 : f2);
        const float g = o == 0 ? 0.f
                      : o == 1 ? 1.f - f
                      : o == -1 ? f
                      : o == 2 ? 2.f - f
                               : 1.f + f;
        const float m = 2.f * (a == 0 ? P.cell_err[0] : (a == 1 ? P.cell_err[1] : P.cell_err[2])) + 1e-4f;
        const float len = a == 0 ? P.cell_len[0] : (a == 1 ? P.cell_len[1] : P.cell_len[2]);
        return fmaxf(0.f, g - m) * len;
    };
    const float r2 = (reach_max * reach_max) * 1.0001f;
    // a cell two away along two axes is at least sqrt(2) cell widths (less the margins)
    // away: in reach only for a reach above about 1.4 cells
    // (an offset f lies in [-err, 1 + err] and the margin is 2 err + 1e-4 cells)
    const float w = P.cell_min * (1.f - 3.f * fmaxf(P.cell_err[0], fmaxf(P.cell_err[1], P.cell_err[2])) - 1e-4f);
    const bool two_axes = r2 > 2.f * w * w;
    for (int a = 0; a < 3; ++a) {
        // b < c: the other two axes; an axis before a stays within one cell (a is the
        // first axis at which the cell lies two away)
        const int b = a == 0 ? 1 : 0, c = a == 2 ? 1 : 2;
        for (int side = -2; side <= 2; side += 4) {
            const float ga = gap(a, side);
            if (ga * ga > r2) continue;
            const int bl = (b < a || !two_axes) ? -1 : -2;
            const int cl = (c < a || !two_axes) ? -1 : -2;
            for (int ob = bl; ob <= -bl; ++ob) {
                const float gb = gap(b, ob);
                if (ga * ga + gb * gb > r2) continue;
                for (int oc = cl; oc <= -cl; ++oc) {
                    const float gc = gap(c, oc);
                    if (ga * ga + gb * gb + gc * gc > r2) continue;
                    const int nx = cx + (a == 0 ? side : ob);
                    const int ny = cy + (a == 0 ? ob : (a == 1 ? side : oc));
                    const int nz = cz + (a == 2 ? side : oc);
                    if (nx < 0 || nx >= P.grid[0] || ny < 0 || ny >= P.grid[1] || nz < 0 ||
                        nz >= P.grid[2])
                        continue;
                    const int2 e = __ldg(&table[P.cell_base + flat_cell(P, nx, ny, nz)]);
                    for (int j = e.x; j < e.y; ++j) visit(j, __ldg(&pos[j]));
                }
            }
        }
    }
}

// Which of the outer cells (two away along one axis) a grain's list has to look into, as
// list_far_shell decides it per cell: bits 0-1 x lower / upper, 2-3 y, 4-5 z. Bit 6: the
// reach covers cells two away along two axes, which only list_far_shell walks.
__device__ __forceinline__ unsigned list_outer_faces(const DevParams& P, float4 pi, int cx, int cy,
                                                     int cz) {
    const float reach = (pi.w + P.rmax) + P.skin;
    if (!(reach > P.cell_min)) return 0u;
    const float r2 = (reach * reach) * 1.0001f;
    const float w = P.cell_min * (1.f - 3.f * fmaxf(P.cell_err[0], fmaxf(P.cell_err[1], P.cell_err[2])) - 1e-4f);
    if (r2 > 2.f * w * w) return 1u << 6;
    const float p3[3] = {pi.x, pi.y, pi.z};
    const int c3[3] = {cx, cy, cz};
    unsigned faces = 0u;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float f = ((p3[a] - P.lo[a]) * P.inv_len[a]) * static_cast<float>(P.grid[a]) -
                        static_cast<float>(c3[a]);
        const float m = 2.f * P.cell_err[a] + 1e-4f;
        const float lower = fmaxf(0.f, 1.f + f - m) * P.cell_len[a];
        const float upper = fmaxf(0.f, 2.f - f - m) * P.cell_len[a];
        if (!(lower * lower > r2)) faces |= 1u << (2 * a);
        if (!(upper * upper > r2)) faces |= 2u << (2 * a);
    }
    return faces;
}

// Slots of the cells (nx, ny, z0 .. z1), at most five: consecutive, or [0, 0) if empty.
__device__ __forceinline__ int2 table_row(const DevParams& P, const int2* __restrict__ table, int nx,
                                          int ny, int z0, int z1) {
    const bool col = nx >= 0 && nx < P.grid[0] && ny >= 0 && ny < P.grid[1];
    const int2* t = table + P.cell_base +
                    (static_cast<uint32_t>(nx) * static_cast<uint32_t>(P.grid[1]) + static_cast<uint32_t>(ny)) *
                        static_cast<uint32_t>(P.grid[2]);
    int2 e[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int z = z0 + k;
        e[k] = col && z <= z1 && z >= 0 && z < P.grid[2] ? __ldg(&t[z]) : make_int2(-1, -1);
    }
    int lo = 0x7fffffff, hi = 0;
#pragma unroll
    for (int k = 0; k < 5; ++k)
        if (e[k].x >= 0) {
            lo = min(lo, e[k].x);
            hi = max(hi, e[k].y);
        }
    return lo < hi ? make_int2(lo, hi) : make_int2(0, 0);
}

// The list of every grain, from the run table of the build's sorted state: the
// contact kernel's stencil walk with the skin added to the contact distance, widened by the
// outer cells in reach. The sorted state is copied back into the step's buffers on the way.
//
// The cells to look into form rows along z: the nine of the stencil, longer by a cell where
// a z face is in reach, and three beyond each x or y face in reach; a lane walks its own
// outer rows, whichever faces they lie at (cell by cell, each of the 54 outer cells cost the
// warp its test, table load and loop). With LPG lanes to a grain the rows' slot ranges go
// to shared memory and the lanes walk the candidates as one sequence, LPG apart and four
// each at a time; for one lane that costs more than row by row (175 us: 4,700 warp
// instructions per 32 grains). Bound by issue. 1,000,003 packed grains 126 us (before 175),
// 2^20 falling 82 (110), 100,003 packed 23 (31), 5,003 packed 10 (23).
constexpr int kListRows = 21;

template <bool BATCH, int LPG>
__global__ void __launch_bounds__(kBlock)
k_list_build(DevParams P0, SceneTab T, const float4* __restrict__ pos,
             const int2* __restrict__ table, int* __restrict__ nbr, int* __restrict__ nbr_cnt,
             float4* __restrict__ xbuild, uint32_t* __restrict__ ctrl, ListCopy cp, Skip skip) {
    if (skipped(skip)) return;
    constexpr int kPer = kBlock / LPG;
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ int2 rows[LPG > 1 ? kListRows : 1][LPG > 1 ? kPer : 1];
    const int g = static_cast<int>(threadIdx.x) / LPG, sub = static_cast<int>(threadIdx.x) % LPG;
    const int s = blockIdx.x * kPer + g;
    const int n = P0.n;
    const bool live = s < n;
    if (LPG == 1 && !live) return;
    const DevParams& P = BATCH ? T.params[live ? T.scene[s] : 0] : P0;
    float4 pi = make_float4(0.f, 0.f, 0.f, 0.f);
    int cx = 0, cy = 0, cz = 0;
    if (live) {
        pi = pos[s];
        if (sub == 0) {
            cp.pos_out[s] = pi;
            cp.vel_out[s] = cp.vel[s];
            cp.ids_out[s] = cp.ids[s];
            if (cp.hcnt) cp.hcnt_out[s] = cp.hcnt[s];
            if (BATCH) cp.scene_out[s] = cp.scene[s];
        }
        cell_coords(P, pi.x, pi.y, pi.z, cx, cy, cz);
    }
    const unsigned faces = live ? list_outer_faces(P, pi, cx, cy, cz) : 0u;
    const int z0 = cz - 1 - ((faces >> 4) & 1), z1 = cz + 1 + ((faces >> 5) & 1);
    int cnt = 0;
    auto reach = [&](int j, float4 pj) {
        float3 d;
        const float ns = pair_norm_sq(pi, pj, d);
        const float far = (pi.w + pj.w) + P.skin;
        return j != s && ns < far * far;
    };
    if (LPG == 1) {
        auto visit = [&](int j, float4 pj) {
            if (!reach(j, pj)) return;
            if (cnt < kNbrCap) nbr[static_cast<int64_t>(cnt) * n + s] = j;
            ++cnt;
        };
        auto walk = [&](int2 q) {
            int j = q.x;
            for (; q.y - j > 1; j += 2) {
                const float4 p0 = __ldg(&pos[j]), p1 = __ldg(&pos[j + 1]);
                visit(j, p0);
                visit(j + 1, p1);
            }
            if (j < q.y) visit(j, __ldg(&pos[j]));
        };
        // the nine stencil rows, a column of x at a time, then each lane's own outer rows
        for (int dx = -1; dx <= 1; ++dx) {
            int2 q[3];
#pragma unroll
            for (int t = 0; t < 3; ++t) q[t] = table_row(P, table, cx + dx, cy + t - 1, z0, z1);
#pragma unroll
            for (int t = 0; t < 3; ++t) walk(q[t]);
        }
        for (unsigned more = faces & 15u; more; more &= more - 1u) {
            const int face = __ffs(static_cast<int>(more)) - 1;
            const int out = face & 1 ? 2 : -2;
            int2 q[3];
#pragma unroll
            for (int t = 0; t < 3; ++t)
                q[t] = table_row(P, table, cx + (face < 2 ? out : t - 1), cy + (face < 2 ? t - 1 : out),
                                 cz - 1, cz + 1);
#pragma unroll
            for (int t = 0; t < 3; ++t) walk(q[t]);
        }
    } else {
        for (int q = sub; q < kListRows; q += LPG) {
            // 3 rows at dx = -2, 5 at each of -1, 0, 1, and 3 at 2
            const int dx = q < 3 ? -2 : q < 18 ? (q - 3) / 5 - 1 : 2;
            const int dy = q < 3 ? q - 1 : q < 18 ? (q - 3) % 5 - 2 : q - 19;
            const bool wanted = live && (dx != -2 || (faces & 1u)) && (dx != 2 || (faces & 2u)) &&
                                (dy != -2 || (faces & 4u)) && (dy != 2 || (faces & 8u));
            const bool face = dx == -2 || dx == 2 || dy == -2 || dy == 2;
            rows[q][g] = wanted ? table_row(P, table, cx + dx, cy + dy, face ? cz - 1 : z0, face ? cz + 1 : z1)
                                : make_int2(0, 0);
        }
        __syncwarp();
        int r = -1, j = sub, hi = 0;
        for (;;) {
            int jj[4];
            float4 pp[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                while (j >= hi && r < kListRows) {
                    const int over = j - hi;      // how far into the next row
                    if (++r < kListRows) {
                        const int2 q = rows[r][g];
                        j = q.x + over;
                        hi = q.y;
                    }
                }
                jj[u] = r < kListRows ? j : -1;
                j += LPG;
            }
            if (!__any_sync(kAll, jj[0] >= 0)) break;
#pragma unroll
            for (int u = 0; u < 4; ++u) pp[u] = jj[u] >= 0 ? __ldg(&pos[jj[u]]) : pi;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool hit = jj[u] >= 0 && reach(jj[u], pp[u]);
                // the group's lanes hold consecutive candidates
                const unsigned shift = (threadIdx.x & 31u) - static_cast<unsigned>(sub);
                const unsigned mine = (__ballot_sync(kAll, hit) >> shift) & (kAll >> (32 - LPG));
                const int at = cnt + __popc(mine & ((1u << sub) - 1u));
                cnt += __popc(mine);
                if (hit && at < kNbrCap) nbr[static_cast<int64_t>(at) * n + s] = jj[u];
            }
        }
    }
    if (!live || sub != 0) return;
    if (faces & (1u << 6)) {
        auto visit = [&](int q, float4 pq) {
            if (!reach(q, pq)) return;
            if (cnt < kNbrCap) nbr[static_cast<int64_t>(cnt) * n + s] = q;
            ++cnt;
        };
        list_far_shell(P, table, pos, pi, cx, cy, cz, visit);
    }
    nbr_cnt[s] = cnt;
    xbuild[s] = pi;
    if (cnt > kNbrCap) atomicOr(&ctrl[kLcOverflow], 1u);
}

__global__ void __launch_bounds__(kBlock)
k_list_copy(int n, const float4* __restrict__ pos, const float4* __restrict__ vel,
            const int* __restrict__ ids, const int* __restrict__ hcnt,
            const int* __restrict__ scene, float4* __restrict__ pos_out,
            float4* __restrict__ vel_out, int* __restrict__ ids_out, int* __restrict__ hcnt_out,
            int* __restrict__ scene_out, Skip skip) {
    if (skipped(skip)) return;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    pos_out[s] = pos[s];
    vel_out[s] = vel[s];
    ids_out[s] = ids[s];
    if (hcnt) hcnt_out[s] = hcnt[s];
    if (scene) scene_out[s] = scene[s];
}

// Position of a partner in the canonical visiting order: the stencil offset of its
// current cell (dx, then dy, then dz, ascending), then its id.
__device__ __forceinline__ unsigned long long visit_key(const DevParams& P, int cx, int cy,
                                                        int cz, float4 pj, int jd) {
    int jx, jy, jz;
    cell_coords(P, pj.x, pj.y, pj.z, jx, jy, jz);
    const int sidx = ((jx - cx + 1) * 3 + (jy - cy + 1)) * 3 + (jz - cz + 1);
    return (static_cast<unsigned long long>(static_cast<unsigned>(sidx)) << 32) |
           static_cast<unsigned>(jd);
}

// |x1 - x0|^2 as float bits; NaN compares above every float, so a diverging grain
// reports +inf and forces a build.
__device__ __forceinline__ uint32_t disp_sq_bits(float3 x1, float3 x0) {
    const float ex = x1.x - x0.x, ey = x1.y - x0.y, ez = x1.z - x0.z;
    const float d2 = ex * ex + ey * ey + ez * ez;
    return d2 >= 0.f ? __float_as_uint(d2) : 0x7f800000u;
}
__device__ __forceinline__ uint32_t disp_sq_bits(float3 x1, float4 x0) {
    return disp_sq_bits(x1, make_float3(x0.x, x0.y, x0.z));
}

// Warp maxima of a Picard iteration's displacements from the build into list_ctrl.
__device__ __forceinline__ void list_disp_report(uint32_t* ctrl, uint32_t disp_bits) {
    disp_bits = __reduce_max_sync(0xffffffffu, disp_bits);
    if ((threadIdx.x & 31) == 0 && disp_bits != 0u) atomicMax(&ctrl[kLcDisp], disp_bits);
}

// Asks L1 for the line holding p; nothing is read into registers, so a later __ldg of
// p finds it on chip without holding registers in between.
__device__ __forceinline__ void prefetch_l1(const void* p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// The contacts (bitmask over list entries) of a grain that a cell crossing re-ordered, in
// canonical order: each pass takes the smallest visiting key above the last. (Inlined: an
// out-of-line call copies the parameter structs to local memory at kernel entry, which
// was measured to cost more than the code it moves away.)
template <bool HIST>
__device__ __forceinline__ void list_contacts_sorted_mask(const DevParams& P, const ListArgs& A,
                                                       int s, int n, unsigned long long hits,
                                                       float4 pi, float3 vel, float mi, int cx,
                                                       int cy, int cz, float3& f, HistRow& h) {
    const float ri = pi.w;
    long long done = -1;
    for (;;) {
        long long best = 0x7fffffffffffffffll;
        int be = -1;
        for (unsigned long long m = hits; m; m &= m - 1ull) {
            const int e = __ffsll(static_cast<long long>(m)) - 1;
            const int j = __ldg(&A.nbr[static_cast<int64_t>(e) * n + s]);
            const long long key = static_cast<long long>(
                visit_key(P, cx, cy, cz, __ldg(&A.pos[j]), __ldg(&A.ids[j])));
            if (key > done && key < best) {
                best = key;
                be = e;
            }
        }
        if (be < 0) break;
        done = best;
        const int j = __ldg(&A.nbr[static_cast<int64_t>(be) * n + s]);
        const float4 pj = __ldg(&A.pos[j]);
        float3 d;
        const float ns = pair_norm_sq(pi, pj, d);
        const float norm = sqrtf(ns);
        const float dist = pair_dist(norm, ri, pj.w);
        const float4 vj = __ldg(&A.vel[j]);
        pair_force<HIST>(P, d, norm, dist, vel, mi, vj, static_cast<int>(best & 0xffffffffll),
                         f, h, A.counters);
    }
}

// The contacts of a grain whose list overflowed, from the run table of the build that
// ran this step (the stencil walk of the searched kernel).
template <bool HIST>
__device__ __forceinline__ void list_contacts_table(const DevParams& P, const ListArgs& A, int s,
                                                 float4 pi, float3 vel, float mi, float cut,
                                                 int cx, int cy, int cz, float3& f, HistRow& h) {
    const float ri = pi.w;
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
                const float dist = pair_dist(norm, ri, pj.w);
                if (!(dist < 0.f)) continue;
                const float4 vj = __ldg(&A.vel[j]);
                const int partner = HIST ? __ldg(&A.ids[j]) : 0;
                pair_force<HIST>(P, d, norm, dist, vel, mi, vj, partner, f, h, A.counters);
            }
        }
    }
}

// Whether a list entry at pj touches the grain at pi. The exact test takes a square root;
// it decides only for pairs within 1e-5 of touching or closer: dist < 0 needs
// |d| < r_i + r_j up to a few roundings of 2^-24, so a pair beyond that margin is no contact.
__device__ __forceinline__ bool entry_hit(float4 pi, float4 pj) {
    float3 d;
    const float ns = pair_norm_sq(pi, pj, d);
    const float rs = pi.w + pj.w;
    return ns <= rs * rs * 1.00001f && pair_dist(sqrtf(ns), pi.w, pj.w) < 0.f;
}

// A slot of a frozen scene: its state copied through.
template <bool HIST>
__device__ __forceinline__ void list_copy_frozen(const ListArgs& A, int s, int scene, float4 pi,
                                                 float4 vi, int id, bool order_out) {
    A.pos_out[s] = pi;
    A.vel_out[s] = vi;
    if (order_out) {
        A.ids_out[s] = id;
        A.scene_out[s] = scene;
    }
    A.acc_out[s] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (HIST) A.hcnt_out[s] = 0;
}

// The integrator and the displacement measures of one grain under the force f, with
// `out_count` springs written. order_out: write the slot's id (and scene) too.
template <bool HIST, bool BATCH, bool PICARD>
__device__ __forceinline__ void list_integrate(const DevParams& P, const ListArgs& A, int s,
                                               int scene, float4 pi, float4 vi, int id, float3 f,
                                               int out_count, float4 xb, bool exact,
                                               bool order_out, uint32_t& disp_bits,
                                               uint32_t& step_bits, uint32_t& res_bits) {
    const float mi = vi.w;
    const float3 pos = make_float3(pi.x, pi.y, pi.z);
    if (HIST) A.hcnt_out[s] = out_count;
    const float3 a = make_float3(f.x / mi, f.y / mi, f.z / mi);
    float3 v1, x1;
    if (!PICARD) {
        v1 = make_float3(fmaf(P.dt, a.x, vi.x), fmaf(P.dt, a.y, vi.y), fmaf(P.dt, a.z, vi.z));
        x1 = make_float3(fmaf(P.dt, v1.x, pos.x), fmaf(P.dt, v1.y, pos.y), fmaf(P.dt, v1.z, pos.z));
    } else {
        const float4 xn = A.xn[s], vn = A.vn[s];
        v1 = make_float3(fmaf(P.dt, a.x, vn.x), fmaf(P.dt, a.y, vn.y), fmaf(P.dt, a.z, vn.z));
        x1 = make_float3(fmaf(P.dt, v1.x, xn.x), fmaf(P.dt, v1.y, xn.y), fmaf(P.dt, v1.z, xn.z));
        res_bits = max(res_bits, __float_as_uint(fabsf(x1.x - pos.x)));
        res_bits = max(res_bits, __float_as_uint(fabsf(x1.y - pos.y)));
        res_bits = max(res_bits, __float_as_uint(fabsf(x1.z - pos.z)));
    }
    A.pos_out[s] = make_float4(x1.x, x1.y, x1.z, pi.w);
    A.vel_out[s] = make_float4(v1.x, v1.y, v1.z, mi);
    if (order_out) {
        A.ids_out[s] = id;
        if (BATCH) A.scene_out[s] = scene;
    }
    A.acc_out[s] = make_float4(a.x, a.y, a.z, 0.f);
    if (exact) disp_bits = max(disp_bits, disp_sq_bits(x1, xb));
    if (!PICARD) step_bits = max(step_bits, disp_sq_bits(x1, pos));
}

// End of a Picard iteration's kernel: residual, validity and iteration counters.
__device__ __forceinline__ void list_picard_report(const ListArgs& A, uint32_t res_bits, bool viol) {
    // max of non-negative float bits (NaN above +inf, so it is kept)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) res_bits = max(res_bits, __shfl_xor_sync(0xffffffffu, res_bits, o));
    if ((threadIdx.x & 31) == 0 && res_bits != 0u) atomicMax(A.res_slot, res_bits);
    if (__any_sync(0xffffffffu, viol) && (threadIdx.x & 31) == 0) atomicOr(&A.list_ctrl[kLcViol], 1u);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *A.picard_used = A.iter + 1;
        A.counters[kCntPicardIters] += 1ull;
    }
}

// One grain of the list contact kernels, its per-slot values already loaded: contacts
// from the list in canonical order (or the run table when the list overflowed), the
// integrator, the displacement measures (maxima folded into disp_bits / step_bits /
// res_bits, viol or-ed). warp_listed: some grain of the calling warp has a list entry
// (warp-uniform). order_out: write the slot's id (and scene) too. Between builds
// the slot order is fixed and the ids of both state buffers agree, so only the first
// step after a build (whose gather reordered one buffer) and Picard write them.
template <bool HIST, bool BATCH, bool PICARD, bool PREFETCH = false>
__device__ __forceinline__ void list_grain(const DevParams& P0, const ListArgs& A, int s, int n,
                                           int scene, float4 pi, float4 vi, int id, int cnt,
                                           float4 xb, int hcnt_in, bool exact, bool order_out,
                                           bool warp_listed, uint32_t& disp_bits,
                                           uint32_t& step_bits, uint32_t& res_bits, bool& viol) {
    const DevParams& P = BATCH ? A.scene_params[scene] : P0;
    if (PICARD) {
        // the rhs of a Picard step pairs the last iterate's velocity with its forces
        A.rhs_vel[s] = vi;
        A.rhs_ids[s] = id;
        if (A.iter > 0) {
            const float ex = pi.x - xb.x, ey = pi.y - xb.y, ez = pi.z - xb.z;
            viol |= !(ex * ex + ey * ey + ez * ez < A.viol_thr);
            // an overflowed list's grain walks the run table, which is that of the step's start
            viol |= cnt > kNbrCap;
        }
    }
    if (BATCH && P.frozen) {
        list_copy_frozen<HIST>(A, s, scene, pi, vi, id, order_out);
    } else {
        const float3 pos = make_float3(pi.x, pi.y, pi.z);
        const float3 vel = make_float3(vi.x, vi.y, vi.z);
        const float ri = pi.w, mi = vi.w;
        float3 f = make_float3(0.f, 0.f, 0.f);
        HistRow h;
        if (HIST) {
            h.in = A.hist_in + static_cast<int64_t>(id) * kHistCap;
            h.in_count = hcnt_in;
            h.out = A.hist_out + static_cast<int64_t>(id) * kHistCap;
            h.out_count = 0;
            // the first stored spring is probed first: on its way while the list is scanned
            if (PREFETCH && hcnt_in > 0) prefetch_l1(h.in);
        }
        wall_forces<HIST>(P, pos, vel, ri, mi, f, h, A.counters);
        // the list contacts, skipped as a whole by warps in which no grain has a list
        // entry (ballistic grains: the contact code's registers stay out of their path)
        if (warp_listed) {
            const float3 f_walls = f;
            const int out_walls = HIST ? h.out_count : 0;
            const float cut = contact_cutoff_sq(ri, P.rmax);
            // the grain's cell orders its contacts; a grain without list entries needs none
            int cx = 0, cy = 0, cz = 0;
            if (cnt > 0) cell_coords(P, pi.x, pi.y, pi.z, cx, cy, cz);
            bool ordered = true;
            if (cnt <= kNbrCap) {
                // scan: which entries are contacts, four entries' loads in flight at a
                // time (index loads, then the partners' positions), one bit each
                unsigned long long hits = 0ull;
                for (int e0 = 0; e0 < cnt; e0 += 4) {
                    int jj[4];
                    float4 pp[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        jj[u] = e0 + u < cnt ? __ldg(&A.nbr[static_cast<int64_t>(e0 + u) * n + s]) : s;
#pragma unroll
                    for (int u = 0; u < 4; ++u) pp[u] = __ldg(&A.pos[jj[u]]);
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const bool hit = e0 + u < cnt && entry_hit(pi, pp[u]);
                        hits |= hit ? (1ull << (e0 + u)) : 0ull;
                        // the contact's partner id and velocity are read after the scan
                        if (PREFETCH && hit) {
                            prefetch_l1(&A.ids[jj[u]]);
                            prefetch_l1(&A.vel[jj[u]]);
                        }
                    }
                }
                // the contacts, in list order, while they arrive in canonical order (the
                // partner's values are re-read: L1 hits, same arithmetic as the scan)
                const unsigned long long all_hits = hits;
                unsigned long long last = 0ull;
                while (hits) {
                    const int e = __ffsll(static_cast<long long>(hits)) - 1;
                    hits &= hits - 1ull;
                    const int j = __ldg(&A.nbr[static_cast<int64_t>(e) * n + s]);
                    const float4 pj = __ldg(&A.pos[j]);
                    float3 d;
                    const float ns = pair_norm_sq(pi, pj, d);
                    const float norm = sqrtf(ns);
                    const float dist = pair_dist(norm, ri, pj.w);
                    const int jd = __ldg(&A.ids[j]);
                    const unsigned long long key = visit_key(P, cx, cy, cz, pj, jd);
                    if (key < last) {
                        ordered = false;
                        break;
                    }
                    last = key;
                    const float4 vj = __ldg(&A.vel[j]);
                    pair_force<HIST>(P, d, norm, dist, vel, mi, vj, jd, f, h, A.counters);
                }
                if (!ordered) {
                    // a cell crossing re-ordered this grain's contacts: redo them in
                    // canonical order
                    f = f_walls;
                    if (HIST) {
                        // springs without a slot so far are counted again below
                        const int seen = __popcll(all_hits) - __popcll(hits) - 1;
                        const int over = out_walls + seen - kHistCap;
                        if (over > 0)
                            atomicAdd(&A.counters[kCntHistOverflow], 0ull - static_cast<unsigned long long>(over));
                        h.out_count = out_walls;
                    }
                    atomicAdd(&A.counters[kCntListResort], 1ull);
                    list_contacts_sorted_mask<HIST>(P, A, s, n, all_hits, pi, vel, mi, cx, cy, cz,
                                                    f, h);
                }
            } else {
                // list overflow: this step built the lists, so the run table is fresh
                list_contacts_table<HIST>(P, A, s, pi, vel, mi, cut, cx, cy, cz, f, h);
            }
        }
        list_integrate<HIST, BATCH, PICARD>(P, A, s, scene, pi, vi, id, f, HIST ? h.out_count : 0,
                                            xb, exact, order_out, disp_bits, step_bits, res_bits);
    }
}

// MINB resident blocks per SM: 5 caps registers at 48 (more warps, a few spills), 4 at
// 64 (no spills); the autotuner picks. The 64-register form also prefetches, into L1,
// each contact's partner id and velocity when the scan finds it, and the grain's first
// stored spring (measured: 2% on a settled column; at 48 registers the prefetches'
// addresses added spills and cost more than they saved).
// PICARD: one backward-Euler / Picard iteration (src/backward_euler_picard_kernel.cu:4-17):
// forces at the iterate (pos, vel), integration from the step-start state (xn, vn), the
// residual max |x_{k+1} - x_k|; an iterate that has left the lists' validity bound marks
// the step for a redo.
template <bool HIST, bool BATCH, int MINB, bool PICARD>
__global__ void __launch_bounds__(kBlock, MINB)
k_force_list(DevParams P0, ListArgs A) {
    if (PICARD ? skipped(A.skip) : list_step_waits(A)) return;
    const int n = P0.n;
    uint32_t disp_bits = 0u, step_bits = 0u;
    uint32_t res_bits = 0u;
    bool viol = false;
    // build positions are read only on the steps that measure the exact displacement;
    // ids only right after a build
    const bool exact = PICARD || A.list_ctrl[kLcExact] != 0u;
    const bool order_out = PICARD || A.list_ctrl[kLcDecision] != 0u;
    // a grid-stride loop: semi-implicit Euler launches one wave (its fused build decision
    // then waits once per block, not once per block of a many-wave grid); Picard launches
    // one slot per thread
    for (int base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        const int s = base + threadIdx.x;
        const bool live = s < n;
        // every per-slot load issued up front: they are independent, and the kernel is
        // bound by their latency when lists are short
        int scene = 0, id = 0, cnt = 0, hcnt_in = 0;
        float4 pi = make_float4(0.f, 0.f, 0.f, 0.f), vi = pi, xb = pi;
        if (live) {
            scene = BATCH ? A.scene[s] : 0;
            pi = A.pos[s];
            vi = A.vel[s];
            id = A.ids[s];
            cnt = A.nbr_cnt[s];
            hcnt_in = HIST ? A.hcnt_in[s] : 0;
            if (exact) xb = A.xbuild[s];
        }
        const bool warp_listed = __any_sync(0xffffffffu, cnt != 0);
        if (live)
            list_grain<HIST, BATCH, PICARD, MINB == 4 && !PICARD>(
                P0, A, s, n, scene, pi, vi, id, cnt, xb, hcnt_in, exact, order_out, warp_listed,
                disp_bits, step_bits, res_bits, viol);
    }
    if (PICARD) {
        list_disp_report(A.list_ctrl, disp_bits);
        list_picard_report(A, res_bits, viol);
    } else {
        list_tail_decide(A, exact, disp_bits, step_bits);
    }
}

// ---- bulk-staged list kernel -------------------------------------------------------
// Persistent warps over tiles of 32 slots. Each warp keeps two tiles in flight: lane 0
// issues the tile's per-slot arrays (x, v, ids, list count, spring count, scene, and
// the build positions on measuring steps) as 1-D bulk copies (cp.async.bulk, the TMA
// engine; each copy reads this GPU's memory into the issuing CTA only) into the warp's
// shared stage, completing on an mbarrier; the lanes compute the tile before while the
// next arrives. The per-slot loads, whose
// latency binds the per-lane kernel, leave the critical path. Contacts, forces and the
// integrator are the per-lane kernel's (list_grain), so the results are identical.
constexpr int kStageWarps = kBlock / 32;
constexpr int kStageTile = 32;
struct __align__(16) SlotStage {
    float4 pos[kStageTile];
    float4 vel[kStageTile];
    float4 xb[kStageTile];
    int ids[kStageTile];
    int cnt[kStageTile];
    int hcnt[kStageTile];
    int scene[kStageTile];
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
// global -> this CTA's shared memory, completing `bytes` on bar (16-byte aligned
// addresses, size a multiple of 16)
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes,
                                         uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0u;
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait for a phase: false after limit_ns without completion.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint64_t limit_ns) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    while (!mbar_try_wait(bar, parity))
        if (global_ns() - t0 > limit_ns) return false;
    return true;
}

template <bool HIST, bool BATCH>
__device__ __forceinline__ void stage_issue(const ListArgs& A, int tile, bool exact,
                                            SlotStage& S, uint64_t* bar) {
    const int s0 = tile * kStageTile;
    constexpr uint32_t f4 = kStageTile * sizeof(float4), i4 = kStageTile * sizeof(int);
    const uint32_t bytes = 2u * f4 + 2u * i4 + (HIST ? i4 : 0u) + (BATCH ? i4 : 0u) +
                           (exact ? f4 : 0u);
    mbar_expect_tx(bar, bytes);
    bulk_g2s(S.pos, A.pos + s0, f4, bar);
    bulk_g2s(S.vel, A.vel + s0, f4, bar);
    bulk_g2s(S.ids, A.ids + s0, i4, bar);
    bulk_g2s(S.cnt, A.nbr_cnt + s0, i4, bar);
    if (HIST) bulk_g2s(S.hcnt, A.hcnt_in + s0, i4, bar);
    if (BATCH) bulk_g2s(S.scene, A.scene + s0, i4, bar);
    if (exact) bulk_g2s(S.xb, A.xbuild + s0, f4, bar);
}

// MINB: resident blocks per SM (5: 48 registers per thread, 4: 64). Tiles: warp w of W
// takes tiles w, w + W, w + 2W, ... (claiming the last rounds from a shared counter
// instead was measured slower: the claims serialize on one address just when every
// warp needs its next tile).
template <bool HIST, bool BATCH, int MINB>
__global__ void __launch_bounds__(kBlock, MINB)
k_force_list_staged(DevParams P0, ListArgs A) {
    if (list_step_waits(A)) return;
    __shared__ SlotStage stage[kStageWarps][2];
    __shared__ uint64_t bars[kStageWarps][2];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int n = P0.n;
    const int tiles = (n + kStageTile - 1) / kStageTile;
    const int whole = n / kStageTile;  // tiles with 32 slots go through the stages
    const int W = gridDim.x * kStageWarps;
    const int first = blockIdx.x * kStageWarps + w;
    const bool exact = A.list_ctrl[kLcExact] != 0u;
    const bool order_out = A.list_ctrl[kLcDecision] != 0u;  // first step after a build
    const uint32_t wait_us = A.list_ctrl[kLcWaitUs];
    const uint64_t limit_ns = wait_us ? 1000ull * wait_us : 1000000000ull;
    const bool stall_test = A.list_ctrl[kLcStallTest] != 0u;
    SlotStage* S = stage[w];
    uint64_t* bar = bars[w];
    // tiles of iterations it (cur, in stage it & 1) and it + 1 (nxt), in registers
    int cur = first, nxt = first + W;
    if (lane == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_init_fence();
        if (cur < whole) {
            if (stall_test) mbar_expect_tx(&bar[0], 16u);   // nothing will arrive
            else stage_issue<HIST, BATCH>(A, cur, exact, S[0], &bar[0]);
        }
        if (nxt < whole) stage_issue<HIST, BATCH>(A, nxt, exact, S[1], &bar[1]);
    }
    __syncwarp();
    uint32_t disp_bits = 0u, step_bits = 0u, res_bits = 0u;
    bool viol = false, failed = false;
    int it = 0;
    for (;; ++it) {
        const int st = it & 1;
        const int t = cur;
        if (t >= tiles) break;
        const int s = t * kStageTile + lane;
        float4 pi = make_float4(0.f, 0.f, 0.f, 0.f), vi = pi, xb = pi;
        int id = 0, cnt = 0, hcnt_in = 0, scene = 0;
        if (t < whole) {
            const bool ok = __all_sync(0xffffffffu, mbar_wait(&bar[st], (it >> 1) & 1, limit_ns));
            if (!ok) {
                failed = true;
                break;
            }
            const SlotStage& T = S[st];
            pi = T.pos[lane];
            vi = T.vel[lane];
            id = T.ids[lane];
            cnt = T.cnt[lane];
            if (HIST) hcnt_in = T.hcnt[lane];
            if (BATCH) scene = T.scene[lane];
            if (exact) xb = T.xb[lane];
            __syncwarp();
            // the stage is read: refill it with the tile two ahead
            const int tn = nxt + W;
            if (lane == 0 && tn < whole) stage_issue<HIST, BATCH>(A, tn, exact, S[st], &bar[st]);
            cur = nxt;
            nxt = tn;
        } else {
            // the ragged last tile: plain loads, nothing after it
            cur = nxt;
            nxt = tiles;
            if (s < n) {
                pi = A.pos[s];
                vi = A.vel[s];
                id = A.ids[s];
                cnt = A.nbr_cnt[s];
                if (HIST) hcnt_in = A.hcnt_in[s];
                if (BATCH) scene = A.scene[s];
                if (exact) xb = A.xbuild[s];
            }
        }
        const bool warp_listed = __any_sync(0xffffffffu, cnt != 0);
        if (s < n)
            list_grain<HIST, BATCH, false>(P0, A, s, n, scene, pi, vi, id, cnt, xb, hcnt_in,
                                           exact, order_out, warp_listed, disp_bits,
                                           step_bits, res_bits, viol);
    }
    if (failed) {
        // a stage never completed: flag it and drain what this warp still has in flight
        // (bounded); the step is left unfinished for the host to report
        if (lane == 0) {
            atomicAdd(&A.counters[kCntStageTimeout], 1ull);
            if (cur < whole) mbar_wait(&bar[it & 1], (it >> 1) & 1, limit_ns);
            if (nxt < whole) mbar_wait(&bar[(it + 1) & 1], ((it + 1) >> 1) & 1, limit_ns);
        }
        disp_bits = step_bits = 0u;   // and its displacements unreported
    }
    list_tail_decide(A, exact, disp_bits, step_bits);
}

// ---- list build with the tile's neighbour window staged in shared memory ----------
// One block per 256 consecutive sorted slots (single scene). Every grain's candidates
// lie in its nine stencil rows (three z-consecutive cells of one column each, one slot
// range per row); over the tile, row r's ranges lie inside [min lo_r, max hi_r). Those
// nine hulls, merged where they overlap (consecutive columns of one x-plane are
// consecutive in slot order), are copied into shared memory once by bulk copies
// (cp.async.bulk, this GPU's memory into this CTA, completing on an mbarrier), and the
// threads read their candidates there: 27 position loads per grain from L2 become a
// few per grain. A window above kWinCap positions, or a copy that does not complete
// within the bounded wait, falls back to global loads. Same lists, same order.
constexpr int kWinCap = 2560;   // positions (40 KB): five blocks per SM

__global__ void __launch_bounds__(kBlock)
k_list_build_tiled(DevParams P, const float4* __restrict__ pos, const int2* __restrict__ table,
                   int* __restrict__ nbr, int* __restrict__ nbr_cnt, float4* __restrict__ xbuild,
                   uint32_t* __restrict__ ctrl, ListCopy cp, Skip skip,
                   unsigned long long* __restrict__ counters) {
    if (skipped(skip)) return;
    __shared__ float4 win[kWinCap];
    __shared__ int hull_lo[9], hull_hi[9], row_off[9];
    __shared__ int staged;
    __shared__ __align__(8) uint64_t bar;
    const int n = P.n;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = s < n;
    if (threadIdx.x < 9) {
        hull_lo[threadIdx.x] = 0x7fffffff;
        hull_hi[threadIdx.x] = 0;
    }
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_init_fence();
    }
    float4 pi = make_float4(0.f, 0.f, 0.f, 0.f);
    int lo[9], hi[9];
#pragma unroll
    for (int r = 0; r < 9; ++r) {
        lo[r] = 0x7fffffff;
        hi[r] = 0;
    }
    if (live) {
        pi = pos[s];
        cp.pos_out[s] = pi;
        cp.vel_out[s] = cp.vel[s];
        cp.ids_out[s] = cp.ids[s];
        if (cp.hcnt) cp.hcnt_out[s] = cp.hcnt[s];
        int cx, cy, cz;
        cell_coords(P, pi.x, pi.y, pi.z, cx, cy, cz);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int nx = cx + r - 1;
            if (nx >= 0 && nx < P.grid[0]) row_ranges(P, table, nx, cy, cz, lo + 3 * r, hi + 3 * r);
        }
    }
    __syncthreads();   // hull initialisation and the barrier's init visible
    if (live) {
#pragma unroll
        for (int r = 0; r < 9; ++r) {
            if (lo[r] < hi[r]) {
                atomicMin(&hull_lo[r], lo[r]);
                atomicMax(&hull_hi[r], hi[r]);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        // merge the nine hulls into disjoint ranges (ascending), stage them if they fit
        int idx[9], m = 0;
        for (int r = 0; r < 9; ++r)
            if (hull_lo[r] < hull_hi[r]) idx[m++] = r;
        for (int a = 1; a < m; ++a) {          // insertion sort by hull start
            const int v = idx[a];
            int b = a - 1;
            while (b >= 0 && hull_lo[idx[b]] > hull_lo[v]) {
                idx[b + 1] = idx[b];
                --b;
            }
            idx[b + 1] = v;
        }
        int mlo[9], mhi[9], nm = 0, total = 0;
        for (int a = 0; a < m; ++a) {
            const int r = idx[a];
            if (nm > 0 && hull_lo[r] <= mhi[nm - 1]) {
                mhi[nm - 1] = max(mhi[nm - 1], hull_hi[r]);
            } else {
                mlo[nm] = hull_lo[r];
                mhi[nm] = hull_hi[r];
                ++nm;
            }
        }
        for (int k = 0; k < nm; ++k) total += mhi[k] - mlo[k];
        const bool fits = nm > 0 && total <= kWinCap;
        staged = fits ? 1 : 0;
        if (fits) {
            int base[9];
            int acc = 0;
            for (int k = 0; k < nm; ++k) {
                base[k] = acc;
                acc += mhi[k] - mlo[k];
            }
            for (int a = 0; a < m; ++a) {
                const int r = idx[a];
                int k = 0;
                while (!(hull_lo[r] >= mlo[k] && hull_hi[r] <= mhi[k])) ++k;
                row_off[r] = base[k] - mlo[k];
            }
            mbar_expect_tx(&bar, static_cast<uint32_t>(total) * 16u);
            for (int k = 0; k < nm; ++k)
                bulk_g2s(&win[base[k]], pos + mlo[k], static_cast<uint32_t>(mhi[k] - mlo[k]) * 16u, &bar);
        }
    }
    __syncthreads();
    bool use_win = staged != 0;
    if (use_win) {
        const bool ok = mbar_wait(&bar, 0u, 1000000000ull);
        if (!__syncthreads_and(ok)) {
            if (threadIdx.x == 0) atomicAdd(&counters[kCntStageTimeout], 1ull);
            use_win = false;
        }
    }
    if (!live) return;
    int cnt = 0;
    auto visit = [&](int j, float4 pj) {
        if (j == s) return;
        float3 d;
        const float ns = pair_norm_sq(pi, pj, d);
        const float reach = (pi.w + pj.w) + P.skin;
        if (ns < reach * reach) {
            if (cnt < kNbrCap) nbr[static_cast<int64_t>(cnt) * n + s] = j;
            ++cnt;
        }
    };
#pragma unroll
    for (int r = 0; r < 9; ++r) {
        int j = lo[r];
        const int e = hi[r];
        if (use_win) {
            if (j < e) {
                const float4* w = win + row_off[r];
                for (; j < e; ++j) visit(j, w[j]);
            }
        } else {
            for (; e - j > 1; j += 2) {
                const float4 a = __ldg(&pos[j]);
                const float4 b = __ldg(&pos[j + 1]);
                visit(j, a);
                visit(j + 1, b);
            }
            if (j < e) visit(j, __ldg(&pos[j]));
        }
    }
    if ((pi.w + P.rmax) + P.skin > P.cell_min) {
        // the outer shell, from global memory (the window holds the stencil only)
        int cx, cy, cz;
        cell_coords(P, pi.x, pi.y, pi.z, cx, cy, cz);
        list_far_shell(P, table, pos, pi, cx, cy, cz, visit);
    }
    nbr_cnt[s] = cnt;
    xbuild[s] = pi;
    if (cnt > kNbrCap) atomicOr(&ctrl[kLcOverflow], 1u);
}

// The last executed Picard iteration k wrote the B buffers when k is even and the
// scratch buffers when k is odd (iterations alternate, starting in B).
__global__ void __launch_bounds__(kBlock)
k_list_finalize(int n, const int* __restrict__ used, const float4* __restrict__ xpos,
                const float4* __restrict__ xvel, float4* __restrict__ pos,
                float4* __restrict__ vel) {
    if ((*used & 1) != 0) return;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    pos[s] = xpos[s];
    vel[s] = xvel[s];
}

__global__ void k_list_picard_check(uint32_t* __restrict__ ctrl,
                                    unsigned long long* __restrict__ counters, int use_cond,
                                    cudaGraphConditionalHandle cond) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const bool redo = ctrl[kLcViol] != 0u;
    ctrl[kLcViol] = 0u;
    ctrl[kLcRedo] = redo ? __float_as_uint(1.f) : 0u;
    if (redo) {
        ctrl[kLcForce] = 1u;  // the redo re-sorts the state: build next step
        counters[kCntPicardRedos] += 1ull;
        counters[kCntHistOverflow] = counters[kCntHistBefore];  // the redo counts its own
    }
    if (use_cond) cudaGraphSetConditional(cond, redo ? 1u : 0u);
}

// Contact-parallel list kernel: a warp finds the contacts of its grains, then its lanes
// evaluate those contacts together, one each (distance, dashpot, spring lookup, Coulomb
// cap), and every grain adds its own contacts' terms in order. A lane evaluating its
// grain's contacts alone runs as many rounds of that long code as the busiest of its 32
// grains has contacts, with about one lane in four active.
//
// LPG lanes share one grain (a warp holds 32 / LPG grains): they scan its list side by
// side, and the walls, the accumulation and the integrator run on the first of them.
//
// Per warp: the scan leaves each grain a bitmask of the list entries in contact; a prefix
// sum over the grains numbers the warp's contacts; up to 32 at a time (whole grains) they
// are queued in shared memory as (owner lane, entry) and evaluated, the new springs going
// to their final rows and the terms to shared memory, from where each owner adds its run.
// List order is the canonical order unless a cell crossing changed it: where a contact's
// visiting key is below its predecessor's, the grain's contacts take their places by the
// rank of their keys. (The per-lane kernels redo such a grain alone, a chain of about 30 us
// for the busiest: a few hundred such grains in a million set the kernel's time.)
//
// The slots' own values come through shared memory by asynchronous copies issued one
// group ahead, which hides their latency without holding registers. What the stages take of
// the SM's 256 KB L1 loses: with 16.6 KB a block (the 164 KB carve-out) the steps of large
// scenes took 1% longer than with 15.6 KB (132 KB), with 20.7 KB (list entries staged too,
// 196 KB) 5% longer. Only batches stage the scene.
//
// Bound by load latency and issue (1,475 warp instructions per 32 packed grains, 328 per 32
// falling ones; half the chip's warps, an instruction every second cycle). Measured at 64
// registers, 8 blocks per SM (80 and 6 for Picard, whose grid is not one wave of equal work)
// against the per-lane kernel, single step graphs: 2^20 falling grains 41.3 us a step against
// 42.3; 1,000,003 packed grains (8 list entries, 0.4 springs each) 134 against 176; 200,003
// packed, 8 Picard iterations 230 against 492. In chains, with the build, now 36.0, 119 and
// 225. A settled 2^20-grain layer (1.5 entries, a floor spring each) takes 108, the per-lane
// kernel at 64 registers 96: there the tuner takes that one; 32,768 settled grains 14.9
// against 15.9.
constexpr int kCoopBlock = 128;
constexpr int kCoopWarps = kCoopBlock / 32;

template <bool BATCH>
struct __align__(16) CoopStage {
    float4 pos[32], vel[32];
    int id[32], cnt[32], hcnt[32];
    int scene[BATCH ? 32 : 1];
};
template <>
struct __align__(16) CoopStage<false> {
    float4 pos[32], vel[32];
    int id[32], cnt[32], hcnt[32];
    static constexpr int* scene = nullptr;
};
template <bool BATCH>
struct __align__(16) CoopWarp {
    CoopStage<BATCH> stage[2];
    float4 term[32][2];            // (nrm, fp), (t, cvn)
    unsigned short queue[32];      // owner lane << 6 | list entry
};

__device__ __forceinline__ void async_copy16(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void async_copy4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// This lane's share of the copies of one slot group into S: the lane that carries grain s
// copies its values. One copy group per call, possibly empty.
template <bool HIST, bool BATCH, int LPG>
__device__ __forceinline__ void coop_stage(const ListArgs& A, CoopStage<BATCH>& S, int s, int n) {
    const int lane = threadIdx.x & 31, g = lane / LPG;
    if (lane % LPG == 0 && s < n) {
        async_copy16(&S.pos[g], &A.pos[s]);
        async_copy16(&S.vel[g], &A.vel[s]);
        async_copy4(&S.cnt[g], &A.nbr_cnt[s]);
        async_copy4(&S.id[g], &A.ids[s]);
        if (HIST) async_copy4(&S.hcnt[g], &A.hcnt_in[s]);
        if (BATCH) async_copy4(&S.scene[g], &A.scene[s]);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// The contacts of one grain on its own lane: a list that overflowed (this step built the
// lists, so the run table is fresh), or more contacts than one round holds. (Out of line it
// cost the packed step 7%: the call's saved registers.)
struct AloneResult {
    float3 f;
    int out_count;
};
template <bool HIST>
__device__ __forceinline__ AloneResult coop_alone(const DevParams& P, const ListArgs& A, float4 pi, float4 vi,
                                               int id, int hcnt_in, int s, int n, int cnt,
                                               unsigned long long hits, float3 f, int out_count) {
    HistRow h;
    if (HIST) {
        h.in = A.hist_in + static_cast<int64_t>(id) * kHistCap;
        h.in_count = hcnt_in;
        h.out = A.hist_out + static_cast<int64_t>(id) * kHistCap;
    }
    h.out_count = out_count;
    const float3 vel = make_float3(vi.x, vi.y, vi.z);
    int cx, cy, cz;
    cell_coords(P, pi.x, pi.y, pi.z, cx, cy, cz);
    if (cnt > kNbrCap)
        list_contacts_table<HIST>(P, A, s, pi, vel, vi.w, contact_cutoff_sq(pi.w, P.rmax), cx, cy, cz, f, h);
    else
        list_contacts_sorted_mask<HIST>(P, A, s, n, hits, pi, vel, vi.w, cx, cy, cz, f, h);
    return {f, h.out_count};
}

// One slot per group of LPG lanes (all lanes of the warp together; s may be >= n).
template <bool HIST, bool BATCH, bool PICARD, int LPG>
__device__ __forceinline__ void coop_slot(const DevParams& P0, const ListArgs& A, CoopWarp<BATCH>& W,
                                          const CoopStage<BATCH>& S, int s, int n, bool exact,
                                          bool order_out, uint32_t& disp_bits, uint32_t& step_bits,
                                          uint32_t& res_bits, bool& viol) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, sub = lane % LPG, g = lane / LPG;
    const bool live = s < n;
    const int scene = BATCH && live ? S.scene[g] : 0;
    const DevParams& P = BATCH ? A.scene_params[scene] : P0;
    const bool frozen = BATCH && live && P.frozen;
    const bool own = live && sub == 0;      // the lane that carries the grain
    const bool work = own && !frozen;
    int cnt = live && !frozen ? S.cnt[g] : 0;
    float3 f = make_float3(0.f, 0.f, 0.f);
    int out_walls = 0, out_count = 0;
    if (PICARD && own) {
        // the rhs of a Picard step pairs the last iterate's velocity with its forces
        A.rhs_vel[s] = S.vel[g];
        A.rhs_ids[s] = S.id[g];
        if (A.iter > 0) {
            const float4 xb = A.xbuild[s], x = S.pos[g];
            const float ex = x.x - xb.x, ey = x.y - xb.y, ez = x.z - xb.z;
            viol |= !(ex * ex + ey * ey + ez * ez < A.viol_thr) || cnt > kNbrCap;
        }
    }
    if (work) {
        const float4 x = S.pos[g], v = S.vel[g];
        HistRow h;
        if (HIST) {
            h.in = A.hist_in + static_cast<int64_t>(S.id[g]) * kHistCap;
            h.in_count = S.hcnt[g];
            h.out = A.hist_out + static_cast<int64_t>(S.id[g]) * kHistCap;
            h.out_count = 0;
        }
        wall_forces<HIST>(P, make_float3(x.x, x.y, x.z), make_float3(v.x, v.y, v.z), x.w, v.w, f, h,
                          A.counters);
        if (HIST) out_walls = out_count = h.out_count;
    }
    if (__any_sync(kAll, cnt != 0)) {
        // scan: this lane's entries, four entries' loads in flight at a time
        unsigned long long hits = 0ull;
        const int scan = cnt <= kNbrCap ? cnt : 0;
        const float4 pi = S.pos[g];
        for (int e0 = sub; e0 < scan; e0 += 4 * LPG) {
            int jj[4];
            float4 pp[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = e0 + u * LPG;
                jj[u] = e < scan ? __ldg(&A.nbr[static_cast<int64_t>(e) * n + s]) : s;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) pp[u] = __ldg(&A.pos[jj[u]]);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = e0 + u * LPG;
                if (e < scan && entry_hit(pi, pp[u])) hits |= 1ull << e;
            }
        }
#pragma unroll
        for (int o = 1; o < LPG; o <<= 1) hits |= __shfl_xor_sync(kAll, hits, o);
        if (cnt > kNbrCap || __popcll(hits) > 32) {
            if (work) {
                const AloneResult r = coop_alone<HIST>(P, A, S.pos[g], S.vel[g], S.id[g],
                                                       HIST ? S.hcnt[g] : 0, s, n, cnt, hits, f, out_count);
                f = r.f;
                out_count = r.out_count;
            }
            hits = 0ull;
        }
        if (__any_sync(kAll, hits != 0ull)) {
            // number the warp's contacts, grain by grain
            const int c = __popcll(hits);
            int upto = sub == 0 ? c : 0;
#pragma unroll
            for (int o = LPG; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(kAll, upto, o);
                if (lane >= o) upto += y;
            }
            if (LPG > 1) upto = __shfl_sync(kAll, upto, lane - sub);
            const int off = upto - c;
            const int total = __shfl_sync(kAll, upto, 31);
            unsigned long long left = sub == 0 ? hits : 0ull;
            int at = off;
            for (int base = 0, end; base < total; base = end) {
                // up to 32 contacts, all of each grain's (none has more than 32 here)
                end = static_cast<int>(__reduce_max_sync(kAll, static_cast<unsigned>(upto <= base + 32 ? upto : 0)));
                for (; left && at < end; ++at) {
                    W.queue[at - base] = static_cast<unsigned short>(
                        (lane << 6) | (__ffsll(static_cast<long long>(left)) - 1));
                    left &= left - 1ull;
                }
                __syncwarp();
                const bool active = base + lane < end;
                const int q = active ? W.queue[lane] : 0;
                const int o = q >> 6, e = q & 63;
                const int so = __shfl_sync(kAll, s, o);
                const int oo = __shfl_sync(kAll, off, o);
                const int first = HIST ? __shfl_sync(kAll, out_walls, o) : 0;
                int r = base + lane - oo;   // the contact's place among its grain's
                unsigned long long key = 0ull;
                PairTerms t;
                float3 xi = make_float3(0.f, 0.f, 0.f);
                int io = 0, jd = 0;
                if (active) {
                    const int go = o / LPG;
                    const DevParams& Q = BATCH ? A.scene_params[S.scene[go]] : P0;
                    const int j = __ldg(&A.nbr[static_cast<int64_t>(e) * n + so]);
                    const float4 po = S.pos[go], vo = S.vel[go];
                    const float4 pj = __ldg(&A.pos[j]), vj = __ldg(&A.vel[j]);
                    jd = __ldg(&A.ids[j]);
                    if (HIST) {
                        io = S.id[go];
                        const int row = S.hcnt[go];
                        if (row > 0) {
                            // rows keep the visiting order, so a lasting contact is about
                            // where it was
                            HistRow h;
                            h.in = A.hist_in + static_cast<int64_t>(io) * kHistCap;
                            h.in_count = row;
                            h.cursor = min(first + r, row - 1);
                            xi = find_spring(h, jd);
                        }
                    }
                    int cx, cy, cz;
                    cell_coords(Q, po.x, po.y, po.z, cx, cy, cz);
                    key = visit_key(Q, cx, cy, cz, pj, jd);
                    float3 d;
                    const float ns = pair_norm_sq(po, pj, d);
                    const float norm = sqrtf(ns);
                    const float dist = pair_dist(norm, po.w, pj.w);
                    t = pair_terms<HIST>(Q, d, norm, dist, make_float3(vo.x, vo.y, vo.z), vo.w, vj, xi);
                }
                const unsigned long long up_key = __shfl_up_sync(kAll, key, 1);
                const int up_owner = __shfl_up_sync(kAll, o, 1);
                const unsigned bad = __reduce_or_sync(
                    kAll, active && lane > 0 && up_owner == o && key < up_key ? 1u << o : 0u);
                if (bad) {
                    // a cell crossing re-ordered these grains' contacts: each takes the place
                    // of its key's rank
                    int rank = 0;
                    const int owner = active ? o : -1;
                    for (int k = 0; k < 32; ++k) {
                        const unsigned long long key_k = __shfl_sync(kAll, key, k);
                        const int owner_k = __shfl_sync(kAll, owner, k);
                        if (owner_k == o && key_k < key) ++rank;
                    }
                    if ((bad >> o) & 1u) r = rank;
                    if (lane == 0)
                        atomicAdd(&A.counters[kCntListResort], static_cast<unsigned long long>(__popc(bad)));
                }
                if (active) {
                    const int place = oo + r - base;
                    W.term[place][0] = make_float4(t.nrm.x, t.nrm.y, t.nrm.z, t.fp);
                    W.term[place][1] = make_float4(t.t.x, t.t.y, t.t.z, t.cvn);
                    if (HIST && first + r < kHistCap)
                        A.hist_out[static_cast<int64_t>(io) * kHistCap + first + r] =
                            make_float4(xi.x, xi.y, xi.z, __int_as_float(jd));
                }
                __syncwarp();
                if (sub == 0) {
                    // a grain of this round has all its contacts in it
                    const int e1 = upto <= end ? upto - base : 0;
                    for (int k = max(off - base, 0); k < e1; ++k) {
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
            if (HIST && work && c > 0) {
                out_count = min(out_walls + c, kHistCap);
                if (out_walls + c > kHistCap)
                    atomicAdd(&A.counters[kCntHistOverflow],
                              static_cast<unsigned long long>(out_walls + c - kHistCap));
            }
        }
    }
    if (work) {
        // the slot's values are read again from the stage, not held in registers meanwhile
        const float4 x = S.pos[g], v = S.vel[g];
        const float4 xb = exact ? A.xbuild[s] : x;
        list_integrate<HIST, BATCH, PICARD>(P, A, s, scene, x, v, S.id[g], f,
                                            out_count, xb, exact, order_out, disp_bits,
                                            step_bits, res_bits);
    } else if (own) {
        list_copy_frozen<HIST>(A, s, scene, S.pos[g], S.vel[g], S.id[g], order_out);
    }
}

// Grid-stride over groups of slots; semi-implicit Euler in one wave, so that the fused
// build decision waits once per resident block.
template <bool HIST, bool BATCH, bool PICARD, int LPG>
__global__ void __launch_bounds__(kCoopBlock, PICARD ? 6 : 8)
k_force_list_coop(const __grid_constant__ DevParams P0, const __grid_constant__ ListArgs A) {
    if (PICARD && skipped(A.skip)) return;
    if (!PICARD) {
        // an early launch: nothing of the step before is touched until it has ended
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    __shared__ CoopWarp<BATCH> warps[kCoopWarps];
    CoopWarp<BATCH>& W = warps[threadIdx.x >> 5];
    const int n = P0.n;
    const bool waits = !PICARD && list_step_waits(A);
    const bool exact = PICARD || A.list_ctrl[kLcExact] != 0u;
    const bool order_out = PICARD || A.list_ctrl[kLcDecision] != 0u;  // first step after a build
    uint32_t disp_bits = 0u, step_bits = 0u, res_bits = 0u;
    bool viol = false;
    // the next group's values are on their way while this one is computed
    constexpr int per = kCoopBlock / LPG;   // slots per block
    const int stride = gridDim.x * per;
    int s = blockIdx.x * per + static_cast<int>(threadIdx.x) / LPG;
    coop_stage<HIST, BATCH, LPG>(A, W.stage[0], s, n);
    if (waits) {
        // (asked after the first copies are issued: one round trip less before the work)
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        return;
    }
    int st = 0;
    for (int base = blockIdx.x * per; base < n; base += stride, s += stride, st ^= 1) {
        __syncwarp();                       // the other stage has been read
        coop_stage<HIST, BATCH, LPG>(A, W.stage[st ^ 1], s + stride, n);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();                       // every lane's copies have arrived
        coop_slot<HIST, BATCH, PICARD, LPG>(P0, A, W, W.stage[st], s, n, exact, order_out, disp_bits,
                                            step_bits, res_bits, viol);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (PICARD) {
        list_disp_report(A.list_ctrl, disp_bits);
        list_picard_report(A, res_bits, viol);
    } else {
        list_tail_decide(A, exact, disp_bits, step_bits);
    }
}

__global__ void __launch_bounds__(kBlock)
k_list_length(int n, const int* __restrict__ cnt, unsigned long long* __restrict__ out) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long v = s < n ? static_cast<unsigned long long>(min(cnt[s], kNbrCap + 1)) : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(out, v);
}

}  // namespace

void launch_list_decide(uint32_t* list_ctrl, float thr, bool always_exact,
                        unsigned long long* counters, unsigned long long* pend, bool use_cond,
                        cudaGraphConditionalHandle cond, cudaStream_t st) {
    k_list_decide<<<1, 32, 0, st>>>(list_ctrl, thr, always_exact ? 1 : 0, counters, pend,
                                    use_cond ? 1 : 0, cond);
}

void launch_cell_load(const DevParams& P, const float4* pos, const float4* xbuild, uint32_t* load,
                      uint32_t* list_ctrl, Skip skip, cudaStream_t st) {
    k_cell_clear<<<blocks_for(P.n), kBlock, 0, st>>>(P, xbuild, load, skip);
    k_cell_load<<<blocks_for(P.n), kBlock, 0, st>>>(P, pos, load, list_ctrl, skip);
}

void launch_list_build(const DevParams& P, SceneTab T, const float4* pos, const int2* table,
                       int* nbr, int* nbr_cnt, float4* xbuild, uint32_t* list_ctrl,
                       const ListCopy& cp, Skip skip, unsigned long long* counters, bool tiled,
                       cudaStream_t st) {
    if (tiled && !T.params) {
        k_list_build_tiled<<<blocks_for(P.n), kBlock, 0, st>>>(P, pos, table, nbr, nbr_cnt, xbuild,
                                                               list_ctrl, cp, skip, counters);
        return;
    }
    auto go = [&](auto lanes) {
        constexpr int L = decltype(lanes)::value;
        const int nb = blocks_for(P.n, kBlock / L);
        if (T.params)
            k_list_build<true, L><<<nb, kBlock, 0, st>>>(P, T, pos, table, nbr, nbr_cnt, xbuild,
                                                         list_ctrl, cp, skip);
        else
            k_list_build<false, L><<<nb, kBlock, 0, st>>>(P, T, pos, table, nbr, nbr_cnt, xbuild,
                                                          list_ctrl, cp, skip);
    };
    // Lanes per grain: as many as the chip has room for while a build is one warp's latency.
    // Upload, build and one step with 32 / 8 / 1 lanes: 1,000 grains 84 / 87 / 92 us, 5,000
    // 93.2 / 95.0 / 96.8, 8,000 96.2 / 95.9 / 98.9, 20,000 107.8 / 96.6 / 100.2, 30,000
    // 121 / 107.6 / 107.5, 50,000 142 / 111 / 106.
    if (P.n < 6144) go(std::integral_constant<int, 32>());
    else if (P.n < 24576) go(std::integral_constant<int, 8>());
    else go(std::integral_constant<int, 1>());
}

void launch_list_copy(int n, const float4* pos, const float4* vel, const int* ids,
                      const int* hcnt, const int* scene, float4* pos_out, float4* vel_out,
                      int* ids_out, int* hcnt_out, int* scene_out, Skip skip, cudaStream_t st) {
    k_list_copy<<<blocks_for(n), kBlock, 0, st>>>(n, pos, vel, ids, hcnt, scene, pos_out,
                                                  vel_out, ids_out, hcnt_out, scene_out, skip);
}

// Blocks of one full wave of a kernel at `block` threads (a multiple of 32 up to 256):
// the SM count times the resident blocks per SM, cached per kernel, device and block
// size (devices beyond the first 64 query each time).
template <auto Kernel>
int one_wave(int block) {
    constexpr int kDevs = 64;
    static int cache[kDevs][9] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    int local = 0;
    int& occ = (dev >= 0 && dev < kDevs) ? cache[dev][(block / 32) % 9] : local;
    if (occ == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, Kernel, block, 0);
        occ = occ < 1 ? 1 : occ;
    }
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms * occ;
}

template <bool HIST, bool BATCH, int MINB>
void force_list_staged(const DevParams& P, const ListArgs& a, cudaStream_t st) {
    // persistent: as many blocks as fit at once, at most one warp per tile
    const int tiles = (P.n + kStageTile - 1) / kStageTile;
    const int want = (tiles + kStageWarps - 1) / kStageWarps;
    const int nb = std::min(want, one_wave<k_force_list_staged<HIST, BATCH, MINB>>(kBlock));
    k_force_list_staged<HIST, BATCH, MINB><<<nb < 1 ? 1 : nb, kBlock, 0, st>>>(P, a);
}

template <bool HIST, bool BATCH, int MINB, bool PICARD>
void force_list_launch(const DevParams& P, const ListArgs& a, cudaStream_t st, int block) {
    int nb = blocks_for(P.n, block);
    // semi-implicit Euler: one wave (grid-stride), so the fused build decision's
    // per-block wait happens once per resident block
    if (!PICARD) nb = std::min(nb, one_wave<k_force_list<HIST, BATCH, MINB, PICARD>>(block));
    k_force_list<HIST, BATCH, MINB, PICARD><<<nb, block, 0, st>>>(P, a);
}

template <int MINB, bool PICARD>
void force_list_variant(const DevParams& P, const ListArgs& a, cudaStream_t st, int block) {
    const bool batch = a.scene_params != nullptr;
    if (P.history) {
        if (batch) force_list_launch<true, true, MINB, PICARD>(P, a, st, block);
        else force_list_launch<true, false, MINB, PICARD>(P, a, st, block);
    } else {
        if (batch) force_list_launch<false, true, MINB, PICARD>(P, a, st, block);
        else force_list_launch<false, false, MINB, PICARD>(P, a, st, block);
    }
}

template <bool HIST, bool BATCH, bool PICARD, int LPG>
void force_list_coop_launch(const DevParams& P, const ListArgs& a, cudaStream_t st) {
    const int per = kCoopBlock / LPG;
    const int wave = one_wave<k_force_list_coop<HIST, BATCH, PICARD, LPG>>(kCoopBlock);
    const int nb = std::min((P.n + per - 1) / per, wave);
    // An early launch hides the next step's launch where both grids are resident at once (up to
    // 75776 grains): 32768 falling grains 11.1 -> 10.7 us a step, 5120 in 24-step runs 776 ->
    // 760 us. Blocks that wait for room gain nothing (2^20 grains 0.5%) or cost (24 scenes,
    // 600 thousand grains, -1.7%).
    const bool overlap = !PICARD && a.early != 0 && 2 * nb <= wave;
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(nb);
    cfg.blockDim = dim3(kCoopBlock);
    cfg.stream = st;
    cfg.attrs = &early;
    cfg.numAttrs = overlap ? 1 : 0;
    cudaLaunchKernelEx(&cfg, k_force_list_coop<HIST, BATCH, PICARD, LPG>, P, a);
}

template <bool PICARD, int LPG>
void force_list_coop_lanes(const DevParams& P, const ListArgs& a, cudaStream_t st) {
    const bool batch = a.scene_params != nullptr;
    if (P.history) {
        if (batch) force_list_coop_launch<true, true, PICARD, LPG>(P, a, st);
        else force_list_coop_launch<true, false, PICARD, LPG>(P, a, st);
    } else {
        if (batch) force_list_coop_launch<false, true, PICARD, LPG>(P, a, st);
        else force_list_coop_launch<false, false, PICARD, LPG>(P, a, st);
    }
}

template <bool PICARD>
void force_list_coop(const DevParams& P, const ListArgs& a, cudaStream_t st) {
    // Four lanes a grain where one each would leave most of the chip idle and the step is
    // one warp's latency: 2^10 packed grains with springs 20.1 vs 21.4 us a step, 5,000 22.0
    // vs 23.9, 10,000 24.3 vs 26.0, 20,000 25.5 vs 26.1, 40,000 30.4 vs 27.0.
    if (P.n < 16384) force_list_coop_lanes<PICARD, 4>(P, a, st);
    else force_list_coop_lanes<PICARD, 1>(P, a, st);
}

void launch_list_finalize(int n, const int* picard_used, const float4* xpos,
                          const float4* xvel, float4* pos, float4* vel, cudaStream_t st) {
    k_list_finalize<<<blocks_for(n), kBlock, 0, st>>>(n, picard_used, xpos, xvel, pos, vel);
}

void launch_list_picard_check(uint32_t* list_ctrl, unsigned long long* counters, bool use_cond,
                              cudaGraphConditionalHandle cond, cudaStream_t st) {
    k_list_picard_check<<<1, 32, 0, st>>>(list_ctrl, counters, use_cond ? 1 : 0, cond);
}

void launch_force_list(const DevParams& P, const ListArgs& a, cudaStream_t st, int block,
                       int min_blocks, bool picard) {
    if (min_blocks == 0) {
        if (picard) force_list_coop<true>(P, a, st);
        else force_list_coop<false>(P, a, st);
        return;
    }
    if (picard) {
        // the per-lane kernel (the bulk-staged one has no Picard form)
        if (min_blocks == 4) force_list_variant<4, true>(P, a, st, block == 0 ? kBlock : block);
        else force_list_variant<5, true>(P, a, st, block);
        return;
    }
    if (min_blocks == 1 || min_blocks == 2) {
        // bulk-staged persistent kernel (kBlock threads; 1: 48 registers, 2: 64)
        const bool batch = a.scene_params != nullptr;
        const bool r64 = min_blocks == 2;
        if (P.history) {
            if (batch) r64 ? force_list_staged<true, true, 4>(P, a, st) : force_list_staged<true, true, 5>(P, a, st);
            else r64 ? force_list_staged<true, false, 4>(P, a, st) : force_list_staged<true, false, 5>(P, a, st);
        } else {
            if (batch) r64 ? force_list_staged<false, true, 4>(P, a, st) : force_list_staged<false, true, 5>(P, a, st);
            else r64 ? force_list_staged<false, false, 4>(P, a, st) : force_list_staged<false, false, 5>(P, a, st);
        }
        return;
    }
    if (min_blocks == 4) {
        force_list_variant<4, false>(P, a, st, block);
    } else {
        force_list_variant<5, false>(P, a, st, block);
    }
}

void launch_list_length(int n, const int* nbr_cnt, unsigned long long* out, cudaStream_t st) {
    k_list_length<<<blocks_for(n), kBlock, 0, st>>>(n, nbr_cnt, out);
}

}  // namespace wd
