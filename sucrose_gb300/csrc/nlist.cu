// Verlet half list on the device: the reference's build_nlist / needs_rebuild
// (fortran/system.f90:895-1051) re-designed as integer cell binning.
//
// Pair set contract: a pair (i < j) is listed iff the reference's FP64 test
// accepts it: RIJ = R(I) - R(J); RIJ -= ANINT(RIJ/box)*box when periodic;
// SUM(RIJ*RIJ) < (rc+skin)^2 (:980-989), evaluated on the FP32 state promoted
// to FP64. The FP32 filter decides only pairs clear of the threshold by a
// relative guard band of 1e-4; every other candidate is re-tested with the
// reference's exact FP64 operation sequence (no contraction).
//
// Layout in HBM: a single system's cooperative build writes every particle's
// full row into nb_pad, rows in cell order, row-major with row_cap entries
// each: the neighbours above (j > i) from the front, those below from the back.
// The half rows (the front parts) are copied into the flattened pair arrays
// pair_i / pair_j, rows in particle order, which the pair-parallel kernels walk
// 32 pairs per warp. Replica contexts write half rows column-major in each
// replica's section of nb_pad.
#include <algorithm>
#include <climits>
#include <cmath>
#include <vector>

#include <cooperative_groups.h>

#include "cell_axis.h"
#include "f32x2.cuh"
#include "sg_internal.cuh"
#include "step_epi.cuh"

namespace cg = cooperative_groups;

namespace {

// Up to this many particles the full rows list particles, and the row driver
// reads their positions where they are (half a megabyte, most of it in L1 before
// long); with more it copies them into cell order first, a launch of 1.2 us and
// up. What the copy gains grows with the rows' length, for particles in random order
// (any fluid after a while); on rows of a hundred or so, and for particles in
// spatial order, it costs 1 to 7 % at every size. Pair stage of a captured step, us,
// with / without the copy, random order: LJ at cut-off 4 (270 a row) 16 384
// particles 24.1 / 23.2, 27 436 32.3 / 32.3, 131 072 123 / 125, a million 883 / 937;
// at 6 (900 a row) 131 072 329 / 346, 500 000 1207 / 1351; dipoles 16 384 49.4 /
// 51.7, 37 044 78.6 / 86.8, 500 000 872 / 1024; LJ at 2.5 (77 a row) 2 916 9.7 /
// 8.9, 37 044 18.1 / 16.0, a million 250 / 249; charged spheres (115 a row) 131 072
// 73.9 / 70.9.
#define SG_ROWS_DIRECT 32768

constexpr int SCAN_BLOCK = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_BLOCK * SCAN_ITEMS;

// flags layout
// F_HALF: the build that the flat half list was last written for
enum { F_REBUILD = 0, F_OVERFLOW = 1, F_NPAIRS = 2, F_BUILDS = 3, F_HALF = 4 };

struct ListGeom {
    float3 box, inv_box;
    double bx, by, bz;
    double rl2;       // (rc+skin)^2
    float rl2_lo, rl2_hi;
    float half_sq;    // (0.4998 min(box))^2, rounded down: a pair with a half-box component is at least this far
    int periodic;
    int nc[3];
};

// Reference FP64 acceptance test, operation by operation (system.f90:980-989).
__device__ __forceinline__ bool ref_accept(float4 pi, float4 pj, const ListGeom& g) {
    double dx = __dsub_rn((double)pi.x, (double)pj.x);
    double dy = __dsub_rn((double)pi.y, (double)pj.y);
    double dz = __dsub_rn((double)pi.z, (double)pj.z);
    if (g.periodic) {
        dx = __dsub_rn(dx, __dmul_rn(round(__ddiv_rn(dx, g.bx)), g.bx));
        dy = __dsub_rn(dy, __dmul_rn(round(__ddiv_rn(dy, g.by)), g.by));
        dz = __dsub_rn(dz, __dmul_rn(round(__ddiv_rn(dz, g.bz)), g.bz));
    }
    double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    return r2 < g.rl2;
}

// FP32 filter, exact FP64 decision inside the guard band.
__device__ __forceinline__ bool accept_pair(float4 pi, float4 pj, const ListGeom& g) {
    float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
    bool halfcase = false;
    if (g.periodic) {
        // a component within 2e-4 of half a box may round the other way in
        // FP64: such pairs take the exact test (the distance to the nearest
        // integer of d / L is read off the rounding the image needs anyway)
        const float tx = dx * g.inv_box.x, ty = dy * g.inv_box.y, tz = dz * g.inv_box.z;
        const float nx = roundf(tx), ny = roundf(ty), nz = roundf(tz);
        halfcase = fabsf(tx - nx) > 0.4998f || fabsf(ty - ny) > 0.4998f || fabsf(tz - nz) > 0.4998f;
        dx -= nx * g.box.x;
        dy -= ny * g.box.y;
        dz -= nz * g.box.z;
    }
    float r2 = dx * dx + dy * dy + dz * dz;
    if (!halfcase) {
        if (r2 < g.rl2_lo) return true;
        if (r2 > g.rl2_hi) return false;
    } else {
        if (g.half_sq > g.rl2_hi) return false;   // beyond the list radius whichever image FP64 picks
        // the other image of such a component changes r^2 by 4e-4 of the side's
        // square at most (a list radius of more than half a side: small boxes,
        // where every eight-hundredth pair comes here)
        const float d = 1.3e-3f * fmaxf(g.box.x * g.box.x, fmaxf(g.box.y * g.box.y, g.box.z * g.box.z));
        if (r2 + d < g.rl2_lo) return true;
        if (r2 - d > g.rl2_hi) return false;
    }
    return ref_accept(pi, pj, g);
}

// Relative half-width of the r^2 band where the FP32 test defers to the FP64
// one. The FP32 r^2 of the same FP32 positions is within ~(1.1e-6 L / r_list
// + 3e-7) of the FP64 value (the FP32 box in the image shift dominates), so
// the band is 1e-4, widened for boxes over ~25 list radii.
inline double guard_band(double box_max, double rl2) { return std::max(1e-4, 4e-6 * box_max / std::sqrt(rl2)); }

// Geometry of replica r (batched contexts): its box, list radius and grid. All
// tabulated: the band's square root and quotient took every warp of the row search
// some ninety FP64 instructions (252 us of row search in a step without them 234).
__device__ __forceinline__ ListGeom geom_for(const ListGeom& base, const RepDev& rp, int r) {
    ListGeom g = base;
    const float4 b = rp.box[r], ib = rp.inv_box[r];
    g.box = make_float3(b.x, b.y, b.z);
    g.inv_box = make_float3(ib.x, ib.y, ib.z);
    g.bx = rp.boxd[3 * r];
    g.by = rp.boxd[3 * r + 1];
    g.bz = rp.boxd[3 * r + 2];
    g.rl2 = rp.rl2[r];
    const float2 band = rp.rl2_band[r];
    g.rl2_lo = band.x;
    g.rl2_hi = band.y;
    g.half_sq = rp.half_sq[r];
    const int4 gr = rp.grid[r];
    g.nc[0] = max(gr.x, 1);
    g.nc[1] = max(gr.y, 1);
    g.nc[2] = max(gr.z, 1);
    return g;
}

__device__ __forceinline__ int wrapc(int c, int n) {
    c %= n;
    return c < 0 ? c + n : c;
}

__device__ __forceinline__ int cell_of(float4 p, const ListGeom& g, int& cx, int& cy, int& cz) {
    cx = wrapc((int)floorf((p.x + 0.5f * g.box.x) * (g.nc[0] * g.inv_box.x)), g.nc[0]);
    cy = wrapc((int)floorf((p.y + 0.5f * g.box.y) * (g.nc[1] * g.inv_box.y)), g.nc[1]);
    cz = wrapc((int)floorf((p.z + 0.5f * g.box.z) * (g.nc[2] * g.inv_box.z)), g.nc[2]);
    return (cz * g.nc[1] + cy) * g.nc[0] + cx;
}

// ---------------------------------------------------------------- trigger --
// needs_rebuild (system.f90:1005-1039) in FP64 on the FP32 state: any
// particle with 4 |dr|^2 > trigger_sq requests a rebuild (the maximum over
// particles exceeds the bound iff some particle does). The test itself is
// check_displacement (step_epi.cuh), which the captured step also runs inside
// its initial half step.
__global__ void k_check(int n, const float4* __restrict__ pos, CheckArgs c) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    check_displacement(i, pos[i], c);
}

// Replica contexts: the rows of the replicas that rebuild, in items of up to 32
// rows of one replica, (replica, first row): a step asks for a few per cent of an
// ensemble's replicas, and a pass over all rows to find theirs costs more than
// the rows (29 000 blocks of 32 rows some 40 us, three times that at the row
// search's registers).
constexpr int REP_ROWS = 32;
struct RepItems {
    int2* item;
    int* count;
};

// Before a replica build: block 0 lists the items, the others clear the cells.
__global__ void __launch_bounds__(1024) k_begin(int* flags, int* cell_count, int* cell_fill, int ncells,
                                                const int* __restrict__ rep_off, const int* __restrict__ rep_flag,
                                                int R, RepItems items) {
    if (!flags[F_REBUILD]) return;
    if (blockIdx.x > 0) {
        for (int c = (blockIdx.x - 1) * blockDim.x + threadIdx.x; c < ncells; c += (gridDim.x - 1) * blockDim.x) {
            cell_count[c] = 0;
            cell_fill[c] = 0;
        }
        return;
    }
    __shared__ int sums[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int before = 0;
    for (int r0 = 0; r0 < R; r0 += 1024) {
        const int r = r0 + threadIdx.x;
        const int o = r < R ? rep_off[r] : 0, e = r < R && rep_flag[r] ? rep_off[r + 1] : o;
        const int k = (e - o + REP_ROWS - 1) / REP_ROWS;
        int end = k;
#pragma unroll
        for (int q = 1; q < 32; q <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, end, q);
            if (lane >= q) end += y;
        }
        if (lane == 31) sums[warp] = end;
        __syncthreads();
        int w = sums[lane], all = w;
#pragma unroll
        for (int q = 1; q < 32; q <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, all, q);
            if (lane >= q) all += y;
        }
        const int total = __shfl_sync(0xffffffffu, all, 31);
        int at = before + __shfl_sync(0xffffffffu, all - w, warp) + end - k;
        for (int i = o; i < e; i += REP_ROWS) items.item[at++] = make_int2(r, i);
        before += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        *items.count = before;
        flags[F_OVERFLOW] = 0;
    }
}

// This warp's row of its next item (a lane each): calls f(replica, row).
template <class F>
__device__ __forceinline__ void for_item_rows(const RepItems& items, const int* __restrict__ rep_off, F f) {
    const int lane = threadIdx.x & 31, nwarps = (gridDim.x * blockDim.x) >> 5, count = *items.count;
    for (int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < count; k += nwarps) {
        const int2 it = items.item[k];
        const int i = it.y + lane;
        if (i < min(it.y + REP_ROWS, rep_off[it.x + 1])) f(it.x, i);
    }
}

__global__ void k_bin(const float4* __restrict__ pos, ListGeom g0, int* particle_cell, int* cell_count,
                      const int* flags, RepDev rp, RepItems items) {
    if (!flags[F_REBUILD]) return;
    for_item_rows(items, rp.off, [&](int r, int i) {
        const int4 gr = rp.grid[r];
        // a replica under three cells per side is searched all-pairs, not binned
        int c = -1, cx, cy, cz;
        if (gr.x) {
            c = gr.w + cell_of(pos[i], geom_for(g0, rp, r), cx, cy, cz);
            atomicAdd(&cell_count[c], 1);
        }
        particle_cell[i] = c;
    });
}

// Cell members in arrival order (atomic slots) into the scratch array.
__global__ void k_fill(const int* __restrict__ particle_cell, const int* __restrict__ cell_start, int* cell_fill,
                       int* cell_unsorted, const int* flags, RepDev rp, RepItems items) {
    if (!flags[F_REBUILD]) return;
    for_item_rows(items, rp.off, [&](int, int i) {
        const int c = particle_cell[i];
        if (c >= 0) cell_unsorted[cell_start[c] + atomicAdd(&cell_fill[c], 1)] = i;
    });
}

// Order each cell's particles by index so that rows are deterministic: one
// warp per cell, each member placed at its rank (the number of smaller
// indices in the cell; indices are distinct).
__global__ void k_sort_cells(int ncells, const int* __restrict__ cell_start, const int* __restrict__ cell_unsorted,
                             int* cell_particles, const int* flags) {
    if (!flags[F_REBUILD]) return;
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (c >= ncells) return;
    const int b = cell_start[c], e = cell_start[c + 1];
    for (int k = b + lane; k < e; k += 32) {
        const int v = cell_unsorted[k];
        int rank = 0;
        for (int t = b; t < e; ++t) rank += cell_unsorted[t] < v;
        cell_particles[b + rank] = v;
    }
}

// Padded-row addressing: slot k of particle i's row is nb_pad[base + k * stride].
struct PadRep {
    const int* max_nb;          // [R] row capacity of each replica
    const long long* pad_off;   // [R] first slot of each replica's section
    int* need;                  // [R] longest row seen on overflow
};

__device__ __forceinline__ void row_done(int i, int cnt, int cap, int* nb_count, int* flags, const RepDev& rp,
                                         const PadRep& pr) {
    nb_count[i] = min(cnt, cap);
    if (cnt > cap) {
        atomicMax(&flags[F_OVERFLOW], cnt);
        if (rp.rep_of) atomicMax(&pr.need[rp.rep_of[i]], cnt);
    }
}

// A replica's acceptance test on the original positions, for the few pairs that
// the row search cannot decide in FP32. Not inlined: FP64 quotients and roundings
// at every place of use took the registers of half the resident warps.
__device__ __noinline__ bool rep_exact(const float4* __restrict__ pos, int i, int j, const ListGeom& g0,
                                       const RepDev& rp, int r) {
    const ListGeom g = geom_for(g0, rp, r);
    return accept_pair(pos[i], pos[j], g);
}

// Half rows of the replicas that rebuild: a block takes an item of 32 rows, a
// warp four of them, 32 candidates at a time, one a lane and row, two rows in
// packed FP32, appended in candidate order by their ballot. In a replica under
// three cells a side the candidates are the later particles, and each load of
// them serves the four rows; in a binned one they are the members of the
// stencil's cells that come after the row's particle, end to end.
// Bound: latency (the candidates' loads) where few replicas rebuild, issue where
// all do. Measured, us, a thread to a row / now: 1, 16 and 437 Gay-Berne replicas
// (about 1 100 particles, box under three cells) 241, 400, 2324 / 25, 51, 758; 39
// of a list radius over half the box, where components near half a side all took
// the FP64 test, 707 / 47; 36 binned ones 603 / 216; 1 and 512 Lennard-Jones ones
// 161, 551 / 23, 555; the tenth of 1 024 replicas that one step rebuilds 750 / 230.
// 128 registers, two blocks an SM: three and four spill (265 and 305 us there).
// A pair is within the radius for sure, or beyond it, but for the guard band and
// for a component near half a side (accept_pair); where the list radius is less
// than half of every side, the latter is beyond the radius with either image.
__global__ void __launch_bounds__(256, 2)
    k_rep_rows(const float4* __restrict__ pos, ListGeom g0, const int* __restrict__ cell_start,
               const int* __restrict__ cell_particles, int* nb_pad, int* nb_count, int* flags, RepDev rp, PadRep pr,
               RepItems items) {
    if (!flags[F_REBUILD]) return;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const int count = *items.count;
    for (int item = blockIdx.x; item < count; item += gridDim.x) {
        const int2 it = items.item[item];
        const int r = it.x, o = rp.off[r], e = rp.off[r + 1];
        const int first = it.y + 4 * warp, rows = min(4, e - first);
        if (rows <= 0) continue;
        const float3 box = f3(rp.box[r]), inv_box = f3(rp.inv_box[r]);
        const float2 band = rp.rl2_band[r];
        const bool wide = !(rp.half_sq[r] > band.y);   // components near half a side matter
        const int4 gr = rp.grid[r];
        const int stride = e - o;
        int* const out = nb_pad + (size_t)pr.pad_off[r] + (first - o);
        const int cap = pr.max_nb[r];
        f2 px[2], py[2], pz[2];
        int cnt[4] = {0, 0, 0, 0};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float4 a = pos[first + min(2 * h, rows - 1)], b = pos[first + min(2 * h + 1, rows - 1)];
            px[h] = f2_of(a.x, b.x);
            py[h] = f2_of(a.y, b.y);
            pz[h] = f2_of(a.z, b.z);
        }
        // rows 2 h and 2 h + 1 against their candidates j0, j1 (-1: none) at x, y, z
        auto pair_rows = [&](int h, f2 x, f2 y, f2 z, int j0, int j1) {
            const f2 big = all_w<f2>(12582912.f);   // 1.5 * 2^23: the sum's rounding is to an integer
            float near0 = 0.f, near1 = 0.f;         // how far d / side is from an integer, at most
            auto image = [&](f2 d, float side, float inv_side) {
                const f2 t = d * all_w<f2>(inv_side), n = (t + big) - big;
                if (wide) {
                    float a, b;
                    f2_split(t - n, a, b);
                    near0 = fmaxf(near0, fabsf(a));
                    near1 = fmaxf(near1, fabsf(b));
                }
                return fma_w(n, all_w<f2>(-side), d);
            };
            const f2 dx = image(px[h] - x, box.x, inv_box.x), dy = image(py[h] - y, box.y, inv_box.y),
                     dz = image(pz[h] - z, box.z, inv_box.z);
            float r0, r1;
            f2_split(fma_w(dz, dz, fma_w(dy, dy, dx * dx)), r0, r1);
            // !(>): a non-finite distance goes on to the exact test
            bool in0 = j0 >= 0 && (!(r0 > band.y) || near0 > 0.4998f), in1 = j1 >= 0 && (!(r1 > band.y) || near1 > 0.4998f);
            if (in0 && !(r0 < band.x && !(near0 > 0.4998f))) in0 = rep_exact(pos, first + 2 * h, j0, g0, rp, r);
            if (in1 && !(r1 < band.x && !(near1 > 0.4998f))) in1 = rep_exact(pos, first + 2 * h + 1, j1, g0, rp, r);
            const unsigned m0 = __ballot_sync(full, in0), m1 = __ballot_sync(full, in1);
            const int at0 = cnt[2 * h] + __popc(m0 & below), at1 = cnt[2 * h + 1] + __popc(m1 & below);
            if (in0 && at0 < cap) out[(size_t)at0 * stride + 2 * h] = j0;
            if (in1 && at1 < cap) out[(size_t)at1 * stride + 2 * h + 1] = j1;
            cnt[2 * h] += __popc(m0);
            cnt[2 * h + 1] += __popc(m1);
        };
        if (!gr.x) {
            float4 c = pos[min(first + 1 + lane, e - 1)];
            for (int j = first + 1 + lane; j - lane < e; j += 32) {
                const float4 q = c;
                c = pos[min(j + 32, e - 1)];   // the next ones are in flight meanwhile
                const f2 x = all_w<f2>(q.x), y = all_w<f2>(q.y), z = all_w<f2>(q.z);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    pair_rows(h, x, y, z, j < e && j > first + 2 * h && 2 * h < rows ? j : -1,
                              j < e && j > first + 2 * h + 1 && 2 * h + 1 < rows ? j : -1);
            }
        } else {
            // the stencil's cells, a lane each, from the first member (members
            // ascend) that comes after the row's particle: the non-empty ones, end
            // to end, make the row's stream. The four rows' streams advance together.
            int from[4], start[4], most = 0, total[4];   // this lane's cell: its place - its start in the stream
            const ListGeom g = geom_for(g0, rp, r);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                int cx, cy, cz, lo = 0, stop = 0;
                const float4 p = pos[first + min(k, rows - 1)];
                cell_of(p, g, cx, cy, cz);
                if (lane < 27 && k < rows) {
                    const int zz = wrapc(cz + lane / 9 - 1, g.nc[2]), yy = wrapc(cy + lane / 3 % 3 - 1, g.nc[1]);
                    const int c = gr.w + (zz * g.nc[1] + yy) * g.nc[0] + wrapc(cx + lane % 3 - 1, g.nc[0]);
                    lo = cell_start[c];
                    stop = cell_start[c + 1];
                }
                from[k] = lo;
                start[k] = stop;
            }
            // lower bounds, the four rows' steps together
            {
                int hi[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) hi[k] = start[k];
                while (__any_sync(full, from[0] < hi[0] || from[1] < hi[1] || from[2] < hi[2] || from[3] < hi[3])) {
                    int mid[4], v[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        mid[k] = (from[k] + hi[k]) >> 1;
                        v[k] = from[k] < hi[k] ? cell_particles[mid[k]] : 0;
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (from[k] < hi[k]) {
                            if (v[k] > first + k) hi[k] = mid[k];
                            else from[k] = mid[k] + 1;
                        }
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int len = start[k] - from[k];
                int end = len;
#pragma unroll
                for (int q = 1; q < 32; q <<= 1) {
                    const int y = __shfl_up_sync(full, end, q);
                    if (lane >= q) end += y;
                }
                total[k] = __shfl_sync(full, end, 31);
                most = max(most, total[k]);
                // the non-empty cells to the first lanes
                const unsigned some = __ballot_sync(full, len > 0);
                const int src = __fns(some, 0, lane + 1);   // (all ones beyond the last)
                const int place = __shfl_sync(full, from[k] - (end - len), src & 31);
                const int at = __shfl_sync(full, end - len, src & 31);
                from[k] = place;
                start[k] = lane < __popc(some) ? at : INT_MAX;
            }
            // candidate v0 + lane: the cell whose start is the last one not beyond it
            auto candidate = [&](int k, int v0) {
                const unsigned before = __ballot_sync(full, start[k] <= v0);
                const unsigned in = start[k] > v0 && start[k] < v0 + 32 ? 1u << (start[k] - v0) : 0u;
                const unsigned starts = __reduce_or_sync(full, in);
                const int cell = __popc(before) - 1 + __popc(starts & (below | 1u << lane));
                const int at = __shfl_sync(full, from[k], cell & 31) + v0 + lane;
                return v0 + lane < total[k] ? cell_particles[at] : -1;
            };
            int j[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) j[k] = candidate(k, 0);
            for (int v0 = 0; v0 < most; v0 += 32) {
                float4 c[4];
                int jj[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    jj[k] = j[k];
                    c[k] = pos[max(j[k], 0)];
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) j[k] = candidate(k, v0 + 32);   // the next ones
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    pair_rows(h, f2_of(c[2 * h].x, c[2 * h + 1].x), f2_of(c[2 * h].y, c[2 * h + 1].y),
                              f2_of(c[2 * h].z, c[2 * h + 1].z), jj[2 * h], jj[2 * h + 1]);
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < rows && lane == k) row_done(first + k, cnt[k], cap, nb_count, flags, rp, pr);
    }
}

// ---- exclusive scan of m ints into out[0..m], out[m] = total -----------------
__global__ void k_scan_tiles(const int* __restrict__ in, int m, int* out, int* tile_sums, const int* flags) {
    if (flags && !flags[F_REBUILD]) return;
    __shared__ int warp_sums[SCAN_BLOCK / 32];
    int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    int v[SCAN_ITEMS];
    int s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        v[k] = (base + k < m) ? in[base + k] : 0;
        s += v[k];
    }
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[w] = x;
    __syncthreads();
    if (w == 0) {
        int ws = warp_sums[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, ws, o);
            if (lane >= o) ws += y;
        }
        warp_sums[lane] = ws;
    }
    __syncthreads();
    int excl = x - s + (w > 0 ? warp_sums[w - 1] : 0);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        if (base + k < m) out[base + k] = excl;
        excl += v[k];
    }
    if (threadIdx.x == SCAN_BLOCK - 1) tile_sums[blockIdx.x] = warp_sums[31];
}

// Single block: exclusive scan of the tile sums in place, total at [ntiles].
__global__ void k_scan_sums(int* tile_sums, int ntiles, const int* flags) {
    if (flags && !flags[F_REBUILD]) return;
    __shared__ int sh[SCAN_BLOCK + 1];
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < ntiles; base += SCAN_BLOCK) {
        int t = base + threadIdx.x;
        int v = t < ntiles ? tile_sums[t] : 0;
        sh[threadIdx.x] = v;
        __syncthreads();
        for (int o = 1; o < SCAN_BLOCK; o <<= 1) {
            int y = threadIdx.x >= o ? sh[threadIdx.x - o] : 0;
            __syncthreads();
            sh[threadIdx.x] += y;
            __syncthreads();
        }
        if (t < ntiles) tile_sums[t] = carry + sh[threadIdx.x] - v;
        __syncthreads();
        if (threadIdx.x == 0) carry += sh[SCAN_BLOCK - 1];
        __syncthreads();
    }
    if (threadIdx.x == 0) tile_sums[ntiles] = carry;
}

__global__ void k_scan_add(int* out, int m, const int* __restrict__ tile_sums, int ntiles, int* total_dst,
                           const int* flags) {
    if (flags && !flags[F_REBUILD]) return;
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < m) out[t] += tile_sums[t / SCAN_TILE];
    if (t == 0) {
        out[m] = tile_sums[ntiles];
        if (total_dst) *total_dst = tile_sums[ntiles];
    }
}

// Replica of the first pair of every 32-pair chunk of the row order: the
// largest r with row_off[off[r]] <= 32 c (pair kernels start their search there).
// With s_r = row_off[off[r]] the first pair of replica r, the chunks c with
// s_r <= 32 c < s_(r+1) are replica r's: c in [ceil(s_r / 32), ceil(s_(r+1) / 32)).
// A warp per replica writes its range (a replica without pairs has none, and
// its chunk goes to the next replica with pairs, the largest r as required).
__global__ void k_chunk_rep(const int* __restrict__ row_off, const int* __restrict__ rep_off, int R,
                            const int* flags, int* chunk_rep) {
    if (!flags[F_REBUILD]) return;
    const int lane = threadIdx.x & 31;
    const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
    for (int r = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); r < R; r += nwarps) {
        const int c0 = (row_off[rep_off[r]] + 31) >> 5;
        const int c1 = (row_off[rep_off[r + 1]] + 31) >> 5;   // rep_off[R] = n: the total
        for (int c = c0 + lane; c < c1; c += 32) chunk_rep[c] = r;
    }
}

// Rows into the flat pair arrays. A single system stores them in row order
// (pair index = row_off[i] + k). A replica context stores each replica's rows
// in the replica's own section (it starts where the replica's padded rows
// start), so only replicas that rebuilt are rewritten: the pair at row-order
// index v of replica r sits at pad_off[r] + v - row_off[off[r]].
// Four warps take an item of 32 rows, each of them every fourth group of 32
// columns, through shared memory: slot k of the 32 rows is one coalesced
// read of the column-major padded rows, and each row's 32 entries one coalesced
// write of the flat arrays. Its first warp notes the rows' positions as those
// of the list. (A warp to 32 rows: 439 us for 437 Gay-Berne replicas, 45 for 16 of
// them, 60 for 512 Lennard-Jones ones; now 330, 15 and 61.)
__global__ void __launch_bounds__(256) k_compact(const float4* __restrict__ pos, float4* __restrict__ last,
                                                 const int* __restrict__ nb_pad, const int* __restrict__ nb_count,
                                                 const int* __restrict__ row_off, int* pair_i, int* pair_j,
                                                 const int* flags, RepDev rp, PadRep pr, RepItems items) {
    if (!flags[F_REBUILD]) return;
    __shared__ int tile[8][32][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int count = *items.count;
    for (int item = 2 * blockIdx.x + (w >> 2); item < count; item += 2 * gridDim.x) {
        const int2 it = items.item[item];
        const int r = it.x, first = rp.off[r], i0 = it.y, i = i0 + lane;   // this lane's row, in every warp
        const size_t base = (size_t)pr.pad_off[r] + (size_t)(i - first), stride = (size_t)(rp.off[r + 1] - first);
        size_t o = 0;
        int c = 0;
        if (i < rp.off[r + 1]) {
            o = (size_t)pr.pad_off[r] + (size_t)(row_off[i] - row_off[first]);
            c = nb_count[i];
            if ((w & 3) == 0) last[i] = pos[i];
        }
        const int cmax = __reduce_max_sync(0xffffffffu, c);
        int (*t)[33] = tile[w];
        for (int k0 = 32 * (w & 3); k0 < cmax; k0 += 32 * 4) {
            // read: lane = row, slots k0 .. k0 + 31, eight loads in flight
            for (int kk = 0; kk < 32; kk += 8) {
                int v[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = k0 + kk + q < c ? nb_pad[base + (size_t)(k0 + kk + q) * stride] : 0;
#pragma unroll
                for (int q = 0; q < 8; ++q) t[kk + q][lane] = v[q];
            }
            __syncwarp();
            // write: row by row, lane = slot
            for (int rr = 0; rr < 32; ++rr) {
                const int cr = __shfl_sync(0xffffffffu, c, rr);
                const unsigned long long orr = __shfl_sync(0xffffffffu, (unsigned long long)o, rr);
                const int k = k0 + lane;
                if (k < cr) {
                    pair_i[orr + k] = i0 + rr;
                    pair_j[orr + k] = t[lane][rr];
                }
            }
            __syncwarp();
        }
    }
}

// Request flags: the global one and, in a replica context, one per replica.
// After a build (rep_builds given) it and each replica that rebuilt are counted.
__global__ void k_clear_request(int* flags, int* rep_flag, int R, int* rep_builds) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (rep_builds && flags[F_REBUILD]) flags[F_BUILDS] += 1;
        flags[F_REBUILD] = 0;
    }
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < R; r += gridDim.x * blockDim.x) {
        if (rep_builds && rep_flag[r]) rep_builds[r] += 1;
        rep_flag[r] = 0;
    }
}
__global__ void k_set_request(int* flags, int* rep_flag, int R) {
    if (blockIdx.x == 0 && threadIdx.x == 0) flags[F_REBUILD] = 1;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < R; r += gridDim.x * blockDim.x) rep_flag[r] = 1;
}

// ------------------------------------------------ single-system rebuild --
// The whole rebuild of a single system in one cooperative kernel: its phases
// (bin, scan of the cell counts, fill, sort, row search, scan of the row
// lengths, compaction, finish) are separated by grid-wide barriers instead of
// kernel boundaries. A step without a rebuild then runs one launch that exits
// at its first instruction, where the captured step would otherwise evaluate a
// graph conditional node or a dozen flag-gated kernels. Arrays written in one
// phase and read in a later one are read with plain (coherent) loads, never
// through the read-only path. Without cells (a box under three cells per side,
// open boundaries) the first four phases are one copy.
struct CoopBuild {
    int n, ncells, ncells_cap, max_nb, row_cap, row_lanes;   // ncells == 0: no cells
    int want_half;                                           // write the flat half list too
    int by_particle;                                         // entries are particles, not places
    const float4* pos;
    ListGeom g;
    int* cell_count;
    int* cell_fill;
    int* cell_start;
    int* cell_unsorted;
    int* cell_particles;
    int* particle_cell;
    float4* pos_cell;
    unsigned* nb_pad;
    int2* nb_count;
    int* nb_half;
    int* row_off;
    int* pair_i;
    int* pair_j;
    float4* last;
    int* flags;
    int* tmp;   // gridDim.x block totals of the scans
};

// Cell of a position and the position's image in the box (cell_axis.h).
__device__ __forceinline__ int cell_and_image(float4& p, const ListGeom& g) {
    const int cx = cell_axis(p.x, g.nc[0], g.box.x, g.inv_box.x, g.bx);
    const int cy = cell_axis(p.y, g.nc[1], g.box.y, g.inv_box.y, g.by);
    const int cz = cell_axis(p.z, g.nc[2], g.box.z, g.inv_box.z, g.bz);
    return (cz * g.nc[1] + cy) * g.nc[0] + cx;
}

__device__ __forceinline__ float warp_min(unsigned m, float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(m, v, o));
    return v;
}

// Row t's lengths: neighbours stored above and below; found counts those past
// the row's capacity too.
__device__ __forceinline__ void row_counts(const CoopBuild& a, int t, int i, int up, int down, int found) {
    a.nb_count[t] = make_int2(up, down);
    a.nb_half[i] = min(up, a.max_nb);
    if (up > a.max_nb) atomicMax(&a.flags[F_OVERFLOW], up);
    // a full row past its capacity asks for rows a third longer at least
    if (found > a.row_cap) atomicMax(&a.flags[F_OVERFLOW], max(found - found / 3, a.max_nb + 1));
}

// The row search of a warp: 32 / S consecutive rows in cell order, S lanes to
// a row. Candidates stream past the warp: each lane loads one, tests it
// against the bounding box of the warp's rows, and those within the list
// radius of the box queue in shared memory; 32 queued candidates are then
// tested against every row, S of them by each row's lanes at a time, read from
// shared memory as broadcasts. A test is a difference, a squared distance and
// one comparison (ten instructions; the image is a shift per run of
// candidates), against some forty, and a load of its own, where each lane
// walked its own candidates. A pair whose FP32 distance is within the guard
// band takes the reference's FP64 test on the original positions, so the pair
// set is the same. With three or more cells a side the list radius is at most
// a third of the box: at most one image of a candidate is in range, however
// often a run repeats a cell.
// Bound: issue and latency of the streaming and of the append loops (a row's
// accepted candidates, about one in eight of those tested). Measured, a whole
// rebuild, us, a warp or a thread per row over its own 27 cells, half rows only /
// this search, full rows, with each candidate's run found by bisection / and by
// following the runs: a million LJ particles 3515 / 860 / 860, 131 072 charged
// spheres 574 / 160 / 158, 32 768 Gay-Berne 370 / 236 / 224, 4 999 of them 180 /
// 132 / 115, 65 536 ECP 111 / 58.8 / 60.1 (cells of three particles: a run of
// candidates is shorter than a warp), 20 000 at radius 3.8 175 / 100 / 94.
struct RowQueue {
    float4 p[64];   // image, particle index
    int s[64];      // the entry to store: place in cell order, or particle
};

template <int S, bool CELLS>
__device__ __forceinline__ void search_rows(const CoopBuild& a, RowQueue& q, int gw, int nwarps) {
    constexpr int R = 32 / S;   // rows of a warp, and candidates of a lane per 32
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, sub = lane % S;
    const ListGeom& g = a.g;
    const float hi = g.rl2_hi, lo = g.rl2_lo;
    const float3 iL = CELLS || !g.periodic ? make_float3(0.f, 0.f, 0.f) : g.inv_box;
    const int nx = g.nc[0], ny = g.nc[1], nz = g.nc[2];
    for (int chunk = gw; chunk * R < a.n; chunk += nwarps) {
        const int t = chunk * R + lane / S;
        const bool valid = t < a.n;
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
        int i = -1, cx = 0, line = -1;
        if (valid) {
            p = a.pos_cell[t];
            i = __float_as_int(p.w);
            if (CELLS) {
                const int c = a.particle_cell[i];
                line = c / nx;
                cx = c - line * nx;
            }
        }
        unsigned* row = a.nb_pad + (size_t)(valid ? t : 0) * a.row_cap;
        int up = 0, down = 0, found = 0;
        // the rows of one line of cells at a time (nearly always one or two lines)
        unsigned todo = __ballot_sync(full, valid);
        while (todo) {
            const int lead = __ffs(todo) - 1;
            const int ln = __shfl_sync(full, line, lead);
            const bool mine = valid && line == ln;
            todo &= ~__ballot_sync(full, mine);
            const int x0 = __reduce_min_sync(full, mine ? cx : nx) - 1, x1 = __reduce_max_sync(full, mine ? cx : -1) + 1;
            const float big = 3e18f;
            float3 b0, b1;
            b0.x = warp_min(full, mine ? p.x : big);
            b0.y = warp_min(full, mine ? p.y : big);
            b0.z = warp_min(full, mine ? p.z : big);
            b1.x = -warp_min(full, mine ? -p.x : big);
            b1.y = -warp_min(full, mine ? -p.y : big);
            b1.z = -warp_min(full, mine ? -p.z : big);
            int qn = 0;
            // the first 32 queued candidates (n < 32: the last ones) against the rows
            auto drain = [&](int n) {
                unsigned m = 0u, sure = 0u;   // within the radius but for the guard band, and surely
#pragma unroll
                for (int b = 0; b < R; ++b) {
                    const float4 c = q.p[b * S + sub];
                    float dx = p.x - c.x, dy = p.y - c.y, dz = p.z - c.z;
                    if (!CELLS) {   // nearest image; without periodic boundaries iL is zero
                        dx -= rintf(dx * iL.x) * g.box.x;
                        dy -= rintf(dy * iL.y) * g.box.y;
                        dz -= rintf(dz * iL.z) * g.box.z;
                    }
                    const float r2 = dx * dx + dy * dy + dz * dz;
                    // !(>): a non-finite distance takes the exact test, as the reference decides it
                    if (!(r2 > hi)) m |= 1u << b;
                    if (r2 < lo) sure |= 1u << b;
                }
                const int nb = (n - sub + S - 1) / S;   // this lane's candidates
                m = !mine || nb <= 0 ? 0u : m & (0xffffffffu >> (32 - nb));
                for (unsigned w = m & ~sure; w; w &= w - 1) {
                    const int b = __ffs(w) - 1, j = __float_as_int(q.p[b * S + sub].w);
                    if (j == i || !ref_accept(a.pos[min(i, j)], a.pos[max(i, j)], g)) m &= ~(1u << b);
                }
                if constexpr (S == 1) {
                    for (; m; m &= m - 1) {
                        const int k = __ffs(m) - 1, j = __float_as_int(q.p[k].w);
                        if (j == i) continue;
                        if (up + down < a.row_cap) row[j > i ? up++ : a.row_cap - ++down] = (unsigned)q.s[k];
                        ++found;
                    }
                } else {
                    unsigned above = 0u, below = 0u;   // the queue places this lane keeps
                    for (; m; m &= m - 1) {
                        const int k = (__ffs(m) - 1) * S + sub, j = __float_as_int(q.p[k].w);
                        if (j > i) above |= 1u << k;
                        if (j < i) below |= 1u << k;
                    }
                    // the row's lanes append in queue order
                    unsigned keep = above | below, aa = above, bb = below;
#pragma unroll
                    for (int o = 1; o < S; o <<= 1) {
                        aa |= __shfl_xor_sync(full, aa, o);
                        bb |= __shfl_xor_sync(full, bb, o);
                    }
                    const int na = __popc(aa), nd = __popc(bb);
                    found += na + nd;
                    if (up + down + na + nd <= a.row_cap) {
                        for (; keep; keep &= keep - 1) {
                            const int k = __ffs(keep) - 1;
                            const unsigned before = (1u << k) - 1u;
                            row[above >> k & 1u ? up + __popc(aa & before)
                                                : a.row_cap - 1 - down - __popc(bb & before)] = (unsigned)q.s[k];
                        }
                        up += na;
                        down += nd;
                    }
                }
                __syncwarp();
                // move the rest down
                float4 rp;
                int rs = 0;
                const bool rest = n == 32 && lane < qn - 32;
                if (rest) {
                    rp = q.p[32 + lane];
                    rs = q.s[32 + lane];
                }
                __syncwarp();
                if (rest) {
                    q.p[lane] = rp;
                    q.s[lane] = rs;
                }
                qn -= n;
                __syncwarp();
            };
            // the stencil as up to 27 runs of consecutive cells, a lane each: a
            // line of cells of the nine, before, inside or past the ends of the
            // box in x, cut to what the box of the rows can reach
            int len = 0, first = 0, image = 0;   // image: 1 + shift in boxes, two bits an axis
            if (!CELLS) {
                len = lane == 0 ? a.n : 0;
                image = 21;
            } else if (lane < 27) {
                const int cz = ln / ny, cy = ln - cz * ny;
                int zz = cz + lane / 9 - 1, yy = cy + lane / 3 % 3 - 1;
                const float fz = 1e-6f * g.box.z, fy = 1e-6f * g.box.y, fx = 1e-6f * g.box.x;   // rounding of the binning
                const float wz = g.box.z / nz, wy = g.box.y / ny, wx = nx * g.inv_box.x;
                const float zl = zz * wz - 0.5f * g.box.z - fz, yl = yy * wy - 0.5f * g.box.y - fy;
                const float ez = fmaxf(fmaxf(zl - b1.z, b0.z - (zl + wz + 2.f * fz)), 0.f);
                const float ey = fmaxf(fmaxf(yl - b1.y, b0.y - (yl + wy + 2.f * fy)), 0.f);
                const float rem = hi * 1.00001f - ey * ey - ez * ez;
                if (rem >= 0.f) {
                    const float rr = sqrtf(rem) * 1.00001f + fx;
                    const int xa = max(x0, (int)floorf((b0.x - rr + 0.5f * g.box.x) * wx));
                    const int xb = min(x1, (int)floorf((b1.x + rr + 0.5f * g.box.x) * wx));
                    int iz = 1, iy = 1;
                    if (zz < 0) { zz += nz; iz = 0; }
                    else if (zz >= nz) { zz -= nz; iz = 2; }
                    if (yy < 0) { yy += ny; iy = 0; }
                    else if (yy >= ny) { yy -= ny; iy = 2; }
                    const int part = lane % 3;
                    const int lo_c = part == 0 ? (xa < 0 ? nx - 1 : nx) : part == 1 ? max(xa, 0) : 0;
                    const int hi_c = part == 0 ? nx - 1 : part == 1 ? min(xb, nx - 1) : (xb >= nx ? 0 : -1);
                    if (lo_c <= hi_c) {
                        const int base = (zz * ny + yy) * nx;
                        first = a.cell_start[base + lo_c];
                        len = a.cell_start[base + hi_c + 1] - first;
                        image = part | iy << 2 | iz << 4;
                    }
                }
            }
            int end = len;   // runs end to end: candidates [end - len, end) of the stream
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(full, end, o);
                if (lane >= o) end += y;
            }
            const int total = __shfl_sync(full, end, 31);
            // the runs that have any, to the first lanes (through the queue, empty now)
            {
                const unsigned some = __ballot_sync(full, len > 0);
                if (len > 0) {
                    const int at = __popc(some & ((1u << lane) - 1u));
                    q.s[at] = end;
                    q.s[32 + at] = first - (end - len);
                    q.p[at].x = __int_as_float(image);
                }
                __syncwarp();
                const bool on = lane < __popc(some);
                end = on ? q.s[lane] : INT_MAX;
                first = on ? q.s[32 + lane] : 0;
                image = on ? __float_as_int(q.p[lane].x) : 0;
                __syncwarp();
            }
            // this lane's run of the stream, which it leaves when v passes the end
            int run = 0, run_end = __shfl_sync(full, end, 0), run_first = __shfl_sync(full, first, 0),
                run_image = __shfl_sync(full, image, 0);
            auto locate = [&](int v, int& k, int& im) {
                while (__any_sync(full, v >= run_end)) {   // (ends with the last run's INT_MAX neighbour)
                    if (v >= run_end) ++run;
                    run_end = __shfl_sync(full, end, run);
                    run_first = __shfl_sync(full, first, run);
                    run_image = __shfl_sync(full, image, run);
                }
                k = run_first + v;
                im = run_image;
            };
            int k, im;
            float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
            locate(lane, k, im);
            if (lane < total) c = a.pos_cell[k];
            for (int v0 = 0; v0 < total; v0 += 32) {
                const int ks = k;
                float4 cs = c;
                const int is = im;
                if (v0 + 32 < total) {   // the next ones in flight while these are tested
                    locate(v0 + 32 + lane, k, im);
                    if (v0 + 32 + lane < total) c = a.pos_cell[k];
                }
                bool in = v0 + lane < total;
                if (CELLS) {
                    cs.x += (float)((is & 3) - 1) * g.box.x;
                    cs.y += (float)((is >> 2 & 3) - 1) * g.box.y;
                    cs.z += (float)((is >> 4) - 1) * g.box.z;
                    const float ex = fmaxf(fmaxf(b0.x - cs.x, cs.x - b1.x), 0.f);
                    const float ey = fmaxf(fmaxf(b0.y - cs.y, cs.y - b1.y), 0.f);
                    const float ez = fmaxf(fmaxf(b0.z - cs.z, cs.z - b1.z), 0.f);
                    in = in && !(ex * ex + ey * ey + ez * ez > hi * 1.00001f);
                }
                const unsigned inm = __ballot_sync(full, in);
                if (in) {
                    const int slot = qn + __popc(inm & ((1u << lane) - 1u));
                    q.p[slot] = cs;
                    q.s[slot] = a.by_particle ? __float_as_int(cs.w) : ks;
                }
                qn += __popc(inm);
                __syncwarp();
                if (qn >= 32) drain(32);
            }
            if (qn > 0) drain(qn);
        }
        if (valid && sub == 0) row_counts(a, t, i, up, down, found);
    }
}

// Exclusive scan of in[0, m) into out[0, m] (out[m] = total, also *total_dst)
// by the whole grid: each block scans a contiguous tile, the tiles' totals
// give each block its offset after a grid barrier.
__device__ __forceinline__ void coop_scan(cg::grid_group& grid, const int* in, int m, int* out, int* total_dst, int* tmp) {
    __shared__ int sh[32];
    __shared__ int sh_off;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int T = (m + (int)gridDim.x - 1) / (int)gridDim.x;
    const int lo = min(m, (int)blockIdx.x * T), hi = min(m, lo + T);
    const int per = (T + (int)blockDim.x - 1) / (int)blockDim.x;
    const int tlo = min(hi, lo + (int)threadIdx.x * per), thi = min(hi, tlo + per);
    int s = 0;
    for (int k = tlo; k < thi; ++k) s += in[k];
    int x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    if (w == 0) {
        int v = lane < nw ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
        }
        if (lane < nw) sh[lane] = v;
    }
    __syncthreads();
    const int excl = x - s + (w ? sh[w - 1] : 0);
    const int btot = sh[nw - 1];
    if (threadIdx.x == 0) tmp[blockIdx.x] = btot;
    grid.sync();
    int o = 0;
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += blockDim.x) o += __ldcg(tmp + b);   // L2: rewritten per scan
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) o += __shfl_xor_sync(0xffffffffu, o, d);
    __syncthreads();
    if (lane == 0) sh[w] = o;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int k = 0; k < nw; ++k) t += sh[k];
        sh_off = t;
    }
    __syncthreads();
    int run = sh_off + excl;
    for (int k = tlo; k < thi; ++k) {
        const int v = in[k];
        out[k] = run;
        run += v;
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        const int tot = sh_off + btot;
        out[m] = tot;
        if (total_dst) *total_dst = tot;
    }
    __syncthreads();   // sh is reused by the next scan
}

// The same rows by a thread each, for cells of few particles: 32 rows of a
// warp then span so many cells that most candidates of their box are far from
// any one row, while a row's own 27 cells hold only a few. The stencil's x
// cells are read as runs (three consecutive cells, or two runs at the ends).
// 96 000 beads at 0.6 a cell: the rebuild takes 47 us this way, 189 with
// search_rows (which takes 62 against 72 us on ECP rows, 4.2 a cell).
__device__ __forceinline__ void thread_row(const CoopBuild& a, int t) {
    const ListGeom& g = a.g;
    const int nx = g.nc[0], ny = g.nc[1], nz = g.nc[2];
    const float4 p = a.pos_cell[t];
    const int i = __float_as_int(p.w);
    const int c = a.particle_cell[i];
    const int line = c / nx, cx = c - line * nx, cz = line / ny, cy = line - cz * ny;
    unsigned* row = a.nb_pad + (size_t)t * a.row_cap;
    int up = 0, down = 0, found = 0;
    for (int d = 0; d < 9; ++d) {
        int zz = cz + d / 3 - 1, yy = cy + d % 3 - 1;
        float sz = 0.f, sy = 0.f;
        if (zz < 0) { zz += nz; sz = -g.box.z; }
        else if (zz >= nz) { zz -= nz; sz = g.box.z; }
        if (yy < 0) { yy += ny; sy = -g.box.y; }
        else if (yy >= ny) { yy -= ny; sy = g.box.y; }
        const int base = (zz * ny + yy) * nx;
        // up to two runs: cells cx-1 .. cx+1, split where they pass an end
        const bool left = cx == 0, right = cx == nx - 1;
        for (int run = 0; run < (left || right ? 2 : 1); ++run) {
            int lo = cx - 1, hi = cx + 1;
            float sx = 0.f;
            if (left) {
                if (run == 0) { lo = hi = nx - 1; sx = -g.box.x; }
                else lo = 0;
            } else if (right) {
                if (run == 0) hi = nx - 1;
                else { lo = hi = 0; sx = g.box.x; }
            }
            const int e = a.cell_start[base + hi + 1];
            for (int k = a.cell_start[base + lo]; k < e; ++k) {
                const float4 v = a.pos_cell[k];
                const float dx = p.x - (v.x + sx), dy = p.y - (v.y + sy), dz = p.z - (v.z + sz);
                const float r2 = dx * dx + dy * dy + dz * dz;
                if (r2 > g.rl2_hi) continue;
                const int j = __float_as_int(v.w);
                if (j == i || !(r2 < g.rl2_lo || ref_accept(a.pos[min(i, j)], a.pos[max(i, j)], g))) continue;
                if (up + down < a.row_cap) row[j > i ? up++ : a.row_cap - ++down] = (unsigned)(a.by_particle ? j : k);
                ++found;
            }
        }
    }
    row_counts(a, t, i, up, down, found);
}

// The half rows (neighbours above) into the flat pair arrays, 8 lanes per row.
// The pair-parallel kernels and the list's own readers need them; a million LJ
// particles' build takes 0.88 ms without and 1.16 ms with them.
__device__ __forceinline__ void half_rows(const CoopBuild& a, int gt, int gs) {
    const int sub = gt & 7;
    for (int t = gt >> 3; t < a.n; t += gs >> 3) {
        const int i = a.cell_particles[t], h = a.nb_half[i], o = a.row_off[i];
        const unsigned* row = a.nb_pad + (size_t)t * a.row_cap;
        for (int k = sub; k < h; k += 8) {
            const int e = (int)row[k];
            a.pair_i[o + k] = i;
            a.pair_j[o + k] = a.by_particle ? e : a.cell_particles[e];
        }
    }
}

__global__ void __launch_bounds__(256, 4) k_build_coop(CoopBuild a) {
    if (!a.flags[F_REBUILD]) return;   // grid-uniform: cleared only after the last barrier
    __shared__ RowQueue queue[8];
    cg::grid_group grid = cg::this_grid();
    const int gt = blockIdx.x * blockDim.x + threadIdx.x, gs = gridDim.x * blockDim.x;
    const int gw = gt >> 5, nwarps = gs >> 5;
    RowQueue& q = queue[threadIdx.x >> 5];
    if (gt == 0) a.flags[F_OVERFLOW] = 0;
    if (a.ncells) {
        // bin (cell_count is zero: the previous build cleared it after its scan)
        for (int c = gt; c < a.ncells; c += gs) a.cell_fill[c] = 0;
        for (int i = gt; i < a.n; i += gs) {
            float4 p = a.pos[i];
            const int c = cell_and_image(p, a.g);
            a.particle_cell[i] = c;
            atomicAdd(&a.cell_count[c], 1);
        }
        grid.sync();
        coop_scan(grid, a.cell_count, a.ncells, a.cell_start, nullptr, a.tmp);
        grid.sync();
        // members in arrival order; the counts are cleared for the next build
        for (int i = gt; i < a.n; i += gs) {
            const int c = a.particle_cell[i];
            a.cell_unsorted[a.cell_start[c] + atomicAdd(&a.cell_fill[c], 1)] = i;
        }
        for (int c = gt; c < a.ncells_cap; c += gs) a.cell_count[c] = 0;
        grid.sync();
        // each cell's members by index (a thread per member, which goes to its
        // rank: indices are distinct), their images in the same order
        for (int k = gt; k < a.n; k += gs) {
            const int v = a.cell_unsorted[k], c = a.particle_cell[v];
            const int b = a.cell_start[c], e = a.cell_start[c + 1];
            int rank = 0;
            for (int t = b; t < e; ++t) rank += a.cell_unsorted[t] < v;
            a.cell_particles[b + rank] = v;
            float4 p = a.pos[v];
            cell_and_image(p, a.g);
            p.w = __int_as_float(v);
            a.pos_cell[b + rank] = p;
        }
        grid.sync();
        switch (a.row_lanes) {
            case 0:
                for (int t = gt; t < a.n; t += gs) thread_row(a, t);
                break;
            case 1: search_rows<1, true>(a, q, gw, nwarps); break;
            case 4: search_rows<4, true>(a, q, gw, nwarps); break;
            default: search_rows<16, true>(a, q, gw, nwarps); break;
        }
    } else {
        for (int i = gt; i < a.n; i += gs) {
            float4 p = a.pos[i];
            if (a.g.periodic) cell_and_image(p, a.g);   // one cell: the image in the box
            p.w = __int_as_float(i);
            a.pos_cell[i] = p;
            a.cell_particles[i] = i;
        }
        grid.sync();
        if (a.row_lanes == 1) search_rows<1, false>(a, q, gw, nwarps);
        else search_rows<16, false>(a, q, gw, nwarps);
    }
    grid.sync();
    coop_scan(grid, a.nb_half, a.n, a.row_off, a.flags + F_NPAIRS, a.tmp);
    grid.sync();
    if (a.want_half) half_rows(a, gt, gs);
    for (int i = gt; i < a.n; i += gs) a.last[i] = a.pos[i];
    if (gt == 0) {
        const int builds = a.flags[F_BUILDS] + 1;
        a.flags[F_BUILDS] = builds;
        if (a.want_half) a.flags[F_HALF] = builds;
        a.flags[F_REBUILD] = 0;   // every block read it at entry, before the first barrier
    }
}

// The flat half list of the current rows, for callers that need it after
// builds that did not write it.
__global__ void __launch_bounds__(256) k_half_list(CoopBuild a) {
    if (a.flags[F_HALF] == a.flags[F_BUILDS]) return;
    half_rows(a, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}
__global__ void k_half_mark(int* flags) { flags[F_HALF] = flags[F_BUILDS]; }

int clear_grid(const sg_ctx* ctx) { return std::max(1, std::min(64, (ctx->nrep + 255) / 256)); }

// (0.4998 min(box))^2 with a margin, as a float that never exceeds the true value
float half_sq_of(const double* b) {
    const double h = 0.4998 * std::min(b[0], std::min(b[1], b[2]));
    return (float)(h * h * (1.0 - 1e-5));
}

ListGeom make_geom(const sg_ctx* ctx) {
    ListGeom g;
    g.box = make_float3((float)ctx->box[0], (float)ctx->box[1], (float)ctx->box[2]);
    g.inv_box = make_float3((float)(1.0 / ctx->box[0]), (float)(1.0 / ctx->box[1]), (float)(1.0 / ctx->box[2]));
    g.bx = ctx->box[0]; g.by = ctx->box[1]; g.bz = ctx->box[2];
    g.rl2 = ctx->nl.rl2;
    const double band = guard_band(std::max(ctx->box[0], std::max(ctx->box[1], ctx->box[2])), ctx->nl.rl2);
    g.rl2_lo = (float)(ctx->nl.rl2 * (1.0 - band));
    g.rl2_hi = (float)(ctx->nl.rl2 * (1.0 + band));
    g.half_sq = half_sq_of(ctx->box);
    g.periodic = ctx->periodic;
    for (int d = 0; d < 3; ++d) g.nc[d] = ctx->nl.ncell[d] > 0 ? ctx->nl.ncell[d] : 1;
    return g;
}

int scan(sg_ctx* ctx, const int* in, int m, int* out, int* total_dst, const int* flags) {
    int ntiles = (m + SCAN_TILE - 1) / SCAN_TILE;
    if (ntiles < 1) ntiles = 1;
    k_scan_tiles<<<ntiles, SCAN_BLOCK, 0, ctx->stream>>>(in, m, out, ctx->nl.scan_tmp, flags);
    k_scan_sums<<<1, SCAN_BLOCK, 0, ctx->stream>>>(ctx->nl.scan_tmp, ntiles, flags);
    k_scan_add<<<(m + 255) / 256 + 1, 256, 0, ctx->stream>>>(out, m, ctx->nl.scan_tmp, ntiles, total_dst, flags);
    SG_LAUNCH_CHECK(ctx, "scan");
    return SG_OK;
}

int alloc_rows(sg_ctx* ctx, int max_nb) {
    sg_nlist_state& nl = ctx->nl;
    if (nl.nb_pad) cudaFree(nl.nb_pad);
    if (nl.pair_i) cudaFree(nl.pair_i);
    if (nl.pair_j) cudaFree(nl.pair_j);
    if (nl.chunk_rep) cudaFree(nl.chunk_rep);
    nl.nb_pad = nl.pair_i = nl.pair_j = nl.chunk_rep = nullptr;
    ctx->graph_epoch++;
    nl.max_nb = max_nb;
    nl.pair_capacity = (int64_t)max_nb * ctx->n;
    if (ctx->nrep) {
        // each replica's rows in a section of their own, sized by its own capacity
        const int R = ctx->nrep;
        std::vector<long long> pad(R);
        long long total = 0;
        for (int r = 0; r < R; ++r) {
            pad[r] = total;
            total += (long long)nl.h_rep_max_nb[r] * (ctx->h_rep_off[r + 1] - ctx->h_rep_off[r]);
        }
        nl.pair_capacity = total;
        nl.h_rep_pad_off = pad;
        nl.max_nb = *std::max_element(nl.h_rep_max_nb.begin(), nl.h_rep_max_nb.end());
        if (total <= (long long)INT32_MAX) {
            SG_CUDA(ctx, cudaMemcpy(nl.rep_max_nb, nl.h_rep_max_nb.data(), sizeof(int) * R, cudaMemcpyHostToDevice));
            SG_CUDA(ctx, cudaMemcpy(nl.rep_pad_off, pad.data(), sizeof(long long) * R, cudaMemcpyHostToDevice));
            SG_CUDA(ctx, cudaMemset(nl.rep_need, 0, sizeof(int) * R));
        }
    }
    if (nl.pair_capacity > (int64_t)INT32_MAX)
        return sg_fail(ctx, SG_ECAPACITY, "neighbour list capacity %lld exceeds 2^31", (long long)nl.pair_capacity);
    // a single system's full rows hold half as much again (a row of low index
    // lists nearly all of its neighbours, so max_nb already covers a full row
    // of the mean density and more), in whole 16-byte pieces
    nl.row_cap = ctx->nrep ? 0 : (std::min(max_nb + max_nb / 2, ctx->n) + 3) / 4 * 4;
    nl.by_particle = !ctx->nrep && ctx->n <= SG_ROWS_DIRECT;
    SG_CUDA(ctx, cudaMalloc(&nl.nb_pad, sizeof(int) * (ctx->nrep ? (size_t)nl.pair_capacity
                                                                 : (size_t)nl.row_cap * (size_t)ctx->n)));
    SG_CUDA(ctx, cudaMalloc(&nl.pair_i, sizeof(int) * (size_t)nl.pair_capacity));
    SG_CUDA(ctx, cudaMalloc(&nl.pair_j, sizeof(int) * (size_t)nl.pair_capacity));
    if (ctx->nrep) SG_CUDA(ctx, cudaMalloc(&nl.chunk_rep, sizeof(int) * (size_t)(nl.pair_capacity / 32 + 2)));
    return SG_OK;
}

// Grid of the cooperative build (every block resident at once) and its
// scratch, sized once per context.
int coop_setup(sg_ctx* ctx) {
    sg_nlist_state& nl = ctx->nl;
    if (nl.coop_grid) return SG_OK;
    int per_sm = 0;
    SG_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_build_coop, 256, 0));
    if (per_sm < 1) return sg_fail(ctx, SG_ECUDA, "the cooperative list build does not fit an SM");
    const int grid = per_sm * ctx->num_sms;
    SG_CUDA(ctx, cudaMalloc(&nl.coop_tmp, sizeof(int) * (size_t)(grid + 1)));
    nl.coop_grid = grid;
    ctx->graph_epoch++;
    return SG_OK;
}

#define SG_LIST_SPARSE 2
// Lanes per row of a single system's search (search_rows): enough warps to
// fill the chip, since each walks its candidates one after another, and no
// more than that, since fewer rows then share a warp's candidates: four times
// the lanes at 32 768 to 131 072 particles took 8 to 40 % longer (ECP 127
// against 90 us, charged spheres 283 against 233). Cells of fewer than two
// particles: 0, a thread per row.
int row_lanes_for(const sg_ctx* ctx, int use_cells, int ncells) {
    const int64_t want = 16ll * ctx->num_sms;   // warps
    if (!use_cells) return ctx->n >= 32 * want ? 1 : 16;
    if (ctx->n < SG_LIST_SPARSE * (int64_t)ncells) return 0;
    return ctx->n >= 32 * want ? 1 : ctx->n >= 8 * want ? 4 : 16;
}

CoopBuild build_args(const sg_ctx* ctx, const ListGeom& g) {
    CoopBuild a;
    const sg_nlist_state& nl = ctx->nl;
    a.n = ctx->n;
    a.want_half = nl.half_in_build;
    a.by_particle = nl.by_particle;
    a.ncells = nl.use_cells ? nl.ncells : 0;
    a.ncells_cap = nl.ncells_cap;
    a.max_nb = nl.max_nb;
    a.row_cap = nl.row_cap;
    a.row_lanes = nl.row_lanes;
    a.pos = ctx->pos;
    a.g = g;
    a.cell_count = nl.cell_count;
    a.cell_fill = nl.cell_fill;
    a.cell_start = nl.cell_start;
    a.cell_unsorted = nl.cell_unsorted;
    a.cell_particles = nl.cell_particles;
    a.particle_cell = nl.particle_cell;
    a.pos_cell = nl.pos_cell;
    a.nb_pad = (unsigned*)nl.nb_pad;
    a.nb_count = (int2*)nl.nb_count;
    a.nb_half = nl.nb_half;
    a.row_off = nl.row_off;
    a.pair_i = nl.pair_i;
    a.pair_j = nl.pair_j;
    a.last = nl.pos_last;
    a.flags = nl.dev_flags;
    a.tmp = nl.coop_tmp;
    return a;
}

// Enqueue the (flag-gated) build kernels.
int enqueue_build(sg_ctx* ctx) {
    sg_nlist_state& nl = ctx->nl;
    const int n = ctx->n;
    ListGeom g = make_geom(ctx);
    const PadRep pad{nl.rep_max_nb, nl.rep_pad_off, nl.rep_need};
    if (!ctx->nrep) {
        // a single system: the cooperative kernel
        if (int rc = coop_setup(ctx)) return rc;
        CoopBuild a = build_args(ctx, g);
        void* args[] = {&a};
        // as many blocks as the row search has warps of rows, up to what is
        // resident at once: blocks without rows would wait at each barrier
        // while the search runs
        const int64_t row_threads = (int64_t)n * std::max(nl.row_lanes, 1);
        const int grid = (int)std::min<int64_t>(nl.coop_grid, (row_threads + 255) / 256);
        SG_CUDA(ctx, cudaLaunchCooperativeKernel((const void*)k_build_coop, grid, 256, args, 0, ctx->stream));
        return SG_OK;
    }
    // replica contexts: flag-gated kernels
    const RepItems items{nl.rep_items + 1, (int*)nl.rep_items};
    const int grid = 8 * ctx->num_sms;
    k_begin<<<1 + std::max(1, std::min(1024, (nl.ncells + 1023) / 1024)), 1024, 0, ctx->stream>>>(
            nl.dev_flags, nl.cell_count, nl.cell_fill, nl.ncells, ctx->rep.off, nl.rep_flag, ctx->nrep, items);
    k_bin<<<grid, 256, 0, ctx->stream>>>(ctx->pos, g, nl.particle_cell, nl.cell_count, nl.dev_flags, ctx->rep, items);
    if (int rc = scan(ctx, nl.cell_count, nl.ncells, nl.cell_start, nullptr, nl.dev_flags)) return rc;
    k_fill<<<grid, 256, 0, ctx->stream>>>(nl.particle_cell, nl.cell_start, nl.cell_fill, nl.cell_unsorted,
                                          nl.dev_flags, ctx->rep, items);
    k_sort_cells<<<(nl.ncells + 7) / 8, 256, 0, ctx->stream>>>(nl.ncells, nl.cell_start, nl.cell_unsorted,
                                                                nl.cell_particles, nl.dev_flags);
    k_rep_rows<<<grid, 256, 0, ctx->stream>>>(ctx->pos, g, nl.cell_start, nl.cell_particles, nl.nb_pad, nl.nb_count,
                                              nl.dev_flags, ctx->rep, pad, items);
    if (int rc = scan(ctx, nl.nb_count, n, nl.row_off, nl.dev_flags + F_NPAIRS, nl.dev_flags)) return rc;
    k_compact<<<grid, 256, 0, ctx->stream>>>(ctx->pos, nl.pos_last, nl.nb_pad, nl.nb_count, nl.row_off, nl.pair_i,
                                             nl.pair_j, nl.dev_flags, ctx->rep, pad, items);
    k_chunk_rep<<<ctx->num_sms * 8, 256, 0, ctx->stream>>>(nl.row_off, ctx->rep.off, ctx->nrep, nl.dev_flags,
                                                          nl.chunk_rep);
    k_clear_request<<<clear_grid(ctx), 256, 0, ctx->stream>>>(nl.dev_flags, nl.rep_flag, ctx->nrep, nl.rep_builds);
    SG_LAUNCH_CHECK(ctx, "nlist build");
    return SG_OK;
}

// Synchronous build with automatic regrowth on overflow.
int build_sync(sg_ctx* ctx) {
    for (int attempt = 0; attempt < 8; ++attempt) {
        k_set_request<<<clear_grid(ctx), 256, 0, ctx->stream>>>(ctx->nl.dev_flags, ctx->nl.rep_flag, ctx->nrep);
        if (int rc = enqueue_build(ctx)) return rc;
        if (int rc = sg_mail(ctx)) return rc;
        const int* flags = ctx->mail->flags;
        if (flags[F_OVERFLOW] == 0) return SG_OK;
        int want = ((flags[F_OVERFLOW] * 5 / 4) + 31) / 32 * 32;
        if (ctx->nrep) {
            // grow only the replicas whose rows overflowed
            const int R = ctx->nrep;
            std::vector<int> need(R);
            SG_CUDA(ctx, cudaMemcpy(need.data(), ctx->nl.rep_need, sizeof(int) * R, cudaMemcpyDeviceToHost));
            for (int r = 0; r < R; ++r)
                if (need[r] > ctx->nl.h_rep_max_nb[r])
                    ctx->nl.h_rep_max_nb[r] = std::min(((need[r] * 5 / 4) + 31) / 32 * 32,
                                                       ctx->h_rep_off[r + 1] - ctx->h_rep_off[r]);
        }
        if (int rc = alloc_rows(ctx, want)) return rc;
    }
    return sg_fail(ctx, SG_ECAPACITY, "neighbour list did not fit after regrowth");
}

}  // namespace

int sg_nlist_enqueue_check(sg_ctx* ctx) {
    k_check<<<(ctx->n + 255) / 256, 256, 0, ctx->stream>>>(ctx->n, ctx->pos, check_args(ctx));
    SG_LAUNCH_CHECK(ctx, "k_check");
    return SG_OK;
}

int sg_nlist_enqueue_build(sg_ctx* ctx) { return enqueue_build(ctx); }

// keep: later builds write the flat half list themselves (captured steps are
// captured again). Without it one kernel writes it now if it is out of date.
int sg_need_half_list(sg_ctx* ctx, bool keep) {
    sg_nlist_state& nl = ctx->nl;
    if (ctx->nrep || nl.half_in_build || !nl.initialized) return SG_OK;
    if (keep) {
        nl.half_in_build = 1;
        ctx->graph_epoch++;
    }
    const int grid = (int)std::min<int64_t>(8ll * ctx->num_sms, ((int64_t)ctx->n * 8 + 255) / 256);
    k_half_list<<<grid, 256, 0, ctx->stream>>>(build_args(ctx, make_geom(ctx)));
    k_half_mark<<<1, 1, 0, ctx->stream>>>(nl.dev_flags);
    SG_LAUNCH_CHECK(ctx, "k_half_list");
    return SG_OK;
}

int sg_nlist_free(sg_ctx* ctx) {
    sg_nlist_state& nl = ctx->nl;
    void* bufs[] = {nl.cell_count, nl.cell_start, nl.cell_fill, nl.cell_particles, nl.particle_cell, nl.nb_count,
                    nl.nb_pad, nl.row_off, nl.scan_tmp, nl.pair_i, nl.pair_j, nl.dev_flags, nl.pos_last, nl.pos_cell,
                    nl.rep_max_nb, nl.rep_pad_off, nl.rep_need, nl.rep_flag, nl.rep_builds, nl.rep_items, nl.cell_unsorted,
                    nl.chunk_rep, nl.coop_tmp, nl.nb_half, nl.spin_cell};
    for (void* b : bufs)
        if (b) cudaFree(b);
    nl = sg_nlist_state();
    return SG_OK;
}

// The box of a single-system context changed (sg_set_box, the barostat):
// cells must stay at least one list radius wide. A shrinking box gets fewer
// cells (within the allocated count); a growing one keeps its cells, which
// are then wider than needed. Under three cells per side the build falls
// back to the all-pairs rows. The current pair list is left as it is, as
// the reference's list is: the next needs_rebuild decides.
int sg_nlist_box_changed(sg_ctx* ctx) {
    sg_nlist_state& nl = ctx->nl;
    if (!nl.initialized || ctx->nrep) return SG_OK;
    const double rskin = nl.cutoff + nl.skin;
    int want[3];
    bool cells = ctx->periodic != 0 && nl.ncells_cap > 1;
    for (int d = 0; d < 3; ++d) {
        want[d] = (int)std::floor(ctx->box[d] / (rskin * (1.0 + 1e-4)));
        if (want[d] < 3) cells = false;
    }
    if (cells) {
        const long long prod = (long long)want[0] * want[1] * want[2];
        bool fits = prod <= nl.ncells_cap;
        if (!fits) {   // grew: keep the current grid if its cells are still wide enough
            fits = true;
            for (int d = 0; d < 3; ++d) {
                want[d] = nl.use_cells ? nl.ncell[d] : want[d];
                if (ctx->box[d] / want[d] < rskin * (1.0 + 1e-4)) fits = false;
            }
            if (!nl.use_cells) fits = false;
        }
        cells = fits;
    }
    if (cells) {
        for (int d = 0; d < 3; ++d) nl.ncell[d] = want[d];
        nl.use_cells = 1;
    } else {
        nl.ncell[0] = nl.ncell[1] = nl.ncell[2] = 1;
        nl.use_cells = 0;
    }
    nl.ncells = nl.ncell[0] * nl.ncell[1] * nl.ncell[2];
    nl.row_lanes = row_lanes_for(ctx, nl.use_cells, nl.ncells);
    ctx->graph_epoch++;
    return SG_OK;
}

extern "C" {

static int alloc_list(sg_ctx* ctx, int max_nb);

int sg_nlist_init(sg_ctx* ctx, double skin, double cutoff, int32_t trigger_mode) {
    if (!ctx) return SG_EINVAL;
    if (ctx->nrep) return sg_fail(ctx, SG_EINVAL, "a replica context takes sg_rep_nlist_init");
    if (!(skin >= 0.0) || !(cutoff > 0.0)) return sg_fail(ctx, SG_EINVAL, "skin must be >= 0 and cutoff > 0");
    if (ctx->box[0] <= 0.0) return sg_fail(ctx, SG_ENOTREADY, "sg_set_box must precede sg_nlist_init");
    for (int d = 0; d < 3; ++d)
        if (cutoff > ctx->box[d] / 2.0)
            return sg_fail(ctx, SG_ECUTOFF_GT_HALFBOX, "A cutoff of %.2f is too large for the box dimensions %.2f %.2f %.2f",
                           cutoff, ctx->box[0], ctx->box[1], ctx->box[2]);
    SG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    sg_nlist_free(ctx);
    ctx->graph_epoch++;
    sg_nlist_state& nl = ctx->nl;
    const int n = ctx->n;
    nl.cutoff = cutoff;
    nl.skin = skin;
    nl.trigger_mode = trigger_mode;
    double rskin = cutoff + skin;
    nl.rl2 = rskin * rskin;
    nl.trigger_sq = trigger_mode == 0 ? nl.rl2 : skin * skin;
    for (int d = 0; d < 3; ++d) nl.ncell[d] = (int)std::floor(ctx->box[d] / (rskin * (1.0 + 1e-4)));
    nl.use_cells = ctx->periodic && nl.ncell[0] >= 3 && nl.ncell[1] >= 3 && nl.ncell[2] >= 3;
    if (!nl.use_cells) nl.ncell[0] = nl.ncell[1] = nl.ncell[2] = 1;
    nl.ncells = nl.ncell[0] * nl.ncell[1] * nl.ncell[2];
    nl.row_lanes = row_lanes_for(ctx, nl.use_cells, nl.ncells);
    double vol = ctx->box[0] * ctx->box[1] * ctx->box[2];
    double rho = n / vol;
    // rows hold the j > i neighbours in index order, so a particle of low
    // index can list nearly all of its neighbours: size for the full count
    double expect = (4.0 / 3.0) * M_PI * rskin * rskin * rskin * rho;
    nl.mean_row = expect;
    int max_nb = (int)std::ceil(expect * 1.3 + 32.0);
    max_nb = (max_nb + 31) / 32 * 32;
    if (max_nb > n) max_nb = std::max(1, n);
    return alloc_list(ctx, max_nb);
}

// Buffers of a list with nl.ncells cells and rows of max_nb, then a build.
static int alloc_list(sg_ctx* ctx, int max_nb) {
    sg_nlist_state& nl = ctx->nl;
    const int n = ctx->n;
    int ntiles = std::max((n + SCAN_TILE - 1) / SCAN_TILE, (nl.ncells + SCAN_TILE - 1) / SCAN_TILE) + 2;
    nl.ncells_cap = nl.ncells;
    SG_CUDA(ctx, cudaMalloc(&nl.cell_count, sizeof(int) * (size_t)nl.ncells));
    // zero before the first build: the cooperative build clears the counts after use
    SG_CUDA(ctx, cudaMemsetAsync(nl.cell_count, 0, sizeof(int) * (size_t)nl.ncells, ctx->stream));
    SG_CUDA(ctx, cudaMalloc(&nl.cell_start, sizeof(int) * ((size_t)nl.ncells + 1)));
    SG_CUDA(ctx, cudaMalloc(&nl.cell_fill, sizeof(int) * (size_t)nl.ncells));
    SG_CUDA(ctx, cudaMalloc(&nl.cell_particles, sizeof(int) * (size_t)n));
    SG_CUDA(ctx, cudaMalloc(&nl.cell_unsorted, sizeof(int) * (size_t)n));
    SG_CUDA(ctx, cudaMalloc(&nl.pos_cell, sizeof(float4) * (size_t)n));
    SG_CUDA(ctx, cudaMalloc(&nl.particle_cell, sizeof(int) * (size_t)n));
    SG_CUDA(ctx, cudaMalloc(&nl.nb_count, sizeof(int) * (ctx->nrep ? 1 : 2) * (size_t)n));
    if (!ctx->nrep) SG_CUDA(ctx, cudaMalloc(&nl.nb_half, sizeof(int) * (size_t)n));
    SG_CUDA(ctx, cudaMalloc(&nl.row_off, sizeof(int) * ((size_t)n + 1)));
    SG_CUDA(ctx, cudaMalloc(&nl.scan_tmp, sizeof(int) * (size_t)(ntiles + 1)));
    SG_CUDA(ctx, cudaMalloc(&nl.dev_flags, sizeof(int) * 8));
    SG_CUDA(ctx, cudaMalloc(&nl.pos_last, sizeof(float4) * (size_t)n));
    SG_CUDA(ctx, cudaMemsetAsync(nl.dev_flags, 0, sizeof(int) * 8, ctx->stream));
    if (int rc = alloc_rows(ctx, max_nb)) return rc;
    nl.initialized = 1;
    return build_sync(ctx);
}

// Per-replica lists of a batched context: each replica gets its own cell grid
// (or one cell when its box is under three list radii per side), its own list
// radius (cutoff[f] + skin[f] of its potential family f) and its own trigger.
int sg_rep_nlist_init(sg_ctx* ctx, const double* skin, const double* cutoff, int32_t trigger_mode) {
    if (!ctx || !skin || !cutoff) return SG_EINVAL;
    if (!ctx->nrep) return sg_fail(ctx, SG_EINVAL, "not a replica context");
    const int R = ctx->nrep;
    std::vector<double> rl2(R), trig(R);
    std::vector<int4> grid(R);
    std::vector<int> max_nb_r(R);
    int total_cells = 0;
    for (int r = 0; r < R; ++r) {
        const int f = ctx->h_rep_family[r];
        const double* b = &ctx->h_rep_box[3 * r];
        if (!(skin[f] >= 0.0) || !(cutoff[f] > 0.0)) return sg_fail(ctx, SG_EINVAL, "bad skin / cutoff for family %d", f);
        for (int d = 0; d < 3; ++d)
            if (cutoff[f] > b[d] / 2.0)
                return sg_fail(ctx, SG_ECUTOFF_GT_HALFBOX, "replica %d: a cutoff of %.2f is too large for the box %.2f",
                               r, cutoff[f], b[d]);
        const double rs = cutoff[f] + skin[f];
        rl2[r] = rs * rs;
        trig[r] = trigger_mode == 0 ? rl2[r] : skin[f] * skin[f];
        int nc[3];
        bool cells = true;
        for (int d = 0; d < 3; ++d) {
            nc[d] = (int)std::floor(b[d] / (rs * (1.0 + 1e-4)));
            if (nc[d] < 3) cells = false;
        }
        grid[r] = cells ? make_int4(nc[0], nc[1], nc[2], total_cells) : make_int4(0, 0, 0, total_cells);
        total_cells += cells ? nc[0] * nc[1] * nc[2] : 1;
        const int nr = ctx->h_rep_off[r + 1] - ctx->h_rep_off[r];

        const double rho = nr / (b[0] * b[1] * b[2]);
        // full neighbour count: index-ordered half rows of low index reach it
        const double expect = (4.0 / 3.0) * M_PI * rs * rs * rs * rho;
        int mnb = (int)std::ceil(expect * 1.3 + 32.0);
        max_nb_r[r] = std::max(1, std::min((mnb + 31) / 32 * 32, nr));
    }
    SG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    sg_nlist_free(ctx);
    ctx->graph_epoch++;
    std::vector<float2> bands(R);
    for (int r = 0; r < R; ++r) {
        const double* b = &ctx->h_rep_box[3 * r];
        const double band = guard_band(std::max(b[0], std::max(b[1], b[2])), rl2[r]);
        bands[r] = make_float2((float)(rl2[r] * (1.0 - band)), (float)(rl2[r] * (1.0 + band)));
    }
    SG_CUDA(ctx, cudaMemcpy((void*)ctx->rep.rl2_band, bands.data(), sizeof(float2) * R, cudaMemcpyHostToDevice));
    SG_CUDA(ctx, cudaMemcpy((void*)ctx->rep.rl2, rl2.data(), sizeof(double) * R, cudaMemcpyHostToDevice));
    SG_CUDA(ctx, cudaMemcpy((void*)ctx->rep.trig, trig.data(), sizeof(double) * R, cudaMemcpyHostToDevice));
    SG_CUDA(ctx, cudaMemcpy((void*)ctx->rep.grid, grid.data(), sizeof(int4) * R, cudaMemcpyHostToDevice));
    sg_nlist_state& nl = ctx->nl;
    nl.trigger_mode = trigger_mode;
    nl.use_cells = 1;
    nl.ncell[0] = nl.ncell[1] = nl.ncell[2] = 1;
    nl.ncells = total_cells;
    nl.row_lanes = 0;
    nl.h_rep_max_nb = max_nb_r;
    SG_CUDA(ctx, cudaMalloc(&nl.rep_max_nb, sizeof(int) * R));
    SG_CUDA(ctx, cudaMalloc(&nl.rep_pad_off, sizeof(long long) * R));
    SG_CUDA(ctx, cudaMalloc(&nl.rep_need, sizeof(int) * R));
    SG_CUDA(ctx, cudaMalloc(&nl.rep_flag, sizeof(int) * R));
    SG_CUDA(ctx, cudaMemset(nl.rep_flag, 0, sizeof(int) * R));
    int max_items = 0;
    for (int r = 0; r < R; ++r) max_items += (ctx->h_rep_off[r + 1] - ctx->h_rep_off[r] + REP_ROWS - 1) / REP_ROWS;
    SG_CUDA(ctx, cudaMalloc(&nl.rep_items, sizeof(int2) * (1 + (size_t)max_items)));
    SG_CUDA(ctx, cudaMalloc(&nl.rep_builds, sizeof(int) * R));
    SG_CUDA(ctx, cudaMemset(nl.rep_builds, 0, sizeof(int) * R));
    return alloc_list(ctx, *std::max_element(max_nb_r.begin(), max_nb_r.end()));
}

int sg_nlist_build(sg_ctx* ctx) {
    if (!ctx) return SG_EINVAL;
    if (!ctx->nl.initialized) return sg_fail(ctx, SG_ENOTREADY, "sg_nlist_init must precede sg_nlist_build");
    return build_sync(ctx);
}

int sg_nlist_needs_rebuild(sg_ctx* ctx, int32_t* flag) {
    if (!ctx || !flag) return SG_EINVAL;
    if (!ctx->nl.initialized) return sg_fail(ctx, SG_ENOTREADY, "sg_nlist_init must precede sg_nlist_needs_rebuild");
    k_clear_request<<<clear_grid(ctx), 256, 0, ctx->stream>>>(ctx->nl.dev_flags, ctx->nl.rep_flag, ctx->nrep,
                                                              nullptr);
    k_check<<<(ctx->n + 255) / 256, 256, 0, ctx->stream>>>(ctx->n, ctx->pos, check_args(ctx));
    SG_LAUNCH_CHECK(ctx, "k_check");
    if (int rc = sg_mail(ctx, !ctx->nrep)) return rc;
    *flag = ctx->mail->flags[F_REBUILD];
    if (ctx->nrep)
        k_clear_request<<<clear_grid(ctx), 256, 0, ctx->stream>>>(ctx->nl.dev_flags, ctx->nl.rep_flag, ctx->nrep,
                                                                  nullptr);
    return SG_OK;
}

int sg_nlist_update(sg_ctx* ctx) {
    if (!ctx) return SG_EINVAL;
    if (!ctx->nl.initialized) return sg_fail(ctx, SG_ENOTREADY, "sg_nlist_init must precede sg_nlist_update");
    k_check<<<(ctx->n + 255) / 256, 256, 0, ctx->stream>>>(ctx->n, ctx->pos, check_args(ctx));
    SG_LAUNCH_CHECK(ctx, "k_check");
    return enqueue_build(ctx);
}

int sg_nlist_count(sg_ctx* ctx, int64_t* npairs) {
    if (!ctx || !npairs) return SG_EINVAL;
    if (!ctx->nl.initialized) return sg_fail(ctx, SG_ENOTREADY, "no neighbour list");
    if (int rc = sg_mail(ctx)) return rc;
    const int* flags = ctx->mail->flags;
    if (flags[F_OVERFLOW]) return sg_fail(ctx, SG_ECAPACITY, "neighbour list overflowed (row of %d)", flags[F_OVERFLOW]);
    *npairs = flags[F_NPAIRS];
    return SG_OK;
}

int sg_nlist_replica_builds(sg_ctx* ctx, int64_t* counts) {
    if (!ctx || !counts) return SG_EINVAL;
    if (!ctx->nl.initialized || !ctx->nl.rep_builds)
        return sg_fail(ctx, SG_ENOTREADY, "no per-replica lists (sg_rep_nlist_init first)");
    std::vector<int> c(ctx->nrep);
    SG_CUDA(ctx, cudaMemcpyAsync(c.data(), ctx->nl.rep_builds, sizeof(int) * c.size(), cudaMemcpyDeviceToHost,
                                 ctx->stream));
    SG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (int r = 0; r < ctx->nrep; ++r) counts[r] = c[r];
    return SG_OK;
}

int sg_nlist_builds(sg_ctx* ctx, int64_t* builds) {
    if (!ctx || !builds) return SG_EINVAL;
    if (!ctx->nl.initialized) return sg_fail(ctx, SG_ENOTREADY, "no neighbour list");
    if (int rc = sg_mail(ctx)) return rc;
    const int* flags = ctx->mail->flags;
    *builds = flags[F_BUILDS];
    return SG_OK;
}

}  // extern "C"

// Storage index of every pair in row order (identity for a single system;
// replica sections otherwise), with the row offsets.
int sg_pair_storage_index(sg_ctx* ctx, int64_t k, std::vector<int>& off, std::vector<int64_t>& where) {
    const int n = ctx->n;
    off.assign(n + 1, 0);
    SG_CUDA(ctx, cudaMemcpyAsync(off.data(), ctx->nl.row_off, sizeof(int) * (n + 1), cudaMemcpyDeviceToHost, ctx->stream));
    SG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    where.resize(k);
    if (!ctx->nrep) {
        for (int64_t v = 0; v < k; ++v) where[v] = v;
        return SG_OK;
    }
    for (int r = 0; r < ctx->nrep; ++r) {
        const int64_t v0 = off[ctx->h_rep_off[r]], v1 = off[ctx->h_rep_off[r + 1]];
        for (int64_t v = v0; v < v1; ++v) where[v] = ctx->nl.h_rep_pad_off[r] + (v - v0);
    }
    return SG_OK;
}

// Row-order copy of a device array of per-pair values.
template <class T>
static int gather_pairs(sg_ctx* ctx, const T* dev, int64_t k, T* out) {
    if (k <= 0) return SG_OK;
    if (!ctx->nrep) {
        SG_CUDA(ctx, cudaMemcpyAsync(out, dev, sizeof(T) * k, cudaMemcpyDeviceToHost, ctx->stream));
        SG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        return SG_OK;
    }
    std::vector<int> off;
    std::vector<int64_t> where;
    if (int rc = sg_pair_storage_index(ctx, k, off, where)) return rc;
    std::vector<T> all((size_t)ctx->nl.pair_capacity);
    SG_CUDA(ctx, cudaMemcpyAsync(all.data(), dev, sizeof(T) * all.size(), cudaMemcpyDeviceToHost, ctx->stream));
    SG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (int64_t v = 0; v < k; ++v) out[v] = all[where[v]];
    return SG_OK;
}

int sg_gather_pair_floats(sg_ctx* ctx, const float* dev, int64_t k, float* out) { return gather_pairs(ctx, dev, k, out); }

extern "C" {

int sg_nlist_pairs(sg_ctx* ctx, int32_t* pi, int32_t* pj, int64_t capacity, int64_t* npairs) {
    if (!ctx || !npairs) return SG_EINVAL;
    int64_t k = 0;
    if (int rc = sg_nlist_count(ctx, &k)) return rc;
    *npairs = k;
    if (k > capacity || (k > 0 && (!pi || !pj))) return sg_fail(ctx, SG_ECAPACITY, "pair capacity too small");
    if (int rc = sg_need_half_list(ctx, false)) return rc;
    if (int rc = gather_pairs(ctx, ctx->nl.pair_i, k, pi)) return rc;
    return gather_pairs(ctx, ctx->nl.pair_j, k, pj);
}

int sg_nlist_export(sg_ctx* ctx, int32_t* nlist, int64_t capacity, int32_t* offset, int64_t* npairs, int32_t one_based) {
    if (!ctx || !offset || !npairs) return SG_EINVAL;
    int64_t k = 0;
    if (int rc = sg_nlist_count(ctx, &k)) return rc;
    *npairs = k;
    if (k > capacity || (!nlist && k > 0)) return sg_fail(ctx, SG_ECAPACITY, "export capacity %lld < %lld pairs",
                                                          (long long)capacity, (long long)k);
    if (int rc = sg_need_half_list(ctx, false)) return rc;
    const int n = ctx->n;
    std::vector<int> off(n + 1), pj(k > 0 ? k : 1);
    SG_CUDA(ctx, cudaMemcpyAsync(off.data(), ctx->nl.row_off, sizeof(int) * (n + 1), cudaMemcpyDeviceToHost, ctx->stream));
    SG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (int rc = gather_pairs(ctx, ctx->nl.pair_j, k, pj.data())) return rc;
    for (int i = 0; i < n; ++i) std::sort(pj.begin() + off[i], pj.begin() + off[i + 1]);
    for (int64_t t = 0; t < k; ++t) nlist[t] = pj[t] + (one_based ? 1 : 0);
    if (one_based) {
        // offset(I) = start of row I, offset(N) = K+1 (system.f90:977,1000)
        for (int i = 0; i < n - 1; ++i) offset[i] = off[i] + 1;
        offset[n - 1] = (int)k + 1;
    } else {
        for (int i = 0; i <= n; ++i) offset[i] = off[i];
    }
    return SG_OK;
}

}  // extern "C"
