// Prior-map grid and batched point-to-plane ICP for global localisation, on sm_100a.
//
// Reference: python/livox_warp/mapgrid.py -- Grid / grid_flat / grid_at / cell_centre :35-65, nearest_point :68-102,
// k_seed :105-114, k_unpack :117-125, k_jfa :128-158, k_df :161-170, PriorGrid.build :272-296;
// python/livox_warp/localize.py -- k_icp_batch :126-167, k_reduce_batch :170-179, k_eval_batch :182-205,
// GlobalLocalizer._icp :517-553, _evaluate :555-565.
//
// The grid build seeds each cell with a 64-bit key (distance in mm << 32 | point index) instead of the
// reference's 32-bit (mm << 23 | index), which held at most 2^23 - 1 map points, and floods between two
// buffers instead of in place, so the flood's result does not depend on thread timing.
//
// The batched ICP runs every hypothesis -- each with its own scan, of any length -- in one cooperative launch:
// tiles of one hypothesis' points accumulate float32 terms into float64 tile partials; after a grid barrier
// each hypothesis sums its tiles in a fixed order and solves its 6x6 system (Cholesky, float64); after a second
// barrier every CTA reads the largest step of the iteration and the schedule stage ends when it is below 2e-4
// (localize.py:536-552). The evaluation counts of localize.py:182-205 follow in the same launch.
#include <cmath>
#include <type_traits>

#include "lw_common.cuh"
#include "lw_linalg.cuh"

namespace lw {

// ---- grid geometry (mapgrid.py:35-65) --------------------------------------------------------------------
__device__ __forceinline__ int64_t grid_flat(const lw_prior_grid& g, int ix, int iy, int iz) {
    if (ix < 0 || iy < 0 || iz < 0 || ix >= g.nx || iy >= g.ny || iz >= g.nz) return -1;
    return ((int64_t)iz * g.ny + iy) * g.nx + ix;
}

__device__ __forceinline__ void grid_idx(const lw_prior_grid& g, float x, float y, float z, int& ix, int& iy, int& iz) {
    ix = ifloor((x - g.origin[0]) * g.inv_cell);
    iy = ifloor((y - g.origin[1]) * g.inv_cell);
    iz = ifloor((z - g.origin[2]) * g.inv_cell);
}

__device__ __forceinline__ void cell_centre(const lw_prior_grid& g, int64_t c, float& x, float& y, float& z) {
    int64_t ix = c % g.nx, r = c / g.nx;
    int64_t iy = r % g.ny, iz = r / g.ny;
    x = g.origin[0] + ((float)ix + 0.5f) * g.cell;
    y = g.origin[1] + ((float)iy + 0.5f) * g.cell;
    z = g.origin[2] + ((float)iz + 0.5f) * g.cell;
}

__device__ __forceinline__ float4 ld_pt(const float4* __restrict__ xyzp, int64_t i) { return __ldg(xyzp + i); }

constexpr float BOX_SLACK = 1.0e-4f;  // m: covers the float rounding of cell assignment and of the box offsets

// The map point nearest to w (mapgrid.py:68-102): exact within one cell -- the first point, in the reference's
// scan order (dz, dy, dx, then index), at the smallest distance below one cell -- otherwise the closest of the
// 27 cells' flooded seeds, or -1 beyond the band.
//
// Same result, fewer reads: the own cell is scanned first, and its smallest distance ub bounds the answer; a
// neighbour cell whose box lies farther than ub from w (less BOX_SLACK) holds no point that could be the first
// minimum, so its points are skipped. The seeds are still compared for every cell while nothing within one cell
// has been found, as the reference does. The own cell's contribution in the scan order is its own first minimum.
__device__ int nearest_point(const lw_prior_grid& g, float wx, float wy, float wz) {
    const float4* __restrict__ P = reinterpret_cast<const float4*>(g.xyz);
    int ix, iy, iz;
    grid_idx(g, wx, wy, wz, ix, iy, iz);
    const float cell2 = g.cell * g.cell;
    // w's offsets from its own cell's lower faces
    const float fx = (wx - g.origin[0]) - (float)ix * g.cell;
    const float fy = (wy - g.origin[1]) - (float)iy * g.cell;
    const float fz = (wz - g.origin[2]) - (float)iz * g.cell;
    int own = -1;
    float own_d2 = cell2;
    const int64_t c0 = grid_flat(g, ix, iy, iz);
    if (c0 >= 0) {
        const int k0 = __ldg(g.start + c0), k1 = __ldg(g.start + c0 + 1);
        for (int k = k0; k < k1; ++k) {
            const float4 q = ld_pt(P, k);
            const float ex = wx - q.x, ey = wy - q.y, ez = wz - q.z;
            const float d2 = ex * ex + ey * ey + ez * ez;
            if (d2 < own_d2) {
                own_d2 = d2;
                own = k;
            }
        }
    }
    const float ub = own_d2 * 1.00001f;
    int best = -1;
    float bd = cell2;
    int seed = -1;
    float sd = 1.0e30f;
    for (int dz = -1; dz <= 1; ++dz) {
        const float lz = fmaxf((dz < 0 ? fz : (dz > 0 ? g.cell - fz : 0.0f)) - BOX_SLACK, 0.0f);
        for (int dy = -1; dy <= 1; ++dy) {
            const float ly = fmaxf((dy < 0 ? fy : (dy > 0 ? g.cell - fy : 0.0f)) - BOX_SLACK, 0.0f);
            for (int dx = -1; dx <= 1; ++dx) {
                const int64_t c = grid_flat(g, ix + dx, iy + dy, iz + dz);
                if (c < 0) continue;
                if (dx == 0 && dy == 0 && dz == 0) {
                    if (own >= 0 && own_d2 < bd) {
                        bd = own_d2;
                        best = own;
                    }
                } else {
                    const float lx = fmaxf((dx < 0 ? fx : (dx > 0 ? g.cell - fx : 0.0f)) - BOX_SLACK, 0.0f);
                    if (lx * lx + ly * ly + lz * lz <= ub) {
                        const int k0 = __ldg(g.start + c), k1 = __ldg(g.start + c + 1);
                        for (int k = k0; k < k1; ++k) {
                            const float4 q = ld_pt(P, k);
                            const float ex = wx - q.x, ey = wy - q.y, ez = wz - q.z;
                            const float d2 = ex * ex + ey * ey + ez * ez;
                            if (d2 < bd) {
                                bd = d2;
                                best = k;
                            }
                        }
                    }
                }
                if (best < 0) {
                    const int s = __ldg(g.nn + c);
                    if (s >= 0) {
                        const float4 q = ld_pt(P, s);
                        const float ex = wx - q.x, ey = wy - q.y, ez = wz - q.z;
                        const float d2 = ex * ex + ey * ey + ez * ez;
                        if (d2 < sd) {
                            sd = d2;
                            seed = s;
                        }
                    }
                }
            }
        }
    }
    return best >= 0 ? best : seed;
}

// nearest_point for a query whose answer a moment ago, or in the pose before, was point `prev` (-1: unknown). Points are
// sorted by cell with x fastest, so the scan order (dz, dy, dx, then index) is the order of the indices and the three cells of
// a row are one run of points. Where prev lies surely within the 27 cells (closer than a cell less twice BOX_SLACK), its
// distance bounds the answer before anything is scanned, and rows and cells whose boxes lie farther are passed over; the
// first minimum is then found among the rest as before. While nothing lies within a cell the 27 seeds are compared in
// order, a seed equal to the last one once.
// The runs to scan are listed first (runs: 9 slots of shared memory per lane, this lane's column) and then walked, two points
// a step: a warp takes as many steps as its busiest lane has points, where walking row by row takes the busiest lane's of
// every row.
__device__ int nearest_warm(const lw_prior_grid& g, float wx, float wy, float wz, int prev, int2 (*runs)[32]) {
    const float4* __restrict__ P = reinterpret_cast<const float4*>(g.xyz);
    int ix, iy, iz;
    grid_idx(g, wx, wy, wz, ix, iy, iz);
    if (ix < -1 || iy < -1 || iz < -1 || ix > g.nx || iy > g.ny || iz > g.nz) return -1;  // none of the 27 is in the grid
    const float cell2 = g.cell * g.cell;
    const float fx = (wx - g.origin[0]) - (float)ix * g.cell;
    const float fy = (wy - g.origin[1]) - (float)iy * g.cell;
    const float fz = (wz - g.origin[2]) - (float)iz * g.cell;
    const int64_t nx = g.nx, nxy = nx * g.ny;
    const int64_t c0 = iz * nxy + iy * nx + ix;
    const bool own_in = ix >= 0 && iy >= 0 && iz >= 0 && ix < g.nx && iy < g.ny && iz < g.nz;
    float ub = cell2;
    if (prev >= 0 && prev < g.n) {
        const float4 q = ld_pt(P, prev);
        const float ex = wx - q.x, ey = wy - q.y, ez = wz - q.z;
        const float d2 = ex * ex + ey * ey + ez * ez;
        const float sure = g.cell - 2.0f * BOX_SLACK;
        if (sure > 0.0f && d2 < sure * sure) ub = d2;
    } else if (own_in) {
        const int k1 = __ldg(g.start + c0 + 1);
        for (int k = __ldg(g.start + c0); k < k1; ++k) {
            const float4 q = ld_pt(P, k);
            const float ex = wx - q.x, ey = wy - q.y, ez = wz - q.z;
            ub = fminf(ub, ex * ex + ey * ey + ez * ez);
        }
    }
    ub *= 1.00001f;
    auto gap2 = [&](float f, int o) {
        const float l = fmaxf((o < 0 ? f : (o > 0 ? g.cell - f : 0.0f)) - BOX_SLACK, 0.0f);
        return l * l;
    };
    const float xl = gap2(fx, -1), xr = gap2(fx, 1);
    const int lane = threadIdx.x & 31;
    int n = 0;
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz) {
        const float z2 = gap2(fz, dz);
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy) {
            const float yz2 = gap2(fy, dy) + z2;
            const int lo = max(xl + yz2 > ub ? ix : ix - 1, 0), hi = min(xr + yz2 > ub ? ix : ix + 1, g.nx - 1);
            const bool in = yz2 <= ub && lo <= hi && iz + dz >= 0 && iz + dz < g.nz && iy + dy >= 0 && iy + dy < g.ny;
            if (in) {
                const int32_t* row = g.start + (c0 + dz * nxy + dy * nx - ix);
                const int k0 = __ldg(row + lo), k1 = __ldg(row + hi + 1);
                if (k0 < k1) runs[n++][lane] = make_int2(k0, k1);
            }
        }
    }
    int best = -1;
    float bd = cell2;
    int j = 0, k = 0, k1 = 0;
    while (true) {
        if (k >= k1) {
            if (j >= n) break;
            const int2 r = runs[j++][lane];
            k = r.x;
            k1 = r.y;
        }
        const int l = min(k + 1, k1 - 1);
        const float4 q = ld_pt(P, k), r = ld_pt(P, l);
        const float ex = wx - q.x, ey = wy - q.y, ez = wz - q.z;
        const float d2 = ex * ex + ey * ey + ez * ez;
        const float fx2 = wx - r.x, fy2 = wy - r.y, fz2 = wz - r.z;
        const float e2 = fx2 * fx2 + fy2 * fy2 + fz2 * fz2;
        if (d2 < bd) {
            bd = d2;
            best = k;
        }
        if (e2 < bd) {
            bd = e2;
            best = l;
        }
        k += 2;
    }
    if (best >= 0) return best;
    int seed = -1, last = -1;
    float sd = 1.0e30f;
    // a row of three seeds at a time, the next row's already on their way
    auto row_of = [&](int r, int (&v)[3]) {
        const int z = iz + r / 3 - 1, y = iy + r % 3 - 1;
        const bool in = r < 9 && z >= 0 && y >= 0 && z < g.nz && y < g.ny;
        const int32_t* row = g.nn + (in ? z * nxy + y * nx : 0);
#pragma unroll
        for (int o = 0; o < 3; ++o) {
            const int x = ix + o - 1;
            v[o] = in && x >= 0 && x < g.nx ? __ldg(row + x) : -1;
        }
    };
    int next[3];
    row_of(0, next);
#pragma unroll 1
    for (int r = 0; r < 9; ++r) {
        const int s0 = next[0], s1 = next[1], s2 = next[2];
        row_of(r + 1, next);
        const bool b0 = s0 >= 0 && s0 != last;
        last = s0 >= 0 ? s0 : last;
        const bool b1 = s1 >= 0 && s1 != last;
        last = s1 >= 0 ? s1 : last;
        const bool b2 = s2 >= 0 && s2 != last;
        last = s2 >= 0 ? s2 : last;
        if (!(b0 || b1 || b2)) continue;
        const float4 q0 = ld_pt(P, b0 ? s0 : last), q1 = ld_pt(P, b1 ? s1 : last), q2 = ld_pt(P, b2 ? s2 : last);
        auto take = [&](bool on, int s, float4 q) {
            const float ex = wx - q.x, ey = wy - q.y, ez = wz - q.z;
            const float d2 = ex * ex + ey * ey + ez * ez;
            if (on && d2 < sd) {
                sd = d2;
                seed = s;
            }
        };
        take(b0, s0, q0);
        take(b1, s1, q1);
        take(b2, s2, q2);
    }
    return seed;
}

// ---- grid build (mapgrid.py:105-170, 272-296) -------------------------------------------------------------
__global__ void k_seed_clear(lw_prior_grid g) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < g.ncell; c += (int64_t)gridDim.x * blockDim.x)
        g.seed[c] = ~0ULL;
}

__global__ void k_seed(lw_prior_grid g) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < g.n; i += (int64_t)gridDim.x * blockDim.x) {
        const float4 p = ld_pt(reinterpret_cast<const float4*>(g.xyz), i);
        int ix, iy, iz;
        grid_idx(g, p.x, p.y, p.z, ix, iy, iz);
        int64_t c = grid_flat(g, ix, iy, iz);
        if (c < 0) continue;
        float cx, cy, cz;
        cell_centre(g, c, cx, cy, cz);
        int dmm = (int)(len3(p.x - cx, p.y - cy, p.z - cz) * 1000.0f);
        if (dmm > 255) dmm = 255;
        atomicMin((unsigned long long*)(g.seed + c), ((unsigned long long)dmm << 32) | (unsigned long long)i);
    }
}

__global__ void k_unpack(lw_prior_grid g) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < g.ncell; c += (int64_t)gridDim.x * blockDim.x) {
        uint64_t v = g.seed[c];
        g.nn2[c] = v == ~0ULL ? -1 : (int32_t)(v & 0xFFFFFFFFULL);
    }
}

// One flood step from `in` to `out`: the nearest of the seeds held STEP cells away in the 26 directions. Bound by instruction
// issue: a thread per cell of a 32 x 8 patch of a z layer, so that no cell index is divided, in 32 bits where the grid's
// cells fit (IDX); patches that lie STEP inside the grid read their neighbours without range checks; a seed equal to the
// last one compared is passed over (it cannot win twice; neighbours along x mostly hold the same). A flat index with its
// 64-bit divisions and a check per neighbour took 0.57 ms per step on 11.5M cells, 32-bit indices with the checks 0.37.
constexpr int JFA_X = 32, JFA_Y = 8;
// LAST also writes the distance field: the winner's distance in whole cm, 255 beyond the band (mapgrid.py:161-170).
template <class IDX, int STEP, bool LAST>
__global__ void __launch_bounds__(JFA_X * JFA_Y) k_jfa(lw_prior_grid g, const int32_t* __restrict__ in,
                                                       int32_t* __restrict__ out, int tiles_x, int tiles_y) {
    const int x0 = (int)(blockIdx.x % tiles_x) * JFA_X, tile = blockIdx.x / tiles_x;
    const int y0 = tile % tiles_y * JFA_Y, iz = tile / tiles_y;
    const int ix = x0 + threadIdx.x, iy = y0 + threadIdx.y;
    const bool inside = x0 >= STEP && y0 >= STEP && iz >= STEP && x0 + JFA_X + STEP <= g.nx && y0 + JFA_Y + STEP <= g.ny &&
                        iz + STEP < g.nz;
    if (ix >= g.nx || iy >= g.ny) return;
    const IDX nxy = (IDX)g.nx * g.ny, c = iz * nxy + (IDX)iy * g.nx + ix;
    // the 27 seeds first (independent loads), then the distances
    int seed[27];
    if (inside) {
#pragma unroll
        for (int r = 0; r < 9; ++r) {
            const int32_t* row = in + (c + (IDX)(r / 3 - 1) * STEP * nxy + (IDX)(r % 3 - 1) * STEP * g.nx);
            seed[3 * r] = __ldg(row - STEP);
            seed[3 * r + 1] = __ldg(row);
            seed[3 * r + 2] = __ldg(row + STEP);
        }
    } else {
#pragma unroll
        for (int k = 0; k < 27; ++k) {
            const int jx = ix + (k % 3 - 1) * STEP, jy = iy + (k / 3 % 3 - 1) * STEP, jz = iz + (k / 9 - 1) * STEP;
            const bool in_grid = jx >= 0 && jy >= 0 && jz >= 0 && jx < g.nx && jy < g.ny && jz < g.nz;
            seed[k] = in_grid ? __ldg(in + (jz * nxy + (IDX)jy * g.nx + jx)) : -1;
        }
    }
    int any = seed[0];
#pragma unroll
    for (int k = 1; k < 27; ++k) any = max(any, seed[k]);
    int best = seed[13];
    float bd = 1.0e30f;
    if (any >= 0) {
        const float4* __restrict__ P = reinterpret_cast<const float4*>(g.xyz);
        // cell_centre's expressions
        const float px = g.origin[0] + ((float)ix + 0.5f) * g.cell;
        const float py = g.origin[1] + ((float)iy + 0.5f) * g.cell;
        const float pz = g.origin[2] + ((float)iz + 0.5f) * g.cell;
        if (best >= 0) {
            const float4 q = ld_pt(P, best);
            const float ex = px - q.x, ey = py - q.y, ez = pz - q.z;
            bd = ex * ex + ey * ey + ez * ez;
        }
        int last = -1;
#pragma unroll
        for (int k = 0; k < 27; ++k) {
            const int s = seed[k];
            if (k == 13 || s < 0 || s == best || s == last) continue;
            last = s;
            const float4 q = ld_pt(P, s);
            const float ex = px - q.x, ey = py - q.y, ez = pz - q.z;
            const float d2 = ex * ex + ey * ey + ez * ez;
            if (d2 < bd) {
                bd = d2;
                best = s;
            }
        }
    }
    out[c] = best;
    if (LAST) {
        const int v = best < 0 ? 255 : (int)(sqrtf(bd) * 100.0f + 0.5f);
        g.df[c] = (uint8_t)(v < 255 ? v : 255);
    }
}

template <class IDX>
static void jfa_step(const lw_prior_grid& g, const int32_t* in, int32_t* out, int step, bool last, unsigned tiles, int tx,
                     int ty, cudaStream_t s) {
    const dim3 cta(JFA_X, JFA_Y);
    if (step == 8)
        k_jfa<IDX, 8, false><<<tiles, cta, 0, s>>>(g, in, out, tx, ty);
    else if (step == 4)
        k_jfa<IDX, 4, false><<<tiles, cta, 0, s>>>(g, in, out, tx, ty);
    else if (step == 2)
        k_jfa<IDX, 2, false><<<tiles, cta, 0, s>>>(g, in, out, tx, ty);
    else if (!last)
        k_jfa<IDX, 1, false><<<tiles, cta, 0, s>>>(g, in, out, tx, ty);
    else
        k_jfa<IDX, 1, true><<<tiles, cta, 0, s>>>(g, in, out, tx, ty);
}

// start[c], the first point of cell c or of the next occupied cell after it, n beyond the last. A warp per run of ST_RUN
// cells: it finds the occupied cells that lie in its run by binary search, and each lane its own among those few (a warp per
// occupied cell filling the gap before it left the widest gaps to single warps: 0.2 ms on 11.5M cells).
constexpr int ST_RUN = 1024;

// The first j in [lo, hi) with cells[j] >= c, hi if none.
__device__ __forceinline__ int64_t first_cell(const int32_t* __restrict__ cells, int64_t lo, int64_t hi, int64_t c) {
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if ((int64_t)__ldg(cells + mid) < c)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

__global__ void k_starts(const int32_t* __restrict__ cells, const int32_t* __restrict__ first, int64_t u, int64_t n,
                         int64_t ncell, int32_t* __restrict__ start) {
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w * ST_RUN <= ncell; w += nwarps) {
        const int64_t c0 = w * ST_RUN, c1 = min(c0 + ST_RUN, ncell + 1);
        const int64_t j0 = first_cell(cells, 0, u, c0), j1 = first_cell(cells, j0, u, c1);
        for (int64_t c = c0 + lane; c < c1; c += 32) {
            const int64_t j = first_cell(cells, j0, j1, c);
            start[c] = j < u ? __ldg(first + j) : (int32_t)n;
        }
    }
}

// Distance of each point (posed by T) to the nearest map point, 1e3 beyond the band (mapgrid.py:173-194).
struct Pose12 {
    float m[12];
};

__global__ void k_distances(lw_prior_grid g, const float* __restrict__ pts, int64_t n, Pose12 T, float* __restrict__ out) {
    const float* M = T.m;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float wx, wy, wz;
        xform(M, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], wx, wy, wz);
        int s = nearest_point(g, wx, wy, wz);
        float d = 1.0e3f;
        if (s >= 0) {
            const float4 q = ld_pt(reinterpret_cast<const float4*>(g.xyz), s);
            d = len3(wx - q.x, wy - q.y, wz - q.z);
        }
        out[i] = d;
    }
}

// ---- batched point-to-plane ICP (localize.py:126-205, 517-565) --------------------------------------------

constexpr int LTERMS = 30;  // H 21, b 6, count, err, weight
constexpr float PLANAR = 0.5f;  // mapgrid.py:32

struct LocPose {
    float R[9], tr[3], c[3];
};

// Per-hypothesis float pose, re-centred on the hypothesis' translation (float32 keeps its precision). The poses
// change between iterations of the same launch, so they are read through L2 (__ldcg), never the L1 cache.
__device__ __forceinline__ void loc_pose(const double* T, LocPose& P) {
    for (int i = 0; i < 3; ++i) {
        for (int j = 0; j < 3; ++j) P.R[i * 3 + j] = (float)__ldcg(T + i * 4 + j);
        const double t = __ldcg(T + i * 4 + 3);
        P.c[i] = (float)t;
        P.tr[i] = (float)(t - (double)P.c[i]);
    }
}

// The hypothesis and point range of a tile, checked against the batch: h = -1 for a tile to skip.
__device__ __forceinline__ void tile_range(const lw_loc_batch& b, int tile, int n_hyp, int& h, int& lo, int& hi) {
    h = __ldg(b.tile_hyp + tile);
    lo = __ldg(b.tile_lo + tile);
    if (h < 0 || h >= n_hyp || lo < 0) {
        h = -1;
        lo = hi = 0;
        return;
    }
    hi = (int)min((int64_t)__ldg(b.scan_end + h), b.pts_cap);
}

// One (hypothesis, point) pair's terms (localize.py:144-167) added to a[k * S], k < LTERMS (S = 1: registers;
// S = 32: a warp's per-lane columns in shared memory).
// KNOWN: the point's nearest map point s was found before; else it is searched for here.
template <int S, bool KNOWN>
__device__ __forceinline__ void loc_terms(const lw_prior_grid& g, const LocPose& P, float4 p, int s, float max_d2,
                                          float c2, float alpha, float* a) {
    float lx = P.R[0] * p.x + P.R[1] * p.y + P.R[2] * p.z + P.tr[0];
    float ly = P.R[3] * p.x + P.R[4] * p.y + P.R[5] * p.z + P.tr[1];
    float lz = P.R[6] * p.x + P.R[7] * p.y + P.R[8] * p.z + P.tr[2];
    float wx = lx + P.c[0], wy = ly + P.c[1], wz = lz + P.c[2];
    if (!KNOWN) s = nearest_point(g, wx, wy, wz);
    if (s < 0 || (KNOWN && s >= g.n)) return;
    const float4 q = ld_pt(reinterpret_cast<const float4*>(g.xyz), s);
    float r0 = wx - q.x, r1 = wy - q.y, r2 = wz - q.z;
    if (r0 * r0 + r1 * r1 + r2 * r2 > max_d2) return;
    const float3 nv = make_float3(__ldg(g.nrm + 3 * (int64_t)s), __ldg(g.nrm + 3 * (int64_t)s + 1),
                                  __ldg(g.nrm + 3 * (int64_t)s + 2));
    float M[6];
    if (q.w > PLANAR && len3(nv.x, nv.y, nv.z) > 0.5f) {
        // the normal at full weight, along the surface only a little
        float b = 1.0f - alpha;
        M[0] = nv.x * nv.x * b + alpha;
        M[1] = nv.x * nv.y * b;
        M[2] = nv.x * nv.z * b;
        M[3] = nv.y * nv.y * b + alpha;
        M[4] = nv.y * nv.z * b;
        M[5] = nv.z * nv.z * b + alpha;
    } else {
        // an edge or clutter: a weak point-to-point pull
        M[0] = M[3] = M[5] = alpha * 4.0f;
        M[1] = M[2] = M[4] = 0.0f;
    }
    float Mr0 = fmaf(M[0], r0, fmaf(M[1], r1, M[2] * r2));
    float Mr1 = fmaf(M[1], r0, fmaf(M[3], r1, M[4] * r2));
    float Mr2 = fmaf(M[2], r0, fmaf(M[4], r1, M[5] * r2));
    float d2 = fmaf(r0, Mr0, fmaf(r1, Mr1, r2 * Mr2));
    float wgt = 1.0f / (1.0f + d2 / c2);
    wgt = wgt * wgt;  // Geman-McClure
    // J = [I | A] with A = -[l]x, so H = w [[M, M A], [A^T M, A^T M A]] and b = w [M r; A^T M r]
    // (the upper triangle in row-major order, the layout of accumulate(), odom.py:244-259)
    const float A[3][3] = {{0.f, lz, -ly}, {-lz, 0.f, lx}, {ly, -lx, 0.f}};
    const float Ms[3][3] = {{M[0], M[1], M[2]}, {M[1], M[3], M[4]}, {M[2], M[4], M[5]}};
    float MA[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int j = 0; j < 3; ++j) MA[r][j] = fmaf(Ms[r][0], A[0][j], fmaf(Ms[r][1], A[1][j], Ms[r][2] * A[2][j]));
    int idx = 0;
#pragma unroll
    for (int pp = 0; pp < 6; ++pp)
#pragma unroll
        for (int qq = pp; qq < 6; ++qq) {
            float h;
            if (qq < 3)
                h = Ms[pp][qq];
            else if (pp < 3)
                h = MA[pp][qq - 3];
            else
                h = fmaf(A[0][pp - 3], MA[0][qq - 3], fmaf(A[1][pp - 3], MA[1][qq - 3], A[2][pp - 3] * MA[2][qq - 3]));
            a[idx * S] = fmaf(wgt, h, a[idx * S]);
            ++idx;
        }
    a[21 * S] = fmaf(wgt, Mr0, a[21 * S]);
    a[22 * S] = fmaf(wgt, Mr1, a[22 * S]);
    a[23 * S] = fmaf(wgt, Mr2, a[23 * S]);
#pragma unroll
    for (int j = 0; j < 3; ++j)
        a[(24 + j) * S] = fmaf(wgt, fmaf(A[0][j], Mr0, fmaf(A[1][j], Mr1, A[2][j] * Mr2)), a[(24 + j) * S]);
    a[27 * S] += 1.0f;
    a[28 * S] = fmaf(wgt, d2, a[28 * S]);
    a[29 * S] += wgt;
}

// The float64 step of hypothesis h from its summed terms sv (localize.py:537-550) applied to its pose; returns
// the step's size max(|dt|, 5 |dr|), 0 when it is skipped. Kept out of line: it runs on one thread per
// hypothesis per iteration, and inlined its arrays would set the register budget of the whole kernel.
__device__ __noinline__ double loc_solve(const double* sv, double* Th, int min_count) {
    double moved = 0.0;
    if (sv[27] >= (double)min_count) {
        // re-centred sums -> the twist about the world origin: H = A^T Hc A, b = A^T bc
        double c[3] = {(double)(float)__ldcg(Th + 3), (double)(float)__ldcg(Th + 7),
                       (double)(float)__ldcg(Th + 11)};
        double Hc[36], H[36], bc[6], bw[6];
        int idx = 0;
        for (int p = 0; p < 6; ++p)
            for (int q = p; q < 6; ++q) {
                Hc[p * 6 + q] = Hc[q * 6 + p] = sv[idx];
                ++idx;
            }
        for (int p = 0; p < 6; ++p) bc[p] = sv[21 + p];
        const double K[9] = {0.0, c[2], -c[1], -c[2], 0.0, c[0], c[1], -c[0], 0.0};
        double HA[36];
        for (int p = 0; p < 6; ++p)
            for (int q = 0; q < 6; ++q) {
                double x = Hc[p * 6 + q];
                if (q >= 3)
                    for (int k = 0; k < 3; ++k) x += Hc[p * 6 + k] * K[k * 3 + q - 3];
                HA[p * 6 + q] = x;
            }
        for (int p = 0; p < 6; ++p) {
            for (int q = 0; q < 6; ++q) {
                double x = HA[p * 6 + q];
                if (p >= 3)
                    for (int k = 0; k < 3; ++k) x += K[k * 3 + p - 3] * HA[k * 6 + q];
                H[p * 6 + q] = x;
            }
            double x = bc[p];
            if (p >= 3)
                for (int k = 0; k < 3; ++k) x += K[k * 3 + p - 3] * bc[k];
            bw[p] = x;
        }
        // A = H + diag(1e-3 dg + 1e-9), delta = solve(A, -b)
        double Lf[36], rhs[6], delta[6];
        for (int p = 0; p < 6; ++p) {
            H[p * 7] += 1e-3 * H[p * 7] + 1e-9;
            rhs[p] = -bw[p];
        }
        bool ok = true;
        for (int j = 0; j < 6 && ok; ++j) {
            double d = H[j * 6 + j];
            for (int k = 0; k < j; ++k) d -= Lf[j * 6 + k] * Lf[j * 6 + k];
            if (!(d > 0.0)) {
                ok = false;
                break;
            }
            d = sqrt(d);
            Lf[j * 6 + j] = d;
            for (int r = j + 1; r < 6; ++r) {
                double x = H[r * 6 + j];
                for (int k = 0; k < j; ++k) x -= Lf[r * 6 + k] * Lf[j * 6 + k];
                Lf[r * 6 + j] = x / d;
            }
        }
        if (ok) {
            double y[6];
            for (int r = 0; r < 6; ++r) {
                double s = rhs[r];
                for (int k = 0; k < r; ++k) s -= Lf[r * 6 + k] * y[k];
                y[r] = s / Lf[r * 6 + r];
            }
            for (int r = 5; r >= 0; --r) {
                double s = y[r];
                for (int k = r + 1; k < 6; ++k) s -= Lf[k * 6 + r] * delta[k];
                delta[r] = s / Lf[r * 6 + r];
            }
            double T[16];
            for (int k = 0; k < 16; ++k) T[k] = __ldcg(Th + k);
            apply_twist(T, delta);
            for (int k = 0; k < 16; ++k) Th[k] = T[k];
            double nt = sqrt(delta[0] * delta[0] + delta[1] * delta[1] + delta[2] * delta[2]);
            double nr = sqrt(delta[3] * delta[3] + delta[4] * delta[4] + delta[5] * delta[5]);
            moved = fmax(nt, 5.0 * nr);
        }
    }
    return moved;
}

struct LocArgs {
    int n_hyp, n_tiles, n_stages;  // counts, or capacities when b.dims is set
    int tile;                      // points per warp tile
    float max_d2[8], c2[8];
    int iters[8];
    float alpha;
    float radii[3];
    int min_count;  // a hypothesis with fewer matched points skips its update (localize.py:538)
};

constexpr int LOC_BLOCK = 256;
constexpr unsigned FULL = 0xffffffffu;

// Reduce-scatter over a warp: afterwards lane j holds the sum over the 32 lanes of v[j]. Each of the five steps
// hands half of the remaining slots to the partner lane (31 shuffles in all, against 5 per slot for 32 butterfly
// reductions).
__device__ __forceinline__ float warp_reduce_scatter32(float (&v)[32], int lane) {
#pragma unroll
    for (int half = 16; half >= 1; half >>= 1) {
        const bool up = (lane & half) != 0;
#pragma unroll
        for (int k = 0; k < half; ++k) {
            const float send = up ? v[k] : v[k + half];
            const float keep = up ? v[k + half] : v[k];
            v[k] = keep + __shfl_xor_sync(FULL, send, half);
        }
    }
    return v[0];
}

// The tiles of pass `pass` for the calling warp, taken `grab` at a time (one atomic, broadcast to the warp). A tile per atomic
// made the atomics on the one counter, about 3 ns each, take as long as the searches themselves: 0.26 ms for 88,000
// tiles. A grab is a quarter of a warp's share, and the last quarter of the tiles goes out singly, so that no warp is a
// whole grab behind at the barrier: 256 scans 13.4 -> 12.9 ms (singles for the last tenth 13.2, five eighths 13.0, pairs
// 13.2).
struct TileTaker {
    int t = 0, left = 0;
    __device__ __forceinline__ int next(const lw_loc_batch& b, int pass, int lane, int grab, int n_tiles) {
        if (left == 0) {
            int v = 0;
            if (lane == 0) v = atomicAdd(b.next + pass, 1);
            v = __shfl_sync(FULL, v, 0);
            const int big = (int)((int64_t)n_tiles * 3 / 4) / grab;
            t = v < big ? v * grab : big * grab + (v - big);
            left = v < big ? grab : 1;
        }
        --left;
        return t++;
    }
};

// A hypothesis' scan points, a CTA each, gathered into 25 cm boxes of the sensor frame in Morton order (32 boxes per axis,
// wrapping) by a counting sort: ws.sorted holds (x, y, z, place in the scan) in slots hyp_tile[h] * tile on, and
// ws.match is set to "unknown". Only neighbourhood matters: the order within a box is whatever the atomics give.
constexpr int LS_BITS = 5, LS_BOXES = 1 << (3 * LS_BITS), LS_T = 1024;

__device__ __forceinline__ unsigned spread5(unsigned v) {  // bits 0..4 to every third
    v = (v | (v << 8)) & 0x100Fu;
    v = (v | (v << 4)) & 0x10C3u;
    return (v | (v << 2)) & 0x1249u;
}

__global__ void __launch_bounds__(LS_T) k_loc_sort(lw_loc_batch b, lw_loc_ws ws, int n_hyp_ub, int n_tiles_ub, int tile) {
    extern __shared__ int box[];  // [LS_BOXES]
    __shared__ int sm[33];
    const int n_hyp = b.dims ? min(__ldg(b.dims), n_hyp_ub) : n_hyp_ub;
    const int n_tiles = b.dims ? min(__ldg(b.dims + 1), n_tiles_ub) : n_tiles_ub;
    if ((int64_t)n_tiles * tile > ws.cap) return;
    for (int h = blockIdx.x; h < n_hyp; h += gridDim.x) {
        const int t0 = max(b.hyp_tile[h], 0), t1 = min(b.hyp_tile[h + 1], n_tiles);
        if (t0 >= t1) continue;
        const int lo = b.tile_lo[t0];
        if (lo < 0) continue;
        const int hi = (int)min((int64_t)b.scan_end[h], b.pts_cap);
        const int n = min(hi - lo, (t1 - t0) * tile);
        if (n <= 0) continue;
        auto box_of = [&](float4 p) {
            const unsigned x = (unsigned)ifloor(p.x * 4.0f) & 31u, y = (unsigned)ifloor(p.y * 4.0f) & 31u,
                           z = (unsigned)ifloor(p.z * 4.0f) & 31u;
            return (int)(spread5(x) | (spread5(y) << 1) | (spread5(z) << 2));
        };
        __syncthreads();
        for (int k = threadIdx.x; k < LS_BOXES; k += LS_T) box[k] = 0;
        __syncthreads();
        const float4* pts = reinterpret_cast<const float4*>(b.pts) + lo;
        for (int i = threadIdx.x; i < n; i += LS_T) atomicAdd(&box[box_of(__ldg(pts + i))], 1);
        __syncthreads();
        // exclusive scan of the boxes, LS_BOXES / LS_T consecutive ones per thread
        constexpr int PER = LS_BOXES / LS_T;
        int sum = 0;
        for (int k = 0; k < PER; ++k) sum += box[threadIdx.x * PER + k];
        int tot;
        int at = block_excl(sum, sm, &tot);
        for (int k = 0; k < PER; ++k) {
            const int c = box[threadIdx.x * PER + k];
            box[threadIdx.x * PER + k] = at;
            at += c;
        }
        __syncthreads();
        float4* out = reinterpret_cast<float4*>(ws.sorted) + (int64_t)t0 * tile;
        int32_t* match = ws.match + (int64_t)t0 * tile;
        for (int i = threadIdx.x; i < n; i += LS_T) {
            const float4 p = __ldg(pts + i);
            out[atomicAdd(&box[box_of(p)], 1)] = make_float4(p.x, p.y, p.z, __int_as_float(i));
            match[i] = -1;
        }
    }
}

// MINB: CTAs of LOC_BLOCK threads the register budget must let reside per SM. With 2 or 3 the per-lane term
// sums of a tile and the tile's pose live in registers; with 4 to 6 they live in shared memory (a [30][32]
// column block and one pose per warp, 31 KB per CTA), which frees ~47 registers across the nearest-point search
// so that two to three times the 2-CTA warp count stays resident.
//
// With a workspace (ws) each iteration first finds every point's nearest map point, in an order in which a warp's 32 points
// are neighbours (k_loc_sort) -- scans come in the order they were fired, whose 32 points lie in as many places: a
// quarter of the loads hit L1 and half the lanes idled -- starting from the point's match of the iteration before; the
// terms are then summed from the matches in the scan's own order, so that every sum and pose is the one without a workspace,
// bit for bit. 256 scans of 2,000-20,000 points, 31 iterations: 12.8 ms, 23.1 without; an iteration is 0.19-0.35 ms of searches
// (bound by L1's one line a cycle: every lane's loads are lines of their own, about 570 a tile), 0.08 of sums, 0.03 of
// the tile partials' sums and solves, 0.08 of waiting at the three barriers. The sorted points are read past L1, which
// the map's lines need.
// WS: a workspace was handed in (whether a batch's tiles fit it is known on the device alone). Without one, as in an
// evaluation, the kernel is compiled without the sorted ways, whose registers and shared memory are in its way: 20,000 points
// at 8 poses 487 us with them, 474 without.
template <int MINB, bool WS>
__global__ void __launch_bounds__(LOC_BLOCK, MINB)
    k_loc_icp(lw_prior_grid g, lw_loc_batch b, lw_loc_ws ws, LocArgs la) {
    constexpr bool SMEM_ACC = MINB >= 4;
    __shared__ __align__(16) float s_acc[SMEM_ACC ? LOC_BLOCK / 32 : 1][SMEM_ACC ? LTERMS : 1][32];
    __shared__ LocPose s_pose[SMEM_ACC ? LOC_BLOCK / 32 : 1];
    __shared__ int2 s_runs[SMEM_ACC || !WS ? 1 : LOC_BLOCK / 32][WS ? 9 : 1][32];
    __shared__ double sv[32];
    __shared__ int s_stop;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int n_hyp = b.dims ? min(__ldg(b.dims), la.n_hyp) : la.n_hyp;
    const int n_tiles = b.dims ? min(__ldg(b.dims + 1), la.n_tiles) : la.n_tiles;
    const bool sorted = WS && (int64_t)n_tiles * la.tile <= ws.cap;
    // a search's runs: in the term sums' columns, which are free while searching
    int2(*runs)[32] = SMEM_ACC ? reinterpret_cast<int2(*)[32]>(&s_acc[tid >> 5][0][0]) : s_runs[SMEM_ACC || !WS ? 0 : tid >> 5];
    static_assert(sizeof(int2) * 9 * 32 <= sizeof(float) * LTERMS * 32, "a search's runs fit the term sums' columns");
    const int warp_id = (blockIdx.x * LOC_BLOCK + tid) >> 5, n_warps = gridDim.x * (LOC_BLOCK / 32);
    const int grab = max(1, min(8, n_tiles / (4 * n_warps)));
    int it_total = 0;
    for (int stage = 0; stage < la.n_stages; ++stage) {
        const float max_d2 = la.max_d2[stage];
        const float c2 = la.c2[stage];
        for (int it = 0; it < la.iters[stage]; ++it, ++it_total) {
            // phase A: warp tiles, handed out in order of arrival, -> float64 tile partials. A tile's partial
            // does not depend on which warp computed it, so the sums of phase B are deterministic.
            if (sorted) {
                for (TileTaker take;;) {
                    const int tile = take.next(b, it_total, lane, grab, n_tiles);
                    if (tile >= n_tiles) break;
                    int h, lo, hi;
                    tile_range(b, tile, n_hyp, h, lo, hi);
                    if (h < 0) continue;
                    LocPose Pr;
                    LocPose& P = SMEM_ACC ? s_pose[tid >> 5] : Pr;
                    if (!SMEM_ACC || lane == 0) loc_pose(b.T + 16 * h, P);
                    __syncwarp();
                    const int64_t slot0 = (int64_t)tile * la.tile;
                    int32_t* match = ws.match + (int64_t)max(__ldg(b.hyp_tile + h), 0) * la.tile;
                    const int count = min(hi - lo, la.tile);
                    for (int i = lane; i < count; i += 32) {
                        const float4 p = __ldcs(reinterpret_cast<const float4*>(ws.sorted) + slot0 + i);
                        const int place = __float_as_int(p.w);
                        if (place < 0 || (match - ws.match) + place >= ws.cap) continue;  // tables that do not fit together
                        int32_t* m = match + place;
                        const float lx = P.R[0] * p.x + P.R[1] * p.y + P.R[2] * p.z + P.tr[0];
                        const float ly = P.R[3] * p.x + P.R[4] * p.y + P.R[5] * p.z + P.tr[1];
                        const float lz = P.R[6] * p.x + P.R[7] * p.y + P.R[8] * p.z + P.tr[2];
                        __stcg(m, nearest_warm(g, lx + P.c[0], ly + P.c[1], lz + P.c[2], __ldcg(m), runs));
                    }
                    __syncwarp();  // the pose slot is rewritten by the warp's next tile
                }
                if (!grid_barrier(b.bar, b.err, 3)) return;
            }
            TileTaker take;
            for (int turn = warp_id;; turn += n_warps) {
                // the sums alone are even work: tiles in turn; with the searches in them tiles go to the next free warp
                const int tile = sorted ? turn : take.next(b, it_total, lane, grab, n_tiles);
                if (tile >= n_tiles) break;
                int h, lo, hi;
                tile_range(b, tile, n_hyp, h, lo, hi);
                float v[32];
#pragma unroll
                for (int k = 0; k < 32; ++k) v[k] = 0.0f;
                if (h >= 0) {
                    // the tile's pose is the same for the whole warp: with SMEM_ACC it is kept in shared memory
                    // (broadcast reads) instead of 15 registers per lane
                    LocPose Pr;
                    LocPose& P = SMEM_ACC ? s_pose[tid >> 5] : Pr;
                    if (!SMEM_ACC || lane == 0) loc_pose(b.T + 16 * h, P);
                    __syncwarp();
                    const int end = min(hi, lo + la.tile);
                    if constexpr (SMEM_ACC) {
                        float* col = &s_acc[tid >> 5][0][lane];
#pragma unroll
                        for (int k = 0; k < LTERMS; ++k) col[k * 32] = 0.0f;
                        if (sorted)
                            for (int i = lo + lane; i < end; i += 32)
                                loc_terms<32, true>(g, P, __ldg(reinterpret_cast<const float4*>(b.pts) + i),
                                                    __ldcg(ws.match + (int64_t)tile * la.tile + (i - lo)), max_d2, c2,
                                                    la.alpha, col);
                        else
                            for (int i = lo + lane; i < end; i += 32)
                                loc_terms<32, false>(g, P, __ldg(reinterpret_cast<const float4*>(b.pts) + i), -1, max_d2,
                                                     c2, la.alpha, col);
#pragma unroll
                        for (int k = 0; k < LTERMS; ++k) v[k] = col[k * 32];
                        __syncwarp();  // the pose slot is rewritten by the warp's next tile
                    } else {
                        if (sorted)
                            for (int i = lo + lane; i < end; i += 32)
                                loc_terms<1, true>(g, P, __ldg(reinterpret_cast<const float4*>(b.pts) + i),
                                                   __ldcg(ws.match + (int64_t)tile * la.tile + (i - lo)), max_d2, c2,
                                                   la.alpha, v);
                        else
                            for (int i = lo + lane; i < end; i += 32)
                                loc_terms<1, false>(g, P, __ldg(reinterpret_cast<const float4*>(b.pts) + i), -1, max_d2,
                                                    c2, la.alpha, v);
                    }
                }
                const float sum = warp_reduce_scatter32(v, lane);
                if (lane < LTERMS) b.tile_part[(int64_t)tile * 32 + lane] = (double)sum;
            }
            if (!grid_barrier(b.bar, b.err, 1)) return;
            // phase B: per hypothesis, sum its tiles in order and solve (localize.py:537-550)
            for (int h = blockIdx.x; h < n_hyp; h += gridDim.x) {
                const int t0 = max(b.hyp_tile[h], 0), t1 = min(b.hyp_tile[h + 1], n_tiles);
                if (tid < LTERMS) {
                    double s = 0.0;
                    // in tile order, 32 loads in flight (a scan has hundreds of tiles)
                    int t = t0;
                    for (; t + 32 <= t1; t += 32) {
                        double v[32];
#pragma unroll
                        for (int u = 0; u < 32; ++u) v[u] = __ldcg(b.tile_part + (int64_t)(t + u) * 32 + tid);
#pragma unroll
                        for (int u = 0; u < 32; ++u) s += v[u];
                    }
                    for (; t < t1; ++t) s += __ldcg(b.tile_part + (int64_t)t * 32 + tid);
                    sv[tid] = s;
                }
                __syncthreads();
                if (tid == 0) {
                    b.count[h] = (int)sv[27];
                    const double moved = loc_solve(sv, b.T + 16 * h, la.min_count);
                    // the largest step of the iteration, as ordered bits of a non-negative float
                    atomicMax(b.moved + it_total, __float_as_int((float)moved));
                }
                __syncthreads();
            }
            if (!grid_barrier(b.bar, b.err, 2)) return;
            if (tid == 0) s_stop = __int_as_float(__ldcg(b.moved + it_total)) < 2e-4f ? 1 : 0;
            __syncthreads();
            if (s_stop) {
                ++it_total;
                break;
            }
        }
    }
    // evaluation (localize.py:182-205): points within each radius of their nearest map point, per hypothesis
    for (TileTaker take;;) {
        const int tile = take.next(b, it_total, lane, grab, n_tiles);
        if (tile >= n_tiles) break;
        int h, lo, hi;
        tile_range(b, tile, n_hyp, h, lo, hi);
        if (h < 0) continue;
        float M[12];
        for (int k = 0; k < 12; ++k) M[k] = (float)__ldcg(b.T + 16 * h + k);
        int c0 = 0, c1 = 0, c2 = 0;
        const int end = min(hi, lo + la.tile);
        const int64_t slot0 = (int64_t)tile * la.tile;
        const int32_t* match = sorted ? ws.match + (int64_t)max(__ldg(b.hyp_tile + h), 0) * la.tile : nullptr;
        for (int i = lo + lane; i < end; i += 32) {
            float4 p = __ldg(sorted ? reinterpret_cast<const float4*>(ws.sorted) + slot0 + (i - lo)
                                    : reinterpret_cast<const float4*>(b.pts) + i);
            float wx, wy, wz;
            xform(M, p.x, p.y, p.z, wx, wy, wz);
            const int place = sorted ? __float_as_int(p.w) : -1;
            const bool known = place >= 0 && (match - ws.match) + place < ws.cap;
            int s = sorted ? nearest_warm(g, wx, wy, wz, known ? __ldcg(match + place) : -1, runs) : nearest_point(g, wx, wy, wz);
            if (s >= 0) {
                const float4 q = ld_pt(reinterpret_cast<const float4*>(g.xyz), s);
                float d = len3(wx - q.x, wy - q.y, wz - q.z);
                c0 += d < la.radii[0];
                c1 += d < la.radii[1];
                c2 += d < la.radii[2];
            }
        }
        c0 = __reduce_add_sync(FULL, c0);
        c1 = __reduce_add_sync(FULL, c1);
        c2 = __reduce_add_sync(FULL, c2);
        if (lane == 0) {
            atomicAdd(b.eval + 3 * h + 0, c0);
            atomicAdd(b.eval + 3 * h + 1, c1);
            atomicAdd(b.eval + 3 * h + 2, c2);
        }
    }
    if (blockIdx.x == 0 && tid == 0) *b.iters_run = it_total;
}

// Clears what the launch accumulates into. The barrier's arrival count is zeroed too: a launch that gave up at a
// barrier may have left it part counted (its generation word needs no reset).
__global__ void k_loc_reset(lw_loc_batch b, int n_hyp, int max_iters) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < max_iters; i += gridDim.x * blockDim.x) b.moved[i] = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= max_iters; i += gridDim.x * blockDim.x) b.next[i] = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 3 * n_hyp; i += gridDim.x * blockDim.x) b.eval[i] = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *b.err = 0;
        b.bar[0] = 0u;
    }
}

}  // namespace lw

using namespace lw;

namespace lw {

// ---- coarse hypothesis scores (localize.py:55-123, k_score_grid / k_score_list) -----------------------------
// A thread per hypothesis, the scan points staged in shared memory in chunks (every thread reads the same point at
// once). The soft count sum over points with d < tau of (1 - d^2 / tau^2) is kept as two integers -- the number of
// such points and the sum of d^2 (d is a whole number of cm) -- and formed once at the end in float64: exact and
// independent of the summation order, where the reference adds float32 terms in point order (the two differ by
// that sum's rounding only). Headings' cosine and sine come from the host (YawTab) so that every implementation
// poses the points with the same float32 values.
constexpr int SC_THREADS = 256;
constexpr int SC_CHUNK = 1024;

struct YawTab {
    float c[LW_SCORE_MAX_YAW], s[LW_SCORE_MAX_YAW];
};

__device__ __forceinline__ void score_chunk(const lw_prior_grid& g, const float* __restrict__ px,
                                            const float* __restrict__ py, const float* __restrict__ pz, int m,
                                            float cx, float cy, float cz, float co, float si, float tau, int& n_in,
                                            int& sum_d2) {
    const uint8_t* __restrict__ df = g.df;
#pragma unroll 4
    for (int k = 0; k < m; ++k) {
        const float wx = cx + co * px[k] - si * py[k];
        const float wy = cy + si * px[k] + co * py[k];
        const float wz = cz + pz[k];
        int ix, iy, iz;
        grid_idx(g, wx, wy, wz, ix, iy, iz);
        const int64_t j = grid_flat(g, ix, iy, iz);
        if (j >= 0) {
            const int d = __ldg(df + j);
            if ((float)d < tau) {
                ++n_in;
                sum_d2 += d * d;
            }
        }
    }
}

__device__ __forceinline__ void stage_pts(const float* __restrict__ pts, int base, int m, float* px, float* py,
                                          float* pz) {
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
        px[k] = pts[3 * (int64_t)(base + k) + 0];
        py[k] = pts[3 * (int64_t)(base + k) + 1];
        pz[k] = pts[3 * (int64_t)(base + k) + 2];
    }
}

__device__ __forceinline__ float soft_count(int n_in, int sum_d2, float tau) {
    return (float)((double)n_in - (double)sum_d2 / ((double)tau * (double)tau));
}

// Thread layout: each thread takes SC_POS consecutive rows of one column, positions ip = c + stride * r with
// r = SC_POS (32 rg + lane) + j, j < SC_POS, at one heading; the warps of a CTA take consecutive headings. When
// positions ip and ip + stride are neighbours along x with the same y and z (stride = ny for a meshgrid with y
// inner), a warp's posed copies of a point differ only in x -- one row of the x-fastest distance field, a few
// cache lines per gather. Each hypothesis' score is the same whatever the layout.
//
// The kernel is bound by the instructions it issues, so what a warp's positions share is worked out once: a warp's
// positions lie in few (y, z) rows (one or two where the x runs are long), and for each row and each of 16 points one lane
// computes the rotated offsets, the posed y and z, their cells and the row's address, into shared memory. What is left
// per position and point is the x chain, two positions to a packed instruction, with the floor taken by one addition that
// rounds down (sc_cell) instead of a quarter-rate conversion. Rows outside the grid and dead positions get an x far outside
// it and need no test of their own. 3.5M hypotheses x 1024 points of an office: 4.87 -> 2.27 ms, at 84% of the issue slots.
// A warp whose positions are spread over many rows (list order along y) gains nothing from the table: its hypotheses are
// left to k_score_rest, and so are all of them when a point is not finite. Four CTAs an SM and eight points in flight:
// five CTAs take 2.33 ms; positions 32 apart in a thread, 2.4; branches around the gathers, 4.0.
constexpr int SC_POS = 2;
constexpr int SC_ROWS = 8;        // (y, z) rows a warp keeps
constexpr int SC_TAB = 16;        // points per table
constexpr float SC_FAR = 1.0e30f; // an x outside every grid
constexpr float SC_HUGE = 1.0e18f;
constexpr int SC_MAX_NX = 1 << 22;
constexpr float SC_PENDING = -3.0e38f;  // no score: scores are -1 or more

struct ScoreRow {
    float ax, bx;        // the rotated offset's two x terms
    const uint8_t* row;  // the distance field's row
};

__device__ __forceinline__ uint64_t f2_pack(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_add_down(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// The cells of two posed x's: floor(f) for f in [-2^22, 2^22), because f + 1.5 x 2^23 rounded down is floor(f) + 1.5 x 2^23
// there; for any other f, infinities included, a number of 2^22 or more.
__device__ __forceinline__ uint2 sc_cell(uint64_t wx, uint64_t neg_origin, uint64_t inv_cell) {
    const uint64_t f = f2_mul(f2_add(wx, neg_origin), inv_cell);
    const uint64_t t = f2_add_down(f, f2_pack(RINT_MAGIC, RINT_MAGIC));
    uint2 u;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(u.x), "=r"(u.y) : "l"(t));
    return make_uint2(u.x - (uint32_t)RINT_BITS, u.y - (uint32_t)RINT_BITS);
}

// SC_TAB points against a thread's two positions. SAME: both lie in the row e0.
template <bool SAME>
__device__ __forceinline__ void score_rows(const ScoreRow* e0, const ScoreRow* e1, int m, uint64_t cx, uint64_t neg_origin,
                                           uint64_t inv_cell, uint32_t nx, int tau_ceil, int (&n_in)[SC_POS],
                                           int (&sum_d2)[SC_POS]) {
#pragma unroll 8
    for (int k = 0; k < m; ++k) {
        const float4 v0 = *reinterpret_cast<const float4*>(e0 + k);
        const float4 v1 = SAME ? v0 : *reinterpret_cast<const float4*>(e1 + k);
        const uint64_t wx = f2_add(f2_add(cx, f2_pack(v0.x, v1.x)), f2_pack(v0.y, v1.y));
        const uint2 u = sc_cell(wx, neg_origin, inv_cell);
        const uint64_t r0 = f2_pack(v0.z, v0.w), r1 = SAME ? r0 : f2_pack(v1.z, v1.w);
        int d0 = 1024, d1 = 1024;
        if (u.x < nx) d0 = __ldg(reinterpret_cast<const uint8_t*>(r0) + u.x);
        if (u.y < nx) d1 = __ldg(reinterpret_cast<const uint8_t*>(r1) + u.y);
        if (d0 < tau_ceil) {  // d < tau for a whole number of cm
            ++n_in[0];
            sum_d2[0] += d0 * d0;
        }
        if (d1 < tau_ceil) {
            ++n_in[1];
            sum_d2[1] += d1 * d1;
        }
    }
}

__global__ void __launch_bounds__(SC_THREADS, 4) k_score_grid(const __grid_constant__ lw_prior_grid g,
                                                           const float* __restrict__ pts, int n_pts,
                                                           const float* __restrict__ pos, int64_t n_pos,
                                                           int64_t stride, int64_t n_rg, int n_yaw,
                                                           const YawTab yt, float tau, int tau_ceil, float free_cm,
                                                           float* __restrict__ out) {
    static_assert(SC_POS == 2, "a thread's positions are one pair");
    __shared__ float px[SC_CHUNK], py[SC_CHUNK], pz[SC_CHUNK];
    __shared__ __align__(16) ScoreRow tab[SC_THREADS / 32][SC_ROWS][SC_TAB + 1];  // + 1: rows start in different banks
    const unsigned full = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int iyaw = (int)(wid % n_yaw);
    const int64_t q = wid / n_yaw;
    const int64_t c = q / n_rg, r0 = ((q - c * n_rg) * 32 + lane) * SC_POS;
    const float co = yt.c[iyaw], si = yt.s[iyaw];
    float cx[SC_POS], cy[SC_POS], cz[SC_POS];
    bool live[SC_POS];
    int row[SC_POS];
#pragma unroll
    for (int j = 0; j < SC_POS; ++j) {
        const int64_t ip = c + stride * (r0 + j);
        live[j] = c < stride && ip < n_pos;
        row[j] = -1;
        cx[j] = SC_FAR;
        cy[j] = cz[j] = 0.f;
        if (live[j]) {
            const float x = pos[3 * ip], y = pos[3 * ip + 1], z = pos[3 * ip + 2];
            int ix, iy, iz;
            grid_idx(g, x, y, z, ix, iy, iz);
            const int64_t cc = grid_flat(g, ix, iy, iz);
            // the sensor outside the grid or inside a mapped surface
            if (cc < 0 || (float)g.df[cc] < free_cm) {
                out[ip * n_yaw + iyaw] = -1.0f;
                live[j] = false;
            } else {
                cx[j] = x;
                cy[j] = y;
                cz[j] = z;
            }
        }
    }
    // the warp's distinct (y, z), lane k keeping row k's
    float ty = 0.f, tz = 0.f;
    int rows = 0;
    const bool plain = g.nx <= SC_MAX_NX;
    for (; rows < SC_ROWS && plain; ++rows) {
        bool open[SC_POS];
#pragma unroll
        for (int j = 0; j < SC_POS; ++j)
            open[j] = live[j] && row[j] < 0 && fabsf(cx[j]) < SC_HUGE && fabsf(cy[j]) < SC_HUGE && fabsf(cz[j]) < SC_HUGE;
        const unsigned w = __ballot_sync(full, open[0] || open[1]);
        if (w == 0) break;
        const int from = __ffs(w) - 1;
        const float y = __shfl_sync(full, open[0] ? cy[0] : cy[1], from);
        const float z = __shfl_sync(full, open[0] ? cz[0] : cz[1], from);
#pragma unroll
        for (int j = 0; j < SC_POS; ++j)
            if (open[j] && cy[j] == y && cz[j] == z) row[j] = rows;
        if (lane == rows) {
            ty = y;
            tz = z;
        }
    }
    // positions left over, one not finite, or rows of fewer than eight positions: k_score_rest
    const int positions = __popc(__ballot_sync(full, live[0])) + __popc(__ballot_sync(full, live[1]));
    bool fits = __all_sync(full, (!live[0] || row[0] >= 0) && (!live[1] || row[1] >= 0)) &&
                (rows <= 2 || 8 * rows <= positions);
    const bool any0 = row[0] >= 0, any1 = row[1] >= 0;
    const bool same = __all_sync(full, row[0] == row[1] || !any0 || !any1);
    const int s0 = any0 ? row[0] : (any1 ? row[1] : 0), s1 = any1 ? row[1] : s0;
    const uint64_t cx2 = f2_pack(any0 ? cx[0] : SC_FAR, any1 ? cx[1] : SC_FAR);
    const uint64_t neg_origin = f2_pack(-g.origin[0], -g.origin[0]), inv_cell = f2_pack(g.inv_cell, g.inv_cell);
    int n_in[SC_POS], sum_d2[SC_POS];
#pragma unroll
    for (int j = 0; j < SC_POS; ++j) n_in[j] = sum_d2[j] = 0;
    for (int base = 0; base < n_pts; base += SC_CHUNK) {
        const int m = min(SC_CHUNK, n_pts - base);
        __syncthreads();
        stage_pts(pts, base, m, px, py, pz);
        bool odd = false;
        for (int k = threadIdx.x; k < m; k += blockDim.x)
            odd |= !(fabsf(px[k]) < SC_HUGE && fabsf(py[k]) < SC_HUGE && fabsf(pz[k]) < SC_HUGE);
        if (__syncthreads_or(odd)) {
            fits = false;
            break;
        }
        if (fits) {
            for (int k0 = 0; k0 < m && rows > 0; k0 += SC_TAB) {
                const int n = min(SC_TAB, m - k0);
                __syncwarp();
                for (int r = 0; r < rows; r += 2) {  // 16 points of two rows at a time
                    const int mine = r + (lane >> 4), k = lane & (SC_TAB - 1);
                    const float y = __shfl_sync(full, ty, mine & 31), z = __shfl_sync(full, tz, mine & 31);
                    if (mine < rows && k < n) {
                        // the reference's expressions (localize.py:89)
                        const float x0 = px[k0 + k], y0 = py[k0 + k];
                        const float wy = y + si * x0 + co * y0, wz = z + pz[k0 + k];
                        const int iy = ifloor((wy - g.origin[1]) * g.inv_cell);
                        const int iz = ifloor((wz - g.origin[2]) * g.inv_cell);
                        const bool in = iy >= 0 && iz >= 0 && iy < g.ny && iz < g.nz;
                        ScoreRow e;
                        e.ax = in ? co * x0 : SC_FAR;
                        e.bx = -(si * y0);
                        e.row = g.df + (in ? ((int64_t)iz * g.ny + iy) * (int64_t)g.nx : 0);
                        tab[warp][mine][k] = e;
                    }
                }
                __syncwarp();
                if (same)
                    score_rows<true>(tab[warp][s0], tab[warp][s0], n, cx2, neg_origin, inv_cell, (uint32_t)g.nx, tau_ceil,
                                     n_in, sum_d2);
                else
                    score_rows<false>(tab[warp][s0], tab[warp][s1], n, cx2, neg_origin, inv_cell, (uint32_t)g.nx, tau_ceil,
                                      n_in, sum_d2);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < SC_POS; ++j)
        if (live[j]) out[(c + stride * (r0 + j)) * n_yaw + iyaw] = fits ? soft_count(n_in[j], sum_d2[j], tau) : SC_PENDING;
}

// The hypotheses k_score_grid left pending, in the same layout, each thread working out its own row or two: six CTAs an SM
// of it hide the gathers better than a second way through k_score_grid would (1.00 against 1.34 ms for 0.6M hypotheses x
// 1024 points in list order).
template <bool WIDE>
__global__ void __launch_bounds__(SC_THREADS, 6) k_score_rest(lw_prior_grid g, const float* __restrict__ pts, int n_pts,
                                                           const float* __restrict__ pos, int64_t n_pos,
                                                           int64_t stride, int64_t n_rg, int n_yaw,
                                                           const YawTab yt, float tau, int tau_ceil,
                                                           float* __restrict__ out) {
    using idx_t = typename std::conditional<WIDE, int64_t, int32_t>::type;
    __shared__ float px[SC_CHUNK], py[SC_CHUNK], pz[SC_CHUNK];
    const int lane = threadIdx.x & 31;
    const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int iyaw = (int)(wid % n_yaw);
    const int64_t q = wid / n_yaw;
    const int64_t c = q / n_rg, r0 = ((q - c * n_rg) * 32 + lane) * SC_POS;
    const float co = yt.c[iyaw], si = yt.s[iyaw];
    float cx[SC_POS];
    bool live[SC_POS], in_b[SC_POS];
    float ya = 0.f, za = 0.f, yb = 0.f, zb = 0.f;
    int rows = 0;  // distinct (y, z) among the live positions
#pragma unroll
    for (int j = 0; j < SC_POS; ++j) {
        const int64_t ip = c + stride * (r0 + j);
        live[j] = c < stride && ip < n_pos && out[ip * n_yaw + iyaw] == SC_PENDING;
        in_b[j] = false;
        cx[j] = 0.f;
        if (live[j]) {
            const float x = pos[3 * ip], y = pos[3 * ip + 1], z = pos[3 * ip + 2];
            cx[j] = x;
            if (rows == 0) {
                ya = y;
                za = z;
                rows = 1;
            } else if (y != ya || z != za) {
                yb = y;
                zb = z;
                rows = 2;
                in_b[j] = y == yb && z == zb;
            }
        }
    }
    if (!__syncthreads_or(rows > 0)) return;
    int n_in[SC_POS], sum_d2[SC_POS];
#pragma unroll
    for (int j = 0; j < SC_POS; ++j) n_in[j] = sum_d2[j] = 0;
    const uint8_t* __restrict__ df = g.df;
    for (int base = 0; base < n_pts; base += SC_CHUNK) {
        const int m = min(SC_CHUNK, n_pts - base);
        __syncthreads();
        stage_pts(pts, base, m, px, py, pz);
        __syncthreads();
        if (rows == 0) continue;
#pragma unroll 2
        for (int k = 0; k < m; ++k) {
            // the reference's expressions (localize.py:89), the shared parts once per row
            const float ax = co * px[k], bx = si * py[k], ey = si * px[k], fy = co * py[k];
            const float wya = ya + ey + fy, wza = za + pz[k];
            const int iya = ifloor((wya - g.origin[1]) * g.inv_cell), iza = ifloor((wza - g.origin[2]) * g.inv_cell);
            const bool oka = iya >= 0 && iza >= 0 && iya < g.ny && iza < g.nz;
            const idx_t rowa = ((idx_t)iza * g.ny + iya) * (idx_t)g.nx;
            idx_t rowb = 0;
            bool okb = false;
            if (rows == 2) {
                const float wyb = yb + ey + fy, wzb = zb + pz[k];
                const int iyb = ifloor((wyb - g.origin[1]) * g.inv_cell), izb = ifloor((wzb - g.origin[2]) * g.inv_cell);
                okb = iyb >= 0 && izb >= 0 && iyb < g.ny && izb < g.nz;
                rowb = ((idx_t)izb * g.ny + iyb) * (idx_t)g.nx;
            }
#pragma unroll
            for (int j = 0; j < SC_POS; ++j) {
                const float wx = cx[j] + ax - bx;
                const int ix = ifloor((wx - g.origin[0]) * g.inv_cell);
                const bool ok = in_b[j] ? okb : oka;
                if (live[j] && ok && ix >= 0 && ix < g.nx) {
                    const int d = __ldg(df + (in_b[j] ? rowb : rowa) + ix);
                    if (d < tau_ceil) {  // d < tau for a whole number of cm
                        ++n_in[j];
                        sum_d2[j] += d * d;
                    }
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < SC_POS; ++j)
        if (live[j]) out[(c + stride * (r0 + j)) * n_yaw + iyaw] = soft_count(n_in[j], sum_d2[j], tau);
}


// Local maxima of the coarse scores (localize.py:450-483, _local_maxima): hypothesis h = ((iz nx + ix) ny + iy)
// n_yaw + iyaw is one when its score is positive, at least min_score, and no less than any of its 26 neighbours in
// (x, y, heading) at its height -- neighbours outside the x / y range are skipped, headings wrap. Survivors are
// appended (index, score) in no particular order; the caller orders them.
__global__ void k_score_maxima(const float* __restrict__ sc, int nz, int nx, int ny, int n_yaw, float min_score,
                               int cap, int64_t* __restrict__ idx, float* __restrict__ val, int* __restrict__ count) {
    const int64_t n = (int64_t)nz * nx * ny * n_yaw;
    for (int64_t h = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; h < n; h += (int64_t)gridDim.x * blockDim.x) {
        const float mine = sc[h];
        if (!(mine > 0.0f) || mine < min_score) continue;
        const int iyaw = (int)(h % n_yaw);
        const int64_t p = h / n_yaw;
        const int iy = (int)(p % ny);
        const int ix = (int)((p / ny) % nx);
        const int64_t base = p - (int64_t)iy - (int64_t)ix * ny;  // iz's first position
        bool best = true;
        for (int ox = -1; ox <= 1 && best; ++ox) {
            const int jx = ix + ox;
            if (jx < 0 || jx >= nx) continue;
            for (int oy = -1; oy <= 1 && best; ++oy) {
                const int jy = iy + oy;
                if (jy < 0 || jy >= ny) continue;
                const int64_t q = (base + (int64_t)jx * ny + jy) * n_yaw;
                for (int oa = -1; oa <= 1; ++oa) {
                    if (ox == 0 && oy == 0 && oa == 0) continue;
                    const int ja = (iyaw + oa + n_yaw) % n_yaw;
                    if (__ldg(sc + q + ja) > mine) {
                        best = false;
                        break;
                    }
                }
            }
        }
        if (!best) continue;
        const int k = atomicAdd(count, 1);
        if (k < cap) {
            idx[k] = h;
            val[k] = mine;
        }
    }
}

__global__ void __launch_bounds__(SC_THREADS) k_score_list(lw_prior_grid g, const float* __restrict__ pts, int n_pts,
                                                           const float4* __restrict__ hyp, int64_t n_hyp, float tau,
                                                           float* __restrict__ out) {
    __shared__ float px[SC_CHUNK], py[SC_CHUNK], pz[SC_CHUNK];
    const int64_t h = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = h < n_hyp;
    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
    float co = 1.f, si = 0.f;
    if (live) {
        q = hyp[h];
        // cos / sin in float64, rounded once: the heading as the host would pose it
        co = (float)cos((double)q.w);
        si = (float)sin((double)q.w);
    }
    int n_in = 0, sum_d2 = 0;
    for (int base = 0; base < n_pts; base += SC_CHUNK) {
        const int m = min(SC_CHUNK, n_pts - base);
        __syncthreads();
        stage_pts(pts, base, m, px, py, pz);
        __syncthreads();
        if (live) score_chunk(g, px, py, pz, m, q.x, q.y, q.z, co, si, tau, n_in, sum_d2);
    }
    if (live) out[h] = soft_count(n_in, sum_d2, tau);
}

}  // namespace lw

static int check_grid(const lw_prior_grid* g, const char* who) {
    if (!g || !g->xyz || !g->start || !g->nn || g->nx <= 0 || g->ny <= 0 || g->nz <= 0 || g->cell <= 0.0f)
        return set_error(LW_EINVAL, "%s: incomplete prior grid", who);
    if ((int64_t)g->nx * g->ny * g->nz != g->ncell) return set_error(LW_EINVAL, "%s: ncell != nx*ny*nz", who);
    if (((uintptr_t)g->xyz & 15) != 0) return set_error(LW_EINVAL, "%s: xyz must be 16-byte aligned", who);
    if (g->n >= 0x7FFFFFFF) return set_error(LW_ECAPACITY, "%s: %lld map points exceed int32 indices", who, (long long)g->n);
    return LW_OK;
}

extern "C" {

int lw_prior_grid_build(lw_prior_grid* g, void* stream) {
    int r = check_grid(g, "lw_prior_grid_build");
    if (r != LW_OK) return r;
    if (!g->seed || !g->nn2 || !g->df) return set_error(LW_EINVAL, "lw_prior_grid_build: missing build scratch");
    cudaStream_t s = (cudaStream_t)stream;
    int gc = blocks_for(g->ncell, 256, 16 * device_sms());
    int gp = blocks_for(g->n, 256, 16 * device_sms());
    const int tiles_x = (g->nx + JFA_X - 1) / JFA_X, tiles_y = (g->ny + JFA_Y - 1) / JFA_Y;
    const int64_t tiles = (int64_t)tiles_x * tiles_y * g->nz;
    if (tiles > 0x7FFFFFFF) return set_error(LW_ECAPACITY, "lw_prior_grid_build: %lld tiles", (long long)tiles);
    ProfScope prof("grid_build", s);
    k_seed_clear<<<gc, 256, 0, s>>>(*g);
    k_seed<<<gp, 256, 0, s>>>(*g);
    k_unpack<<<gc, 256, 0, s>>>(*g);
    const int steps[5] = {8, 4, 2, 1, 1};  // mapgrid.py:31
    int32_t* a = g->nn2;  // an odd number of steps: from nn2 the last lands in nn
    int32_t* bbuf = g->nn;
    for (int k = 0; k < 5; ++k) {
        if (g->ncell < 0x7FFFFFFF)
            jfa_step<int32_t>(*g, a, bbuf, steps[k], k == 4, (unsigned)tiles, tiles_x, tiles_y, s);
        else
            jfa_step<int64_t>(*g, a, bbuf, steps[k], k == 4, (unsigned)tiles, tiles_x, tiles_y, s);
        int32_t* t = a;
        a = bbuf;
        bbuf = t;
    }
    LW_LAUNCHED("lw_prior_grid_build");
    count_launches(8);
    return LW_OK;
}

// An array that never falls, holds first[j] at cells[j] and first[j + 1] one further on is first[j + 1] from there to
// cells[j + 1]: the two ends of every occupied cell tell for all cells.
int lw_prior_starts_match(const int32_t* start, const int32_t* cells, const int32_t* first, int64_t u, int64_t n,
                          int64_t ncell) {
    if (!start || !cells || !first || u <= 0 || ncell <= 0 || start[0] != 0 || start[ncell] != n) return 0;
    int64_t last = -1;
    for (int64_t j = 0; j < u; ++j) {
        const int64_t c = cells[j], end = j + 1 < u ? first[j + 1] : n;
        if (c <= last || c >= ncell || start[c] != first[j] || start[c + 1] != end) return 0;
        last = c;
    }
    return 1;
}

int lw_prior_starts(const int32_t* cells, const int32_t* first, int64_t u, int64_t n, int64_t ncell, int32_t* start,
                    void* stream) {
    if (u < 0 || n < 0 || n > 0x7FFFFFFF || ncell < 0 || !start || (u > 0 && (!cells || !first)))
        return set_error(LW_EINVAL, "lw_prior_starts: bad arguments");
    k_starts<<<blocks_for((ncell / ST_RUN + 1) * 32, 256, 32 * device_sms()), 256, 0, (cudaStream_t)stream>>>(cells, first, u, n, ncell,
                                                                                               start);
    LW_LAUNCHED("lw_prior_starts");
    count_launches(1);
    return LW_OK;
}

int lw_prior_distances(const lw_prior_grid* g, const float* pts, int64_t n, const double* T_host, float* out,
                       void* stream) {
    int r = check_grid(g, "lw_prior_distances");
    if (r != LW_OK) return r;
    if (!pts || !T_host || !out) return set_error(LW_EINVAL, "lw_prior_distances: null argument");
    if (n <= 0) return LW_OK;
    Pose12 T;
    for (int k = 0; k < 12; ++k) T.m[k] = (float)T_host[k];
    k_distances<<<blocks_for(n, 256, 16 * device_sms()), 256, 0, (cudaStream_t)stream>>>(*g, pts, n, T, out);
    LW_LAUNCHED("lw_prior_distances");
    count_launches(1);
    return LW_OK;
}

int lw_score_grid(const lw_prior_grid* g, const float* pts, int32_t n_pts, const float* pos, int64_t n_pos,
                  int64_t pos_stride, int32_t n_yaw, float yaw0, float dyaw, float tau_cm, float free_cm, float* out,
                  void* stream) {
    int r = check_grid(g, "lw_score_grid");
    if (r != LW_OK) return r;
    if (!g->df || n_pts < 0 || n_pos < 0 || (n_pts > 0 && !pts) || (n_pos > 0 && (!pos || !out)))
        return set_error(LW_EINVAL, "lw_score_grid: bad arguments");
    if (n_yaw < 1 || n_yaw > LW_SCORE_MAX_YAW)
        return set_error(LW_EINVAL, "lw_score_grid: n_yaw %d outside [1, %d]", n_yaw, LW_SCORE_MAX_YAW);
    if (!(tau_cm > 0.0f)) return set_error(LW_EINVAL, "lw_score_grid: tau_cm must be positive");
    if ((int64_t)n_pts * 255 * 255 > 0x7FFFFFFF)
        return set_error(LW_ECAPACITY, "lw_score_grid: %d points overflow the int32 sums", n_pts);
    if (pos_stride < 1) return set_error(LW_EINVAL, "lw_score_grid: pos_stride must be >= 1");
    if (n_pos == 0) return LW_OK;
    const int64_t stride = pos_stride < n_pos ? pos_stride : n_pos;
    const int64_t n_rg = ((n_pos + stride - 1) / stride + 32 * SC_POS - 1) / (32 * SC_POS);  // per column
    const int64_t threads = stride * n_rg * (int64_t)n_yaw * 32;
    YawTab yt;
    lw_score_yaw_table(n_yaw, yaw0, dyaw, yt.c, yt.s);
    const int tau_ceil = tau_cm > 1024.0f ? 1024 : (int)ceilf(tau_cm);  // distances are whole cm in [0, 255]
    const unsigned blocks = (unsigned)((threads + SC_THREADS - 1) / SC_THREADS);
    k_score_grid<<<blocks, SC_THREADS, 0, (cudaStream_t)stream>>>(*g, pts, n_pts, pos, n_pos, stride, n_rg, n_yaw, yt, tau_cm,
                                                                  tau_ceil, free_cm, out);
    if (g->ncell < 0x7FFFFFFF)
        k_score_rest<false><<<blocks, SC_THREADS, 0, (cudaStream_t)stream>>>(*g, pts, n_pts, pos, n_pos, stride, n_rg, n_yaw,
                                                                             yt, tau_cm, tau_ceil, out);
    else
        k_score_rest<true><<<blocks, SC_THREADS, 0, (cudaStream_t)stream>>>(*g, pts, n_pts, pos, n_pos, stride, n_rg, n_yaw,
                                                                            yt, tau_cm, tau_ceil, out);
    LW_LAUNCHED("lw_score_grid");
    count_launches(2);
    return LW_OK;
}

int lw_score_list(const lw_prior_grid* g, const float* pts, int32_t n_pts, const float* hyp, int64_t n_hyp,
                  float tau_cm, float* out, void* stream) {
    int r = check_grid(g, "lw_score_list");
    if (r != LW_OK) return r;
    if (!g->df || n_pts < 0 || n_hyp < 0 || (n_pts > 0 && !pts) || (n_hyp > 0 && (!hyp || !out)))
        return set_error(LW_EINVAL, "lw_score_list: bad arguments");
    if (((uintptr_t)hyp & 15) != 0) return set_error(LW_EINVAL, "lw_score_list: hyp must be 16-byte aligned");
    if (!(tau_cm > 0.0f)) return set_error(LW_EINVAL, "lw_score_list: tau_cm must be positive");
    if ((int64_t)n_pts * 255 * 255 > 0x7FFFFFFF)
        return set_error(LW_ECAPACITY, "lw_score_list: %d points overflow the int32 sums", n_pts);
    if (n_hyp == 0) return LW_OK;
    k_score_list<<<(unsigned)((n_hyp + SC_THREADS - 1) / SC_THREADS), SC_THREADS, 0, (cudaStream_t)stream>>>(
        *g, pts, n_pts, reinterpret_cast<const float4*>(hyp), n_hyp, tau_cm, out);
    LW_LAUNCHED("lw_score_list");
    count_launches(1);
    return LW_OK;
}

int lw_score_maxima(const float* scores, int32_t nz, int32_t nx, int32_t ny, int32_t n_yaw, float min_score,
                    int32_t cap, int64_t* idx, float* val, int32_t* count_dev, void* stream) {
    if (!scores || !idx || !val || !count_dev || nz < 0 || nx < 0 || ny < 0 || n_yaw < 1 || cap < 0)
        return set_error(LW_EINVAL, "lw_score_maxima: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    if (cudaMemsetAsync(count_dev, 0, sizeof(int32_t), s) != cudaSuccess)
        return set_error(LW_ECUDA, "lw_score_maxima: clearing the count failed");
    const int64_t n = (int64_t)nz * nx * ny * n_yaw;
    if (n == 0) return LW_OK;
    k_score_maxima<<<blocks_for(n, 256, 16 * device_sms()), 256, 0, s>>>(scores, nz, nx, ny, n_yaw, min_score, cap,
                                                                        idx, val, count_dev);
    LW_LAUNCHED("lw_score_maxima");
    count_launches(1);
    return LW_OK;
}

void lw_score_yaw_table(int32_t n_yaw, float yaw0, float dyaw, float* c, float* s) {
    for (int j = 0; j < n_yaw; ++j) {
        const float yaw = yaw0 + (float)j * dyaw;  // float32, as localize.py:82
        c[j] = (float)std::cos((double)yaw);
        s[j] = (float)std::sin((double)yaw);
    }
}

int lw_loc_icp_batch(const lw_prior_grid* g, lw_loc_batch* b, int32_t n_hyp, int32_t n_tiles, int32_t tile,
                     int32_t n_stages, const double* dmax, const int32_t* iters, float alpha, int32_t min_count,
                     int32_t blocks_per_sm, int32_t grid, void* stream) {
    return lw_loc_icp_batch_ws(g, b, n_hyp, n_tiles, tile, n_stages, dmax, iters, alpha, min_count, blocks_per_sm, grid,
                               nullptr, stream);
}

int lw_loc_icp_batch_ws(const lw_prior_grid* g, lw_loc_batch* b, int32_t n_hyp, int32_t n_tiles, int32_t tile,
                        int32_t n_stages, const double* dmax, const int32_t* iters, float alpha, int32_t min_count,
                        int32_t blocks_per_sm, int32_t grid, const lw_loc_ws* ws, void* stream) {
    int r = check_grid(g, "lw_loc_icp_batch");
    if (r != LW_OK) return r;
    if (!b || (n_stages > 0 && (!dmax || !iters)) || n_stages < 0 || n_stages > 8 || n_hyp < 1 || n_tiles < 1)
        return set_error(LW_EINVAL, "lw_loc_icp_batch: bad arguments");
    if (!b->pts || !b->scan_end || !b->tile_hyp || !b->tile_lo || !b->hyp_tile || !b->T || !b->tile_part ||
        !b->moved || !b->next || !b->count || !b->eval || !b->bar || !b->err || !b->iters_run || b->pts_cap < 0)
        return set_error(LW_EINVAL, "lw_loc_icp_batch: incomplete batch buffers");
    if (tile < 32 || tile > 2048 || tile % 32 != 0)
        return set_error(LW_EINVAL, "lw_loc_icp_batch: tile must be a multiple of 32 in [32, 2048]");
    if (!g->nrm) return set_error(LW_EINVAL, "lw_loc_icp_batch: the grid needs normals");
    LocArgs la{};
    la.n_hyp = n_hyp;
    la.n_tiles = n_tiles;
    la.n_stages = n_stages;
    la.tile = tile;
    int total_iters = 0;
    for (int k = 0; k < n_stages; ++k) {
        if (iters[k] < 0 || !(dmax[k] > 0.0)) return set_error(LW_EINVAL, "lw_loc_icp_batch: stage %d", k);
        la.max_d2[k] = (float)(dmax[k] * dmax[k]);  // localize.py:541: dmax * dmax
        const double half = dmax[k] * 0.5;
        la.c2[k] = (float)(half * half);  // localize.py:530: (dmax * 0.5) ** 2
        la.iters[k] = iters[k];
        total_iters += iters[k];
    }
    if (total_iters > b->moved_cap) return set_error(LW_ECAPACITY, "lw_loc_icp_batch: %d iterations > moved_cap", total_iters);
    la.alpha = alpha;
    la.radii[0] = 0.03f;  // EVAL_RADII (localize.py:47)
    la.radii[1] = 0.05f;
    la.radii[2] = 0.10f;
    la.min_count = min_count;
    cudaStream_t s = (cudaStream_t)stream;
    int sms = device_sms();
    if (blocks_per_sm == 0) blocks_per_sm = 3;
    if (blocks_per_sm < 2 || blocks_per_sm > 6)
        return set_error(LW_EINVAL, "lw_loc_icp_batch: blocks_per_sm must be 0 or 2..6");
    // one search per point repays the sorting only where it is repeated
    lw_loc_ws w{};
    if (ws && ws->sorted && ws->match && total_iters > 1) w = *ws;
    if (((uintptr_t)w.sorted & 15) != 0)
        return set_error(LW_EINVAL, "lw_loc_icp_batch_ws: the sorted points must be 16-byte aligned");
    using Kernel = void (*)(lw_prior_grid, lw_loc_batch, lw_loc_ws, LocArgs);
    static const Kernel kernels[2][5] = {
        {k_loc_icp<2, false>, k_loc_icp<3, false>, k_loc_icp<4, false>, k_loc_icp<5, false>, k_loc_icp<6, false>},
        {k_loc_icp<2, true>, k_loc_icp<3, true>, k_loc_icp<4, true>, k_loc_icp<5, true>, k_loc_icp<6, true>}};
    const Kernel fn = kernels[w.sorted ? 1 : 0][blocks_per_sm - 2];
    int per_sm = 0;
    LW_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, LOC_BLOCK, 0));
    if (per_sm < 1) return set_error(LW_EINVAL, "lw_loc_icp_batch: the kernel does not fit on an SM");
    int max_grid = per_sm * sms;
    if (grid <= 0 || grid > max_grid) grid = max_grid;
    if (grid > b->grid_cap) grid = b->grid_cap;
    ProfScope prof("loc_icp", s);
    k_loc_reset<<<16, 256, 0, s>>>(*b, n_hyp, total_iters);
    if (w.sorted) {
        static bool attr_set[64] = {};
        int dev = 0;
        LW_CUDA(cudaGetDevice(&dev));
        if (dev < 0 || dev >= 64 || !attr_set[dev]) {
            LW_CUDA(cudaFuncSetAttribute(k_loc_sort, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         LS_BOXES * (int)sizeof(int)));
            if (dev >= 0 && dev < 64) attr_set[dev] = true;
        }
        k_loc_sort<<<n_hyp < 4 * sms ? n_hyp : 4 * sms, LS_T, LS_BOXES * sizeof(int), s>>>(*b, w, n_hyp, n_tiles, tile);
        count_launches(1);
    }
    // a cooperative launch (every CTA resident: the grid barriers rely on it), made through cudaLaunchKernelEx
    // so that it can also be captured into a CUDA graph
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(LOC_BLOCK);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    LW_CUDA(cudaLaunchKernelEx(&cfg, fn, *g, *b, w, la));
    LW_LAUNCHED("lw_loc_icp_batch");
    count_launches(2);
    return LW_OK;
}

}  // extern "C"

