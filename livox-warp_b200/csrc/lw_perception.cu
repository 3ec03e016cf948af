// Ground segmentation and Euclidean clustering of the visible points on sm_100a.
//
// Reference: python/livox_warp/perception.py -- cell_of :32-36, k_gnd_min :39-43, k_gnd_support :46-58,
// k_gnd_label :61-111, Perception.ground :458-483; k_cl_insert :114-139, k_cc_init/step/jump :142-179,
// k_cc_reset/stats/flag/compact/gather :182-271, Perception.cluster / _voxelize / _label / _compact :487-567.
//
// Ground: the same three passes over a toroidal 2048 x 2048 grid; a fourth pass puts back the cells the points
// touched, so the 32 MB grid is cleared once at construction instead of on every call.
// Clusters: the non-ground points' voxels are gathered into bricks with occupancy masks (lw_bricks.cuh) and numbered brick
// by brick, with exact fixed-point sums per voxel; the nodes are the voxels in the order of their first point
// (deterministic). Neighbours (centroids within `connect`) are met by walking the masks of the 27 bricks around a
// voxel and joined on the spot by a lock-free union-find that always hooks the larger root under the smaller, so every
// component is labelled by its smallest node index -- the fixed point the reference's min-label propagation converges
// to -- independent of thread order. No edge list is kept.
//
// Layout of the caller's buffers during a call: keys and acc hold the bricks' keys, masks and bases in the first
// brick_slots(n) slots; per voxel (in number order) st_sum holds the sums, dense the first point, edge_off
// the node, st_lo the centroid and st_hi the brick's slot until the components' boxes replace the last two.
#include "lw_bricks.cuh"
#include "lw_common.cuh"

namespace lw {

constexpr int GRID = 2048;
constexpr int CTILE = 1024;

__device__ __forceinline__ int cell_of(float x, float y, float inv_cell) {
    int cx = ifloor(x * inv_cell) & (GRID - 1);
    int cy = ifloor(y * inv_cell) & (GRID - 1);
    return cy * GRID + cx;
}

struct GroundArgs {
    float inv_cell, thick, thresh, slope_step, nz_min;
    int min_sup, use_nrm;
};

template <int STRIDE>
__device__ __forceinline__ void ld3(const float* __restrict__ p, int64_t i, float& x, float& y, float& z) {
    x = p[i * STRIDE + 0];
    y = p[i * STRIDE + 1];
    z = p[i * STRIDE + 2];
}

template <int STRIDE>
__global__ void k_gnd_min(const float* __restrict__ xyz, const int* n_dev, int64_t n_ub, GroundArgs a,
                          float* __restrict__ cell_min) {
    int64_t n = n_dev ? (int64_t)*n_dev : n_ub;
    if (n > n_ub) n = n_ub;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float x, y, z;
        ld3<STRIDE>(xyz, i, x, y, z);
        atomic_min_float(cell_min + cell_of(x, y, a.inv_cell), z);
    }
}

template <int STRIDE>
__global__ void k_gnd_support(const float* __restrict__ xyz, const int* n_dev, int64_t n_ub, GroundArgs a,
                              const float* __restrict__ cell_min, int* __restrict__ cell_sup) {
    int64_t n = n_dev ? (int64_t)*n_dev : n_ub;
    if (n > n_ub) n = n_ub;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float x, y, z;
        ld3<STRIDE>(xyz, i, x, y, z);
        int c = cell_of(x, y, a.inv_cell);
        if (z - cell_min[c] < a.thick) atomicAdd(cell_sup + c, 1);
    }
}

template <int STRIDE>
__global__ void k_gnd_label(const float* __restrict__ xyz, const float* __restrict__ nrm, const int* n_dev,
                            int64_t n_ub, GroundArgs a, const float* __restrict__ cell_min,
                            const int* __restrict__ cell_sup, int* __restrict__ out_gnd, float* __restrict__ out_hag) {
    int64_t n = n_dev ? (int64_t)*n_dev : n_ub;
    if (n > n_ub) n = n_ub;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float x, y, z;
        ld3<STRIDE>(xyz, i, x, y, z);
        int cx = ifloor(x * a.inv_cell), cy = ifloor(y * a.inv_cell);
        float g = 1.0e30f, g_floor = 1.0e30f;
        for (int dy = -2; dy <= 2; ++dy)
            for (int dx = -2; dx <= 2; ++dx) {
                int c = ((cy + dy) & (GRID - 1)) * GRID + ((cx + dx) & (GRID - 1));
                if (cell_sup[c] >= a.min_sup) {
                    int cheb = max(abs(dx), abs(dy));
                    float cand = cell_min[c] + a.slope_step * (float)cheb;
                    if (cand < g) {
                        g = cand;
                        g_floor = cell_min[c];
                    }
                }
            }
        if (g > 1.0e29f) {
            out_gnd[i] = 0;
            out_hag[i] = 0.0f;
            continue;
        }
        float h = z - g;
        int is_gnd = 0;
        if (h < a.thresh) {
            is_gnd = 1;
            // a steep normal within the ground band is the foot of a wall, unless the point is right at ground level
            if (a.use_nrm != 0 && h > 0.2f * a.thresh) {
                if (fabsf(nrm[i * 3 + 2]) < a.nz_min) is_gnd = 0;
            }
        }
        out_gnd[i] = is_gnd;
        out_hag[i] = is_gnd != 0 ? h : z - g_floor;
    }
}

template <int STRIDE>
__global__ void k_gnd_reset(const float* __restrict__ xyz, const int* n_dev, int64_t n_ub, GroundArgs a,
                            float* __restrict__ cell_min, int* __restrict__ cell_sup) {
    int64_t n = n_dev ? (int64_t)*n_dev : n_ub;
    if (n > n_ub) n = n_ub;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float x, y, z;
        ld3<STRIDE>(xyz, i, x, y, z);
        int c = cell_of(x, y, a.inv_cell);
        cell_min[c] = 1.0e30f;
        cell_sup[c] = 0;
    }
}

// =====================================================================================================
// Clusters
// =====================================================================================================

struct ClArgs {
    float inv_v;
    int mask, use_gnd;
    int64_t slots;  // brick slots used
    int per;        // voxels that a warp of k_cl_brick and a CTA of k_cl_join take at a time
    int sms;
    float connect2;
    int reach;
    float min_pts;
    int max_out;
};

// The bricks' masks and bases, in the caller's acc: [slots] 64-bit masks, [slots] 32-bit bases, [slots] common labels.
__device__ __forceinline__ uint64_t* cl_masks(const lw_cluster_buf& cb) { return reinterpret_cast<uint64_t*>(cb.acc); }
__device__ __forceinline__ int32_t* cl_bases(const lw_cluster_buf& cb, int64_t slots) {
    return reinterpret_cast<int32_t*>(cb.acc + slots);
}

// Rewritten per voxel: its brick's slot, until the boxes take st_hi over.
__device__ __forceinline__ int32_t* cl_brick(const lw_cluster_buf& cb) { return reinterpret_cast<int32_t*>(cb.st_hi); }

__global__ void k_cl_clear(lw_cluster_buf cb, ClArgs a) {
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < a.slots; s += (int64_t)gridDim.x * blockDim.x) {
        cb.keys[s] = EMPTY_KEY;
        cl_masks(cb)[s] = 0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *cb.m = 0;
}

// Pass 1: non-ground points claim their voxel's brick and mark the voxel.
template <int STRIDE>
__global__ void k_cl_insert(const float* __restrict__ xyz, const int* __restrict__ gnd, const int* n_dev,
                            int64_t n_ub, ClArgs a, lw_cluster_buf cb) {
    int64_t n = n_dev ? (int64_t)*n_dev : n_ub;
    if (n > n_ub) n = n_ub;
    const int lane = threadIdx.x & 31;
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < n; i0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = i0 + lane;
        const bool live = i < n && !(a.use_gnd && gnd[i] != 0);
        int bit = 0;
        int64_t key = EMPTY_KEY;
        if (live) {
            float x, y, z;
            ld3<STRIDE>(xyz, i, x, y, z);
            key = brick_of(ifloor(x * a.inv_v), ifloor(y * a.inv_v), ifloor(z * a.inv_v), bit);
        }
        const int s = enter_brick(live, key, bit, cb.keys, a.mask, [&](int slot, uint64_t bits) {
            uint64_t* m = cl_masks(cb) + slot;
            if ((~*(volatile uint64_t*)m & bits) != 0) atomicOr((unsigned long long*)m, (unsigned long long)bits);
        });
        if (i < n) cb.slot_of_pt[i] = s;
    }
}

// Pass 2: number the voxels.
__global__ void __launch_bounds__(CTILE) k_cl_number(lw_cluster_buf cb, ClArgs a) {
    const uint64_t* masks = cl_masks(cb);
    brick_number(cb.keys, [&](int s) { return masks[s]; }, cl_bases(cb, a.slots), a.slots, cb.m, cl_brick(cb), cb.pt_cap, [&](int64_t v) {
        cb.dense[v] = NO_INDEX;
        cb.st_sum[4 * v + 0] = cb.st_sum[4 * v + 1] = cb.st_sum[4 * v + 2] = cb.st_sum[4 * v + 3] = 0;
    });
}

// Pass 3: exact fixed-point sums per voxel (BULK: by one 32-byte reduction a point, as in k_nb_sum; it needs st_sum 16-byte
// aligned, other buffers take the atomics), and the lowest point index (it orders the nodes; read before its atomic
// minimum: a value read can only be too high, and then the atomic decides).
constexpr int CL_SUM_CTA = 256;

template <int STRIDE, bool BULK>
__global__ void __launch_bounds__(CL_SUM_CTA) k_cl_sum(const float* __restrict__ xyz, const int* n_dev, int64_t n_ub,
                                                       ClArgs a, lw_cluster_buf cb) {
    int64_t n = n_dev ? (int64_t)*n_dev : n_ub;
    if (n > n_ub) n = n_ub;
    const float FW = (float)LW_FIX_W;
    __shared__ __align__(16) int64_t row[CL_SUM_CTA][4];
    int64_t* const mine = row[threadIdx.x];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int s = cb.slot_of_pt[i];
        if (s < 0) continue;
        float x, y, z;
        ld3<STRIDE>(xyz, i, x, y, z);
        int bit;
        brick_of(ifloor(x * a.inv_v), ifloor(y * a.inv_v), ifloor(z * a.inv_v), bit);
        const int64_t v = (int64_t)cl_bases(cb, a.slots)[s] + popc64(cl_masks(cb)[s] & ((1ull << bit) - 1));
        if (BULK) {
            bulk_read_wait();
            reinterpret_cast<longlong2*>(mine)[0] = make_longlong2(to_fix(x, FW), to_fix(y, FW));
            reinterpret_cast<longlong2*>(mine)[1] = make_longlong2(to_fix(z, FW), 1);
            bulk_add<4>(cb.st_sum + 4 * v, mine);
        } else {
            atomic_add_i64(cb.st_sum + 4 * v + 0, to_fix(x, FW));
            atomic_add_i64(cb.st_sum + 4 * v + 1, to_fix(y, FW));
            atomic_add_i64(cb.st_sum + 4 * v + 2, to_fix(z, FW));
            atomic_add_i64(cb.st_sum + 4 * v + 3, 1);
        }
        if ((int)i < *(volatile int32_t*)(cb.dense + v)) atomicMin(cb.dense + v, (int)i);
        cb.slot_of_pt[i] = (int)v;
    }
    if (BULK) bulk_wait();
}

template <int STRIDE>
void cl_sum(const float* xyz, const int* n_dev, int64_t n_ub, const ClArgs& a, const lw_cluster_buf& cb, cudaStream_t s) {
    const int grid = blocks_for(n_ub, CL_SUM_CTA, 8 * a.sms);
    if (((uintptr_t)cb.st_sum & 15) == 0)
        k_cl_sum<STRIDE, true><<<grid, CL_SUM_CTA, 0, s>>>(xyz, n_dev, n_ub, a, cb);
    else
        k_cl_sum<STRIDE, false><<<grid, CL_SUM_CTA, 0, s>>>(xyz, n_dev, n_ub, a, cb);
}

// Pass 4/5: the nodes are the voxels in the order of their first point: per-tile counts, then the scatter.
__device__ __forceinline__ int cl_opens(const lw_cluster_buf& cb, int64_t i, int64_t n, int& v) {
    v = i < n ? cb.slot_of_pt[i] : -1;
    return v >= 0 && cb.dense[v] == (int)i;
}

__global__ void k_cl_node_count(const int* n_dev, int64_t n_ub, lw_cluster_buf cb) {
    int64_t n = n_dev ? (int64_t)*n_dev : n_ub;
    if (n > n_ub) n = n_ub;
    int v;
    int c = __syncthreads_count(cl_opens(cb, (int64_t)blockIdx.x * CTILE + threadIdx.x, n, v));
    if (threadIdx.x == 0) cb.tiles[blockIdx.x] = c;
}

__device__ __forceinline__ int tiles_before(const int* __restrict__ tiles, int b) {
    __shared__ int red[32];
    int s = 0;
    for (int j = threadIdx.x; j < b; j += blockDim.x) s += tiles[j];
    s = warp_sum_i(s);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    int tot = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
    __syncthreads();
    return tot;
}

__global__ void k_cl_node_scatter(const int* n_dev, int64_t n_ub, lw_cluster_buf cb) {
    __shared__ int sm[33];
    int64_t n = n_dev ? (int64_t)*n_dev : n_ub;
    if (n > n_ub) n = n_ub;
    int v;
    const int f = cl_opens(cb, (int64_t)blockIdx.x * CTILE + threadIdx.x, n, v);
    int base = tiles_before(cb.tiles, blockIdx.x);
    int tot;
    int r = block_rank(f, sm, &tot);
    if (!f) return;
    const int j = base + r;
    cb.node_slot[j] = v;
    cb.edge_off[v] = j;
    const int64_t* acc = cb.st_sum + 4 * (int64_t)v;
    double w = (double)acc[3];
    cb.v_w[j] = (int)acc[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float c = (float)((double)acc[d] / (w * LW_FIX_W));
        cb.v_xyz[3 * (int64_t)j + d] = c;
        cb.st_lo[3 * (int64_t)v + d] = c;  // in number order, for the walk over neighbours
    }
}

constexpr int UF_HOPS = 1 << 20;

// The root of x, or -1 after UF_HOPS hops. HALVE shortens the path on the way (not while labels are being put at their
// roots: a late shortening would put one back).
template <bool HALVE = true>
__device__ __forceinline__ int uf_find(int* parent, int x) {
    for (int it = 0; it < UF_HOPS; ++it) {
        // through L2: another SM's hook must be seen, or a lost CAS would be retried on the same stale root
        int p = __ldcg(parent + x);
        if (p == x) return x;
        int gp = __ldcg(parent + p);
        if (HALVE && gp != p) __stcg(parent + x, gp);  // x is no root, and any ancestor will do as its parent
        x = p;
    }
    return -1;
}

// The one label of all voxels of a brick (from k_cl_brick), -1 when they have several.
__device__ __forceinline__ int32_t* cl_common(const lw_cluster_buf& cb, int64_t slots) {
    return reinterpret_cast<int32_t*>(cb.acc + slots) + slots;
}

// Put nodes x and y (any nodes of their components) in one component: hooks the larger root under the smaller; a CAS that
// loses a race (another hook won: progress) retries with the new roots.
__device__ __forceinline__ void uf_join(const lw_cluster_buf& cb, int x, int y) {
    for (int it = 0; it < UF_HOPS; ++it) {
        x = uf_find(cb.label, x);
        y = uf_find(cb.label, y);
        if (x < 0 || y < 0) break;
        if (x == y) return;
        const int hi = max(x, y), lo = min(x, y);
        if (atomicCAS(cb.label + hi, hi, lo) == hi) return;
    }
    atomicExch(cb.err, 1);
}

// Pass 6: the components within each brick, a warp per brick and no atomics: every voxel's links to the brick's (at most 64)
// voxels as a bit mask, closed over the links; the label is the component's smallest node. A brick of one component, as
// most are, gets its label as the brick's common one.
constexpr int CL_WARPS = 4;

__global__ void __launch_bounds__(32 * CL_WARPS) k_cl_brick(ClArgs a, lw_cluster_buf cb) {
    __shared__ float4 pos_s[CL_WARPS][64];  // x, y, z, bit
    __shared__ int node_s[CL_WARPS][64];
    __shared__ uint64_t link_s[CL_WARPS][64];
    const int m = *cb.m;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float4* pos = pos_s[warp];
    int* node = node_s[warp];
    uint64_t* link = link_s[warp];
    const int64_t nwarps = (int64_t)gridDim.x * CL_WARPS;
    for (int64_t w = (int64_t)blockIdx.x * CL_WARPS + warp; w * a.per < m; w += nwarps) {
        const int64_t v0 = w * a.per + lane;
        const int slot0 = lane < a.per && v0 < m ? cl_brick(cb)[v0] : -1;
        // the bricks whose first voxel is among the warp's
        unsigned leads = __ballot_sync(0xffffffffu, slot0 >= 0 && cl_bases(cb, a.slots)[max(slot0, 0)] == (int)v0);
        for (; leads; leads &= leads - 1) {
            const int src = __ffs(leads) - 1;
            const int slot = __shfl_sync(0xffffffffu, slot0, src);
            const int64_t base = w * a.per + src;
            const uint64_t mask = cl_masks(cb)[slot];
            const int n = popc64(mask);
            for (int k = lane; k < n; k += 32) {
                const int64_t v = base + k;
                pos[k] = make_float4(cb.st_lo[3 * v], cb.st_lo[3 * v + 1], cb.st_lo[3 * v + 2],
                                     __int_as_float(nth_bit(mask, k)));
                node[k] = cb.edge_off[v];
            }
            __syncwarp();
            const uint64_t full = n == 64 ? ~0ull : (1ull << n) - 1;
            for (int k = lane; k < n; k += 32) {
                const float4 p = pos[k];
                const uint64_t near = brick_window(__float_as_int(p.w), 0, 0, 0, a.reach);
                uint64_t l = 1ull << k;
                for (int q = 0; q < n; ++q) {
                    const float4 o = pos[q];
                    const float ex = o.x - p.x, ey = o.y - p.y, ez = o.z - p.z;
                    if (ex * ex + ey * ey + ez * ez <= a.connect2 && (near >> __float_as_int(o.w) & 1)) l |= 1ull << q;
                }
                link[k] = l;
            }
            __syncwarp();
            bool whole = true;
            for (int k = lane; k < n; k += 32) {
                uint64_t c = link[k], done = 1ull << k;
                while (c != full && c != done) {
                    const int q = __ffsll((long long)(c & ~done)) - 1;
                    done |= 1ull << q;
                    c |= link[q];
                }
                whole = whole && c == full;
                int label = NO_INDEX;
                for (uint64_t t = c; t; t &= t - 1) label = min(label, node[__ffsll((long long)t) - 1]);
                cb.label[node[k]] = label;
            }
            whole = __all_sync(0xffffffffu, whole);
            if (lane == 0) cl_common(cb, a.slots)[slot] = whole ? cb.label[node[0]] : -1;
            __syncwarp();
        }
    }
}

// Pass 7: the voxels, in brick order, joined with every neighbour of another brick numbered above theirs. Two bricks of one
// component each need a single pair that connects: the walk notes one, and the pairs of a CTA's bricks are then joined
// side by side, a thread each -- a join is a chain of dependent loads, and made where a lane meets its pair it holds up the
// other 31. On 0.3M nodes of a scanned floor counting, writing, scanning and joining edge lists took 2.0 ms and
// joining each pair when met 0.65 ms.
__global__ void __launch_bounds__(BRICK_CTA) k_cl_join(ClArgs a, lw_cluster_buf cb) {
    __shared__ BrickRows rows;
    __shared__ int32_t common[BRICK_ROWS][27];
    __shared__ int32_t met[BRICK_ROWS][27];
    __shared__ int32_t low[BRICK_ROWS];
    const int m = *cb.m;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int R = a.reach;
    for (int64_t j0 = (int64_t)blockIdx.x * a.per; j0 < m; j0 += (int64_t)gridDim.x * a.per) {
        const int64_t v = j0 + lane;
        const bool live = lane < a.per && v < m;
        const int slot = live ? cl_brick(cb)[v] : -1;
        float px = 0.f, py = 0.f, pz = 0.f;
        int me = 0;
        if (live) {
            px = cb.st_lo[3 * v];
            py = cb.st_lo[3 * v + 1];
            pz = cb.st_lo[3 * v + 2];
            me = cb.edge_off[v];
        }
        brick_rows(
            cb.keys, cl_bases(cb, a.slots), a.mask,
            [&](int s, int r, int c, int lead) {
                const int l = cl_common(cb, a.slots)[s];
                common[r][c] = l;
                met[r][c] = -1;
                // numbered below, or both of one component that is the same already: nothing to join
                if (c != 13) {
                    if (cl_bases(cb, a.slots)[s] < cl_bases(cb, a.slots)[lead]) return (uint64_t)0;
                    const int o = cl_common(cb, a.slots)[lead];
                    if (l >= 0 && o >= 0 && __ldcg(cb.label + l) == __ldcg(cb.label + o)) return (uint64_t)0;
                }
                return cl_masks(cb)[s];
            },
            slot, rows,
            [&](int row) {
                const int bit = nth_bit(rows.mask[row][13], (int)v - rows.base[row][13]);
                const bool own_one = common[row][13] >= 0;
#pragma unroll 1
                for (int c = warp; c < 27; c += BRICK_WARPS) {
                    const uint64_t all = rows.mask[row][c];
                    if (all == 0 || c == 13) continue;
                    uint64_t near = all & brick_window(bit, c % 3 - 1, c / 3 % 3 - 1, c / 9 - 1, R);
                    const int base = rows.base[row][c];
                    const bool one = own_one && common[row][c] >= 0;
                    while (near) {
                        if (one && *(volatile int32_t*)&met[row][c] >= 0) break;
                        const int b = __ffsll((long long)near) - 1;
                        near &= near - 1;
                        const int64_t k = base + popc64(all & ((1ull << b) - 1));
                        const float ex = cb.st_lo[3 * k] - px, ey = cb.st_lo[3 * k + 1] - py,
                                    ez = cb.st_lo[3 * k + 2] - pz;
                        if (!(ex * ex + ey * ey + ez * ez <= a.connect2)) continue;
                        if (one) {
                            *(volatile int32_t*)&met[row][c] = 1;
                            break;
                        }
                        uf_join(cb, me, cb.edge_off[k]);
                    }
                }
            },
            [&](int r, int c, bool found) {
                // a brick's own root and those of the bricks it met all go under the smallest, each hook on a word of its own;
                // where another CTA hooked one of them meanwhile all go round again (the smallest must not be lost sight of)
                const bool in = found && common[r][13] >= 0 && (c == 13 || met[r][c] >= 0);
                int x = in ? common[r][c] : 0;
                for (int it = 0; it < UF_HOPS; ++it) {
                    if (threadIdx.x < BRICK_ROWS) low[threadIdx.x] = NO_INDEX;
                    __syncthreads();
                    if (in) {
                        x = uf_find(cb.label, x);
                        if (x >= 0)
                            atomicMin(&low[r], x);
                        else
                            atomicExch(cb.err, 1);
                    }
                    __syncthreads();
                    const bool open = in && x >= 0 && x != low[r] && atomicCAS(cb.label + x, x, low[r]) != x;
                    if (x < 0) x = 0;
                    if (!__syncthreads_or(open)) break;
                }
            });
    }
}

__global__ void k_cl_uf_flatten(lw_cluster_buf cb) {
    const int m = *cb.m;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < m; j += gridDim.x * blockDim.x) {
        const int r = uf_find<false>(cb.label, j);
        if (r < 0) atomicExch(cb.err, 1);
        cb.label[j] = max(r, 0);
#pragma unroll
        for (int d = 0; d < 3; ++d) cb.st_lo[3 * (int64_t)j + d] = cb.st_hi[3 * (int64_t)j + d] = cb.v_xyz[3 * (int64_t)j + d];
    }
}

// Per-root statistics: exact fixed-point sums and point counts (in the root's own voxel sums), float min / max of the
// node centroids. Most nodes of a scene share one root, so a warp takes up to 32 x CL_RUN consecutive nodes, each lane gathers
// what belongs to the warp's usual root in registers and the warp adds it with ten atomics; the other nodes add their own
// (1.0 ms for 0.3M nodes when every node did, on the same ten words).
// A round is a chain of loads, so there are several only where every SM gets eight warps all the same: 210,000 points in 300
// clumps take 36 us by rounds counted by the points, 5 by the nodes; a room of 400,000 points, 15 and 3.
constexpr int CL_RUN = 16;

__global__ void k_cl_stats(lw_cluster_buf cb, ClArgs a) {
    const int m = *cb.m;
    const int run = max(1, min(CL_RUN, m / (32 * 8 * a.sms)));
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t j0 = warp * 32 * run; j0 < m; j0 += nwarps * 32 * run) {
        long long sum[4] = {0, 0, 0, 0};
        float lo[3] = {1.0e30f, 1.0e30f, 1.0e30f}, hi[3] = {-1.0e30f, -1.0e30f, -1.0e30f};
        int usual = -1;
        for (int u = 0; u < run; ++u) {
            const int64_t j = j0 + 32 * u + lane;
            const int r = j < m ? cb.label[j] : -1;
            const bool other = r >= 0 && r != (int)j;  // a root's own sums are in place
            const unsigned some = __ballot_sync(0xffffffffu, other);
            if (some == 0) continue;
            if (usual < 0) {
                // the first such lane's root, or, where most of the others have another, the first of those lanes'
                usual = __shfl_sync(0xffffffffu, r, __ffs(some) - 1);
                const unsigned same = __ballot_sync(0xffffffffu, other && r == usual);
                if (2 * __popc(same) < __popc(some)) {
                    const unsigned rest = some & ~same;
                    usual = __shfl_sync(0xffffffffu, r, __ffs(rest) - 1);
                }
            }
            if (!other) continue;
            const int64_t* acc = cb.st_sum + 4 * (int64_t)cb.node_slot[j];
            const float x[3] = {cb.v_xyz[3 * j], cb.v_xyz[3 * j + 1], cb.v_xyz[3 * j + 2]};
            if (r == usual) {
#pragma unroll
                for (int d = 0; d < 4; ++d) sum[d] += acc[d];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    lo[d] = fminf(lo[d], x[d]);
                    hi[d] = fmaxf(hi[d], x[d]);
                }
            } else {
                int64_t* su = cb.st_sum + 4 * (int64_t)cb.node_slot[r];
#pragma unroll
                for (int d = 0; d < 4; ++d) atomic_add_i64(su + d, acc[d]);
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    atomic_min_float(cb.st_lo + 3 * (int64_t)r + d, x[d]);
                    atomic_max_float(cb.st_hi + 3 * (int64_t)r + d, x[d]);
                }
            }
        }
        if (usual < 0) continue;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
            for (int d = 0; d < 4; ++d) sum[d] += __shfl_xor_sync(0xffffffffu, sum[d], o);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
                hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
            }
        }
        if (lane == 0) {
            int64_t* su = cb.st_sum + 4 * (int64_t)cb.node_slot[usual];
#pragma unroll
            for (int d = 0; d < 4; ++d) atomic_add_i64(su + d, sum[d]);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                atomic_min_float(cb.st_lo + 3 * (int64_t)usual + d, lo[d]);
                atomic_max_float(cb.st_hi + 3 * (int64_t)usual + d, hi[d]);
            }
        }
    }
}

// Dense ids for the roots with at least min_pts points, in node order (<= max_out of them).
__device__ __forceinline__ int cl_kept(const lw_cluster_buf& cb, const ClArgs& a, int m, int j) {
    return j < m && cb.label[j] == j && (float)cb.st_sum[4 * (int64_t)cb.node_slot[j] + 3] >= a.min_pts;
}

__global__ void k_cl_flag(lw_cluster_buf cb, ClArgs a) {
    int c = __syncthreads_count(cl_kept(cb, a, *cb.m, blockIdx.x * CTILE + threadIdx.x));
    if (threadIdx.x == 0) cb.tiles[blockIdx.x] = c;
}

__global__ void k_cl_compact(lw_cluster_buf cb, ClArgs a) {
    __shared__ int sm[33];
    const int m = *cb.m;
    int j = blockIdx.x * CTILE + threadIdx.x;
    const int f = cl_kept(cb, a, m, j);
    int base = tiles_before(cb.tiles, blockIdx.x);
    int tot;
    int r = block_rank(f, sm, &tot);
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        cb.n_clusters[0] = base + tot < a.max_out ? base + tot : a.max_out;
        cb.n_clusters[1] = base + tot;  // before the cap
    }
    if (j < m) cb.dense[j] = -1;
    if (f) {
        int d = base + r;
        if (d < a.max_out) {
            cb.dense[j] = d;
            const int64_t* su = cb.st_sum + 4 * (int64_t)cb.node_slot[j];
            double w = (double)su[3];
            cb.out_cnt[d] = (float)su[3];
            for (int k = 0; k < 3; ++k) {
                cb.out_cen[3 * d + k] = (float)((double)su[k] / (w * LW_FIX_W));
                cb.out_lo[3 * d + k] = cb.st_lo[3 * (int64_t)j + k];
                cb.out_hi[3 * d + k] = cb.st_hi[3 * (int64_t)j + k];
            }
        }
    }
}

// Per point: its cluster id (or -1).
__global__ void k_cl_gather(const int* n_dev, int64_t n_ub, lw_cluster_buf cb, int* __restrict__ out_cid) {
    int64_t n = n_dev ? (int64_t)*n_dev : n_ub;
    if (n > n_ub) n = n_ub;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        int v = cb.slot_of_pt[i];
        out_cid[i] = v < 0 ? -1 : cb.dense[cb.label[cb.edge_off[v]]];
    }
}

}  // namespace lw

using namespace lw;

extern "C" {

int lw_ground(const float* xyz, int32_t xyz_stride, const float* nrm, const int32_t* n_dev, int64_t n_ub, float cell,
              float thick, int32_t min_sup, float thresh, float slope_step, int32_t use_normals, float nz_min,
              float* cell_min, int32_t* cell_sup, int32_t* out_gnd, float* out_hag, void* stream) {
    if (!xyz || !cell_min || !cell_sup || !out_gnd || !out_hag || (use_normals && !nrm) ||
        (xyz_stride != 3 && xyz_stride != 4))
        return set_error(LW_EINVAL, "lw_ground: bad arguments");
    if (n_ub <= 0) return LW_OK;
    cudaStream_t s = (cudaStream_t)stream;
    GroundArgs a;
    a.inv_cell = 1.0f / fmaxf(cell, 0.05f);
    a.thick = thick;
    a.thresh = thresh;
    a.slope_step = slope_step;
    a.nz_min = nz_min;
    a.min_sup = min_sup;
    a.use_nrm = use_normals ? 1 : 0;
    int grid = blocks_for(n_ub, 256, 8 * device_sms());
    ProfScope prof("ground", s);
    if (xyz_stride == 4) {
        k_gnd_min<4><<<grid, 256, 0, s>>>(xyz, n_dev, n_ub, a, cell_min);
        k_gnd_support<4><<<grid, 256, 0, s>>>(xyz, n_dev, n_ub, a, cell_min, cell_sup);
        k_gnd_label<4><<<grid, 256, 0, s>>>(xyz, nrm, n_dev, n_ub, a, cell_min, cell_sup, out_gnd, out_hag);
        k_gnd_reset<4><<<grid, 256, 0, s>>>(xyz, n_dev, n_ub, a, cell_min, cell_sup);
    } else {
        k_gnd_min<3><<<grid, 256, 0, s>>>(xyz, n_dev, n_ub, a, cell_min);
        k_gnd_support<3><<<grid, 256, 0, s>>>(xyz, n_dev, n_ub, a, cell_min, cell_sup);
        k_gnd_label<3><<<grid, 256, 0, s>>>(xyz, nrm, n_dev, n_ub, a, cell_min, cell_sup, out_gnd, out_hag);
        k_gnd_reset<3><<<grid, 256, 0, s>>>(xyz, n_dev, n_ub, a, cell_min, cell_sup);
    }
    LW_LAUNCHED("lw_ground");
    count_launches(4);
    return LW_OK;
}

int lw_cluster(const float* xyz, int32_t xyz_stride, const int32_t* gnd, int32_t use_ground, const int32_t* n_dev,
               int64_t n_ub, float voxel, float connect, float min_pts, int32_t max_out, lw_cluster_buf* cb,
               int32_t* out_cid, void* stream) {
    if (!xyz || !cb || !out_cid || (use_ground && !gnd) || (xyz_stride != 3 && xyz_stride != 4))
        return set_error(LW_EINVAL, "lw_cluster: bad arguments");
    if ((cb->cap & (cb->cap - 1)) != 0) return set_error(LW_EINVAL, "lw_cluster: table capacity not a power of two");
    if (n_ub > cb->pt_cap) return set_error(LW_ECAPACITY, "lw_cluster: %lld points exceed the buffers' %lld",
                                           (long long)n_ub, (long long)cb->pt_cap);
    if (n_ub <= 0) return LW_OK;
    cudaStream_t s = (cudaStream_t)stream;
    ClArgs a;
    a.inv_v = 1.0f / fmaxf(voxel, 0.01f);
    a.slots = brick_slots(n_ub, cb->cap);
    a.mask = (int)(a.slots - 1);
    a.use_gnd = use_ground ? 1 : 0;
    a.connect2 = connect * connect;
    a.reach = (int)ceilf(connect * a.inv_v);
    if (a.reach < 1) a.reach = 1;
    if (a.reach > 4) return set_error(LW_EINVAL, "lw_cluster: connect / voxel = %g needs a %d-voxel reach (max 4)",
                                      (double)(connect * a.inv_v), a.reach);
    a.min_pts = min_pts;
    a.max_out = max_out;
    const int sms = device_sms();
    a.per = brick_voxels(n_ub, sms);
    a.sms = sms;
    int grid = blocks_for(n_ub, 256, 8 * sms);
    int nt = blocks_for(n_ub, CTILE);
    ProfScope prof("cluster", s);
    k_cl_clear<<<blocks_for(a.slots, 256, 16 * sms), 256, 0, s>>>(*cb, a);
    if (xyz_stride == 4)
        k_cl_insert<4><<<grid, 256, 0, s>>>(xyz, gnd, n_dev, n_ub, a, *cb);
    else
        k_cl_insert<3><<<grid, 256, 0, s>>>(xyz, gnd, n_dev, n_ub, a, *cb);
    k_cl_number<<<blocks_for(a.slots, CTILE), CTILE, 0, s>>>(*cb, a);
    if (xyz_stride == 4)
        cl_sum<4>(xyz, n_dev, n_ub, a, *cb, s);
    else
        cl_sum<3>(xyz, n_dev, n_ub, a, *cb, s);
    k_cl_node_count<<<nt, CTILE, 0, s>>>(n_dev, n_ub, *cb);
    k_cl_node_scatter<<<nt, CTILE, 0, s>>>(n_dev, n_ub, *cb);
    // at most one node per point
    const int gridj = blocks_for(n_ub, a.per, 64 * sms);
    k_cl_brick<<<blocks_for(n_ub, a.per * CL_WARPS, 64 * sms), 32 * CL_WARPS, 0, s>>>(a, *cb);
    k_cl_join<<<gridj, BRICK_CTA, 0, s>>>(a, *cb);
    k_cl_uf_flatten<<<grid, 256, 0, s>>>(*cb);
    // four warps to a CTA: two rounds of eight warps an SM, or CL_RUN rounds of 32 nodes a warp, whichever are more
    const int full = blocks_for(n_ub, 128 * CL_RUN, 16 * sms);
    k_cl_stats<<<blocks_for(n_ub, 128, full > 4 * sms ? full : 4 * sms), 128, 0, s>>>(*cb, a);
    k_cl_flag<<<nt, CTILE, 0, s>>>(*cb, a);
    k_cl_compact<<<nt, CTILE, 0, s>>>(*cb, a);
    k_cl_gather<<<grid, 256, 0, s>>>(n_dev, n_ub, *cb, out_cid);
    LW_LAUNCHED("lw_cluster");
    count_launches(13);
    return LW_OK;
}

}  // extern "C"
