// Neighbourhood summaries of the visible points on sm_100a: a weighted neighbour count, a PCA normal and the
// curvature per point, from a voxel summary a third of the radius wide.
//
// Reference: python/livox_warp/gpu.py -- k_nb_insert :781-800, k_nb_flag / k_nb_compact :803-826, k_nb_voxel
// :829-876, k_nb_gather :879-904, Pipeline.neighborhoods :1531-1557.
//
// Determinism: the reference adds float coordinates into its voxels with float atomics and sums each voxel's
// neighbours in the order a hash-grid query returns them, so its answers depend on thread timing. Here the voxel
// sums are int64 fixed point (exact), the neighbours of a voxel are the voxels whose centroid lies within the radius
// -- all within 3 voxels along each axis (a centroid lies inside its voxel, and voxels are radius / 3 wide), found
// through the masks of the 27 bricks around it (lw_bricks.cuh) -- and their weighted offsets and outer products are
// summed as int64 fixed point too; the covariance and its eigen-decomposition are float64. Every point's count,
// normal and curvature is then independent of thread order and of where keys land in the table. (A table smaller than two
// slots a point can run out of room; which points it then leaves out depends on their order of arrival.)
//
// Layout of the caller's buffers: keys, v_slot / vidx and v_w hold the bricks' keys, masks' halves and bases in the first
// brick_slots(n) slots (so a call clears what its points can fill, not the whole table); acc holds voxel v's sums and
// then, in its place, the record (x, y, z, weight); v_cnt holds a voxel's brick slot until its count replaces it.
#include "lw_common.cuh"
#include "lw_bricks.cuh"
#include "lw_linalg.cuh"

namespace lw {

constexpr double NB_FIX_D = 1048576.0;         // units per metre of a neighbour offset (2^20)
constexpr double NB_FIX_DD = 1099511627776.0;  // units per m^2 of an offset product (2^40)
constexpr int NB_REACH = 3;                    // voxels per axis: radius / (radius / 3)

struct NbArgs {
    float inv_h, r2;
    int mask, want_normals;
    int per;       // voxels per CTA
    int64_t vcap;  // voxel records the buffers hold
    double sensor[3];
};

template <int STRIDE>
__device__ __forceinline__ void nb_ld(const float* __restrict__ xyz, int64_t i, float& x, float& y, float& z) {
    x = xyz[STRIDE * i];
    y = xyz[STRIDE * i + 1];
    z = xyz[STRIDE * i + 2];
}

__global__ void k_nb_clear(lw_nbr_buf nb, int64_t slots) {
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < slots; s += (int64_t)gridDim.x * blockDim.x) {
        nb.keys[s] = EMPTY_KEY;
        nb.v_slot[s] = 0;
        nb.vidx[s] = 0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *nb.m = 0;
}

template <int STRIDE>
__device__ __forceinline__ int64_t nb_brick(const float* __restrict__ xyz, int64_t i, const NbArgs& a, float& x, float& y,
                                            float& z, int& bit) {
    nb_ld<STRIDE>(xyz, i, x, y, z);
    return brick_of(ifloor(x * a.inv_h), ifloor(y * a.inv_h), ifloor(z * a.inv_h), bit);  // floor(w * inv_h), gpu.py:243
}

// Each point claims its voxel's brick and marks the voxel.
template <int STRIDE>
__global__ void k_nb_insert(const float* __restrict__ xyz, const int* n_dev, int64_t n_ub, NbArgs a, lw_nbr_buf nb) {
    int64_t n = n_dev ? (int64_t)*n_dev : n_ub;
    if (n > n_ub) n = n_ub;
    auto mark_half = [](int32_t* half, unsigned bits) {
        if (bits != 0 && (~*(volatile unsigned*)half & bits) != 0) atomicOr(reinterpret_cast<unsigned*>(half), bits);
    };
    const int lane = threadIdx.x & 31;
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < n; i0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = i0 + lane;
        const bool live = i < n;
        float x, y, z;
        int bit = 0;
        int64_t key = EMPTY_KEY;
        if (live) key = nb_brick<STRIDE>(xyz, i, a, x, y, z, bit);
        const int s = enter_brick(live, key, bit, nb.keys, a.mask, [&](int slot, uint64_t bits) {
            mark_half(nb.v_slot + slot, (unsigned)bits);
            mark_half(nb.vidx + slot, (unsigned)(bits >> 32));
        });
        if (live) nb.slot_of_pt[i] = s;
    }
}

__device__ __forceinline__ uint64_t nb_mask(const lw_nbr_buf& nb, int s) {
    return (uint64_t)(uint32_t)nb.v_slot[s] | ((uint64_t)(uint32_t)nb.vidx[s] << 32);
}

__global__ void __launch_bounds__(1024) k_nb_number(lw_nbr_buf nb, int64_t slots, int64_t vcap) {
    brick_number(nb.keys, [&](int s) { return nb_mask(nb, s); }, nb.v_w, slots, nb.m,
                 reinterpret_cast<int32_t*>(nb.v_cnt), vcap, [&](int64_t v) {
                     longlong2* a = reinterpret_cast<longlong2*>(nb.acc + 4 * v);
                     a[0] = a[1] = make_longlong2(0, 0);
                 });
}

// Each point adds its coordinates to its voxel in fixed point and keeps the voxel's number. Neighbouring voxels are
// neighbours in memory, and the L2 takes one operation a cycle on a line: where many points share few voxels (200,000 in 27)
// four 64-bit atomics a point take 302 us (the whole pass 406 us; 109 when the voxels' sums lay apart in a hash), one
// 32-byte bulk reduction 72 (122). A room of 400,000 points in 4,800 voxels: 14 and 10 us.
constexpr int NB_SUM_CTA = 256;

template <int STRIDE>
__global__ void __launch_bounds__(NB_SUM_CTA) k_nb_sum(const float* __restrict__ xyz, const int* n_dev, int64_t n_ub,
                                                       NbArgs a, lw_nbr_buf nb) {
    int64_t n = n_dev ? (int64_t)*n_dev : n_ub;
    if (n > n_ub) n = n_ub;
    const float FW = (float)LW_FIX_W;
    __shared__ __align__(16) int64_t row[NB_SUM_CTA][4];
    int64_t* const mine = row[threadIdx.x];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int s = nb.slot_of_pt[i];
        if (s < 0) continue;
        float x, y, z;
        int bit;
        nb_brick<STRIDE>(xyz, i, a, x, y, z, bit);
        const int64_t v = (int64_t)nb.v_w[s] + popc64(nb_mask(nb, s) & ((1ull << bit) - 1));
        if (v < a.vcap) {
            bulk_read_wait();
            reinterpret_cast<longlong2*>(mine)[0] = make_longlong2(to_fix(x, FW), to_fix(y, FW));
            reinterpret_cast<longlong2*>(mine)[1] = make_longlong2(to_fix(z, FW), 1);
            bulk_add<4>(nb.acc + 4 * v, mine);
        }
        nb.slot_of_pt[i] = v < a.vcap ? (int)v : -1;
    }
    bulk_wait();
}

__device__ __forceinline__ int64_t nb_voxels(const lw_nbr_buf& nb, int64_t vcap) {
    return min((int64_t)*(const unsigned*)nb.m, vcap);
}

// The voxels' means, exact from the fixed-point sums (the reference divides float sums, gpu.py:823), and weights.
__global__ void k_nb_mean(lw_nbr_buf nb, int64_t vcap) {
    const int64_t m = nb_voxels(nb, vcap);
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < m; v += (int64_t)gridDim.x * blockDim.x) {
        const longlong2* acc = reinterpret_cast<const longlong2*>(nb.acc + 4 * v);
        const longlong2 p = acc[0], q = acc[1];
        const double w = (double)q.y;
        const float x = (float)((double)p.x / (w * LW_FIX_W)), y = (float)((double)p.y / (w * LW_FIX_W)),
                    z = (float)((double)q.x / (w * LW_FIX_W));
        *reinterpret_cast<float4*>(nb.acc + 4 * v) = make_float4(x, y, z, __int_as_float((int)q.y));
    }
}

// The voxels in brick order (gpu.py:829-876): every voxel whose centroid lies within the radius adds its points' weight,
// weighted offset and weighted outer product in fixed point; from them the count, and with want_normals the
// covariance's smallest-eigenvalue vector turned toward the sensor and the curvature (smallest eigenvalue / trace).
// Bound by latency and issue of the candidates' walk at a third of the lanes (each lane has its own window), so by the
// warps in flight: 64 registers (8 CTAs per SM) 0.54 ms on 0.5M voxels of a scanned floor, 92 registers 0.66 ms; queueing a
// lane's candidates and working the queues off on full warps was slower (0.72 ms), as were sums without float -> int64
// conversions, which take more registers. A warp per voxel probing 343 offsets, its lane 0 decomposing alone, took 3.15 ms.
__global__ void __launch_bounds__(BRICK_CTA, 8) k_nb_voxel(NbArgs a, lw_nbr_buf nb) {
    __shared__ BrickRows rows;
    __shared__ long long part[BRICK_WARPS - 1][10][32];
    const int64_t m = nb_voxels(nb, a.vcap);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t j0 = (int64_t)blockIdx.x * a.per; j0 < m; j0 += (int64_t)gridDim.x * a.per) {
        const int64_t j = lane < a.per ? j0 + lane : m;
        const int slot = j < m ? __float_as_int(nb.v_cnt[j]) : -1;
        const float4 P = j < m ? *reinterpret_cast<const float4*>(nb.acc + 4 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
        long long W = 0, s1[3] = {0, 0, 0}, s2[6] = {0, 0, 0, 0, 0, 0};
        brick_rows(nb.keys, nb.v_w, a.mask, [&](int s, int, int, int) { return nb_mask(nb, s); }, slot, rows, [&](int row) {
            const int bit = nth_bit(rows.mask[row][13], (int)j - rows.base[row][13]);
#pragma unroll 1
            for (int c = warp; c < 27; c += BRICK_WARPS) {
                const uint64_t all = rows.mask[row][c];
                uint64_t near = all & brick_window(bit, c % 3 - 1, c / 3 % 3 - 1, c / 9 - 1, NB_REACH);
                const int base = rows.base[row][c];
                while (near) {
                    const int b = __ffsll((long long)near) - 1;
                    near &= near - 1;
                    const int64_t k = base + popc64(all & ((1ull << b) - 1));
                    if (k >= m) continue;
                    const float4 Q = *reinterpret_cast<const float4*>(nb.acc + 4 * k);
                    const float ex = Q.x - P.x, ey = Q.y - P.y, ez = Q.z - P.z;
                    if (ex * ex + ey * ey + ez * ez > a.r2) continue;
                    const int w = __float_as_int(Q.w);
                    const float FD = (float)NB_FIX_D, FDD = (float)NB_FIX_DD;
                    W += w;
                    s1[0] += (long long)w * __float2int_rn(ex * FD);  // at most 4 m: 2^22 units
                    s1[1] += (long long)w * __float2int_rn(ey * FD);
                    s1[2] += (long long)w * __float2int_rn(ez * FD);
                    s2[0] += w * to_fix(ex * ex, FDD);
                    s2[1] += w * to_fix(ex * ey, FDD);
                    s2[2] += w * to_fix(ex * ez, FDD);
                    s2[3] += w * to_fix(ey * ey, FDD);
                    s2[4] += w * to_fix(ey * ez, FDD);
                    s2[5] += w * to_fix(ez * ez, FDD);
                }
            }
        }, NoAfter());
        if (warp > 0) {
            long long(*p)[32] = part[warp - 1];
            p[0][lane] = W;
#pragma unroll
            for (int c = 0; c < 3; ++c) p[1 + c][lane] = s1[c];
#pragma unroll
            for (int c = 0; c < 6; ++c) p[4 + c][lane] = s2[c];
        }
        __syncthreads();
        if (warp > 0 || j >= m) continue;  // the next round's first barrier comes after this round's reads of part
#pragma unroll
        for (int q = 0; q < BRICK_WARPS - 1; ++q) {
            W += part[q][0][lane];
#pragma unroll
            for (int c = 0; c < 3; ++c) s1[c] += part[q][1 + c][lane];
#pragma unroll
            for (int c = 0; c < 6; ++c) s2[c] += part[q][4 + c][lane];
        }
        nb.v_cnt[j] = (float)W;
        if (a.want_normals == 0) continue;
        // toward the sensor, in float64 from the float coordinates
        double tx = a.sensor[0] - (double)P.x, ty = a.sensor[1] - (double)P.y, tz = a.sensor[2] - (double)P.z;
        const double tl = sqrt(tx * tx + ty * ty + tz * tz);
        if (tl > 0.0) {
            tx /= tl;
            ty /= tl;
            tz /= tl;
        }
        const double inv = 1.0 / fmax((double)W, 1.0);
        const double mu[3] = {(double)s1[0] / NB_FIX_D * inv, (double)s1[1] / NB_FIX_D * inv,
                              (double)s1[2] / NB_FIX_D * inv};
        const int up[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
        double C[9], ev[3], Q[9];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) C[r * 3 + c] = (double)s2[up[r * 3 + c]] / NB_FIX_DD * inv - mu[r] * mu[c];
        jacobi_eig<3>(C, ev, Q);
        int kmin = 0;
        if (ev[1] < ev[kmin]) kmin = 1;
        if (ev[2] < ev[kmin]) kmin = 2;
        // selects instead of indexing keep ev and Q in registers
        auto at = [](const double* v, int k) { return k == 0 ? v[0] : (k == 1 ? v[1] : v[2]); };
        double nx = at(Q, kmin), ny = at(Q + 3, kmin), nz = at(Q + 6, kmin);
        const double nl = sqrt(nx * nx + ny * ny + nz * nz);
        if (nl > 0.0) {
            nx /= nl;
            ny /= nl;
            nz /= nl;
        }
        if (nx * tx + ny * ty + nz * tz < 0.0) {
            nx = -nx;
            ny = -ny;
            nz = -nz;
        }
        const double tr = ev[0] + ev[1] + ev[2];
        if (tr <= 1.0e-12) {  // a lone voxel: no surface to fit
            nx = tx;
            ny = ty;
            nz = tz;
        }
        nb.v_nrm[3 * j + 0] = (float)nx;
        nb.v_nrm[3 * j + 1] = (float)ny;
        nb.v_nrm[3 * j + 2] = (float)nz;
        nb.v_curv[j] = (float)(fmax(at(ev, kmin), 0.0) / fmax(tr, 1.0e-12));
    }
}

// Each point takes its voxel's answers (gpu.py:879-904); a point whose voxel did not fit in the table reads as
// crowded (count 2^30), flat and facing up, so nothing hides it.
__global__ void k_nb_gather(const int* n_dev, int64_t n_ub, int want_normals, lw_nbr_buf nb, int32_t* __restrict__ cnt,
                            float* __restrict__ nrm, float* __restrict__ curv) {
    int64_t n = n_dev ? (int64_t)*n_dev : n_ub;
    if (n > n_ub) n = n_ub;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int s = nb.slot_of_pt[i];
        if (s < 0) {
            cnt[i] = 1 << 30;
            if (want_normals) {
                nrm[3 * i] = 0.0f;
                nrm[3 * i + 1] = 0.0f;
                nrm[3 * i + 2] = 1.0f;
                curv[i] = 0.0f;
            }
            continue;
        }
        const int v = s;
        cnt[i] = (int)(nb.v_cnt[v] + 0.5f);
        if (want_normals) {
            nrm[3 * i] = nb.v_nrm[3 * (int64_t)v];
            nrm[3 * i + 1] = nb.v_nrm[3 * (int64_t)v + 1];
            nrm[3 * i + 2] = nb.v_nrm[3 * (int64_t)v + 2];
            curv[i] = nb.v_curv[v];
        }
    }
}

}  // namespace lw

using namespace lw;

extern "C" {

int lw_neighborhoods(const float* xyz, int32_t xyz_stride, const int32_t* n_dev, int64_t n_ub, float radius,
                     int32_t want_normals, const float* sensor, lw_nbr_buf* nb, int32_t* out_cnt, float* out_nrm,
                     float* out_curv, void* stream) {
    if (!nb || !nb->keys || !nb->acc || !nb->vidx || !nb->v_slot || !nb->slot_of_pt || !nb->v_xyz || !nb->v_w ||
        !nb->v_cnt || !nb->v_nrm || !nb->v_curv || !nb->tiles || !nb->m)
        return set_error(LW_EINVAL, "lw_neighborhoods: incomplete buffers");
    if ((nb->cap & (nb->cap - 1)) != 0 || nb->cap <= 0 || nb->cap > (1LL << 30))
        return set_error(LW_EINVAL, "lw_neighborhoods: table capacity must be a power of two");
    if (!(radius > 0.0f) || radius > 4.0f)
        return set_error(LW_EINVAL, "lw_neighborhoods: radius %g outside (0, 4] m", (double)radius);
    if ((xyz_stride != 3 && xyz_stride != 4) || (n_ub > 0 && (!xyz || !out_cnt)) ||
        (want_normals && n_ub > 0 && (!out_nrm || !out_curv || !sensor)))
        return set_error(LW_EINVAL, "lw_neighborhoods: bad arguments");
    if (n_ub > nb->pt_cap)
        return set_error(LW_ECAPACITY, "lw_neighborhoods: %lld points exceed the buffers' %lld", (long long)n_ub,
                         (long long)nb->pt_cap);
    cudaStream_t s = (cudaStream_t)stream;
    NbArgs a{};
    a.inv_h = 3.0f / radius;  // voxels a third of the radius wide (gpu.py:1539)
    a.r2 = radius * radius;
    const int64_t slots = brick_slots(n_ub, nb->cap);
    a.mask = (int)(slots - 1);
    a.want_normals = want_normals ? 1 : 0;
    for (int k = 0; k < 3; ++k) a.sensor[k] = sensor ? (double)sensor[k] : 0.0;
    lw_nbr_buf b = *nb;
    a.vcap = b.cap;
    if ((uintptr_t)b.acc & 8) {  // the voxel records are read 16 bytes at a time
        b.acc += 1;
        a.vcap -= 1;
    }
    const int sms = device_sms();
    a.per = brick_voxels(n_ub, sms);
    if (n_ub <= 0) {
        LW_CUDA(cudaMemsetAsync(nb->m, 0, sizeof(int32_t), s));
        return LW_OK;
    }
    k_nb_clear<<<blocks_for(slots, 256, 16 * sms), 256, 0, s>>>(b, slots);
    static_assert(NB_SUM_CTA == 256, "one grid for the passes over the points");
    const int grid = blocks_for(n_ub, 256, 8 * sms);
    if (xyz_stride == 4)
        k_nb_insert<4><<<grid, 256, 0, s>>>(xyz, n_dev, n_ub, a, b);
    else
        k_nb_insert<3><<<grid, 256, 0, s>>>(xyz, n_dev, n_ub, a, b);
    k_nb_number<<<blocks_for(slots, 1024), 1024, 0, s>>>(b, slots, a.vcap);
    if (xyz_stride == 4)
        k_nb_sum<4><<<grid, NB_SUM_CTA, 0, s>>>(xyz, n_dev, n_ub, a, b);
    else
        k_nb_sum<3><<<grid, NB_SUM_CTA, 0, s>>>(xyz, n_dev, n_ub, a, b);
    // at most one voxel per point
    k_nb_mean<<<grid, 256, 0, s>>>(b, a.vcap);
    k_nb_voxel<<<blocks_for(n_ub, a.per, 64 * sms), BRICK_CTA, 0, s>>>(a, b);
    k_nb_gather<<<grid, 256, 0, s>>>(n_dev, n_ub, a.want_normals, b, out_cnt, out_nrm, out_curv);
    LW_LAUNCHED("lw_neighborhoods");
    count_launches(7);
    return LW_OK;
}

}  // extern "C"
