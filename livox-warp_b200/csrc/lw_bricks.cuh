// Voxels gathered into bricks of 4 x 4 x 4: a hash of bricks, each with a 64-bit mask of its occupied voxels, and the
// voxels numbered brick by brick, so that voxel `bit` of a brick is number base + popcount(mask below bit).
//
// Why: finding a voxel's neighbours in a hash of voxels takes one probe per offset of the neighbourhood -- 343 for a
// reach of 3 voxels, 729 for 4, nearly all of them misses. A neighbourhood of up to 4 voxels' reach lies in 27 bricks:
// 27 probes, shared by all voxels of a brick, then a walk over the set bits of the masks, which meets only occupied
// voxels; and those lie next to each other in memory.
//
// Coordinates are the 21-bit fields of the voxel key (gpu.py:231-239), so neighbourhoods wrap where keys do.
#pragma once
#include <type_traits>

#include "lw_common.cuh"

namespace lw {

constexpr int64_t BRICK_MASK = (1LL << 19) - 1;  // a 21-bit field without its two low bits

__device__ __forceinline__ int64_t brick_key(int64_t bx, int64_t by, int64_t bz) {
    return (bx & BRICK_MASK) | ((by & BRICK_MASK) << 19) | ((bz & BRICK_MASK) << 38);
}

// The brick of voxel (ix, iy, iz) and the voxel's bit in it: x + 4 y + 16 z of the low coordinate bits.
__device__ __forceinline__ int64_t brick_of(int ix, int iy, int iz, int& bit) {
    const int64_t x = ((int64_t)ix + KEY_BIAS) & KEY_MASK, y = ((int64_t)iy + KEY_BIAS) & KEY_MASK,
                  z = ((int64_t)iz + KEY_BIAS) & KEY_MASK;
    bit = (int)(x & 3) | ((int)(y & 3) << 2) | ((int)(z & 3) << 4);
    return brick_key(x >> 2, y >> 2, z >> 2);
}

// The table of the bricks. Its load may come to a half (a cloud sparser than a brick), and the bricks of a floor are a regular
// lattice, which slot_hash -- one multiplication, one shift -- lays in clumps: 2^20 bricks of a flat grid in 2^21 slots
// lost 250 to a window of 64 probes, differing ones with the order of arrival. So the keys are mixed by two rounds, which
// leave the longest chain of the same grid at 34 (45 over all lattices and halls tried, up to 3M bricks), and the window
// is 256: a random table at half load has a chain that long once in 10^15 calls. A table smaller than twice
// the points serves as far as it goes (loads up to 0.8); bricks it has no room for are reported as such.
constexpr int BRICK_PROBES = 256;

__host__ __device__ __forceinline__ int brick_hash(int64_t k) {
    uint64_t h = (uint64_t)k * HASH_MULT;
    h ^= h >> 32;
    h *= HASH_MULT;
    h ^= h >> 29;
    return (int)(h & 0x7FFFFFFFULL);
}

// Slot of the brick, or -1.
__device__ __forceinline__ int find_brick(int64_t key, const int64_t* __restrict__ keys, int mask) {
    return find_from<BRICK_PROBES>(brick_hash(key), key, keys, mask);
}

// Slot of the brick, claimed if it has none yet; -1 when its window is full.
__device__ __forceinline__ int claim_brick(int64_t key, int64_t* keys, int mask) {
    bool claimed;
    return claim_from<BRICK_PROBES>(brick_hash(key), key, keys, mask, &claimed);
}

// Slots a hash of at most n bricks takes: the power of two from 2 n up, at least 1024 and at most cap.
inline int64_t brick_slots(int64_t n, int64_t cap) {
    int64_t h = 1024;
    while (h < 2 * n) h *= 2;
    return h < cap ? h : cap;
}

__device__ __forceinline__ int popc64(uint64_t v) { return __popcll(v); }

// The slot of each lane's brick (every lane calls; live: the lane has a point; -1 without room), claimed where it has none
// yet, and the points' voxels marked: mark(s, bits) sets `bits` in the mask of the brick in slot s.
// Every point finds the table empty when a call starts, and the L2 takes one operation a cycle on a word: with a claim and a
// mark a point, 200,000 points of one brick take 60 us. So a brick is claimed by one of the warp's lanes in it, and marked by
// that one too where eight or more share it: 8 us.
constexpr int BRICK_SHARED = 8;

template <class Mark>
__device__ __forceinline__ int enter_brick(bool live, int64_t key, int bit, int64_t* keys, int mask, const Mark& mark) {
    constexpr unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned group = __match_any_sync(full, (unsigned long long)(live ? key : EMPTY_KEY));
    const int leader = __ffs(group) - 1;
    int s = -1;
    if (live && lane == leader) s = claim_brick(key, keys, mask);
    s = __shfl_sync(full, s, leader);
    uint64_t bits = live && s >= 0 ? 1ull << bit : 0ull;
    for (unsigned b = __ballot_sync(full, live && lane == leader && __popc(group) >= BRICK_SHARED); b; b &= b - 1) {
        const int lead = __ffs(b) - 1;
        const bool in = leader == lead;
        const unsigned lo = __reduce_or_sync(full, in ? (unsigned)bits : 0u);
        const unsigned hi = __reduce_or_sync(full, in ? (unsigned)(bits >> 32) : 0u);
        if (in) bits = lane == lead ? (uint64_t)lo | (uint64_t)hi << 32 : 0ull;
    }
    if (bits) mark(s, bits);
    return s;
}

// The n-th set bit of a mask, from 0.
__device__ __forceinline__ int nth_bit(uint64_t mask, int n) {
    uint32_t h = (uint32_t)mask;
    int bit = 0;
    if (n >= __popc(h)) {
        n -= __popc(h);
        h = (uint32_t)(mask >> 32);
        bit = 32;
    }
    for (int k = 0; k < n; ++k) h &= h - 1;
    return bit + __ffs(h) - 1;
}

// The low coordinates (0..3) of the brick `o` away whose distance from l is at most R, as a 4-bit pattern (R <= 4).
__device__ __forceinline__ unsigned brick_span(int l, int o, int R) {
    const int lo = max(0, l - R - 4 * o), hi = min(3, l + R - 4 * o);
    return hi < lo ? 0u : (0xFu >> (3 - hi)) & (0xFu << lo);
}

// The voxels of the brick (ox, oy, oz) away within R of bit `bit` along every axis.
__device__ __forceinline__ uint64_t brick_window(int bit, int ox, int oy, int oz, int R) {
    const uint64_t x = brick_span(bit & 3, ox, R) * 0x1111111111111111ull;
    const unsigned py = brick_span((bit >> 2) & 3, oy, R), pz = brick_span(bit >> 4, oz, R);
    const uint64_t row = ((py & 1u) * 0xFu) | ((py >> 1 & 1u) * 0xF0u) | ((py >> 2 & 1u) * 0xF00u) |
                         ((py >> 3 & 1u) * 0xF000u);
    const uint64_t y = row * 0x0001000100010001ull;
    const uint64_t z = ((pz & 1u) * 0xFFFFull) | ((pz >> 1 & 1u) * 0xFFFF0000ull) |
                       ((uint64_t)(pz >> 2 & 1u) * 0xFFFFull << 32) | ((uint64_t)(pz >> 3 & 1u) * 0xFFFFull << 48);
    return x & y & z;
}

// The 27 bricks around each of up to BRICK_ROWS bricks, for one CTA's voxels.
constexpr int BRICK_ROWS = 4, BRICK_WARPS = 4;
constexpr int BRICK_CTA = 32 * BRICK_WARPS;  // threads of a CTA that walks neighbourhoods: 32 voxels, BRICK_WARPS threads each
struct BrickRows {
    uint64_t mask[BRICK_ROWS][27];
    int32_t base[BRICK_ROWS][27];
};

// Voxels that a CTA walking neighbourhoods takes at a time: 32, or 8 up to 64 points an SM -- one wave of such CTAs, eight to an
// SM -- where 32 would leave most of the chip idle and each CTA with a chain of up to 32 lone bricks to look up, four at a
// time. A perception frame of 500 / 6,000 sparse points: 357 / 501 us with 32, 274 / 410 with 8 (274 / 414 before there were
// bricks); from 12,000 on 32 is as good.
inline int brick_voxels(int64_t n, int sms) { return n > 64 * (int64_t)sms ? 32 : 8; }

// For the up to 32 voxels of a CTA, lane l of every warp serving voxel l, in the order of their numbers (slot: the voxel's
// brick, -1 for none; every thread calls), run(row) with the bricks around the lane's own brick in rows.mask[row],
// rows.base[row]. Voxels of a brick are neighbours in number, so 32 of them lie in a few bricks, whose 27 neighbours are
// looked up side by side, BRICK_ROWS bricks at a time. The warps share out the 27 bricks (warp w takes w, w + BRICK_WARPS, ...):
// a scene's voxels alone leave too few warps in flight to hide the walk's loads.
// mask_of(s, r, c, lead) is the mask of the brick in slot s of the hash (keys, base, hash_mask), found for rows[r][c]
// around the brick in slot lead.
// after(r, c, found): called by every thread once the lanes are done with the bricks looked up, found where the thread's own
// lookup (r, c) met a brick.
struct NoAfter {};
template <class MaskOf, class Run, class After>
__device__ __forceinline__ void brick_rows(const int64_t* keys, const int32_t* base, int hash_mask, const MaskOf& mask_of,
                                           int slot, BrickRows& rows, const Run& run, const After& after) {
    static_assert(BRICK_ROWS * 27 <= BRICK_CTA, "one lookup per thread");
    const int lane = threadIdx.x & 31;
    const int prev = __shfl_up_sync(0xffffffffu, slot, 1);
    const unsigned leaders = __ballot_sync(0xffffffffu, slot >= 0 && (lane == 0 || slot != prev));
    const int mine = __popc(leaders & (0xffffffffu >> (31 - lane))) - 1;  // my brick's place among the leaders
    const int nrows = __popc(leaders);
    unsigned left = leaders;
    for (int r0 = 0; r0 < nrows; r0 += BRICK_ROWS) {
        const int here = min(BRICK_ROWS, nrows - r0);
        const int r = threadIdx.x / 27, c = threadIdx.x - 27 * r;
        int lead = 0, s = -1;
#pragma unroll
        for (int q = 0; q < BRICK_ROWS; ++q) {
            const int ls = __shfl_sync(0xffffffffu, slot, left ? __ffs(left) - 1 : 0);
            left &= left - 1;
            lead = q == r ? ls : lead;
        }
        if (r < here) {
            const int64_t k = keys[lead];
            const int64_t nk = brick_key((k & BRICK_MASK) + (c % 3 - 1), (k >> 19 & BRICK_MASK) + (c / 3 % 3 - 1),
                                         (k >> 38 & BRICK_MASK) + (c / 9 - 1));
            s = c == 13 ? lead : find_brick(nk, keys, hash_mask);
            rows.mask[r][c] = s < 0 ? 0ull : mask_of(s, r, c, lead);
            rows.base[r][c] = s < 0 ? 0 : base[s];
        }
        __syncthreads();
        if (slot >= 0 && mine >= r0 && mine < r0 + here) run(mine - r0);
        __syncthreads();
        if constexpr (!std::is_same<After, NoAfter>::value) {
            after(r, c, s >= 0);
            __syncthreads();  // after() may read what other threads' lookups left: not before all are done with it
        }
    }
}

// Number the voxels brick by brick: a CTA per 1024 brick slots takes a run of numbers for its bricks (which run depends
// on timing, so no result may depend on a voxel's number), writes each brick's base, each voxel's brick slot
// (voxel_slot [vcap]) and whatever init(v) sets up for voxel v < vcap.
template <class MaskOf, class Init>
__device__ __forceinline__ void brick_number(const int64_t* __restrict__ keys, const MaskOf& mask_of,
                                             int32_t* __restrict__ base, int64_t slots, int* counter,
                                             int32_t* __restrict__ voxel_slot, int64_t vcap, const Init& init) {
    __shared__ int sm[33];
    __shared__ int first;
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool used = s < slots && keys[s] != EMPTY_KEY;
    const int c = used ? popc64(mask_of((int)s)) : 0;
    int tot;
    const int r = block_excl(c, sm, &tot);
    if (tot == 0) return;
    if (threadIdx.x == 0) first = atomicAdd(counter, tot);
    __syncthreads();
    if (used) {
        base[s] = first + r;
        for (int k = 0; k < c; ++k)
            if (first + r + k < vcap) voxel_slot[first + r + k] = (int)s;
    }
    for (int k = threadIdx.x; k < tot; k += blockDim.x)
        if (first + k < vcap) init((int64_t)first + k);
}

}  // namespace lw
