// Broad phase of a world step: collider world AABBs and the fat-AABB update
// (reference src/systems/BroadPhaseSystem.cpp:155-185,
// src/collision/shapes/CollisionShape.cpp:54-90, SphereShape.cpp:49-58,
// src/collision/broadphase/DynamicAABBTree.cpp:186-214), and the set of
// overlapping pairs of fat AABBs with the pair filters of
// CollisionDetectionSystem::updateOverlappingPairs (:270-343).
//
// The reference keeps the fat AABBs in an incrementally balanced tree and
// queries it for the colliders that moved; the pairs it holds after each step
// are exactly the pairs of overlapping fat AABBs that pass the filters (a
// pair is created or dropped only when one of its colliders is reinserted,
// which is when its fat AABB changes).  Here that set is computed directly,
// two ways:
//   - LBVH (the default): 30-bit Morton codes of the fat-AABB centres with
//     the group (world) in the bits above, an LSD radix sort, the radix tree
//     over the sorted keys (ties broken by sorted position) built and boxed
//     bottom-up in one pass, and one walk per collider (32 Morton-consecutive
//     ones a warp) that looks for partners later in the sorted order, so each
//     pair is found once; the partners found are kept and written out at the
//     collider's offset by a second kernel;
//   - sort and sweep along one axis: an LSD radix sort of the colliders by
//     (group, fat min on the sweep axis), then each collider scans forward
//     while the next minimum is within its maximum.
// Both give the output in a deterministic order.
#include <cuda_runtime.h>

#include "broadphase_launch.h"
#include "rp3dg_math.cuh"
#include "shape_aabb.cuh"

namespace rp3dg {

namespace {

// ---- world AABB + fat AABB update, one collider per thread --------------
__global__ void __launch_bounds__(128) bp_update_kernel(const BpArgs a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n_update) return;
    if (a.enabled && !a.enabled[i]) {
        a.moved[i] = 0;
        return;
    }
    const int32_t si = a.shape[i];
    if (uint32_t(si) >= a.nb_shapes) {
        atomicOr(a.error, 1u);
        a.moved[i] = 0;
        return;
    }
    const rp3dg_shape s = a.shapes[si];
    const float4 p4 = a.wpos[i], q4 = a.wori[i];
    v3 amin, amax;
    shape_transformed_aabb(s.kind, s.params[0], a.bounds[2 * si], a.bounds[2 * si + 1],
                           X(V(p4.x, p4.y, p4.z), Q(q4.x, q4.y, q4.z, q4.w)), amin, amax);
    // DynamicAABBTree::updateObject: keep the fat AABB while it contains the
    // new one (AABB::contains), else inflate the new one by 4% of its extent
    // on each side (DYNAMIC_TREE_FAT_AABB_INFLATE_PERCENTAGE 0.08 x 0.5)
    const float4 fmn = a.fat_min[i], fmx = a.fat_max[i];
    const bool inside = fmn.x <= amin.x && fmn.y <= amin.y && fmn.z <= amin.z && fmx.x >= amax.x &&
                        fmx.y >= amax.y && fmx.z >= amax.z;
    const bool force = a.force && a.force[i];
    if (!force && inside) {
        a.moved[i] = 0;
        return;
    }
    const v3 ext = V(amax.x - amin.x, amax.y - amin.y, amax.z - amin.z);
    const v3 gap = V(0.5f * (0.08f * ext.x), 0.5f * (0.08f * ext.y), 0.5f * (0.08f * ext.z));
    a.fat_min[i] = make_float4(amin.x - gap.x, amin.y - gap.y, amin.z - gap.z, 0.0f);
    a.fat_max[i] = make_float4(amax.x + gap.x, amax.y + gap.y, amax.z + gap.z, 0.0f);
    a.moved[i] = 1;
}

// Exclusive scan of n uint32 in place, one block of 1024 threads (each
// thread scans a contiguous segment).
__global__ void __launch_bounds__(1024) scan_small(uint32_t* __restrict__ v, uint32_t n, uint32_t* __restrict__ total) {
    __shared__ uint32_t part[1024];
    const uint32_t per = (n + 1023) / 1024;
    const uint32_t b = threadIdx.x * per, e = b + per < n ? b + per : n;
    uint32_t s = 0;
    for (uint32_t i = b; i < e; i++) s += v[i];
    part[threadIdx.x] = s;
    __syncthreads();
    for (uint32_t off = 1; off < 1024; off <<= 1) {
        const uint32_t x = threadIdx.x >= off ? part[threadIdx.x - off] : 0u;
        __syncthreads();
        part[threadIdx.x] += x;
        __syncthreads();
    }
    uint32_t run = threadIdx.x ? part[threadIdx.x - 1] : 0u;
    for (uint32_t i = b; i < e; i++) {
        const uint32_t x = v[i];
        v[i] = run;
        run += x;
    }
    if (total && threadIdx.x == 1023) *total = part[1023];
}

// ---- radix sort of 64-bit keys with 32-bit values (LSD, 10-bit digits) ---
//
// Two kernels a pass: digit counts per tile of 2,048 keys (tile-major), and a
// scatter whose blocks add up the counts of the tiles before theirs
// themselves: a row of 1,024 counts a tile, read coalesced, 49 rows for
// 100,000 keys (a one-block scan between the two took 17 us a pass).  Above
// SORT_SUM_TILES tiles, where the rows read grow with the square, a kernel
// turns the counts into running sums first.  Ten bits make three passes of a
// 30-bit Morton code: 18 us a pass for 100,000 keys, latency of the rows and
// of the ranking; tiles of 1,024 keys took 23.
constexpr int SORT_BITS = 10;
constexpr uint32_t SORT_RADIX = 1u << SORT_BITS;
constexpr int SORT_THREADS = 256;
constexpr int SORT_ITEMS = 8;
constexpr uint32_t SORT_TILE = SORT_THREADS * SORT_ITEMS;   // 2048 keys per block
constexpr int SORT_WARPS = SORT_THREADS / 32;
constexpr uint32_t SORT_SUM_TILES = 512;
static_assert(SORT_RADIX == 4 * SORT_THREADS, "four digits a thread");

RD uint32_t digit_of(unsigned long long k, int shift) { return uint32_t(k >> shift) & (SORT_RADIX - 1u); }

__global__ void __launch_bounds__(SORT_THREADS) sort_hist(const unsigned long long* __restrict__ keys, uint32_t n,
                                                          int shift, uint32_t* __restrict__ hist) {
    __shared__ __align__(16) uint32_t h[SORT_RADIX];
    for (uint32_t d = threadIdx.x; d < SORT_RADIX; d += SORT_THREADS) h[d] = 0;
    __syncthreads();
    const uint32_t base = blockIdx.x * SORT_TILE;
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; k++) {
        const uint32_t idx = base + k * SORT_THREADS + threadIdx.x;
        if (idx < n) atomicAdd(&h[digit_of(keys[idx], shift)], 1u);
    }
    __syncthreads();
    reinterpret_cast<uint4*>(hist + size_t(blockIdx.x) * SORT_RADIX)[threadIdx.x] = reinterpret_cast<uint4*>(h)[threadIdx.x];
}

// Many tiles: each digit's counts become running sums over the tiles, its
// total goes to `totals`; one digit a thread.
__global__ void __launch_bounds__(32) sort_tile_sums(uint32_t* __restrict__ hist, uint32_t ntiles, uint32_t* __restrict__ totals) {
    const uint32_t d = blockIdx.x * 32u + threadIdx.x;
    uint32_t run = 0;
#pragma unroll 8
    for (uint32_t t = 0; t < ntiles; t++) {
        const uint32_t v = hist[size_t(t) * SORT_RADIX + d];
        hist[size_t(t) * SORT_RADIX + d] = run;
        run += v;
    }
    totals[d] = run;
}

// Stable scatter: each warp ranks its 256 consecutive keys of the tile in
// order (lanes with equal digits via __match_any_sync), warps are ordered by
// the per-digit counts of the warps before them, tiles by the counts of the
// tiles before them.
template <bool SUMMED>
__global__ void __launch_bounds__(SORT_THREADS, 2) sort_scatter(const unsigned long long* __restrict__ keys_in,
                                                             const uint32_t* __restrict__ vals_in,
                                                             unsigned long long* __restrict__ keys_out,
                                                             uint32_t* __restrict__ vals_out, uint32_t n, int shift,
                                                             const uint32_t* __restrict__ hist, uint32_t ntiles,
                                                             const uint32_t* __restrict__ totals) {
    __shared__ uint16_t cnt[SORT_WARPS][SORT_RADIX];
    __shared__ __align__(16) uint32_t offs[SORT_RADIX];
    __shared__ uint32_t wsum[SORT_WARPS];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (uint32_t d = lane; d < SORT_RADIX; d += 32) cnt[warp][d] = 0;
    __syncwarp();
    const uint32_t base = blockIdx.x * SORT_TILE + warp * (SORT_ITEMS * 32);
    unsigned long long k_[SORT_ITEMS];
    uint32_t v_[SORT_ITEMS], rank[SORT_ITEMS], dg[SORT_ITEMS];
    const uint32_t lt = (1u << lane) - 1u;
    // this thread's four digits: keys before this tile, keys in all
    {
        const uint4* rows = reinterpret_cast<const uint4*>(hist) + threadIdx.x;
        uint4 pre = make_uint4(0, 0, 0, 0), tot = pre;
        if (SUMMED) {
            pre = rows[size_t(blockIdx.x) * (SORT_RADIX / 4)];
            tot = reinterpret_cast<const uint4*>(totals)[threadIdx.x];
        } else {
            // 16 rows in flight
            for (uint32_t t0 = 0; t0 < ntiles; t0 += 16) {
                uint4 v[16];
#pragma unroll
                for (uint32_t k = 0; k < 16; k++)
                    v[k] = t0 + k < ntiles ? rows[size_t(t0 + k) * (SORT_RADIX / 4)] : make_uint4(0, 0, 0, 0);
#pragma unroll
                for (uint32_t k = 0; k < 16; k++) {
                    const uint32_t m = t0 + k < blockIdx.x ? 0xffffffffu : 0u;
                    tot.x += v[k].x; tot.y += v[k].y; tot.z += v[k].z; tot.w += v[k].w;
                    pre.x += v[k].x & m; pre.y += v[k].y & m; pre.z += v[k].z & m; pre.w += v[k].w & m;
                }
            }
        }
        const uint32_t sum = tot.x + tot.y + tot.z + tot.w;
        uint32_t inc = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= uint32_t(o)) inc += x;
        }
        if (lane == 31) wsum[warp] = inc;
        __syncthreads();
        uint32_t run = inc - sum;
        for (uint32_t w = 0; w < warp; w++) run += wsum[w];
        uint4 o;
        o.x = run + pre.x; run += tot.x;
        o.y = run + pre.y; run += tot.y;
        o.z = run + pre.z; run += tot.z;
        o.w = run + pre.w;
        reinterpret_cast<uint4*>(offs)[threadIdx.x] = o;
    }
#pragma unroll
    for (int r = 0; r < SORT_ITEMS; r++) {
        const uint32_t idx = base + r * 32 + lane;
        k_[r] = idx < n ? keys_in[idx] : 0ull;
        v_[r] = idx < n ? vals_in[idx] : 0u;
    }
#pragma unroll
    for (int r = 0; r < SORT_ITEMS; r++) {
        const bool valid = base + r * 32 + lane < n;
        const uint32_t d = valid ? digit_of(k_[r], shift) : SORT_RADIX;
        dg[r] = d;
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        const uint32_t before = valid ? cnt[warp][d] : 0u;
        rank[r] = before + __popc(peers & lt);
        __syncwarp();
        if (valid && (peers & lt) == 0) cnt[warp][d] = uint16_t(before + __popc(peers));
        __syncwarp();
    }
    __syncthreads();
    // per digit: counts of the earlier warps of this block
    for (uint32_t d = threadIdx.x; d < SORT_RADIX; d += SORT_THREADS) {
        uint32_t run = 0;
        for (int w = 0; w < SORT_WARPS; w++) {
            const uint32_t c = cnt[w][d];
            cnt[w][d] = uint16_t(run);
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < SORT_ITEMS; r++) {
        const uint32_t d = dg[r];
        if (d < SORT_RADIX) {
            const uint32_t pos = offs[d] + cnt[warp][d] + rank[r];
            keys_out[pos] = k_[r];
            vals_out[pos] = v_[r];
        }
    }
}

// ---- sweep ---------------------------------------------------------------

// float -> unsigned key with the same order (negative floats reversed)
RD uint32_t ordered_bits(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__global__ void __launch_bounds__(128) sap_keys(const BpArgs a, int axis) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const float4 mn = a.fat_min[i];
    const float x = axis == 0 ? mn.x : (axis == 1 ? mn.y : mn.z);
    uint32_t g = a.group ? uint32_t(a.group[i]) : 0u;
    if (a.group_bits < 32 && (g >> a.group_bits) != 0u) {
        atomicOr(a.error, 8u);  // group outside 0..nb_groups-1: its pairs are not searched correctly
        g &= (1u << a.group_bits) - 1u;
    }
    a.keys[i] = (static_cast<unsigned long long>(g) << 32) | ordered_bits(x);
    a.vals[i] = i;
}

// Sorted copies of what the sweep reads, sweep axis first.
__global__ void __launch_bounds__(128) sap_gather(const BpArgs a, int axis) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n) return;
    const uint32_t i = a.vals[p];
    const float4 mn = a.fat_min[i], mx = a.fat_max[i];
    float4 lo = mn, hi = mx;
    if (axis == 1) { lo = make_float4(mn.y, mn.x, mn.z, 0.0f); hi = make_float4(mx.y, mx.x, mx.z, 0.0f); }
    if (axis == 2) { lo = make_float4(mn.z, mn.y, mn.x, 0.0f); hi = make_float4(mx.z, mx.y, mx.x, 0.0f); }
    lo.w = __int_as_float(a.body[i]);
    const uint32_t cat = a.category ? a.category[i] : 0xffffu;
    const uint32_t msk = a.mask ? a.mask[i] : 0xffffu;
    hi.w = __uint_as_float((cat << 16) | msk);
    a.s_lo[p] = lo;
    a.s_hi[p] = hi;
    a.s_group[p] = a.group ? a.group[i] : 0;
}

template <bool WRITE>
__global__ void __launch_bounds__(128) sap_sweep(const BpArgs a) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n) return;
    const float4 lo = a.s_lo[p], hi = a.s_hi[p];
    const int32_t g = a.s_group[p];
    const int32_t body = __float_as_int(lo.w);
    const uint32_t bits = __float_as_uint(hi.w);
    const uint32_t cat = bits >> 16, msk = bits & 0xffffu;
    uint32_t count = 0;
    uint32_t out = WRITE ? a.pair_offset[p] : 0u;
    const uint32_t ci = WRITE ? a.vals[p] : 0u;
    for (uint32_t q = p + 1; q < a.n; q++) {
        const float4 lo2 = a.s_lo[q];
        if (lo2.x > hi.x || a.s_group[q] != g) break;   // sorted by (group, min): nothing further overlaps
        const float4 hi2 = a.s_hi[q];
        // AABB::testCollision (AABB.h:179-187) on the two other axes
        if (hi.y < lo2.y || hi2.y < lo.y) continue;
        if (hi.z < lo2.z || hi2.z < lo.z) continue;
        if (__float_as_int(lo2.w) == body) continue;            // same body
        const uint32_t bits2 = __float_as_uint(hi2.w);
        if ((msk & (bits2 >> 16)) == 0u || (cat & (bits2 & 0xffffu)) == 0u) continue;
        if (WRITE) {
            if (out < a.capacity) {
                const uint32_t cj = a.vals[q];
                a.pairs[2 * out] = int32_t(ci < cj ? ci : cj);
                a.pairs[2 * out + 1] = int32_t(ci < cj ? cj : ci);
            }
            out++;
        } else {
            count++;
        }
    }
    if (!WRITE) a.pair_offset[p] = count;
}

uint32_t blocks128(uint32_t n) { return (n + 127) / 128; }

// ---- LBVH -----------------------------------------------------------------

RD float3 aabb_centre(const float4 mn, const float4 mx) {
    return make_float3(0.5f * (mn.x + mx.x), 0.5f * (mn.y + mx.y), 0.5f * (mn.z + mx.z));
}

// Scene bounds of the centres, as ordered bits: maxima in [3..5], minima
// complemented in [0..2] (so that zero is the start of both).  A few blocks
// with one atomic a value each: with one a warp, 100,000 centres queued 19,000
// atomics on six words (15 us).
constexpr uint32_t BOUNDS_BLOCKS = 148;
__global__ void __launch_bounds__(256) lbvh_bounds(const BpArgs a, uint32_t* __restrict__ bounds) {
    __shared__ uint32_t part[8][6];
    uint32_t m[6] = {0u, 0u, 0u, 0u, 0u, 0u};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
        const float3 c = aabb_centre(a.fat_min[i], a.fat_max[i]);
        const uint32_t x = ordered_bits(c.x), y = ordered_bits(c.y), z = ordered_bits(c.z);
        m[0] = max(m[0], ~x); m[1] = max(m[1], ~y); m[2] = max(m[2], ~z);
        m[3] = max(m[3], x); m[4] = max(m[4], y); m[5] = max(m[5], z);
    }
    for (int k = 0; k < 6; k++) {
        m[k] = __reduce_max_sync(0xffffffffu, m[k]);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5][k] = m[k];
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        uint32_t v = 0;
        for (int w = 0; w < 8; w++) v = max(v, part[w][threadIdx.x]);
        atomicMax(bounds + threadIdx.x, v);
    }
}

RD float from_ordered_bits(uint32_t u) { return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u); }

// 10 bits per axis spread to every third bit
RD uint32_t spread3(uint32_t v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

RD uint32_t quantize10(float x, float lo, float inv) {
    float q = (x - lo) * inv;
    q = q < 0.0f ? 0.0f : (q > 1023.0f ? 1023.0f : q);   // NaN centres land in cell 0
    return uint32_t(q);
}

__global__ void __launch_bounds__(128) lbvh_keys(const BpArgs a, const uint32_t* __restrict__ bounds) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    float lo[3], inv[3];
    for (int k = 0; k < 3; k++) {
        lo[k] = from_ordered_bits(~bounds[k]);
        const float ext = from_ordered_bits(bounds[3 + k]) - lo[k];
        inv[k] = ext > 0.0f ? 1023.0f / ext : 0.0f;
    }
    const float3 c = aabb_centre(a.fat_min[i], a.fat_max[i]);
    const uint32_t m = (spread3(quantize10(c.x, lo[0], inv[0])) << 2) | (spread3(quantize10(c.y, lo[1], inv[1])) << 1) |
                       spread3(quantize10(c.z, lo[2], inv[2]));
    uint32_t g = a.group ? uint32_t(a.group[i]) : 0u;
    if (a.group_bits < 32 && (g >> a.group_bits) != 0u) {
        atomicOr(a.error, 8u);  // group outside 0..nb_groups-1
        g &= (1u << a.group_bits) - 1u;
    }
    a.keys[i] = (static_cast<unsigned long long>(g) << 30) | m;
    a.vals[i] = i;
}

// The radix tree over the sorted keys, bottom-up in one pass (after Apetrei,
// "Fast and Simple Agglomerative LBVH Construction", 2014): a leaf's thread
// walks up, and joins the range it covers, [l, r], with the neighbour it
// shares the longer prefix with.  Internal node s lies between the sorted
// positions s and s + 1.  A child leaves its box, its id (leaf at sorted
// position p: n - 1 + p) and its last position in its half of the parent's
// record; the first to arrive stops, the second goes on with both (the other
// half was written before the fence that precedes the counter's increment).
// Equal prefixes of equal keys are told apart by the positions.
__global__ void __launch_bounds__(128) lbvh_build(const unsigned long long* __restrict__ keys, const float4* __restrict__ s_lo,
                                                  const float4* __restrict__ s_hi, uint32_t n, LbvhNode* __restrict__ nodes,
                                                  uint32_t* __restrict__ first, uint32_t* __restrict__ visits,
                                                  uint32_t* __restrict__ root) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n || n < 2) return;
    uint32_t l = p, r = p;
    int32_t id = int32_t(n) - 1 + int32_t(p);
    float4 lo = s_lo[p], hi = s_hi[p];
    unsigned long long kl = keys[p], kr = kl;
    while (l != 0 || r != n - 1) {
        bool right;   // join the neighbour on the right
        if (l == 0) right = true;
        else if (r == n - 1) right = false;
        else {
            const unsigned long long xr = kr ^ keys[r + 1], xl = keys[l - 1] ^ kl;
            right = xr != xl ? xr < xl : (r ^ (r + 1)) < ((l - 1) ^ l);
        }
        const uint32_t parent = right ? r : l - 1;
        LbvhNode* nd = nodes + parent;
        lo.w = __int_as_float(id);
        hi.w = __int_as_float(int32_t(r));
        __stcg(right ? &nd->lo0 : &nd->lo1, lo);
        __stcg(right ? &nd->hi0 : &nd->hi1, hi);
        if (right) __stcg(first + parent, l);
        __threadfence();
        if (atomicAdd(visits + parent, 1u) == 0u) return;
        __threadfence();
        const float4 olo = __ldcg(right ? &nd->lo1 : &nd->lo0), ohi = __ldcg(right ? &nd->hi1 : &nd->hi0);
        if (right) {
            r = uint32_t(__float_as_int(ohi.w));
            kr = keys[r];
        } else {
            l = __ldcg(first + parent);
            kl = keys[l];
        }
        lo = make_float4(fminf(lo.x, olo.x), fminf(lo.y, olo.y), fminf(lo.z, olo.z), 0.0f);
        hi = make_float4(fmaxf(hi.x, ohi.x), fmaxf(hi.y, ohi.y), fmaxf(hi.z, ohi.z), 0.0f);
        id = int32_t(parent);
    }
    *root = uint32_t(id);
}

constexpr int LBVH_STACK = 128;   // > the deepest tree 96-bit keys can give
// A warp in which LBVH_DENSE_LANES colliders have LBVH_DENSE partners walks for
// those together.  20,000 colliders in clumps of 100, 300, 500, 5,000, us: a walk
// each 394, 948, 1,425, 13,300; together 446, 630, 922, 6,500 (the walks given up
// at 64 partners are what the first loses); given up at 48 or 32, clumps of 50 to
// 70 lose as much (265 -> 273, 300).
constexpr uint32_t LBVH_DENSE = 64, LBVH_DENSE_LANES = 4;
constexpr uint32_t LBVH_BLOCK = 128;
// Up to this many blocks the writing kernel's blocks add up the totals before
// theirs; above it they are scanned first.
constexpr uint32_t LBVH_SUM_BLOCKS = 2048;

// AABB::testCollision (AABB.h:179-187): inclusive on every axis
RD bool aabb_overlap(const float4 alo, const float4 ahi, const float4 blo, const float4 bhi) {
    if (ahi.x < blo.x || bhi.x < alo.x) return false;
    if (ahi.y < blo.y || bhi.y < alo.y) return false;
    if (ahi.z < blo.z || bhi.z < alo.z) return false;
    return true;
}

// A collider that looks for partners: its box, filters and group.
struct LbvhQuery {
    float4 lo, hi;
    int32_t body, g;
    uint32_t cat, msk;
    uint32_t end;   // last position of the group
    RD LbvhQuery(const BpArgs& a, uint32_t p) {
        const uint32_t n = a.n;
        lo = a.s_lo[p];
        hi = a.s_hi[p];
        body = __float_as_int(lo.w);
        const uint32_t bits = __float_as_uint(hi.w);
        cat = bits >> 16;
        msk = bits & 0xffffu;
        g = 0;
        end = n - 1;
        if (a.group) {
            g = a.s_group[p];
            uint32_t l = p, h = n - 1;
            while (l < h) {
                const uint32_t m = l + (h - l + 1) / 2;
                if (a.s_group[m] > g) h = m - 1;
                else l = m;
            }
            end = l;
        }
    }
    // the filters of the collider at position j, whose box overlaps
    RD bool accepts(const BpArgs& a, uint32_t j, float4 lo2, float4 hi2) const {
        const uint32_t bits2 = __float_as_uint(hi2.w);
        return __float_as_int(lo2.w) != body && (msk & (bits2 >> 16)) != 0u && (cat & (bits2 & 0xffffu)) != 0u &&
               (!a.group || a.s_group[j] == g);
    }
};

// The partners of the collider at sorted position p that lie behind it, in
// ascending position: the walk takes left children first, and both children
// of a node are tested from its one record.  With groups only positions up to
// the group's end are looked at. `found` answers whether to go on.
template <class Found>
RD void lbvh_walk(const BpArgs& a, uint32_t p, uint32_t root, Found found) {
    const int32_t nl = int32_t(a.n) - 1;
    const LbvhQuery q(a, p);
    auto leaf = [&](uint32_t j) { return !q.accepts(a, j, a.s_lo[j], a.s_hi[j]) || found(j); };
    int32_t stack[LBVH_STACK];
    int sp = 0;
    int32_t node = int32_t(root);
    for (;;) {
        if (node < 0) {
            if (sp == 0) break;
            node = stack[--sp];
            if (node >= nl) {
                if (!leaf(uint32_t(node - nl))) break;
                node = -1;
                continue;
            }
        }
        const LbvhNode* nd = a.lbvh_nodes + node;
        const float4 lo0 = nd->lo0, hi0 = nd->hi0, lo1 = nd->lo1, hi1 = nd->hi1;
        const int32_t c0 = __float_as_int(lo0.w), last0 = __float_as_int(hi0.w), c1 = __float_as_int(lo1.w);
        const int32_t last1 = __float_as_int(hi1.w);
        const bool hit0 = last0 > int32_t(p) && aabb_overlap(q.lo, q.hi, lo0, hi0);
        const bool hit1 = last1 > int32_t(p) && uint32_t(last0) < q.end && aabb_overlap(q.lo, q.hi, lo1, hi1);
        node = -1;
        if (hit0 && c0 >= nl && !leaf(uint32_t(c0 - nl))) break;
        if (hit0 && c0 < nl) {
            node = c0;
            if (hit1) {
                if (sp == LBVH_STACK) {
                    atomicOr(a.error, 16u);   // cannot happen for trees of 96-bit keys
                    break;
                }
                stack[sp++] = c1;
            }
        } else if (hit1) {
            if (c1 < nl) node = c1;
            else if (!leaf(uint32_t(c1 - nl))) break;
        }
    }
}

// The same for the active colliders of a warp together, on one stack whose
// entries carry the lanes that want them: each lane meets the nodes of its own
// walk, and the lanes that meet one share its read.  For colliders with many
// partners, whose own walks part at every leaf: 2,000 colliders that all
// overlap took 5.6 ms with a walk each, 2.8 so.
template <class Found>
RD void lbvh_packet(const BpArgs& a, uint32_t p, bool active, uint32_t root, int2* stack, Found found) {
    const int32_t nl = int32_t(a.n) - 1;
    const uint32_t lane = threadIdx.x & 31u;
    const LbvhQuery q(a, active ? p : 0u);
    const uint32_t want = __ballot_sync(0xffffffffu, active);
    auto leaf = [&](uint32_t j, uint32_t lanes) {
        if ((lanes >> lane & 1u) && q.accepts(a, j, a.s_lo[j], a.s_hi[j])) found(j);
    };
    __syncwarp();
    if (lane == 0) stack[0] = make_int2(int32_t(root), int32_t(want));
    int sp = want ? 1 : 0;
    while (sp > 0) {
        __syncwarp();
        const int2 top = stack[--sp];
        __syncwarp();
        if (top.x >= nl) {
            leaf(uint32_t(top.x - nl), uint32_t(top.y));
            continue;
        }
        const LbvhNode* nd = a.lbvh_nodes + top.x;
        const float4 lo0 = nd->lo0, hi0 = nd->hi0, lo1 = nd->lo1, hi1 = nd->hi1;
        const int32_t c0 = __float_as_int(lo0.w), last0 = __float_as_int(hi0.w), c1 = __float_as_int(lo1.w);
        const int32_t last1 = __float_as_int(hi1.w);
        const bool mine = (uint32_t(top.y) >> lane & 1u) != 0u;
        const uint32_t m0 = __ballot_sync(0xffffffffu, mine && last0 > int32_t(p) && aabb_overlap(q.lo, q.hi, lo0, hi0));
        const uint32_t m1 = __ballot_sync(0xffffffffu, mine && last1 > int32_t(p) && uint32_t(last0) < q.end &&
                                                           aabb_overlap(q.lo, q.hi, lo1, hi1));
        if (m0 && c0 >= nl) leaf(uint32_t(c0 - nl), m0);
        const int push1 = m1 ? 1 : 0, push0 = m0 && c0 < nl ? 1 : 0;
        if (sp + 2 > LBVH_STACK) {
            if (lane == 0) atomicOr(a.error, 16u);   // cannot happen for trees of 96-bit keys
            break;
        }
        if (lane == 0) {
            if (push1) stack[sp] = make_int2(c1, int32_t(m1));
            if (push0) stack[sp + push1] = make_int2(c0, int32_t(m0));
        }
        sp += push0 + push1;
    }
    __syncwarp();
}

// Bound: the latency of the dependent node reads.  100,000 colliders: 44 us,
// plus 9 to write the pairs (a count and a write walk of 32-lane packets took
// 138 + 137 us, the whole search 560 us; 174 now).
//
// Search: a collider's partners, the first LBVH_KEEP of them to `found`
// (entry k of position p at k * n + p), their number to pair_offset[p], each
// block's total to block_pairs.  A walk that finds LBVH_DENSE partners is given
// up, and its collider's partners counted with the warp's other dense ones.
__global__ void __launch_bounds__(LBVH_BLOCK) lbvh_search(const BpArgs a) {
    __shared__ int2 stack[LBVH_BLOCK / 32][LBVH_STACK];
    const uint32_t p = blockIdx.x * LBVH_BLOCK + threadIdx.x;
    uint32_t count = 0;
    bool dense = false;
    if (p < a.n && a.n >= 2)
        lbvh_walk(a, p, *a.lbvh_root, [&](uint32_t j) {
            if (count < LBVH_KEEP) a.lbvh_found[size_t(count) * a.n + p] = j;
            dense = ++count == LBVH_DENSE;
            return !dense;
        });
    const uint32_t dense_lanes = uint32_t(__popc(__ballot_sync(0xffffffffu, dense)));
    if (dense_lanes) {
        uint32_t all = 0;
        if (dense_lanes >= LBVH_DENSE_LANES)
            lbvh_packet(a, p, dense, *a.lbvh_root, stack[threadIdx.x >> 5], [&](uint32_t) { all++; });
        else if (dense)
            lbvh_walk(a, p, *a.lbvh_root, [&](uint32_t) { all++; return true; });
        if (dense) count = all;
    }
    if (p < a.n) a.pair_offset[p] = count;
    __shared__ uint32_t part[LBVH_BLOCK / 32];
    const uint32_t sum = __reduce_add_sync(0xffffffffu, count);
    if ((threadIdx.x & 31u) == 0) part[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (uint32_t w = 0; w < LBVH_BLOCK / 32; w++) t += part[w];
        a.block_pairs[blockIdx.x] = t;
    }
}

// The pairs in order of sorted position: every block adds up the totals of
// the blocks before it (SCANNED: they are running sums already), scans its
// own counts and writes its pairs; a collider with more than LBVH_KEEP
// partners walks again for the rest, the colliders of a warp together when
// enough of them are dense.
template <bool SCANNED>
__global__ void __launch_bounds__(LBVH_BLOCK) lbvh_emit(const BpArgs a) {
    __shared__ uint32_t part[LBVH_BLOCK / 32], s_base;
    __shared__ int2 stack[LBVH_BLOCK / 32][LBVH_STACK];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t p = blockIdx.x * LBVH_BLOCK + threadIdx.x;
    if (SCANNED) {
        if (threadIdx.x == 0) s_base = a.block_pairs[blockIdx.x];
    } else {
        uint32_t before = 0;
        for (uint32_t b = threadIdx.x; b < blockIdx.x; b += LBVH_BLOCK) before += a.block_pairs[b];
        before = __reduce_add_sync(0xffffffffu, before);
        if (lane == 0) part[warp] = before;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t t = 0;
            for (uint32_t w = 0; w < LBVH_BLOCK / 32; w++) t += part[w];
            s_base = t;
        }
        __syncthreads();
    }
    const uint32_t count = p < a.n ? a.pair_offset[p] : 0u;
    uint32_t inc = count;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= uint32_t(o)) inc += x;
    }
    if (lane == 31) part[warp] = inc;
    __syncthreads();
    uint32_t out = s_base + inc - count;
    for (uint32_t w = 0; w < warp; w++) out += part[w];
    if (!SCANNED && blockIdx.x == gridDim.x - 1 && threadIdx.x == LBVH_BLOCK - 1) *a.pair_count = out + count;
    if (!__any_sync(0xffffffffu, count != 0)) return;
    const uint32_t ci = a.vals[p < a.n ? p : a.n - 1];
    auto put = [&](uint32_t j) {
        if (out < a.capacity) {
            const uint32_t cj = a.vals[j];
            a.pairs[2 * size_t(out)] = int32_t(ci < cj ? ci : cj);
            a.pairs[2 * size_t(out) + 1] = int32_t(ci < cj ? cj : ci);
        }
        out++;
    };
    for (uint32_t k = 0; k < count && k < LBVH_KEEP; k++) put(a.lbvh_found[size_t(k) * a.n + p]);
    uint32_t k = 0;
    if (uint32_t(__popc(__ballot_sync(0xffffffffu, count >= LBVH_DENSE))) >= LBVH_DENSE_LANES) {
        lbvh_packet(a, p, count > LBVH_KEEP, *a.lbvh_root, stack[warp], [&](uint32_t j) {
            if (k++ >= LBVH_KEEP) put(j);
        });
    } else if (count > LBVH_KEEP) {
        lbvh_walk(a, p, *a.lbvh_root, [&](uint32_t j) {
            if (k++ >= LBVH_KEEP) put(j);
            return true;
        });
    }
}

}  // namespace

cudaError_t launch_bp_update(const BpArgs& a, cudaStream_t s, uint64_t* launches) {
    if (a.n_update == 0) return cudaSuccess;
    bp_update_kernel<<<blocks128(a.n_update), 128, 0, s>>>(a);
    (*launches)++;
    return cudaGetLastError();
}

size_t sort_scratch_words(uint32_t n) { return size_t(SORT_RADIX) * ((n + SORT_TILE - 1) / SORT_TILE + 1); }
size_t lbvh_block_words(uint32_t n) { return (n + LBVH_BLOCK - 1) / LBVH_BLOCK; }

cudaError_t launch_exclusive_scan(uint32_t* v, uint32_t n, uint32_t* total, cudaStream_t s) {
    if (n == 0) return total ? cudaMemsetAsync(total, 0, sizeof(uint32_t), s) : cudaSuccess;
    scan_small<<<1, 1024, 0, s>>>(v, n, total);
    return cudaGetLastError();
}

cudaError_t launch_bp_pairs(const BpArgs& a, int axis, cudaStream_t s, uint64_t* launches) {
    if (a.n == 0) return cudaMemsetAsync(a.pair_count, 0, sizeof(uint32_t), s);
    const bool lbvh = axis < 0;
    if (lbvh) {
        // centre bounds, then the visit counters
        const cudaError_t e = cudaMemsetAsync(a.lbvh_bounds, 0, (8 + size_t(a.n)) * sizeof(uint32_t), s);
        if (e != cudaSuccess) return e;
        const uint32_t nb = (a.n + 255) / 256;
        lbvh_bounds<<<nb < BOUNDS_BLOCKS ? nb : BOUNDS_BLOCKS, 256, 0, s>>>(a, a.lbvh_bounds);
        lbvh_keys<<<blocks128(a.n), 128, 0, s>>>(a, a.lbvh_bounds);
        *launches += 2;
    } else {
        sap_keys<<<blocks128(a.n), 128, 0, s>>>(a, axis);
        (*launches)++;
    }
    // radix sort: (group, Morton code) = 30 + group bits, or (group, min) =
    // 32 float bits + the group bits in use
    const uint32_t ntiles = (a.n + SORT_TILE - 1) / SORT_TILE;
    uint32_t* totals = a.sort_hist + size_t(ntiles) * SORT_RADIX;
    unsigned long long *kin = a.keys, *kout = a.keys_tmp;
    uint32_t *vin = a.vals, *vout = a.vals_tmp;
    const int end_bit = (lbvh ? 30 : 32) + a.group_bits;
    for (int shift = 0; shift < end_bit; shift += SORT_BITS) {
        sort_hist<<<ntiles, SORT_THREADS, 0, s>>>(kin, a.n, shift, a.sort_hist);
        if (ntiles > SORT_SUM_TILES) {
            sort_tile_sums<<<SORT_RADIX / 32, 32, 0, s>>>(a.sort_hist, ntiles, totals);
            sort_scatter<true><<<ntiles, SORT_THREADS, 0, s>>>(kin, vin, kout, vout, a.n, shift, a.sort_hist, ntiles, totals);
            (*launches)++;
        } else {
            sort_scatter<false><<<ntiles, SORT_THREADS, 0, s>>>(kin, vin, kout, vout, a.n, shift, a.sort_hist, ntiles, nullptr);
        }
        *launches += 2;
        unsigned long long* tk = kin; kin = kout; kout = tk;
        uint32_t* tv = vin; vin = vout; vout = tv;
    }
    BpArgs b = a;
    b.keys = kin;
    b.vals = vin;
    sap_gather<<<blocks128(a.n), 128, 0, s>>>(b, lbvh ? 0 : axis);
    *launches += 1;
    if (lbvh) {
        if (a.n > 1) {
            lbvh_build<<<blocks128(a.n), 128, 0, s>>>(kin, b.s_lo, b.s_hi, a.n, a.lbvh_nodes, a.lbvh_first, a.lbvh_visits,
                                                      a.lbvh_root);
            (*launches)++;
        }
        const uint32_t nb = uint32_t(lbvh_block_words(a.n));
        lbvh_search<<<nb, LBVH_BLOCK, 0, s>>>(b);
        if (nb > LBVH_SUM_BLOCKS) {
            scan_small<<<1, 1024, 0, s>>>(b.block_pairs, nb, a.pair_count);
            lbvh_emit<true><<<nb, LBVH_BLOCK, 0, s>>>(b);
            (*launches)++;
        } else {
            lbvh_emit<false><<<nb, LBVH_BLOCK, 0, s>>>(b);
        }
        *launches += 2;
        return cudaGetLastError();
    }
    sap_sweep<false><<<blocks128(a.n), 128, 0, s>>>(b);
    scan_small<<<1, 1024, 0, s>>>(b.pair_offset, a.n, a.pair_count);
    sap_sweep<true><<<blocks128(a.n), 128, 0, s>>>(b);
    *launches += 3;
    return cudaGetLastError();
}

}  // namespace rp3dg
