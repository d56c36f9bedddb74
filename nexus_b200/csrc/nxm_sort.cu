// Block activation and particle sort (src_mpm/grid/grid.rs:26-191,
// src_mpm_shaders/grid/sort.rs:104-491, src_mpm_shaders/grid/grid.rs:447-578).
//
// Same results as the reference: the set of active blocks (every particle's
// 2x2x2 block neighbourhood), the per-block slab buckets (4 primary z-slabs,
// 6 extra buckets), the +1 neighbour header ids and the sorted id list.
//
// Inside a slab the particles are also grouped by associated cell (64 counters
// a block, z-major, so the slabs are runs of 16 cells): P2G takes a cell per
// lane and G2P's neighbouring lanes read the same halo nodes.
// Header order and the order inside a bucket come from atomics, as in the
// reference; the canonical pass (deterministic mode) orders every bucket by
// ascending particle id.  The extras (a particle listed again in each +1
// neighbour block its stencil reaches) are only built when asked for: the
// gather-form P2G reads them, the scatter-form P2G does not.
//
// B200 specifics: every particle pass is a persistent grid-stride loop that
// keeps whole warps together, so that __match_any_sync can merge the atomics
// of lanes that hit the same block (or the same block bucket): one hash probe
// or one atomicAdd per distinct key per warp instead of one per particle.
// The block key of each particle is cached in `pcode` (8 bytes) by the
// previous step's G2P, so activation does not re-read the particle
// records.  Counters, headers and the hash live in L2.
#include "nxm_device.cuh"
#include "nxm_kernels.h"

// k_count<false> / k_finalize<false> skip the extras loop by design.
#pragma nv_diag_suppress 128

namespace nxm {
namespace {

__device__ __forceinline__ void set_status(Counters* c, uint32_t bit) { atomicOr(&c->status, bit); }

__device__ __forceinline__ void assoc_shift(int i, int& dx, int& dy, int& dz) {
    // grid.rs:175-212 blocks_associated_to_block: z fastest.
    dx = (i >> 2) & 1;
    dy = (i >> 1) & 1;
    dz = i & 1;
}

// Insert `key` (block kx,ky,kz); allocates a header on first insertion.
// Primary blocks take ids [0, num_primary); neighbour-pass blocks take ids
// base + [0, num_extra) with base = num_primary.
__device__ void hash_insert(const DevPtrs& P, uint32_t key, int kx, int ky, int kz, bool primary, uint32_t base,
                            uint32_t hash_mask, uint32_t block_cap) {
    uint32_t slot = hash_key(key) & hash_mask;
    for (uint32_t it = 0; it <= hash_mask; ++it) {
        uint32_t cur = __ldcg(&P.hkey[slot]);
        if (cur == key) return;
        if (cur == NONE) {
            uint32_t old = atomicCAS(&P.hkey[slot], NONE, key);
            if (old == NONE) {
                uint32_t id = primary ? atomicAdd(&P.counters->num_primary, 1u)
                                      : base + atomicAdd(&P.counters->num_extra, 1u);
                if (id >= block_cap) {
                    set_status(P.counters, STATUS_BLOCK_CAPACITY);
                    P.hval[slot] = NONE;
                    return;
                }
                P.bvid[id] = make_int4(kx, ky, kz, (int)key);
                P.hval[slot] = id;
                return;
            }
            if (old == key) return;
        }
        slot = (slot + 1) & hash_mask;
    }
    set_status(P.counters, STATUS_HASH_FULL);
}

__device__ __forceinline__ uint32_t hash_find(const DevPtrs& P, uint32_t key, uint32_t hash_mask) {
    uint32_t slot = hash_key(key) & hash_mask;
    for (uint32_t it = 0; it <= hash_mask; ++it) {
        uint32_t cur = __ldg(&P.hkey[slot]);
        if (cur == key) return __ldg(&P.hval[slot]);
        if (cur == NONE) return NONE;
        slot = (slot + 1) & hash_mask;
    }
    return NONE;
}

// Warp-aggregated atomicAdd: lanes with equal `key` (NONE = no-op) share one
// atomic; each gets base + its rank among the equal lanes (lane order).
__device__ __forceinline__ uint32_t warp_agg_add(uint32_t key, uint32_t* addr) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t peers = __match_any_sync(0xFFFFFFFFu, key);
    uint32_t leader = __ffs(peers) - 1;
    uint32_t rank = __popc(peers & ((1u << lane) - 1u));
    uint32_t base = 0;
    if (key != NONE && lane == leader) base = atomicAdd(addr, (uint32_t)__popc(peers));
    base = __shfl_sync(peers, base, leader);
    return base + rank;
}

// Warp-aggregated atomicAdd without a result (fire-and-forget).
__device__ __forceinline__ void warp_agg_red(uint32_t key, uint32_t* addr) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, key);
    if (key != NONE && lane == (uint32_t)(__ffs(peers) - 1)) atomicAdd(addr, (uint32_t)__popc(peers));
}

// The contiguous particle range [lo, hi) of this warp (a multiple of 32 long):
// with particles stored in block order, a warp's consecutive passes mostly see
// the same block, which lets the passes below skip repeated hash work.
__device__ __forceinline__ void warp_range(uint32_t n, uint32_t& lo, uint32_t& hi) {
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t per_warp = ((n + nwarps - 1) / nwarps + 31u) & ~31u;
    lo = min(warp * per_warp, n);
    hi = min(lo + per_warp, n);
}

// kSortBatch (a template parameter of the particle passes): passes of 32
// particles whose loads a warp issues together (2, 4 or 8; tuned per state).

__device__ __forceinline__ bool spills(uint32_t ax, uint32_t ay, uint32_t az, int sx, int sy, int sz) {
    // sort.rs:320-329, EXTRA_PARTICLE_MIN_SHIFT = 2
    return (sx == 0 || ax >= 2) && (sy == 0 || ay >= 2) && (sz == 0 || az >= 2);
}
__device__ __forceinline__ uint32_t extra_bucket(uint32_t az, int sz) {
    // sort.rs:56-62
    int local = (int)az - sz * 4;
    if (local < -2) local = -2;
    return NUM_PRIMARY_BUCKETS + (uint32_t)(local + 2);
}

// ---------------------------------------------------------------------------

// Clears the hash and the step counters; the last CTA also refreshes the
// colliders' world centres of mass from their poses (rigid_impulses.rs:167-185),
// which the grid update reads.
__global__ void k_sort_reset(DevPtrs P, uint32_t hash_cap) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < hash_cap; i += gridDim.x * blockDim.x)
        P.hkey[i] = NONE;
    if (P.colliders && blockIdx.x == gridDim.x - 1) {
        const Params& prm = *P.params;
        const uint32_t ncol = prm.scene_blocks ? prm.ncol : min(prm.ncol, (uint32_t)MAX_COLLIDERS);
        for (uint32_t i = threadIdx.x; i < ncol; i += blockDim.x) {
            DevCollider& c = P.colliders[i];
            const quat q = quat{c.rot[0], c.rot[1], c.rot[2], c.rot[3]};
            const v3 com = qrot(q, mk(c.local_com[0], c.local_com[1], c.local_com[2])) + mk(c.tra[0], c.tra[1], c.tra[2]);
            c.com[0] = com.x; c.com[1] = com.y; c.com[2] = com.z;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        P.counters->num_primary = 0;
        P.counters->num_extra = 0;
        P.counters->num_blocks = 0;
        P.counters->sorted_len = 0;
        P.counters->unsorted = 0;
        P.counters->rigid_len = 0;
        P.counters->p2g_next = 0;
    }
}

// sort.rs:104-121 gpu_touch_primary_blocks.  Block keys come from the cache
// written by the previous step (or from the positions after an upload).
// Each warp walks a contiguous range of particles, so consecutive passes
// mostly see the block they inserted last: a pass whose lanes all carry the
// key inserted by the previous pass skips the hash entirely.
template <int kSortBatch>
__global__ void __launch_bounds__(256) k_touch_primary(DevPtrs P) {
    after_previous();
    const uint32_t n = P.params->n;
    const float dx = P.params->dx;
    const uint32_t hmask = P.params->hash_capacity - 1;
    const uint32_t bcap = P.params->block_capacity;
    const bool cached = P.counters->codes_valid != 0;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t lo, hi;
    warp_range(n, lo, hi);
    uint32_t known = NONE;  // a key this warp has already inserted
    for (uint32_t base = lo; base < hi; base += 32u * kSortBatch) {
        uint32_t keys[kSortBatch];
#pragma unroll
        for (int j = 0; j < kSortBatch; ++j) {
            const uint32_t p = base + 32u * j + lane;
            uint32_t key = NONE;
            if (p < hi) {
                if (cached) {
                    key = __ldg(&P.pcode[p].x);
                } else {
                    float4 xm = __ldg(reinterpret_cast<const float4*>(&P.in.kin[p]));
                    CellInfo ci = cell_info(dx, mk(xm.x, xm.y, xm.z));
                    int3 o = make_int3(0, 0, 0);
                    if (P.params->scene_blocks) o = scene_base_of(*P.params, P.pscene[P.pid_in ? P.pid_in[p] : p]);
                    key = pack_key(ci.bx + o.x, ci.by + o.y, ci.bz + o.z);
                    P.pcode[p] = make_uint2(key, ci.ax | (ci.ay << 2) | (ci.az << 4));
                }
            }
            keys[j] = key;
        }
#pragma unroll
        for (int j = 0; j < kSortBatch; ++j) {
            const uint32_t b32 = base + 32u * j;
            if (b32 >= hi) break;
            const bool active = b32 + lane < hi;
            const uint32_t key = keys[j];
            const uint32_t need = (active && key != known) ? key : NONE;
            if (!__all_sync(0xFFFFFFFFu, need == NONE)) {
                const uint32_t peers = __match_any_sync(0xFFFFFFFFu, need);
                if (need != NONE && lane == (uint32_t)(__ffs(peers) - 1))
                    hash_insert(P, key, key_x(key), key_y(key), key_z(key), true, 0, hmask, bcap);
            }
            // the last active lane's key is now in the table
            known = __shfl_sync(0xFFFFFFFFu, key, min(31u, hi - 1u - b32));
        }
    }
}

// sort.rs:133-163 gpu_touch_neighbor_blocks: one thread per (base block, neighbour).
__global__ void __launch_bounds__(256) k_touch_nbh(DevPtrs P) {
    after_previous();
    const uint32_t hmask = P.params->hash_capacity - 1;
    const uint32_t bcap = P.params->block_capacity;
    const uint32_t nprim = min(__ldcg(&P.counters->num_primary), bcap);
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nprim * 7u; t += gridDim.x * blockDim.x) {
        const uint32_t b = t / 7u;
        const int i = (int)(t % 7u) + 1;
        const int4 v = P.bvid[b];
        int sx, sy, sz;
        assoc_shift(i, sx, sy, sz);
        const int kx = v.x + sx, ky = v.y + sy, kz = v.z + sz;
        hash_insert(P, pack_key(kx, ky, kz), kx, ky, kz, false, nprim, hmask, bcap);
    }
}

// sort.rs:261-279 gpu_update_nbh_block_ids, plus zeroing of the block's
// bucket counters and P2G accumulation nodes.  One thread per node.  Without
// extras only primary blocks have cell counts (kCells: which blocks' to clear).
enum CellBlocks { kNoCells, kPrimaryCells, kAllCells };
template <CellBlocks kCells>
__global__ void __launch_bounds__(256) k_block_prep(DevPtrs P) {
    after_previous();
    const uint32_t hmask = P.params->hash_capacity - 1;
    const uint32_t bcap = P.params->block_capacity;
    const uint32_t nprim = min(__ldcg(&P.counters->num_primary), bcap);
    const uint32_t total = min(nprim + __ldcg(&P.counters->num_extra), bcap);
    if (blockIdx.x == 0 && threadIdx.x == 0) P.counters->num_blocks = total;
    const uint32_t nthreads = total * 64u;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nthreads; t += gridDim.x * blockDim.x) {
        const uint32_t b = t >> 6, k = t & 63u;
        if (P.nodes) P.nodes[t] = make_float4(0.f, 0.f, 0.f, 0.f);
        // the scatter P2G of CPIC accumulates the incompatible field too
        if (P.nodes_inc && P.params->use_cpic) P.nodes_inc[t] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (kCells == kAllCells || (kCells == kPrimaryCells && b < nprim)) P.cells[t] = 0;
        if (k < NUM_NBH) {
            int4 v = P.bvid[b];
            int sx, sy, sz;
            assoc_shift((int)k + 1, sx, sy, sz);
            P.nbh[b * NUM_NBH + k] = hash_find(P, pack_key(v.x + sx, v.y + sy, v.z + sz), hmask);
        } else if (k < NUM_NBH + NUM_BUCKETS) {
            P.cursors[b * NUM_BUCKETS + (k - NUM_NBH)] = 0;
        } else if (k == 63u && P.rp_count) {
            P.rp_count[b] = 0;
        }
    }
}

// sort.rs:287-349 gpu_update_block_particle_count.
template <bool kExtras, int kSortBatch>
__global__ void __launch_bounds__(256) k_count(DevPtrs P) {
    after_previous();
    const uint32_t n = P.params->n;
    const uint32_t hmask = P.params->hash_capacity - 1;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t lo, hi;
    warp_range(n, lo, hi);
    uint32_t known_key = NONE, known_h0 = NONE;  // the last key this warp looked up
    for (uint32_t base = lo; base < hi; base += 32u * kSortBatch) {
        uint2 codes[kSortBatch];
#pragma unroll
        for (int j = 0; j < kSortBatch; ++j) {
            const uint32_t p = base + 32u * j + lane;
            codes[j] = p < hi ? P.pcode[p] : make_uint2(NONE, 0u);
        }
#pragma unroll
        for (int j = 0; j < kSortBatch; ++j) {
            const uint32_t b32 = base + 32u * j;
            if (b32 >= hi) break;
            const uint32_t p = b32 + lane;
            const bool active = p < hi;
            const uint2 code = codes[j];
            const uint32_t key = active ? code.x : NONE;
            uint32_t h0;
            if (__all_sync(0xFFFFFFFFu, !active || key == known_key)) {
                h0 = active ? known_h0 : NONE;
            } else {  // one probe per distinct block key in the warp
                const uint32_t peers = __match_any_sync(0xFFFFFFFFu, key);
                const uint32_t leader = __ffs(peers) - 1;
                uint32_t h = NONE;
                if (active && lane == leader) h = hash_find(P, key, hmask);
                h0 = __shfl_sync(0xFFFFFFFFu, h, leader);
            }
            const uint32_t last = min(31u, hi - 1u - b32);
            known_key = __shfl_sync(0xFFFFFFFFu, key, last);
            known_h0 = __shfl_sync(0xFFFFFFFFu, h0, last);
            const uint32_t ckey = (h0 != NONE) ? h0 * 64u + code.y : NONE;
            if (active) {
                P.phdr[p] = ckey;
                if (h0 == NONE) set_status(P.counters, STATUS_MISSING_BLOCK);
            }
            warp_agg_red(ckey, ckey != NONE ? &P.cells[ckey] : nullptr);
            if (!kExtras) continue;
            const uint32_t ax = code.y & 3u, ay = (code.y >> 2) & 3u, az = (code.y >> 4) & 3u;
            for (int i = 1; i < 8; ++i) {
                int sx, sy, sz;
                assoc_shift(i, sx, sy, sz);
                uint32_t hn = NONE, e = 0;
                if (h0 != NONE && spills(ax, ay, az, sx, sy, sz)) {
                    hn = P.nbh[h0 * NUM_NBH + (i - 1)];
                    if (hn == NONE) set_status(P.counters, STATUS_MISSING_BLOCK);
                    e = extra_bucket(az, sz);
                }
                const uint32_t k2 = (hn != NONE) ? hn * 16u + e : NONE;
                warp_agg_red(k2, k2 != NONE ? &P.cursors[hn * NUM_BUCKETS + e] : nullptr);
            }
        }
    }
}

// prefix sum (src_rbd/utils/prefix_sum.rs) over the block totals, then
// sort.rs:382-420 gpu_copy_scan_values_to_first_particles, as a two-pass
// tiled scan: pass 1 gives each block its offset inside a tile of kScanTile
// blocks and each tile its total; pass 2 adds the tile's offset (the sum of
// the tile totals before it) and turns the bucket counts into cursors.  These
// two serve the slab sort of launch_sort_positions.
constexpr uint32_t kScanThreads = 256;
constexpr uint32_t kScanPer = kScanTile / kScanThreads;  // blocks per thread

// Exclusive CTA-wide scan of one value per thread; returns the CTA total in *total.
__device__ __forceinline__ uint32_t cta_exclusive_scan(uint32_t v, uint32_t* warp_tot, uint32_t* total) {
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    if (lane == 31) warp_tot[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        const uint32_t nw = blockDim.x >> 5;
        uint32_t w = lane < nw ? warp_tot[lane] : 0u;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xFFFFFFFFu, wi, o);
            if (lane >= (uint32_t)o) wi += y;
        }
        if (lane < nw) warp_tot[lane] = wi - w;
        if (lane == 31) warp_tot[32] = wi;
    }
    __syncthreads();
    const uint32_t out = warp_tot[wid] + incl - v;
    *total = warp_tot[32];
    __syncthreads();
    return out;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(DevPtrs P) {
    __shared__ uint32_t warp_tot[33];
    const uint32_t total = P.counters->num_blocks;
    const uint32_t ntiles = (total + kScanTile - 1) / kScanTile;
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const uint32_t b0 = tile * kScanTile + threadIdx.x * kScanPer;
        uint32_t bt[kScanPer];
        uint32_t t = 0;
#pragma unroll
        for (uint32_t j = 0; j < kScanPer; ++j) {
            const uint32_t b = b0 + j;
            uint32_t s = 0;
            if (b < total) {
#pragma unroll
                for (int k = 0; k < NUM_BUCKETS; ++k) s += P.cursors[b * NUM_BUCKETS + k];
            }
            bt[j] = s;
            t += s;
        }
        uint32_t tile_total;
        uint32_t run = cta_exclusive_scan(t, warp_tot, &tile_total);
#pragma unroll
        for (uint32_t j = 0; j < kScanPer; ++j) {
            const uint32_t b = b0 + j;
            if (b < total) P.scan_tmp[b] = run;
            run += bt[j];
        }
        if (threadIdx.x == 0) P.tile_sums[tile] = tile_total;
    }
}

__global__ void __launch_bounds__(kScanThreads) k_scan_apply(DevPtrs P) {
    __shared__ uint32_t warp_tot[33];
    const uint32_t total = P.counters->num_blocks;
    const uint32_t ntiles = (total + kScanTile - 1) / kScanTile;
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        uint32_t part = 0;
        for (uint32_t i = threadIdx.x; i < tile; i += kScanThreads) part += P.tile_sums[i];
        uint32_t offset;
        cta_exclusive_scan(part, warp_tot, &offset);
        const uint32_t b0 = tile * kScanTile + threadIdx.x * kScanPer;
        // all loads first: the stores below may alias them as far as the compiler knows
        uint32_t cnt[kScanPer][NUM_BUCKETS], rel[kScanPer];
#pragma unroll
        for (uint32_t j = 0; j < kScanPer; ++j) {
            const uint32_t b = b0 + j;
            rel[j] = b < total ? P.scan_tmp[b] : 0u;
#pragma unroll
            for (int k = 0; k < NUM_BUCKETS; ++k) cnt[j][k] = b < total ? P.cursors[b * NUM_BUCKETS + k] : 0u;
        }
#pragma unroll
        for (uint32_t j = 0; j < kScanPer; ++j) {
            const uint32_t b = b0 + j;
            if (b >= total) break;
            const uint32_t first = offset + rel[j];
            uint32_t running = first;
            P.first[b] = first;
#pragma unroll
            for (int k = 0; k < NUM_BUCKETS; ++k) {
                if (k == NUM_PRIMARY_BUCKETS) P.nprim[b] = running - first;
                P.cursors[b * NUM_BUCKETS + k] = running;
                running += cnt[j][k];
            }
            P.nwx[b] = running - first;
            if (b == total - 1) {
                P.counters->sorted_len = running;
                if (running > P.params->sorted_capacity) set_status(P.counters, STATUS_SORT_CAPACITY);
            }
        }
    }
}

// The same two passes for the cell sort, one warp per block: a block's total
// is the sum of its 64 cell counts (and 6 extra buckets); the second pass
// turns the cell counts into cursors (a warp scan, two cells a lane) and
// writes the slab ends.  Without extras only the primary blocks, which come
// first, have counts: the others start where the list ends.
constexpr uint32_t kCellPerWarp = 8;  // blocks per warp of a scan CTA
static_assert(kCellTile == kCellPerWarp * (kScanThreads / 32), "a tile per scan CTA");

template <bool kExtras>
__global__ void __launch_bounds__(kScanThreads) k_scan_cell_tiles(DevPtrs P) {
    after_previous();
    __shared__ uint32_t warp_tot[33];
    __shared__ uint32_t btot[kCellTile];
    const uint32_t total = __ldcg(&P.counters->num_blocks);
    const uint32_t counted = kExtras ? total : min(__ldcg(&P.counters->num_primary), total);
    const uint32_t ntiles = (counted + kCellTile - 1) / kCellTile;
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint2* cells = reinterpret_cast<const uint2*>(P.cells);
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const uint32_t b0 = tile * kCellTile;
        uint32_t v[kCellPerWarp];
#pragma unroll
        for (uint32_t j = 0; j < kCellPerWarp; ++j) {
            const uint32_t b = b0 + wid * kCellPerWarp + j;
            v[j] = 0u;
            if (b < counted) {
                const uint2 c = __ldcg(&cells[b * 32u + lane]);
                v[j] = c.x + c.y;
                if (kExtras && lane < NUM_EXTRA_BUCKETS)
                    v[j] += __ldcg(&P.cursors[b * NUM_BUCKETS + NUM_PRIMARY_BUCKETS + lane]);
            }
        }
#pragma unroll
        for (uint32_t j = 0; j < kCellPerWarp; ++j) {
            const uint32_t t = __reduce_add_sync(0xFFFFFFFFu, v[j]);
            if (lane == 0) btot[wid * kCellPerWarp + j] = t;
        }
        __syncthreads();
        const uint32_t mine = threadIdx.x < kCellTile ? btot[threadIdx.x] : 0u;
        uint32_t tile_total;
        const uint32_t off = cta_exclusive_scan(mine, warp_tot, &tile_total);
        if (threadIdx.x < kCellTile && b0 + threadIdx.x < total) P.scan_tmp[b0 + threadIdx.x] = off;
        if (threadIdx.x == 0) P.tile_sums[tile] = tile_total;
    }
}

// The cursors, header fields and run starts of block b, whose particles start
// at `first` (a warp; cnt: the counts of cells 2 lane and 2 lane + 1, ext: of
// extra bucket `lane`).  Returns where the next block's start.
template <bool kExtras>
__device__ __forceinline__ uint32_t write_block_cursors(const DevPtrs& P, uint32_t b, uint32_t total, uint32_t first,
                                                        uint2 cnt, uint32_t ext, uint32_t lane) {
    uint2* cells = reinterpret_cast<uint2*>(P.cells);
    uint32_t incl = cnt.x + cnt.y;
    uint32_t einc = ext;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
        if (kExtras && o < 8) {
            const uint32_t e = __shfl_up_sync(0xFFFFFFFFu, einc, o);
            if (lane >= (uint32_t)o) einc += e;
        }
    }
    const uint32_t start = first + incl - cnt.x - cnt.y;
    cells[b * 32u + lane] = make_uint2(start, start + cnt.x);
    const uint32_t prim_end = first + __shfl_sync(0xFFFFFFFFu, incl, 31);
    const uint32_t end = kExtras ? prim_end + __shfl_sync(0xFFFFFFFFu, einc, NUM_EXTRA_BUCKETS - 1) : prim_end;
    // slab ends (a slab is 16 cells, 8 lanes); the extra buckets' cursors, empty without extras
    if ((lane & 7u) == 7u) P.cursors[b * NUM_BUCKETS + (lane >> 3)] = first + incl;
    if (lane < NUM_EXTRA_BUCKETS)
        P.cursors[b * NUM_BUCKETS + NUM_PRIMARY_BUCKETS + lane] = prim_end + einc - ext;
    if (lane == 0) {
        P.first[b] = first;
        P.nprim[b] = prim_end - first;
        P.nwx[b] = end - first;
        if (b == total - 1) {
            P.counters->sorted_len = end;
            if (end > P.params->sorted_capacity) set_status(P.counters, STATUS_SORT_CAPACITY);
        }
    }
    // the runs of kRangeChunk sorted positions that start inside this block
    if (P.chunk_blk)
        for (uint32_t c = (first + kRangeChunk - 1u) / kRangeChunk + lane; c * kRangeChunk < end && c < P.chunk_cap;
             c += 32u)
            P.chunk_blk[c] = b;
    return end;
}

// The header of block b without particles, of a list that ends at `len` (a warp).
__device__ __forceinline__ void write_block_empty(const DevPtrs& P, uint32_t b, uint32_t total, uint32_t len,
                                                  uint32_t lane) {
    if (lane < NUM_BUCKETS) P.cursors[b * NUM_BUCKETS + lane] = len;
    if (lane == 0) {
        P.first[b] = len;
        P.nprim[b] = 0u;
        P.nwx[b] = 0u;
        if (b == total - 1) {
            P.counters->sorted_len = len;
            if (len > P.params->sorted_capacity) set_status(P.counters, STATUS_SORT_CAPACITY);
        }
    }
}

template <bool kExtras>
__global__ void __launch_bounds__(kScanThreads) k_scan_cell_apply(DevPtrs P) {
    after_previous();
    __shared__ uint32_t warp_tot[33];
    const uint32_t total = __ldcg(&P.counters->num_blocks);
    const uint32_t counted = kExtras ? total : min(__ldcg(&P.counters->num_primary), total);
    const uint32_t ntiles = (total + kCellTile - 1) / kCellTile, summed = (counted + kCellTile - 1) / kCellTile;
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    uint2* cells = reinterpret_cast<uint2*>(P.cells);
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const uint32_t b0 = tile * kCellTile + wid * kCellPerWarp;
        // all loads first: the stores below may alias them as far as the compiler knows
        uint2 cnt[kCellPerWarp];
        uint32_t ext[kCellPerWarp];
#pragma unroll
        for (uint32_t j = 0; j < kCellPerWarp; ++j) {
            cnt[j] = make_uint2(0u, 0u);
            ext[j] = 0u;
            if (b0 + j < counted) {
                cnt[j] = __ldcg(&cells[(b0 + j) * 32u + lane]);
                if (kExtras && lane < NUM_EXTRA_BUCKETS)
                    ext[j] = __ldcg(&P.cursors[(b0 + j) * NUM_BUCKETS + NUM_PRIMARY_BUCKETS + lane]);
            }
        }
        const uint32_t rel =
            tile < summed && lane < kCellPerWarp && b0 + lane < total ? __ldcg(&P.scan_tmp[b0 + lane]) : 0u;
        uint32_t part = 0;
        for (uint32_t i = threadIdx.x; i < min(tile, summed); i += kScanThreads) part += __ldcg(&P.tile_sums[i]);
        uint32_t offset;
        cta_exclusive_scan(part, warp_tot, &offset);
#pragma unroll
        for (uint32_t j = 0; j < kCellPerWarp; ++j) {
            const uint32_t b = b0 + j;
            if (b >= total) break;
            const uint32_t first = offset + __shfl_sync(0xFFFFFFFFu, rel, j);
            if (b < counted) write_block_cursors<kExtras>(P, b, total, first, cnt[j], ext[j], lane);
            else write_block_empty(P, b, total, first, lane);
        }
    }
}

// Both passes in one CTA, for states of few blocks (without extras): its warps
// share the blocks out evenly, sum them, scan the sums and write the cursors,
// which takes less than a second launch does (one state of 4,096 particles: sort
// 39 us with two kernels, 34 us with this one; above some 2,000 blocks the one
// CTA's walk costs more than the launch).
constexpr uint32_t kOneCtaBlocks = 2048;
constexpr uint32_t kOneCtaThreads = 1024;
__global__ void __launch_bounds__(kOneCtaThreads) k_scan_cells(DevPtrs P) {
    after_previous();
    __shared__ uint32_t warp_tot[33];
    const uint32_t total = P.counters->num_blocks;
    const uint32_t counted = min(P.counters->num_primary, total);
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t per = (counted + 31u) / 32u;  // blocks per warp, at most 64
    const uint32_t b0 = min(wid * per, counted), b1 = min(b0 + per, counted);
    uint2* cells = reinterpret_cast<uint2*>(P.cells);
    uint32_t sum = 0;
    for (uint32_t b = b0; b < b1; b += 8u) {
        uint2 c[8];
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) c[j] = b + j < b1 ? __ldcg(&cells[(b + j) * 32u + lane]) : make_uint2(0u, 0u);
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) sum += c[j].x + c[j].y;
    }
    sum = __reduce_add_sync(0xFFFFFFFFu, sum);
    if (lane == 0) warp_tot[wid] = sum;
    __syncthreads();
    if (wid == 0) {
        const uint32_t v = warp_tot[lane];
        uint32_t incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        warp_tot[lane] = incl - v;
        if (lane == 31) warp_tot[32] = incl;
    }
    __syncthreads();
    for (uint32_t b = counted + wid; b < total; b += 32u) write_block_empty(P, b, total, warp_tot[32], lane);
    uint32_t first = warp_tot[wid];
    for (uint32_t b = b0; b < b1; b += 8u) {
        uint2 c[8];
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) c[j] = b + j < b1 ? __ldcg(&cells[(b + j) * 32u + lane]) : make_uint2(0u, 0u);
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            if (b + j >= b1) break;
            first = write_block_cursors<false>(P, b + j, total, first, c[j], 0u, lane);
        }
    }
}

// sort.rs:430-491 gpu_finalize_particles_sort.
template <bool kExtras, int kSortBatch>
__global__ void __launch_bounds__(256) k_finalize(DevPtrs P) {
    after_previous();
    const uint32_t n = P.params->n;
    const uint32_t scap = P.params->sorted_capacity;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint32_t lo, hi;
    warp_range(n, lo, hi);
    for (uint32_t base = lo; base < hi; base += 32u * kSortBatch) {
        // the cell atomics of all passes in flight together, then the scatter
        uint32_t key[kSortBatch], leader[kSortBatch], rank[kSortBatch], got[kSortBatch];
#pragma unroll
        for (int j = 0; j < kSortBatch; ++j) {
            const uint32_t p = base + 32u * j + lane;
            key[j] = p < hi ? P.phdr[p] : NONE;
        }
#pragma unroll
        for (int j = 0; j < kSortBatch; ++j) {
            const uint32_t peers = __match_any_sync(0xFFFFFFFFu, key[j]);
            leader[j] = __ffs(peers) - 1;
            rank[j] = __popc(peers & lt_mask);
            got[j] = 0u;
            if (key[j] != NONE && lane == leader[j])
                got[j] = atomicAdd(&P.cells[key[j]], (uint32_t)__popc(peers));
        }
#pragma unroll
        for (int j = 0; j < kSortBatch; ++j) {
            const uint32_t p = base + 32u * j + lane;
            const uint32_t slot = __shfl_sync(0xFFFFFFFFu, got[j], leader[j]) + rank[j];
            if (key[j] != NONE && slot < scap) P.sorted[slot] = p;
            if (!kExtras) continue;
            const uint32_t h0 = key[j] >> 6, ax = key[j] & 3u, ay = (key[j] >> 2) & 3u, az = (key[j] >> 4) & 3u;
            for (int i = 1; i < 8; ++i) {
                int sx, sy, sz;
                assoc_shift(i, sx, sy, sz);
                uint32_t hn = NONE, e = 0;
                if (key[j] != NONE && spills(ax, ay, az, sx, sy, sz)) {
                    hn = P.nbh[h0 * NUM_NBH + (i - 1)];
                    e = extra_bucket(az, sz);
                }
                const uint32_t k2 = (hn != NONE) ? hn * 16u + e : NONE;
                const uint32_t s2 = warp_agg_add(k2, k2 != NONE ? &P.cursors[hn * NUM_BUCKETS + e] : nullptr);
                if (k2 != NONE && s2 < scap) P.sorted[s2] = p;
            }
        }
    }
}

// Canonical order: every (block, bucket) segment sorted by ascending id, by
// ranks (particle ids are distinct inside a block).  A block's whole list (some
// 1,700 ids at 8 particles a cell) is taken into shared memory, every bucket
// from a multiple of four, and the CTA's threads each rank some ids against
// their bucket, four at a time; longer lists are sorted bucket by bucket.
// Bound by the comparisons: 100,003 particles 28 us (one bucket after another,
// a thread per id: 36 us; a warp per bucket: 31 us).
constexpr uint32_t kSegMax = 4096;
constexpr uint32_t kSegList = kSegMax - 4 * NUM_BUCKETS - 4;
__global__ void __launch_bounds__(256) k_sort_segments(DevPtrs P) {
    after_previous();
    __shared__ uint4 buf4[kSegMax / 4];
    __shared__ uint32_t ends[NUM_BUCKETS + 1];  // of the buckets in the block's list; ends[0] = 0
    uint32_t* buf = reinterpret_cast<uint32_t*>(buf4);
    const uint32_t total = P.counters->num_blocks;
    for (uint32_t b = blockIdx.x; b < total; b += gridDim.x) {
        const uint32_t first = P.first[b], len = P.nwx[b];
        if (threadIdx.x <= NUM_BUCKETS)
            ends[threadIdx.x] = threadIdx.x ? P.cursors[b * NUM_BUCKETS + threadIdx.x - 1] - first : 0u;
        __syncthreads();
        if (len <= kSegList) {
            // bucket k starts at the next multiple of four, four words of room a bucket
            const auto at = [&](uint32_t k) { return (ends[k] + 4u * k + 3u) & ~3u; };
            const auto bucket = [&](uint32_t i) {
                uint32_t k = 0;
                while (k + 1u < NUM_BUCKETS && i >= ends[k + 1u]) ++k;
                return k;
            };
            for (uint32_t i = threadIdx.x; i < len; i += blockDim.x) {
                const uint32_t k = bucket(i);
                buf[at(k) + i - ends[k]] = P.sorted[first + i];
            }
            if (threadIdx.x < 4u * NUM_BUCKETS) {  // the words after a bucket's last compare as larger
                const uint32_t k = threadIdx.x >> 2, j = threadIdx.x & 3u, n = ends[k + 1u] - ends[k];
                if (n + j < ((n + 3u) & ~3u)) buf[at(k) + n + j] = NONE;
            }
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < len; i += blockDim.x) {
                const uint32_t k = bucket(i), s = at(k), n = ends[k + 1u] - ends[k];
                const uint32_t v = buf[s + i - ends[k]];
                uint32_t rank = 0;
                for (uint32_t j = s / 4u; j < (s + n + 3u) / 4u; ++j) {
                    const uint4 q = buf4[j];
                    rank += (q.x < v) + (q.y < v) + (q.z < v) + (q.w < v);
                }
                P.sorted[first + ends[k] + rank] = v;
            }
        } else {
            for (uint32_t k = 0; k < NUM_BUCKETS; ++k) {
                const uint32_t start = first + ends[k], n = ends[k + 1u] - ends[k];
                if (n > 1u && n <= kSegMax) {
                    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) buf[i] = P.sorted[start + i];
                    __syncthreads();
                    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
                        const uint32_t v = buf[i];
                        uint32_t rank = 0;
                        for (uint32_t j = 0; j < n; ++j) rank += buf[j] < v ? 1u : 0u;
                        P.sorted[start + rank] = v;
                    }
                    __syncthreads();
                } else if (n > kSegMax && threadIdx.x == 0) {
                    set_status(P.counters, STATUS_SORT_CAPACITY);
                }
            }
        }
        __syncthreads();
    }
}

inline int grid_for(int sm_count, int per_sm) { return sm_count * per_sm; }
// At most `per_sm` CTAs of 256 threads an SM, and no more than `items` threads
// need (a small scene's launch is mostly the cost of starting its CTAs).
inline int grid_for(int sm_count, int per_sm, uint64_t items) {
    const uint64_t want = (items + 255u) / 256u, cap = (uint64_t)sm_count * per_sm;
    return (int)(want < 1u ? 1u : (want < cap ? want : cap));
}


// ---------------------------------------------------------------------------
// Primary-only sort of plain float4 positions (no per-particle scratch: the
// key is recomputed from the position in each pass and the primary block is
// found again through the hash).  Used by the allocation-free entry point.

__device__ __forceinline__ uint32_t key_of(const float4* pos, uint32_t p, float dx, uint32_t* assoc) {
    const float4 x = __ldg(&pos[p]);
    const CellInfo ci = cell_info(dx, mk(x.x, x.y, x.z));
    *assoc = ci.ax | (ci.ay << 2) | (ci.az << 4);
    return pack_key(ci.bx, ci.by, ci.bz);
}

__global__ void __launch_bounds__(256) k_touch_primary_pos(DevPtrs P, const float4* __restrict__ pos) {
    const uint32_t n = P.params->n;
    const float dx = P.params->dx;
    const uint32_t hmask = P.params->hash_capacity - 1;
    const uint32_t bcap = P.params->block_capacity;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t base = warp * 32u; base < n; base += nwarps * 32u) {
        const uint32_t p = base + lane;
        uint32_t assoc = 0, key = NONE;
        if (p < n) key = key_of(pos, p, dx, &assoc);
        uint32_t peers = __match_any_sync(0xFFFFFFFFu, key);
        if (p < n && lane == (uint32_t)(__ffs(peers) - 1))
            hash_insert(P, key, key_x(key), key_y(key), key_z(key), true, 0, hmask, bcap);
    }
}

template <bool kScatter>
__global__ void __launch_bounds__(256) k_bucket_pos(DevPtrs P, const float4* __restrict__ pos) {
    const uint32_t n = P.params->n;
    const float dx = P.params->dx;
    const uint32_t hmask = P.params->hash_capacity - 1;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t base = warp * 32u; base < n; base += nwarps * 32u) {
        const uint32_t p = base + lane;
        uint32_t h0 = NONE, assoc = 0;
        if (p < n) {
            h0 = hash_find(P, key_of(pos, p, dx, &assoc), hmask);
            if (h0 == NONE) set_status(P.counters, STATUS_MISSING_BLOCK);
        }
        const uint32_t az = (assoc >> 4) & 3u;
        const uint32_t key = (h0 != NONE) ? h0 * 16u + az : NONE;
        const uint32_t slot = warp_agg_add(key, key != NONE ? &P.cursors[h0 * NUM_BUCKETS + az] : nullptr);
        if (kScatter && key != NONE && slot < P.params->sorted_capacity) P.sorted[slot] = p;
    }
}

}  // namespace


void launch_sort_positions(const DevPtrs& P, const LaunchCfg& c, const float4* pos, cudaStream_t s) {
    const int g = grid_for(c.sm_count, 8);
    int reset_grid = (int)((c.hash_capacity + 255u) / 256u);
    if (reset_grid > g) reset_grid = g;
    if (reset_grid < 1) reset_grid = 1;
    k_sort_reset<<<reset_grid, 256, 0, s>>>(P, c.hash_capacity);
    k_touch_primary_pos<<<g, 256, 0, s>>>(P, pos);
    k_touch_nbh<<<g, 256, 0, s>>>(P);
    k_block_prep<kNoCells><<<g, 256, 0, s>>>(P);
    k_bucket_pos<false><<<g, 256, 0, s>>>(P, pos);
    k_scan_tiles<<<c.sm_count, kScanThreads, 0, s>>>(P);
    k_scan_apply<<<c.sm_count, kScanThreads, 0, s>>>(P);
    k_bucket_pos<true><<<g, 256, 0, s>>>(P, pos);
}


// ---------------------------------------------------------------------------
// CPIC rigid particles (src_mpm/grid/grid.rs:95-121, sort.rs:165-249, 493-667).
// ---------------------------------------------------------------------------

namespace {

// Block (global key coordinates: in batched mode offset by the scene of the
// sample's collider, as the particles' keys are) and associated cell of rigid
// particle i.
__device__ __forceinline__ CellInfo rigid_cell(const DevPtrs& P, uint32_t i, float dx) {
    const float4 w = P.rp_world[i];
    CellInfo ci = cell_info(dx, mk(w.x, w.y, w.z));
    if (P.params->scene_blocks) {
        const uint32_t sid = P.colliders[__float_as_uint(w.w) >> kRigidTriBits].scene;
        const int3 o = scene_base_of(*P.params, sid);
        ci.bx += o.x;
        ci.by += o.y;
        ci.bz += o.z;
    }
    return ci;
}

// sort.rs:200-249 gpu_mark_rigid_particles_needing_block: a rigid particle
// needs its own block when that block is missing while one of its +1
// neighbours exists (without it the particle could not be listed there).
// Runs on the hash as the particle passes left it, before any insertion.
__global__ void __launch_bounds__(256) k_rigid_mark(DevPtrs P) {
    after_previous();
    const uint32_t hmask = P.params->hash_capacity - 1;
    const float dx = P.params->dx;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < P.nrp; i += gridDim.x * blockDim.x) {
        const CellInfo ci = rigid_cell(P, i, dx);
        int k = 0;
        for (; k < 8; ++k) {
            int sx, sy, sz;
            assoc_shift(k, sx, sy, sz);
            if (hash_find(P, pack_key(ci.bx + sx, ci.by + sy, ci.bz + sz), hmask) != NONE) break;
        }
        P.rp_need[i] = (k > 0 && k < 8) ? 1u : 0u;
    }
}

// sort.rs:165-198 gpu_touch_rigid_particle_blocks: the marked particles'
// blocks join the neighbour-pass blocks (ids after the primaries).
__global__ void __launch_bounds__(256) k_rigid_touch(DevPtrs P) {
    after_previous();
    const uint32_t hmask = P.params->hash_capacity - 1;
    const uint32_t bcap = P.params->block_capacity;
    const uint32_t nprim = min(__ldcg(&P.counters->num_primary), bcap);
    const float dx = P.params->dx;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < P.nrp; i += gridDim.x * blockDim.x) {
        if (!P.rp_need[i]) continue;
        const CellInfo ci = rigid_cell(P, i, dx);
        hash_insert(P, pack_key(ci.bx, ci.by, ci.bz), ci.bx, ci.by, ci.bz, false, nprim, hmask, bcap);
    }
}

// The blocks a rigid particle is listed in: its own block (NONE if missing:
// the particle is skipped) and each existing +1 neighbour its 3-cell range
// reaches (sort.rs:509-553).  Returns how many; out[0] is the own block.
__device__ __forceinline__ int rigid_blocks(const DevPtrs& P, uint32_t i, float dx, uint32_t hmask, uint32_t out[8]) {
    const CellInfo ci = rigid_cell(P, i, dx);
    const uint32_t h0 = hash_find(P, pack_key(ci.bx, ci.by, ci.bz), hmask);
    if (h0 == NONE) return 0;
    int n = 0;
    out[n++] = h0;
    for (int k = 1; k < 8; ++k) {
        int sx, sy, sz;
        assoc_shift(k, sx, sy, sz);
        if (!spills(ci.ax, ci.ay, ci.az, sx, sy, sz)) continue;
        const uint32_t hb = P.nbh[h0 * NUM_NBH + k - 1];
        if (hb != NONE) out[n++] = hb;
    }
    return n;
}

// sort.rs:493-556 gpu_update_block_rigid_particle_count.
__global__ void __launch_bounds__(256) k_rigid_count(DevPtrs P) {
    after_previous();
    const uint32_t hmask = P.params->hash_capacity - 1;
    const float dx = P.params->dx;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < P.nrp; i += gridDim.x * blockDim.x) {
        uint32_t hb[8];
        const int n = rigid_blocks(P, i, dx, hmask, hb);
        for (int k = 0; k < n; ++k) atomicAdd(&P.rp_count[hb[k]], 1u);
    }
}

// Each block with rigid entries takes a contiguous range of the list (the
// reference lays the ranges out by a prefix sum, sort.rs:558-600; p2g_cdf
// reads one block's range, so the order of the ranges is free): one atomic
// per warp on the list length, a warp scan for the lanes' offsets.  The
// count becomes the placement cursor.
__global__ void __launch_bounds__(256) k_rigid_alloc(DevPtrs P) {
    after_previous();
    const uint32_t nb = __ldcg(&P.counters->num_blocks);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < nb; base += stride) {
        const uint32_t b = base + lane;
        const uint32_t cnt = b < nb ? P.rp_count[b] : 0u;
        uint32_t incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= (uint32_t)o) incl += v;
        }
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
        uint32_t start = 0;
        if (lane == 31u && total) start = atomicAdd(&P.counters->rigid_len, total);
        start = __shfl_sync(0xFFFFFFFFu, start, 31);
        if (b < nb) {
            P.rp_first[b] = start + incl - cnt;
            P.rp_count[b] = 0;
        }
    }
}

// sort.rs:602-667 gpu_finalize_rigid_particles_sort: the same block set as
// the count pass, so every claimed slot stays inside its block's range.
__global__ void __launch_bounds__(256) k_rigid_finalize(DevPtrs P) {
    after_previous();
    const uint32_t hmask = P.params->hash_capacity - 1;
    const float dx = P.params->dx;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < P.nrp; i += gridDim.x * blockDim.x) {
        uint32_t hb[8];
        const int n = rigid_blocks(P, i, dx, hmask, hb);
        for (int k = 0; k < n; ++k) {
            const uint32_t slot = atomicAdd(&P.rp_count[hb[k]], 1u);
            P.rp_sorted[P.rp_first[hb[k]] + slot] = i;
        }
    }
}

}  // namespace

namespace fast {

bool one_cta_scan(const LaunchCfg& c) { return c.block_capacity <= kOneCtaBlocks; }

int sort_launches(const LaunchCfg& c, bool with_extras, bool canonical) {
    return (canonical ? 9 : 8) - (!with_extras && one_cta_scan(c) ? 1 : 0);
}

void launch_sort(const DevPtrs& P, const LaunchCfg& c, bool with_extras, bool canonical, cudaStream_t s,
                 bool rigid) {
    const int per_sm = (int)c.t.sort_ctas;
    const int g = grid_for(c.sm_count, per_sm, c.particle_capacity);
    const int gr = grid_for(c.sm_count, per_sm, P.nrp);
    const int reset_grid = grid_for(c.sm_count, per_sm, c.hash_capacity);
    const int scan_grid = grid_for(c.sm_count, 2, ((uint64_t)c.block_capacity + kCellTile - 1) / kCellTile * 256u);
    // a primary block holds a particle, and each has seven +1 neighbours
    const uint64_t primaries = c.block_capacity < c.particle_capacity ? c.block_capacity : c.particle_capacity;
    const int gn = grid_for(c.sm_count, per_sm, primaries * 7u);
    const int gb = grid_for(c.sm_count, per_sm, (uint64_t)c.block_capacity * 64u);
    k_sort_reset<<<reset_grid, 256, 0, s>>>(P, c.hash_capacity);
    switch (c.t.sort_batch) {
    case 2: launch_after(k_touch_primary<2>, g, 256, 0, s, P); break;
    case 8: launch_after(k_touch_primary<8>, g, 256, 0, s, P); break;
    default: launch_after(k_touch_primary<4>, g, 256, 0, s, P); break;
    }
    launch_after(k_touch_nbh, gn, 256, 0, s, P);
    if (rigid) {
        launch_after(k_rigid_mark, gr, 256, 0, s, P);
        launch_after(k_rigid_touch, gr, 256, 0, s, P);
    }
    if (with_extras) launch_after(k_block_prep<kAllCells>, gb, 256, 0, s, P);
    else launch_after(k_block_prep<kPrimaryCells>, gb, 256, 0, s, P);
    switch ((with_extras ? 16 : 0) + c.t.sort_batch) {
    case 2: launch_after(k_count<false, 2>, g, 256, 0, s, P); break;
    case 8: launch_after(k_count<false, 8>, g, 256, 0, s, P); break;
    case 18: launch_after(k_count<true, 2>, g, 256, 0, s, P); break;
    case 20: launch_after(k_count<true, 4>, g, 256, 0, s, P); break;
    case 24: launch_after(k_count<true, 8>, g, 256, 0, s, P); break;
    default: launch_after(k_count<false, 4>, g, 256, 0, s, P); break;
    }
    if (with_extras) {
        launch_after(k_scan_cell_tiles<true>, scan_grid, kScanThreads, 0, s, P);
        launch_after(k_scan_cell_apply<true>, scan_grid, kScanThreads, 0, s, P);
    } else {
        if (one_cta_scan(c)) {
            launch_after(k_scan_cells, 1, kOneCtaThreads, 0, s, P);
        } else {
            launch_after(k_scan_cell_tiles<false>, scan_grid, kScanThreads, 0, s, P);
            launch_after(k_scan_cell_apply<false>, scan_grid, kScanThreads, 0, s, P);
        }
    }
    switch ((with_extras ? 16 : 0) + c.t.sort_batch) {
    case 2: launch_after(k_finalize<false, 2>, g, 256, 0, s, P); break;
    case 8: launch_after(k_finalize<false, 8>, g, 256, 0, s, P); break;
    case 18: launch_after(k_finalize<true, 2>, g, 256, 0, s, P); break;
    case 20: launch_after(k_finalize<true, 4>, g, 256, 0, s, P); break;
    case 24: launch_after(k_finalize<true, 8>, g, 256, 0, s, P); break;
    default: launch_after(k_finalize<false, 4>, g, 256, 0, s, P); break;
    }
    if (canonical) launch_after(k_sort_segments, grid_for(c.sm_count, 4), 256, 0, s, P);
    if (rigid) {
        launch_after(k_rigid_count, gr, 256, 0, s, P);
        launch_after(k_rigid_alloc, grid_for(c.sm_count, per_sm, c.block_capacity), 256, 0, s, P);
        launch_after(k_rigid_finalize, gr, 256, 0, s, P);
    }
}

}  // namespace fast
}  // namespace nxm
