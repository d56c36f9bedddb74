// Fast-path transfers: scatter-form P2G with a shared-memory node tile and
// one vector atomic flush per touched node, plus the grid update and the
// fused G2P + particle update (shared with the deterministic build through
// nxm_transfer.inc.cuh), and the collider pose kernels.
#define NXM_NS fast
#define NXM_FAST true
#include "nxm_transfer.inc.cuh"

#include <type_traits>

namespace nxm {
namespace fast {
namespace {

__device__ __forceinline__ void set_status_f(Counters* c, uint32_t bit) { atomicOr(&c->status, bit); }

__device__ __forceinline__ float4 f4add(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// P2G (solver/p2g.rs:64-351 computes the same node sums in gather form).
//
// One warp per active block (taken from a counter), one cell per lane.  The
// sort lists a block's particles by associated cell, so a lane walks its
// cell's particles and keeps the cell's 27 nodes x (momentum, mass) in
// registers: no particle is staged, binned or exchanged, and no two lanes
// share an accumulator.  The contribution to stencil node s = (i, j, k) is
// w_x[i] w_y[j] w_z[k] (q + (C dx) s, m) with q = m v + C (x_0 - x_p), x_0 =
// node (0,0,0); per z layer k the factors w_z[k] (q + k C_z dx, m), w_z[k] C_x
// dx and w_z[k] C_y dx are formed once.  At the end of a round the lanes add
// their nodes into the warp's 6x6x6 tile (the block plus the first two node
// layers of its +1 neighbours), one stencil offset at a time: distinct cells,
// distinct nodes, so no atomics.  The tile goes to global memory with one
// float4 atomic per non-zero node; nodes were zeroed by the sort.
//
// A round ends with its fullest cell, so the 64 cells are split by count: the
// 32 fullest in the first round, the rest in the second (none when at most 32
// hold particles).  The registers of the 108 sums leave 12 warps an SM.
// A cell far fuller than the others (a collapsed or compressed scene) would
// hold up 31 lanes: it gets a round of its own in which the lanes share its
// particles and add up their sums, where that is less work (pick_heavy).  A step
// of a scene of 8 particles a cell and one cell of 2,000 in every block: 228 us
// with a warp per cell, 784 without such rounds, 163 with them; one cell of 20,000
// alone 768, 7,300, 284 us.
//
// The records of a lane's next particles are in flight while it accumulates:
// asynchronous copies into a ring of kP2gRing slots a lane in shared memory
// (slot words of one kind side by side over the lanes: no bank conflicts), so
// that the registers are left to the sums (168, some block words spilled).
//
// Bound by FP32 issue and the L1 lookups of 32 lanes' separate records.  2 M
// sand + water particles: 168 us with a warp per cell and three lanes' groups a
// stencil column, 111 us a cell per lane, 96 us with the ring, 90 us with the
// next round's records in flight while a round's sums go to the tile (0.15 GB,
// 1.7 TB/s); 48 small scenes 152, 90, 81, 76 us; six coupled ones 70, -, 55, 45.
#ifndef NXM_P2G_MIN_CTAS
#define NXM_P2G_MIN_CTAS 3
#endif
#ifndef NXM_P2G_RING
#define NXM_P2G_RING 4
#endif
constexpr int kP2gWarps = 4;
constexpr int kP2gThreads = 32 * kP2gWarps;
constexpr int kP2gRing = NXM_P2G_RING;  // kP2gRing - 1 records ahead
struct P2gSlot {
    float4 xm[32], vf[32], c0[32], c1[32];  // x, m; v, flags; C 0..3; C 4..7
    float c2[32];                           // C 8
};
// A block with a cell above kHeavyCell particles looks for heavy ones; a round of
// the whole warp for one costs some kHeavyCost particles of a lane (the 540
// shuffles that add up the lanes' sums; 3 or 12 make no difference).
constexpr uint32_t kHeavyCell = 32;
constexpr uint32_t kHeavyCost = 6;
constexpr uint32_t kHeavyRound = 2;  // beside rounds 0 and 1
struct P2gBlock {
    uint32_t ends[65];  // ends[c]: where cell c's particles start in the sorted list
    uint32_t blk[8];    // the block and its +1 neighbours
    int x, y, z;        // scene-local block coordinates
    uint32_t heavy;     // cells above this many particles get a round of the whole warp
    uint32_t left[2];   // the ones still to come (cells 0..31, 32..63)
    uint32_t rounds;    // 1 where the second round's cells are empty
};
struct P2gWarp {
    float4 tile[216];
    P2gSlot ring[kP2gRing];
    P2gBlock block[2];  // of this unit and the next
    uint8_t order[64];
};
constexpr size_t kP2gSmem = sizeof(P2gWarp) * kP2gWarps;

__device__ __forceinline__ void p2g_fetch(const DevPtrs& P, P2gSlot& s, uint32_t lane, uint32_t pid) {
    const float4* k = reinterpret_cast<const float4*>(&P.in.kin[pid]);
    const float4* c = reinterpret_cast<const float4*>(&P.in.aff[pid]);
    async_copy<16>(&s.xm[lane], k);
    async_copy<16>(&s.vf[lane], k + 1);
    async_copy<16>(&s.c0[lane], c);
    async_copy<16>(&s.c1[lane], c + 1);
    async_copy<4>(&s.c2[lane], &P.in.tail[pid].c22);
}

__global__ void __launch_bounds__(kP2gThreads, NXM_P2G_MIN_CTAS) k_p2g(DevPtrs P) {
    after_previous();
    extern __shared__ float4 p2g_smem[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    P2gWarp& sm = reinterpret_cast<P2gWarp*>(p2g_smem)[warp];
    float4* tile = sm.tile;
    uint8_t* order = sm.order;
    const float dx = P.params->dx;
    const float inv_dx = P.params->inv_dx;
    const uint32_t nbp = min(__ldcg(&P.counters->num_primary), __ldcg(&P.counters->num_blocks));
    const uint32_t nwarps = gridDim.x * kP2gWarps;
    // With fewer blocks than half the warps, a block's two rounds go to two warps.
    const bool split = 2u * nbp <= nwarps;
    const uint32_t units = split ? 2u * nbp : nbp;
    for (uint32_t t = lane; t < 216u; t += 32u) tile[t] = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t u = warp * gridDim.x + blockIdx.x;  // the first units go to different SMs
    // The block of a unit: loaded ahead, while the sums of the unit before go to
    // the tile; its first records are then in flight while that tile is flushed.
    uint32_t my_blk = 0, el = 0, eh = 0, first = 0;
    int4 vid = make_int4(0, 0, 0, 0);
    const auto load_block = [&](uint32_t v) {
        const uint32_t b = split ? v >> 1 : v;
        vid = P.bvid[b];
        my_blk = lane - 1u < NUM_NBH ? __ldg(&P.nbh[b * NUM_NBH + lane - 1u]) : b;
        // the cells' ends in the sorted list: lane's cells are `lane` and `lane + 32`
        el = __ldg(&P.cells[b * 64u + lane]);
        eh = __ldg(&P.cells[b * 64u + 32u + lane]);
        first = __ldg(&P.first[b]);
    };
    // The threshold, halving from the fullest cell, of the fewest steps: a heavy cell's particles over 32
    // lanes and its cost, then two rounds of cells of at most the threshold.
    const auto pick_heavy = [&](uint32_t cl, uint32_t ch, uint32_t most) {
        uint32_t best = 2u * most, heavy = NONE;
        for (uint32_t t = most >> 1; t >= kHeavyCell / 4u; t >>= 1) {
            const uint32_t held = __reduce_add_sync(0xFFFFFFFFu, (cl > t ? cl : 0u) + (ch > t ? ch : 0u));
            const uint32_t cells = __popc(__ballot_sync(0xFFFFFFFFu, cl > t)) + __popc(__ballot_sync(0xFFFFFFFFu, ch > t));
            const uint32_t steps = held / 32u + kHeavyCost * cells + 2u * t;
            if (steps < best) {
                best = steps;
                heavy = t;
            }
        }
        return heavy;
    };
    const auto order_cells = [&](P2gBlock& k, uint32_t v) {
        k.ends[lane + 1u] = el;
        k.ends[lane + 33u] = eh;
        if (lane < 8u) k.blk[lane] = my_blk;
        if (lane == 0) {
            k.ends[0] = first;
            const int3 o = scene_base_of_block(*P.params, vid);
            k.x = vid.x - o.x;
            k.y = vid.y - o.y;
            k.z = vid.z - o.z;
        }
        __syncwarp();
        uint32_t cl = el - k.ends[lane], ch = eh - k.ends[lane + 32u];
        const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, max(cl, ch));
        uint32_t heavy = NONE, lo = 0, hi = 0;
        if (most > kHeavyCell) {
            heavy = pick_heavy(cl, ch, most);
            lo = __ballot_sync(0xFFFFFFFFu, cl > heavy);
            hi = __ballot_sync(0xFFFFFFFFu, ch > heavy);
            if (split) (v & 1u ? lo : hi) = 0u;  // the block's two warps share them
            if (cl > heavy) cl = 0u;
            if (ch > heavy) ch = 0u;
        }
        if (lane == 0) {
            k.heavy = heavy;
            k.left[0] = lo;
            k.left[1] = hi;
        }
        // the smallest threshold that at most 32 cells exceed
        const auto above = [&](uint32_t t) {
            return __popc(__ballot_sync(0xFFFFFFFFu, cl > t)) + __popc(__ballot_sync(0xFFFFFFFFu, ch > t));
        };
        uint32_t thr = 0;
        if (above(0) > 32) {
            uint32_t lo = 0, hi = min(most, heavy);
            while (hi - lo > 1u) {
                const uint32_t m = (lo + hi) >> 1;
                if (above(m) > 32) lo = m; else hi = m;
            }
            thr = hi;
        }
        if (lane == 0) k.rounds = thr == 0u ? 1u : 2u;
        {  // the cells above it, then as many at it as fill 32 lanes; the others after them
            const uint32_t need = 32u - above(thr);
            const uint32_t eql = __ballot_sync(0xFFFFFFFFu, cl == thr), eqh = __ballot_sync(0xFFFFFFFFu, ch == thr);
            const bool inl = cl > thr || (cl == thr && __popc(eql & lt) < need);
            const bool inh = ch > thr || (ch == thr && __popc(eql) + __popc(eqh & lt) < need);
            const uint32_t ml = __ballot_sync(0xFFFFFFFFu, inl), mh = __ballot_sync(0xFFFFFFFFu, inh);
            const uint32_t nl = __popc(ml);
            order[inl ? __popc(ml & lt) : 32u + __popc(~ml & lt)] = (uint8_t)lane;
            order[inh ? nl + __popc(mh & lt) : 64u - nl + __popc(~mh & lt)] = (uint8_t)(lane + 32u);
            __syncwarp();
        }
    };
    uint32_t c = 0, n = 0, ahead = 0;  // this lane's cell of the round, its particles, the id after the ring's
    const uint32_t* list = nullptr;
    // round 0 or 1, a cell per lane; kHeavyRound: the lanes share the next heavy cell, each every 32nd particle
    const auto begin_round = [&](P2gBlock& k, uint32_t round) {
        const bool shared = round == kHeavyRound;
        if (shared) {
            const uint32_t word = k.left[0] ? 0u : 1u, bits = k.left[word];
            c = 32u * word + (uint32_t)__ffs(bits) - 1u;
            __syncwarp();  // every lane has read the word
            if (lane == 0) k.left[word] = bits & (bits - 1u);
        } else {
            c = order[round * 32u + lane];
        }
        const uint32_t start = k.ends[c], held = k.ends[c + 1u] - start;
        list = P.sorted + start + (shared ? lane : 0u);
        n = shared ? (held + 31u - lane) >> 5 : (held > k.heavy ? 0u : held);
        const uint32_t apart = shared ? 5u : 0u;
        uint32_t pid[kP2gRing - 1];
#pragma unroll
        for (uint32_t t = 0; t + 1 < kP2gRing; ++t) pid[t] = t < n ? __ldg(&list[t << apart]) : 0u;
        ahead = kP2gRing - 1u < n ? __ldg(&list[(kP2gRing - 1u) << apart]) : 0u;
#pragma unroll
        for (uint32_t t = 0; t + 1 < kP2gRing; ++t) {
            if (t < n) p2g_fetch(P, sm.ring[t], lane, pid[t]);
            async_commit();
        }
    };
    if (u < units) {
        load_block(u);
        order_cells(sm.block[0], u);
        begin_round(sm.block[0], split ? u & 1u : 0u);
    }
    uint32_t turn = 0;
    while (u < units) {
        uint32_t next = units;
        if (units > nwarps && lane == 0) next = nwarps + atomicAdd(&P.counters->p2g_next, 1u);
        P2gBlock& now = sm.block[turn];
        const uint32_t r_end = split ? (u & 1u) + 1u : now.rounds;
        // sums the round begun last, begins the one after it (or loads the next block) and returns which
        const auto sum_round = [&](auto shared_cell, uint32_t round) {
            constexpr bool kShared = decltype(shared_cell)::value;
            constexpr uint32_t kApart = kShared ? 32u : 1u;  // from a lane's particle to its next in the list
            const uint32_t nmax = __reduce_max_sync(0xFFFFFFFFu, n);
            const uint32_t cx = c & 3u, cy = (c >> 2) & 3u, cz = c >> 4;
            const bool held = kShared ? lane == 0u : n != 0u;
            const v3 x0 = mk((float)(now.x * 4 + (int)cx), (float)(now.y * 4 + (int)cy), (float)(now.z * 4 + (int)cz)) * dx;
            float2 axy[27], azm[27];  // sums of node i + 3 j + 9 k: (x, y) and (z, mass)
#pragma unroll
            for (int t = 0; t < 27; ++t) axy[t] = azm[t] = make_float2(0.f, 0.f);
            uint32_t at = 0;  // ring slot of the current particle
#pragma unroll 1
            for (uint32_t it = 0; it < nmax; ++it) {
                async_wait<kP2gRing - 2>();  // this lane's copies of the current slot have landed
                const P2gSlot& cur = sm.ring[at];
                const float4 xm = cur.xm[lane], vf = cur.vf[lane], c0 = cur.c0[lane], c1 = cur.c1[lane];
                const float c22 = cur.c2[lane];
                // the slot read in the previous iteration takes the record kP2gRing - 1 ahead
                if (it + kP2gRing - 1u < n) p2g_fetch(P, sm.ring[at == 0u ? kP2gRing - 1u : at - 1u], lane, ahead);
                async_commit();
                ahead = it + kP2gRing < n ? __ldg(&list[(it + kP2gRing) * kApart]) : 0u;
                at = at + 1u == kP2gRing ? 0u : at + 1u;
                const bool on = it < n && (__float_as_uint(vf.w) & PFLAG_ENABLED) != 0u;
                const v3 r = x0 - mk(xm.x, xm.y, xm.z);
                const v3 wx = kernel_eval_all(-r.x * inv_dx);
                const v3 wy = kernel_eval_all(-r.y * inv_dx);
                const v3 wz = kernel_eval_all(-r.z * inv_dx);
                const float m = xm.w;
                const m3 C = mkm(mk(c0.x, c0.y, c0.z), mk(c0.w, c1.x, c1.y), mk(c1.z, c1.w, c22));
                const v3 q = C * r + mk(vf.x, vf.y, vf.z) * m;
                const m3 K = C * dx;
                if (!on) continue;
                float wxy[9];
#pragma unroll
                for (int t = 0; t < 9; ++t) wxy[t] = vget(wx, t % 3) * vget(wy, t / 3);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float wk = vget(wz, k);
                    const v3 bk = k == 0 ? q : (k == 1 ? q + K.c2 : q + K.c2 * 2.0f);
                    float2 pxy = make_float2(bk.x * wk, bk.y * wk), pzm = make_float2(bk.z * wk, m * wk);
                    const float2 ixy = make_float2(K.c0.x * wk, K.c0.y * wk), izm = make_float2(K.c0.z * wk, 0.f);
                    const float2 jxy = make_float2(K.c1.x * wk, K.c1.y * wk), jzm = make_float2(K.c1.z * wk, 0.f);
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        if (j) {
                            pxy = __fadd2_rn(pxy, jxy);
                            pzm = __fadd2_rn(pzm, jzm);
                        }
                        float2 bxy = pxy, bzm = pzm;
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            if (i) {
                                bxy = __fadd2_rn(bxy, ixy);
                                bzm = __fadd2_rn(bzm, izm);
                            }
                            const float w = wxy[i + 3 * j];
                            const int t = i + 3 * j + 9 * k;
                            axy[t] = __ffma2_rn(make_float2(w, w), bxy, axy[t]);
                            azm[t] = __ffma2_rn(make_float2(w, w), bzm, azm[t]);
                        }
                    }
                }
            }
            float4* node = tile + cx + 6u * cy + 36u * cz;
            // the next round's first records, or the next block, while these sums go to the tile
            uint32_t after = NONE;
            if (!kShared && round + 1u < r_end) after = round + 1u;
            else if (now.left[0] | now.left[1]) after = kHeavyRound;
            if (after != NONE) {
                begin_round(now, after);
            } else {
                u = __shfl_sync(0xFFFFFFFFu, next, 0);
                if (u < units) load_block(u);
            }
            if (kShared) {  // the lanes' sums of the one cell: all to lane 0
#pragma unroll
                for (int t = 0; t < 27; ++t) {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        axy[t].x += __shfl_xor_sync(0xFFFFFFFFu, axy[t].x, o);
                        axy[t].y += __shfl_xor_sync(0xFFFFFFFFu, axy[t].y, o);
                        azm[t].x += __shfl_xor_sync(0xFFFFFFFFu, azm[t].x, o);
                        azm[t].y += __shfl_xor_sync(0xFFFFFFFFu, azm[t].y, o);
                    }
                }
            }
#pragma unroll
            for (int t = 0; t < 27; ++t) {
                const int off = t % 3 + 6 * ((t / 3) % 3) + 36 * (t / 9);
                if (held) {
                    const float4 o = node[off];
                    node[off] = make_float4(o.x + axy[t].x, o.y + axy[t].y, o.z + azm[t].x, o.w + azm[t].y);
                }
                __syncwarp();  // the next offset's nodes are other lanes' nodes of this one
            }
            return after;
        };
        uint32_t round = split ? u & 1u : 0u;
        do round = sum_round(std::false_type{}, round);
        while (round < kHeavyRound);
        while (round == kHeavyRound) round = sum_round(std::true_type{}, round);
        if (u < units) {
            __syncwarp();  // the cell order is read
            order_cells(sm.block[turn ^ 1u], u);
            begin_round(sm.block[turn ^ 1u], split ? u & 1u : 0u);
        }
        // the tile to global memory (clearing it)
        for (uint32_t t = lane; t < 216u; t += 32u) {
            const uint32_t tx = t % 6u, ty = (t / 6u) % 6u, tz = t / 36u;
            const uint32_t ox = tx >= 4u, oy = ty >= 4u, oz = tz >= 4u;
            const uint32_t oct = ox * 4u + oy * 2u + oz;
            const uint32_t blk = now.blk[oct];
            const float4 sum = tile[t];
            if (sum.x != 0.f || sum.y != 0.f || sum.z != 0.f || sum.w != 0.f) {
                tile[t] = make_float4(0.f, 0.f, 0.f, 0.f);
                const uint32_t node = (tx - 4u * ox) + 4u * (ty - 4u * oy) + 16u * (tz - 4u * oz);
                if (blk == NONE) set_status_f(P.counters, STATUS_MISSING_BLOCK);
                else atomicAdd(&P.nodes[blk * 64u + node], sum);
            }
        }
        __syncwarp();
        turn ^= 1u;
    }
}

// The words of a particle that the CPIC P2G reads.
struct P2gRaw {
    f8 k, c;  // x, m, v, flags; C's first eight
    float c22;
};

__device__ __forceinline__ P2gRaw p2g_load_raw(const DevPtrs& P, uint32_t pid) {
    P2gRaw r;
    if (pid == NONE) {
        r.k.v[7] = 0.f;  // flags 0: contributes nothing
        return r;
    }
    r.k = load8(&P.in.kin[pid]);
    r.c = load8(&P.in.aff[pid]);
    r.c22 = __ldg(&P.in.tail[pid].c22);
    return r;
}

// CPIC P2G (solver/p2g.rs:258-310): a particle whose affinity bits are
// incompatible with a node's (aff_compatible) feeds that node's second,
// incompatible field instead.
//
// One CTA per active block (grid-stride).  The block's primary particles are
// staged in shared memory in chunks of kCpicChunk.  A staged record holds
//   q = m v + C (x_0 - x_p)  (x_0 = stencil node (0,0,0)) and m,
//   the three columns of C dx, each carrying one z weight w_z[k] alongside,
//   the nine products w_x[i] w_y[j], the affinity bits,
// so the contribution to stencil node s is w_x[s.x] w_y[s.y] w_z[s.z]
// (q + (C dx) s, m).  The sort lists the particles by associated cell; each
// warp takes an eighth of the chunk (whole cells would leave warps idle where
// a chunk holds few: 200,000 particles at 200 a cell 147 us, so 98 us, and 96,000
// with one cell of 1,000 in every block 139, 55 us), a cell's at a time: lane l < 27
// owns the stencil column (s.x, s.y) = ((l mod 9) mod 3, (l mod 9) / 3) for
// particle group l / 9, so a pass reads three particles (three broadcast
// addresses per load) and each lane accumulates its column's three nodes, the
// compatible and the incompatible sums.  A
// three-way shuffle exchange leaves lane l with the cell's full sum for node
// (s.x, s.y, l / 9), which it adds to the warp's private 6x6x6 node tile (one
// per field): the 27
// lanes own distinct nodes and no other warp writes that tile, so no atomics.
// At the end of the block the warp tiles are summed and each non-empty node
// goes to global memory with one float4 atomic; nodes were zeroed by the sort.
constexpr int kCpicWarps = 8;
constexpr int kCpicThreads = 32 * kCpicWarps;
constexpr int kCpicChunk = kCpicThreads;  // particles staged per pass, one per thread
constexpr int kCpicRec = 28;  // floats per staged particle
// record: [0..3] q.xyz, m | [4..7] (C dx).c0, w_z[0] | [8..11] (C dx).c1, w_z[1]
//       | [12..15] (C dx).c2, w_z[2] | [16 + i + 3 j] w_x[i] w_y[j] | [25] affinity | [26..27] unused
constexpr size_t kCpicSmem = (size_t)2 * kCpicWarps * 216 * 16 + (size_t)kCpicChunk * kCpicRec * 4 + 68 * 4 + 218 * 4;

struct P2gHdr {
    uint32_t first, np;
};

__device__ __forceinline__ P2gHdr p2g_load_hdr(const DevPtrs& P, uint32_t b, uint32_t nbp) {
    P2gHdr h{0u, 0u};
    if (b < nbp) {
        h.first = __ldcg(&P.first[b]);
        h.np = __ldcg(&P.nprim[b]);
    }
    return h;
}

// Work runs over the primary blocks only (ids [0, num_primary); the others
// hold no particles).  Loads run ahead of use: the headers of the blocks two
// grid strides ahead, the sorted id of the next chunk's particle right after
// staging, and its record at the start of the cell phase, so their latency
// overlaps the current chunk's shared-memory work.  Two coupled fields of 27
// sums do not fit a lane's registers, so this mode keeps a cell per warp.
__global__ void __launch_bounds__(kCpicThreads, 2) k_p2g_cpic(DevPtrs P) {
    after_previous();
    static_assert(kCpicThreads >= 216, "one flushed tile node per thread");
    extern __shared__ float4 p2g_smem[];
    float4* tiles = p2g_smem;  // kCpicWarps x 216 nodes of (x, y, z, m)
    float4* tiles_inc = tiles + kCpicWarps * 216;
    float* rec = reinterpret_cast<float*>(tiles + 2 * kCpicWarps * 216);
    int* start = reinterpret_cast<int*>(rec + kCpicChunk * kCpicRec);  // 65 used
    uint32_t* node_aff = reinterpret_cast<uint32_t*>(start + 68);  // 216 tile nodes
    // Nonzero when a tile node of the current block carries an affinity
    // bit; otherwise every particle is compatible with every node and the
    // block runs the plain accumulation (no incompatible sums, no flush).
    // Two flags by block parity: the one of the next block is cleared while
    // the current one is in use (between two end-of-block barriers).
    volatile uint32_t* blk_aff_pair = node_aff + 216;
    uint32_t parity = 0u;

    const float dx = P.params->dx;
    const float inv_dx = P.params->inv_dx;
    const uint32_t nbp = min(__ldcg(&P.counters->num_primary), __ldcg(&P.counters->num_blocks));
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    // cell-phase roles; lanes 27..31 idle (zero weight, never write)
    const bool worker = lane < 27u;
    const uint32_t grp = worker ? lane / 9u : 0u;
    const uint32_t sxy = worker ? lane % 9u : 0u;
    const float fx = (float)(sxy % 3u), fy = (float)(sxy / 3u);
    const uint32_t src1 = worker ? sxy + 9u * ((grp + 1u) % 3u) : lane;
    const uint32_t src2 = worker ? sxy + 9u * ((grp + 2u) % 3u) : lane;
    float4* tile = tiles + warp * 216u;
    float4* tile_inc = tiles_inc + warp * 216u;
    // flush role: tile node `tid` (tid < 216) of octant `foct`
    const uint32_t ftx = tid % 6u, fty = (tid / 6u) % 6u, ftz = tid / 36u;
    const uint32_t fox = ftx >= 4u, foy = fty >= 4u, foz = ftz >= 4u;
    const uint32_t foct = fox * 4u + foy * 2u + foz;
    const uint32_t fnode = (ftx - 4u * fox) + 4u * (fty - 4u * foy) + 16u * (ftz - 4u * foz);
    // particles stay in id order (slot = id): the affinity of this step's g2p_cdf
    const auto load_aff = [&](uint32_t pid) { return pid == NONE ? 0.f : __ldg(&P.pcdf[3u * pid + 1u].w); };

    uint32_t b = blockIdx.x;
    if (b >= nbp) return;
    const uint32_t stride = gridDim.x;
    for (uint32_t t = tid; t < 2u * kCpicWarps * 216u; t += kCpicThreads) tiles[t] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (tid == 0) blk_aff_pair[0] = 0u;
    P2gHdr h = p2g_load_hdr(P, b, nbp);
    P2gHdr hn = p2g_load_hdr(P, b + stride, nbp);
    P2gHdr hnn = p2g_load_hdr(P, b + 2u * stride, nbp);
    uint32_t pid = tid < h.np ? __ldg(&P.sorted[h.first + tid]) : NONE;
    P2gRaw raw = p2g_load_raw(P, pid);
    float aff = load_aff(pid);
    __syncthreads();
    for (;;) {
        int4 vid = P.bvid[b];
        {
            const int3 o = scene_base_of_block(*P.params, vid);  // scene-local block coordinates
            vid.x -= o.x; vid.y -= o.y; vid.z -= o.z;
        }
        const uint32_t fblk = (tid < 216u && foct != 0u) ? __ldg(&P.nbh[b * NUM_NBH + foct - 1u]) : b;
        // this thread's cell: the end of its particles in the block's list
        const uint32_t cell_end = tid < 64u ? __ldg(&P.cells[b * 64u + tid]) - h.first : 0u;
        volatile uint32_t* blk_aff = blk_aff_pair + parity;
        if (tid == 0) blk_aff_pair[parity ^ 1u] = 0u;
        if (tid < 216u) {  // read after the staging barrier below
            const uint32_t na = fblk == NONE ? 0u : __ldg(&P.ncdf[fblk * 64u + fnode].y);
            node_aff[tid] = na;
            if (na & 0x0000FFFFu) *blk_aff = 1u;
        }
        for (uint32_t base = 0; base < h.np; base += kCpicChunk) {
            const uint32_t m_chunk = min(h.np - base, (uint32_t)kCpicChunk);
            // 1. stage this thread's particle (base + tid); a disabled one as zeros
            if (tid < m_chunk) {
                float4* rr = reinterpret_cast<float4*>(rec + tid * kCpicRec);
                if (!(__float_as_uint(raw.k.v[7]) & PFLAG_ENABLED)) {
#pragma unroll
                    for (int w = 0; w < 7; ++w) rr[w] = make_float4(0.f, 0.f, 0.f, 0.f);
                } else {
                    const v3 pt = mk(raw.k.v[0], raw.k.v[1], raw.k.v[2]);
                    const float m = raw.k.v[3];
                    const CellInfo ci = cell_info_near(dx, inv_dx, pt);
                    const v3 r = mk((float)(vid.x * 4 + (int)ci.ax), (float)(vid.y * 4 + (int)ci.ay),
                                    (float)(vid.z * 4 + (int)ci.az)) * dx - pt;
                    const v3 wx = kernel_eval_all(-r.x * inv_dx);
                    const v3 wy = kernel_eval_all(-r.y * inv_dx);
                    const v3 wz = kernel_eval_all(-r.z * inv_dx);
                    const m3 C = mkm(mk(raw.c.v[0], raw.c.v[1], raw.c.v[2]), mk(raw.c.v[3], raw.c.v[4], raw.c.v[5]),
                                     mk(raw.c.v[6], raw.c.v[7], raw.c22));
                    const v3 q = C * r + mk(raw.k.v[4], raw.k.v[5], raw.k.v[6]) * m;
                    rr[0] = make_float4(q.x, q.y, q.z, m);
                    rr[1] = make_float4(C.c0.x * dx, C.c0.y * dx, C.c0.z * dx, wz.x);
                    rr[2] = make_float4(C.c1.x * dx, C.c1.y * dx, C.c1.z * dx, wz.y);
                    rr[3] = make_float4(C.c2.x * dx, C.c2.y * dx, C.c2.z * dx, wz.z);
                    rr[4] = make_float4(wx.x * wy.x, wx.y * wy.x, wx.z * wy.x, wx.x * wy.y);
                    rr[5] = make_float4(wx.y * wy.y, wx.z * wy.y, wx.x * wy.z, wx.y * wy.z);
                    rr[6] = make_float4(wx.z * wy.z, aff, 0.f, 0.f);
                }
            }
            // where each cell's particles lie in this chunk
            if (tid < 64u) start[tid + 1] = (int)min(max(cell_end, base) - base, m_chunk);
            if (tid == 64u) start[0] = 0;
            // sorted id of this thread's particle in the next chunk (this block or the next one)
            uint32_t pid_next = NONE;
            if (base + kCpicChunk < h.np) {
                if (base + kCpicChunk + tid < h.np) pid_next = __ldg(&P.sorted[h.first + base + kCpicChunk + tid]);
            } else if (tid < hn.np) {
                pid_next = __ldg(&P.sorted[hn.first + tid]);
            }
            __syncthreads();
            raw = p2g_load_raw(P, pid_next);
            aff = load_aff(pid_next);
            const bool split = *blk_aff != 0u;
            // 2. an eighth of the chunk per warp, cell by cell, three particles per pass
            const int seg = (int)((m_chunk + kCpicWarps - 1u) / kCpicWarps);
            const int seg0 = min((int)warp * seg, (int)m_chunk), seg1 = min(seg0 + seg, (int)m_chunk);
            const uint32_t before = __popc(__ballot_sync(0xFFFFFFFFu, start[lane + 1] <= seg0)) +
                                    __popc(__ballot_sync(0xFFFFFFFFu, start[lane + 33] <= seg0));
            for (uint32_t c = before; c < 64u && start[c] < seg1; ++c) {
                const int s0 = max(start[c], seg0), s1 = min(start[c + 1], seg1);
                if (s0 >= s1) continue;
                float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f), a1 = a0, a2 = a0;  // s.z = 0, 1, 2
                float4 i0 = a0, i1 = a0, i2 = a0;  // the incompatible sums
                const uint32_t cx = c & 3u, cy = (c >> 2) & 3u, cz = c >> 4;
                const uint32_t col = (cx + sxy % 3u) + 6u * (cy + sxy / 3u) + 36u * cz;  // this lane's s.z = 0 node
                uint32_t na0 = 0u, na1 = 0u, na2 = 0u;
                if (split && worker) {
                    na0 = node_aff[col];
                    na1 = node_aff[col + 36u];
                    na2 = node_aff[col + 72u];
                }
                for (int i = s0; i < s1; i += 3) {
                    const int j = i + (int)grp;
                    const bool valid = worker && j < s1;
                    const float* r = rec + (valid ? j : s0) * kCpicRec;
                    const float4 qm = *reinterpret_cast<const float4*>(r);
                    const float4 k0 = *reinterpret_cast<const float4*>(r + 4);
                    const float4 k1 = *reinterpret_cast<const float4*>(r + 8);
                    const float4 k2 = *reinterpret_cast<const float4*>(r + 12);
                    const float wxy = valid ? r[16 + sxy] : 0.f;
                    float bx = qm.x + k0.x * fx + k1.x * fy;
                    float by = qm.y + k0.y * fx + k1.y * fy;
                    float bz = qm.z + k0.z * fx + k1.z * fy;
                    if (!split) {
                        float w = wxy * k0.w;
                        a0.x += w * bx; a0.y += w * by; a0.z += w * bz; a0.w += w * qm.w;
                        bx += k2.x; by += k2.y; bz += k2.z;
                        w = wxy * k1.w;
                        a1.x += w * bx; a1.y += w * by; a1.z += w * bz; a1.w += w * qm.w;
                        bx += k2.x; by += k2.y; bz += k2.z;
                        w = wxy * k2.w;
                        a2.x += w * bx; a2.y += w * by; a2.z += w * bz; a2.w += w * qm.w;
                    } else {
                        const uint32_t paff = __float_as_uint(r[25]);
                        const auto acc = [&](float4& a, float4& ai, uint32_t na, float w) {
                            const bool comp = aff_compatible(paff, na);
                            const float wc = comp ? w : 0.f, wi = comp ? 0.f : w;
                            a.x += wc * bx; a.y += wc * by; a.z += wc * bz; a.w += wc * qm.w;
                            ai.x += wi * bx; ai.y += wi * by; ai.z += wi * bz; ai.w += wi * qm.w;
                        };
                        acc(a0, i0, na0, wxy * k0.w);
                        bx += k2.x; by += k2.y; bz += k2.z;
                        acc(a1, i1, na1, wxy * k1.w);
                        bx += k2.x; by += k2.y; bz += k2.z;
                        acc(a2, i2, na2, wxy * k2.w);
                    }
                }
                // lane (sxy, g) collects node (sxy, s.z = g) from the three groups:
                // from group g+1 its s.z = g sum, which that lane holds as (its g + 2) mod 3,
                // from group g+2 likewise as (its g + 1) mod 3.
                const auto exchange = [&](float4 x0, float4 x1, float4 x2) {
                    const float4 own = grp == 0u ? x0 : (grp == 1u ? x1 : x2);
                    const float4 out1 = grp == 0u ? x2 : (grp == 1u ? x0 : x1);
                    const float4 out2 = grp == 0u ? x1 : (grp == 1u ? x2 : x0);
                    float4 t;
                    t.x = own.x + __shfl_sync(0xFFFFFFFFu, out1.x, src1) + __shfl_sync(0xFFFFFFFFu, out2.x, src2);
                    t.y = own.y + __shfl_sync(0xFFFFFFFFu, out1.y, src1) + __shfl_sync(0xFFFFFFFFu, out2.y, src2);
                    t.z = own.z + __shfl_sync(0xFFFFFFFFu, out1.z, src1) + __shfl_sync(0xFFFFFFFFu, out2.z, src2);
                    t.w = own.w + __shfl_sync(0xFFFFFFFFu, out1.w, src1) + __shfl_sync(0xFFFFFFFFu, out2.w, src2);
                    return t;
                };
                const float4 t = exchange(a0, a1, a2);
                const uint32_t node = col + 36u * grp;
                if (worker) tile[node] = f4add(tile[node], t);
                if (split) {
                    const float4 ti = exchange(i0, i1, i2);
                    if (worker) tile_inc[node] = f4add(tile_inc[node], ti);
                }
            }
            __syncthreads();
        }
        // 3. sum the warp tiles (clearing them) and flush the block's nodes
        const int nfields = *blk_aff != 0u ? 2 : 1;
        if (tid < 216u) {
            for (int f = 0; f < nfields; ++f) {
                float4* tt = f ? tiles_inc : tiles;
                float4 sum = tt[tid];
                tt[tid] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int w = 1; w < kCpicWarps; ++w) {
                    sum = f4add(sum, tt[w * 216 + tid]);
                    tt[w * 216 + tid] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
                if (sum.x != 0.f || sum.y != 0.f || sum.z != 0.f || sum.w != 0.f) {
                    if (fblk == NONE) set_status_f(P.counters, STATUS_MISSING_BLOCK);
                    else atomicAdd(&(f ? P.nodes_inc : P.nodes)[fblk * 64u + fnode], sum);
                }
            }
        }
        __syncthreads();
        parity ^= 1u;
        b += stride;
        if (b >= nbp) break;
        h = hn;
        hn = hnn;
        hnn = p2g_load_hdr(P, b + 2u * stride, nbp);
    }
}

}  // namespace

void launch_p2g(const DevPtrs& P, const LaunchCfg& c, cudaStream_t s) {
    // at most a warp per round of a block, and no more blocks than particles
    const uint64_t units = 2ull * min(c.block_capacity, c.particle_capacity);
    const uint64_t want = max(units / kP2gWarps, (uint64_t)1);
    const uint64_t cap = (uint64_t)c.sm_count * min(c.t.p2g_ctas, (uint32_t)NXM_P2G_MIN_CTAS);
    cudaFuncSetAttribute(k_p2g, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kP2gSmem);
    launch_after(k_p2g, (int)min(want, cap), kP2gThreads, kP2gSmem, s, P);
}

void launch_p2g_cpic(const DevPtrs& P, const LaunchCfg& c, cudaStream_t s) {
    cudaFuncSetAttribute(k_p2g_cpic, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCpicSmem);
    launch_after(k_p2g_cpic, c.sm_count * 2, kCpicThreads, kCpicSmem, s, P);
}


}  // namespace fast
}  // namespace nxm
