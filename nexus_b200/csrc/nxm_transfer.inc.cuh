// Grid update and G2P + particle update kernels, included twice: by
// nxm_transfer_fast.cu (multiply-adds may fuse) and by nxm_transfer_det.cu
// (built with --fmad=false, every multiply and add rounded separately in the
// reference's order).  NXM_NS names the namespace of the instantiation.
#include "nxm_device.cuh"
#include "nxm_kernels.h"

#ifndef NXM_NS
#error "define NXM_NS before including nxm_transfer.inc.cuh"
#endif
#ifndef NXM_FAST
#error "define NXM_FAST (true: fast build, false: reference operation order)"
#endif
#ifndef NXM_CPIC
#define NXM_CPIC 0  // 1: also build the CPIC branches (deterministic-build kernels only)
#endif

namespace nxm {
namespace NXM_NS {
namespace {

// C and F of the particle in slot p.
__device__ __forceinline__ m3 affine_of(const Particles& a, uint32_t p) {
    const f8 c = load8(&a.aff[p]);
    return mkm(mk(c.v[0], c.v[1], c.v[2]), mk(c.v[3], c.v[4], c.v[5]), mk(c.v[6], c.v[7], a.tail[p].c22));
}
__device__ __forceinline__ m3 def_grad_of(const Particles& a, uint32_t p, float f22) {
    const f8 f = load8(&a.def[p]);
    return mkm(mk(f.v[0], f.v[1], f.v[2]), mk(f.v[3], f.v[4], f.v[5]), mk(f.v[6], f.v[7], f22));
}

__device__ __forceinline__ void set_status(Counters* c, uint32_t bit) { atomicOr(&c->status, bit); }

__device__ __forceinline__ v3 col_vel_at(const DevCollider& c, v3 p) {
    // dynamics/body.rs:239-250 velocity_at_point
    v3 lin = mk(c.linvel[0], c.linvel[1], c.linvel[2]);
    v3 ang = mk(c.angvel[0], c.angvel[1], c.angvel[2]);
    v3 com = mk(c.com[0], c.com[1], c.com[2]);
    return lin + cross(ang, p - com);
}

struct Collision {
    v3 normal;
    float distance;
    uint32_t closest;
};

// Whether analytic collider c (ball, cuboid, capsule) can touch a node of a
// block whose 64 nodes lie within rb of `centre` (rb = 1.5 sqrt(3) dx about
// the block's middle): the exact distance at the centre, then the bound
// distance(node) >= distance(centre) - rb.  A contributing node is inside the
// shape or has its projection within cap on every axis (so within sqrt(3)
// cap): the collider is kept when the centre is inside or the shape lies
// within rb + sqrt(3) cap of it.  The reach carries a relative and an
// absolute margin above the rounding of the per-node queries it stands for.
__device__ __forceinline__ bool analytic_near_block(const DevCollider& c, float cap, float rb, v3 centre) {
    const quat q = quat{c.rot[0], c.rot[1], c.rot[2], c.rot[3]};
    const v3 local = qrot(qconj(q), centre - mk(c.tra[0], c.tra[1], c.tra[2]));
    Proj pr;
    if (c.type == SHAPE_BALL) pr = ball_project_local(c.a[0], local);
    else if (c.type == SHAPE_CUBOID) pr = cuboid_project_local(mk(c.a[0], c.a[1], c.a[2]), local);
    else if (c.type == SHAPE_CAPSULE)
        pr = capsule_project_local(mk(c.a[0], c.a[1], c.a[2]), mk(c.b[0], c.b[1], c.b[2]), c.b[3], local);
    else return true;
    if (pr.inside) return true;
    const v3 d = pr.point - local;
    const float reach = (rb + 1.75f * cap) * 1.001f + 1.0e-5f;
    return !(dot(d, d) > reach * reach);  // a NaN keeps the collider
}

// Whether trimesh collider c can have a triangle within cap of a node of the
// block: the box of its BVH root within rb + cap of the centre (a node's
// query descends only into boxes within cap of the node).  Only the root is
// tested: one lane's deeper query for the whole block costs the warp about
// as much as the 32 per-node queries it would save.
__device__ __forceinline__ bool mesh_near_block(const DevPtrs& P, const DevCollider& c, float cap, float rb,
                                                v3 centre) {
    if (c.bvh_count == 0u) return false;
    const quat ci = qconj(quat{c.rot[0], c.rot[1], c.rot[2], c.rot[3]});
    const v3 local = qrot(ci, centre) + (-qrot(ci, mk(c.tra[0], c.tra[1], c.tra[2])));
    return !(aabb_distance(P.bvh[c.bvh_first], local) > (rb + cap) * 1.001f + 1.0e-5f);
}

// Bit i: collider i (< 32) may touch a node of block `vid` (scene-local
// block coordinates).  Every lane of the warp calls it for the same block;
// lane i tests collider i.  Trimeshes are left out when `skip_meshes`.
__device__ __forceinline__ uint32_t colliders_near_block(const DevPtrs& P, const DevCollider* cols, uint32_t ncol,
                                                        float dx, int4 vid, bool skip_meshes) {
    const uint32_t lane = threadIdx.x & 31u;
    const v3 centre = mk((float)vid.x * 4.0f + 1.5f, (float)vid.y * 4.0f + 1.5f, (float)vid.z * 4.0f + 1.5f) * dx;
    const float cap = dx * 1.5f, rb = 2.6f * dx;
    bool near = false;
    if (lane < ncol) {
        const DevCollider& c = cols[lane];
        near = c.type == SHAPE_TRIMESH ? !skip_meshes && mesh_near_block(P, c, cap, rb, centre)
                                       : analytic_near_block(c, cap, rb, centre);
    }
    return __ballot_sync(0xFFFFFFFFu, near);
}

// A warp's room for the leaves of a mesh search and the ones being tested.
struct MeshWarp {
    uint32_t leaves[kMeshLeaves];
    MeshLeaf stage[32];
};

// `near` (bit i for collider i < 32, from colliders_near_block) leaves out
// the colliders that cannot reach this node: their projections would find
// no point within cap and no inside.
// A trimesh within reach of the block is searched once for the warp's 32 nodes
// (`mesh`: the warp's room for the leaves found), each node then tests those:
// a node's own traversal is a chain of some hundred dependent loads (six scenes
// over a 20,000-triangle floor: grid update 90 us, with the shared search 77 us,
// with the leaves staged in shared memory and the windows in one scan 61 us).
__device__ __forceinline__ Collision collide(const DevPtrs& P, const DevCollider* cols, uint32_t ncol, float dx,
                                             v3 point, uint32_t near, MeshWarp& mesh) {
    const float cap = dx * 1.5f;
    Collision col;
    col.normal = splat(0.f);
    col.distance = MAX_FLT;
    col.closest = 0;
    for (uint32_t i = 0; i < ncol; ++i) {
        if (i < 32u && !(near & (1u << i))) {
            // next candidate: skip the run of unset bits at once
            const uint32_t rest = near & ~((2u << i) - 1u);
            if (rest == 0u) i = 31u;
            else i = (uint32_t)__ffs(rest) - 2u;
            continue;
        }
        const DevCollider& c = cols[i];
        quat q = quat{c.rot[0], c.rot[1], c.rot[2], c.rot[3]};
        v3 tra = mk(c.tra[0], c.tra[1], c.tra[2]);
        // fast build: an unrotated collider (the usual box walls) skips the
        // two rotations (the deterministic build keeps them: they turn -0 into +0)
        const bool ident = NXM_FAST && q.x == 0.f && q.y == 0.f && q.z == 0.f && q.w == 1.f;
        Proj pr;
        if (ident && c.type != SHAPE_TRIMESH) {
            const v3 local = point - tra;
            if (c.type == SHAPE_BALL) pr = ball_project_local(c.a[0], local);
            else if (c.type == SHAPE_CUBOID) pr = cuboid_project_local(mk(c.a[0], c.a[1], c.a[2]), local);
            else if (c.type == SHAPE_CAPSULE)
                pr = capsule_project_local(mk(c.a[0], c.a[1], c.a[2]), mk(c.b[0], c.b[1], c.b[2]), c.b[3], local);
            else { pr.point = local; pr.inside = false; }
            pr.point = pr.point + tra;
        } else if (c.type == SHAPE_TRIMESH) {
            // pose.inverse() * point, as the inverse isometry applies it
            const quat ci = qconj(q);
            const v3 local = qrot(ci, point) + (-qrot(ci, tra));
            __syncwarp();  // the previous mesh's leaves are read
            const uint32_t nl = warp_mesh_leaves(P.bvh, c.bvh_first, c.bvh_count, local, cap, mesh.leaves);
            const bool found = nl != NONE ? mesh_project_leaves(P.tris, P.bvh, mesh.leaves, nl, local, cap, mesh.stage, pr)
                                          : trimesh_project_local(P.tris, P.bvh, c.bvh_first, c.bvh_count, local, cap, pr);
            if (!found) continue;
        } else {
            v3 local = qrot(qconj(q), point - tra);
            if (c.type == SHAPE_BALL) pr = ball_project_local(c.a[0], local);
            else if (c.type == SHAPE_CUBOID) pr = cuboid_project_local(mk(c.a[0], c.a[1], c.a[2]), local);
            else if (c.type == SHAPE_CAPSULE)
                pr = capsule_project_local(mk(c.a[0], c.a[1], c.a[2]), mk(c.b[0], c.b[1], c.b[2]), c.b[3], local);
            else { pr.point = local; pr.inside = false; }
        }
        if (!(ident && c.type != SHAPE_TRIMESH)) pr.point = qrot(q, pr.point) + tra;
        v3 dpt = pr.point - point;
        v3 ad = vabs(dpt);
        bool within = ad.x <= cap && ad.y <= cap && ad.z <= cap;
        if (pr.inside || within) {
            float sign = pr.inside ? -1.0f : 1.0f;
            float distance = length(dpt);
            v3 normal = dpt / (distance * -sign);
            float sd = sign * distance;
            if (sd < col.distance) {
                col.distance = sd;
                col.normal = normal;
                col.closest = i;
            }
        }
    }
    return col;
}

// grid_update.rs:21-88 + grid_update_collide.rs:102-183, one thread per node.
// CTAs of one block's nodes: a block near a mesh takes many times as long as one
// in free flight, and its CTA holds up no other block's warps (256 threads a CTA:
// six coupled scenes 80 us, 48 small scenes 24.6 us; 64: 77 us, 22.5 us).
constexpr int kGridThreads = 64;
__global__ void __launch_bounds__(kGridThreads, 16) k_grid_update(DevPtrs P) {
    after_previous();
    __shared__ DevCollider scol[MAX_COLLIDERS];
    __shared__ MeshWarp mesh[kGridThreads / 32];
    const Params prm = *P.params;
    // batched scenes: each block sees only its scene's colliders (global memory)
    const bool scenes = prm.scene_blocks != 0;
    const uint32_t ncol = prm.use_cpic ? 0u : (scenes ? prm.ncol : min(prm.ncol, (uint32_t)MAX_COLLIDERS));
    if (!scenes)
        for (uint32_t i = threadIdx.x; i < ncol * (sizeof(DevCollider) / 4); i += blockDim.x)
            reinterpret_cast<uint32_t*>(scol)[i] = reinterpret_cast<const uint32_t*>(P.colliders)[i];
    __syncthreads();
    const float dx = prm.dx, dt = prm.dt;
    const v3 g = mk(prm.gravity[0], prm.gravity[1], prm.gravity[2]);
    const float lim = dx / dt;
    const uint32_t total = P.counters->num_blocks * 64u;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        float4 nd = P.nodes[t];
        const float mass = nd.w;
        const float inv_mass = mass > 0.f ? 1.0f / mass : 0.0f;
        v3 v = (mk(nd.x, nd.y, nd.z) + g * (mass * dt)) * inv_mass;
        v = vclamp(v, -lim, lim);
        if (ncol > 0) {
            const uint32_t b = t >> 6, k = t & 63u;
            int4 vid = P.bvid[b];
            const DevCollider* cols = scol;
            uint32_t nc = ncol;
            if (scenes) {
                const uint32_t sid = scene_of_block(prm, vid);
                const uint2 r = sid != NONE ? P.scene_cols[sid] : make_uint2(0u, 0u);
                cols = P.colliders + r.x;
                nc = r.y;
                const int3 o = scene_base_of_block(prm, vid);  // scene-local node position
                vid.x -= o.x; vid.y -= o.y; vid.z -= o.z;
            }
            v3 cell_pt = mk((float)(vid.x * 4 + (int)(k & 3u)), (float)(vid.y * 4 + (int)((k >> 2) & 3u)),
                            (float)(vid.z * 4 + (int)(k >> 4))) * dx;
            // the warp's 32 nodes share one block: its colliders in reach, one lane each
            const uint32_t near = colliders_near_block(P, cols, nc, dx, vid, false);
            Collision c = collide(P, cols, nc, dx, cell_pt, near, mesh[threadIdx.x >> 5]);
            if (c.distance != MAX_FLT) {
                const DevCollider& cc = cols[c.closest];
                v3 bv = col_vel_at(cc, cell_pt);
                v3 delta = v - bv;
                float nv = dot(delta, c.normal);
                const float margin = dx;
                if (c.distance <= margin) {
                    v = bv + bc_project(cc.bc_type, cc.bc_friction, delta, c.normal);
                } else if (-nv * dt > c.distance - margin) {
                    v3 excess = c.normal * (nv + (c.distance - margin) / dt);
                    v = v - excess;
                }
            }
        }
        P.nodes[t] = make_float4(v.x, v.y, v.z, mass);
#if NXM_CPIC
        if (prm.use_cpic) {  // grid_update.rs:55-66: the incompatible field gets the same update
            const float4 ni = P.nodes_inc[t];
            const float mi = ni.w;
            const float inv_mi = mi > 0.f ? 1.0f / mi : 0.0f;
            v3 vi = (mk(ni.x, ni.y, ni.z) + g * (mi * dt)) * inv_mi;
            vi = vclamp(vi, -lim, lim);
            P.nodes_inc[t] = make_float4(vi.x, vi.y, vi.z, mi);
        }
#endif
    }
}

// CPIC context of one block for G2P: the incompatible velocities and node
// distance fields of its 6x6x6 halo, and the colliders it sees.
struct CpicCtx {
    const float4* halo_inc;
    const uint2* halo_cdf;  // affinity bits, closest collider
    const DevCollider* cols;
    uint32_t ncols;
};

// Velocity of shared-halo node t (t = x + 6 y + 36 z, x, y, z in [0, 6)) of
// block b: node (x mod 4, ...) of the block itself or of one of its +1
// neighbours; zero where that neighbour is not active.
__device__ __forceinline__ float4 halo_node(const DevPtrs& P, uint32_t b, uint32_t t) {
    const uint32_t tx = t % 6u, ty = (t / 6u) % 6u, tz = t / 36u;
    const uint32_t ox = tx >= 4u, oy = ty >= 4u, oz = tz >= 4u;
    const uint32_t oct = ox * 4u + oy * 2u + oz;
    const uint32_t blk = oct == 0 ? b : P.nbh[b * NUM_NBH + oct - 1u];
    if (blk == NONE) return make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 nd = P.nodes[blk * 64u + (tx - 4u * ox) + 4u * (ty - 4u * oy) + 16u * (tz - 4u * oz)];
    return make_float4(nd.x, nd.y, nd.z, 0.f);
}

#ifndef NXM_G2P_THREADS
#define NXM_G2P_THREADS 256
#endif
constexpr uint32_t kG2pThreads = NXM_G2P_THREADS;  // threads per G2P CTA

// g2p.rs:150-270 (non-CPIC) fused with particle_update.rs:60-201 for one
// particle: gathers velocity and velocity gradient from the 6x6x6 halo of its
// block (shared memory), then advects, updates F and the model, and writes the
// particle (read from slot `src`, xm / vf = its first two kin words) to slot
// `dst` of the output records, together with the block key of its new position.
// The fast build takes the particle's cell from the sort: its block's
// coordinates (in its scene) and its associated cell there.
// kCpicBlock: the CPIC branches (a block whose halo carries affinity bits);
// the plain instantiation serves every other block without their registers.
// kSlots: `slots` holds 68 bytes a thread of shared memory: the deformation
// record, the model state and the id come there by asynchronous copies while the
// gather runs (instead of waiting in registers), and m A waits there across the
// model update.
struct G2pSlots {
    float4 a[kG2pThreads], b[kG2pThreads], c[kG2pThreads];
    float4 st[kG2pThreads];  // model state words, where any material has some (P.has_state)
    uint32_t id[kG2pThreads];
};
__device__ __forceinline__ float4 reload(const float4* p) {  // a shared-memory read that stays one
    float4 r;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w)
                 : "r"((uint32_t)__cvta_generic_to_shared(p))
                 : "memory");
    return r;
}
// Where a particle's block is told from: its coordinates and key offset as
// values, or in shared memory, read when they are needed.
struct BlockHere {
    int4 v;
    int3 k;
    __device__ __forceinline__ int4 vid() const { return v; }
    __device__ __forceinline__ int3 key() const { return k; }
};
struct BlockStaged {
    const int4* v;
    const int4* k;
    __device__ __forceinline__ int4 vid() const { return *v; }
    __device__ __forceinline__ int3 key() const {
        const float4 r = reload(reinterpret_cast<const float4*>(k));
        return make_int3(__float_as_int(r.x), __float_as_int(r.y), __float_as_int(r.z));
    }
};
template <bool kCpicBlock, bool kSlots, class Block>
__device__ __forceinline__ void g2p_particle(const DevPtrs& P, const Params& prm, const float4* __restrict__ halo,
                                             uint32_t src, uint32_t dst, float4 xm, uint32_t flags, const Block& block,
                                             uint32_t cell, const CpicCtx& cx, volatile float* stash,
                                             G2pSlots* slots) {
    const float dx = prm.dx, dt = prm.dt;
    const float inv_d = prm.inv_d;
    const v3 pt = mk(xm.x, xm.y, xm.z);
    float mass = xm.w;
    // the deformation record, fetched ahead of the gather; pm: F's last, V0, damping, material
    float4 pm;
    m3 F;
    if (kSlots) {
        const float4* f = reinterpret_cast<const float4*>(&P.in.def[src]);
        async_copy<16>(&slots->a[threadIdx.x], f);
        async_copy<16>(&slots->b[threadIdx.x], f + 1);
        async_copy<16>(&slots->c[threadIdx.x], &P.in.mat[src]);
        async_copy<4>(&slots->id[threadIdx.x], &P.pid_in[src]);
        if (P.has_state) async_copy<16>(&slots->st[threadIdx.x], &P.in.pstate[src]);
        async_commit();
    } else {
        pm = *reinterpret_cast<const float4*>(&P.in.mat[src]);
        F = def_grad_of(P.in, src, pm.x);
    }

#if NXM_CPIC
    // particle Cdf (normal, signed distance, affinity) from this step's g2p_cdf pass
    const bool cpic = kCpicBlock;
    float4 crec0 = make_float4(0.f, 0.f, 0.f, 0.f), crec1 = crec0;
    float bfric = 1.0f;
    if (cpic) {
        crec0 = P.pcdf[3u * src];
        crec1 = P.pcdf[3u * src + 1u];
        bfric = P.pcdf[3u * src + 2u].x;
    }
    const uint32_t paff = __float_as_uint(crec1.w);
    const v3 pnormal = mk(crec0.x, crec0.y, crec0.z);
    v3 rigid_vel = splat(0.f);
#else
    (void)cx;
#endif
    (void)cell;
    // ---- G2P (g2p.rs:150-270)
    v3 velocity = splat(0.f);
    m3 grad = mzero();
    float vgd = 0.f;
#if NXM_CPIC
    // a particle with affinity bits may meet incompatible nodes: per-node gather below
    const bool factored = NXM_FAST && !(cpic && paff != 0u);
#else
    const bool factored = NXM_FAST;
#endif
    if ((flags & PFLAG_ENABLED) && factored) {
        // Same sums, factored: with dpt_i = ref + s_i dx,
        //   grad = inv_d (v (x) ref + dx [Sx Sy Sz]),  S_a = sum_i w_i v_i s_i,a
        //   vgd  = inv_d (v . ref + dx (Sx.x + Sy.y + Sz.z))
        // and, the weights being products, summed along x, then y, then z: 240
        // multiply-adds (a weight product per node and the three moments summed
        // over the 27 nodes take 310).
        const float inv_dx = prm.inv_dx;
        const uint32_t ax = cell & 3u, ay = (cell >> 2) & 3u, az = cell >> 4;
        const int4 vid = block.vid();  // scene-local
        v3 ref = mk((float)(vid.x * 4 + (int)ax), (float)(vid.y * 4 + (int)ay), (float)(vid.z * 4 + (int)az)) * dx - pt;
        // a block beyond the packed keys' range carries the aliased coordinates
        if (fmaxf(fmaxf(fabsf(ref.x), fabsf(ref.y)), fabsf(ref.z)) > 4.0f * dx) ref = assoc_cell_of(dx, pt) * dx - pt;
        const v3 wx = kernel_eval_all(-ref.x * inv_dx);
        const v3 wy = kernel_eval_all(-ref.y * inv_dx);
        const v3 wz = kernel_eval_all(-ref.z * inv_dx);
        const float wx2 = 2.0f * wx.z, wy2 = 2.0f * wy.z, wz2 = 2.0f * wz.z;
        const float4* node = halo + ax + 6u * ay + 36u * az;
        v3 sxv = splat(0.f), syv = sxv, szv = sxv;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            v3 a = splat(0.f), bx = a, by = a;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const float4 h0 = node[6 * j + 36 * k], h1 = node[1 + 6 * j + 36 * k], h2 = node[2 + 6 * j + 36 * k];
                const v3 s0 = mk(h0.x, h0.y, h0.z) * wx.x + mk(h1.x, h1.y, h1.z) * wx.y + mk(h2.x, h2.y, h2.z) * wx.z;
                const v3 s1 = mk(h1.x, h1.y, h1.z) * wx.y + mk(h2.x, h2.y, h2.z) * wx2;
                a = a + s0 * vget(wy, j);
                bx = bx + s1 * vget(wy, j);
                if (j) by = by + s0 * (j == 1 ? wy.y : wy2);
            }
            velocity = velocity + a * vget(wz, k);
            sxv = sxv + bx * vget(wz, k);
            syv = syv + by * vget(wz, k);
            if (k) szv = szv + a * (k == 1 ? wz.y : wz2);
        }
        grad = (outer(velocity, ref) + mkm(sxv, syv, szv) * dx) * inv_d;
        vgd = (dot(velocity, ref) + dx * (sxv.x + syv.y + szv.z)) * inv_d;
    } else if (flags & PFLAG_ENABLED) {
        const v3 ref = assoc_cell_of(dx, pt) * dx - pt;
        const v3 w0 = kernel_eval_all(-ref.x / dx);
        const v3 w1 = kernel_eval_all(-ref.y / dx);
        const v3 w2 = kernel_eval_all(-ref.z / dx);
        const CellInfo ci = cell_info(dx, pt);
        const uint32_t packed = ci.ax + 6u * ci.ay + 36u * ci.az;
#pragma unroll
        for (int i = 0; i < 27; ++i) {
            int sx, sy, sz;
            nbh_shift(i, sx, sy, sz);
            const uint32_t hid = packed + (uint32_t)(sx + 6 * sy + 36 * sz);
            const float4 h = halo[hid];
            v3 cv = mk(h.x, h.y, h.z);
            const v3 dpt = ref + mk((float)sx, (float)sy, (float)sz) * dx;
#if NXM_CPIC
            if (cpic) {
                // g2p.rs:206-235: an incompatible node gives its second velocity,
                // projected by its closest body's boundary condition
                const uint2 nc = cx.halo_cdf[hid];
                if (!aff_compatible(paff, nc.x)) {
                    const float4 hi = cx.halo_inc[hid];
                    cv = mk(hi.x, hi.y, hi.z);
                    if (nc.y != NONE) {
                        const DevCollider& c = cx.cols[nc.y];
                        const v3 cell_center = dpt + pt;
                        const v3 bv = col_vel_at(c, cell_center);
                        cv = bv + bc_project(c.bc_type, c.bc_friction * bfric, cv - bv, pnormal);
                    }
                }
            }
#endif
            const float weight = vget(w0, sx) * vget(w1, sy) * vget(w2, sz);
            velocity = velocity + cv * weight;
            grad = grad + outer(cv, dpt) * (weight * inv_d);
            vgd += weight * inv_d * dot(cv, dpt);
        }
#if NXM_CPIC
        if (cpic)  // g2p.rs:248-262: velocity of every body the particle has affinity with
            for (uint32_t ic = 0; ic < 16u && ic < cx.ncols; ++ic)
                if (paff & (1u << ic)) rigid_vel = rigid_vel + col_vel_at(cx.cols[ic], pt);
#endif
    }
#if NXM_CPIC
    if (cpic) P.pcdf[3u * src + 1u] = make_float4(rigid_vel.x, rigid_vel.y, rigid_vel.z, crec1.w);
#endif

    // ---- particle update (particle_update.rs:60-201, non-CPIC: Cdf = 0)
    if (kSlots) {
        async_wait<0>();
        const float4 f0 = slots->a[threadIdx.x], f1 = slots->b[threadIdx.x];
        pm = slots->c[threadIdx.x];
        F = mkm(mk(f0.x, f0.y, f0.z), mk(f0.w, f1.x, f1.y), mk(f1.z, f1.w, pm.x));
    }
    const float init_volume = pm.y, damping = pm.z;
    const uint32_t mid = __float_as_uint(pm.w);
    const Material& mat = P.materials[mid];
    const uint32_t tag = mat.tag;

    v3 v = velocity;
#if NXM_CPIC
    // particle_update.rs:98-102: reproject a penetrating particle
    if (cpic && crec0.w < -0.05f * dx) v = rigid_vel + bc_project(BC_SLIP, 0.0f, v - rigid_vel, pnormal);
#endif
    if (NXM_FAST) {
        // the square root only near or above the limit
        if (dot(v, v) > 0.999f * prm.speed_limit2) {
            const float vl = length(v);
            if (vl > dx / dt) v = ((v / vl) * dx) / dt;
        }
    } else {
        const float vl = length(v);
        if (vl > dx / dt) v = ((v / vl) * dx) / dt;
    }
    if (NXM_FAST) v = v * (1.0f / (1.0f + damping * dt));  // one division instead of three
    else v = v / (1.0f + damping * dt);
    if (flags & PFLAG_FIXED) v = splat(0.f);
    const v3 np_ = pt + v * dt;
#if NXM_CPIC
    if (cpic && crec0.w < -0.05f * dx) {  // particle_update.rs:132-136 penalty, PENALTY_COEFF = 1e3
        const float corrected = fmaxf(crec0.w, -0.3f * dx);
        v = v + pnormal * (dt * -corrected * 1.0e3f);
    }
#endif
    // The new position, velocity and block key follow from the gather alone:
    // written ahead of the constitutive update (fewer values live across it);
    // a particle that the check after it disables is rewritten there.
    const bool nan = (np_.x != np_.x) || (np_.y != np_.y) || (np_.z != np_.z);
    store8(&P.out.kin[dst], np_.x, np_.y, np_.z, mass, v.x, v.y, v.z, __uint_as_float(flags));
    {
        const CellInfo nc = NXM_FAST ? cell_info_near(dx, prm.inv_dx, np_) : cell_info(dx, np_);
        const int3 key_off = block.key();
        P.pcode[dst] = make_uint2(pack_key(nc.bx + key_off.x, nc.by + key_off.y, nc.bz + key_off.z),
                                  nc.ax | (nc.ay << 2) | (nc.az << 4));
    }
    const m3 A = grad;
    if (tag != MODEL_FLUID) {
        F = F + (A * dt) * F;
    } else {
        const float fd0 = F.c0.x;
        float rate = vgd * dt / 3.0f;
        rate = rclamp(rate, -0.1f, 0.1f);
        const float nd = rclamp(fd0 + rate * fd0, 0.5f, 2.0f);
        F = diag(splat(nd));
    }
    float st[4] = {0.f, 0.f, 0.f, 0.f};
    if (mat.has_state) {
        const float4 s4 = kSlots ? slots->st[threadIdx.x] : P.in.pstate[src];
        st[0] = s4.x; st[1] = s4.y; st[2] = s4.z; st[3] = s4.w;
    }
    m3 aff;
    if (kSlots && tag != MODEL_FLUID) {
        const m3 am = A * mass;
        slots->a[threadIdx.x] = make_float4(am.c0.x, am.c0.y, am.c0.z, am.c1.x);
        slots->b[threadIdx.x] = make_float4(am.c1.y, am.c1.z, am.c2.x, am.c2.y);
        slots->c[threadIdx.x].x = am.c2.z;
        const m3 tau = model_update<NXM_FAST>(tag, mat.w, st, F, mzero());
        const float4 a = reload(&slots->a[threadIdx.x]), b = reload(&slots->b[threadIdx.x]);
        const float4 c = reload(&slots->c[threadIdx.x]);
        aff = mkm(mk(a.x, a.y, a.z), mk(a.w, b.x, b.y), mk(b.z, b.w, c.x)) - tau * (init_volume * inv_d * dt);
    } else if (!kSlots && stash && tag != MODEL_FLUID) {
        // m A waits in this thread's shared-memory slots (stride kG2pThreads) across
        // the model update instead of in registers
        const m3 am = A * mass;
        const float* e = &am.c0.x;
#pragma unroll
        for (int i = 0; i < 9; ++i) stash[kG2pThreads * i] = e[i];
        const m3 tau = model_update<NXM_FAST>(tag, mat.w, st, F, mzero());
        float r[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) r[i] = stash[kG2pThreads * i];
        aff = mkm(mk(r[0], r[1], r[2]), mk(r[3], r[4], r[5]), mk(r[6], r[7], r[8])) -
              tau * (init_volume * inv_d * dt);
    } else {
        const m3 tau = model_update<NXM_FAST>(tag, mat.w, st, F, A);
        aff = A * mass - tau * (init_volume * inv_d * dt);
    }
    if (nan || !(det(F) > 0.0f)) {  // disabled: rewrite what was written ahead
        flags &= ~PFLAG_ENABLED;
        F = mident();
        aff = mzero();
        // at its old position: kSlots writes to the other buffer, so it is re-read
        // instead of staying live across the model update; in place (deterministic
        // and CPIC) the record already holds the new one
        v3 op = pt;
        if (kSlots) {
            const PKin& old = P.in.kin[P.sorted[dst]];
            op = mk(old.x, old.y, old.z);
        }
        store8(&P.out.kin[dst], op.x, op.y, op.z, 0.f, 0.f, 0.f, 0.f, __uint_as_float(flags));
        const CellInfo oc = cell_info(dx, op);
        const int3 key_off = block.key();
        P.pcode[dst] = make_uint2(pack_key(oc.bx + key_off.x, oc.by + key_off.y, oc.bz + key_off.z),
                                  oc.ax | (oc.ay << 2) | (oc.az << 4));
    }
    store8(&P.out.aff[dst], aff.c0.x, aff.c0.y, aff.c0.z, aff.c1.x, aff.c1.y, aff.c1.z, aff.c2.x, aff.c2.y);
    *reinterpret_cast<float2*>(&P.out.tail[dst]) = make_float2(aff.c2.z, vgd);
    store8(&P.out.def[dst], F.c0.x, F.c0.y, F.c0.z, F.c1.x, F.c1.y, F.c1.z, F.c2.x, F.c2.y);
    *reinterpret_cast<float4*>(&P.out.mat[dst]) = make_float4(F.c2.z, init_volume, damping, pm.w);
    if (mat.has_state) P.out.pstate[dst] = make_float4(st[0], st[1], st[2], st[3]);
    if (kSlots) P.pid_out[dst] = slots->id[threadIdx.x];
    else if (P.pid_in) P.pid_out[dst] = P.pid_in[src];
}

// dynamics/body.rs Velocity::integrate for one-way coupled bodies
// (rigid_impulses.rs:66-140 with zero impulse and zero inverse mass): the
// pose of every collider the step moves (all, at most 16, or every scene's
// in batched mode) advances by its velocities over dt.  Run by the first
// threads of the G2P launch, one collider each: nothing in G2P reads a
// collider's rotation or translation (the body velocities it reads use the
// centre of mass refreshed at the start of the step), and the next reader is
// the next step's sort.
__device__ __forceinline__ void integrate_colliders(const DevPtrs& P, const Params& prm) {
    const uint32_t ncol = prm.scene_blocks ? prm.ncol : min(prm.ncol, (uint32_t)MAX_COLLIDERS);
    const float dt = prm.dt;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < ncol; i += gridDim.x * blockDim.x) {
        DevCollider& c = P.colliders[i];
        const quat q = quat{c.rot[0], c.rot[1], c.rot[2], c.rot[3]};
        const v3 tra = mk(c.tra[0], c.tra[1], c.tra[2]);
        const v3 init_com = qrot(q, mk(c.local_com[0], c.local_com[1], c.local_com[2])) + tra;
        const v3 sa = mk(c.angvel[0], c.angvel[1], c.angvel[2]) * dt;
        const float ang = length(sa);
        quat dq;
        if (ang == 0.f) {
            dq = quat{0.f, 0.f, 0.f, 1.f};
        } else {
            const v3 ax = sa / ang;
            const float sh = sinf(ang * 0.5f), ch = cosf(ang * 0.5f);
            dq = quat{ax.x * sh, ax.y * sh, ax.z * sh, ch};
        }
        const v3 dl = mk(c.linvel[0], c.linvel[1], c.linvel[2]) * dt;
        const v3 nt = (init_com + qrot(dq, tra - init_com)) + dl;
        quat nr;
        nr.w = dq.w * q.w - dq.x * q.x - dq.y * q.y - dq.z * q.z;
        nr.x = dq.w * q.x + dq.x * q.w + dq.y * q.z - dq.z * q.y;
        nr.y = dq.w * q.y - dq.x * q.z + dq.y * q.w + dq.z * q.x;
        nr.z = dq.w * q.z + dq.x * q.y - dq.y * q.x + dq.z * q.w;
        const float rl = 1.0f / sqrtf(nr.x * nr.x + nr.y * nr.y + nr.z * nr.z + nr.w * nr.w);
        c.rot[0] = nr.x * rl; c.rot[1] = nr.y * rl; c.rot[2] = nr.z * rl; c.rot[3] = nr.w * rl;
        c.tra[0] = nt.x; c.tra[1] = nt.y; c.tra[2] = nt.z;
    }
}

// End of a G2P launch: when reordering, the particles the sort could not
// place (their block was not created: capacity or hash overflow, reported in
// the status word) are copied unchanged to the slots after the sorted ones;
// then the cached block keys are marked valid.
__device__ __forceinline__ void g2p_finish(const DevPtrs& P, const Params& prm) {
    if (P.pid_in) {
        const uint32_t n = prm.n, sl = __ldcg(&P.counters->sorted_len);
        for (uint32_t p = sl < n ? blockIdx.x * blockDim.x + threadIdx.x : n; p < n; p += gridDim.x * blockDim.x) {
            if (__ldcg(&P.phdr[p]) != NONE) continue;
            const uint32_t dst = sl + atomicAdd(&P.counters->unsorted, 1u);
            if (dst >= n) continue;  // not reached: exactly n - sl particles have no header
            P.out.kin[dst] = P.in.kin[p];
            P.out.aff[dst] = P.in.aff[p];
            P.out.tail[dst] = P.in.tail[p];
            P.out.def[dst] = P.in.def[p];
            P.out.mat[dst] = P.in.mat[p];
            P.out.pstate[dst] = P.in.pstate[p];
            P.pid_out[dst] = P.pid_in[p];
            const CellInfo nc = cell_info(prm.dx, mk(P.in.kin[p].x, P.in.kin[p].y, P.in.kin[p].z));
            const int3 o = prm.scene_blocks ? scene_base_of(prm, P.pscene[P.pid_in[p]]) : make_int3(0, 0, 0);
            P.pcode[dst] = make_uint2(pack_key(nc.bx + o.x, nc.by + o.y, nc.bz + o.z),
                                      nc.ax | (nc.ay << 2) | (nc.az << 4));
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) P.counters->codes_valid = 1u;
}

// CTAs per SM the register budget is sized for: at 4 (64 registers) the spills
// around the constitutive update cost more than the fourth CTA's latency hiding
// gives (2 M sand + water: 178 us at 4, 166 us at 3; 48 small scenes 129, 124).
#ifndef NXM_G2P_MIN_CTAS
#define NXM_G2P_MIN_CTAS 3
#endif
// k_g2p_update (a block a CTA) at 4: sparse scenes wait for each block's loads, and
// their step loses more at 3 than crowded ones gain (deterministic, 100,000
// particles over 198,000 blocks: 881 us at 3, 695 at 4; 110,000 in 64 blocks 76, 82).
#ifndef NXM_G2P_BLOCK_CTAS
#define NXM_G2P_BLOCK_CTAS 4
#endif

// One CTA per primary block (ids [0, num_primary); the other blocks hold no
// particles), grid-stride: the halo of the block and its +1 neighbours is
// staged in shared memory, then each thread gathers and updates one of the
// block's primary particles.  The next block's header is loaded one block
// ahead, and each thread's first particle is fetched alongside the halo so
// that the two dependent load chains overlap.  When reordering, sorted entry
// j = first + k goes to output slot j; particles the sort could not place
// (their block was not created: capacity or hash overflow, reported in the
// status word) are copied unchanged to the slots after the sorted ones.
#ifndef NXM_G2P_STASH
#define NXM_G2P_STASH 1  // m A waits in shared memory across the model update (fast build)
#endif
// Below prm.range_min_fill particles a block on average (64 unless tuned), a
// run of the fast G2P (k_g2p_range) would span more blocks than one pass
// stages: such a launch (decided on the device from this step's counts, the
// same in every CTA) runs the per-block loop, where the blocks of a small
// sparse scene are side by side on many CTAs instead of passes in a row on a
// few.
__device__ __forceinline__ bool g2p_sparse(const DevPtrs& P, const Params& prm) {
    const uint32_t nbp = min(__ldcg(&P.counters->num_primary), __ldcg(&P.counters->num_blocks));
    const uint32_t len = min(__ldcg(&P.counters->sorted_len), prm.n);
    return (uint64_t)len < (uint64_t)prm.range_min_fill * nbp;
}

#if !NXM_FAST || NXM_CPIC
// The per-block loop: one CTA per primary block (grid-stride), halo of 216
// nodes in `halo` (CPIC: the incompatible fields and node distance field in
// halo_inc / halo_cdf).
__device__ __forceinline__ void g2p_block_loop(const DevPtrs& P, const Params& prm, float4* halo, float4* halo_inc,
                                               uint2* halo_cdf, volatile float* stash) {
    (void)halo_inc;
    (void)halo_cdf;
    const uint32_t nbp = min(__ldcg(&P.counters->num_primary), __ldcg(&P.counters->num_blocks));
    const uint32_t tid = threadIdx.x;
    const uint32_t ht = tid < 216u ? tid : 0u;  // halo node of this thread
    const uint32_t htx = ht % 6u, hty = (ht / 6u) % 6u, htz = ht / 36u;
    const uint32_t hox = htx >= 4u, hoy = hty >= 4u, hoz = htz >= 4u;
    const uint32_t hoct = hox * 4u + hoy * 2u + hoz;
    const uint32_t hnode = (htx - 4u * hox) + 4u * (hty - 4u * hoy) + 16u * (htz - 4u * hoz);
    uint32_t b = blockIdx.x;
    uint32_t first = 0, np = 0;
    if (b < nbp) {
        first = __ldcg(&P.first[b]);
        np = __ldcg(&P.nprim[b]);
    }
    while (b < nbp) {
        const uint32_t bn = b + gridDim.x;
        uint32_t nfirst = 0, nnp = 0;
        if (bn < nbp) {
            nfirst = __ldcg(&P.first[bn]);
            nnp = __ldcg(&P.nprim[bn]);
        }
        const bool reorder = P.pid_in != nullptr;
        BlockHere block{P.bvid[b], make_int3(0, 0, 0)};
        block.k = scene_base_of_block(prm, block.v);
        block.v.x -= block.k.x; block.v.y -= block.k.y; block.v.z -= block.k.z;
        uint32_t pid = tid < np ? __ldg(&P.sorted[first + tid]) : NONE;
        const uint32_t hblk = (tid < 216u && hoct != 0u) ? __ldg(&P.nbh[b * NUM_NBH + hoct - 1u]) : b;
        float4 xm = make_float4(0.f, 0.f, 0.f, 0.f), vf = xm;
        if (pid != NONE) {
            const float4* kr = reinterpret_cast<const float4*>(&P.in.kin[pid]);
            xm = kr[0];
            vf = kr[1];
        }
        if (tid < 216u) {
            float4 nd = make_float4(0.f, 0.f, 0.f, 0.f);
            if (hblk != NONE) nd = P.nodes[hblk * 64u + hnode];
            halo[tid] = make_float4(nd.x, nd.y, nd.z, 0.f);
        }
        for (uint32_t t = tid + blockDim.x; t < 216u; t += blockDim.x) halo[t] = halo_node(P, b, t);
        CpicCtx cx{nullptr, nullptr, P.colliders, 0u};
#if NXM_CPIC
        // A halo whose nodes carry no affinity bit gave every particle of the
        // block an empty affinity and a zero distance record (g2p_cdf): all
        // nodes are compatible, no body velocity enters and the record stays
        // zero, so the block runs the plain transfer (halo_cdf left null).
        bool cpic_block = false;
        if (prm.use_cpic) {
            uint32_t any = 0u;
            for (uint32_t t = tid; t < 216u; t += blockDim.x) {
                const uint32_t tx = t % 6u, ty = (t / 6u) % 6u, tz = t / 36u;
                const uint32_t ox = tx >= 4u, oy = ty >= 4u, oz = tz >= 4u;
                const uint32_t oct = ox * 4u + oy * 2u + oz;
                const uint32_t blk = oct == 0 ? b : P.nbh[b * NUM_NBH + oct - 1u];
                const uint32_t node = (tx - 4u * ox) + 4u * (ty - 4u * oy) + 16u * (tz - 4u * oz);
                const uint4 nc = blk == NONE ? make_uint4(0u, 0u, NONE, 0u) : P.ncdf[blk * 64u + node];
                halo_cdf[t] = make_uint2(nc.y, nc.z);
                any |= nc.y;
            }
            cpic_block = __syncthreads_or((int)(any & 0x0000FFFFu)) != 0;
        }
        if (cpic_block) {
            for (uint32_t t = tid; t < 216u; t += blockDim.x) {
                const uint32_t tx = t % 6u, ty = (t / 6u) % 6u, tz = t / 36u;
                const uint32_t ox = tx >= 4u, oy = ty >= 4u, oz = tz >= 4u;
                const uint32_t oct = ox * 4u + oy * 2u + oz;
                const uint32_t blk = oct == 0 ? b : P.nbh[b * NUM_NBH + oct - 1u];
                const uint32_t node = (tx - 4u * ox) + 4u * (ty - 4u * oy) + 16u * (tz - 4u * oz);
                halo_inc[t] = blk == NONE ? make_float4(0.f, 0.f, 0.f, 0.f) : P.nodes_inc[blk * 64u + node];
            }
            cx.halo_inc = halo_inc;
            cx.halo_cdf = halo_cdf;
            if (prm.scene_blocks) {
                const uint32_t sid = scene_of_block(prm, P.bvid[b]);
                const uint2 r = sid != NONE ? P.scene_cols[sid] : make_uint2(0u, 0u);
                cx.cols = P.colliders + r.x;
                cx.ncols = min(r.y, (uint32_t)MAX_COLLIDERS);
            } else {
                cx.ncols = min(prm.ncol, (uint32_t)MAX_COLLIDERS);
            }
        }
#endif
        __syncthreads();
        for (uint32_t k = tid; k < np; k += blockDim.x) {
            if (k != tid) {
                pid = P.sorted[first + k];
                const float4* kr = reinterpret_cast<const float4*>(&P.in.kin[pid]);
                xm = kr[0];
                vf = kr[1];
            }
            const uint32_t cell = NXM_FAST ? __ldcg(&P.phdr[pid]) & 63u : 0u;
#if NXM_CPIC
            if (cx.halo_cdf)
                g2p_particle<true, false>(P, prm, halo, pid, reorder ? first + k : pid, xm, __float_as_uint(vf.w), block,
                                          cell, cx, stash, nullptr);
            else
#endif
                g2p_particle<false, false>(P, prm, halo, pid, reorder ? first + k : pid, xm, __float_as_uint(vf.w), block,
                                           cell, cx, stash, nullptr);
        }
        __syncthreads();
        b = bn;
        first = nfirst;
        np = nnp;
    }
}

__global__ void __launch_bounds__(kG2pThreads, NXM_G2P_BLOCK_CTAS) k_g2p_update(DevPtrs P) {
    after_previous();
    __shared__ float4 halo[216];
#if NXM_G2P_STASH
    __shared__ float stash_mem[9 * kG2pThreads];
    volatile float* stash = NXM_FAST ? stash_mem + threadIdx.x : nullptr;
#else
    volatile float* stash = nullptr;
#endif
#if NXM_CPIC
    __shared__ float4 halo_inc[216];
    __shared__ uint2 halo_cdf[216];
#else
    float4* halo_inc = nullptr;
    uint2* halo_cdf = nullptr;
#endif
    const Params prm = *P.params;
    integrate_colliders(P, prm);
    g2p_block_loop(P, prm, halo, halo_inc, halo_cdf, stash);
    g2p_finish(P, prm);
}

#endif

#if NXM_FAST && !NXM_CPIC
// ---- a copy-barrier wait with an iteration limit ----------------------------
// An mbarrier in shared memory as bulk copies complete on; a wait on its phase
// gives up after `limit` rounds, so that a kernel can record STATUS_COPY_TIMEOUT
// instead of waiting on.  Reached by nxm_debug_copy_wait_timeout alone: no step
// kernel copies this way (halos by bulk copies were slower than plain loads).
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// Waits for the barrier's phase `parity` to complete; false when the limit ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t limit) {
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t done;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// The wait made to run out: a barrier that expects bytes no copy will
// deliver (nothing is issued), waited on with `limit` rounds; the kernel
// records STATUS_COPY_TIMEOUT and returns with no copy in flight.
__global__ void k_copy_wait_timeout(Counters* counters, uint32_t limit) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar);
        mbar_expect_tx(&bar, 16u);
    }
    __syncthreads();
    if (!mbar_wait(&bar, 0u, limit) && threadIdx.x == 0) set_status(counters, STATUS_COPY_TIMEOUT);
}

// The fast build's G2P walks the sorted list in runs of kRangeChunk
// positions, one particle per thread, instead of one CTA per block: a block
// holds some 1-600 particles, so per-block rounds of 256 threads run part
// empty (three quarters full on a settled scene); a run fills every thread
// but one run's worth at the end.  The fast path lists no extras, so the
// positions [0, sorted_len) are exactly the primary particles, block after
// block; run c spans the blocks [chunk_blk[c], chunk_blk[c + 1]] (the scan
// records the block of each run's first position; the last run reaches the
// last primary block), usually one or two.  Their halos are staged
// kRangeHalos at a time, and each thread takes its particle's block and
// cell from the word the sort's count pass stored for it (phdr).  A run's span is
// loaded one run ahead, so that a run's own loads (ids, records, halos) are
// issued together.
//
// A launch over sparse blocks (g2p_sparse) takes one block per unit instead
// (its particles in rounds of 256), through the same loop: a unit is a span
// of blocks whose halos are staged in passes and a range of sorted positions
// the threads step through, so the particle update has one call site.
// Neighbouring positions are particles of the same cell or the next, so a
// warp's halo reads are mostly broadcasts.
//
// Bound by instruction issue and the latency of a run's first loads; 2 M sand +
// water particles: 193 us with the 27-node gather and records held in
// registers, 166 us now (0.25 GB, 1.5 TB/s); 500,000 snow particles 82, 73 us.
//
// Halo staging: every thread below 216 loads one node of each staged block
// (its block id from the neighbour table, then the node, both L2 hits).
constexpr uint32_t kRangeHalos = 8;
static_assert(kG2pThreads == kRangeChunk, "one sorted position per thread");
__global__ void __launch_bounds__(kG2pThreads, NXM_G2P_MIN_CTAS) k_g2p_range(DevPtrs P) {
    after_previous();
    __shared__ float4 halo[kRangeHalos * 216];
    __shared__ G2pSlots slots;
    __shared__ int4 svid[kRangeHalos], skey[kRangeHalos];  // the staged blocks' coordinates and key offsets
    // the parameters are read from shared memory where they are used: in
    // registers they would push the particle's own values out to local memory
    __shared__ Params prm;
    if (threadIdx.x < sizeof(Params) / 4)
        reinterpret_cast<uint32_t*>(&prm)[threadIdx.x] = reinterpret_cast<const uint32_t*>(P.params)[threadIdx.x];
    __syncthreads();
    integrate_colliders(P, prm);
    const uint32_t nbp = min(__ldcg(&P.counters->num_primary), __ldcg(&P.counters->num_blocks));
    const uint32_t len = min(__ldcg(&P.counters->sorted_len), prm.n);
    const bool sparse = g2p_sparse(P, prm);
    const uint32_t nunits = !nbp ? 0u : (sparse ? nbp : min((len + kRangeChunk - 1u) / kRangeChunk, P.chunk_cap));
    const uint32_t tid = threadIdx.x;
    // this thread's halo node: its octant and its place in that block
    const uint32_t htx = tid % 6u, hty = (tid / 6u) % 6u, htz = tid / 36u;
    const uint32_t hox = htx >= 4u, hoy = hty >= 4u, hoz = htz >= 4u;
    const uint32_t hnode = (hox * 4u + hoy * 2u + hoz) << 8 | ((htx - 4u * hox) + 4u * (hty - 4u * hoy) + 16u * (htz - 4u * hoz));
    const CpicCtx cx{nullptr, nullptr, P.colliders, 0u};
    // unit u: blocks [x, y], sorted positions [z, w), from two loaded words
    // (dense: the run's first and last block; sparse: first, nprim of the
    // block), loaded one unit ahead by one thread (a ring of four: others may
    // still look at the previous unit)
    __shared__ uint4 unit[4];
    const auto unit_of = [&](uint32_t u) {
        uint4 r = make_uint4(0u, 0u, 0u, 0u);
        if (u >= nunits) return r;
        if (sparse) {
            r.x = r.y = u;
            r.z = __ldcg(&P.first[u]);
            r.w = min(r.z + __ldcg(&P.nprim[u]), len);
        } else {
            r.x = __ldcg(&P.chunk_blk[u]);
            r.y = min(u + 1u < nunits ? __ldcg(&P.chunk_blk[u + 1u]) : nbp - 1u, nbp - 1u);
            r.z = u * kRangeChunk;
            r.w = min(r.z + kRangeChunk, len);
        }
        return r;
    };
    if (tid == 0) unit[0] = unit_of(blockIdx.x);
    __syncthreads();
    uint32_t slot = 0u;
    for (uint32_t u = blockIdx.x; u < nunits; u += gridDim.x, slot = (slot + 1u) & 3u) {
        if (tid == 0) unit[(slot + 1u) & 3u] = unit_of(u + gridDim.x);
        const uint4 cur = unit[slot];
        // this thread's first particle, fetched while the halos load
        uint32_t pid = cur.z + tid < cur.w ? __ldg(&P.sorted[cur.z + tid]) : NONE;
        float4 xm = make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t flags = 0u, home = cur.x << 6;  // home: the particle's block and cell
        const auto load_head = [&] {
            xm = *reinterpret_cast<const float4*>(&P.in.kin[pid]);
            flags = __float_as_uint(P.in.kin[pid].flags);
            home = __ldcg(&P.phdr[pid]);
        };
        if (pid != NONE) load_head();
        bool pending = pid != NONE;  // dense: this thread's one particle not yet updated
        for (uint32_t b = cur.x; b <= unit[slot].y; b += kRangeHalos) {
            const uint32_t cnt = min(unit[slot].y - b + 1u, kRangeHalos);
            if (tid >= kG2pThreads - kRangeHalos && tid - (kG2pThreads - kRangeHalos) < cnt) {  // no halo node of theirs
                const uint32_t i = tid - (kG2pThreads - kRangeHalos);
                const int4 v = P.bvid[b + i];
                const int3 o = scene_base_of_block(prm, v);
                svid[i] = make_int4(v.x - o.x, v.y - o.y, v.z - o.z, v.w);
                skey[i] = make_int4(o.x, o.y, o.z, 0);
            }
            if (tid < 216u) {
                const uint32_t oct = hnode >> 8, at = hnode & 255u;
#pragma unroll 2
                for (uint32_t i = 0; i < cnt; ++i) {
                    const uint32_t blk = oct ? __ldg(&P.nbh[(b + i) * NUM_NBH + oct - 1u]) : b + i;
                    float4 nd = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (blk != NONE) nd = P.nodes[blk * 64u + at];
                    halo[216u * i + tid] = nd;
                }
            }
            __syncthreads();
            // dense: one position per thread; sparse: the block's positions in rounds
            for (uint32_t p = unit[slot].z + tid; p < unit[slot].w; p += kG2pThreads) {
                if (p >= unit[slot].z + kG2pThreads) {
                    pid = __ldg(&P.sorted[p]);
                    load_head();
                }
                const uint32_t at = (home >> 6) - b;
                if (at < cnt) {
                    g2p_particle<false, true>(P, prm, halo + 216u * at, pid, p, xm, flags,
                                              BlockStaged{svid + at, skey + at}, home & 63u, cx, nullptr, &slots);
                    pending = false;
                }
            }
            __syncthreads();
        }
        if (!sparse && pending) set_status(P.counters, STATUS_MISSING_BLOCK);  // not reached: a run holds its blocks
    }
    g2p_finish(P, prm);
}
#endif

}  // namespace

#if NXM_FAST && !NXM_CPIC
void launch_copy_wait_timeout(Counters* counters, uint32_t limit, cudaStream_t s) {
    k_copy_wait_timeout<<<1, 32, 0, s>>>(counters, limit);
}
#endif

// Grids stop at what the state's capacities can use: a CTA a block, or a run of
// the sorted list each (a small scene's launch is mostly the start of its CTAs).
void launch_grid_update(const DevPtrs& P, const LaunchCfg& c, cudaStream_t s) {
    // grid_ctas counts CTAs of 256 threads
    const uint32_t most = (uint32_t)c.sm_count * c.t.grid_ctas * (256 / kGridThreads);
    launch_after(k_grid_update, (int)min(max(c.block_capacity, 1u), most), kGridThreads, 0, s, P);
}

int launch_g2p_update(const DevPtrs& P, const LaunchCfg& c, cudaStream_t s) {
    const uint32_t primaries = min(c.block_capacity, c.particle_capacity);
    const uint32_t units = max(max(primaries, (c.particle_capacity + kRangeChunk - 1u) / kRangeChunk), 1u);
#if NXM_FAST && !NXM_CPIC
    const uint32_t most = (uint32_t)c.sm_count * min(c.t.g2p_ctas, (uint32_t)NXM_G2P_MIN_CTAS);
    launch_after(k_g2p_range, (int)min(units, most), kG2pThreads, 0, s, P);
#else
    launch_after(k_g2p_update, (int)min(units, (uint32_t)c.sm_count * NXM_G2P_BLOCK_CTAS), kG2pThreads, 0, s, P);
#endif
    return 1;
}

}  // namespace NXM_NS
}  // namespace nxm
