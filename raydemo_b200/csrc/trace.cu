// Closest-hit traversal (compiled with --fmad=false).
//
// World level: for every mesh instance, the reference's instance box test
// (bbox_test with safe_invert, CoreRef.cpp:64-86, 272-294) and TransformRay
// (CoreRef.cpp:1605-1617), both reproduced operation for operation. Mesh
// level: the compressed 8-wide BVH, traversed with node groups (a base index
// plus a hit mask of up to 8 children) on a per-thread stack, children in
// octant order, which is roughly front to back; the triangles of the leaf
// children a node step hits (up to 24) are tested at once. Triangles use the
// reference's intersection arithmetic (CoreRef.cpp:11-42) with every product
// and sum rounded on its own, so t, u, v are bit-exact; a tie on t goes to the
// lower triangle index, which makes the result independent of visiting order.
//
// The kernels share the traversal step:
//   k_trace_closest      one thread per ray (a grid over the rays)
//   k_trace_persistent   a resident grid; a lane whose ray is done takes the
//                        next one from a global counter (warp-aggregated), so
//                        more lanes do useful work per instruction on
//                        incoherent rays of very different lengths
//   k_trace_closest_one  its closest-hit, one-triangle-per-step form for
//                        scenes without an instance tree, register-bounded
// The persistent kernels trace a ray with eight lanes, one per child of a
// node and one per triangle of a leaf, where rays are few: launches of at most
// one wave of such groups, and every launch's last rays (a warp with no more
// than four left and none to take). There a ray's steps follow one another
// with nothing to hide them, and a step's latency is what counts.
// The stack holds one node group per tree level at most. It lives in shared
// memory; meshes deeper than that use the DEEP instances, which continue it
// in a local array.
#include <algorithm>
#include <type_traits>

#include "trace.cuh"
#include "traverse.cuh"

namespace rg {
namespace {

using namespace trav;

// shared stack entries of the counting, any-hit and multi-scene launches
constexpr int LOOP_STACK = 16;
constexpr uint32_t MI_DONE = 0xfffffffeu; // no further instance of the ray to look for

// Ray counts up to which a launch traces every ray with eight lanes: as many
// groups of eight as the resident grid has. Measured on B200 (20,000
// triangles, one lane / eight lanes a ray): 100 rays 77 / 57 us, 1,000 109 /
// 75, 10,000 111 / 100, 20,000 116 / 113; beyond one wave of groups the single
// lanes win (40,000 rays 134 / 162).
constexpr uint32_t coop_rays(int blocks, int block) { return (uint32_t)blocks * (uint32_t)block / 8u; }

template <bool COUNT>
__device__ __forceinline__ void flush_counters(uint32_t err, uint32_t nvis, uint32_t ntri, uint32_t *err_out, unsigned long long *counters) {
    if (err) atomicOr(err_out, err);
    if (COUNT) {
        unsigned long long a = nvis, b = ntri;
        for (int off = 16; off; off >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, off);
            b += __shfl_xor_sync(0xffffffffu, b, off);
        }
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(&counters[0], a);
            atomicAdd(&counters[1], b);
        }
    }
}

template <bool COUNT, bool DEEP, bool TLAS = false>
__global__ void __launch_bounds__(TRACE_BLOCK) k_trace_closest(SceneView sv, const float4 *__restrict__ rays, uint32_t n, float4 *__restrict__ hits,
                                                               int32_t *__restrict__ obj_out, uint32_t *__restrict__ err_out,
                                                               unsigned long long *__restrict__ counters, const uint32_t *__restrict__ n_dev,
                                                               const uint32_t *__restrict__ order) {
    __shared__ uint2 s_stack[SMEM_STACK * TRACE_BLOCK];
    Stack<DEEP> st;
    st.smem = s_stack + threadIdx.x;
    st.sp = 0;
    if (n_dev) n = min(n, *n_dev);
    const uint32_t k = blockIdx.x * TRACE_BLOCK + threadIdx.x;
    uint32_t err = 0, nvis = 0, ntri = 0;
    if (k < n) {
        const uint32_t i = order ? __ldg(order + k) : k;
        const float4 r0 = __ldg(rays + 2ull * i), r1 = __ldg(rays + 2ull * i + 1);
        Best best;
        best.t = r0.w;
        best.u = best.v = 0.0f;
        best.prim = -1;
        best.obj = -1;
        trace_scene<COUNT, TLAS>(sv, r0, r1, best, st, err, nvis, ntri);
        hits[i] = make_float4(__int_as_float(best.prim), best.t, best.prim >= 0 ? best.u : 0.0f, best.prim >= 0 ? best.v : 0.0f);
        if (obj_out) obj_out[i] = best.obj;
    }
    flush_counters<COUNT>(err, nvis, ntri, err_out, counters);
}

// Persistent variant. Per lane: the ray it owns (index ri), the next instance
// to try (mi) and, while a mesh is being traversed (in_mesh), the traversal
// state. Each loop iteration of a warp: refill lanes without a ray when
// enough of them are idle, advance lanes to their next instance (or finish
// their ray), then one node step plus the triangles it hit.
// MULTI: rays of several scenes in one launch; ray i belongs to the scene
// whose SceneView is at views + ray_job[i] * view_stride.
// ANY: shadow rays -- a ray ends at its first accepted hit on a solid
// triangle (Traverse_MacroTree_WithStack_AnyHit, CoreRef.cpp:1224-1368).
// ONE: a lane tests one triangle per loop iteration and takes its next node
// only when the triangles of the last one are done, so each iteration is at
// most one node step and one triangle test per lane; otherwise a lane tests
// all the triangles of its node step in the same iteration, and the warp's
// triangle loop runs as long as its longest list.
template <bool COUNT, bool DEEP, bool MULTI, bool ANY, int BLOCK, int SDEPTH, bool TLAS, bool ONE>
__device__ __forceinline__ void trace_persistent(SceneView sv, const float4 *__restrict__ rays, uint32_t n, float4 *__restrict__ hits,
                                                 int32_t *__restrict__ obj_out, uint32_t *__restrict__ err_out,
                                                 unsigned long long *__restrict__ counters, uint32_t *__restrict__ next_ray, int refill_min,
                                                 const uint32_t *__restrict__ n_dev, const uint8_t *__restrict__ views, uint32_t view_stride,
                                                 const uint32_t *__restrict__ ray_job, const uint32_t *__restrict__ order, int stream_hint,
                                                 uint32_t coop_max) {
    if (n_dev) n = min(n, *n_dev);
    __shared__ uint2 s_stack[SDEPTH * BLOCK];
    Stack<DEEP, BLOCK, SDEPTH> st;
    st.smem = s_stack + threadIdx.x;
    st.sp = 0;
    uint32_t err = 0, nvis = 0, ntri = 0;
    uint32_t ri = NO_RAY, mi = 0, visits = 0;
    bool in_mesh = false; // traversing a mesh, or the instance tree (in_tree)
    bool in_tree = false;
    int sp0 = 0; // stack entries below the mesh's own (the tree's groups)
    constexpr bool BEST_SMEM = (SDEPTH * 8 + 12) * BLOCK <= 48 * 1024;
    __shared__ float s_best[BEST_SMEM ? 3 * BLOCK : 1];
    LaneBest<BLOCK, BEST_SMEM> best;
    best.t = 0.0f;
    best.prim = -1;
    if constexpr (BEST_SMEM) best.slot = s_best + threadIdx.x;
    // the ray in world space (origin, reciprocals) and the tree's visit count,
    // kept while the lane is inside an instance (without room in shared memory
    // the count in a register, the ray read again)
    constexpr bool WORLD_SMEM = TLAS && (SDEPTH * 8 + 12 + 28) * BLOCK <= 48 * 1024;
    __shared__ float s_world[WORLD_SMEM ? 7 * BLOCK : 1];
    float *world = s_world + (WORLD_SMEM ? threadIdx.x : 0);
    uint32_t tree_visits = 0;
    LocalRay r = make_local_ray(0.0f, 0.0f, 0.0f, 1.0f, 1.0f, 1.0f);
    MeshRef mr{};
    uint32_t ng_base = 0, ng_bits = 0, tg_base = 0, tg_bits = 0;
    bool pool_empty = false;
    auto scene_of = [&](uint32_t ray) -> const SceneView & {
        return *reinterpret_cast<const SceneView *>(views + (size_t)__ldg(ray_job + ray) * view_stride);
    };
    auto enter = [&](const SceneView &lsv, const InstanceRec *ir, int m, float4 r0, float4 r1) {
        mr = mesh_of(lsv, ir, m);
        r = transform_ray(ir, r0, r1);
        ng_base = 0;
        ng_bits = r.root_bits();
        visits = 0;
    };
    // The start of a lane's ray (its scene's instance tree, or the first
    // instance whose box it enters) or its next instance; false when the ray
    // is done (a ray whose scene has no instance left is done without reading
    // it again; a multi-scene ray reads its scene view first).
    auto next_mesh = [&]() -> bool {
        if (mi >= MI_DONE || !(MULTI || mi < sv.n_inst)) return false;
        // streaming hint: the ray is read once per instance pass and the
        // hit written once, so they may leave L1/L2 first (evict-first),
        // which keeps more of the BVH resident
        const float4 r0 = stream_hint ? __ldcs(rays + 2ull * ri) : __ldg(rays + 2ull * ri);
        const float4 r1 = stream_hint ? __ldcs(rays + 2ull * ri + 1) : __ldg(rays + 2ull * ri + 1);
        const float sx = safe_inv(r1.x), sy = safe_inv(r1.y), sz = safe_inv(r1.z);
        const SceneView &lsv = MULTI ? scene_of(ri) : sv;
        st.sp = 0;
        sp0 = 0;
        tg_bits = 0;
        if (TLAS && lsv.tlas) {
            mi = MI_DONE; // no instance after the tree's
            r = world_ray(r0.x, r0.y, r0.z, sx, sy, sz);
            if (WORLD_SMEM) { // (a group's eight lanes write the same values)
                world[0] = r.ox;
                world[BLOCK] = r.oy;
                world[2 * BLOCK] = r.oz;
                world[3 * BLOCK] = r.ix;
                world[4 * BLOCK] = r.iy;
                world[5 * BLOCK] = r.iz;
            }
            mr = tree_of(lsv);
            ng_base = 0;
            ng_bits = r.root_bits();
            visits = 0;
            in_tree = true;
            return true;
        }
        while (mi < lsv.n_inst) {
            const InstanceRec *ir = lsv.inst + mi;
            float bmin[3], bmax[3];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                bmin[k] = __ldg(&ir->bbox_min[k]);
                bmax[k] = __ldg(&ir->bbox_max[k]);
            }
            mi++;
            if (!ref_bbox_test(r0.x, r0.y, r0.z, sx, sy, sz, best.t, bmin, bmax)) continue;
            enter(lsv, ir, (int)mi - 1, r0, r1);
            if (TLAS) in_tree = false;
            return true;
        }
        return false;
    };
    auto write_hit = [&]() {
        const bool found = best.prim >= 0;
        const float4 h = make_float4(__int_as_float(best.prim), best.t, found ? best.u() : 0.0f, found ? best.v() : 0.0f);
        if (stream_hint) __stcs(hits + ri, h);
        else hits[ri] = h;
        if (obj_out) obj_out[ri] = found ? best.obj_of() : -1;
    };
    // A lane whose tree node has leaf entries left takes the next instance the
    // ray enters; the rest of the node waits on the stack. False: the stack is full.
    auto enter_instance = [&](bool writer) -> bool {
        const SceneView &lsv = MULTI ? scene_of(ri) : sv;
        const int m = next_instance(lsv, r, best.t, tg_base, tg_bits, err);
        if (m < 0) return true;
        bool ok = ng_bits <= 0x00FFFFFFu || st.push_group(make_uint2(ng_base, ng_bits), writer);
        if (tg_bits) ok = st.push_group(make_uint2(tg_base, tg_bits), writer) && ok;
        tg_bits = 0;
        if (!ok) {
            err |= TRACE_ERR_STACK;
            return false;
        }
        const float4 r0 = __ldg(rays + 2ull * ri), r1 = __ldg(rays + 2ull * ri + 1);
        if (WORLD_SMEM) world[6 * BLOCK] = __uint_as_float(visits);
        else tree_visits = visits;
        enter(lsv, lsv.inst + m, m, r0, r1);
        in_tree = false;
        sp0 = st.sp;
        return true;
    };
    // The end of a group: the next one from the stack, the tree when an
    // instance of it is done; false when the mesh (or the tree) is.
    auto next_group = [&]() -> bool {
        if (TLAS && !in_tree && mi == MI_DONE && st.sp == sp0) { // the instance is done: back to the tree
            if (WORLD_SMEM) {
                r = world_ray(world[0], world[BLOCK], world[2 * BLOCK], world[3 * BLOCK], world[4 * BLOCK], world[5 * BLOCK]);
                visits = __float_as_uint(world[6 * BLOCK]);
            } else {
                const float4 r0 = __ldg(rays + 2ull * ri), r1 = __ldg(rays + 2ull * ri + 1);
                r = world_ray(r0.x, r0.y, r0.z, safe_inv(r1.x), safe_inv(r1.y), safe_inv(r1.z));
                visits = tree_visits;
            }
            mr = tree_of(MULTI ? scene_of(ri) : sv);
            in_tree = true;
            sp0 = 0;
        }
        if (st.sp == sp0) return false;
        const uint2 e = st.pop();
        if (!TLAS || e.y > 0x00FFFFFFu) {
            ng_base = e.x;
            ng_bits = e.y;
        } else { // the rest of a tree node's leaf entries
            tg_base = e.x;
            tg_bits = e.y;
        }
        return true;
    };
    // few rays: eight lanes each from the start
    constexpr bool COOP = !COUNT;
    const bool few = COOP && n <= coop_max;
    while (!few) {
        // ---- refill lanes that have no ray
        const uint32_t need = __ballot_sync(0xffffffffu, ri == NO_RAY);
        if (!pool_empty && need != 0 && (__popc(need) >= refill_min || need == 0xffffffffu)) {
            const uint32_t leader = __ffs(need) - 1, lane = threadIdx.x & 31u;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(next_ray, (uint32_t)__popc(need));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (base + __popc(need) >= n) pool_empty = true;
            if (ri == NO_RAY) {
                const uint32_t idx = base + __popc(need & ((1u << lane) - 1u));
                if (idx < n) {
                    ri = order ? __ldg(order + idx) : idx;
                    mi = 0;
                    in_mesh = false;
                    best.t = __ldg(&rays[2ull * ri].w);
                    best.prim = -1;
                }
            }
        }
        if (pool_empty) {
            // the launch's last rays: once a warp has no more than four left, eight lanes each
            const uint32_t live = __ballot_sync(0xffffffffu, ri != NO_RAY);
            if (live == 0 || (COOP && !DEEP && __popc(live) <= 4)) break;
        }
        // A lane without work this iteration falls through to the next one, the
        // warp meeting again (__syncwarp) after each phase, which keeps lanes
        // that took different branches from drifting into different iterations
        // (one triangle per step, 4M-ray launch of the microbench on B200:
        // 4.28 ms without, 3.7 ms with)
        bool idle = ri == NO_RAY;
        // ---- the start of the ray, the next instance, or the end of the ray
        if (!idle && !in_mesh) {
            in_mesh = next_mesh();
            if (!in_mesh) {
                write_hit();
                ri = NO_RAY;
                idle = true;
            }
        }
        __syncwarp();
        // ---- a node visit (the node step bounds a mesh's visits by its node
        // count) for the lanes whose last node's triangles are done
        if (!idle && tg_bits == 0) {
            if (!node_step<COUNT>(mr, r, best.t, ng_base, ng_bits, tg_base, tg_bits, st, visits, err, nvis)) {
                in_mesh = false;
                mi = MI_DONE; // abandon the ray; the error flag reports it
                tg_bits = 0;
                idle = true;
            }
        }
        __syncwarp();
        // ---- instances
        if (TLAS) {
            if (!idle && in_tree && tg_bits && !enter_instance(true)) {
                in_mesh = false;
                mi = MI_DONE;
                idle = true;
            }
            __syncwarp();
        }
        // ---- triangles: one per lane, then (not with ONE) the others
        bool stop = false;
        while (true) {
            if (!idle && tg_bits && !(TLAS && in_tree)) {
                const uint32_t k = __ffs(tg_bits) - 1;
                tg_bits &= tg_bits - 1;
                if (ANY) {
                    if (tri_test<COUNT, true>(mr, r, tg_base + k, best, err, ntri)) {
                        stop = true;
                        tg_bits = 0;
                    }
                } else {
                    tri_test<COUNT>(mr, r, tg_base + k, best, err, ntri);
                }
            }
            if (ONE || !__any_sync(0xffffffffu, !idle && tg_bits && !(TLAS && in_tree))) break;
        }
        __syncwarp();
        if (idle) continue;
        if (ANY && stop) { // a solid triangle blocks the ray: no further instance
            in_mesh = false;
            mi = MI_DONE;
            continue;
        }
        if (tg_bits == 0 && ng_bits <= 0x00FFFFFFu) in_mesh = next_group();
    }
    if constexpr (COOP) {
        // ---- eight lanes per ray: the group's lanes hold the same state, the
        // ray's stack, best hit and world ray being its owner's (a lane of the
        // main loop whose ray it is, or the group's first lane)
        const uint32_t lane = threadIdx.x & 31u, grp = lane >> 3, c = lane & 7u;
        uint32_t live = few ? 0u : __ballot_sync(0xffffffffu, ri != NO_RAY);
        if (!few && live == 0) {
            flush_counters<COUNT>(err, nvis, ntri, err_out, counters);
            return;
        }
        for (uint32_t k = 0; k < grp; k++) live &= live - 1u;
        const bool has = live != 0;
        const uint32_t own = has ? __ffs(live) - 1u : grp * 8u;
        if (!few) { // hand over the ray's state
            auto take = [&](auto &x) { x = __shfl_sync(0xffffffffu, x, own); };
            auto take_flag = [&](bool &x) { x = __shfl_sync(0xffffffffu, (int)x, own) != 0; };
            auto take_ptr = [&](auto *&x) {
                x = reinterpret_cast<std::remove_reference_t<decltype(x)>>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(x), own));
            };
            take(ri);
            take(mi);
            take(visits);
            if constexpr (TLAS && !WORLD_SMEM) take(tree_visits);
            take(sp0);
            take(st.sp);
            take_flag(in_mesh);
            take_flag(in_tree);
            take(best.t);
            take(best.prim);
            if constexpr (!BEST_SMEM) {
                take(best.bu);
                take(best.bv);
                take(best.bobj);
            }
            take(r.ox);
            take(r.oy);
            take(r.oz);
            take(r.dx);
            take(r.dy);
            take(r.dz);
            take(r.ix);
            take(r.iy);
            take(r.iz);
            take(r.oct);
            take_ptr(mr.nodes);
            take_ptr(mr.tris);
            take(mr.prim_base);
            take(mr.node_count);
            take(mr.tri_count);
            take(mr.obj);
            take(ng_base);
            take(ng_bits);
            take(tg_base);
            take(tg_bits);
            if (!has) ri = NO_RAY;
        }
        const int off = (int)own - (int)lane;
        st.smem += off;
        if constexpr (BEST_SMEM) best.slot += off;
        if (WORLD_SMEM) world += off;
        __syncwarp();
        // the groups that take rays: with fewer rays than warps one a warp (its
        // steps then wait for no other ray's), else all four
        const uint32_t takers = n <= gridDim.x * (BLOCK / 32) ? 1u : 0x01010101u;
        while (true) {
            if (few && !pool_empty) {
                const uint32_t need = __ballot_sync(0xffffffffu, ri == NO_RAY) & takers; // the groups' first lanes
                if (need) {
                    uint32_t base = 0;
                    const uint32_t leader = __ffs(need) - 1;
                    if (lane == leader) base = atomicAdd(next_ray, (uint32_t)__popc(need));
                    base = __shfl_sync(0xffffffffu, base, leader);
                    if (base + __popc(need) >= n) pool_empty = true;
                    if ((need >> (grp * 8u)) & 1u) {
                        const uint32_t idx = base + __popc(need & ((1u << (grp * 8u)) - 1u));
                        if (idx < n) {
                            ri = order ? __ldg(order + idx) : idx;
                            mi = 0;
                            in_mesh = false;
                            best.t = __ldg(&rays[2ull * ri].w);
                            best.prim = -1;
                        }
                    }
                }
            }
            if ((!few || pool_empty) && __all_sync(0xffffffffu, ri == NO_RAY)) break;
            bool idle = ri == NO_RAY;
            if (!idle && !in_mesh) {
                in_mesh = next_mesh();
                if (!in_mesh) {
                    if (c == 0) write_hit();
                    ri = NO_RAY;
                    idle = true;
                }
            }
            __syncwarp();
            if (!node_step_coop(!idle && tg_bits == 0, mr, r, best.t, ng_base, ng_bits, tg_base, tg_bits, st, visits, err)) {
                in_mesh = false;
                mi = MI_DONE;
                tg_bits = 0;
                idle = true;
            }
            if (TLAS) {
                if (!idle && in_tree && tg_bits && !enter_instance(c == 0)) {
                    in_mesh = false;
                    mi = MI_DONE;
                    idle = true;
                }
            }
            // triangles: lane c the c-th of the group's list, eight at a time
            bool stop = false;
            const bool tri = !idle && !(TLAS && in_tree);
            while (__any_sync(0xffffffffu, tri && tg_bits)) {
                uint32_t m = tri ? tg_bits : 0u;
                for (uint32_t k = 0; k < c; k++) m &= m - 1u;
                float t = 0.0f, u = 0.0f, v = 0.0f;
                int gp = 0;
                bool solid = false;
                const bool cand = m != 0 && tri_candidate(mr, r, tg_base + __ffs(m) - 1u, best, err, t, u, v, gp, solid);
                if (tri) { // past the eight
                    for (int k = 0; k < 8; k++) tg_bits &= tg_bits - 1u;
                }
                if (__any_sync(0xffffffffu, cand)) {
                    // the group's winner: any hit prefers a solid triangle (it ends the ray); then the
                    // nearest, a tie to the lower triangle
                    uint32_t from = lane;
                    uint32_t rank = !cand ? 2u : (ANY && solid ? 0u : 1u);
                    float wt = t;
                    int wp = gp;
                    for (uint32_t o = 4; o; o >>= 1) {
                        const uint32_t orank = __shfl_xor_sync(0xffffffffu, rank, o), ofrom = __shfl_xor_sync(0xffffffffu, from, o);
                        const float ot = __shfl_xor_sync(0xffffffffu, wt, o);
                        const int op = __shfl_xor_sync(0xffffffffu, wp, o);
                        if (orank < rank || (orank == rank && (ot < wt || (ot == wt && op < wp)))) {
                            rank = orank;
                            from = ofrom;
                            wt = ot;
                            wp = op;
                        }
                    }
                    if (rank < 2u) {
                        best.t = wt;
                        best.prim = wp;
                        if (ANY && rank == 0u) {
                            stop = true;
                            tg_bits = 0;
                        }
                    }
                    if constexpr (BEST_SMEM) {
                        if (rank < 2u && from == lane) best.rest(u, v, mr.obj);
                    } else {
                        u = __shfl_sync(0xffffffffu, u, from);
                        v = __shfl_sync(0xffffffffu, v, from);
                        if (rank < 2u) best.rest(u, v, mr.obj);
                    }
                    __syncwarp();
                }
            }
            __syncwarp(); // the groups' pushes before their pops
            if (idle) continue;
            if (ANY && stop) {
                in_mesh = false;
                mi = MI_DONE;
                continue;
            }
            if (tg_bits == 0 && ng_bits <= 0x00FFFFFFu) in_mesh = next_group();
        }
    }
    flush_counters<COUNT>(err, nvis, ntri, err_out, counters);
}

template <bool COUNT, bool DEEP, bool MULTI = false, bool ANY = false, int BLOCK = TRACE_BLOCK, int SDEPTH = SMEM_STACK, bool TLAS = false,
          bool ONE = false>
__global__ void __launch_bounds__(BLOCK) k_trace_persistent(SceneView sv, const float4 *__restrict__ rays, uint32_t n,
                                                                  float4 *__restrict__ hits, int32_t *__restrict__ obj_out,
                                                                  uint32_t *__restrict__ err_out, unsigned long long *__restrict__ counters,
                                                                  uint32_t *__restrict__ next_ray, int refill_min,
                                                                  const uint32_t *__restrict__ n_dev, const uint8_t *__restrict__ views = nullptr,
                                                                  uint32_t view_stride = 0, const uint32_t *__restrict__ ray_job = nullptr,
                                                                  const uint32_t *__restrict__ order = nullptr, int stream_hint = 0,
                                                                  uint32_t coop_max = 0) {
    trace_persistent<COUNT, DEEP, MULTI, ANY, BLOCK, SDEPTH, TLAS, ONE>(sv, rays, n, hits, obj_out, err_out, counters, next_ray, refill_min,
                                                                        n_dev, views, view_stride, ray_job, order, stream_hint, coop_max);
}

// The closest-hit, one-triangle-per-step form for scenes without an
// instance tree whose BVHs fit the shared stack, with registers bounded so
// that 1024 threads per SM stay resident (64 registers; no spills, where the
// other instances of the kernel would spill at that bound): measured
// 3.23 ms per 4M-ray launch of the microbench on B200 against 3.33 ms at 72
// registers and 896 threads (64 threads per block, 16 stack entries).
template <int BLOCK, int SDEPTH>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK) k_trace_closest_one(SceneView sv, const float4 *__restrict__ rays, uint32_t n,
                                                                          float4 *__restrict__ hits, int32_t *__restrict__ obj_out,
                                                                          uint32_t *__restrict__ err_out,
                                                                          unsigned long long *__restrict__ counters,
                                                                          uint32_t *__restrict__ next_ray, int refill_min,
                                                                          const uint32_t *__restrict__ n_dev,
                                                                          const uint32_t *__restrict__ order, int stream_hint,
                                                                          uint32_t coop_max) {
    trace_persistent<false, false, false, false, BLOCK, SDEPTH, false, true>(sv, rays, n, hits, obj_out, err_out, counters, next_ray,
                                                                              refill_min, n_dev, nullptr, 0, nullptr, order, stream_hint, coop_max);
}

int g_persistent_blocks[2][2] = {{0, 0}, {0, 0}}; // [DEEP][TLAS]

// The closest-hit persistent kernel with a tuned block size and shared stack
// depth (one resident grid: the SM count times the blocks that fit per SM).
template <bool DEEP, bool TLAS, int BLOCK, int SDEPTH, bool ONE>
cudaError_t launch_tuned(const SceneView &sv, const float4 *rays, uint32_t n, float4 *hits, int32_t *obj, uint32_t *err,
                         unsigned long long *counters, cudaStream_t st, const TraceParams &tp) {
    static_assert(SDEPTH * BLOCK * 8 <= 48 * 1024, "static shared memory limit");
    // k_trace_closest_one: with 16 stack entries (at 24 per thread its 1024 threads
    // hold 192 KB of shared stack per SM, and it measured 4.12 ms against 3.38
    // for the unbounded kernel, which keeps more of the SM's L1)
    constexpr bool FAST = ONE && !DEEP && !TLAS && SDEPTH <= 16;
    static int blocks = 0;
    if (blocks == 0) {
        int dev = 0, sms = 0, per_sm = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) {
            if (FAST)
                e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_trace_closest_one<BLOCK, SDEPTH>, BLOCK, 0);
            else
                e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_trace_persistent<false, DEEP, false, false, BLOCK, SDEPTH, TLAS, ONE>,
                                                                  BLOCK, 0);
        }
        if (e != cudaSuccess) return e;
        blocks = sms * (per_sm > 0 ? per_sm : 1);
    }
    if (!tp.next_zeroed) {
        const cudaError_t e = cudaMemsetAsync(tp.next_ray, 0, sizeof(uint32_t), st);
        if (e != cudaSuccess) return e;
    }
    const uint32_t coop = coop_rays(blocks, BLOCK);
    // few rays, the count known here: no more blocks than give each a warp
    const uint32_t grid = n <= coop ? std::min<uint32_t>(blocks, (n + BLOCK / 32 - 1) / (BLOCK / 32)) : (uint32_t)blocks;
    if (FAST)
        k_trace_closest_one<BLOCK, SDEPTH><<<grid, BLOCK, 0, st>>>(sv, rays, n, hits, obj, err, counters, tp.next_ray, tp.refill_min, tp.count,
                                                                     tp.order, tp.stream_hint, coop);
    else
        k_trace_persistent<false, DEEP, false, false, BLOCK, SDEPTH, TLAS, ONE><<<grid, BLOCK, 0, st>>>(
            sv, rays, n, hits, obj, err, counters, tp.next_ray, tp.refill_min, tp.count, nullptr, 0, nullptr, tp.order, tp.stream_hint, coop);
    return cudaGetLastError();
}

template <bool DEEP, bool TLAS>
cudaError_t launch_tuned_dispatch(const SceneView &sv, const float4 *rays, uint32_t n, float4 *hits, int32_t *obj, uint32_t *err,
                                  unsigned long long *counters, cudaStream_t st, const TraceParams &tp) {
#define RG_TUNED(B, D)                                                                                                                  \
    if (tp.block == B && tp.smem_stack == D)                                                                                            \
        return tp.one_tri ? launch_tuned<DEEP, TLAS, B, D, true>(sv, rays, n, hits, obj, err, counters, st, tp)                          \
                          : launch_tuned<DEEP, TLAS, B, D, false>(sv, rays, n, hits, obj, err, counters, st, tp);
    RG_TUNED(64, 16) RG_TUNED(64, 24) RG_TUNED(64, 32)
    RG_TUNED(128, 16) RG_TUNED(128, 24) RG_TUNED(128, 32)
    RG_TUNED(256, 16) RG_TUNED(256, 24)
#undef RG_TUNED
    return cudaErrorInvalidValue;
}

template <bool DEEP, bool TLAS>
cudaError_t launch_impl(const SceneView &sv, const float4 *rays, uint32_t n, float4 *hits, int32_t *obj, uint32_t *err,
                        unsigned long long *counters, bool count, cudaStream_t st, const TraceParams &tp) {
    constexpr int B = TRACE_BLOCK, D = LOOP_STACK;
    if (!tp.persistent && !tp.views && !tp.any) {
        const uint32_t grid = (n + TRACE_BLOCK - 1) / TRACE_BLOCK;
        if (count)
            k_trace_closest<true, DEEP, TLAS><<<grid, TRACE_BLOCK, 0, st>>>(sv, rays, n, hits, obj, err, counters, tp.count, tp.order);
        else
            k_trace_closest<false, DEEP, TLAS><<<grid, TRACE_BLOCK, 0, st>>>(sv, rays, n, hits, obj, err, counters, tp.count, tp.order);
        return cudaGetLastError();
    }
    if (!tp.next_ray) return cudaErrorInvalidValue;
    if (!count && !tp.views && !tp.any)
        return launch_tuned_dispatch<DEEP, TLAS>(sv, rays, n, hits, obj, err, counters, st, tp);
    int &blocks = g_persistent_blocks[DEEP ? 1 : 0][TLAS ? 1 : 0];
    if (blocks == 0) {
        int dev = 0, sms = 0, per_sm = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_trace_persistent<false, DEEP, false, false, B, D, TLAS>, TRACE_BLOCK, 0);
        if (e != cudaSuccess) return e;
        blocks = sms * (per_sm > 0 ? per_sm : 1);
    }
    if (!tp.next_zeroed) {
        const cudaError_t e = cudaMemsetAsync(tp.next_ray, 0, sizeof(uint32_t), st);
        if (e != cudaSuccess) return e;
    }
    const uint32_t coop = coop_rays(blocks, TRACE_BLOCK);
    // shadow rays and rays of several scenes (no counting variants), with one
    // triangle test per step or a node's triangles at once
#define RG_LAUNCH_P(MULTI_, ANY_, ONE_)                                                                                                 \
    k_trace_persistent<false, DEEP, MULTI_, ANY_, B, D, TLAS, ONE_><<<blocks, TRACE_BLOCK, 0, st>>>(                                    \
        sv, rays, n, hits, obj, err, counters, tp.next_ray, tp.refill_min, tp.count, tp.views, tp.view_stride, tp.ray_job, nullptr, 0, coop)
    if (tp.any) {
        if (tp.views) {
            if (tp.one_tri) RG_LAUNCH_P(true, true, true);
            else RG_LAUNCH_P(true, true, false);
        } else {
            if (tp.one_tri) RG_LAUNCH_P(false, true, true);
            else RG_LAUNCH_P(false, true, false);
        }
        return cudaGetLastError();
    }
    if (tp.views) {
        if (tp.one_tri) RG_LAUNCH_P(true, false, true);
        else RG_LAUNCH_P(true, false, false);
        return cudaGetLastError();
    }
#undef RG_LAUNCH_P
    k_trace_persistent<true, DEEP, false, false, B, D, TLAS><<<blocks, TRACE_BLOCK, 0, st>>>(
        sv, rays, n, hits, obj, err, counters, tp.next_ray, tp.refill_min, tp.count, nullptr, 0, nullptr, tp.order);
    return cudaGetLastError();
}

} // namespace

cudaError_t launch_trace_closest(const SceneView &sv, const float4 *rays, uint32_t n, float4 *hits, int32_t *obj, uint32_t *err,
                                 unsigned long long *counters, bool count, cudaStream_t st, const TraceParams &tp) {
    if (n == 0) return cudaSuccess;
    // one group per level at most: the shared-memory stack suffices up to its
    // depth in levels
    const bool special = count || tp.views || tp.any;
    const uint32_t sdepth = tp.persistent || tp.views || tp.any ? (special ? (uint32_t)LOOP_STACK : (uint32_t)tp.smem_stack) : (uint32_t)SMEM_STACK;
    if (tp.tlas) {
        if (tp.max_depth < sdepth) return launch_impl<false, true>(sv, rays, n, hits, obj, err, counters, count, st, tp);
        return launch_impl<true, true>(sv, rays, n, hits, obj, err, counters, count, st, tp);
    }
    if (tp.max_depth < sdepth) return launch_impl<false, false>(sv, rays, n, hits, obj, err, counters, count, st, tp);
    return launch_impl<true, false>(sv, rays, n, hits, obj, err, counters, count, st, tp);
}

} // namespace rg
