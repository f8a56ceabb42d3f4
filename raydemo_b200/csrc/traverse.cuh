// Device-side traversal shared by the trace kernels and the shading kernels:
// the instance-level test and transform, the compressed wide-BVH node step,
// the triangle test and whole-mesh traversal. See trace.cu for the design.
#pragma once

#include "trace.cuh"

namespace rg {
namespace trav {

constexpr int TRACE_BLOCK = 128;
constexpr int SMEM_STACK = 24; // entries per thread in shared memory
constexpr int LMEM_STACK = 40; // further entries in a local array (DEEP instances only)
constexpr uint32_t NO_RAY = 0xffffffffu;
constexpr float SLAB_SLACK = 9.5367431640625e-07f; // 2^-20, see node_step

// Three-input max / min (sm_100). NaN inputs are dropped, as fmaxf/fminf drop them.
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Byte k of word as the float 2^15 + byte (0x4700bb00): exact, one permute.
__device__ __forceinline__ float byte_to_float(uint32_t word, uint32_t k) {
    return __uint_as_float(__byte_perm(word, 0x47000000u, 0x7604u | (k << 4)));
}

// Pairs of floats in one 64-bit register and their packed arithmetic
// (sm_100): each half is rounded as the scalar operation rounds it.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// The reference's slab test, exactly (bbox_test, CoreRef.cpp:64-86).
__device__ __forceinline__ bool ref_bbox_test(float ox, float oy, float oz, float ix, float iy, float iz, float t, const float *bmin,
                                              const float *bmax) {
    float lo_x = __fmul_rn(ix, __fsub_rn(bmin[0], ox)), hi_x = __fmul_rn(ix, __fsub_rn(bmax[0], ox));
    if (lo_x > hi_x) { const float tmp = lo_x; lo_x = hi_x; hi_x = tmp; }
    float lo_y = __fmul_rn(iy, __fsub_rn(bmin[1], oy)), hi_y = __fmul_rn(iy, __fsub_rn(bmax[1], oy));
    if (lo_y > hi_y) { const float tmp = lo_y; lo_y = hi_y; hi_y = tmp; }
    float lo_z = __fmul_rn(iz, __fsub_rn(bmin[2], oz)), hi_z = __fmul_rn(iz, __fsub_rn(bmax[2], oz));
    if (lo_z > hi_z) { const float tmp = lo_z; lo_z = hi_z; hi_z = tmp; }
    float tmin = lo_x > lo_y ? lo_x : lo_y;
    if (lo_z > tmin) tmin = lo_z;
    float tmax = hi_x < hi_y ? hi_x : hi_y;
    if (hi_z < tmax) tmax = hi_z;
    tmax = __fmul_rn(tmax, 1.00000024f);
    return tmin <= tmax && tmin <= t && tmax > 0;
}

// safe_invert, CoreRef.cpp:272-294
__device__ __forceinline__ float safe_inv(float v) {
    float r = __frcp_rn(v);
    if (v <= FLT_EPS_ && v >= 0) r = 3.402823466e+38F;
    else if (v >= -FLT_EPS_ && v < 0) r = -3.402823466e+38F;
    return r;
}

struct Best {
    float t, u, v;
    int prim, obj;
    __device__ __forceinline__ void rest(float u_, float v_, int obj_) {
        u = u_;
        v = v_;
        obj = obj_;
    }
    __device__ __forceinline__ int obj_of() const { return obj; }
};

// The best hit of a lane of the persistent kernel: what the tests compare
// stays in registers; u, v and the instance, written on an accepted hit and
// read when the ray ends, are in shared memory (word k of this thread at
// slot[k * STRIDE]). Three registers less keep the 64-register instance
// of the kernel from spilling.
// IN_SMEM false (block shapes whose stack fills the static shared memory):
// everything in registers.
template <int STRIDE, bool IN_SMEM>
struct LaneBest;

template <int STRIDE>
struct LaneBest<STRIDE, false> {
    float t;
    int prim;
    float bu, bv;
    int bobj;
    __device__ __forceinline__ void rest(float u, float v, int obj) {
        bu = u;
        bv = v;
        bobj = obj;
    }
    __device__ __forceinline__ float u() const { return bu; }
    __device__ __forceinline__ float v() const { return bv; }
    __device__ __forceinline__ int obj_of() const { return bobj; }
};

template <int STRIDE>
struct LaneBest<STRIDE, true> {
    float t;
    int prim;
    float *slot;
    __device__ __forceinline__ void rest(float u, float v, int obj) {
        slot[0] = u;
        slot[STRIDE] = v;
        slot[2 * STRIDE] = __int_as_float(obj);
    }
    __device__ __forceinline__ float u() const { return slot[0]; }
    __device__ __forceinline__ float v() const { return slot[STRIDE]; }
    __device__ __forceinline__ int obj_of() const { return __float_as_int(slot[2 * STRIDE]); }
};

// Ray in the space of the instance being traversed.
struct LocalRay {
    float ox, oy, oz, dx, dy, dz, ix, iy, iz;
    // bit a (0..2) set: the direction is negative on axis a; bit 3 + a set: it
    // is zero there (the node step tests that axis by containment)
    uint32_t oct;
    __device__ __forceinline__ uint32_t root_bits() const { return (1u << (24 + (oct & 7u))) | 1u; } // the root as slot 0 of a virtual parent
};

struct MeshRef {
    const WideNode *nodes;
    const TriRec *tris;
    uint32_t prim_base, node_count, tri_count;
    int obj;
};

// Per-thread stack of node groups: entry k of this thread at
// smem[k * STRIDE] (STRIDE = the block's thread count), DEPTH entries in
// shared memory; the DEEP variant continues it in a local array, to
// SMEM_STACK + LMEM_STACK entries in all.
template <bool DEEP, int STRIDE = TRACE_BLOCK, int DEPTH = SMEM_STACK>
struct Stack;

template <int STRIDE, int DEPTH>
struct Stack<false, STRIDE, DEPTH> {
    uint2 *smem;
    int sp;
    __device__ __forceinline__ bool push(uint2 e) {
        if (sp >= DEPTH) return false;
        smem[sp * STRIDE] = e;
        sp++;
        return true;
    }
    __device__ __forceinline__ uint2 pop() {
        sp--;
        return smem[sp * STRIDE];
    }
    // eight lanes with one stack (the same smem): one of them writes
    __device__ __forceinline__ bool push_group(uint2 e, bool writer) {
        if (sp >= DEPTH) return false;
        if (writer) smem[sp * STRIDE] = e;
        sp++;
        return true;
    }
};

template <int STRIDE, int DEPTH>
struct Stack<true, STRIDE, DEPTH> {
    static constexpr int LOCAL = SMEM_STACK + LMEM_STACK - DEPTH;
    uint2 *smem;
    uint2 lmem[LOCAL];
    int sp;
    __device__ __forceinline__ bool push(uint2 e) {
        if (sp >= DEPTH + LOCAL) return false;
        if (sp < DEPTH) smem[sp * STRIDE] = e;
        else lmem[sp - DEPTH] = e;
        sp++;
        return true;
    }
    __device__ __forceinline__ uint2 pop() {
        sp--;
        return sp < DEPTH ? smem[sp * STRIDE] : lmem[sp - DEPTH];
    }
    // eight lanes with one stack: one writes the shared part, each its own copy of the rest
    __device__ __forceinline__ bool push_group(uint2 e, bool writer) {
        if (sp >= DEPTH + LOCAL) return false;
        if (sp >= DEPTH) lmem[sp - DEPTH] = e;
        else if (writer) smem[sp * STRIDE] = e;
        sp++;
        return true;
    }
};

__device__ __forceinline__ LocalRay make_local_ray(float ox, float oy, float oz, float dx, float dy, float dz) {
    LocalRay r;
    r.ox = ox; r.oy = oy; r.oz = oz;
    r.dx = dx; r.dy = dy; r.dz = dz;
    r.ix = __frcp_rn(dx); // 1.0f / d, CoreRef.cpp:1215
    r.iy = __frcp_rn(dy);
    r.iz = __frcp_rn(dz);
    r.oct = (r.ix < 0.0f ? 1u : 0u) | (r.iy < 0.0f ? 2u : 0u) | (r.iz < 0.0f ? 4u : 0u);
    if (dx == 0.0f || dy == 0.0f || dz == 0.0f) r.oct |= (dx == 0.0f ? 8u : 0u) | (dy == 0.0f ? 16u : 0u) | (dz == 0.0f ? 32u : 0u);
    return r;
}

// TransformRay, CoreRef.cpp:1605-1617, with the instance's inverse transform.
__device__ __forceinline__ LocalRay transform_ray(const InstanceRec *ir, float4 r0, float4 r1) {
    float x[12];
#pragma unroll
    for (int k = 0; k < 12; k++) x[k] = __ldg(&ir->inv_xform[k]);
    const float tox = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(x[0], r0.x), __fmul_rn(x[3], r0.y)), __fmul_rn(x[6], r0.z)), x[9]);
    const float toy = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(x[1], r0.x), __fmul_rn(x[4], r0.y)), __fmul_rn(x[7], r0.z)), x[10]);
    const float toz = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(x[2], r0.x), __fmul_rn(x[5], r0.y)), __fmul_rn(x[8], r0.z)), x[11]);
    const float tdx = __fadd_rn(__fadd_rn(__fmul_rn(x[0], r1.x), __fmul_rn(x[3], r1.y)), __fmul_rn(x[6], r1.z));
    const float tdy = __fadd_rn(__fadd_rn(__fmul_rn(x[1], r1.x), __fmul_rn(x[4], r1.y)), __fmul_rn(x[7], r1.z));
    const float tdz = __fadd_rn(__fadd_rn(__fmul_rn(x[2], r1.x), __fmul_rn(x[5], r1.y)), __fmul_rn(x[8], r1.z));
    return make_local_ray(tox, toy, toz, tdx, tdy, tdz);
}

__device__ __forceinline__ MeshRef mesh_of(const SceneView &sv, const InstanceRec *ir, int m) {
    MeshRef mr;
    mr.nodes = sv.nodes + __ldg(&ir->node_base);
    mr.tris = sv.leaf_tris + __ldg(&ir->tri_base);
    mr.prim_base = __ldg(&ir->prim_base);
    mr.node_count = __ldg(&ir->node_count);
    mr.tri_count = __ldg(&ir->tri_count);
    mr.obj = m;
    return mr;
}

// The ray in world space, as the instance tree is traversed: the reciprocals
// are the instance test's own (safe_invert), so a component of 1e-7 or less
// counts as zero there and here. With all three that small nothing is left to
// order the axes by: the planes alone decide (they come out unbounded where
// they overflow).
__device__ __forceinline__ LocalRay world_ray(float ox, float oy, float oz, float ix, float iy, float iz) {
    LocalRay r;
    r.ox = ox; r.oy = oy; r.oz = oz;
    r.dx = r.dy = r.dz = 0.0f;
    r.ix = ix; r.iy = iy; r.iz = iz;
    r.oct = (ix < 0.0f ? 1u : 0u) | (iy < 0.0f ? 2u : 0u) | (iz < 0.0f ? 4u : 0u);
    const float big = 3.402823466e+38F;
    const uint32_t zero = (fabsf(ix) == big ? 8u : 0u) | (fabsf(iy) == big ? 16u : 0u) | (fabsf(iz) == big ? 32u : 0u);
    if (zero != 56u) r.oct |= zero;
    return r;
}

// The instance tree as the node step takes it. A leaf entry's test is the
// reference's own instance test (bbox_test with safe_invert), so no instance
// is entered that the reference culls; the nodes above accept whatever that
// test accepts. With the test's reciprocals, its near plane errs by 2u of its
// t and its far plane, widened by 1 + 4u, by 7u; the node step's slack of 16u
// (|B| + 33024|A|), 3u of which its own rounding takes, covers both, and the
// node's planes lie a quantum outside the instance's box besides.
__device__ __forceinline__ MeshRef tree_of(const SceneView &sv) {
    MeshRef mr;
    mr.nodes = sv.tlas;
    mr.tris = nullptr;
    mr.prim_base = 0;
    mr.node_count = sv.tlas_count;
    mr.tri_count = sv.n_inst;
    mr.obj = -1;
    return mr;
}

// The next instance of a leaf group of the tree (tg_base, tg_bits) that the
// ray enters with the current best t, taken out of the group; -1 for none.
__device__ __forceinline__ int next_instance(const SceneView &sv, const LocalRay &w, float best_t, uint32_t tg_base, uint32_t &tg_bits,
                                             uint32_t &err) {
    while (tg_bits) {
        const uint32_t e = tg_base + __ffs(tg_bits) - 1u;
        tg_bits &= tg_bits - 1u;
        const uint32_t m = e < sv.n_inst ? __ldg(sv.tlas_inst + e) : 0xffffffffu;
        if (m >= sv.n_inst) {
            err |= TRACE_ERR_TLAS;
            continue;
        }
        const InstanceRec *ir = sv.inst + m;
        const float4 lo = __ldg(reinterpret_cast<const float4 *>(ir->bbox_min)), hi = __ldg(reinterpret_cast<const float4 *>(ir->bbox_max));
        const float bmin[3] = {lo.x, lo.y, lo.z}, bmax[3] = {hi.x, hi.y, hi.z};
        if (ref_bbox_test(w.ox, w.oy, w.oz, w.ix, w.iy, w.iz, best_t, bmin, bmax)) return (int)m;
    }
    return -1;
}

// Children of a node whose slab on every zero axis of the ray (oct bits 3..5)
// holds the ray's origin: on such an axis the ray never leaves its origin's
// coordinate, so a box that does not span it is missed at every t. The decoded
// planes p + q 2^e are exact floats (the product and sum below round nothing)
// and lie a quantum outside the child's triangles, so no triangle whose box
// spans the origin is dropped. Bytes are read again from the node: this runs
// for rays that are parallel to an axis plane only.
__device__ __forceinline__ uint32_t zero_axis_children(const WideNode *nd, uint32_t oct, float ox, float oy, float oz) {
    uint32_t keep = 0xFFu;
#pragma unroll 1
    for (int a = 0; a < 3; a++) {
        if (!((oct >> (3 + a)) & 1u)) continue;
        const float o = a == 0 ? ox : (a == 1 ? oy : oz);
        const float p = __ldg(&nd->p[a]), sc = __uint_as_float((uint32_t)__ldg(&nd->e[a]) << 23);
#pragma unroll 1
        for (int c = 0; c < 8; c++) {
            const float lo = __fmaf_rn((float)__ldg(&nd->qlo[a][c]), sc, p), hi = __fmaf_rn((float)__ldg(&nd->qhi[a][c]), sc, p);
            if (o < lo || o > hi) keep &= ~(1u << c); // (a NaN origin keeps every child)
        }
    }
    return keep;
}

// Node step: takes the next child of node group (ng_base, ng_bits), tests
// its 8 children and returns their hits as a node group (internal children,
// bits 24..31, with the node's imask in bits 0..7) and a triangle group
// (bits 0..23). Returns false (and sets err) on a corrupt index.
template <bool COUNT, typename ST>
__device__ __forceinline__ bool node_step(const MeshRef &mr, const LocalRay &r, float best_t, uint32_t &ng_base, uint32_t &ng_bits,
                                          uint32_t &tg_base, uint32_t &tg_bits, ST &st, uint32_t &visits, uint32_t &err,
                                          uint32_t &nvis) {
    const uint32_t j = __ffs(ng_bits >> 24) - 1;
    ng_bits &= ~(1u << (24 + j));
    const uint32_t s = (j ^ r.oct) & 7u;
    const uint32_t ni = ng_base + __popc((ng_bits & 0xFFu) & ((1u << s) - 1u));
    if (ng_bits > 0x00FFFFFFu && !st.push(make_uint2(ng_base, ng_bits))) {
        err |= TRACE_ERR_STACK;
        return false;
    }
    // A tree visits each node at most once; a bad index or a longer walk
    // means a corrupt structure: flag it and stop this ray.
    if (ni >= mr.node_count || ++visits > mr.node_count) {
        err |= (ni >= mr.node_count) ? TRACE_ERR_BOUNDS : TRACE_ERR_LIMIT;
        return false;
    }
    // a zero direction component leaves its axis' planes NaN, that is unbounded:
    // without this a ray parallel to an axis plane entered every node its
    // other two axes allow, thousands of them, and one such ray among the 4M of
    // a launch decided the launch's time (5.4 ms with one seed's rays and 14 with
    // another's, against 3.2 without such a ray, on B200)
    const uint32_t keep = r.oct > 7u ? zero_axis_children(mr.nodes + ni, r.oct, r.ox, r.oy, r.oz) : 0xFFu;
    const uint4 *np = reinterpret_cast<const uint4 *>(mr.nodes + ni);
    const uint4 w0 = __ldg(np), w1 = __ldg(np + 1), w2 = __ldg(np + 2), w3 = __ldg(np + 3), w4 = __ldg(np + 4);
    if (COUNT) nvis++;
    const uint32_t imask = w0.w >> 24;
    // Slab parameter of plane q on one axis: t(q) = q * A + B with
    // A = 2^e * inv_d (exact: a power-of-two scaling) and B = (p - o) * inv_d.
    // It is evaluated as one FMA on the byte read as the float v = 2^15 + q:
    // t = v * A + (B - 2^15 A), v * A exact inside the FMA. Rounding
    // B - 2^15 A, then -/+ slack, then the FMA's result errs by less than
    // 3u(|B| + 33024|A|) (u = 2^-24); the slack 2^-20 (|B| + 33024|A|)
    // moves the near planes down and the far planes up by more than that,
    // so the test accepts every box that the exact slab test on the decoded
    // box accepts, and with the instance tree what the instance test accepts
    // (tree_of). (An overflowing 2^15 A gives NaN planes: that axis is left
    // unbounded, still conservative.)
    // The step is bound by instruction issue. The set-up of the x and y axes
    // goes through packed arithmetic; the children's FMAs stay scalar, packed
    // ones measured slower (the pairs' registers spill at 64 a thread: 3.41
    // against 3.18 ms per 4M-ray launch; at 72 a thread 3.26).
    const float scx = __uint_as_float((w0.w & 0xFFu) << 23), scy = __uint_as_float(((w0.w >> 8) & 0xFFu) << 23),
                scz = __uint_as_float(((w0.w >> 16) & 0xFFu) << 23);
    const unsigned long long ixy = pack2(r.ix, r.iy);
    const unsigned long long Axy = mul2(pack2(scx, scy), ixy);
    const unsigned long long Bxy = mul2(add2(pack2(__uint_as_float(w0.x), __uint_as_float(w0.y)), pack2(-r.ox, -r.oy)), ixy);
    float Ax, Ay, Bx, By;
    unpack2(Axy, Ax, Ay);
    unpack2(Bxy, Bx, By);
    const float Az = __fmul_rn(scz, r.iz), Bz = __fmul_rn(__fsub_rn(__uint_as_float(w0.z), r.oz), r.iz);
    const unsigned long long Sxy = pack2(__fmaf_rn(fabsf(Ax), 33024.0f, fabsf(Bx)), __fmaf_rn(fabsf(Ay), 33024.0f, fabsf(By)));
    const float Sz = __fmaf_rn(fabsf(Az), 33024.0f, fabsf(Bz));
    const unsigned long long B0xy = fma2(Axy, pack2(-32768.0f, -32768.0f), Bxy);
    const float B0z = __fmaf_rn(-32768.0f, Az, Bz);
    constexpr float SLACK = SLAB_SLACK;
    const unsigned long long Bnxy = fma2(Sxy, pack2(-SLACK, -SLACK), B0xy), Bfxy = fma2(Sxy, pack2(SLACK, SLACK), B0xy);
    const float Bnz = __fmaf_rn(Sz, -SLACK, B0z), Bfz = __fmaf_rn(Sz, SLACK, B0z);
    float Bnx, Bny, Bfx, Bfy;
    unpack2(Bnxy, Bnx, Bny);
    unpack2(Bfxy, Bfx, Bfy);
    // Near/far plane words by direction sign, so that a NaN slab value
    // (origin on a plane of a box the ray runs parallel to) leaves that axis
    // unbounded, which keeps the test conservative. Planes: lo x = w2.xy,
    // lo y = w2.zw, lo z = w3.xy, hi x = w3.zw, hi y = w4.xy, hi z = w4.zw.
    const bool nx = r.oct & 1u, ny = r.oct & 2u, nz = r.oct & 4u;
    const uint32_t nxa = nx ? w3.z : w2.x, nxb = nx ? w3.w : w2.y, fxa = nx ? w2.x : w3.z, fxb = nx ? w2.y : w3.w;
    const uint32_t nya = ny ? w4.x : w2.z, nyb = ny ? w4.y : w2.w, fya = ny ? w2.z : w4.x, fyb = ny ? w2.w : w4.y;
    const uint32_t nza = nz ? w4.z : w3.x, nzb = nz ? w4.w : w3.y, fza = nz ? w3.x : w4.z, fzb = nz ? w3.y : w4.w;
    uint32_t miss = 0; // sign bits of (far - near) shifted in, the last slot first: slots whose box the ray misses
#pragma unroll
    for (int c = 7; c >= 0; c--) {
        const uint32_t k = (uint32_t)(c & 3);
        const float tnx = __fmaf_rn(byte_to_float(c < 4 ? nxa : nxb, k), Ax, Bnx), tfx = __fmaf_rn(byte_to_float(c < 4 ? fxa : fxb, k), Ax, Bfx);
        const float tny = __fmaf_rn(byte_to_float(c < 4 ? nya : nyb, k), Ay, Bny), tfy = __fmaf_rn(byte_to_float(c < 4 ? fya : fyb, k), Ay, Bfy);
        const float tnz = __fmaf_rn(byte_to_float(c < 4 ? nza : nzb, k), Az, Bnz), tfz = __fmaf_rn(byte_to_float(c < 4 ? fza : fzb, k), Az, Bfz);
        // [max(near planes, 0), min(far planes, best_t)] non-empty: the slab
        // test with the ray's interval folded in (best_t >= 0); the difference
        // is never negative when it is (inf - inf gives NaN, sign clear)
        const float tmin = max3f(tnx, tny, fmaxf(tnz, 0.0f));
        const float tmax = min3f(tfx, tfy, fminf(tfz, best_t));
        miss = __funnelshift_l(__float_as_uint(__fsub_rn(tmax, tmin)), miss, 1);
    }
    uint32_t hit8 = ~miss & keep;
    // internal children: bit 24 + (slot ^ octant), so that the node group
    // is taken in the ray's octant order
    uint32_t inner = hit8 & imask;
    if (r.oct & 1u) inner = ((inner & 0x55u) << 1) | ((inner >> 1) & 0x55u);
    if (r.oct & 2u) inner = ((inner & 0x33u) << 2) | ((inner >> 2) & 0x33u);
    if (r.oct & 4u) inner = ((inner & 0x0Fu) << 4) | ((inner >> 4) & 0x0Fu);
    uint32_t hitmask = inner << 24;
    // leaf children: their triangle bits (an empty slot has meta 0 and adds nothing)
    for (uint32_t lv = hit8 & ~imask; lv; lv &= lv - 1u) {
        const uint32_t sl = __ffs(lv) - 1u;
        const uint32_t meta = ((sl < 4u ? w1.z : w1.w) >> (8u * (sl & 3u))) & 0xFFu;
        hitmask |= (meta >> 5) << (meta & 31u);
    }
    ng_base = w1.x;
    ng_bits = (hitmask & 0xFF000000u) | imask;
    tg_base = w1.y;
    tg_bits = hitmask & 0x00FFFFFFu;
    return true;
}

// Node step of a ray that eight lanes trace together (lane c of the group
// tests child c; the ray's state is the same in all eight). The steps of one
// ray follow one another, so their latency, not their throughput, decides the
// time of a launch with few rays and of every launch's last rays: testing the
// children side by side takes a step's dependent instructions from about 200
// to 60. Called by whole warps; `go`: this group's ray takes a step.
// Arithmetic and results as node_step; false on a corrupt index.
template <typename ST>
__device__ __forceinline__ bool node_step_coop(bool go, const MeshRef &mr, const LocalRay &r, float best_t, uint32_t &ng_base,
                                               uint32_t &ng_bits, uint32_t &tg_base, uint32_t &tg_bits, ST &st, uint32_t &visits,
                                               uint32_t &err) {
    const uint32_t lane = threadIdx.x & 31u, c = lane & 7u;
    bool ok = true, hit = false;
    uint32_t imask = 0, child_base = 0, tri_base = 0, meta_lo = 0, meta_hi = 0;
    if (go) {
        const uint32_t j = __ffs(ng_bits >> 24) - 1;
        ng_bits &= ~(1u << (24 + j));
        const uint32_t s = (j ^ r.oct) & 7u;
        const uint32_t ni = ng_base + __popc((ng_bits & 0xFFu) & ((1u << s) - 1u));
        if (ng_bits > 0x00FFFFFFu && !st.push_group(make_uint2(ng_base, ng_bits), c == 0)) {
            err |= TRACE_ERR_STACK;
            ok = false;
        } else if (ni >= mr.node_count || ++visits > mr.node_count) {
            err |= (ni >= mr.node_count) ? TRACE_ERR_BOUNDS : TRACE_ERR_LIMIT;
            ok = false;
        } else {
            const WideNode *nd = mr.nodes + ni;
            const uint4 w0 = __ldg(reinterpret_cast<const uint4 *>(nd)), w1 = __ldg(reinterpret_cast<const uint4 *>(nd) + 1);
            const uint8_t *q = reinterpret_cast<const uint8_t *>(nd) + 32 + c; // qlo[axis][c] at 8 axis, qhi 24 further
            const uint32_t lx = __ldg(q), ly = __ldg(q + 8), lz = __ldg(q + 16), hx = __ldg(q + 24), hy = __ldg(q + 32), hz = __ldg(q + 40);
            imask = w0.w >> 24;
            child_base = w1.x;
            tri_base = w1.y;
            meta_lo = w1.z;
            meta_hi = w1.w;
            float tn[3], tf[3];
#pragma unroll
            for (int a = 0; a < 3; a++) { // as node_step
                const float p = __uint_as_float(a == 0 ? w0.x : (a == 1 ? w0.y : w0.z));
                const float sc = __uint_as_float(((w0.w >> (8 * a)) & 0xFFu) << 23);
                const float inv = a == 0 ? r.ix : (a == 1 ? r.iy : r.iz), o = a == 0 ? r.ox : (a == 1 ? r.oy : r.oz);
                const uint32_t lo = a == 0 ? lx : (a == 1 ? ly : lz), hi = a == 0 ? hx : (a == 1 ? hy : hz);
                const bool neg = (r.oct >> a) & 1u;
                const float A = __fmul_rn(sc, inv), B = __fmul_rn(__fsub_rn(p, o), inv);
                const float S = __fmaf_rn(fabsf(A), 33024.0f, fabsf(B)), B0 = __fmaf_rn(-32768.0f, A, B);
                tn[a] = __fmaf_rn(__uint_as_float(0x47000000u | ((neg ? hi : lo) << 8)), A, __fmaf_rn(S, -SLAB_SLACK, B0));
                tf[a] = __fmaf_rn(__uint_as_float(0x47000000u | ((neg ? lo : hi) << 8)), A, __fmaf_rn(S, SLAB_SLACK, B0));
                if ((r.oct >> (3 + a)) & 1u) { // zero_axis_children
                    const float pl = __fmaf_rn((float)lo, sc, p), ph = __fmaf_rn((float)hi, sc, p);
                    if (o < pl || o > ph) ok = false;
                }
            }
            const float tmin = max3f(tn[0], tn[1], fmaxf(tn[2], 0.0f)), tmax = min3f(tf[0], tf[1], fminf(tf[2], best_t));
            hit = ok && !(__float_as_int(__fsub_rn(tmax, tmin)) < 0);
            ok = true;
        }
    }
    const uint32_t hit8 = (__ballot_sync(0xffffffffu, hit) >> (lane & 24u)) & 0xFFu;
    if (go && ok) {
        uint32_t inner = hit8 & imask;
        if (r.oct & 1u) inner = ((inner & 0x55u) << 1) | ((inner >> 1) & 0x55u);
        if (r.oct & 2u) inner = ((inner & 0x33u) << 2) | ((inner >> 2) & 0x33u);
        if (r.oct & 4u) inner = ((inner & 0x0Fu) << 4) | ((inner >> 4) & 0x0Fu);
        uint32_t leaf = 0;
        for (uint32_t lv = hit8 & ~imask; lv; lv &= lv - 1u) {
            const uint32_t sl = __ffs(lv) - 1u;
            const uint32_t meta = ((sl < 4u ? meta_lo : meta_hi) >> (8u * (sl & 3u))) & 0xFFu;
            leaf |= (meta >> 5) << (meta & 31u);
        }
        ng_base = child_base;
        ng_bits = (inner << 24) | imask;
        tg_base = tri_base;
        tg_bits = leaf & 0x00FFFFFFu;
    }
    return ok;
}

// The reference's triangle arithmetic (_IntersectTri, CoreRef.cpp:18-40) on
// one precomputed record (t0, t1, t2) and a ray given by origin and
// direction: true when the ray's line passes the edge tests; then
// t = dett / det, u = detu / det and v = detv / det, each as the product with
// the correctly rounded reciprocal rdet, as the reference computes them.
__device__ __forceinline__ bool tri_core(const float4 &t0, const float4 &t1, const float4 &t2, float ox, float oy, float oz, float dx,
                                         float dy, float dz, float &rdet, float &dett, float &detu, float &detv) {
    const float nu = t0.x, nv = t0.y, npl = t0.z, pu = t0.w, pv = t1.x, e0u = t1.z, e0v = t1.w, e1u = t2.x, e1v = t2.y;
    const int iw = __float_as_int(t1.y) & TRI_W_BITS;
    const float du = iw == 0 ? dy : dx, dv = iw == 2 ? dy : dz, dw = iw == 0 ? dx : (iw == 1 ? dy : dz);
    const float ou = iw == 0 ? oy : ox, ov = iw == 2 ? oy : oz, ow = iw == 0 ? ox : (iw == 1 ? oy : oz);
    const float det = __fadd_rn(__fadd_rn(__fmul_rn(du, nu), __fmul_rn(dv, nv)), dw);
    dett = __fsub_rn(npl, __fadd_rn(__fadd_rn(__fmul_rn(ou, nu), __fmul_rn(ov, nv)), ow));
    const float Du = __fsub_rn(__fmul_rn(du, dett), __fmul_rn(__fsub_rn(pu, ou), det));
    const float Dv = __fsub_rn(__fmul_rn(dv, dett), __fmul_rn(__fsub_rn(pv, ov), det));
    detu = __fsub_rn(__fmul_rn(e1v, Du), __fmul_rn(e1u, Dv));
    detv = __fsub_rn(__fmul_rn(e0u, Dv), __fmul_rn(e0v, Du));
    const float tmpdet0 = __fsub_rn(__fsub_rn(det, detu), detv);
    if ((tmpdet0 > -HIT_EPS && detu > -HIT_EPS && detv > -HIT_EPS) || (tmpdet0 < HIT_EPS && detu < HIT_EPS && detv < HIT_EPS)) {
        rdet = __frcp_rn(det); // 1.0f / det, correctly rounded
        return true;
    }
    return false;
}

// A triangle test of a group's lane against the ray's best hit so far: true
// when it is the closer one (tri_test's rule), with its t, u, v and index.
template <typename BEST>
__device__ __forceinline__ bool tri_candidate(const MeshRef &mr, const LocalRay &r, uint32_t li, const BEST &best, uint32_t &err, float &t,
                                              float &u, float &v, int &gp, bool &solid) {
    if (li >= mr.tri_count) {
        err |= TRACE_ERR_BOUNDS;
        return false;
    }
    const float4 *tp = reinterpret_cast<const float4 *>(mr.tris + li);
    const float4 t0 = __ldg(tp), t1 = __ldg(tp + 1), t2 = __ldg(tp + 2);
    float rdet, dett, detu, detv;
    if (!tri_core(t0, t1, t2, r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, rdet, dett, detu, detv)) return false;
    t = __fmul_rn(dett, rdet);
    gp = (int)(mr.prim_base + __float_as_uint(t2.z));
    u = __fmul_rn(detu, rdet);
    v = __fmul_rn(detv, rdet);
    solid = (__float_as_int(t1.y) & TRI_SOLID_BIT) != 0;
    return t > 0.0f && (t < best.t || (t == best.t && best.prim >= 0 && gp <= best.prim && (gp < best.prim || mr.obj < best.obj_of())));
}

// One triangle test; updates best when it is the closer hit. With SOLID,
// returns whether that hit is on a solid triangle (TRI_SOLID_BIT), which ends
// a shadow ray's search (IntersectTris_AnyHit, CoreRef.cpp:804-829).
template <bool COUNT, bool SOLID = false, typename BEST>
__device__ __forceinline__ bool tri_test(const MeshRef &mr, const LocalRay &r, uint32_t li, BEST &best, uint32_t &err, uint32_t &ntri) {
    if (li >= mr.tri_count) {
        err |= TRACE_ERR_BOUNDS;
        return false;
    }
    const float4 *tp = reinterpret_cast<const float4 *>(mr.tris + li);
    const float4 t0 = __ldg(tp), t1 = __ldg(tp + 1), t2 = __ldg(tp + 2);
    if (COUNT) ntri++;
    float rdet, dett, detu, detv;
    if (tri_core(t0, t1, t2, r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, rdet, dett, detu, detv)) {
        const float t = __fmul_rn(dett, rdet);
        const int gp = (int)(mr.prim_base + __float_as_uint(t2.z));
        // a tie goes to the lower triangle index, then to the lower instance:
        // independent of the visiting order
        if (t > 0.0f && (t < best.t || (t == best.t && best.prim >= 0 && gp <= best.prim && (gp < best.prim || mr.obj < best.obj_of())))) {
            best.t = t;
            best.prim = gp;
            best.rest(__fmul_rn(detu, rdet), __fmul_rn(detv, rdet), mr.obj);
            if (SOLID) return (__float_as_int(t1.y) & TRI_SOLID_BIT) != 0;
        }
    }
    return false;
}

// Whole traversal of one mesh for one ray (the one-thread-per-ray kernel).
// The current node group always has a child left at the top of the loop: the
// root's, then the group a node step returns or one taken from the stack.
template <bool COUNT, typename ST>
__device__ __forceinline__ void trace_mesh(const MeshRef &mr, const LocalRay &r, Best &best, ST &st, uint32_t &err,
                                           uint32_t &nvis, uint32_t &ntri) {
    uint32_t ng_base = 0, ng_bits = r.root_bits();
    uint32_t tg_base = 0, tg_bits = 0, visits = 0;
    const int sp0 = st.sp; // the caller's entries below
    while (true) {
        if (!node_step<COUNT>(mr, r, best.t, ng_base, ng_bits, tg_base, tg_bits, st, visits, err, nvis)) return;
        while (tg_bits) {
            const uint32_t k = __ffs(tg_bits) - 1;
            tg_bits &= tg_bits - 1;
            tri_test<COUNT>(mr, r, tg_base + k, best, err, ntri);
        }
        if (ng_bits <= 0x00FFFFFFu) {
            if (st.sp == sp0) return;
            const uint2 e = st.pop();
            ng_base = e.x;
            ng_bits = e.y;
        }
    }
}

// Shadow-ray traversal of one mesh (Traverse_MicroTree_WithStack_AnyHit,
// CoreRef.cpp:1470-1577): closest-hit order, stopping at the first accepted
// hit on a solid triangle. Returns true when it stopped there.
template <typename ST>
__device__ __forceinline__ bool trace_mesh_any(const MeshRef &mr, const LocalRay &r, Best &best, ST &st, uint32_t &err) {
    uint32_t ng_base = 0, ng_bits = r.root_bits();
    uint32_t tg_base = 0, tg_bits = 0, visits = 0, nvis = 0, ntri = 0;
    st.sp = 0;
    while (true) {
        if (!node_step<false>(mr, r, best.t, ng_base, ng_bits, tg_base, tg_bits, st, visits, err, nvis)) return false;
        while (tg_bits) {
            const uint32_t k = __ffs(tg_bits) - 1;
            tg_bits &= tg_bits - 1;
            if (tri_test<false, true>(mr, r, tg_base + k, best, err, ntri)) return true;
        }
        if (ng_bits <= 0x00FFFFFFu) {
            if (st.sp == 0) return false;
            const uint2 e = st.pop();
            ng_base = e.x;
            ng_bits = e.y;
        }
    }
}

// Closest hit of one ray (r0, r1) against the whole scene, one thread: the
// instances of the tree where the scene has one, else all in turn.
template <bool COUNT, bool TLAS, typename ST>
__device__ __forceinline__ void trace_scene(const SceneView &sv, float4 r0, float4 r1, Best &best, ST &st, uint32_t &err, uint32_t &nvis,
                                            uint32_t &ntri) {
    const float sx = safe_inv(r1.x), sy = safe_inv(r1.y), sz = safe_inv(r1.z);
    if (TLAS && sv.tlas) {
        const MeshRef tree = tree_of(sv);
        const LocalRay w = world_ray(r0.x, r0.y, r0.z, sx, sy, sz);
        uint32_t ng_base = 0, ng_bits = w.root_bits(), tg_base = 0, tg_bits = 0, visits = 0, none = 0;
        st.sp = 0;
        while (true) {
            if (ng_bits > 0x00FFFFFFu && !node_step<false>(tree, w, best.t, ng_base, ng_bits, tg_base, tg_bits, st, visits, err, none)) return;
            const int floor_sp = st.sp;
            for (int m; (m = next_instance(sv, w, best.t, tg_base, tg_bits, err)) >= 0;) {
                // the mesh's groups go on top of the tree's
                const InstanceRec *ir = sv.inst + m;
                trace_mesh<COUNT>(mesh_of(sv, ir, m), transform_ray(ir, r0, r1), best, st, err, nvis, ntri);
                st.sp = floor_sp;
            }
            if (ng_bits <= 0x00FFFFFFu) {
                if (st.sp == 0) return;
                const uint2 e = st.pop();
                ng_base = e.x;
                ng_bits = e.y;
            }
        }
    }
    for (uint32_t m = 0; m < sv.n_inst; m++) {
        const InstanceRec *ir = sv.inst + m;
        float bmin[3], bmax[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            bmin[k] = __ldg(&ir->bbox_min[k]);
            bmax[k] = __ldg(&ir->bbox_max[k]);
        }
        if (!ref_bbox_test(r0.x, r0.y, r0.z, sx, sy, sz, best.t, bmin, bmax)) continue;
        st.sp = 0;
        trace_mesh<COUNT>(mesh_of(sv, ir, (int)m), transform_ray(ir, r0, r1), best, st, err, nvis, ntri);
    }
}

} // namespace trav
} // namespace rg
