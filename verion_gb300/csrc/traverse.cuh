// Software ray traversal of the quantised 8-wide BVH (bvh8.h) on sm_103a, standing in for the
// hardware ray queries of Verion's kernels: `traceClosest` (shaders/include/pt_core.slang:684-700,
// closest opaque hit, TMin 0, TMax 1e30) and the shadow-ray query inside `occluded` (:580-613,
// accept the first hit and end the search).
//
// Hit rule, identical in the CPU oracle: a triangle is hit at distance t when the watertight test
// of Woop, Benthin and Wald ("Watertight Ray/Triangle Intersection", JCGT 2013) accepts it and
// 0 < t < tmax. The closest hit is the smallest t; equal distances go to the lower global triangle
// index, so the answer does not depend on the order the tree is walked in.
//
// Child boxes are tested in the node-local form of Ylitie, Karras and Laine (HPG 2017), one FMA per
// plane, with an explicit bound on its rounding error added outwards, so a box the ray touches is
// never rejected and the culling cannot change the answer.
#pragma once
#include "bvh8.h"
#include "vec3.h"

namespace vgt {

struct TRay {
    V3 o, d;
    float ix, iy, iz; // reciprocal direction for the slab test (tiny components clamped)
    uint32_t oct;     // sign octant of the direction
    int kx, ky, kz;   // watertight test axis permutation
    float sx, sy, sz; // watertight test shear
};

__device__ __forceinline__ float slab_rcp(float d)
{
    float a = fabsf(d);
    if (a < bvh8::MIN_DIR)
        d = copysignf(bvh8::MIN_DIR, d);
    return 1.0f / d;
}

__device__ __forceinline__ TRay make_ray(V3 o, V3 d)
{
    TRay r;
    r.o = o;
    r.d = d;
    r.ix = slab_rcp(d.x);
    r.iy = slab_rcp(d.y);
    r.iz = slab_rcp(d.z);
    r.oct = (d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u);
    float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    int kz = 0;
    if (ay > ax)
        kz = 1;
    if (az > (kz == 0 ? ax : ay))
        kz = 2;
    int kx = kz + 1 == 3 ? 0 : kz + 1;
    int ky = kx + 1 == 3 ? 0 : kx + 1;
    float dz = comp(d, kz);
    if (dz < 0.0f) {
        int t = kx;
        kx = ky;
        ky = t;
    }
    r.kx = kx;
    r.ky = ky;
    r.kz = kz;
    r.sx = comp(d, kx) / dz;
    r.sy = comp(d, ky) / dz;
    r.sz = 1.0f / dz;
    return r;
}

// A triangle's vertices relative to a ray's origin, in the ray's axis permutation.
struct TriRel {
    float ax, ay, az, bx, by, bz, cx, cy, cz;
};

__device__ __forceinline__ TriRel tri_relative(V3 o, int kx, int ky, int kz, V3 v0, V3 v1, V3 v2)
{
    V3 A = v0 - o, B = v1 - o, C = v2 - o;
    return TriRel{comp(A, kx), comp(A, ky), comp(A, kz), comp(B, kx), comp(B, ky),
                  comp(B, kz), comp(C, kx), comp(C, ky), comp(C, kz)};
}

// Watertight test of a ray of shear (sx, sy, sz). On success returns true with the distance t = T / det and the
// edge functions (U, V, W weigh vertices 0, 1, 2; divided by det they are the barycentrics). (Tried: a sign and
// magnitude test ahead of the division, rejecting where the quotient could only be rejected
// against the closest hit so far; it measured 1.5% slower per extend launch.)
__device__ __forceinline__ bool tri_test(const TriRel& v, float sx, float sy, float sz, float& t, float& U, float& V,
                                         float& W, float& det)
{
    float Ax = v.ax - sx * v.az;
    float Ay = v.ay - sy * v.az;
    float Bx = v.bx - sx * v.bz;
    float By = v.by - sy * v.bz;
    float Cx = v.cx - sx * v.cz;
    float Cy = v.cy - sy * v.cz;
    U = Cx * By - Cy * Bx;
    V = Ax * Cy - Ay * Cx;
    W = Bx * Ay - By * Ax;
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        // Edge hit: redo the 2x2 determinants in double precision (the paper's fallback).
        double cxby = (double)Cx * (double)By, cybx = (double)Cy * (double)Bx;
        double axcy = (double)Ax * (double)Cy, aycx = (double)Ay * (double)Cx;
        double bxay = (double)Bx * (double)Ay, byax = (double)By * (double)Ax;
        U = (float)(cxby - cybx);
        V = (float)(axcy - aycx);
        W = (float)(bxay - byax);
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f))
        return false;
    det = U + V + W;
    if (det == 0.0f)
        return false;
    float Az = sz * v.az;
    float Bz = sz * v.bz;
    float Cz = sz * v.cz;
    float T = U * Az + V * Bz + W * Cz;
    t = T / det;
    return t > 0.0f;
}

__device__ __forceinline__ bool tri_test(const TRay& r, V3 v0, V3 v1, V3 v2, float& t, float& U, float& V, float& W,
                                         float& det)
{
    return tri_test(tri_relative(r.o, r.kx, r.ky, r.kz, v0, v1, v2), r.sx, r.sy, r.sz, t, U, V, W, det);
}

struct TraceHit {
    bool hit;
    uint32_t inst, prim;
    float t;
    float b1, b2;           // barycentric weights of vertices 1 and 2
    uint32_t nodes, tests;  // nodes visited and triangles tested (dropped by the compiler unless read)
};

// The byte as a float plus 2^15, exactly: the byte placed in bits 8-15 of the mantissa of 2^15 (one
// byte permute; the last place of the float there is 2^-8). The node test folds the 2^15 into the
// constant of its FMA, so a plane costs a permute and an FMA, with no subtraction.
__device__ __forceinline__ float byte_f15(uint32_t lo, uint32_t hi, int i)
{
    uint32_t w = i < 4 ? lo : hi;
    return __uint_as_float(__byte_perm(w, 0x47000000u, 0x7604u + ((uint32_t)(i & 3) << 4)));
}

__device__ __forceinline__ float max3(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

__device__ __forceinline__ float min3(float a, float b, float c)
{
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Index of the highest set bit (x != 0).
__device__ __forceinline__ uint32_t high_bit(uint32_t x) { return 31u - (uint32_t)__clz((int)x); }

// x << (s mod 32): the shift count's upper bits are ignored, so a packed byte needs no mask.
__device__ __forceinline__ uint32_t shl_wrap(uint32_t x, uint32_t s) { return __funnelshift_l(0u, x, s); }

// What the box test reads of a ray: its origin, and per axis the reciprocal direction that its near and
// its far plane are divided by (one and the same for a single ray; the ends of an interval of directions
// for a beam of rays from one origin, whose components must not change sign within it).
struct Slabs {
    V3 o;
    float nx, ny, nz, fx, fy, fz;
    uint32_t oct;
};

__device__ __forceinline__ Slabs slabs_of(const TRay& r)
{
    return Slabs{r.o, r.ix, r.iy, r.iz, r.ix, r.iy, r.iz, r.oct};
}

// Child-box tests of one BVH8 node (words w0, w1.zw = meta, w2..w4, bvh8.h) for a ray with the
// closest hit so far at best_t. Returns the hit children in one word: bits 24-31 the internal ones
// (bit 24 + (slot XOR octant XOR 7): the highest set bit is the child to visit first), bits 0-23 the
// triangles of the hit leaf slots, from the node's triangle base.
//
// Node-local ray (Ylitie et al. 2017): t(q) = A + q S per axis with A = (p - o) / d and S = 2^e / d,
// one FMA per plane. The plane p + q 2^e is exact; A and S carry at most a few roundings, a
// relative 2^-21 at most. The FMA takes 2^15 + q (byte_f15) and the constant A - 2^15 S, whose
// rounding is at most 2^-9 |S| + 2^-24 |A|. So every t is moved outwards by
// err = 2^-21 |A| + 2^-8 |S|, a bound on all of it: the test never rejects a box the ray enters, and
// the hits stay those of brute force. The margin of 1/256 of a quantisation step adds no measurable
// node visits; the byte's exact value (a subtraction per plane, 48 per node) needed 2^-13 of a step.
//
// Each child ends in one predicated OR of its meta byte's bits: no branch, whatever the lanes hit.
__device__ __forceinline__ uint32_t node_test(const Slabs& r, uint4 w0, uint32_t meta_lo, uint32_t meta_hi, uint4 w2,
                                              uint4 w3, uint4 w4, float best_t)
{
    float px = __uint_as_float(w0.x), py = __uint_as_float(w0.y), pz = __uint_as_float(w0.z);
    uint32_t em = w0.w;
    float scx = __uint_as_float((em & 0xffu) << 23);
    float scy = __uint_as_float(((em >> 8) & 0xffu) << 23);
    float scz = __uint_as_float(((em >> 16) & 0xffu) << 23);
    bool px_pos = r.nx >= 0.0f, py_pos = r.ny >= 0.0f, pz_pos = r.nz >= 0.0f;
    // Near and far quantised planes per axis (low words at w2.x .. high words at w4.w).
    uint32_t nxl = px_pos ? w2.x : w3.z, nxh = px_pos ? w2.y : w3.w;
    uint32_t fxl = px_pos ? w3.z : w2.x, fxh = px_pos ? w3.w : w2.y;
    uint32_t nyl = py_pos ? w2.z : w4.x, nyh = py_pos ? w2.w : w4.y;
    uint32_t fyl = py_pos ? w4.x : w2.z, fyh = py_pos ? w4.y : w2.w;
    uint32_t nzl = pz_pos ? w3.x : w4.z, nzh = pz_pos ? w3.y : w4.w;
    uint32_t fzl = pz_pos ? w4.z : w3.x, fzh = pz_pos ? w4.w : w3.y;
    float dx = px - r.o.x, dy = py - r.o.y, dz = pz - r.o.z;
    float snx = scx * r.nx, sny = scy * r.ny, snz = scz * r.nz;
    float sfx = scx * r.fx, sfy = scy * r.fy, sfz = scz * r.fz;
    float anx = dx * r.nx, any_ = dy * r.ny, anz = dz * r.nz;
    float afx = dx * r.fx, afy = dy * r.fy, afz = dz * r.fz;
    constexpr float EA = 4.76837158e-7f, ES = 3.90625e-3f; // 2^-21, 2^-8
    anx = fmaf(-32768.0f, snx, anx - fmaf(EA, fabsf(anx), ES * fabsf(snx)));
    any_ = fmaf(-32768.0f, sny, any_ - fmaf(EA, fabsf(any_), ES * fabsf(sny)));
    anz = fmaf(-32768.0f, snz, anz - fmaf(EA, fabsf(anz), ES * fabsf(snz)));
    afx = fmaf(-32768.0f, sfx, afx + fmaf(EA, fabsf(afx), ES * fabsf(sfx)));
    afy = fmaf(-32768.0f, sfy, afy + fmaf(EA, fabsf(afy), ES * fabsf(sfy)));
    afz = fmaf(-32768.0f, sfz, afz + fmaf(EA, fabsf(afz), ES * fabsf(sfz)));
    uint32_t flip = (r.oct ^ 7u) * 0x01010101u;
    uint32_t found = 0;
#pragma unroll
    for (int half = 0; half < 2; half++) {
        uint32_t meta = half ? meta_hi : meta_lo;
        // Bytes of internal slots have bits 3 and 4 set (bit index 24 + slot): flip their slot.
        uint32_t inner = (meta & (meta << 1)) & 0x10101010u;
        uint32_t at = meta ^ (((inner >> 4) * 7u) & flip);
        uint32_t bits = (meta >> 5) & 0x07070707u;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            int i = 4 * half + j;
            float tnx = fmaf(byte_f15(nxl, nxh, i), snx, anx);
            float tny = fmaf(byte_f15(nyl, nyh, i), sny, any_);
            float tnz = fmaf(byte_f15(nzl, nzh, i), snz, anz);
            float tfx = fmaf(byte_f15(fxl, fxh, i), sfx, afx);
            float tfy = fmaf(byte_f15(fyl, fyh, i), sfy, afy);
            float tfz = fmaf(byte_f15(fzl, fzh, i), sfz, afz);
            float tn = fmaxf(max3(tnx, tny, tnz), 0.0f);
            float tf = fminf(min3(tfx, tfy, tfz), best_t);
            uint32_t b = shl_wrap((bits >> (8 * j)) & 0xffu, at >> (8 * j));
            found |= tn <= tf ? b : 0u;
        }
    }
    return found;
}

// A ray's way through the tree. group: the node group being visited, .x its first child's index,
// .y its internal-child mask (bits 0-7) and the children still to visit (bits 24-31, node_test's
// order). tri_base, tri_bits: the triangles of the last visited node still to test. hit_tri: the
// closest hit's triangle record (NO_TRI: none).
constexpr uint32_t NO_TRI = 0xffffffffu;

struct Walk {
    TRay r;
    float tmax;             // the closest hit so far, or the ray's end
    uint32_t hit_tri;
    uint32_t item;          // queue traversal: the ray's queue entry
    uint32_t node;          // the next node to visit
    uint2 group;
    uint32_t tri_base, tri_bits;
    int sp;
    bool any;               // HITS_EITHER: this ray ends at its first hit
    float b1, b2;           // barycentric weights of vertices 1 and 2 at the hit (dropped unless read)
    uint32_t nodes, tests;  // nodes visited and triangles tested (dropped unless read)
};

// What a traversal looks for: every ray's closest hit, any hit, or one of the two by the ray (Walk::any).
enum Hits { HITS_CLOSEST, HITS_ANY, HITS_EITHER };

__device__ __forceinline__ void walk_begin(Walk& w, V3 o, V3 d, float tmax)
{
    w.r = make_ray(o, d);
    w.tmax = tmax;
    w.hit_tri = NO_TRI;
    w.node = 0;
    w.group = make_uint2(0u, 0u);
    w.tri_base = w.tri_bits = 0;
    w.sp = 0;
    w.b1 = w.b2 = 0.0f;
    w.nodes = w.tests = 0;
}

// Visits w.node: its hit internal children become the walk's node group, what the group before it
// had left goes to the stack (next_node), its hit leaf slots' triangles become the pending ones.
__device__ __forceinline__ void node_visit(const uint4* __restrict__ nodes, Walk& w, const Slabs& slabs)
{
    const uint4* np = nodes + (size_t)w.node * bvh8::NODE_VEC4;
    uint4 w0 = __ldg(np), w1 = __ldg(np + 1), w2 = __ldg(np + 2), w3 = __ldg(np + 3), w4 = __ldg(np + 4);
    w.nodes++;
    uint32_t found = node_test(slabs, w0, w1.z, w1.w, w2, w3, w4, w.tmax);
    w.group = make_uint2(w1.x, (found & 0xff000000u) | (w0.w >> 24));
    w.tri_base = w1.y;
    w.tri_bits = found & 0x00ffffffu;
}

// Tests one pending triangle. Returns true when an any-hit walk has its hit.
template <Hits H>
__device__ __forceinline__ bool test_one(const float4* __restrict__ tris, Walk& w)
{
    uint32_t j = high_bit(w.tri_bits);
    w.tri_bits ^= 1u << j;
    uint32_t k = w.tri_base + j;
    const float4* tp = tris + (size_t)k * bvh8::TRI_VEC4;
    float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
    float t, U, V, W, det;
    w.tests++;
    if (tri_test(w.r, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(c.x, c.y, c.z), t, U, V, W, det)) {
        bool take = t < w.tmax;
        if (H != HITS_ANY && t == w.tmax && w.hit_tri != NO_TRI)
            take = __float_as_uint(c.w) < __float_as_uint(__ldg(&tris[(size_t)w.hit_tri * bvh8::TRI_VEC4 + 2].w));
        if (take) {
            w.hit_tri = k;
            w.tmax = t;
            w.b1 = V / det;
            w.b2 = W / det;
            return H == HITS_ANY || (H == HITS_EITHER && w.any);
        }
    }
    return false;
}

// Picks the next node: the first child left in the walk's group, else in the top group of the stack;
// what the group has left then goes (back) to the stack. Returns true when the walk has finished
// (nothing left, or the stack overflowed: the error flag is then set).
__device__ __forceinline__ bool next_node(Walk& w, uint2* stack, uint32_t* err)
{
    uint2 g = w.group;
    if (g.y < 0x01000000u) {
        if (w.sp == 0)
            return true;
        g = stack[--w.sp];
    }
    uint32_t b = high_bit(g.y);
    g.y ^= 1u << b;
    uint32_t slot = (b ^ w.r.oct ^ 7u) & 7u;
    w.node = g.x + __popc(g.y & ((1u << slot) - 1u));
    if (g.y >= 0x01000000u) {
        if (w.sp >= (int)bvh8::STACK_SIZE) {
            atomicOr(err, bvh8::ERR_STACK);
            return true;
        }
        stack[w.sp++] = g;
    }
    return false;
}

// One node visit: box tests, the node's triangles, then the next node. Returns true when the walk has
// finished (nothing left, or an any-hit walk has its hit). (Tried: one triangle a step, a lane with
// more of them skipping the node test of the steps that follow, so that the triangle test runs once
// a step instead of as often as the warp's busiest lane needs: 7% slower on the 1M-triangle workload.)
template <Hits H>
__device__ __forceinline__ bool walk_step(const uint4* __restrict__ nodes, const float4* __restrict__ tris, Walk& w,
                                          uint2* stack, uint32_t* err)
{
    node_visit(nodes, w, slabs_of(w.r));
    while (w.tri_bits)
        if (test_one<H>(tris, w))
            return true;
    return next_node(w, stack, err);
}

__device__ __forceinline__ TraceHit walk_hit(const float4* __restrict__ tris, const Walk& w)
{
    TraceHit h;
    h.hit = w.hit_tri != NO_TRI;
    h.inst = h.prim = 0;
    if (h.hit) {
        const float4* tp = tris + (size_t)w.hit_tri * bvh8::TRI_VEC4;
        h.inst = __float_as_uint(__ldg(&tp[0].w));
        h.prim = __float_as_uint(__ldg(&tp[1].w));
    }
    h.t = w.tmax;
    h.b1 = w.b1;
    h.b2 = w.b2;
    h.nodes = w.nodes;
    h.tests = w.tests;
    return h;
}

// The answer of a queue item without a ray.
__device__ __forceinline__ TraceHit no_hit(float tmax)
{
    TraceHit h;
    h.hit = false;
    h.inst = h.prim = 0;
    h.t = tmax;
    h.b1 = h.b2 = 0.0f;
    h.nodes = h.tests = 0;
    return h;
}

// Closest hit (ANY = false) or any hit (ANY = true) with 0 < t < tmax.
template <bool ANY>
__device__ __forceinline__ TraceHit trace_bvh(const uint4* __restrict__ nodes, const float4* __restrict__ tris, V3 o,
                                              V3 d, float tmax, uint32_t* err)
{
    uint2 stack[bvh8::STACK_SIZE];
    Walk w;
    walk_begin(w, o, d, tmax);
    while (!walk_step<ANY ? HITS_ANY : HITS_CLOSEST>(nodes, tris, w, stack, err)) {
    }
    return walk_hit(tris, w);
}

// ---------------------------------------------------------------------------------------------
// Warp-cooperative leaf testing. In walk_step every lane tests its node's triangles itself, so a
// warp runs its triangle loop as often as its busiest lane needs while the other lanes idle: on the
// 1M-triangle workload about a third of the lanes are active per instruction. Here a step is split
// in three: every lane tests its node's child boxes (node_visit), then the warp tests all the
// (ray, triangle) pairs its lanes collected, one pair per lane (coop_tris), and then every lane
// picks its next node (next_node). The visiting order per ray is walk_step's, and the hit rule does
// not depend on which lane tests a triangle, so the results and the counters are the same.
// Measured on the 1M-triangle workload (1080p, depth 16, before the node test lost its branches): the extend
// stage took 0.447 ms per launch this way against 0.407 ms with each lane testing its own triangles, so it is
// off by default: the per-step scan, owner search and shared-memory reductions cost more issue slots than the
// divergent triangle loop they replace.
//
// A pair lane reads the owner's ray from shared memory (written once per ray) and reports a hit
// with a 64-bit shared-memory atomicMin of (t bits << 32 | global triangle index) on the owner's
// slot: for t > 0 the float bits order like the floats, so the minimum is the closest hit with the
// lower index on ties, the rule of trace_bvh. The winning lane then leaves the hit's triangle
// record and barycentrics in the owner's slot. Any-hit rays only need a flag.

// Shared state of one warp (block size 128: four per block).
struct CoopWarp {
    float4 ra[32];               // owner ray: origin xyz, watertight axes kx | ky << 2 | kz << 4
    float4 rb[32];               // owner ray: shear sx, sy, sz; tmax (any-hit)
    unsigned long long key[32];  // closest-hit candidates, min-reduced
    uint4 info[32];              // the winner's triangle record, 0, b1, b2 bits; any-hit: x = hit
};
constexpr uint32_t COOP_WARPS = 4; // warps per block of the cooperative kernels (128 threads)

__device__ __forceinline__ void coop_publish_ray(CoopWarp& cw, uint32_t lane, const TRay& r, float tmax)
{
    cw.ra[lane] = make_float4(r.o.x, r.o.y, r.o.z, __uint_as_float((uint32_t)(r.kx | (r.ky << 2) | (r.kz << 4))));
    cw.rb[lane] = make_float4(r.sx, r.sy, r.sz, tmax);
}

// Tests every (ray, triangle) pair the warp's lanes collected in this step: lane i owns the
// triangles tri_base + bit of `bits` (its node's hit leaf slots). Called by all 32 lanes of a
// converged warp. Closest hit: the owner's walk takes the closest of them (or keeps its hit) and
// lowers its tmax. Any hit: returns true for an owner with a hit below its tmax (the walk then
// records the hit flag only).
template <bool ANY>
__device__ __forceinline__ bool coop_tris(CoopWarp& cw, uint32_t lane, uint32_t bits, uint32_t tri_base, Walk& w,
                                          const float4* __restrict__ tris)
{
    const uint32_t FULLM = 0xffffffffu;
    uint32_t cnt = __popc(bits);
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t v = __shfl_up_sync(FULLM, incl, o);
        if (lane >= (uint32_t)o)
            incl += v;
    }
    uint32_t total = __shfl_sync(FULLM, incl, 31);
    if (total == 0)
        return false;
    uint32_t excl = incl - cnt;
    unsigned long long init = 0;
    if (cnt) {
        w.tests += cnt;
        if (ANY) {
            cw.info[lane].x = 0u;
        } else {
            uint32_t gid = 0;
            if (w.hit_tri != NO_TRI)
                gid = __float_as_uint(__ldg(&tris[(size_t)w.hit_tri * bvh8::TRI_VEC4 + 2].w));
            init = ((unsigned long long)__float_as_uint(w.tmax) << 32) | gid;
            cw.key[lane] = init;
        }
    }
    __syncwarp();
    for (uint32_t q0 = 0; q0 < total; q0 += 32) {
        uint32_t q = q0 + lane;
        // Owner of pair q: the number of lanes whose inclusive count is <= q (a binary search over
        // the lanes' non-decreasing counts).
        uint32_t L = 0;
#pragma unroll
        for (uint32_t b = 16; b > 0; b >>= 1) {
            uint32_t v = __shfl_sync(FULLM, incl, L + b - 1);
            if (v <= q)
                L += b;
        }
        uint32_t obits = __shfl_sync(FULLM, bits, L);
        uint32_t oexcl = __shfl_sync(FULLM, excl, L);
        uint32_t obase = __shfl_sync(FULLM, tri_base, L);
        bool mine = false;
        unsigned long long key = 0;
        float V = 0.0f, Wb = 0.0f, det = 1.0f;
        uint32_t ktri = 0;
        if (q < total) {
            for (uint32_t j = q - oexcl; j > 0; j--)
                obits &= obits - 1;
            ktri = obase + __ffs(obits) - 1;
            const float4* tp = tris + (size_t)ktri * bvh8::TRI_VEC4;
            float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
            float4 ra = cw.ra[L], rb = cw.rb[L];
            TRay r;
            r.o = v3(ra.x, ra.y, ra.z);
            uint32_t kk = __float_as_uint(ra.w);
            r.kx = (int)(kk & 3u);
            r.ky = (int)((kk >> 2) & 3u);
            r.kz = (int)((kk >> 4) & 3u);
            r.sx = rb.x;
            r.sy = rb.y;
            r.sz = rb.z;
            float t, U;
            if (tri_test(r, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(c.x, c.y, c.z), t, U, V, Wb, det)) {
                if (ANY) {
                    if (t < rb.w)
                        cw.info[L].x = 1u;
                } else {
                    key = ((unsigned long long)__float_as_uint(t) << 32) | __float_as_uint(c.w);
                    atomicMin(&cw.key[L], key);
                    mine = true;
                }
            }
        }
        if (!ANY) {
            __syncwarp();
            // The lane whose candidate is the owner's minimum so far leaves its hit there.
            if (mine && cw.key[L] == key)
                cw.info[L] = make_uint4(ktri, 0u, __float_as_uint(V / det), __float_as_uint(Wb / det));
        }
        __syncwarp();
    }
    if (cnt == 0)
        return false;
    if (ANY)
        return cw.info[lane].x != 0u;
    unsigned long long best = cw.key[lane];
    if (best < init) {
        uint4 in = cw.info[lane];
        w.tmax = __uint_as_float((uint32_t)(best >> 32));
        w.hit_tri = in.x;
        w.b1 = __uint_as_float(in.z);
        w.b2 = __uint_as_float(in.w);
    }
    return false;
}

// trace_queue (below) with warp-cooperative leaf testing (same dynamic fetch, same results). `cw` is this
// warp's shared state.
template <bool ANY, typename GetRay, typename PutHit>
__device__ __forceinline__ void trace_queue_coop(const uint4* __restrict__ nodes, const float4* __restrict__ tris,
                                                 uint32_t* fetch, uint32_t count, uint32_t* err, uint32_t refill,
                                                 uint32_t steps, CoopWarp& cw, GetRay get, PutHit put)
{
    const uint32_t FULLM = 0xffffffffu;
    uint32_t lane = threadIdx.x & 31u;
    uint32_t lt = (1u << lane) - 1u;
    uint2 stack[bvh8::STACK_SIZE];
    Walk w;
    bool active = false, exhausted = false;
    for (;;) {
        uint32_t need = __ballot_sync(FULLM, !active);
        if (!exhausted && (need == FULLM || (uint32_t)__popc(need) >= refill)) {
            uint32_t n = __popc(need);
            uint32_t base = 0;
            if (lane == 0)
                base = atomicAdd(fetch, n);
            base = __shfl_sync(FULLM, base, 0);
            exhausted = base + n >= count;
            if (!active) {
                uint32_t idx = base + __popc(need & lt);
                if (idx < count) {
                    V3 o, d;
                    float tmax;
                    if (get(idx, o, d, tmax, w.any)) {
                        walk_begin(w, o, d, tmax);
                        w.item = idx;
                        active = true;
                        coop_publish_ray(cw, lane, w.r, tmax);
                    } else {
                        put(idx, no_hit(tmax));
                    }
                }
            }
        }
        if (__ballot_sync(FULLM, active) == 0) {
            if (exhausted)
                break;
            continue;
        }
        __syncwarp();
#pragma unroll 1
        for (uint32_t s = 0; s < steps; s++) {
            uint32_t bits = 0;
            if (active) {
                node_visit(nodes, w, slabs_of(w.r));
                bits = w.tri_bits;
                w.tri_bits = 0;
            }
            bool hit = coop_tris<ANY>(cw, lane, bits, w.tri_base, w, tris);
            if (active) {
                if (ANY && hit)
                    w.hit_tri = 0; // any-hit: the flag alone
                if ((ANY && hit) || next_node(w, stack, err)) {
                    put(w.item, walk_hit(tris, w));
                    active = false;
                }
            }
            if (__ballot_sync(FULLM, active) == 0)
                break;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Queue traversal with dynamic ray fetch: a warp keeps one ray per lane and, whenever at least
// `refill` lanes have finished theirs, hands those lanes the next rays of the queue (one atomic per
// refill), so the warp does not idle on its longest ray (Aila and Laine, "Understanding the
// Efficiency of Ray Traversal on GPUs", HPG 2009). Each lane runs at most `steps` node visits
// between refills. Results are those of trace_bvh: the hit rule does not depend on the visiting order.
//
// get(i, o, d, tmax, any) loads queue item i into a ray (with HITS_EITHER also whether any hit will do)
// and returns false when it has no ray (it then completes at once with a miss); put(i, hit) stores the
// result of item i.

// The body of trace_queue and trace_queue_scenes: with SCENES, `get` also names the BVH of each ray
// (its node and triangle arrays), which the lane keeps while it walks that ray.
template <Hits H, bool SCENES, typename GetRay, typename PutHit>
__device__ __forceinline__ void trace_queue_impl(const uint4* __restrict__ nodes0, const float4* __restrict__ tris0,
                                                 uint32_t* fetch, uint32_t count, uint32_t* err, uint32_t refill,
                                                 uint32_t steps, GetRay get, PutHit put)
{
    const uint32_t FULLM = 0xffffffffu;
    const uint4* nodes = nodes0;
    const float4* tris = tris0;
    uint32_t lane = threadIdx.x & 31u;
    uint32_t lt = (1u << lane) - 1u;
    uint2 stack[bvh8::STACK_SIZE];
    Walk w;
    bool active = false, exhausted = false;
    for (;;) {
        uint32_t need = __ballot_sync(FULLM, !active);
        if (!exhausted && (need == FULLM || (uint32_t)__popc(need) >= refill)) {
            uint32_t n = __popc(need);
            uint32_t base = 0;
            if (lane == 0)
                base = atomicAdd(fetch, n);
            base = __shfl_sync(FULLM, base, 0);
            exhausted = base + n >= count;
            if (!active) {
                uint32_t idx = base + __popc(need & lt);
                if (idx < count) {
                    V3 o, d;
                    float tmax;
                    bool ok;
                    if constexpr (SCENES)
                        ok = get(idx, o, d, tmax, w.any, nodes, tris);
                    else
                        ok = get(idx, o, d, tmax, w.any);
                    if (ok) {
                        walk_begin(w, o, d, tmax);
                        w.item = idx;
                        active = true;
                    } else {
                        put(idx, no_hit(tmax));
                    }
                }
            }
        }
        if (__ballot_sync(FULLM, active) == 0) {
            if (exhausted)
                break;
            continue;
        }
        if (active) {
#pragma unroll 1
            for (uint32_t s = 0; s < steps; s++) {
                if (walk_step<H>(nodes, tris, w, stack, err)) {
                    put(w.item, walk_hit(tris, w));
                    active = false;
                    break;
                }
            }
        }
    }
}

template <Hits H, typename GetRay, typename PutHit>
__device__ __forceinline__ void trace_queue(const uint4* __restrict__ nodes, const float4* __restrict__ tris,
                                            uint32_t* fetch, uint32_t count, uint32_t* err, uint32_t refill,
                                            uint32_t steps, GetRay get, PutHit put)
{
    trace_queue_impl<H, false>(nodes, tris, fetch, count, err, refill, steps, get, put);
}

// trace_queue over the rays of several scenes: get(idx, o, d, tmax, any, nodes, tris) also sets the
// ray's BVH arrays.
template <Hits H, typename GetRay, typename PutHit>
__device__ __forceinline__ void trace_queue_scenes(uint32_t* fetch, uint32_t count, uint32_t* err, uint32_t refill,
                                                   uint32_t steps, GetRay get, PutHit put)
{
    trace_queue_impl<H, true>(nullptr, nullptr, fetch, count, err, refill, steps, get, put);
}

} // namespace vgt
