// Primary-hit AOV kernels: shaders/normals.slang:41-110 (interpolated normal facing the viewer) and
// shaders/aov.slang:86-188 (albedo, depth, object / material id through the pixel centre, and
// coverage of 16 stratified rays followed through translucent surfaces). One thread per pixel.
//
// The camera record is the reference's (crates/verion-gpu/src/pack.rs:97-108): width, height,
// tan(fov/2), pad, the camera-to-world 3x4 rows, lens shift x and y.
#pragma once
#include "pt_device.cuh"

namespace vga {

using namespace vgd;

struct CameraRecord {
    float v[18];
};

// aov.slang:79-86: camera-space position on the plane z = -1 of pixel position (px, py).
__device__ __forceinline__ float planeU(const CameraRecord& cam, float px, uint32_t w, float t, float aspect)
{
    return (2.0f * px / (float)w - 1.0f + cam.v[16]) * aspect * t;
}

__device__ __forceinline__ float planeV(const CameraRecord& cam, float py, uint32_t h, float t)
{
    return (1.0f - 2.0f * py / (float)h + cam.v[17]) * t;
}

// Camera-space unit direction through (u, v) on that plane, world direction in dir.
__device__ __forceinline__ V3 planeDir(const CameraRecord& cam, float u, float v, V3& dir)
{
    V3 d = normalize(v3(u, v, -1.0f));
    float r[3];
#pragma unroll
    for (int k = 0; k < 3; k++)
        r[k] = cam.v[4 + 4 * k] * d.x + cam.v[5 + 4 * k] * d.y + cam.v[6 + 4 * k] * d.z;
    dir = v3(r[0], r[1], r[2]);
    return d;
}

// The same through pixel position (px, py).
__device__ __forceinline__ V3 pixelDir(const CameraRecord& cam, float px, float py, uint32_t w, uint32_t h, float t,
                                       float aspect, V3& dir)
{
    return planeDir(cam, planeU(cam, px, w, t, aspect), planeV(cam, py, h, t), dir);
}

// The hit triangle's world vertices and the barycentric weights of vertices 1 and 2 at distance t.
__device__ __forceinline__ void hitGeometry(const Ctx& c, Hit hq, V3 org, V3 dir, V3& p0, V3& p1, V3& p2, float& b1,
                                            float& b2, uint32_t& i0, uint32_t& i1, uint32_t& i2)
{
    uint32_t inst = hq.inst * 16;
    uint32_t tri = __ldg(c.s.instances + inst + 1) + 3 * hq.prim;
    uint32_t vo = __ldg(c.s.instances + inst);
    i0 = __ldg(c.s.indices + tri) + vo;
    i1 = __ldg(c.s.indices + tri + 1) + vo;
    i2 = __ldg(c.s.indices + tri + 2) + vo;
    p0 = transformPoint(c, inst + 4, vertexPos(c, i0));
    p1 = transformPoint(c, inst + 4, vertexPos(c, i1));
    p2 = transformPoint(c, inst + 4, vertexPos(c, i2));
    V3 e1 = p1 - p0, e2 = p2 - p0, e3 = org + dir * hq.t - p0;
    float d11 = dot(e1, e1), d12 = dot(e1, e2), d22 = dot(e2, e2);
    float den = fmaxf(d11 * d22 - d12 * d12, 1.0e-20f);
    b1 = (d22 * dot(e3, e1) - d12 * dot(e3, e2)) / den;
    b2 = (d11 * dot(e3, e2) - d12 * dot(e3, e1)) / den;
}

// normals.slang:41-110
static __global__ void __launch_bounds__(128) aov_normals(const __grid_constant__ Ctx c, CameraRecord cam, float* out)
{
    uint32_t w = (uint32_t)cam.v[0], h = (uint32_t)cam.v[1];
    uint32_t x = blockIdx.x * 16 + (threadIdx.x & 15u), y = blockIdx.y * 8 + (threadIdx.x >> 4);
    if (x >= w || y >= h)
        return;
    float t = cam.v[2];
    float aspect = cam.v[0] / cam.v[1];
    float u = (2.0f * ((float)x + 0.5f) / (float)w - 1.0f + cam.v[16]) * aspect * t;
    float v = (1.0f - 2.0f * ((float)y + 0.5f) / (float)h + cam.v[17]) * t;
    V3 d = normalize(v3(u, v, -1.0f));
    float dr[3], orr[3];
#pragma unroll
    for (int r = 0; r < 3; r++) {
        dr[r] = cam.v[4 + 4 * r] * d.x + cam.v[5 + 4 * r] * d.y + cam.v[6 + 4 * r] * d.z;
        orr[r] = cam.v[7 + 4 * r];
    }
    V3 org = v3(orr[0], orr[1], orr[2]);
    V3 dir = normalize(v3(dr[0], dr[1], dr[2]));
    Hit hq = traceClosest(c, org, dir);
    V3 n = v3(0.0f);
    if (hq.hit) {
        V3 p0, p1, p2;
        float b1, b2;
        uint32_t i0, i1, i2;
        hitGeometry(c, hq, org, dir, p0, p1, p2, b1, b2, i0, i1, i2);
        V3 ng = normalize(cross(p1 - p0, p2 - p0));
        n = ng;
        V3 nsObj = (1.0f - b1 - b2) * vertexNormal(c, i0) + b1 * vertexNormal(c, i1) + b2 * vertexNormal(c, i2);
        if (dot(nsObj, nsObj) > 1.0e-12f) {
            n = normalize(transformNormal(c, hq.inst * 16 + 4, nsObj));
            if (dot(n, ng) < 0.0f)
                n = -n;
        }
        if (dot(ng, dir) > 0.0f)
            n = -n;
    }
    size_t o = 3 * ((size_t)y * w + x);
    out[o] = n.x;
    out[o + 1] = n.y;
    out[o + 2] = n.z;
}

// aov.slang:86-188 but for the coverage (aov_coverage_*). Albedo and depth go to planes of their own or
// interleaved, by their strides. Also clears the counters of the coverage's rest (two words).
static __global__ void __launch_bounds__(128) aov_main(const __grid_constant__ Ctx c, CameraRecord cam,
                                                       float* albedo, uint32_t albedo_stride, float* depths,
                                                       uint32_t depth_stride, uint32_t* object_ids,
                                                       uint32_t* material_ids, uint32_t* rest_counters)
{
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 2)
        rest_counters[threadIdx.x] = 0;
    uint32_t w = (uint32_t)cam.v[0], h = (uint32_t)cam.v[1];
    uint32_t x = blockIdx.x * 16 + (threadIdx.x & 15u), y = blockIdx.y * 8 + (threadIdx.x >> 4);
    if (x >= w || y >= h)
        return;
    float t = cam.v[2];
    float aspect = cam.v[0] / cam.v[1];
    V3 org = v3(cam.v[7], cam.v[11], cam.v[15]);
    V3 dir;
    V3 d = pixelDir(cam, (float)x + 0.5f, (float)y + 0.5f, w, h, t, aspect, dir);
    dir = normalize(dir);
    Hit hq = traceClosest(c, org, dir);
    V3 alb = v3(0.0f);
    float depth = 0.0f;
    uint32_t id = 0, matId = 0;
    if (hq.hit) {
        uint32_t inst = hq.inst * 16;
        id = hq.inst + 1;
        uint32_t mat = __ldg(c.s.instances + inst + 2);
        matId = mat + 1;
        depth = hq.t * -d.z;
        uint32_t mi = mat * 24;
        alb = v3(__ldg(c.s.materials + mi), __ldg(c.s.materials + mi + 1), __ldg(c.s.materials + mi + 2));
        uint32_t texBase = (uint32_t)__ldg(c.s.materials + mi + 10);
        if (texBase > 0) {
            V3 p0, p1, p2;
            float b1, b2;
            uint32_t i0, i1, i2;
            hitGeometry(c, hq, org, dir, p0, p1, p2, b1, b2, i0, i1, i2);
            float u0x = __ldg(c.s.uvs + 2 * i0), u0y = __ldg(c.s.uvs + 2 * i0 + 1);
            float u1x = __ldg(c.s.uvs + 2 * i1), u1y = __ldg(c.s.uvs + 2 * i1 + 1);
            float u2x = __ldg(c.s.uvs + 2 * i2), u2y = __ldg(c.s.uvs + 2 * i2 + 1);
            float ux = u0x + b1 * (u1x - u0x) + b2 * (u2x - u0x);
            float uy = u0y + b1 * (u1y - u0y) + b2 * (u2y - u0y);
            uint32_t ti = (texBase - 1) * 4;
            alb *= bilinear(c, __ldg(c.s.tex_info + ti), __ldg(c.s.tex_info + ti + 1), __ldg(c.s.tex_info + ti + 2),
                               ux, uy);
        }
    }
    size_t pixel = (size_t)y * w + x;
    albedo[albedo_stride * pixel] = alb.x;
    albedo[albedo_stride * pixel + 1] = alb.y;
    albedo[albedo_stride * pixel + 2] = alb.z;
    depths[depth_stride * pixel] = depth;
    object_ids[pixel] = id;
    material_ids[pixel] = matId;
}

// World direction of coverage sample k (of 4 x 4) of pixel (x, y), as its ray is traced.
__device__ __forceinline__ V3 sampleDir(const CameraRecord& cam, uint32_t x, uint32_t y, uint32_t k, uint32_t w, uint32_t h,
                                        float t, float aspect)
{
    V3 sdir;
    pixelDir(cam, (float)x + ((float)(k % 4) + 0.5f) / 4.0f, (float)y + ((float)(k / 4) + 0.5f) / 4.0f, w, h, t, aspect,
             sdir);
    return normalize(sdir);
}

// How a triangle covers the samples of a pixel, whose shears lie in a box (centre m, half size h): the edge
// functions of the watertight test are linear in the shear, so over the box each stays within its centre value
// +- r, r with an allowance for both computations' rounding (2^-19 of the terms' magnitudes). COVER_NONE: one is
// surely positive and another surely negative. COVER_ALL: all are surely of one sign, and every vertex is in
// front of the origin, so the distance is positive. COVER_SOME: to be tested sample by sample.
enum Cover { COVER_NONE, COVER_ALL, COVER_SOME };

__device__ __forceinline__ Cover cover_box(const vgt::TriRel& v, float mx, float my, float hx, float hy, float sz_lo, float sz_hi)
{
    float ex = fabsf(mx) + hx, ey = fabsf(my) + hy;
    float pa = fmaf(ex, fabsf(v.az), fabsf(v.ax)), qa = fmaf(ey, fabsf(v.az), fabsf(v.ay));
    float pb = fmaf(ex, fabsf(v.bz), fabsf(v.bx)), qb = fmaf(ey, fabsf(v.bz), fabsf(v.by));
    float pc = fmaf(ex, fabsf(v.cz), fabsf(v.cx)), qc = fmaf(ey, fabsf(v.cz), fabsf(v.cy));
    auto edge = [&](float px, float py, float pz, float qx, float qy, float qz, float mag, float& lo, float& hi) {
        // (p - s pz) x (q - s qz) = p x q + sx (py qz - pz qy) + sy (pz qx - px qz)
        float gx = fmaf(py, qz, -(pz * qy)), gy = fmaf(pz, qx, -(px * qz));
        float at = fmaf(mx, gx, fmaf(my, gy, fmaf(px, qy, -(py * qx))));
        float r = fmaf(hx, fabsf(gx), fmaf(hy, fabsf(gy), 1.9073486e-6f * mag));
        lo = at - r;
        hi = at + r;
    };
    float ulo, uhi, vlo, vhi, wlo, whi;
    edge(v.cx, v.cy, v.cz, v.bx, v.by, v.bz, fmaf(pc, qb, qc * pb), ulo, uhi);
    edge(v.ax, v.ay, v.az, v.cx, v.cy, v.cz, fmaf(pa, qc, qa * pc), vlo, vhi);
    edge(v.bx, v.by, v.bz, v.ax, v.ay, v.az, fmaf(pb, qa, qb * pa), wlo, whi);
    bool pos = ulo > 0.0f || vlo > 0.0f || wlo > 0.0f, neg = uhi < 0.0f || vhi < 0.0f || whi < 0.0f;
    if (pos && neg)
        return COVER_NONE;
    // (1e-30: far above where their products with a distance could vanish.)
    bool all = (ulo > 1.0e-30f && vlo > 1.0e-30f && wlo > 1.0e-30f) || (uhi < -1.0e-30f && vhi < -1.0e-30f && whi < -1.0e-30f);
    // Distances of the vertices along the ray, at the ends of the samples' scales.
    float near = fminf(fminf(fminf(v.az * sz_lo, v.az * sz_hi), fminf(v.bz * sz_lo, v.bz * sz_hi)), fminf(v.cz * sz_lo, v.cz * sz_hi));
    float far = fmaxf(fmaxf(fmaxf(v.az * sz_lo, v.az * sz_hi), fmaxf(v.bz * sz_lo, v.bz * sz_hi)), fmaxf(v.cz * sz_lo, v.cz * sz_hi));
    return all && near > 1.0e-6f && far < 1.0e20f ? COVER_ALL : COVER_SOME;
}

// aov.slang:150-181: the coverage of 16 stratified rays followed through translucent surfaces.
static __global__ void __launch_bounds__(128) aov_coverage_layers(const __grid_constant__ Ctx c, CameraRecord cam,
                                                                  float* coverage)
{
    uint32_t w = (uint32_t)cam.v[0], h = (uint32_t)cam.v[1];
    uint32_t x = blockIdx.x * 16 + (threadIdx.x & 15u), y = blockIdx.y * 8 + (threadIdx.x >> 4);
    if (x >= w || y >= h)
        return;
    V3 org = v3(cam.v[7], cam.v[11], cam.v[15]);
    float cover = 0.0f;
    for (uint32_t k = 0; k < 16; k++) {
        V3 so = org;
        V3 sd = sampleDir(cam, x, y, k, w, h, cam.v[2], cam.v[0] / cam.v[1]);
        float seen = 0.0f, through = 1.0f;
        for (uint32_t layer = 0; layer < 8 && through > 0.0f; layer++) {
            vgt::TraceHit q = vgt::trace_bvh<false>(c.s.nodes, c.s.tris, so, sd, 1.0e30f, c.err);
            if (!q.hit)
                break;
            float op = opacityAt(c, q.inst, q.prim, q.b1, q.b2);
            seen += through * op;
            through *= 1.0f - op;
            so = so + sd * (q.t + 1.0e-4f);
        }
        cover += seen;
    }
    coverage[(size_t)y * w + x] = cover / 16.0f;
}

// The same where every surface is solid (DeviceScene::solid: a sample counts 1 if its ray hits anything):
// one walk of the tree per pixel. Its box test takes all of the pixel's 16 rays as one beam: they share
// their origin, and in each axis the near plane is divided by the largest and the far plane by the
// smallest of their direction components, so a box that any of them meets is visited (a superset of what
// each ray's own walk visits, and a hit of any triangle is what each ray's walk looks for: the counts
// are the same). A triangle found is classified against the samples' box first (cover_box); one that covers
// some of it is tested against the samples still open, by the rays' own test. The walk ends when all 16 are
// covered. Lanes go on to their next leaf before the warp tests triangles. Bound by issue: where the pixel is
// no larger than a few triangles, 16 walks of some 13 nodes become one of about 15.
//
// Where it is larger the beam meets every box in the pixel, and the warp waits for its worst one. So a walk that
// has cost COVER_WORK (node visits, and COVER_SOME_WORK for each triangle tested sample by sample) is given up, and
// the pixel goes to `rest` with its open samples, as does one whose directions change sign in an axis (a line or two of
// pixels): aov_coverage_rest traces those rays one by one. A block is a tile of 16 x 8 pixels, the launch's from
// first_tile on, row by row of tiles.
// Whole calls in us with COVER_WORK 16 / 64 / 256 (COVER_SOME_WORK 4, at 16: 2), and with 16 closest-hit walks a pixel and
// no beam: the 1M-triangle scene at 16x16 336 / 502 / 1004, 818; 64x48 386 / 572 / 1044, 1021; 641x359 884 / 852 / 1027,
// 3194; 1920x1080 3627 / 2680 / 2632, 19,673; the 110k-triangle scene at 16x16 300 / 433 / 783, 680; 1920x1080 1762 / 1614 /
// 1576, 18,033. Without a bound the 1M scene took 35.3 ms at 16x16 and 7.3 at 64x48.
constexpr uint32_t COVER_WORK = 64, COVER_SOME_WORK = 4;
constexpr uint32_t COVER_TILES = 1u << 16; // most tiles of one launch: at most 2^23 pixels and 2^27 rays in `rest`

// A pixel of the launch (the tile's number in it x 128 + the thread) and its samples still open.
struct CoverRest {
    uint2* pixels;
    uint32_t* count;
    uint32_t* fetch;
};

// Pixel of thread `tid` of tile `tile`: a warp's are 4 x 8.
static __device__ __forceinline__ void coverPixel(uint32_t w, uint32_t tile, uint32_t tid, uint32_t& x, uint32_t& y)
{
    uint32_t tiles_x = (w + 15u) / 16u;
    x = tile % tiles_x * 16 + (tid >> 5) * 4 + (tid & 3u);
    y = tile / tiles_x * 8 + ((tid >> 2) & 7u);
}

static __global__ void __launch_bounds__(128, 6) aov_coverage_solid(const __grid_constant__ Ctx c, CameraRecord cam,
                                                                    float* coverage, uint32_t first_tile, CoverRest rest)
{
    __shared__ float4 rays[16][128]; // shear x, y, z and the axis permutation of each thread's samples
    uint32_t tid = threadIdx.x;
    uint32_t w = (uint32_t)cam.v[0], h = (uint32_t)cam.v[1], x, y;
    coverPixel(w, first_tile + blockIdx.x, tid, x, y);
    bool inside = x < w && y < h, open = inside;
    uint32_t covered = 0;
    float t = cam.v[2], aspect = cam.v[0] / cam.v[1];
    V3 org = v3(cam.v[7], cam.v[11], cam.v[15]);
    V3 lo = v3(3.0e38f), hi = v3(-3.0e38f);
    float us[4], vs[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; k++) {
        us[k] = planeU(cam, (float)x + ((float)k + 0.5f) / 4.0f, w, t, aspect);
        vs[k] = planeV(cam, (float)y + ((float)k + 0.5f) / 4.0f, h, t);
    }
    // The samples' shears, their box, and the axis permutation when all have the same.
    V3 slo = v3(3.0e38f), shi = v3(-3.0e38f);
    int kx = 0, ky = 0, kz = 0;
    bool same = inside;
#pragma unroll
    for (uint32_t k = 0; k < 16; k++) {
        V3 d;
        planeDir(cam, us[k % 4], vs[k / 4], d);
        d = normalize(d);
        vgt::TRay r = vgt::make_ray(org, d);
        rays[k][tid] = make_float4(r.sx, r.sy, r.sz, 0.0f);
        if (k == 0)
            kx = r.kx, ky = r.ky, kz = r.kz;
        same = same && kx == r.kx && ky == r.ky && kz == r.kz;
        slo = v3(fminf(slo.x, r.sx), fminf(slo.y, r.sy), fminf(slo.z, r.sz));
        shi = v3(fmaxf(shi.x, r.sx), fmaxf(shi.y, r.sy), fmaxf(shi.z, r.sz));
        lo = v3(fminf(lo.x, d.x), fminf(lo.y, d.y), fminf(lo.z, d.z));
        hi = v3(fmaxf(hi.x, d.x), fmaxf(hi.y, d.y), fmaxf(hi.z, d.z));
        if (bad3(d))
            lo = v3(-3.0e38f); // no beam
    }
    auto one_sign = [](float a, float b) { return a > bvh8::MIN_DIR || (b < -bvh8::MIN_DIR && a > -2.0f); };
    if (same && one_sign(lo.x, hi.x) && one_sign(lo.y, hi.y) && one_sign(lo.z, hi.z)) {
        float mx = 0.5f * (slo.x + shi.x), my = 0.5f * (slo.y + shi.y);
        float hx = 1.000001f * (0.5f * (shi.x - slo.x)) + 1.0e-6f * fabsf(mx);
        float hy = 1.000001f * (0.5f * (shi.y - slo.y)) + 1.0e-6f * fabsf(my);
        // Positive components: near / hi, far / lo; negative ones: near / lo, far / hi.
        vgt::Slabs b;
        b.o = org;
        b.nx = 1.0f / (lo.x > 0.0f ? hi.x : lo.x), b.fx = 1.0f / (lo.x > 0.0f ? lo.x : hi.x);
        b.ny = 1.0f / (lo.y > 0.0f ? hi.y : lo.y), b.fy = 1.0f / (lo.y > 0.0f ? lo.y : hi.y);
        b.nz = 1.0f / (lo.z > 0.0f ? hi.z : lo.z), b.fz = 1.0f / (lo.z > 0.0f ? lo.z : hi.z);
        b.oct = (lo.x < 0.0f ? 1u : 0u) | (lo.y < 0.0f ? 2u : 0u) | (lo.z < 0.0f ? 4u : 0u);
        uint2 stack[bvh8::STACK_SIZE];
        vgt::Walk k;
        k.r.oct = b.oct;
        k.tmax = 1.0e30f;
        k.node = 0;
        k.sp = 0;
        k.nodes = 0;
        uint32_t work = 0;
        bool done = false;
        while (!done && covered != 0xffffu && work < COVER_WORK) {
            do {
                vgt::node_visit(c.s.nodes, k, b);
                work++;
                done = vgt::next_node(k, stack, c.err);
            } while (!done && k.tri_bits == 0 && work < COVER_WORK);
            while (k.tri_bits && covered != 0xffffu) {
                uint32_t j = vgt::high_bit(k.tri_bits);
                k.tri_bits ^= 1u << j;
                const float4* tp = c.s.tris + (size_t)(k.tri_base + j) * bvh8::TRI_VEC4;
                float4 p0 = __ldg(tp), p1 = __ldg(tp + 1), p2 = __ldg(tp + 2);
                vgt::TriRel v = vgt::tri_relative(org, kx, ky, kz, v3(p0.x, p0.y, p0.z), v3(p1.x, p1.y, p1.z), v3(p2.x, p2.y, p2.z));
                Cover cv = cover_box(v, mx, my, hx, hy, slo.z, shi.z);
                if (cv == COVER_ALL)
                    covered = 0xffffu;
                if (cv == COVER_SOME) {
                    work += COVER_SOME_WORK;
                    for (uint32_t left = covered ^ 0xffffu; left; left &= left - 1) {
                        uint32_t i = (uint32_t)__ffs((int)left) - 1u;
                        float4 q = rays[i][tid];
                        float th, U, V, W, det;
                        if (vgt::tri_test(v, q.x, q.y, q.z, th, U, V, W, det) && th < 1.0e30f)
                            covered |= 1u << i;
                    }
                }
            }
        }
        open = !done && covered != 0xffffu;
    }
    if (inside)
        coverage[(size_t)y * w + x] = (float)__popc(covered) / 16.0f;
    __syncwarp();
    uint32_t b = __ballot_sync(vgk::FULL, open), base = 0, lane = tid & 31u;
    if (b == 0)
        return;
    if (lane == 0)
        base = atomicAdd(rest.count, __popc(b));
    base = __shfl_sync(vgk::FULL, base, 0);
    if (open)
        rest.pixels[base + __popc(b & ((1u << lane) - 1u))] = make_uint2(blockIdx.x * 128 + tid, covered ^ 0xffffu);
}

// The rays that aov_coverage_solid left, any hit with dynamic fetch: an image of few pixels fills the chip with them
// too. A hit adds its sixteenth, exactly and in any order.
static __global__ void __launch_bounds__(128, VG_TRACE_MIN_BLOCKS) aov_coverage_rest(const __grid_constant__ Ctx c, CameraRecord cam,
                                                                                    float* coverage, uint32_t first_tile,
                                                                                    CoverRest rest)
{
    uint32_t w = (uint32_t)cam.v[0], h = (uint32_t)cam.v[1];
    auto pixel = [&](uint32_t i, uint32_t& x, uint32_t& y) {
        uint2 e = rest.pixels[i >> 4];
        coverPixel(w, first_tile + (e.x >> 7), e.x & 127u, x, y);
        return ((e.y >> (i & 15u)) & 1u) != 0;
    };
    vgk::trace_queue_any<vgt::HITS_ANY, false>(
        c, rest.fetch, *rest.count * 16u, vgk::TRACE_REFILL, vgk::TRACE_STEPS,
        [&](uint32_t i, V3& o, V3& d, float& tmax, bool&) {
            uint32_t x, y;
            o = v3(cam.v[7], cam.v[11], cam.v[15]);
            tmax = 1.0e30f;
            if (!pixel(i, x, y))
                return false;
            d = sampleDir(cam, x, y, i & 15u, w, h, cam.v[2], cam.v[0] / cam.v[1]);
            return true;
        },
        [&](uint32_t i, const vgt::TraceHit& q) {
            uint32_t x, y;
            if (q.hit && pixel(i, x, y))
                atomicAdd(coverage + (size_t)y * w + x, 0.0625f);
        });
}

} // namespace vga
