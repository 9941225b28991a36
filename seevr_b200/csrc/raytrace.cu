// raytrace.cu — the path tracer of raytrace.comp (Raytracer.render,
// raytracer.zig:159-200) over the triangle LBVH, writing a headless RGBA32F
// buffer in place of the Vulkan storage image.
//
// Each sample path of raytrace.comp (16 samples per pixel, up to 16
// bounces, Russian roulette after the first, Lambert / metal / glass
// materials, sky colour on a miss; raytrace.comp:37-282) keeps the shader's
// arithmetic, but the work is laid out for the GPU rather than as the
// shader's thread per pixel:
//   - a pre-pass packs the BVH into one 32-byte record per node (bounds and
//     child or leaf words: one sector per visit instead of five scattered
//     loads) and the triangles into 48-byte records in leaf order (v0 and
//     the two edges the intersection test forms, with the triangle index),
//     so a leaf's triangles are one contiguous read;
//   - the binary tree is collapsed into wide nodes of four children (each node's
//     grandchildren, in the shader's visiting order), a 128-byte record per visit:
//     half the dependent fetches of a path to a leaf, and no fetch for the leaf;
//   - a persistent grid of lanes runs sample paths; a lane whose path ends takes
//     the next (pixel, sample) from a warp-aggregated ticket.  A warp's lanes step
//     through their trees together, and those whose ray is done wait until enough
//     do (kShadeLanes) for their hits to be shaded together, so a warp neither
//     waits for its longest ray nor shades one hit at a time;
//   - each path's colour is stored per sample and a resolve pass sums a
//     pixel's 16 samples in sample order, as the shader's loop does.
// Leaves are visited in the shader's order (left pushed before right), every
// expression keeps its evaluation order and the library is built without FMA
// contraction, so the image equals the CPU restatement's bit for bit.  (The
// shader reaches a leaf if every box on its path is hit nearer than the closest
// hit so far.  A child's box lies in its parent's, so by monotone rounding its
// entry is no nearer and its exit no farther, and the closest hit only comes
// nearer: the leaf's own box, tested when its turn comes, decides alone.  Where
// that does not hold, the shader's own traversal of the binary tree runs: for a
// tree whose boxes do not nest or are not finite or that overruns the shader's
// stack (k_rt_check), and for rays with a component of zero or
// NaN.)  Three functions whose GLSL
// precision is implementation-defined are pinned here, and the restatement
// uses the same definitions:
//   - sin/cos of the hemisphere angle: reduction by quadrant (pi/2 split in
//     two parts, Cody and Waite's method) and Maclaurin polynomials on
//     [-pi/4, pi/4] to x^9 / x^10 (truncation below 2e-9);
//   - pow(x, 5.0) in Schlick's Fresnel: ((x*x)*(x*x))*x;
//   - the field-of-view scale tan(30 degrees): computed on the host in
//     double and rounded to float.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>

#include "../../include/seevr.h"
#include "common.cuh"

namespace seevr {
namespace {

constexpr float kPi = 3.14159265f;
constexpr int kMaxBounces = 16;
constexpr int kSamples = 16;

struct RtArgs {
    float* image;
    const float* verts;
    const uint32_t* idx;
    const float* node_min;
    const float* node_max;
    const uint32_t* left;
    const uint32_t* right;
    const uint32_t* count;
    const uint32_t* prim;
    const uint32_t* tri_geom;
    const uint32_t* geom_material;
    const float* albedo;
    const float* roughness;
    const float* metallic;
    const float* emission;
    const float* ior;
    f3 cam_pos, cam_dir, cam_right, cam_up;
    uint32_t width, height, frame, num_tris;
    float fov_scale;
};

// PCG hash (raytrace.comp:43-47)
__device__ __forceinline__ uint32_t pcg(uint32_t seed) {
    const uint32_t state = seed * 747796405u + 2891336453u;
    const uint32_t word = ((state >> ((state >> 28) + 4u)) ^ state) * 277803737u;
    return (word >> 22) ^ word;
}
// rand_f (raytrace.comp:49-51): the literal 4294967295.0 is a float, 2^32
__device__ __forceinline__ float rand_f(uint32_t seed) { return float(pcg(seed)) / 4294967296.0f; }

// sin and cos of x >= 0 (see the header comment)
__device__ __forceinline__ void sincos_pinned(float x, float& s, float& c) {
    const float kHalfPiHi = 1.57079637050628662109375f;       // float(pi/2)
    const float kHalfPiLo = -4.37113900018624283e-8f;          // pi/2 - kHalfPiHi
    const float q = float(int(x * 0.636619772f + 0.5f));      // nearest quadrant
    const float r = (x - q * kHalfPiHi) - q * kHalfPiLo;
    const float r2 = r * r;
    const float sp = r * (1.0f + r2 * (-1.0f / 6.0f + r2 * (1.0f / 120.0f + r2 * (-1.0f / 5040.0f +
                                                                                  r2 * (1.0f / 362880.0f)))));
    const float cp = 1.0f + r2 * (-0.5f + r2 * (1.0f / 24.0f + r2 * (-1.0f / 720.0f +
                                                                    r2 * (1.0f / 40320.0f +
                                                                          r2 * (-1.0f / 3628800.0f)))));
    switch (int(q) & 3) {
        case 0: s = sp; c = cp; break;
        case 1: s = cp; c = -sp; break;
        case 2: s = -sp; c = -cp; break;
        default: s = -cp; c = sp; break;
    }
}

// GLSL built-ins with their specified definitions
__device__ __forceinline__ f3 mix3(f3 x, f3 y, float a) { return add(scale(1.0f - a, x), scale(a, y)); }
__device__ __forceinline__ f3 reflect3(f3 i, f3 n) { return sub(i, scale(2.0f * dot(n, i), n)); }
__device__ __forceinline__ f3 refract3(f3 i, f3 n, float eta) {
    const float d = dot(n, i);
    const float k = 1.0f - eta * eta * (1.0f - d * d);
    if (k < 0.0f) return mk(0.f, 0.f, 0.f);
    return sub(scale(eta, i), scale(eta * d + sqrtf(k), n));
}
__device__ __forceinline__ f3 mul3(f3 a, f3 b) { return f3{a.x * b.x, a.y * b.y, a.z * b.z}; }

// ray_tri (raytrace.comp:55-69): Moller-Trumbore, t > 0.001; the edges
// e1 = v1 - v0 and e2 = v2 - v0 come precomputed from the packed triangle
__device__ __forceinline__ float ray_tri(f3 ro, f3 rd, f3 v0, f3 e1, f3 e2) {
    const f3 h = cross(rd, e2);
    const float a = dot(e1, h);
    if (fabsf(a) < 1e-8f) return -1.0f;
    const float f = 1.0f / a;
    const f3 s = sub(ro, v0);
    const float u = f * dot(s, h);
    if (u < 0.0f || u > 1.0f) return -1.0f;
    const f3 q = cross(s, e1);
    const float v = f * dot(rd, q);
    if (v < 0.0f || u + v > 1.0f) return -1.0f;
    const float t = f * dot(e2, q);
    return t > 0.001f ? t : -1.0f;
}

// ray_aabb (raytrace.comp:73-81) with GLSL min/max
__device__ __forceinline__ bool ray_aabb(f3 ro, f3 inv_d, f3 bmin, f3 bmax, float closest) {
    const f3 t1 = mul3(sub(bmin, ro), inv_d), t2 = mul3(sub(bmax, ro), inv_d);
    const f3 tmin = vmin(t1, t2), tmax = vmax(t1, t2);
    const float enter = gmax(gmax(tmin.x, tmin.y), tmin.z);
    const float exit_ = gmin(gmin(tmax.x, tmax.y), tmax.z);
    return exit_ >= enter && enter < closest && exit_ > 0.0f;
}

// One BVH node: bounds, with the left child (or a leaf's first primitive
// slot) in lo.w and the right child (or 0x80000000 | a leaf's count) in hi.w.
struct NodeP {
    float4 lo, hi;
};
// One triangle in leaf order: v0 with the triangle index, e1, e2.
struct TriP {
    float4 a, b, c;
};
constexpr uint32_t kLeafBit = 0x80000000u;

__global__ void k_rt_pack_nodes(RtArgs g, uint32_t nnodes, NodeP* __restrict__ out) {
    for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < nnodes; n += gridDim.x * blockDim.x) {
        const f3 lo = ld3(g.node_min, n), hi = ld3(g.node_max, n);
        const uint32_t cnt = g.count[n];
        const uint32_t w = cnt > 0 ? (kLeafBit | cnt) : g.right[n];
        out[n].lo = make_float4(lo.x, lo.y, lo.z, __uint_as_float(g.left[n]));
        out[n].hi = make_float4(hi.x, hi.y, hi.z, __uint_as_float(w));
    }
}

__global__ void k_rt_pack_tris(RtArgs g, TriP* __restrict__ out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < g.num_tris; i += gridDim.x * blockDim.x) {
        const uint32_t ti = g.prim[i];
        const f3 v0 = ld3(g.verts, g.idx[size_t(ti) * 3]);
        const f3 v1 = ld3(g.verts, g.idx[size_t(ti) * 3 + 1]);
        const f3 v2 = ld3(g.verts, g.idx[size_t(ti) * 3 + 2]);
        const f3 e1 = sub(v1, v0), e2 = sub(v2, v0);
        out[i].a = make_float4(v0.x, v0.y, v0.z, __uint_as_float(ti));
        out[i].b = make_float4(e1.x, e1.y, e1.z, 0.0f);
        out[i].c = make_float4(e2.x, e2.y, e2.z, 0.0f);
    }
}

// trace (raytrace.comp:85-131) over the packed records: the same visiting
// order (left pushed before right) and stack bound (32 entries, pushes
// guarded by sp < 31)
__device__ void trace(const NodeP* __restrict__ nodes, const TriP* __restrict__ tris, f3 ro, f3 rd,
                      float& closest, f3& normal, uint32_t& hit, bool& front) {
    closest = 1e10f;
    normal = mk(0.f, 1.f, 0.f);
    hit = 0xFFFFFFFFu;
    front = true;
    const f3 inv_d = mk(1.0f / rd.x, 1.0f / rd.y, 1.0f / rd.z);
    uint32_t stack[32];
    stack[0] = 0;
    int sp = 1;
    while (sp > 0) {
        --sp;
        const uint32_t node = stack[sp];
        const float4 lo = __ldg(&nodes[node].lo), hi = __ldg(&nodes[node].hi);
        if (!ray_aabb(ro, inv_d, mk(lo.x, lo.y, lo.z), mk(hi.x, hi.y, hi.z), closest)) continue;
        const uint32_t lf = __float_as_uint(lo.w), wd = __float_as_uint(hi.w);
        if (wd & kLeafBit) {
            const uint32_t cnt = wd & ~kLeafBit;
            for (uint32_t i = 0; i < cnt; ++i) {
                const float4 a = __ldg(&tris[lf + i].a), b = __ldg(&tris[lf + i].b),
                             c = __ldg(&tris[lf + i].c);
                const f3 e1 = mk(b.x, b.y, b.z), e2 = mk(c.x, c.y, c.z);
                const float t = ray_tri(ro, rd, mk(a.x, a.y, a.z), e1, e2);
                if (t > 0.0f && t < closest) {
                    closest = t;
                    const f3 n = normalize(cross(e1, e2));
                    front = dot(n, rd) < 0.0f;
                    normal = front ? n : neg(n);
                    hit = __float_as_uint(a.w);
                }
            }
        } else {
            if (sp < 31) stack[sp++] = lf;
            if (sp < 31) stack[sp++] = wd;
        }
    }
}

// ---- wide nodes ----------------------------------------------------------------
// The four grandchildren of a node in visiting order (the right child's right, the
// right child's left, ...; a leaf child counts as one), bounds by axis.  id: an
// inner node, kLeafBit | the slot of a one-triangle leaf, kMulti | the node of a leaf
// with another count, or kNone.
struct Wide {
    float4 lx, ly, lz, hx, hy, hz;
    uint4 id;
    uint4 pad;
};
static_assert(sizeof(Wide) == 128, "one record, four sectors");
constexpr uint32_t kMulti = 0x40000000u, kNodeMask = 0x3FFFFFFFu;
// The shader's stack holds the left siblings of a path's right turns and drops what
// comes after 31 entries: nothing, if no inner node lies more right turns deep than
constexpr uint32_t kMaxRights = 29;
constexpr uint32_t kMaxDepth = 48;  // of a leaf, by the stack below
constexpr int kWideStack = 3 * (kMaxDepth / 2) + 4;  // three entries a level, four being written

// parent[child] = node (cleared to kNone before); *bad is raised for a tree that is
// not one: a child out of range or with two parents.
__global__ void k_rt_parents(RtArgs g, uint32_t nnodes, uint32_t* __restrict__ parent,
                             uint32_t* __restrict__ bad) {
    for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < nnodes; n += gridDim.x * blockDim.x) {
        if (g.count[n] > 0) continue;
        const uint32_t c[2] = {g.left[n], g.right[n]};
        for (uint32_t q = 0; q < 2; ++q)
            if (c[q] >= nnodes || atomicExch(&parent[c[q]], n) != kNone) *bad = 1u;
    }
}

// Raises *bad unless every node reached has finite bounds inside its parent's and a
// place within the depths above.
__global__ void k_rt_check(RtArgs g, const NodeP* __restrict__ nodes, uint32_t nnodes,
                           const uint32_t* __restrict__ parent, uint32_t* __restrict__ bad) {
    for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < nnodes; n += gridDim.x * blockDim.x) {
        const float4 lo = nodes[n].lo, hi = nodes[n].hi;
        const uint32_t p = parent[n];
        if (p == kNone && n != 0) continue;  // not reached from the root
        // (a difference of equal infinities or with a NaN is NaN)
        const float f = (lo.x - lo.x) + (lo.y - lo.y) + (lo.z - lo.z) + (hi.x - hi.x) +
                        (hi.y - hi.y) + (hi.z - hi.z);
        bool ok = f == 0.0f && g.count[n] < kMulti && (n != 0 || p == kNone);
        if (p != kNone && p < nnodes) {
            const float4 pl = nodes[p].lo, ph = nodes[p].hi;
            ok = ok && pl.x <= lo.x && pl.y <= lo.y && pl.z <= lo.z && ph.x >= hi.x &&
                 ph.y >= hi.y && ph.z >= hi.z;
        }
        if (g.count[n] > 0) {  // a leaf: the way up
            uint32_t depth = 0, rights = 0;
            for (uint32_t q = p, c = kNone; q != kNone && q < nnodes && depth <= kMaxDepth;
                 c = q, q = parent[q]) {
                ++depth;
                rights += c != kNone && g.right[q] == c;  // the edge to an inner node
            }
            ok = ok && depth <= kMaxDepth && rights <= kMaxRights;
        }
        if (!ok) *bad = 1u;
    }
}

__global__ void k_rt_wide(RtArgs g, const NodeP* __restrict__ nodes, uint32_t nnodes,
                          const uint32_t* __restrict__ bad, Wide* __restrict__ out) {
    if (*bad) return;
    for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < nnodes; n += gridDim.x * blockDim.x) {
        if (g.count[n] > 0) continue;
        uint32_t id[4] = {kNone, kNone, kNone, kNone};
        float b[6][4] = {};
        uint32_t at = 0;
        auto put = [&](uint32_t c) {
            const float4 lo = nodes[c].lo, hi = nodes[c].hi;
            const uint32_t cnt = g.count[c];
            id[at] = cnt == 1u ? kLeafBit | __float_as_uint(lo.w) : cnt > 1u ? kMulti | c : c;
            b[0][at] = lo.x; b[1][at] = lo.y; b[2][at] = lo.z;
            b[3][at] = hi.x; b[4][at] = hi.y; b[5][at] = hi.z;
            ++at;
        };
        const uint32_t kids[2] = {g.right[n], g.left[n]};  // right first: it is on top of the stack
        for (uint32_t q = 0; q < 2; ++q) {
            const uint32_t c = kids[q];
            if (g.count[c] > 0) {
                put(c);
            } else {
                put(g.right[c]);
                put(g.left[c]);
            }
        }
        Wide w;
        w.lx = make_float4(b[0][0], b[0][1], b[0][2], b[0][3]);
        w.ly = make_float4(b[1][0], b[1][1], b[1][2], b[1][3]);
        w.lz = make_float4(b[2][0], b[2][1], b[2][2], b[2][3]);
        w.hx = make_float4(b[3][0], b[3][1], b[3][2], b[3][3]);
        w.hy = make_float4(b[4][0], b[4][1], b[4][2], b[4][3]);
        w.hz = make_float4(b[5][0], b[5][1], b[5][2], b[5][3]);
        w.id = make_uint4(id[0], id[1], id[2], id[3]);
        w.pad = make_uint4(0u, 0u, 0u, 0u);
        out[n] = w;
    }
}

// A ray's closest hit so far.
struct Hit {
    float t;
    f3 normal;
    uint32_t tri;
    bool front;
};
__device__ __forceinline__ void hit_triangle(const TriP* __restrict__ tris, uint32_t slot, f3 ro,
                                             f3 rd, Hit& h) {
    const float4 a = __ldg(&tris[slot].a), b = __ldg(&tris[slot].b), c = __ldg(&tris[slot].c);
    const f3 e1 = mk(b.x, b.y, b.z), e2 = mk(c.x, c.y, c.z);
    const float t = ray_tri(ro, rd, mk(a.x, a.y, a.z), e1, e2);
    if (t > 0.0f && t < h.t) {
        h.t = t;
        const f3 n = normalize(cross(e1, e2));
        h.front = dot(n, rd) < 0.0f;
        h.normal = h.front ? n : neg(n);
        h.tri = __float_as_uint(a.w);
    }
}
// ray_aabb's test but for the closest hit; the entry.  (Finite operands: fminf and
// fmaxf give GLSL's min and max but for the sign of a zero.)
__device__ __forceinline__ bool enters(f3 ro, f3 inv, float lx, float ly, float lz, float hx, float hy,
                                       float hz, float& enter) {
    const float ax = (lx - ro.x) * inv.x, bx = (hx - ro.x) * inv.x;
    const float ay = (ly - ro.y) * inv.y, by = (hy - ro.y) * inv.y;
    const float az = (lz - ro.z) * inv.z, bz = (hz - ro.z) * inv.z;
    enter = fmaxf(fmaxf(fminf(ax, bx), fminf(ay, by)), fminf(az, bz));
    const float exit_ = fminf(fminf(fmaxf(ax, bx), fmaxf(ay, by)), fmaxf(az, bz));
    return exit_ >= enter && exit_ > 0.0f;
}

__device__ __forceinline__ f3 sky_color(f3 rd) {  // raytrace.comp:135-138
    const float t = 0.5f * (rd.y + 1.0f);
    return scale(0.8f, mix3(mk(1.f, 1.f, 1.f), mk(0.5f, 0.7f, 1.0f), t));
}

__device__ __forceinline__ f3 sample_hemisphere(f3 n, uint32_t seed1, uint32_t seed2) {  // 142-153
    const float r1 = rand_f(seed1), r2 = rand_f(seed2);
    const float phi = 2.0f * kPi * r1;
    const float cos_t = sqrtf(r2), sin_t = sqrtf(1.0f - r2);
    const f3 up = fabsf(n.y) > 0.99f ? mk(1.f, 0.f, 0.f) : mk(0.f, 1.f, 0.f);
    const f3 tan1 = normalize(cross(up, n));
    const f3 tan2 = cross(n, tan1);
    float sp, cp;
    sincos_pinned(phi, sp, cp);
    return normalize(add(add(scale(cp, scale(sin_t, tan1)), scale(cos_t, n)), scale(sp, scale(sin_t, tan2))));
}

__device__ __forceinline__ float schlick(float cos_theta, float r0) {  // 157-159
    const float x = 1.0f - cos_theta;
    return r0 + (1.0f - r0) * (((x * x) * (x * x)) * x);
}

constexpr uint32_t kRtThreads = 128;
// Triangles from which wide nodes are built and traversed: below, a lane's ray is so
// short that waiting for others costs more than it saves.  Frames of 640x480 with the
// binary / the wide tree: 24 triangles 444 / 569 us, 1,060 613 / 680, 1,584 699 / 675,
// 15,732 1,656 / 1,262.
constexpr uint32_t kWideFrom = 1500;
// Lanes of a warp whose ray is done at which their hits are shaded, and lanes at inner
// nodes up to which a warp goes on to the leaves.  A frame is bound by issue (68% of
// the slots) with few lanes active per instruction (6 of 32 before), so both are
// chosen for full warps: 640x480 over 134,156 triangles 6.0 ms (9.5 ms with the
// binary tree one bounce per step); 7.0 ms with 6 and 4, 7.9 ms with 20 and 0.
constexpr int kShadeLanes = 20;
constexpr int kInnerLanes = 10;

// The camera ray of sample si of pixel (px, py) (raytrace.comp:176-190).
__device__ __forceinline__ void camera_ray(const RtArgs& g, uint32_t px, uint32_t py, uint32_t si,
                                           uint32_t& seed, f3& ro, f3& rd) {
    const float aspect = float(g.width) / float(g.height);
    seed = px + py * g.width + g.frame * g.width * g.height + si * 12345u;
    const float jx = rand_f(seed) - 0.5f;
    const float jy = rand_f(seed + 1u) - 0.5f;
    const float u = (2.0f * (float(px) + 0.5f + jx) / float(g.width) - 1.0f) * aspect * g.fov_scale;
    const float v = -(2.0f * (float(py) + 0.5f + jy) / float(g.height) - 1.0f) * g.fov_scale;
    rd = normalize(add(add(g.cam_dir, scale(u, g.cam_right)), scale(v, g.cam_up)));
    ro = g.cam_pos;
}

// Sample paths (raytrace.comp:192-270).  Item q
// is sample q % 16 of pixel q / 16 (row-major), so a warp's first paths are
// two neighbouring pixels' samples; its colour goes to samples[3q..3q+2].
// Without kWide: a lane traces the binary tree, one bounce per step of the warp.
template <bool kWide>
__global__ void __launch_bounds__(kRtThreads) k_rt_paths(RtArgs g, const NodeP* __restrict__ nodes,
                                                         const Wide* __restrict__ wide,
                                                         const TriP* __restrict__ tris,
                                                         float* __restrict__ samples,
                                                         uint32_t* __restrict__ ticket,
                                                         const uint32_t* __restrict__ bad,
                                                         uint32_t nitems) {
    const uint32_t lane = threadIdx.x & 31u;
    const unsigned full = 0xFFFFFFFFu;
    const bool plain = kWide && *bad != 0u;  // only the shader's own traversal
    enum : uint32_t { kIdle, kTracing, kWaiting };
    uint32_t mode = kIdle;
    bool drained = false;
    uint32_t item = 0, seed = 0, bounce = 0;
    f3 ro = mk(0.f, 0.f, 0.f), rd = ro, inv = ro, throughput = ro, color = ro;
    Hit h{};
    uint2 stack[kWide ? kWideStack : 1];  // node or leaf, bits of its entry
    int sp = 0;
    uint32_t cur = kNone;  // the node or leaf the lane is at
    // Pushes the children of the inner node cur that the ray enters, last to first, so
    // that the first is on top.
    auto visit = [&] {
        const Wide* w = wide + cur;
        const float4 lx = __ldg(&w->lx), ly = __ldg(&w->ly), lz = __ldg(&w->lz), hx = __ldg(&w->hx),
                     hy = __ldg(&w->hy), hz = __ldg(&w->hz);
        const uint4 id = __ldg(&w->id);
        auto push = [&](uint32_t c, float x0, float y0, float z0, float x1, float y1, float z1) {
            float en;
            const bool in = enters(ro, inv, x0, y0, z0, x1, y1, z1, en);
            stack[sp] = make_uint2(c, __float_as_uint(en));  // kept if sp moves on
            sp += (in & (en < h.t) & (c != kNone)) ? 1 : 0;
        };
        push(id.w, lx.w, ly.w, lz.w, hx.w, hy.w, hz.w);
        push(id.z, lx.z, ly.z, lz.z, hx.z, hy.z, hz.z);
        push(id.y, lx.y, ly.y, lz.y, hx.y, hy.y, hz.y);
        push(id.x, lx.x, ly.x, lz.x, hx.x, hy.x, hz.x);
    };
    // Starts the ray (ro, rd).
    auto launch = [&] {
        if constexpr (!kWide) {
            mode = kTracing;
            return;
        }
        h.t = 1e10f;
        h.normal = mk(0.f, 1.f, 0.f);
        h.tri = 0xFFFFFFFFu;
        h.front = true;
        inv = mk(1.0f / rd.x, 1.0f / rd.y, 1.0f / rd.z);
        const float f = (inv.x - inv.x) + (inv.y - inv.y) + (inv.z - inv.z) + (ro.x - ro.x) +
                        (ro.y - ro.y) + (ro.z - ro.z);
        if (plain || f != 0.0f) {
            trace(nodes, tris, ro, rd, h.t, h.normal, h.tri, h.front);
            mode = kWaiting;
        } else {
            cur = 0;
            sp = 0;
            mode = kTracing;
        }
    };
    while (true) {
        if (!drained) {  // idle lanes take the next items
            const unsigned need = __ballot_sync(full, mode == kIdle);
            if (need) {
                const uint32_t leader = __ffs(need) - 1;
                uint32_t base = 0;
                if (lane == leader) base = atomicAdd(ticket, uint32_t(__popc(need)));
                base = __shfl_sync(full, base, leader);
                if (base + __popc(need) >= nitems) drained = true;
                if (mode == kIdle) {
                    const uint32_t q = base + __popc(need & ((1u << lane) - 1u));
                    if (q < nitems) {
                        item = q;
                        const uint32_t pix = q >> 4;
                        camera_ray(g, pix % g.width, pix / g.width, q & 15u, seed, ro, rd);
                        throughput = mk(1.f, 1.f, 1.f);
                        color = mk(0.f, 0.f, 0.f);
                        bounce = 0;
                        launch();
                    }
                }
            }
        }
        // ---- steps of the rays, until enough of them are done ----
        const int busy = __popc(__ballot_sync(full, mode != kIdle));
        if (busy == 0) break;
        if constexpr (!kWide) {
            if (mode == kTracing) {
                trace(nodes, tris, ro, rd, h.t, h.normal, h.tri, h.front);
                mode = kWaiting;
            }
        } else {
            // the nearest entry left on the stack that is still nearer than the hit
            auto pop = [&] {
                cur = kNone;
                while (sp > 0) {
                    const uint2 e = stack[--sp];
                    if (__uint_as_float(e.y) < h.t) {
                        cur = e.x;
                        break;
                    }
                }
                if (cur == kNone) mode = kWaiting;
            };
            while (true) {
                const int tracing = __popc(__ballot_sync(full, mode == kTracing));
                if (tracing == 0 || busy - tracing >= kShadeLanes) break;
                // inner nodes, until few lanes are at one
                while (true) {
                    const bool inner = mode == kTracing && cur < kMulti;
                    if (__popc(__ballot_sync(full, inner)) <= kInnerLanes) break;
                    if (!inner) continue;
                    visit();
                    pop();
                }
                if (mode == kTracing) {
                    if (cur & kLeafBit) {
                        hit_triangle(tris, cur & ~kLeafBit, ro, rd, h);
                    } else if (cur & kMulti) {
                        const NodeP n = nodes[cur & kNodeMask];
                        const uint32_t lf = __float_as_uint(n.lo.w), cnt = __float_as_uint(n.hi.w) & ~kLeafBit;
                        for (uint32_t i = 0; i < cnt; ++i) hit_triangle(tris, lf + i, ro, rd, h);
                    } else {
                        visit();
                    }
                    pop();
                }
            }
        }
        if (mode != kWaiting) continue;

        const float t = h.t;
        const f3 normal = h.normal;
        const uint32_t hit = h.tri;
        const bool front = h.front;
        bool done = false;
        if (t >= 1e9f) {
            color = add(color, mul3(throughput, sky_color(rd)));
            done = true;
        } else {
            const uint32_t mi = g.geom_material[g.tri_geom[hit]];
            const f3 albedo = ld3(g.albedo, mi);
            const float rough = g.roughness[mi], metal = g.metallic[mi], ior = g.ior[mi];
            const f3 emission = ld3(g.emission, mi);
            color = add(color, mul3(throughput, emission));
            if (emission.x + emission.y + emission.z > 0.0f) done = true;
            const f3 hp = add(ro, scale(t, rd));
            if (!done && bounce > 0) {  // Russian roulette
                const float p = gmax(throughput.x, gmax(throughput.y, throughput.z));
                if (rand_f(seed + bounce * 7u) > p) done = true;
                else throughput = mk(throughput.x / p, throughput.y / p, throughput.z / p);
            }
            if (!done) {
                seed = pcg(seed);
                if (ior > 0.0f) {  // glass
                    const float eta = front ? (1.0f / ior) : ior;
                    const float cos_i = fabsf(dot(rd, normal));
                    const float sin2_t = eta * eta * (1.0f - cos_i * cos_i);
                    float r0 = (1.0f - ior) / (1.0f + ior);
                    r0 = r0 * r0;
                    const float fresnel = schlick(cos_i, r0);
                    const bool tir = sin2_t > 1.0f;
                    if (rand_f(seed + 5u) < fresnel || tir) {
                        rd = reflect3(rd, normal);
                        ro = add(hp, scale(0.001f, normal));
                    } else {
                        rd = refract3(rd, normal, eta);
                        ro = sub(hp, scale(0.001f, normal));
                    }
                    throughput = mul3(throughput, albedo);
                } else if (metal > 0.5f) {  // metal
                    const f3 refl = reflect3(rd, normal);
                    const f3 diff = sample_hemisphere(normal, seed, seed + 1u);
                    rd = normalize(mix3(refl, diff, rough * rough));
                    throughput = mul3(throughput, albedo);
                    ro = add(hp, scale(0.001f, normal));
                } else {  // dielectric
                    const f3 refl = reflect3(rd, normal);
                    const f3 diff = sample_hemisphere(normal, seed, seed + 1u);
                    const float cos_theta = gmax(dot(neg(rd), normal), 0.0f);
                    const float fresnel = schlick(cos_theta, 0.04f);
                    if (rand_f(seed + 3u) < fresnel) {
                        rd = normalize(mix3(refl, diff, rough * rough));
                    } else {
                        rd = diff;
                        throughput = mul3(throughput, albedo);
                    }
                    ro = add(hp, scale(0.001f, normal));
                }
                if (++bounce >= uint32_t(kMaxBounces)) done = true;
            }
        }
        if (done) {
            st3(samples, item, color);
            mode = kIdle;
        } else {
            launch();
        }
    }
}

// A pixel's samples summed in sample order and averaged (raytrace.comp:272-281).
__global__ void k_rt_resolve(RtArgs g, const float* __restrict__ samples) {
    const uint32_t npix = g.width * g.height;
    for (uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x; pix < npix; pix += gridDim.x * blockDim.x) {
        f3 pixel = mk(0.f, 0.f, 0.f);
        for (uint32_t si = 0; si < uint32_t(kSamples); ++si) pixel = add(pixel, ld3(samples, pix * 16u + si));
        const float inv = float(kSamples);
        float* o = g.image + size_t(pix) * 4;
        o[0] = pixel.x / inv;
        o[1] = pixel.y / inv;
        o[2] = pixel.z / inv;
        o[3] = 1.0f;
    }
}

// The work arrays come from a memory pool of the library's own per device,
// which keeps freed memory for the next frame (the device's default pool
// returns it to the system at every synchronisation, and mapping it again
// costs milliseconds per frame).
cudaMemPool_t work_pool(int dev) {
    static std::mutex mu;
    static cudaMemPool_t pools[64] = {};
    if (dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (!pools[dev]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t p = nullptr;
        if (cudaMemPoolCreate(&p, &props) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        uint64_t keep = ~uint64_t(0);
        cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
        pools[dev] = p;
    }
    return pools[dev];
}

}  // namespace
}  // namespace seevr

using namespace seevr;

extern "C" {

float seevr_raytrace_fov_scale(void) {
    // tan(30 degrees) as raytrace.comp:172 computes its argument in float
    const float arg = 30.0f * kPi / 180.0f;
    return float(std::tan(double(arg)));
}

seevr_status seevr_raytrace(const seevr_rt_bindings* b, const seevr_rt_params* p, void* stream) {
    if (!b || !p) {
        set_last_error("bindings or params is NULL");
        return SEEVR_ERR_INVALID_ARGUMENT;
    }
    for (int i = 0; i < SEEVR_RT_NUM_BINDINGS; ++i)
        if (!b->ptr[i]) {
            set_last_error("raytrace binding " + std::to_string(i) + " is NULL");
            return SEEVR_ERR_INVALID_ARGUMENT;
        }
    if (p->width == 0 || p->height == 0) return SEEVR_OK;
    if (p->num_triangles == 0) {
        set_last_error("num_triangles is 0: the tree has no root");
        return SEEVR_ERR_INVALID_ARGUMENT;
    }
    RtArgs g;
    g.image = static_cast<float*>(b->ptr[SEEVR_RT_IMAGE]);
    g.verts = static_cast<const float*>(b->ptr[SEEVR_RT_VERTICES]);
    g.idx = static_cast<const uint32_t*>(b->ptr[SEEVR_RT_INDICES]);
    g.node_min = static_cast<const float*>(b->ptr[SEEVR_RT_NODE_MIN]);
    g.node_max = static_cast<const float*>(b->ptr[SEEVR_RT_NODE_MAX]);
    g.left = static_cast<const uint32_t*>(b->ptr[SEEVR_RT_LEFT]);
    g.right = static_cast<const uint32_t*>(b->ptr[SEEVR_RT_RIGHT]);
    g.count = static_cast<const uint32_t*>(b->ptr[SEEVR_RT_COUNT]);
    g.prim = static_cast<const uint32_t*>(b->ptr[SEEVR_RT_PRIM]);
    g.tri_geom = static_cast<const uint32_t*>(b->ptr[SEEVR_RT_TRI_GEOM]);
    g.geom_material = static_cast<const uint32_t*>(b->ptr[SEEVR_RT_GEOM_MATERIAL]);
    g.albedo = static_cast<const float*>(b->ptr[SEEVR_RT_MAT_ALBEDO]);
    g.roughness = static_cast<const float*>(b->ptr[SEEVR_RT_MAT_ROUGHNESS]);
    g.metallic = static_cast<const float*>(b->ptr[SEEVR_RT_MAT_METALLIC]);
    g.emission = static_cast<const float*>(b->ptr[SEEVR_RT_MAT_EMISSION]);
    g.ior = static_cast<const float*>(b->ptr[SEEVR_RT_MAT_IOR]);
    g.cam_pos = f3{p->cam_pos[0], p->cam_pos[1], p->cam_pos[2]};
    g.cam_dir = f3{p->cam_dir[0], p->cam_dir[1], p->cam_dir[2]};
    g.cam_right = f3{p->cam_right[0], p->cam_right[1], p->cam_right[2]};
    g.cam_up = f3{p->cam_up[0], p->cam_up[1], p->cam_up[2]};
    g.width = p->width;
    g.height = p->height;
    g.frame = p->frame_num;
    g.num_tris = p->num_triangles;
    g.fov_scale = seevr_raytrace_fov_scale();
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint64_t npix = uint64_t(p->width) * p->height;
    if (npix * kSamples >= (1ull << 32)) {
        set_last_error("width * height * 16 samples must stay below 2^32");
        return SEEVR_ERR_INVALID_ARGUMENT;
    }
    const uint32_t nitems = uint32_t(npix * kSamples);
    const uint32_t nnodes = 2 * p->num_triangles - 1;
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const bool few = p->num_triangles < kWideFrom;  // the binary tree only
    const auto paths = few ? k_rt_paths<false> : k_rt_paths<true>;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, paths, kRtThreads, 0);
    // work arrays, stream-ordered: wide and binary nodes, triangles, per-sample
    // colours, parents, the path ticket
    const size_t wide_bytes = few ? 0 : size_t(nnodes) * sizeof(Wide), node_bytes = size_t(nnodes) * sizeof(NodeP),
                 tri_bytes = size_t(p->num_triangles) * sizeof(TriP);
    const size_t sample_bytes = (size_t(nitems) * 3 * sizeof(float) + 15) & ~size_t(15);
    const size_t parent_bytes = size_t(nnodes) * sizeof(uint32_t);
    const size_t work_bytes = wide_bytes + node_bytes + tri_bytes + sample_bytes + parent_bytes + 16;
    void* work = nullptr;
    const cudaMemPool_t pool = work_pool(dev);
    cudaError_t e = pool ? cudaMallocFromPoolAsync(&work, work_bytes, pool, st)
                         : cudaMallocAsync(&work, work_bytes, st);
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_last_error(std::string("raytrace work arrays: ") + cudaGetErrorString(e));
        return SEEVR_ERR_OUT_OF_MEMORY;
    }
    char* w = static_cast<char*>(work);
    Wide* wide = reinterpret_cast<Wide*>(w);
    NodeP* nodes = reinterpret_cast<NodeP*>(w + wide_bytes);
    TriP* tris = reinterpret_cast<TriP*>(w + wide_bytes + node_bytes);
    float* samples = reinterpret_cast<float*>(w + wide_bytes + node_bytes + tri_bytes);
    uint32_t* parent = reinterpret_cast<uint32_t*>(w + wide_bytes + node_bytes + tri_bytes + sample_bytes);
    uint32_t* ticket = parent + nnodes;  // and whether the tree is unfit for wide nodes
    uint32_t* bad = ticket + 1;
    const uint32_t cap = uint32_t(std::max(sms, 1)) * 8u;
    const uint32_t nblocks = std::min((nnodes + 255) / 256, cap);
    cudaMemsetAsync(ticket, 0, 2 * sizeof(uint32_t), st);
    k_rt_pack_nodes<<<nblocks, 256, 0, st>>>(g, nnodes, nodes);
    k_rt_pack_tris<<<std::min((p->num_triangles + 255) / 256, cap), 256, 0, st>>>(g, tris);
    if (!few) {
        cudaMemsetAsync(parent, 0xFF, parent_bytes, st);
        k_rt_parents<<<nblocks, 256, 0, st>>>(g, nnodes, parent, bad);
        k_rt_check<<<nblocks, 256, 0, st>>>(g, nodes, nnodes, parent, bad);
        k_rt_wide<<<nblocks, 256, 0, st>>>(g, nodes, nnodes, bad, wide);
    }
    const uint32_t resident = uint32_t(std::max(sms, 1)) * uint32_t(std::max(per_sm, 1));
    const uint32_t blocks = std::min((nitems + kRtThreads - 1) / kRtThreads, resident);
    paths<<<blocks, kRtThreads, 0, st>>>(g, nodes, wide, tris, samples, ticket, bad, nitems);
    k_rt_resolve<<<std::min(uint32_t((npix + 255) / 256), cap), 256, 0, st>>>(g, samples);
    e = cudaGetLastError();
    cudaFreeAsync(work, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        set_last_error(std::string("raytrace: ") + cudaGetErrorString(e));
        return SEEVR_ERR_CUDA;
    }
    return SEEVR_OK;
}

}  // extern "C"
