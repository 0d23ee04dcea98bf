// Device-side traversal of the 8-wide quantized BVH (bvh8.cpp), shared by the ray-cast
// entry points (cast.cu) and the path tracer's extend / shadow kernels (render.cu).
//
// Traversal follows the compressed-wide-BVH scheme of Ylitie, Karras and Laine (HPG 2017):
// a node group (child base, hit bits) and a triangle group (triangle base, hit bits) per
// lane, a per-lane stack of pending node groups, children visited in the ray-octant order
// fixed at build time.  A warp steps together (warp_step): each lane tests one pending triangle,
// if it has any, then, if none is left, the next node (8 child boxes).
//
// The triangle test is the reference's Möller-Trumbore (triangle_primitive_mt.inl:100-131)
// with its operation order: cross products as in simd.inl:173-187 (AVX2 path: one product
// rounded, one fused), dot products as in simd.inl:165-171 ((x + y) + z), and an IEEE
// reciprocal of the determinant in place of the reference's rcpss + Newton step
// (scalar.inl:67-71).  Every operation is an explicit _rn intrinsic so that nvcc does not
// contract them; results are bit-identical to the CPU restatement in oracle/.
//
// A triangle is hit when the test passes with min_t <= t <= max_t and the hit point
// o + t * d (one FMA per axis) lies within the triangle's bounds widened by the tree's hit
// margin (2^-17 of the scene size).  The second condition never rejects a genuine hit; it
// rejects the rounding noise the test returns for zero-area triangles, whose "hits" can lie
// anywhere along the ray.  Closest hit keeps, among all hit triangles, the one with the
// smallest t, ties going to the smaller triangle index: the answer does not depend on tree
// shape or traversal order.
#pragma once

#include <cstdint>

#include "bvh8.hpp"

namespace spb::gpu {

constexpr uint32_t Stack_size = Max_wide_depth;
constexpr uint32_t Miss       = 0xFFFFFFFFu;

struct Ray_state {
    float    ox, oy, oz;
    float    dx, dy, dz;
    float    ix, iy, iz;
    float    tmin, tbest;
    float    u, v;
    uint32_t best_id;
    uint32_t oct_inv;
};

// Reciprocal of a direction component for the slab test; components below 2^-80 in
// magnitude are replaced by +-2^-80 so that every slab distance stays finite.
__device__ __forceinline__ float safe_rcp(float d) {
    float const tiny = 8.27180613e-25f;  // 2^-80
    float const m    = fabsf(d) < tiny ? copysignf(tiny, d) : d;
    return __frcp_rn(m);
}

__device__ __forceinline__ float dot3(float ax, float ay, float az, float bx, float by,
                                      float bz) {
    return __fadd_rn(__fadd_rn(__fmul_rn(ax, bx), __fmul_rn(ay, by)), __fmul_rn(az, bz));
}

// cross(a, b) with the reference's AVX2 operation order (simd.inl:173-187).
__device__ __forceinline__ void cross3(float ax, float ay, float az, float bx, float by,
                                       float bz, float& rx, float& ry, float& rz) {
    rx = __fmaf_rn(bz, ay, -__fmul_rn(az, by));
    ry = __fmaf_rn(bx, az, -__fmul_rn(ax, bz));
    rz = __fmaf_rn(by, ax, -__fmul_rn(ay, bx));
}

// Möller-Trumbore with inclusive bounds (triangle_primitive_mt.inl:100-131).
__device__ __forceinline__ bool triangle_test(Ray_state const& r, float4 a, float4 e1, float4 e2,
                                              float tmax, float& t, float& u, float& v) {
    float const tx = __fsub_rn(r.ox, a.x);
    float const ty = __fsub_rn(r.oy, a.y);
    float const tz = __fsub_rn(r.oz, a.z);

    float px, py, pz;
    cross3(r.dx, r.dy, r.dz, e2.x, e2.y, e2.z, px, py, pz);
    float qx, qy, qz;
    cross3(tx, ty, tz, e1.x, e1.y, e1.z, qx, qy, qz);

    float const det = dot3(e1.x, e1.y, e1.z, px, py, pz);
    float const tvp = dot3(tx, ty, tz, px, py, pz);
    float const dqv = dot3(r.dx, r.dy, r.dz, qx, qy, qz);
    float const eqv = dot3(e2.x, e2.y, e2.z, qx, qy, qz);

    float const inv = __frcp_rn(det);

    u        = __fmul_rn(tvp, inv);
    v        = __fmul_rn(dqv, inv);
    t        = __fmul_rn(eqv, inv);
    float uv = __fadd_rn(u, v);

    return (u >= 0.f) & (u <= 1.f) & (v >= 0.f) & (uv <= 1.f) & (t >= r.tmin) & (t <= tmax);
}

// The hit point o + t * d lies within the triangle's bounds widened by margin.
__device__ __forceinline__ bool within_bounds(Ray_state const& r, float4 a, float4 e1, float4 e2,
                                              float t, float margin) {
    float const p[3]  = {__fmaf_rn(t, r.dx, r.ox), __fmaf_rn(t, r.dy, r.oy),
                         __fmaf_rn(t, r.dz, r.oz)};
    float const va[3] = {a.x, a.y, a.z};
    float const vb[3] = {__fadd_rn(a.x, e1.x), __fadd_rn(a.y, e1.y), __fadd_rn(a.z, e1.z)};
    float const vc[3] = {__fadd_rn(a.x, e2.x), __fadd_rn(a.y, e2.y), __fadd_rn(a.z, e2.z)};
    bool inside = true;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float const lo = __fsub_rn(fminf(va[k], fminf(vb[k], vc[k])), margin);
        float const hi = __fadd_rn(fmaxf(va[k], fmaxf(vb[k], vc[k])), margin);
        inside &= (p[k] >= lo) & (p[k] <= hi);
    }
    return inside;
}

// Per-lane traversal state kept in registers; the node-group stack itself is a separate
// array (local memory), so that dynamic indexing into it does not pull these scalars out of
// registers.
struct Traversal {
    uint2    group;      // node group: child base, internal-child hit bits << 24 | imask
    uint2    tri_group;  // triangle group: triangle base, triangle hit bits
    uint32_t tri_valid;  // the triangles its node has (Wide_node::tri_valid)
    uint32_t sp;
};

// Two FP32 FMAs in one instruction (sm_100a): the same roundings as two __fmaf_rn.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{.reg .b64 a, b, c, d;\n\t"
        "mov.b64 a, {%2, %3};\n\t"
        "mov.b64 b, {%4, %5};\n\t"
        "mov.b64 c, {%6, %7};\n\t"
        "fma.rn.f32x2 d, a, b, c;\n\t"
        "mov.b64 {%0, %1}, d;}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("{.reg .b64 a, b, d;\n\t"
        "mov.b64 a, {%2, %3};\n\t"
        "mov.b64 b, {%4, %5};\n\t"
        "add.rn.f32x2 d, a, b;\n\t"
        "mov.b64 {%0, %1}, d;}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// 32 bytes in one load (sm_100a).
struct Load32 {
    uint32_t w[8];
};
__device__ __forceinline__ Load32 load32(void const* p) {
    Load32 v;
    asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]), "=r"(v.w[4]), "=r"(v.w[5]), "=r"(v.w[6]),
          "=r"(v.w[7])
        : "l"(p));
    return v;
}

// Two bytes of a word as floats, exactly: 2^23 + b, then 2^23 taken off both at once.  The even
// child's byte comes by a byte permutation, the odd child's by a dot product with a unit vector:
// the walk is bound by the ALU pipe, and the dot product runs on another (all permutations 6 %
// slower on incoherent rays, a quarter or three quarters dot products 2-3 %).
__device__ __forceinline__ float2 bounds_pair(uint32_t w, uint32_t perm, uint32_t unit) {
    uint32_t const e = __byte_perm(w, 0x4B000000u, perm);
    uint32_t const o = __dp4a(w, unit, 0x4B000000u);
    return add2(make_float2(__uint_as_float(e), __uint_as_float(o)), make_float2(-8388608.f, -8388608.f));
}

// Bit i of x moved to bit i ^ o (x 8 bits, o 3 bits).
__device__ __forceinline__ uint32_t permute_octant(uint32_t x, uint32_t o) {
    x = (o & 1u) ? ((x & 0x55u) << 1) | ((x >> 1) & 0x55u) : x;
    x = (o & 2u) ? ((x & 0x33u) << 2) | ((x >> 2) & 0x33u) : x;
    x = (o & 4u) ? ((x & 0x0Fu) << 4) | ((x >> 4) & 0x0Fu) : x;
    return x;
}

// Bit i of x (8 bits) to bits 3 i, 3 i + 1 and 3 i + 2.
__device__ __forceinline__ uint32_t spread_leaves(uint32_t x) {
    x = (x * 0x101u) & 0x00F00Fu;
    x = (x * 0x011u) & 0x0C30C3u;
    x = (x * 0x005u) & 0x249249u;
    return x * 7u;
}

// Intersects the ray with the 8 child boxes of a node: sets the lane's group of hit internal
// children (bits 24..31 of group.y permuted by the ray octant, above the node's mask of internal
// children) and its group of hit leaf triangles.
__device__ __forceinline__ void node_test(Ray_state const& r, Wide_node const* __restrict__ node, Traversal& tv) {
    char const* const p = reinterpret_cast<char const*>(node);
    Load32 const      h = load32(p);
    Load32 const      q = load32(p + 32);
    Load32 const      z = load32(p + 64);

    float const ajx = __uint_as_float(h.w[6]) * r.ix;
    float const ajy = __uint_as_float(h.w[7]) * r.iy;
    float const ajz = __uint_as_float(z.w[4]) * r.iz;
    float const ogx = (__uint_as_float(h.w[0]) - r.ox) * r.ix;
    float const ogy = (__uint_as_float(h.w[1]) - r.oy) * r.iy;
    float const ogz = (__uint_as_float(h.w[2]) - r.oz) * r.iz;
    float2 const adjx = make_float2(ajx, ajx), adjy = make_float2(ajy, ajy), adjz = make_float2(ajz, ajz);
    float2 const orgx = make_float2(ogx, ogx), orgy = make_float2(ogy, ogy), orgz = make_float2(ogz, ogz);

    // near and far planes by the direction's signs
    uint32_t const pnx = r.ix < 0.f ? 0x7651u : 0x7650u, pfx = pnx ^ 1u;
    uint32_t const pny = r.iy < 0.f ? 0x7651u : 0x7650u, pfy = pny ^ 1u;
    uint32_t const pnz = r.iz < 0.f ? 0x7651u : 0x7650u, pfz = pnz ^ 1u;
    uint32_t const unx = r.ix < 0.f ? 0x01000000u : 0x00010000u, ufx = unx ^ 0x01010000u;
    uint32_t const uny = r.iy < 0.f ? 0x01000000u : 0x00010000u, ufy = uny ^ 0x01010000u;
    uint32_t const unz = r.iz < 0.f ? 0x01000000u : 0x00010000u, ufz = unz ^ 0x01010000u;

    // The sign of far - near says whether a child is missed, so a far end of -0 (a hit at -0) must
    // not meet a near end of +0: it becomes +0.
    float const tbest = __fadd_rn(r.tbest, 0.f);
    uint32_t    miss  = 0;
#pragma unroll
    for (int k = 3; k >= 0; --k) {
        float2 const tnx = fma2(bounds_pair(q.w[k], pnx, unx), adjx, orgx);
        float2 const tny = fma2(bounds_pair(q.w[4 + k], pny, uny), adjy, orgy);
        float2 const tnz = fma2(bounds_pair(z.w[k], pnz, unz), adjz, orgz);
        float2 const tfx = fma2(bounds_pair(q.w[k], pfx, ufx), adjx, orgx);
        float2 const tfy = fma2(bounds_pair(q.w[4 + k], pfy, ufy), adjy, orgy);
        float2 const tfz = fma2(bounds_pair(z.w[k], pfz, ufz), adjz, orgz);
        float const  tn0 = fmaxf(fmaxf(tnx.x, tny.x), fmaxf(tnz.x, r.tmin));
        float const  tf0 = fminf(fminf(tfx.x, tfy.x), fminf(tfz.x, tbest));
        float const  tn1 = fmaxf(fmaxf(tnx.y, tny.y), fmaxf(tnz.y, r.tmin));
        float const  tf1 = fminf(fminf(tfx.y, tfy.y), fminf(tfz.y, tbest));
        // shifted in: set where the ray misses the child
        miss = __funnelshift_l(__float_as_uint(tf1 - tn1), miss, 1);
        miss = __funnelshift_l(__float_as_uint(tf0 - tn0), miss, 1);
    }
    uint32_t const hit   = ~miss & 0xFFu;
    uint32_t const imask = h.w[3] >> 24;
    tv.group     = make_uint2(h.w[4], (permute_octant(hit & imask, r.oct_inv) << 24) | imask);
    tv.tri_valid = h.w[3] & 0x00FFFFFFu;
    tv.tri_group = make_uint2(h.w[5], spread_leaves(hit) & tv.tri_valid);
}

// Whether the ray's [min_t, max_t] overlaps the box [lo, hi]: a slab test in double precision
// whose reciprocals are the ray's slab reciprocals (start_ray) refined by one Newton step, so
// that rounding cannot reject a ray that passes through the box by more than about 1e-14 of
// its distance to it.  A NaN anywhere makes the test pass (fmin and fmax ignore NaN), leaving
// such rays to the traversal.  Used with the tree's scene box (Wide_bvh::scene_lo/hi), which
// is padded by 128 hit margins: every ray it rejects ends as a miss of the full traversal too.
__device__ __forceinline__ bool enters_box(Ray_state const& r, float3 lo, float3 hi) {
    float const o[3]   = {r.ox, r.oy, r.oz};
    float const d[3]   = {r.dx, r.dy, r.dz};
    float const inv[3] = {r.ix, r.iy, r.iz};
    float const l[3]   = {lo.x, lo.y, lo.z};
    float const h[3]   = {hi.x, hi.y, hi.z};
    double      tn     = r.tmin;
    double      tf     = r.tbest;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float const  tiny = 8.27180613e-25f;  // 2^-80, as safe_rcp
        double const m    = fabsf(d[k]) < tiny ? copysignf(tiny, d[k]) : d[k];
        double       i    = inv[k];
        i                 = i * fma(-m, i, 2.0);
        double const a    = (double(l[k]) - double(o[k])) * i;
        double const b    = (double(h[k]) - double(o[k])) * i;
        tn                = fmax(tn, fmin(a, b));
        tf                = fmin(tf, fmax(a, b));
    }
    return tn <= tf;
}

// Loads one ray (math::ray order: origin, min_t / direction, max_t) and resets the state.
__device__ __forceinline__ void start_ray(Ray_state& r, Traversal& tv, float4 ro, float4 rd) {
    r.ox      = ro.x;
    r.oy      = ro.y;
    r.oz      = ro.z;
    r.tmin    = ro.w;
    r.dx      = rd.x;
    r.dy      = rd.y;
    r.dz      = rd.z;
    r.tbest   = rd.w;
    r.ix      = safe_rcp(rd.x);
    r.iy      = safe_rcp(rd.y);
    r.iz      = safe_rcp(rd.z);
    r.u       = 0.f;
    r.v       = 0.f;
    r.best_id = Miss;
    uint32_t const o = (r.ix < 0.f ? 1u : 0u) | (r.iy < 0.f ? 2u : 0u) | (r.iz < 0.f ? 4u : 0u);
    r.oct_inv        = 7u - o;
    tv.group         = make_uint2(0, 0x80000000u);  // the root, as the only child of a group
    tv.tri_group     = make_uint2(0, 0);
    tv.tri_valid     = 0;
    tv.sp            = 0;
}

// ---- two-level traversal (instancing) ----
// The top-level tree's leaf records are instances (Wide_triangle::id = instance index).  A lane
// reaching one pushes what is left of its top-level traversal (pending node group, then pending
// leaves), transforms its ray into the instance's object space -- the direction by the linear
// part only, not renormalised, so that t is the same parameter in both spaces and min_t,
// the closest hit so far and every hit distance carry over -- and walks the instance's own tree
// from its root.  When that tree is spent (the stack back at the depth where it began), the
// world ray is restored and the top-level traversal resumes.  A stack entry whose top byte is
// zero is a group of pending top-level leaves (node groups are pushed only while they still
// have children to visit, in the top byte).

// What the traversal reads of an instance: its world-to-object map (rows: object_k =
// dot(row_k.xyz, world) + row_k.w), the root node of its tree and that tree's hit margin.
struct Instance_trace {
    float4   w2o[3];
    uint32_t root;
    float    hit_margin;
    uint32_t pad[2];
};
static_assert(sizeof(Instance_trace) == 64, "Instance_trace is 64 bytes");

// A lane's two-level state: the world-space ray, kept while the lane is inside an instance;
// the instance it is in (Miss at the top level); the stack depth at which that instance's tree
// began; the instance of the closest hit so far; the hit margin of the current tree.
struct Instance_state {
    float    wox, woy, woz;
    float    wdx, wdy, wdz;
    uint32_t inst;
    uint32_t base_sp;
    uint32_t best_inst;
    float    margin;
};

__device__ __forceinline__ void start_instances(Ray_state const& r, Instance_state& is) {
    is.wox       = r.ox;
    is.woy       = r.oy;
    is.woz       = r.oz;
    is.wdx       = r.dx;
    is.wdy       = r.dy;
    is.wdz       = r.dz;
    is.inst      = Miss;
    is.base_sp   = 0;
    is.best_inst = Miss;
    is.margin    = 0.f;
}

// The ray's origin and direction replaced (slab reciprocals and octant recomputed).
__device__ __forceinline__ void set_ray(Ray_state& r, float ox, float oy, float oz, float dx,
                                        float dy, float dz) {
    r.ox = ox;
    r.oy = oy;
    r.oz = oz;
    r.dx = dx;
    r.dy = dy;
    r.dz = dz;
    r.ix = safe_rcp(dx);
    r.iy = safe_rcp(dy);
    r.iz = safe_rcp(dz);
    uint32_t const o = (r.ix < 0.f ? 1u : 0u) | (r.iy < 0.f ? 2u : 0u) | (r.iz < 0.f ? 4u : 0u);
    r.oct_inv        = 7u - o;
}

__device__ __forceinline__ bool push_group(uint2* stack, Traversal& tv, uint2 group) {
    if (tv.sp < Stack_size) {
        stack[tv.sp++] = group;
        return true;
    }
    return false;
}

// The pending triangles of a lane's group as a stack entry: bit i for the i-th triangle from its
// base (next_group reads it back with every triangle valid).
__device__ __forceinline__ uint2 pack_leaves(Traversal const& tv) {
    uint32_t packed = 0;
    for (uint32_t rest = tv.tri_group.y; rest != 0; rest &= rest - 1) {
        packed |= 1u << __popc(tv.tri_valid & ((rest & (0u - rest)) - 1u));
    }
    return make_uint2(tv.tri_group.x, packed);
}

// Tests the next pending triangle of the lane's triangle group (which must have one), or, at the
// top level of a two-level tree, enters the next pending instance.  Returns true when the ray is
// finished: any hit found, or the stack guard tripped (overflow counts it; it cannot for trees of
// depth <= Max_wide_depth, nor for two-level trees whose depths add up to at most that), in which
// case the ray ends as a miss instead of writing out of bounds.
// Filter: triangles whose class word (Wide_triangle::tri_class) shares a bit with skip_class
// are ignored (the path tracer skips medium boundaries for shadow rays, and surfaces when it
// walks the boundaries along a shadow ray).
// Instances: two-level traversal (is, instances); the top-level tree's leaves are instances.
template <bool Any_hit, bool Filter = false, bool Instances = false>
__device__ __forceinline__ bool triangle_step(Ray_state& r, Traversal& tv, uint2* stack,
                                              float4 const* __restrict__ triangles,
                                              float hit_margin, uint32_t* overflow,
                                              uint32_t skip_class = 0,
                                              Instance_state* is = nullptr,
                                              Instance_trace const* __restrict__ instances = nullptr) {
    bool           done = false;
    // the triangles are stored in the order of their bits in the node's tri_valid
    uint32_t const below = tv.tri_group.y ^ (tv.tri_group.y - 1);  // the lowest bit and those below it
    uint32_t const k     = __popc(tv.tri_valid & below) - 1;
    tv.tri_group.y &= ~below;
    float4 const* tri   = triangles + 4 * size_t(tv.tri_group.x + k);
    Load32 const  t0    = load32(tri);
    float4 const  a     = make_float4(__uint_as_float(t0.w[0]), __uint_as_float(t0.w[1]), __uint_as_float(t0.w[2]), __uint_as_float(t0.w[3]));
    bool          enter = false;
    if constexpr (Instances) {
        enter = is->inst == Miss;
    }
    if (enter) {
        if constexpr (Instances) {
            // A top-level leaf: keep the rest of the top-level traversal, enter the instance.
            uint32_t const inst = __float_as_uint(a.w);
            bool           ok   = true;
            if (tv.group.y & 0xFF000000u) {
                ok = push_group(stack, tv, tv.group);
            }
            if (ok && tv.tri_group.y != 0) {
                ok = push_group(stack, tv, pack_leaves(tv));
            }
            if (!ok) {
                atomicAdd(overflow, 1u);
                r.best_id = Miss;
                done      = true;
            } else {
                Instance_trace const& it = instances[inst];
                float4 const          m0 = __ldg(&it.w2o[0]);
                float4 const          m1 = __ldg(&it.w2o[1]);
                float4 const          m2 = __ldg(&it.w2o[2]);
                uint32_t const        root = __ldg(&it.root);
                is->margin  = __ldg(&it.hit_margin);
                is->inst    = inst;
                is->base_sp = tv.sp;
                set_ray(r, fmaf(m0.x, is->wox, fmaf(m0.y, is->woy, fmaf(m0.z, is->woz, m0.w))),
                        fmaf(m1.x, is->wox, fmaf(m1.y, is->woy, fmaf(m1.z, is->woz, m1.w))),
                        fmaf(m2.x, is->wox, fmaf(m2.y, is->woy, fmaf(m2.z, is->woz, m2.w))),
                        fmaf(m0.x, is->wdx, fmaf(m0.y, is->wdy, m0.z * is->wdz)),
                        fmaf(m1.x, is->wdx, fmaf(m1.y, is->wdy, m1.z * is->wdz)),
                        fmaf(m2.x, is->wdx, fmaf(m2.y, is->wdy, m2.z * is->wdz)));
                tv.group     = make_uint2(root, 0x80000000u);
                tv.tri_group = make_uint2(0, 0);
            }
        }
    } else {
        float4 const e1 = make_float4(__uint_as_float(t0.w[4]), __uint_as_float(t0.w[5]), __uint_as_float(t0.w[6]), __uint_as_float(t0.w[7]));
        float4 const e2 = __ldg(tri + 2);
        float        t, u, v;
        float        margin = hit_margin;
        if constexpr (Instances) {
            margin = is->margin;
        }
        bool const candidate = !Filter || !(__float_as_uint(e1.w) & skip_class);
        if (candidate && triangle_test(r, a, e1, e2, r.tbest, t, u, v) &&
            within_bounds(r, a, e1, e2, t, margin)) {
            uint32_t const id = __float_as_uint(a.w);
            if (Any_hit) {
                r.best_id = id;
                if constexpr (Instances) {
                    is->best_inst = is->inst;
                }
                done = true;
            } else {
                // t <= the closest t so far; equal distances go to the smaller
                // (instance, triangle) pair.
                bool closer = t < r.tbest;
                if constexpr (Instances) {
                    closer = closer || is->inst < is->best_inst ||
                             (is->inst == is->best_inst && id < r.best_id);
                } else {
                    closer = closer || id < r.best_id;
                }
                if (closer) {
                    r.tbest   = t;
                    r.best_id = id;
                    r.u       = u;
                    r.v       = v;
                    if constexpr (Instances) {
                        is->best_inst = is->inst;
                    }
                }
            }
        }
    }
    return done;
}

// Replaces a spent node group by the next one from the stack (or, at the top level of a
// two-level tree, by a group of pending leaves).  Leaving an instance restores the world ray.
template <bool Instances = false>
__device__ __forceinline__ void next_group(Ray_state& r, Traversal& tv, uint2* stack, Instance_state* is) {
    if (!(tv.group.y & 0xFF000000u)) {
        if constexpr (Instances) {
            if (is->inst != Miss && tv.sp == is->base_sp) {
                // The instance's tree is spent: back to the world ray.
                set_ray(r, is->wox, is->woy, is->woz, is->wdx, is->wdy, is->wdz);
                is->inst = Miss;
            }
        }
        if (tv.sp > 0) {
            uint2 const e = stack[--tv.sp];
            if (Instances && !(e.y & 0xFF000000u)) {
                tv.tri_group = e;
                tv.tri_valid = 0x00FFFFFFu;
            } else {
                tv.group = e;
            }
        }
    }
}

// Visits the next child node of the lane's node group (which must have one).  Returns true when
// the stack guard tripped, as triangle_step does.
__device__ __forceinline__ bool node_step(Ray_state& r, Traversal& tv, uint2* stack,
                                          Wide_node const* __restrict__ nodes, uint32_t* overflow) {
    uint32_t const b = 31u - __clz(tv.group.y & 0xFF000000u);
    tv.group.y &= ~(1u << b);
    uint32_t const slot = (b - 24u) ^ r.oct_inv;
    uint32_t const rel  = __popc(tv.group.y & 0xFFu & ((1u << slot) - 1u));
    uint32_t const node = tv.group.x + rel;
    if (tv.group.y & 0xFF000000u) {
        if (!push_group(stack, tv, tv.group)) {
            atomicAdd(overflow, 1u);
            r.best_id = Miss;
            return true;
        }
    }
    node_test(r, nodes + node, tv);
    return false;
}

// Whether nothing is left to visit.
template <bool Instances = false>
__device__ __forceinline__ bool spent(Traversal const& tv, Instance_state const* is) {
    bool s = tv.tri_group.y == 0 && !(tv.group.y & 0xFF000000u) && tv.sp == 0;
    if constexpr (Instances) {
        s = s && is->inst == Miss;
    }
    return s;
}

// One traversal step of a whole warp (all 32 lanes call it; inactive ones pass active = false and
// only take part in the convergence barriers): every lane tests a pending triangle, if it has
// one, then, if it has none left, visits its next node.  The barriers hold the lanes together at
// the start of each phase.  Returns true for a lane whose ray is finished.
template <bool Any_hit, bool Filter = false, bool Instances = false>
__device__ __forceinline__ bool warp_step(bool active, Ray_state& r, Traversal& tv, uint2* stack,
                                          Wide_node const* __restrict__ nodes,
                                          float4 const* __restrict__ triangles, float hit_margin,
                                          uint32_t* overflow, uint32_t skip_class = 0,
                                          Instance_state* is = nullptr,
                                          Instance_trace const* __restrict__ instances = nullptr) {
    bool done = false;
    if (active && tv.tri_group.y != 0) {
        done = triangle_step<Any_hit, Filter, Instances>(r, tv, stack, triangles, hit_margin, overflow, skip_class,
                                                         is, instances);
    }
    __syncwarp();
    bool const walk = active && !done && tv.tri_group.y == 0;
    if (walk) {
        next_group<Instances>(r, tv, stack, is);
    }
    __syncwarp();
    if (walk && (tv.group.y & 0xFF000000u)) {
        done = node_step(r, tv, stack, nodes, overflow);
    }
    __syncwarp();
    return done || (active && spent<Instances>(tv, is));
}

}  // namespace spb::gpu
