// Device building blocks shared by the trace and render kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace lmgpu {

constexpr float kInf = 1e10f;  // include/lm/math.h:54
constexpr float kEps = 1e-3f;  // include/lm/math.h:55
constexpr float kPi = 3.14159265358979323846f;

// ---------------------------------------------------------------------------------------------
// fp32 vector math. The `ieee` namespace spells out every multiply and add with the _rn
// intrinsics, which the compiler never contracts into FMA, in glm's operation order; it is used
// wherever results must match the host restatement bit for bit (ray generation, triangle test).
struct f3 { float x, y, z; };
__host__ __device__ inline f3 mk(float x, float y, float z) { return {x, y, z}; }
__device__ inline f3 operator+(f3 a, f3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ inline f3 operator-(f3 a, f3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ inline f3 operator-(f3 a) { return {-a.x, -a.y, -a.z}; }
__device__ inline f3 operator*(f3 a, f3 b) { return {a.x * b.x, a.y * b.y, a.z * b.z}; }
__device__ inline f3 operator*(f3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ inline f3 operator*(float s, f3 a) { return {a.x * s, a.y * s, a.z * s}; }
__device__ inline f3 operator/(f3 a, float s) { return {a.x / s, a.y / s, a.z / s}; }
// Shading math fuses with explicit fmaf (the library is compiled with --fmad=false, so nothing is
// fused implicitly and every kernel inlining these gets the same bits).
__device__ inline float dot(f3 a, f3 b) { return fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x)); }
__device__ inline f3 cross(f3 a, f3 b) {
    return {fmaf(a.y, b.z, -(b.y * a.z)), fmaf(a.z, b.x, -(b.z * a.x)), fmaf(a.x, b.y, -(b.x * a.y))};
}
// a*s + b*t + c*r per component (barycentric interpolation, basis expansion)
__device__ inline f3 mix3(f3 a, float s, f3 b, float t, f3 c, float r) {
    return {fmaf(c.x, r, fmaf(b.x, t, a.x * s)), fmaf(c.y, r, fmaf(b.y, t, a.y * s)), fmaf(c.z, r, fmaf(b.z, t, a.z * s))};
}
__device__ inline f3 normalize(f3 v) { return v * (1.0f / sqrtf(dot(v, v))); }
__device__ inline float length(f3 v) { return sqrtf(dot(v, v)); }
__device__ inline float cmax(f3 v) { return fmaxf(fmaxf(v.x, v.y), v.z); }
__device__ inline bool is_zero(f3 v) { return v.x == 0.f && v.y == 0.f && v.z == 0.f; }

namespace ieee {
__device__ inline float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ inline float add(float a, float b) { return __fadd_rn(a, b); }
__device__ inline float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ inline float div(float a, float b) { return __fdiv_rn(a, b); }
__device__ inline f3 sub3(f3 a, f3 b) { return {sub(a.x, b.x), sub(a.y, b.y), sub(a.z, b.z)}; }
__device__ inline f3 add3(f3 a, f3 b) { return {add(a.x, b.x), add(a.y, b.y), add(a.z, b.z)}; }
__device__ inline f3 scale3(f3 a, float s) { return {mul(a.x, s), mul(a.y, s), mul(a.z, s)}; }
// glm compute_dot: (x*x' + y*y') + z*z'
__device__ inline float dot3(f3 a, f3 b) { return add(add(mul(a.x, b.x), mul(a.y, b.y)), mul(a.z, b.z)); }
// glm cross: (x.y*y.z - y.y*x.z, x.z*y.x - y.z*x.x, x.x*y.y - y.x*x.y)
__device__ inline f3 cross3(f3 x, f3 y) {
    return {sub(mul(x.y, y.z), mul(y.y, x.z)), sub(mul(x.z, y.x), mul(y.z, x.x)), sub(mul(x.x, y.y), mul(y.x, x.y))};
}
// glm normalize: v * inversesqrt(dot(v, v)), inversesqrt(x) = 1 / sqrt(x)
__device__ inline f3 normalize3(f3 v) { return scale3(v, div(1.0f, __fsqrt_rn(dot3(v, v)))); }
}  // namespace ieee

// ---------------------------------------------------------------------------------------------
// Philox4x32-10 (Salmon et al., SC 2011), keyed per path:
//   key = (seed, 0x6c6d6770), counter = (4*vertex + slot/4, path_lo, path_hi, 0)
// Slots of one vertex: 0-7 light sample, 8-11 direction, 12 Russian roulette, 13-14 component.
struct U4 { float v[4]; };
#ifndef LMGPU_PHILOX_UNROLL
#define LMGPU_PHILOX_UNROLL 10
#endif
constexpr int kPhiloxUnroll = LMGPU_PHILOX_UNROLL;  // rounds unrolled per loop trip (code size vs loop overhead)
__device__ inline U4 philox_block(uint32_t seed, uint64_t path, uint32_t block) {
    uint32_t c0 = block, c1 = uint32_t(path), c2 = uint32_t(path >> 32), c3 = 0u;
    uint32_t k0 = seed, k1 = 0x6c6d6770u;
#pragma unroll kPhiloxUnroll
    for (int r = 0; r < 10; r++) {
        const uint32_t lo0 = 0xD2511F53u * c0, hi0 = __umulhi(0xD2511F53u, c0);
        const uint32_t lo1 = 0xCD9E8D57u * c2, hi1 = __umulhi(0xCD9E8D57u, c2);
        const uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
        c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
        k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
    }
    const float s = 1.0f / 16777216.0f;
    return U4{{float(c0 >> 8) * s, float(c1 >> 8) * s, float(c2 >> 8) * s, float(c3 >> 8) * s}};
}

// ---------------------------------------------------------------------------------------------
// 8-wide BVH (layout in bvh_build.h).
struct Bvh8 {
    const uint4* nodes;   // 5 words per node
    const float4* tris;   // 3 words per triangle
    int32_t depth;        // levels; bounds the traversal stack
    uint32_t num_nodes;   // node index bound
    // Two-level trees (instancing): per instance 4 float4, the rows of its local-from-world
    // transform and {root node, first hit index, 0, 0} as bits; null for single-level trees.
    const float4* inst;
    uint32_t max_visits;  // node visits one ray can make; more flag corruption
};

struct TraceHit {
    float t, u, v;
    int32_t id;
};

// Moller-Trumbore exactly as accel_sahbvh.cpp:58-75 in fp32 (IEEE ops, no FMA). Returns true and
// fills t/u/v if accepted in [tl, th].
__device__ inline bool tri_test(f3 o, f3 d, f3 p1, f3 e1, f3 e2, float tl, float th, float& t, float& u, float& v) {
    using ieee::add; using ieee::mul; using ieee::div;
    const f3 p = ieee::cross3(d, e2);
    const f3 tv = ieee::sub3(o, p1);
    const f3 q = ieee::cross3(tv, e1);
    const float det = ieee::dot3(e1, p);
    const float ad = fabsf(det);
    const float s = copysignf(1.0f, det);
    const float uu = mul(ieee::dot3(tv, p), s);
    const float vv = mul(ieee::dot3(d, q), s);
    if (ad < 1e-8f || uu < 0.0f || vv < 0.0f || add(uu, vv) > ad) return false;
    const float tt = div(ieee::dot3(e2, q), det);
    if (tt < tl || th < tt) return false;
    t = tt;
    u = div(uu, ad);
    v = div(vv, ad);
    return true;
}

// Three-input min / max (one instruction each on sm_100 and later; exact, like the two-input
// forms, so the slab test's result does not change).
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float fmin3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Two fp32 FMAs in one instruction (sm_100 and later), each rounded as fmaf rounds it.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ uint64_t pack2(uint32_t a, uint32_t b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ float2 fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    float2 v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(r));
    return v;
}

// Ray traversal of the 8-wide BVH. Closest hit: the smallest t over every triangle whose test
// accepts the ray in [tmin, tmax], ties broken toward the smaller flattened index. Any hit
// (`any_hit`): ends at the first accepted triangle. The per-thread stack of sibling groups
// lives in shared memory: stk[i * stride] for i < bvh.depth. Child boxes carry a margin of one
// quantum and the slab comparison widens by 2^-18 relative, which bounds the rounding of the
// one-FMA slab distances (see Slabs), so no triangle the exact test would accept is culled.
//
// The traversal is a resumable state (Trav) advanced one step at a time, so a persistent kernel
// can interleave rays on a lane (dynamic ray fetch); trace_bvh8 runs one ray to the end. The
// result is the same however the steps of a ray and of different rays are interleaved.
//
// Two-level trees (kTwoLevel): a top-level child whose node carries the instance marker
// (exponent byte 0xFF) stands for one instance. Visiting it saves the world ray, moves the ray
// into the instance's local frame (o' = M^-1 o, d' = M^-1 d, not renormalized, so t keeps its
// meaning and best.t stays valid), records the stack level and continues at the instance's BLAS
// root; hit indices get the instance's first hit index added. When the traversal pops back to
// the recorded level the world ray is restored and the top level resumes. One instancing level,
// as accel::embreeinstanced builds (accel_embree_instanced.cpp:84-230).
struct Trav {
    f3 o, d, inv;
    float tmin;
    uint32_t oct;
    int sp;
    uint32_t node;  // the node to visit next; kNoNode: none is left
    uint32_t nvis, ntri;
    TraceHit best;
    // two-level only (never read, so never allocated, in single-level code)
    f3 wo, wd;
    int inst_sp;
    int32_t id_base;
    // entered leaf triangles still to be tested: of one node, and (single-level trees) of a later one
    uint32_t tri_base, tri_mask, tri_base2, tri_mask2;
};
constexpr uint32_t kNoNode = 0xffffffffu;

// Lanes per ray and rays per warp of the cooperative traversal (see coop_loop), and the lanes of lane
// `lane`'s group.
constexpr int kCoopLanes = 8, kCoopRays = 32 / kCoopLanes;
__device__ __forceinline__ unsigned group_mask(unsigned lane) { return 0xffu << (lane & unsigned(32 - kCoopLanes)); }

__device__ inline void trav_set_ray(Trav& s, f3 o, f3 d) {
    s.o = o;
    s.d = d;
    // Slab reciprocals from a direction whose zero (or tiny) components are replaced by +-1e-20,
    // keeping the sign: every slab distance stays finite (an exact zero would give infinities and
    // then NaN in the one-FMA form, which would disable culling on that axis). The triangle test
    // still uses the true direction.
    const float dxs = fabsf(d.x) > 1e-20f ? d.x : copysignf(1e-20f, d.x);
    const float dys = fabsf(d.y) > 1e-20f ? d.y : copysignf(1e-20f, d.y);
    const float dzs = fabsf(d.z) > 1e-20f ? d.z : copysignf(1e-20f, d.z);
    s.inv = {1.0f / dxs, 1.0f / dys, 1.0f / dzs};
    s.oct = (signbit(d.x) ? 1u : 0u) | (signbit(d.y) ? 2u : 0u) | (signbit(d.z) ? 4u : 0u);
}

__device__ inline void trav_init(Trav& s, f3 o, f3 d, float tmin, float tmax) {
    trav_set_ray(s, o, d);
    // -0 for a zero: the box comparison is the sign of far * kWiden - near, and a hit at t = -0 (a ray
    // that starts on a surface) as the far side against +0 gives -0, a miss of boxes with hits at the
    // same t and a smaller index; against -0 it gives +0.
    s.tmin = -(0.0f - tmin);
    s.best = TraceHit{tmax, 0.f, 0.f, -1};
    s.sp = 0;
    s.node = 0;
    s.nvis = 0;
    s.ntri = 0;
    s.inst_sp = -1;
    s.id_base = 0;
    s.tri_mask = s.tri_mask2 = 0u;
}

// Slab distances of one node for one ray, with one FMA per plane. Plane q of an axis lies at
// p + q*s; with a = s*inv and b = (p - o)*inv, t = q*a + b. The byte is unpacked straight into
// the float X = 2^23 + 256*q (one byte permute), so t = fma(X, a/256, b - 2^15*a): the large
// offset cancels exactly inside the FMA. Error: about 5 ulp relative plus 0.003 quanta absolute;
// the builder leaves one quantum of margin around every child box and the comparison widens the
// far side by 2^-18 relative (kWiden), so the test never culls a box the exact ray enters.
struct Slabs {
    float ax, ay, az, bx, by, bz;
};
constexpr float kWiden = 1.0000038f;
__device__ __forceinline__ Slabs node_slabs(const uint4& w0, const Trav& s) {
    const float ax = __uint_as_float((w0.w & 0xffu) << 23) * s.inv.x;
    const float ay = __uint_as_float(((w0.w >> 8) & 0xffu) << 23) * s.inv.y;
    const float az = __uint_as_float(((w0.w >> 16) & 0xffu) << 23) * s.inv.z;
    const float bx = (__uint_as_float(w0.x) - s.o.x) * s.inv.x;
    const float by = (__uint_as_float(w0.y) - s.o.y) * s.inv.y;
    const float bz = (__uint_as_float(w0.z) - s.o.z) * s.inv.z;
    return Slabs{ax * 0.00390625f, ay * 0.00390625f, az * 0.00390625f,
                 fmaf(-32768.0f, ax, bx), fmaf(-32768.0f, ay, by), fmaf(-32768.0f, az, bz)};
}

// The children of a node whose boxes the ray enters in [tmin, best.t], one bit per slot (plane
// words: qlo x y z, then qhi x y z, two words each).
__device__ __forceinline__ uint32_t node_children(const uint4& w0, const uint4& w2, const uint4& w3, const uint4& w4, const Trav& s) {
    const Slabs S = node_slabs(w0, s);
    const uint64_t ax2 = pack2(S.ax, S.ax), ay2 = pack2(S.ay, S.ay), az2 = pack2(S.az, S.az);
    const uint64_t bx2 = pack2(S.bx, S.bx), by2 = pack2(S.by, S.by), bz2 = pack2(S.bz, S.bz);
    // near/far plane bytes per axis, chosen by the ray's octant
    const bool ox = s.oct & 1u, oy = s.oct & 2u, oz = s.oct & 4u;
    const uint32_t nx0 = ox ? w3.z : w2.x, nx1 = ox ? w3.w : w2.y, fx0 = ox ? w2.x : w3.z, fx1 = ox ? w2.y : w3.w;
    const uint32_t ny0 = oy ? w4.x : w2.z, ny1 = oy ? w4.y : w2.w, fy0 = oy ? w2.z : w4.x, fy1 = oy ? w2.w : w4.y;
    const uint32_t nz0 = oz ? w4.z : w3.x, nz1 = oz ? w4.w : w3.y, fz0 = oz ? w3.x : w4.z, fz1 = oz ? w3.y : w4.w;
    // The trace kernels are bound by instruction issue (70-79 % of the slots, the nodes in L1 and L2),
    // a node's 48 planes being most of it: two slots per instruction (fma.f32x2), and the comparison
    // near <= far * kWiden as the sign of far * kWiden - near shifted into the mask, slot 7 first (zeros:
    // see trav_init)
    // (2^20 diffuse bounces in a soup of 60k triangles: 781 -> 710 us; one FMA per plane 2 % and
    // compares with set bits 3 % slower). Empty slots hold inverted boxes
    // (qlo = 255, qhi = 0) that no ray enters; one accepted through rounding is a leaf of zero
    // triangles.
    uint32_t miss = 0u;
#pragma unroll
    for (int k = 6; k >= 0; k -= 2) {
        const uint32_t s0 = 0x5404u | (uint32_t(k & 3) << 4), s1 = s0 + 0x10u;  // bytes: 00, q, 00, 4B
        auto planes = [&](uint32_t w, uint64_t a, uint64_t b) {
            return fma2(pack2(__byte_perm(w, 0x4B00u, s0), __byte_perm(w, 0x4B00u, s1)), a, b);
        };
        const float2 xn = planes(k < 4 ? nx0 : nx1, ax2, bx2), xf = planes(k < 4 ? fx0 : fx1, ax2, bx2);
        const float2 yn = planes(k < 4 ? ny0 : ny1, ay2, by2), yf = planes(k < 4 ? fy0 : fy1, ay2, by2);
        const float2 zn = planes(k < 4 ? nz0 : nz1, az2, bz2), zf = planes(k < 4 ? fz0 : fz1, az2, bz2);
        const float n0 = fmax3(xn.x, yn.x, fmaxf(zn.x, s.tmin)), n1 = fmax3(xn.y, yn.y, fmaxf(zn.y, s.tmin));
        const float f0 = fmin3(xf.x, yf.x, fminf(zf.x, s.best.t)), f1 = fmin3(xf.y, yf.y, fminf(zf.y, s.best.t));
        miss = __funnelshift_l(__float_as_uint(fmaf(f1, kWiden, -n1)), miss, 1);
        miss = __funnelshift_l(__float_as_uint(fmaf(f0, kWiden, -n0)), miss, 1);
    }
    return ~miss & 0xffu;
}

// The triangles of a leaf child, from its meta byte (the low byte of `meta`): count << 5 | offset.
__device__ __forceinline__ uint32_t leaf_bits(uint32_t meta) {
    uint32_t m;
    asm("bmsk.clamp.b32 %0, %1, %2;" : "=r"(m) : "r"(meta & 31u), "r"((meta >> 5) & 7u));
    return m;
}

// The triangles of the entered leaf children, one bit per triangle after the node's first one.
__device__ __forceinline__ uint32_t leaf_triangles(const uint4& w1, uint32_t leaves) {
    uint32_t tmask = 0u;
    while (leaves) {
        const int k = __ffs(leaves) - 1;
        leaves &= leaves - 1;
        tmask |= leaf_bits(__byte_perm(w1.z, w1.w, uint32_t(k)));
    }
    return tmask;
}

// Tests the first triangle of s.tri_mask. Any hit: true if the ray hits it.
template <bool kAnyHit, bool kCount, bool kTwoLevel>
__device__ __forceinline__ bool trav_test_tri(const Bvh8& bvh, Trav& s) {
    const int j = __ffs(s.tri_mask) - 1;
    s.tri_mask &= s.tri_mask - 1u;
    const float4* tp = bvh.tris + size_t(s.tri_base + uint32_t(j)) * 3;
    const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
    if (kCount) s.ntri++;
    float t, u, v;
    if (tri_test(s.o, s.d, mk(a.x, a.y, a.z), mk(a.w, b.x, b.y), mk(b.z, b.w, c.x), s.tmin, s.best.t, t, u, v)) {
        const int32_t id = (kTwoLevel ? s.id_base : 0) + int32_t(__float_as_uint(c.y));
        if (kAnyHit) {
            s.best = TraceHit{t, u, v, id};
            return true;
        }
        if (t < s.best.t || s.best.id < 0 || id < s.best.id) s.best = TraceHit{t, u, v, id};
    }
    return false;
}

// The instance pseudo-node (w0, w1): the ray continues in the instance's frame at its BLAS root.
__device__ __forceinline__ void trav_enter_instance(const Bvh8& bvh, Trav& s, const uint4& w1) {
    const float4* ip = bvh.inst + size_t(w1.x) * 4;
    const float4 r0 = __ldg(ip), r1 = __ldg(ip + 1), r2 = __ldg(ip + 2);
    const uint4 m = __ldg(reinterpret_cast<const uint4*>(ip + 3));
    s.wo = s.o;
    s.wd = s.d;
    const f3 lo = {r0.x * s.o.x + r0.y * s.o.y + r0.z * s.o.z + r0.w, r1.x * s.o.x + r1.y * s.o.y + r1.z * s.o.z + r1.w,
                   r2.x * s.o.x + r2.y * s.o.y + r2.z * s.o.z + r2.w};
    const f3 ld = {r0.x * s.d.x + r0.y * s.d.y + r0.z * s.d.z, r1.x * s.d.x + r1.y * s.d.y + r1.z * s.d.z,
                   r2.x * s.d.x + r2.y * s.d.y + r2.z * s.d.z};
    trav_set_ray(s, lo, ld);
    s.inst_sp = s.sp;
    s.id_base = int32_t(m.y);
    s.node = m.x;
}

// Chooses s.node: the nearest of the entered inner children `inner` (slots of the node whose
// children start at `base`, with child mask `imask`), else of the sibling group on top of the
// stack, else kNoNode. False on a stack overflow. kGroup: all lanes of a cooperative group call this on
// the same ray and stack column; the first of them stores.
template <bool kTwoLevel, bool kGroup = false>
__device__ __forceinline__ bool trav_next(const Bvh8& bvh, Trav& s, uint32_t base, uint32_t imask, uint32_t inner, uint2* stk,
                                          int stride) {
    const unsigned lane = threadIdx.x & 31u;
    if (inner == 0u) {
        if (kTwoLevel && s.sp == s.inst_sp) {  // the instance is done: back to the world ray
            trav_set_ray(s, s.wo, s.wd);
            s.inst_sp = -1;
            s.id_base = 0;
        }
        if (s.sp == 0) {
            s.node = kNoNode;
            return true;
        }
        s.sp--;
        const uint2 g = stk[s.sp * stride];
        // what is left of the entry goes back to the same place: not before the whole group has read it
        if (kGroup) __syncwarp(group_mask(lane));
        base = g.x;
        imask = g.y >> 8;
        inner = g.y & 0xffu;
    }
    // nearest first by octant order: the slot with the smallest slot ^ octant, as a one-bit mask
    uint32_t first = inner, part = first & ((s.oct & 4u) ? 0xf0u : 0x0fu);
    first = part ? part : first;
    part = first & ((s.oct & 2u) ? 0xccu : 0x33u);
    first = part ? part : first;
    part = first & ((s.oct & 1u) ? 0xaau : 0x55u);
    first = part ? part : first;
    s.node = base + __popc(imask & (first - 1u));
    inner ^= first;
    if (inner != 0u) {
        if (s.sp >= bvh.depth) return false;
        if (!kGroup || lane % kCoopLanes == 0u) stk[s.sp * stride] = make_uint2(base, (imask << 8) | inner);
        s.sp++;
    }
    return true;
}

// Visits s.node (testing the triangles of every leaf child the ray enters) and moves to the next
// node. Returns true when the traversal has ended; s.best is then the result. Sets *err (and
// ends) on a stack overflow (1) or a visit count above the node count (2), which only a corrupt
// BVH can cause.
template <bool kAnyHit, bool kCount, bool kTwoLevel = false>
__device__ __forceinline__ bool trav_step(const Bvh8& bvh, Trav& s, uint2* stk, int stride, int* err) {
    if (s.node >= bvh.num_nodes || s.nvis >= bvh.max_visits) { *err = 2; return true; }
    const uint4* np = bvh.nodes + size_t(s.node) * 5;
    const uint4 w0 = __ldg(np), w1 = __ldg(np + 1);
    s.nvis++;
    if (kTwoLevel && (w0.w & 0xffu) == 0xffu) {
        trav_enter_instance(bvh, s, w1);
        return false;
    }
    const uint4 w2 = __ldg(np + 2), w3 = __ldg(np + 3), w4 = __ldg(np + 4);
    const uint32_t hit = node_children(w0, w2, w3, w4, s), imask = w0.w >> 24;
    s.tri_base = w1.y;
    s.tri_mask = leaf_triangles(w1, hit & ~imask);
    while (s.tri_mask)
        if (trav_test_tri<kAnyHit, kCount, kTwoLevel>(bvh, s)) return true;
    if (!trav_next<kTwoLevel>(bvh, s, w1.x, imask, hit & imask, stk, stride)) { *err = 1; return true; }
    return s.node == kNoNode;
}

// trav_step's node part alone, for single-level trees (after the speculative traversal of Aila & Laine,
// HPG 2009): visits s.node and only records the triangles of the entered leaf children. A ray
// may visit further nodes while one node's triangles wait (not while two nodes' do), so a warp can
// choose the step that most of its lanes can take; a visit before a nearer hit is known may enter
// more nodes, the result is the same. Returns true when no node and no triangle is left.
__device__ __forceinline__ bool trav_node(const Bvh8& bvh, Trav& s, uint2* stk, int stride, int* err) {
    if (s.node >= bvh.num_nodes || s.nvis >= bvh.max_visits) { *err = 2; return true; }
    const uint4* np = bvh.nodes + size_t(s.node) * 5;
    const uint4 w0 = __ldg(np), w1 = __ldg(np + 1), w2 = __ldg(np + 2), w3 = __ldg(np + 3), w4 = __ldg(np + 4);
    s.nvis++;
    const uint32_t hit = node_children(w0, w2, w3, w4, s), imask = w0.w >> 24;
    const uint32_t tmask = leaf_triangles(w1, hit & ~imask);
    if (s.tri_mask) {
        s.tri_base2 = w1.y;
        s.tri_mask2 = tmask;
    } else {
        s.tri_base = w1.y;
        s.tri_mask = tmask;
    }
    if (!trav_next<false>(bvh, s, w1.x, imask, hit & imask, stk, stride)) { *err = 1; return true; }
    return s.node == kNoNode && s.tri_mask == 0u;
}

// One ray to the end. Adds the node visits and triangle tests to *nodes_visited / *tris_tested
// when kCount.
template <bool kAnyHit, bool kCount, bool kTwoLevel = false>
__device__ inline TraceHit trace_bvh8(const Bvh8& bvh, f3 o, f3 d, float tmin, float tmax, uint2* stk, int stride,
                                      uint32_t* nodes_visited, uint32_t* tris_tested, int* err) {
    Trav s;
    trav_init(s, o, d, tmin, tmax);
    while (!trav_step<kAnyHit, kCount, kTwoLevel>(bvh, s, stk, stride, err)) {
    }
    if (kCount) { *nodes_visited += s.nvis; *tris_tested += s.ntri; }
    return s.best;
}

__device__ inline unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Dynamic ray fetch for the persistent trace kernels: `self` hands out queue entries (zero at
// launch). The launch zeroes the counter `reset` (where set) at its start, for a kernel that runs
// after it and that no kernel in flight uses. refill: see Tuning. With `stamp`, the launch writes its
// start and end times there ([0], [1], in ns); `done` counts its finished blocks (zero between
// launches).
struct Fetch {
    int* self;
    int* reset;
    int refill;
    unsigned long long* stamp;
    int* done;
};
__device__ __forceinline__ void trace_begin(const Fetch& f) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    if (f.reset) *f.reset = 0;
    if (f.stamp) f.stamp[0] = globaltimer_ns();
}
// Called by all threads of the block at the launch's end.
__device__ __forceinline__ void trace_end(const Fetch& f) {
    if (!f.stamp) return;
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(f.done, 1) == int(gridDim.x) - 1) {
        *f.done = 0;
        f.stamp[1] = globaltimer_ns();
    }
}

// Cooperative traversal: eight lanes per ray, four rays per warp, for launches and queue ends that
// leave fewer rays than lanes. A lane tests one child box and one triangle, so a visit takes about
// a third of the instructions of a lane that tests all of them, and a node's triangles are tested
// together; what remains is the chain of dependent loads. The box and triangle tests are the
// one-lane steps' and the smallest (t, index) wins as there, so the results are the same. The
// longest rays take 100-200 steps of about 0.6 us, so a launch's last rays cost 100 us and more
// whatever its size: 16k rays into a soup of 60k triangles 114 -> 89 us, 200k 195 -> 179 us, the
// light-traced frame (18 trace launches) 3.68 -> 3.31 ms with the smaller blocks of its kernels.
// Tests the triangles s.tri_mask of each group's ray (same in the group's lanes); any hit: true in
// the lanes of a group whose ray hits one. Called by full warps; groups without a ray: mask 0.
template <bool kAnyHit, bool kTwoLevel>
__device__ __forceinline__ bool coop_tris(const Bvh8& bvh, Trav& s) {
    const unsigned sub = threadIdx.x & (kCoopLanes - 1);
    bool found = false;
    // a node has at most 24 triangles (8 children of at most 3)
#pragma unroll 1
    for (int r = 0; r < 32 && __ballot_sync(0xffffffffu, s.tri_mask != 0u); r += kCoopLanes) {
        float t = INFINITY, u = 0.f, v = 0.f;
        int32_t id = INT32_MAX;
        if ((s.tri_mask >> sub) & 1u) {
            const float4* tp = bvh.tris + size_t(s.tri_base + uint32_t(r) + sub) * 3;
            const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
            float tt, tu, tv;
            if (tri_test(s.o, s.d, mk(a.x, a.y, a.z), mk(a.w, b.x, b.y), mk(b.z, b.w, c.x), s.tmin, s.best.t, tt, tu, tv)) {
                t = tt;
                u = tu;
                v = tv;
                id = (kTwoLevel ? s.id_base : 0) + int32_t(__float_as_uint(c.y));
            }
        }
        s.tri_mask >>= kCoopLanes;
        if (__ballot_sync(0xffffffffu, id != INT32_MAX) == 0u) continue;
#pragma unroll
        for (int o = 1; o < kCoopLanes; o <<= 1) {
            const float ot = __shfl_xor_sync(0xffffffffu, t, o), ou = __shfl_xor_sync(0xffffffffu, u, o);
            const float ov = __shfl_xor_sync(0xffffffffu, v, o);
            const int32_t oi = __shfl_xor_sync(0xffffffffu, id, o);
            if (ot < t || (!(t < ot) && oi < id)) {
                t = ot;
                u = ou;
                v = ov;
                id = oi;
            }
        }
        if (id != INT32_MAX && (kAnyHit || t < s.best.t || s.best.id < 0 || id < s.best.id)) {
            s.best = TraceHit{t, u, v, id};
            if (kAnyHit) {
                found = true;
                s.tri_mask = 0u;
            }
        }
    }
    return found;
}

// Runs the groups' rays to their ends: `live` groups hold entry k in state s (the same in all lanes
// of the group), `stk` is the stack column of the ray. Called by full warps.
template <bool kAnyHit, bool kTwoLevel, typename End>
__device__ __forceinline__ void coop_loop(const Bvh8& bvh, Trav& s, bool live, int k, uint2* stk, int stride, int* lerr, End end) {
    const unsigned sub = threadIdx.x & (kCoopLanes - 1);
    // triangles pending from one-lane steps
    const uint32_t later = live ? s.tri_mask2 : 0u;
    if (!live) s.tri_mask = 0u;
    bool done = coop_tris<kAnyHit, kTwoLevel>(bvh, s);
    if (!kTwoLevel) {
        s.tri_base = s.tri_base2;
        s.tri_mask = done ? 0u : later;
        done = coop_tris<kAnyHit, kTwoLevel>(bvh, s) || done;
    }
    if (live && s.node == kNoNode) done = true;
    while (true) {
        if (live && done) {
            if (sub == 0u) end(k, s);
            live = false;
        }
        __syncwarp();  // stack entries written by one lane are read by its group
        if (__ballot_sync(0xffffffffu, live) == 0u) return;
        done = false;
        uint4 w0 = make_uint4(0u, 0u, 0u, 0u), w1 = w0;
        bool test = false, enter = false;
        if (live) {
            if (s.node >= bvh.num_nodes || s.nvis >= bvh.max_visits) {
                *lerr = 2;
                done = true;
            } else {
                const uint4* np = bvh.nodes + size_t(s.node) * 5;
                w0 = __ldg(np);
                w1 = __ldg(np + 1);
                s.nvis++;
                if (kTwoLevel && (w0.w & 0xffu) == 0xffu) {
                    trav_enter_instance(bvh, s, w1);
                } else {
                    test = true;
                    // this lane's child: its near and far plane bytes (qlo x y z, then qhi x y z)
                    const unsigned char* q = reinterpret_cast<const unsigned char*>(np + 2) + sub;
                    const int ox = (s.oct & 1u) ? 24 : 0, oy = (s.oct & 2u) ? 24 : 0, oz = (s.oct & 4u) ? 24 : 0;
                    auto plane = [&](int at, float a, float b) {
                        return fmaf(__uint_as_float(0x4B000000u | (uint32_t(__ldg(q + at)) << 8)), a, b);
                    };
                    const Slabs S = node_slabs(w0, s);
                    const float n = fmax3(plane(ox, S.ax, S.bx), plane(8 + oy, S.ay, S.by), fmaxf(plane(16 + oz, S.az, S.bz), s.tmin));
                    const float f = fmin3(plane(24 - ox, S.ax, S.bx), plane(32 - oy, S.ay, S.by),
                                          fminf(plane(40 - oz, S.az, S.bz), s.best.t));
                    enter = !signbit(fmaf(f, kWiden, -n));
                }
            }
        }
        const uint32_t hit = (__ballot_sync(0xffffffffu, enter) >> (threadIdx.x & (32 - kCoopLanes))) & 0xffu;
        const uint32_t imask = w0.w >> 24;
        uint32_t tm = ((hit & ~imask) >> sub) & 1u ? leaf_bits(__byte_perm(w1.z, w1.w, sub)) : 0u;
        tm |= __shfl_xor_sync(0xffffffffu, tm, 1);
        tm |= __shfl_xor_sync(0xffffffffu, tm, 2);
        tm |= __shfl_xor_sync(0xffffffffu, tm, 4);
        s.tri_base = w1.y;
        s.tri_mask = tm;
        if (coop_tris<kAnyHit, kTwoLevel>(bvh, s)) done = true;
        if (test && !done) {
            if (!trav_next<kTwoLevel, true>(bvh, s, w1.x, imask, hit & imask, stk, stride)) {
                *lerr = 1;
                done = true;
            }
            if (s.node == kNoNode) done = true;
        }
    }
}

// Persistent traversal with dynamic ray fetch (Aila & Laine, HPG 2009): every lane of a warp
// holds one ray in flight; once fewer than f.refill lanes still trace, the idle lanes take the
// next entries of the queue (one atomic per warp), so a warp no longer waits for its slowest
// ray. begin(k, s) loads entry k into the traversal state; tree(k) is the BVH it traverses;
// end(k, s) consumes the finished traversal. Called by every thread of full warps; `warps`: the
// warps that share the queue.
template <bool kAnyHit, bool kCount, bool kTwoLevel, typename Begin, typename Tree, typename End>
__device__ __forceinline__ void fetch_loop(int n, int warps, const Fetch& f, uint2* stk, int stride, int* lerr, Begin begin,
                                           Tree tree, End end) {
    const int lane = int(threadIdx.x & 31u);
    const unsigned below = (1u << lane) - 1u;
    // fewer rays than lanes: spread them over the warps, at least what a cooperative warp takes
    const int lanes = n >= 32 * warps ? 32 : max(kCoopRays, (n + warps - 1) / warps);
    Trav s;
    s.tri_mask = s.tri_mask2 = 0u;
    Bvh8 B{};
    int k = 0;
    bool active = false, held = false, exhausted = false;  // held: a ray whose end is still to be called
    while (true) {
        if (!exhausted) {
            const unsigned idle = __ballot_sync(0xffffffffu, !active && lane < lanes);
            if (idle) {
                const int leader = __ffs(idle) - 1;
                int base = 0;
                if (lane == leader) base = atomicAdd(f.self, __popc(idle));
                base = __shfl_sync(0xffffffffu, base, leader);
                if (base + __popc(idle) >= n) exhausted = true;  // warp-uniform
                if ((idle >> lane) & 1u) {
                    k = base + __popc(idle & below);
                    if (k < n) {
                        begin(k, s);
                        B = tree(k);
                        active = held = true;
                    }
                }
            }
        }
        unsigned act = __ballot_sync(0xffffffffu, active);
        if (act == 0u) {
            if (exhausted) return;
            continue;
        }
        const int keep = exhausted ? (kCount ? 1 : kCoopRays + 1) : min(f.refill, lanes);
        while (__popc(act) >= keep) {
            bool done = false;
            if constexpr (kTwoLevel || kCount) {
                // two-level trees keep whole-node steps (a triangle must be tested before its instance
                // is left); counted rays visit and test as trace_bvh8 does
                if (active) done = trav_step<kAnyHit, kCount, kTwoLevel>(B, s, stk, stride, lerr);
            } else {
                // A triangle step when at least half as many lanes have a triangle as could visit a node.
                // A lane's ray on a triangle idles a node step's 190 instructions and the reverse 110.
                // 2^20 bounces in a soup of 60k triangles / 16 batched jobs: every lane with a triangle
                // tests it before the next node 684 us / 18.3 ms; this rule at half 641 / 16.7, at one
                // 677 / 17.4; eight lanes, whatever the number active, 678 / 17.8.
                const unsigned tris = __ballot_sync(0xffffffffu, active && s.tri_mask != 0u);
                const unsigned nodes = __ballot_sync(0xffffffffu, active && s.tri_mask2 == 0u && s.node != kNoNode);
                if (2 * __popc(tris) >= __popc(nodes) || nodes == 0u) {
                    if (active && s.tri_mask) {
                        done = trav_test_tri<kAnyHit, kCount, false>(B, s);
                        if (s.tri_mask == 0u) {
                            s.tri_base = s.tri_base2;
                            s.tri_mask = s.tri_mask2;
                            s.tri_mask2 = 0u;
                        }
                        done = done || (s.tri_mask == 0u && s.node == kNoNode);
                    }
                } else {
                    if (active && s.tri_mask2 == 0u && s.node != kNoNode) done = trav_node(B, s, stk, stride, lerr);
                }
            }
            if (done) active = false;
            act = __ballot_sync(0xffffffffu, active);
        }
        // finished rays are handed on here, several lanes at a time, rather than one by one in the loop
        // (2^20 bounces in a soup 643 -> 616 us, 16.6M-path frame 9.83 -> 9.56 ms)
        if (held && !active) {
            end(k, s);
            held = false;
        }
        if (!kCount && exhausted && act != 0u) {
            // hand the last rays to groups of eight lanes
            unsigned m = act;
            for (int g = lane / kCoopLanes; g > 0; g--) m &= m - 1u;
            const bool live = m != 0u;
            const int src = live ? __ffs(m) - 1 : lane;
            auto from = [&](auto& x) { x = __shfl_sync(0xffffffffu, x, src); };
            from(s.o.x); from(s.o.y); from(s.o.z);
            from(s.d.x); from(s.d.y); from(s.d.z);
            from(s.inv.x); from(s.inv.y); from(s.inv.z);
            from(s.tmin); from(s.oct); from(s.sp); from(s.node); from(s.nvis);
            from(s.best.t); from(s.best.u); from(s.best.v); from(s.best.id);
            from(s.tri_base); from(s.tri_mask); from(s.tri_base2); from(s.tri_mask2);
            if (kTwoLevel) {
                from(s.wo.x); from(s.wo.y); from(s.wo.z);
                from(s.wd.x); from(s.wd.y); from(s.wd.z);
                from(s.inst_sp); from(s.id_base);
            }
            from(k);
            if (live) B = tree(k);
            __syncwarp();
            coop_loop<kAnyHit, kTwoLevel>(B, s, live, k, stk + (src - lane), stride, lerr, end);
            return;
        }
    }
}

}  // namespace lmgpu
