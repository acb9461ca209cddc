// The ray-march kernel (shared by the march_*.cu translation units): a GB300 restatement of CPURaycaster::directRendering
// (modules/base/processors/render/cpuraycaster.cpp:210-326) with the GLSL-only
// compositing and shading rules of rc_singlevolume.frag:116-312.
//
// Design:
//  * persistent grid (a few CTAs per SM); each warp pulls 8x4 ray tiles from
//    a global counter, so a warp's 32 rays are adjacent on screen and walk
//    the same bricks. Small frames give each ray 2 to 8 lanes, and larger ones
//    hand the rays left over when the tiles run out to a second kernel with 8
//    lanes a ray (launch_t has the rule and the figures);
//  * the transfer function sits in shared memory as its RGBA8 entries plus
//    a table of 256 alphas (one per alpha byte) that already carry the
//    opacity correction 1-(1-a)^(step*200), computed on the host with the
//    same powf the CPU path calls; r/255, g/255, b/255 are the exact 8-bit
//    normalisation. 17 KB per CTA at 4096 entries, so most of the SM's
//    unified L1 / shared array stays L1 for the voxel gathers;
//  * voxels come from the bricked layout (32^3 core + apron), so a stencil
//    never crosses a brick; empty bricks (per-brick min/max against the TF)
//    are skipped without reading voxels while t still advances sample by
//    sample, which keeps results identical to the unskipped march;
//  * every operation on the sample path is an explicitly rounded FP32
//    intrinsic in the reference's order (no FMA contraction), so positions,
//    trilinear values, TF indices, compositing and the t > tend stop match
//    the FP32 CPU path bit for bit;
//  * what bounds it: neither HBM (3 % of peak on 512^3 shaded DVR) nor any one
//    pipe, but issue slots and load latency along each ray's serial chain, with
//    22 (512^3 shells) to 13 (sparse tubes) of 32 lanes active. So a sample is
//    made of as few instructions and dependent loads as its rounding allows:
//    the default brick's geometry is compile-time (BS = 32), products and
//    lerps run on FP32 pairs (f32x2), the TF coordinate is a corrected product
//    instead of a division, one distance byte decides emptiness, the box exit
//    is two FMAs an axis on per-ray constants. Together, us per frame before
//    and after (bits unchanged): 512^3 u16 shaded DVR at 1080p 678 -> 475, its
//    MIP 830 -> 661, pre-integrated 854 -> 605, 2048x2048x1024 tubes at 4K
//    21,600 -> 15,430, 64 mixed requests 15,100 -> 11,030; then the lanes a
//    ray and the queue, shaded DVR 475 -> 388, pre-integrated 605 -> 487,
//    64^3 u8 at 256^2 81 -> 48;
//  * gradients (central differences, mod_gradients.frag:202-214) are six
//    lookups at +-1/dim in texture space, clamped like the intensity sample
//    and read from the centre's brick apron (another brick only when rounding
//    puts a tap two voxels away); they interpolate raw voxel values with FMA
//    lerps. Phong (mod_shading.frag:134-151) runs in registers with fast
//    reciprocal square roots and __powf. Shading only colours samples whose
//    alpha is already decided, so it changes no discrete decision; its
//    colours differ from the CPU path by ~1e-6.
#pragma once
#include <algorithm>
#include <cstdint>
#include <mutex>
#include <vector>

#include "vrc_internal.h"

namespace vrc {
namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int LOOP_CAP = 255 * 255;  // cpuraycaster.cpp:239

__device__ __forceinline__ float m_(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float a_(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float s_(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float d_(float a, float b) { return __fdiv_rn(a, b); }

// Exact voxel normalisation v / 255 and v / 65535 (VolumeRAM's
// getVoxelNormalized: float division, correctly rounded), without a
// division or an integer-to-float conversion instruction.
// For D = 2^k - 1, 1/D = 2^-k (1 + 2^-k + 2^-2k + ...), so
//   v / D = v (2^-k + 2^-2k) + v (2^-3k [+ 2^-4k + 2^-5k for k = 8]) + tail,
// tail >= 0 and smaller than the spacing of the fused sum's grid (2^-48 for
// k = 16, 2^-40 for k = 8). The fused sum lies on that grid, as do all
// rounding midpoints of the result, and it is never a midpoint itself: for a
// result in [2^e, 2^(e+1)), v would need a factor 2^(e + 24) (k = 16) or
// 2^(e + 16) (k = 8), more than v < 2^(e + k + 1) holds. So the tail cannot
// change the rounding: fma(v, A, v * B) = RN(v / D) for every v in [0, D]. (Checked exhaustively by the test suite.) v as a float: the bits
// 0x4B000000 | v are the float 2^23 + v.
__device__ __forceinline__ float small_uint_to_float(unsigned v) {
    return __fsub_rn(__int_as_float(0x4B000000u | v), 8388608.f);
}
// Pairs of FP32 in one 64-bit register pair: add / mul / fma of both halves
// in one issue slot, each half rounded as the scalar instruction rounds it
// (never a product that an addition follows: a pair of those came out fused).
// The march is bound by instruction issue and load latency, so the sample's
// eight normalisations and products and the gradient's lerps run on pairs.
using f2 = unsigned long long;
__device__ __forceinline__ f2 pk(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float lo2(f2 v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return a;
}
__device__ __forceinline__ float hi2(f2 v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return b;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// a + t * (b - a) of both halves (t the same or one per half)
__device__ __forceinline__ f2 lerp2(f2 t, f2 a, f2 b) { return fma2(t, sub2(b, a), a); }

__device__ __forceinline__ float magic_uint(unsigned v) { return __int_as_float(0x4B000000u | v); }  // 2^23 + v

// norm: v / 255, v / 65535; raw2: two stored values as floats; norm2: two
// normalised values from raw2's.
template <int DT> struct Vox;
template <> struct Vox<VRC_U8> {
    using T = uint8_t;
    static __device__ __forceinline__ float norm(T v) {
        const float x = small_uint_to_float(v);
        return __fmaf_rn(x, 0x1.01p-8f, __fmul_rn(x, 0x1.0101p-24f));
    }
    static __device__ __forceinline__ f2 raw2(T a, T b) {
        return add2(pk(magic_uint(a), magic_uint(b)), pk(-8388608.f, -8388608.f));
    }
    static __device__ __forceinline__ f2 norm2(f2 x) {
        return fma2(x, pk(0x1.01p-8f, 0x1.01p-8f), mul2(x, pk(0x1.0101p-24f, 0x1.0101p-24f)));
    }
};
template <> struct Vox<VRC_U16> {
    using T = uint16_t;
    static __device__ __forceinline__ float norm(T v) {
        const float x = small_uint_to_float(v);
        return __fmaf_rn(x, 0x1.0001p-16f, __fmul_rn(x, 0x1p-48f));
    }
    static __device__ __forceinline__ f2 raw2(T a, T b) {
        return add2(pk(magic_uint(a), magic_uint(b)), pk(-8388608.f, -8388608.f));
    }
    static __device__ __forceinline__ f2 norm2(f2 x) {
        return fma2(x, pk(0x1.0001p-16f, 0x1.0001p-16f), mul2(x, pk(0x1p-48f, 0x1p-48f)));
    }
};
template <> struct Vox<VRC_F32> {
    using T = float;
    static __device__ __forceinline__ float norm(T v) { return v; }
    static __device__ __forceinline__ f2 raw2(T a, T b) { return pk(a, b); }
    static __device__ __forceinline__ f2 norm2(f2 x) { return x; }
};

struct F3 {
    float x, y, z;
};

// The eight stored values around a sample as floats: c<x><y> holds the pair
// (z = 0, z = 1). S, S2: row and slice stride of the brick.
struct Raw8 {
    f2 c00, c10, c01, c11;
};
template <int DT>
__device__ __forceinline__ Raw8 load8(const typename Vox<DT>::T* __restrict__ b, int S, int S2) {
    using V = Vox<DT>;
    return Raw8{V::raw2(__ldg(b), __ldg(b + S2)), V::raw2(__ldg(b + 1), __ldg(b + S2 + 1)),
                V::raw2(__ldg(b + S), __ldg(b + S2 + S)), V::raw2(__ldg(b + S + 1), __ldg(b + S2 + S + 1))};
}

// VolumeRAM::getVoxelNormalizedLinear (volumeram.cpp:89-96): each voxel times
// its x, y and z weight, summed in the order 000 100 110 010 001 101 111 011;
// the products of a z pair run together, the sum one after the other.
template <int DT>
__device__ __forceinline__ float tri8(const Raw8& r, float fx, float fy, float fz) {
    using V = Vox<DT>;
    const float ox = s_(1.f, fx), oy = s_(1.f, fy), oz = s_(1.f, fz);
    const f2 wx0 = pk(ox, ox), wx1 = pk(fx, fx), wy0 = pk(oy, oy), wy1 = pk(fy, fy), wz = pk(oz, fz);
    const f2 a = mul2(mul2(mul2(V::norm2(r.c00), wx0), wy0), wz);
    const f2 b = mul2(mul2(mul2(V::norm2(r.c10), wx1), wy0), wz);
    const f2 c = mul2(mul2(mul2(V::norm2(r.c11), wx1), wy1), wz);
    const f2 d = mul2(mul2(mul2(V::norm2(r.c01), wx0), wy1), wz);
    float s = a_(lo2(a), lo2(b));
    s = a_(s, lo2(c));
    s = a_(s, lo2(d));
    s = a_(s, hi2(a));
    s = a_(s, hi2(b));
    s = a_(s, hi2(c));
    return a_(s, hi2(d));
}

template <int DT>
__device__ __forceinline__ float tri_at(const typename Vox<DT>::T* __restrict__ b, int o, int S, int S2, float fx,
                                        float fy, float fz) {
    return tri8<DT>(load8<DT>(b + o, S, S2), fx, fy, fz);
}

// (x > lo ? x : lo) < hi ? ... : hi, also for NaN (lo)
__device__ __forceinline__ float clampf_(float x, float lo, float hi) { return fminf(fmaxf(x, lo), hi); }

// RealWorldMapping::realWorldToNormalized on the TF domain: 0 below it, 1
// above, (rw - lo) / (hi - lo) inside, correctly rounded. With rcp = RN(1 / (hi
// - lo)) given, the quotient is the product a * rcp corrected twice by its
// exact residual: after the first correction it is within one ulp, and then
// the second gives RN(a / b) (Markstein, IBM J. Res. Dev. 34(1), 1990,
// theorem on q + r * RN(1/b)). The host gives rcp only for 2^-60 <= hi - lo <=
// 2^60: the residual of any a >= 2^-100 is then exact, and a smaller a selects
// entry 0 whatever its last bit. 5 instructions instead of a division's call
// sequence. rcp = 0: divide.
__device__ __forceinline__ float rw_to_tf(float rw, float lo, float hi, float rcp) {
    if (rcp != 0.f) {
        const float a = s_(clampf_(rw, lo, hi), lo), b = s_(hi, lo);
        float q = m_(a, rcp);
        q = __fmaf_rn(__fmaf_rn(-q, b, a), rcp, q);
        return __fmaf_rn(__fmaf_rn(-q, b, a), rcp, q);
    }
    if (rw < lo) return 0.f;
    if (rw > hi) return 1.f;
    if (lo == hi) return 0.f;
    return d_(s_(rw, lo), s_(hi, lo));
}

// iround(x * (w - 1)) for x in [0, 1] (or NaN: entry 0): x * (w - 1) + 0.5 is
// not negative and below w, so truncation is the floor and no clamp is needed
__device__ __forceinline__ int tf_index(float x, int w) { return (int)a_(m_(x, (float)(w - 1)), 0.5f); }

__device__ __forceinline__ float len3(float x, float y, float z) {
    float s = m_(x, x);
    s = a_(s, m_(y, y));
    s = a_(s, m_(z, z));
    return __fsqrt_rn(s);
}

__device__ __forceinline__ F3 normalize3(F3 v) {
    const float l = len3(v.x, v.y, v.z);
    if (l == 0.f) return F3{0.f, 0.f, 0.f};
    const float r = d_(1.f, l);
    return F3{m_(v.x, r), m_(v.y, r), m_(v.z, r)};
}

__device__ __forceinline__ float dot3(F3 a, F3 b) {
    float s = m_(a.x, b.x);
    s = a_(s, m_(a.y, b.y));
    s = a_(s, m_(a.z, b.z));
    return s;
}

// ---- shading path ----------------------------------------------------
// Shading feeds only the colour of samples with alpha > 0; it has no
// discrete decision and its pow is not correctly rounded on any platform, so
// it uses fused multiply-adds, fast reciprocal square roots and __powf. The
// resulting colour differs from the CPU path by ~1e-6 relative.
__device__ __forceinline__ F3 fnormalize(F3 v) {
    const float l2 = __fmaf_rn(v.x, v.x, __fmaf_rn(v.y, v.y, __fmul_rn(v.z, v.z)));
    if (l2 == 0.f) return F3{0.f, 0.f, 0.f};
    const float r = rsqrtf(l2);
    return F3{v.x * r, v.y * r, v.z * r};
}
__device__ __forceinline__ float fdot(F3 a, F3 b) { return __fmaf_rn(a.x, b.x, __fmaf_rn(a.y, b.y, __fmul_rn(a.z, b.z))); }

// Trilinear interpolation of raw voxel values with FMA lerps (gradient taps).
template <int DT>
__device__ __forceinline__ float tri_raw(const typename Vox<DT>::T* __restrict__ b, int o, int S, int S2, float fx,
                                         float fy, float fz) {
    const float v000 = (float)__ldg(b + o), v100 = (float)__ldg(b + o + 1);
    const float v010 = (float)__ldg(b + o + S), v110 = (float)__ldg(b + o + S + 1);
    const float v001 = (float)__ldg(b + o + S2), v101 = (float)__ldg(b + o + S2 + 1);
    const float v011 = (float)__ldg(b + o + S2 + S), v111 = (float)__ldg(b + o + S2 + S + 1);
    const float x00 = __fmaf_rn(fx, v100 - v000, v000), x10 = __fmaf_rn(fx, v110 - v010, v010);
    const float x01 = __fmaf_rn(fx, v101 - v001, v001), x11 = __fmaf_rn(fx, v111 - v011, v011);
    const float y0 = __fmaf_rn(fy, x10 - x00, x00), y1 = __fmaf_rn(fy, x11 - x01, x01);
    return __fmaf_rn(fz, y1 - y0, y0);
}

// Start of brick `brick`: in the pool directly, or, for a host-resident pool
// with a device cache (brick_slot != nullptr), in the cache slot the table
// names. A brick the cache does not hold (slot -1) is read in the mapped
// host pool, so every brick stays readable whatever the cache holds -- or,
// with a level of detail attached, not at all: nullptr, and the caller
// samples the half-resolution level instead.
template <bool POOL, typename T>
__device__ __forceinline__ const T* brick_base(const MarchParams& P, const T* __restrict__ bricks, long long brick) {
    if (!POOL) return bricks + brick * P.L.brick_stride;
    const int slot = __ldg(P.brick_slot + brick);
    if (slot >= 0) return bricks + (long long)slot * P.L.brick_stride;
    return P.lod_bricks ? nullptr : reinterpret_cast<const T*>(P.host_pool) + brick * P.L.brick_stride;
}

// Records that a brick was read this frame (cache refinement). Lanes of the
// warp reading the same brick share one atomic.
__device__ __forceinline__ void mark_used(const MarchParams& P, long long brick) {
    const unsigned peers = __match_any_sync(__activemask(), (unsigned long long)brick);
    if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicOr(P.brick_used + (brick >> 5), 1u << (brick & 31));
}

// The half-resolution level at texture-space point (sx, sy, sz), sampled
// like the full level (clamped voxel position, trilinear from the brick
// holding the floor voxel): normalised (RAW false) or raw values. This is
// the coarser octree level Voreen's octree raycaster reads where a brick is
// not on the GPU (singleoctreeraycaster.cl), here the 2x2x2 mean of
// VolumeOctree's half-sampled parent bricks (volumeoctree.cpp:188-202).
template <int DT, bool RAW>
__device__ __noinline__ float lod_tap(const MarchParams& P, float sx, float sy, float sz) {
    using T = typename Vox<DT>::T;
    const BrickLayout& L = P.L;
    const float vx = clampf_(s_(m_(P.lod_dimf[0], sx), 0.5f), 0.f, P.lod_dim_m1[0]);
    const float vy = clampf_(s_(m_(P.lod_dimf[1], sy), 0.5f), 0.f, P.lod_dim_m1[1]);
    const float vz = clampf_(s_(m_(P.lod_dimf[2], sz), 0.5f), 0.f, P.lod_dim_m1[2]);
    const float flx = floorf(vx), fly = floorf(vy), flz = floorf(vz);
    const int ix = (int)flx, iy = (int)fly, iz = (int)flz;
    const int bx = ix >> L.shift, by = iy >> L.shift, bz = iz >> L.shift;
    const long long brick = ((long long)bz * P.lod_nb[1] + by) * P.lod_nb[0] + bx;
    const T* b = reinterpret_cast<const T*>(P.lod_bricks) + brick * L.brick_stride;
    const int o = ((iz - (bz << L.shift) + APRON_LO) * L.S + (iy - (by << L.shift) + APRON_LO)) * L.S +
                  (ix - (bx << L.shift) + APRON_LO);
    const float fx = s_(vx, flx), fy = s_(vy, fly), fz = s_(vz, flz);
    return RAW ? tri_raw<DT>(b, o, L.S, L.S * L.S, fx, fy, fz) : tri_at<DT>(b, o, L.S, L.S * L.S, fx, fy, fz);
}

// The same from a full-resolution voxel position (gradient and previous-sample
// taps of a brick without a cache slot). These taps read the coarser level
// and so approximate the full-resolution values whatever the rounding of
// their texture-space position; a fast division serves.
template <int DT, bool RAW>
__device__ __forceinline__ float lod_tap_voxel(const MarchParams& P, float vx, float vy, float vz) {
    return lod_tap<DT, RAW>(P, __fdividef(vx + 0.5f, P.dimf[0]), __fdividef(vy + 0.5f, P.dimf[1]),
                            __fdividef(vz + 0.5f, P.dimf[2]));
}

template <int DT, bool POOL>
__device__ __noinline__ float tap_raw_any_brick(const MarchParams& P, const typename Vox<DT>::T* __restrict__ bricks,
                                                float vx, float vy, float vz) {
    const BrickLayout& L = P.L;
    const float flx = floorf(vx), fly = floorf(vy), flz = floorf(vz);
    const int ix = (int)flx, iy = (int)fly, iz = (int)flz;
    const int bx = ix >> L.shift, by = iy >> L.shift, bz = iz >> L.shift;
    const long long brick = ((long long)bz * L.nb[1] + by) * L.nb[0] + bx;
    const int o = ((iz - (bz << L.shift) + APRON_LO) * L.S + (iy - (by << L.shift) + APRON_LO)) * L.S +
                  (ix - (bx << L.shift) + APRON_LO);
    if (POOL && P.brick_used) atomicOr(P.brick_used + (brick >> 5), 1u << (brick & 31));
    const typename Vox<DT>::T* b = brick_base<POOL>(P, bricks, brick);
    if (POOL && !b) return lod_tap_voxel<DT, true>(P, vx, vy, vz);
    return tri_raw<DT>(b, o, L.S, L.S * L.S, vx - flx, vy - fly, vz - flz);
}

// One central-difference lookup displaced along one axis: tap position `vt`
// (clamped voxel coordinate on that axis, as calcGradientA's texture lookup
// gives it) with the centre's coordinates on the other axes. Reads from the
// centre's brick when the stencil fits in its apron.
template <int DT, int AXIS, bool POOL>
__device__ __forceinline__ float grad_tap(const MarchParams& P, const typename Vox<DT>::T* __restrict__ bricks,
                                          const typename Vox<DT>::T* __restrict__ b, int o, int lc, int ic, float vt,
                                          float vx, float vy, float vz, float fx, float fy, float fz) {
    const float fl = floorf(vt);
    const int it = (int)fl;
    const int lt = lc + (it - ic);
    const int S = P.L.S, S2 = P.L.S * P.L.S;
    if ((!POOL || b) && lt >= 0 && lt <= P.L.B + 1) {
        const int stride = AXIS == 0 ? 1 : (AXIS == 1 ? S : S2);
        const float ft = vt - fl;
        return tri_raw<DT>(b, o + (it - ic) * stride, S, S2, AXIS == 0 ? ft : fx, AXIS == 1 ? ft : fy,
                           AXIS == 2 ? ft : fz);
    }
    return tap_raw_any_brick<DT, POOL>(P, bricks, AXIS == 0 ? vt : vx, AXIS == 1 ? vt : vy, AXIS == 2 ? vt : vz);
}

// phongShading (mod_shading.frag:134-151), ka = kd = TF colour, ks = 1.
__device__ __forceinline__ F3 phong_fast(const MarchParams& P, F3 n, F3 pos, F3 col) {
    const F3 N = fnormalize(n);
    F3 L{P.light_phys[0] - pos.x, P.light_phys[1] - pos.y, P.light_phys[2] - pos.z};
    const F3 V = fnormalize(F3{P.cam_phys[0] - pos.x, P.cam_phys[1] - pos.y, P.cam_phys[2] - pos.z});
    const float d2 = fdot(L, L);
    const float rd = d2 > 0.f ? rsqrtf(d2) : 0.f;
    const float d = d2 * rd;
    L = F3{L.x * rd, L.y * rd, L.z * rd};
    const float ndl = fmaxf(fdot(N, L), 0.f);
    const F3 Hh = fnormalize(F3{V.x + L.x, V.y + L.y, V.z + L.z});
    const float ndh = fmaxf(fdot(N, Hh), 0.f);
    const float spec = __powf(ndh, P.shininess);
    F3 out{__fmaf_rn(col.x * P.dif[0], ndl, __fmaf_rn(P.spec[0], spec, col.x * P.amb[0])),
           __fmaf_rn(col.y * P.dif[1], ndl, __fmaf_rn(P.spec[1], spec, col.y * P.amb[1])),
           __fmaf_rn(col.z * P.dif[2], ndl, __fmaf_rn(P.spec[2], spec, col.z * P.amb[2]))};
    if (P.atten_on) {
        const float att = fminf(__fdividef(1.f, __fmaf_rn(P.att[2] * d, d, __fmaf_rn(P.att[1], d, P.att[0]))), 1.f);
        out = F3{out.x * att, out.y * att, out.z * att};
    }
    return out;
}

// Analytic entry/exit for pixel (px, py): the pixel-centre ray through the
// unit texture cube, clipped to the near/far planes. Returns false for
// background.
__device__ bool analytic_entry_exit(const MarchParams& P, int px, int py, float4& e, float4& l) {
    const float nx = s_(d_(m_(2.f, a_((float)px, 0.5f)), (float)P.W), 1.f);
    const float ny = s_(d_(m_(2.f, a_((float)py, 0.5f)), (float)P.H), 1.f);
    float pn[4], pf[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const float* M = P.inv_mvp + 4 * r;
        const float base = a_(m_(M[0], nx), m_(M[1], ny));
        pn[r] = a_(s_(base, M[2]), M[3]);
        pf[r] = a_(a_(base, M[2]), M[3]);
    }
    float o[3], d[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        o[i] = d_(pn[i], pn[3]);
        d[i] = s_(d_(pf[i], pf[3]), o[i]);
    }
    float s0 = 0.f, s1 = 1.f;
    bool hit = true;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        if (d[i] == 0.f) {
            if (o[i] < P.box_lo[i] || o[i] > P.box_hi[i]) hit = false;
        } else {
            float a = d_(s_(P.box_lo[i], o[i]), d[i]), b = d_(s_(P.box_hi[i], o[i]), d[i]);
            if (a > b) {
                const float t = a;
                a = b;
                b = t;
            }
            s0 = fmaxf(s0, a);
            s1 = fminf(s1, b);
        }
    }
    if (!hit || !(s0 < s1)) {
        e = make_float4(0.f, 0.f, 0.f, 0.f);
        l = e;
        return false;
    }
    float en[3], ex[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        float a = clampf_(a_(o[i], m_(s0, d[i])), P.box_lo[i], P.box_hi[i]);
        float b = clampf_(a_(o[i], m_(s1, d[i])), P.box_lo[i], P.box_hi[i]);
        if (P.quantize) {
            a = d_(floorf(a_(m_(a, 65535.f), 0.5f)), 65535.f);
            b = d_(floorf(a_(m_(b, 65535.f), 0.5f)), 65535.f);
        }
        en[i] = a;
        ex[i] = b;
    }
    e = make_float4(en[0], en[1], en[2], 1.f);
    l = make_float4(ex[0], ex[1], ex[2], 1.f);
    return true;
}

__device__ __forceinline__ F3 entry_point_at(const MarchParams& P, int x, int y) {
    x = min(max(x, 0), P.W - 1);
    y = min(max(y, 0), P.H - 1);
    float4 e, l;
    if (P.ee_mode == VRC_EE_BUFFERS) {
        e = P.entry[(size_t)y * P.W + x];
    } else {
        analytic_entry_exit(P, x, y, e, l);
    }
    return F3{e.x, e.y, e.z};
}

// fixClipBorderGradient (mod_gradients.frag:39-46); only samples at t = 0
// with alpha > 0 come here, so it stays out of line
__device__ __noinline__ F3 clip_border_gradient(const MarchParams& P, F3 s, F3 dir, int px, int py) {
    const F3 a = entry_point_at(P, px + 2, py), b = entry_point_at(P, px, py + 2);
    const F3 v0 = normalize3(F3{s_(a.x, s.x), s_(a.y, s.y), s_(a.z, s.z)});
    const F3 v1 = normalize3(F3{s_(b.x, s.x), s_(b.y, s.y), s_(b.z, s.z)});
    F3 g{s_(m_(v0.y, v1.z), m_(v0.z, v1.y)), s_(m_(v0.z, v1.x), m_(v0.x, v1.z)), s_(m_(v0.x, v1.y), m_(v0.y, v1.x))};
    if (!(dot3(g, dir) < 0.f)) g = F3{-g.x, -g.y, -g.z};
    return g;
}

__device__ __forceinline__ void write_out(const MarchParams& P, size_t pix, float4 r) {
    if (P.out_format == VRC_OUT_RGBA32F) {
        reinterpret_cast<float4*>(P.out)[pix] = r;
    } else if (P.out_format == VRC_OUT_RGBA8) {
        auto q = [](float v) -> unsigned {
            v = fminf(fmaxf(v, 0.f), 1.f);
            return (unsigned)floorf(v * 255.f + 0.5f);
        };
        reinterpret_cast<uchar4*>(P.out)[pix] = make_uchar4(q(r.x), q(r.y), q(r.z), q(r.w));
    } else {
        auto q = [](float v) -> unsigned {
            v = fminf(fmaxf(v, 0.f), 1.f);
            return (unsigned)floorf(v * 65535.f + 0.5f);
        };
        reinterpret_cast<ushort4*>(P.out)[pix] = make_ushort4(q(r.x), q(r.y), q(r.z), q(r.w));
    }
}

// Samples of one ray by what became of them, two counts of at most 255^2 to a
// register: fetched in the low half, shaded in the high half; skip runs in the
// low half, pre-integration's reads of a skipped previous sample (fetched
// samples too) in the high half.
struct RayCounts {
    unsigned fetched_shaded = 0, runs = 0;
};

// Adds a tile's rays to the warp's totals in shared memory: the totals take no
// registers while a ray marches. `loop`: the samples of this lane's ray.
struct WarpTotals {
    unsigned long long samples, fetched, shaded, runs;
};
__device__ __forceinline__ void add_tile(WarpTotals& w, int loop, const RayCounts& c) {
    // at most 32 x 2 x 255^2 each
    const unsigned a = __reduce_add_sync(FULL, (unsigned)loop);
    const unsigned b = __reduce_add_sync(FULL, (c.fetched_shaded & 0xffffu) + (c.runs >> 16));
    const unsigned d = __reduce_add_sync(FULL, c.fetched_shaded >> 16);
    const unsigned e = __reduce_add_sync(FULL, c.runs & 0xffffu);
    if ((threadIdx.x & 31) == 0) {
        w.samples += a;
        w.fetched += b;
        w.shaded += d;
        w.runs += e;
    }
}

// MIP: true when no sample of a cell whose largest normalised value is `m`
// can exceed the ray's maximum real-world intensity `max_int`, so the cell
// changes nothing (compositeMIP replaces the result only for a larger value).
// A trilinear sample exceeds its largest voxel by at most ~13 ulp of rounding
// (three products, seven sums, weights summing to at most (1 + u)^3); m is
// raised by 2e-6 relative, well above that, and the real-world mapping is
// monotone (scale >= 0, checked on the host), so the test is exact.
__device__ __forceinline__ bool mip_cell_below(const MarchParams& P, float m, float max_int) {
    const float mb = m + fabsf(m) * 2e-6f;
    return a_(m_(mb, P.rwm_scale), P.rwm_offset) <= max_int;
}

// Largest ray parameter up to which every sample's floor voxel stays in skip
// cell (cx, cy, cz): per axis, where the unclamped voxel coordinate
// dim * (first + t * dir) - 0.5 reaches the cell face it moves toward, pulled
// in by skip_margin voxels to absorb rounding (the margin exceeds the error of
// the sample-position arithmetic and of the fast division here by orders of
// magnitude). Cells on the volume border have no face on their outer side:
// clamping keeps samples there.
__device__ __forceinline__ float cell_exit_t(const MarchParams& P, float4 f, float dx, float dy, float dz, int cx,
                                             int cy, int cz, int shift, const int* nc) {
    const int C = 1 << shift;
    const float fo[3] = {f.x, f.y, f.z}, di[3] = {dx, dy, dz};
    const int ci[3] = {cx, cy, cz};
    float tmax = INFINITY;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float a = P.dimf[i] * fo[i] - 0.5f, b = P.dimf[i] * di[i];
        if (b > 0.f && ci[i] < nc[i] - 1) {
            tmax = fminf(tmax, __fdividef((float)((ci[i] + 1) * C) - P.skip_margin - a, b));
        } else if (b < 0.f && ci[i] > 0) {
            tmax = fminf(tmax, __fdividef((float)(ci[i] * C) + P.skip_margin - a, b));
        }
    }
    return tmax;
}

// The same for a box of cells [c - r, c + r] on each axis, the ray's part
// computed once: an axis with voxel position a + t * b is left at
//   b > 0:  ((c + r + 1) * C - margin - a) / b = c * C/b + r * C/b + (C - margin - a)/b
//   b < 0:  ((c - r) * C + margin - a) / b     = c * C/b - r * C/b + (margin - a)/b,
// two FMAs on per-ray constants. Each term is below the volume's edge in
// voxels, so FP32 rounding moves the face by less than 4 * 2^-23 of that
// edge; the margin is 0.01 + 2e-5 of it. An axis the ray does not move along
// gives infinities or NaN, which fminf drops where they mean "never left".
// A face on the grid's border is never left (samples beyond it clamp to the
// border cells): at() counts it like others, which costs samples within the
// volume nothing but the last half voxel at a near face; border() drops it and
// is taken where at() gives a ray no advance.
struct BoxExit {
    float k1[3], k0[3];
    __device__ __forceinline__ void set(const MarchParams& P, float4 f, float dx, float dy, float dz) {
        const float fo[3] = {f.x, f.y, f.z}, di[3] = {dx, dy, dz};
        const float C = (float)(1 << P.cshift);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float a = P.dimf[i] * fo[i] - 0.5f, rb = __fdividef(1.f, P.dimf[i] * di[i]);
            k1[i] = C * rb;
            k0[i] = ((rb > 0.f ? C - P.skip_margin : P.skip_margin) - a) * rb;
        }
    }
    __device__ __forceinline__ float at(int cx, int cy, int cz, int r) const {
        const float fr = (float)r;
        const float tx = __fmaf_rn((float)cx, k1[0], __fmaf_rn(fr, fabsf(k1[0]), k0[0]));
        const float ty = __fmaf_rn((float)cy, k1[1], __fmaf_rn(fr, fabsf(k1[1]), k0[1]));
        const float tz = __fmaf_rn((float)cz, k1[2], __fmaf_rn(fr, fabsf(k1[2]), k0[2]));
        return fminf(fminf(tx, ty), tz);
    }
    __device__ __forceinline__ float border(const MarchParams& P, int cx, int cy, int cz, int r) const {
        const float fr = (float)r;
        const int c[3] = {cx, cy, cz};
        float t = INFINITY;
#pragma unroll
        for (int i = 0; i < 3; ++i)
            if (k1[i] > 0.f ? c[i] + r < P.nc[i] - 1 : c[i] - r > 0)
                t = fminf(t, __fmaf_rn((float)c[i], k1[i], __fmaf_rn(fr, fabsf(k1[i]), k0[i])));
        return t;
    }
};

// Advances (t, loop) over the samples of an empty run in closed form: every
// sample with t <= lim is processed (and changes nothing). The FP32 sum
// t + step, for t on the grid of its binade [T, 2T) with spacing u, is exactly
// t + q with q = round(step / u) * u = fl(T + step) - T, unless step / u ends
// in .5 (a rounding tie, left to the caller's exact loop). So n steps inside
// the binade give exactly t + n * q, the value the reference's one-at-a-time
// accumulation t += samplingStepSize produces. n is the number of whole steps
// that fit before lim and before the binade's last step; the quotient's error
// (at most 65025 steps times 2^-22) stays below that step. The caller finishes
// with exact single steps (one or two, and one across the binade's end).
template <bool TRACK = false>
__device__ __forceinline__ void jump_empty_run(float& t, int& loop, float step, float lim, float* tprev = nullptr) {
    const float T = __int_as_float(__float_as_int(t) & 0x7f800000);
    const float q = s_(a_(T, step), T);
    if (!(T > 0x1p-90f) || step >= T || !(q > 0.f) || fabsf(s_(step, q)) == m_(T, 0x1p-24f)) return;
    const float x = m_(s_(fminf(lim, s_(m_(2.f, T), q)), t), __fdividef(1.f, q));
    const int n = min((int)x, LOOP_CAP - loop);
    if (n <= 0) return;
    if (TRACK) *tprev = __fmaf_rn((float)(n - 1), q, t);  // the last sample jumped over
    t = __fmaf_rn((float)n, q, t);
    loop += n;
}

// The samples after one in an empty cell, up to lim: processed without effect.
__device__ __forceinline__ void skip_run(float& t, int& loop, float step, float lim) {
    t = a_(t, step);
    ++loop;
    while (t <= lim && loop < LOOP_CAP) {
        jump_empty_run(t, loop, step, lim);
        if (t <= lim && loop < LOOP_CAP) {
            t = a_(t, step);
            ++loop;
        }
    }
}

// Normalised trilinear value at a clamped voxel position, read from the
// brick holding its floor voxel, in the exact order of the intensity sample.
template <int DT, bool POOL>
__device__ __forceinline__ float tap_norm(const MarchParams& P, const typename Vox<DT>::T* __restrict__ bricks,
                                          float vx, float vy, float vz) {
    const BrickLayout& L = P.L;
    const float flx = floorf(vx), fly = floorf(vy), flz = floorf(vz);
    const int ix = (int)flx, iy = (int)fly, iz = (int)flz;
    const int bx = ix >> L.shift, by = iy >> L.shift, bz = iz >> L.shift;
    const long long brick = ((long long)bz * L.nb[1] + by) * L.nb[0] + bx;
    const int lx = ix - (bx << L.shift) + APRON_LO, ly = iy - (by << L.shift) + APRON_LO,
              lz = iz - (bz << L.shift) + APRON_LO;
    if (POOL && P.brick_used) atomicOr(P.brick_used + (brick >> 5), 1u << (brick & 31));
    const typename Vox<DT>::T* b = brick_base<POOL>(P, bricks, brick);
    if (POOL && !b) return lod_tap_voxel<DT, false>(P, vx, vy, vz);
    return tri_at<DT>(b, (lz * L.S + ly) * L.S + lx, L.S, L.S * L.S, s_(vx, flx),
                      s_(vy, fly), s_(vz, flz));
}

// Texture-space point -> clamped voxel position (cpuraycaster.cpp:243).
__device__ __forceinline__ float to_voxel(const MarchParams& P, int axis, float s) {
    return clampf_(s_(m_(P.dimf[axis], s), 0.5f), 0.f, P.dim_m1[axis]);
}

// calcGradientA (mod_gradients.frag:202-214) with exactly rounded taps, in
// the order the CPU restatement evaluates it: six normalised trilinear
// lookups at +-1/dim in texture space, (v(-) - v(+)) * 0.5/spacing * rwmScale.
template <int DT, bool POOL>
__device__ F3 gradient_exact(const MarchParams& P, const typename Vox<DT>::T* __restrict__ bricks, float sx, float sy,
                             float sz, float vx, float vy, float vz) {
    const float v0 = tap_norm<DT, POOL>(P, bricks, to_voxel(P, 0, a_(sx, P.offs[0])), vy, vz);
    const float v1 = tap_norm<DT, POOL>(P, bricks, vx, to_voxel(P, 1, a_(sy, P.offs[1])), vz);
    const float v2 = tap_norm<DT, POOL>(P, bricks, vx, vy, to_voxel(P, 2, a_(sz, P.offs[2])));
    const float v3 = tap_norm<DT, POOL>(P, bricks, to_voxel(P, 0, s_(sx, P.offs[0])), vy, vz);
    const float v4 = tap_norm<DT, POOL>(P, bricks, vx, to_voxel(P, 1, s_(sy, P.offs[1])), vz);
    const float v5 = tap_norm<DT, POOL>(P, bricks, vx, vy, to_voxel(P, 2, s_(sz, P.offs[2])));
    return F3{m_(m_(s_(v3, v0), P.spacing_rcp_half[0]), P.rwm_scale),
              m_(m_(s_(v4, v1), P.spacing_rcp_half[1]), P.rwm_scale),
              m_(m_(s_(v5, v2), P.spacing_rcp_half[2]), P.rwm_scale)};
}

// compositeMIDAhelper (mod_compositing.frag:109-125): delta = max intensity
// increase, beta = 1 - delta * (1 + gamma), then a DVR step weighted by beta.
__device__ __forceinline__ float4 mida_step(float4 r, float v, float4 c, float maxi, float gamma) {
    const float delta = v > maxi ? s_(v, maxi) : 0.f;
    const float beta = s_(1.f, m_(delta, a_(1.f, gamma)));
    const float wa = m_(s_(1.f, m_(beta, r.w)), c.w);
    return make_float4(a_(m_(beta, r.x), m_(wa, c.x)), a_(m_(beta, r.y), m_(wa, c.y)), a_(m_(beta, r.z), m_(wa, c.z)),
                       a_(m_(beta, r.w), wa));
}

// The geometry of a brick: compile-time for the default 32^3 bricks (BS = 32:
// shifts, strides and the 32 voxel addresses of a shaded sample become
// immediates), at run time otherwise (BS = 0).
template <int BS> struct BrickGeom {
    static_assert(BS == 0 || BS == 32, "brick edge");
    static __device__ __forceinline__ int shift(const BrickLayout& L) { return BS ? 5 : L.shift; }
    static __device__ __forceinline__ int S(const BrickLayout& L) { return BS ? BS + APRON_LO + APRON_HI : L.S; }
    static __device__ __forceinline__ int S2(const BrickLayout& L) { return S(L) * S(L); }
    static __device__ __forceinline__ long long stride(const BrickLayout& L) {
        constexpr int E = BS + APRON_LO + APRON_HI;
        return BS ? (E * E * E + 63) / 64 * 64 : L.brick_stride;
    }
};

// A sample: texture-space point s, clamped voxel position v, its floor.
struct SamplePos {
    float sx, sy, sz, vx, vy, vz, flx, fly, flz;
    int ix, iy, iz;
    __device__ __forceinline__ void set(const MarchParams& P, float4 f, float dx, float dy, float dz, float t) {
        sx = a_(f.x, m_(t, dx));
        sy = a_(f.y, m_(t, dy));
        sz = a_(f.z, m_(t, dz));
        vx = to_voxel(P, 0, sx);
        vy = to_voxel(P, 1, sy);
        vz = to_voxel(P, 2, sz);
        flx = floorf(vx);
        fly = floorf(vy);
        flz = floorf(vz);
        ix = (int)flx;
        iy = (int)fly;
        iz = (int)flz;
    }
};

// calcGradientA (mod_gradients.frag:202-214) where some tap is not one voxel
// from the sample's floor voxel (the volume's faces, or rounding): the taps
// are read from the sample's brick where its apron holds them, else from
// their own bricks. Rare, so out of line.
template <int DT, bool POOL>
__device__ __noinline__ F3 gradient_at_edges(const MarchParams& P, const typename Vox<DT>::T* __restrict__ bricks,
                                             const typename Vox<DT>::T* __restrict__ b, float sx, float sy, float sz) {
    const BrickLayout& L = P.L;
    const int S = L.S, S2 = L.S * L.S;
    const float vx = to_voxel(P, 0, sx), vy = to_voxel(P, 1, sy), vz = to_voxel(P, 2, sz);
    const float flx = floorf(vx), fly = floorf(vy), flz = floorf(vz);
    const int ix = (int)flx, iy = (int)fly, iz = (int)flz;
    const float fx = s_(vx, flx), fy = s_(vy, fly), fz = s_(vz, flz);
    const int lx = (ix & (L.B - 1)) + APRON_LO, ly = (iy & (L.B - 1)) + APRON_LO, lz = (iz & (L.B - 1)) + APRON_LO;
    const int o = (lz * S + ly) * S + lx;
    const float vxp = to_voxel(P, 0, a_(sx, P.offs[0])), vxm = to_voxel(P, 0, s_(sx, P.offs[0]));
    const float vyp = to_voxel(P, 1, a_(sy, P.offs[1])), vym = to_voxel(P, 1, s_(sy, P.offs[1]));
    const float vzp = to_voxel(P, 2, a_(sz, P.offs[2])), vzm = to_voxel(P, 2, s_(sz, P.offs[2]));
    const float v0 = grad_tap<DT, 0, POOL>(P, bricks, b, o, lx, ix, vxp, vx, vy, vz, fx, fy, fz);
    const float v1 = grad_tap<DT, 1, POOL>(P, bricks, b, o, ly, iy, vyp, vx, vy, vz, fx, fy, fz);
    const float v2 = grad_tap<DT, 2, POOL>(P, bricks, b, o, lz, iz, vzp, vx, vy, vz, fx, fy, fz);
    const float v3 = grad_tap<DT, 0, POOL>(P, bricks, b, o, lx, ix, vxm, vx, vy, vz, fx, fy, fz);
    const float v4 = grad_tap<DT, 1, POOL>(P, bricks, b, o, ly, iy, vym, vx, vy, vz, fx, fy, fz);
    const float v5 = grad_tap<DT, 2, POOL>(P, bricks, b, o, lz, iz, vzm, vx, vy, vz, fx, fy, fz);
    return F3{(v3 - v0) * P.gscale[0], (v4 - v1) * P.gscale[1], (v5 - v2) * P.gscale[2]};
}

// calcGradientA of a sample: six lookups at +-1/dim in texture space, each
// clamped like the intensity sample, interpolated on raw values. p: its
// position, (fx, fy, fz) the fractions, b its brick, vox the address of its
// floor voxel, c the eight raw values there. Usually each tap's floor voxel is
// one voxel from the sample's; the six stencils then cover the eight values
// and 24 more (four on each side), read in one straight block and
// interpolated from registers. The bits of a sample's gradient do not depend
// on which thread or loop computes it.
template <int DT, int BS, bool POOL>
__device__ __forceinline__ F3 central_gradient(const MarchParams& P, const typename Vox<DT>::T* __restrict__ bricks,
                                               const typename Vox<DT>::T* __restrict__ b,
                                               const typename Vox<DT>::T* __restrict__ vox, const Raw8& c,
                                               const SamplePos& p, float fx, float fy, float fz) {
    using V = Vox<DT>;
    const int S = BrickGeom<BS>::S(P.L), S2 = BrickGeom<BS>::S2(P.L);
    const float vxp = to_voxel(P, 0, a_(p.sx, P.offs[0])), vxm = to_voxel(P, 0, s_(p.sx, P.offs[0]));
    const float vyp = to_voxel(P, 1, a_(p.sy, P.offs[1])), vym = to_voxel(P, 1, s_(p.sy, P.offs[1]));
    const float vzp = to_voxel(P, 2, a_(p.sz, P.offs[2])), vzm = to_voxel(P, 2, s_(p.sz, P.offs[2]));
    const float fxp = floorf(vxp), fyp = floorf(vyp), fzp = floorf(vzp);
    const float fxm = floorf(vxm), fym = floorf(vym), fzm = floorf(vzm);
    // floors are whole numbers below 2^24: differences of 1 are exact
    const bool usual = s_(fxp, p.flx) == 1.f && s_(fyp, p.fly) == 1.f && s_(fzp, p.flz) == 1.f &&
                       s_(p.flx, fxm) == 1.f && s_(p.fly, fym) == 1.f && s_(p.flz, fzm) == 1.f;
    if ((POOL && !b) || !usual) return gradient_at_edges<DT, POOL>(P, bricks, b, p.sx, p.sy, p.sz);
    // v<axis><side> pairs over z (0, 1); the z sides as the pair (-1, 2)
#define VRC_Z(X, Y) V::raw2(__ldg(vox + (X) + (Y) * S), __ldg(vox + (X) + (Y) * S + S2))
#define VRC_E(X, Y) V::raw2(__ldg(vox + (X) + (Y) * S - S2), __ldg(vox + (X) + (Y) * S + 2 * S2))
    const f2 fx2 = pk(fx, fx), fy2 = pk(fy, fy);
    const float gxp = vxp - fxp, gxm = vxm - fxm, gyp = vyp - fyp, gym = vym - fym;
    const f2 xm0 = VRC_Z(-1, 0), xm1 = VRC_Z(-1, 1), xp0 = VRC_Z(2, 0), xp1 = VRC_Z(2, 1);
    const f2 ym0 = VRC_Z(0, -1), ym1 = VRC_Z(1, -1), yp0 = VRC_Z(0, 2), yp1 = VRC_Z(1, 2);
    const f2 xp = lerp2(fy2, lerp2(pk(gxp, gxp), c.c10, xp0), lerp2(pk(gxp, gxp), c.c11, xp1));
    const f2 xm = lerp2(fy2, lerp2(pk(gxm, gxm), xm0, c.c00), lerp2(pk(gxm, gxm), xm1, c.c01));
    const f2 e0 = lerp2(fx2, c.c00, c.c10), e1 = lerp2(fx2, c.c01, c.c11);
    const f2 yp = lerp2(pk(gyp, gyp), e1, lerp2(fx2, yp0, yp1));
    const f2 ym = lerp2(pk(gym, gym), lerp2(fx2, ym0, ym1), e0);
    // the z sides after the others: 24 loads in flight at once cost the 80
    // registers spills (512^3 tubes 16.2 ms a 4K frame against 15.4)
    asm volatile("" ::: "memory");
    const f2 z00 = VRC_E(0, 0), z10 = VRC_E(1, 0), z01 = VRC_E(0, 1), z11 = VRC_E(1, 1);
    const f2 f = lerp2(fy2, e0, e1);
    const f2 z = lerp2(fy2, lerp2(fx2, z00, z10), lerp2(fx2, z01, z11));
#undef VRC_Z
#undef VRC_E
    const float v0 = __fmaf_rn(fz, hi2(xp) - lo2(xp), lo2(xp)), v3 = __fmaf_rn(fz, hi2(xm) - lo2(xm), lo2(xm));
    const float v1 = __fmaf_rn(fz, hi2(yp) - lo2(yp), lo2(yp)), v4 = __fmaf_rn(fz, hi2(ym) - lo2(ym), lo2(ym));
    const float v2 = __fmaf_rn(vzp - fzp, hi2(z) - hi2(f), hi2(f)), v5 = __fmaf_rn(vzm - fzm, lo2(f) - lo2(z), lo2(z));
    return F3{(v3 - v0) * P.gscale[0], (v4 - v1) * P.gscale[1], (v5 - v2) * P.gscale[2]};
}

// The Phong colour of a sample with gradient g and TF colour c.
__device__ __forceinline__ void shade(const MarchParams& P, const SamplePos& p, F3 g, float4& c) {
    const F3 pos{a_(m_(s_(m_(p.sx, P.dimf[0]), 0.5f), P.spacing[0]), P.vol_offset[0]),
                 a_(m_(s_(m_(p.sy, P.dimf[1]), 0.5f), P.spacing[1]), P.vol_offset[1]),
                 a_(m_(s_(m_(p.sz, P.dimf[2]), 0.5f), P.spacing[2]), P.vol_offset[2])};
    const F3 sh = phong_fast(P, g, pos, F3{c.x, c.y, c.z});
    c.x = sh.x;
    c.y = sh.y;
    c.z = sh.z;
}

// One sample with alpha > 0 onto the ray's result (rc_singlevolume.frag,
// mod_compositing.frag): c its colour and alpha, rw its real-world intensity.
// FHP and FHN take the value to show in c.
template <int COMP>
__device__ __forceinline__ void composite(const MarchParams& P, float4& res, float& max_int, float4 c, float rw) {
    if (COMP == VRC_DVR || COMP == COMP_DVR_PREINT) {
        const float w = m_(s_(1.f, res.w), c.w);
        res.x = a_(res.x, m_(w, c.x));
        res.y = a_(res.y, m_(w, c.y));
        res.z = a_(res.z, m_(w, c.z));
        res.w = a_(res.w, w);
    } else if (COMP == VRC_MIP) {
        if (rw > max_int) {
            res = c;
            max_int = rw;
        }
    } else if (COMP == VRC_ISO) {
        if (c.w >= s_(P.iso, 0.02f) && c.w <= a_(P.iso, 0.02f)) res = make_float4(c.x, c.y, c.z, 1.f);
    } else if (COMP == VRC_MOP) {
        // compositeMOP (mod_compositing.frag:97-107)
        if (c.w > res.w) res = c;
    } else if (COMP == VRC_MIDA) {
        // compositeMIDA (mod_compositing.frag:127-146); as there, only
        // the MIP half (gamma > 0) ever raises the maximum intensity
        const float gm = P.mida_gamma;
        if (gm <= 0.f) {
            res = mida_step(res, rw, c, max_int, gm);
        } else {
            float4 mip = res;
            if (rw > max_int) {
                mip = c;
                max_int = rw;
            }
            const float4 md = mida_step(res, rw, c, max_int, 0.f);
            const float og = s_(1.f, gm);
            res = make_float4(a_(m_(gm, mip.x), m_(og, md.x)), a_(m_(gm, mip.y), m_(og, md.y)),
                              a_(m_(gm, mip.z), m_(og, md.z)), a_(m_(gm, mip.w), m_(og, md.w)));
        }
    } else {  // compositeFHP / compositeFHN (mod_compositing.frag:168-196): the first sample
        if (res.x == 0.f && res.y == 0.f && res.z == 0.f) res = c;
    }
}

// The auxiliary output of a pixel whose first sample with alpha > 0 lies at t
// with squared gradient magnitude g2 (no such sample: (1, 0), written with the
// pixel before its ray marches).
__device__ __forceinline__ void write_aux(const MarchParams& P, int px, int py, float t, float tend, float g2) {
    P.aux[(size_t)py * P.W + px] = make_float2(__fdividef(t, fmaxf(tend, 1e-20f)), sqrtf(g2) * P.aux_gscale);
}

// Ray direction and end (cpuraycaster.cpp:216-232); degenerate rays take one sample.
__device__ __forceinline__ float ray_setup(const MarchParams& P, float4 f, float4 l, float& dx, float& dy, float& dz) {
    dx = s_(l.x, f.x);
    dy = s_(l.y, f.y);
    dz = s_(l.z, f.z);
    const bool dir0 = dx == 0.f && dy == 0.f && dz == 0.f;
    const bool last0 = l.x == 0.f && l.y == 0.f && l.z == 0.f;
    const bool first0 = f.x == 0.f && f.y == 0.f && f.z == 0.f;
    if (dir0 && !last0 && !first0) return d_(P.step, 2.f);
    const float tend = len3(dx, dy, dz);
    const float rl = d_(1.f, tend);
    dx = m_(dx, rl);
    dy = m_(dy, rl);
    dz = m_(dz, rl);
    return tend;
}

// Colour of a sample's TF coordinate x: the entry's bytes / 255 (exact), alpha
// from the per-byte table.
template <bool GLOBAL_TF>
__device__ __forceinline__ float4 tf_colour(const MarchParams& P, const uchar4* __restrict__ s_tf,
                                            const float* __restrict__ s_alpha, float rw) {
    const int i = (int)a_(m_(rw_to_tf(rw, P.tf_lo, P.tf_hi, P.tf_rcp), P.tf_wm1), 0.5f);
    const uchar4 e8 = GLOBAL_TF ? __ldg(s_tf + i) : s_tf[i];
    const f2 rg = Vox<VRC_U8>::norm2(Vox<VRC_U8>::raw2(e8.x, e8.y));
    return make_float4(lo2(rg), hi2(rg), Vox<VRC_U8>::norm(e8.z), GLOBAL_TF ? __ldg(s_alpha + e8.w) : s_alpha[e8.w]);
}

// The empty-space test of one sample: whether its cell is empty for the ray
// and, if so, up to which t the following samples are too.
//  * A TF-empty cell with the cells' distance field given (occ_dist: 0 for an
//    occupied cell) is the centre of an empty box: one byte decides, and the
//    box's exit ends the run. Reading the byte alone instead of the bit map
//    first takes one of two dependent loads out of every run.
//  * MIP: a cell that cannot raise the ray's maximum is left too, or its
//    whole brick where that cannot either.
//  * Without the field (pre-integration with steps of a voxel or more) the bit
//    map decides, and the brick's bit gives the longer run.
template <int COMP>
__device__ __forceinline__ bool empty_cell(const MarchParams& P, const BoxExit& bx, float4 f, float dx, float dy,
                                           float dz, const SamplePos& p, float t, float max_int, float& tsafe) {
    constexpr bool MIPS = COMP == VRC_MIP;
    // cell and brick indices fit 32 bits (checked when the volume is uploaded)
    const int fcx = p.ix >> P.cshift, fcy = p.iy >> P.cshift, fcz = p.iz >> P.cshift;
    const unsigned fc = ((unsigned)fcz * (unsigned)P.nc[1] + (unsigned)fcy) * (unsigned)P.nc[0] + (unsigned)fcx;
    const bool mip_skip = MIPS && P.mip_skip;
    bool tf_empty;
    if (P.occ_dist) {
        const int d = (int)__ldg(P.occ_dist + fc);
        tf_empty = d > 0;
        if (tf_empty) {
            const int r = d - 1;
            tsafe = bx.at(fcx, fcy, fcz, r);
            if (!(tsafe > t)) tsafe = bx.border(P, fcx, fcy, fcz, r);
            return true;
        }
        if (!mip_skip) return false;
    } else {
        tf_empty = ((__ldg(P.occupancy + (fc >> 5)) >> (fc & 31)) & 1u) == 0u;
    }
    if (!(tf_empty || (mip_skip && mip_cell_below(P, __ldg(P.cell_max + fc), max_int)))) return false;
    if (P.occ_coarse) {
        // a brick holds its cells' value ranges, so it can be empty (or below
        // the maximum) only where the cell is
        const int cx = p.ix >> P.cshift_coarse, cy = p.iy >> P.cshift_coarse, cz = p.iz >> P.cshift_coarse;
        const unsigned c = ((unsigned)cz * (unsigned)P.ncc[1] + (unsigned)cy) * (unsigned)P.ncc[0] + (unsigned)cx;
        if (((__ldg(P.occ_coarse + (c >> 5)) >> (c & 31)) & 1u) == 0u ||
            (mip_skip && mip_cell_below(P, __ldg(P.brick_max + c), max_int))) {
            tsafe = cell_exit_t(P, f, dx, dy, dz, cx, cy, cz, P.cshift_coarse, P.ncc);
            return true;
        }
    }
    tsafe = cell_exit_t(P, f, dx, dy, dz, fcx, fcy, fcz, P.cshift, P.nc);
    return true;
}

// What a ray's samples so far have left; t, loop: the next sample. In the
// queue of unfinished rays: two float4 (pre-integration has no maximum, the
// other modes no previous sample).
struct RayState {
    float4 res;
    float max_int, t;
    int loop;
    bool hit;         // the auxiliary output has the first sample with alpha > 0
    float t_prev;     // pre-integration: the sample before t, and whether its cell was empty
    bool prev_empty;
    __device__ __forceinline__ void begin(const MarchParams& P) {
        res = make_float4(0.f, 0.f, 0.f, 0.f);
        max_int = t = t_prev = 0.f;
        loop = 0;
        hit = P.aux == nullptr;
        prev_empty = false;
    }
    template <bool PI> __device__ __forceinline__ void store(float4* q, int pix) const {
        q[0] = res;
        q[1] = make_float4(PI ? t_prev : max_int, t, __int_as_float(loop | (hit ? 1 << 30 : 0) | (prev_empty ? 1 << 29 : 0)),
                           __int_as_float(pix));
    }
    template <bool PI> __device__ __forceinline__ int load(const float4* q) {
        res = q[0];
        const float4 r = q[1];
        (PI ? t_prev : max_int) = r.x;
        t = r.y;
        const int bits = __float_as_int(r.z);
        loop = bits & ((1 << 29) - 1);
        hit = ((bits >> 30) & 1) != 0;
        prev_empty = ((bits >> 29) & 1) != 0;
        return __float_as_int(r.w);
    }
};

// One ray on one thread: the loop of cpuraycaster.cpp:239-317 with the GLSL
// compositing. STOP: the ray is left unfinished (false) a sample or run after
// *stop becomes set. GLOBAL_TF: the table is in global memory.
template <int DT, int COMP, int SHADE, int BS, bool POOL, bool STOP, bool GLOBAL_TF = false>
__device__ __forceinline__ bool march_ray(const MarchParams& P, const uchar4* __restrict__ s_tf,
                                          const float* __restrict__ s_alpha, float4 f, float4 l, int px, int py,
                                          const volatile int* stop, RayState& st, RayCounts& cnt) {
    using T = typename Vox<DT>::T;
    using G = BrickGeom<BS>;
    const T* __restrict__ bricks = reinterpret_cast<const T*>(P.bricks);
    const float step = P.step;
    float dx, dy, dz;
    const float tend = ray_setup(P, f, l, dx, dy, dz);
    // pre-integrated classification (cpuraycaster.cpp:255-261); no early ray
    // termination for mip / mop / mida (volumeraycaster.cpp:226-228)
    constexpr bool PI = COMP == COMP_DVR_PREINT;
    constexpr bool ERT = !(COMP == VRC_MIP || COMP == VRC_MOP || COMP == VRC_MIDA);
    BoxExit bx;
    bx.set(P, f, dx, dy, dz);
    float4& res = st.res;
    float &max_int = st.max_int, &t = st.t;
    int& loop = st.loop;
    bool& hit = st.hit;
    st.begin(P);
    float last = 0.f;  // lastIntensity (cpuraycaster.cpp:235), TF-normalised
    // pre-integration: whether the previous sample lay in an empty cell, and
    // whether `last` still has to be read at t_last (the last skipped sample)
    bool& prev_empty = st.prev_empty;
    bool last_stale = false;
    float& t_last = st.t_prev;
    long long marked = -1;             // last brick recorded as read (cache refinement)
    // POOL: the brick of the last fetched sample and its start (a slot lookup
    // each); a device-resident pool's address is two multiply-adds
    int cached_brick = -1;
    const T* cached_base = nullptr;
    bool finished = false;
    int stopped = 0;
    while (!finished && loop < LOOP_CAP) {
        // read for the next pass: the load's latency stays off the chain
        if (STOP) {
            if (stopped) return false;
            stopped = *stop;
        }
        SamplePos p;
        p.set(P, f, dx, dy, dz, t);
        bool skip_after = false;  // pre-integration: skip the samples after this one in its empty cell
        float skip_lim = 0.f;
        if (P.occupancy) {
            float tsafe = 0.f;
            const bool empty = empty_cell<COMP>(P, bx, f, dx, dy, dz, p, t, max_int, tsafe);
            if (PI && empty && P.pi_chain && prev_empty) {
                // This sample and the previous one lie in empty cells that
                // share a voxel (a step moves less than a voxel per axis), so
                // their value ranges overlap and every table entry between
                // the two samples has alpha 0: skip it and the rest of its
                // cell; `last` is read when a sample is next classified.
                ++cnt.runs;
                float tp = t;
                t = a_(t, step);
                ++loop;
                const float lim = fminf(tsafe, tend);
                while (t <= lim && loop < LOOP_CAP) {
                    jump_empty_run<true>(t, loop, step, lim, &tp);
                    if (t <= lim && loop < LOOP_CAP) {
                        tp = t;
                        t = a_(t, step);
                        ++loop;
                    }
                }
                finished = t > tend;
                last_stale = true;
                t_last = tp;
                continue;
            } else if (PI && empty) {
                // A pre-integrated colour also depends on the previous sample,
                // which may lie outside the cell: classify this sample as
                // usual, skip the ones after it that stay in the cell (both
                // ends of their segments are in the cell, so every table
                // entry they reach has alpha 0).
                skip_after = true;
                skip_lim = fminf(tsafe, tend);
            } else if (empty) {
                // This sample lies in a cell where every reachable TF entry has
                // alpha 0: it changes nothing. So do all following samples that
                // provably stay in the cell; only t and the count advance.
                ++cnt.runs;
                skip_run(t, loop, step, fminf(tsafe, tend));
                finished = t > tend;
                continue;
            }
        }
        {
            const int sh = G::shift(P.L);
            const int bX = p.ix >> sh, bY = p.iy >> sh, bZ = p.iz >> sh;
            const int brick = (bZ * P.L.nb[1] + bY) * P.L.nb[0] + bX;
            const T* __restrict__ b;
            if (POOL) {
                if (brick != cached_brick) {
                    cached_brick = brick;
                    cached_base = brick_base<POOL>(P, bricks, (long long)brick);
                }
                b = cached_base;
                if (P.brick_used && brick != marked) {
                    marked = brick;
                    mark_used(P, brick);
                }
            } else {
                b = bricks + (long long)brick * G::stride(P.L);
            }
            ++cnt.fetched_shaded;
            const float fx = s_(p.vx, p.flx), fy = s_(p.vy, p.fly), fz = s_(p.vz, p.flz);
            const int S = G::S(P.L);
            const int o = ((p.iz - (bZ << sh) + APRON_LO) * S + (p.iy - (bY << sh) + APRON_LO)) * S +
                          (p.ix - (bX << sh) + APRON_LO);
            const T* __restrict__ vox = b + o;
            Raw8 raw;
            float intensity;
            if (!POOL || b) {
                raw = load8<DT>(vox, S, G::S2(P.L));
                intensity = tri8<DT>(raw, fx, fy, fz);
            } else {
                raw = Raw8{};
                intensity = lod_tap<DT, false>(P, p.sx, p.sy, p.sz);
            }
            const float rw = a_(m_(intensity, P.rwm_scale), P.rwm_offset);
            float4 c;
            if (PI) {
                if (last_stale) {  // the previous sample was skipped: read its TF coordinate
                    cnt.runs += 0x10000u;
                    const float px_ = a_(f.x, m_(t_last, dx)), py_ = a_(f.y, m_(t_last, dy)),
                                pz_ = a_(f.z, m_(t_last, dz));
                    const float rwp = a_(m_(tap_norm<DT, POOL>(P, bricks, to_voxel(P, 0, px_), to_voxel(P, 1, py_),
                                                        to_voxel(P, 2, pz_)),
                                            P.rwm_scale),
                                         P.rwm_offset);
                    last = rw_to_tf(rwp, P.tf_lo, P.tf_hi, P.tf_rcp);
                    last_stale = false;
                }
                prev_empty = skip_after;  // this sample is classified; its cell was empty iff skip_after
                // PreIntegrationTable::classify(last, cur) (preintegrationtable.cpp:256-279)
                const float cur = rw_to_tf(rw, P.tf_lo, P.tf_hi, P.tf_rcp);
                c = __ldg(P.pi_table + (size_t)tf_index(cur, P.pi_res) * P.pi_res + tf_index(last, P.pi_res));
                last = cur;
            } else {
                c = tf_colour<GLOBAL_TF>(P, s_tf, s_alpha, rw);
            }
            if (c.w > 0.f) {
                float gmag2 = 0.f;
                if (SHADE == VRC_SHADE_PHONG) {
                    cnt.fetched_shaded += 0x10000u;
                    const F3 g = t == 0.f ? clip_border_gradient(P, F3{p.sx, p.sy, p.sz}, F3{dx, dy, dz}, px, py)
                                          : central_gradient<DT, BS, POOL>(P, bricks, b, vox, raw, p, fx, fy, fz);
                    if (!hit) gmag2 = g.x * g.x + g.y * g.y + g.z * g.z;
                    shade(P, p, g, c);
                }
                if (!hit) {
                    hit = true;
                    write_aux(P, px, py, t, tend, gmag2);
                }
                if (COMP == VRC_FHP) {
                    c = make_float4(p.sx, p.sy, p.sz, 1.f);  // texture-space position
                } else if (COMP == VRC_FHN) {
                    // normalize(gradient) / 2 + 0.5, the gradient exactly
                    // rounded; a zero gradient gives 0.5. Only the first shows.
                    if (res.x == 0.f && res.y == 0.f && res.z == 0.f) {
                        const F3 g = t == 0.f ? clip_border_gradient(P, F3{p.sx, p.sy, p.sz}, F3{dx, dy, dz}, px, py)
                                              : gradient_exact<DT, POOL>(P, bricks, p.sx, p.sy, p.sz, p.vx, p.vy, p.vz);
                        const F3 n = normalize3(g);
                        c = make_float4(a_(d_(n.x, 2.f), 0.5f), a_(d_(n.y, 2.f), 0.5f), a_(d_(n.z, 2.f), 0.5f), 1.f);
                    }
                }
                composite<COMP>(P, res, max_int, c, rw);
            }
        }
        if (ERT && res.w >= P.ert) {
            res.w = 1.f;
            finished = true;
        }
        if (PI && STOP) t_last = t;  // where another kernel reads the previous sample
        t = a_(t, step);
        ++loop;
        finished = finished || (t > tend);
        if (PI && skip_after && !finished) {
            // skip the rest of the empty cell's samples; the next classified
            // sample needs the TF coordinate of the last one skipped
            ++cnt.runs;
            float tp = 0.f;
            bool skipped = false;
            while (t <= skip_lim && loop < LOOP_CAP) {
                const int l0 = loop;
                jump_empty_run<true>(t, loop, step, skip_lim, &tp);
                skipped = skipped || loop > l0;
                if (t <= skip_lim && loop < LOOP_CAP) {
                    tp = t;
                    skipped = true;
                    t = a_(t, step);
                    ++loop;
                }
            }
            finished = t > tend;
            if (skipped) {  // `last` is read when a sample is next classified
                last_stale = true;
                t_last = tp;
            }
        }
    }
    return true;
}

// One ray on G neighbouring lanes: lane k of the group takes the k-th of the
// next G samples, and the group then composites them in order, every lane the
// same (lane 0's result is the ray's). All lanes of the warp call it together;
// `alive` is the same in a group, and so are f, l, px, py. A ray's chain of
// dependent loads gets G times shorter where its samples are occupied, for G
// times the lanes on a run through empty space.
//
// Pre-integration: a sample is classified unless it and the one before it lie
// in empty cells a step of less than a voxel apart (as in march_ray; with
// longer steps every sample of a pass is), with the TF coordinate of the lane
// before. The last sample's coordinate goes on to the next pass; where it was
// not read, or samples were jumped over, lane 0 reads it when it is needed.
template <int DT, int COMP, int SHADE, int BS, int G>
__device__ __forceinline__ void march_ray_group(const MarchParams& P, const uchar4* __restrict__ s_tf,
                                                const float* __restrict__ s_alpha, bool alive, float4 f, float4 l,
                                                int px, int py, RayState& st, RayCounts& cnt) {
    using T = typename Vox<DT>::T;
    using BG = BrickGeom<BS>;
    constexpr bool PI = COMP == COMP_DVR_PREINT;
    constexpr bool ERT = !(COMP == VRC_MIP || COMP == VRC_MOP || COMP == VRC_MIDA);
    constexpr unsigned GM = (1u << G) - 1u;
    const T* __restrict__ bricks = reinterpret_cast<const T*>(P.bricks);
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), base = lane & ~(G - 1);
    const float step = P.step;
    float dx, dy, dz;
    const float tend = ray_setup(P, f, l, dx, dy, dz);
    BoxExit bx;
    bx.set(P, f, dx, dy, dz);
    float4& res = st.res;
    float &max_int = st.max_int, &t = st.t;
    int& loop = st.loop;
    bool& hit = st.hit;
    float last = 0.f;             // pre-integration: TF coordinate of the sample before t
    bool stale = PI && loop > 0;  // ... still to be read at st.t_prev
    bool finished = !alive;
    while (__any_sync(FULL, !finished)) {
        // this lane's sample: t advanced `sub` times, as the one-at-a-time loop does
        float tl = t, tn = t;
#pragma unroll
        for (int k = 1; k < G; ++k) {
            tn = a_(tn, step);
            if (k == sub) tl = tn;
        }
        tn = a_(tn, step);
        const bool valid = !finished && loop + sub < LOOP_CAP && (sub == 0 || !(tl > tend));
        float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
        float rw = 0.f, tsafe = 0.f, gmag2 = 0.f, cur = 0.f;
        bool empty = false;
        unsigned gval, gemp, gcls, gread;  // per group: valid samples, empty, classified, read
        SamplePos p;
        // A sample's voxels and intensity; classify(raw, ...) then colours it
        // from values still in registers.
        auto read = [&](auto classify) {
            const int sh = BG::shift(P.L), S = BG::S(P.L);
            const int bX = p.ix >> sh, bY = p.iy >> sh, bZ = p.iz >> sh;
            const T* __restrict__ b = bricks + (long long)((bZ * P.L.nb[1] + bY) * P.L.nb[0] + bX) * BG::stride(P.L);
            const float fx = s_(p.vx, p.flx), fy = s_(p.vy, p.fly), fz = s_(p.vz, p.flz);
            const T* __restrict__ vox = b + ((p.iz - (bZ << sh) + APRON_LO) * S + (p.iy - (bY << sh) + APRON_LO)) * S +
                                        (p.ix - (bX << sh) + APRON_LO);
            const Raw8 raw = load8<DT>(vox, S, BG::S2(P.L));
            rw = a_(m_(tri8<DT>(raw, fx, fy, fz), P.rwm_scale), P.rwm_offset);
            classify(b, vox, raw, fx, fy, fz);
        };
        auto shade_sample = [&](const T* b, const T* vox, const Raw8& raw, float fx, float fy, float fz) {
            if (SHADE == VRC_SHADE_PHONG && c.w > 0.f) {
                const F3 g = tl == 0.f ? clip_border_gradient(P, F3{p.sx, p.sy, p.sz}, F3{dx, dy, dz}, px, py)
                                       : central_gradient<DT, BS, false>(P, bricks, b, vox, raw, p, fx, fy, fz);
                if (!hit) gmag2 = g.x * g.x + g.y * g.y + g.z * g.z;
                shade(P, p, g, c);
            }
        };
        if (valid) {
            p.set(P, f, dx, dy, dz, tl);
            if (P.occupancy) empty = empty_cell<COMP>(P, bx, f, dx, dy, dz, p, tl, max_int, tsafe);
            if (!PI && !empty)
                read([&](const T* b, const T* vox, const Raw8& raw, float fx, float fy, float fz) {
                    c = tf_colour<false>(P, s_tf, s_alpha, rw);
                    shade_sample(b, vox, raw, fx, fy, fz);
                });
        }
        gval = (__ballot_sync(FULL, valid) >> base) & GM, gemp = (__ballot_sync(FULL, empty) >> base) & GM;
        gcls = gread = gval & ~gemp;
        if (PI) {
            gcls = P.pi_chain ? gval & ~(gemp & (gemp << 1 | (st.prev_empty ? 1u : 0u))) : gval;
            gread = gcls | gcls >> 1;  // the sample before each classified one too
            if (stale && (gcls & 1u) && sub == 0) {
                cnt.runs += 0x10000u;
                const float x = a_(f.x, m_(st.t_prev, dx)), y = a_(f.y, m_(st.t_prev, dy)), z = a_(f.z, m_(st.t_prev, dz));
                const float v = tap_norm<DT, false>(P, bricks, to_voxel(P, 0, x), to_voxel(P, 1, y), to_voxel(P, 2, z));
                last = rw_to_tf(a_(m_(v, P.rwm_scale), P.rwm_offset), P.tf_lo, P.tf_hi, P.tf_rcp);
            }
            // every lane of the warp takes part in handing the coordinates up,
            // so the colour is looked up, and shaded from voxels read again,
            // after it
            if ((gread >> sub) & 1u)
                read([&](const T*, const T*, const Raw8&, float, float, float) {
                    cur = rw_to_tf(rw, P.tf_lo, P.tf_hi, P.tf_rcp);
                });
            const float up = __shfl_up_sync(FULL, cur, 1, G);
            if ((gcls >> sub) & 1u) {
                c = __ldg(P.pi_table + (size_t)tf_index(cur, P.pi_res) * P.pi_res + tf_index(sub > 0 ? up : last, P.pi_res));
                if (SHADE == VRC_SHADE_PHONG && c.w > 0.f) read(shade_sample);
            }
        }
        const bool reads = (gread >> sub) & 1u;
        const unsigned vis = __ballot_sync(FULL, c.w > 0.f);
        const unsigned gvis = (vis >> base) & GM;
        int used = __popc(gval);  // samples of this pass that the ray takes
        bool stop = false;
        if (vis != 0u || (ERT && P.ert <= 0.f)) {
#pragma unroll
            for (int k = 0; k < G; ++k) {
                const float4 ck = make_float4(__shfl_sync(FULL, c.x, k, G), __shfl_sync(FULL, c.y, k, G),
                                              __shfl_sync(FULL, c.z, k, G), __shfl_sync(FULL, c.w, k, G));
                const float rk = COMP == VRC_MIP || COMP == VRC_MIDA ? __shfl_sync(FULL, rw, k, G) : 0.f;
                if (!stop && ((gcls >> k) & 1u)) {
                    if ((gvis >> k) & 1u) composite<COMP>(P, res, max_int, ck, rk);
                    if (ERT && res.w >= P.ert) {
                        res.w = 1.f;
                        stop = true;
                        used = k + 1;
                    }
                }
            }
            const int first = __ffs(gvis) - 1;  // none: -1
            if (!hit && first >= 0 && first < used) {
                hit = true;
                if (sub == first) write_aux(P, px, py, tl, tend, gmag2);
            }
        }
        if (sub < used && reads) {
            ++cnt.fetched_shaded;
            if (SHADE == VRC_SHADE_PHONG && c.w > 0.f) cnt.fetched_shaded += 0x10000u;
        }
        loop += used;
        finished = finished || stop || used < G || tn > tend || loop >= LOOP_CAP;
        t = tn;
        const float ts = __shfl_sync(FULL, tsafe, G - 1, G);
        if (PI) {
            last = __shfl_sync(FULL, cur, G - 1, G);
            st.t_prev = __shfl_sync(FULL, tl, G - 1, G);
            stale = !(gread >> (G - 1));
            st.prev_empty = (gemp >> (G - 1)) != 0u;
        }
        if (!finished && (gemp >> (G - 1)) != 0u) {
            // the last sample's cell is empty: so are the samples up to its exit
            if (sub == 0) ++cnt.runs;
            const float lim = fminf(ts, tend);
            while (t <= lim && loop < LOOP_CAP) {
                const int before_jump = loop;
                jump_empty_run<PI>(t, loop, step, lim, &st.t_prev);
                if (PI && loop > before_jump) stale = true;
                if (t <= lim && loop < LOOP_CAP) {
                    if (PI) {
                        st.t_prev = t;
                        stale = true;
                    }
                    t = a_(t, step);
                    ++loop;
                }
            }
            finished = t > tend || loop >= LOOP_CAP;
        }
    }
}

// The TF in shared memory: 256 alphas, then the RGBA8 entries (17 KB at 4096
// entries, leaving most of the SM's 256 KB to the L1 that serves the voxel
// gathers).
__device__ __forceinline__ void stage_tf(const MarchParams& P, float* s_alpha, uchar4* s_tf) {
    if (P.tf_width > 0) {
        for (int i = threadIdx.x; i < P.tf_width; i += blockDim.x) s_tf[i] = P.tf_rgba8[i];
        for (int i = threadIdx.x; i < 256; i += blockDim.x) s_alpha[i] = P.tf_alpha[i];
    }
    __syncthreads();
}

// Entry and exit point of a pixel; false for background.
__device__ __forceinline__ bool pixel_ray(const MarchParams& P, int px, int py, float4& f, float4& l) {
    if (P.ee_mode == VRC_EE_BUFFERS) {
        const size_t pix = (size_t)py * P.W + px;
        f = P.entry[pix];
        l = P.exitp[pix];
    } else {
        analytic_entry_exit(P, px, py, f, l);
    }
    return !(f.x == 0.f && f.y == 0.f && f.z == 0.f && f.w == 0.f && l.x == 0.f && l.y == 0.f && l.z == 0.f &&
             l.w == 0.f);
}

__device__ __forceinline__ void add_counters(const MarchParams& P, const WarpTotals& w) {
    if (!P.counters || (threadIdx.x & 31) != 0) return;
    atomicAdd(P.counters + 0, w.samples);
    atomicAdd(P.counters + 1, w.fetched);
    atomicAdd(P.counters + 2, w.shaded);
    atomicAdd(P.counters + 3, w.runs);
}

#ifndef VRC_MARCH_MIN_BLOCKS
#define VRC_MARCH_MIN_BLOCKS 3
#endif

// One ray per lane. QUEUE: when the tiles run out, the warps of a CTA leave
// their unfinished rays to march_queue_kernel: the longest rays of a frame
// (those that graze a shell, the whole of a MIP) take as long on one lane each
// as a tenth of the pixels do, so the frame would end on a few slow warps.
template <int DT, int COMP, int SHADE, int BS, bool POOL, bool QUEUE>
__global__ void __launch_bounds__(256, VRC_MARCH_MIN_BLOCKS) march_kernel(const __grid_constant__ MarchParams P) {
    extern __shared__ float4 s_raw[];
    float* s_alpha = reinterpret_cast<float*>(s_raw);
    uchar4* s_tf = reinterpret_cast<uchar4*>(s_alpha + 256);
    __shared__ WarpTotals totals[8];
    __shared__ int s_stop;
    if (threadIdx.x == 0) s_stop = 0;
    stage_tf(P, s_alpha, s_tf);
    const int lane = threadIdx.x & 31;
    const int ntiles = P.tiles_x * P.tiles_y;
    WarpTotals& mine = totals[threadIdx.x >> 5];
    if (lane == 0) mine = WarpTotals{};
    for (;;) {
        int tile = 0;
        if (lane == 0) tile = (int)atomicAdd(P.tile_counter, 1u);
        tile = __shfl_sync(FULL, tile, 0);
        if (tile >= ntiles) break;
        const int tx = tile % P.tiles_x, ty = tile / P.tiles_x;
        const int tw = 1 << P.tile_wshift;
        const int px = P.rx0 + tx * tw + (lane & (tw - 1));
        const int py = P.ry0 + ty * (32 >> P.tile_wshift) + (lane >> P.tile_wshift);
        RayState st;
        st.begin(P);
        RayCounts cnt;
        bool done = true;
        const size_t pix = (size_t)py * P.W + px;
        if (px < P.rx1 && py < P.ry1) {
            if (P.aux) P.aux[pix] = make_float2(1.f, 0.f);
            float4 f, l;
            if (pixel_ray(P, px, py, f, l))
                done = march_ray<DT, COMP, SHADE, BS, POOL, QUEUE>(P, s_tf, s_alpha, f, l, px, py, &s_stop, st, cnt);
            if (done) write_out(P, pix, st.res);
        }
        add_tile(mine, done ? st.loop : 0, cnt);
        if (QUEUE) {
            const unsigned left = __ballot_sync(FULL, !done);
            if (left) {
                unsigned at = 0;
                if (lane == 0) at = atomicAdd(P.queue_count, (unsigned)__popc(left));
                at = __shfl_sync(FULL, at, 0) + __popc(left & ((1u << lane) - 1u));
                if (!done) st.store<COMP == COMP_DVR_PREINT>(P.queue + 2 * (size_t)at, (int)pix);
            }
        }
    }
    if (QUEUE && lane == 0) *const_cast<volatile int*>(&s_stop) = 1;
    add_counters(P, mine);
}

// G lanes per ray, a warp takes 32 / G pixels: tiles of the frame, or the
// queue march_kernel left.
template <int G> struct GroupTile {
    static constexpr int W = G == 8 ? 2 : 4, H = 32 / G / W;
};
template <int DT, int COMP, int SHADE, int BS, int G, bool QUEUE>
__global__ void __launch_bounds__(256, VRC_MARCH_MIN_BLOCKS) march_group_kernel(const __grid_constant__ MarchParams P) {
    extern __shared__ float4 s_raw[];
    float* s_alpha = reinterpret_cast<float*>(s_raw);
    uchar4* s_tf = reinterpret_cast<uchar4*>(s_alpha + 256);
    const int lane = threadIdx.x & 31, ray = lane / G;
    const unsigned queued = QUEUE ? *P.queue_count : 0u;
    const int ntiles = QUEUE ? (int)((queued + 32 / G - 1) / (32 / G)) : P.tiles_x * P.tiles_y;
    if (QUEUE && (int)blockIdx.x * 8 >= ntiles) return;
    stage_tf(P, s_alpha, s_tf);
    __shared__ WarpTotals totals[8];
    WarpTotals& mine = totals[threadIdx.x >> 5];
    if (lane == 0) mine = WarpTotals{};
    for (;;) {
        int tile = 0;
        if (lane == 0) tile = (int)atomicAdd(QUEUE ? P.queue_count + 1 : P.tile_counter, 1u);
        tile = __shfl_sync(FULL, tile, 0);
        if (tile >= ntiles) break;
        RayState st;
        st.begin(P);
        int px, py;
        bool inside;
        if (QUEUE) {
            const unsigned q = (unsigned)tile * (32 / G) + ray;
            inside = q < queued;
            const int pix = inside ? st.load<COMP == COMP_DVR_PREINT>(P.queue + 2 * (size_t)q) : 0;
            py = pix / P.W;
            px = pix - py * P.W;
        } else {
            px = P.rx0 + (tile % P.tiles_x) * GroupTile<G>::W + ray % GroupTile<G>::W;
            py = P.ry0 + (tile / P.tiles_x) * GroupTile<G>::H + ray / GroupTile<G>::W;
            inside = px < P.rx1 && py < P.ry1;
        }
        const size_t pix = (size_t)py * P.W + px;
        const bool writes = inside && (lane & (G - 1)) == 0;
        if (!QUEUE && writes && P.aux) P.aux[pix] = make_float2(1.f, 0.f);
        __syncwarp();  // before any lane of the group writes the pixel's first hit
        float4 f = make_float4(0.f, 0.f, 0.f, 0.f), l = f;
        const bool alive = inside && pixel_ray(P, px, py, f, l);
        if (__any_sync(FULL, alive)) {
            RayCounts cnt;
            march_ray_group<DT, COMP, SHADE, BS, G>(P, s_tf, s_alpha, alive, f, l, px, py, st, cnt);
            add_tile(mine, writes ? st.loop : 0, cnt);
        }
        if (writes) write_out(P, pix, st.res);
    }
    add_counters(P, mine);
}

// Resident CTAs per SM of one kernel for a dynamic shared memory size,
// queried once per (kernel, device, size), and the kernel's shared memory limit
// and carve-out set for `largest`, the most it is launched with: the attribute calls and the
// occupancy query cost more host time than a frame's launch. Every march
// instantiation has the same function type, so entries are keyed by the
// kernel's address.
template <typename K>
cudaError_t resident_ctas(K k, size_t smem, size_t largest, int* per_sm) {
    struct Entry {
        const void* fn;
        int dev;
        size_t smem;
        int per_sm;
    };
    static std::mutex m;
    static std::vector<Entry> seen;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const void* fn = reinterpret_cast<const void*>(k);
    std::lock_guard<std::mutex> lock(m);
    for (const Entry& x : seen)
        if (x.fn == fn && x.dev == dev && x.smem == smem) {
            *per_sm = x.per_sm;
            return cudaSuccess;
        }
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)largest);
    if (e != cudaSuccess) return e;
    int n = 0, reserved = 0, per_sm_bytes = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, 256, smem);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&per_sm_bytes, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    // Shared memory gets what the resident CTAs' tables take and no more: left
    // alone, the driver gave it 135 KB of the SM's array where three CTAs use
    // 55 KB, and the gathers' L1 that much less. One step below the need
    // costs a resident CTA (512^3 MIP, 4 CTAs: 781 us against 701), one above
    // costs L1 (512^3 shaded DVR, 3 CTAs: 525 us against 508).
    if (e == cudaSuccess && n > 0 && per_sm_bytes > 0) {
        const long long need = (long long)n * ((long long)largest + reserved);
        const int percent = (int)std::min<long long>(100, (100 * need + per_sm_bytes - 1) / per_sm_bytes);
        e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, percent);
    }
    if (e != cudaSuccess) return e;
    seen.push_back(Entry{fn, dev, smem, n});
    *per_sm = n;
    return cudaSuccess;
}

inline size_t tf_smem(const MarchParams& p) { return 256 * sizeof(float) + (size_t)p.tf_width * sizeof(uchar4); }

// Persistent launch: as many CTAs as are resident at once, or as 8 warps a
// CTA need for the tiles.
template <typename K>
cudaError_t launch_persistent(K k, const MarchParams& p, long long tiles, int num_sms, cudaStream_t s) {
    int per_sm = 0;
    // the largest table (4096 entries) once per device; smaller ones fit under
    // it (a kernel that stages no table, pre-integration, has the 256 alphas)
    const size_t largest = 256 * sizeof(float) + (p.tf_width > 0 ? (size_t)4096 * sizeof(uchar4) : 0);
    cudaError_t e = resident_ctas(k, tf_smem(p), largest, &per_sm);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    long long grid = (long long)num_sms * per_sm;
    const long long need = (tiles + 7) / 8;
    if (grid > need) grid = need < 1 ? 1 : need;
    k<<<(unsigned)grid, 256, tf_smem(p), s>>>(p);
    if (p.launches) ++*p.launches;
    return cudaGetLastError();
}

template <int DT, int COMP, int SHADE, int BS, int G>
cudaError_t launch_group(const MarchParams& p, int num_sms, cudaStream_t s) {
    MarchParams q = p;
    q.tiles_x = (p.rx1 - p.rx0 + GroupTile<G>::W - 1) / GroupTile<G>::W;
    q.tiles_y = (p.ry1 - p.ry0 + GroupTile<G>::H - 1) / GroupTile<G>::H;
    return launch_persistent(march_group_kernel<DT, COMP, SHADE, BS, G, false>, q, (long long)q.tiles_x * q.tiles_y,
                             num_sms, s);
}

// How a frame's rays are spread over lanes, by its 32-pixel tiles against the
// warps the GPU holds (24 per SM). A frame ends when its longest ray does, and
// on one lane such a ray takes as long as a thousand tiles: CT volume, 512^3
// u16, shaded DVR, us by image and lanes per ray 1 / 2 / 4 / 8 / queue:
//    160x90    (460 tiles)     229  174  117   84    96
//    560x315   (5,530)         262  194  129  117   125
//    800x450   (11,300)        237  181  157  162   141
//    960x540   (16,200)        233  185  177  202   151
//    1920x1080 (64,800)        314  353  427  682   256
//    2560x1440 (115,200)       422  518  722 1179   371
//    3840x2160 (259,200)       720 1014 1553 2584   710
// (a 512x512x256 tube volume turns from 4 lanes to the queue between 11,300
// and 16,200 tiles too). More lanes a ray cost more on runs through empty
// space, which each lane of the group repeats, so they lose where the GPU is
// full. The queue: one lane a ray, and the rays unfinished when the tiles run
// out go on with 8 lanes each (half of a tube frame's gain with 4); it costs
// the marching loop 3 % of its rate, which 4K frames do not get back.
// Pre-integrated frames follow the same lines (1080p 605 -> 487).
// MIP, MOP and MIDA go on to the end of the volume, so their rays are long
// everywhere and the queue only adds to the work (512^3 MIP at 1080p 655 ->
// 782 us, 1280x720 628 -> 970); they take 4 lanes up to 16,200 tiles (MIP 611
// -> 394), 2 up to 28,800 (MIP 628 -> 595, MOP 534 -> 405), then one.
// A brick cache's use marks depend on which samples are read, and first-hit
// rays end early: one lane.
template <int DT, int COMP, int SHADE, int BS, bool POOL>
cudaError_t launch_t(const MarchParams& p, int num_sms, cudaStream_t s) {
    const long long tiles = (long long)p.tiles_x * p.tiles_y;
    constexpr bool ERT = COMP == VRC_DVR || COMP == VRC_ISO || COMP == COMP_DVR_PREINT;
    constexpr bool ALL = COMP == VRC_MIP || COMP == VRC_MOP || COMP == VRC_MIDA;
    if constexpr (BS == 32 && !POOL && (ERT || ALL)) {
        const long long warps = 24LL * num_sms;
        if (2 * tiles <= 3 * warps) return launch_group<DT, COMP, SHADE, BS, 8>(p, num_sms, s);
        if (tiles <= 3 * warps || (ALL && 2 * tiles <= 9 * warps))
            return launch_group<DT, COMP, SHADE, BS, 4>(p, num_sms, s);
        if constexpr (ALL) {
            if (tiles <= 8 * warps) return launch_group<DT, COMP, SHADE, BS, 2>(p, num_sms, s);
        } else if (p.queue && tiles <= 50 * warps) {
            cudaError_t e = launch_persistent(march_kernel<DT, COMP, SHADE, BS, POOL, true>, p, tiles, num_sms, s);
            if (e != cudaSuccess) return e;
            return launch_persistent(march_group_kernel<DT, COMP, SHADE, BS, 8, true>, p, tiles, num_sms, s);
        }
    }
    return launch_persistent(march_kernel<DT, COMP, SHADE, BS, POOL, false>, p, tiles, num_sms, s);
}

template <int DT, int COMP, int SHADE>
cudaError_t launch_pool(const MarchParams& p, int num_sms, cudaStream_t s) {
    // POOL: a host-resident brick pool read through the device cache's slot
    // table (and its level of detail); device-resident pools compile without it
    if (p.brick_slot) return launch_t<DT, COMP, SHADE, 0, true>(p, num_sms, s);
    return p.L.B == 32 ? launch_t<DT, COMP, SHADE, 32, false>(p, num_sms, s)
                       : launch_t<DT, COMP, SHADE, 0, false>(p, num_sms, s);
}

template <int DT, int COMP>
cudaError_t launch_sh(const MarchParams& p, int shading, int num_sms, cudaStream_t s) {
    return shading == VRC_SHADE_PHONG ? launch_pool<DT, COMP, VRC_SHADE_PHONG>(p, num_sms, s)
                                      : launch_pool<DT, COMP, VRC_SHADE_NONE>(p, num_sms, s);
}

}  // namespace
}  // namespace vrc
