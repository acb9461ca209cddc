// Volume ingest: linear VolumeRAM layout -> bricked device layout, per-brick
// min/max, and the per-(volume, TF) brick occupancy used for empty-space
// skipping.
//
// Reference behaviour this replaces / follows:
//   VolumeGL upload (linear 3D texture)       src/core/datastructures/volume/volumegl.cpp:126-168
//   per-region min/max with 1-voxel overlap   modules/base/processors/proxygeometry/optimizedproxygeometry.cpp:894-987
//   region emptiness from TF opacity          optimizedproxygeometry.cpp:878-880
// The brick test here is exact for the march: a brick is empty when every TF
// entry its trilinear samples can select has alpha 0.
#include <algorithm>
#include <cstdint>

#include "vrc_internal.h"

namespace vrc {
namespace {

// One CTA per brick (grid-stride), four stored voxels a thread and store. HBM
// is the bound (a voxel read, 1.31 written); what it took before was index
// arithmetic: two 64-bit divisions and a store per voxel. The edge is
// compile-time, so a position in the brick divides by constants, and four
// consecutive voxels span at most two rows. 512^3 u16: 1095 -> 177 us (the floor at the copy rate: 91).
template <typename T> struct SlicesOf {
    const T* base;
    int first, at, ring;
    explicit SlicesOf(const Slices& s) : base((const T*)s.base), first(s.first), at(s.at), ring(s.ring) {}
    // row y of slice z
    __device__ __forceinline__ const T* row(int z, int y, int X, int Y) const {
        int i = z - first + at;
        if (i >= ring) i -= ring;
        return base + ((long long)i * Y + y) * X;
    }
};

template <typename T, int B>
__global__ void __launch_bounds__(256) brick_build_kernel(SlicesOf<T> lin, BrickLayout L, long long b0, long long b1,
                                                          T* __restrict__ bricks) {
    constexpr int S = B + APRON_LO + APRON_HI, S2 = S * S, S3 = S2 * S;
    struct alignas(4 * sizeof(T)) Quad {
        T v[4];
    };
    const int X1 = L.dims[0] - 1, Y1 = L.dims[1] - 1, Z1 = L.dims[2] - 1;
    for (long long b = b0 + blockIdx.x; b < b1; b += gridDim.x) {
        const unsigned bu = (unsigned)b, nb0 = (unsigned)L.nb[0], nb1 = (unsigned)L.nb[1];  // fewer than 2^31 bricks
        const int x0 = (int)(bu % nb0) * B - APRON_LO, y0 = (int)(bu / nb0 % nb1) * B - APRON_LO,
                  z0 = (int)(bu / nb0 / nb1) * B - APRON_LO;
        T* out = bricks + b * L.brick_stride;
        auto row = [&](int y, int z) {
            return lin.row(min(max(z0 + z, 0), Z1), min(max(y0 + y, 0), Y1), L.dims[0], L.dims[1]);
        };
        // the last quad may reach past S^3 into the brick's padding (the stride is a multiple of 64)
        for (int i = threadIdx.x; i < (S3 + 3) / 4; i += 256) {
            const int r = 4 * i, z = r / S2, y = r % S2 / S, x = r % S;
            const T* p = row(y, z);
            const T* q = y + 1 < S ? row(y + 1, z) : row(0, z + 1);  // the row after it
            Quad o;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const bool next = x + k >= S;
                o.v[k] = __ldg((next ? q : p) + min(max(x0 + (next ? x + k - S : x + k), 0), X1));
            }
            *reinterpret_cast<Quad*>(out + r) = o;
        }
    }
}

template <typename T> __device__ __forceinline__ float raw_to_float(T v) { return (float)v; }

// Voxel (x, y, z) of a bricked volume (core voxels, no apron lookup needed).
template <typename T>
__device__ __forceinline__ T brick_voxel(const T* __restrict__ bricks, const BrickLayout& L, int x, int y, int z) {
    const int bx = x >> L.shift, by = y >> L.shift, bz = z >> L.shift;
    const long long b = ((long long)bz * L.nb[1] + by) * L.nb[0] + bx;
    return bricks[b * L.brick_stride +
                  ((z - (bz << L.shift) + APRON_LO) * L.S + (y - (by << L.shift) + APRON_LO)) * L.S +
                  (x - (bx << L.shift) + APRON_LO)];
}

// HalfSampleMean (volumeoctree.cpp:188-202) on the stored type: integers
// summed exactly, divided by 8 with truncation; floats summed in z, y, x
// order and scaled by 1/8.
template <typename T> struct HalfSum { using A = uint32_t; };
template <> struct HalfSum<float> { using A = float; };
template <typename T> __device__ __forceinline__ T half_mean(typename HalfSum<T>::A s) { return (T)(s / 8u); }
template <> __device__ __forceinline__ float half_mean<float>(float s) { return __fmul_rn(s, 0.125f); }

template <typename T>
__global__ void half_sample_kernel(const T* __restrict__ bricks, BrickLayout L, int d1x, int d1y, int d1z,
                                   T* __restrict__ out) {
    const long long total = (long long)d1x * d1y * d1z;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int x1 = (int)(i % d1x), y1 = (int)((i / d1x) % d1y), z1 = (int)(i / ((long long)d1x * d1y));
        typename HalfSum<T>::A sum = 0;
        for (int dz = 0; dz < 2; ++dz)
            for (int dy = 0; dy < 2; ++dy)
                for (int dx = 0; dx < 2; ++dx) {
                    const int x = min(2 * x1 + dx, L.dims[0] - 1), y = min(2 * y1 + dy, L.dims[1] - 1),
                              z = min(2 * z1 + dz, L.dims[2] - 1);
                    sum += (typename HalfSum<T>::A)brick_voxel(bricks, L, x, y, z);
                }
        out[i] = half_mean<T>(sum);
    }
}

// One thread per cell: min/max over the cell's voxels plus one voxel on the
// high side of every axis (clamped), i.e. the trilinear support of all
// samples whose floor voxel lies in the cell. Any cell edge and row length.
template <typename T>
__global__ void cell_minmax_kernel(SlicesOf<T> lin, int X, int Y, int Z, int C, int ncx, int ncy, long long c0,
                                   long long c1, float norm, float* cmin, float* cmax) {
    for (long long c = c0 + blockIdx.x * (long long)blockDim.x + threadIdx.x; c < c1;
         c += (long long)gridDim.x * blockDim.x) {
        const int cx = (int)(c % ncx), cy = (int)((c / ncx) % ncy), cz = (int)(c / ((long long)ncx * ncy));
        const int x0 = cx * C, y0 = cy * C, z0 = cz * C;
        const int x1 = min(x0 + C, X - 1), y1 = min(y0 + C, Y - 1), z1 = min(z0 + C, Z - 1);
        float mn = INFINITY, mx = -INFINITY;
        for (int z = z0; z <= z1; ++z)
            for (int y = y0; y <= y1; ++y) {
                const T* row = lin.row(z, y, X, Y);
                for (int x = x0; x <= x1; ++x) {
                    const float v = raw_to_float(row[x]);
                    mn = fminf(mn, v);
                    mx = fmaxf(mx, v);
                }
            }
        cmin[c] = norm > 0.f ? __fdiv_rn(mn, norm) : mn;
        cmax[c] = norm > 0.f ? __fdiv_rn(mx, norm) : mx;
    }
}

__device__ __forceinline__ unsigned min2(unsigned a, unsigned b) {
    unsigned r;
    asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ unsigned max2(unsigned a, unsigned b) {
    unsigned r;
    asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// Running min/max of 9 consecutive voxels of several rows: integers as pairs
// of 16 bits, floats one by one.
template <typename T> struct Run9 {
    unsigned mn[5], mx[5];  // voxels (0, 1) (2, 3) (4, 5) (6, 7) (8, 8)
    __device__ __forceinline__ void begin() {
        for (int i = 0; i < 5; ++i) mn[i] = 0xffffffffu, mx[i] = 0u;
    }
    __device__ __forceinline__ void add(const T* __restrict__ row, int x0, int x8) {
        unsigned v[5];
        if (sizeof(T) == 2) {
            const uint4 q = __ldg(reinterpret_cast<const uint4*>(row + x0));
            v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
        } else {
            const uint2 q = __ldg(reinterpret_cast<const uint2*>(row + x0));
            v[0] = __byte_perm(q.x, 0, 0x4140), v[1] = __byte_perm(q.x, 0, 0x4342);
            v[2] = __byte_perm(q.y, 0, 0x4140), v[3] = __byte_perm(q.y, 0, 0x4342);
        }
        const unsigned last = __ldg(row + x8);
        v[4] = last | last << 16;
#pragma unroll
        for (int i = 0; i < 5; ++i) mn[i] = min2(mn[i], v[i]), mx[i] = max2(mx[i], v[i]);
    }
    // voxels 2i, 2i + 1, 2i + 2
    __device__ __forceinline__ float lo(int i) const {
        return (float)min(min(mn[i] & 0xffffu, mn[i] >> 16), mn[i + 1] & 0xffffu);
    }
    __device__ __forceinline__ float hi(int i) const {
        return (float)max(max(mx[i] & 0xffffu, mx[i] >> 16), mx[i + 1] & 0xffffu);
    }
};
template <> struct Run9<float> {
    float mn[9], mx[9];
    __device__ __forceinline__ void begin() {
        for (int i = 0; i < 9; ++i) mn[i] = INFINITY, mx[i] = -INFINITY;
    }
    __device__ __forceinline__ void add(const float* __restrict__ row, int x0, int x8) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(row + x0)),
                     b = __ldg(reinterpret_cast<const float4*>(row + x0 + 4));
        const float v[9] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, __ldg(row + x8)};
#pragma unroll
        for (int i = 0; i < 9; ++i) mn[i] = fminf(mn[i], v[i]), mx[i] = fmaxf(mx[i], v[i]);
    }
    __device__ __forceinline__ float lo(int i) const { return fminf(fminf(mn[2 * i], mn[2 * i + 1]), mn[2 * i + 2]); }
    __device__ __forceinline__ float hi(int i) const { return fmaxf(fmaxf(mx[2 * i], mx[2 * i + 1]), mx[2 * i + 2]); }
};

// The 2^3 cells of volumes whose rows are multiples of 8 voxels (and start on
// 16 bytes): four cells a thread from nine rows of 8 + 1 voxels, one wide load
// a row, integers compared as pairs. HBM is the bound (the volume read, two
// floats a cell written). 512^3 u16: 480 -> 82 us (floor: 59).
template <typename T>
__global__ void __launch_bounds__(256) cell2_minmax_kernel(SlicesOf<T> lin, int X, int Y, int Z, int ncy, unsigned g0,
                                                           unsigned g1, float norm, float* __restrict__ cmin,
                                                           float* __restrict__ cmax) {
    const unsigned gx = (unsigned)X / 8u;
    for (unsigned long long i = g0 + blockIdx.x * 256ull + threadIdx.x; i < g1; i += gridDim.x * 256ull) {
        const unsigned r = (unsigned)i / gx;
        const int x0 = (int)((unsigned)i - r * gx) * 8, y0 = 2 * (int)(r % (unsigned)ncy), z0 = 2 * (int)(r / (unsigned)ncy);
        const int x8 = min(x0 + 8, X - 1);
        Run9<T> run;
        run.begin();
#pragma unroll
        for (int dz = 0; dz < 3; ++dz)
#pragma unroll
            for (int dy = 0; dy < 3; ++dy)
                run.add(lin.row(min(z0 + dz, Z - 1), min(y0 + dy, Y - 1), X, Y), x0, x8);
        float4 mn = make_float4(run.lo(0), run.lo(1), run.lo(2), run.lo(3));
        float4 mx = make_float4(run.hi(0), run.hi(1), run.hi(2), run.hi(3));
        if (norm > 0.f) {
            mn = make_float4(__fdiv_rn(mn.x, norm), __fdiv_rn(mn.y, norm), __fdiv_rn(mn.z, norm), __fdiv_rn(mn.w, norm));
            mx = make_float4(__fdiv_rn(mx.x, norm), __fdiv_rn(mx.y, norm), __fdiv_rn(mx.z, norm), __fdiv_rn(mx.w, norm));
        }
        reinterpret_cast<float4*>(cmin)[i] = mn;
        reinterpret_cast<float4*>(cmax)[i] = mx;
    }
}

// Min/max of cells of F times the edge from their F^3 cells: each of those
// covers its voxels and one more on the high side, so together they cover the
// larger cell and one voxel on its high side, and the normalisation is
// monotone -- the values are those of a pass over the voxels. Reading the
// volume again for each level took 567 us at 512^3 u16 and the bricks another
// 412; the chain takes 35 us.
template <int F>
__global__ void coarser_minmax_kernel(const float* __restrict__ fmin, const float* __restrict__ fmax, int fx, int fy, int fz,
                                      int ncx, int ncy, long long ncells, float* __restrict__ cmin,
                                      float* __restrict__ cmax) {
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncells;
         c += (long long)gridDim.x * blockDim.x) {
        const unsigned cu = (unsigned)c;  // below 2^32 cells
        const int cx = (int)(cu % (unsigned)ncx), cy = (int)(cu / (unsigned)ncx % (unsigned)ncy),
                  cz = (int)(cu / (unsigned)ncx / (unsigned)ncy);
        float mn = INFINITY, mx = -INFINITY;
#pragma unroll
        for (int dz = 0; dz < F; ++dz)
#pragma unroll
            for (int dy = 0; dy < F; ++dy) {
                const long long row = ((long long)min(F * cz + dz, fz - 1) * fy + min(F * cy + dy, fy - 1)) * fx;
#pragma unroll
                for (int dx = 0; dx < F; ++dx) {
                    const long long i = row + min(F * cx + dx, fx - 1);
                    mn = fminf(mn, __ldg(fmin + i));
                    mx = fmaxf(mx, __ldg(fmax + i));
                }
            }
        cmin[c] = mn;
        cmax[c] = mx;
    }
}

// As the march (march_core.cuh: rw_to_tf, tf_index).
__device__ __forceinline__ float rw_to_tf(float rw, float lo, float hi, float rcp) {
    if (rcp != 0.f) {
        const float a = __fsub_rn(fminf(fmaxf(rw, lo), hi), lo), b = __fsub_rn(hi, lo);
        float q = __fmul_rn(a, rcp);
        q = __fmaf_rn(__fmaf_rn(-q, b, a), rcp, q);
        return __fmaf_rn(__fmaf_rn(-q, b, a), rcp, q);
    }
    if (rw < lo) return 0.f;
    if (rw > hi) return 1.f;
    if (lo == hi) return 0.f;
    return __fdiv_rn(__fsub_rn(rw, lo), __fsub_rn(hi, lo));
}
__device__ __forceinline__ int tf_index(float x, int w) { return (int)__fadd_rn(__fmul_rn(x, (float)(w - 1)), 0.5f); }

// Bit c of the map is set if any TF entry with index in
// [idx(min_c) - 1, idx(max_c) + 1] has alpha > 0 (alpha_prefix[i] = number of
// entries below i with alpha > 0). HBM is the bound: the two tables, 8 bytes a
// cell. One lane per cell, a ballot per word, four words a warp at a time; a
// thread per word read 32 cells in a row each, 128 bytes apart across the
// warp (512^3 at 2^3 cells: 141 -> 40 us; floor: 20).
__global__ void __launch_bounds__(256) occupancy_kernel(const float* __restrict__ bmin, const float* __restrict__ bmax,
                                                        long long n, const int* __restrict__ prefix, int w, float rs,
                                                        float ro, float lo, float hi, float rcp, uint32_t* occ) {
    const int lane = threadIdx.x & 31;
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long base = (blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5)) * 128; base < n;
         base += warps * 128) {
        float mn[4], mx[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const long long c = base + 32 * j + lane;
            mn[j] = c < n ? __ldg(bmin + c) : INFINITY;
            mx[j] = c < n ? __ldg(bmax + c) : INFINITY;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float r0 = __fadd_rn(__fmul_rn(mn[j], rs), ro), r1 = __fadd_rn(__fmul_rn(mx[j], rs), ro);
            const int i0 = max(tf_index(rw_to_tf(fminf(r0, r1), lo, hi, rcp), w) - 1, 0);
            const int i1 = min(tf_index(rw_to_tf(fmaxf(r0, r1), lo, hi, rcp), w) + 1, w - 1);
            const bool visible = base + 32 * j + lane < n && __ldg(prefix + i1 + 1) - __ldg(prefix + i0) > 0;
            const uint32_t bits = __ballot_sync(0xffffffffu, visible);
            if (lane == j && base + 32 * j < n) occ[(base >> 5) + j] = bits;
        }
    }
}

// Chebyshev distance to the nearest occupied cell, capped at OCC_DIST_CAP:
// d(c) = min over occupied o of max(|cx-ox|, |cy-oy|, |cz-oz|). The max of
// the axis offsets composes per axis, so three passes give it exactly:
// along x the distance to the nearest occupied cell of the row, then along
// y and along z the min over offsets k of max(|k|, previous pass at c + k).
// Offsets beyond the cap only give values above it, so each pass looks at
// |k| < OCC_DIST_CAP. Of small maps, where the scratch is short and for caps
// other than 16 (others: the bit planes below). Four cells of a row a thread; a word of four bytes a
// load where rows are multiples of four cells (WORDS), else bytes.
//
// Along x: the row's bits from 16 below the four cells to 47 above them in one
// 64-bit window, the distances by counting zeros (caps above 16: cell by cell).
// 512^3 at 2^3 cells: 332 -> 26 us (up to 32 loads a cell before).
template <bool WORDS>
__global__ void __launch_bounds__(256) occ_dist_x_kernel(const uint32_t* __restrict__ occ, int nx, int ny, int nz,
                                                         uint8_t* __restrict__ out) {
    const unsigned nx4 = ((unsigned)nx + 3u) / 4u;
    const unsigned long long total = (unsigned long long)nx4 * ny * nz;
    const long long nwords = ((long long)nx * ny * nz + 31) / 32;
    for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < total; i += gridDim.x * 256ull) {
        const unsigned row = (unsigned)i / nx4;
        const int x = (int)((unsigned)i - row * nx4) * 4;
        const long long first = (long long)row * nx, c = first + x;
        uint32_t d = 0;
        if (OCC_DIST_CAP <= 16) {
            const long long s = c - 16, w0 = s >> 5;
            const int sh = (int)(s & 31);
            const uint32_t a = w0 >= 0 ? __ldg(occ + w0) : 0u;
            const uint32_t b = w0 + 1 >= 0 && w0 + 1 < nwords ? __ldg(occ + w0 + 1) : 0u;
            const uint32_t e = w0 + 2 < nwords ? __ldg(occ + w0 + 2) : 0u;
            unsigned long long win = (unsigned long long)__funnelshift_r(b, e, sh) << 32 | __funnelshift_r(a, b, sh);
            if (x < 16) win &= ~0ull << (16 - x);                       // bits of the row before
            if (nx - x < 48) win &= (1ull << (nx - x + 16)) - 1ull;  // ... and after
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const unsigned below = (unsigned)__clzll((long long)(win << (47 - j)));
                const unsigned above = (unsigned)__ffsll((long long)(win >> (16 + j))) - 1u;  // none: 2^32 - 1
                d |= min(min(below, above), (unsigned)OCC_DIST_CAP) << (8 * j);
            }
        } else {
            for (int j = 0; j < 4 && x + j < nx; ++j) {
                int v = OCC_DIST_CAP;
                for (int k = 0; k < v; ++k) {
                    const long long lo = x + j - k >= 0 ? c + j - k : -1, hi = x + j + k < nx ? c + j + k : -1;
                    if ((lo >= 0 && (__ldg(occ + (lo >> 5)) >> (lo & 31)) & 1u) ||
                        (hi >= 0 && (__ldg(occ + (hi >> 5)) >> (hi & 31)) & 1u))
                        v = k;
                }
                d |= (uint32_t)v << (8 * j);
            }
        }
        if (WORDS) {
            *reinterpret_cast<uint32_t*>(out + c) = d;
        } else {
            for (int j = 0; j < 4 && x + j < nx; ++j) out[c + j] = (uint8_t)(d >> (8 * j));
        }
    }
}

// Along y (AXIS 1) or z (AXIS 2): the four cells as two pairs of 16 bits, min
// and max a pair at a time, up to STEP offsets' loads in flight on both sides;
// a thread stops once no offset can lower one of its cells. 512^3 at 2^3
// cells: 233 + 220 -> 66 + 72 us for the two passes (a byte load, a min and a max
// a cell and offset before).
template <int AXIS, bool WORDS>
__global__ void __launch_bounds__(256) occ_dist_axis_kernel(const uint8_t* __restrict__ in, int nx, int ny, int nz,
                                                            uint8_t* __restrict__ out) {
    constexpr int STEP = 5;
    const unsigned nx4 = ((unsigned)nx + 3u) / 4u;
    const unsigned long long total = (unsigned long long)nx4 * ny * nz;
    const long long stride = AXIS == 1 ? nx : (long long)nx * ny;
    const int len = AXIS == 1 ? ny : nz;
    for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < total; i += gridDim.x * 256ull) {
        const unsigned row = (unsigned)i / nx4;
        const int x = (int)((unsigned)i - row * nx4) * 4, cells = min(nx - x, 4);
        const int pos = AXIS == 1 ? (int)(row % (unsigned)ny) : (int)(row / (unsigned)ny);
        const uint8_t* p = in + (long long)row * nx + x;
        auto load = [&](const uint8_t* q) -> uint32_t {
            if (WORDS) return __ldg(reinterpret_cast<const uint32_t*>(q));
            uint32_t v = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j < cells) v |= (uint32_t)__ldg(q + j) << (8 * j);
            return v;
        };
        const uint32_t v0 = load(p);
        unsigned a = __byte_perm(v0, 0, 0x4140), b = __byte_perm(v0, 0, 0x4342);
        for (int k0 = 1; k0 < OCC_DIST_CAP; k0 += STEP) {
            const unsigned m = max2(a, b);
            if ((int)max(m & 0xffffu, m >> 16) <= k0) break;
            uint32_t lo[STEP], hi[STEP];
#pragma unroll
            for (int j = 0; j < STEP; ++j) {  // beyond the grid, or the cap: nothing
                const int k = k0 + j;
                lo[j] = k < OCC_DIST_CAP && pos - k >= 0 ? load(p - k * stride) : 0xffffffffu;
                hi[j] = k < OCC_DIST_CAP && pos + k < len ? load(p + k * stride) : 0xffffffffu;
            }
#pragma unroll
            for (int j = 0; j < STEP; ++j) {
                const unsigned kk = (unsigned)(k0 + j) * 0x10001u;
                a = min2(a, max2(kk, min2(__byte_perm(lo[j], 0, 0x4140), __byte_perm(hi[j], 0, 0x4140))));
                b = min2(b, max2(kk, min2(__byte_perm(lo[j], 0, 0x4342), __byte_perm(hi[j], 0, 0x4342))));
            }
        }
        const uint32_t d = __byte_perm(a, b, 0x6420);
        uint8_t* q = out + (long long)row * nx + x;
        if (WORDS) {
            *reinterpret_cast<uint32_t*>(q) = d;
        } else {
            for (int j = 0; j < cells; ++j) q[j] = (uint8_t)(d >> (8 * j));
        }
    }
}

// The same map from bit planes, 32 cells a word. The box of radius r around a
// cell holds an occupied cell or not: one bit, and a cell's distance is the
// number of radii 0 .. 15 whose bit is 0. The bits of radius r are the occupancy
// dilated by r along each axis, shifts and ORs of words instead of a min and a
// max a pair of cells and offset.
constexpr int DIST_PLANES = 16;

// Word i of row y (cells 32 i ..) with 16 cells on either side as 64 bits: the OR
// of rows y - r .. y + r takes in two rows a step; along x, a union of shifts by
// s of a run of c cells each way, s at most 2 c + 1, is one of c + s. A CTA takes
// 8 words of 32 rows and has their and the 30 rows' windows beside them in shared
// memory. Planes [r][z][y][i], rows padded to words. Issue slots bound it, some
// 25 a plane. 512^3 at 2^3 cells: x and y 92 -> 15.5 us (each row's window
// made anew by each of the 31 threads that take it: 45).
constexpr int PLANE_WORDS = 8, PLANE_ROWS = 32;
__global__ void __launch_bounds__(256) occ_planes_xy_kernel(const uint32_t* __restrict__ occ, int nx, int ny, int nz, int tiles_x,
                                                            int tiles_y, uint32_t* __restrict__ planes) {
    constexpr int REACH = DIST_PLANES - 1, ROWS = PLANE_ROWS + 2 * REACH;
    __shared__ unsigned long long win[ROWS][PLANE_WORDS];
    const int nw = (nx + 31) / 32;
    const size_t plane = (size_t)nw * ny * nz;
    const long long last = ((long long)nx * ny * nz + 31) / 32 - 1;
    const int lane = threadIdx.x % PLANE_WORDS, row = threadIdx.x / PLANE_WORDS;
    const long long tiles = (long long)tiles_x * tiles_y * nz;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int i = (int)(t % tiles_x) * PLANE_WORDS + lane, y0 = (int)(t / tiles_x % tiles_y) * PLANE_ROWS;
        const int z = (int)(t / tiles_x / tiles_y), x = i * 32;
        // beside the row (and, at either end of the map, a clamped word's bits): nothing
        const unsigned long long mask = (x == 0 ? ~0xffffull : ~0ull) & (nx - x < 48 ? (1ull << (nx - x + 16)) - 1ull : ~0ull);
        for (int k = row; k < ROWS; k += PLANE_ROWS) {
            const int y = y0 + k - REACH;
            unsigned long long v = 0;
            if (i < nw && (unsigned)y < (unsigned)ny) {
                const long long s = ((long long)z * ny + y) * nx + x - 16, w = s >> 5;
                const int sh = (int)(s & 31);
                const uint32_t a = __ldg(occ + max(w, 0ll)), b = __ldg(occ + min(w + 1, last)), c = __ldg(occ + min(w + 2, last));
                v = ((unsigned long long)__funnelshift_r(b, c, sh) << 32 | __funnelshift_r(a, b, sh)) & mask;
            }
            win[k][lane] = v;
        }
        __syncthreads();
        if (i < nw && y0 + row < ny) {
            uint32_t* out = planes + ((size_t)z * ny + y0 + row) * nw + i;
            unsigned long long col = 0;
#pragma unroll
            for (int r = 0; r < DIST_PLANES; ++r, out += plane) {
                col |= win[row + REACH - r][lane] | win[row + REACH + r][lane];
                unsigned long long v = col;
#pragma unroll
                for (int c = 0; c < r;) {
                    const int s = 2 * c + 1 < r - c ? 2 * c + 1 : r - c;
                    v |= v << s | v >> s;
                    c += s;
                }
                *out = (uint32_t)(v >> 16);
            }
        }
        __syncthreads();
    }
}

// Bits i .. i + 3 of w, one to a byte.
__device__ __forceinline__ uint32_t bits_to_bytes(uint32_t w, int i) {
    return ((w >> i & 0xfu) * 0x00204081u) & 0x01010101u;
}

// Along z: a CTA takes 32 words of 8 slices. Warp g ORs the windows of radii g
// and 15 - g, together the same work for every warp, from the words that the
// eight windows share and the runs on either side of them; then it takes slice
// g. A distance's bit s is the parity of the radii r with 2^s dividing r + 1
// whose bit is 0. Bytes leave 16 at a time, or (WIDE false: rows that are no
// multiple of 16 cells) by way of shared memory, a word's 32 cells a store.
// Bound by L2 and by latency. 512^3 at 2^3 cells: z 72 -> 21 us; 500^3: 141 -> 33
// (all radii one after another in a thread: 33 and 130).
constexpr int PLANES_Z = 8;
template <bool WIDE>
__global__ void __launch_bounds__(256) occ_planes_z_kernel(const uint32_t* __restrict__ planes, int nx, int ny, int nz,
                                                           uint8_t* __restrict__ out) {
    __shared__ uint32_t hit[PLANES_Z][DIST_PLANES][32];
    const unsigned nw = ((unsigned)nx + 31u) / 32u, slice = nw * (unsigned)ny, chunks = (slice + 31u) / 32u;
    const unsigned tiles = chunks * (((unsigned)nz + PLANES_Z - 1) / PLANES_Z);
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    for (unsigned t = blockIdx.x; t < tiles; t += gridDim.x) {
        const unsigned at = t % chunks * 32u + lane;
        const int z0 = (int)(t / chunks) * PLANES_Z;
        if (at < slice) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int r = half ? DIST_PLANES - 1 - g : g;
                const uint32_t* p = planes + (size_t)r * slice * nz + at;
                auto word = [&](int z) { return (unsigned)z < (unsigned)nz ? __ldg(p + (size_t)z * slice) : 0u; };
                uint32_t o[PLANES_Z];
                if (half || r >= PLANES_Z / 2) {
                    uint32_t lo[PLANES_Z], hi[PLANES_Z];  // of slices j .. 6, and of 2 r + 1 .. 2 r + j
#pragma unroll
                    for (int j = 0; j < PLANES_Z - 1; ++j) {
                        lo[j] = word(z0 - r + j);
                        hi[j + 1] = word(z0 + r + 1 + j);
                    }
                    uint32_t all = 0;
#pragma unroll 8
                    for (int k = PLANES_Z - 1; k <= 2 * r; ++k) all |= word(z0 - r + k);
                    lo[PLANES_Z - 1] = hi[0] = 0;
#pragma unroll
                    for (int j = PLANES_Z - 2; j >= 0; --j) lo[j] |= lo[j + 1];
#pragma unroll
                    for (int j = 0; j < PLANES_Z; ++j) {
                        if (j) hi[j] |= hi[j - 1];
                        o[j] = all | lo[j] | hi[j];
                    }
                } else {  // the windows need not overlap
#pragma unroll
                    for (int j = 0; j < PLANES_Z; ++j) o[j] = 0;
#pragma unroll
                    for (int k = 0; k < 2 * PLANES_Z - 2; ++k) {
                        const uint32_t w = k < PLANES_Z + 2 * r ? word(z0 - r + k) : 0u;
#pragma unroll
                        for (int j = 0; j < PLANES_Z; ++j)
                            if (j <= k) o[j] |= k <= j + 2 * r ? w : 0u;
                    }
                }
#pragma unroll
                for (int j = 0; j < PLANES_Z; ++j) hit[j][r][lane] = o[j];
            }
        }
        __syncthreads();
        const int z = z0 + g;
        if (z < nz) {
            uint32_t d[5] = {}, b[8];
            if (at < slice) {
#pragma unroll
                for (int r = 0; r < DIST_PLANES; ++r) {
                    const uint32_t o = hit[g][r][lane];
#pragma unroll
                    for (int s = 0; s < 5; ++s)
                        if ((r + 1) % (1 << s) == 0) d[s] ^= o;
                }
            }
            d[4] = ~d[4];  // one radius; the others have an even number of them
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                b[i] = 0;
#pragma unroll
                for (int s = 0; s < 5; ++s) b[i] += bits_to_bytes(d[s], 4 * i) << s;
            }
            uint8_t* q = out + (size_t)z * ny * nx;
            if (WIDE) {
                const unsigned y = at / nw;
                const int x = (int)(at - y * nw) * 32;
                if (at < slice) {
                    uint4* q16 = reinterpret_cast<uint4*>(q + (size_t)y * nx + x);
                    q16[0] = make_uint4(b[0], b[1], b[2], b[3]);
                    if (nx - x > 16) q16[1] = make_uint4(b[4], b[5], b[6], b[7]);
                }
            } else {
                uint32_t* stage = &hit[g][0][0];  // this warp's slice, read
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i) stage[lane * 9 + i] = b[i];
                __syncwarp();
                const unsigned first = at - lane, words = min(32u, slice - first);
                unsigned y = first / nw, i = first - y * nw;
                for (unsigned k = 0; k < words; ++k) {
                    const int x = (int)i * 32 + lane;
                    if (x < nx) q[(size_t)y * nx + x] = reinterpret_cast<const uint8_t*>(stage + k * 9)[lane];
                    if (++i == nw) { i = 0; ++y; }
                }
            }
        }
        __syncthreads();
    }
}

// Maps of fewer words keep the passes: level with them (32^3 cells 9.9 us against
// 11.3, 48^3 10.5 against 12) and the planes want 64 bytes of scratch a word.
// 128^3 cells 13 us against 30, 256^3 37 against 164, 250^3 48 against 303.
constexpr long long PLANES_MIN_WORDS = 4096;

int grid_for(long long n, int block) {
    long long g = (n + block - 1) / block;
    if (g > 152LL * 64) g = 152LL * 64;
    if (g < 1) g = 1;
    return (int)g;
}

}  // namespace

// One CTA per cached brick: 16-byte copies from the (host-resident) pool.
// One CTA per cached brick; four 16-byte loads in flight per thread, since
// the source is host memory read over the C2C link.
__global__ void brick_gather_kernel(const uint4* __restrict__ pool, const long long* __restrict__ ids,
                                    const long long* __restrict__ slots, long long words, uint4* __restrict__ cache) {
    const uint4* src = pool + ids[blockIdx.x] * words;
    uint4* dst = cache + slots[blockIdx.x] * words;
    long long i = threadIdx.x;
    for (; i + 3 * blockDim.x < words; i += 4 * blockDim.x) {
        const uint4 a = src[i], b = src[i + blockDim.x], c = src[i + 2 * blockDim.x], d = src[i + 3 * blockDim.x];
        dst[i] = a;
        dst[i + blockDim.x] = b;
        dst[i + 2 * blockDim.x] = c;
        dst[i + 3 * blockDim.x] = d;
    }
    for (; i < words; i += blockDim.x) dst[i] = src[i];
}

cudaError_t launch_brick_gather(const void* pool, const long long* ids, const long long* dst, long long n,
                                size_t brick_stride_bytes, void* cache, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (n > 0x7fffffffLL || brick_stride_bytes % 16) return cudaErrorInvalidValue;
    brick_gather_kernel<<<(unsigned)n, 256, 0, s>>>(static_cast<const uint4*>(pool), ids, dst,
                                                    (long long)(brick_stride_bytes / 16), static_cast<uint4*>(cache));
    return cudaGetLastError();
}

template <typename T>
static cudaError_t brick_build_t(const Slices& lin, const BrickLayout& L, int layer0, int layer1, T* bricks, cudaStream_t s) {
    const SlicesOf<T> v(lin);
    const long long layer = (long long)L.nb[0] * L.nb[1], b0 = layer0 * layer, b1 = layer1 * layer;
    const unsigned g = (unsigned)std::min<long long>(b1 - b0, 1 << 20);
    switch (L.B) {
        case 8: brick_build_kernel<T, 8><<<g, 256, 0, s>>>(v, L, b0, b1, bricks); break;
        case 16: brick_build_kernel<T, 16><<<g, 256, 0, s>>>(v, L, b0, b1, bricks); break;
        case 32: brick_build_kernel<T, 32><<<g, 256, 0, s>>>(v, L, b0, b1, bricks); break;
        case 64: brick_build_kernel<T, 64><<<g, 256, 0, s>>>(v, L, b0, b1, bricks); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_brick_build(const Slices& linear, int dtype, const BrickLayout& L, int layer0, int layer1, void* bricks,
                               cudaStream_t s) {
    switch (dtype) {
        case VRC_U8: return brick_build_t(linear, L, layer0, layer1, (uint8_t*)bricks, s);
        case VRC_U16: return brick_build_t(linear, L, layer0, layer1, (uint16_t*)bricks, s);
        default: return brick_build_t(linear, L, layer0, layer1, (float*)bricks, s);
    }
}

cudaError_t launch_half_sample(const void* bricks, int dtype, const BrickLayout& L, const int dims1[3], void* out,
                               cudaStream_t s) {
    const long long total = (long long)dims1[0] * dims1[1] * dims1[2];
    const int g = grid_for(total, 256);
    switch (dtype) {
        case VRC_U8:
            half_sample_kernel<uint8_t><<<g, 256, 0, s>>>((const uint8_t*)bricks, L, dims1[0], dims1[1], dims1[2],
                                                          (uint8_t*)out);
            break;
        case VRC_U16:
            half_sample_kernel<uint16_t><<<g, 256, 0, s>>>((const uint16_t*)bricks, L, dims1[0], dims1[1], dims1[2],
                                                           (uint16_t*)out);
            break;
        default:
            half_sample_kernel<float><<<g, 256, 0, s>>>((const float*)bricks, L, dims1[0], dims1[1], dims1[2],
                                                        (float*)out);
            break;
    }
    return cudaGetLastError();
}

template <typename T>
static cudaError_t cell_minmax_t(const Slices& lin, const int d[3], int C, int cz0, int cz1, float norm, float* cmin,
                                 float* cmax, cudaStream_t s) {
    const int ncx = (d[0] + C - 1) / C, ncy = (d[1] + C - 1) / C;
    const long long layer = (long long)ncx * ncy, c0 = cz0 * layer, c1 = cz1 * layer;
    const SlicesOf<T> v(lin);
    if (C == 2 && d[0] % 8 == 0 && reinterpret_cast<uintptr_t>(lin.base) % 16 == 0)
        cell2_minmax_kernel<T><<<grid_for((c1 - c0) / 4, 256), 256, 0, s>>>(v, d[0], d[1], d[2], ncy, (unsigned)(c0 / 4),
                                                                            (unsigned)(c1 / 4), norm, cmin, cmax);
    else
        cell_minmax_kernel<T><<<grid_for(c1 - c0, 128), 128, 0, s>>>(v, d[0], d[1], d[2], C, ncx, ncy, c0, c1, norm, cmin, cmax);
    return cudaGetLastError();
}

cudaError_t launch_cell_minmax(const Slices& linear, int dtype, const int d[3], int C, int cz0, int cz1, float* cmin,
                               float* cmax, cudaStream_t s) {
    switch (dtype) {
        case VRC_U8: return cell_minmax_t<uint8_t>(linear, d, C, cz0, cz1, 255.f, cmin, cmax, s);
        case VRC_U16: return cell_minmax_t<uint16_t>(linear, d, C, cz0, cz1, 65535.f, cmin, cmax, s);
        default: return cell_minmax_t<float>(linear, d, C, cz0, cz1, 0.f, cmin, cmax, s);
    }
}

cudaError_t launch_coarser_minmax(const float* fmin, const float* fmax, const int fnc[3], int factor, const int nc[3],
                                  float* cmin, float* cmax, cudaStream_t s) {
    const long long n = (long long)nc[0] * nc[1] * nc[2];
    const int g = grid_for(n, 128);
    if (factor == 2)
        coarser_minmax_kernel<2><<<g, 128, 0, s>>>(fmin, fmax, fnc[0], fnc[1], fnc[2], nc[0], nc[1], n, cmin, cmax);
    else if (factor == 4)
        coarser_minmax_kernel<4><<<g, 128, 0, s>>>(fmin, fmax, fnc[0], fnc[1], fnc[2], nc[0], nc[1], n, cmin, cmax);
    else
        return cudaErrorInvalidValue;
    return cudaGetLastError();
}

cudaError_t launch_occupancy(const float* bmin, const float* bmax, long long ncells, const int* alpha_prefix,
                             int tf_width, float rwm_scale, float rwm_offset, float tf_lo, float tf_hi,
                             uint32_t* occ, cudaStream_t s) {
    occupancy_kernel<<<grid_for((ncells + 3) / 4, 256), 256, 0, s>>>(bmin, bmax, ncells, alpha_prefix, tf_width, rwm_scale,
                                                                     rwm_offset, tf_lo, tf_hi,
                                                                     tf_reciprocal(tf_lo, tf_hi), occ);
    return cudaGetLastError();
}

// The planes' words, and whether they gain.
static long long plane_words(const int nc[3]) { return (long long)((nc[0] + 31) / 32) * nc[1] * nc[2]; }
size_t occ_distance_scratch(const int nc[3]) {
    const long long words = plane_words(nc);
    if (OCC_DIST_CAP != DIST_PLANES || words < PLANES_MIN_WORDS || words >= (1ll << 28)) return 0;
    return (size_t)words * 4 * DIST_PLANES;
}
static bool takes_planes(const int nc[3], size_t tmp_bytes) {
    const size_t need = occ_distance_scratch(nc);
    return need && tmp_bytes >= need;
}
int occ_distance_launches(const int nc[3], size_t tmp_bytes) { return takes_planes(nc, tmp_bytes) ? 2 : 3; }

cudaError_t launch_occ_distance(const uint32_t* occ, const int nc[3], uint8_t* dist, uint8_t* tmp, size_t tmp_bytes,
                                cudaStream_t s) {
    if (takes_planes(nc, tmp_bytes) && reinterpret_cast<uintptr_t>(tmp) % 4 == 0) {
        uint32_t* planes = reinterpret_cast<uint32_t*>(tmp);
        const int nw = (nc[0] + 31) / 32, tx = (nw + PLANE_WORDS - 1) / PLANE_WORDS, ty = (nc[1] + PLANE_ROWS - 1) / PLANE_ROWS;
        occ_planes_xy_kernel<<<grid_for((long long)tx * ty * nc[2], 1), 256, 0, s>>>(occ, nc[0], nc[1], nc[2], tx, ty, planes);
        const int gz = grid_for(((long long)nw * nc[1] + 31) / 32 * ((nc[2] + PLANES_Z - 1) / PLANES_Z), 1);
        if ((reinterpret_cast<uintptr_t>(dist) | (uintptr_t)nc[0]) % 16 == 0)
            occ_planes_z_kernel<true><<<gz, 256, 0, s>>>(planes, nc[0], nc[1], nc[2], dist);
        else
            occ_planes_z_kernel<false><<<gz, 256, 0, s>>>(planes, nc[0], nc[1], nc[2], dist);
        return cudaGetLastError();
    }
    const int g = grid_for((long long)((nc[0] + 3) / 4) * nc[1] * nc[2], 256);
    const bool words = nc[0] % 4 == 0 && reinterpret_cast<uintptr_t>(dist) % 4 == 0 && reinterpret_cast<uintptr_t>(tmp) % 4 == 0;
    if (words) {
        occ_dist_x_kernel<true><<<g, 256, 0, s>>>(occ, nc[0], nc[1], nc[2], dist);
        occ_dist_axis_kernel<1, true><<<g, 256, 0, s>>>(dist, nc[0], nc[1], nc[2], tmp);
        occ_dist_axis_kernel<2, true><<<g, 256, 0, s>>>(tmp, nc[0], nc[1], nc[2], dist);
    } else {
        occ_dist_x_kernel<false><<<g, 256, 0, s>>>(occ, nc[0], nc[1], nc[2], dist);
        occ_dist_axis_kernel<1, false><<<g, 256, 0, s>>>(dist, nc[0], nc[1], nc[2], tmp);
        occ_dist_axis_kernel<2, false><<<g, 256, 0, s>>>(tmp, nc[0], nc[1], nc[2], dist);
    }
    return cudaGetLastError();
}

}  // namespace vrc
