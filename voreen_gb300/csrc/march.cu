// Frame-level launch dispatch of the ray march (one translation unit per
// compositing family: march_dvr.cu, march_mip_iso.cu, march_mop_mida.cu,
// march_first_hit.cu), the analytic entry/exit kernel and the batched
// persistent render.
#include "march_core.cuh"

namespace vrc {
namespace {

__global__ void entry_exit_kernel(MarchParams P, float4* entry, float4* exitp) {
    const int px = blockIdx.x * blockDim.x + threadIdx.x, py = blockIdx.y;
    if (px >= P.W) return;
    float4 e, l;
    analytic_entry_exit(P, px, py, e, l);
    entry[(size_t)py * P.W + px] = e;
    exitp[(size_t)py * P.W + px] = l;
}

}  // namespace

cudaError_t launch_march(const MarchParams& p, int dtype, int compositing, int shading, int num_sms,
                         cudaStream_t s) {
    switch (compositing) {
        case VRC_MIP:
        case VRC_ISO: return launch_march_mip_iso(p, dtype, compositing, shading, num_sms, s);
        case VRC_MOP:
        case VRC_MIDA: return launch_march_mop_mida(p, dtype, compositing, shading, num_sms, s);
        case VRC_FHP:
        case VRC_FHN: return launch_march_first_hit(p, dtype, compositing, num_sms, s);
        default: return launch_march_dvr(p, dtype, shading, num_sms, s);
    }
}

cudaError_t launch_entry_exit(const MarchParams& p, float4* entry, float4* exitp, cudaStream_t s) {
    dim3 grid((p.W + 127) / 128, p.H);
    entry_exit_kernel<<<grid, 128, 0, s>>>(p, entry, exitp);
    return cudaGetLastError();
}

}  // namespace vrc

// ---- batched persistent render ------------------------------------------
// Many requests (uneven volumes, dtypes, image sizes) in one persistent
// launch: warps claim ray tiles from a global counter over the concatenated
// tile lists (requests ordered by dtype, then longest first), copy the request's parameters
// into shared memory when they move to another request, and march with the
// request's dtype. Per-request completion times are stamped with the global
// timer (state layout: [0] tile counter, [1] start ns, [2] samples,
// [3 + r] request r's last tile completion ns).
//
// Issue slots bound it (48 % active at 21 of 32 lanes), and what it spent them
// on beside the march: the three dtypes' loops inlined in one body spilled 284
// bytes at 80 registers, a fence and an atomic per tile to stamp its time, and
// parameters read from shared memory. So each dtype marches in a function of
// its own (its registers are its own, and it knows that the parameters lie in
// shared memory), a warp stamps a request when it leaves it, and the requests
// are grouped by dtype. 64 mixed requests: 11.03 -> 9.15 ms.
namespace vrc {
namespace {

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__global__ void batch_begin_kernel(unsigned long long* state, int nreq) {
    for (int i = threadIdx.x; i < 3 + nreq; i += blockDim.x) state[i] = 0ull;
    __syncthreads();
    if (threadIdx.x == 0) state[1] = global_ns();
}

// Shared memory of a batch CTA, one of each per warp.
struct BatchShared {
    MarchParams par[8];
    WarpTotals totals[8];
};
extern __shared__ float4 s_batch[];

template <int DT, int COMP, int SHADE, int BS>
__device__ __noinline__ void batch_tile(int warp, int tile) {
    BatchShared& sh = *reinterpret_cast<BatchShared*>(s_batch);
    const MarchParams& P = sh.par[warp];
    const int lane = threadIdx.x & 31;
    const int tw = 1 << P.tile_wshift;
    const int px = P.rx0 + (tile % P.tiles_x) * tw + (lane & (tw - 1));
    const int py = P.ry0 + (tile / P.tiles_x) * (32 >> P.tile_wshift) + (lane >> P.tile_wshift);
    RayState st;
    st.begin(P);
    RayCounts cnt;
    if (px < P.rx1 && py < P.ry1) {
        const size_t pix = (size_t)py * P.W + px;
        float4 f, l;
        if (pixel_ray(P, px, py, f, l))
            march_ray<DT, COMP, SHADE, BS, false, false, true>(P, P.tf_rgba8, P.tf_alpha, f, l, px, py, nullptr, st, cnt);
        write_out(P, pix, st.res);
    }
    add_tile(sh.totals[warp], st.loop, cnt);
}

template <int COMP, int SHADE, int BS>
__global__ void __launch_bounds__(256, VRC_MARCH_MIN_BLOCKS)
    march_batch_kernel(const BatchReq* __restrict__ reqs, int nreq, const unsigned* __restrict__ tile_prefix,
                       unsigned total_tiles, unsigned long long* state) {
    BatchShared& sh = *reinterpret_cast<BatchShared*>(s_batch);
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    if (lane == 0) sh.totals[wib] = WarpTotals{};
    int cur = -1, dtype = 0;
    for (;;) {
        unsigned tile = 0;
        if (lane == 0) tile = atomicAdd(reinterpret_cast<unsigned*>(state), 1u);
        tile = __shfl_sync(FULL, tile, 0);
        int r = nreq;
        if (tile < total_tiles) {
            int lo = 0, hi = nreq;  // largest r with tile_prefix[r] <= tile
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (tile_prefix[mid] <= tile) lo = mid;
                else hi = mid;
            }
            r = lo;
        }
        if (r != cur) {
            __syncwarp();
            if (cur >= 0 && lane == 0) {  // this warp's last tile of the request it leaves is written
                __threadfence();
                atomicMax(state + 3 + cur, global_ns());
            }
            if (r == nreq) break;
            const int* src = reinterpret_cast<const int*>(&reqs[r].P);
            int* dst = reinterpret_cast<int*>(&sh.par[wib]);
            for (int i = lane; i < (int)(sizeof(MarchParams) / sizeof(int)); i += 32) dst[i] = src[i];
            dtype = reqs[r].dtype;
            __syncwarp();
            cur = r;
        }
        const int lt = (int)(tile - tile_prefix[r]);
        if (dtype == VRC_U8) batch_tile<VRC_U8, COMP, SHADE, BS>(wib, lt);
        else if (dtype == VRC_U16) batch_tile<VRC_U16, COMP, SHADE, BS>(wib, lt);
        else batch_tile<VRC_F32, COMP, SHADE, BS>(wib, lt);
        __syncwarp();
    }
    if (lane == 0) atomicAdd(state + 2, sh.totals[wib].samples);
}

template <int COMP, int SHADE, int BS>
cudaError_t launch_batch_t(const BatchReq* reqs, int nreq, const unsigned* prefix, unsigned total,
                           unsigned long long* state, int num_sms, cudaStream_t s) {
    auto k = march_batch_kernel<COMP, SHADE, BS>;
    int per_sm = 0;
    cudaError_t e = resident_ctas(k, sizeof(BatchShared), sizeof(BatchShared), &per_sm);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    long long grid = (long long)num_sms * per_sm;
    const long long need = ((long long)total + 7) / 8;
    if (grid > need) grid = need < 1 ? 1 : need;
    k<<<(unsigned)grid, 256, sizeof(BatchShared), s>>>(reqs, nreq, prefix, total, state);
    return cudaGetLastError();
}

// Every request of the default brick edge: its geometry is compile-time.
template <int COMP, int SHADE>
cudaError_t launch_batch_b(const BatchReq* reqs, int nreq, const unsigned* prefix, unsigned total,
                           unsigned long long* state, bool bricks32, int num_sms, cudaStream_t s) {
    return bricks32 ? launch_batch_t<COMP, SHADE, 32>(reqs, nreq, prefix, total, state, num_sms, s)
                    : launch_batch_t<COMP, SHADE, 0>(reqs, nreq, prefix, total, state, num_sms, s);
}

}  // namespace

cudaError_t launch_batch_begin(unsigned long long* state, int nreq, cudaStream_t s) {
    batch_begin_kernel<<<1, 256, 0, s>>>(state, nreq);
    return cudaGetLastError();
}

cudaError_t launch_march_batch(const BatchReq* reqs, int nreq, const unsigned* prefix, unsigned total,
                               unsigned long long* state, int compositing, int shading, bool bricks32, int num_sms,
                               cudaStream_t s) {
    const bool ph = shading == VRC_SHADE_PHONG;
    switch (compositing) {
        case VRC_MIP:
            return ph ? launch_batch_b<VRC_MIP, VRC_SHADE_PHONG>(reqs, nreq, prefix, total, state, bricks32, num_sms, s)
                      : launch_batch_b<VRC_MIP, VRC_SHADE_NONE>(reqs, nreq, prefix, total, state, bricks32, num_sms, s);
        case VRC_ISO:
            return ph ? launch_batch_b<VRC_ISO, VRC_SHADE_PHONG>(reqs, nreq, prefix, total, state, bricks32, num_sms, s)
                      : launch_batch_b<VRC_ISO, VRC_SHADE_NONE>(reqs, nreq, prefix, total, state, bricks32, num_sms, s);
        default:
            return ph ? launch_batch_b<VRC_DVR, VRC_SHADE_PHONG>(reqs, nreq, prefix, total, state, bricks32, num_sms, s)
                      : launch_batch_b<VRC_DVR, VRC_SHADE_NONE>(reqs, nreq, prefix, total, state, bricks32, num_sms, s);
    }
}

}  // namespace vrc
