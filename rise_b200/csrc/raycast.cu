// raycast.cu -- batched closest-hit and any-hit kernels for sm_100a.
//
// Persistent kernels: one grid of (SMs x resident blocks).  Each warp runs the
// while-while traversal of raycast.cuh; lanes refill themselves with new rays
// from a warp-local chunk as soon as their ray finishes, so SIMT lanes stay
// busy on the long tail of incoherent rays.  Rays are read as two 16-byte
// vector loads and hits written as one 16-byte store; the traversal stack
// lives in shared memory ([depth][thread], conflict-free).
#include <algorithm>
#include <atomic>

#include "core.h"
#include "raycast.cuh"

namespace rtb200 {

__device__ __forceinline__ Ray LoadRay(const rtb200_ray* rays, int i)
{
    const float4 a = ldg4(rays + i);
    const float4 b = ldg4(reinterpret_cast<const float*>(rays + i) + 4);
    Ray r;
    r.o[0] = a.x; r.o[1] = a.y; r.o[2] = a.z; r.tmin = a.w;
    r.d[0] = b.x; r.d[1] = b.y; r.d[2] = b.z; r.tmax = b.w;
    return r;
}

// Leaves tested per lane per traversal round in the batch kernels (measured
// best for both closest and any hit on incoherent rays).
constexpr int kCastLeaves = 2;
// Lanes of a warp that may still lack a postponed leaf when the descent stops:
// waiting for the last few to find one leaves most lanes idle.  8, 12, 14, 16 and
// 18 lanes: closest hit of 4,194,304 incoherent rays over binary16 boxes 3314,
// 3091, 3086, 3128, 3217 us, any hit 1649, 1543, 1524, 1548, 1581; of 100,003 rays
// with the joint tail (COOP) 161 us with 12 and 170 with 14.  (Closest hits with
// integer child keys; with whole distances 12 lanes take 2971 and 157 us.)
template <bool ANY, bool COOP>
constexpr int kCastLack = ANY && !COOP ? 14 : 12;

// Stores a finished ray's answer: its occlusion flag, or its closest hit with
// the distance re-measured in FP64.  The ray is read again: its direction is
// not kept during the walk.
template <bool ANY>
__device__ __forceinline__ void StoreAnswer(const TraceState& s, const GpuTri* __restrict__ tris,
                                            const rtb200_ray* __restrict__ rays, int ray,
                                            rtb200_hit* __restrict__ hits, uint8_t* __restrict__ occ)
{
    if (ANY) {
        occ[ray] = s.bestSlot >= 0 ? 1 : 0;
        return;
    }
    float4 out = make_float4(-1.0f, __int_as_float(-1), 0.0f, 0.0f);
    if (s.bestSlot >= 0) {
        float4 A, B, C;
        LoadVertices(tris, s.bestSlot, A, B, C);
        const Ray r = LoadRay(rays, ray);
        out.x = (float)RefineT(r.o, r.d, A, B, C);
        out.y = __int_as_float(TriIndex(tris, s.bestSlot));
        out.z = s.ba;
        out.w = s.bb;
    }
    *reinterpret_cast<float4*>(hits + ray) = out;
}

// COOP: the last rays of a warp are finished by all its lanes (CoopFinish);
// the rule for its use is in Launch.
template <class NodeT, bool ANY, bool SPILL, bool COOP>
__global__ void __launch_bounds__(kTraceBlock, 8)
KTrace(const NodeT* __restrict__ nodes, const GpuTri* __restrict__ tris,
       const rtb200_ray* __restrict__ rays, unsigned n, int ntri, rtb200_hit* __restrict__ hits,
       uint8_t* __restrict__ occ, unsigned chunk, unsigned* counter, unsigned* err)
{
    __shared__ int sstack[kStackRows * kTraceBlock];
    int spill[SPILL ? kTraceSpill : 1];
    const TraceStack stk = MakeStack(sstack + threadIdx.x, spill);
    WarpFeed feed = FeedStart(n, chunk);
    TraceState s;
    if (COOP) s.sp = stk.bottom, s.over = 0;
    int ray = -1;
    for (;;) {
        const int got = FeedTake(feed, ray < 0, n, chunk, counter);
        if (got >= 0) {
            ray = got;
            StartRay(s, LoadRay(rays, ray), stk.bottom);
        }
        const unsigned live = __ballot_sync(kFull, ray >= 0);
        if (!live) return;
        if (COOP && __popc(live) <= kCoopRays && FeedDry(feed) && CoopReady<SPILL>(s, stk, live)) break;
        if (ray >= 0 && TraceRound<NodeT, ANY, SPILL, kCastLeaves, kCastLack<ANY, COOP>>(s, nodes, tris, ntri, stk, err)) {
            StoreAnswer<ANY>(s, tris, rays, ray, hits, occ);
            ray = -1;
        }
    }
    if (COOP) {
        if (CoopFinish<NodeT, ANY, SPILL, false>(s, stk, ray >= 0, nodes, tris, ntri, sstack + (threadIdx.x & ~31u), err)) {
            StoreAnswer<ANY>(s, tris, rays, ray, hits, occ);
            ray = -1;
        }
        // What it left: nothing, but where triangles lie at about one distance.
        if (!ANY && ray >= 0) {
            LaneRest<NodeT, SPILL>(s, nodes, tris, ntri, stk, err);
            StoreAnswer<ANY>(s, tris, rays, ray, hits, occ);
        }
    }
}

namespace {

// Node visits per lane between ray refills of the eight-wide kernel.
constexpr int kW8Budget = 16;

template <bool ANY>
__global__ void __launch_bounds__(kTraceBlock, 8)
KTraceW8(const WNode8* __restrict__ nodes, const GpuTri* __restrict__ tris, const rtb200_ray* __restrict__ rays,
         unsigned n, rtb200_hit* __restrict__ hits, uint8_t* __restrict__ occ, unsigned chunk, unsigned* counter,
         unsigned* err)
{
    __shared__ uint2 sstack[kW8Stack * kTraceBlock];
    uint2* stk = sstack + threadIdx.x;
    WarpFeed feed = FeedStart(n, chunk);
    W8State s;
    int ray = -1;
    for (;;) {
        const int got = FeedTake(feed, ray < 0, n, chunk, counter);
        if (got >= 0) {
            ray = got;
            StartRayW8(s, LoadRay(rays, ray));
        }
        if (__all_sync(kFull, ray < 0)) break;
        if (ray >= 0 && TraceW8<ANY>(s, nodes, tris, stk, err, kW8Budget)) {
            if (ANY) {
                occ[ray] = s.bestSlot >= 0 ? 1 : 0;
            } else {
                float4 out;
                if (s.bestSlot >= 0) {
                    float4 A, B, C;
                    LoadVertices(tris, s.bestSlot, A, B, C);
                    out.x = (float)RefineT(s.p.o, s.d, A, B, C);
                    out.y = __int_as_float(TriIndex(tris, s.bestSlot));
                    out.z = s.ba;
                    out.w = s.bb;
                } else {
                    out = make_float4(-1.0f, __int_as_float(-1), 0.0f, 0.0f);
                }
                *reinterpret_cast<float4*>(hits + ray) = out;
            }
            ray = -1;
        }
    }
}

template <class K>
int GridFor(K kernel, int num_sms)
{
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kTraceBlock, 0) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    return per_sm * num_sms;
}

// One launch over `n` rays with the work counter and error word given.  The
// full grid is the kernel's occupancy times the SM count, cached per
// instantiation and device (devices of one process may differ).  Batches of
// up to 32 rays per resident warp launch only the warps that get a ray and
// never touch the counter; larger ones clear it first.
constexpr int kGridDevices = 64;

template <class K>
cudaError_t PlanFeed(K kernel, std::atomic<int>* grids, const rtb200_ctx* ctx, unsigned n, unsigned* counter,
                     cudaStream_t stream, int& grid, unsigned& chunk)
{
    constexpr unsigned kWarps = kTraceBlock / 32;
    const int dev = ctx->device;
    grid = (dev >= 0 && dev < kGridDevices) ? grids[dev].load(std::memory_order_relaxed) : 0;
    if (!grid) {
        grid = GridFor(kernel, ctx->num_sms);
        if (dev >= 0 && dev < kGridDevices) grids[dev].store(grid, std::memory_order_relaxed);
    }
    chunk = FeedChunk(n, (unsigned)grid * kWarps);
    const unsigned blocks = ((n + chunk - 1) / chunk + kWarps - 1) / kWarps;
    if (blocks <= (unsigned)grid) {
        grid = (int)blocks;
        return cudaSuccess;
    }
    return cudaMemsetAsync(counter, 0, sizeof(unsigned), stream);
}

// Batches of up to this many rays per SM (the resident warps' first 128 rays
// each) use the kernels whose warps finish their last rays together.  Without
// and with (binary16 boxes, 300k-triangle soup): 20,000 rays 155 and 85 us,
// 100,003 245 and 157, 500,000 442 and 393.  Beyond, the last rays count for less
// and the joint walk's registers and checks for more: 1,000,000 rays on 1M triangles
// 818 and 805 us, 4,194,304 2971 and 3087, 786,432 camera rays 209 and 223.
constexpr unsigned kCoopBatchPerSm = 4096;

template <class NodeT, bool ANY, bool SPILL, bool COOP>
cudaError_t LaunchKernel(const rtb200_scene* s, const rtb200_ray* d_rays, unsigned n, rtb200_hit* hits, uint8_t* occ,
                         unsigned* counter, unsigned* err, cudaStream_t stream)
{
    static std::atomic<int> grids[kGridDevices];
    int grid;
    unsigned chunk;
    const cudaError_t e = PlanFeed(KTrace<NodeT, ANY, SPILL, COOP>, grids, s->ctx, n, counter, stream, grid, chunk);
    if (e != cudaSuccess) return e;
    KTrace<NodeT, ANY, SPILL, COOP><<<grid, kTraceBlock, 0, stream>>>((const NodeT*)s->d_nodes, s->d_tris, d_rays, n,
                                                                      (int)s->tri_material.size(), hits, occ, chunk,
                                                                      counter, err);
    return cudaGetLastError();
}

template <class NodeT, bool ANY>
cudaError_t Launch(const rtb200_scene* s, const rtb200_ray* d_rays, unsigned n, rtb200_hit* hits, uint8_t* occ,
                   unsigned* counter, unsigned* err, cudaStream_t stream)
{
    const bool spill = s->stack_bound > kTraceStack;
    if (n <= kCoopBatchPerSm * (unsigned)s->ctx->num_sms)
        return spill ? LaunchKernel<NodeT, ANY, true, true>(s, d_rays, n, hits, occ, counter, err, stream)
                     : LaunchKernel<NodeT, ANY, false, true>(s, d_rays, n, hits, occ, counter, err, stream);
    return spill ? LaunchKernel<NodeT, ANY, true, false>(s, d_rays, n, hits, occ, counter, err, stream)
                 : LaunchKernel<NodeT, ANY, false, false>(s, d_rays, n, hits, occ, counter, err, stream);
}

template <bool ANY>
cudaError_t DispatchPart(const rtb200_scene* s, const rtb200_ray* d_rays, unsigned n, rtb200_hit* hits, uint8_t* occ,
                         unsigned* counter, unsigned* err, cudaStream_t stream)
{
    if (s->layout == RTB200_BVH_W8) {
        static std::atomic<int> grids[kGridDevices];
        int grid;
        unsigned chunk;
        const cudaError_t e = PlanFeed(KTraceW8<ANY>, grids, s->ctx, n, counter, stream, grid, chunk);
        if (e != cudaSuccess) return e;
        KTraceW8<ANY><<<grid, kTraceBlock, 0, stream>>>((const WNode8*)s->d_nodes, s->d_tris, d_rays, n, hits, occ,
                                                        chunk, counter, err);
        return cudaGetLastError();
    }
    if (s->layout == RTB200_BVH_Q8) return Launch<QNode4, ANY>(s, d_rays, n, hits, occ, counter, err, stream);
    if (s->layout == RTB200_BVH_F16) return Launch<HNode4, ANY>(s, d_rays, n, hits, occ, counter, err, stream);
    return Launch<GpuNode4, ANY>(s, d_rays, n, hits, occ, counter, err, stream);
}

template <bool ANY>
cudaError_t Dispatch(const rtb200_scene* s, const rtb200_ray* d_rays, int64_t n, rtb200_hit* hits, uint8_t* occ,
                     unsigned long long* counter, unsigned* err, cudaStream_t stream)
{
    cudaError_t e = cudaSuccess;
    for (int64_t at = 0; at < n && e == cudaSuccess; at += kFeedRays)
        e = DispatchPart<ANY>(s, d_rays + at, (unsigned)std::min<int64_t>(kFeedRays, n - at),
                              ANY ? nullptr : hits + at, ANY ? occ + at : nullptr, (unsigned*)counter, err, stream);
    return e;
}

}  // namespace

cudaError_t LaunchCastClosest(const rtb200_scene* s, const rtb200_ray* d_rays, int64_t n,
                              rtb200_hit* d_hits, cudaStream_t stream)
{
    return Dispatch<false>(s, d_rays, n, d_hits, nullptr, s->d_counter, s->d_err, stream);
}

cudaError_t LaunchCastClosestScratch(const rtb200_scene* s, const rtb200_ray* d_rays, int64_t n,
                                     rtb200_hit* d_hits, unsigned long long* counter, unsigned* err,
                                     cudaStream_t stream)
{
    return Dispatch<false>(s, d_rays, n, d_hits, nullptr, counter, err, stream);
}

cudaError_t LaunchCastAnyScratch(const rtb200_scene* s, const rtb200_ray* d_rays, int64_t n, uint8_t* d_occ,
                                 unsigned long long* counter, unsigned* err, cudaStream_t stream)
{
    return Dispatch<true>(s, d_rays, n, nullptr, d_occ, counter, err, stream);
}

cudaError_t LaunchCastAny(const rtb200_scene* s, const rtb200_ray* d_rays, int64_t n,
                          uint8_t* d_occ, cudaStream_t stream)
{
    return Dispatch<true>(s, d_rays, n, nullptr, d_occ, s->d_counter, s->d_err, stream);
}

}  // namespace rtb200
