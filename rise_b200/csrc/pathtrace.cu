// pathtrace.cu -- wavefront hero-wavelength spectral path tracer for sm_100a.
//
// Restates, as a wavefront, the reference's HWSS path loop
// (src/Library/Shaders/PathTracingIntegrator.cpp:3939-4821 IntegrateFromHitHWSS,
// :4855-5126 IntegrateRayHWSS) driven per pixel sample by
// PathTracingSpectralRasterizer::IntegratePixelSpectral
// (src/Library/Rendering/PathTracingSpectralRasterizer.cpp:121-198).
//
// A fixed pool of path slots lives in HBM as SoA.  One iteration is five to ten
// launches over device-side queues (no host round trip):
//   KConnect any hit for the shadow-ray queue of the iteration before;
//            unoccluded contributions are added to the path's per-wavelength
//            radiance
//   KAssign  rotate the queue counters, split the free slots among the jobs
//            that have samples left
//   KRegen   splat finished paths into the film, start new camera samples
//   KExtend  closest hit for every active path (warp while-while traversal)
//   KClassify sort the active paths by the material they hit, where scenes mix
//            shading classes
//   KShade   emission + MIS, next-event estimation to area lights and the
//            sky (shadow-ray queue), hero-wavelength BSDF sampling with
//            companion-wavelength weights, Russian roulette; after KClassify one
//            launch per class
//   KEscape  the sky's radiance for paths that left the scene (after KClassify)
// Appends to queues are warp-aggregated (one atomic per warp and queue).
//
// Over deep trees (PtLaunch::coop) the paths that go on are extended on the
// iteration's stream beside KConnect, KAssign, KRegen and the extension of the new
// paths on a side stream: five launches for one shading class over a small tree,
// ten for mixed ones over a deep tree.  What runs side by side shares no counter:
// the continuing paths' KExtend reads kCntNext of the last iteration's parity and
// feeds from trace_ctr[2 + parity], while KAssign clears kCntNext of this parity
// and trace_ctr[0], [1] and [2 + the other parity]; the new paths' KExtend feeds
// from trace_ctr[1], KConnect from trace_ctr[0].  The shading kernels run side by
// side after a join and append to the same queues, with atomics.
#include <cfloat>

#include "bsdf.cuh"
#include "core.h"
#include "env_map.h"
#include "pathtrace.h"
#include "pt_device.cuh"
#include "raycast.cuh"

namespace rtb200 {

constexpr int kShadeBlock = 256;
// Leaves tested per lane per traversal round in KExtend / KConnect (measured
// best for the path tracer's mixed secondary and shadow rays).
constexpr int kPathLeaves = 1;
// Lanes that may lack a leaf when the descent stops (raycast.cu).  Over deep
// trees (COOP) 16: 800k-triangle scene at 8 spp 25.8 ms with 12, 24.8 with 16 and
// 18, 26.1 with 24; over small ones 12: Cornell box at 16 spp 2.76, 2.77, 2.78,
// 2.81 ms.
template <bool COOP>
constexpr int kPathLack = COOP ? 16 : 12;
constexpr float kInv4Pi = 0.07957747154594767f;

// ---- light BVH -------------------------------------------------------------

// LightBVH::NodeImportance (Lights/LightBVH.cpp:169-217) for full-sphere
// cones: power / max(squared distance from p to the node's box, 1e-4).
__device__ __forceinline__ float LightImportance(const PtLightNode* __restrict__ nodes, int i, V3 p)
{
    const float4 a = __ldg(reinterpret_cast<const float4*>(nodes + i));       // lo xyz, hi x
    const float4 b = __ldg(reinterpret_cast<const float4*>(nodes + i) + 1);   // hi yz, power, right
    if (!(b.z > 0.0f)) return 0.0f;
    const float lo[3] = {a.x, a.y, a.z}, hi[3] = {a.w, b.x, b.y}, q[3] = {p.x, p.y, p.z};
    float d2 = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float d = q[k] < lo[k] ? lo[k] - q[k] : (q[k] > hi[k] ? q[k] - hi[k] : 0.0f);
        d2 += d * d;
    }
    return b.z / fmaxf(d2, 1e-4f);
}

// LightBVH::Sample (LightBVH.cpp:423-482): from the root, pick a child in
// proportion to its importance, reusing the rescaled random number; returns
// the luminary and its selection probability (0: nothing to pick).
__device__ int SampleLightBvh(const PtLightNode* __restrict__ nodes, V3 p, float xi, float& pdf)
{
    pdf = 1.0f;
    int i = 0;
    for (int guard = 0; guard < 64; ++guard) {
        const int4 c = __ldg(reinterpret_cast<const int4*>(nodes + i) + 2);   // light, count, start, pad
        if (c.y <= 1) return c.x;
        const int right = __float_as_int(__ldg(reinterpret_cast<const float4*>(nodes + i) + 1).w);
        const float il = LightImportance(nodes, i + 1, p), ir = LightImportance(nodes, right, p);
        const float total = il + ir;
        if (!(total > 0.0f)) { pdf = 0.0f; return -1; }
        const float pl = il / total;
        if (xi < pl) {
            pdf *= pl;
            xi = xi / pl;
            i = i + 1;
        } else {
            pdf *= 1.0f - pl;
            xi = (xi - pl) / (1.0f - pl);
            i = right;
        }
    }
    pdf = 0.0f;
    return -1;
}

// LightBVH::Pdf (LightBVH.cpp:484-531): the probability that SampleLightBvh
// picks the luminary at leaf position `pos` from p.
__device__ float LightBvhPdf(const PtLightNode* __restrict__ nodes, int pos, V3 p)
{
    float pdf = 1.0f;
    int i = 0;
    for (int guard = 0; guard < 64; ++guard) {
        const int4 c = __ldg(reinterpret_cast<const int4*>(nodes + i) + 2);
        if (c.y <= 1) return pdf;
        const int right = __float_as_int(__ldg(reinterpret_cast<const float4*>(nodes + i) + 1).w);
        const float il = LightImportance(nodes, i + 1, p), ir = LightImportance(nodes, right, p);
        const float total = il + ir;
        if (!(total > 0.0f)) return 0.0f;
        const float pl = il / total;
        const int4 lc = __ldg(reinterpret_cast<const int4*>(nodes + i + 1) + 2);
        if (pos >= lc.z && pos < lc.z + lc.y) {
            pdf *= pl;
            i = i + 1;
        } else {
            pdf *= 1.0f - pl;
            i = right;
        }
    }
    return 0.0f;
}

// ---- image environment (env_map.h), out of line: rarely taken, and inlined
// it would add to the shading kernels' register pressure ----------------------

__device__ __noinline__ EnvSpec EnvLookupAt(const PtEnvMap* E, V3 d) { return EnvLookup(*E, d.x, d.y, d.z); }
__device__ __noinline__ float EnvPdfAt(const PtEnvMap* E, V3 d) { return EnvPdf(*E, d.x, d.y, d.z); }
__device__ __noinline__ float EnvSampleAt(const PtEnvMap* E, float u1, float u2, V3& d)
{
    return EnvSample(*E, u1, u2, d.x, d.y, d.z);
}

// ---- film ------------------------------------------------------------------

// XYZ of one finished sample: sum over active wavelengths of
// XYZ(lambda_i) * L_i, scaled by (lmax - lmin) / k_y / active
// (PathTracingSpectralRasterizer.cpp:141-198); a pixel sample of several
// spectral samples is their mean (1 / nSpectralSamples on the mean films; the
// filtered film's weights normalise it by themselves).
__device__ __forceinline__ void Splat(const PtJobDev& J, float4 L, float hero, uint4 m)
{
    const PtSettings& S = J.set;
    float lam[4];
    Wavelengths(hero, S.lmin, S.lmax, lam);
    const unsigned term = (m.z >> kTermShift) & 0xfu;
    float X = 0, Y = 0, Z = 0;
    int active = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float x, y, z;
        if (!(term & (1u << i)) && Cmf(lam[i], x, y, z)) {
            const float l = Get(L, i);
            X += x * l; Y += y * l; Z += z * l;
            ++active;
        }
    }
    if (active == 0) return;
    const float s = S.ynorm / (float)active * (S.filter == kFilterSplat ? 1.0f : S.inv_spectral);
    if (J.lum && Y != 0.0f) {
        // Adaptive sampling: the pixel's luminance sums for its convergence test.
        const double y = (double)(Y * s);
        atomicAdd(J.lum + 2 * (size_t)m.x, y);
        atomicAdd(J.lum + 2 * (size_t)m.x + 1, y * y);
    }
    if (S.filter != kFilterSplat) {
        float* px = J.film + 3 * (size_t)m.x;
        if (X != 0.0f) atomicAdd(px + 0, X * s);
        if (Y != 0.0f) atomicAdd(px + 1, Y * s);
        if (Z != 0.0f) atomicAdd(px + 2, Z * s);
        return;
    }
    // FilteredFilm::Splat (Rendering/FilteredFilm.cpp:42-98): the sample's
    // screen position (the camera's, see KRegen: uniform in its pixel, pixel
    // centres on integer coordinates) adds w XYZ and w to every pixel within the Gaussian's
    // support, w = exp(-r^2 / 2 sigma^2) / (2 pi sigma^2)
    // (GaussianPixelFilter.h:67-78).
    const int W = J.cam.width, H = J.cam.height;
    const int px = (int)(m.x % (uint32_t)W), py = (int)(m.x / (uint32_t)W);
    // The camera's jitter numbers again (hash key or Sobol seed in m.w, sample in m.y).
    const bool sobol = S.sampler != kSamplerHash, shuf = S.sampler == kSamplerSobolShuffled;
    const float ox = sobol ? SobolSample(m.y, 0, m.w, shuf) : Rand(m.w, 0);
    const float oy = sobol ? SobolSample(m.y, 1, m.w, shuf) : Rand(m.w, 1);
    const float sx = (float)px + ox - 0.5f, sy = (float)py + 0.5f - oy;
    const float hw = S.filt_half;
    const int x0 = max(0, (int)floorf(sx - hw)), x1 = min(W - 1, (int)floorf(sx + hw));
    const int y0 = max(0, (int)floorf(sy - hw)), y1 = min(H - 1, (int)floorf(sy + hw));
    X *= s; Y *= s; Z *= s;
    for (int qy = y0; qy <= y1; ++qy) {
        const float dy = sy - (float)qy;
        if (fabsf(dy) > hw) continue;
        for (int qx = x0; qx <= x1; ++qx) {
            const float dx = sx - (float)qx;
            if (fabsf(dx) > hw) continue;
            const float w = S.filt_norm * expf(-(dx * dx + dy * dy) * S.filt_inv2s2);
            float* f = J.film + 4 * ((size_t)qy * W + qx);
            AtomicAdd4(f, X * w, Y * w, Z * w, w);
        }
    }
}

// ---- kernels ---------------------------------------------------------------

// A path's job: the kernel argument where the engine renders one job (ONE),
// whose scene, camera and settings are then operands from the constant bank,
// else an entry of the job table, each use of which is a load (Cornell box at 16
// spp 2.87 ms from the table, 2.77 from the argument; adaptive 200 x 150 image
// 3.53 and 3.38).
template <bool ONE>
__device__ __forceinline__ const PtJobDev& JobOf(const PtJobDev* __restrict__ jobs, const PtJobDev& one, int jid)
{
    if constexpr (ONE) return one;
    else return jobs[jid];
}

// First in every kernel of an iteration: waits for the stream's previous kernel
// to end, when this one was launched ahead of that (Chain below).  The launch
// latency is then off the path: a 120 x 80 image at 4 spp 1.95 -> 1.78 ms, the
// Cornell box 3.02 -> 2.86 ms device time.  Letting the next kernel's blocks in
// as soon as the last of this one's run (a trigger here) took that back: they
// wait in the way of kernels on the side streams (2.98 ms).
__device__ __forceinline__ void ChainStart() { cudaGridDependencySynchronize(); }

// Inclusive prefix sum over a block of 1024 threads, or over one warp.
template <bool WARP>
__device__ __forceinline__ int Scan(int v, int* warp_sums)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(kFull, v, o);
        if (lane >= o) v += u;
    }
    if (WARP) return v;
    if (lane == 31) warp_sums[w] = v;
    __syncthreads();
    if (w == 0) {
        int s = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(kFull, s, o);
            if (lane >= o) s += u;
        }
        warp_sums[lane] = s;
    }
    __syncthreads();
    const int r = v + (w > 0 ? warp_sums[w - 1] : 0);
    __syncthreads();
    return r;
}

// Split this iteration's free slots among the jobs that still have camera
// samples (one block, one thread per job).  Every such job first gets a
// quarter of an equal share (capped by what it has left), so none starves;
// the rest goes to jobs in order of fewest samples left (shortest remaining
// first: in a serving mix the first progressive levels of new requests finish
// before long high-spp levels).  Each job's range of free-queue entries and
// first sample index go to Q.assign and its issued counter advances by its
// share.  Block prefix sums replace per-warp atomics on one counter per job.
// Images do not depend on this schedule: a sample's random numbers depend
// only on its job, pixel and sample index.
template <bool WARP>
__device__ __forceinline__ void AssignJobs(const PtJobDev* __restrict__ jobs, const int* __restrict__ ids,
                                           const PtQueues& Q, int iter, int njobs, int n)
{
    __shared__ int sums[32];
    __shared__ unsigned long long s_left[kPtMaxJobs];   // samples left per job (for the order)
    __shared__ int s_sorted[kPtMaxJobs];
    __shared__ int s_live, s_first;
    const auto sync = [] { if (WARP) __syncwarp(); else __syncthreads(); };
    const int t = threadIdx.x, last = WARP ? 31 : kPtMaxJobs - 1;
    int jid = -1, rem = 0;
    unsigned long long issued = 0, left_all = 0;
    if (t < njobs) {
        jid = ids[(t + iter) % njobs];
        const PtJobDev& J = jobs[jid];
        issued = *J.sample_ctr;
        if (issued < J.total) {
            left_all = J.total - issued;
            rem = (int)min(left_all, (unsigned long long)n);
        }
    }
    const int live = Scan<WARP>(rem > 0 ? 1 : 0, sums);
    if (t == last) s_live = live;
    sync();
    const int share = s_live > 0 ? n / s_live / 4 : 0;
    const int first = min(rem, share);
    const int firstIncl = Scan<WARP>(first, sums);
    if (t == last) s_first = firstIncl;
    s_left[t] = left_all;
    sync();
    const int left = n - s_first;
    const int more = rem - first;
    // Rank by samples left (ties by position), then a prefix sum in that order.
    int rank = 0;
    if (t < njobs)
        for (int k = 0; k < njobs; ++k) rank += (s_left[k] < left_all) || (s_left[k] == left_all && k < t);
    if (t < njobs) s_sorted[rank] = more;
    sync();
    const int v = t < njobs ? s_sorted[t] : 0;
    const int inclSorted = Scan<WARP>(v, sums);
    sync();
    s_sorted[t] = inclSorted - v;   // exclusive prefix in rank order
    sync();
    const int extra = t < njobs ? max(0, min(more, left - s_sorted[rank])) : 0;
    const int take = first + extra;
    const int takeIncl = Scan<WARP>(take, sums);
    if (t < njobs) {
        PtAssign a;
        a.base = issued;
        a.off = takeIncl - take;
        a.jid = jid;
        Q.assign[t] = a;
        if (take > 0) *jobs[jid].sample_ctr = issued + (unsigned long long)take;
    }
    if (t == last) Q.cnt[kCntAssigned] = takeIncl;
}

// Also rotates the queue counters of the last iteration into this one's: a
// launch of its own for that, and a memset of the feed counters, cost 4 us an
// iteration.  With up to 32 jobs one warp does the work.
__global__ void __launch_bounds__(kPtMaxJobs)
KAssign(const PtJobDev* __restrict__ jobs, const int* __restrict__ ids, PtQueues Q, int iter)
{
    const int parity = iter & 1;
    ChainStart();
    const int njobs = Q.cnt[kCntJobs], n = Q.cnt[kCntFreeNext];
    __syncthreads();
    if (threadIdx.x == 0) {
        int* cnt = Q.cnt;
        for (int c = 0; c < kShadeClasses; ++c) cnt[kCntClass + c] = 0;
        Counter64(cnt, kCntSegments) += (unsigned)cnt[kCntActive];
        Counter64(cnt, kCntShadowRays) += (unsigned)cnt[kCntShadow];
        cnt[kCntActive] = cnt[kCntFreshRays] = cnt[kCntNext + (parity ^ 1)];
        cnt[kCntNext + parity] = 0;
        cnt[kCntFree] = n;
        cnt[kCntFreeNext] = 0;
        cnt[kCntShadow] = 0;
        Q.trace_ctr[0] = Q.trace_ctr[1] = Q.trace_ctr[2 + (parity ^ 1)] = 0ull;
    }
    if (njobs > 32) AssignJobs<false>(jobs, ids, Q, iter, njobs, n);
    else if (threadIdx.x < 32) AssignJobs<true>(jobs, ids, Q, iter, njobs, n);
}

template <bool ONE>
__global__ void __launch_bounds__(kShadeBlock)
KRegen(const PtJobDev* __restrict__ jobs, PtPaths P, PtQueues Q, const __grid_constant__ PtJobDev one)
{
    ChainStart();
    const int njobs = Q.cnt[kCntJobs];
    const int n = Q.cnt[kCntFree];
    const int nassigned = Q.cnt[kCntAssigned];
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int base = warp * 32; base < n; base += nwarps * 32) {
        const int i = base + lane;
        const bool valid = i < n;
        const int slot = valid ? Q.free_[i] : -1;
        int fin_job = -1;
        if (valid) {
            float4 aux, meta;
            LoadPair(P.state + slot, aux, meta);
            const uint4 m = Bits(meta);
            if (m.z & kFlagFinishing) {
                fin_job = __float_as_int(aux.z);
                Splat(JobOf<ONE>(jobs, one, fin_job), P.rad[slot].b, aux.x, m);
                SetFlags(P, slot, m.z & ~kFlagFinishing);
            }
        }
        // Finished samples, one atomic per job present in the warp.
        const unsigned grp = __match_any_sync(kFull, fin_job);
        if (fin_job >= 0 && lane == __ffs(grp) - 1) atomicAdd(JobOf<ONE>(jobs, one, fin_job).done_ctr, (unsigned long long)__popc(grp));
        // New camera samples: free entry i < nassigned belongs to the job
        // whose assigned range holds it (KAssign).
        bool got = false;
        if (valid && i < nassigned) {
            int lo = 0, hi = njobs - 1;   // largest k with assign[k].off <= i
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (Q.assign[mid].off <= i) lo = mid; else hi = mid - 1;
            }
            const PtAssign a = Q.assign[lo];
            const int jid = a.jid;
            const PtJobDev& J = JobOf<ONE>(jobs, one, jid);
            const unsigned long long g = a.base + (unsigned long long)(i - a.off);
            {   // PinholeCamera::GenerateRay (Cameras/PinholeCamera.cpp:182-210)
                // 64-bit division only where the request needs it.
                const uint32_t npix = (uint32_t)J.npix;
                const uint32_t pass = J.total >> 32 ? (uint32_t)(g / npix) : (uint32_t)g / npix;
                const uint32_t slot_px = (uint32_t)g - pass * npix;
                const uint32_t pixel = J.px_list ? __ldg(J.px_list + slot_px) : slot_px;
                const uint32_t sample = (uint32_t)(J.sample_begin + pass);
                const int px = (int)(pixel % (uint32_t)J.cam.width), py = (int)(pixel / (uint32_t)J.cam.width);
                const bool sobol = J.set.sampler != kSamplerHash, shuf = J.set.sampler == kSamplerSobolShuffled;
                // Hash key, or the pixel's Sobol seed (camera dimensions 0-2).
                const uint32_t key = sobol ? SobolPixelSeed((uint32_t)px, (uint32_t)py, J.set.seed)
                                           : PathKey(J.set.seed, pixel, sample);
                // Screen position in pixel units, pixel centres on integer
                // coordinates, rows counted downwards: the reference's
                // ptOnScreen = (x + u - 1/2, (height - y) + v - 1/2) for the
                // box filter and the filtered film
                // (PathTracingSpectralRasterizer.cpp:321-331, BoxPixelFilter.h:54-58),
                // or the pixel centre moved by the truncated Gaussian's
                // inverse CDF for a narrow Gaussian (GaussianPixelFilter.h:109-127).
                const float ox = sobol ? SobolSample(sample, 0, key, shuf) : Rand(key, 0);
                const float oy = sobol ? SobolSample(sample, 1, key, shuf) : Rand(key, 1);
                float fx, fy;
                if (J.set.filter == kFilterWarp) {
                    const float v = fmaxf(J.set.filt_trunc + (1.0f - J.set.filt_trunc) * ox, 1e-30f);
                    const float r = J.set.filt_sigma * sqrtf(-2.0f * logf(v));
                    float sn, cs;
                    sincospif(2.0f * oy, &sn, &cs);
                    fx = (float)px + r * cs;
                    fy = (float)py - r * sn;
                } else {
                    fx = (float)px + ox - 0.5f;
                    fy = (float)py + 0.5f - oy;
                }
                const float sx = 2.0f * fx / (float)J.cam.width - 1.0f;
                const float sy = 1.0f - 2.0f * fy / (float)J.cam.height;
                const V3 d = normalize(mk(J.cam.fwd[0] + sx * J.cam.right[0] + sy * J.cam.up[0],
                                          J.cam.fwd[1] + sx * J.cam.right[1] + sy * J.cam.up[1],
                                          J.cam.fwd[2] + sx * J.cam.right[2] + sy * J.cam.up[2]));
                // Wavelength: the hero of an equidistant bundle, or one
                // wavelength, binned as the reference's single-wavelength loop
                // bins it (lambda_begin + int(u * n) * step,
                // PathTracingSpectralRasterizer.cpp:180-183); the companions of a
                // single-wavelength path start terminated.
                const float uw = sobol ? SobolSample(sample, 2, key, shuf) : Rand(key, 2);
                const float hero = J.set.num_wl && J.set.single
                                       ? J.set.lmin + (float)min((int)(uw * (float)J.set.num_wl), J.set.num_wl - 1) *
                                                          J.set.wl_step
                                       : J.set.lmin + uw * (J.set.lmax - J.set.lmin);
                StorePair(P.ray + slot, make_float4(J.cam.pos[0], J.cam.pos[1], J.cam.pos[2], 0.0f),
                          make_float4(d.x, d.y, d.z, __int_as_float(0x7f800000)));
                StorePair(P.rad + slot, make_float4(1.0f, 1.0f, 1.0f, 1.0f), make_float4(0.0f, 0.0f, 0.0f, 0.0f));
                StorePair(P.state + slot, make_float4(hero, 0.0f, __int_as_float(jid), 0.0f),
                          Floats(make_uint4(pixel, sample,
                                            kFlagConsiderEmission | (J.set.single ? (0xeu << kTermShift) : 0u), key)));
                got = true;
            }
        }
        // Slots left without work stay queued for the next iteration, so
        // jobs submitted later find them.
        const bool idle = valid && !got;
        int* const queues[2] = {&Q.cnt[kCntActive], &Q.cnt[kCntFreeNext]};
        const int count[2] = {got, idle};
        int at[2];
        WarpAppend(queues, count, at);
        if (got) Q.active[at[0]] = slot;
        if (idle) Q.free_next[at[1]] = slot;
    }
}

// The extension kernel over all active paths, those that continue from the last
// iteration, or this iteration's new ones behind them in the queue; or the
// connection kernel.
enum class TraceKind { Extend, ExtendOld, ExtendNew, Connect };

// Closest hit for active paths.
// Same while-while walk as KTrace; the hit stores the leaf-order triangle slot
// for shading.
// UNIFORM: every job shares the scene `us` (kernel argument, no per-path
// lookup of the job's scene).
template <class NodeT, bool SPILL, bool UNIFORM, bool COOP>
__global__ void __launch_bounds__(kTraceBlock, 8)
KExtend(const PtJobDev* __restrict__ jobs, PtPaths P, PtQueues Q, PtScene us, int parity, TraceKind kind)
{
    const NodeT* nodes = UNIFORM ? (const NodeT*)us.nodes : nullptr;
    const GpuTri* tris = UNIFORM ? us.tris : nullptr;
    int ntri = UNIFORM ? us.ntri : 0;
    __shared__ int sstack[kStackRows * kTraceBlock];
    int spill[SPILL ? kTraceSpill : 1];
    const TraceStack stk = MakeStack(sstack + threadIdx.x, spill);
    ChainStart();
    const bool going_on = kind == TraceKind::ExtendOld;
    const unsigned first = kind == TraceKind::ExtendNew ? (unsigned)Q.cnt[kCntFreshRays] : 0u;
    const unsigned n = (unsigned)Q.cnt[going_on ? kCntNext + (parity ^ 1) : (int)kCntActive] - first;
    unsigned* counter = (unsigned*)(Q.trace_ctr + (going_on ? 2 + parity : 1));
    const unsigned chunk = FeedChunk(n, (gridDim.x * blockDim.x) >> 5);
    WarpFeed feed = FeedStart(n, chunk);
    TraceState s;
    if (COOP) s.sp = stk.bottom, s.over = 0;
    int qi = -1;
    int slot = -1;
    for (;;) {
        const int got = FeedTake(feed, qi < 0, n, chunk, counter);
        if (got >= 0) {
            qi = (int)first + got;
            slot = Q.active[qi];
            if (!UNIFORM) {
                const PtScene& S = jobs[PathJob(P, slot)].scene;
                nodes = (const NodeT*)S.nodes;
                tris = S.tris;
                ntri = S.ntri;
            }
            float4 o, d;
            LoadPair(P.ray + slot, o, d);
            Ray r;
            r.o[0] = o.x; r.o[1] = o.y; r.o[2] = o.z; r.tmin = o.w;
            r.d[0] = d.x; r.d[1] = d.y; r.d[2] = d.z; r.tmax = d.w;
            StartRay(s, r, stk.bottom);
        }
        const unsigned live = __ballot_sync(kFull, qi >= 0);
        if (!live) return;
        if (COOP && __popc(live) <= kCoopRays && FeedDry(feed) && CoopReady<SPILL>(s, stk, live)) break;
        if (qi >= 0 && TraceRound<NodeT, false, SPILL, kPathLeaves, kPathLack<COOP>>(s, nodes, tris, ntri, stk, Q.err)) {
            P.hit[slot] = make_float4(s.best, __int_as_float(s.bestSlot), s.ba, s.bb);
            qi = -1;
        }
    }
    if (COOP) {
        const bool done = CoopFinish<NodeT, false, SPILL, !UNIFORM>(s, stk, qi >= 0, nodes, tris, ntri,
                                                                    sstack + (threadIdx.x & ~31u), Q.err);
        if (qi >= 0 && !done) LaneRest<NodeT, SPILL>(s, nodes, tris, ntri, stk, Q.err);
        if (qi >= 0) P.hit[slot] = make_float4(s.best, __int_as_float(s.bestSlot), s.ba, s.bb);
    }
}

// Adds an unoccluded shadow entry's contribution to its path's radiance.
__device__ __forceinline__ void AddShadow(const PtPaths& P, const ShadowEntry& e)
{
    float* l = &P.rad[__float_as_int(e.d.w)].b.x;
    // One wavelength's contribution, or a sample that all four share.
    if ((e.c.x != 0.0f) + (e.c.y != 0.0f) + (e.c.z != 0.0f) + (e.c.w != 0.0f) > 1) {
        AtomicAdd4(l, e.c.x, e.c.y, e.c.z, e.c.w);
        return;
    }
    if (e.c.x != 0.0f) atomicAdd(l + 0, e.c.x);
    if (e.c.y != 0.0f) atomicAdd(l + 1, e.c.y);
    if (e.c.z != 0.0f) atomicAdd(l + 2, e.c.z);
    if (e.c.w != 0.0f) atomicAdd(l + 3, e.c.w);
}

// Any hit for the shadow-ray queue; unoccluded entries add their
// contribution to the path's radiance.
template <class NodeT, bool SPILL, bool UNIFORM, bool COOP>
__global__ void __launch_bounds__(kTraceBlock, 8)
KConnect(const PtJobDev* __restrict__ jobs, PtPaths P, PtQueues Q, PtScene us)
{
    const NodeT* nodes = UNIFORM ? (const NodeT*)us.nodes : nullptr;
    const GpuTri* tris = UNIFORM ? us.tris : nullptr;
    int ntri = UNIFORM ? us.ntri : 0;
    __shared__ int sstack[kStackRows * kTraceBlock];
    int spill[SPILL ? kTraceSpill : 1];
    const TraceStack stk = MakeStack(sstack + threadIdx.x, spill);
    ChainStart();
    const unsigned n = (unsigned)Q.cnt[kCntShadow];
    const unsigned chunk = FeedChunk(n, (gridDim.x * blockDim.x) >> 5);
    WarpFeed feed = FeedStart(n, chunk);
    TraceState s;
    if (COOP) s.sp = stk.bottom, s.over = 0;
    int qi = -1;
    for (;;) {
        const int got = FeedTake(feed, qi < 0, n, chunk, (unsigned*)Q.trace_ctr);
        if (got >= 0) {
            qi = got;
            const ShadowEntry e = Q.shadow[qi];
            if (!UNIFORM) {
                const PtScene& S = jobs[PathJob(P, __float_as_int(e.d.w))].scene;
                nodes = (const NodeT*)S.nodes;
                tris = S.tris;
                ntri = S.ntri;
            }
            Ray r;
            r.o[0] = e.o.x; r.o[1] = e.o.y; r.o[2] = e.o.z; r.tmin = 0.0f;
            r.d[0] = e.d.x; r.d[1] = e.d.y; r.d[2] = e.d.z; r.tmax = e.o.w;
            StartRay(s, r, stk.bottom);
        }
        const unsigned live = __ballot_sync(kFull, qi >= 0);
        if (!live) return;
        if (COOP && __popc(live) <= kCoopRays && FeedDry(feed) && CoopReady<SPILL>(s, stk, live)) break;
        if (qi >= 0 && TraceRound<NodeT, true, SPILL, kPathLeaves, kPathLack<COOP>>(s, nodes, tris, ntri, stk, Q.err)) {
            if (s.bestSlot < 0) AddShadow(P, Q.shadow[qi]);
            qi = -1;
        }
    }
    if (COOP) {
        CoopFinish<NodeT, true, SPILL, !UNIFORM>(s, stk, qi >= 0, nodes, tris, ntri, sstack + (threadIdx.x & ~31u), Q.err);
        if (qi >= 0 && s.bestSlot < 0) AddShadow(P, Q.shadow[qi]);
    }
}

// Wavelength-independent BSDF data of a next-event direction v seen from r:
// the GGX pair, or for Lambertian the same-side gate and pdf |nv|/pi
// (LambertianBRDF::valueNM + LambertianSPF::Pdf, ShouldReflect at
// LambertianBRDF.cpp:44-75).  The sampling pdf is wavelength-independent.
__device__ __forceinline__ GgxPair NeePair(int mtype, const GgxPoint& gp, V3 ns, V3 ng, V3 r, V3 v)
{
    if (mtype == kMatGGX) return GgxPairAt(gp, dot(r, ns) < 0.0f ? -ns : ns, ng, r, v);
    GgxPair q;
    const float nr = dot(ns, r), nv = dot(ns, v);
    const bool same = (nr >= kNearZero && nv >= kNearZero) || (nr <= -kNearZero && nv <= -kNearZero);
    q.ok = same && dot(v, ng) > 0.0f && dot(r, ng) > 0.0f;
    q.sf = q.rh = q.ms = 0.0f;
    q.pdf = q.ok ? fabsf(nv) * kInvPi : 0.0f;
    return q;
}

// Top of a path's index-of-refraction stack (entries from x upward, -1 past
// the top); the stack is read only when it holds a mesh.
__device__ __forceinline__ int MediaTop(int4 m)
{
    return m.w >= 0 ? m.w : (m.z >= 0 ? m.z : (m.y >= 0 ? m.y : m.x));
}

// The index a stack entry stands for: its dielectric's at the hero
// wavelength, as IORStack::push records it (DielectricSPF.cpp:198-207).
__device__ __noinline__ float MeshIor(const PtScene& S, int mesh, float lam)
{
    const PtMaterial M = S.mats[__ldg(S.mesh_mat + mesh)];
    return M.eta >= 0 ? Spec(S.spectra, M.eta, lam) : M.ior;
}

// The shading point's spectra at its four wavelengths, looked up once: the
// Lambertian reflectance or the GGX specular colour, the conductor's optical
// constants and its Fresnel average for the medium around the hit.
struct PointSpectra {
    float4 refl, eta, k, favg;
};

__device__ __forceinline__ GgxParams GgxOf(const PtMaterial& M, const PointSpectra& ps, int j, float amb)
{
    return GgxFrom(M, Get(ps.refl, j), Get(ps.eta, j), Get(ps.k, j), Get(ps.favg, j), amb);
}

// The BSDF value at wavelength j for a next-event pair.
__device__ __forceinline__ float NeeValue(int mtype, const PtMaterial& M, const PointSpectra& ps, int j,
                                          const GgxPair& q, float eavg, float amb)
{
    if (!q.ok) return 0.0f;
    if (mtype == kMatGGX) return GgxValueAt(q, GgxOf(M, ps, j, amb), eavg);
    return Get(ps.refl, j) * kInvPi;
}

// Radiance of the sky, or the image environment, that an escaped path sees:
// uniform sky (IntegrateRayHWSS :5076-5120 for camera rays; :4235-4303 with MIS
// against sky NEE for continuations), or the image environment, weighted
// against its importance sampling by EnvironmentSampler::Pdf (:4255-4283).
template <bool ENV>
__device__ __forceinline__ void AddSky(const PtScene& S, const PtSettings& set, int depth, V3 d, float bsdfPdf,
                                       unsigned term, const float (&lam)[4], const float4& thr, float4& L)
{
    if (ENV && S.env_map && (depth > 0 || set.env_visible)) {
        const EnvSpec es = EnvLookupAt(S.env_map, d);
        float w = 1.0f;
        if (bsdfPdf > 0.0f) {
            const float ep = EnvPdfAt(S.env_map, d);
            if (ep > 0.0f) w = PowerHeuristic(bsdfPdf, ep);
        }
        for (int k = 0; k < 4; ++k)
            if (!(term & (1u << k))) Set(L, k, Get(L, k) + Get(thr, k) * EnvSpectrum(es, lam[k]) * w);
    } else if (set.env >= 0 && (depth > 0 || set.env_visible)) {
        const float w = bsdfPdf > 0.0f ? PowerHeuristic(bsdfPdf, kInv4Pi) : 1.0f;
        for (int k = 0; k < 4; ++k)
            if (!(term & (1u << k))) Set(L, k, Get(L, k) + Get(thr, k) * Spec(S.spectra, set.env, lam[k]) * w);
    }
}

// Sort the active paths into shading classes (Lambertian, GGX, dielectric,
// escaped) so KShade's warps each run one material model.
__global__ void __launch_bounds__(kShadeBlock)
KClassify(const PtJobDev* __restrict__ jobs, PtPaths P, PtQueues Q)
{
    ChainStart();
    const int n = Q.cnt[kCntActive];
    const int stride = gridDim.x * blockDim.x;
    for (int base = blockIdx.x * blockDim.x; base < n; base += stride) {
        const int i = base + threadIdx.x;
        int cls = -1, slot = -1;
        if (i < n) {
            slot = Q.active[i];
            const int hslot = __float_as_int(P.hit[slot].y);
            cls = kClassEscaped;
            if (hslot >= 0) {
                const PtScene& S = jobs[PathJob(P, slot)].scene;
                cls = S.mats[S.attr[hslot].mat & kAttrMatMask].type;
            }
        }
        int* const queues[kShadeClasses] = {&Q.cnt[kCntClass], &Q.cnt[kCntClass + 1], &Q.cnt[kCntClass + 2],
                                            &Q.cnt[kCntClass + kClassEscaped]};
        const int count[kShadeClasses] = {cls == 0, cls == 1, cls == 2, cls == kClassEscaped};
        int at[kShadeClasses];
        WarpAppend(queues, count, at);
        if (cls >= 0) Q.shade[cls * Q.capacity + at[cls]] = slot;
    }
}

// Escaped paths after KClassify: the sky's radiance, and the end of the path.
// In KShade<0> they left half of the lanes of a Lambertian warp idle (16 of 32
// active): 189 us an iteration of the 800k-triangle scene together, 109 and 24
// apart.
template <bool ENV, bool ONE>
__global__ void __launch_bounds__(kShadeBlock)
KEscape(const PtJobDev* __restrict__ jobs, PtPaths P, PtQueues Q, const __grid_constant__ PtJobDev one)
{
    ChainStart();
    const int n = Q.cnt[kCntClass + kClassEscaped];
    const int* __restrict__ src = Q.shade + kClassEscaped * Q.capacity;
    const int lane = threadIdx.x & 31;
    for (int base = blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += gridDim.x * blockDim.x) {
        const bool valid = base + lane < n;
        int slot = -1;
        if (valid) {
            slot = src[base + lane];
            float4 aux, meta, thr, L;
            LoadPair(P.state + slot, aux, meta);
            LoadPair(P.rad + slot, thr, L);
            const uint4 m = Bits(meta);
            const float4 rd = P.ray[slot].b;
            const PtJobDev& J = JobOf<ONE>(jobs, one, __float_as_int(aux.z));
            float lam[4];
            Wavelengths(aux.x, J.set.lmin, J.set.lmax, lam);
            AddSky<ENV>(J.scene, J.set, (int)(m.z & kFlagDepthMask), xyz(rd), aux.y, (m.z >> kTermShift) & 0xfu, lam,
                        thr, L);
            P.rad[slot].b = L;
            SetFlags(P, slot, m.z | kFlagFinishing);
        }
        int* const queues[1] = {&Q.cnt[kCntFreeNext]};
        const int count[1] = {valid};
        int at[1];
        WarpAppend(queues, count, at);
        if (valid) Q.free_next[at[0]] = slot;
    }
}

// CLS >= 0: every path to shade hit a material of shading class CLS (0
// Lambertian, 1 GGX, 2 dielectric) or escaped, so the other models' code is
// left out and the kernel needs fewer registers; the paths come from
// KClassify's queue of that class (from_class, no escaped ones) or, for scenes
// of one class, straight from the active queue.  CLS = -1 shades any material from the active queue.
// ENV: compiled with the image-environment code (some job's scene has one).
template <int CLS, bool ENV, bool ONE>
__global__ void __launch_bounds__(kShadeBlock, CLS == 1 || CLS < 0 ? 2 : 3)
KShade(const PtJobDev* __restrict__ jobs, PtPaths P, PtQueues Q, int from_class, int parity,
       const __grid_constant__ PtJobDev one)
{
    ChainStart();
    const int n = (CLS >= 0 && from_class) ? Q.cnt[kCntClass + (CLS < 0 ? 0 : CLS)] : Q.cnt[kCntActive];
    const int* __restrict__ src = (CLS >= 0 && from_class) ? Q.shade + (CLS < 0 ? 0 : CLS) * Q.capacity : Q.active;
    // Next events found by the threads of a block, up to four light and four sky
    // samples each (direction, distance, contribution).  They wait here until
    // the warp has all of its paths' and appends them to the shadow queue at
    // once, instead of with an atomic and the wait for it each; a path's entries
    // land side by side, so the connection kernel's lanes trace neighbouring
    // rays (800k-triangle scene at 8 spp: 33.2 -> 31.7 ms).
    __shared__ float4 s_dir[8][kShadeBlock];
    __shared__ float s_con[8][kShadeBlock];
    const int tid = threadIdx.x;
    for (int base = blockIdx.x * blockDim.x + (tid & ~31); base < n; base += gridDim.x * blockDim.x) {
        const bool valid = base + (tid & 31) < n;
        const int slot = valid ? src[base + (tid & 31)] : -1;
        unsigned events = 0;     // next events found: light sample k in bit k, sky sample k in bit 4 + k
        bool shared_event = false;   // each carries all four wavelengths (samples 0 only)
        bool cont = false;
        V3 p, nface;
        bool ng_flipped = false;
        if (valid) {
            float4 aux, meta, ro, rd, thr, L;
            LoadPair(P.state + slot, aux, meta);
            LoadPair(P.ray + slot, ro, rd);
            LoadPair(P.rad + slot, thr, L);
            const PtJobDev& J = JobOf<ONE>(jobs, one, __float_as_int(aux.z));
            const PtScene& S = J.scene;
            const PtSettings& set = J.set;
            uint4 m = Bits(meta);
            const float4 h = P.hit[slot];
            const int depth = (int)(m.z & kFlagDepthMask);
            // Random numbers: hash key or Sobol seed in meta.w, sample index in meta.y.
            VertexRng rng{m.w, m.y, depth, set.sampler, 0u, 0u, 0u};
            const float bsdfPdf = aux.y;
            unsigned term = (m.z >> kTermShift) & 0xfu;
            float lam[4];
            Wavelengths(aux.x, set.lmin, set.lmax, lam);
            const V3 d = xyz(rd);
            const int hslot = __float_as_int(h.y);

            do {
                if (hslot < 0) {
                    AddSky<ENV>(S, set, depth, d, bsdfPdf, term, lam, thr, L);
                    break;
                }
                // Runaway-throughput guard (IntegrateFromHitHWSS :4094-4110).
                {
                    float mx = 0.0f;
                    bool bad = false;
                    for (int k = 0; k < 4; ++k) {
                        const float v = Get(thr, k);
                        if (!isfinite(v)) bad = true;
                        mx = fmaxf(mx, fabsf(v));
                    }
                    if (bad || mx > 1e6f) break;
                }
                const float t = h.x;
                p = xyz(ro) + d * t;
                float4 A, B, C;
                LoadVertices(S.tris, hslot, A, B, C);
                nface = normalize(cross(xyz(B) - xyz(A), xyz(C) - xyz(A)));
                const PtTriAttr at = S.attr[hslot];
                const int mi = at.mat & kAttrMatMask;
                // Shading normal: the vertex normals interpolated at the hit,
                // n0 + (n1 - n0) a + (n2 - n0) b normalised, else the face normal
                // (TriangleMeshGeometryIndexedSpecializations.h:194-199,
                // Object.cpp:543); the geometric normal is the face normal turned
                // to the shading normal's side.
                V3 ns0 = nface;
                if (at.mat & kAttrSmooth) {
                    const uint4 q = __ldg(S.tri_normals + hslot);
                    const V3 n0 = OctDecode(q.x), n1 = OctDecode(q.y), n2 = OctDecode(q.z);
                    ns0 = normalize(n0 + (n1 - n0) * h.z + (n2 - n0) * h.w);
                }
                ng_flipped = dot(nface, ns0) < 0.0f;
                V3 ng = ng_flipped ? -nface : nface;
                V3 ns = ns0;
                // Double-sided meshes turn both towards the incoming ray
                // (TriangleMeshGeometryIndexed.cpp:170-188).
                if (at.mat & kAttrDoubleSided) {
                    if (dot(ns, d) > 0.0f) ns = -ns;
                    if (dot(ng, d) > 0.0f) {
                        ng = -ng;
                        ng_flipped = !ng_flipped;
                    }
                }
                const V3 gnv = dot(ng, d) < 0.0f ? ng : -ng;   // geometric normal facing the ray
                const PtMaterial M = S.mats[mi];
                const int mtype = CLS < 0 ? M.type : CLS;
                // The path's index-of-refraction stack (IORStack.h); its top is
                // the medium around the hit, the ambient index of a conductor
                // (PathTracingIntegrator.cpp:4315-4322).  Lambertian shading
                // needs neither.
                int4 med = make_int4(-1, -1, -1, -1);
                float amb = 1.0f;
                if (CLS != 0 && (m.z & kFlagInMedium)) {
                    med = P.media[slot];
                    amb = MeshIor(S, MediaTop(med), lam[0]);
                }
                bool media_changed = false;

                // PART 1: emission with MIS against light sampling (:4424-4518).
                if (M.emit >= 0 && (m.z & kFlagConsiderEmission) && dot(-d, ng) > 0.0f) {
                    float w = 1.0f;
                    if (bsdfPdf > 0.0f && at.light >= 0) {
                        const PtLight lg = S.lights[at.light];
                        const float cosL = fabsf(dot(d, ng));
                        // Selection probability from the previous vertex (the ray's origin).
                        const float psel = (set.light_bvh && S.light_nodes) ? LightBvhPdf(S.light_nodes, lg.bvh_pos, xyz(ro))
                                                                             : lg.pdf;
                        if (cosL > 0.0f && lg.area > 0.0f) w = PowerHeuristic(bsdfPdf, psel * (t * t) / (lg.area * cosL));
                    }
                    for (int k = 0; k < 4; ++k)
                        if (!(term & (1u << k))) Set(L, k, Get(L, k) + Get(thr, k) * Spec(S.spectra, M.emit, lam[k]) * w);
                }

                float4 kray = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                V3 nd;
                float npdf = 0.0f;       // continuation pdf for the next emission MIS (0 = delta)
                unsigned nflags = kFlagConsiderEmission;
                int btype = kBounceDiffuse;   // ScatteredRay type of the continuation

                if (mtype == kMatDielectric) {
                    // Smooth dielectric: Fresnel choice between reflection and
                    // refraction (DielectricSPF.cpp:120-300) at the hero's index.
                    // With a constant index every wavelength follows the hero's
                    // direction with the same weight, so the bundle continues
                    // together; where a companion's index differs from the hero's
                    // (by more than 1e-8, GetSpecularInfoNM), the companions end
                    // and the hero goes on alone (TerminateSecondary,
                    // PathTracingIntegrator.cpp:4658-4677).
                    const float ior = M.eta >= 0 ? Spec(S.spectra, M.eta, lam[0]) : M.ior;
                    if (M.eta >= 0 && (term & 0xeu) != 0xeu) {
                        #pragma unroll 1
                        for (int k = 1; k < 4; ++k) {
                            if (!(term & (1u << k)) && fabsf(Spec(S.spectra, M.eta, lam[k]) - ior) > 1e-8f) {
                                term |= 0xeu;
                                m.z |= 0xeu << kTermShift;
                                break;
                            }
                        }
                    }
                    // Inside or outside from the stack, not the facing
                    // (DielectricSPF.cpp:406-418): inside, the ray leaves for the
                    // medium under this mesh's entry (:177-183); outside, it comes
                    // from the stack's top (:198-207).  w is ri.onb.w(), the
                    // shading normal turned towards the ray on a double-sided mesh.
                    const int mesh = at.light >= 0 ? S.lights[at.light].mesh : ~at.light;
                    int e[kPtMediaDepth] = {med.x, med.y, med.z, med.w};
                    int depthIn = 0, pos = -1;
                    #pragma unroll
                    for (int i = 0; i < kPtMediaDepth; ++i) {
                        if (e[i] >= 0) depthIn = i + 1;
                        if (e[i] == mesh) pos = i;
                    }
                    const bool fromInside = pos >= 0;
                    float exitIor = 1.0f;
                    if (fromInside) {
                        const int below = pos == depthIn - 1 ? (depthIn >= 2 ? e[depthIn - 2] : -1) : e[depthIn - 1];
                        if (below >= 0) exitIor = MeshIor(S, below, lam[0]);
                    }
                    const float n1 = fromInside ? ior : amb, n2 = fromInside ? exitIor : ior;
                    const V3 w = ns;
                    const V3 nEff = fromInside ? -w : w;
                    const V3 geomN = dot(ng, nEff) >= 0.0f ? ng : -ng;
                    // Snell's law with the normal turned against the ray
                    // (Optics.cpp:84-98); Fresnel on absolute cosines (:101-159).
                    const V3 nf = dot(w, d) > 0.0f ? -w : w;
                    const float cosI = -dot(d, nf);
                    const float eta = n1 / n2;
                    const float s2t = eta * eta * fmaxf(0.0f, 1.0f - cosI * cosI);
                    const bool snell = 1.0f - s2t >= kNearZero;
                    float R = 1.0f;
                    V3 tdir = mk(0.0f, 0.0f, 0.0f);
                    if (snell) {
                        const float cosT = sqrtf(1.0f - s2t);
                        tdir = normalize(d * eta + nf * (eta * cosI - cosT));
                        R = DielectricR(cosI, cosT, n1, n2);
                    }
                    // ScatterNM's two numbers (DielectricSPF.cpp:421) tilt the
                    // transmitted direction by a Phong lobe of the material's
                    // exponent: acos(u^(1/(n+1))) off it, uniform in azimuth
                    // (GenerateScatteredRay, :248-272; none at 0 or >= 1e6).
                    const float u1 = rng.next(16), u2 = rng.next(17);
                    bool refr = snell;
                    if (refr && M.alpha > 0.0f && M.alpha < 1e6f) {
                        const float a = acosf(powf(u1, 1.0f / (M.alpha + 1.0f)));
                        if (a > 0.0f && a < 0.5f * kPi) {
                            V3 tx, ty;
                            Basis(tdir, tx, ty);
                            float sp, cp, sa, ca;
                            __sincosf(2.0f * kPi * u2, &sp, &cp);
                            sincosf(a, &sa, &ca);
                            tdir = normalize(tdir * ca + (tx * cp + ty * sp) * sa);
                        }
                    }
                    // The transmitted ray must cross to the far side of w's
                    // crossing (:274-279); the reflected one must stay above the
                    // geometric normal on that side, and under total internal
                    // reflection mirrors about it instead (:221-243).
                    if (refr && !(dot(tdir, nEff) < -kNearZero)) refr = false;
                    V3 rdir = normalize(d - w * (2.0f * dot(d, w)));
                    bool refl = true;
                    if (!(dot(rdir, geomN) > 0.0f)) {
                        if (R >= 1.0f) rdir = normalize(d - geomN * (2.0f * dot(d, geomN)));
                        else refl = false;
                    }
                    // RandomlySelect over (transmitted 1 - R, reflected R)
                    // (ScatteredRayContainer.cpp:43-70); a lobe the reference
                    // drops ends the path here with the same expectation.  The
                    // transmitted ray carries the stack with this mesh pushed or
                    // removed (PathTracingIntegrator.cpp:4814-4816).
                    if (rng.next(18) < 1.0f - R) {
                        if (!refr) break;
                        nd = tdir;
                        btype = kBounceTransmission;
                        if (fromInside) {
                            #pragma unroll
                            for (int i = 0; i < kPtMediaDepth - 1; ++i)
                                if (i >= pos) e[i] = e[i + 1];
                            e[kPtMediaDepth - 1] = -1;
                        } else {
                            if (depthIn == kPtMediaDepth) break;   // deeper than the stack kept per path
                            #pragma unroll
                            for (int i = 0; i < kPtMediaDepth; ++i)
                                if (i == depthIn) e[i] = mesh;
                        }
                        med = make_int4(e[0], e[1], e[2], e[3]);
                        media_changed = true;
                    } else {
                        if (!refl) break;
                        nd = rdir;
                        btype = kBounceGlossy;
                    }
                    for (int k = 0; k < 4; ++k) Set(kray, k, (term & (1u << k)) ? 0.0f : 1.0f);
                    nflags |= kFlagSpecular;
                } else {
                    const V3 r = -d;
                    GgxPoint gp{1.0f, 0.0f, 0.0f, 0.0f};
                    PointSpectra ps;
                    ps.refl = ps.eta = ps.k = ps.favg = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (mtype == kMatGGX) {
                        gp = GgxPointAt(M.alpha, fabsf(dot(r, ns)));
                        #pragma unroll 1
                        for (int k = 0; k < 4; ++k) {
                            const float e = M.eta >= 0 ? Spec(S.spectra, M.eta, lam[k]) : M.ior;
                            const float kk = M.kappa >= 0 ? Spec(S.spectra, M.kappa, lam[k]) : 0.0f;
                            Set(ps.refl, k, M.refl >= 0 ? Spec(S.spectra, M.refl, lam[k]) : 1.0f);
                            Set(ps.eta, k, e);
                            Set(ps.k, k, kk);
                            Set(ps.favg, k, GgxFavg(M, S.spectra, lam[k], amb, e, kk));
                        }
                    } else {
                        #pragma unroll 1
                        for (int k = 0; k < 4; ++k) Set(ps.refl, k, Spec(S.spectra, M.refl, lam[k]));
                    }
                    // PART 2: next-event estimation (LightSampler::EvaluateDirectLightingNM,
                    // LightSampler.cpp:1942-2361): one area-light sample and one sky
                    // sample per wavelength (reference) or one shared sample.
                    const int nsamp = set.nee_per_lambda ? 4 : 1;
                    shared_event = !set.nee_per_lambda;
                    const auto stage = [&](int event, int k, const float4& c, const V3& dir, float tmax) {
                        events |= 1u << event;
                        s_dir[event][tid] = make_float4(dir.x, dir.y, dir.z, tmax);
                        if (set.nee_per_lambda) {
                            s_con[event][tid] = Get(c, k);
                        } else {
                            for (int j = 0; j < 4; ++j) s_con[event + j][tid] = Get(c, j);
                        }
                    };
                    #pragma unroll 1
                    for (int k = 0; k < nsamp; ++k) {
                        if (set.nee_per_lambda && (term & (1u << k))) continue;
                        // Wavelengths that share this light sample.
                        const int j0 = set.nee_per_lambda ? k : 0, j1 = set.nee_per_lambda ? k + 1 : 4;
                        if (set.n_lights > 0) {
                            const float ul = rng.next(4 * k + 0);
                            int li = 0;
                            float psel;
                            if (set.light_bvh && S.light_nodes) {
                                li = SampleLightBvh(S.light_nodes, p, ul, psel);
                            } else {
                                // Alias table (AliasTable::Sample): one number
                                // picks an entry and decides between it and its alias.
                                const float sc = ul * (float)set.n_lights;
                                const int idx = min((int)sc, set.n_lights - 1);
                                const PtLightAlias al = S.light_alias[idx];
                                li = (sc - (float)idx < al.prob) ? idx : al.alias;
                                psel = S.lights[li].pdf;
                            }
                            // No sample when nothing can be picked, nor from a luminary to itself.
                            if (li >= 0 && S.lights[li].kind == 1 && psel > 0.0f) {
                                // Point light (LightSampler.cpp:2097-2130): luminance of
                                // colour x power, cos / d^2, no MIS (a delta light).
                                const PtLight lg = S.lights[li];
                                V3 toL = mk(lg.pos[0], lg.pos[1], lg.pos[2]) - p;
                                const float dist = sqrtf(dot(toL, toL));
                                toL = toL * (1.0f / dist);
                                const float cosS = dot(toL, ns);
                                if (dist > 0.0f && cosS > 0.0f) {
                                    float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                                    bool any = false;
                                    const GgxPair bq = NeePair(mtype, gp, ns, gnv, r, toL);
                                    #pragma unroll 1
                                    for (int j = j0; j < j1; ++j) {
                                        if (term & (1u << j)) continue;
                                        const float f = NeeValue(mtype, M, ps, j, bq, gp.eavg, amb);
                                        const float v = Get(thr, j) * lg.le * f * cosS / (dist * dist) / psel;
                                        Set(c, j, v);
                                        any |= v != 0.0f;
                                    }
                                    if (any) stage(k, k, c, toL, dist - 0.001f);
                                }
                            } else if (li >= 0 && li != at.light && psel > 0.0f) {
                                const PtLight lg = S.lights[li];
                                const float ux = rng.next(4 * k + 1);
                                const float uy = rng.next(4 * k + 2);
                                const float uz = rng.next(4 * k + 3);
                                // First triangle whose area CDF reaches uz: binary
                                // search (std::lower_bound over the areas CDF,
                                // TriangleMeshGeometryIndexed.cpp:207-217).
                                int tsel = lg.first, hi = lg.first + lg.count - 1;
                                while (tsel < hi) {
                                    const int mid = (tsel + hi) >> 1;
                                    if (__ldg(&S.light_tris[mid].cdf) >= uz) hi = mid;
                                    else tsel = mid + 1;
                                }
                                const PtLightTri lt = S.light_tris[tsel];
                                // GeometricUtilities::PointOnTriangle (GeometricUtilities.cpp:543-569).
                                const float sa = sqrtf(1.0f - ux);
                                const float alpha = 1.0f - sa, beta = sa * uy;
                                const V3 e1 = mk(lt.e1[0], lt.e1[1], lt.e1[2]), e2 = mk(lt.e2[0], lt.e2[1], lt.e2[2]);
                                const V3 pl = mk(lt.v0[0], lt.v0[1], lt.v0[2]) + e1 * alpha + e2 * beta;
                                const V3 nl = normalize(cross(e1, e2));
                                V3 toL = pl - p;
                                const float dist = sqrtf(dot(toL, toL));
                                toL = toL * (1.0f / dist);
                                const float cosS = dot(toL, ns);
                                const float cosL = dot(-toL, nl);
                                if (cosL > 0.0f && cosS > 0.0f) {
                                    const float geom = lg.area * cosL / (dist * dist);
                                    const float plight = psel * (dist * dist) / (lg.area * cosL);
                                    float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                                    bool any = false;
                                    const GgxPair bq = NeePair(mtype, gp, ns, gnv, r, toL);
                                    const float pb = bq.pdf;
                                    #pragma unroll 1
                                    for (int j = j0; j < j1; ++j) {
                                        if (term & (1u << j)) continue;
                                        const float f = NeeValue(mtype, M, ps, j, bq, gp.eavg, amb);
                                        const float w = (pb > 0.0f ? PowerHeuristic(plight, pb) : 1.0f) / psel;
                                        const float v = Get(thr, j) * Spec(S.spectra, lg.emit, lam[j]) * cosS * geom * f * w;
                                        Set(c, j, v);
                                        any |= v != 0.0f;
                                    }
                                    if (any) stage(k, k, c, toL, dist - 0.001f);
                                }
                            } else if (!(li >= 0 && S.lights[li].kind == 1 && psel > 0.0f)) {
                                // Nothing to sample, or the luminary being shaded:
                                // the reference still draws the point's three
                                // numbers (LightSampler.cpp:2064-2096).
                                rng.skip(3);
                            }
                        }
                        if (set.env >= 0 || (ENV && S.env_map)) {
                            // Environment NEE (LightSampler.cpp:2271-2359): the
                            // image environment's importance table
                            // (EnvironmentSampler::Sample), or for a uniform sky
                            // uniform directions with pdf 1/(4 pi).
                            const float u1 = rng.next(20 + 2 * k);
                            const float u2 = rng.next(21 + 2 * k);
                            V3 dir;
                            float epdf;
                            EnvSpec es{0.0f, 0.0f, 0.0f, 0.0f};
                            if (ENV && S.env_map) {
                                epdf = EnvSampleAt(S.env_map, u1, u2, dir);
                                if (epdf > 0.0f) es = EnvLookupAt(S.env_map, dir);
                            } else {
                                const float z = 1.0f - 2.0f * u1;
                                const float rr = sqrtf(fmaxf(0.0f, 1.0f - z * z));
                                float sp, cp;
                                __sincosf(2.0f * kPi * u2, &sp, &cp);
                                dir = mk(rr * cp, rr * sp, z);
                                epdf = kInv4Pi;
                            }
                            const float cosE = dot(dir, ns);
                            if (cosE > 0.0f && epdf > 0.0f) {
                                float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                                bool any = false;
                                const GgxPair bq = NeePair(mtype, gp, ns, gnv, r, dir);
                                const float pb = bq.pdf;
                                #pragma unroll 1
                                for (int j = j0; j < j1; ++j) {
                                    if (term & (1u << j)) continue;
                                    const float f = NeeValue(mtype, M, ps, j, bq, gp.eavg, amb);
                                    const float w = pb > 0.0f ? PowerHeuristic(epdf, pb) : 1.0f;
                                    const float le = (ENV && S.env_map) ? EnvSpectrum(es, lam[j])
                                                                        : Spec(S.spectra, set.env, lam[j]);
                                    const float v = Get(thr, j) * le * f * cosE / epdf * w;
                                    Set(c, j, v);
                                    any |= v != 0.0f;
                                }
                                if (any) stage(4 + k, k, c, dir, __int_as_float(0x7f800000));
                            }
                        }
                    }

                    // PART 3: hero-wavelength BSDF sample (:4597-4719).
                    const V3 w = dot(d, ns) > kNearZero ? -ns : ns;   // viewer side
                    const V3 gn = gnv;
                    V3 tx, ty;
                    Basis(w, tx, ty);
                    // GGXSPF::ScatterNM draws the lobe choice before the
                    // direction (GGXSPF.cpp:478-520); LambertianSPF the direction.
                    const float ulobe = mtype == kMatGGX ? rng.next(18) : 0.0f;
                    const float u1 = rng.next(16), u2 = rng.next(17);
                    if (mtype == kMatGGX) {
                        const GgxParams g0 = GgxOf(M, ps, 0, amb);
                        const float cosR = dot(r, w);
                        const float ws = g0.spec;
                        const float wms = ws * (1.0f - gp.essR);
                        const float total = ws + wms;
                        if (!(total > 1e-10f)) break;
                        const float pSpec = ws / total, pMS = wms / total;
                        const float msz = gp.msz;
                        float khero = 0.0f;
                        if (ulobe < pSpec) {
                            btype = kBounceGlossy;
                            const V3 mh = VndfSample(r, tx, ty, w, g0.alpha, u1, u2);
                            const float rm = dot(r, mh);
                            if (!(rm > 0.0f)) break;
                            nd = normalize(mh * (2.0f * rm) - r);
                            const float cosO = dot(nd, w);
                            if (!(cosO > 0.0f && dot(nd, gn) > 0.0f)) break;
                            const float vpdf = VndfPdf(r, nd, w, g0.alpha);
                            if (!(vpdf > 1e-10f)) break;
                            npdf = (wms * MsPdf(cosO, g0.alpha, msz) + ws * vpdf) / total;
                            const float G2 = 1.0f / (1.0f + GgxLambda(g0.alpha, cosR) + GgxLambda(g0.alpha, cosO));
                            const float G1 = 1.0f / (1.0f + GgxLambda(g0.alpha, cosR));
                            khero = g0.spec * ConductorF(rm, amb, g0.eta, g0.k) * G2 / (G1 * pSpec);
                        } else {
                            // Multiple-scattering lobe: mu_o from (1 - E(mu_o)) mu_o,
                            // uniform azimuth (GGXSPF.cpp:604-675).
                            const float eavg = gp.eavg;
                            if (!(pMS > 1e-10f && 1.0f - eavg > 1e-10f)) break;
                            const float cost = MsSampleCos(g0.alpha, u1);
                            const float sint = sqrtf(fmaxf(0.0f, 1.0f - cost * cost));
                            float sp, cp;
                            __sincosf(2.0f * kPi * u2, &sp, &cp);
                            nd = normalize(tx * (cp * sint) + ty * (sp * sint) + w * cost);
                            const float cosO = dot(nd, w);
                            if (!(cosO > 0.0f && dot(nd, gn) > 0.0f)) break;
                            const float mpdf = MsPdf(cosO, g0.alpha, msz);
                            if (!(mpdf > 1e-14f)) break;
                            npdf = (wms * mpdf + ws * VndfPdf(r, nd, w, g0.alpha)) / total;
                            const float fms = Fms(g0.spec * g0.favg, eavg) * (1.0f - LookupEss(cosO, g0.alpha)) *
                                              (1.0f - gp.essR) / (kPi * (1.0f - eavg));
                            khero = fms * cosO / (mpdf * pMS);
                        }
                        if (!(npdf > 0.0f)) break;
                        Set(kray, 0, (term & 1u) ? 0.0f : khero);
                        const float cosV = fabsf(dot(nd, ns));
                        // Companions evaluate the BSDF in the hero's direction and
                        // divide by the hero's pdf (:4676-4714).
                        const GgxPair cq = GgxPairAt(gp, w, gnv, r, nd);
                        #pragma unroll 1
                        for (int k = 1; k < 4; ++k) {
                            if (term & (1u << k)) continue;
                            Set(kray, k, GgxValueAt(cq, GgxOf(M, ps, k, amb), gp.eavg) * cosV / npdf);
                        }
                    } else {
                        // Lambertian: cosine-weighted direction, kray = rho(lambda),
                        // pdf = cos/pi (LambertianSPF.cpp:90-160).
                        const float phi = 2.0f * kPi * u1;
                        const float sint = sqrtf(u2), cost = sqrtf(1.0f - u2);
                        float sp, cp;
                        __sincosf(phi, &sp, &cp);
                        nd = normalize(tx * (cp * sint) + ty * (sp * sint) + w * cost);
                        npdf = fabsf(dot(nd, w)) * kInvPi;
                        // Geometric-horizon gate (LambertianSPF.cpp:141-151).
                        if (!(dot(nd, gn) > 0.0f)) break;
                        for (int k = 0; k < 4; ++k) Set(kray, k, (term & (1u << k)) ? 0.0f : Get(ps.refl, k));
                    }
                    // The integrator's choice among the scattered rays
                    // (ScatteredRayContainer::RandomlySelect; one ray here).
                    rng.skip(1);
                }
                // Russian roulette on the max over wavelengths (:4738-4769,
                // PathTransportUtilities.h:86-110).
                float prevMax = 0.0f, currMax = 0.0f;
                for (int k = 0; k < 4; ++k) {
                    if (term & (1u << k)) continue;
                    prevMax = fmaxf(prevMax, fabsf(Get(thr, k)));
                    currMax = fmaxf(currMax, fabsf(Get(thr, k) * Get(kray, k)));
                }
                if (currMax <= kNearZero) break;
                if (depth >= set.rr_min_depth) {
                    const float prob = fminf(1.0f, currMax / fmaxf(prevMax, set.rr_threshold));
                    if (rng.next(19) >= prob) break;
                    if (prob > 0.0f && prob < 1.0f) {
                        const float s = 1.0f / prob;
                        kray = make_float4(kray.x * s, kray.y * s, kray.z * s, kray.w * s);
                    }
                }
                // Per-type bounce limits (PropagateBounceLimits,
                // PathTransportUtilities.h:170-221), checked after Russian roulette
                // as the reference does (:4770-4790).
                unsigned bounces = __float_as_uint(aux.w);
                {
                    const unsigned c = ((bounces >> (8 * btype)) & 0xffu) + 1u;
                    if ((int)c > set.max_bounce[btype]) break;
                    bounces = (bounces & ~(0xffu << (8 * btype))) | (c << (8 * btype));
                }
                if (depth + 1 >= set.max_depth) break;
                thr = make_float4(thr.x * kray.x, thr.y * kray.y, thr.z * kray.z, thr.w * kray.w);
                const V3 no = OffsetRay(p, nface, nd);
                StorePair(P.ray + slot, make_float4(no.x, no.y, no.z, 0.0f),
                          make_float4(nd.x, nd.y, nd.z, __int_as_float(0x7f800000)));
                m.z = (m.z & ~(kFlagDepthMask | kFlagSpecular)) | (unsigned)(depth + 1) | nflags;
                if (media_changed) {
                    P.media[slot] = med;
                    m.z = med.x >= 0 ? (m.z | kFlagInMedium) : (m.z & ~kFlagInMedium);
                }
                StorePair(P.state + slot, make_float4(aux.x, npdf, aux.z, __uint_as_float(bounces)), Floats(m));
                cont = true;
            } while (false);

            if (cont) {
                StorePair(P.rad + slot, thr, L);
            } else {
                P.rad[slot].b = L;
                SetFlags(P, slot, m.z | kFlagFinishing);
            }
        }
        int* const queues[3] = {&Q.cnt[kCntShadow], &Q.cnt[kCntNext + parity], &Q.cnt[kCntFreeNext]};
        const int count[3] = {__popc(events), cont, valid && !cont};
        int at[3];
        WarpAppend(queues, count, at);
        if (cont) Q.active_next[at[1]] = slot;
        else if (valid) Q.free_next[at[2]] = slot;
        while (events) {
            const int ev = __ffs(events) - 1, k = ev & 3;
            events &= events - 1u;
            const float4 dir = s_dir[ev][tid];
            const V3 o = OffsetRay(p, ng_flipped ? -nface : nface, xyz(dir));
            ShadowEntry e;
            e.o = make_float4(o.x, o.y, o.z, dir.w);
            e.d = make_float4(dir.x, dir.y, dir.z, __int_as_float(slot));
            if (shared_event) {
                e.c = make_float4(s_con[ev][tid], s_con[ev + 1][tid], s_con[ev + 2][tid], s_con[ev + 3][tid]);
            } else {
                const float c = s_con[ev][tid];
                e.c = make_float4(k == 0 ? c : 0.0f, k == 1 ? c : 0.0f, k == 2 ? c : 0.0f, k == 3 ? c : 0.0f);
            }
            Q.shadow[at[0]++] = e;
        }
    }
}

__global__ void KIota(int* p, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = i;
}

// Kahan-compensated fold of this call's film into the running sums.
__global__ void KFold(float* pass, float* sum, float* comp, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float y = pass[i] - comp[i];
        const float s = sum[i];
        const float t = s + y;
        comp[i] = (t - s) - y;
        sum[i] = t;
        pass[i] = 0.0f;
    }
}

// Fold into the FP64 running sum used past 4096 spp; `first` moves the
// compensated FP32 sum over.
__global__ void KFoldWide(float* pass, float* sum, float* comp, double* wide, int n, int first)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double w = first ? (double)sum[i] - (double)comp[i] : wide[i];
        wide[i] = w + (double)pass[i];
        pass[i] = 0.0f;
        if (first) sum[i] = comp[i] = 0.0f;
    }
}

__device__ __forceinline__ double FilmValue(const float* __restrict__ sum, const float* __restrict__ comp,
                                            const double* __restrict__ wide, int k)
{
    return wide ? wide[k] : (double)sum[k] - (double)comp[k];
}

// relMSE of the resolved film (FP32 compensated or FP64 sums; 3 channels:
// sum / spp, 4 channels: weighted sum / weight, 0 where the weight is at most
// 1e-10) against `ref` (XYZ per pixel): sum over pixels and channels of
// (x - r)^2 / (r^2 + 1e-2), in FP64.
__global__ void KRelMse(const float* __restrict__ sum, const float* __restrict__ comp, const double* __restrict__ wide,
                        const unsigned* __restrict__ counts, const float* __restrict__ ref, int npix, int channels,
                        double inv_spp, double* out)
{
    double acc = 0.0;
    const int n3 = 3 * npix;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += gridDim.x * blockDim.x) {
        double x;
        if (channels == 3) {
            const unsigned c = counts ? counts[i / 3] : 1u;
            x = c ? FilmValue(sum, comp, wide, i) * (counts ? 1.0 / (double)c : inv_spp) : 0.0;
        } else {
            const int p = i / 3;
            const double w = FilmValue(sum, comp, wide, 4 * p + 3);
            x = fabs(w) > 1e-10 ? FilmValue(sum, comp, wide, 4 * p + i - 3 * p) / w : 0.0;
        }
        const double r = ref[i];
        acc += (x - r) * (x - r) / (r * r + 1e-2);
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(kFull, acc, o);
    __shared__ double part[32];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        acc = threadIdx.x < (blockDim.x >> 5) ? part[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(kFull, acc, o);
        if (threadIdx.x == 0) atomicAdd(out, acc);
    }
}

// Adaptive sampling after a batch of `batch` samples for each listed pixel
// (PathTracingSpectralRasterizer.cpp:379-408 with the Welford mean / M2
// formed from the sums of Y and Y^2): adds the batch to the pixel's count,
// tests convergence once it has 32 samples, and appends pixels still below
// the maximum and not converged to `next`.
__global__ void KConverge(const unsigned* __restrict__ list, int n, const double* __restrict__ lum,
                          unsigned* __restrict__ count, int batch, int max_spp, double threshold,
                          unsigned* __restrict__ next, int* __restrict__ n_next)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned p = list[i];
        const unsigned c = count[p] + (unsigned)batch;
        count[p] = c;
        bool converged = false;
        if (c >= 32) {
            const double N = (double)c, s1 = lum[2 * (size_t)p], s2 = lum[2 * (size_t)p + 1];
            const double mean = s1 / N;
            const double m2 = fmax(s2 - s1 * mean, 0.0);
            const double se = sqrt(m2 / (N - 1.0) / N), ma = fabs(mean);
            if (ma > 1e-12) converged = se / ma < threshold * (1.0 - 4.0 / N);
            else converged = m2 < 1e-12 && c >= 64;
        }
        if (!converged && (int)c < max_spp) next[atomicAdd(n_next, 1)] = p;
    }
}

// ---- host launchers ----------------------------------------------------------

namespace {

// Launch that may start while the stream's previous kernel still runs: the
// kernel begins with ChainStart.
template <class... P, class... A>
void Chain(void (*kernel)(P...), int grid, int block, cudaStream_t st, A... args)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

template <class K>
int TraceGrid(K kernel, int sms)
{
    int per = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kTraceBlock, 0) != cudaSuccess || per < 1) per = 1;
    return per * sms;
}
}  // namespace

// Grids cached per instantiation.
template <class NodeT, bool SPILL, bool UNIFORM, bool COOP>
void LaunchTraceKernels(const PtLaunch& L, cudaStream_t st, TraceKind kind, int parity)
{
    if (kind != TraceKind::Connect) {
        static int g = 0;
        if (!g) g = TraceGrid(KExtend<NodeT, SPILL, UNIFORM, COOP>, L.sms);
        Chain(KExtend<NodeT, SPILL, UNIFORM, COOP>, g, kTraceBlock, st, L.jobs, L.paths, L.queues, L.scene, parity, kind);
    } else {
        static int g = 0;
        if (!g) g = TraceGrid(KConnect<NodeT, SPILL, UNIFORM, COOP>, L.sms);
        Chain(KConnect<NodeT, SPILL, UNIFORM, COOP>, g, kTraceBlock, st, L.jobs, L.paths, L.queues, L.scene);
    }
}

template <class NodeT, bool SPILL, bool UNIFORM>
void LaunchTraceCoop(const PtLaunch& L, cudaStream_t st, TraceKind kind, int parity)
{
    if (L.coop) LaunchTraceKernels<NodeT, SPILL, UNIFORM, true>(L, st, kind, parity);
    else LaunchTraceKernels<NodeT, SPILL, UNIFORM, false>(L, st, kind, parity);
}

template <class NodeT>
void LaunchTraceLayout(const PtLaunch& L, cudaStream_t st, TraceKind kind, int parity)
{
    if (L.spill) {
        if (L.uniform) LaunchTraceCoop<NodeT, true, true>(L, st, kind, parity);
        else LaunchTraceCoop<NodeT, true, false>(L, st, kind, parity);
    } else {
        if (L.uniform) LaunchTraceCoop<NodeT, false, true>(L, st, kind, parity);
        else LaunchTraceCoop<NodeT, false, false>(L, st, kind, parity);
    }
}

void LaunchTrace(const PtLaunch& L, cudaStream_t st, TraceKind kind, int parity)
{
    if (L.layout == RTB200_BVH_Q8) LaunchTraceLayout<QNode4>(L, st, kind, parity);
    else if (L.layout == RTB200_BVH_F16) LaunchTraceLayout<HNode4>(L, st, kind, parity);
    else LaunchTraceLayout<GpuNode4>(L, st, kind, parity);
}

cudaError_t PtSetGgxTables(const float* ess, const float* eavg, const float* msz, const float* mscum,
                           const float* favg_x, const float* favg_w)
{
    cudaError_t e = cudaMemcpyToSymbol(g_ess, ess, sizeof(float) * kLut * kLut);
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_eavg, eavg, sizeof(float) * kLut);
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_msz, msz, sizeof(float) * kLut);
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_mscum, mscum, sizeof(float) * kLut * (kLut + 2));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_favg_x, favg_x, sizeof(float) * kFavgNodes);
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_favg_w, favg_w, sizeof(float) * kFavgNodes);
    return e;
}

template <int CLS>
void LaunchShade(const PtLaunch& L, int from_class, int parity, cudaStream_t st)
{
    const int grid = L.sms * 8;
    auto* kernel = L.env_image ? (L.one ? KShade<CLS, true, true> : KShade<CLS, true, false>)
                               : (L.one ? KShade<CLS, false, true> : KShade<CLS, false, false>);
    Chain(kernel, grid, kShadeBlock, st, L.jobs, L.paths, L.queues, from_class, parity, L.job);
}

cudaError_t PtIteration(const PtLaunch& L, int iter, cudaStream_t st)
{
    const int shadeGrid = L.sms * 8;
    const int parity = iter & 1;
    // The last iteration's shadow rays, and then this one's new paths, beside the
    // paths that go on: neither needs the other before shading.  Over small trees
    // (L.coop) the rays end sooner than the second extension and the joins take:
    // Cornell box at 16 spp 2.95 ms side by side and 2.86 one after the other,
    // 800k-triangle scene at 8 spp 25.8 and 26.6, 120 x 80 image of a 20k-triangle
    // scene 1.70 and 1.78.
    const cudaStream_t rays = L.coop ? L.side[0] : st;
    if (L.coop) {
        cudaEventRecord(L.fork, st);
        cudaStreamWaitEvent(rays, L.fork, 0);
        LaunchTrace(L, st, TraceKind::ExtendOld, parity);
    }
    LaunchTrace(L, rays, TraceKind::Connect, parity);
    Chain(KAssign, 1, kPtMaxJobs, rays, L.jobs, L.ids, L.queues, iter);
    Chain(L.one ? KRegen<true> : KRegen<false>, shadeGrid, kShadeBlock, rays, L.jobs, L.paths, L.queues, L.job);
    LaunchTrace(L, rays, L.coop ? TraceKind::ExtendNew : TraceKind::Extend, parity);
    if (L.coop) {
        cudaEventRecord(L.join[0], rays);
        cudaStreamWaitEvent(st, L.join[0], 0);
    }
    if (L.classify) {
        Chain(KClassify, shadeGrid, kShadeBlock, st, L.jobs, L.paths, L.queues);
        // The classes side by side: a late iteration's few paths are a wait for
        // one warp's instructions in each (9,600 pixels at 4 spp: 57, 27 and 9 us).
        cudaEventRecord(L.fork, st);
        cudaStreamWaitEvent(L.side[0], L.fork, 0);
        cudaStreamWaitEvent(L.side[1], L.fork, 0);
        LaunchShade<1>(L, 1, parity, st);
        LaunchShade<0>(L, 1, parity, L.side[0]);
        auto* escape = L.env_image ? (L.one ? KEscape<true, true> : KEscape<true, false>)
                                   : (L.one ? KEscape<false, true> : KEscape<false, false>);
        Chain(escape, shadeGrid, kShadeBlock, L.side[1], L.jobs, L.paths, L.queues, L.job);
        // Dielectrics shade no next events.
        Chain(L.one ? KShade<2, false, true> : KShade<2, false, false>, shadeGrid, kShadeBlock, L.side[1], L.jobs,
              L.paths, L.queues, 1, parity, L.job);
        for (int k = 0; k < 2; ++k) {
            cudaEventRecord(L.join[k], L.side[k]);
            cudaStreamWaitEvent(st, L.join[k], 0);
        }
    } else if (L.shade_class == 0) {
        LaunchShade<0>(L, 0, parity, st);
    } else if (L.shade_class == 1) {
        LaunchShade<1>(L, 0, parity, st);
    } else if (L.shade_class == 2) {
        // A dielectric-only scene: this kernel also shades the escaped rays.
        LaunchShade<2>(L, 0, parity, st);
    } else {
        LaunchShade<-1>(L, 0, parity, st);
    }
    return cudaGetLastError();
}

cudaError_t PtIota(int* p, int n, int sms, cudaStream_t st)
{
    KIota<<<sms * 4, 256, 0, st>>>(p, n);
    return cudaGetLastError();
}

cudaError_t PtFoldWide(float* pass, float* sum, float* comp, double* wide, int n, bool first, int sms,
                       cudaStream_t st)
{
    KFoldWide<<<sms * 4, 256, 0, st>>>(pass, sum, comp, wide, n, first ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t PtRelMse(const float* sum, const float* comp, const double* wide, const unsigned* counts,
                     const float* ref, int npix, int channels, double inv_spp, double* out, int sms, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(double), st);
    if (e != cudaSuccess) return e;
    KRelMse<<<sms * 2, 256, 0, st>>>(sum, comp, wide, counts, ref, npix, channels, inv_spp, out);
    return cudaGetLastError();
}

cudaError_t PtConverge(const unsigned* list, int n, const double* lum, unsigned* count, int batch, int max_spp,
                       double threshold, unsigned* next, int* n_next, int sms, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(n_next, 0, sizeof(int), st);
    if (e != cudaSuccess || n == 0) return e;
    KConverge<<<std::min(sms * 8, (n + 255) / 256), 256, 0, st>>>(list, n, lum, count, batch, max_spp, threshold,
                                                                  next, n_next);
    return cudaGetLastError();
}

cudaError_t PtFold(float* pass, float* sum, float* comp, int n, int sms, cudaStream_t st)
{
    KFold<<<sms * 4, 256, 0, st>>>(pass, sum, comp, n);
    return cudaGetLastError();
}

}  // namespace rtb200
