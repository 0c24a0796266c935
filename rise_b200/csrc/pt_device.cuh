// pt_device.cuh -- device helpers of the spectral path tracer: counter-based
// random numbers, spectra and CIE lookups, HWSS wavelengths, small vector
// algebra, ray-origin offsetting, MIS weights and warp-aggregated appends.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "cie1931.h"
#include "pt_types.h"

namespace rtb200 {

constexpr float kPi = 3.14159265358979323846f;
constexpr float kInvPi = 0.31830988618379067154f;
constexpr float kNearZero = 1e-12f;   // NEARZERO, Utilities/Math3D/Constants.h:33

// The colour-matching functions, a row (x, y, z, 0) per wavelength, in global
// memory: every lane of a warp reads its own wavelength, which constant memory
// would serialise (24 scalar reads a sample; KRegen spent most of its time
// there).  Defined here: this header is compiled into exactly one translation
// unit (pathtrace.cu).
struct alignas(16) CieTable {
    float v[RTB200_CIE_COUNT][4];
};
constexpr CieTable MakeCieTable()
{
    constexpr float x[] = {RTB200_CIE_XBAR}, y[] = {RTB200_CIE_YBAR}, z[] = {RTB200_CIE_ZBAR};
    CieTable t{};
    for (int i = 0; i < RTB200_CIE_COUNT; ++i) {
        t.v[i][0] = x[i];
        t.v[i][1] = y[i];
        t.v[i][2] = z[i];
    }
    return t;
}
__device__ const CieTable g_cie = MakeCieTable();

// ---- random numbers ---------------------------------------------------------
// Counter-based: every number is a hash of (seed, pixel, sample, dimension),
// so the oracle draws the identical sequence on the CPU.

__device__ __forceinline__ uint32_t Mix32(uint32_t x)
{
    x ^= x >> 16; x *= 0x7feb352du;
    x ^= x >> 15; x *= 0x846ca68bu;
    x ^= x >> 16;
    return x;
}

__device__ __forceinline__ uint32_t PathKey(uint32_t seed, uint32_t pixel, uint32_t sample)
{
    return Mix32(Mix32(seed ^ 0x9e3779b9u ^ Mix32(pixel)) ^ sample);
}

__device__ __forceinline__ float Rand(uint32_t key, uint32_t dim)
{
    return (float)(Mix32(key ^ (dim * 0x9e3779b9u + 0x7f4a7c15u)) >> 8) * (1.0f / 16777216.0f);
}

// Dimension layout: camera jitter 0-1, hero wavelength 2; bounce `depth`
// uses 8 + 32*depth + j: light sample i at j = 4i..4i+3 (light, x, y,
// triangle), BSDF direction j = 16, 17, lobe / Fresnel choice 18, Russian
// roulette 19, sky sample i at j = 20 + 2i, 21 + 2i.
__device__ __forceinline__ uint32_t Dim(int depth, int j) { return 8u + 32u * (uint32_t)depth + (uint32_t)j; }

// ---- the reference's sampler: Owen-scrambled padded Sobol ------------------
// SobolSequence (Sampling/SobolSequence.h:55-206): dimension d of sample i is
// Sobol dimension d & 1 of i (dimension 0 the bit-reversed index, dimension 1
// the XOR of the direction numbers v_0 = 2^31, v_{k+1} = v_k ^ (v_k >> 1) over
// the set bits of i), Owen-scrambled by the Laine-Karras hash seeded with
// HashCombine(seed, d) (Burley 2020, "Practical Hash-based Owen Scrambling").

// HashCombine: a ^= b + golden + (a << 6) + (a >> 2), then MurmurHash3's
// fmix32 finaliser.
__device__ __forceinline__ uint32_t HashCombine(uint32_t a, uint32_t b)
{
    a ^= b + 0x9e3779b9u + (a << 6) + (a >> 2);
    a ^= a >> 16; a *= 0x85ebca6bu;
    a ^= a >> 13; a *= 0xc2b2ae35u;
    a ^= a >> 16;
    return a;
}

// Sobol dimension 1 of i, bit-reversed.  Over GF(2) the direction numbers are
// the powers of (1 + x) applied to 1 (bit 31 - k holding x^k), so the XOR over
// the set bits of i is the polynomial i shifted by one, i(1 + x); splitting i
// into halves, (1 + x)^(2^k) = 1 + x^(2^k) adds the upper half to the lower, at
// every size.  Ten instructions where the sum over the bits of a shuffled
// index, which has all 32, took a loop of 32 steps.
__device__ __forceinline__ uint32_t SobolDim1Reversed(uint32_t i)
{
    i ^= i >> 16;
    i ^= (i >> 8) & 0x00ff00ffu;
    i ^= (i >> 4) & 0x0f0f0f0fu;
    i ^= (i >> 2) & 0x33333333u;
    i ^= (i >> 1) & 0x55555555u;
    return i;
}

// Owen scrambling by the Laine-Karras hash on the bit-reversed value v.
__device__ __forceinline__ uint32_t OwenScrambleReversed(uint32_t v, uint32_t s)
{
    v ^= v * 0x3d20adeau;
    v += s;
    v *= (s >> 16) | 1u;
    v ^= v * 0x05526c56u;
    v ^= v * 0x53a22864u;
    return __brev(v);
}

// shuffle: the sample index is first Owen-scrambled with a seed per
// dimension pair (2k, 2k + 1), Burley's decorrelation of padded dimensions
// ("Practical Hash-based Owen Scrambling", JCGT 9(4), 2020, section 4), so
// different pairs no longer replay one Sobol pair under another scramble;
// the reference pads without it.
__device__ __forceinline__ uint32_t SobolShuffle(uint32_t index, uint32_t pair, uint32_t seed)
{
    return OwenScrambleReversed(__brev(index), HashCombine(HashCombine(seed, 0x5bd1e995u), pair));
}

// Dimension `dim` of the (shuffled) index.
__device__ __forceinline__ float SobolValue(uint32_t index, uint32_t dim, uint32_t seed)
{
    const uint32_t v = OwenScrambleReversed((dim & 1u) ? SobolDim1Reversed(index) : index, HashCombine(seed, dim));
    return (float)(v >> 8) * (1.0f / 16777216.0f);   // the top 24 bits: < 1 in FP32
}

__device__ __forceinline__ float SobolSample(uint32_t index, uint32_t dim, uint32_t seed, bool shuffle)
{
    return SobolValue(shuffle ? SobolShuffle(index, dim >> 1, seed) : index, dim, seed);
}

// Sobol seed of a pixel: the reference's HashCombine(x, y); a nonzero job seed
// is mixed in so that renders with different seeds are independent.
__device__ __forceinline__ uint32_t SobolPixelSeed(uint32_t x, uint32_t y, uint32_t seed)
{
    const uint32_t s = HashCombine(x, y);
    return seed ? HashCombine(s, seed) : s;
}

// Random numbers of one path vertex.  Hash mode: Rand(key, Dim(depth, j))
// with the fixed layout above.  Sobol mode: the reference's
// StartStream(16 + depth) then dimensions in the order they are drawn
// (`cur`), so each call site names its hash-layout slot j and the Sobol
// dimension follows the draw order; skip(n) consumes dimensions that the
// reference draws but this vertex does not use.
struct VertexRng {
    uint32_t key;      // hash key, or the pixel's Sobol seed
    uint32_t index;    // sample index (Sobol)
    int depth;
    int mode;          // kSamplerHash / kSamplerSobol / kSamplerSobolShuffled
    uint32_t cur;
    // The last dimension pair drawn from (dimensions start at 512) and its
    // shuffled index: a pair's two numbers come one after the other.
    uint32_t pair, shuffled;
    __device__ __forceinline__ float next(int j)
    {
        if (mode == kSamplerHash) return Rand(key, Dim(depth, j));
        const uint32_t dim = (16u + (uint32_t)depth) * 32u + cur++;
        if (mode == kSamplerSobol) return SobolValue(index, dim, key);
        if ((dim >> 1) != pair) {
            pair = dim >> 1;
            shuffled = SobolShuffle(index, pair, key);
        }
        return SobolValue(shuffled, dim, key);
    }
    __device__ __forceinline__ void skip(int n) { cur += (uint32_t)n; }
};

// ---- spectra -----------------------------------------------------------------

// Spectrum table: one float4 header per spectrum id, then the samples.
// Header {0, 380, 780, offset}: 81 samples on the 5 nm grid, linear between
// them (InterpSPDIndices, src/Library/Utilities/Color/ColorUtils.cpp:270-300),
// 0 outside 380..780 nm.  Header {n, begin, end, offset}: a binned packet of
// n amplitudes over [begin, end], the bin holding nm returned as is, 0
// outside (SpectralPacket::ValueAtNM, Utilities/Color/SpectralPacket.h:285-297;
// nm == end reads the last bin).  Header {-1, 380, 780, offset}: an RGB
// colour's sigmoid polynomial (c0, c1, c2, scale), scale * s(c0 t^2 + c1 t +
// c2) with t = (nm - 380) / 400 (RGBSigmoidPolynomial::Eval,
// Utilities/Color/RGBSigmoidPolynomial.h:58-70).  Header {-2, 0, 1e30,
// offset}: a black body (temperature, scale): scale * C1 / l^5 /
// (exp(C2 / (l T)) - 1) with l = nm * 1e-9 m, C1 = 2 pi h c^2, C2 = h c / k
// (BlackBodyPainter::GetColorNM, Painters/BlackBodyPainter.cpp:26-43,103-106).
// offset is the samples' float index (bits).
__device__ __forceinline__ float Spec(const float* table, int id, float nm)
{
    if (id < 0) return 0.0f;
    const float4 h = __ldg(reinterpret_cast<const float4*>(table) + id);
    const float* s = table + __float_as_int(h.w);
    if (!(nm >= h.y) || nm > h.z) return 0.0f;
    if (h.x == -2.0f) {
        // C1 / l^5 with l in nm: 2 pi h c^2 * 1e45 / nm^5; C2 / (l T) = h c / k * 1e9 / (nm T).
        const float T = __ldg(s), k = __ldg(s + 1);
        const float n2 = nm * nm;
        const float first = 3.7417749e29f / (n2 * n2 * nm);
        return k * first / (expf(1.4387687e7f / (nm * T)) - 1.0f);
    }
    if (h.x < 0.0f) {
        const float4 c = make_float4(__ldg(s), __ldg(s + 1), __ldg(s + 2), __ldg(s + 3));
        const float t = (nm - 380.0f) / 400.0f;
        const float x = c.x * t * t + c.y * t + c.z;
        return c.w * (0.5f + x / (2.0f * sqrtf(1.0f + x * x)));
    }
    if (h.x == 0.0f) {
        const float x = (nm - 380.0f) * 0.2f;
        const int i = (int)floorf(x);
        const int j = i + 1 > 80 ? 80 : i + 1;
        const float w = x - (float)i;
        return __ldg(s + i) + w * (__ldg(s + j) - __ldg(s + i));
    }
    const int n = (int)h.x;
    const int i = min((int)((nm - h.y) * h.x / (h.z - h.y)), n - 1);
    return __ldg(s + i);
}

// ColorUtils::XYZFromNM (ColorUtils.cpp:313-325).
__device__ __forceinline__ bool Cmf(float nm, float& X, float& Y, float& Z)
{
    if (!(nm >= 380.0f) || nm > 780.0f) return false;
    const float x = (nm - 380.0f) * 0.2f;
    const int i = (int)floorf(x);
    const int j = i + 1 > 80 ? 80 : i + 1;
    const float w = x - (float)i;
    const float4 a = __ldg(reinterpret_cast<const float4*>(g_cie.v[i]));
    const float4 b = __ldg(reinterpret_cast<const float4*>(g_cie.v[j]));
    X = a.x + w * (b.x - a.x);
    Y = a.y + w * (b.y - a.y);
    Z = a.z + w * (b.z - a.z);
    return true;
}

// SampledWavelengths::SampleEquidistant
// (src/Library/Utilities/Color/SampledWavelengths.h:79-106).  The offset from
// lmin lies in [0, 1.75 range], where fmod by the range is at most one exact
// subtraction.
__device__ __forceinline__ void Wavelengths(float hero, float lmin, float lmax, float lam[4])
{
    const float range = lmax - lmin;
    const float delta = range * 0.25f;
    lam[0] = hero;
#pragma unroll
    for (int i = 1; i < 4; ++i) {
        const float x = hero - lmin + (float)i * delta;
        lam[i] = lmin + (x >= range ? x - range : x);
    }
}

__device__ __forceinline__ float Get(const float4& v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)); }
__device__ __forceinline__ void Set(float4& v, int i, float x)
{
    if (i == 0) v.x = x; else if (i == 1) v.y = x; else if (i == 2) v.z = x; else v.w = x;
}

// ---- small vector helpers ---------------------------------------------------

struct V3 { float x, y, z; };
__device__ __forceinline__ V3 mk(float x, float y, float z) { return {x, y, z}; }
__device__ __forceinline__ V3 operator+(V3 a, V3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ V3 operator-(V3 a, V3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V3 operator*(V3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ V3 operator-(V3 a) { return {-a.x, -a.y, -a.z}; }
__device__ __forceinline__ float dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 cross(V3 a, V3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
__device__ __forceinline__ V3 normalize(V3 a) { return a * rsqrtf(fmaxf(dot(a, a), 1e-30f)); }
__device__ __forceinline__ V3 xyz(float4 v) { return {v.x, v.y, v.z}; }

// Unit vector from its octahedral encoding (OctEncode in pt_types.h).
__device__ __forceinline__ V3 OctDecode(unsigned q)
{
    const float u = (float)(short)(q & 0xffffu) * (1.0f / 32767.0f);
    const float v = (float)(short)(q >> 16) * (1.0f / 32767.0f);
    float x = u, y = v;
    const float z = 1.0f - fabsf(u) - fabsf(v);
    if (z < 0.0f) {
        x = (1.0f - fabsf(v)) * (u >= 0.0f ? 1.0f : -1.0f);
        y = (1.0f - fabsf(u)) * (v >= 0.0f ? 1.0f : -1.0f);
    }
    return normalize(mk(x, y, z));
}

// Orthonormal basis around unit n (Duff et al., JCGT 6(1), 2017).
__device__ __forceinline__ void Basis(V3 n, V3& t, V3& b)
{
    const float sign = copysignf(1.0f, n.z);
    const float a = -1.0f / (sign + n.z);
    const float c = n.x * n.y * a;
    t = mk(1.0f + sign * n.x * n.x * a, sign * c, -sign * n.x);
    b = mk(c, sign + n.y * n.y * a, -n.y);
}

// Ray origin pushed off the surface on the side of `dir` by a few float ulps
// (Waechter and Binder, "A Fast and Robust Method for Avoiding
// Self-Intersection", Ray Tracing Gems, 2019).  The reference advances the
// origin by 1e-8 along the ray in double precision
// (PathTracingIntegrator.cpp:4812); in FP32 that step is below one ulp.
__device__ __forceinline__ V3 OffsetRay(V3 p, V3 ng, V3 dir)
{
    const V3 n = dot(dir, ng) >= 0.0f ? ng : -ng;
    const float kOrigin = 1.0f / 32.0f, kFloat = 1.0f / 65536.0f, kInt = 256.0f;
    const int ox = (int)(kInt * n.x), oy = (int)(kInt * n.y), oz = (int)(kInt * n.z);
    const V3 pi = mk(__int_as_float(__float_as_int(p.x) + (p.x < 0 ? -ox : ox)),
                     __int_as_float(__float_as_int(p.y) + (p.y < 0 ? -oy : oy)),
                     __int_as_float(__float_as_int(p.z) + (p.z < 0 ? -oz : oz)));
    return mk(fabsf(p.x) < kOrigin ? p.x + kFloat * n.x : pi.x,
              fabsf(p.y) < kOrigin ? p.y + kFloat * n.y : pi.y,
              fabsf(p.z) < kOrigin ? p.z + kFloat * n.z : pi.z);
}

// PathTransportUtilities::PowerHeuristic (Utilities/PathTransportUtilities.h:251).
__device__ __forceinline__ float PowerHeuristic(float a, float b)
{
    const float a2 = a * a;
    return a2 / (a2 + b * b);
}

// Adds four floats to a 16-byte aligned address, each atomically, in one operation
// (splats of a Gaussian film, light samples shared by the wavelengths: an adaptive
// 200 x 150 image 3.39 -> 3.30 ms).
__device__ __forceinline__ void AtomicAdd4(float* p, float x, float y, float z, float w)
{
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

// A path's pair in one access.
__device__ __forceinline__ void LoadPair(const PathPair* p, float4& a, float4& b)
{
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void StorePair(PathPair* p, const float4& a, const float4& b)
{
    asm volatile("st.global.v8.f32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};" ::"f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w),
                 "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w), "l"(p)
                 : "memory");
}
__device__ __forceinline__ uint4 Bits(const float4& v)
{
    return make_uint4(__float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w));
}
__device__ __forceinline__ float4 Floats(const uint4& v)
{
    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
// The path's job and its flags alone.
__device__ __forceinline__ int PathJob(const PtPaths& P, int slot) { return __float_as_int(P.state[slot].a.z); }
__device__ __forceinline__ void SetFlags(const PtPaths& P, int slot, unsigned flags)
{
    P.state[slot].b.z = __uint_as_float(flags);
}

// Appends to up to four queues at once, called by a whole warp: a lane adds
// n[q] entries to queue q and gets its first index in at[q].  The counts
// (below 1024 a warp, 256 with four queues) are summed in one packed scan and
// the counters advanced by one instruction, an atomic per queue and warp.
template <int N>
__device__ __forceinline__ void WarpAppend(int* const (&counter)[N], const int (&n)[N], int (&at)[N])
{
    static_assert(N <= 4, "packed counts");
    constexpr int kBits = N <= 3 ? 10 : 8;
    constexpr unsigned kMask = (1u << kBits) - 1u;
    const int lane = threadIdx.x & 31;
    unsigned mine = 0;
#pragma unroll
    for (int q = 0; q < N; ++q) mine |= (unsigned)n[q] << (kBits * q);
    unsigned incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    const unsigned total = __shfl_sync(0xffffffffu, incl, 31);
    int base = 0;
#pragma unroll
    for (int q = 0; q < N; ++q) {
        const int t = (int)((total >> (kBits * q)) & kMask);
        if (lane == q && t) base = atomicAdd(counter[q], t);
    }
    const unsigned excl = incl - mine;
#pragma unroll
    for (int q = 0; q < N; ++q) at[q] = __shfl_sync(0xffffffffu, base, q) + (int)((excl >> (kBits * q)) & kMask);
}

}  // namespace rtb200
