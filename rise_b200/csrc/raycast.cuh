// raycast.cuh -- device-side BVH traversal and triangle tests for sm_100a.
//
// Shared by the batch ray-cast kernels (raycast.cu) and the wavefront path
// tracer (pathtrace.cu).  The traversal replaces the reference's single-ray
// BVH4 walk (src/Library/Acceleration/BVH.h:1304-1471) over the same
// collapsed tree with a warp-cooperative "while-while" walk: lanes first
// descend internal nodes until every lane holds a postponed leaf, then test
// leaves together, and a lane whose ray is finished takes the next ray from a
// warp-local chunk of the batch.  The reference's double-precision
// Moller-Trumbore leaf test (src/Library/Intersection/RayTriangleIntersection.cpp:21-68)
// becomes the FP32 watertight test of Woop, Benthin and Wald (JCGT 2(1), 2013);
// the closest hit is re-measured in FP64 with the reference's formula, so the
// reported distance is the reference's distance rounded once to FP32.
#pragma once
#include <climits>
#include <cstdint>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "bvh_build.h"

namespace rtb200 {

constexpr unsigned kErrStackOverflow = 1u;
constexpr int kEmpty = INT_MIN;      // no node / no leaf
constexpr int kTraceBlock = 128;     // threads per block of the trace kernels
// Traversal stack per thread: the first kTraceStack entries in shared memory
// (kStackRows: 22 KB per block, 8 blocks of 128 threads stay resident per SM next
// to 64 registers).  Kernels instantiated with SPILL continue it in local memory for
// scenes whose TraceStackBound exceeds kTraceStack; the others carry no local
// array at all.
constexpr int kTraceStack = kTraceStackShared;
constexpr int kTraceSpill = kTraceStackMax - kTraceStackShared;
constexpr unsigned kFull = 0xffffffffu;

struct Ray {
    float o[3];
    float tmin;
    float d[3];
    float tmax;
};

struct RayPre {
    float o[3];
    float inv[3];
    float tmin;
    // Watertight shear: byte offsets of the triangle's coordinate rows (GpuTri)
    // along the permuted axes x, y and z (z the direction's largest component).
    int rx, ry, rz;
    float sx, sy, sz;
};

__device__ __forceinline__ float4 ldg4(const void* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ int4 ldg4i(const void* p) { return __ldg(reinterpret_cast<const int4*>(p)); }

// Two 16-byte vectors in one 32-byte load (p 32-byte aligned).  The lane walk
// over a large tree is bound by L1 (88 % of its throughput), and a node in half
// as many loads traces 4,194,304 incoherent rays in 3176 us instead of 3346
// (binary16), 3400 / 3499 (8-bit) and 4131 / 4398 (FP32 boxes).  Triangles stay
// 48 bytes and three loads: 64-byte ones in two loads cannot be read in the
// order of the ray's axes, and the selects cost 20 %.
__device__ __forceinline__ void ldg8(const void* p, int4& a, int4& b)
{
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
        : "l"(p));
}

__device__ __forceinline__ float Comp(const float* v, int k) { return k == 0 ? v[0] : (k == 1 ? v[1] : v[2]); }

__device__ __forceinline__ void Prepare(const Ray& r, RayPre& p)
{
    for (int k = 0; k < 3; ++k) {
        p.o[k] = r.o[k];
        // Zero components map to FLT_MAX like the reference (BVH.h:1221-1224).
        p.inv[k] = (r.d[k] == 0.0f) ? 3.402823466e+38f : __frcp_rn(r.d[k]);
    }
    p.tmin = r.tmin;
    const float ax = fabsf(r.d[0]), ay = fabsf(r.d[1]), az = fabsf(r.d[2]);
    int kz = (ax > ay) ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
    int kx = kz + 1; if (kx == 3) kx = 0;
    int ky = kx + 1; if (ky == 3) ky = 0;
    const float dz = Comp(r.d, kz);
    if (dz < 0.0f) { int t = kx; kx = ky; ky = t; }
    p.rx = 16 * kx; p.ry = 16 * ky; p.rz = 16 * kz;
    p.sx = Comp(r.d, kx) / dz;
    p.sy = Comp(r.d, ky) / dz;
    p.sz = dz == 0.0f ? 1.0f / dz : Comp(p.inv, kz);   // the reciprocal above, both correctly rounded
}

// A triangle's rows along the ray's permuted axes: x, y and z hold that
// coordinate of v0, v1 and v2, w the triangle's index and last-of-leaf flag.
struct TriRows {
    float4 x, y, z;
};

__device__ __forceinline__ TriRows LoadRows(const GpuTri* tris, int slot, const RayPre& p)
{
    const char* tb = reinterpret_cast<const char*>(tris + slot);
    return TriRows{ldg4(tb + p.rx), ldg4(tb + p.ry), ldg4(tb + p.rz)};
}

__device__ __forceinline__ int TriIndex(const GpuTri* tris, int slot)
{
    return __ldg(&tris[slot].x.w) & kTriIndexMask;
}

// The ray's origin along its permuted axes.
__device__ __forceinline__ void PermutedOrigin(const RayPre& p, float& ox, float& oy, float& oz)
{
    ox = p.rx == 0 ? p.o[0] : (p.rx == 16 ? p.o[1] : p.o[2]);
    oy = p.ry == 0 ? p.o[0] : (p.ry == 16 ? p.o[1] : p.o[2]);
    oz = p.rz == 0 ? p.o[0] : (p.rz == 16 ? p.o[1] : p.o[2]);
}

// A candidate hit: t = num / den (den > 0) and the quotient rounded, with the
// barycentrics (alpha, beta) of v1 and v2, the reference's (a, b) convention.
struct TriHit {
    float num, den;
    float t, a, b;
};

// A hit is nearer than tmax when its products say so: the rounded quotients of
// two triangles can be equal where these are not.
__device__ __forceinline__ bool Nearer(const TriHit& h, float tmax) { return !(h.num >= tmax * h.den); }

// Watertight ray/triangle test.  Returns true for a hit with tmin < t < tmax.
// (ox, oy, oz) is PermutedOrigin.
__device__ __forceinline__ bool Watertight(const RayPre& p, const TriRows& r, float ox, float oy, float oz, float tmax,
                                           TriHit& h)
{
    const float Az = r.z.x - oz, Bz = r.z.y - oz, Cz = r.z.z - oz;
    const float Ax = (r.x.x - ox) - p.sx * Az, Ay = (r.y.x - oy) - p.sy * Az;
    const float Bx = (r.x.y - ox) - p.sx * Bz, By = (r.y.y - oy) - p.sy * Bz;
    const float Cx = (r.x.z - ox) - p.sx * Cz, Cy = (r.y.z - oy) - p.sy * Cz;
    float U = Cx * By - Cy * Bx;
    float V = Ax * Cy - Ay * Cx;
    float W = Bx * Ay - By * Ax;
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        // Edge case: redo the 2D edge functions in FP64 (paper, section 3).
        U = (float)((double)Cx * (double)By - (double)Cy * (double)Bx);
        V = (float)((double)Ax * (double)Cy - (double)Ay * (double)Cx);
        W = (float)((double)Bx * (double)Ay - (double)By * (double)Ax);
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
    const float det = U + V + W;
    const float adet = fabsf(det);
    // det is the Moller-Trumbore determinant e1 . (d x e2) divided by the
    // dominant direction component, |det_MT| = adet / |sz|: the reference
    // rejects |det_MT| < 1e-12 (RayTriangleIntersection.cpp:40-42), which
    // also drops triangles with edges below ~1e-6.
    if (!(adet >= 1e-12f * fabsf(p.sz))) return false;
    const float T = U * (p.sz * Az) + V * (p.sz * Bz) + W * (p.sz * Cz);
    h.num = copysignf(1.0f, det) * T;
    h.den = adet;
    if (h.num <= p.tmin * h.den || !Nearer(h, tmax)) return false;
    const float rcp = 1.0f / det;
    h.t = T * rcp;
    h.a = V * rcp;
    h.b = W * rcp;
    return true;
}

// The reference's double-precision Moller-Trumbore distance for a triangle
// already known to be hit (RayTriangleIntersection.cpp:36-60).
__device__ __forceinline__ double RefineT(const float* o, const float* d, const float4& A4,
                                          const float4& B4, const float4& C4)
{
    const double ea[3] = {(double)B4.x - A4.x, (double)B4.y - A4.y, (double)B4.z - A4.z};
    const double eb[3] = {(double)C4.x - A4.x, (double)C4.y - A4.y, (double)C4.z - A4.z};
    const double dd[3] = {d[0], d[1], d[2]};
    const double pv[3] = {dd[1] * eb[2] - dd[2] * eb[1], dd[2] * eb[0] - dd[0] * eb[2], dd[0] * eb[1] - dd[1] * eb[0]};
    const double det = ea[0] * pv[0] + ea[1] * pv[1] + ea[2] * pv[2];
    const double tv[3] = {(double)o[0] - A4.x, (double)o[1] - A4.y, (double)o[2] - A4.z};
    const double qv[3] = {tv[1] * ea[2] - tv[2] * ea[1], tv[2] * ea[0] - tv[0] * ea[2], tv[0] * ea[1] - tv[1] * ea[0]};
    return (eb[0] * qv[0] + eb[1] * qv[1] + eb[2] * qv[2]) / det;
}

// The three vertices of a triangle (w unused).
__device__ __forceinline__ void LoadVertices(const GpuTri* tris, int slot, float4& A, float4& B, float4& C)
{
    const char* tb = reinterpret_cast<const char*>(tris + slot);
    const float4 x = ldg4(tb), y = ldg4(tb + 16), z = ldg4(tb + 32);
    A = make_float4(x.x, y.x, z.x, 0.0f);
    B = make_float4(x.y, y.y, z.y, 0.0f);
    C = make_float4(x.z, y.z, z.z, 0.0f);
}

// ---- node decoders --------------------------------------------------------

// A node's children: c[i] the link of child i (kEmpty when EXACT and missed),
// key[i] its entry distance as float bits.  EXACT (closest hit): all the bits, and
// those of +inf for a miss.  Otherwise (any hit, whose answer no order changes):
// bits with the child's number in the two low ones, so that keys order as
// integers from -0 up and are all distinct, and kMiss for a miss.
constexpr int kMiss = INT_MAX;
constexpr int kInfBits = 0x7f800000;
struct ChildHits {
    int key[4];
    int c[4];
};

// Three-input minimum / maximum (one instruction on sm_100a).
__device__ __forceinline__ float Max3(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float Min3(float a, float b, float c)
{
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// The key of child i, entered at tn if it is hit (ChildHits).
template <bool EXACT>
__device__ __forceinline__ int HitKey(float tn, bool hit, int i, int& link)
{
    if (EXACT) {
        link = hit ? link : kEmpty;
        return hit ? __float_as_int(tn) : kInfBits;
    }
    return hit ? ((__float_as_int(tn) & ~3) | i) : kMiss;
}

// Entry and exit distance of one child from the six plane offsets (plane
// minus origin): the reference slab arithmetic (BVH.h:738-763).  The
// reference takes min / max of the two plane distances per axis; with a
// finite reciprocal (zero components map to FLT_MAX) the near plane is the
// low one for a positive reciprocal and the high one otherwise, so picking
// the planes by the ray's direction signs gives bit-identical distances
// without the per-axis min / max.
//
// The walk is bound by instruction issue (75 % of the issue slots, 14 of 32
// lanes active), so the work of a visit is counted in instructions: products
// run two to an instruction.  With the mixed subtraction and the triangle rows
// (GpuTri), and the loads and the stack below: 4,194,304 incoherent closest-hit
// rays on a 1M-triangle soup 3810 -> 2991 us over binary16 boxes, 3909 -> 3139
// over 8-bit and 4527 -> 4140 over FP32 ones, which are bound by L1 instead.
template <bool EXACT>
__device__ __forceinline__ int SlabKey(float nx, float ny, float nz, float fx, float fy, float fz, const RayPre& p,
                                       float best, int i, bool present, int& link)
{
    const float2 ixy = make_float2(p.inv[0], p.inv[1]), izz = make_float2(p.inv[2], p.inv[2]);
    const float2 n = __fmul2_rn(make_float2(nx, ny), ixy), f = __fmul2_rn(make_float2(fx, fy), ixy);
    const float2 z = __fmul2_rn(make_float2(nz, fz), izz);
    const float tn = Max3(n.x, n.y, fmaxf(z.x, p.tmin));
    const float tf = Min3(f.x, f.y, fminf(z.y, best));
    return HitKey<EXACT>(tn, tn <= tf && present, i, link);
}

// FP32 node: the low and high planes of an axis come in one load.
template <bool EXACT>
__device__ __forceinline__ void SlabF32(const GpuNode4* nodes, int ni, const RayPre& p, float best, ChildHits& h)
{
    const float* base = reinterpret_cast<const float*>(nodes + ni);
    int4 lx, hx, ly, hy, lz, hz;
    ldg8(base, lx, hx);
    ldg8(base + 8, ly, hy);
    ldg8(base + 16, lz, hz);
    const int4 child = ldg4i(base + 24);   // empty slots hold kEmpty; counts are not read
    const bool gx = p.inv[0] < 0.0f, gy = p.inv[1] < 0.0f, gz = p.inv[2] < 0.0f;
    const float lxa[4] = {__int_as_float(lx.x), __int_as_float(lx.y), __int_as_float(lx.z), __int_as_float(lx.w)};
    const float hxa[4] = {__int_as_float(hx.x), __int_as_float(hx.y), __int_as_float(hx.z), __int_as_float(hx.w)};
    const float lya[4] = {__int_as_float(ly.x), __int_as_float(ly.y), __int_as_float(ly.z), __int_as_float(ly.w)};
    const float hya[4] = {__int_as_float(hy.x), __int_as_float(hy.y), __int_as_float(hy.z), __int_as_float(hy.w)};
    const float lza[4] = {__int_as_float(lz.x), __int_as_float(lz.y), __int_as_float(lz.z), __int_as_float(lz.w)};
    const float hza[4] = {__int_as_float(hz.x), __int_as_float(hz.y), __int_as_float(hz.z), __int_as_float(hz.w)};
    h.c[0] = child.x; h.c[1] = child.y; h.c[2] = child.z; h.c[3] = child.w;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        h.key[i] = SlabKey<EXACT>((gx ? hxa[i] : lxa[i]) - p.o[0], (gy ? hya[i] : lya[i]) - p.o[1],
                                  (gz ? hza[i] : lza[i]) - p.o[2], (gx ? lxa[i] : hxa[i]) - p.o[0],
                                  (gy ? lya[i] : hya[i]) - p.o[1], (gz ? lza[i] : hza[i]) - p.o[2], p, best, i,
                                  h.c[i] != kEmpty, h.c[i]);
}

// An 8-bit integer of a packed word as a float, exactly, without the
// half-rate integer conversion: the byte under the exponent of 2^23, less 2^23.
__device__ __forceinline__ float ByteMagic(unsigned w, int i)
{
    return __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7650u | (unsigned)i));
}

// Quantised node: child slabs from 8-bit bounds, t = q * (2^e / d) + (origin - o) / d.
template <bool EXACT>
__device__ __forceinline__ void SlabQ8(const QNode4* nodes, int ni, const RayPre& p, float best, ChildHits& h)
{
    const int4* base = reinterpret_cast<const int4*>(nodes + ni);
    int4 w0, w1, w2, w3;
    ldg8(base, w0, w1);
    ldg8(base + 2, w2, w3);
    const float org[3] = {__int_as_float(w0.x), __int_as_float(w0.y), __int_as_float(w0.z)};
    const unsigned meta = (unsigned)w0.w;
    const int e[3] = {(int)(int8_t)(meta & 0xff), (int)(int8_t)((meta >> 8) & 0xff), (int)(int8_t)((meta >> 16) & 0xff)};
    // Near / far quantised planes per axis by the direction's sign (see SlabKey).
    const unsigned qlo[3] = {(unsigned)w1.x, (unsigned)w1.y, (unsigned)w1.z};
    const unsigned qhi[3] = {(unsigned)w1.w, (unsigned)w2.x, (unsigned)w2.y};
    unsigned qn[3], qf[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const bool neg = p.inv[k] < 0.0f;
        qn[k] = neg ? qhi[k] : qlo[k];
        qf[k] = neg ? qlo[k] : qhi[k];
    }
    h.c[0] = w2.z; h.c[1] = w2.w; h.c[2] = w3.x; h.c[3] = w3.y;
    const int cnt[4] = {(int)(int16_t)(w3.z & 0xffff), (int)(int16_t)((unsigned)w3.z >> 16),
                        (int)(int16_t)(w3.w & 0xffff), (int)(int16_t)((unsigned)w3.w >> 16)};
    float a[3], s[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        a[k] = (org[k] - p.o[k]) * p.inv[k];
        s[k] = __int_as_float((e[k] + 127) << 23) * p.inv[k];
    }
    const float2 axy = make_float2(a[0], a[1]), azz = make_float2(a[2], a[2]);
    const float2 sxy = make_float2(s[0], s[1]), szz = make_float2(s[2], s[2]);
    const float2 bias = make_float2(-8388608.0f, -8388608.0f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 n = __ffma2_rn(__fadd2_rn(make_float2(ByteMagic(qn[0], i), ByteMagic(qn[1], i)), bias), sxy, axy);
        const float2 f = __ffma2_rn(__fadd2_rn(make_float2(ByteMagic(qf[0], i), ByteMagic(qf[1], i)), bias), sxy, axy);
        const float2 z = __ffma2_rn(__fadd2_rn(make_float2(ByteMagic(qn[2], i), ByteMagic(qf[2], i)), bias), szz, azz);
        const float tn = Max3(n.x, n.y, fmaxf(z.x, p.tmin));
        const float tf = Min3(f.x, f.y, fminf(z.y, best));
        h.key[i] = HitKey<EXACT>(tn, tn <= tf && cnt[i] >= 0, i, h.c[i]);
    }
}

// One half of a word minus an FP32 value: the conversion is exact and the
// mixed-precision subtraction rounds once, so it equals convert-then-subtract
// in one instruction (3405 -> 3334 us on the 4,194,304-ray batch below).
__device__ __forceinline__ float HalfMinus(unsigned w, int hi, float o)
{
    float d;
    asm("sub.rn.f32.f16 %0, %1, %2;" : "=f"(d) : "h"((unsigned short)(hi ? w >> 16 : w)), "f"(o));
    return d;
}

// Half-precision node: the FP32 slab test on child boxes widened to binary16
// (outward), planes picked by the direction's sign as in SlabKey.
template <bool EXACT>
__device__ __forceinline__ void SlabF16(const HNode4* nodes, int ni, const RayPre& p, float best, ChildHits& h)
{
    const int4* base = reinterpret_cast<const int4*>(nodes + ni);
    int4 w0, w1, w2, w3;
    ldg8(base, w0, w1);
    ldg8(base + 2, w2, w3);
    // Words (two halves each): lo x, y, z then hi x, y, z, children 0-1 and 2-3.
    const unsigned lo[3][2] = {{(unsigned)w0.x, (unsigned)w0.y}, {(unsigned)w0.z, (unsigned)w0.w},
                               {(unsigned)w1.x, (unsigned)w1.y}};
    const unsigned hi[3][2] = {{(unsigned)w1.z, (unsigned)w1.w}, {(unsigned)w2.x, (unsigned)w2.y},
                               {(unsigned)w2.z, (unsigned)w2.w}};
    unsigned n[3][2], f[3][2];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const bool neg = p.inv[k] < 0.0f;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            n[k][j] = neg ? hi[k][j] : lo[k][j];
            f[k][j] = neg ? lo[k][j] : hi[k][j];
        }
    }
    h.c[0] = w3.x; h.c[1] = w3.y; h.c[2] = w3.z; h.c[3] = w3.w;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        h.key[i] = SlabKey<EXACT>(HalfMinus(n[0][i >> 1], i & 1, p.o[0]), HalfMinus(n[1][i >> 1], i & 1, p.o[1]),
                                  HalfMinus(n[2][i >> 1], i & 1, p.o[2]), HalfMinus(f[0][i >> 1], i & 1, p.o[0]),
                                  HalfMinus(f[1][i >> 1], i & 1, p.o[1]), HalfMinus(f[2][i >> 1], i & 1, p.o[2]), p,
                                  best, i, h.c[i] != kEmpty, h.c[i]);
}

// Child c of a node alone: its key and, in `link`, its link.  The same
// arithmetic as the whole node's, for walks that give a child to each lane.
template <bool EXACT>
__device__ __forceinline__ int ChildF32(const GpuNode4* nodes, int ni, int c, const RayPre& p, float best, int& link)
{
    // Float offsets of lox, hix, loy, hiy, loz, hiz: 0, 4, 8, 12, 16, 20.
    const float* base = reinterpret_cast<const float*>(nodes + ni) + c;
    const int nx = p.inv[0] < 0.0f ? 4 : 0, ny = p.inv[1] < 0.0f ? 12 : 8, nz = p.inv[2] < 0.0f ? 20 : 16;
    link = __float_as_int(__ldg(base + 24));
    return SlabKey<EXACT>(__ldg(base + nx) - p.o[0], __ldg(base + ny) - p.o[1], __ldg(base + nz) - p.o[2],
                          __ldg(base + (4 - nx)) - p.o[0], __ldg(base + (20 - ny)) - p.o[1],
                          __ldg(base + (36 - nz)) - p.o[2], p, best, c, link != kEmpty, link);
}
template <bool EXACT>
__device__ __forceinline__ int ChildF16(const HNode4* nodes, int ni, int c, const RayPre& p, float best, int& link)
{
    const unsigned short* base = reinterpret_cast<const unsigned short*>(nodes + ni) + c;
    const int nx = p.inv[0] < 0.0f ? 12 : 0, ny = p.inv[1] < 0.0f ? 16 : 4, nz = p.inv[2] < 0.0f ? 20 : 8;
    link = __ldg(&nodes[ni].child[c]);
    return SlabKey<EXACT>(HalfMinus(__ldg(base + nx), 0, p.o[0]), HalfMinus(__ldg(base + ny), 0, p.o[1]),
                          HalfMinus(__ldg(base + nz), 0, p.o[2]), HalfMinus(__ldg(base + (12 - nx)), 0, p.o[0]),
                          HalfMinus(__ldg(base + (20 - ny)), 0, p.o[1]), HalfMinus(__ldg(base + (28 - nz)), 0, p.o[2]),
                          p, best, c, link != kEmpty, link);
}
template <bool EXACT>
__device__ __forceinline__ int ChildQ8(const QNode4* nodes, int ni, int c, const RayPre& p, float best, int& link)
{
    const QNode4* n = nodes + ni;
    const int4 w0 = ldg4i(n);
    const float org[3] = {__int_as_float(w0.x), __int_as_float(w0.y), __int_as_float(w0.z)};
    float tl[3], th[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int e = (int)(int8_t)((unsigned)w0.w >> (8 * k));
        const float q0 = (float)__ldg(&n->qlo[k][c]), q1 = (float)__ldg(&n->qhi[k][c]);
        const float a = (org[k] - p.o[k]) * p.inv[k], sc = __int_as_float((e + 127) << 23) * p.inv[k];
        const bool neg = p.inv[k] < 0.0f;
        tl[k] = fmaf(neg ? q1 : q0, sc, a);
        th[k] = fmaf(neg ? q0 : q1, sc, a);
    }
    link = __ldg(&n->child[c]);
    const float tn = Max3(tl[0], tl[1], fmaxf(tl[2], p.tmin));
    const float tf = Min3(th[0], th[1], fminf(th[2], best));
    return HitKey<EXACT>(tn, tn <= tf && __ldg(&n->count[c]) >= 0, c, link);
}

template <class NodeT>
struct Slab;
template <>
struct Slab<GpuNode4> {
    template <bool EXACT>
    __device__ __forceinline__ static void Run(const GpuNode4* n, int i, const RayPre& p, float b, ChildHits& h)
    {
        SlabF32<EXACT>(n, i, p, b, h);
    }
    template <bool EXACT>
    __device__ __forceinline__ static int One(const GpuNode4* n, int i, int c, const RayPre& p, float b, int& link)
    {
        return ChildF32<EXACT>(n, i, c, p, b, link);
    }
};
template <>
struct Slab<QNode4> {
    template <bool EXACT>
    __device__ __forceinline__ static void Run(const QNode4* n, int i, const RayPre& p, float b, ChildHits& h)
    {
        SlabQ8<EXACT>(n, i, p, b, h);
    }
    template <bool EXACT>
    __device__ __forceinline__ static int One(const QNode4* n, int i, int c, const RayPre& p, float b, int& link)
    {
        return ChildQ8<EXACT>(n, i, c, p, b, link);
    }
};
template <>
struct Slab<HNode4> {
    template <bool EXACT>
    __device__ __forceinline__ static void Run(const HNode4* n, int i, const RayPre& p, float b, ChildHits& h)
    {
        SlabF16<EXACT>(n, i, p, b, h);
    }
    template <bool EXACT>
    __device__ __forceinline__ static int One(const HNode4* n, int i, int c, const RayPre& p, float b, int& link)
    {
        return ChildF16<EXACT>(n, i, c, p, b, link);
    }
};

__device__ __forceinline__ void CSwap(int& a, int& b)
{
    const int lo = min(a, b);
    b = max(a, b);
    a = lo;
}

// The link of the child a key names.
__device__ __forceinline__ int Child(const ChildHits& h, int key)
{
    const int lo = (key & 1) ? h.c[1] : h.c[0], hi = (key & 1) ? h.c[3] : h.c[2];
    return (key & 2) ? hi : lo;
}

// After the call (ta, ca) holds the nearer entry; equal ones stay.
__device__ __forceinline__ void CSwap(float& ta, int& ca, float& tb, int& cb)
{
    const bool sw = tb < ta;
    const float t = sw ? tb : ta;
    const int c = sw ? cb : ca;
    tb = sw ? ta : tb;
    cb = sw ? ca : cb;
    ta = t;
    ca = c;
}

// The children nearest first: with EXACT their links (kEmpty after the last hit
// one), else their keys (kMiss).  The closest-hit walk keeps the first of
// several triangles at one distance, so its order is part of its answer: by the
// whole entry distances, with children at equal ones (coincident meshes have
// the same boxes) in the order in which this network leaves them.  Keys that
// gave two bits to the child's number turned 65,252 of 287,982 hits on three
// coincident meshes to another of the three, and were no faster: decoding the
// links took what the shorter sort gave (4,194,304 rays as above: binary16 3122
// and 2991 us, 8-bit 3247 and 3139, FP32 4137 and 4140).  Any hit needs no such
// order, and its keys sort in ten min / max.
template <bool EXACT>
__device__ __forceinline__ void Order(const ChildHits& h, int& k0, int& k1, int& k2, int& k3)
{
    if (EXACT) {
        float t0 = __int_as_float(h.key[0]), t1 = __int_as_float(h.key[1]);
        float t2 = __int_as_float(h.key[2]), t3 = __int_as_float(h.key[3]);
        k0 = h.c[0]; k1 = h.c[1]; k2 = h.c[2]; k3 = h.c[3];
        CSwap(t0, k0, t1, k1);
        CSwap(t2, k2, t3, k3);
        CSwap(t0, k0, t2, k2);
        CSwap(t1, k1, t3, k3);
        CSwap(t1, k1, t2, k2);
        return;
    }
    k0 = h.key[0]; k1 = h.key[1]; k2 = h.key[2]; k3 = h.key[3];
    CSwap(k0, k1);
    CSwap(k2, k3);
    CSwap(k0, k2);
    CSwap(k1, k3);
    CSwap(k1, k2);
}

// Per-lane traversal state of one ray.
struct TraceState {
    RayPre p;
    float best;        // current tmax
    int bestSlot;      // leaf-order triangle slot of the closest hit
    float ba, bb;      // its barycentrics
    int node;          // next internal node, a leaf entry (~first), or kEmpty
    int leaf;          // postponed leaf entry (~first) or kEmpty
    unsigned sp;       // shared-memory address of the next free stack entry
    int over;          // entries in local memory (SPILL kernels)
};

// Bytes between the entries of a thread's stack in shared memory.
constexpr unsigned kStackStep = 4u * kTraceBlock;

__device__ __forceinline__ void StartRay(TraceState& s, const Ray& r, unsigned bottom)
{
    Prepare(r, s.p);
    s.best = r.tmax;
    s.bestSlot = -1;
    s.ba = s.bb = 0.0f;
    s.node = 0;
    s.leaf = kEmpty;
    s.sp = bottom;
    s.over = 0;
}

// The stack: a thread's column of the shared-memory part, [row][thread], held
// as 32-bit shared addresses.  Row 0 holds kEmpty for good, so popping an empty
// stack needs no test; `bottom` is row 1.  `spill` is the thread's
// local-memory continuation.  Against indexing with a test per access:
// 4,194,304 incoherent rays 3172 -> 3085 us closest and 1626 -> 1545 any hit over
// binary16, 3394 -> 3240 and 1694 -> 1609 over 8-bit boxes; FP32 boxes, bound by
// L1, unchanged.
struct TraceStack {
    unsigned bottom;
    int* spill;
};
constexpr int kStackRows = kTraceStack + 4;   // and three beyond the bound
static_assert(8 * (kStackRows * kTraceBlock * 4 + 1024) <= 228 * 1024, "8 blocks per SM");

__device__ __forceinline__ void StoreShared(unsigned at, int v)
{
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(at), "r"(v) : "memory");
}
__device__ __forceinline__ int LoadShared(unsigned at)
{
    int v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
    return v;
}

__device__ __forceinline__ TraceStack MakeStack(int* column, int* spill)
{
    *column = kEmpty;
    return TraceStack{(unsigned)__cvta_generic_to_shared(column) + kStackStep, spill};
}

// Push of the SPILL kernels.  Overflow (a bound computed wrongly) drops the
// entry and raises the error flag, which the host turns into an error status.
__device__ __forceinline__ void Push(TraceState& s, const TraceStack& st, int v, unsigned* err)
{
    if (s.sp < st.bottom + kTraceStack * kStackStep) {
        StoreShared(s.sp, v);
        s.sp += kStackStep;
    } else if (s.over < kTraceSpill) {
        st.spill[s.over++] = v;
    } else {
        atomicOr(err, kErrStackOverflow);
    }
}

template <bool SPILL>
__device__ __forceinline__ int Pop(TraceState& s, const TraceStack& st)
{
    if (SPILL && s.over > 0) return st.spill[--s.over];
    s.sp -= kStackStep;
    return LoadShared(s.sp);
}

// One round of while-while traversal for every active lane: descend internal
// nodes until fewer than LACK active lanes still lack a postponed
// leaf (or have run out of nodes), then test at most LEAVES leaves per lane
// as one flat walk over their triangles; a leaf met after that is kept for the
// next round, whose descent starts with it.  Measured on incoherent rays
// (4-wide nodes, where sibling leaves are common): with uncapped leaf chains
// and a descent that waited for every lane, 25 % of the lanes were active in
// the leaf loop and 42 % in the descent; the cap, the flat walk and the early
// stop together trace 70 % more rays per second.  ANY: stop at the first
// accepted hit.  Returns true when this lane's ray is finished.
template <class NodeT, bool ANY, bool SPILL, int LEAVES, int LACK>
__device__ __forceinline__ bool TraceRound(TraceState& s, const NodeT* __restrict__ nodes,
                                           const GpuTri* __restrict__ tris, int ntri, const TraceStack& stk, unsigned* err)
{
    // Descend internal nodes, first postponing a leaf left from the last round.
    for (;;) {
        if (s.node < 0 && s.node != kEmpty && s.leaf == kEmpty) {
            s.leaf = s.node;
            s.node = Pop<SPILL>(s, stk);
        }
        if (s.node < 0) break;
        ChildHits h;
        Slab<NodeT>::template Run<!ANY>(nodes, s.node, s.p, s.best, h);
        // The nearest hit child becomes the next node; the others are pushed
        // far to near (pushing them unsorted saved instructions and cost 11 %
        // in visits).
        constexpr int kNone = ANY ? kMiss : kEmpty;
        const auto link = [&](int k) { return ANY ? Child(h, k) : k; };
        int k0, k1, k2, k3;
        Order<!ANY>(h, k0, k1, k2, k3);
        if (!SPILL) {
            // One test for all three: the rows go on past the bound.
            if (s.sp > stk.bottom + kTraceStack * kStackStep) {
                atomicOr(err, kErrStackOverflow);
                k1 = k2 = k3 = kNone;
            }
            if (k3 != kNone) {
                StoreShared(s.sp, link(k3));
                s.sp += kStackStep;
            }
            if (k2 != kNone) {
                StoreShared(s.sp, link(k2));
                s.sp += kStackStep;
            }
            if (k1 != kNone) {
                StoreShared(s.sp, link(k1));
                s.sp += kStackStep;
            }
        } else {
            if (k3 != kNone) Push(s, stk, link(k3), err);
            if (k2 != kNone) Push(s, stk, link(k2), err);
            if (k1 != kNone) Push(s, stk, link(k1), err);
        }
        s.node = (k0 != kNone) ? link(k0) : Pop<SPILL>(s, stk);
        // Postpone the first leaf met; keep descending until most lanes have one.
        if (s.node < 0 && s.node != kEmpty && s.leaf == kEmpty) {
            s.leaf = s.node;
            s.node = Pop<SPILL>(s, stk);
        }
        if (__popc(__ballot_sync(__activemask(), s.leaf == kEmpty)) < LACK) break;
    }
    // Test leaves: one walk over the triangles of up to LEAVES leaves.
    int nleaf = 0;
    int slot = s.leaf != kEmpty ? ~s.leaf : -1;
    float ox, oy, oz;
    PermutedOrigin(s.p, ox, oy, oz);
    while (slot >= 0) {
        const TriRows r = LoadRows(tris, slot, s.p);
        TriHit hit;
        if (Watertight(s.p, r, ox, oy, oz, s.best, hit)) {
            if (ANY) {
                s.bestSlot = slot;
                s.node = kEmpty;
                s.leaf = kEmpty;
                return true;
            }
            s.best = hit.t;
            s.bestSlot = slot;
            s.ba = hit.a;
            s.bb = hit.b;
        }
        // The last triangle of a leaf is flagged; the array bound is a second
        // stop so a leaf walk never leaves the buffer.
        if (__float_as_int(r.x.w) < 0 || slot + 1 >= ntri) {
            s.leaf = kEmpty;
            slot = -1;
            if (++nleaf < LEAVES && s.node < 0 && s.node != kEmpty) {
                s.leaf = s.node;
                s.node = Pop<SPILL>(s, stk);
                slot = ~s.leaf;
            }
        } else {
            ++slot;
        }
    }
    return s.node == kEmpty && s.leaf == kEmpty;
}

// ---- the last rays of a warp, one at a time by all its lanes ----------------
//
// A warp whose supply has run dry and that holds few rays takes them in turn:
// its lanes form eight groups of four, each group pops one entry of the ray's
// stack, tests a node's four children (a child per lane) or four triangles of
// a leaf, and the hit children go back on the stack, nearest on top within a
// node.  One step does the work of up to eight dependent steps of the lane
// walk, so a small batch, and the end of a large one, waits for memory a few
// times instead of once per node and triangle (1,000 rays on a 100k-triangle
// soup: 103 -> 21 us).
//
// A closest hit is the lane walk's, triangle for triangle: which walk ends a ray
// depends on its neighbours and on timing, and must not show where triangles lie
// at one distance.  The joint walk tests leaves as they come to hand, so where
// another triangle is about as far as the nearest (kCloseUnits) it says so and leaves
// the ray to its lane, whose walk goes on from where it was, bounded by the
// distance found (LaneRest).  Taking any of several equal hits gave another triangle
// to 1,266 of 600,000 rays on a soup whose triangles lie there twice, to 535 of
// them from run to run.  Walking every ray jointly but in the lane walk's order took
// 20,000 rays on a 300k-triangle soup 105 us; this takes 85 and any of them took 91.
// Where all triangles lie twelve times, 20,000 rays take 269 us (any: 100, in the
// lane walk alone 1,140).
//
// Everything lives in the warp's part of the stack memory: with D the deepest
// lane stack, rows D + 1 .. D + m keep the state of the m rays, a row each,
// and the rows above are the shared stack.

// Rays left in a warp when its lanes join forces.  100,003 rays on a
// 300k-triangle soup: 245 us without and 157 with 8 rays (3, 5 and 8 rays compared
// with integer child keys and any of equal hits: 200, 181 and 167 us).
constexpr int kCoopRays = 8;

// Triangles about as far as each other: their rounded distances are at most this
// many units in the last place apart.  A distance T / det is rounded twice and the
// lane walk compares products rounded once, so beyond three units (a unit is at
// least 2^-24 of the distance) the nearer one wins in any order.  kCloseHits is as
// much as a share or more.
constexpr int kCloseUnits = 4;
constexpr float kCloseHits = 1.0f / 1048576.0f;   // 2^-20
// Share of a distance by which a box may be entered behind a triangle in it.  Both
// are rounded: the box's entry to a few units in 2^24, the triangle's distance by
// its barycentrics' error (2^-24 d^2 / s^2, at most 1, at distance d and size s)
// times its extent s, at most 2^-12 d and a small factor.  Boxes are culled with
// this much to spare, so that no triangle about as far as the best goes unseen.
constexpr float kBoxSlack = 1.0f / 128.0f;

// Words of a ray's state row.
enum CoopWord : int {
    kCoO = 0, kCoInv = 3, kCoTmin = 6, kCoRows = 7, kCoS = 8, kCoBest = 11, kCoSlot = 12, kCoA = 13, kCoB = 14,
    kCoNode = 15, kCoLeaf = 16, kCoSp = 17, kCoLane = 18, kCoNodes = 19, kCoTris = 21, kCoNtri = 23,
    kCoClose = 24, kCoAnswer = 25   // best, slot, a, b found
};

// Orders floats as integers.
__device__ __forceinline__ int OrderedBits(float t)
{
    const int i = __float_as_int(t);
    return i ^ ((i >> 31) & 0x7fffffff);
}

// Whether a warp whose lanes with `live` set still hold a ray should finish
// them together: few rays, and room above the lane stacks for their state
// rows, the shared stack's seeds and a first full step.
template <bool SPILL>
__device__ __forceinline__ bool CoopReady(const TraceState& s, const TraceStack& stk, unsigned live)
{
    constexpr int kBound = SPILL ? kTraceStackMax : kTraceStack;
    const int m = __popc(live);
    int depth = 0;
    if ((live >> (threadIdx.x & 31u)) & 1u)
        depth = SPILL && s.over > 0 ? kTraceStack : (int)((s.sp - stk.bottom) / kStackStep);
    const int D = __reduce_max_sync(kFull, depth);
    return (kTraceStack - D - m) * 32 >= D + 2 + 24 + kBound;
}

// Walks the m rays whose state rows start at row D + 1.
template <class NodeT, bool ANY, bool SPILL>
__device__ __forceinline__ void CoopWalk(int* rows, int D, int m, unsigned* err)
{
    constexpr int kBound = SPILL ? kTraceStackMax : kTraceStack;   // TraceStackBound of the scene is at most this
    const unsigned lane = threadIdx.x & 31u;
    const int cap = (kTraceStack - D - m) * 32;
    const auto word = [&](int row, int col) -> int& { return rows[row * kTraceBlock + col]; };
    const int first = D + 1 + m;   // row of the shared stack's entry 0
    const auto entry = [&](int i) -> int& { return rows[(first + (i >> 5)) * kTraceBlock + (i & 31)]; };
    const unsigned group = lane >> 2, c = lane & 3u;
    for (int k = 0; k < m; ++k) {
        const int row = D + 1 + k;
        RayPre p;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            p.o[j] = __int_as_float(word(row, kCoO + j));
            p.inv[j] = __int_as_float(word(row, kCoInv + j));
        }
        p.tmin = __int_as_float(word(row, kCoTmin));
        const int rr = word(row, kCoRows);
        p.rx = rr & 0xff; p.ry = (rr >> 8) & 0xff; p.rz = rr >> 16;
        p.sx = __int_as_float(word(row, kCoS));
        p.sy = __int_as_float(word(row, kCoS + 1));
        p.sz = __int_as_float(word(row, kCoS + 2));
        float best = __int_as_float(word(row, kCoBest));
        const NodeT* nd = reinterpret_cast<const NodeT*>(((unsigned long long)(unsigned)word(row, kCoNodes + 1) << 32) |
                                                         (unsigned)word(row, kCoNodes));
        const GpuTri* tr = reinterpret_cast<const GpuTri*>(((unsigned long long)(unsigned)word(row, kCoTris + 1) << 32) |
                                                           (unsigned)word(row, kCoTris));
        const int nt = word(row, kCoNtri);
        const int owner = word(row, kCoLane), sp0 = word(row, kCoSp);
        const int node0 = word(row, kCoNode), leaf0 = word(row, kCoLeaf);
        float ox, oy, oz;
        PermutedOrigin(p, ox, oy, oz);
        // Seeds: the lane's stack (bottom first), its next node, its postponed leaf.
        for (int i = (int)lane; i < sp0; i += 32) entry(i) = word(i + 1, owner);
        int sp = sp0;
        if (node0 != kEmpty) {
            if (lane == 0) entry(sp) = node0;
            ++sp;
        }
        if (leaf0 != kEmpty) {
            if (lane == 0) entry(sp) = leaf0;
            ++sp;
        }
        __syncwarp();
        while (sp > 0) {
            // Eight entries at once while that leaves a depth-first walk of one
            // entry's subtree (at most kBound more) room above them.
            const int take = max(1, min(min(8, sp), (cap - kBound - sp) / 3));
            // Group `take - 1` holds the top entry, so its children end up on top.
            const int e = (int)group < take ? entry(sp - take + (int)group) : kEmpty;
            sp -= take;
            __syncwarp();
            int key = kMiss, link = kEmpty;
            if (e >= 0)
                key = Slab<NodeT>::template One<false>(nd, e, (int)c, p, ANY ? best : best + kBoxSlack * fabsf(best), link);
            int at = (e < 0 && e != kEmpty) ? ~e + (int)c : -1;
            bool found = false;
            while (__any_sync(kFull, at >= 0)) {
                bool last = false, hit = false;
                TriHit h{0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
                if (at >= 0) {
                    const TriRows r = LoadRows(tr, min(at, nt - 1), p);
                    last = __float_as_int(r.x.w) < 0 || at >= nt - 1;
                    hit = Watertight(p, r, ox, oy, oz, ANY ? best : best + kCloseHits * fabsf(best), h);
                }
                // Lanes past the leaf's last triangle looked at another leaf's.
                const unsigned lasts = (__ballot_sync(kFull, last) >> (group * 4u)) & 0xfu;
                hit = hit && !(lasts & ((1u << c) - 1u));
                const unsigned cand = __ballot_sync(kFull, hit);
                if (cand) {
                    const int ord = hit ? OrderedBits(h.t) : INT_MAX;
                    const int lo = __reduce_min_sync(kFull, ord);
                    const unsigned near = __ballot_sync(kFull, ord <= lo + kCloseUnits);
                    const int from = __ffs(__ballot_sync(kFull, ord == lo)) - 1;
                    if (lane == 0) word(row, kCoClose) = (near & (near - 1u)) || OrderedBits(best) <= lo + kCloseUnits;
                    if (ANY || lo < OrderedBits(best)) {
                        best = __shfl_sync(kFull, h.t, from);
                        const int slot = __shfl_sync(kFull, at, from);
                        const float ba = __shfl_sync(kFull, h.a, from), bb = __shfl_sync(kFull, h.b, from);
                        if (lane == 0) {
                            word(row, kCoAnswer) = __float_as_int(best);
                            word(row, kCoAnswer + 1) = slot;
                            word(row, kCoAnswer + 2) = __float_as_int(ba);
                            word(row, kCoAnswer + 3) = __float_as_int(bb);
                        }
                    }
                    found = true;
                    if (ANY) break;
                }
                at = at >= 0 && !lasts ? at + 4 : -1;
            }
            if (ANY && found) break;
            // Push the hit children: a lower group's below a higher group's,
            // within a group the farther ones first.
            const unsigned hits = __ballot_sync(kFull, key != kMiss);
            int rank = 0;
#pragma unroll
            for (int x = 1; x < 4; ++x) {
                const int other = __shfl_xor_sync(kFull, key, x);
                rank += other != kMiss && other > key;
            }
            const int pos = sp + __popc(hits & ((1u << (group * 4u)) - 1u)) + rank;
            if (key != kMiss) {
                if (pos < cap) entry(pos) = link;
                else atomicOr(err, kErrStackOverflow);
            }
            sp = min(sp + __popc(hits), cap);
            __syncwarp();
        }
        __syncwarp();
    }
}

// Ends the rays of the lanes with `live` set, whose state is s and for which
// CoopReady holds; every lane of the warp calls it.  `rows` is the warp's column 0
// of the stack memory.  Returns whether the lane's ray is done: then s.best,
// s.bestSlot, s.ba and s.bb hold its answer and the rest of s is undefined.  A ray
// with several triangles about as far as the nearest is left to the lane walk, with
// its state as it was but for a nearer bound.  OWN: lanes trace different scenes.
template <class NodeT, bool ANY, bool SPILL, bool OWN, class NodePtr, class TriPtr>
__device__ __forceinline__ bool CoopFinish(TraceState& s, const TraceStack& stk, bool live, NodePtr& nodes,
                                           TriPtr& tris, int& ntri, int* rows, unsigned* err)
{
    const unsigned lane = threadIdx.x & 31u;
    const unsigned mask = __ballot_sync(kFull, live);
    const int m = __popc(mask);
    const int depth = live ? (int)((s.sp - stk.bottom) / kStackStep) : 0;
    const int D = __reduce_max_sync(kFull, depth);
    const auto word = [&](int row, int col) -> int& { return rows[row * kTraceBlock + col]; };
    const int mine = D + 1 + __popc(mask & ((1u << lane) - 1u));   // this lane's state row
    if (live) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            word(mine, kCoO + k) = __float_as_int(s.p.o[k]);
            word(mine, kCoInv + k) = __float_as_int(s.p.inv[k]);
        }
        word(mine, kCoTmin) = __float_as_int(s.p.tmin);
        word(mine, kCoRows) = s.p.rx | (s.p.ry << 8) | (s.p.rz << 16);
        word(mine, kCoS) = __float_as_int(s.p.sx);
        word(mine, kCoS + 1) = __float_as_int(s.p.sy);
        word(mine, kCoS + 2) = __float_as_int(s.p.sz);
        word(mine, kCoBest) = __float_as_int(s.best);
        word(mine, kCoSlot) = s.bestSlot;
        word(mine, kCoA) = __float_as_int(s.ba);
        word(mine, kCoB) = __float_as_int(s.bb);
        word(mine, kCoNode) = s.node;
        word(mine, kCoLeaf) = s.leaf;
        word(mine, kCoSp) = depth;
        word(mine, kCoLane) = (int)lane;
        word(mine, kCoNodes) = (int)(unsigned)(unsigned long long)nodes;
        word(mine, kCoNodes + 1) = (int)((unsigned long long)nodes >> 32);
        word(mine, kCoTris) = (int)(unsigned)(unsigned long long)tris;
        word(mine, kCoTris + 1) = (int)((unsigned long long)tris >> 32);
        word(mine, kCoNtri) = ntri;
        word(mine, kCoClose) = 0;
        word(mine, kCoAnswer) = __float_as_int(s.best);
        word(mine, kCoAnswer + 1) = s.bestSlot;
        word(mine, kCoAnswer + 2) = __float_as_int(s.ba);
        word(mine, kCoAnswer + 3) = __float_as_int(s.bb);
    }
    __syncwarp();
    CoopWalk<NodeT, ANY, SPILL>(rows, D, m, err);
    const float best = __int_as_float(word(mine, kCoAnswer));
    if (!ANY) {
        // The lane's state again, from its row and for every lane, so that it takes
        // no registers meanwhile; lanes without a ray read what they never use.
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            s.p.o[k] = __int_as_float(word(mine, kCoO + k));
            s.p.inv[k] = __int_as_float(word(mine, kCoInv + k));
        }
        s.p.tmin = __int_as_float(word(mine, kCoTmin));
        const int rr = word(mine, kCoRows);
        s.p.rx = rr & 0xff; s.p.ry = (rr >> 8) & 0xff; s.p.rz = rr >> 16;
        s.p.sx = __int_as_float(word(mine, kCoS));
        s.p.sy = __int_as_float(word(mine, kCoS + 1));
        s.p.sz = __int_as_float(word(mine, kCoS + 2));
        s.node = word(mine, kCoNode);
        s.leaf = word(mine, kCoLeaf);
        s.sp = stk.bottom + (unsigned)word(mine, kCoSp) * kStackStep;
        s.over = 0;
        if (OWN) {
            nodes = reinterpret_cast<const NodeT*>(((unsigned long long)(unsigned)word(mine, kCoNodes + 1) << 32) |
                                                   (unsigned)word(mine, kCoNodes));
            tris = reinterpret_cast<const GpuTri*>(((unsigned long long)(unsigned)word(mine, kCoTris + 1) << 32) |
                                                   (unsigned)word(mine, kCoTris));
            ntri = word(mine, kCoNtri);
        }
    }
    const bool again = !ANY && word(mine, kCoClose);
    s.best = again ? fminf(__int_as_float(word(mine, kCoBest)), best + kBoxSlack * fabsf(best)) : best;
    s.bestSlot = word(mine, again ? kCoSlot : kCoAnswer + 1);
    s.ba = __int_as_float(word(mine, again ? kCoA : kCoAnswer + 2));
    s.bb = __int_as_float(word(mine, again ? kCoB : kCoAnswer + 3));
    // Every lane has read its row before a walk that goes on overwrites it.
    __syncwarp();
    return live && !again;
}

// Ends the closest-hit walk of a ray that CoopFinish left, by its lane alone: the
// lane walk without its rounds and votes, which so few rays do not need (its
// code a second time in the kernels slowed their main loop: 100,003 rays 171 us
// instead of 157).
template <class NodeT, bool SPILL>
__device__ __forceinline__ void LaneRest(TraceState& s, const NodeT* __restrict__ nodes, const GpuTri* __restrict__ tris,
                                         int ntri, const TraceStack& stk, unsigned* err)
{
    const auto push = [&](int v) {
        if (SPILL) {
            Push(s, stk, v, err);
        } else if (s.sp < stk.bottom + kTraceStack * kStackStep) {
            StoreShared(s.sp, v);
            s.sp += kStackStep;
        } else {
            atomicOr(err, kErrStackOverflow);
        }
    };
    float ox, oy, oz;
    PermutedOrigin(s.p, ox, oy, oz);
    int cur = s.node;
    if (s.leaf != kEmpty) {
        if (cur != kEmpty) push(cur);
        cur = s.leaf;
    }
    if (cur == kEmpty) cur = Pop<SPILL>(s, stk);
    while (cur != kEmpty) {
        if (cur >= 0) {
            ChildHits h;
            Slab<NodeT>::template Run<true>(nodes, cur, s.p, s.best, h);
            int k0, k1, k2, k3;
            Order<true>(h, k0, k1, k2, k3);
            if (k3 != kEmpty) push(k3);
            if (k2 != kEmpty) push(k2);
            if (k1 != kEmpty) push(k1);
            cur = k0 != kEmpty ? k0 : Pop<SPILL>(s, stk);
            continue;
        }
        for (int slot = ~cur;; ++slot) {
            const TriRows r = LoadRows(tris, slot, s.p);
            TriHit hit;
            if (Watertight(s.p, r, ox, oy, oz, s.best, hit)) {
                s.best = hit.t;
                s.bestSlot = slot;
                s.ba = hit.a;
                s.bb = hit.b;
            }
            if (__float_as_int(r.x.w) < 0 || slot + 1 >= ntri) break;
        }
        cur = Pop<SPILL>(s, stk);
    }
}

// ---- eight-wide compressed nodes (WNode8, bvh_wide.cpp) -------------------
// Per-lane traversal after Ylitie, Karras and Laine (HPG 2017): a node group
// (first internal child's index; hit children in bits 24-31 in visiting
// order, the node's internal-child mask in bits 0-7) and a triangle group
// (first triangle; hit triangles in bits 0-23).  A node's hit children are
// visited in slot order s ^ oct, oct the ray's non-negative direction signs,
// which the build made roughly near to far; groups wait on a stack of one
// entry per tree level, bounded at commit.

constexpr int kW8Stack = kW8StackEntries;   // uint2 entries per thread in shared memory
constexpr int kW8Levels = kW8MaxLevels;      // node groups the stack keeps room for

struct W8State {
    RayPre p;
    float d[3];
    float best;
    int bestSlot;
    float ba, bb;
    unsigned oct;
    uint2 ng;          // node group
    int sp;
    int visits;        // iterations spent on this ray (bounded)
};

// A ray takes at most this many iterations (each visits one node or tests
// one triangle group; a tree of n triangles has fewer than n nodes), else its
// traversal stops with the error flag raised.
constexpr int kW8MaxIterations = 1 << 22;

__device__ __forceinline__ void StartRayW8(W8State& s, const Ray& r)
{
    Prepare(r, s.p);
    s.d[0] = r.d[0]; s.d[1] = r.d[1]; s.d[2] = r.d[2];
    s.best = r.tmax;
    s.bestSlot = -1;
    s.ba = s.bb = 0.0f;
    s.oct = (r.d[0] >= 0.0f ? 1u : 0u) | (r.d[1] >= 0.0f ? 2u : 0u) | (r.d[2] >= 0.0f ? 4u : 0u);
    // The root as the one internal child (slot 0) of a virtual parent at 0.
    s.ng = make_uint2(0u, (1u << (24 + s.oct)) | 1u);
    s.sp = 0;
    s.visits = 0;
}

// Child slabs of one node: the node group of its hit internal children and
// the triangle group of its hit leaf slots.
__device__ __forceinline__ void IntersectW8(const WNode8* __restrict__ nodes, unsigned ni, const RayPre& p,
                                            unsigned oct, float best, uint2& ng, uint2& tg)
{
    const uint4* base = reinterpret_cast<const uint4*>(nodes + ni);
    const uint4 w0 = __ldg(base), w1 = __ldg(base + 1), w2 = __ldg(base + 2), w3 = __ldg(base + 3),
                w4 = __ldg(base + 4);
    const float org[3] = {__uint_as_float(w0.x), __uint_as_float(w0.y), __uint_as_float(w0.z)};
    const unsigned em = w0.w;
    const int e[3] = {(int)(int8_t)(em & 0xffu), (int)(int8_t)((em >> 8) & 0xffu), (int)(int8_t)((em >> 16) & 0xffu)};
    const unsigned imask = em >> 24;
    // Bounds per axis as two words of four bytes (slots 0-3, 4-7); near and
    // far planes by the direction's sign (see SlabKey).
    const unsigned lo[3][2] = {{w2.x, w2.y}, {w2.z, w2.w}, {w3.x, w3.y}};
    const unsigned hi[3][2] = {{w3.z, w3.w}, {w4.x, w4.y}, {w4.z, w4.w}};
    unsigned qn[3][2], qf[3][2];
    float a[3], sc[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const bool neg = p.inv[k] < 0.0f;
        qn[k][0] = neg ? hi[k][0] : lo[k][0];
        qn[k][1] = neg ? hi[k][1] : lo[k][1];
        qf[k][0] = neg ? lo[k][0] : hi[k][0];
        qf[k][1] = neg ? lo[k][1] : hi[k][1];
        a[k] = (org[k] - p.o[k]) * p.inv[k];
        sc[k] = __int_as_float((e[k] + 127) << 23) * p.inv[k];
    }
    unsigned hitsN = 0u, hitsT = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int h = i >> 2, sh = 8 * (i & 3);
        float tl[3], th[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            tl[k] = fmaf((float)((qn[k][h] >> sh) & 0xffu), sc[k], a[k]);
            th[k] = fmaf((float)((qf[k][h] >> sh) & 0xffu), sc[k], a[k]);
        }
        const float tn = Max3(tl[0], tl[1], fmaxf(tl[2], p.tmin));
        const float tf = Min3(th[0], th[1], fminf(th[2], best));
        if (tn <= tf) {
            if ((imask >> i) & 1u) {
                hitsN |= 1u << (24 + (i ^ oct));
            } else {
                const unsigned meta = ((i < 4 ? w1.z : w1.w) >> sh) & 0xffu;
                hitsT |= (meta >> 5) << (meta & 31u);
            }
        }
    }
    ng = make_uint2(w1.x, hitsN | imask);
    tg = make_uint2(w1.y, hitsT);
}

// Lanes below which a warp postpones its triangle tests (pushes the
// triangle group and keeps descending), after Ylitie et al.
constexpr int kW8TriLanes = 8;

// Traverses for at most `budget` iterations; returns true when the ray is
// finished.  The current group `ng` is a node group (hits in bits 24-31) or,
// popped from the stack, a postponed triangle group (bits 0-23 only).  A
// triangle group is postponed while fewer than kW8TriLanes lanes of the warp
// have triangles to test and the stack keeps room for one node group per
// level (kW8Levels).  ANY: stop at the first accepted hit.
template <bool ANY>
__device__ __forceinline__ bool TraceW8(W8State& s, const WNode8* __restrict__ nodes,
                                        const GpuTri* __restrict__ tris, uint2* stk, unsigned* err, int budget)
{
    for (int it = 0; it < budget; ++it) {
        if (++s.visits > kW8MaxIterations) {
            atomicOr(err, kErrStackOverflow);
            return true;
        }
        uint2 tg = make_uint2(0u, 0u);
        if (s.ng.y & 0xff000000u) {
            const unsigned j = (unsigned)__ffs(s.ng.y >> 24) - 1u;
            s.ng.y &= ~(1u << (24 + j));
            const unsigned slot = j ^ s.oct;
            const unsigned ni = s.ng.x + (unsigned)__popc(s.ng.y & 0xffu & ((1u << slot) - 1u));
            if (s.ng.y & 0xff000000u) {
                if (s.sp < kW8Stack) { stk[s.sp * kTraceBlock] = s.ng; ++s.sp; }
                else atomicOr(err, kErrStackOverflow);
            }
            IntersectW8(nodes, ni, s.p, s.oct, s.best, s.ng, tg);
        } else {
            tg = s.ng;   // a postponed triangle group (or nothing)
            s.ng = make_uint2(0u, 0u);
        }
        float ox, oy, oz;
        PermutedOrigin(s.p, ox, oy, oz);
        while (tg.y) {
            // Postpone only with a node group to continue with, so a popped
            // triangle group is always tested (the ray keeps progressing).
            if ((s.ng.y & 0xff000000u) && s.sp < kW8Stack - kW8Levels &&
                __popc(__ballot_sync(__activemask(), true)) < kW8TriLanes) {
                stk[s.sp * kTraceBlock] = tg;
                ++s.sp;
                break;
            }
            const unsigned k = (unsigned)__ffs(tg.y) - 1u;
            tg.y &= tg.y - 1u;
            const unsigned slot = tg.x + k;
            const TriRows r = LoadRows(tris, (int)slot, s.p);
            TriHit hit;
            if (Watertight(s.p, r, ox, oy, oz, s.best, hit)) {
                s.bestSlot = (int)slot;
                if (ANY) return true;
                s.best = hit.t;
                s.ba = hit.a;
                s.bb = hit.b;
            }
        }
        if (!(s.ng.y & 0xff000000u)) {
            if (s.sp == 0) return true;
            --s.sp;
            s.ng = stk[s.sp * kTraceBlock];
        }
    }
    return false;
}

// Warp-cooperative ray supply: warp w of W starts with the w-th run of
// `chunk` rays, and a lane whose ray is finished takes the next index of its
// warp's run; past the first W runs a warp takes further runs from the global
// counter (one atomic per run), which counts rays past the first W runs.
struct WarpFeed {
    unsigned next, end, base;
    bool exhausted;
};

// Rays of one launch at most, so that ray numbers and counters fit 32 bits.
constexpr long long kFeedRays = 1ll << 30;

// Rays per run.  Up to 32 rays per resident warp every warp takes an equal
// share, so a small batch spreads over the whole chip instead of filling a
// few warps (100,003 rays on a 300k-triangle soup took 478 us as 782 warps of
// 128 rays and take 256 as 4,736 of 22; 1,000 rays 424 and 109 us).  Beyond
// that a run is an eighth of a warp's share, at least 32 and at most 128 rays,
// so that the last runs end close together without giving up the order of
// coherent rays (786,432 camera rays: 211 us; 272 with a half, 233 with a
// quarter of a share; 228 with runs of 16).
__host__ __device__ inline unsigned FeedChunk(unsigned n, unsigned warps)
{
    if (n <= 32 * warps) return (n + warps - 1) / warps;
    const unsigned c = n / (8 * warps);
    return c < 32 ? 32 : (c > 128 ? 128 : c);
}

__device__ __forceinline__ WarpFeed FeedStart(unsigned n, unsigned chunk)
{
    const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = (gridDim.x * blockDim.x) >> 5;
    WarpFeed f;
    f.base = warps * chunk;
    f.next = min(warp * chunk, n);
    f.end = min(f.next + chunk, n);
    f.exhausted = f.base >= n;
    return f;
}

// No ray is left to hand out.
__device__ __forceinline__ bool FeedDry(const WarpFeed& f) { return f.exhausted && f.next >= f.end; }

// Returns this lane's new ray index or -1.  `want` lanes ask for work.
__device__ __forceinline__ int FeedTake(WarpFeed& f, bool want, unsigned n, unsigned chunk, unsigned* counter)
{
    const unsigned lane = threadIdx.x & 31u;
    const unsigned wm = __ballot_sync(kFull, want);
    if (!wm) return -1;
    const unsigned need = __popc(wm);
    const unsigned rank = __popc(wm & ((1u << lane) - 1u));
    const unsigned avail = f.end - f.next;
    int mine = -1;
    if (rank < avail) mine = (int)(f.next + rank);
    if (avail < need && !f.exhausted) {
        unsigned base = 0;
        if (lane == 0) base = f.base + atomicAdd(counter, chunk);
        base = __shfl_sync(kFull, base, 0);
        if (base >= n) {
            f.exhausted = true;
            f.next = f.end;
        } else {
            const unsigned end = min(base + chunk, n);
            const unsigned extra = need - avail;
            if (rank >= avail && base + (rank - avail) < end) mine = (int)(base + (rank - avail));
            f.next = min(base + extra, end);
            f.end = end;
            if (end == n) f.exhausted = true;
        }
    } else {
        f.next += min(avail, need);
    }
    return want ? mine : -1;
}

}  // namespace rtb200
