// raycast_common.cuh - device side of the GigaVoxels ray walk, shared by the
// forward ray cast, the checkpointing forward and the adjoint replay.
//
// Floating point: every translation unit that includes this header is
// compiled with -fmad=false -prec-div=true -prec-sqrt=true and without
// fast-math, so each +,-,*,/ and sqrt below is one IEEE binary32 operation in
// the written order.  Fused operations are written as such: the linear
// interpolations of the filter (fma2 in lerp4 and lerp_x, as the oracle's
// lerp is fused); the corrections of fixed_div and markstein_div
// (fixed_div.h), whose quotients equal the IEEE division; and the bounds of
// brick_empty, which only pick samples that are zero.  The host oracle performs
// the same sequence, which makes descent decisions, step counts, LOD choices and
// node-usage lists bit-identical.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "cellmask.cuh"
#include "dxt.h"
#include "fixed_div.h"
#include "kernels.cuh"
#include "lod_bound.h"

namespace vv {
namespace rc {

constexpr uint32_t kResident = 0x80000000u;
constexpr uint32_t kConstant = 0x40000000u;

struct F3 {
    float x, y, z;
};
__device__ __forceinline__ F3 f3(float x, float y, float z) { return F3{x, y, z}; }
__device__ __forceinline__ F3 ld3(const float* a) { return F3{a[0], a[1], a[2]}; }
__device__ __forceinline__ F3 add(F3 a, F3 b) { return F3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ F3 sub(F3 a, F3 b) { return F3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ F3 mul(F3 a, F3 b) { return F3{a.x * b.x, a.y * b.y, a.z * b.z}; }
__device__ __forceinline__ F3 muls(F3 a, float s) { return F3{a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ F3 divv(F3 a, F3 b) { return F3{a.x / b.x, a.y / b.y, a.z / b.z}; }
__device__ __forceinline__ float dot3(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
// normalize(v) = v * (1 / sqrt(dot(v,v))), correctly rounded sqrt and divide.
__device__ __forceinline__ F3 normalize3(F3 v) {
    float r = 1.0f / sqrtf(dot3(v, v));
    return muls(v, r);
}

__device__ __forceinline__ void set_status(int* status, int code) {
    if (status) atomicCAS(status, 0, code);
}

// 2^e for e in [-126, 127], exactly: the normal power of two built from its
// exponent bits (ldexpf covers every case and costs more instructions).  Every
// use below scales by a tree level, well inside that range.
__device__ __forceinline__ float pow2i(int e) { return __int_as_float((e + 127) << 23); }

// pow(x, 2^k) as k squarings (the sample-ratio powers of the shader).
__device__ __forceinline__ float pow_pow2(float x, int k) {
    for (int i = 0; i < k; ++i) x = x * x;
    return x;
}

// Texel loads per storage format: 4 channels as float (RGBA8 as 0..255).
template <int FMT>
struct Texel;
// Byte k of v as a float, exactly: the bit pattern 0x4B0000bb is 2^23 + b.
// (A byte-select and an add instead of an integer-to-float conversion, which
// runs at a quarter of the add rate.)  Selectors: result bytes (low to high) =
// byte k of v, 0, 0, 0x4B.
__device__ __forceinline__ float byte_as_float(uint32_t v, uint32_t sel) {
    return __uint_as_float(__byte_perm(v, 0x4B000000u, sel)) - 8388608.0f;
}
template <>
struct Texel<VV_FMT_RGBA8> {
    static constexpr float kScale = 1.0f / 255.0f;
};
template <>
struct Texel<VV_FMT_FP16> {
    static constexpr float kScale = 1.0f;
    __device__ __forceinline__ static float4 load(const void* pool, uint32_t i) {
        uint2 v = __ldg((const uint2*)pool + i);
        __half2 a = *reinterpret_cast<__half2*>(&v.x), b = *reinterpret_cast<__half2*>(&v.y);
        float2 fa = __half22float2(a), fb = __half22float2(b);
        return make_float4(fa.x, fa.y, fb.x, fb.y);
    }
};
template <>
struct Texel<VV_FMT_BF16> {
    static constexpr float kScale = 1.0f;
    __device__ __forceinline__ static float4 load(const void* pool, uint32_t i) {
        uint2 v = __ldg((const uint2*)pool + i);
        return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xFFFF0000u),
                           __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xFFFF0000u));
    }
};
template <>
struct Texel<VV_FMT_FP32> {
    static constexpr float kScale = 1.0f;
    __device__ __forceinline__ static float4 load(const void* pool, uint32_t i) {
        return __ldg((const float4*)pool + i);
    }
};

// Block-compressed pools (dxt.h): texel i = slot * 1000 + (z*10 + y)*10 + x
// decoded from its 4x4 block of slice z, as RGBA8 values.
__device__ __forceinline__ void dxt_address(uint32_t i, uint32_t& block, int& t) {
    const uint32_t slot = i / 1000u, r = i - slot * 1000u;
    const uint32_t z = r / 100u, yx = r - z * 100u, y = yx / 10u, x = yx - y * 10u;
    block = slot * (uint32_t)dxt::kBlocksPerSlot + (uint32_t)dxt::block_of((int)x, (int)y, (int)z);
    t = dxt::texel_of((int)x, (int)y);
}
template <>
struct Texel<VV_FMT_DXT5> {
    static constexpr float kScale = 1.0f / 255.0f;
};
template <>
struct Texel<VV_FMT_DXT1> {
    static constexpr float kScale = 1.0f / 255.0f;
    __device__ __forceinline__ static float4 load(const void* pool, uint32_t i) {
        uint32_t b;
        int t;
        dxt_address(i, b, t);
        const uint2 v = __ldg((const uint2*)pool + b);
        const uint32_t w[2] = {v.x, v.y};
        const uint32_t c = dxt::decode_dxt1(w, t);
        return make_float4(byte_as_float(c, 0x7440u), byte_as_float(c, 0x7441u), byte_as_float(c, 0x7442u), 0.0f);
    }
};

// Two binary32 operations per instruction (sm_100a packed f32x2), each lane
// rounded as the scalar operation rounds: the same values in half the issue
// slots, which is what bounds the walk.
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// A texel as two channel pairs.
struct Pair4 {
    unsigned long long xy, zw;
};
__device__ __forceinline__ Pair4 pair4(float4 v) { return Pair4{pack2(v.x, v.y), pack2(v.z, v.w)}; }
// fmaf(t, b - a, a) of every channel, tt = (t, t)
__device__ __forceinline__ Pair4 lerp4(Pair4 a, Pair4 b, unsigned long long tt) {
    return Pair4{fma2(tt, sub2(b.xy, a.xy), a.xy), fma2(tt, sub2(b.zw, a.zw), a.zw)};
}

// The trilinear filter of eight texels (x fastest) with weights f, and the
// format's scale.  RGBA8 texels come as 2^23 + byte: the x lerp's difference
// of two of them is the bytes' difference exactly, so only its addend loses
// the bias.
template <int FMT>
struct RawTexel {
    using T = float4;
    __device__ __forceinline__ static T load(const void* pool, uint32_t i) { return Texel<FMT>::load(pool, i); }
    __device__ __forceinline__ static Pair4 lerp_x(T a, T b, unsigned long long tt) {
        return lerp4(pair4(a), pair4(b), tt);
    }
};
template <>
struct RawTexel<VV_FMT_RGBA8> {
    using T = uint32_t;
    __device__ __forceinline__ static T load(const void* pool, uint32_t i) { return __ldg((const uint32_t*)pool + i); }
    __device__ __forceinline__ static Pair4 biased(uint32_t v) {
        return Pair4{pack2(__uint_as_float(__byte_perm(v, 0x4B000000u, 0x7440u)),
                           __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7441u))),
                     pack2(__uint_as_float(__byte_perm(v, 0x4B000000u, 0x7442u)),
                           __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7443u)))};
    }
    __device__ __forceinline__ static Pair4 lerp_x(T a, T b, unsigned long long tt) {
        const unsigned long long bias = pack2(-8388608.0f, -8388608.0f);
        const Pair4 pa = biased(a), pb = biased(b);
        return Pair4{fma2(tt, sub2(pb.xy, pa.xy), add2(pa.xy, bias)), fma2(tt, sub2(pb.zw, pa.zw), add2(pa.zw, bias))};
    }
};
// DXT5 texels are decoded to RGBA8 words and filtered as those.
template <>
struct RawTexel<VV_FMT_DXT5> : RawTexel<VV_FMT_RGBA8> {
    __device__ __forceinline__ static T decode(const void* pool, uint32_t block, int t) {
        const uint4 v = __ldg((const uint4*)pool + block);
        return dxt::texel_dxt5(v.x, v.y, v.z, v.w, t);
    }
    __device__ __forceinline__ static T load(const void* pool, uint32_t i) {
        uint32_t b;
        int t;
        dxt_address(i, b, t);
        return decode(pool, b, t);
    }
};
template <int FMT>
__device__ __forceinline__ float4 filter8(const typename RawTexel<FMT>::T v[8], float fx, float fy, float fz) {
    using R = RawTexel<FMT>;
    const unsigned long long tx = pack2(fx, fx), ty = pack2(fy, fy), tz = pack2(fz, fz);
    const Pair4 c0 = lerp4(R::lerp_x(v[0], v[1], tx), R::lerp_x(v[2], v[3], tx), ty);
    const Pair4 c1 = lerp4(R::lerp_x(v[4], v[5], tx), R::lerp_x(v[6], v[7], tx), ty);
    Pair4 c = lerp4(c0, c1, tz);
    if (Texel<FMT>::kScale != 1.0f) {
        const unsigned long long k = pack2(Texel<FMT>::kScale, Texel<FMT>::kScale);
        c = Pair4{mul2(c.xy, k), mul2(c.zw, k)};
    }
    const float2 a = unpack2(c.xy), b = unpack2(c.zw);
    return make_float4(a.x, a.y, b.x, b.y);
}
// dst + T * src per channel (a product and a sum; the packed forms of the two
// were seen to give the fused result, so they stay scalar)
__device__ __forceinline__ float4 composite(float T, float4 src, float4 dst) {
    return make_float4(T * src.x + dst.x, T * src.y + dst.y, T * src.z + dst.z, T * src.w + dst.w);
}

// One axis of GL_LINEAR + CLAMP_TO_EDGE (GL 3.3 spec 3.8.8): texel centres at
// i+0.5, i0 = floor(u*N - 0.5), weight = frac.  Returns brick-linear
// coordinates (slot, local) of both taps.
struct Axis {
    int s0, l0, s1, l1;
    float f;
};
__device__ __forceinline__ Axis axis_taps(float u, float N, int n) {
    float t = u * N - 0.5f;
    t = fminf(fmaxf(t, -1.0f), N);
    float fi = floorf(t);
    Axis a;
    a.f = t - fi;
    int i0 = (int)fi, i1 = i0 + 1;
    i0 = min(max(i0, 0), n - 1);
    i1 = min(max(i1, 0), n - 1);
    a.s0 = i0 / 10;
    a.l0 = i0 - 10 * a.s0;
    a.s1 = i1 / 10;
    a.l1 = i1 - 10 * a.s1;
    return a;
}

__device__ __forceinline__ void touch(uint32_t* bits, uint32_t i) { atomicOr(bits + (i >> 5), 1u << (i & 31u)); }

// The trilinear fetch of the brick-pool texture at uvw, any taps.  Out of
// line: the walk comes here only for samples whose taps leave their slot.
template <int FMT, bool COUNT>
__device__ __noinline__ float4 sample_brick(const RaycastParams& p, F3 uvw) {
    const float* N = p.u.brick_pool_dimension;
    const int nx = p.slots[0] * 10, ny = p.slots[1] * 10, nz = p.slots[2] * 10;
    Axis ax = axis_taps(uvw.x, N[0], nx);
    Axis ay = axis_taps(uvw.y, N[1], ny);
    Axis az = axis_taps(uvw.z, N[2], nz);
    const uint32_t SX = (uint32_t)p.slots[0], SY = (uint32_t)p.slots[1];
    typename RawTexel<FMT>::T v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const uint32_t sx = (uint32_t)((k & 1) ? ax.s1 : ax.s0), sy = (uint32_t)((k & 2) ? ay.s1 : ay.s0),
                       sz = (uint32_t)((k & 4) ? az.s1 : az.s0);
        const int lx = (k & 1) ? ax.l1 : ax.l0, ly = (k & 2) ? ay.l1 : ay.l0, lz = (k & 4) ? az.l1 : az.l0;
        const uint32_t slot = (sz * SY + sy) * SX + sx;
        v[k] = RawTexel<FMT>::load(p.bricks, slot * 1000u + (uint32_t)((lz * 10 + ly) * 10 + lx));
        if (COUNT) touch(p.brick_touch, slot);
    }
    return filter8<FMT>(v, ax.f, ay.f, az.f);
}

// The brick-pool slot a brick segment samples: its first texel per axis, its
// first texel and its empty-cell mask (or nullptr).
struct SlotView {
    int bias[3];  // kFloorBits + first texel per axis
    uint32_t texel0;
    const uint32_t* cmask;
};
// floor(t) for |t| < 2^22 in one addition rounded down: the sum with 1.5 * 2^23
// holds the integer in its low bits (a float-to-integer conversion runs at a
// quarter of the rate).  Any other t gives an integer far outside a slot.
constexpr float kFloorMagic = 12582912.0f;
constexpr int kFloorBits = 0x4B400000;

// Local index of the first tap of the sample at uvw per axis, in [0, 8] when
// all eight taps lie in the slot; t (the texel coordinate) kept per axis.
struct TapCell {
    float t[3], fl[3];
    int l[3];
    __device__ __forceinline__ TapCell(const RaycastParams& p, const SlotView& sv, F3 uvw) {
        const float* N = p.u.brick_pool_dimension;
        t[0] = uvw.x * N[0] - 0.5f;
        t[1] = uvw.y * N[1] - 0.5f;
        t[2] = uvw.z * N[2] - 0.5f;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            fl[a] = __fadd_rd(t[a], kFloorMagic);
            l[a] = __float_as_int(fl[a]) - sv.bias[a];
        }
    }
    __device__ __forceinline__ bool in_slot() const {
        return max(max((unsigned)l[0], (unsigned)l[1]), (unsigned)l[2]) <= 8u;
    }
};

// Whether the sample at uvw has to be fetched: false when its taps lie in the
// slot and the slot's mask marks their cell all zero (the sample is then
// exactly zero and compositing it changes nothing).
__device__ __forceinline__ bool sample_needed(const RaycastParams& p, const SlotView& sv, F3 uvw) {
    const TapCell c(p, sv, uvw);
    const bool in = c.in_slot();
    const uint32_t i = in ? (uint32_t)((c.l[2] * kCellsPerAxis + c.l[1]) * kCellsPerAxis + c.l[0]) : 0u;
    const uint32_t w = __ldg(sv.cmask + (i >> 5));
    return !(in && ((w >> (i & 31u)) & 1u));
}

// The sample at uvw: the in-slot filter (from stex, the slot's RGBA8 texels
// in shared memory, when given), else the general one.
template <int FMT, bool STAGED = false>
__device__ __forceinline__ float4 fetch_sample(const RaycastParams& p, const SlotView& sv, F3 uvw,
                                               const uint32_t* stex = nullptr) {
    const TapCell c(p, sv, uvw);
    if (!c.in_slot()) return sample_brick<FMT, false>(p, uvw);
    const uint32_t l000 = (uint32_t)((c.l[2] * 10 + c.l[1]) * 10 + c.l[0]);
    typename RawTexel<FMT>::T v[8];
    if (STAGED && stex) {
        static_assert(!STAGED || FMT == VV_FMT_RGBA8, "staging holds RGBA8 slots");
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t w = stex[l000 + (k & 1) + 10 * ((k >> 1) & 1) + 100 * (k >> 2)];
            memcpy(&v[k], &w, sizeof(w));
        }
    } else if constexpr (FMT == VV_FMT_DXT5) {
        // the taps' blocks from the local texel (4x4 texels of a slice each)
        const uint32_t blocks = sv.texel0 / 1000u * (uint32_t)dxt::kBlocksPerSlot;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int x = c.l[0] + (k & 1), y = c.l[1] + ((k >> 1) & 1), z = c.l[2] + (k >> 2);
            v[k] = RawTexel<FMT>::decode(p.bricks, blocks + (uint32_t)dxt::block_of(x, y, z), dxt::texel_of(x, y));
        }
    } else {
        const uint32_t i000 = sv.texel0 + l000;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            v[k] = RawTexel<FMT>::load(p.bricks, i000 + (k & 1) + 10 * ((k >> 1) & 1) + 100 * (k >> 2));
    }
    return filter8<FMT>(v, c.t[0] - (c.fl[0] - kFloorMagic), c.t[1] - (c.fl[1] - kFloorMagic),
                        c.t[2] - (c.fl[2] - kFloorMagic));
}

// A colour as RGBA8 unorm: round(clamp(c, 0, 1) * 255) per channel, to the
// nearest (ties to even); NaN stores 0.
__device__ __forceinline__ uint32_t unorm8(float c) {
    return __float2uint_rn(__fmul_rn(fminf(fmaxf(c, 0.0f), 1.0f), 255.0f));
}
__device__ __forceinline__ uint32_t pack_unorm8(float4 c) {
    return unorm8(c.x) | (unorm8(c.y) << 8) | (unorm8(c.z) << 16) | (unorm8(c.w) << 24);
}

// t / step for step = RS * 2^e.  With RS a power of two (rstep = 1 / RS)
// the quotient is t times a power of two: the same real number, so the same
// rounded result, as the division.
__device__ __forceinline__ float div_step(const RaycastParams& p, float t, float step, int e) {
    return p.rstep != 0.0f ? t * (p.rstep * pow2i(-e)) : t / step;
}

// ComputeMinRayBoxIntersection (GigaVoxelsNoLighting.frag:124-180): exit
// time over the planes facing away from the ray, 4.0 if none, t == 0 ignored.
__device__ __forceinline__ float min_exit(F3 p, F3 d, F3 mn, F3 mx) {
    float tmin = 4.0f;
    // planes 0..2: min faces with normals -x,-y,-z
    const float pa[3] = {p.x, p.y, p.z}, da[3] = {d.x, d.y, d.z};
    const float mna[3] = {mn.x, mn.y, mn.z}, mxa[3] = {mx.x, mx.y, mx.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float dn = -da[a];
        if (dn > 0.0f) {
            float t = (pa[a] - mna[a]) / dn;
            if (t < tmin && fabsf(t) > 0.0f) tmin = t;
        }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float dn = da[a];
        if (dn > 0.0f) {
            float t = -(pa[a] - mxa[a]) / dn;
            if (t < tmin && fabsf(t) > 0.0f) tmin = t;
        }
    }
    return tmin;
}

// (out of line for the unit box's walk, which seldom comes here; a call in the
// walk of the other boxes leaves a warp's lanes apart for good: their adjoint
// took 5.7 ms instead of 1.6, 960x540 of the 1024^3 terrain)
static __device__ __noinline__ float min_exit_call(F3 p, F3 d, F3 mn, F3 mx) { return min_exit(p, d, mn, mx); }

// The exit time of one axis is num / |d|, num the distance to the plane ahead,
// from y = exit_rcp(d) = RN(1 / |d|) (markstein_div, fixed_div.h: five
// operations for the IEEE quotient).  exit_time takes the division for a num
// below kExitSmall, and for |d| below 2^-60 any other num gives a quotient of
// at least 4, which no exit time is: y = 0 then makes it 0, which exit_time
// ignores the same way.
constexpr float kExitSmall = 3.4694469519536142e-18f;  // 2^-58
__device__ __forceinline__ float exit_rcp(float d) {
    const float b = fabsf(d);
    return b >= 8.6736173798840355e-19f ? 1.0f / b : 0.0f;  // 2^-60
}
// min_exit over the planes ahead of the ray (the only ones that face away
// from it), `ahead` one plane per axis; three independent quotients.
__device__ __forceinline__ float exit_time(F3 p, F3 d, F3 rinv, F3 lo, float size) {
    const F3 num = f3(d.x < 0.0f ? p.x - lo.x : (lo.x + size) - p.x, d.y < 0.0f ? p.y - lo.y : (lo.y + size) - p.y,
                      d.z < 0.0f ? p.z - lo.z : (lo.z + size) - p.z);
    if (fminf(fminf(num.x, num.y), num.z) < kExitSmall)
        return min_exit_call(p, d, lo, f3(lo.x + size, lo.y + size, lo.z + size));
    const float tx = markstein_div(num.x, fabsf(d.x), rinv.x), ty = markstein_div(num.y, fabsf(d.y), rinv.y),
                tz = markstein_div(num.z, fabsf(d.z), rinv.z);
    // 0: an axis the ray does not move along
    return fminf(fminf(tx != 0.0f ? tx : 4.0f, ty != 0.0f ? ty : 4.0f), fminf(tz != 0.0f ? tz : 4.0f, 4.0f));
}

__device__ __forceinline__ bool inside_box(F3 p, F3 mn, F3 mx) {
    return p.x > mn.x && p.y > mn.y && p.z > mn.z && mx.x > p.x && mx.y > p.y && mx.z > p.z;
}

template <bool COUNT>
__device__ __forceinline__ uint2 fetch_node(const RaycastParams& p, uint32_t x, uint32_t y, uint32_t z,
                                            bool& ok) {
    if (x >= (uint32_t)p.node_dim[0] || y >= (uint32_t)p.node_dim[1] || z >= (uint32_t)p.node_dim[2]) {
        ok = false;
        return make_uint2(0u, 0u);
    }
    const uint32_t bx = (uint32_t)p.node_dim[0] >> 1, by = (uint32_t)p.node_dim[1] >> 1;
    uint32_t blk = ((z >> 1) * by + (y >> 1)) * bx + (x >> 1);
    uint32_t idx = blk * 8u + ((x & 1u) | ((y & 1u) << 1) | ((z & 1u) << 2));
    if (COUNT) touch(p.node_touch, idx);
    return __ldg(p.nodes + idx);
}

// Grid position of node i of the pool.
__device__ __forceinline__ void node_position(const RaycastParams& p, uint32_t i, uint32_t& x, uint32_t& y, uint32_t& z) {
    const uint32_t blk = i >> 3, bz = block_div(blk, p.slice), r = blk - bz * p.slice.d, by = block_div(r, p.row);
    x = 2u * (r - by * p.row.d) + (i & 1u);
    y = 2u * by + ((i >> 1) & 1u);
    z = 2u * bz + ((i >> 2) & 1u);
}

// Index of the child in block `link` by the top bit of each axis' digits:
// 8 * block + (x | y << 1 | z << 2).
__device__ __forceinline__ uint32_t child_index(uint32_t link, uint32_t hx, uint32_t hy, uint32_t hz) {
    return __funnelshift_l(hx, __funnelshift_l(hy, __funnelshift_l(hz, link, 1), 1), 1);
}

// The child of node `idx` at `depth` that holds pos, into idx, where the
// walk's record does not give it (walknode.h: an odd or bad pointer) or the
// position's fixed-point digits have run out; false out of the grid.
static __device__ __noinline__ bool odd_child(const RaycastParams& p, F3 pos, int depth, uint32_t& idx) {
    const float sc = pow2i(depth);
    const F3 q = f3(pos.x * sc, pos.y * sc, pos.z * sc);
    const uint32_t w = __ldg(&p.nodes[idx].x);
    const uint32_t x = ((w >> 20) & 0x3FFu) + (q.x - floorf(q.x) >= 0.5f ? 1u : 0u),
                   y = ((w >> 10) & 0x3FFu) + (q.y - floorf(q.y) >= 0.5f ? 1u : 0u),
                   z = (w & 0x3FFu) + (q.z - floorf(q.z) >= 0.5f ? 1u : 0u);
    if (x >= (uint32_t)p.node_dim[0] || y >= (uint32_t)p.node_dim[1] || z >= (uint32_t)p.node_dim[2]) return false;
    const uint32_t bx = (uint32_t)p.node_dim[0] >> 1, by = (uint32_t)p.node_dim[1] >> 1;
    idx = (((z >> 1) * by + (y >> 1)) * bx + (x >> 1)) * 8u + ((x & 1u) | ((y & 1u) << 1) | ((z & 1u) << 2));
    return true;
}

// ---------------------------------------------------------------------------
// The ray walk of GigaVoxelsNoLighting.frag main (:490-751) after the ray
// set-up: leaf segments, each a descent from the root to the node that stops
// it (:563-622, :722-746) followed by TraverseConstant (:230-282) or
// TraverseBrick (:311-359) and the break test (:673-679).  The descent is its
// own loop, so the lanes of a warp descend together and march together.
// A visitor observes the walk:
//   bool segment_begin(const RayState&)   false ends the walk
//   bool sample(int kind, float4 src, F3 bpos, float T, int index)
//                                          before a sample is composited;
//                                          false ends the walk after it
//   void segment_end<UNIT>(const RaycastParams&, const RayState&)
//   void begin_record / end_record, box_segment: around the segments that take
//                                          samples, for the adjoint's records
//   void fail(int code)
// STEPS is the number of samples a march looks ahead (march_brick); the
// results do not depend on it.

struct WalkConsts {
    F3 C, vmin, vmax, up, left, bdim, pdim;
    float RS, astop, lod, pixel_size, rvh;
    int L, max_iter;
    uint2 root;  // the root's walk record (unit box) or words
};

struct RayState {
    F3 pos, dir;
    F3 rinv;        // exit_rcp of dir
    float4 dst;
    int iter;
    int nsamples;   // samples composited so far
    // octTreeNodePtr (not reset between segments): in the unit box the index of
    // the node, else x << 20 | y << 10 | z
    uint32_t nptr;
};

enum { kSampleConst = 0, kSampleBrick = 1 };

// Whether a draw takes the unit box's walk: its volume box is [0,1]^3 and the
// pool has walk records.
__device__ __forceinline__ bool unit_walk(const RaycastParams& p) {
    const vv_uniforms& u = p.u;
    return p.walk && u.vol_extent_min[0] == 0.0f && u.vol_extent_min[1] == 0.0f && u.vol_extent_min[2] == 0.0f &&
           u.vol_extent_max[0] == 1.0f && u.vol_extent_max[1] == 1.0f && u.vol_extent_max[2] == 1.0f;
}

__device__ __forceinline__ WalkConsts walk_consts(const RaycastParams& p, uint2 root) {
    const vv_uniforms& u = p.u;
    WalkConsts k;
    k.C = ld3(u.camera_position);
    k.vmin = ld3(u.vol_extent_min);
    k.vmax = ld3(u.vol_extent_max);
    k.up = ld3(u.camera_up);
    k.left = ld3(u.camera_left);
    k.bdim = ld3(u.brick_dimension);
    k.pdim = ld3(u.brick_pool_dimension);
    k.RS = u.ray_step_size;
    k.astop = u.alpha_stop;
    k.lod = u.lod_scalar;
    k.pixel_size = u.pixel_size;
    k.rvh = u.root_voxel_half_size;
    k.L = u.oct_tree_depth_minus_one;
    k.max_iter = p.max_iter;
    k.root = root;
    return k;
}

// The fragment's RayPosition: the box entry point of pixel (px,py)'s ray
// (GigaVoxels.vert) or its near-plane point (NearPlaneQuad.vert); false when
// the pixel has no fragment.
__device__ __forceinline__ bool ray_origin(const vv_uniforms& u, const WalkConsts& k, int px, int py, F3& pos) {
    const float fx = (float)px + 0.5f, fy = (float)py + 0.5f;
    const F3 d = f3(u.near_origin[0] + fx * u.near_dx[0] + fy * u.near_dy[0],
                    u.near_origin[1] + fx * u.near_dx[1] + fy * u.near_dy[1],
                    u.near_origin[2] + fx * u.near_dx[2] + fy * u.near_dy[2]);
    if (u.camera_inside) {
        pos = add(k.C, d);
        return true;
    }
    const float da[3] = {d.x, d.y, d.z}, ca[3] = {k.C.x, k.C.y, k.C.z};
    const float mn[3] = {k.vmin.x, k.vmin.y, k.vmin.z}, mx[3] = {k.vmax.x, k.vmax.y, k.vmax.z};
    float tenter = -INFINITY, texit = INFINITY;
    int axis = -1;
    bool frag = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (da[a] != 0.0f) {
            float t0 = (mn[a] - ca[a]) / da[a];
            float t1 = (mx[a] - ca[a]) / da[a];
            float tn = t0 < t1 ? t0 : t1, tf = t0 < t1 ? t1 : t0;
            if (tn > tenter) {
                tenter = tn;
                axis = a;
            }
            if (tf < texit) texit = tf;
        } else if (!(ca[a] > mn[a] && ca[a] < mx[a])) {
            frag = false;
        }
    }
    if (axis < 0 || !(tenter <= texit) || !(tenter > 0.0f)) frag = false;
    if (!frag) return false;
    float pa[3] = {ca[0] + da[0] * tenter, ca[1] + da[1] * tenter, ca[2] + da[2] * tenter};
#pragma unroll
    for (int a = 0; a < 3; ++a)
        if (a == axis) pa[a] = da[a] > 0.0f ? mn[a] : mx[a];
    pos = f3(pa[0], pa[1], pa[2]);
    return true;
}

// Ray set-up after the origin (:500-510): direction, jitter, inside test.
__device__ __forceinline__ bool ray_start(const RaycastParams& p, const WalkConsts& k, int px, int py, F3 pos,
                                          RayState& s) {
    const vv_uniforms& u = p.u;
    s.dir = normalize3(sub(pos, k.C));
    const int J = u.jitter_tex_size;
    const float jitter = (float)p.jitter[(py % J) * J + (px % J)] / 255.0f;
    s.pos = add(pos, muls(muls(s.dir, k.RS), jitter));
    s.rinv = f3(exit_rcp(s.dir.x), exit_rcp(s.dir.y), exit_rcp(s.dir.z));
    s.dst = make_float4(0.f, 0.f, 0.f, 0.f);
    s.iter = 0;
    s.nsamples = 0;
    s.nptr = 0u;
    return inside_box(s.pos, k.vmin, k.vmax);
}

// The path of the ray's last descent, per thread in shared memory: the child
// link (walknode.h) of the node of each level it went on from, `stride`
// elements apart per level.  A later descent whose position lies in the same
// level-r node, and whose LOD test lodb::clear_range shows to continue at
// every level down to r, starts at that node's child: the levels it skips
// would take exactly the recorded path (same nodes, every stop condition
// false), so the walk is unchanged.  (Starting at node r itself, by its index,
// cost one more dependent load and visit of three a segment.)
constexpr int kPathLevels = 11;  // levels 0..10
struct StageBuf;
struct PathSlots {
    uint32_t* link;
    int stride;
    StageBuf* stage;  // the warp's staged brick (VV_RAYCAST_STAGED), else nullptr
};

// ---- brick staging (VV_RAYCAST_STAGED, RGBA8 pools) ------------------------
//
// Each warp owns one 10^3-texel RGBA8 slot copy in shared memory.  When the
// lanes that reach a brick segment together share a slot (__match_any_sync),
// the largest such group copies that slot's 4000 bytes with one
// cp.async.bulk (global -> this CTA's own shared memory) and
// samples it from shared memory; other lanes read the pool as usual.
//   state = tag << 32 | mask: tag = the slot the buffer holds (kNoSlot while
//   a copy is in flight), mask = the lanes reading it.  A group joins a
//   buffer that holds its slot, or refills an unread one; both by one
//   atomicCAS of its leader, so a copy never overwrites texels being read.
// The only wait is the copy's own mbarrier (bounded: on timeout the status
// is set, the buffer stays claimed and the lanes read the pool).
constexpr uint32_t kNoSlot = 0xFFFFFFFFu;
constexpr int kStageMinLanes = 4;  // smallest group worth a copy
struct __align__(16) StageBuf {
    uint32_t texels[1000];
    unsigned long long state;
    unsigned long long bar;
    uint32_t phase;  // completed copies (the mbarrier's phase parity)
};

// Lane 0 of the warp, before any lane returns.
__device__ __forceinline__ void stage_init(StageBuf* sb) {
    sb->state = (unsigned long long)kNoSlot << 32;
    sb->phase = 0u;
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&sb->bar);
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Called by the converged lanes entering a brick segment; `slot` is the
// lane's slot or kNoSlot.  True: the lane reads its slot from sb->texels
// until stage_release.
__device__ __forceinline__ bool stage_acquire(StageBuf* sb, const void* pool, uint32_t slot, int* status) {
    const unsigned am = __activemask();
    const unsigned peers = __match_any_sync(am, slot);
    const int lane = (int)(threadIdx.x & 31u);
    const int leader = __ffs(peers) - 1;
    // 1: joined a buffer holding the slot, 2: claimed it for a copy
    int act = 0;
    if (lane == leader && slot != kNoSlot) {
        unsigned long long st = *(volatile unsigned long long*)&sb->state;
        for (int tries = 0; tries < 4; ++tries) {
            unsigned long long want;
            int a;
            if ((uint32_t)(st >> 32) == slot) {
                want = st | peers;
                a = 1;
            } else if ((uint32_t)st == 0u && __popc(peers) >= kStageMinLanes) {
                want = ((unsigned long long)kNoSlot << 32) | peers;
                a = 2;
            } else {
                break;
            }
            const unsigned long long old = atomicCAS(&sb->state, st, want);
            if (old == st) {
                act = a;
                break;
            }
            st = old;
        }
        __threadfence_block();
    }
    act = __shfl_sync(peers, act, leader);
    if (act == 2) {
        const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&sb->bar);
        const uint32_t parity = sb->phase & 1u;
        if (lane == leader) {
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(sb->texels);
            const uint32_t* src = (const uint32_t*)pool + (size_t)slot * 1000u;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], 4000;" ::"r"(bar) : "memory");
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 4000, [%2];" ::"r"(dst),
                "l"(src), "r"(bar)
                : "memory");
        }
        uint32_t done = 0u;
        for (int i = 0; i < (1 << 20) && !done; ++i) {
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done)
                : "r"(bar), "r"(parity)
                : "memory");
        }
        done = __all_sync(peers, done != 0u);
        if (!done) {
            set_status(status, VV_ERR_TIMEOUT);
            return false;
        }
        __syncwarp(peers);
        if (lane == leader) {
            sb->phase = sb->phase + 1u;
            __threadfence_block();
            atomicExch(&sb->state, ((unsigned long long)slot << 32) | peers);
        }
        __syncwarp(peers);
        return true;
    }
    return act == 1;
}

// The lane stops reading the staged slot.
__device__ __forceinline__ void stage_release(StageBuf* sb) {
    __threadfence_block();
    atomicAnd(&sb->state, ~(1ull << (threadIdx.x & 31u)));
}

// ---- lighting (GigaVoxels.frag with ComputeLighting) ----------------------

// texture(BrickGradientsSampler, p).rgb (:316): the trilinear filter of
// sample_brick over the gradient pool (FP32 gradients, or RGBA8 / 255).
template <int GFMT>
__device__ __forceinline__ F3 sample_gradient(const RaycastParams& p, F3 uvw) {
    const float* N = p.u.brick_pool_dimension;
    const Axis ax = axis_taps(uvw.x, N[0], p.slots[0] * 10);
    const Axis ay = axis_taps(uvw.y, N[1], p.slots[1] * 10);
    const Axis az = axis_taps(uvw.z, N[2], p.slots[2] * 10);
    const uint32_t SX = (uint32_t)p.slots[0], SY = (uint32_t)p.slots[1];
    typename RawTexel<GFMT>::T v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const uint32_t sx = (uint32_t)((k & 1) ? ax.s1 : ax.s0), sy = (uint32_t)((k & 2) ? ay.s1 : ay.s0),
                       sz = (uint32_t)((k & 4) ? az.s1 : az.s0);
        const int lx = (k & 1) ? ax.l1 : ax.l0, ly = (k & 2) ? ay.l1 : ay.l0, lz = (k & 4) ? az.l1 : az.l0;
        v[k] = RawTexel<GFMT>::load(p.grads, ((sz * SY + sy) * SX + sx) * 1000u + (uint32_t)((lz * 10 + ly) * 10 + lx));
    }
    const float4 c = filter8<GFMT>(v, ax.f, ay.f, az.f);
    return f3(c.x, c.y, c.z);
}

// pow(x, 100) as x^64 * x^32 * x^4 by squarings (the shininess power).
__device__ __forceinline__ float pow100(float x) {
    const float x2 = x * x, x4 = x2 * x2, x8 = x4 * x4, x16 = x8 * x8, x32 = x16 * x16, x64 = x32 * x32;
    return (x64 * x32) * x4;
}

// shading (:293-312) with k_Ambient 0.05, k_Diffuse = k_Specular = 1,
// k_Shininess 100, added to src.rgb when the gradient normalizes (:370-384).
__device__ __forceinline__ void light_sample(const RaycastParams& p, F3 bpos, F3 dir, F3 light_dir, float4& src) {
    F3 n = p.grad_fmt == VV_FMT_RGBA8  ? sample_gradient<VV_FMT_RGBA8>(p, bpos)
           : p.grad_fmt == VV_FMT_DXT1 ? sample_gradient<VV_FMT_DXT1>(p, bpos)
                                       : sample_gradient<VV_FMT_FP32>(p, bpos);
    if (p.u.gradients_unsigned) n = sub(muls(n, 2.0f), f3(1.0f, 1.0f, 1.0f));  // LookupGradient :318-322
    n = normalize3(n);
    if (isnan(n.x) || isnan(n.y) || isnan(n.z)) return;  // homogeneous region: no lighting
    const F3 rgb = f3(src.x, src.y, src.z);
    const F3 to_camera = muls(dir, -1.0f);
    const F3 halfway = normalize3(add(light_dir, to_camera));
    const float diffuse_light = fmaxf(dot3(light_dir, n), 0.0f);
    F3 diffuse = f3(0.0f, 0.0f, 0.0f), specular = f3(0.0f, 0.0f, 0.0f);
    if (diffuse_light > 0.0f) {
        diffuse = muls(rgb, diffuse_light);
        specular = muls(rgb, pow100(fmaxf(dot3(halfway, n), 0.0f)));
    }
    const F3 ambient = muls(rgb, 0.05f);
    const F3 sh = add(add(ambient, diffuse), specular);
    src.x = src.x + sh.x;
    src.y = src.y + sh.y;
    src.z = src.z + sh.z;
}

// The lower corner of the depth-d node of the unit box that holds pos, whose
// fixed-point form (1 + pos rounded to zero, see walk_round_unit) is ix, iy, iz.
__device__ __forceinline__ F3 unit_corner(F3 pos, uint32_t ix, uint32_t iy, uint32_t iz, int d) {
    if (d <= 23) {
        const uint32_t m = 0xFFFFFFFFu << (23 - d);
        return f3(__uint_as_float(ix & m) - 1.0f, __uint_as_float(iy & m) - 1.0f, __uint_as_float(iz & m) - 1.0f);
    }
    const float sc = pow2i(d), rs = pow2i(-d);
    return f3(floorf(pos.x * sc) * rs, floorf(pos.y * sc) * rs, floorf(pos.z * sc) * rs);
}

// The slot whose texels a brick pointer covers with a border of one (slot
// origin + 1 per axis), or kNoSlot for another pointer.
__device__ __forceinline__ uint32_t slot_of(const RaycastParams& p, uint32_t bw) {
    const uint32_t x = (bw >> 20) & 0x3FFu, y = (bw >> 10) & 0x3FFu, z = bw & 0x3FFu;
    const uint32_t sx = (x - 1u) / 10u, sy = (y - 1u) / 10u, sz = (z - 1u) / 10u;  // (a pointer of 0 wraps)
    if (sx * 10u + 1u != x || sy * 10u + 1u != y || sz * 10u + 1u != z || sx >= (uint32_t)p.slots[0] ||
        sy >= (uint32_t)p.slots[1] || sz >= (uint32_t)p.slots[2])
        return kNoSlot;
    return (sz * (uint32_t)p.slots[1] + sy) * (uint32_t)p.slots[0] + sx;
}

// Whether n samples of a brick segment that enters its node at the relative
// position brp all fall in empty cells of slot `slot`, by the projections of
// the occupied cells (cellmask.cuh).  The texel coordinates of the first and
// the last sample bound those between, per axis; they are off from the
// shader's sums by less than 0.01 texel for up to 128 samples (a sum of
// coordinates below 1 in pools of at most 1020 texels rounds by 6e-5 texel).
// A count out of 1..pass_steps (set_divisors; a quotient by a tiny step
// overflows) shows nothing.
__device__ __forceinline__ bool brick_empty(const RaycastParams& p, const WalkConsts& k, F3 brp, F3 dir, int n,
                                            uint32_t slot) {
    const uint32_t occ = __ldg(p.cell_mask + (size_t)slot * kCellMaskWords + kOccupancyWord);
    const float m = (float)(n - 1);
    const F3 u0 = f3(fmaf(brp.x, k.bdim.x, 0.5f), fmaf(brp.y, k.bdim.y, 0.5f), fmaf(brp.z, k.bdim.z, 0.5f));
    const F3 u1 = f3(fmaf(m * dir.x, p.bstep_texel[0], u0.x), fmaf(m * dir.y, p.bstep_texel[1], u0.y),
                     fmaf(m * dir.z, p.bstep_texel[2], u0.z));
    bool in = (unsigned)(n - 1) < (unsigned)p.pass_steps, empty = false;
    const float a0[3] = {u0.x, u0.y, u0.z}, a1[3] = {u1.x, u1.y, u1.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float lo = fminf(a0[a], a1[a]) - 0.02f, hi = fmaxf(a0[a], a1[a]) + 0.02f;
        in = in && lo >= 0.0f && hi < 9.0f;
        // bits of the slabs [floor(lo), floor(hi)], by the floor of TapCell
        const int l = __float_as_int(__fadd_rd(lo, kFloorMagic)) & 15, h = __float_as_int(__fadd_rd(hi, kFloorMagic)) & 15;
        empty = empty || (((2u << h) - (1u << l)) & (occ >> (9 * a)) & 0x1FFu) == 0u;
    }
    return in && empty;
}

// A brick segment about to be marched (TraverseBrick, :311-359): the first
// sample's brick-pool position, the steps and the slot.
struct BrickMarch {
    F3 bpos, bstep, wstep;
    float step;
    int n;  // samples to the exit
    uint32_t slot_id;
    SlotView sv;
    // bw: the brick's pool pointer; brp: the relative position in its node
    template <bool COUNT>
    __device__ __forceinline__ void set(const RaycastParams& p, const WalkConsts& k, const RayState& s, uint32_t bw, F3 brp,
                                        int brick_depth, float t) {
        // the six quotients by the pool dimensions from their reciprocals (fixed_div.h)
        const uint32_t ptr[3] = {(bw >> 20) & 0x3FFu, (bw >> 10) & 0x3FFu, bw & 0x3FFu};
        const F3 bptr = f3(fixed_div((float)ptr[0], k.pdim.x, p.rpdim[0]), fixed_div((float)ptr[1], k.pdim.y, p.rpdim[1]),
                           fixed_div((float)ptr[2], k.pdim.z, p.rpdim[2]));
        const F3 brb = mul(brp, k.bdim);
        bpos = add(bptr, f3(fixed_div(brb.x, k.pdim.x, p.rpdim[0]), fixed_div(brb.y, k.pdim.y, p.rpdim[1]),
                            fixed_div(brb.z, k.pdim.z, p.rpdim[2])));
        const float ratio = pow2i(k.L - brick_depth);
        wstep = muls(muls(s.dir, k.RS), ratio);
        bstep = mul(s.dir, ld3(p.u.brick_step_vector));
        step = k.RS * ratio;
        n = (int)div_step(p, t, step, k.L - brick_depth) + 1;
        // taps inside this brick's slot skip the general texel addressing
        sv.texel0 = 0u;
        sv.cmask = nullptr;  // (not in footprint counts)
        sv.bias[0] = sv.bias[1] = sv.bias[2] = 0;  // no texel coordinate is in this slot
        slot_id = slot_of(p, bw);
        if (slot_id != kNoSlot) {
            sv.texel0 = slot_id * 1000u;
#pragma unroll
            for (int a = 0; a < 3; ++a) sv.bias[a] = kFloorBits - 1 + (int)ptr[a];
            if (!COUNT && p.cell_mask) sv.cmask = p.cell_mask + (size_t)slot_id * kCellMaskWords;
        }
    }
};
// A brick segment whose samples are all in empty cells is stepped over: the
// position takes the shader's sums, nothing is composited.  False, and nothing
// done, when that is not shown.
__device__ __forceinline__ bool step_over_brick(const RaycastParams& p, const WalkConsts& k, RayState& s, F3 corner,
                                                uint32_t bw, int brick_depth, float t) {
    const uint32_t slot = slot_of(p, bw);
    if (slot == kNoSlot) return false;
    const float ratio = pow2i(k.L - brick_depth);
    const int n = (int)div_step(p, t, k.RS * ratio, k.L - brick_depth) + 1;
    if (!brick_empty(p, k, muls(sub(s.pos, corner), pow2i(brick_depth)), s.dir, n, slot)) return false;
    const F3 wstep = muls(muls(s.dir, k.RS), ratio);
    for (int i = 0; i < n; ++i) s.pos = add(s.pos, wstep);
    s.nsamples += n;
    return true;
}

// lightDir = normalize(LightPosition - rayWorldPosition) at entry (:337)
template <bool LIT>
__device__ __forceinline__ F3 entry_light(const RaycastParams& p, const RayState& s) {
    return LIT ? normalize3(sub(ld3(p.u.light_position), s.pos)) : f3(0.0f, 0.0f, 0.0f);
}
// One sample composited (the zero of an empty cell only counted: T * 0 + dst is
// dst but for an infinite T, and lighting adds nothing to it); false when the
// visitor ends the walk after it.
template <bool LIT, class V>
__device__ __forceinline__ bool take_sample(const RaycastParams& p, RayState& s, V& vis, float4 src, F3 bpos, F3 light_dir,
                                            bool empty) {
    src.w = 1.0f - (1.0f - src.w);
    if (LIT && !empty) light_sample(p, bpos, s.dir, light_dir, src);
    const float T = 1.0f - s.dst.w;
    const bool go = vis.sample(kSampleBrick, src, bpos, T, s.nsamples);
    if (!empty) s.dst = composite(T, src, s.dst);
    ++s.nsamples;
    return go;
}

// The march, a lane on its own; false when the visitor ends the walk.  Samples
// of empty cells are not fetched: the 256^3 volume in a box of three quarters at
// 512x512, every sample fetched 408 us, DXT5 1123, lit 839; so 317, 554, 435.
template <int FMT, bool COUNT, class V, bool LIT>
__device__ __forceinline__ bool march_brick(const RaycastParams& p, const WalkConsts& k, RayState& s, V& vis, BrickMarch& b) {
    const F3 light_dir = entry_light<LIT>(p, s);
    bool go = true;
    for (int i = 0; i < b.n && go; ++i) {
        s.pos = add(s.pos, b.wstep);
        if (s.dst.w > k.astop) {
            s.pos = add(s.pos, muls(s.dir, (float)(b.n - (i + 1)) * b.step));
            break;
        }
        const bool empty = !COUNT && b.sv.cmask && !sample_needed(p, b.sv, b.bpos);
        float4 src = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (!empty) src = COUNT ? sample_brick<FMT, COUNT>(p, b.bpos) : fetch_sample<FMT>(p, b.sv, b.bpos);
        go = take_sample<LIT>(p, s, vis, src, b.bpos, light_dir, empty);
        b.bpos = add(b.bpos, b.bstep);
    }
    return go;
}

// The march of the lanes `lanes` of a warp together.  Most samples fall in
// empty cells: each lane steps over them by the position sums alone (the
// shader's, one per step and in its order) to its next sample that has to be
// fetched, where the lanes meet.  The warp then filters once for all of them:
// as often as its busiest lane needs it, not at every step at which any lane
// does.  AHEAD cells are tested at a time, their mask loads in flight together.
template <int FMT, class V, int AHEAD, bool LIT, bool STAGED>
__device__ __forceinline__ bool march_brick_warp(const RaycastParams& p, const WalkConsts& k, RayState& s, V& vis,
                                                 BrickMarch& b, unsigned lanes, StageBuf* stage) {
    const F3 light_dir = entry_light<LIT>(p, s);
    const bool staged = STAGED && stage_acquire(stage, p.bricks, b.slot_id, p.status);
    const uint32_t* stex = staged ? stage->texels : nullptr;
    bool go = true;
    int left = b.n;  // samples not yet taken
    if (left > 0 && s.dst.w > k.astop) {  // opaque before the first one: the ray moves to the exit
        s.pos = add(add(s.pos, b.wstep), muls(s.dir, (float)(left - 1) * b.step));
        left = 0;
    }
    int ahead = 0;        // of those left, tested
    uint32_t needed = 0;  // bit j: the j-th of the tested has to be fetched
    while (__any_sync(lanes, left > 0)) {
        bool need = left > 0;
        if (!V::kEverySample && need && b.sv.cmask) {
            if (AHEAD == 1) {
                while (left > 0 && !sample_needed(p, b.sv, b.bpos)) {
                    s.pos = add(s.pos, b.wstep);
                    b.bpos = add(b.bpos, b.bstep);
                    ++s.nsamples;
                    --left;
                }
                need = left > 0;
            } else {
                for (;;) {
                    if (ahead == 0) {
                        F3 q = b.bpos;
                        needed = 0u;
#pragma unroll
                        for (int j = 0; j < AHEAD; ++j) {
                            if (sample_needed(p, b.sv, q)) needed |= 1u << j;
                            q = add(q, b.bstep);
                        }
                        ahead = min(AHEAD, left);
                        needed &= (1u << ahead) - 1u;
                    }
                    const int skip = needed ? __ffs(needed) - 1 : ahead;
                    for (int j = 0; j < skip; ++j) {
                        s.pos = add(s.pos, b.wstep);
                        b.bpos = add(b.bpos, b.bstep);
                    }
                    s.nsamples += skip;
                    left -= skip;
                    ahead -= skip;
                    needed >>= skip;
                    if (needed || left == 0) break;
                }
                need = left > 0;
                --ahead;
                needed >>= 1;
            }
        }
        __syncwarp(lanes);
        if (need) {
            s.pos = add(s.pos, b.wstep);
            float4 src = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const bool empty = V::kEverySample && b.sv.cmask && !sample_needed(p, b.sv, b.bpos);
            if (!empty) src = fetch_sample<FMT, STAGED>(p, b.sv, b.bpos, stex);
            go = take_sample<LIT>(p, s, vis, src, b.bpos, light_dir, empty);
            b.bpos = add(b.bpos, b.bstep);
            --left;
            if (left > 0 && s.dst.w > k.astop) {  // the step at which the stop is seen, then the rest at once
                s.pos = add(add(s.pos, b.wstep), muls(s.dir, (float)(left - 1) * b.step));
                left = 0;
            }
            if (!go) left = 0;
        }
    }
    if (staged) stage_release(stage);
    return go;
}

// TraverseConstant (:230-282) of a node at `depth`, to the exit time t.  An
// empty node (alpha / 255 < 0.005) is stepped over; the samples of another are
// composited: false when the visitor ends the walk.
__device__ __forceinline__ bool constant_empty(uint32_t w1) { return (w1 >> 24) < 2u; }
__device__ __forceinline__ void step_over_constant(const RaycastParams& p, const WalkConsts& k, RayState& s, int depth,
                                                   float t) {
    const float step = k.RS * pow2i(k.L - depth);
    const int n = (int)div_step(p, t, step, k.L - depth) + 1;
    s.pos = add(s.pos, muls(s.dir, (float)n * step));
}
// The sample of a constant node.
__device__ __forceinline__ float4 constant_sample(const WalkConsts& k, uint32_t w1, int depth) {
    const float ratio = pow2i(k.L - depth);
    const float aw = (float)(w1 >> 24) / 255.0f;
    return make_float4((float)(w1 & 255u) / 255.0f * ratio, (float)((w1 >> 8) & 255u) / 255.0f * ratio,
                       (float)((w1 >> 16) & 255u) / 255.0f * ratio, 1.0f - pow_pow2(1.0f - aw, k.L - depth));
}
template <class V>
__device__ __forceinline__ bool march_constant(const RaycastParams& p, const WalkConsts& k, RayState& s, V& vis,
                                               uint32_t w1, int depth, float t) {
    const float ratio = pow2i(k.L - depth);
    const float step = k.RS * ratio;
    const int n = (int)div_step(p, t, step, k.L - depth) + 1;
    bool go = true;
    const F3 wstep = muls(s.dir, step);
    const float4 src = constant_sample(k, w1, depth);
    for (int i = 0; i < n && go; ++i) {
        s.pos = add(s.pos, wstep);
        if (s.dst.w > k.astop) {
            const int rem = n - (i + 1);
            s.pos = add(s.pos, muls(s.dir, (float)rem * step));
            break;
        }
        const float T = 1.0f - s.dst.w;
        go = vis.sample(kSampleConst, src, s.pos, T, s.nsamples);
        s.dst = composite(T, src, s.dst);
        ++s.nsamples;
    }
    return go;
}

// ComputeVoxelSize (:429-441) * LodScalar against PixelSize, in the shader's
// order: whether the descent stops at a node of half voxel size vhalf.
__device__ __forceinline__ bool lod_stops(const WalkConsts& k, F3 pos, float vhalf) {
    const F3 uh = muls(k.up, vhalf), lh = muls(k.left, vhalf);
    const F3 ll = normalize3(sub(add(sub(pos, uh), lh), k.C));
    const F3 ur = normalize3(sub(sub(add(pos, uh), lh), k.C));
    const float proj = (1.0f - dot3(ll, ur)) * k.lod;
    return k.pixel_size > proj;
}

// One leaf segment in a volume box other than [0,1]^3, or with footprint
// counts: the descent from the root with the node's extent and the relative
// position tracked in binary32 as the shader does.
template <int FMT, bool COUNT, class V, bool LIT>
__device__ __forceinline__ bool walk_segment_box(const RaycastParams& p, const WalkConsts& k, RayState& s, V& vis) {
    if (!vis.segment_begin(s)) return false;
    vis.box_segment(s);
    bool ok = true;
    uint2 node = k.root;
    F3 ext_min = k.vmin, ext_max = k.vmax;
    float node_size = 1.0f, vhalf = k.rvh;
    F3 rbp = s.pos, cur_brp = s.pos;
    uint32_t cur_bw = k.root.y;
    int depth = 0, brick_depth = 0;
    bool is_const, loaded;
    for (;;) {
        if (++s.iter > k.max_iter) {
            vis.fail(VV_ERR_TIMEOUT);
            return false;
        }
        is_const = (node.x & kConstant) != 0u;
        loaded = (node.x & kResident) != 0u;
        if (loaded) {
            cur_bw = node.y;
            cur_brp = rbp;
            brick_depth = depth;
        }
        const uint32_t cx = (node.x >> 20) & 0x3FFu, cy = (node.x >> 10) & 0x3FFu, cz = node.x & 0x3FFu;
        if ((!is_const && !loaded) || (cx == 0u && cy == 0u && cz == 0u)) break;
        if (lod_stops(k, s.pos, vhalf)) break;
        const F3 boff = muls(rbp, 2.0f);
        const uint32_t ox = boff.x >= 1.0f ? 1u : 0u;
        const uint32_t oy = boff.y >= 1.0f ? 1u : 0u;
        const uint32_t oz = boff.z >= 1.0f ? 1u : 0u;
        rbp = sub(boff, f3((float)ox, (float)oy, (float)oz));
        const uint32_t x = cx + ox, y = cy + oy, z = cz + oz;
        ++depth;
        node_size = node_size * 0.5f;
        ext_min = add(ext_min, muls(f3((float)ox, (float)oy, (float)oz), node_size));
        ext_max = sub(ext_max, muls(f3(1.0f - (float)ox, 1.0f - (float)oy, 1.0f - (float)oz), node_size));
        vhalf = vhalf * 0.5f;
        node = fetch_node<COUNT>(p, x, y, z, ok);
        if (!ok) {
            vis.fail(VV_ERR_BOUNDS);
            return false;
        }
        s.nptr = (x << 20) | (y << 10) | z;
    }
    const float t = min_exit(s.pos, s.dir, ext_min, ext_max);
    if (is_const) {
        if (constant_empty(node.y)) step_over_constant(p, k, s, depth, t);
        else if (!march_constant(p, k, s, vis, node.y, depth, t)) return false;
    } else {
        BrickMarch b;
        b.set<COUNT>(p, k, s, cur_bw, cur_brp, brick_depth, t);
        if (!march_brick<FMT, COUNT, V, LIT>(p, k, s, vis, b)) return false;
    }
    vis.template segment_end<false>(p, s);
    if (s.dst.w > k.astop && (is_const || loaded)) return false;
    // restart from the root (:688-720); the node pointer keeps its value
    return inside_box(s.pos, k.vmin, k.vmax);
}
// Where a ray's last descent stopped: its depth (0: no path kept), the fixed-point
// position it was made for and the levels of its path that hold a brick.
struct WalkResume {
    int prev_depth = 0;
    uint32_t ix = 0u, iy = 0u, iz = 0u, res = 0u;
};

// The walk of a warp's rays in the unit box; all 32 lanes call it, `alive` the
// ones that have a ray.
//
// The walk is bound by the warp instructions it issues, and left to itself a
// warp comes apart: lanes that left a loop early ran on alone, at 14 lanes a
// descent and 5 a brick (256^3 terrain, 512x512).  So the lanes meet by vote
// before every descent, after it and before every march.  Most segments are
// descents to an empty constant node and a step to its far side (11 of 15
// segments of a ray there, 17 of 19 at 2048^3), so lanes that have reached a
// brick wait until the visitor's kGather of them have, or no lane can go on
// without, and then march together.  256^3 at 512x512 / 2048^3 at 3840x2160, whole draw:
// 0.368 / 8.87 ms before; 0.289 / 6.36 ms when every brick is marched at once
// (kGather 1), 0.280 / 6.20 at 8, 0.287 / 6.15 at 16, 0.315 / 6.65 when every
// lane is waited for.
//
// A position in [0,1) plus one, rounded to zero, holds its first 23 binary
// digits in the significand: digit 22-d picks the child at depth d (what the
// shader's repeated doubling of the relative position gives), the common
// prefix of two positions is the part of the path they share, and a node's
// lower corner is its position's prefix: all integer operations, one per
// axis.  Beyond depth 22 (a chain of nodes takes one block a level, so a pool
// may hold one of any depth) the digits come from the scaled position itself.
// The pool pointer of the deepest resident node (at depth d) of the last
// descent, whose position the resume state holds.
constexpr uint32_t kOnPath = 0xFFFFFFFFu;
__device__ __forceinline__ uint32_t brick_pointer(const RaycastParams& p, const PathSlots& path, const WalkResume& wr,
                                                  int d, uint32_t brick_idx) {
    if (brick_idx == kOnPath)
        brick_idx = d == 0 ? 0u : child_index(path.link[(d - 1) * path.stride], wr.ix << (8 + d), wr.iy << (8 + d),
                                              wr.iz << (8 + d));
    return __ldg(&p.walk[brick_idx].y);
}

struct NoRefill {
    static constexpr bool kOn = false;
    template <class V>
    __device__ __forceinline__ void take(RayState&, V&, WalkResume&, bool, bool&) {}
};
template <int FMT, class V, int AHEAD, bool LIT, bool STAGED, class R>
__device__ __forceinline__ void walk_warp(const RaycastParams& p, const WalkConsts& k, RayState& s, V& vis,
                                          const PathSlots& path, bool alive, R&& refill) {
    constexpr unsigned kAll = 0xFFFFFFFFu;
    WalkResume wr;
    uint2 node = k.root;
    uint32_t brick_idx = 0u;  // the deepest resident node of the path, or kOnPath: by the kept path
    int depth = 0, brick_depth = 0;
    bool is_const = false, loaded = false;
    bool pending = false;  // the lane's segment takes samples
    // lanes to wait for, of the rays the warp has
    const int gather = refill.kOn ? V::kGather : max(1, V::kGather * __popc(__ballot_sync(kAll, alive)) / 32);
    float t = 0.0f;
    for (;;) {
        for (;;) {
            if (refill.kOn) refill.take(s, vis, wr, alive || pending, alive);
            if (__popc(__ballot_sync(kAll, pending)) >= gather) break;
            bool go = alive && !pending;
            if (go) go = alive = vis.segment_begin(s);
            const unsigned lanes = __ballot_sync(kAll, go);
            if (lanes == 0u) break;
            if (go) {
                int skip_lo = 0, skip_hi;
                const lodb::V3 at{s.pos.x, s.pos.y, s.pos.z};
                skip_hi = lodb::deep_levels(p.lodk, at);
                if (skip_hi < 0) {
                    lodb::clear_range(p.lodk, at, skip_lo, skip_hi);
                    if (skip_hi < skip_lo) skip_lo = skip_hi = 1 << 20;  // none
                }
                const uint32_t ix = __float_as_uint(__fadd_rz(s.pos.x, 1.0f)),
                               iy = __float_as_uint(__fadd_rz(s.pos.y, 1.0f)),
                               iz = __float_as_uint(__fadd_rz(s.pos.z, 1.0f));
                uint32_t res = 0u;  // levels of the path whose node is resident
                uint32_t idx = 0u;  // the node
                node = k.root;
                depth = 0;
                brick_idx = 0u;
                if (wr.prev_depth > 0 && skip_lo == 0) {
                    // the deepest node the last descent went on from that holds
                    // this position too and from which this one surely goes on
                    const uint32_t diff = (ix ^ wr.ix) | (iy ^ wr.iy) | (iz ^ wr.iz);
                    const int r = min(min(wr.prev_depth - 1, __clz(diff) - 9), skip_hi);
                    if (r >= 0 && s.iter + r + 1 <= k.max_iter) {
                        depth = r + 1;
                        idx = child_index(path.link[r * path.stride], ix << (9 + r), iy << (9 + r), iz << (9 + r));
                        node = __ldg(p.walk + idx);
                        s.nptr = idx;
                        s.iter += depth;
                        res = wr.res & ((2u << r) - 1u);
                        brick_idx = res ? kOnPath : 0u;
                    }
                }
                // ---- descent to the node that stops it.  The next binary digit
                // of the position per axis is kept in the top bit of hx, hy, hz.
                uint32_t hx = ix << (9 + depth), hy = iy << (9 + depth), hz = iz << (9 + depth);
                const int last = depth + k.max_iter - s.iter;  // depths from here on are past the iteration bound
                const int first = depth;
                const unsigned shown = (unsigned)(skip_hi - skip_lo);
                int error = VV_OK;
                bool odd = false;  // a child that its link does not give: no path to resume
                int deep = 0;      // the last resident level past the 32 of res, but for the last node's
                for (;;) {
                    if (depth >= last) {
                        error = VV_ERR_TIMEOUT;
                        break;
                    }
                    if (node.x & kResident) {
                        res |= 1u << (depth & 31);
                        brick_idx = idx;
                    }
                    const uint32_t link = node.x & kLinkMask;
                    if (node.x < kConstant || link == 0u) break;  // neither constant nor resident, or no children
                    // the LOD test, only when the other two stop conditions do
                    // not decide (it has no side effects), and not at the
                    // levels lodb::clear_range has shown to continue
                    if ((unsigned)(depth - skip_lo) > shown && lod_stops(k, s.pos, k.rvh * pow2i(-depth))) break;
                    if (depth < kPathLevels) path.link[depth * path.stride] = link;
                    if (depth < 23 && link < kLinkOdd) {
                        idx = child_index(link, hx, hy, hz);
                    } else {
                        odd = true;
                        if (depth > 31 && (node.x & kResident)) deep = depth;
                        if (!odd_child(p, s.pos, depth, idx)) {
                            error = VV_ERR_BOUNDS;
                            break;
                        }
                    }
                    ++depth;
                    hx += hx;
                    hy += hy;
                    hz += hz;
                    node = __ldg(p.walk + idx);
                }
                s.iter += depth - first + 1;
                if (depth > first) s.nptr = idx;
                is_const = (node.x & kConstant) != 0u;
                loaded = (node.x & kResident) != 0u;
                __syncwarp(lanes);
                wr.prev_depth = depth < kPathLevels && !odd ? depth : 0;
                wr.ix = ix;
                wr.iy = iy;
                wr.iz = iz;
                wr.res = res;
                // (levels past 31 share the bits of res: a chain of nodes may be that deep)
                brick_depth = loaded ? depth : max(deep, 31 - __clz(res));  // (deep is 0 without one)
                t = exit_time(s.pos, s.dir, s.rinv, unit_corner(s.pos, ix, iy, iz, depth), pow2i(-depth));
                if (error != VV_OK) {
                    vis.fail(error);
                    alive = false;
                } else if (is_const && constant_empty(node.y)) {
                    step_over_constant(p, k, s, depth, t);
                    vis.template segment_end<true>(p, s);
                    // restart from the root (:688-720); the node pointer keeps its value
                    alive = !(s.dst.w > k.astop) && inside_box(s.pos, k.vmin, k.vmax);
                } else if (!V::kEverySample && !is_const && p.cell_mask && !(s.dst.w > k.astop)) {
                    const uint32_t bw = brick_pointer(p, path, wr, brick_depth, brick_idx);
                    if (V::kRecords) vis.begin_record(s);
                    pending = !step_over_brick(p, k, s, unit_corner(s.pos, ix, iy, iz, brick_depth), bw, brick_depth, t);
                    if (!pending) {
                        if (V::kRecords) vis.end_record(s, 0, bw, brick_depth);
                        vis.template segment_end<true>(p, s);
                        alive = inside_box(s.pos, k.vmin, k.vmax);
                    }
                } else {
                    pending = true;
                }
            }
        }
        const unsigned bricks = __ballot_sync(kAll, pending && !is_const);
        if (!__any_sync(kAll, pending)) break;
        if (pending) {
            bool go;
            if (V::kRecords) vis.begin_record(s);
            if (is_const) {
                go = march_constant(p, k, s, vis, node.y, depth, t);
                if (V::kRecords) vis.end_record(s, 1, node.y, depth);
            } else {
                // the position relative to the brick's node, the fractional part of its scaled position
                const F3 lo = unit_corner(s.pos, wr.ix, wr.iy, wr.iz, brick_depth);
                const uint32_t bw = brick_pointer(p, path, wr, brick_depth, brick_idx);
                BrickMarch b;
                b.set<false>(p, k, s, bw, muls(sub(s.pos, lo), pow2i(brick_depth)), brick_depth, t);
                go = march_brick_warp<FMT, V, AHEAD, LIT, STAGED>(p, k, s, vis, b, bricks, path.stage);
                if (V::kRecords) vis.end_record(s, 0, bw, brick_depth);
            }
            if (go) vis.template segment_end<true>(p, s);
            alive = go && !(s.dst.w > k.astop && (is_const || loaded)) && inside_box(s.pos, k.vmin, k.vmax);
            pending = false;
        }
    }
}

// walk() runs a ray's segments until its walk has ended; all 32 lanes of a warp
// call it, `alive` the ones that have a ray.  UNIT: the volume box is [0,1]^3
// (unit_walk), as compute_uniforms makes it; each pixel body keeps the other
// boxes in a function of its own, out of line, so that they cost the unit box
// neither registers nor instruction cache.
template <int FMT, bool COUNT, class V, bool UNIT, int AHEAD, bool LIT = false, bool STAGED = false>
__device__ __forceinline__ void walk(const RaycastParams& p, const WalkConsts& k, RayState& s, V& vis,
                                     const PathSlots& path, bool alive) {
    if (UNIT) {
        walk_warp<FMT, V, AHEAD, LIT, STAGED>(p, k, s, vis, path, alive, NoRefill{});
    } else if (alive) {
        while (walk_segment_box<FMT, COUNT, V, LIT>(p, k, s, vis)) {
        }
    }
}

// Visitor of the forward draw: AddToNodeUsageList (:454-488) for the leaf
// segments whose traversal index falls in this pixel's window (:663-671).
// Entries go straight to the pixel's 12 usage words in memory (zeroed
// before the walk), which keeps 12 registers free during the walk.
struct UsageVisitor {
    static constexpr int kGather = 8;
    static constexpr bool kRecords = false;  // (hooks of the adjoint's records)
    __device__ __forceinline__ void begin_record(const RayState&) {}
    __device__ __forceinline__ void end_record(const RayState&, int, uint32_t, int) {}
    __device__ __forceinline__ void box_segment(const RayState&) {}
    static constexpr bool kEverySample = false;  // samples of empty cells change nothing it records
    uint32_t* out;  // this pixel's usage words, or nullptr
    int list_slot, nl_count, pushed, start_push, max_push;
    int* status;
    __device__ __forceinline__ bool segment_begin(const RayState&) { return true; }
    __device__ __forceinline__ bool sample(int, const float4&, F3, float, int) { return true; }
    template <bool UNIT>
    __device__ __forceinline__ void segment_end(const RaycastParams& p, const RayState& s) {
        if (nl_count >= start_push && nl_count < start_push + 12 && pushed < max_push) {
            ++pushed;
            uint32_t x, y, z;
            if (UNIT) node_position(p, s.nptr, x, y, z);
            else x = s.nptr >> 20, y = (s.nptr >> 10) & 0x3FFu, z = s.nptr & 0x3FFu;
            const uint32_t bits = ((x + 1u) << 20) | ((y + 1u) << 10) | (z + 1u);
            if (out) out[list_slot] = bits;
            list_slot = list_slot == 11 ? 0 : list_slot + 1;
        }
        if (++nl_count >= 48) nl_count = 0;
    }
    __device__ __forceinline__ void fail(int code) { set_status(status, code); }
};

// The set-up of pixel (px,py)'s draw: its usage-list record zeroed and the
// visitor pointed at it, dst cleared, and the fragment's ray started; false
// when the pixel has no fragment or its ray starts outside the volume (its
// walk is then empty).
__device__ __forceinline__ bool start_pixel(const RaycastParams& p, const WalkConsts& k, int px, int py,
                                            RayState& s, UsageVisitor& vis) {
    const vv_uniforms& u = p.u;
    const size_t pix = (size_t)py * u.width + px;
    vis.out = nullptr;
    if (p.usage) {
        uint4* o = p.usage + pix * 3;
        o[0] = o[1] = o[2] = make_uint4(0u, 0u, 0u, 0u);
        vis.out = reinterpret_cast<uint32_t*>(o);
    }
    vis.list_slot = 0;
    vis.nl_count = 0;
    vis.pushed = 0;
    vis.start_push = (px % 2) * 12 + (py % 2) * 24;
    vis.max_push = u.max_nodes_to_push;
    vis.status = p.status;
    s.dst = make_float4(0.f, 0.f, 0.f, 0.f);
    F3 pos;
    return ray_origin(u, k, px, py, pos) && ray_start(p, k, px, py, pos, s);
}

// FragColor of pixel `pix` (:751): float4, or RGBA8 unorm.
__device__ __forceinline__ void finish_pixel(const RaycastParams& p, size_t pix, const RayState& s) {
    if (p.color) {
        if (p.color8) ((uint32_t*)p.color)[pix] = pack_unorm8(s.dst);
        else p.color[pix] = s.dst;
    }
}

// One pixel of the forward draw: the fragment's ray walk, FragColor and the
// three RGBA32UI usage-list layers (:490-751).  All lanes of a warp call it;
// pixels outside the frame do nothing.
template <int FMT, bool COUNT, bool UNIT, int AHEAD, bool LIT, bool STAGED>
__device__ __forceinline__ void pixel_body(const RaycastParams& p, int px, int py, const PathSlots& path) {
    const bool inside = px < p.u.width && py < p.u.height;
    bool ok = true;
    const WalkConsts k = walk_consts(p, UNIT ? __ldg(p.walk) : fetch_node<COUNT>(p, 0, 0, 0, ok));
    UsageVisitor vis;
    RayState s;
    const bool alive = inside && start_pixel(p, k, px, py, s, vis);
    walk<FMT, COUNT, UsageVisitor, UNIT, AHEAD, LIT, STAGED>(p, k, s, vis, path, alive);
    if (inside) finish_pixel(p, (size_t)py * p.u.width + px, s);
}
template <int FMT, bool LIT>
__device__ __noinline__ void pixel_body_box(const RaycastParams& p, int px, int py) {
    pixel_body<FMT, false, false, 1, LIT, false>(p, px, py, PathSlots{nullptr, 0, nullptr});
}
template <int FMT, bool COUNT, int AHEAD, bool LIT = false, bool STAGED = false>
__device__ __forceinline__ void render_pixel(const RaycastParams& p, int px, int py, const PathSlots& path) {
    if (COUNT) pixel_body<FMT, true, false, 1, LIT, false>(p, px, py, path);
    else if (unit_walk(p)) pixel_body<FMT, false, true, AHEAD, LIT, STAGED>(p, px, py, path);
    else pixel_body_box<FMT, LIT>(p, px, py);
}

// The pixel of a thread of a 128-thread CTA whose warps take RAYS pixels each
// (warp_tile_w x warp_tile_h; lanes past them get a pixel outside any frame).
//
// A launch with few rays leaves most schedulers without a warp while one warp
// serves the different paths of 32 rays; its time is that of its slowest warp.
// With fewer rays a warp each path is shorter and the machine fuller (ray cast
// alone, us, 96x64 of the 128^3 / 256^3 / 1024^3 terrain: 132 / 190 / 212 with
// 32 rays, 113 / 124 / 188 with 16, 101 / 120 / 179 with 8, 91 / 105 / 140 with
// 4; 160x120: 117 / 205 / 312, 115 / 154 / 252, 109 / 152 / 230, 106 / 135 /
// 199; 256x192: 140 / 202 / 298, 124 / 169 / 263, 140 / 212 / 273, 155 / 220 /
// 260; 384x288: 156 / 232 / 308, 149 / 195 / 306, 189 / 278 / 335; 512x512:
// 174 / 292 / 336, 213 / 292 / 346), until the warps are more than the
// machine holds: the lines of rays_per_warp.  Other draws and the adjoint have
// the first line in the same place (4 / 16 / 32 rays, lit 192x128 205 / 210 /
// 257, 256x192 281 / 208 / 259; DXT5 228 / 230 / 282, 334 / 240 / 288; FP32 154 /
// 171 / 203, 200 / 169 / 204; forward and adjoint of 160x120 544 / 535 / 572, of
// two 128x128 833 / 688 / 666), the second lower: 384x288 lit 506 / 272 / 257,
// DXT5 605 / 337 / 304, forward and adjoint 1604 / 1171 / 1069, up to a tenth
// under the one line that all of them share.
__host__ __device__ constexpr int warp_tile_w(int rays) { return rays == 32 ? 8 : rays == 16 ? 4 : 2; }
__host__ __device__ constexpr int warp_tile_h(int rays) { return rays == 32 ? 4 : rays == 16 ? 4 : 2; }
inline int rays_per_warp(long long rays) { return rays <= 24576 ? 4 : rays <= 114688 ? 16 : 32; }
template <int RAYS>
__device__ __forceinline__ void warp_pixel(int& px, int& py) {
    constexpr int w = warp_tile_w(RAYS), h = warp_tile_h(RAYS);
    const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
    px = blockIdx.x * (2 * w) + (warp & 1) * w + lane % w;
    py = blockIdx.y * (2 * h) + (warp >> 1) * h + lane / w;
    if (RAYS < 32 && lane >= RAYS) px = 1 << 24;
}
inline dim3 warp_grid(int rays, int width, int height, int views = 1) {
    const int w = 2 * warp_tile_w(rays), h = 2 * warp_tile_h(rays);
    return dim3((unsigned)((width + w - 1) / w), (unsigned)((height + h - 1) / h), (unsigned)views);
}

// Persistent ray cast that keeps the lanes of a warp busy: each warp takes
// 8x4 pixel tiles from a device counter and walks their rays (walk_warp); a
// lane whose ray has ended takes the next pixel of the warp's tile (ballot +
// popc rank) before the next descent, instead of idling until the warp's
// slowest ray ends.  Same pixels, same walk, same results as render_pixel;
// volumes in the unit box.
struct TileRefill {
    static constexpr bool kOn = true;
    const RaycastParams& p;
    const WalkConsts& k;
    unsigned int* counter;
    int tiles_x, tiles;
    int tile, taken;  // the warp's tile and how many of its pixels are handed out
    bool more;        // tiles left
    bool has;         // the lane holds pixel `pix`
    size_t pix;
    __device__ __forceinline__ TileRefill(const RaycastParams& p_, const WalkConsts& k_, unsigned int* counter_)
        : p(p_), k(k_), counter(counter_), tile(0), taken(32), more(true), has(false), pix(0) {
        tiles_x = (p.u.width + 7) >> 3;
        tiles = tiles_x * ((p.u.height + 3) >> 2);
    }
    // All lanes of the warp; busy: the lane's ray goes on.  A lane that is not
    // finishes its pixel and takes the next one; alive: it has a ray.
    __device__ __forceinline__ void take(RayState& s, UsageVisitor& vis, WalkResume& wr, bool busy, bool& alive) {
        const unsigned lane = threadIdx.x & 31u;
        if (!busy && has) {
            finish_pixel(p, pix, s);
            has = false;
        }
        unsigned idle = __ballot_sync(0xFFFFFFFFu, !busy);
        while (idle && more) {
            if (taken == 32) {
                unsigned t = 0u;
                if (lane == 0u) t = atomicAdd(counter, 1u);
                tile = (int)__shfl_sync(0xFFFFFFFFu, t, 0);
                taken = 0;
                if (tile >= tiles) {
                    more = false;
                    break;
                }
            }
            const int n = min(__popc(idle), 32 - taken);
            const int rank = __popc(idle & ((1u << lane) - 1u));
            if (!busy && rank < n) {
                const int q = taken + rank;
                const int px = (tile % tiles_x) * 8 + (q & 7), py = (tile / tiles_x) * 4 + (q >> 3);
                if (px < p.u.width && py < p.u.height) {
                    pix = (size_t)py * p.u.width + px;
                    wr = WalkResume{};
                    alive = busy = has = start_pixel(p, k, px, py, s, vis);
                    if (!has) finish_pixel(p, pix, s);
                }
            }
            taken += n;
            idle = __ballot_sync(0xFFFFFFFFu, !busy);
        }
    }
};
template <int FMT>
__device__ __forceinline__ void render_refill(const RaycastParams& p, unsigned int* counter, const PathSlots& path) {
    const WalkConsts k = walk_consts(p, __ldg(p.walk));
    RayState s;
    UsageVisitor vis;
    TileRefill refill(p, k, counter);
    walk_warp<FMT, UsageVisitor, 1, false, false>(p, k, s, vis, path, false, refill);
}

}  // namespace rc
}  // namespace vv
