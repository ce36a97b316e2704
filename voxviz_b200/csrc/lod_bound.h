// lod_bound.h - a certificate that the descent's LOD test continues.
//
// The descent of GigaVoxelsNoLighting.frag (:563-622) stops at a node when
// PixelSize > ComputeVoxelSize (:429-441) * LodScalar, evaluated here in
// binary32 as
//     uh = up*vh, lh = left*vh                     (vh = rvh * 2^-level)
//     ll = normalize(pos - uh + lh - C), ur = normalize(pos + uh - lh - C)
//     stop iff pixel_size > (1 - dot(ll, ur)) * lod
// with normalize(v) = v * (1/sqrt(dot(v,v))), no contraction.
//
// lod_bound_clears() shows, for a ray position, that this test is FALSE
// (the descent continues) at every level j in [j0, m], without evaluating
// it.  With a = pos - C, d = vh*(up - left) (exact: vh is a power of two),
// the test measures R = 1 - cos(theta), theta the angle between a - d and
// a + d, and
//     R >= sin^2(theta)/2 >= 2 vh^2 |a x w|^2 / (|a|^2 + vh^2 |w|^2)^2 = Rlow
// (w = up - left).  For levels with vh |w| <= |a|/4 the binary32 sequence
// returns at least lod * (R - theta * Dmax - 11.2 u)(1 - u) (u = 2^-24):
// Dmax bounds the angle error of its two directions (rounding of
// pos - uh + lh - C per component <= u (2 max|pos| + max|a| + 5 vh) with
// pos in the unit box, plus 1.8 u from normalising) and 11.2 u the length
// and dot-product rounding.  Rlow is evaluated with approximate reciprocal
// square root and division (<= 2 ulp each on the device; exact on the
// host); the (1 - 1e-4) factors cover that.  If the bound clears
// pixel_size at level m and theta >= 5 Dmax there, it clears it at every
// shallower level down to j0, the first level with vh |w| <= |a|/4, since
// R grows faster with theta than theta * Dmax.
//
// Shared by the kernels and by the host check in tests/ (which compares it
// with the exact binary32 sequence on random and adversarial inputs).
#pragma once

#include <stdint.h>

#include <cmath>
#include <cstring>

#ifdef __CUDACC__
#define VV_HD __host__ __device__ __forceinline__
#else
#define VV_HD inline
#endif

namespace vv {
namespace lodb {

struct V3 {
    float x, y, z;
};

VV_HD V3 sub3(V3 a, V3 b) { return V3{a.x - b.x, a.y - b.y, a.z - b.z}; }
VV_HD float dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
VV_HD V3 cross(V3 a, V3 b) { return V3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }

VV_HD float fast_rsqrt(float x) {
#ifdef __CUDA_ARCH__
    float r;  // x is a normal number wherever this is used
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / std::sqrt(x);
#endif
}
VV_HD float vabs(float x) { return x < 0.0f ? -x : x; }
VV_HD float vmax(float a, float b) { return a > b ? a : b; }
VV_HD uint32_t float_bits(float f) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(f);
#else
    uint32_t b;
    std::memcpy(&b, &f, 4);
    return b;
#endif
}
// x * 2^e for a normal power-of-two scale (exact); on the device 2^e is built
// from its exponent bits (e in [-126, 127])
VV_HD float scale2(float x, int e) {
#ifdef __CUDA_ARCH__
    return x * __int_as_float((e + 127) << 23);
#else
    return std::ldexp(x, e);
#endif
}

constexpr int kDeepTries = 3;

// Per-frame constants (made once on the host).
struct Consts {
    V3 C, w;          // camera position, w = up - left
    float W;          // |w|^2
    float t0;         // 4 rvh |w| rounded up: t0 / |a| bounds 4 vh |w| / |a| at level 0
    float ra_shallow; // 1/|a| up to which the levels above j0 are shown to continue (see clear_range)
    float d0, d1;     // Dmax <= d0 / |a| + d1
    float theta;      // theta <= theta * vh / |a|
    float need;       // pixel_size / lod and the rounding terms: what R - theta Dmax has to reach
    float guess;      // 0.97 rvh^2 / need
    float rvh;
    int max_level;
    bool ok;
    // deep_levels: the deepest level's half voxel size squared and times theta,
    // the smallest |a|^2 it covers (NaN: none; a far camera's |a|^2 may be infinite)
    float quick_vh2, quick_theta, quick_min;
};

// Every rounding of a bound's own evaluation (a few ulp, approximate
// reciprocal square roots included) is covered by the factors 1.001 on upper
// and 1 - 3e-4 on lower bounds.
VV_HD Consts make_consts(V3 C, V3 up, V3 left, float rvh, float lod, float pixel_size, int max_level, bool unit_box) {
    const float u = 5.9604645e-8f;  // 2^-24
    Consts k;
    k.C = C;
    k.w = sub3(up, left);
    k.W = dot(k.w, k.w);
    const float wn = (k.W > 0.0f ? 1.0f / fast_rsqrt(k.W) : 0.0f) * 1.001f;  // |w| rounded up
    const float cmax = vmax(vabs(C.x), vmax(vabs(C.y), vabs(C.z)));
    k.rvh = rvh;
    k.max_level = max_level;
    k.ok = unit_box && lod > 0.0f && lod < 1e30f && pixel_size < 1e30f && rvh > 0.0f && k.W > 0.5f && k.W < 8.0f &&
           cmax < 1e6f;
    k.t0 = 4.0f * rvh * wn * 1.001f;
    // rounding of pos -+ uh +- lh - C per component with vh |w| <= |a|/4:
    // u (2 max|pos| + max|a| + 5 vh + 2 cmax), max|a| <= |a|, 5 vh <= 1.25 |a| / |w|;
    // e0 + e1 |a| bounds its norm
    const float e0 = 1.7321f * u * (2.0f + 2.0f * cmax) * 1.02f;
    const float e1 = 1.7321f * u * (1.0f + 1.25f * 1.003f / wn) * 1.02f;
    k.d0 = 2.0f * 1.34f * e0 * 1.02f;
    k.d1 = 2.0f * (1.34f * e1 + 1.8f * u) * 1.02f;
    k.theta = 2.7f * wn * 1.001f;
    const float px = pixel_size / lod;
    k.need = px * (1.0f + 2e-4f) + 11.3f * u;
    k.guess = k.need > 1e-30f ? 0.97f * rvh * rvh / k.need : 1e30f * rvh * rvh;
    // levels above j0 (vh <= rvh there): a direction is off by at most
    // 1.01 sqrt(3) eps / (0.316 |a|) + 1.8 u, eps = u (3 + 8 rvh + |a| + 2 cmax);
    // both together move 1 - cos, which is over 0.0051, by s0 / |a| + s1
    const float s0 = 2.0f * 1.01f * 1.7321f / 0.316f * u * (3.0f + 8.0f * rvh + 2.0f * cmax) * 1.02f;
    const float s1 = 2.0f * (1.01f * 1.7321f / 0.316f * u + 1.8f * u) * 1.02f;
    const float room = 0.0051f - s1 - 13.2f * u - px * (1.0f + 2e-4f);
    k.ra_shallow = room > 0.0f ? room / s0 * (1.0f - 1e-3f) : 0.0f;
    // deep_levels: the deepest level's half voxel size vh, and |a| at least
    // 16 vh' |w| for the size vh' of the highest level tried, so that
    // vh'^2 |w|^2 / |a|^2 <= 1/256 (and vh' |w| <= |a|/4), and either no level
    // above j0 or those shown; theta >= 5 Dmax from R >= need
    const float vh = scale2(rvh, -max_level);
    k.quick_vh2 = 2.0f * vh * vh * (1.0f - 2.0f / 256.0f) * (1.0f - 6e-4f);
    k.quick_theta = 1.001f * k.theta * vh;
    float amin = 16.0f * vh * (float)(1 << (kDeepTries - 1)) * wn;
    if (amin < k.t0) {
        const float shallow = k.ra_shallow > 0.0f ? 1.001f / k.ra_shallow : 1e18f;
        if (amin < shallow) amin = shallow < k.t0 ? shallow : k.t0;
    }
    const float dm = k.d0 / (amin > 1e-6f ? amin : 1e-6f) + k.d1;
    k.quick_min = k.ok && max_level >= kDeepTries && max_level < 60 && amin > 1e-6f && k.need >= 12.6f * dm * dm
                      ? amin * amin * 1.001f : NAN;
    return k;
}

// The deepest level of the last kDeepTries up to which the LOD test surely
// continues from level 0 on, or -1: clear_range's bound, with |a| bounded by
// (1 + |a|^2) / 2 in place of its square root (no reciprocals).
VV_HD int deep_levels(const Consts& k, V3 pos) {
    const V3 a = sub3(pos, k.C);
    const float A = dot(a, a);
    const float aw = dot(a, k.w), AW = A * k.W;
    const float S = AW - aw * aw;
    if (!(A >= k.quick_min && S >= 0.1002f * AW)) return -1;
    const float base = 1.0005f * k.need * A * A;
    float r = k.quick_vh2 * S, d = 1.0005f * A * k.quick_theta * (k.d0 + k.d1 * (0.5f + 0.5f * A));
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int i = 0; i < kDeepTries; ++i) {
        if (r >= base + d) return k.max_level - i;
        r = r * 4.0f;  // the next level up: vh doubled
        d = d * 2.0f;
    }
    return -1;
}

// Levels [lo, hi] at which the LOD test surely continues for position pos
// (inside the unit box); lo > hi when nothing is shown.  The deepest level is
// picked from R ~ G vh^2 with 3 % to spare and, when its own bound falls
// short (near the camera), the one above it.
VV_HD void clear_range(const Consts& k, V3 pos, int& lo, int& hi) {
    lo = 1;
    hi = 0;
    if (!k.ok) return;
    const V3 a = sub3(pos, k.C);
    const float A = dot(a, a);
    // |a x w|^2 = |a|^2 |w|^2 - (a.w)^2; with sin(angle(a, w)) >= 0.316 its
    // cancellation leaves it within 1e-5
    const float aw = dot(a, k.w), AW = A * k.W;
    const float S = AW - aw * aw;
    if (!(A > 1e-12f) || !(S >= 0.1002f * AW)) return;
    const float ra = fast_rsqrt(A);
    const float invA = ra * ra;
    // j0: the smallest j with 2^j >= t >= 4 rvh |w| / |a|
    const float t = k.t0 * ra;
    int j0 = 0;
    if (t > 1.0f) {
        const uint32_t b = float_bits(t);
        j0 = (int)((b >> 23) & 255u) - 126;  // t < 2^j0
    }
    // Levels below j0 (vh |w| > |a|/4): sin(theta) = 2|a||d| sin(phi) /
    // (|a - d||a + d|) >= 2 * 0.25 * 0.316 / 1.25^2 at vh |w| = |a|/4 and theta
    // grows with vh, so R >= 1 - cos(0.101) > 0.0051, and |a -+ d| >= |a| sin(phi).
    const bool shallow = j0 == 0 || ra <= k.ra_shallow;
    if (shallow) {  // whatever the deeper levels give, [0, j0) is shown
        lo = 0;
        hi = j0 - 1;
    }
    const float G = 2.0f * S * invA * invA;  // R ~ G vh^2
    const float q = G * k.guess;
    if (!(q >= 1.0f)) return;
    int m = ((int)((float_bits(q) >> 23) & 255u) - 127) >> 1;  // floor(log2(q) / 2)
    m = m < k.max_level ? m : k.max_level;
    const float dmax = k.d0 * ra + k.d1;
    const float tm = k.theta * ra;
    for (int tries = 0; tries < 2 && m >= j0; ++tries, --m) {
        const float vh = scale2(k.rvh, -m);
        const float vh2 = vh * vh;
        // 2 vh^2 S / (A + vh^2 W)^2 >= G vh^2 (1 - 2 vh^2 W / A)
        const float Rlow = G * vh2 * (1.0f - 2.0f * vh2 * k.W * invA) * (1.0f - 3e-4f);
        // theta >= sqrt(2 R) >= 5 Dmax, and the bound itself
        if (2.0f * Rlow >= 25.1f * dmax * dmax && Rlow - tm * vh * dmax * 1.001f >= k.need) {
            lo = shallow ? 0 : j0;
            hi = m;
            return;
        }
    }
}

}  // namespace lodb
}  // namespace vv
