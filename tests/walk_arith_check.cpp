// Host checks of the arithmetic that the unit-box walk takes in place of the
// shader's own: markstein_div (fixed_div.h) against IEEE division, block_div
// and walk_link (walknode.h) against their definitions, and
// lodb::deep_levels (lod_bound.h) against the exact binary32 LOD test, and the
// one-texel DXT5 decode (dxt.h) against the block's.
// Prints "<checks> <mismatches>" per part; built and run by
// tests/test_walk_arith.py.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

#include "../voxviz_b200/csrc/dxt.h"
#include "../voxviz_b200/csrc/fixed_div.h"
#include "../voxviz_b200/csrc/lod_bound.h"
#include "../voxviz_b200/csrc/walknode.h"

using vv::lodb::V3;

static float from_bits(uint32_t b) {
    float f;
    std::memcpy(&f, &b, 4);
    return f;
}
static V3 add(V3 a, V3 b) { return V3{a.x + b.x, a.y + b.y, a.z + b.z}; }
static V3 sub(V3 a, V3 b) { return V3{a.x - b.x, a.y - b.y, a.z - b.z}; }
static V3 muls(V3 a, float s) { return V3{a.x * s, a.y * s, a.z * s}; }
static float dot3(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
static V3 normalize3(V3 v) { return muls(v, 1.0f / std::sqrt(dot3(v, v))); }
static V3 cross3(V3 a, V3 b) { return V3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
static float exact_proj(V3 pos, V3 C, V3 up, V3 left, float vh, float lod) {
    const V3 uh = muls(up, vh), lh = muls(left, vh);
    const V3 ll = normalize3(sub(add(sub(pos, uh), lh), C)), ur = normalize3(sub(sub(add(pos, uh), lh), C));
    return (1.0f - dot3(ll, ur)) * lod;
}

int main() {
    std::mt19937_64 rng(11);
    std::uniform_real_distribution<float> U(0.f, 1.f);
    long checks = 0, bad = 0, total_bad = 0;
    // divisors: every significand in steps and random ones, exponents from 2^-60 up to 1
    for (long i = 0; i < 20000000; ++i) {
        const uint32_t mb = (i & 1) ? (uint32_t)(rng() & 0x7FFFFFu) : (uint32_t)((i * 2654435761u) & 0x7FFFFFu);
        const float b = std::ldexp(from_bits(0x3F800000u | mb), -(int)(rng() % 61));
        // exit distances, and the all-ones and power-of-two significands
        uint32_t ma = (uint32_t)(rng() & 0x7FFFFFu);
        if (i % 17 == 0) ma = 0x7FFFFFu;
        if (i % 19 == 0) ma = 0u;
        const float a = std::ldexp(from_bits(0x3F800000u | ma), -(int)(rng() % 59));
        const float y = 1.0f / b, q = vv::markstein_div(a, b, y), e = a / b;
        ++checks;
        if (std::memcmp(&q, &e, 4) != 0) ++bad;
    }
    std::printf("%ld %ld\n", checks, bad);
    total_bad += bad;
    checks = bad = 0;
    for (uint32_t d = 1; d < (1u << 18) + 1; d = d < 600 ? d + 1 : d * 9 / 8 + 1) {
        const vv::BlockDiv b = vv::make_block_div(d);
        for (int t = 0; t < 2000; ++t) {
            const uint32_t n = (uint32_t)(rng() & 0x7FFFFFFu), m = n / d * d;
            for (uint32_t v : {n, m, m + d - 1, m ? m - 1 : 0u, 0x7FFFFFFu}) {
                if (v > 0x7FFFFFFu) continue;
                ++checks;
                if (vv::block_div(v, b) != v / d) ++bad;
            }
        }
    }
    for (int t = 0; t < 2000000; ++t) {
        const int dx = 2 + 2 * (int)(rng() % 512), dy = 2 + 2 * (int)(rng() % 512), dz = 2 + 2 * (int)(rng() % 512);
        const uint32_t w = (uint32_t)rng() & ((t & 3) ? 0xFFFFFFFFu : 0xC7F1FC7Fu), r = vv::walk_link(w, dx, dy, dz);
        const uint32_t x = (w >> 20) & 1023u, y = (w >> 10) & 1023u, z = w & 1023u, link = r & vv::kLinkMask;
        bool ok = (r >> 30) == (w >> 30);
        if (!(x | y | z)) ok = ok && link == 0;
        else if ((x | y | z) & 1u) ok = ok && link == vv::kLinkOdd;
        else if ((int)x >= dx || (int)y >= dy || (int)z >= dz) ok = ok && link == vv::kLinkBad;
        else {
            const uint32_t blk = ((z >> 1) * (uint32_t)(dy / 2) + (y >> 1)) * (uint32_t)(dx / 2) + (x >> 1);
            ok = ok && link != 0 && (link == blk || (blk >= vv::kLinkOdd && link == vv::kLinkOdd));
        }
        ++checks;
        if (!ok) ++bad;
    }
    std::printf("%ld %ld\n", checks, bad);
    total_bad += bad;
    checks = bad = 0;
    const float rvh = 1.0f / 16.0f;
    for (long it = 0; it < 1500000; ++it) {
        const V3 C{U(rng) * 3.f - 1.f, U(rng) * 3.f - 1.f, U(rng) * 1.6f - 0.2f}, pos{U(rng), U(rng), U(rng)};
        V3 look = sub(pos, C);
        const float ln = std::sqrt(dot3(look, look));
        if (ln < 1e-4f) continue;
        look = normalize3(add(muls(look, 1.0f / ln), muls(V3{U(rng) - 0.5f, U(rng) - 0.5f, U(rng) - 0.5f}, 0.8f)));
        V3 left = cross3(V3{0.f, 0.f, 1.f}, look);
        if (dot3(left, left) < 1e-6f) continue;
        left = normalize3(left);
        const V3 up = normalize3(cross3(look, left));
        const int L = 3 + (int)(U(rng) * 8);
        const float lod = U(rng) < 0.8f ? 1.0f : 0.25f + 2.f * U(rng);
        // pixel sizes: any, one ulp above a deep level's projection (it stops there), below it
        const float proj = exact_proj(pos, C, up, left, std::ldexp(rvh, -(L - (int)(it / 3 % 4))), lod);
        const float pix = it % 3 == 0 ? std::pow(10.f, -8.5f + 4.f * U(rng))
                          : it % 3 == 1 ? std::nextafter(proj, 1e30f) : proj * (0.8f + 0.2f * U(rng));
        const vv::lodb::Consts k = vv::lodb::make_consts(C, up, left, rvh, lod, pix, L, true);
        const int hi = vv::lodb::deep_levels(k, pos);
        if (hi < 0) continue;
        ++checks;
        for (int l = 0; l <= hi; ++l)
            if (pix > exact_proj(pos, C, up, left, std::ldexp(rvh, -l), lod)) {
                ++bad;
                break;
            }
    }
    std::printf("%ld %ld\n", checks, bad);
    total_bad += bad;
    checks = bad = 0;
    for (uint32_t e = 0; e < 65536u * 8u; ++e) {  // every pair of alpha endpoints and code, colours along
        const uint32_t a = e & 65535u, code = e >> 16;
        uint64_t codes = 0;
        for (int t = 0; t < 16; ++t) codes |= (uint64_t)((code + t) & 7u) << (3 * t);
        const uint32_t w[4] = {a | (uint32_t)(codes << 16), (uint32_t)(codes >> 16), (uint32_t)rng(), (uint32_t)rng()};
        for (int t = 0; t < 16; ++t, ++checks)
            if (vv::dxt::texel_dxt5(w[0], w[1], w[2], w[3], t) != vv::dxt::decode_dxt5(w, t)) ++bad;
    }
    for (uint32_t e = 0; e < (1u << 22); ++e, ++checks) {  // colour endpoints
        const uint32_t w[4] = {(uint32_t)rng(), (uint32_t)rng(), (uint32_t)rng(), (uint32_t)rng()};
        const int t = (int)(e & 15u);
        if (vv::dxt::texel_dxt5(w[0], w[1], w[2], w[3], t) != vv::dxt::decode_dxt5(w, t)) ++bad;
    }
    std::printf("%ld %ld\n", checks, bad);
    total_bad += bad;
    return total_bad ? 1 : 0;
}
