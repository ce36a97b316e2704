// adjoint.cu - differentiable ray cast: checkpointing forward and adjoint.
//
// The forward composites  dst_{k+1} = dst_k + T_k * src_k,  T_k = 1 - dst_k.a
// (GigaVoxelsNoLighting.frag:280,354).  Its adjoint with g = dL/d dst is
//   dL/d src_k = g_{k+1} * T_k
//   g_k.rgb    = g_{k+1}.rgb,   g_k.a = g_{k+1}.a - dot(g_{k+1}, src_k)
// and a brick sample is the trilinear blend of 8 texels, so each texel gets
// its blend weight times dL/d src_k.  Walking the samples backwards needs
// T_k, which is not recoverable from the final colour once a sample is
// opaque, so the forward keeps a record of each leaf segment that took
// samples: where the ray was and what it had composited (alpha alone: the
// colour so far enters nothing), which brick or constant, and how many
// samples.  The adjoint goes through a ray's records from the last to the
// first, takes a segment's samples again (in pieces of at most 64, the last
// piece first), keeps the piece in local memory and back-propagates through it
// in reverse: no descent is repeated.  The last quarter of a ray's records, and
// all of them where the unit box's walk is not taken, are points to walk from
// instead (one whenever 32 or more samples were composited since the last), for
// rays that cross more segments than there are records.  The control flow (descent, step counts, early
// termination) is that of the forward and is held fixed, as any reverse-mode
// derivative of this shader does.
#include "ckpt_layout.h"
#include "raycast_common.cuh"

namespace vv {

using namespace rc;

namespace {

// The views of a launch: views of one size over the same pools.
constexpr int kMaxDiffViews = 16;  // 480 bytes each of the launch parameters
template <int VIEWS>
struct DiffViews {
    RaycastParams p[VIEWS];
};

constexpr int kCkptEvery = 32;
constexpr int kPiece = 64;

// A record, 24 bytes: the ray's position at the start of the segment and its
// dst.a there; a brick's pointer or a constant's word, and samples | depth <<
// 16 | kind << 24 (a walk record: the index of its first sample, and its kind).
struct Ckpt {
    float2 p0, p1;
    uint2 w;
};
static_assert(sizeof(Ckpt) == kRecordBytes && alignof(Ckpt) == 8, "records are 24 bytes of 8-byte vectors");
enum { kRecBrick = 0, kRecConst = 1, kRecWalk = 2 };

struct CkptVisitor {
    static constexpr int kGather = 8;
    static constexpr bool kEverySample = false;
    static constexpr bool kRecords = true;
    Ckpt* out;
    int cap, count, last;
    int segments;  // records of segments there may be; then walk records
    int* status;
    __device__ __forceinline__ void start(Ckpt* out_, int per_ray, int* status_) {
        out = out_;
        cap = record_cap(per_ray);
        count = 0;
        last = -kCkptEvery;
        segments = cap - max(1, cap / 4);
        status = status_;
    }
    __device__ __forceinline__ void put(const RayState& s, uint32_t w0, uint32_t w1) {
        Ckpt c;
        c.p0 = make_float2(s.pos.x, s.pos.y);
        c.p1 = make_float2(s.pos.z, s.dst.w);
        c.w = make_uint2(w0, w1);
        out[count] = c;
    }
    // (also the box walk's records)
    __device__ __forceinline__ void box_segment(const RayState& s) {
        if (s.nsamples - last >= kCkptEvery && count < cap) {
            put(s, (uint32_t)s.nsamples, (uint32_t)kRecWalk << 24);
            ++count;
            last = s.nsamples;
        }
    }
    __device__ __forceinline__ bool segment_begin(const RayState&) { return true; }
    // Before and after a segment that may take samples.
    __device__ __forceinline__ void begin_record(const RayState& s) {
        if (count < segments) {
            put(s, 0u, 0u);
            last = s.nsamples;
        } else {
            if (segments >= 0) {  // the first walk record
                segments = -1;
                last = s.nsamples - kCkptEvery;
            }
            box_segment(s);
        }
    }
    __device__ __forceinline__ void end_record(const RayState& s, int kind, uint32_t word, int depth) {
        const int n = s.nsamples - last;
        if (count >= segments || n <= 0) return;
        if (n > 0xFFFF || depth > 0xFF) {  // does not fit: walked from here on
            out[count++].w = make_uint2((uint32_t)last, (uint32_t)kRecWalk << 24);
            segments = -1;
        } else {
            out[count++].w = make_uint2(word, (uint32_t)n | ((uint32_t)depth << 16) | ((uint32_t)kind << 24));
        }
    }
    __device__ __forceinline__ bool sample(int, const float4&, F3, float, int) { return true; }
    template <bool UNIT>
    __device__ __forceinline__ void segment_end(const RaycastParams&, const RayState&) {}
    __device__ __forceinline__ void fail(int code) { set_status(status, code); }
};

// The samples of one piece, compactly: T (the transmittance before the
// sample, negated for a constant-node sample: T > 0 or +0 for brick samples),
// the sample's alpha, r = dot(dL/dc.rgb, src.rgb) (dL/dc.rgb is constant
// along the ray) and the brick position.  24 bytes a sample.
struct Piece {
    float T[kPiece];
    float a[kPiece];
    float r[kPiece];
    F3 bpos[kPiece];
    __device__ __forceinline__ void put(int i, int kind, const float4& v, F3 b, float t, float4 g) {
        T[i] = kind == kSampleBrick ? t : -t;
        a[i] = v.w;
        // the first three products of the g.a update, in its order
        r[i] = g.x * v.x + g.y * v.y + g.z * v.z;
        bpos[i] = b;
    }
};
// A walk from a point, for the samples [first, last) of the ray.
struct ReplayVisitor {
    static constexpr int kGather = 32;
    static constexpr bool kEverySample = true;  // the gradient scatters empty samples too
    static constexpr bool kRecords = false;
    Piece* piece;
    int first, last, n;
    float4 g;  // dL/dc
    __device__ __forceinline__ bool segment_begin(const RayState& s) { return s.nsamples < last; }
    __device__ __forceinline__ bool sample(int kind, const float4& v, F3 b, float t, int index) {
        if (index >= first && n < kPiece) piece->put(n++, kind, v, b, t, g);
        return index + 1 < last;
    }
    template <bool UNIT>
    __device__ __forceinline__ void segment_end(const RaycastParams&, const RayState&) {}
    __device__ __forceinline__ void fail(int) {}
    __device__ __forceinline__ void begin_record(const RayState&) {}
    __device__ __forceinline__ void end_record(const RayState&, int, uint32_t, int) {}
    __device__ __forceinline__ void box_segment(const RayState&) {}
};

// The row of the gradient that holds `slot`: the slot itself (dense), or,
// with a slot map, the row claimed by the first sample that reaches the
// slot (-1 in the map: unclaimed; -2: being claimed; -3: no row left).
// The claiming thread never waits, so a waiting thread's bound is never
// reached on valid data; reaching it, or running out of rows, sets the
// device status and drops the contribution.
__device__ __forceinline__ int grad_row(const GradTarget& gt, uint32_t slot, int* status) {
    if (!gt.slot_map) return (int)slot;
    int* m = gt.slot_map + slot;
    int r = *(volatile int*)m;
    if (r >= 0) return r;
    if (r == -1 && atomicCAS(m, -1, -2) == -1) {
        const int nr = atomicAdd(gt.rows_used, 1);
        if (nr >= gt.rows_cap) {
            atomicExch(m, -3);
            set_status(status, VV_ERR_OOM);
            return -1;
        }
        __threadfence();
        atomicExch(m, nr);
        return nr;
    }
    for (int i = 0; i < (1 << 22); ++i) {
        r = *(volatile int*)m;
        if (r >= 0) return r;
        if (r == -3) return -1;
        __nanosleep(64);
    }
    set_status(status, VV_ERR_TIMEOUT);
    return -1;
}

// gradient element i += v (binary32 rows: one vector reduction, red.v4.f32,
// which returns nothing - atomicAdd(float4*) returns the old value and so
// holds four registers until the L2 answers - into the warp's copy of the
// rows; binary64 rows: four double atomics).
template <bool F64>
__device__ __forceinline__ void texel_atomic(const GradTarget& gt, size_t i, float4 v) {
    if (F64) {
        double* g = (double*)gt.grad + 4 * i;
        atomicAdd(g + 0, (double)v.x);
        atomicAdd(g + 1, (double)v.y);
        atomicAdd(g + 2, (double)v.z);
        atomicAdd(g + 3, (double)v.w);
    } else {
        float4* g = (float4*)gt.grad + i;
        // the warp's copy: its index in the CTA, then the CTA's column parity
        const unsigned c = ((threadIdx.x >> 5) | ((blockIdx.x & 1u) << 2)) & (unsigned)(gt.copies - 1);
        if (c) g = gt.spread + (size_t)(c - 1u) * (size_t)gt.spread_rows * 1000u + i;
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(g), "f"(v.x), "f"(v.y), "f"(v.z),
                     "f"(v.w)
                     : "memory");
    }
}

// dL/d texel += w_j * d for the 8 taps of the sample at uvw (the addressing
// of sample_brick, clamps included: clamped taps share a texel).  The slot
// map is read once per slot change: (c_slot, c_row) is the thread's last
// slot and its row.  Taps in one slot (the usual case): WSUM groups the
// lanes whose samples lie in the same cell (one __match_any_sync a sample:
// the same 8 texels) and sums each tap over the group in lane order, lane r
// of n taking the taps r, r + n, ... (it reads each member's weights and
// gradient, 7 shuffles, instead of its 4 products a tap, 32, and the taps of
// a group go out together: backward of six 1080p views 4.1, 2.8, 5.9, 4.0, 5.4
// and 0.95 ms, from 4.8, 3.2, 10.5, 7.5, 7.1 and 1.1); without WSUM each lane starts its 8 taps at a
// different one (fewer lanes of one instruction on one texel).
template <bool F64, bool WSUM>
__device__ __forceinline__ void scatter_texels(const RaycastParams& p, F3 uvw, float4 d, const GradTarget& gt,
                                               uint32_t& c_slot, int& c_row) {
    const float* N = p.u.brick_pool_dimension;
    const Axis ax = axis_taps(uvw.x, N[0], p.slots[0] * 10);
    const Axis ay = axis_taps(uvw.y, N[1], p.slots[1] * 10);
    const Axis az = axis_taps(uvw.z, N[2], p.slots[2] * 10);
    const uint32_t SX = (uint32_t)p.slots[0], SY = (uint32_t)p.slots[1];
    const int lane = (int)(threadIdx.x & 31u);
    if (ax.s0 == ax.s1 && ay.s0 == ay.s1 && az.s0 == az.s1) {
        const uint32_t slot = ((uint32_t)az.s0 * SY + (uint32_t)ay.s0) * SX + (uint32_t)ax.s0;
        if (slot != c_slot) {
            c_row = grad_row(gt, slot, p.status);
            c_slot = slot;
        }
        if (c_row < 0) return;
        const uint32_t t0 = (uint32_t)((az.l0 * 10 + ay.l0) * 10 + ax.l0);
        const uint32_t dx = (uint32_t)(ax.l1 - ax.l0), dy = (uint32_t)(10 * (ay.l1 - ay.l0)),
                       dz = (uint32_t)(100 * (az.l1 - az.l0));
        const size_t base = (size_t)c_row * 1000u + t0;
        if (WSUM) {
            const uint64_t key = ((uint64_t)(uint32_t)c_row << 16) | (t0 << 3) | (dx << 2) | ((dy ? 1u : 0u) << 1) |
                                 (dz ? 1u : 0u);
            const unsigned peers = __match_any_sync(__activemask(), key);
            const int n = __popc(peers), rank = __popc(peers & ((1u << lane) - 1u));
            if (n == 1) {
#pragma unroll
                for (int t = 0; t < 8; ++t) {
                    const int bx = t & 1, by = (t >> 1) & 1, bz = t >> 2;
                    const float w = (bx ? ax.f : 1.0f - ax.f) * (by ? ay.f : 1.0f - ay.f) * (bz ? az.f : 1.0f - az.f);
                    const float4 v = make_float4(w * d.x, w * d.y, w * d.z, w * d.w);
                    if (v.x != 0.f || v.y != 0.f || v.z != 0.f || v.w != 0.f)
                        texel_atomic<F64>(gt, base + (bx ? dx : 0u) + (by ? dy : 0u) + (bz ? dz : 0u), v);
                }
                return;
            }
            for (int t = rank; t - rank < 8; t += n) {
                const int bx = t & 1, by = (t >> 1) & 1, bz = (t >> 2) & 1;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                for (unsigned m = peers; m; m &= m - 1) {
                    const int src = __ffs(m) - 1;
                    const float fx = __shfl_sync(peers, ax.f, src), fy = __shfl_sync(peers, ay.f, src),
                                fz = __shfl_sync(peers, az.f, src);
                    const float w = (bx ? fx : 1.0f - fx) * (by ? fy : 1.0f - fy) * (bz ? fz : 1.0f - fz);
                    v.x += w * __shfl_sync(peers, d.x, src);
                    v.y += w * __shfl_sync(peers, d.y, src);
                    v.z += w * __shfl_sync(peers, d.z, src);
                    v.w += w * __shfl_sync(peers, d.w, src);
                }
                if (t < 8 && (v.x != 0.f || v.y != 0.f || v.z != 0.f || v.w != 0.f))
                    texel_atomic<F64>(gt, base + (bx ? dx : 0u) + (by ? dy : 0u) + (bz ? dz : 0u), v);
            }
        } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int t = (q + lane) & 7;
                const int bx = t & 1, by = (t >> 1) & 1, bz = t >> 2;
                const float w = (bx ? ax.f : 1.0f - ax.f) * (by ? ay.f : 1.0f - ay.f) * (bz ? az.f : 1.0f - az.f);
                if (w == 0.0f) continue;
                texel_atomic<F64>(gt, base + (bx ? dx : 0u) + (by ? dy : 0u) + (bz ? dz : 0u),
                                  make_float4(w * d.x, w * d.y, w * d.z, w * d.w));
            }
        }
        return;
    }
    // taps in two or more slots
#pragma unroll 1
    for (int t = 0; t < 8; ++t) {
        const int bx = t & 1, by = (t >> 1) & 1, bz = t >> 2;
        const float w = (bx ? ax.f : 1.0f - ax.f) * (by ? ay.f : 1.0f - ay.f) * (bz ? az.f : 1.0f - az.f);
        if (w == 0.0f) continue;
        const int sx = bx ? ax.s1 : ax.s0, lx = bx ? ax.l1 : ax.l0;
        const int sy = by ? ay.s1 : ay.s0, ly = by ? ay.l1 : ay.l0;
        const int sz = bz ? az.s1 : az.s0, lz = bz ? az.l1 : az.l0;
        const uint32_t slot = ((uint32_t)sz * SY + (uint32_t)sy) * SX + (uint32_t)sx;
        if (slot != c_slot) {
            c_row = grad_row(gt, slot, p.status);
            c_slot = slot;
        }
        if (c_row < 0) continue;
        texel_atomic<F64>(gt, (size_t)c_row * 1000u + (uint32_t)((lz * 10 + ly) * 10 + lx),
                          make_float4(w * d.x, w * d.y, w * d.z, w * d.w));
    }
}

// scatter_texels for a sample of a segment whose slot's gradient row is `row`
// (-1: none): the taps' cell comes from the segment's slot.  False (and
// nothing) when the taps leave the slot.
template <bool F64>
__device__ __forceinline__ bool scatter_cell(const RaycastParams& p, const SlotView& sv, F3 uvw, float4 d,
                                             const GradTarget& gt, int row) {
    const TapCell c(p, sv, uvw);
    if (!c.in_slot()) return false;
    if (row < 0) return true;
    const float fx = c.t[0] - (c.fl[0] - kFloorMagic), fy = c.t[1] - (c.fl[1] - kFloorMagic),
                fz = c.t[2] - (c.fl[2] - kFloorMagic);
    const size_t base = (size_t)row * 1000u + (uint32_t)((c.l[2] * 10 + c.l[1]) * 10 + c.l[0]);
    const int lane = (int)(threadIdx.x & 31u);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        // each lane starts at another tap: fewer lanes of one instruction on one texel
        const int tap = (q + lane) & 7;
        const int bx = tap & 1, by = (tap >> 1) & 1, bz = tap >> 2;
        const float w = (bx ? fx : 1.0f - fx) * (by ? fy : 1.0f - fy) * (bz ? fz : 1.0f - fz);
        if (w == 0.0f) continue;
        texel_atomic<F64>(gt, base + (uint32_t)(bx + 10 * by + 100 * bz), make_float4(w * d.x, w * d.y, w * d.z, w * d.w));
    }
    return true;
}

}  // namespace

// One pixel of the checkpointing forward.
template <int FMT, bool UNIT>
__device__ __forceinline__ void forward_pixel(const RaycastParams& p, int px, int py, int2* hdr, Ckpt* ckpt,
                                              int per_ray, const PathSlots& path) {
    const vv_uniforms& u = p.u;
    const bool inside = px < u.width && py < u.height;
    const size_t pix = inside ? (size_t)py * u.width + px : 0;
    bool ok = true;
    const WalkConsts k = walk_consts(p, UNIT ? __ldg(p.walk) : fetch_node<false>(p, 0, 0, 0, ok));
    CkptVisitor vis;
    vis.start(ckpt + pix * ray_records(per_ray), per_ray, p.status);
    RayState s;
    s.dst = make_float4(0.f, 0.f, 0.f, 0.f);
    s.nsamples = 0;
    F3 pos;
    const bool alive = inside && ray_origin(u, k, px, py, pos) && ray_start(p, k, px, py, pos, s);
    walk<FMT, false, CkptVisitor, UNIT, 1>(p, k, s, vis, path, alive);
    if (!inside) return;
    if (p.color) p.color[pix] = s.dst;
    hdr[pix] = make_int2(vis.count, s.nsamples);
}
template <int FMT>
__device__ __noinline__ void forward_pixel_box(const RaycastParams& p, int px, int py, int2* hdr, Ckpt* ckpt,
                                               int per_ray) {
    forward_pixel<FMT, false>(p, px, py, hdr, ckpt, per_ray, PathSlots{nullptr, 0, nullptr});
}

// 7 resident CTAs (28 warps) per SM, at most 72 registers per thread: the
// occupancy that measured fastest for the plain ray cast.  FP32 texels (32
// registers a sample) take 5: a fit step 18.8 ms against 20.3 at 7, 18.9 at 4.
template <int FMT, int VIEWS, int RAYS>
__global__ void __launch_bounds__(128, FMT == VV_FMT_FP32 ? 5 : 7)
    forward_ckpt_kernel(const __grid_constant__ DiffViews<VIEWS> dv, char* ckpts, size_t stride, size_t hdr_size,
                        int per_ray) {
    const RaycastParams& p = dv.p[VIEWS > 1 ? blockIdx.z : 0];
    int2* hdr = (int2*)(ckpts + (VIEWS > 1 ? blockIdx.z * stride : 0));
    Ckpt* ckpt = (Ckpt*)((char*)hdr + hdr_size);
    int px, py;
    warp_pixel<RAYS>(px, py);
    __shared__ uint32_t path[kPathLevels][128];
    if (unit_walk(p))
        forward_pixel<FMT, true>(p, px, py, hdr, ckpt, per_ray,
                                 PathSlots{&path[0][threadIdx.x], 128, nullptr});
    else
        forward_pixel_box<FMT>(p, px, py, hdr, ckpt, per_ray);
}

// The state a walk record restarts from.
__device__ __forceinline__ RayState walk_state(const RayState& s0, const Ckpt& c) {
    RayState s = s0;
    s.pos = f3(c.p0.x, c.p0.y, c.p1.x);
    s.dst = make_float4(0.f, 0.f, 0.f, c.p1.y);
    s.iter = 0;  // (the bound on iterations: the forward came through with this part of them)
    s.nsamples = (int)c.w.x;
    s.nptr = 0u;
    return s;
}

// The piece [first, last) of a ray whose records ran out, walked from its walk
// record; all lanes of the warp call it, `on` the ones that have such a piece.
// Out of line: few rays cross more sampled segments than there are records.
template <int FMT>
__device__ __noinline__ int replay_tail(const RaycastParams& p, const WalkConsts& k, const RayState& s0, const Ckpt& c,
                                        Piece* piece, float4 g, int first, int last, bool on, PathSlots path) {
    ReplayVisitor rv;
    rv.piece = piece;
    rv.first = first;
    rv.last = last;
    rv.n = 0;
    rv.g = g;
    RayState s = walk_state(s0, c);
    walk<FMT, false, ReplayVisitor, true, 1>(p, k, s, rv, path, on);
    return rv.n;
}

// One pixel of the adjoint in the unit box; all lanes of a warp call it.  F64:
// binary64 gradient rows; WSUM: the lanes of a cell summed before the atomics
// (scatter_texels).
template <int FMT, bool F64, bool WSUM>
__device__ __forceinline__ void backward_pixel(const RaycastParams& p, int px, int py, const int2* hdr,
                                               const Ckpt* ckpt, int per_ray, const float4* dl_dcolor,
                                               const GradTarget& gt, const PathSlots& path) {
    const vv_uniforms& u = p.u;
    const bool inside = px < u.width && py < u.height;
    const size_t pix = inside ? (size_t)py * u.width + px : 0;
    int2 h = make_int2(0, 0);
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
    if (inside) {
        h = hdr[pix];
        g = dl_dcolor[pix];
    }
    const int C = h.x, total = h.y;
    const WalkConsts k = walk_consts(p, __ldg(p.walk));
    RayState s0;
    F3 pos = f3(0.f, 0.f, 0.f);
    bool more = C != 0 && total != 0 && (g.x != 0.f || g.y != 0.f || g.z != 0.f || g.w != 0.f) &&
                ray_origin(u, k, px, py, pos);
    ray_start(p, k, inside ? px : 0, inside ? py : 0, pos, s0);  // direction of this ray
    const Ckpt* ck = ckpt + pix * ray_records(per_ray);
    uint32_t c_slot = 0xFFFFFFFFu;  // the last slot scattered into and its gradient row
    int c_row = -1;
    Piece piece;
    // pieces of the ray's records, the last first.  The lanes of a warp take
    // their pieces together: they meet before every replay and every scatter
    // (left to itself each lane runs ahead on its own, at 8 threads a warp
    // instruction instead of 15).
    int c = C - 1, m = -1;
    int end = total;  // of a walk record's samples
    while (__any_sync(0xFFFFFFFFu, more)) {
        int n = 0;  // samples of the piece
        bool tail = false;
        int first = 0, last = 0;
        Ckpt cc;
        cc.p0 = cc.p1 = make_float2(0.f, 0.f);
        cc.w = make_uint2(0u, 0u);
        BrickMarch b;
        b.slot_id = kNoSlot;
        if (more) {
            cc = ck[c];
            tail = (cc.w.y >> 24) == kRecWalk;
            const int count = tail ? end - (int)cc.w.x : (int)(cc.w.y & 0xFFFFu);
            if (m < 0) m = (count - 1) / kPiece;
            first = m * kPiece;
            last = min(count, first + kPiece);
        }
        if (__any_sync(0xFFFFFFFFu, tail)) {  // (copies: the originals stay in registers)
            const WalkConsts kt = k;
            const RayState st = s0;
            const Ckpt ct = cc;
            n = replay_tail<FMT>(p, kt, st, ct, &piece, g, (int)ct.w.x + first, (int)ct.w.x + last, tail, path);
        }
        if (more && !tail) {
            n = last - first;
            const int depth = (int)(cc.w.y >> 16) & 255;
            float da = cc.p1.y;
            if ((cc.w.y >> 24) == kRecConst) {
                const float4 src = constant_sample(k, cc.w.x, depth);
                for (int i = 0; i < last; ++i) {
                    const float T = 1.0f - da;
                    if (i >= first) piece.put(i - first, kSampleConst, src, f3(0.f, 0.f, 0.f), T, g);
                    da = T * src.w + da;
                }
            } else {
                RayState s = s0;
                s.pos = f3(cc.p0.x, cc.p0.y, cc.p1.x);
                const F3 lo = unit_corner(s.pos, __float_as_uint(__fadd_rz(s.pos.x, 1.0f)),
                                          __float_as_uint(__fadd_rz(s.pos.y, 1.0f)),
                                          __float_as_uint(__fadd_rz(s.pos.z, 1.0f)), depth);
                b.set<false>(p, k, s, cc.w.x, muls(sub(s.pos, lo), pow2i(depth)), depth, 0.0f);
                for (int i = 0; i < last; ++i) {
                    float4 src = make_float4(0.f, 0.f, 0.f, 0.f);
                    const float T = 1.0f - da;
                    // (an empty sample leaves the alpha as it is, also where T is infinite)
                    if (!b.sv.cmask || sample_needed(p, b.sv, b.bpos)) {
                        src = fetch_sample<FMT>(p, b.sv, b.bpos);
                        src.w = 1.0f - (1.0f - src.w);
                        da = T * src.w + da;
                    }
                    if (i >= first) piece.put(i - first, kSampleBrick, src, b.bpos, T, g);
                    b.bpos = add(b.bpos, b.bstep);
                }
            }
        }
        __syncwarp();
        if (more) {
            // the segment's row, its own: scatter_texels moves (c_slot, c_row) to
            // the slot of a sample that left the segment's
            int row = -1;
            if (b.slot_id != kNoSlot) {
                row = b.slot_id == c_slot ? c_row : grad_row(gt, b.slot_id, p.status);
                c_slot = b.slot_id;
                c_row = row;
            }
            for (int j = n - 1; j >= 0; --j) {
                const float tj = piece.T[j];
                const float t = fabsf(tj);
                if (!(__float_as_uint(tj) >> 31)) {
                    const float4 d = make_float4(g.x * t, g.y * t, g.z * t, g.w * t);
                    if (WSUM || b.slot_id == kNoSlot || !scatter_cell<F64>(p, b.sv, piece.bpos[j], d, gt, row))
                        scatter_texels<F64, WSUM>(p, piece.bpos[j], d, gt, c_slot, c_row);
                }
                // g.a -= dot(g, src), the products summed in the order x, y, z, w
                g.w = g.w - (piece.r[j] + g.w * piece.a[j]);
            }
            if (--m < 0) {
                if (tail) end = (int)cc.w.x;
                more = --c >= 0;
            }
        }
    }
}

// The same where the unit box's walk is not taken: every record is walked from.
template <int FMT, bool F64, bool WSUM>
__device__ __forceinline__ void backward_pixel_box(const RaycastParams& p, int px, int py, const int2* hdr,
                                                const Ckpt* ckpt, int per_ray, const float4* dl_dcolor,
                                                const GradTarget& gt) {
    const vv_uniforms& u = p.u;
    if (px >= u.width || py >= u.height) return;
    const size_t pix = (size_t)py * u.width + px;
    const int2 h = hdr[pix];
    float4 g = dl_dcolor[pix];
    if (h.x == 0 || h.y == 0 || (g.x == 0.f && g.y == 0.f && g.z == 0.f && g.w == 0.f)) return;
    bool ok = true;
    const WalkConsts k = walk_consts(p, fetch_node<false>(p, 0, 0, 0, ok));
    RayState s0;
    F3 pos;
    if (!ray_origin(u, k, px, py, pos)) return;
    ray_start(p, k, px, py, pos, s0);
    const Ckpt* ck = ckpt + pix * ray_records(per_ray);
    uint32_t c_slot = 0xFFFFFFFFu;
    int c_row = -1;
    Piece piece;
    ReplayVisitor rv;
    rv.piece = &piece;
    int b = h.y;
    for (int c = h.x - 1; c >= 0; --c) {
        const int a = (int)ck[c].w.x;
        for (int m = (b - a - 1) / kPiece; m >= 0; --m) {
            RayState s = walk_state(s0, ck[c]);
            rv.first = a + m * kPiece;
            rv.last = min(b, rv.first + kPiece);
            rv.n = 0;
            rv.g = g;
            walk<FMT, false, ReplayVisitor, false, 1>(p, k, s, rv, PathSlots{nullptr, 0, nullptr}, true);
            for (int j = rv.n - 1; j >= 0; --j) {
                const float tj = piece.T[j], t = fabsf(tj);
                if (!(__float_as_uint(tj) >> 31))
                    scatter_texels<F64, WSUM>(p, piece.bpos[j], make_float4(g.x * t, g.y * t, g.z * t, g.w * t), gt,
                                              c_slot, c_row);
                g.w = g.w - (piece.r[j] + g.w * piece.a[j]);
            }
        }
        b = a;
    }
}

// 4 resident CTAs per SM (128 registers).  What bounds it is the latency of
// its loads (texels, and the pieces in local memory) behind a small L1, not
// warps to switch to: one forward and adjoint of the 1080p frame 6.67 ms at 6
// CTAs, 6.02 at 5, 5.53 at 4, 5.72 at 3; a fit step of eight 512x512 views of
// FP32 bricks 27.0, 24.2, 20.2 and 20.0 ms.  Also measured and left: the 8
// texels of a cell summed in registers along the ray (2.3 times fewer
// reductions, 7.0 and 23.8 ms: more instructions, and the reductions are not
// the bound any more), pieces of 32 samples (5.58, 22.1), two samples' texels
// in flight together (0.98-1.00 of the speed), positions summed again instead
// of kept (1.02 and 0.87 of it).
//
// Each warp has a block of pixels of its own and each lane starts at another
// tap.  Close to the terrain, where thousands of samples fall on one texel, the
// reductions' contention is the bound: backward of two such 1080p views (34445
// and 14119 bricks touched) 16.8 and 9.7 ms with neither, 12.2 and 7.8 with the
// taps alone, 14.4 and 9.1 with the blocks alone, 10.2 and 7.1 with both; the
// usual views (5.3 and 4.9) take 4.6 and 4.0 with the blocks, 4.8 and 4.3 with
// both; fit steps are within 4 %.
template <int FMT, bool F64, bool WSUM, int VIEWS, int RAYS>
__global__ void __launch_bounds__(128, 4)
    backward_kernel(const __grid_constant__ DiffViews<VIEWS> dv, const char* ckpts, size_t stride, size_t hdr_size,
                    int per_ray, const float4* dl, const __grid_constant__ GradTarget gt) {
    const RaycastParams& p = dv.p[VIEWS > 1 ? blockIdx.z : 0];
    const int2* hdr = (const int2*)(ckpts + (VIEWS > 1 ? blockIdx.z * stride : 0));
    const Ckpt* ckpt = (const Ckpt*)((const char*)hdr + hdr_size);
    const float4* dl_dcolor = dl + (VIEWS > 1 ? (size_t)blockIdx.z * p.u.width * p.u.height : 0);
    int px, py;
    warp_pixel<RAYS>(px, py);
    __shared__ uint32_t path[kPathLevels][128];
    backward_pixel<FMT, F64, WSUM>(p, px, py, hdr, ckpt, per_ray, dl_dcolor, gt,
                                   PathSlots{&path[0][threadIdx.x], 128, nullptr});
}

// The views of other boxes, in a kernel of its own: as a function that the
// kernel above called for such a view it ran a lane at a time.  One backward of
// the 1024^3 terrain in a box of three quarters at 960x540 / the 512^3 one at
// 1920x1080 / the 256^3 one at 256x256: 6.27 / 6.20 / 1.28 ms as a function, 1.61
// / 3.88 / 0.53 ms here (6 CTAs per SM, 80 registers; 5 the same).  17 views of
// 96x96 in one launch of 16 and one: fit step 2.34 ms, a launch each 13.0.
template <int FMT, bool F64, bool WSUM, int VIEWS>
__global__ void __launch_bounds__(128, 6)
    backward_box_kernel(const __grid_constant__ DiffViews<VIEWS> dv, const char* ckpts, size_t stride, size_t hdr_size,
                        int per_ray, const float4* dl, const __grid_constant__ GradTarget gt, int rays) {
    const RaycastParams& p = dv.p[VIEWS > 1 ? blockIdx.z : 0];
    const char* ck = ckpts + (VIEWS > 1 ? blockIdx.z * stride : 0);
    const float4* dl_dcolor = dl + (VIEWS > 1 ? (size_t)blockIdx.z * p.u.width * p.u.height : 0);
    int px, py;
    if (rays == 4) warp_pixel<4>(px, py);
    else if (rays == 16) warp_pixel<16>(px, py);
    else warp_pixel<32>(px, py);
    backward_pixel_box<FMT, F64, WSUM>(p, px, py, (const int2*)ck, (const Ckpt*)(ck + hdr_size), per_ray, dl_dcolor, gt);
}

// grad[e] += copy_k[e] for the extra copies k of the rows in use (all rows
// without a row counter), each copy element zeroed after it is read (the
// copies are all zero between reductions).  All loads of an element are
// issued before its stores (streaming: the copies are not read again soon).
template <int EXTRA>
__global__ void spread_reduce_kernel(float4* __restrict__ grad, float4* __restrict__ spread,
                                     const int* __restrict__ rows_used, int rows) {
    const size_t n = (size_t)(rows_used ? min(*rows_used, rows) : rows) * 1000u;
    const size_t stride = (size_t)rows * 1000u;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        float4 v[EXTRA];
#pragma unroll
        for (int k = 0; k < EXTRA; ++k) v[k] = __ldcs(spread + (size_t)k * stride + e);
        float4 s = grad[e];
#pragma unroll
        for (int k = 0; k < EXTRA; ++k) s = make_float4(s.x + v[k].x, s.y + v[k].y, s.z + v[k].z, s.w + v[k].w);
        grad[e] = s;
#pragma unroll
        for (int k = 0; k < EXTRA; ++k) __stcs(spread + (size_t)k * stride + e, zero);
    }
}

cudaError_t launch_spread_reduce(const GradTarget& grad, cudaStream_t s) {
    if (grad.copies <= 1) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    const dim3 blocks((unsigned)(sms * 16)), threads(256);
    switch (grad.copies) {
        case 2: spread_reduce_kernel<1><<<blocks, threads, 0, s>>>((float4*)grad.grad, grad.spread, grad.rows_used,
                                                                   grad.spread_rows); break;
        case 4: spread_reduce_kernel<3><<<blocks, threads, 0, s>>>((float4*)grad.grad, grad.spread, grad.rows_used,
                                                                   grad.spread_rows); break;
        case 8: spread_reduce_kernel<7><<<blocks, threads, 0, s>>>((float4*)grad.grad, grad.spread, grad.rows_used,
                                                                   grad.spread_rows); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

size_t ckpt_bytes(int w, int h, int per_ray) { return ckpt_buffer_bytes(w, h, per_ray); }

namespace {

// One launch for a call's views, up to kMaxDiffViews: a view of a fit (512x512
// and less) does not fill the machine, and its slowest rays end alone.
template <int FMT, int VIEWS>
cudaError_t forward_views(const RaycastParams* p, int n, char* ckpt, size_t stride, int per_ray, cudaStream_t s) {
    const int W = p->u.width, H = p->u.height;
    DiffViews<VIEWS> dv;
    for (int v = 0; v < n; ++v) dv.p[v] = p[v];
    const size_t hdr = ckpt_header_bytes(W, H);
    const int rays = rays_per_warp((long long)n * W * H);
    const dim3 grid = warp_grid(rays, W, H, n);
    if (rays == 4) forward_ckpt_kernel<FMT, VIEWS, 4><<<grid, 128, 0, s>>>(dv, ckpt, stride, hdr, per_ray);
    else if (rays == 16) forward_ckpt_kernel<FMT, VIEWS, 16><<<grid, 128, 0, s>>>(dv, ckpt, stride, hdr, per_ray);
    else forward_ckpt_kernel<FMT, VIEWS, 32><<<grid, 128, 0, s>>>(dv, ckpt, stride, hdr, per_ray);
    return cudaGetLastError();
}

template <int FMT, bool F64, bool WSUM, int VIEWS>
cudaError_t backward_views(const RaycastParams* p, int n, const char* ckpt, size_t stride, int per_ray,
                           const float4* dl, const GradTarget& gt, cudaStream_t s) {
    const int W = p->u.width, H = p->u.height;
    DiffViews<VIEWS> dv;
    for (int v = 0; v < n; ++v) dv.p[v] = p[v];
    const size_t hdr = ckpt_header_bytes(W, H);
    // (the forms for checks and comparisons take full warps)
    const int rays = F64 || WSUM ? 32 : rays_per_warp((long long)n * W * H);
    const dim3 grid = warp_grid(rays, W, H, n);
    if constexpr (!F64 && !WSUM) {
        if (rays == 4) {
            backward_kernel<FMT, F64, WSUM, VIEWS, 4><<<grid, 128, 0, s>>>(dv, ckpt, stride, hdr, per_ray, dl, gt);
            return cudaGetLastError();
        }
        if (rays == 16) {
            backward_kernel<FMT, F64, WSUM, VIEWS, 16><<<grid, 128, 0, s>>>(dv, ckpt, stride, hdr, per_ray, dl, gt);
            return cudaGetLastError();
        }
    }
    backward_kernel<FMT, F64, WSUM, VIEWS, 32><<<grid, 128, 0, s>>>(dv, ckpt, stride, hdr, per_ray, dl, gt);
    return cudaGetLastError();
}

// Views that take the unit box's walk, or views that do not.
template <int FMT, bool F64, bool WSUM, int VIEWS>
cudaError_t backward_run(const RaycastParams* p, int n, const char* ckpt, size_t stride, int per_ray, const float4* dl,
                         const GradTarget& gt, cudaStream_t s) {
    if (takes_unit_walk(*p)) return backward_views<FMT, F64, WSUM, VIEWS>(p, n, ckpt, stride, per_ray, dl, gt, s);
    const int W = p->u.width, H = p->u.height;
    DiffViews<VIEWS> dv;
    for (int v = 0; v < n; ++v) dv.p[v] = p[v];
    const int rays = F64 || WSUM ? 32 : rays_per_warp((long long)n * W * H);
    backward_box_kernel<FMT, F64, WSUM, VIEWS><<<warp_grid(rays, W, H, n), 128, 0, s>>>(
        dv, ckpt, stride, ckpt_header_bytes(W, H), per_ray, dl, gt, rays);
    return cudaGetLastError();
}

template <int FMT>
cudaError_t backward_form(const RaycastParams* p, int n, const char* ckpt, size_t stride, int per_ray, const float4* dl,
                          const GradTarget& gt, cudaStream_t s) {
    const size_t npix = (size_t)p->u.width * p->u.height;
    const int most = gt.f64 || gt.warp_sum ? 1 : kMaxDiffViews;
    cudaError_t e = cudaSuccess;
    for (int v = 0, m; v < n && e == cudaSuccess; v += m) {
        for (m = 1; m < most && v + m < n && takes_unit_walk(p[v + m]) == takes_unit_walk(p[v]);) ++m;
        const char* ck = ckpt + (size_t)v * stride;
        const float4* d = dl + (size_t)v * npix;
        if (m > 1) e = backward_run<FMT, false, false, kMaxDiffViews>(p + v, m, ck, stride, per_ray, d, gt, s);
        else if (gt.f64 && gt.warp_sum) e = backward_run<FMT, true, true, 1>(p + v, 1, ck, stride, per_ray, d, gt, s);
        else if (gt.f64) e = backward_run<FMT, true, false, 1>(p + v, 1, ck, stride, per_ray, d, gt, s);
        else if (gt.warp_sum) e = backward_run<FMT, false, true, 1>(p + v, 1, ck, stride, per_ray, d, gt, s);
        else e = backward_run<FMT, false, false, 1>(p + v, 1, ck, stride, per_ray, d, gt, s);
    }
    return e;
}

template <int FMT>
cudaError_t forward_form(const RaycastParams* p, int n, char* ckpt, size_t stride, int per_ray, cudaStream_t s) {
    cudaError_t e = cudaSuccess;
    for (int v = 0; v < n && e == cudaSuccess; v += kMaxDiffViews) {
        const int m = n - v < kMaxDiffViews ? n - v : kMaxDiffViews;
        char* ck = ckpt + (size_t)v * stride;
        e = m > 1 ? forward_views<FMT, kMaxDiffViews>(p + v, m, ck, stride, per_ray, s)
                  : forward_views<FMT, 1>(p + v, 1, ck, stride, per_ray, s);
    }
    return e;
}

}  // namespace

cudaError_t launch_forward_ckpt(int fmt, const RaycastParams* p, int n, void* ckpt, size_t stride, int per_ray,
                                cudaStream_t s) {
    switch (fmt) {
        case VV_FMT_RGBA8: return forward_form<VV_FMT_RGBA8>(p, n, (char*)ckpt, stride, per_ray, s);
        case VV_FMT_FP16: return forward_form<VV_FMT_FP16>(p, n, (char*)ckpt, stride, per_ray, s);
        case VV_FMT_BF16: return forward_form<VV_FMT_BF16>(p, n, (char*)ckpt, stride, per_ray, s);
        case VV_FMT_FP32: return forward_form<VV_FMT_FP32>(p, n, (char*)ckpt, stride, per_ray, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_backward(int fmt, const RaycastParams* p, int n, const void* ckpt, size_t stride, int per_ray,
                            const float4* dl_dcolor, const GradTarget& grad, cudaStream_t s) {
    const char* ck = (const char*)ckpt;
    switch (fmt) {
        case VV_FMT_RGBA8: return backward_form<VV_FMT_RGBA8>(p, n, ck, stride, per_ray, dl_dcolor, grad, s);
        case VV_FMT_FP16: return backward_form<VV_FMT_FP16>(p, n, ck, stride, per_ray, dl_dcolor, grad, s);
        case VV_FMT_BF16: return backward_form<VV_FMT_BF16>(p, n, ck, stride, per_ray, dl_dcolor, grad, s);
        case VV_FMT_FP32: return backward_form<VV_FMT_FP32>(p, n, ck, stride, per_ray, dl_dcolor, grad, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace vv
