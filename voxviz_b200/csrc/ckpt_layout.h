// ckpt_layout.h - where a view's checkpoint records lie in its buffer: 8 bytes
// of header a pixel (records, samples), rounded up to 16 so that the views of a
// call, one after another, all start at that alignment, then the records of the
// pixels, two of 24 bytes for each of the caller's per_ray slots.  A caller may
// ask for up to 2^31 - 1 slots a ray (a frame of a few pixels): offsets are 64
// bits wide, and a ray keeps at most 2^31 - 1 records.
#pragma once

#include <stddef.h>
#include <stdint.h>

#if defined(__CUDACC__)
#define VV_CKPT_HD __host__ __device__ __forceinline__
#else
#define VV_CKPT_HD inline
#endif

namespace vv {

constexpr int kRecordsPerSlot = 2;
constexpr size_t kRecordBytes = 24;

// Records of one ray in the buffer, and how many of them it may use.
VV_CKPT_HD size_t ray_records(int per_ray) { return (size_t)per_ray * (size_t)kRecordsPerSlot; }
VV_CKPT_HD int record_cap(int per_ray) {
    return per_ray > 0x7FFFFFFF / kRecordsPerSlot ? 0x7FFFFFFF : per_ray * kRecordsPerSlot;
}
VV_CKPT_HD size_t ckpt_header_bytes(int w, int h) { return ((size_t)w * (size_t)h * 8u + 15u) / 16u * 16u; }
VV_CKPT_HD size_t ckpt_buffer_bytes(int w, int h, int per_ray) {
    return ckpt_header_bytes(w, h) + (size_t)w * (size_t)h * ray_records(per_ray) * kRecordBytes;
}

}  // namespace vv
