// Host check of voxviz_b200/csrc/ckpt_layout.h, built and run by
// tests/test_ckpt_layout.py: a ray's last record ends inside the buffer, no ray
// reaches into the next one's, and no number of slots overflows.
#include <cstdio>
#include <initializer_list>

#include "../voxviz_b200/csrc/ckpt_layout.h"

int main() {
    long checks = 0, bad = 0;
    for (const int per_ray : {1, 2, 3, 16, 1 << 20, (1 << 30) - 1, 1 << 30, (1 << 30) + 1, 0x7FFFFFFF})
        for (const int w : {1, 2, 3, 63, 1920})
            for (const int h : {1, 5, 1080}) {
                const unsigned __int128 records = (unsigned __int128)2 * per_ray, pixels = (unsigned __int128)w * h;
                const unsigned __int128 bytes = (pixels * 8 + 15) / 16 * 16 + pixels * records * 24;
                const int cap = vv::record_cap(per_ray);
                ++checks;
                if (vv::ckpt_buffer_bytes(w, h, per_ray) != bytes || vv::ray_records(per_ray) != records || cap <= 0 ||
                    (unsigned __int128)cap > records || vv::ckpt_header_bytes(w, h) % 16 != 0)
                    ++bad;
                // (the walk records' share and the segment records', adjoint.cu)
                const int walks = cap / 4 > 1 ? cap / 4 : 1;
                if (cap - walks < 1 || cap - walks >= cap) ++bad;
            }
    printf("%ld %ld\n", checks, bad);
    return bad ? 1 : 0;
}
