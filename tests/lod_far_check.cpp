// Host check of voxviz_b200/csrc/lod_bound.h for cameras outside the range its
// bounds are shown for (1e6 and beyond, up to where squares overflow): the LOD
// test stops there, so neither certificate may clear a level.  Built and run by
// tests/test_lod_far.py; prints "<checks> <violations>".
#include <cmath>
#include <cstdio>
#include <initializer_list>

#include "../voxviz_b200/csrc/lod_bound.h"

using vv::lodb::V3;

int main() {
    long checks = 0, bad = 0;
    for (double far = 1.1e6; far < 1e38; far *= 3.0)
        for (int axis = 0; axis < 3; ++axis)
            for (int sign = -1; sign <= 1; sign += 2)
                for (int depth = 1; depth <= 11; ++depth) {
                    float c[3] = {0.5f, 0.5f, 0.5f};
                    c[axis] = (float)(sign * far);
                    const V3 C{c[0], c[1], c[2]};
                    // up and left across the view direction: |a x w| is all of |a| |w|
                    const V3 up = axis == 0 ? V3{0, 1, 0} : V3{1, 0, 0}, left = axis == 2 ? V3{0, 1, 0} : V3{0, 0, 1};
                    for (const float px : {1e-7f, 1e-3f, 1.0f}) {
                        const vv::lodb::Consts k = vv::lodb::make_consts(C, up, left, 0.0625f, 1.0f, px, depth, true);
                        const V3 pos{0.5f, 0.5f, 0.5f};
                        int lo, hi;
                        vv::lodb::clear_range(k, pos, lo, hi);
                        ++checks;
                        if (vv::lodb::deep_levels(k, pos) >= 0 || lo <= hi) ++bad;
                    }
                }
    printf("%ld %ld\n", checks, bad);
    return bad ? 1 : 0;
}
