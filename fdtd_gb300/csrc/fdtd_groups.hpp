// How the points of a soft source are grouped into the items of the fused
// passes.  No CUDA in here, so that it can be compiled and checked without a GPU.
#pragma once

namespace fdtd {

// End of the group that starts at point `first`: the points [first, end) are
// taken while their bounding box holds at most kGroupFill cells per point, so
// that few cells look for a point of theirs in vain and a table of the box's
// cells stays small.  at(q, a): coordinate a of point q; the points come in
// cell order.  A diagonal line through the grid, us per step, one group with a
// bisection in every cell of its box and groups of 8 cells per point: 256^3
// float32 386 -> 282, 320^3 791 -> 573, 180^3 float32c 214 -> 179, 2D 900^2
// 42.1 -> 34.5.  2 and 4 cells per point measured the same within 2 %, but 320^3
// 604 with 2.
constexpr long long kGroupFill = 8;

template <class At>
inline int group_end(int first, int last, At at) {
    int lo[3], hi[3];
    for (int a = 0; a < 3; ++a) lo[a] = hi[a] = at(first, a);
    int e = first + 1;
    for (; e < last; ++e) {
        long long box = 1;
        for (int a = 0; a < 3; ++a) {
            const int x = at(e, a);
            lo[a] = x < lo[a] ? x : lo[a];
            hi[a] = x > hi[a] ? x : hi[a];
            box *= hi[a] - lo[a] + 1;
        }
        if (box > kGroupFill * (e - first + 1)) break;
    }
    return e;
}

}  // namespace fdtd
