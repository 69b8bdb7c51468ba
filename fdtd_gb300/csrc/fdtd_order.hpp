// The order in which a cell's absorbing layers are corrected: that of their
// registration (fdtd/grid.py:284-293, 311-320), as the flat half steps follow it.
// No CUDA in here, so that it can be compiled and checked without a GPU.
#pragma once

namespace fdtd {

// The axes of an order, four bits each from the first one corrected.
constexpr int kOrderXYZ = 0x210;

// Order of n layers given by their axes in registration order: x, y, z
// wherever the layers allow it (axes without a layer go anywhere), else the
// axes as registered.  False where layers of two axes interleave, so that no
// one order serves every cell.
inline bool layer_order(int n, const int *axis, int &order) {
    bool plain = true, grouped = true;
    for (int s = 0; s < n; ++s)
        for (int t = s + 1; t < n; ++t) {
            plain = plain && axis[s] <= axis[t];
            grouped = grouped && (axis[s] != axis[t] || axis[t] == axis[t - 1]);
        }
    order = kOrderXYZ;
    if (plain || !grouped) return grouped;
    int at = 0, listed = 0;
    order = 0;
    for (int s = 0; s < n + 3; ++s) {
        const int a = s < n ? axis[s] : s - n;
        if (listed >> a & 1) continue;
        listed |= 1 << a;
        order |= a << 4 * at++;
    }
    return true;
}

}  // namespace fdtd
