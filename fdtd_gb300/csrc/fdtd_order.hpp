// The order in which a cell's absorbing layers are corrected: that of their
// registration (fdtd/grid.py:284-293, 311-320), as the flat half steps follow it.
// No CUDA in here, so that it can be compiled and checked without a GPU.
#pragma once

#ifdef __CUDACC__
#define FDTD_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define FDTD_HOST_DEVICE inline
#endif

namespace fdtd {

// The axes of an order, four bits each from the first one corrected.
constexpr int kOrderXYZ = 0x210;
constexpr int kOrderBySide = 0;  // layers of two axes interleave: cell_order

// Places of the layers by axis and side (0 low, 1 high) in registration order.
struct LayerRank {
    unsigned char at[3][2];
};

// Order of n layers (at most one per axis and side) given in registration
// order: x, y, z wherever the layers allow it (axes without a layer go
// anywhere), else the axes as registered; kOrderBySide where layers of two
// axes interleave, so that no one order serves every cell.
inline int layer_order(int n, const int *axis, const int *high, LayerRank &rank) {
    bool plain = true, grouped = true;
    for (int a = 0; a < 3; ++a) rank.at[a][0] = rank.at[a][1] = (unsigned char)(6 + a);  // no layer
    for (int s = 0; s < n; ++s) {
        rank.at[axis[s]][high[s]] = (unsigned char)s;
        for (int t = s + 1; t < n; ++t) {
            plain = plain && axis[s] <= axis[t];
            grouped = grouped && (axis[s] != axis[t] || axis[t] == axis[t - 1]);
        }
    }
    if (plain) return kOrderXYZ;
    if (!grouped) return kOrderBySide;
    int at = 0, listed = 0, order = 0;
    for (int s = 0; s < n + 3; ++s) {
        const int a = s < n ? axis[s] : s - n;
        if (listed >> a & 1) continue;
        listed |= 1 << a;
        order |= a << 4 * at++;
    }
    return order;
}

// Order of a cell's layers under kOrderBySide, given the side that it can be in
// along each axis (a cell meets at most one layer per axis; axes on which it
// meets none go anywhere).
FDTD_HOST_DEVICE int cell_order(const LayerRank &rank, bool xhigh, bool yhigh, bool zhigh) {
    const int x = xhigh ? rank.at[0][1] : rank.at[0][0], y = yhigh ? rank.at[1][1] : rank.at[1][0],
              z = zhigh ? rank.at[2][1] : rank.at[2][0];
    const int px = (y < x) + (z < x), py = (x < y) + (z < y), pz = (x < z) + (y < z);
    return 0 << 4 * px | 1 << 4 * py | 2 << 4 * pz;
}

}  // namespace fdtd
