// Flat transposed half steps (float32 plans whose layers run inside the pass):
// k_adj_H and k_adj_E with one thread per cell of a flattened plane, marching
// along x as the flat half steps of the forward run do (fdtd_flat.cuh), and
// for the same reasons.  The transposed H half reads the backward neighbours
// of w = courant inv_mu lam_H and marches up, the transposed E half the
// forward neighbours of u = courant inv_eps lam_E and marches down.  The
// arithmetic of each cell and its order are those of adj_bulk_H / adj_slab_H
// and adj_bulk_E / adj_slab_E.
//
// 128^3 with 12-cell layers: transposed E half 47 -> 32 us, H half 45 -> 24; a
// gradient of 60 steps 14.3 -> 12.6 ms, 192x192x96 of 40 steps 15.5 -> 13.1.
// Four blocks of 64 registers; three of 80 measured 240 against 221 us per step
// of the whole gradient.
#pragma once

#include "fdtd_adjoint.cuh"
#include "fdtd_flat.cuh"

namespace fdtd {

// A thread's layer normal to one axis: the pair of the present plane in the
// current auxiliaries (q null: none) and in the next ones, the step to the
// neighbour along the normal, the coefficients of this place and of the
// neighbour's, and whether the two terms apply (slab-local index rules).
template <class T>
struct AdjLayer {
    const FlatPair<T> *q;
    FlatPair<T> *n;
    long nbr;
    T b, c, cn;
    bool own, next;
};

// TH: the transposed H half (lam_E from lam_H), else the transposed E half.
template <class T, bool TH>
__device__ __forceinline__ void adj_layer_coefs(AdjLayer<T> &L, const T *b, const T *c, int l, int th) {
    L.b = b[l];
    L.c = c[l];
    L.own = TH ? l <= th - 2 : l >= 1;
    L.next = TH ? l >= 1 : l <= th - 2;
    L.cn = L.next ? c[TH ? l - 1 : l + 1] : T(0);
}

template <class T, bool TH>
__device__ __forceinline__ AdjLayer<T> adj_layer_at(const SlabK (&lay)[2], const void *const (&old)[3][2],
                                                    void *const (&now)[3][2], int axis, int l, bool low, long pair,
                                                    long stride) {
    const SlabK &A = lay[0], &B = lay[1];
    AdjLayer<T> L;
    L.q = (const FlatPair<T> *)(low ? old[axis][0] : old[axis][1]) + pair;
    L.n = (FlatPair<T> *)(low ? now[axis][0] : now[axis][1]) + pair;
    L.nbr = TH ? -stride : stride;
    adj_layer_coefs<T, TH>(L, (const T *)(TH ? (low ? A.bH : B.bH) : (low ? A.bE : B.bE)),
                           (const T *)(TH ? (low ? A.cH : B.cH) : (low ? A.cE : B.cE)), l, low ? A.th : B.th);
    return L;
}

// One layer's terms on a cell: v1, v2 are the scaled values that drive its
// first and second auxiliary, n1, n2 the neighbour's; d0 and d1 are taken from
// the two tangential components by the caller.
template <class T, bool TH>
__device__ __forceinline__ void adj_layer(const AdjLayer<T> &L, FlatPair<T> p, FlatPair<T> pn, T v1, T v2, T n1, T n2,
                                          T &d0, T &d1) {
    const T f = T(1);
    T a0, a1;
    d0 = T(0);
    d1 = T(0);
    if (TH) {
        a0 = p.p0 + f * v1;
        a1 = p.p1 - f * v2;
        if (L.own) {
            d0 = L.c * a0;
            d1 = L.c * a1;
        }
        if (L.next) {
            const T p0 = pn.p0 + f * n1;
            const T p1 = pn.p1 - f * n2;
            d0 -= L.cn * p0;
            d1 -= L.cn * p1;
        }
    } else {
        a0 = p.p0 - f * v1;
        a1 = p.p1 + f * v2;
        if (L.own) {
            d0 = -(L.c * a0);
            d1 = -(L.c * a1);
        }
        if (L.next) {
            const T q0 = pn.p0 - f * n1;
            const T q1 = pn.p1 + f * n2;
            d0 += L.cn * q0;
            d1 += L.cn * q1;
        }
    }
    *L.n = FlatPair<T>{L.b * a0, L.b * a1};
}

// Auxiliaries of the layers by axis and side: current (read) and next.
struct AdjFlat {
    const void *old[3][2];
    void *now[3][2];
};

// The scaled field at a cell and its y and z neighbours, and the field updated.
// The scaled products are rounded before they are added, as in the other
// transposed kernels (which select between them and zero first).
template <class T>
struct AdjCell {
    T ax, ay, az, yx, yz, zx, zy, f0, f1, f2;
};

template <class T, int MAT>
__device__ __forceinline__ void adj_load(AdjCell<T> &v, const T *n, const T *f, const T *m, const unsigned char *id,
                                         long oy, long oz, long iy, long iz, const T *lut, int nlut, T c,
                                         const T (&mu)[3]) {
    T a[3] = {n[0], n[1], n[2]}, y[2] = {n[oy], n[oy + 2]}, z[2] = {n[oz], n[oz + 1]};
    v.f0 = f[0];
    v.f1 = f[1];
    v.f2 = f[2];
    T ma[3], my[2], mz[2];
    if constexpr (MAT == MAT_FULL) {
        ma[0] = m[0];
        ma[1] = m[1];
        ma[2] = m[2];
        my[0] = m[oy];
        my[1] = m[oy + 2];
        mz[0] = m[oz];
        mz[1] = m[oz + 1];
    } else if constexpr (MAT == MAT_IDS) {
        const int i0 = id[0], i1 = id[iy], i2 = id[iz];  // (an index past the table reads zeros)
#pragma unroll
        for (int q = 0; q < 3; ++q) ma[q] = i0 < nlut ? lut[3 * i0 + q] : T(0);
        my[0] = i1 < nlut ? lut[3 * i1] : T(0);
        my[1] = i1 < nlut ? lut[3 * i1 + 2] : T(0);
        mz[0] = i2 < nlut ? lut[3 * i2] : T(0);
        mz[1] = i2 < nlut ? lut[3 * i2 + 1] : T(0);
    }
    if constexpr (MAT == MAT_UNIFORM) {
        v.ax = __fmul_rn(mu[0], a[0]);
        v.ay = __fmul_rn(mu[1], a[1]);
        v.az = __fmul_rn(mu[2], a[2]);
        v.yx = __fmul_rn(mu[0], y[0]);
        v.yz = __fmul_rn(mu[2], y[1]);
        v.zx = __fmul_rn(mu[0], z[0]);
        v.zy = __fmul_rn(mu[1], z[1]);
    } else {
        v.ax = __fmul_rn(c * ma[0], a[0]);
        v.ay = __fmul_rn(c * ma[1], a[1]);
        v.az = __fmul_rn(c * ma[2], a[2]);
        v.yx = __fmul_rn(c * my[0], y[0]);
        v.yz = __fmul_rn(c * my[1], y[1]);
        v.zx = __fmul_rn(c * mz[0], z[0]);
        v.zy = __fmul_rn(c * mz[1], z[1]);
    }
}

// lam of a cell with all six neighbours in the grid; (bx.. on the plane before).
template <class T, bool TH>
__device__ __forceinline__ void adj_plain(AdjCell<T> &v, T by, T bz) {
    if (TH) {
        const T dy_z = v.az - v.yz, dz_y = v.ay - v.zy, dz_x = v.ax - v.zx;
        const T dx_z = v.az - bz, dx_y = v.ay - by, dy_x = v.ax - v.yx;
        v.f0 -= dy_z - dz_y;
        v.f1 -= dz_x - dx_z;
        v.f2 -= dx_y - dy_x;
    } else {
        const T dy_z = v.yz - v.az, dz_y = v.zy - v.ay, dz_x = v.zx - v.ax;
        const T dx_z = bz - v.az, dx_y = by - v.ay, dy_x = v.yx - v.ax;
        v.f0 += dy_z - dz_y;
        v.f1 += dz_x - dx_z;
        v.f2 += dx_y - dy_x;
    }
}

// Blocks as in k_flat: chunk b mod n of the plane, x chunk b / n.
template <class T, bool TH, int MAT>
__global__ void __launch_bounds__(kFlatBlock, 4) k_adj_flat(const __grid_constant__ GridK g,
                                                            const __grid_constant__ AdjFlat aux) {
    constexpr int dir = TH ? 1 : -1;
    const unsigned nch = g.flat_chunks, xc = blockIdx.x / nch, chunk = blockIdx.x - xc * nch;
    const int xa = (int)xc * g.XC, xb = min(g.nx, xa + g.XC);
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const FlatPlace pl = flat_place(g, chunk);
    const int j = pl.j, k = pl.k;
    const long jk = (long)j * nz + k, nyz = (long)ny * nz;
    // the neighbour read lies behind (TH) or ahead; `own` terms drop on the far face
    const bool ynb = TH ? j > 0 : j < ny - 1, znb = TH ? k > 0 : k < nz - 1;
    const bool yow = TH ? j < ny - 1 : j > 0, zow = TH ? k < nz - 1 : k > 0;
    const long iy = ynb ? -dir * nz : 0, iz = znb ? -dir : 0;
    const int i0 = TH ? xa : xb - 1;
    bool ylow, zlow;
    const int ly = flat_side(g.lay[1], j, ylow), lz = flat_side(g.lay[2], k, zlow);
    const bool special =
        __any_sync(0xffffffffu, pl.in && (!ynb || !znb || !yow || !zow || ly >= 0 || lz >= 0));
    if (!pl.in) return;

    const T c = courant_of<T>(g);
    const T *lut = (const T *)(TH ? g.mlut_H : g.mlut_E);
    const int nlut = TH ? g.nlut_H : g.nlut_E;
    T mu[3] = {T(0), T(0), T(0)};
    if constexpr (MAT == MAT_UNIFORM) {
#pragma unroll
        for (int q = 0; q < 3; ++q) mu[q] = c * lut[q];
    }
    const long first = (long)i0 * nyz + jk, step = dir * 3 * nyz, istep = dir * nyz;
    const T *pn = (const T *)(TH ? g.H : g.E) + 3 * first;
    T *pf = (T *)(TH ? g.E : g.H) + 3 * first;
    const T *pm = MAT == MAT_FULL ? (const T *)(TH ? g.imu : g.ie) + 3 * first : nullptr;
    const unsigned char *pid = MAT == MAT_IDS ? (TH ? g.mid_H : g.mid_E) + first : nullptr;
    T by = T(0), bz = T(0);  // scaled, on the plane before
    if (TH ? i0 > 0 : i0 < nx - 1) {
        T m1 = mu[1], m2 = mu[2];
        if constexpr (MAT == MAT_FULL) {
            m1 = c * pm[1 - step];
            m2 = c * pm[2 - step];
        } else if constexpr (MAT == MAT_IDS) {
            const int id = pid[-istep];
            m1 = id < nlut ? c * lut[3 * id + 1] : T(0);
            m2 = id < nlut ? c * lut[3 * id + 2] : T(0);
        }
        by = __fmul_rn(m1, pn[1 - step]);
        bz = __fmul_rn(m2, pn[2 - step]);
    }

    AdjLayer<T> Y{nullptr, nullptr, 0, T(0), T(0), T(0), false, false}, W = Y, X = Y;
    int ystep = 0, wstep = 0;
    if (special) {
        if (ly >= 0) {
            const int th = ylow ? g.lay[1][0].th : g.lay[1][1].th;
            Y = adj_layer_at<T, TH>(g.lay[1], aux.old, aux.now, 1, ly, ylow, ((long)i0 * th + ly) * nz + k, nz);
            ystep = dir * th * nz;
        }
        if (lz >= 0) {
            const int thp = zlow ? g.lay[2][0].thp : g.lay[2][1].thp;
            W = adj_layer_at<T, TH>(g.lay[2], aux.old, aux.now, 2, lz, zlow, ((long)i0 * ny + j) * thp + lz, 1);
            wstep = dir * ny * thp;
        }
    }
    const bool hy = Y.q != nullptr, hw = W.q != nullptr;

    const int end = TH ? xb : xa - 1;
    int i = i0;
    while (i != end) {
        // planes up to the next face of a layer normal to x, or of the grid
        int stop = end, side = -1;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int lo = g.lay[0][h].start, hi = lo + g.lay[0][h].th;
            if (lo == hi) continue;
            if (i >= lo && i < hi) {
                stop = TH ? min(stop, hi) : max(stop, lo - 1);
                side = h;
            } else if (TH ? lo > i : hi <= i) {
                stop = TH ? min(stop, lo) : max(stop, hi - 1);
            }
        }
        if (!special && side < 0 && i > 0 && i < nx - 1) {
            // (the grid's last plane along the march goes to the full loop)
            const int last = TH ? min(stop, nx - 1) : max(stop, 0);
#pragma unroll 1
            for (; (last - i) * dir >= 2; i += 2 * dir) {
                AdjCell<T> v, w;
                adj_load<T, MAT>(v, pn, pf, pm, pid, 3 * iy, 3 * iz, iy, iz, lut, nlut, c, mu);
                adj_load<T, MAT>(w, pn + step, pf + step, pm + step, pid + istep, 3 * iy, 3 * iz, iy, iz, lut, nlut, c,
                                 mu);
                adj_plain<T, TH>(v, by, bz);
                pf[0] = v.f0;
                pf[1] = v.f1;
                pf[2] = v.f2;
                adj_plain<T, TH>(w, v.ay, v.az);
                pf[step] = w.f0;
                pf[step + 1] = w.f1;
                pf[step + 2] = w.f2;
                by = w.ay;
                bz = w.az;
                pn += 2 * step;
                pf += 2 * step;
                if constexpr (MAT == MAT_FULL) pm += 2 * step;
                if constexpr (MAT == MAT_IDS) pid += 2 * istep;
            }
#pragma unroll 1
            for (; i != last; i += dir) {
                AdjCell<T> v;
                adj_load<T, MAT>(v, pn, pf, pm, pid, 3 * iy, 3 * iz, iy, iz, lut, nlut, c, mu);
                adj_plain<T, TH>(v, by, bz);
                pf[0] = v.f0;
                pf[1] = v.f1;
                pf[2] = v.f2;
                by = v.ay;
                bz = v.az;
                pn += step;
                pf += step;
                if constexpr (MAT == MAT_FULL) pm += step;
                if constexpr (MAT == MAT_IDS) pid += istep;
            }
            if (i == stop) continue;
        }
        const bool hx = side >= 0;
        long xpair = 0;
        if (hx) {
            xpair = (long)(i - g.lay[0][side].start) * nyz + jk;
            X.q = (const FlatPair<T> *)(side == 0 ? aux.old[0][0] : aux.old[0][1]) + xpair;
            X.n = (FlatPair<T> *)(side == 0 ? aux.now[0][0] : aux.now[0][1]) + xpair;
            X.nbr = -dir * nyz;
        }
#pragma unroll 1
        for (; i != stop; i += dir) {
            AdjCell<T> v;
            adj_load<T, MAT>(v, pn, pf, pm, pid, 3 * iy, 3 * iz, iy, iz, lut, nlut, c, mu);
            FlatPair<T> qx{T(0), T(0)}, qxn = qx, qy = qx, qyn = qx, qw = qx, qwn = qx;
            if (hx) {
                const SlabK &S = g.lay[0][side];
                adj_layer_coefs<T, TH>(X, (const T *)(TH ? S.bH : S.bE), (const T *)(TH ? S.cH : S.cE), i - S.start,
                                       S.th);
                qx = *X.q;
                if (X.next) qxn = X.q[X.nbr];
            }
            if (hy) {
                qy = *Y.q;
                if (Y.next) qyn = Y.q[Y.nbr];
            }
            if (hw) {
                qw = *W.q;
                if (W.next) qwn = W.q[W.nbr];
            }
            // differences: the own term drops on the far face, the neighbour's on the near one
            const bool xnb = TH ? i > 0 : i < nx - 1, xow = TH ? i < nx - 1 : i > 0;
            const T zero = T(0);
            if (TH) {
                const T dy_z = (yow ? v.az : zero) - (ynb ? v.yz : zero);
                const T dz_y = (zow ? v.ay : zero) - (znb ? v.zy : zero);
                const T dz_x = (zow ? v.ax : zero) - (znb ? v.zx : zero);
                const T dx_z = (xow ? v.az : zero) - (xnb ? bz : zero);
                const T dx_y = (xow ? v.ay : zero) - (xnb ? by : zero);
                const T dy_x = (yow ? v.ax : zero) - (ynb ? v.yx : zero);
                v.f0 -= dy_z - dz_y;
                v.f1 -= dz_x - dx_z;
                v.f2 -= dx_y - dy_x;
            } else {
                const T dy_z = (ynb ? v.yz : zero) - (yow ? v.az : zero);
                const T dz_y = (znb ? v.zy : zero) - (zow ? v.ay : zero);
                const T dz_x = (znb ? v.zx : zero) - (zow ? v.ax : zero);
                const T dx_z = (xnb ? bz : zero) - (xow ? v.az : zero);
                const T dx_y = (xnb ? by : zero) - (xow ? v.ay : zero);
                const T dy_x = (ynb ? v.yx : zero) - (yow ? v.ax : zero);
                v.f0 += dy_z - dz_y;
                v.f1 += dz_x - dx_z;
                v.f2 += dx_y - dy_x;
            }
            // the layers in boundary order; one normal to a takes d0 from
            // component a+2 and d1 from a+1
            auto layer = [&](int a) {
                T d0, d1;
                if (a == 0) {
                    if (hx) {
                        adj_layer<T, TH>(X, qx, qxn, v.ay, v.az, by, bz, d0, d1);
                        v.f2 -= d0;
                        v.f1 -= d1;
                    }
                } else if (a == 1) {
                    if (hy) {
                        adj_layer<T, TH>(Y, qy, qyn, v.az, v.ax, v.yz, v.yx, d0, d1);
                        v.f0 -= d0;
                        v.f2 -= d1;
                    }
                } else if (hw) {
                    adj_layer<T, TH>(W, qw, qwn, v.ax, v.ay, v.zx, v.zy, d0, d1);
                    v.f1 -= d0;
                    v.f0 -= d1;
                }
            };
            if (g.lay_order == kOrderXYZ) {
                layer(0);
                layer(1);
                layer(2);
            } else {
                int o = g.lay_order;
                if (o == kOrderBySide)
                    o = cell_order(g.lay_rank, i >= g.lay[0][0].th, j >= g.lay[1][0].th, k >= g.lay[2][0].th);
#pragma unroll 1
                for (int r = 0; r < 3; ++r, o >>= 4) layer(o & 15);
            }
            pf[0] = v.f0;
            pf[1] = v.f1;
            pf[2] = v.f2;
            by = v.ay;
            bz = v.az;
            pn += step;
            pf += step;
            if constexpr (MAT == MAT_FULL) pm += step;
            if constexpr (MAT == MAT_IDS) pid += istep;
            if (hx) {
                X.q += istep;
                X.n += istep;
            }
            if (hy) {
                Y.q += ystep;
                Y.n += ystep;
            }
            if (hw) {
                W.q += wstep;
                W.n += wstep;
            }
        }
    }
}

}  // namespace fdtd
