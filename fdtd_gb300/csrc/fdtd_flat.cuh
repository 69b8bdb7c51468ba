// Flat half steps: one thread per cell, marching along x.
//
// A plane of a field is one contiguous run of ny nz cells.  A block takes
// kFlatBlock consecutive cells of the tile box's plane and steps them through
// a chunk of planes, so every lane holds a cell whatever nz is (odd extents,
// 2D grids), a layer normal to z is a run of lanes and not a few lanes of
// every warp, and a thread's place in the plane, its layers, their
// coefficients and its neighbours' offsets are worked out once per chunk.
// E marches up and H down, so the x neighbour is the plane before and stays in
// registers.  The arithmetic of each cell and its order are those of thread_E
// / thread_H, and so are the bits.
//
// Bound by latency and instruction issue, not by bytes: at 128^3 with 12-cell
// layers (everything in L2) a half step issues 205 (E) and 160 (H) warp
// instructions per 32 cells, 48 % of the issue slots.  us per step with one
// launch per half step (plain object, plane source, plane record), four blocks
// of 64 registers per SM: 52.8; five (48 registers) and three (80) measured 65
// and 77.  Against the register-streaming tiles (four cells per thread, whose
// warps all hold a few cells of each z layer and whose 124 registers leave 16
// warps per SM), the same scene 91 -> 53, 192x192x96 169 -> 92, 131x150x97 83 ->
// 55; in the persistent loop 128^3 89 -> 47, 64^3 15.9 -> 11.9, 131x150x97 71 ->
// 48.  Float32 only: with double or compensated values, and on the slab-free
// interior of a partition, the register tiles stay faster (256^3 float64 1416
// against 1675, float32c 500 against 565).
#pragma once

#include "fdtd_cell.cuh"

namespace fdtd {

constexpr int kFlatBlocks = 4;  // per SM

// A pair of auxiliaries of a layer, or of values.
template <class T>
struct alignas(2 * sizeof(T)) FlatPair {
    T p0, p1;
};

// A thread's layer normal to one axis (q null: none): where the pair of the
// present plane is, the coefficients, and whether the differences drive it
// (not on the layer's plane whose neighbour lies outside it).
template <class T>
struct FlatLayer {
    FlatPair<T> *q;
    T b, c;
    bool inc;
};

// The pair of a layer on one plane, updated with its two differences and
// stored (without the drive: p b + 0 c).
template <class P>
__device__ __forceinline__ void flat_psi(const FlatLayer<typename P::T> &L, FlatPair<typename P::T> &p,
                                         typename P::T d0, typename P::T d1) {
    using T = typename P::T;
    p.p0 = P::psi(p.p0, L.b, L.inc ? d0 : T(0), L.c);
    p.p1 = P::psi(p.p1, L.b, L.inc ? d1 : T(0), L.c);
    if (L.q) *L.q = p;
}

// Column of a block's thread in the plane of the tile box.
struct FlatPlace {
    bool in;
    int j, k;
};
__device__ __forceinline__ FlatPlace flat_place(const GridK &g, unsigned chunk) {
    const int bnz = g.ez - g.oz;
    const long total = (long)(g.ey - g.oy) * bnz;
    const long t = (long)chunk * kFlatBlock + threadIdx.x;
    FlatPlace p;
    p.in = t < total;
    if (total < (1L << 31)) {
        const unsigned row = (unsigned)t / (unsigned)bnz;
        p.j = g.oy + (int)row;
        p.k = g.oz + (int)((unsigned)t - row * (unsigned)bnz);
    } else {
        p.j = g.oy + (int)(t / bnz);
        p.k = g.oz + (int)(t % bnz);
    }
    return p;
}

// First point of a group at or after key (its cells by column, ascending).
__device__ __forceinline__ int point_at(const ItemK &s, long long key) {
    const long long *cells = (const long long *)s.coef[0];
    int a = 0, n = s.aux;
    while (n > 0) {
        const int h = n >> 1;
        if (cells[a + h] < key) {
            a += h + 1;
            n -= h + 1;
        } else {
            n = h;
        }
    }
    return a;
}

// The chunk's listed sources (where the kernel's parameters do not hold them) on
// planes [xa, xb), after the march has stored those planes: one source after
// the other over the planes (each cell gets them in order), so that a thread
// looks at a source once and not once a plane, and finds its column's first
// point in a group by one bisection.  us per step, plane by plane and with a
// bisection per plane inside the march, and now: 128^3 with 40 points 68 -> 46,
// 200 points 118 -> 76; 2D 1500x1100 with a diagonal line 74 -> 33, 128^3 62 ->
// 39, with six of them 355 -> 54.
// Not inlined: the march would lose the registers (192x192x96 E half and H half
// 84 -> 75, 131x150x97 in the persistent loop 53.5 -> 50.6).
template <class P, bool IS_E>
__device__ __noinline__ void flat_listed(const GridK &g, const double *__restrict__ wave, unsigned chunk, int xa,
                                            int xb) {
    using T = typename P::T;
    const FlatPlace pl = flat_place(g, chunk);
    if (!pl.in) return;
    const int nx = g.nx, ny = g.ny, nz = g.nz, j = pl.j, k = pl.k;
    const long nyz = (long)ny * nz, jk = (long)j * nz + k;
    T *F = (T *)(IS_E ? g.E : g.H);
    const int *off = IS_E ? g.srcE_off : g.srcH_off, *idx = IS_E ? g.srcE_idx : g.srcH_idx;
    const int last = off[chunk + 1];
    T none = T(0);
#pragma unroll 1
    for (int it = off[chunk]; it < last; ++it) {
        const ItemK &s = g.items[idx[it]];
        if (j < s.lo[1] || j >= s.hi[1] || k < s.lo[2] || k >= s.hi[2]) continue;
        const int i0 = max(xa, s.lo[0]), end = min(xb, s.hi[0]);
        T *f = F + 3 * jk + s.comp;
        const T wv = (T)wave[s.column];
        if (IS_E && s.kind == kItemSoftGroup) {
            const long long *cells = (const long long *)s.coef[0];
            const double *weights = (const double *)s.coef[1];
            if (cells == nullptr) {
#pragma unroll 1
                for (int i = i0; i < end; ++i)
                    P::add_prod(f[3 * (i * nyz)], none, (T)weights[box_index(s, i, j, k)], wv);
            } else {
                const long long key = (long long)jk * nx;
#pragma unroll 1
                for (int a = point_at(s, key + i0); a < s.aux && cells[a] < key + end; ++a)
                    P::add_prod(f[3 * ((cells[a] - key) * nyz)], none, (T)weights[a], wv);
            }
        } else {
            const bool soft = s.kind == FDTD_ITEM_SOFT;
#pragma unroll 1
            for (int i = i0; i < end; ++i) {
                T &x = f[3 * (i * nyz)];
                if (soft) P::add_prod(x, none, (T)s.weight, wv);
                else P::set(x, none, P::mul((T)s.weight, wv));
            }
        }
    }
}

// Where a thread stands in its march: its cell of the present plane in the
// neighbour field, the field and the material (values or index), and the
// neighbour field on the plane before.
template <class T>
struct FlatMarch {
    const T *pn;
    T *pf;
    const T *pm;
    const unsigned char *pid;
    T by, bz;
};

// A cell of one plane: the neighbour field there and at its y and z
// neighbours, the field, courant times the material.
template <class T>
struct FlatCell {
    T ax, ay, az, yx, yz, zx, zy, f0, f1, f2, m0, m1, m2;
    int id;
};

// The loads of the cell `step` values on from the present plane's.
template <class P, int MAT>
__device__ __forceinline__ void flat_load(FlatCell<typename P::T> &v, const FlatMarch<typename P::T> &s, long step,
                                          long istep, long oy, long oz) {
    const typename P::T *n = s.pn + step, *f = s.pf + step;
    v.ax = n[0];
    v.ay = n[1];
    v.az = n[2];
    v.yx = n[oy];
    v.yz = n[oy + 2];
    v.zx = n[oz];
    v.zy = n[oz + 1];
    v.f0 = f[0];
    v.f1 = f[1];
    v.f2 = f[2];
    if constexpr (MAT == MAT_FULL) {
        v.m0 = s.pm[step];
        v.m1 = s.pm[step + 1];
        v.m2 = s.pm[step + 2];
    } else if constexpr (MAT == MAT_IDS) {
        v.id = (int)s.pid[istep];
    }
}

template <class P, int MAT>
__device__ __forceinline__ void flat_material(FlatCell<typename P::T> &v, const typename P::T *lut, int nlut,
                                              typename P::T courant, const typename P::T (&m)[3]) {
    using T = typename P::T;
    if constexpr (MAT == MAT_UNIFORM) {
        v.m0 = m[0];
        v.m1 = m[1];
        v.m2 = m[2];
    } else {
        if constexpr (MAT == MAT_IDS) {
            const bool in = v.id < nlut;  // an index past the table reads zeros
            v.m0 = in ? lut[3 * v.id] : T(0);
            v.m1 = in ? lut[3 * v.id + 1] : T(0);
            v.m2 = in ? lut[3 * v.id + 2] : T(0);
        }
        v.m0 = P::cm(courant, v.m0);
        v.m1 = P::cm(courant, v.m1);
        v.m2 = P::cm(courant, v.m2);
    }
}

template <class P, bool IS_E>
__device__ __forceinline__ void flat_bulk(FlatCell<typename P::T> &v, typename P::T u0, typename P::T u1,
                                          typename P::T u2) {
    typename P::T none = 0;
    if (IS_E) {
        P::add_prod(v.f0, none, v.m0, u0);
        P::add_prod(v.f1, none, v.m1, u1);
        P::add_prod(v.f2, none, v.m2, u2);
    } else {
        P::sub_prod(v.f0, none, v.m0, u0);
        P::sub_prod(v.f1, none, v.m1, u1);
        P::sub_prod(v.f2, none, v.m2, u2);
    }
}

// Bulk update of a cell with all its neighbours in the grid, but for those
// along z in a 2D grid; (by, bz) is the neighbour field on the plane before.
template <class P, bool IS_E>
__device__ __forceinline__ void flat_plain(FlatCell<typename P::T> &v, typename P::T by, typename P::T bz,
                                           bool flat2d) {
    using T = typename P::T;
    const T xy = IS_E ? v.ay - by : by - v.ay, xz = IS_E ? v.az - bz : bz - v.az;
    const T yx = IS_E ? v.ax - v.yx : v.yx - v.ax, yz = IS_E ? v.az - v.yz : v.yz - v.az;
    const T zx = flat2d ? T(0) : (IS_E ? v.ax - v.zx : v.zx - v.ax);
    const T zy = flat2d ? T(0) : (IS_E ? v.ay - v.zy : v.zy - v.ay);
    flat_bulk<P, IS_E>(v, yz - zy, zx - xz, xy - yx);
}

template <class T>
__device__ __forceinline__ void flat_store(const FlatCell<T> &v, const FlatMarch<T> &s, long step) {
    s.pf[step] = v.f0;
    s.pf[step + 1] = v.f1;
    s.pf[step + 2] = v.f2;
}

// The march moved on by `step` values past cell v.
template <class T, int MAT>
__device__ __forceinline__ void flat_next(FlatMarch<T> &s, const FlatCell<T> &v, long step, long istep) {
    s.by = v.ay;
    s.bz = v.az;
    s.pn += step;
    s.pf += step;
    if constexpr (MAT == MAT_FULL) s.pm += step;
    if constexpr (MAT == MAT_IDS) s.pid += istep;
}

// The low or high layer of an axis at coordinate x: its slab-local index, -1 outside.
__device__ __forceinline__ int flat_side(const SlabK (&lay)[2], int x, bool &low) {
    low = x < lay[0].th;
    const int l = x - lay[1].start;
    return low ? x : (l >= 0 && l < lay[1].th ? l : -1);
}

template <class T, bool IS_E>
__device__ __forceinline__ FlatLayer<T> flat_layer_at(const SlabK (&lay)[2], int l, bool low, long pair) {
    const SlabK &A = lay[0], &B = lay[1];
    FlatLayer<T> L;
    L.q = (FlatPair<T> *)(IS_E ? (low ? A.psiE : B.psiE) : (low ? A.psiH : B.psiH)) + pair;
    L.b = ((const T *)(IS_E ? (low ? A.bE : B.bE) : (low ? A.bH : B.bH)))[l];
    L.c = ((const T *)(IS_E ? (low ? A.cE : B.cE) : (low ? A.cH : B.cH)))[l];
    L.inc = IS_E ? l >= 1 : l <= (low ? A.th : B.th) - 2;
    return L;
}

// Order of a cell's layers where they interleave.  Not inlined: the march would
// lose the registers on every grid (us per step, inlined and not: 64^3 12.3 ->
// 11.9, 131x150x97 50.9 -> 47.2, 2D 1500x1100 30.7 -> 28.6, 128^3 with layers in
// the order z, y, x 42.9 -> 38.9, interleaved 47.8 -> 47.5).
static __device__ __noinline__ int flat_order(const GridK &g, int i, int j, int k) {
    return cell_order(g.lay_rank, i >= g.lay[0][0].th, j >= g.lay[1][0].th, k >= g.lay[2][0].th);
}

// What a thread knows of its column of a tile before it marches.  A block of
// the persistent loop that keeps its tile works it out once per launch.
template <class T>
struct FlatColumn {
    FlatPair<T> *yq, *wq;  // the layers normal to y and z: pair of the march's first plane,
    T yb, yc, wb, wc;      // coefficients,
    int ystep, wstep;      // step to the next plane's pair
    int j, k;
    unsigned omask, smask;  // objects and sources whose y and z ranges hold the cell
    int ob0, ob1;           // the chunk's objects in the lists (past 32 tested plane by plane)
    bool in, yok, zok, special, yinc, winc;
};

template <class P, bool IS_E>
__device__ __forceinline__ FlatColumn<typename P::T> flat_column(const GridK &g, unsigned chunk, int xa, int xb) {
    using T = typename P::T;
    constexpr int dir = IS_E ? 1 : -1;
    const int ny = g.ny, nz = g.nz;
    const FlatPlace pl = flat_place(g, chunk);
    const int j = pl.j, k = pl.k;
    FlatColumn<T> o;
    o.in = pl.in;
    o.j = j;
    o.k = k;
    o.yok = IS_E ? j > 0 : j < ny - 1;
    o.zok = IS_E ? k > 0 : k < nz - 1;
    const int i0 = IS_E ? xa : xb - 1;

    // an object or source whose y and z ranges hold this cell sets a bit, so
    // that a plane tests only those
    o.ob0 = o.ob1 = 0;
    o.omask = o.smask = 0;
    if constexpr (IS_E) {
        o.ob0 = g.obj_off[chunk];
        o.ob1 = g.obj_off[chunk + 1];
        for (int it = o.ob0; it < min(o.ob1, o.ob0 + 32); ++it) {
            const ItemK &b = g.items[g.obj_idx[it]];
            if (b.lo[0] < xb && b.hi[0] > xa && j >= b.lo[1] && j < b.hi[1] && k >= b.lo[2] && k < b.hi[2])
                o.omask |= 1u << (it - o.ob0);
        }
        o.ob1 = max(o.ob1, o.ob0 + 32);
    }
    const FlatSources &src = IS_E ? g.src_E : g.src_H;
#pragma unroll
    for (int q = 0; q < kFlatSources; ++q)
        if (q < src.n && src.item[q].lo[0] < xb && src.item[q].hi[0] > xa && j >= src.item[q].lo[1] &&
            j < src.item[q].hi[1] && k >= src.item[q].lo[2] && k < src.item[q].hi[2])
            o.smask |= 1u << q;
    bool ylow, zlow;
    const int ly = flat_side(g.lay[1], j, ylow), lz = flat_side(g.lay[2], k, zlow);
    o.special =
        __any_sync(0xffffffffu, pl.in && (!o.yok || (!o.zok && nz > 1) || ly >= 0 || lz >= 0 || o.omask != 0 ||
                                          o.smask != 0 || o.ob1 > o.ob0 + 32));
    FlatLayer<T> Y{nullptr, T(0), T(0), false}, W = Y;
    o.ystep = o.wstep = 0;
    if (pl.in && ly >= 0) {
        const int th = ylow ? g.lay[1][0].th : g.lay[1][1].th;
        Y = flat_layer_at<T, IS_E>(g.lay[1], ly, ylow, ((long)i0 * th + ly) * nz + k);
        o.ystep = dir * th * nz;
    }
    if (pl.in && lz >= 0) {
        const int thp = zlow ? g.lay[2][0].thp : g.lay[2][1].thp;
        W = flat_layer_at<T, IS_E>(g.lay[2], lz, zlow, ((long)i0 * ny + j) * thp + lz);
        o.wstep = dir * ny * thp;
    }
    o.yq = Y.q;
    o.yb = Y.b;
    o.yc = Y.c;
    o.yinc = Y.inc;
    o.wq = W.q;
    o.wb = W.b;
    o.wc = W.c;
    o.winc = W.inc;
    return o;
}

// Planes [xa, xb) of a column.  A warp whose cells have all their neighbours in
// the grid and lie in no layer and no object runs the short loop, two planes
// loaded before the first is computed; the others run the full one.
template <class P, bool IS_E, int MAT>
__device__ __forceinline__ void flat_march(const GridK &g, const double *__restrict__ wave, unsigned chunk, int xa,
                                           int xb, const FlatColumn<typename P::T> &col) {
    using T = typename P::T;
    static_assert(sizeof(T) == 4 && !P::COMP, "float32 only: see the head of this file");
    constexpr int dir = IS_E ? 1 : -1;
    if (!col.in) return;
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const int j = col.j, k = col.k;
    const long jk = (long)j * nz + k, nyz = (long)ny * nz;
    const bool yok = col.yok, zok = col.zok, special = col.special;
    // to the y and z neighbours (the cell itself where there is none)
    const long oy = yok ? -dir * 3 * nz : 0, oz = zok ? -dir * 3 : 0;
    const int i0 = IS_E ? xa : xb - 1;
    const int ob0 = col.ob0, ob1 = col.ob1;
    const unsigned omask = col.omask, smask = col.smask;
    const FlatSources &src = IS_E ? g.src_E : g.src_H;
    FlatLayer<T> X{nullptr, T(0), T(0), false}, Y{col.yq, col.yb, col.yc, col.yinc}, W{col.wq, col.wb, col.wc, col.winc};
    const int ystep = col.ystep, wstep = col.wstep;

    const T courant = courant_of<T>(g);
    const T *lut = (const T *)(IS_E ? g.mlut_E : g.mlut_H);
    const int nlut = IS_E ? g.nlut_E : g.nlut_H;
    const long first = (long)i0 * nyz + jk, step = dir * 3 * nyz, istep = dir * nyz;
    FlatMarch<T> s;
    s.pn = (const T *)(IS_E ? g.H : g.E) + 3 * first;
    s.pf = (T *)(IS_E ? g.E : g.H) + 3 * first;
    s.pm = MAT == MAT_FULL ? (const T *)(IS_E ? g.ie : g.imu) + 3 * first : nullptr;
    s.pid = MAT == MAT_IDS ? (IS_E ? g.mid_E : g.mid_H) + first : nullptr;
    T m[3] = {T(0), T(0), T(0)};
    if constexpr (MAT == MAT_UNIFORM) {
#pragma unroll
        for (int q = 0; q < 3; ++q) m[q] = P::cm(courant, lut[q]);
    }
    bool xok = IS_E ? i0 > 0 : i0 < nx - 1;  // only the march's first plane can lack an x neighbour
    s.by = s.bz = T(0);
    if (xok) {
        s.by = s.pn[1 - step];
        s.bz = s.pn[2 - step];
    }

    const int end = IS_E ? xb : xa - 1;  // the march stops before this plane
    int i = i0;
    while (i != end) {
        // planes up to the next face of a layer normal to x
        int stop = end;
        X.q = nullptr;
        const T *tb = nullptr, *tc = nullptr;  // this layer's coefficients
        int edge = -1;                         // its plane that no difference drives
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const SlabK &S = g.lay[0][h];
            const int lo = S.start, hi = S.start + S.th;
            if (lo == hi) continue;
            if (i >= lo && i < hi) {
                stop = IS_E ? min(stop, hi) : max(stop, lo - 1);
                tb = (const T *)(IS_E ? S.bE : S.bH) - lo;
                tc = (const T *)(IS_E ? S.cE : S.cH) - lo;
                edge = IS_E ? lo : hi - 1;
                X.q = (FlatPair<T> *)(IS_E ? S.psiE : S.psiH) + (long)(i - lo) * nyz + jk;
            } else if (IS_E ? lo > i : hi <= i) {
                stop = IS_E ? min(stop, lo) : max(stop, hi - 1);
            }
        }
        if (!special && tb == nullptr && xok) {
#pragma unroll 1
            for (; (stop - i) * dir >= 2; i += 2 * dir) {
                FlatCell<T> v, w;
                flat_load<P, MAT>(v, s, 0, 0, oy, oz);
                flat_load<P, MAT>(w, s, step, istep, oy, oz);
                flat_material<P, MAT>(v, lut, nlut, courant, m);
                flat_plain<P, IS_E>(v, s.by, s.bz, nz == 1);
                flat_store(v, s, 0);
                flat_material<P, MAT>(w, lut, nlut, courant, m);
                flat_plain<P, IS_E>(w, v.ay, v.az, nz == 1);
                flat_store(w, s, step);
                flat_next<T, MAT>(s, w, 2 * step, 2 * istep);
            }
#pragma unroll 1
            for (; i != stop; i += dir) {
                FlatCell<T> v;
                flat_load<P, MAT>(v, s, 0, 0, oy, oz);
                flat_material<P, MAT>(v, lut, nlut, courant, m);
                flat_plain<P, IS_E>(v, s.by, s.bz, nz == 1);
                flat_store(v, s, 0);
                flat_next<T, MAT>(s, v, step, istep);
            }
            continue;
        }
        const bool hx = tb != nullptr, hy = Y.q != nullptr, hw = W.q != nullptr;
#pragma unroll 1
        for (; i != stop; i += dir) {
            FlatCell<T> v;
            flat_load<P, MAT>(v, s, 0, 0, oy, oz);
            FlatPair<T> qx{T(0), T(0)}, qy{T(0), T(0)}, qw{T(0), T(0)};
            if (hx) {
                qx = *X.q;
                X.b = tb[i];
                X.c = tc[i];
                X.inc = i != edge;
            }
            if (hy) qy = *Y.q;
            if (hw) qw = *W.q;
            flat_material<P, MAT>(v, lut, nlut, courant, m);
            // one-sided differences, zero where the neighbour is outside the grid
            const T xy = xok ? (IS_E ? v.ay - s.by : s.by - v.ay) : T(0);
            const T xz = xok ? (IS_E ? v.az - s.bz : s.bz - v.az) : T(0);
            const T yx = yok ? (IS_E ? v.ax - v.yx : v.yx - v.ax) : T(0);
            const T yz = yok ? (IS_E ? v.az - v.yz : v.yz - v.az) : T(0);
            const T zx = zok ? (IS_E ? v.ax - v.zx : v.zx - v.ax) : T(0);
            const T zy = zok ? (IS_E ? v.ay - v.zy : v.zy - v.ay) : T(0);
            const T u0 = yz - zy, u1 = zx - xz, u2 = xy - yx;
            T none = T(0);
            flat_bulk<P, IS_E>(v, u0, u1, u2);
            if constexpr (IS_E) {
                for (unsigned om = omask; om; om &= om - 1) {
                    const ItemK &o = g.items[g.obj_idx[ob0 + __ffs(om) - 1]];
                    if (i >= o.lo[0] && i < o.hi[0])
                        apply_object_cell<P>(o, box_index(o, i, j, k), courant, u0, u1, u2, v.f0, v.f1, v.f2, none,
                                             none, none);
                }
                for (int it = ob0 + 32; it < ob1; ++it) {
                    const ItemK &o = g.items[g.obj_idx[it]];
                    if (in_box(o, i, j, k))
                        apply_object_cell<P>(o, box_index(o, i, j, k), courant, u0, u1, u2, v.f0, v.f1, v.f2, none,
                                             none, none);
                }
            }
            // auxiliaries, then their corrections in boundary order (of a layer
            // normal to c, component c+1 takes -p0 and c+2 takes p1)
            if (hx) flat_psi<P>(X, qx, xz, xy);
            flat_psi<P>(Y, qy, yx, yz);
            flat_psi<P>(W, qw, zy, zx);
            if (g.lay_order == kOrderXYZ) {
                if (hx) pml_correct<P, IS_E>(v.f1, none, v.m1, -qx.p0);
                if (hx) pml_correct<P, IS_E>(v.f2, none, v.m2, qx.p1);
                if (hy) pml_correct<P, IS_E>(v.f2, none, v.m2, -qy.p0);
                if (hy) pml_correct<P, IS_E>(v.f0, none, v.m0, qy.p1);
                if (hw) pml_correct<P, IS_E>(v.f0, none, v.m0, -qw.p0);
                if (hw) pml_correct<P, IS_E>(v.f1, none, v.m1, qw.p1);
            } else {
                int o = g.lay_order;
                if (o == kOrderBySide) o = flat_order(g, i, j, k);
#pragma unroll 1
                for (int r = 0; r < 3; ++r, o >>= 4) {
                    if ((o & 15) == 0 && hx) {
                        pml_correct<P, IS_E>(v.f1, none, v.m1, -qx.p0);
                        pml_correct<P, IS_E>(v.f2, none, v.m2, qx.p1);
                    } else if ((o & 15) == 1 && hy) {
                        pml_correct<P, IS_E>(v.f2, none, v.m2, -qy.p0);
                        pml_correct<P, IS_E>(v.f0, none, v.m0, qy.p1);
                    } else if ((o & 15) == 2 && hw) {
                        pml_correct<P, IS_E>(v.f0, none, v.m0, -qw.p0);
                        pml_correct<P, IS_E>(v.f1, none, v.m1, qw.p1);
                    }
                }
            }
            for (unsigned sm = smask; sm; sm &= sm - 1) {
                const ItemK &o = src.item[__ffs(sm) - 1];
                if (i < o.lo[0] || i >= o.hi[0]) continue;
                T x = o.comp == 0 ? v.f0 : (o.comp == 1 ? v.f1 : v.f2);
                const T wv = (T)wave[o.column];
                if (IS_E && o.kind == kItemSoftGroup)  // (its box is full)
                    P::add_prod(x, none, (T)((const double *)o.coef[1])[box_index(o, i, j, k)], wv);
                else if (o.kind == FDTD_ITEM_SOFT) P::add_prod(x, none, (T)o.weight, wv);
                else P::set(x, none, P::mul((T)o.weight, wv));
                if (o.comp == 0) v.f0 = x;
                else if (o.comp == 1) v.f1 = x;
                else v.f2 = x;
            }
            flat_store(v, s, 0);
            flat_next<T, MAT>(s, v, step, istep);
            X.q += istep;
            if (hy) Y.q += ystep;
            if (hw) W.q += wstep;
            xok = true;
        }
    }
    if (src.n < 0) flat_listed<P, IS_E>(g, wave, chunk, xa, xb);
}

// Block b of a half step: chunk b mod n of the plane, x chunk b / n.  MAT: how
// the material is read.
template <class P, bool IS_E, int MAT>
__global__ void __launch_bounds__(kFlatBlock, kFlatBlocks)
    k_flat(const __grid_constant__ GridK g, const double *__restrict__ wave) {
    const unsigned n = g.flat_chunks, xc = blockIdx.x / n, chunk = blockIdx.x - xc * n;
    const int xa = g.ox + (int)xc * g.XC, xb = min(g.ex, xa + g.XC);
    flat_march<P, IS_E, MAT>(g, wave, chunk, xa, xb, flat_column<P, IS_E>(g, chunk, xa, xb));
}

}  // namespace fdtd
