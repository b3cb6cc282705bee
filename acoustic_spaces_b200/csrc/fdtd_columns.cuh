// The interior air by columns: quads of four adjacent cells marched along z, a column a thread, from a
// list that holds no other cells (fdtd.hpp:242-288 is the update).
#pragma once

#include "fdtd_kernels.cuh"

namespace fdtd {

constexpr int kColumnPlanes = 8;  // planes an item of the interior's list spans at most (4 bits each)

template <typename T>
struct SweepArgs {
    // {the first quad's pitched index, the interior cells of each plane, four bits a plane from the lowest}
    const uint2 *columns;
    uint32_t count, pitch, plane;
    const float *scale;  // with a speed field: each pitched cell's scale
    T *d;                // COMP: the increments
    float axial, diagonal, centre, total, residual;
};

// A quad's new pressures (fdtd.hpp:242-288) from its own pressures h, its neighbours before and
// after along x (left, right the cells beside the quad), y and z, and with the wide stencil the
// twelve edge sums; pv the previous pressures (COMP: the increments).
template <typename T, bool WIDE, bool SCALED, bool COMP>
struct Update {
    T axial, diagonal, centre, total, residual;
    template <class Edges>
    __device__ __forceinline__ void operator()(const Quad<T> &h, T left, T right, const Quad<T> &ym, const Quad<T> &yp,
                                               const Quad<T> &zm, const Quad<T> &zp, const Quad<T> &pv, const Quad<T> &sc,
                                               Edges edges, Quad<T> &next, Quad<T> &step) const {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const T here = h.v[j];
            const T xm = j == 0 ? left : h.v[j - 1], xp = j == 3 ? right : h.v[j + 1];
            if (COMP) {
                const T sum = (xm - here) + (xp - here) + (ym.v[j] - here) + (yp.v[j] - here) + (zm.v[j] - here) +
                              (zp.v[j] - here);
                const T around = WIDE ? edges(j, here) : (T)0;
                T s;
                if (SCALED) {
                    s = WIDE ? pv.v[j] + (sc.v[j] * axial) * sum + (sc.v[j] * diagonal) * around + (sc.v[j] * residual) * here
                             : pv.v[j] + (sc.v[j] * axial) * sum + (sc.v[j] * residual) * here;
                } else {
                    s = WIDE ? pv.v[j] + axial * sum + diagonal * around + residual * here
                             : pv.v[j] + axial * sum + residual * here;
                }
                next.v[j] = here + s;
                step.v[j] = s;
                continue;
            }
            const T sum = xm + xp + ym.v[j] + yp.v[j] + zm.v[j] + zp.v[j];
            const T around = WIDE ? edges(j, (T)0) : (T)0;
            if (SCALED) {
                next.v[j] = WIDE ? ((T)2 - total * sc.v[j]) * here + (sc.v[j] * axial) * sum + (sc.v[j] * diagonal) * around - pv.v[j]
                                 : ((T)2 - total * sc.v[j]) * here + (sc.v[j] * axial) * sum - pv.v[j];
            } else {
                next.v[j] = WIDE ? centre * here + axial * sum + diagonal * around - pv.v[j] : centre * here + axial * sum - pv.v[j];
            }
        }
    }
};

// What a plane of a 7-point column loads beside the pressures it keeps from the plane before: the
// pressures a plane on, a row before and after and beside the quad, and the previous pressures.
template <typename T>
struct PlaneLoads {
    Quad<T> zp, ym, yp, pv;
    T left, right;
    __device__ __forceinline__ void load(const T *b, const T *before, uint32_t i, uint32_t pitch, uint32_t plane) {
        zp = load_quad(b + i + plane);
        ym = load_quad(b + i - pitch);
        yp = load_quad(b + i + pitch);
        pv = load_quad(before + i);
        left = b[i - 1], right = b[i + 4];
    }
};

// A column of quads along z, the 7-point stencil: each plane's loads are issued while the plane
// before is worked out, and a quad's pressures serve the planes before and after it from registers.
// (The cells beside a quad by shuffles from the lanes beside, in place of scalar loads, made a step of
// 2.9M cells 12.6 us in place of 9.0: the lanes' loads then wait for one another.)
template <typename T, bool SCALED, bool COMP>
__device__ __forceinline__ void step_column(const SweepArgs<T> &p, const T *b, T *a, uint2 column) {
    const uint32_t pitch = p.pitch, plane = p.plane;
    const T *before = COMP ? p.d : a;
    const Update<T, false, SCALED, COMP> update{(T)p.axial, (T)p.diagonal, (T)p.centre, (T)p.total, (T)p.residual};
    uint32_t i = column.x, masks = column.y;
    Quad<T> zm = load_quad(b + i - plane), h = load_quad(b + i);
    PlaneLoads<T> now, then;
    now.load(b, before, i, pitch, plane);
    for (;;) {
        const uint32_t mask = masks & 15u;
        masks >>= 4;
        if (masks) then.load(b, before, i + plane, pitch, plane);
        if (mask) {
            Quad<T> next, step;
            update(h, now.left, now.right, now.ym, now.yp, zm, now.zp, now.pv, scales<T, SCALED>(p.scale, i),
                   [](int, T) { return (T)0; }, next, step);
            store_cells<false>(a + i, next, mask);
            if (COMP) store_cells<false>(p.d + i, step, mask);
        }
        if (!masks) return;
        zm = h, h = now.zp, now = then;
        i += plane;
    }
}

// Six cells of a row: a quad and the cells beside it, where a column's interior cells need them (a
// quad at the grid's first cells has no cell before it, and its first cell is on the edge).
template <typename T>
struct Row {
    T v[6];
    __device__ __forceinline__ void load(const T *p, bool left, bool right) {
        const Quad<T> q = load_quad(p);
        v[0] = left ? p[-1] : (T)0, v[5] = right ? p[4] : (T)0;
#pragma unroll
        for (int j = 0; j < 4; ++j) v[1 + j] = q.v[j];
    }
    __device__ __forceinline__ Quad<T> quad() const { return {{v[1], v[2], v[3], v[4]}}; }
};

// The same with the 19-point stencil: three rows of six cells of each of three planes.
template <typename T, bool SCALED, bool COMP>
__device__ __forceinline__ void step_wide_column(const SweepArgs<T> &p, const T *b, T *a, uint2 column) {
    const uint32_t pitch = p.pitch, plane = p.plane;
    const T *before = COMP ? p.d : a;
    const Update<T, true, SCALED, COMP> update{(T)p.axial, (T)p.diagonal, (T)p.centre, (T)p.total, (T)p.residual};
    uint32_t i = column.x, masks = column.y;
    const bool left = (masks & 0x11111111u) != 0, right = (masks & 0x88888888u) != 0;
    Row<T> z[3][3];  // [plane before, this, after][row before, this, after]
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int r = 0; r < 3; ++r) z[k][r].load(b + i + (k - 1) * (int64_t)plane + (r - 1) * (int64_t)pitch, left, right);
    while (masks) {
        const uint32_t mask = masks & 15u;
        masks >>= 4;
#pragma unroll
        for (int r = 0; r < 3; ++r) z[2][r].load(b + i + plane + (r - 1) * (int64_t)pitch, left, right);
        if (mask) {
            const Quad<T> pv = load_quad(before + i);
            Quad<T> next, step;
            update(
                z[1][1].quad(), z[1][1].v[0], z[1][1].v[5], z[1][0].quad(), z[1][2].quad(), z[0][1].quad(), z[2][1].quad(),
                pv, scales<T, SCALED>(p.scale, i),
                [&](int j, T here) {
                    const T *m = z[1][0].v + j, *q = z[1][2].v + j, *l = z[0][1].v + j, *h = z[2][1].v + j;
                    if (COMP)
                        return (m[0] - here) + (m[2] - here) + (q[0] - here) + (q[2] - here) + (l[0] - here) + (l[2] - here) +
                               (h[0] - here) + (h[2] - here) + (z[0][0].v[j + 1] - here) + (z[0][2].v[j + 1] - here) +
                               (z[2][0].v[j + 1] - here) + (z[2][2].v[j + 1] - here);
                    return m[0] + m[2] + q[0] + q[2] + l[0] + l[2] + h[0] + h[2] + z[0][0].v[j + 1] + z[0][2].v[j + 1] +
                           z[2][0].v[j + 1] + z[2][2].v[j + 1];
                },
                next, step);
            store_cells<false>(a + i, next, mask);
            if (COMP) store_cells<false>(p.d + i, step, mask);
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) z[0][r] = z[1][r], z[1][r] = z[2][r];
        i += plane;
    }
}

// The launched sweep, a column a thread and no loop over columns.
//
// What bounds it is DRAM: 12 bytes a cell (COMP 16, double 24), and the cells around a quad come from L1
// and L2. Two thousand threads an SM of 32 registers each, in many short blocks, keep more loads in
// flight than the pipelined tiles of bulk_kernel, and the list spares the cells around rooms that a tile
// takes in. Alone, tiles and columns: the 4 cm room 97 and 90.6 us, outdoors 640 x 176 x 150 40.8 and 37.3, the batch of
// boxes 49.6 and 37.0, the 6 cm room compensated 43.7 and 39.4, a 16M-cell box with a speed field 57.0 and 47.0, the wide
// stencil on 9.7M cells 45.4 and 27.4; in double the 4 cm room 182.8 and 176.7. (A plain box of 47M cells steps
// at 6.3 TB/s in this form, 6.4 being a two-reads-one-write stream's.)
template <typename T, bool SCALED, bool COMP>
__device__ __forceinline__ void march_column(const SweepArgs<T> &p, const T *b, T *a, uint2 column) {
    const uint32_t pitch = p.pitch, plane = p.plane;
    const T *before = COMP ? p.d : a;
    const Update<T, false, SCALED, COMP> update{(T)p.axial, (T)p.diagonal, (T)p.centre, (T)p.total, (T)p.residual};
    uint32_t i = column.x, masks = column.y;
    Quad<T> zm = load_quad(b + i - plane), h = load_quad(b + i);
    for (; masks; masks >>= 4, i += plane) {
        const uint32_t mask = masks & 15u;
        const Quad<T> zp = load_quad(b + i + plane);
        if (mask) {
            Quad<T> next, step;
            update(h, b[i - 1], b[i + 4], load_quad(b + i - pitch), load_quad(b + i + pitch), zm, zp, load_quad(before + i),
                   scales<T, SCALED>(p.scale, i), [](int, T) { return (T)0; }, next, step);
            store_cells<false>(a + i, next, mask);
            if (COMP) store_cells<false>(p.d + i, step, mask);
        }
        zm = h, h = zp;
    }
}

constexpr int kColumnThreads = 256;

template <typename T, bool WIDE, bool SCALED, bool COMP>
__global__ void __launch_bounds__(kColumnThreads) column_kernel(const __grid_constant__ SweepArgs<T> p, const T *b, T *a) {
    const uint32_t c = blockIdx.x * kColumnThreads + threadIdx.x;
    if (c >= p.count) return;
    const uint2 column = __ldg(p.columns + c);
    if constexpr (WIDE)
        step_wide_column<T, SCALED, COMP>(p, b, a, column);
    else
        march_column<T, SCALED, COMP>(p, b, a, column);
}

}  // namespace fdtd
