// The smallest grids: both levels in the shared memory of one cluster of blocks, every step of a piece of
// a run in one launch.
//
// A step of a few thousand cells is all latency: through L2 it costs the pressures' round trip and the
// barrier's (the resident stepper: 1.5-2.6 us). Here the pitched grid's runs of 64 cells go round the
// blocks, so that the walls' rows are shared out evenly, and each block keeps both levels of its cells, its
// rows' tables and its branch velocities in shared memory; a cell's neighbours are read from whichever block
// owns them (ld.shared::cluster), its new pressure is written to its own block's, and the cluster's barrier
// ends the step: 0.85 us on a plain box of 12 cells a side, 1.24 with two branch states a row, 2.2 at 28 a side
// (a run of planes a block instead, the floor's rows on one block: 3.5). The operations of each cell are the
// launched kernels', in their order.
#pragma once

#include "fdtd_resident.cuh"

namespace fdtd {

__device__ __forceinline__ uint32_t cluster_address(uint32_t own, uint32_t rank) {
    uint32_t at;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(own), "r"(rank));
    return at;
}
__device__ __forceinline__ void load_cluster(uint32_t at, float &v) {
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
}
__device__ __forceinline__ void load_cluster(uint32_t at, double &v) {
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(at) : "memory");
}
__device__ __forceinline__ void load_cluster(uint32_t at, Quad<float> &q) {
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(q.v[0]), "=f"(q.v[1]), "=f"(q.v[2]), "=f"(q.v[3])
                 : "r"(at)
                 : "memory");
}
__device__ __forceinline__ void load_cluster(uint32_t at, Quad<double> &q) {
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(q.v[0]), "=d"(q.v[1]) : "r"(at) : "memory");
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(q.v[2]), "=d"(q.v[3]) : "r"(at + 16) : "memory");
}
constexpr uint32_t kClusterBlocks = 16, kClusterRun = 6;
// The block of cell i: runs of 64 cells go round the 16, each round five further on than the one before (walls a
// power of two apart would else fall on a few blocks).
__host__ __device__ __forceinline__ uint32_t cluster_owner(uint32_t i) {
    return ((i >> kClusterRun) + 5 * (i >> (kClusterRun + 4))) & (kClusterBlocks - 1);
}

template <typename T>
struct ClusterArgs {
    Tables g;
    SweepArgs<T> air;  // the coefficients, the scales and the increments (its columns: one plane each, by owner)
    T *u[2], *w[2];    // [1]: the current ones at the launch's start
    uint32_t cells, own_cells;  // the pitched grid's cells and a block's
    // By owner: the rows, {row, its first link and branch state in the block's, its counts: links | states << 8},
    // and where each block's rows and quads begin.
    const uint4 *rows;
    uint32_t row_start[17], quad_start[17];
    const uint32_t *link_start;  // by the grid's rows
    const uint2 *links;
    uint32_t links_at, states_at, rows_at, drive_at;  // where the parts of a block's shared memory begin
    uint32_t most_rows, most_states;
    const float *signal;
    T *gathered;
    uint32_t gathered_count, most_reads, probe_steps, reads_at;
    T *traj_u, *traj_w;
    uint32_t states, steps;
};

// A block's shared memory: two levels (and the increments, and the scales), the links {weight, address of the
// first level's cell in its owner}, the states {weight, now, before, gain} and their velocities, the rows {cell
// within the block, row, first link | links << 24, first state | states << 24}, their coefficients, the drive, and
// the probes' pressures of some steps.
template <typename T, bool SCALED, bool COMP>
constexpr uint32_t kClusterCellBytes = sizeof(T) * (COMP ? 3 : 2) + (SCALED ? 4 : 0);

template <typename T>
constexpr int kClusterThreads = sizeof(T) == 8 ? 512 : 1024;

template <typename T, bool SCALED, bool COMP>
__global__ void __launch_bounds__(kClusterThreads<T>, 1) cluster_kernel(const __grid_constant__ ClusterArgs<T> p) {
    constexpr uint32_t kThreads = kClusterThreads<T>;
    extern __shared__ __align__(128) unsigned char smem[];
    const Tables &g = p.g;
    const uint32_t rank = blockIdx.x, own_cells = p.own_cells, run = (1u << kClusterRun) - 1u;
    T *level = reinterpret_cast<T *>(smem), *increment = level + 2 * own_cells;
    float *scale = reinterpret_cast<float *>(level + (COMP ? 3 : 2) * own_cells);
    uint2 *link = reinterpret_cast<uint2 *>(smem + p.links_at);
    float4 *state = reinterpret_cast<float4 *>(smem + p.states_at);
    T *w = reinterpret_cast<T *>(state + p.most_states);
    uint4 *row = reinterpret_cast<uint4 *>(smem + p.rows_at);
    float4 *coef = reinterpret_cast<float4 *>(row + p.most_rows);
    float *residual = reinterpret_cast<float *>(coef + p.most_rows), *drive = reinterpret_cast<float *>(smem + p.drive_at);
    const uint32_t base = smem_address(smem), level_bytes = own_cells * (uint32_t)sizeof(T);
    // The first level's cell i wherever it lies (a level's is level_bytes further).
    auto local = [&](uint32_t i) { return (i >> (kClusterRun + 4) << kClusterRun) | (i & run); };
    auto address = [&](uint32_t i) {
        return cluster_address(base + local(i) * (uint32_t)sizeof(T), cluster_owner(i));
    };
    auto global = [&](uint32_t c) {
        const uint32_t round = c >> kClusterRun;
        return ((round << 4 | ((rank - 5 * round) & 15u)) << kClusterRun) | (c & run);
    };
    for (uint32_t c = threadIdx.x; c < own_cells; c += kThreads) {
        const uint32_t i = global(c);
        const bool in = i < p.cells;
        level[c] = in ? p.u[0][i] : (T)0, level[own_cells + c] = in ? p.u[1][i] : (T)0;
        if (COMP) increment[c] = in ? p.air.d[i] : (T)0;
        if (SCALED) scale[c] = in ? p.air.scale[i] : 0.0f;
    }
    const uint32_t rows = p.row_start[rank + 1] - p.row_start[rank], quads = p.quad_start[rank + 1] - p.quad_start[rank];
    for (uint32_t k = threadIdx.x; k < rows; k += kThreads) {
        const uint4 e = p.rows[p.row_start[rank] + k];
        const uint32_t r = e.x, i = g.special[r], n = e.w & 255u, m = e.w >> 8, l0 = p.link_start[r], s0 = g.state_start[r];
        row[k] = make_uint4(local(i), r, e.y | n << 24, e.z | m << 24);
        coef[k] = make_float4(g.coef_a[r], g.coef_b[r], g.coef_inv[r], g.source[r]);
        if (COMP) residual[k] = g.row_residual[r];
        for (uint32_t l = 0; l < n; ++l) {
            const uint2 from = p.links[l0 + l];
            link[e.y + l] = make_uint2(from.x, address(i + from.y));
        }
        for (uint32_t j = 0; j < m; ++j) {
            state[e.z + j] = make_float4(g.state_weight[s0 + j], g.state_now[s0 + j], g.state_before[s0 + j], g.state_gain[s0 + j]);
            w[e.z + j] = p.w[0][s0 + j], w[p.most_states + e.z + j] = p.w[1][s0 + j];
        }
    }
    for (uint32_t k = threadIdx.x; k < p.steps; k += kThreads) drive[k] = p.signal[k];
    // The rows on the first warps, the quads after them; a thread's first quad's neighbours are found once.
    const uint32_t row_slots = (rows + 31) / 32 * 32;
    const Update<T, false, SCALED, COMP> update{(T)p.air.axial, (T)p.air.diagonal, (T)p.air.centre, (T)p.air.total,
                                                (T)p.air.residual};
    struct Around {
        uint32_t cell, mask, left, right, ym, yp, zm, zp;
    };
    auto around = [&](uint32_t k) {
        const uint2 q = p.air.columns[p.quad_start[rank] + k];
        const uint32_t i = q.x;
        return Around{local(i), q.y, address(i - 1), address(i + 4), address(i - g.pitch), address(i + g.pitch),
                      address(i - g.plane), address(i + g.plane)};
    };
    uint32_t my_slot = row_slots / kThreads * kThreads + threadIdx.x;  // (the thread's first slot past the rows)
    if (my_slot < row_slots) my_slot += kThreads;
    Around mine{};
    if (my_slot < row_slots + quads) mine = around(my_slot - row_slots);
    // The block's share of the probes' cells, kept for probe_steps steps and then written out together (a
    // store to global memory would hold up each step's barrier).
    const uint32_t reads0 = min(rank * p.most_reads, p.gathered_count), reads = min(p.most_reads, p.gathered_count - reads0);
    T *kept = reinterpret_cast<T *>(smem + p.reads_at);
    const uint32_t my_read = kThreads - 1 - threadIdx.x;
    const uint32_t my_read_at = my_read < reads ? address(g.probe_cells[reads0 + my_read]) : 0u;
    cluster_barrier();
    for (uint32_t step = 0; step < p.steps; ++step) {
        const uint32_t cur = 1u - (step & 1u), now = cur * level_bytes;
        const T *b = level + cur * own_cells;
        T *a = level + (1u - cur) * own_cells;
        for (uint32_t t = threadIdx.x; t < row_slots + quads; t += kThreads) {
            if (t >= row_slots) {
                const Around q = t == my_slot ? mine : around(t - row_slots);
                Quad<T> ym, yp, zm, zp, next, delta, sc;
                T left, right;
                load_cluster(q.zm + now, zm), load_cluster(q.zp + now, zp);
                load_cluster(q.ym + now, ym), load_cluster(q.yp + now, yp);
                load_cluster(q.left + now, left), load_cluster(q.right + now, right);
                if (SCALED) {
                    const float4 s = *reinterpret_cast<const float4 *>(scale + q.cell);
                    sc = {{(T)s.x, (T)s.y, (T)s.z, (T)s.w}};
                }
                update(load_quad(b + q.cell), left, right, ym, yp, zm, zp, load_quad(COMP ? increment + q.cell : a + q.cell), sc,
                       [](int, T) { return (T)0; }, next, delta);
                store_cells<false>(a + q.cell, next, q.mask);
                if (COMP) store_cells<false>(increment + q.cell, delta, q.mask);
                continue;
            }
            if (t >= rows) continue;
            const uint4 e = row[t];
            const uint32_t l0 = e.z & 0xffffffu, n = e.z >> 24, s0 = e.w & 0xffffffu, s1 = s0 + (e.w >> 24);
            const float4 c = coef[t];
            const T here = b[e.x], previous = COMP ? increment[e.x] : a[e.x];
            // (Six links at once, most rows' all, the states' flow while they are on their way.)
            T value[6], weight[6];
#pragma unroll
            for (int l = 0; l < 6; ++l) {
                value[l] = weight[l] = (T)0;
                if ((uint32_t)l < n) {
                    const uint2 k = link[l0 + l];
                    load_cluster(k.y + now, value[l]);
                    weight[l] = (T)__uint_as_float(k.x);
                }
            }
            T *wa = w + (1u - cur) * p.most_states;
            const T *wb = w + cur * p.most_states;
            T flow = 0;
#pragma unroll 2
            for (uint32_t j = s0; j < s1; ++j) {
                const float4 k = state[j];
                const T own = (T)k.y * wb[j] - (T)k.z * wa[j];
                flow += (T)k.x * own;
            }
            T sum = 0;
#pragma unroll
            for (int l = 0; l < 6; ++l)
                if ((uint32_t)l < n) sum += COMP ? weight[l] * (value[l] - here) : weight[l] * value[l];
            for (uint32_t l = 6; l < n; ++l) {
                const uint2 k = link[l0 + l];
                T v;
                load_cluster(k.y + now, v);
                const T x = (T)__uint_as_float(k.x);
                sum += COMP ? x * (v - here) : x * v;
            }
            T change;
            const T push = (T)c.w * (T)drive[step];
            if (COMP) {
                const T delta = (sum + (T)c.y * previous - flow + push) * (T)c.z + (T)residual[t] * here;
                a[e.x] = here + delta;
                increment[e.x] = delta;
                change = delta + previous;
            } else {
                const T next = ((T)c.x * here + sum - (T)c.y * previous - flow + push) * (T)c.z;
                a[e.x] = next;
                if (p.traj_u) p.traj_u[(uint64_t)step * g.specials + e.y] = next;
                change = next - previous;
            }
            const uint32_t global_state = !COMP && p.traj_w ? g.state_start[e.y] : 0u;
#pragma unroll 2
            for (uint32_t j = s0; j < s1; ++j) {
                const float4 k = state[j];
                const T own = (T)k.y * wb[j] - (T)k.z * wa[j];
                const T v = wa[j] + (change * (T)k.w + own);
                wa[j] = v;
                if (!COMP && p.traj_w) p.traj_w[(uint64_t)step * p.states + global_state + (j - s0)] = v;
            }
        }
        const uint32_t slot = step % p.probe_steps;
        for (uint32_t e = my_read; e < reads; e += kThreads) {
            T v;
            load_cluster((e == my_read ? my_read_at : address(g.probe_cells[reads0 + e])) + now, v);
            kept[slot * p.most_reads + e] = v;
        }
        cluster_barrier();
        if (reads && (slot + 1 == p.probe_steps || step + 1 == p.steps)) {
            for (uint32_t e = threadIdx.x; e < (slot + 1) * reads; e += kThreads) {
                const uint32_t k = e / reads, c = e - k * reads;
                p.gathered[(uint64_t)(step - slot + k) * p.gathered_count + reads0 + c] = kept[k * p.most_reads + c];
            }
            __syncthreads();
        }
    }
    // Back go the cells that the block steps and no others: a solid plane may be a neighbour's ghost plane, which a
    // copy fills beside this launch.
    for (uint32_t k = threadIdx.x; k < quads; k += kThreads) {
        const uint2 q = p.air.columns[p.quad_start[rank] + k];
        const uint32_t c = local(q.x);
        store_cells<false>(p.u[0] + q.x, load_quad(level + c), q.y);
        store_cells<false>(p.u[1] + q.x, load_quad(level + own_cells + c), q.y);
        if (COMP) store_cells<false>(p.air.d + q.x, load_quad(increment + c), q.y);
    }
    for (uint32_t k = threadIdx.x; k < rows; k += kThreads) {
        const uint4 e = row[k];
        const uint32_t i = g.special[e.y];
        p.u[0][i] = level[e.x], p.u[1][i] = level[own_cells + e.x];
        if (COMP) p.air.d[i] = increment[e.x];
        const uint32_t s0 = e.w & 0xffffffu, m = e.w >> 24, to = g.state_start[e.y];
        for (uint32_t j = 0; j < m; ++j) p.w[0][to + j] = w[s0 + j], p.w[1][to + j] = w[p.most_states + s0 + j];
    }
}

}  // namespace fdtd
