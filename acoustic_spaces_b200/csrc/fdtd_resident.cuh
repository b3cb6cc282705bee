// The resident stepper: many time steps of a grid in one launch.
//
// Below some tens of millions of cells a step's launches, event waits and drained waves take longer
// than its memory traffic, which the L2 cache serves. Here one launch of as many blocks as fit the
// GPU at once (or, for the smallest grids, one cluster) takes every step of a piece of a run: each
// block keeps a fixed share of the special rows, the matched-layer cells, the interior air and the
// probes' cells, a warp takes 32 of one kind at a time, and one barrier over the blocks ends a
// step. A step reads the current level, writes the other and swaps the two by the step's parity,
// so that one barrier a step is enough. The operations of each cell are the launched kernels' own,
// in their order: the results are equal to the bit.
#pragma once

#include "fdtd_columns.cuh"

namespace fdtd {

template <typename T>
struct ResidentArgs {
    Tables g;
    T *u[2], *w[2], *layer[2];  // [1]: the current ones at the launch's start
    T *d;                       // COMP: the increments
    SweepArgs<T> air;           // the interior air's columns
    const float *signal;  // the drive of the launch's first step
    // The special rows' links row by row (their starts, then {weight, offset} each), and whether each
    // block keeps its rows' tables and branch velocities in shared memory over the steps.
    const uint32_t *link_start;
    const uint2 *links;
    uint32_t staged;
    // The layer's coefficients and, of as many tasks a block as fit (keep_layer), its state are kept in
    // shared memory too: where the rows (after the coefficients) and the state begin, and the
    // coefficients' counts along x, y and z.
    uint32_t keep_layer, rows_at, layer_at, coefs[3];
    T *layer_work;  // the other tasks' state, in the same form (nine quads a quad)
    // The probes' cells of every step, gathered in their order (summed by probe_sum_kernel).
    T *gathered;
    uint32_t gathered_count;
    // Recording (Fields): the first step's places, or null.
    T *traj_u, *traj_w, *traj_layer;
    uint32_t states;
    uint32_t steps;
    uint32_t clustered;     // the launch is one cluster: its barrier in place of the counter
    unsigned int *arrived;  // blocks arrived at the steps' barriers so far
    unsigned int *error;
};

// Every thread of the cluster has arrived, and sees what the others wrote before they did. (Not the aligned form: it
// wants a warp's threads together, and the loops before it end lane by lane.)
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
}

// Every block of the launch has done its part of a step: a count in device memory, cleared before
// the launch (`target`: the blocks times the barriers so far), or the cluster's barrier. False
// after too many tries: the block then reports the error and stops, and so do the others.
__device__ __forceinline__ bool step_barrier(unsigned int *arrived, unsigned int target, uint32_t clustered,
                                             unsigned int *error) {
    if (clustered) {
        cluster_barrier();
        return true;
    }
    int failed = 0;
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;\n" ::"l"(arrived) : "memory");
        failed = 1;
        for (uint32_t spin = 0; spin < kSpinLimit; ++spin) {
            unsigned int now;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(now) : "l"(arrived) : "memory");
            if (now >= target) {
                failed = 0;
                break;
            }
        }
        if (failed) atomicOr(error, 1u);
    }
    return !__syncthreads_or(failed);
}

// ---- the special rows ------------------------------------------------------------------------------

// A block's rows in its shared memory for the whole launch: each row's cell, coefficients and where
// its links (or, with axial links alone, their mask) and branch states lie; the links, the states'
// coefficients and the states' velocities (two sets, as the levels). A barrier leaves nothing of the
// tables in the multiprocessor's cache, and a row read from L2 waits for its cell, then its links'
// directions, then its pressures, and once for every branch state; from shared memory it waits for
// the pressures alone.
template <typename T>
struct RowStage {
    float4 *coef;   // a, b, inv, source
    float4 *state;  // weight, now, before, gain
    T *w;           // [2][states]
    uint2 *link;    // {weight, offset}
    uint32_t *cell, *link_at, *state_at;  // (link_at: the links' mask with axial links alone)
    float *residual;
    uint32_t states;
    __host__ __device__ static uint32_t bytes(uint32_t rows, uint32_t links, uint32_t states) {
        return 16 * (rows + states) + 2 * (uint32_t)sizeof(T) * states + 8 * links + 4 * (4 * rows + 2) + 16;
    }
    __device__ RowStage(unsigned char *at, uint32_t rows, uint32_t links, uint32_t n) : states(n) {
        coef = reinterpret_cast<float4 *>(at), state = coef + rows;
        w = reinterpret_cast<T *>(state + n);
        link = reinterpret_cast<uint2 *>(w + 2 * n);
        cell = reinterpret_cast<uint32_t *>(link + links);
        link_at = cell + rows, state_at = link_at + rows + 1;
        residual = reinterpret_cast<float *>(state_at + rows + 1);
    }
};

// special_row's operations, in its order, from the stage (k the block's row, r the grid's).
template <typename T, int SLOTS, bool COMP>
__device__ __forceinline__ void staged_row(const Tables &g, const RowStage<T> &m, const Fields<T> &f, uint32_t k,
                                           uint32_t cur, uint32_t r, uint32_t first_state) {
    const uint32_t i = m.cell[k];
    const T *b = f.b;
    const T here = b[i], previous = COMP ? f.d[i] : f.a[i], drive = (T)f.signal[0];
    const float4 c = m.coef[k];
    const uint32_t s0 = m.state_at[k], s1 = m.state_at[k + 1];
    constexpr int kValues = SLOTS ? SLOTS : 6;
    const uint32_t l0 = m.link_at[k], n = SLOTS ? m.link_at[k + 1] - l0 : l0;  // (the links, or their mask)
    T value[kValues];
#pragma unroll
    for (int l = 0; l < kValues; ++l) {
        if (SLOTS == 0)
            value[l] = (n >> l) & 1u ? b[i + (uint32_t)g.offset[l]] : (T)0;
        else
            value[l] = (uint32_t)l < n ? b[i + m.link[l0 + l].y] : (T)0;
    }
    // (The branch states' flow, from shared memory, while the pressures are on their way.)
    T *wa = m.w + (1u - cur) * m.states;
    const T *wb = m.w + cur * m.states;
    T flow = 0;
#pragma unroll 2
    for (uint32_t j = s0; j < s1; ++j) {
        const float4 t = m.state[j];
        const T own = (T)t.y * wb[j] - (T)t.z * wa[j];
        flow += (T)t.x * own;
    }
    T sum = 0;
#pragma unroll
    for (int l = 0; l < kValues; ++l) {
        if (SLOTS == 0) {
            const T w = (T)g.link_axial;
            if ((n >> l) & 1u) sum += COMP ? w * (value[l] - here) : w * value[l];
        } else if ((uint32_t)l < n) {
            const T w = (T)__uint_as_float(m.link[l0 + l].x);
            sum += COMP ? w * (value[l] - here) : w * value[l];
        }
    }
    T change;
    if (COMP) {
        const T step = (sum + (T)c.y * previous - flow + (T)c.w * drive) * (T)c.z + (T)m.residual[k] * here;
        f.a[i] = here + step;
        f.d[i] = step;
        change = step + previous;
    } else {
        const T next = ((T)c.x * here + sum - (T)c.y * previous - flow + (T)c.w * drive) * (T)c.z;
        f.a[i] = next;
        if (f.traj_u) f.traj_u[r] = next;
        change = next - previous;
    }
#pragma unroll 2
    for (uint32_t j = s0; j < s1; ++j) {
        const float4 t = m.state[j];
        const T own = (T)t.y * wb[j] - (T)t.z * wa[j];
        const T w = wa[j] + (change * (T)t.w + own);
        wa[j] = w;
        if (!COMP && f.traj_w) f.traj_w[first_state + j] = w;
    }
}

// ---- the steps -------------------------------------------------------------------------------------

// Threads a block, one block a multiprocessor: the registers a column or a layer's quad takes set it.
template <typename T, bool WIDE, bool LAYER>
constexpr int kResidentThreads = (WIDE || LAYER ? 512 : 1024) / (sizeof(T) == 8 ? 2 : 1);

// A block's share of a list, in tasks of 32 (a warp each): its first task and one past its last.
__host__ __device__ __forceinline__ uint32_t share_of(uint32_t count, uint32_t block, uint32_t blocks) {
    return (uint32_t)((uint64_t)((count + 31) / 32) * block / blocks);
}

// A layer quad's nine values in shared memory, 32 quads apart.
template <typename T>
__device__ __forceinline__ void kept_state(const T *kept, LayerState<T> &s) {
#pragma unroll
    for (int a = 0; a < 3; ++a)
        s.part[a] = load_quad(kept + a * 128), s.lo[a] = load_quad(kept + (3 + a) * 128), s.hi[a] = load_quad(kept + (6 + a) * 128);
}
template <typename T>
__device__ __forceinline__ void keep_state(T *kept, const LayerState<T> &s) {
#pragma unroll
    for (int a = 0; a < 3; ++a)
        store_quad<false>(kept + a * 128, s.part[a]), store_quad<false>(kept + (3 + a) * 128, s.lo[a]),
            store_quad<false>(kept + (6 + a) * 128, s.hi[a]);
}

template <typename T, bool WIDE, bool SCALED, bool COMP, bool LAYER>
__global__ void __launch_bounds__(kResidentThreads<T, WIDE, LAYER>, 1)
    resident_kernel(const __grid_constant__ ResidentArgs<T> p) {
    constexpr uint32_t kThreads = kResidentThreads<T, WIDE, LAYER>, kWarps = kThreads / 32;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int32_t offset[18];
    const Tables &g = p.g;
    if (threadIdx.x < 18) offset[threadIdx.x] = g.offset[threadIdx.x];
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    // The block's shares: the special rows first, then the layer's quads, the probes' cells and the
    // columns.
    auto share = [](uint32_t n, uint32_t &first) {
        first = share_of(n, blockIdx.x, gridDim.x);
        return share_of(n, blockIdx.x + 1, gridDim.x) - first;
    };
    uint32_t rows0, layer0 = 0, reads0, air0;
    const uint32_t rows = share(g.specials, rows0), layer = LAYER ? share(g.layer_quads, layer0) : 0u;
    const uint32_t reads = share(p.gathered_count, reads0), air = share(p.air.count, air0);
    const uint32_t all = rows + layer + reads + air;
    // The rows staged in shared memory.
    const uint32_t r0 = min(rows0 * 32, g.specials), r1 = min((rows0 + rows) * 32, g.specials);
    const uint32_t l0 = g.link_mask ? 0u : p.link_start[r0], l1 = g.link_mask ? 0u : p.link_start[r1];
    const uint32_t s0 = g.state_start[r0], s1 = g.state_start[r1];
    const RowStage<T> m(smem + p.rows_at, r1 - r0, l1 - l0, s1 - s0);
    if (p.staged) {
        for (uint32_t k = threadIdx.x; k <= r1 - r0; k += kThreads) {
            const uint32_t r = r0 + k;
            m.state_at[k] = g.state_start[r] - s0;
            if (!g.link_mask) m.link_at[k] = p.link_start[r] - l0;
            if (r == r1) continue;
            if (g.link_mask) m.link_at[k] = g.link_mask[r];
            m.cell[k] = g.special[r];
            m.coef[k] = make_float4(g.coef_a[r], g.coef_b[r], g.coef_inv[r], g.source[r]);
            if (COMP) m.residual[k] = g.row_residual[r];
        }
        for (uint32_t l = threadIdx.x; l < l1 - l0; l += kThreads) m.link[l] = p.links[l0 + l];
        for (uint32_t j = threadIdx.x; j < s1 - s0; j += kThreads) {
            m.state[j] = make_float4(g.state_weight[s0 + j], g.state_now[s0 + j], g.state_before[s0 + j], g.state_gain[s0 + j]);
            m.w[j] = p.w[0][s0 + j], m.w[m.states + j] = p.w[1][s0 + j];
        }
    }
    // The layer's state: nine quads a quad, its own copy of both faces on each axis as the reference
    // keeps it, 32 quads (a task's) together, slot by slot, each its own thread's alone and updated in
    // place, in shared memory or, past what fits there, in the workspace; and its coefficients.
    auto kept_at = [&](uint32_t t) {
        return t < p.keep_layer ? reinterpret_cast<T *>(smem + p.layer_at) + t * 9 * 128 + 4 * lane
                                : p.layer_work + (uint64_t)(layer0 + t) * 9 * 128 + 4 * lane;
    };
    const float4 *coef[3] = {};
    if (LAYER) {
        float4 *at = reinterpret_cast<float4 *>(smem);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            for (uint32_t x = threadIdx.x; x < p.coefs[a]; x += kThreads) at[x] = (a == 0 ? g.layer_coef_x : g.layer_coef[a])[x];
            coef[a] = at, at += p.coefs[a];
        }
        for (uint32_t t = warp; t < layer; t += kWarps) {
            const uint32_t q = (layer0 + t) * 32 + lane;
            if (q >= g.layer_quads) continue;
            const uint4 d = g.layer_quad[q];
            if (!(d.w & 15u)) continue;
            LayerState<T> s;
            load_layer(p.layer[1], g.layer_lanes, q, d, s);
            keep_state(kept_at(t), s);
        }
    }
    __syncthreads();
    // A task's entry of its list (a row's are staged); the first task's stays the same every step, and
    // the next one's is loaded while a task runs.
    auto entry = [&](uint32_t t) {
        uint4 e = make_uint4(0, 0, 0, 0);
        if (t < rows) return e;
        t -= rows;
        if (LAYER && t < layer) {
            const uint32_t q = (layer0 + t) * 32 + lane;
            return q < g.layer_quads ? __ldg(g.layer_quad + q) : e;
        }
        t -= layer;
        if (t < reads) {
            const uint32_t c = (reads0 + t) * 32 + lane;
            if (c < p.gathered_count) e.x = __ldg(g.probe_cells + c);
            return e;
        }
        const uint32_t c = (air0 + t - reads) * 32 + lane;
        if (c < p.air.count) {
            const uint2 column = __ldg(p.air.columns + c);
            e.x = column.x, e.y = column.y;
        }
        return e;
    };
    const uint4 first = warp < all ? entry(warp) : make_uint4(0, 0, 0, 0);
    for (uint32_t k = 0; k < p.steps; ++k) {
        const uint32_t cur = 1u - (k & 1u);
        Fields<T> f{};
        f.b = cur ? p.u[1] : p.u[0], f.a = cur ? p.u[0] : p.u[1];
        f.wb = cur ? p.w[1] : p.w[0], f.wa = cur ? p.w[0] : p.w[1], f.d = p.d;
        f.signal = p.signal + k;
        if (p.traj_u) f.traj_u = p.traj_u + (uint64_t)k * g.specials, f.traj_w = p.traj_w + (uint64_t)k * p.states;
        if (LAYER && p.traj_layer) f.traj_layer = p.traj_layer + (uint64_t)k * 18 * g.layer_lanes;
        uint4 here = first;
        for (uint32_t t = warp; t < all; t += kWarps) {
            const uint4 e = here;
            if (t + kWarps < all) here = entry(t + kWarps);
            if (t < rows) {
                const uint32_t r = (rows0 + t) * 32 + lane;
                if (r >= g.specials) continue;
                if (p.staged) {
                    if (g.link_mask)
                        staged_row<T, 0, COMP>(g, m, f, r - r0, cur, r, s0);
                    else if (!more_links(m.link_at[r - r0 + 1] - m.link_at[r - r0]))
                        staged_row<T, kFewLinks, COMP>(g, m, f, r - r0, cur, r, s0);
                    else
                        staged_row<T, 18, COMP>(g, m, f, r - r0, cur, r, s0);
                } else {
                    if (g.link_mask)
                        special_row<T, 0, COMP, false>(g, f, r, row_entry<0, false>(g, r), offset);
                    else
                        special_row<T, 18, COMP, false>(g, f, r, row_entry<18, false>(g, r), offset);
                }
            } else if (LAYER && t < rows + layer) {
                const uint32_t q = (layer0 + t - rows) * 32 + lane;
                if (!(e.w & 15u)) continue;
                T *kept = kept_at(t - rows);
                LayerState<T> s;
                kept_state(kept, s);
                step_layer<T, SCALED, COMP, false>(g, f, coef, q, e, s);
                keep_state(kept, s);
            } else if (t < rows + layer + reads) {
                const uint32_t c = (reads0 + t - rows - layer) * 32 + lane;
                if (c < p.gathered_count) p.gathered[(uint64_t)k * p.gathered_count + c] = f.b[e.x];
            } else if (e.y) {
                if constexpr (WIDE)
                    step_wide_column<T, SCALED, COMP>(p.air, f.b, f.a, make_uint2(e.x, e.y));
                else
                    step_column<T, SCALED, COMP>(p.air, f.b, f.a, make_uint2(e.x, e.y));
            }
        }
        if (k + 1 < p.steps && !step_barrier(p.arrived, (k + 1) * gridDim.x, p.clustered, p.error)) break;
    }
    __syncthreads();
    if (p.staged) {
        for (uint32_t j = threadIdx.x; j < s1 - s0; j += kThreads)
            p.w[0][s0 + j] = m.w[j], p.w[1][s0 + j] = m.w[m.states + j];
    }
    if (LAYER) {
        // (into the set that is the current one after the launch's steps)
        T *to = p.steps & 1u ? p.layer[0] : p.layer[1];
        for (uint32_t t = warp; t < layer; t += kWarps) {
            const uint32_t q = (layer0 + t) * 32 + lane;
            if (q >= g.layer_quads) continue;
            const uint4 d = g.layer_quad[q];
            if (!(d.w & 15u)) continue;
            LayerState<T> s;
            kept_state(kept_at(t), s);
            store_layer<false>(to, g.layer_lanes, q, d, s);
        }
    }
}

}  // namespace fdtd
