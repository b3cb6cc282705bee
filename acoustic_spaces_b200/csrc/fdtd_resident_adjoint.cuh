// The resident reverse stepper: many reverse steps of the gradient (fdtd_adjoint.cuh) in one launch, as
// the resident stepper takes the forward's. A block keeps its share of the special rows, of the cells
// formed whole, of the layer's cells and of the interior; the rows' tables, their branch states'
// adjoints and the double sums of their gradient stay in its shared memory over the steps. Every
// cell's operations are the launched kernels', in their order.
#pragma once

#include "fdtd_adjoint.cuh"
#include "fdtd_resident.cuh"

namespace fdtd {

template <typename T>
struct ReverseArgs {
    AdjointTables t;
    SweepArgs<T> sweep;
    // Each launch's first step reads lam[0] (the level after) and its companions and writes lam[1]; the
    // next the other way round.
    T *lam[2], *om[2], *tilde[2], *hat[2];
    // The trajectory and dL/dy, both by the step's number: step m reads levels m .. m + 2.
    const T *traj_u, *traj_w;
    const double *dloss;
    uint64_t stride;
    uint32_t first;  // the launch's first step's number; it counts down from there
    uint32_t steps;
    double *g_ci, *g_cb, *g_now, *g_before, *g_gain;
    LayerNext<T> next;  // (its hat and its tangent's place are set a step)
    T *waiting;         // with the tables: the steps' Q^, L^, H^ (layer_pending_kernel)
    uint32_t tangent_factors;
    uint32_t cells_at;  // where the cells formed whole begin in shared memory
    uint32_t clustered;
    unsigned int *arrived, *error;
};

// A block's rows: {cell, first reader, first state, layer mask | 128 if probes read it} each, their coefficients,
// readers, branch states and sums.
template <typename T>
struct AdjointStage {
    double *g_row;    // [2][rows]: coef_inv, coef_b
    double *g_state;  // [3][states]: now, before, gain
    float4 *state;    // weight, now, before, gain
    uint4 *row;
    T *reader_coef, *om;  // om: [2][states]
    float2 *coef;         // inv, b
    uint32_t *reader;     // bit 31: a row's L~, else a cell's adjoint
    uint32_t rows, states;
    __host__ __device__ static uint32_t bytes(uint32_t rows, uint32_t readers, uint32_t states) {
        return 16 * (rows + 1) + 40 * states + 16 * (rows + 1) + (uint32_t)sizeof(T) * (readers + 2 * states) + 8 * rows +
               4 * readers + 64;
    }
    __device__ AdjointStage(unsigned char *at, uint32_t n, uint32_t readers, uint32_t m) : rows(n), states(m) {
        row = reinterpret_cast<uint4 *>(at);
        state = reinterpret_cast<float4 *>(row + n + 1);
        g_row = reinterpret_cast<double *>(state + m);
        g_state = g_row + 2 * n;
        coef = reinterpret_cast<float2 *>(g_state + 3 * m);
        om = reinterpret_cast<T *>(coef + n);
        reader_coef = om + 2 * m;
        reader = reinterpret_cast<uint32_t *>(reader_coef + readers);
    }
};

// A block's cells formed whole: {cell, neighbours left out, first entry, layer mask | 128 if probes read it}
// each, their scales and their entries (a row, its coefficient).
template <typename T>
struct WholeStage {
    uint4 *cell;
    T *coef;
    uint32_t *row;
    float *scale;
    __host__ __device__ static uint32_t bytes(uint32_t cells, uint32_t entries) {
        return 16 * (cells + 1) + (4 + (uint32_t)sizeof(T)) * entries + 4 * cells + 64;
    }
    __device__ WholeStage(unsigned char *at, uint32_t n, uint32_t entries) {
        cell = reinterpret_cast<uint4 *>(at);
        coef = reinterpret_cast<T *>(cell + n + 1);
        row = reinterpret_cast<uint32_t *>(coef + entries);
        scale = reinterpret_cast<float *>(row + entries);
    }
};

// special_adjoint_row's operations, in its order (k the block's row, r the grid's; cur: the states' set
// of the level after).
template <typename T>
__device__ __forceinline__ void staged_adjoint_row(const ReverseArgs<T> &p, const AdjointStage<T> &m, uint32_t k, uint32_t r,
                                                   uint32_t first_state, uint32_t cur, const T *lam_next, const T *tilde,
                                                   const T *hat, T *lam_out, T *tilde_out, uint32_t step) {
    const AdjointTables &t = p.t;
    const uint4 own = m.row[k];
    const uint32_t i = own.x, s0 = own.z, s1 = m.row[k + 1].z;
    const T u_prev = p.traj_u[(uint64_t)step * t.specials + r], u_next = p.traj_u[(uint64_t)(step + 2) * t.specials + r];
    const T lam2 = lam_out[i], U = tilde[r];
    const T ci = (T)m.coef[k].x, cb = (T)m.coef[k].y;
    T *om_out = m.om + (1u - cur) * m.states;
    const T *om_next = m.om + cur * m.states;
    T gathered = 0;
    for (uint32_t e = own.y, end = m.row[k + 1].y; e < end; e += 8) {
        T value[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t at = e + j < end ? m.reader[e + j] : 0u;
            value[j] = e + j < end ? ((at >> 31) ? tilde[at & 0x7fffffffu] : lam_next[at]) : (T)0;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (e + j < end) gathered += m.reader_coef[e + j] * value[j];
    }
    T tilde2 = lam2, gain_om2 = 0;
    for (uint32_t j = s0; j < s1; ++j) {
        const T term = (T)m.state[j].w * om_out[j];
        tilde2 += term;
        gain_om2 += term;
    }
    if (own.w & 127u) gathered += layer_terms<T>(t, hat, i, own.w & 127u);
    T lam = gathered - (ci * cb * tilde2 + gain_om2);
    if (own.w & 128u) {
        const double probed = probe_terms(t, t.special_read_start[r], t.special_read_start[r + 1], p.dloss, p.stride, step);
        if (probed != 0.0) lam += (T)probed;
    }
    lam_out[i] = lam;
    T next_tilde = lam;
    m.g_row[k] += (double)U * ((double)u_next / (double)ci);
    m.g_row[m.rows + k] += -(double)U * (double)ci * (double)u_prev;
    for (uint32_t j = s0; j < s1; ++j) {
        const float4 c = m.state[j];
        const T W = (T)c.x, now = (T)c.y, before = (T)c.z;
        const T om1 = om_next[j], om2 = om_out[j];
        const T om = -ci * W * now * U + now * om1 + ci * W * before * tilde2 + ((T)1 - before) * om2;
        om_out[j] = om;
        next_tilde += (T)c.w * om;
        const double own_bar = (double)om1 - (double)W * (double)ci * (double)U;
        const uint64_t at = (uint64_t)step * t.states + first_state + j;
        const double w_n = (double)p.traj_w[at + t.states], w_prev = (double)p.traj_w[at];
        m.g_state[j] += own_bar * w_n;
        m.g_state[m.states + j] += -own_bar * w_prev;
        m.g_state[2 * m.states + j] += (double)om1 * ((double)u_next - (double)u_prev);
    }
    tilde_out[r] = next_tilde;
}

// correct_cell's operations, in its order.
template <typename T>
__device__ __forceinline__ void staged_whole_cell(const ReverseArgs<T> &p, const WholeStage<T> &m, uint32_t k, uint32_t c,
                                                  const T *lam_next, const T *tilde, const T *hat, T *lam_out,
                                                  uint32_t step) {
    const AdjointTables &t = p.t;
    const uint4 own = m.cell[k];
    const uint32_t cell = own.x, special = own.y;
    T around[6], edges = 0, sum = 0;
#pragma unroll
    for (int d = 0; d < 6; ++d) around[d] = special & (1u << d) ? (T)0 : lam_next[cell + (uint32_t)t.offset[d]];
    const T here = lam_next[cell], lam2 = lam_out[cell];
#pragma unroll
    for (int d = 0; d < 6; ++d)
        if (!(special & (1u << d))) sum += around[d];
    if (t.wide) {
#pragma unroll
        for (int d = 6; d < 18; ++d)
            if (!(special & (1u << d))) edges += lam_next[cell + (uint32_t)t.offset[d]];
    }
    T centre = (T)t.centre, axial = (T)t.axial, diagonal = (T)t.diagonal, sc = (T)1;
    if (t.corrected_scale) {
        sc = (T)m.scale[k];
        centre = (T)2 - (T)t.total * sc;
        axial = sc * (T)t.axial;
        diagonal = sc * (T)t.diagonal;
    }
    T value = centre * here + axial * sum + diagonal * edges - lam2;
    for (uint32_t e = own.z, end = m.cell[k + 1].z; e < end; ++e) value += m.coef[e] * tilde[m.row[e]];
    if (own.w & 127u) value += sc * layer_terms<T>(t, hat, cell, own.w & 127u);
    if (own.w & 128u) {
        const double probed = probe_terms(t, t.corrected_read_start[c], t.corrected_read_start[c + 1], p.dloss, p.stride, step);
        if (probed != 0.0) value += (T)probed;
    }
    lam_out[cell] = value;
}

constexpr int kReverseThreads = 512;

template <typename T, bool WIDE, bool SCALED, bool LAYER>
__global__ void __launch_bounds__(kReverseThreads, 1) reverse_kernel(const __grid_constant__ ReverseArgs<T> p) {
    constexpr uint32_t kThreads = kReverseThreads, kWarps = kThreads / 32;
    extern __shared__ __align__(128) unsigned char smem[];
    const AdjointTables &t = p.t;
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    auto share = [](uint32_t n, uint32_t &first) {
        first = share_of(n, blockIdx.x, gridDim.x);
        return share_of(n, blockIdx.x + 1, gridDim.x) - first;
    };
    uint32_t rows0, layer0 = 0, whole0, air0;
    const uint32_t rows = share(t.specials, rows0), layer = LAYER ? share(t.layers, layer0) : 0u;
    const uint32_t whole = share(t.corrected, whole0), air = share(p.sweep.count, air0);
    const uint32_t all = rows + layer + whole + air;
    // The stages.
    const uint32_t r0 = min(rows0 * 32, t.specials), r1 = min((rows0 + rows) * 32, t.specials);
    const uint32_t e0 = t.reader_start[r0], e1 = t.reader_start[r1], s0 = t.state_start[r0], s1 = t.state_start[r1];
    const AdjointStage<T> m(smem, r1 - r0, e1 - e0, s1 - s0);
    for (uint32_t k = threadIdx.x; k <= r1 - r0; k += kThreads) {
        const uint32_t r = r0 + k;
        uint4 own = make_uint4(0, t.reader_start[r] - e0, t.state_start[r] - s0, 0);
        if (r < r1) {
            own.x = t.special[r];
            own.w = (LAYER ? (uint32_t)t.special_layer_mask[r] : 0u) |
                    (t.special_read_start[r] < t.special_read_start[r + 1] ? 128u : 0u);
            m.coef[k] = make_float2(t.coef_inv[r], t.coef_b[r]);
            m.g_row[k] = p.g_ci[r], m.g_row[m.rows + k] = p.g_cb[r];
        }
        m.row[k] = own;
    }
    for (uint32_t e = threadIdx.x; e < e1 - e0; e += kThreads) {
        m.reader[e] = t.reader_index[e0 + e] | ((uint32_t)t.reader_kind[e0 + e] << 31);
        m.reader_coef[e] = (T)t.reader_coef[e0 + e];
    }
    for (uint32_t j = threadIdx.x; j < s1 - s0; j += kThreads) {
        m.state[j] = make_float4(t.state_weight[s0 + j], t.state_now[s0 + j], t.state_before[s0 + j], t.state_gain[s0 + j]);
        m.om[j] = p.om[0][s0 + j], m.om[m.states + j] = p.om[1][s0 + j];
        m.g_state[j] = p.g_now[s0 + j], m.g_state[m.states + j] = p.g_before[s0 + j];
        m.g_state[2 * m.states + j] = p.g_gain[s0 + j];
    }
    const uint32_t c0 = min(whole0 * 32, t.corrected), c1 = min((whole0 + whole) * 32, t.corrected);
    const uint32_t w0 = t.corrected ? t.corrected_start[c0] : 0u, w1 = t.corrected ? t.corrected_start[c1] : 0u;
    const WholeStage<T> n(smem + p.cells_at, c1 - c0, w1 - w0);
    if (t.corrected)
        for (uint32_t k = threadIdx.x; k <= c1 - c0; k += kThreads) {
            const uint32_t c = c0 + k;
            uint4 own = make_uint4(0, 0, t.corrected_start[c] - w0, 0);
            if (c < c1) {
                own.x = t.corrected_cell[c], own.y = t.corrected_mask[c];
                own.w = (LAYER ? (uint32_t)t.corrected_layer_mask[c] : 0u) |
                        (t.corrected_read_start[c] < t.corrected_read_start[c + 1] ? 128u : 0u);
                if (t.corrected_scale) n.scale[k] = t.corrected_scale[c];
            }
            n.cell[k] = own;
        }
    for (uint32_t e = threadIdx.x; e < w1 - w0; e += kThreads) {
        n.row[e] = t.corrected_row[w0 + e];
        n.coef[e] = (T)t.corrected_coef[w0 + e];
    }
    __syncthreads();
    for (uint32_t j = 0; j < p.steps; ++j) {
        const uint32_t cur = j & 1u, step = p.first - j;
        const T *lam_next = cur ? p.lam[1] : p.lam[0], *tilde = cur ? p.tilde[1] : p.tilde[0];
        T *lam_out = cur ? p.lam[0] : p.lam[1], *tilde_out = cur ? p.tilde[0] : p.tilde[1];
        const T *hat = LAYER ? (cur ? p.hat[1] : p.hat[0]) : nullptr;
        for (uint32_t k = warp; k < all; k += kWarps) {
            if (k < rows) {
                const uint32_t r = (rows0 + k) * 32 + lane;
                if (r < t.specials) staged_adjoint_row<T>(p, m, r - r0, r, s0, cur, lam_next, tilde, hat, lam_out, tilde_out, step);
            } else if (k < rows + whole) {
                const uint32_t c = (whole0 + k - rows) * 32 + lane;
                if (c < t.corrected) staged_whole_cell<T>(p, n, c - c0, c, lam_next, tilde, hat, lam_out, step);
            } else if (LAYER && k < rows + whole + layer) {
                const uint32_t c = (layer0 + k - rows - whole) * 32 + lane;
                // (With the tables, Q^, L^, H^ wait for the launch's end, those of the step before the
                // segment for that segment; along a tangent, the products with the step's factors.)
                LayerNext<T> next = p.next;
                next.hat = cur ? p.hat[0] : p.hat[1];
                if (step > 0) {
                    next.pending = p.waiting ? p.waiting + (uint64_t)j * 9 * t.layers : nullptr;
                    if (next.tangent_base) next.tangent_offset = (uint64_t)(step - 1) * p.tangent_factors;
                }
                layer_adjoint_cell<T>(t, c, lam_next, tilde, hat, lam_out, p.dloss, p.stride, step, next);
            } else {
                const uint32_t c = (air0 + k - rows - whole - layer) * 32 + lane;
                if (c < p.sweep.count) {
                    const uint2 column = __ldg(p.sweep.columns + c);
                    if constexpr (WIDE)
                        step_wide_column<T, SCALED, false>(p.sweep, lam_next, lam_out, column);
                    else
                        step_column<T, SCALED, false>(p.sweep, lam_next, lam_out, column);
                }
            }
        }
        if (j + 1 < p.steps && !step_barrier(p.arrived, (j + 1) * gridDim.x, p.clustered, p.error)) break;
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < r1 - r0; k += kThreads) p.g_ci[r0 + k] = m.g_row[k], p.g_cb[r0 + k] = m.g_row[m.rows + k];
    for (uint32_t j = threadIdx.x; j < s1 - s0; j += kThreads) {
        p.om[0][s0 + j] = m.om[j], p.om[1][s0 + j] = m.om[m.states + j];
        p.g_now[s0 + j] = m.g_state[j], p.g_before[s0 + j] = m.g_state[m.states + j];
        p.g_gain[s0 + j] = m.g_state[2 * m.states + j];
    }
}

}  // namespace fdtd
