// history.cuh — device code of the time histories: per-part states and
// accelerometer node samples (src/solver.rs:114-187 part_states and
// sample_accelerometers), shared by the record kernels and the resident step
// kernel.
#pragma once
#include "kernels.cuh"

namespace crush {
namespace {

constexpr int HIST_TREE = 256;  // columns of the part sums' tree
static_assert(HIST_LONG == HIST_BLOCKS * HIST_TREE, "a node per column");

// Whether slot `slot` takes a record now: its run's first record, a step
// that is a multiple of history_steps, or the last step of a finished crash;
// never twice at one step.
template <class C>
__device__ __forceinline__ bool hist_due(const HistoryArrays& h, const C* ctl, int slot, int mode) {
    if (!h.slot_on[slot]) return false;
    if (mode == HIST_INITIAL) return true;
    if (ctl->step == h.last_step[slot]) return false;
    return mode == HIST_FINAL ? ctl->done != 0 : ctl->step % h.steps == 0;
}

// Nodal acceleration (net force / mass, with the added mass of mass
// scaling), zero at fixed nodes (src/solver.rs:333-341).
__device__ __forceinline__ double hist_acc(const NodeArrays& nd, const double* f_ext, long long n, int d) {
    if (nd.fixed[n]) return 0.0;
    const long long k = 3 * n + d;
    return (f_ext[k] - nd.f_int[k]) * nd.inv_mass[n];
}

__device__ __forceinline__ void cross3(const double* a, const double* b, double* c) {
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
}
__device__ __forceinline__ double norm3(const double* a) { return sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]); }

// Body-fixed axes from three nodes at X + u (LocalFrame::axes,
// src/model.rs:45-61): e1 along origin -> x_axis, e3 normal to the plane of
// e1 and origin -> plane, e2 = e3 x e1; degenerate inputs fall back to the
// global axes as there. Rows are the axes.
__device__ void frame_axes(const NodeArrays& nd, const uint32_t* fn, double ax[3][3]) {
    double o[3], e1[3], p[3];
    for (int d = 0; d < 3; ++d) {
        o[d] = nd.pos[3ll * fn[0] + d] + nd.u[3ll * fn[0] + d];
        e1[d] = (nd.pos[3ll * fn[1] + d] + nd.u[3ll * fn[1] + d]) - o[d];
        p[d] = (nd.pos[3ll * fn[2] + d] + nd.u[3ll * fn[2] + d]) - o[d];
    }
    if (norm3(e1) < 1e-300) {
        e1[0] = 1.0;
        e1[1] = 0.0;
        e1[2] = 0.0;
    }
    const double n1 = norm3(e1);
    for (int d = 0; d < 3; ++d) e1[d] /= n1;
    double c[3];
    cross3(p, e1, c);
    if (norm3(c) < 1e-12 * fmax(norm3(p), 1e-300)) {
        const bool use_x = fabs(e1[0]) < 0.9;
        p[0] = use_x ? 1.0 : 0.0;
        p[1] = use_x ? 0.0 : 1.0;
        p[2] = 0.0;
    }
    double e3[3], e2[3];
    cross3(e1, p, e3);
    const double n3 = norm3(e3);
    for (int d = 0; d < 3; ++d) e3[d] /= n3;
    cross3(e3, e1, e2);
    for (int d = 0; d < 3; ++d) {
        ax[0][d] = e1[d];
        ax[1][d] = e2[d];
        ax[2][d] = e3[d];
    }
}

// Accumulators of the part sums: mass, momentum-like sums and kinetic energy.
struct HistSums {
    double a[HIST_PART_VALUES];
};
__device__ __forceinline__ void hist_add(HistSums& x, const HistSums& y) {
#pragma unroll
    for (int k = 0; k < HIST_PART_VALUES; ++k) x.a[k] += y.a[k];
}
// Nodes i, i + HIST_TREE, ... below i1 of the unit's list.
__device__ __forceinline__ HistSums hist_column(const HistoryArrays& h, const NodeArrays& nd, const double* f_ext, long long i, long long i1) {
    HistSums s;
#pragma unroll
    for (int k = 0; k < HIST_PART_VALUES; ++k) s.a[k] = 0.0;
    for (; i < i1; i += HIST_TREE) {
        const long long n = h.pu_nodes[i];
        const double m = nd.mass[n];
        s.a[0] += m;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double v = nd.v[3 * n + d];
            s.a[1 + d] += m * v;
            s.a[4 + d] += m * nd.u[3 * n + d];
            s.a[7 + d] += m * hist_acc(nd, f_ext, n, d);
            s.a[10] += 0.5 * m * v * v;
        }
    }
    return s;
}

// Partial sums of chunk b of part unit pu by one warp: HIST_TREE columns of
// nodes added in a fixed binary tree (column c and c + HIST_TREE / 2 first,
// neighbours last). Lane l holds columns l + 32 j; the tree over j runs in its
// registers, two columns at a time, and the tree over the lanes by shuffles.
// Bound by the latency of one round of node loads (a vehicle's part has 10-40
// nodes per chunk, so one column per lane): a warp per chunk takes 7.1 us for
// the 126 units of 18 barrier probes, a block with the tree in shared memory
// took 30.5 us.
__device__ __forceinline__ void hist_part_warp(const HistoryArrays& h, const NodeArrays& nd, const double* f_ext, int pu, int b, int lane) {
    const long long lo = h.pu_off[pu], len = (long long)h.pu_off[pu + 1] - lo;
    const long long per = (len + HIST_BLOCKS - 1) / HIST_BLOCKS;
    const long long i0 = lo + b * per, i1 = min(lo + len, i0 + per);
    HistSums s = hist_column(h, nd, f_ext, i0 + lane, i1);
    static_assert(HIST_TREE == 256, "eight columns per lane");
    if (i1 - i0 > 32) {  // warp-uniform; below, the other columns are empty (+ 0.0)
        hist_add(s, hist_column(h, nd, f_ext, i0 + lane + 128, i1));
        HistSums t = hist_column(h, nd, f_ext, i0 + lane + 64, i1);
        hist_add(t, hist_column(h, nd, f_ext, i0 + lane + 192, i1));
        hist_add(s, t);
        HistSums o = hist_column(h, nd, f_ext, i0 + lane + 32, i1);
        hist_add(o, hist_column(h, nd, f_ext, i0 + lane + 160, i1));
        t = hist_column(h, nd, f_ext, i0 + lane + 96, i1);
        hist_add(t, hist_column(h, nd, f_ext, i0 + lane + 224, i1));
        hist_add(o, t);
        hist_add(s, o);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int k = 0; k < HIST_PART_VALUES; ++k) s.a[k] += __shfl_down_sync(0xffffffffu, s.a[k], off);
    if (lane == 0) {
        double* o = h.partial + ((long long)pu * HIST_BLOCKS + b) * HIST_PART_VALUES;
#pragma unroll
        for (int k = 0; k < HIST_PART_VALUES; ++k) o[k] = s.a[k];
    }
}

// The same sums by HIST_TREE threads, a column each, for the part units of
// large meshes (more than HIST_LONG nodes): a warp's lanes would each add eight
// columns of many nodes one after the other. `sh`: HIST_PART_VALUES x HIST_TREE
// doubles. A step of 279,936 elements with a record takes 161 us, 259 us by
// warps (126 without a record); of 55,566 elements 47 and 71 (38).
__device__ __forceinline__ bool hist_long(const HistoryArrays& h, int pu) { return h.pu_off[pu + 1] - h.pu_off[pu] > (uint32_t)HIST_LONG; }
__device__ __forceinline__ void hist_sync() { asm volatile("bar.sync 1, %0;" ::"n"(HIST_TREE) : "memory"); }
__device__ __noinline__ void hist_part_block(const HistoryArrays& h, const NodeArrays& nd, const double* f_ext, int pu, int b, double* sh) {
    const long long lo = h.pu_off[pu], len = (long long)h.pu_off[pu + 1] - lo;
    const long long per = (len + HIST_BLOCKS - 1) / HIST_BLOCKS;
    const long long i0 = lo + b * per, i1 = min(lo + len, i0 + per);
    const HistSums s = hist_column(h, nd, f_ext, i0 + threadIdx.x, i1);
#pragma unroll
    for (int k = 0; k < HIST_PART_VALUES; ++k) sh[k * HIST_TREE + threadIdx.x] = s.a[k];
    hist_sync();
    const int lane = threadIdx.x & 31;
    for (int k = threadIdx.x >> 5; k < HIST_PART_VALUES; k += HIST_TREE / 32) {
        const double* c = sh + k * HIST_TREE + lane;
        double x = ((c[0] + c[128]) + (c[64] + c[192])) + ((c[32] + c[160]) + (c[96] + c[224]));
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
        if (lane == 0) h.partial[((long long)pu * HIST_BLOCKS + b) * HIST_PART_VALUES + k] = x;
    }
    hist_sync();  // sh is free again
}

// Record r of part unit pu by one warp: lane k < HIST_PART_VALUES adds value k
// of the chunks in order (its loads all in flight), then divides the means by
// the mass as src/solver.rs:131-139 does. A record of 18 barrier probes takes
// 5.6 us, one thread per part took 13.7 us.
__device__ __forceinline__ void hist_finish_warp(const HistoryArrays& h, int pu, long long r, int lane) {
    double s = 0.0;
    if (lane < HIST_PART_VALUES) {
        const double* p = h.partial + (long long)pu * HIST_BLOCKS * HIST_PART_VALUES + lane;
        double x[HIST_BLOCKS];
#pragma unroll
        for (int b = 0; b < HIST_BLOCKS; ++b) x[b] = p[b * HIST_PART_VALUES];
#pragma unroll
        for (int b = 0; b < HIST_BLOCKS; ++b) s += x[b];
    }
    const double mass = __shfl_sync(0xffffffffu, s, 0);
    const double inv = mass > 0.0 ? 1.0 / mass : 0.0;
    if (lane < HIST_PART_VALUES) h.part_rec[((long long)pu * h.max_rec + r) * HIST_PART_VALUES + lane] = lane > 0 && lane < 10 ? s * inv : s;
}

// Record r of accelerometer node j.
__device__ __forceinline__ void hist_node(const HistoryArrays& h, const NodeArrays& nd, const double* f_ext, int j, long long r) {
    const long long n = h.an_node[j];
    double x[3], u[3], v[3], a[3];
    for (int d = 0; d < 3; ++d) {
        u[d] = nd.u[3 * n + d];
        x[d] = nd.pos[3 * n + d] + u[d];
        v[d] = nd.v[3 * n + d];
        a[d] = hist_acc(nd, f_ext, n, d);
    }
    double* o = h.node_rec + ((long long)j * h.max_rec + r) * HIST_NODE_VALUES;
    for (int d = 0; d < 3; ++d) {
        o[d] = x[d];
        o[3 + d] = u[d];
        o[6 + d] = v[d];
        o[9 + d] = a[d];
    }
    const int f = h.an_frame[j];
    if (f < 0) {
        for (int d = 0; d < 3; ++d) {
            o[12 + d] = u[d];
            o[15 + d] = v[d];
            o[18 + d] = a[d];
        }
    } else {
        double ax[3][3];
        frame_axes(nd, h.fr_nodes + 3ll * f, ax);
        for (int i = 0; i < 3; ++i) {  // rotate, src/solver.rs:143-145
            o[12 + i] = ax[i][0] * u[0] + ax[i][1] * u[1] + ax[i][2] * u[2];
            o[15 + i] = ax[i][0] * v[0] + ax[i][1] * v[1] + ax[i][2] * v[2];
            o[18 + i] = ax[i][0] * a[0] + ax[i][1] * a[1] + ax[i][2] * a[2];
        }
    }
}

}  // namespace
}  // namespace crush
