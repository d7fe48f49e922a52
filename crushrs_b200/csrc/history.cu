// history.cu — time histories on the device, recorded inside the step
// sequence every history_steps steps (src/solver.rs:283-286 and :349-358), so
// a run that records every step needs no device-to-host copy per step.
#include "history.cuh"

namespace crush {

namespace {

constexpr int HIST_TPB = 256;

// Warp per (part unit, chunk): the chunk's sums into partial[pu][chunk]; where
// a context has long part units, a block per chunk of those (and of every
// eighth of the others, for eight chunks).
__global__ void __launch_bounds__(HIST_TPB) k_hist_parts(HistoryArrays h, NodeArrays nd, const Control* ctls,
                                                         const double* __restrict__ f_ext, int mode, const double* __restrict__ f_ext_odd) {
    __shared__ double sh[HIST_PART_VALUES * HIST_TREE];
    static_assert(HIST_TPB == HIST_TREE && HIST_BLOCKS % (HIST_TPB / 32) == 0, "a column per thread, a block's chunks of one part");
    const int first = h.any_long ? blockIdx.x : blockIdx.x * (HIST_TPB / 32);  // the block's first (part unit, chunk)
    const int pu = first / HIST_BLOCKS, b = first % HIST_BLOCKS;
    const bool is_long = h.any_long && hist_long(h, pu);
    if (h.any_long && !is_long && b % (HIST_TPB / 32) != 0) return;  // block-uniform, as the next
    const int slot = h.pu_slot[pu];
    if (!hist_due(h, ctls + slot, slot, mode)) return;
    const bool odd = mode == HIST_FINAL && f_ext_odd && ((ctls[slot].step - 1) & 1);
    if (is_long) hist_part_block(h, nd, odd ? f_ext_odd : f_ext, pu, b, sh);
    else hist_part_warp(h, nd, odd ? f_ext_odd : f_ext, pu, b + (threadIdx.x >> 5), threadIdx.x & 31);
}

// Block per slot: the record's part states (a warp per part), accelerometer
// samples, its time and step, and the slot's record count.
__global__ void __launch_bounds__(HIST_TPB) k_hist_finish(HistoryArrays h, NodeArrays nd, const Control* ctls,
                                                          const double* __restrict__ f_ext, int mode, const double* __restrict__ f_ext_odd) {
    const int slot = blockIdx.x;
    const Control* ctl = ctls + slot;
    if (!hist_due(h, ctl, slot, mode)) return;  // block-uniform
    if (mode == HIST_FINAL && f_ext_odd && ((ctl->step - 1) & 1)) f_ext = f_ext_odd;
    const long long r = h.rec_count[slot];
    const bool keep = r < h.slot_max[slot];
    if (keep) {
        for (int pu = h.slot_pu_off[slot] + (threadIdx.x >> 5); pu < h.slot_pu_off[slot + 1]; pu += HIST_TPB / 32)
            hist_finish_warp(h, pu, r, threadIdx.x & 31);
        for (int j = h.slot_an_off[slot] + threadIdx.x; j < h.slot_an_off[slot + 1]; j += HIST_TPB) hist_node(h, nd, f_ext, j, r);
    }
    __syncthreads();  // every thread has read rec_count
    if (threadIdx.x == 0) {
        if (keep) {
            h.rec_time[(long long)slot * h.max_rec + r] = ctl->t;
            h.rec_step[(long long)slot * h.max_rec + r] = ctl->step;
        }
        h.rec_count[slot] = r + 1;
        h.last_step[slot] = ctl->step;
    }
}

}  // namespace

void launch_history(cudaStream_t s, const HistoryArrays& h, const NodeArrays& nd, const Control* ctls, const double* f_ext, int mode,
                    const double* f_ext_odd) {
    if (h.n_pu > 0)
        k_hist_parts<<<(unsigned)(h.n_pu * HIST_BLOCKS / (h.any_long ? 1 : HIST_TPB / 32)), HIST_TPB, 0, s>>>(h, nd, ctls, f_ext, mode,
                                                                                                          f_ext_odd);
    k_hist_finish<<<(unsigned)h.n_slots, HIST_TPB, 0, s>>>(h, nd, ctls, f_ext, mode, f_ext_odd);
}

}  // namespace crush
