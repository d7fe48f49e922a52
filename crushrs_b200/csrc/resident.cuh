// resident.cuh — the whole step loop of a small context in one kernel
// (included by kernels.cu, whose per-entity functions it calls).
//
// A crash of a few thousand elements is bound by latency: its step is a chain
// of seven kernels that each wait a few microseconds for memory with most of
// the chip idle, plus the gaps between them. Here a cooperative grid of one
// block per SM stays resident for many steps. A step is three phases with a
// grid barrier after each, one more at a stable-dt check and two more when a
// contact has a dynamic grid:
//   gather   the contact reactions of a node and its half step
//   forces   the element forces beside the faces' geometry at the new X + u
//   full     the full update beside the contact search, which emits the next
//            step's reaction events at once (its dt is known unless a
//            stable-dt check or a reduction stop rule comes first)
// The end of a step (and the stable-dt decision) runs in the last block to
// arrive at the step's last barrier, before it lets the others go. Work is
// dealt to warps in tasks of 32 threads, neighbouring tasks to different SMs,
// so that a few tasks use as many SMs as there are. The arithmetic and its
// order are those of the separate kernels (the same functions), so a run may
// change between the two at any step and its bits do not depend on it.
//
// Bound by latency: a barrier takes 1.4 us, a phase three to eight dependent
// reads of L2 (a barrier empties L1) and one warp's instruction stream. A
// step of the 1290-element head-on takes 18 us, 33 us as a graph of kernels
// (20,176 elements: 25 against 46 us). On a plain step (no stable-dt check, no
// reduction stop rule) every block advances its own copy of the crashes'
// time and done flags in shared memory, which keeps the step's end (1.8 us
// between two barriers) and a read of the control block per phase off the path.
#pragma once

// Threads per block: 256 with up to 255 registers each while an element per
// thread and a warp per searched entry fit, else 512 with 128 (launch_resident).
constexpr int RES_SMALL = 256, RES_LARGE = 512;
constexpr int RES_ST_LANES = 4;       // lanes per static-grid entry (as many as emit a hit's events)
constexpr int RES_GRID_LANES = 32;    // lanes per dynamic-grid entry
// Grid barrier: every block adds one to `count` and waits until all have.
// With a serial part, the last block to arrive runs it, with everything the
// others wrote before it visible, and lets them go by `gen`. Without one, the
// blocks watch the count itself, a round trip less. False when a block gave up
// waiting: every block then leaves the kernel (those that did not see it give
// up at their next barrier, which the ones that left never reach). A barrier
// that some block passed had every block arrive, so a launch that gives up
// leaves one phase half done and nothing of the next.
struct ResidentBarrier {
    ResidentSync* y;
    int limit;  // polls before a block gives up
    unsigned target, gen;

    __device__ __forceinline__ int wait(const unsigned* word, unsigned want) {
        for (int polls = 0; polls < limit; ++polls) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
            if ((int)(v - want) >= 0) return 1;
        }
        y->error = 1;
        return 0;
    }
    __device__ __forceinline__ unsigned arrive() {
        unsigned k;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(k) : "l"(&y->count) : "memory");
        return k;
    }
    __device__ __forceinline__ bool operator()() {
        __syncthreads();
        target += gridDim.x;
        int ok = 1;
        if (threadIdx.x == 0) {
            arrive();
            ok = wait(&y->count, target);
        }
        return __syncthreads_and(ok);
    }
    template <class Serial>
    __device__ __forceinline__ bool operator()(int* s_state, Serial serial) {
        __syncthreads();
        target += gridDim.x;
        ++gen;
        if (threadIdx.x == 0) *s_state = arrive() == target - 1;
        __syncthreads();
        int ok = 1;
        if (*s_state) {
            serial();
            __syncthreads();
            if (threadIdx.x == 0) asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&y->gen), "r"(gen) : "memory");
        } else if (threadIdx.x == 0) {
            ok = wait(&y->gen, gen);
        }
        return __syncthreads_and(ok);
    }
};

// Warp tasks of one job: tasks [0, n) dealt round-robin over the grid's
// warps, starting where the phase's jobs before it stopped.
struct TaskDeal {
    int gw, warps, base;
    template <class F>
    __device__ __forceinline__ void operator()(int n, F f) {
        int t = gw - base % warps;
        if (t < 0) t += warps;
        for (; t < n; t += warps) f(t);
        base += n;
    }
};

// One entry of an exhaustively searched contact by a warp: the lanes test the
// boxes of its faces (each lane's loads in flight together) and list the faces
// that pass in `cand`; then the narrow tests of the list run one per lane, so
// that their long f64 chains run side by side however the candidates fall, and
// the smallest face that hits wins (every lane returns it, -1 for none).
// BRUTE_MAX_FACES faces at most: a byte each.
constexpr int RES_BOX_BATCH = 4;
__device__ __forceinline__ int resident_brute(const ContactArrays& ca, const NodeArrays& nd, const ControlView* view, const BruteEntry& be,
                                              int lane, uint8_t* cand, double* sd_out) {
    const long long n = be.node, s = be.s;
    const double p[3] = {nd.pos[3 * n] + nd.u[3 * n], nd.pos[3 * n + 1] + nd.u[3 * n + 1], nd.pos[3 * n + 2] + nd.u[3 * n + 2]};
    const double md = ca.max_distance[be.contact];
    const int nf = be.n_faces;
    const FaceGeo* geo = ca.geo + be.face0;
    if (view[be.slot].done) return -1;  // warp-uniform
    int count = 0;
    for (int f0 = 0; f0 < nf; f0 += 32 * RES_BOX_BATCH) {
        bool in[RES_BOX_BATCH];
#pragma unroll
        for (int k = 0; k < RES_BOX_BATCH; ++k) {
            const int f = f0 + 32 * k + lane;
            const FaceGeo& g = geo[f < nf ? f : 0];
            const double l0 = g.lo[0], l1 = g.lo[1], l2 = g.lo[2], h0 = g.hi[0], h1 = g.hi[1], h2 = g.hi[2];
            in[k] = f < nf && !(p[0] < l0 || p[0] > h0 || p[1] < l1 || p[1] > h1 || p[2] < l2 || p[2] > h2);
        }
#pragma unroll
        for (int k = 0; k < RES_BOX_BATCH; ++k) {
            const unsigned m = __ballot_sync(0xffffffffu, in[k]);
            if (in[k]) cand[count + __popc(m & ((1u << lane) - 1u))] = (uint8_t)(f0 + 32 * k + lane);
            count += __popc(m);
        }
    }
    __syncwarp();
    int best = INT_MAX;
    double best_sd = 0.0;
    for (int k = lane; k < count; k += 32) {  // ascending: a lane's first hit is its smallest
        const int f = cand[k];
        double sd;
        if (face_hit(geo[f], p, md, &sd)) {
            best = f;
            best_sd = sd;
            break;
        }
    }
    __syncwarp();  // the list is free again
    const int first = __reduce_min_sync(0xffffffffu, best);
    if (first == INT_MAX) {
        if (lane == 0) ca.hit[s] = -1;
        return -1;
    }
    const int owner = __ffs(__ballot_sync(0xffffffffu, best == first)) - 1;
    *sd_out = __shfl_sync(0xffffffffu, best_sd, owner);
    if (lane == 0) {
        ca.hit[s] = first;
        ca.hit_sd[s] = *sd_out;
    }
    return first;
}

// The next step's force and events of a hit just found: `best` is lane 0's of
// the LANES lanes that share entry s (every lane of the warp calls).
template <int LANES>
__device__ __forceinline__ void resident_emit(const ContactArrays& ca, const ControlView* view, const double* masses, long long s, int best,
                                              double sd, int lane) {
    best = __shfl_sync(0xffffffffu, best, 0, LANES);
    sd = __shfl_sync(0xffffffffu, sd, 0, LANES);
    if (best < 0 || lane >= FORCE_LANES) return;
    const int c = ca.slave_contact[s];
    const ControlView* ctl = view + ca.contact_slot[c];
    if (last_step_by_count_or_time(ctl)) return;  // stops here: takes no next step
    record_hit(ca, s, c, ca.slaves[s], best, sd, next_step_dt(ctl), masses, ca.geo[ca.face_off[c] + best], 1, lane);
}

// A node's contact reactions (unless it is heavy), then its half step
// (half_body's arithmetic). Only contact nodes have external forces.
__device__ __forceinline__ void resident_gather_half(const ContactArrays& ca, const NodeArrays& nd, const ControlView* view,
                                                     const uint32_t* node_cn, long long n) {
    if (n >= nd.n) return;
    const uint32_t cn = node_cn[n];
    const ControlView* ctl = view + nd.node_slot[n];
    const bool fixed = nd.fixed[n] != 0;
    const double im = nd.inv_mass[n];
    double fi[3], v[3], u0[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        fi[d] = nd.f_int[3 * n + d];
        v[d] = nd.v[3 * n + d];
        u0[d] = nd.u[3 * n + d];
    }
    if (ctl->done) return;
    double fe[3] = {0.0, 0.0, 0.0};
    if (cn != CN_NONE && !fixed) {
        const uint4* list = reinterpret_cast<const uint4*>(ca.ev_list + (long long)cn * EV_CAP);
        const uint4 row[EV_CAP / 4] = {list[0], list[1], list[2], list[3]};  // beside the count
        const int cnt = ca.ev_count[cn];
        if (cnt > EV_CAP) return;  // the block that sums it takes its half step
        gather_events(ca, cn, cnt, row, fe[0], fe[1], fe[2]);
#pragma unroll
        for (int d = 0; d < 3; ++d) nd.f_ext[3 * n + d] = fe[d];
    }
    const double dt = step_dt(ctl);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double a = (fe[d] - fi[d]) * im;
        double vh = v[d] + 0.5 * dt * a;
        double u = u0[d] + dt * vh;
        if (fixed) {
            u = 0.0;
            vh = 0.0;
            nd.v[3 * n + d] = 0.0;
        }
        nd.v_half[3 * n + d] = vh;
        nd.u[3 * n + d] = u;
    }
}

// A node's full update: full_body's arithmetic for its three components, its
// incidence read once.
template <bool ELASTIC>
__device__ __forceinline__ void resident_full(const ElementArrays& el, const NodeArrays& nd, const ControlView* view, long long n) {
    if (n >= nd.n) return;
    const ControlView* ctl = view + nd.node_slot[n];
    const bool fixed = nd.fixed[n] != 0;
    const double im = nd.inv_mass[n];
    const uint4 r0 = __ldg(nd.hc_ell + 2 * n), r1 = __ldg(nd.hc_ell + 2 * n + 1);
    double fe[3], vh[3], f[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        fe[d] = nd.f_ext[3 * n + d];
        vh[d] = nd.v_half[3 * n + d];
    }
    if (r0.x != HC_ELL_MORE) {
        const uint32_t sl[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
        float c[8][3];
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int d = 0; d < 3; ++d) c[j][d] = sl[j] != HC_ELL_NONE ? el.corner[3ull * sl[j] + d] : 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (sl[j] != HC_ELL_NONE)
#pragma unroll
                for (int d = 0; d < 3; ++d) f[d] += (double)c[j][d];
    } else {
#pragma unroll
        for (int d = 0; d < 3; ++d) f[d] = gather_component(nd, el.corner, n, d);
    }
    if (ELASTIC)
#pragma unroll
        for (int d = 0; d < 3; ++d) f[d] = add_scalar_corners(el, nd, n, d, f[d]);
    if (ctl->done) return;
    const double dt = step_dt(ctl);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double a = (fe[d] - f[d]) * im;
        const double v = (vh[d] + 0.5 * dt * a) * ctl->damping;
        nd.v[3 * n + d] = fixed ? 0.0 : v;
        nd.f_int[3 * n + d] = f[d];
    }
}

// A static-grid entry by RES_ST_LANES lanes: nothing outside the union of the
// fixed faces' key boxes, else the faces of its point's bucket, smallest first
// (contact_slave_body's static part). Every lane of the warp calls; the face, or
// -1, in the first lane of the entry.
__device__ __forceinline__ int resident_static(const ContactArrays& ca, const NodeArrays& nd, const ControlView* view, long long s, bool live,
                                               int lane, double* sd_out) {
    int best = INT_MAX;
    double best_sd = 0.0, sd;
    if (live) {
        const int c = ca.slave_contact[s];
        const long long n = ca.slaves[s];
        const double p[3] = {nd.pos[3 * n] + nd.u[3 * n], nd.pos[3 * n + 1] + nd.u[3 * n + 1], nd.pos[3 * n + 2] + nd.u[3 * n + 2]};
        const double* box = ca.st_box + 6 * c;
        live = !view[ca.contact_slot[c]].done;
        if (live && p[0] >= box[0] && p[0] <= box[3] && p[1] >= box[1] && p[1] <= box[4] && p[2] >= box[2] && p[2] <= box[5]) {
            const double md = ca.max_distance[c];
            const FaceGeo* geo = ca.geo + ca.face_off[c];
            const long long st0 = ca.st_tab_off[c];
            const long long bk = st0 + (point_cell_hash(p, ca.cell[c], 0) & (unsigned)(ca.st_tab_off[c + 1] - st0 - 1));
            const uint32_t e0 = ca.st_off[bk + c], e1 = ca.st_off[bk + c + 1];
            for (uint32_t k = e0 + lane; k < e1; k += RES_ST_LANES) {  // ascending faces: a lane's first hit is its smallest
                const int f = ca.st_entries[k];
                if (face_hit(geo[f], p, md, &sd)) {
                    best = f;
                    best_sd = sd;
                    break;
                }
            }
        }
    }
#pragma unroll
    for (int off = RES_ST_LANES / 2; off > 0; off >>= 1) {
        const int ob = __shfl_down_sync(0xffffffffu, best, off, RES_ST_LANES);
        const double osd = __shfl_down_sync(0xffffffffu, best_sd, off, RES_ST_LANES);
        if (ob < best) {
            best = ob;
            best_sd = osd;
        }
    }
    if (!live || lane != 0) return -1;
    if (best == INT_MAX) {
        ca.hit[s] = -1;
        return -1;
    }
    ca.hit[s] = best;
    ca.hit_sd[s] = best_sd;
    *sd_out = best_sd;
    return best;
}
// A dynamic-grid entry (or one of a contact without any grid) by a warp:
// contact_slave_body's dynamic part with one list of candidates, so that a
// single narrow test serves all of them. Every lane calls; the face, or -1, in
// lane 0. (A step of the 20,048-element T-bone takes 29 us, 31 us with the
// buckets of the levels scanned one after the other.)
__device__ __forceinline__ int resident_grid(const ContactArrays& ca, const NodeArrays& nd, const ControlView* view, long long s, bool live,
                                             int l, double* sd_out) {
    int best = INT_MAX;
    double best_sd = 0.0;
    bool reset_big = false;
    if (live) {
        const int c = ca.slave_contact[s];
        const long long n = ca.slaves[s];
        const int tab = ca.tab_off[c], tab1 = ca.tab_off[c + 1];
        reset_big = l == 0 && tab1 > tab;
        const double p[3] = {nd.pos[3 * n] + nd.u[3 * n], nd.pos[3 * n + 1] + nd.u[3 * n + 1], nd.pos[3 * n + 2] + nd.u[3 * n + 2]};
        const double md = ca.max_distance[c];
        const long long fb = ca.face_off[c];
        const FaceGeo* geo = ca.geo + fb;
        live = !view[ca.contact_slot[c]].done;
        // the candidates: the smallest big face that hit (one more for lane 0),
        // then the point's bucket of every level in use, or all the faces
        const int big = live && tab1 > tab ? ca.big_best[s] : BIG_NONE;
        const int used = tab1 > tab ? ca.levels_used[c] : 0;
        const unsigned mask = (unsigned)(tab1 - tab - 1);
        unsigned e0[GRID_LEVELS] = {0u, 0u};
        int cnt[GRID_LEVELS] = {0, 0};
        if (live && tab1 > tab) {
            double cs = ca.cell[c];
#pragma unroll
            for (int level = 0; level < GRID_LEVELS; ++level, cs *= 4.0)
                if (used & (1 << level)) {
                    const int b = tab + (int)(point_cell_hash(p, cs, level) & mask);
                    e0[level] = ca.boff[b];
                    cnt[level] = ca.blen[b];
                }
        }
        const int lead = big != BIG_NONE ? 1 : 0;
        const int total = !live ? 0 : tab1 > tab ? lead + cnt[0] + cnt[1] : (int)(ca.face_off[c + 1] - fb);
        for (int k = l; k < total; k += RES_GRID_LANES) {
            int f = k;
            if (tab1 > tab) f = k < lead ? big : k < lead + cnt[0] ? ca.entries[e0[0] + k - lead] : ca.entries[e0[1] + k - lead - cnt[0]];
            double sd;
            if (f < best && face_hit(geo[f], p, md, &sd)) {
                best = f;
                best_sd = sd;
            }
        }
    }
#pragma unroll
    for (int off = RES_GRID_LANES / 2; off > 0; off >>= 1) {
        const int ob = __shfl_down_sync(0xffffffffu, best, off, RES_GRID_LANES);
        const double osd = __shfl_down_sync(0xffffffffu, best_sd, off, RES_GRID_LANES);
        if (ob < best) {
            best = ob;
            best_sd = osd;
        }
    }
    static_assert(GRID_LEVELS == 2, "two levels' buckets");
    if (reset_big) ca.big_best[s] = BIG_NONE;
    if (!live || l != 0) return -1;
    if (best == INT_MAX) {
        ca.hit[s] = -1;
        return -1;
    }
    ca.hit[s] = best;
    ca.hit_sd[s] = best_sd;
    *sd_out = best_sd;
    return best;
}
// ELASTIC: the context has elastic elements with a free node; without, their
// code stays out of the kernel.
template <int RES_TPB, bool ELASTIC>
__global__ void __launch_bounds__(RES_TPB, 1) k_steps(const __grid_constant__ ResidentArgs A) {
    __shared__ HeavyShared heavy;
    __shared__ FaceGeo big_face;
    __shared__ double big_box[6];
    __shared__ int s_state, s_chunks[ACTIVE_SPACES];
    __shared__ uint8_t s_cand[RES_TPB / 32][BRUTE_MAX_FACES + 1];
    // OCT_SHARED per eight threads, when elastic elements take eight lanes, then
    // a control view per slot
    extern __shared__ double oct_shared[];
    constexpr int RES_WARPS = RES_TPB / 32;
    ControlView* view = reinterpret_cast<ControlView*>(oct_shared + (ELASTIC && A.sc_oct ? OCT_SHARED * RES_TPB / 8 : 0));
    static_assert(RES_TPB >= HEAVY_TPB && VEH_TPB == HEAVY_TPB && sizeof(heavy.sf) >= 2 * sizeof(double) * VEH_TPB, "block sums");
    static_assert(RES_TPB >= HIST_TREE && sizeof(heavy) >= sizeof(double) * HIST_PART_VALUES * HIST_TREE && alignof(HeavyShared) >= 8,
                  "a history's part sums");
    const bool summing = threadIdx.x < HEAVY_TPB;  // the threads of the block-wide sums
    const bool odd_jobs = blockIdx.x == gridDim.x - 1;  // the block that does what one block does
    const int lane = threadIdx.x & 31;
    const ElementArrays& el = A.el;
    Control* ctls = A.ctls;
    const int n_slots = A.ca[0].n_slots;
    const bool contacts = A.ca[0].n_contacts > 0, grids = A.ca[0].n_grid_slaves > 0;
    // The dynamic grids' three passes (count with the geometry, allocate,
    // insert) run all or none: a count that no insert takes back would add to
    // the next search's. None without an entry to look up (bodies that miss
    // each other, or start apart by more than the contact's reach).
    const bool cells = grids && A.ca[0].n_buckets > 0;
    ResidentBarrier barrier{A.sync, A.polls, 0, 0};
    if (A.sync->dead) return;  // an earlier launch of the run gave up
    // emitted: the search emitted this step's events. pending_end: the last
    // step's end is still to be written to the control blocks. pending_record:
    // a record's partial sums are still to be added up.
    bool emitted = false, pending_end = false, pending_record = false;
    long long ended = A.step0;  // the last step whose phases are through

    // chunk c of space sp holds the entities [256 c, 256 c + 256)
    auto entity = [&](int sp, int task, int mult, int* l) -> long long {
        const int g = task * 32 + lane, per = CHUNK * mult, item = g / per, within = g - item * per;
        const long long chunk = A.lists ? A.lists[A.space_off[sp] + item] : item;
        *l = within % mult;
        return chunk * CHUNK + within / mult;
    };
    auto tasks = [&](int sp, int mult) { return s_chunks[sp] * (CHUNK / 32) * mult; };
    auto load_view = [&] {  // every block, behind a barrier with a serial part
        for (int sl = threadIdx.x; sl < n_slots; sl += RES_TPB) {
            const Control& c = ctls[sl];
            view[sl] = ControlView{c.t, c.end_time, c.dt_cfl, c.damping, c.dt_floor, c.step, c.max_steps, c.done, c.mass_scale_now};
        }
        if (threadIdx.x < ACTIVE_SPACES)
            s_chunks[threadIdx.x] = A.lists ? A.ab.counts[threadIdx.x] : (int)((A.space_n[threadIdx.x] + CHUNK - 1) / CHUNK);
    };
    // The crashes still running, block-wide; orders the view for the block as well.
    auto running = [&] {
        int n = 0;
        for (int sl = 0; sl < n_slots; sl += RES_TPB) n += __syncthreads_count(sl + threadIdx.x < n_slots && !view[sl + threadIdx.x].done);
        return n;
    };
    // The chunks that still hold a running crash, in one block (over the chunks
    // that hold entities, not a serving context's whole room: 50,000 chunks of a
    // room of 2 M elements).
    auto rebuild = [&] {
        for (int k = threadIdx.x; k < ACTIVE_SPACES; k += RES_TPB) A.ab.counts[k] = 0;
        __syncthreads();
        const int total = A.chunk_off[ACTIVE_SPACES];
        for (int k0 = 0; k0 < total; k0 += RES_TPB) {
            const int k = k0 + threadIdx.x;
            long long t = A.ab.n_chunks;  // none
            if (k < total) {
                int sp = 0;
                while (k >= A.chunk_off[sp + 1]) ++sp;
                t = A.space_off[sp] + (k - A.chunk_off[sp]);
            }
            build_active_body(A.ab, ctls, t);
        }
        __syncthreads();
    };
    auto finalize = [&] {
        for (int sl = threadIdx.x; sl < n_slots; sl += RES_TPB) dt_finalize_slot(ctls + sl, A.mass_flag);
    };
    auto end_step = [&](long long step, bool sep) {  // the step's end in the control blocks (one block)
        if (threadIdx.x == 0) *A.mass_flag = 0;
        for (int sl = threadIdx.x; sl < n_slots; sl += RES_TPB) {
            Control* ctl = ctls + sl;
            if (!ctl->done) step_end_slot(ctl, sl, A.ca[step & 1], A.va, sep ? 1 : 0);
            A.done_out[sl] = ctl->done;
        }
    };
    auto record_sums = [&](TaskDeal& deal) {  // of the record whose partial sums are in place
        deal(A.hist.n_pu, [&](int pu) {
            const int slot = A.hist.pu_slot[pu];
            const long long r = A.hist.rec_count[slot];
            if (hist_due(A.hist, view + slot, slot, HIST_STEP) && r < A.hist.slot_max[slot]) hist_finish_warp(A.hist, pu, r, lane);
        });
    };
    auto record_close = [&] {  // one block, behind record_sums
        for (int slot = threadIdx.x; slot < n_slots; slot += RES_TPB) {
            if (!hist_due(A.hist, view + slot, slot, HIST_STEP)) continue;
            const long long r = A.hist.rec_count[slot];
            if (r < A.hist.slot_max[slot]) {
                A.hist.rec_time[(long long)slot * A.hist.max_rec + r] = view[slot].t;
                A.hist.rec_step[(long long)slot * A.hist.max_rec + r] = view[slot].step;
            }
            A.hist.rec_count[slot] = r + 1;
            A.hist.last_step[slot] = view[slot].step;
        }
    };

    bool go = barrier(&s_state, [&] {
        if (A.lists && A.step0 % 20 == 0) rebuild();
        if (A.adaptive && A.step0 % A.check_steps == 0) finalize();
    });
    if (go) load_view();
    int n_running = running(), n_listed = n_running;  // now, and when the lists were built
    go = go && n_running > 0;
    TaskDeal deal{(int)((threadIdx.x >> 5) * gridDim.x + blockIdx.x), (int)gridDim.x * RES_WARPS, 0};
    for (int i = 0; go && i < A.n_steps; ++i) {
        const long long step = A.step0 + i;
        const ContactArrays& ca = A.ca[step & 1];
        const ContactArrays& cn = A.ca[(step + 1) & 1];
        const NodeArrays& nd = A.nd[step & 1];
        const bool check = A.adaptive && step % A.check_steps == 0, check_next = A.adaptive && (step + 1) % A.check_steps == 0;
        const bool sep = A.any_separation && (step + 1) % 10 == 0 && A.va.n_vehicles > 0;
        // Whether the next step's dt and the crashes that take it are known
        // without the control blocks: no stable-dt check, no stop rule that
        // looks at the whole state, not the launch's last step.
        const bool plain = i + 1 < A.n_steps && !check_next && !sep && (step + 1) % 20 != 0;
        deal.base = 0;

        // Contact forces, where the search did not emit them, and mass scaling.
        if ((contacts && !emitted) || check) {
            if (contacts && !emitted)
                deal(tasks(6, FORCE_LANES), [&](int t) {
                    int l;
                    const long long s = entity(6, t, FORCE_LANES, &l);
                    if (s < A.n_slaves) contact_force_body(ca, view, 1, 0.0, nd.mass, 1, 0, s, l);
                });
            if (check)
                deal(tasks(2, 1), [&](int t) {
                    int l;
                    mass_scaling_body(el, nd, view, 0, entity(2, t, 1, &l));
                });
            if (!(go = barrier())) break;
            deal.base = 0;
        }

        // Reactions and half step; the search's bookkeeping starts clear.
        const int n_heavy = contacts ? *ca.gather_count : 0;
        deal(tasks(2, 1), [&](int t) {
            int l;
            resident_gather_half(ca, nd, view, A.node_cn, entity(2, t, 1, &l));
        });
        if (pending_record) record_sums(deal);
        for (int w = blockIdx.x; summing && w < n_heavy; w += gridDim.x) {
            const long long k = ca.gather_work[w], n = ca.cnode[k];
            const ControlView* ctl = view + nd.node_slot[n];
            const double acc = heavy_node(ca, 0, ca.n_contacts, k, ca.ev_count[k], heavy);
            if (threadIdx.x < 3 && !ctl->done) {  // a heavy node is a free one (fixed nodes take no events)
                const long long q = 3 * n + threadIdx.x;
                const double dt = step_dt(ctl);
                const double a = (acc - nd.f_int[q]) * nd.inv_mass[n];
                const double vh = nd.v[q] + 0.5 * dt * a;
                nd.f_ext[q] = acc;
                nd.v_half[q] = vh;
                nd.u[q] = nd.u[q] + dt * vh;
            }
            heavy_sync();
        }
        if (odd_jobs) {
            if (contacts)
                for (long long k = threadIdx.x; k < 2 * ca.contact_room + 1; k += RES_TPB) ca.grid_state[k] = 0;
            if (pending_end) end_step(ended, false);
        }
        pending_end = false;
        if (!(go = barrier())) break;
        deal.base = 0;

        // Element forces and the moving faces' geometry.
        if (odd_jobs) {
            if (contacts) contact_reset_block(ca);
            if (pending_record) record_close();
        }
        pending_record = false;
        deal(tasks(0, 1), [&](int t) {
            int l;
            forces_body<false>(el, nd, ctls, view, 1, entity(0, t, 1, &l));
        });
        if (ELASTIC && A.sc_oct)
            deal(tasks(8, 8), [&](int t) {
                int l;
                const long long k = entity(8, t, 8, &l);
                scalar_force_oct(el, nd, ctls, view, 1, k < el.n_sc ? (long long)el.sc_list[k] : -1,
                                 oct_shared + OCT_SHARED * (threadIdx.x / 8));
            });
        else if (ELASTIC)
            deal(tasks(8, 1), [&](int t) {
                int l;
                const long long k = entity(8, t, 1, &l);
                scalar_force_body<true>(el, nd, ctls, view, 1, k < el.n_sc ? (long long)el.sc_list[k] : el.sc_count);
            });
        if (cells)
            deal(tasks(5, FACE_LANES), [&](int t) {
                int l;
                const long long k = entity(5, t, FACE_LANES, &l);
                contact_face_body<FACE_LANES>(ca, nd, view, 0, ca.dyn_faces, ca.n_dyn_faces, 1, 1, k, l);
            });
        else
            deal(tasks(5, 1), [&](int t) {
                int l;
                const long long k = entity(5, t, 1, &l);
                contact_face_body<1>(ca, nd, view, 0, ca.dyn_faces, ca.n_dyn_faces, 1, 0, k, l);
            });
        if (!(go = barrier())) break;
        deal.base = 0;

        // Full update beside the search of the next step's contacts.
        deal(tasks(9, 32), [&](int t) {
            int l;
            const long long e = entity(9, t, 32, &l);
            if (e >= ca.n_brute_entries) return;
            const BruteEntry be = ca.brute_entries[e];
            double sd = 0.0;
            const int best = resident_brute(cn, nd, view, be, lane, s_cand[threadIdx.x >> 5], &sd);
            if (plain) resident_emit<32>(cn, view, nd.mass, be.s, best, sd, lane);
        });
        deal(tasks(7, RES_ST_LANES), [&](int t) {
            int l;
            const long long e = entity(7, t, RES_ST_LANES, &l);
            const bool live = e < ca.n_st_slaves;
            const long long s = live ? (long long)ca.st_slaves[e] : 0;
            double sd = 0.0;
            const int best = resident_static(cn, nd, view, s, live, l, &sd);
            if (plain) resident_emit<RES_ST_LANES>(cn, view, nd.mass, s, best, sd, l);
        });
        if (check_next)
            deal(tasks(1, 1), [&](int t) {
                int l;
                elem_dt_body(el, nd, ctls, view, nd.u, 1, entity(1, t, 1, &l));
            });
        deal(tasks(2, 1), [&](int t) {
            int l;
            resident_full<ELASTIC>(el, nd, view, entity(2, t, 1, &l));
        });
        if ((step + 1) % 20 == 0)
            deal(tasks(2, 1), [&](int t) {
                int l;
                nonfinite_body(nd, ctls, view, entity(2, t, 1, &l));
            });
        if (grids) {
            if (cells) {
                deal((int)((ca.n_buckets - ca.tab_off[A.contact0] + 31) / 32),
                     [&](int t) { grid_alloc_body(ca, A.contact0, ca.n_contacts, (long long)t * 32 + lane); });
                contact_big_block(ca, nd, big_face, big_box);
                if (!(go = barrier())) break;
                deal.base = 0;
                deal(tasks(5, 32), [&](int t) {
                    int l;
                    const long long k = entity(5, t, 32, &l);
                    contact_insert_body(ca, 0, ca.dyn_faces, ca.n_dyn_faces, k, l);
                });
                if (!(go = barrier())) break;
                deal.base = 0;
            }
            deal(tasks(3, RES_GRID_LANES), [&](int t) {
                int l;
                const long long e = entity(3, t, RES_GRID_LANES, &l);
                const bool live = e < ca.n_grid_slaves;
                const long long s = live ? (long long)ca.grid_slaves[e] : 0;
                double sd = 0.0;
                const int best = resident_grid(cn, nd, view, s, live, l, &sd);
                if (plain) resident_emit<RES_GRID_LANES>(cn, view, nd.mass, s, best, sd, l);
            });
        }
        if (sep) {
            if (!(go = barrier())) break;
            for (int k = blockIdx.x; summing && k < A.va.n_vehicles * A.va.vx_blocks; k += gridDim.x) {
                vehicle_vx_block(A.va, nd.mass, nd.v, ctls, k, &heavy.sf[0][0], &heavy.sf[0][0] + VEH_TPB);
                heavy_sync();
            }
        }
        emitted = plain;
        ended = step;

        // The step's end. On a plain step every block moves its own view on,
        // and one block writes the control blocks during the next phase;
        // otherwise the control blocks decide, with the next step's stable-dt
        // decision and chunk lists.
        if (plain) {
            if (!(go = barrier())) break;
            for (int sl = threadIdx.x; sl < n_slots; sl += RES_TPB) {
                ControlView c = view[sl];
                if (c.done) continue;
                c.done = last_step_by_count_or_time(&c) ? 1 : 0;
                const double dt = step_dt(&c);
                c.step += 1;
                c.t = c.t + dt;
                c.mass_scale_now = 0;
                view[sl] = c;
            }
            pending_end = true;
        } else {
            // crashes only ever stop during a launch, so the same number is the same lists
            const bool relist = A.lists && (step + 1) % 20 == 0 && i + 1 < A.n_steps;
            go = barrier(&s_state, [&] {
                end_step(step, sep);
                __syncthreads();  // the mass flag is clear before a slot sets it
                if (check_next && i + 1 < A.n_steps) finalize();
                if (relist) {
                    int n = 0;
                    for (int sl = 0; sl < n_slots; sl += RES_TPB)
                        n += __syncthreads_count(sl + threadIdx.x < n_slots && !ctls[sl + threadIdx.x].done);
                    if (n != n_listed) rebuild();
                }
            });
            if (!go) break;
            load_view();
        }
        n_running = running();
        if ((step + 1) % 20 == 0) n_listed = n_running;
        if (A.hist_on && (step + 1) % A.hist.steps == 0) {
            deal.base = 0;
            deal(A.hist.n_pu * HIST_BLOCKS, [&](int t) {
                const int pu = t / HIST_BLOCKS, slot = A.hist.pu_slot[pu];
                if (A.hist.any_long && hist_long(A.hist, pu)) return;
                if (hist_due(A.hist, view + slot, slot, HIST_STEP)) hist_part_warp(A.hist, nd, nd.f_ext, pu, t % HIST_BLOCKS, lane);
            });
            for (int t = blockIdx.x; A.hist.any_long && threadIdx.x < HIST_TREE && t < A.hist.n_pu * HIST_BLOCKS; t += gridDim.x) {
                const int pu = t / HIST_BLOCKS, slot = A.hist.pu_slot[pu];
                if (hist_long(A.hist, pu) && hist_due(A.hist, view + slot, slot, HIST_STEP))
                    hist_part_block(A.hist, nd, nd.f_ext, pu, t % HIST_BLOCKS, reinterpret_cast<double*>(&heavy));
            }
            deal((A.hist.n_an + 31) / 32, [&](int t) {
                const int j = t * 32 + lane;
                if (j >= A.hist.n_an) return;
                const int slot = nd.node_slot[A.hist.an_node[j]];
                const long long r = A.hist.rec_count[slot];
                if (hist_due(A.hist, view + slot, slot, HIST_STEP) && r < A.hist.slot_max[slot]) hist_node(A.hist, nd, nd.f_ext, j, r);
            });
            pending_record = true;
            if (!(go = barrier())) break;
        }
        if (n_running == 0) break;
    }
    if (!go) return;
    // every crash is done, or the launch's last step was not a plain one
    if (pending_end && odd_jobs) end_step(ended, false);
    if (pending_record) {
        deal.base = 0;
        record_sums(deal);
        barrier(&s_state, record_close);
    }
}

// Behind every launch of k_steps: after one that gave up, the bookkeeping that
// a contact search expects clear, which its half-done phase may have left set
// (grid counts, event lists, big-face hits); the run's later launches then
// return at once.
__global__ void k_steps_failed(ResidentSync* y, int* failed, ContactArrays ca, long long n_slaves) {
    if (!y->error) return;
    y->dead = 1;
    *failed = 1;
    const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, n = (long long)gridDim.x * blockDim.x;
    if (ca.n_contacts == 0) return;
    for (long long i = i0; i < ca.n_buckets; i += n) ca.counts[i] = 0;
    for (long long i = i0; i < ca.n_cnodes; i += n) ca.ev_count[i] = 0;
    for (long long i = i0; i < n_slaves; i += n) ca.big_best[i] = BIG_NONE;
    if (i0 == 0) {
        *ca.ev_pool_n = 0;
        *ca.gather_count = 0;
    }
}
