// The device loop's parts that its forms share: the loop's kernels of their own (one a part of the step, captured in
// graphs) and the resident loop (several steps in one cooperative launch). Compiled into both builds of the step, so
// what the exact build rounds twice is written so that contraction cannot round it once.
#pragma once

#include "w2b_common.cuh"
#include "w2b_tma.cuh"

namespace w2b {

// ------------------------------------------------------------------ the resident loop's grid barrier

constexpr int RESIDENT_THREADS = 256;
// CTAs a SM the launch bound plans for, by the strips' height. Fewer leave more registers a thread: 4-row strips serve
// the smallest grids, where nothing but a warp's own chain counts (62 x 62 cells: 11.4 us a step with two, 11.9 with
// three, 13.2 with four); 8-row ones need their CTAs (256 x 256: 17.1 with three, 18.6 with four, 19.2 with two); 16-row
// ones do best with two where the resident loop is the best form at all (a valley of 108 tiles: 20.7 against 25.0 with
// three and 27.0 with four).
constexpr int resident_ctas(int rows) { return rows == 8 ? 3 : 2; }
constexpr uint32_t GRID_WAIT_LIMIT = 1u << 21;  // polls of a barrier before a CTA gives up, one to two seconds

__device__ __forceinline__ GridState* grid_state(Ctl* ctl) {
    return reinterpret_cast<GridState*>(reinterpret_cast<char*>(ctl) + GRID_STATE_AT);
}
__device__ __forceinline__ int32_t* follow_flag(Ctl* ctl) {
    return reinterpret_cast<int32_t*>(reinterpret_cast<char*>(ctl) + FOLLOW_AT);
}

// Every CTA of a cooperative launch: what each wrote before it, in either proxy's eyes, is what all read after it.
// met: this launch's arrivals so far, the same in every CTA. False: some CTA did not come in time (reported; the
// caller leaves, and so does every other CTA, each by its own count).
// meanwhile: what every thread does after its CTA has arrived, before it waits.
template <class Meanwhile>
__device__ __forceinline__ bool grid_barrier(uint32_t* arrived, int32_t* status, uint32_t& met, Meanwhile meanwhile) {
    met += gridDim.x;
    asm volatile("fence.proxy.async;" ::: "memory");  // the state is written by threads and read by bulk copies
    __syncthreads();
    bool late = false;
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrived) : "memory");
    meanwhile();
    if (threadIdx.x == 0) {
        uint32_t seen, polls = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(arrived) : "memory");
            late = ++polls > GRID_WAIT_LIMIT;
        } while (seen < met && !late);
        if (late) atomicExch(status, W2B_ETIMEOUT);
        asm volatile("fence.proxy.async;" ::: "memory");
    }
    return !__syncthreads_or(late);
}
__device__ __forceinline__ bool grid_barrier(GridState* grid, Ctl* ctl, uint32_t& met) {
    return grid_barrier(&grid->arrived, &ctl->status, met, [] {});
}

// The end of a resident launch: the last CTA to leave puts the barrier's counters back to zero.
__device__ __forceinline__ void grid_leave(GridState* grid) {
    if (threadIdx.x == 0 && atomicAdd(&grid->left, 1u) == gridDim.x - 1) {
        grid->arrived = 0;
        grid->left = 0;
    }
}

// ------------------------------------------------------------------ envelope, boundary cells, tally, lines

// The envelope of one own cell (wadi2d/engine/maxima.py:75-92; the CPU twin forms the centre speed in float64): what it
// reads, every load issued before any store, so that a thread's loads make one round trip; then the entries that
// change. un, vn: the face velocities after the step.
struct EnvelopeIn {
    float d0, h0, s0, z0, a0, ue, uw, vs, vn;
};
__device__ __forceinline__ EnvelopeIn envelope_load(const StepArgs& A, int fid, int k, const float* un,
                                                    const float* vn) {
    return EnvelopeIn{A.env[0][fid], A.env[1][fid], A.env[2][fid], A.env[3][fid], A.env[4][fid],
                      un[k + 1],     un[k],         vn[k + A.px],  vn[k]};
}
__device__ __forceinline__ void envelope_apply(const StepArgs& A, int fid, const EnvelopeIn& E, float dk, float hk,
                                               float time, float arrive, float deep) {
    // max(old, new) as fmax32 forms it keeps old exactly when old >= new
    if (!(E.d0 >= dk)) A.env[0][fid] = dk;
    if (!(E.h0 >= hk)) A.env[1][fid] = hk;
    if (dk > deep) {
        const double uc = 0.5 * (double)(E.uw + E.ue);
        const double vc = 0.5 * (double)(E.vn + E.vs);
        const double sp = sqrt(__dadd_rn(__dmul_rn(uc, uc), __dmul_rn(vc, vc)));
        if (!((double)E.s0 >= sp)) A.env[2][fid] = (float)sp;
        const double hz = sp * (double)dk;
        if (!((double)E.z0 >= hz)) A.env[3][fid] = (float)hz;
    }
    if (E.a0 < 0.0f && dk >= arrive) A.env[4][fid] = time;
}
__device__ __forceinline__ void envelope_cell(const StepArgs& A, int fid, int k, float dk, float hk, float time,
                                              float arrive, float deep, const float* un, const float* vn) {
    envelope_apply(A, fid, envelope_load(A, fid, k, un, vn), dk, hk, time, arrive, deep);
}

// The run that native cell k belongs to.
__device__ __forceinline__ int run_of_native(const StepArgs& A, int k) {
    return A.nruns == 1 ? 0 : A.tile_run[tile_of_native(A, k)];
}

// The boundary cells of every running run after its step (wadi2d/solver/gpu/kernels/cells.cu:95-111), whether their tile is
// stepped or asleep, and their envelope entries. host_flags: a host-driven step's of run 0 (0 in the device loop). What a
// cell needs is a chain of loads from L2, so all that do not depend on one another are issued together.
__device__ __forceinline__ void boundary_items(const StepArgs& A, const StepView& V, int gtid, int gstride,
                                               int host_flags = 0) {
    for (int m = gtid; m < A.nb; m += gstride) {
        const int k = A.bcell[m], kind = A.bkind[m];
        const float h0 = A.bh0[m], d0 = A.bd0[m];
        const float arrive = A.ctl->arrive, deep = A.ctl->deep;
        const int fid = fid_of_native(A, k);
        const int run = A.nruns == 1 ? 0 : A.tile_run[fid / TILE2];
        const int flags = host_flags ? host_flags : __ldcg(V.flags + run);
        const int n = 1 - __ldcg(V.parity + run);
        const float time = __ldcg(V.max_time + run);
        if (!(flags & F_RUN)) continue;
        float* h_next = A.hh[n];
        float hk = kind == 0 ? h0 : 0.0f, dk = kind == 0 ? d0 : 0.0f;
        if (kind > 1) {
            const int r = A.bref[m];
            hk = h_next[r];
            dk = fmax32(A.d[r] + d0, 0.0f);
        }
        h_next[k] = hk;
        A.d[k] = dk;
        if (flags & F_MAX) envelope_cell(A, fid, k, dk, hk, time, arrive, deep, A.uu[0][n], A.uu[1][n]);
    }
}

// The FP64 tally (wadi2d/engine/maxima.py:53-62) and the design lines (wadi2d/engine/monitor.py:229-232) of a step:
// tally faces, then a warp a line. A line's Q is the sum of sign q over its faces, FP64, lane-strided then a fixed
// shuffle tree; its running peak of |Q| and the time at the end of the step.
__device__ __forceinline__ void tally_items(const StepArgs& A, const StepView& V, int gtid, int gstride) {
    for (int m = gtid; m < A.ntally; m += gstride) {
        const int face = A.tface[m];
        const int run = run_of_native(A, face);
        if (!(__ldcg(V.flags + run) & F_RUN)) continue;
        const float qv = __ldcg((A.taxis[m] ? A.q[1] : A.q[0]) + face);
        A.ttotal[m] = __dadd_rn(A.ttotal[m], __dmul_rn(__ldcg(V.dt_tally + run), (double)(A.tsign[m] * qv)));
    }
    const int lane = threadIdx.x & 31;
    const int gwarp = gtid >> 5, nwarps = gstride >> 5;
    for (int l = gwarp; l < A.nlines; l += nwarps) {
        const int s = A.lstart[l], e = A.lstart[l + 1];
        if (s >= e) continue;
        const int run = run_of_native(A, A.lface[s]);
        if (!(__ldcg(V.flags + run) & F_RUN)) continue;
        double acc = 0.0;
        for (int m = s + lane; m < e; m += 32) {
            const int f = A.lface[m];
            acc = __dadd_rn(acc, __dmul_rn((double)A.lsign[m], (double)__ldcg((A.laxis[m] ? A.q[1] : A.q[0]) + f)));
        }
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        if (lane == 0) {
            A.lq[l] = acc;
            const double a = fabs(acc);
            if (a > A.lpeak[l]) {
                A.lpeak[l] = a;
                A.ltime[l] = __ldcg(V.t_new + run);
            }
        }
    }
}

// ------------------------------------------------------------------ clocks and settings

// A running run's clock after its step of settings V (wadi2d/solver/stepper.py:113-124): the swap of its halves (into
// W, which may be V), t, the step counts, the step rule on refresh steps (dt_min and non-finite checks). True: the run
// stops, so its tiles leave the work list at this step's rebuild. Every run's wave maximum goes on to W, for either set
// holds the last refresh step's (run_settings clears it where the next step refreshes).
__device__ __forceinline__ bool run_clock(const StepArgs& A, const StepView& V, const StepView& W, int r) {
    Ctl* ctl = A.ctl;
    const RunTab& R = A.R;
    const int flags = V.flags[r];
    const uint32_t bits = __ldcg(V.wave_bits + r);
    if (!(flags & F_RUN)) {
        W.wave_bits[r] = bits;
        W.parity[r] = V.parity[r];
        return false;
    }
    W.parity[r] = V.parity[r] ^ 1;
    R.t[r] = R.t[r] + R.dt_step[r];
    R.nsteps[r] += 1;
    R.steps_run[r] += 1;
    if (flags & F_WAVE) {
        const float wave = __uint_as_float(bits);
        R.wave_last[r] = wave;
        const double w = (double)wave;
        if (!isfinite(w)) {
            R.status[r] = W2B_ENONFINITE;
        } else {
            const double lim = ctl->cfl * (double)R.dx[r] / (ctl->wave_floor > w ? ctl->wave_floor : w);
            R.dt[r] = ctl->dt_max < lim ? ctl->dt_max : lim;
            if (R.dt[r] < ctl->dt_min) R.status[r] = W2B_EDTMIN;
        }
    }
    W.wave_bits[r] = bits;
    return !live_run(R, r, ctl);
}

// The settings of run r's next step (wadi2d/solver/stepper.py:106-111) into W; its share of Ctl::any.
__device__ __forceinline__ uint32_t run_settings(const StepArgs& A, const StepView& W, int r) {
    Ctl* ctl = A.ctl;
    const RunTab& R = A.R;
    if (!live_run(R, r, ctl)) {
        W.flags[r] = 0;
        return 0u;
    }
    const int refresh = R.refresh_due[r] || (R.nsteps[r] % ctl->dt_every == 0);
    R.refresh_due[r] = 0;
    const int activate = (int)(R.nsteps[r] % ctl->active_every == 0);
    double dt = R.dt[r];
    const double rest = R.t_end[r] - R.t[r];
    if (rest < dt) dt = rest;
    if (ctl->dt_max < dt) dt = ctl->dt_max;
    R.dt_step[r] = dt;
    W.dtf[r] = (float)dt;
    const double t_new = R.t[r] + dt;
    W.t_new[r] = t_new;
    W.dt_tally[r] = t_new - R.t[r];
    W.max_time[r] = (float)t_new;
    const int want_max = ctl->max_every > 0 && ((R.nsteps[r] + 1) % ctl->max_every == 0);
    const int act = activate && ctl->adaptive;
    W.flags[r] = F_RUN | (refresh ? F_WAVE : 0) | (activate ? F_WET : 0) | (want_max ? F_MAX : 0) | (act ? F_ACT : 0);
    if (refresh) W.wave_bits[r] = 0u;
    return ANY_RUN | (refresh ? ANY_WAVE : 0u) | (act ? ANY_ACT : 0u) | (want_max ? ANY_MAX : 0u);
}

// The wave of each tile of a run that refreshes at the step of settings W: its face units take their maxima into it.
// The threads of one CTA.
__device__ __forceinline__ void clear_waves(const StepArgs& A, const StepView& W) {
#pragma unroll 4
    for (int t = threadIdx.x; t < A.ntiles; t += blockDim.x)
        if (W.flags[A.tile_run[t]] & F_WAVE) A.wave[t] = 0.0f;
}

// The device loop, one CTA, while the others update the state: every run's clock after the step of settings V, the
// settings of the next step into W, their flags into *to, and whether this step ends with a rebuild of the lists (any:
// this step's flags). A step that no run takes hands each run's half on.
__device__ __forceinline__ void next_settings(const StepArgs& A, const StepView& V, const StepView& W, uint32_t any,
                                              uint32_t* to, GridState* grid) {
    uint32_t mine = 0u;
    bool prune = false;
    for (int r = threadIdx.x; r < A.nruns; r += blockDim.x) {
        prune |= run_clock(A, V, W, r);
        mine |= run_settings(A, W, r);
    }
    uint32_t next = 0u;
    for (const uint32_t bit : {ANY_RUN, ANY_WAVE, ANY_ACT, ANY_MAX})
        if (__syncthreads_or(mine & bit)) next |= bit;
    prune = __syncthreads_or(prune);
    if (threadIdx.x == 0) {
        *to = next;
        if (any & ANY_RUN) A.ctl->m_stored = 0;
        grid->rebuild = prune || (any & ANY_ACT);
    }
    if (next & ANY_WAVE) clear_waves(A, W);
}

// The second set of settings into the first (one CTA, no other reading either).
__device__ __forceinline__ void adopt_settings(const StepArgs& A) {
    const StepView V = step_view(A.R, 1), W = step_view(A.R, 0);
    for (int r = threadIdx.x; r < A.nruns; r += blockDim.x) {
        W.dt_tally[r] = V.dt_tally[r];
        W.t_new[r] = V.t_new[r];
        W.dtf[r] = V.dtf[r];
        W.max_time[r] = V.max_time[r];
        W.flags[r] = V.flags[r];
        W.parity[r] = V.parity[r];
        W.wave_bits[r] = V.wave_bits[r];
    }
}

// ------------------------------------------------------------------ the lists

// Exclusive scan of n over one CTA of whole warps; returns this thread's offset and the total in *total.
__device__ __forceinline__ int block_scan(int n, int* warp_sums, int* total) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = (int)(blockDim.x >> 5);
    int v = n;
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    if (lane == 31) warp_sums[wid] = v;
    __syncthreads();
    if (wid == 0) {
        int w = lane < nw ? warp_sums[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += u;
        }
        warp_sums[lane] = w;  // inclusive sums of warps
    }
    __syncthreads();
    const int before = (wid > 0 ? warp_sums[wid - 1] : 0) + v - n;
    *total = warp_sums[nw - 1];
    __syncthreads();
    return before;
}

// rebuild_active(check=True), wadi2d/solver/stepper.py:56-92, for the runs that rebuild at the step of settings V
// (rebuild: some do): wet or kept tiles and their eight neighbours are active; a tile sleeps after SLEEP_CHECKS checks
// in a row that did not want it; tiles that join the list are listed in woken for their wet share to be written. Then
// the work list: the active tiles of the runs that take another step, rebuilt whenever the active list or the set of
// stepping runs (prune) changed. only_work: the work list alone, before the first step of the device loop. One CTA.
static __device__ __noinline__ void rebuild_lists(const StepArgs& A, const StepView& V, bool only_work, bool rebuild,
                                                  bool prune) {
    Ctl* ctl = A.ctl;
    if (!only_work && !rebuild) {
        // no tile woke at this step: the plan pass that follows has nothing to do
        if (threadIdx.x == 0) ctl->nwoken = 0;
        if (!prune) return;
    }
    const int nt = A.ntiles;
    int* wet_eff = A.scratch;
    int* flags = A.scratch + nt;
    __shared__ int sums[32];
    if (rebuild) {
        for (int t = threadIdx.x; t < nt; t += blockDim.x)
            wet_eff[t] = t != 0 && (__ldcg(A.wet + t) != 0 || A.keep[t] != 0);
        __syncthreads();
        for (int t = threadIdx.x; t < nt; t += blockDim.x) {
            if (t == 0) {
                flags[0] = 0;
                continue;
            }
            const int cur = A.is_act[t];
            if (!(V.flags[A.tile_run[t]] & F_ACT)) {  // this tile's run does not rebuild at this step
                flags[t] = cur;
                continue;
            }
            int act = wet_eff[t];
            for (int n = 0; n < 8; ++n) act |= wet_eff[A.nbr[8 * t + n]];
            if (act)
                A.idle[t] = 0;
            else
                A.idle[t] += 1;
            act |= cur && A.idle[t] < SLEEP_CHECKS;
            flags[t] = act | ((act && !cur) << 1);
            A.is_act[t] = act;
        }
        __syncthreads();
        int nact = 0, nwoken = 0;
        for (int base = 0; base < nt; base += blockDim.x) {
            const int t = base + threadIdx.x;
            const int f = t < nt ? flags[t] : 0;
            int tot_a, tot_w;
            const int oa = block_scan(f & 1, sums, &tot_a);
            const int ow = block_scan((f >> 1) & 1, sums, &tot_w);
            if (f & 1) A.active[nact + oa] = t;
            if (f & 2) A.woken[nwoken + ow] = t;
            nact += tot_a;
            nwoken += tot_w;
        }
        if (threadIdx.x == 0) {
            ctl->nact = nact;
            ctl->nwoken = nwoken;
        }
    }
    // the work list, in tile order: active tiles whose run takes another step
    int nwork = 0;
    for (int base = 0; base < nt; base += blockDim.x) {
        const int t = base + threadIdx.x;
        const int f = t > 0 && t < nt && A.is_act[t] && live_run(A.R, A.tile_run[t], ctl);
        int tot;
        const int o = block_scan(f, sums, &tot);
        if (f) A.work[nwork + o] = t;
        nwork += tot;
    }
    if (threadIdx.x == 0) ctl->nwork = nwork;
}

// refresh_plan (wadi2d/solver/gpu/kernels/cells.cu:66-78) of the listed tiles from entry `first` on, `stride` apart,
// from the current mean depth (parity: each run's current half). CTAs of 256 threads.
__device__ __forceinline__ void plan_tiles(const StepArgs& A, const int32_t* parity, const int32_t* list, int count,
                                           int first, int stride) {
    const int tid = threadIdx.x, ii = tid & 31;
    for (int a = first; a < count; a += stride) {
        const int t = __ldcg(list + a);
        const int tj = A.tiles[2 * t], ti = A.tiles[2 * t + 1];
        const int base = (tj * TILE + GY) * A.px + ti * TILE + GX;
        const int ts = table_of(A, t);
        const float2* pairs_t = A.dtab2 + (size_t)ts * (A.rows - 1) * TILE2;
        const float* h = A.hh[__ldcg(parity + A.tile_run[t])];
        for (int c = 0; c < 4; ++c) {
            const int jj = (tid >> 5) * 4 + c;
            const int local = jj * TILE + ii;
            const int k = base + jj * A.px + ii;
            A.om[k] = cell_plan(h[k], A.hc[ts * TILE2 + local], pairs_t + local, A.rows);
        }
    }
}

}  // namespace w2b
