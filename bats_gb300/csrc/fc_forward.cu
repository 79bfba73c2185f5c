// Fully-connected LIF forward: event scan + closed-form threshold crossings.
//
// Replaces get_spike_weights + compute_spike_times
// (bats/CudaKernels/Wrappers/Inference/get_spike_weights.py:9-18,
//  bats/CudaKernels/Wrappers/Inference/compute_spike_times.py:11-32,
//  bats/CudaKernels/CuFiles/Inference/compute_spike_times.cu:86-138).
//
// Grid (ceil(N_post / TILE), B): one CTA per (post-neuron tile, sample). The reference gathers a
// dense (B, N_post, S) weight array first; here a producer warp streams, for every event of the
// sample in time order, its window constants and the weight-row segment wt[j, tile] (TILE floats) into a
// ring of shared-memory stages (the rows with bulk copies, cp.async.bulk, completing on an mbarrier), running
// up to STAGES * SEV events ahead of the consumers, so no weight load sits on the consumers' path.
// Each consumer thread owns one post neuron and runs the reference's recurrence
// a += w*exp(t/tau_s), b += w*exp(t/tau), crossing search in (t_event, t_next_event].
// Per stage the consumer first accumulates all SEV events and evaluates the provable screen
// (may_cross) on each intermediate state; only if some event may cross does it replay the stage from its
// saved state with the exact solver. The accumulation is the same FMA sequence either way, so the
// results are those of the reference's one-event-at-a-time loop.
//
// Variants, all bit-identical: the stage screen (SCREEN, BATS_FWD_STAGE_SCREEN) first tests a whole
// stage with one membrane bound per neuron (quiet layers); the persistent work-queue kernel
// (bats_lif_forward_fc_queue) runs the same per-item code over (sample, tile) items taken longest
// samples first by resident CTAs (uneven batches); the lanes kernel gives a warp to one (sample, neuron)
// and 32 events at a time (narrow layers, small batches).
#include <algorithm>
#include <cmath>
#include <limits>
#include "common.cuh"
#include "pipeline.cuh"
#include "abi_util.h"

namespace bats {

// Shared memory of one CTA: a ring of STAGES stages of SEV events, each with its weight-row segments (bulk copies),
// its window constants and times (written by the producer), and the full / empty mbarriers.
template <int TILE, int SEV, int STAGES>
struct FwdSmem {
    float rows[STAGES][SEV][TILE];
    CrossWindow win[STAGES][SEV];
    float t[STAGES][SEV + 1];  // t[u + 1]: the end of event u's window
    uint64_t full[STAGES];
    uint64_t empty[STAGES];
    int abort;
    int stop_at;              // ring position of the marker that ended an item early (forward_produce)
    int finished[TILE / 32];  // per consumer warp: the last work item whose remaining events it does not need
};

// Position in the ring: the running stage count, its slot and the slot's phase parity.
template <int STAGES>
struct RingPos {
    int k = 0, slot = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void next() {
        ++k;
        if (++slot == STAGES) {
            slot = 0;
            phase ^= 1u;
        }
    }
};

template <int TILE, int SEV, int STAGES>
__device__ __forceinline__ void forward_init(FwdSmem<TILE, SEV, STAGES>& sm, int consumer_warps) {
    if (threadIdx.x == 0) {
        for (int q = 0; q < STAGES; ++q) {
            mbar_init(&sm.full[q], 1);
            mbar_init(&sm.empty[q], consumer_warps);
        }
        sm.abort = 0;
        sm.stop_at = -1;
        for (int w = 0; w < TILE / 32; ++w) sm.finished[w] = -1;
        fence_barrier_init();
    }
}

// Producer warp, one work item: streams the events' weight-row segments wt[j, tile0 : tile0 + TILE] and window
// constants through the ring. Lane l handles event l of each block of 32 (its record is loaded two blocks ahead, its
// window constants are formed once for all consumer warps), and copies its row when the block's stage is due.
// When every consumer warp has marked the item in sm.finished (its neurons all have k_post spikes, so no later event
// can change an output), the item's next stage becomes a marker without data (sm.stop_at, then one arrival on its
// full barrier) and the item ends with it; the consumers acquire every stage up to the marker, so no copy is in
// flight when they leave the item. Returns false when a wait gave up (the CTA abort flag is raised).
template <int TILE, int SEV, int STAGES>
__device__ __forceinline__ bool forward_produce(FwdSmem<TILE, SEV, STAGES>& sm, RingPos<STAGES>& pos, int it,
                                                const Event* __restrict__ evs, int E, const float* __restrict__ wt,
                                                int ld, int tile0, int consumer_warps, const SolveConst& sk, int lane,
                                                int* status) {
    constexpr int SPB = 32 / SEV;  // stages per block of 32 events
    const uint32_t row_bytes = (uint32_t)min(TILE, ld - tile0) * 4u;
    const int n_stages = (E + SEV - 1) / SEV;
    const float4* src = reinterpret_cast<const float4*>(evs);
    const float4 none = make_float4(BATS_INF, 0.0f, 0.0f, BATS_INF);
    float4 nx1 = lane < E ? __ldg(src + lane) : none;
    float4 nx2 = lane + 32 < E ? __ldg(src + lane + 32) : none;
    for (int kb = 0; kb < n_stages; kb += SPB) {
        const float4 ev = nx1;  // (t, j, es, e)
        const int m = kb * SEV + lane;
        nx1 = nx2;
        nx2 = m + 64 < E ? __ldg(src + m + 64) : none;
        float t_next = __shfl_down_sync(0xffffffffu, ev.x, 1), e_next = __shfl_down_sync(0xffffffffu, ev.w, 1);
        const float t_blk = __shfl_sync(0xffffffffu, nx1.x, 0), e_blk = __shfl_sync(0xffffffffu, nx1.w, 0);
        if (lane == 31) {
            t_next = t_blk;
            e_next = e_blk;
        }
        const CrossWindow w = cross_window(ev.z, ev.w, ev.w, e_next, sk);
        const float* row = wt + (long long)__float_as_int(ev.y) * ld + tile0;
#pragma unroll
        for (int i = 0; i < SPB; ++i) {
            if (kb + i >= n_stages) break;
            const bool ok = mbar_wait(&sm.empty[pos.slot], pos.phase ^ 1u, &sm.abort, status);
            if (!__all_sync(0xffffffffu, ok)) return false;
            if (i == 0) {
                const bool fin = lane >= consumer_warps || *(volatile int*)&sm.finished[lane] == it;
                if (__all_sync(0xffffffffu, fin)) {
                    if (lane == 0) {
                        *(volatile int*)&sm.stop_at = pos.k;
                        mbar_arrive(&sm.full[pos.slot]);  // release: stop_at is visible to the acquiring waits
                    }
                    __syncwarp();
                    pos.next();
                    return true;
                }
            }
            const bool mine = lane / SEV == i && m < E;
            if (mine) {
                const int u = lane % SEV;
                sm.win[pos.slot][u] = w;
                sm.t[pos.slot][u] = ev.x;
                if (u == SEV - 1 || m == E - 1) sm.t[pos.slot][u + 1] = t_next;
            }
            __syncwarp();
            if (lane == 0)
                mbar_arrive_expect_tx(&sm.full[pos.slot], (uint32_t)min(SEV, E - (kb + i) * SEV) * row_bytes);
            __syncwarp();
            if (mine) bulk_copy_g2s(&sm.rows[pos.slot][lane % SEV][0], row, row_bytes, &sm.full[pos.slot]);
            pos.next();
        }
    }
    return true;
}

// After an abort: bounded waits for the copies of the last STAGES issued stages, so that no bulk copy into shared
// memory is in flight when the CTA exits.
template <int TILE, int SEV, int STAGES>
__device__ __forceinline__ void forward_drain(FwdSmem<TILE, SEV, STAGES>& sm, int issued) {
    for (int k = max(0, issued - STAGES); k < issued; ++k) {
        volatile int dummy = 0;
        mbar_wait(&sm.full[k % STAGES], (k / STAGES) & 1, &dummy, nullptr);
    }
}

constexpr int STOP_EVERY = 8;  // stages between two looks at whether every neuron of a warp is done

// Consumer warps' part of one work item (sample s, post neurons tile0 .. tile0 + TILE - 1): thread = post neuron.
// Returns false when a wait gave up (the CTA is aborting).
//
// Pass 1 accumulates a stage's events (the reference's FMA sequence) and marks every event after which a crossing
// cannot be ruled out (may_cross): branch-free, so the per-event tests of the stage overlap. Pass 2, for the neurons
// with a marked event, is the reference's event-by-event loop from that event on.
// Until the first stage that does not settle so for the warp's neurons, stages run only the accumulation, tracking the
// smallest a and |a| and the largest b of their states, and skip the per-event tests when stage_no_crossing rules out a
// crossing after any of the stage's events (784 -> 800 silent neurons, 256 samples: 46 -> 33 us). SCREEN: every full stage
// is tried so first; otherwise it is evaluated as without SCREEN. The FMA sequence is the same either way, so results are
// bit-identical. (Tries at growing distances all through the loop made active layers 2.5 % slower.)
// A neuron with k_post spikes is done; a warp whose neurons are all done, or that has none, only passes stages on (see
// forward_produce).
//
// What bounds it: instruction issue (76 % of the issue slots), 590 warp instructions per warp and 8-event stage of an
// active 800 x 800 layer (batch 256, 652 events a sample, 1.4 spikes per warp and stage), 884 with a screen per
// event twice as long, without the left-of-window test in pass 1 (whose false candidates then ran pass 2) and with
// the window constants formed by every consumer warp: 0.587 -> 0.396 ms there, 3.43 -> 2.26 ms on 1024 x 1024 with
// 4096 uneven samples. Two neurons per thread: 0.349 and 2.34 ms, and slower on every smaller grid.
template <int TILE, int SEV, int STAGES, bool SCREEN>
__device__ __forceinline__ bool forward_tile_item(FwdSmem<TILE, SEV, STAGES>& sm, RingPos<STAGES>& pos, int it, int s,
                                                  int tile0, int E, int n_post, int k_post, const SolveConst& sk,
                                                  int* __restrict__ n_spikes, float* __restrict__ a_out,
                                                  float* __restrict__ x_out, float* __restrict__ t_out,
                                                  float* __restrict__ z_out, int* status, int pad) {
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const int n_stages = (E + SEV - 1) / SEV;
    if (tile0 + warp * 32 >= n_post) {  // no neuron (the last tile's warps): only passes stages on
        if (lane == 0) *(volatile int*)&sm.finished[warp] = it;
        for (int k = 0; k < n_stages; ++k) {
            const bool ok = mbar_wait(&sm.full[pos.slot], pos.phase, &sm.abort, status);
            if (!__all_sync(0xffffffffu, ok)) return false;
            const bool stop = *(volatile int*)&sm.stop_at == pos.k;
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.empty[pos.slot]);
            pos.next();
            if (stop) break;
        }
        return true;
    }
    const int i = tile0 + tid;
    const bool active = i < n_post;
    const long long obase = ((long long)s * n_post + (active ? i : 0)) * k_post;
    float a = 0.0f, b = 0.0f;
    int n = 0;
    bool done = !active;
    bool all_done = false;  // warp-uniform
    // A full stage's events accumulated; true if no crossing is possible after any of them.
    auto stage_quiet = [&](const CrossWindow* win, const float* row, float& aa, float& bb) {
        float amin = BATS_INF, bmax = -BATS_INF, amag = BATS_INF;
#pragma unroll
        for (int u = 0; u < SEV; ++u) {
            const float w = row[u * TILE];
            aa = fmaf(w, win[u].es, aa);
            bb = fmaf(w, win[u].e, bb);
            amin = fminf(amin, aa);
            amag = fminf(amag, fabsf(aa));
            bmax = fmaxf(bmax, bb);
        }
        return stage_no_crossing(amin, bmax, amag, aa, bb, win[0].e, sk);
    };
    int k = 0;
    if (!SCREEN) {
        // The quiet beginning: stages that settle for the whole warp by one test per neuron. From the first other one on
        // (which stays where it is) the loop below goes event by event.
        for (; (k + 1) * SEV < E; ++k) {
            const bool ok = mbar_wait(&sm.full[pos.slot], pos.phase, &sm.abort, status);
            if (!__all_sync(0xffffffffu, ok)) return false;
            float aa = a, bb = b;
            const bool quiet = !active || stage_quiet(sm.win[pos.slot], &sm.rows[pos.slot][0][tid], aa, bb);
            if (!__all_sync(0xffffffffu, quiet)) break;
            a = aa;
            b = bb;
            __syncwarp();  // every lane's reads of the slot come before its release
            if (lane == 0) mbar_arrive(&sm.empty[pos.slot]);
            pos.next();
        }
    }
    for (; k < n_stages; ++k) {
        const int slot = pos.slot;
        const bool ok = mbar_wait(&sm.full[slot], pos.phase, &sm.abort, status);
        if (!__all_sync(0xffffffffu, ok)) return false;
        const bool stop = all_done && *(volatile int*)&sm.stop_at == pos.k;  // the marker of an item ended early
        if (!all_done && !done) {
            const int cnt = min(SEV, E - k * SEV);
            const CrossWindow* win = sm.win[slot];
            const float* row = &sm.rows[slot][0][tid];
            float aa = a, bb = b;
            unsigned cand = 0u;
            auto step = [&](int u) {
                const CrossWindow c = win[u];
                const float w = row[u * TILE];
                aa = fmaf(w, c.es, aa);
                bb = fmaf(w, c.e, bb);
                cand |= cross_bit(aa, bb, c, sk, 1u << u);
            };
            bool screened = false;
            if (SCREEN && (k + 1) * SEV < E) {
                screened = stage_quiet(win, row, aa, bb);
                if (!screened) {
                    aa = a;
                    bb = b;
                }
            }
            if (!screened) {
                if (cnt == SEV) {
#pragma unroll
                    for (int u = 0; u < SEV; ++u) step(u);
                } else {  // the sample's last stage
#pragma unroll
                    for (int u = 0; u < SEV; ++u)
                        if (u < cnt) step(u);
                }
            }
            if (cand) {
                // No crossing is possible before the first marked event: its state is reached by plain accumulation.
                const int first = __ffs(cand) - 1;
                aa = a;
                bb = b;
                for (int u = 0; u <= first; ++u) {
                    const float w = row[u * TILE];
                    aa = fmaf(w, win[u].es, aa);
                    bb = fmaf(w, win[u].e, bb);
                }
                bool cross = true;
                for (int u = first;;) {
                    if (cross && solve_candidate<false>(aa, bb, sm.t[slot][u], sm.t[slot][u + 1], win[u], sk, n, k_post,
                                                        obase, a_out, x_out, t_out, z_out)) {
                        done = true;
                        break;
                    }
                    if (++u >= cnt) break;
                    const CrossWindow c = win[u];
                    const float w = row[u * TILE];
                    aa = fmaf(w, c.es, aa);
                    bb = fmaf(w, c.e, bb);
                    cross = may_cross(aa, bb, c, sk);
                }
            }
            a = aa;
            b = bb;
        }
        if ((k & (STOP_EVERY - 1)) == STOP_EVERY - 1 && !all_done) {
            all_done = __all_sync(0xffffffffu, done);
            if (all_done && lane == 0) *(volatile int*)&sm.finished[warp] = it;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.empty[slot]);
        pos.next();
        if (stop) break;
    }
    if (active) n_spikes[(long long)s * n_post + i] = n;
    // +inf past each neuron's spikes. The warp's 32 neurons own contiguous rows of k_post slots, so the
    // warp fills them row by row with the lanes along the row (contiguous stores), not lane by neuron.
    const int i0 = tile0 + warp * 32;
    const int rows = pad ? max(0, min(32, n_post - i0)) : 0;
    const long long wbase = ((long long)s * n_post + i0) * k_post;
    for (int r = 0; r < rows; ++r) {
        const int nr = __shfl_sync(0xffffffffu, n, r);
        for (int q = nr + lane; q < k_post; q += 32) {
            t_out[wbase + (long long)r * k_post + q] = BATS_INF;
            z_out[wbase + (long long)r * k_post + q] = BATS_INF;
        }
    }
    return true;
}

// Resident CTAs the compiler aims at: eight with 128-neuron tiles (48 registers; what their stages leave room for); the
// narrow tiles, whose grids rarely fill the SMs, take the registers they like (1024 -> 20 neurons, 4096 uneven samples:
// 0.83 -> 0.75 ms).
template <int TILE>
constexpr int forward_min_ctas() {
    return TILE == 128 ? 8 : 1;
}

template <int TILE, int SEV, int STAGES, bool SCREEN>
__global__ void __launch_bounds__(TILE + 32, forward_min_ctas<TILE>())
lif_fc_forward_kernel(const Event* __restrict__ ev, const int* __restrict__ ev_count, long long ev_cap,
                      const float* __restrict__ wt, int ld, int n_post, int k_post, SolveConst sk,
                      int* __restrict__ n_spikes, float* __restrict__ a_out, float* __restrict__ x_out,
                      float* __restrict__ t_out, float* __restrict__ z_out, int* __restrict__ status, int pad) {
    pdl_prologue();
    extern __shared__ __align__(128) unsigned char smem_raw[];
    using Smem = FwdSmem<TILE, SEV, STAGES>;
    Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
    constexpr int CONSUMER_WARPS = TILE / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s = blockIdx.y;
    const int tile0 = blockIdx.x * TILE;
    const int E = ev_count[s];
    forward_init(sm, CONSUMER_WARPS);
    __syncthreads();
    RingPos<STAGES> pos;
    if (warp == CONSUMER_WARPS) {
        if (!forward_produce(sm, pos, 0, ev + (long long)s * ev_cap, E, wt, ld, tile0, CONSUMER_WARPS, sk, lane,
                             status))
            forward_drain(sm, pos.k);
        return;
    }
    forward_tile_item<TILE, SEV, STAGES, SCREEN>(sm, pos, 0, s, tile0, E, n_post, k_post, sk, n_spikes, a_out,
                                                      x_out, t_out, z_out, status, pad);
}

// Persistent variant over a work queue, for batches whose samples carry very different numbers of events.
// A work item is (sample, post-neuron tile); the items are numbered in the order of `order` (samples by
// descending event count, from work_order_kernel), the tiles of a sample next to each other, and a grid of
// as many CTAs as fit on the GPU at once takes them from a global counter (`head`, zero at launch) until
// none is left: the longest samples start first and the short ones fill the end, instead of the block
// scheduler's fixed index order leaving a long sample for last. The producer warp claims the next item
// and starts streaming its stages while the consumers finish the current one (the ring's stage count runs
// on across items), so no CTA start-up or pipeline fill sits between items. Items reach the consumers
// through a two-slot mailbox with its own full/empty mbarriers. Each item computes exactly what the
// one-item-per-CTA kernel computes for it, so results are bit-identical to lif_fc_forward_kernel's.
struct WorkItem {
    int s;      // sample, < 0: no work left
    int tile0;  // first post neuron of the tile
    int E;      // events of the sample
    int unused;
};
struct ItemMailbox {
    uint64_t full[2];   // the producer has written item[q] (one arrival)
    uint64_t empty[2];  // every consumer warp has read item[q] (one arrival per warp)
    WorkItem item[2];
};

template <typename Smem>
__host__ __device__ constexpr size_t mailbox_offset() {
    return (sizeof(Smem) + 15) / 16 * 16;
}

template <int TILE, int SEV, int STAGES, bool SCREEN>
__global__ void __launch_bounds__(TILE + 32, forward_min_ctas<TILE>())
lif_fc_forward_queue_kernel(const Event* __restrict__ ev, const int* __restrict__ ev_count, long long ev_cap,
                            const float* __restrict__ wt, int ld, int n_post, int k_post, SolveConst sk,
                            int* __restrict__ n_spikes, float* __restrict__ a_out, float* __restrict__ x_out,
                            float* __restrict__ t_out, float* __restrict__ z_out, int* __restrict__ status, int pad,
                            const int* __restrict__ order, int* __restrict__ head, int n_tiles, int n_items) {
    pdl_prologue();
    extern __shared__ __align__(128) unsigned char smem_raw[];
    using Smem = FwdSmem<TILE, SEV, STAGES>;
    Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
    ItemMailbox& box = *reinterpret_cast<ItemMailbox*>(smem_raw + mailbox_offset<Smem>());
    constexpr int CONSUMER_WARPS = TILE / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int q = 0; q < 2; ++q) {
            mbar_init(&box.full[q], 1);
            mbar_init(&box.empty[q], CONSUMER_WARPS);
        }
    }
    forward_init(sm, CONSUMER_WARPS);  // thread 0: the stage barriers, then the barrier-init fence
    __syncthreads();
    RingPos<STAGES> pos;
    if (warp == CONSUMER_WARPS) {
        for (int it = 0;; ++it) {
            int item = 0;
            if (lane == 0) item = atomicAdd(head, 1);
            item = __shfl_sync(0xffffffffu, item, 0);
            WorkItem w = {-1, 0, 0, 0};
            if (item < n_items) {
                const int r = item / n_tiles;
                w.s = __ldg(order + r);
                w.tile0 = (item - r * n_tiles) * TILE;
                w.E = __ldg(ev_count + w.s);
            }
            const int q = it & 1;
            const bool ok = mbar_wait(&box.empty[q], ((it >> 1) & 1) ^ 1, &sm.abort, status);
            if (!__all_sync(0xffffffffu, ok)) break;
            if (lane == 0) {
                box.item[q] = w;
                mbar_arrive(&box.full[q]);  // release: the item is visible to the consumers' acquiring wait
            }
            if (w.s < 0) break;
            if (!forward_produce(sm, pos, it, ev + (long long)w.s * ev_cap, w.E, wt, ld, w.tile0, CONSUMER_WARPS, sk,
                                 lane, status))
                break;
        }
        if (sm.abort) forward_drain(sm, pos.k);
        return;
    }
    for (int it = 0;; ++it) {
        const int q = it & 1;
        const bool ok = mbar_wait(&box.full[q], (it >> 1) & 1, &sm.abort, status);
        if (!__all_sync(0xffffffffu, ok)) return;
        const volatile int* vi = reinterpret_cast<const volatile int*>(&box.item[q]);
        const int s = vi[0], tile0 = vi[1], E = vi[2];
        __syncwarp();
        if (lane == 0) mbar_arrive(&box.empty[q]);
        if (s < 0) return;
        if (!forward_tile_item<TILE, SEV, STAGES, SCREEN>(sm, pos, it, s, tile0, E, n_post, k_post, sk, n_spikes,
                                                               a_out, x_out, t_out, z_out, status, pad))
            return;
    }
}

// Longest-first order of the samples for lif_fc_forward_queue_kernel, and the reset of its queue head. The
// samples are ranked by descending event count in 512 logarithmic classes (16 per octave: the exponent and
// top four mantissa bits of the float count + 1); the order inside a class is whatever the atomics give,
// which changes only the schedule, never a result. One CTA of 1024 threads. head may be null (bats_sample_order:
// the order alone, for the sort of the layer's output spikes).
__device__ __forceinline__ int count_class(int c) {
    const int key = (int)(__float_as_uint((float)(c + 1)) >> 19) - (127 << 4);  // increasing in c, >= 0
    return 511 - min(511, max(0, key));
}

__global__ void __launch_bounds__(1024) work_order_kernel(const int* __restrict__ ev_count, int batch,
                                                          int* __restrict__ head, int* __restrict__ order) {
    pdl_prologue();
    __shared__ int off[512];
    __shared__ int warp_sum[16];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < 512) off[tid] = 0;
    if (tid == 0 && head) *head = 0;
    __syncthreads();
    for (int s = tid; s < batch; s += blockDim.x) atomicAdd(&off[count_class(ev_count[s])], 1);
    __syncthreads();
    // Exclusive scan of the 512 class sizes: 16 warps of 32 classes, then the warp totals.
    int v = 0, incl = 0;
    if (tid < 512) {
        v = off[tid];
        incl = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += u;
        }
        if (lane == 31) warp_sum[warp] = incl;
    }
    __syncthreads();
    if (tid < 512) {
        int base = 0;
        for (int w = 0; w < warp; ++w) base += warp_sum[w];
        off[tid] = base + incl - v;
    }
    __syncthreads();
    for (int s = tid; s < batch; s += blockDim.x) order[atomicAdd(&off[count_class(ev_count[s])], 1)] = s;
}

// Event-parallel variant for layers with little neuron parallelism (few post neurons, or a small
// batch with long event streams): one warp per (sample, post neuron), the 32 lanes taking 32
// consecutive events. Per block of 32 events:
//   1. the states after each event are formed by the reference's sequential FMA chain
//      (a = fma(w, e^{t/tau_s}, a), b = fma(w, e^{t/tau}, b), event order), every lane running the
//      same chain over the block's (w, exponentials) in warp-private shared memory and keeping the
//      state after its own event;
//   2. every lane evaluates the provable screen (may_cross, its event's constants formed once) on its own state (one ballot);
//   3. candidates are taken in event order by their lane with the exact solver; a spike's reset
//      changes b for the later events of the block, whose b chain is then re-run from the spiking
//      event (a is unaffected by resets) and whose tests are re-evaluated.
// The arithmetic per event is that of the reference's loop, so results are bit-identical to the
// tile kernel's. What bounds it: the latency of a block's chain of dependent steps where there are few warps (the loads,
// hence two blocks ahead), instruction issue where there are many; a 32-event block costs about 230 instructions for one
// neuron, against the tile kernel's ~100 per 32 neurons and event, so the variant pays off when B * N_post is small against
// the GPU's ~5000 resident warps. With the event and its weight loaded together one block ahead (the second waiting for the
// first) and the fuller test: 20 neurons, one sample of 2800 events 60 -> 46 us; 4096 warps of 3600 events 138 -> 117 us; 8192 of
// 2400: 197 -> 173 us. (Copies into a ring in shared memory four blocks ahead: 50, 138 and 201 us, 20 % more instructions.)
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
lif_fc_forward_lanes_kernel(const Event* __restrict__ ev, const int* __restrict__ ev_count, long long ev_cap,
                            const float* __restrict__ wt, int ld, int n_post, int k_post, SolveConst sk,
                            int* __restrict__ n_spikes, float* __restrict__ a_out, float* __restrict__ x_out,
                            float* __restrict__ t_out, float* __restrict__ z_out, int pad) {
    pdl_prologue();
    __shared__ float4 blk[WARPS][32];  // the block's events as (t, w, es, e)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int s = blockIdx.y;
    const int i = blockIdx.x * WARPS + warp;
    if (i >= n_post) return;  // whole warp
    const int E = ev_count[s];
    const Event* evs = ev + (long long)s * ev_cap;
    const long long obase = ((long long)s * n_post + i) * k_post;
    float* ao = a_out + obase;
    float* xo = x_out + obase;
    float* to = t_out + obase;
    float* zo = z_out + obase;
    float a = 0.0f, b = 0.0f;
    int n = 0;
    bool done = false;
    float4* my = blk[warp];
    // Events in registers two blocks ahead and their weights, whose addresses they hold, one: neither load waits on the other.
    const Event* ev_from = evs + lane;
    const float* w_from = wt + i;
    auto event_at = [&](int m) {
        return m + lane < E ? __ldg(reinterpret_cast<const float4*>(ev_from + m)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    };
    auto weight_of = [&](const float4& e, int m) {
        return m + lane < E ? __ldg(w_from + (long long)__float_as_int(e.y) * ld) : 0.0f;
    };
    float4 e4_nx = event_at(0), e4_nx2 = event_at(32);
    float w_nx = weight_of(e4_nx, 0);
    for (int m0 = 0; m0 < E && !done; m0 += 32) {
        const int m = m0 + lane;
        const int cnt = min(32, E - m0);
        const bool in = lane < cnt;
        const float4 e4 = e4_nx;  // (t, j, es, e); zeros past the end
        my[lane] = make_float4(e4.x, w_nx, e4.z, e4.w);
        e4_nx = e4_nx2;
        w_nx = weight_of(e4_nx, m0 + 32);
        e4_nx2 = event_at(m0 + 64);
        // Window end: the next event's time and exponential (+inf after the last event).
        float t_nx = __shfl_sync(0xffffffffu, lane == 0 ? e4_nx.x : e4.x, lane + 1);
        float e_nx = __shfl_sync(0xffffffffu, lane == 0 ? e4_nx.w : e4.w, lane + 1);
        if (m + 1 >= E) {
            t_nx = BATS_INF;
            e_nx = BATS_INF;
        }
        const CrossWindow win = cross_window(e4.z, e4.w, e4.w, e_nx, sk);
        // 1. sequential chain.
        __syncwarp();
        // Lane l stops after event l: its state is the chain's l-th prefix, with no select per step.
        float am = a, bm = b;
#pragma unroll
        for (int k = 0; k < 32; ++k) {
            const float4 q = my[k];
            if (k <= lane) {
                am = fmaf(q.y, q.z, am);
                bm = fmaf(q.y, q.w, bm);
            }
        }
        // 2. provable no-crossing tests of all lanes at once.
        unsigned cand = __ballot_sync(0xffffffffu, in && may_cross(am, bm, win, sk));
        // 3. candidates in event order.
        while (cand) {
            const int u = __ffs(cand) - 1;
            int spiked = 0;
            int full = 0;
            if (lane == u) {
                const int n0 = n;
                full = solve_candidate<false>(am, bm, e4.x, t_nx, win, sk, n, k_post, 0, ao, xo, to, zo) ? 1 : 0;
                spiked = n - n0;
            }
            n = __shfl_sync(0xffffffffu, n, u);
            spiked = __shfl_sync(0xffffffffu, spiked, u);
            if (__shfl_sync(0xffffffffu, full, u)) {
                done = true;
                break;
            }
            if (spiked) {
                float cb2 = __shfl_sync(0xffffffffu, bm, u);
#pragma unroll 4
                for (int k = u + 1; k < cnt; ++k) {
                    const float4 q = my[k];
                    if (k <= lane) cb2 = fmaf(q.y, q.w, cb2);
                }
                bm = lane > u ? cb2 : bm;
                cand = __ballot_sync(0xffffffffu, in && lane > u && may_cross(am, bm, win, sk));
            } else {
                cand &= cand - 1u;
            }
        }
        a = __shfl_sync(0xffffffffu, am, cnt - 1);
        b = __shfl_sync(0xffffffffu, bm, cnt - 1);
        __syncwarp();
    }
    if (lane == 0) n_spikes[(long long)s * n_post + i] = n;
    for (int q = n + lane; pad && q < k_post; q += 32) {
        to[q] = BATS_INF;
        zo[q] = BATS_INF;
    }
}

template <int WARPS>
static int launch_forward_lanes(const void* events, const int* ev_count, long long ev_cap, const float* wt, int ld,
                                int batch, int n_post, int k_post, const SolveConst& sk, int* n_spikes, float* a,
                                float* x, float* times, float* post_exp_tau, int pad, cudaStream_t stream) {
    dim3 grid((n_post + WARPS - 1) / WARPS, batch);
    BATS_CUDA(bats::launch(lif_fc_forward_lanes_kernel<WARPS>, grid, WARPS * 32, 0, stream,
        reinterpret_cast<const Event*>(events), ev_count, ev_cap, wt, ld, n_post, k_post, sk, n_spikes, a, x, times,
        post_exp_tau, pad));
    BATS_CUDA(cudaGetLastError());
    return BATS_OK;
}

template <int TILE, int SEV, int STAGES, bool SCREEN>
static int launch_forward(const void* events, const int* ev_count, long long ev_cap, const float* wt, int ld, int batch,
                          int n_post, int k_post, const SolveConst& sk, int* n_spikes, float* a, float* x,
                          float* times, float* post_exp_tau, int* status, int pad, cudaStream_t stream) {
    const size_t smem = sizeof(FwdSmem<TILE, SEV, STAGES>);
    BATS_CUDA((cudaError_t)max_dynamic_smem_set((const void*)lif_fc_forward_kernel<TILE, SEV, STAGES, SCREEN>,
                                                (int)smem));
    dim3 grid((n_post + TILE - 1) / TILE, batch);
    BATS_CUDA(bats::launch(lif_fc_forward_kernel<TILE, SEV, STAGES, SCREEN>, grid, TILE + 32, smem, stream,
        reinterpret_cast<const Event*>(events), ev_count, ev_cap, wt, ld, n_post, k_post, sk, n_spikes, a, x, times,
        post_exp_tau, status, pad));
    BATS_CUDA(cudaGetLastError());
    return BATS_OK;
}

// Work-queue launch: the order kernel, then a grid of as many CTAs of the persistent kernel as are resident
// at once on this GPU (at most one per work item).
template <int TILE, int SEV, int STAGES, bool SCREEN>
static int launch_forward_queue(const void* events, const int* ev_count, long long ev_cap, const float* wt, int ld,
                                int batch, int n_post, int k_post, const SolveConst& sk, int* n_spikes, float* a,
                                float* x, float* times, float* post_exp_tau, int* status, int pad, int* order,
                                int* head, cudaStream_t stream) {
    using Smem = FwdSmem<TILE, SEV, STAGES>;
    const size_t smem = mailbox_offset<Smem>() + sizeof(ItemMailbox);
    const void* kern = (const void*)lif_fc_forward_queue_kernel<TILE, SEV, STAGES, SCREEN>;
    BATS_CUDA((cudaError_t)max_dynamic_smem_set(kern, (int)smem));
    int dev = 0, n_sm = 0, per_sm = 0;
    BATS_CUDA(cudaGetDevice(&dev));
    BATS_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    BATS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &per_sm, lif_fc_forward_queue_kernel<TILE, SEV, STAGES, SCREEN>, TILE + 32, smem));
    const int n_tiles = (n_post + TILE - 1) / TILE;
    BATS_REQUIRE((long long)batch * n_tiles < (1LL << 31), BATS_ERR_BAD_SHAPE,
                 "lif_forward_fc_queue: batch * post-neuron tiles must stay below 2^31");
    const int n_items = batch * n_tiles;
    const int grid = (int)std::min<long long>(n_items, (long long)std::max(1, per_sm) * std::max(1, n_sm));
    BATS_CUDA(bats::launch(work_order_kernel, 1, 1024, 0, stream, ev_count, batch, head, order));
    BATS_CUDA(cudaGetLastError());
    BATS_CUDA(bats::launch(lif_fc_forward_queue_kernel<TILE, SEV, STAGES, SCREEN>, grid, TILE + 32, smem, stream,
        reinterpret_cast<const Event*>(events), ev_count, ev_cap, wt, ld, n_post, k_post, sk, n_spikes, a, x, times,
        post_exp_tau, status, pad, order, head, n_tiles, n_items));
    BATS_CUDA(cudaGetLastError());
    return BATS_OK;
}

// The stage-screen choice (a run-time flag) mapped onto the kernel template.
template <int TILE, int SEV, int STAGES, typename... Args>
static int launch_tile(bool screen, Args... args) {
    return screen ? launch_forward<TILE, SEV, STAGES, true>(args...)
                  : launch_forward<TILE, SEV, STAGES, false>(args...);
}
template <int TILE, int SEV, int STAGES, typename... Args>
static int launch_queue(bool screen, Args... args) {
    return screen ? launch_forward_queue<TILE, SEV, STAGES, true>(args...)
                  : launch_forward_queue<TILE, SEV, STAGES, false>(args...);
}

SolveConst make_solve_const(float c, float dtt, float tau, float max_sim) {
    SolveConst k;
    k.c = c;
    k.dtt = dtt;
    k.tau = tau;
    k.max_sim = max_sim;
    const double em = std::exp((double)max_sim / (double)tau);
    k.e_max = std::isfinite(em) && em < 3.0e38 ? (float)em : std::numeric_limits<float>::infinity();
    k.inv_c = c > 0.0f ? 1.0f / c : 0.0f;
    k.fast = c > 0.0f && tau > 0.0f;
    set_screen_const(k);
    return k;
}

}  // namespace bats

static int forward_fc_impl(const void* events, const int* ev_count, long long ev_cap, const float* weights_t, int ld,
                           int batch, int n_post, int k_post, float c, float delta_theta_tau, float tau,
                           float max_simulation, int* n_spikes, float* a, float* x, float* times, float* post_exp_tau,
                           int algo, cudaStream_t stream) {
    BATS_REQUIRE(batch >= 0 && n_post >= 0 && k_post > 0 && ld >= n_post && ld % 4 == 0, BATS_ERR_BAD_SHAPE,
                 "lif_forward_fc: bad shape (ld must be >= n_post and a multiple of 4)");
    const int pad = (algo & BATS_FWD_NO_PAD) ? 0 : 1;
    const bool screen = (algo & BATS_FWD_STAGE_SCREEN) != 0;
    algo &= ~(BATS_FWD_NO_PAD | BATS_FWD_STAGE_SCREEN);
    BATS_REQUIRE(algo >= BATS_FWD_AUTO && algo <= BATS_FWD_TILE64, BATS_ERR_BAD_SHAPE, "lif_forward_fc: unknown algo");
    if (batch == 0 || n_post == 0) return BATS_OK;
    BATS_REQUIRE(events && ev_count && weights_t && n_spikes && a && x && times && post_exp_tau, BATS_ERR_NULL,
                 "lif_forward_fc: null pointer");
    BATS_REQUIRE(((uintptr_t)weights_t & 15) == 0 && ((uintptr_t)events & 15) == 0, BATS_ERR_BAD_SHAPE,
                 "lif_forward_fc: weights_t and events must be 16-byte aligned");
    const bats::SolveConst sk = bats::make_solve_const(c, delta_theta_tau, tau, max_simulation);
    const bool pick = algo == BATS_FWD_AUTO;
    if (pick)
        algo = bats_lif_forward_fc_default_algo(batch, n_post, (int)(ev_cap < (1LL << 30) ? ev_cap : (1LL << 30)));
    if (algo == BATS_FWD_LANES)
        return bats::launch_forward_lanes<4>(events, ev_count, ev_cap, weights_t, ld, batch, n_post, k_post, sk,
                                             n_spikes, a, x, times, post_exp_tau, pad, stream);
    int* status = nullptr;
    BATS_CUDA((cudaError_t)bats::device_status(&status));
    if (algo == BATS_FWD_TILE64)
        return bats::launch_tile<64, 16, 6>(screen, events, ev_count, ev_cap, weights_t, ld, batch, n_post, k_post, sk,
                                              n_spikes, a, x, times, post_exp_tau, status, pad, stream);
    if (n_post <= 32)
        return bats::launch_tile<32, 16, 8>(screen, events, ev_count, ev_cap, weights_t, ld, batch, n_post, k_post, sk,
                                               n_spikes, a, x, times, post_exp_tau, status, pad, stream);
    if (n_post <= 64)
        return bats::launch_tile<64, 16, 6>(screen, events, ev_count, ev_cap, weights_t, ld, batch, n_post, k_post, sk,
                                              n_spikes, a, x, times, post_exp_tau, status, pad, stream);
    // 64-neuron tiles with 8-event stages where 128-neuron tiles would be filled less than 1 / 1.15 as well, up to about 20
    // CTAs per SM (300 neurons, 256 samples, 150 / 800 events: 92 against 113 us, 237 against 279; 131 neurons, 128 samples, 3500
    // events: 0.9 of the time; 131 neurons, 1024 samples, above the line: 135 / 144, 467 / 449).
    const long long w64 = (n_post + 63) / 64, w128 = 2 * ((n_post + 127) / 128);
    if (pick && 100 * w128 >= 115 * w64 && w64 * batch <= 152 * 20)
        return bats::launch_tile<64, 8, 6>(screen, events, ev_count, ev_cap, weights_t, ld, batch, n_post, k_post, sk,
                                             n_spikes, a, x, times, post_exp_tau, status, pad, stream);
    // 8-event stages: half the shared memory of 16-event stages (26 KB), so 8 CTAs (32 consumer warps) fit on an SM
    // instead of 4, and a replay after a possible crossing covers fewer events.
    return bats::launch_tile<128, 8, 6>(screen, events, ev_count, ev_cap, weights_t, ld, batch, n_post, k_post, sk,
                                          n_spikes, a, x, times, post_exp_tau, status, pad, stream);
}

extern "C" int bats_lif_forward_fc_default_algo(int batch, int n_post, int ev_cap) {
    (void)ev_cap;
    // Warp per (sample, neuron): its time grows with the number of warps, that of the tile kernel with the number of tiles
    // and, below about a wave, with nothing. The lines are where both meet, per sub-partition of a 152-SM GPU; measured
    // with input lists of 150 / 800 / 3500 events, lanes against tile in us:
    //   at most 8 neurons (three quarters of a tile idle): always (4 neurons, 4096 samples: 199 / 343)
    //   at most 16: 20 warps (12 neurons, 1024 samples 66 / 74, 168 / 164; 16 and 4096: 715 / 433, above the line)
    //   at most 32: 16 warps (32 neurons, 256 samples: 50 / 87, 118 / 148, 259 / 363; 512 samples: 214 / 160, above)
    //     These are output layers, which spike, on batches of uneven samples, where a tile lasts as long as its longest one: 32
    //     neurons, 256 samples of 2400 events, sigma of their logarithm 0.3, 6 spikes a neuron 262 / 380 to 575. Layers that
    //     stay silent pay (24 neurons, 256 samples of 718 events 54 / 40, of 2880 197 / 127), and so do even batches of few
    //     spikes (32 neurons, 256 samples of 719, 2 spikes 70 / 50); no host knows either. (Tiles through the quiet beginning
    //     and a second launch of warps per neuron from there: silent 132 us at 2880 events, but 30 us on top of every spiking layer.)
    //   wider: 8 warps (131 neurons, 32 samples: 31 / 64, 70 / 156, 136 / 388; silent layers 15 / 21, 44 / 58; twice as
    //   many warps are still faster where the neurons spike, 52 / 70, 120 / 158, but not where they are silent, 79 / 58)
    const long long warps = (long long)batch * n_post;
    const long long per_sub = n_post <= 8 ? warps : n_post <= 16 ? 20 : n_post <= 32 ? 16 : 8;
    return warps <= 152LL * 4 * per_sub ? BATS_FWD_LANES : BATS_FWD_TILE;
}

extern "C" int bats_lif_forward_fc(const void* events, const int* ev_count, long long ev_cap, const float* weights_t,
                                   int ld, int batch, int n_post, int k_post, float c, float delta_theta_tau,
                                   float tau, float max_simulation, int* n_spikes, float* a, float* x, float* times,
                                   float* post_exp_tau, cudaStream_t stream) {
    return forward_fc_impl(events, ev_count, ev_cap, weights_t, ld, batch, n_post, k_post, c, delta_theta_tau, tau,
                           max_simulation, n_spikes, a, x, times, post_exp_tau, BATS_FWD_AUTO, stream);
}

extern "C" int bats_lif_forward_fc_algo(const void* events, const int* ev_count, long long ev_cap,
                                        const float* weights_t, int ld, int batch, int n_post, int k_post, float c,
                                        float delta_theta_tau, float tau, float max_simulation, int* n_spikes,
                                        float* a, float* x, float* times, float* post_exp_tau, int algo,
                                        cudaStream_t stream) {
    return forward_fc_impl(events, ev_count, ev_cap, weights_t, ld, batch, n_post, k_post, c, delta_theta_tau, tau,
                           max_simulation, n_spikes, a, x, times, post_exp_tau, algo, stream);
}

extern "C" int bats_sample_order(const int* ev_count, int batch, int* order, cudaStream_t stream) {
    BATS_REQUIRE(batch >= 0, BATS_ERR_BAD_SHAPE, "sample_order: bad shape");
    if (batch == 0) return BATS_OK;
    BATS_REQUIRE(ev_count && order, BATS_ERR_NULL, "sample_order: null pointer");
    BATS_CUDA(bats::launch(bats::work_order_kernel, 1, 1024, 0, stream, ev_count, batch, (int*)nullptr, order));
    BATS_CUDA(cudaGetLastError());
    return BATS_OK;
}

extern "C" size_t bats_lif_forward_fc_queue_workspace_bytes(int batch) {
    // The queue head (own 256-byte line), then the sample order.
    return 256 + ((size_t)(batch > 0 ? batch : 0) * sizeof(int) + 255) / 256 * 256;
}

extern "C" int bats_lif_forward_fc_queue(const void* events, const int* ev_count, long long ev_cap,
                                         const float* weights_t, int ld, int batch, int n_post, int k_post, float c,
                                         float delta_theta_tau, float tau, float max_simulation, int* n_spikes,
                                         float* a, float* x, float* times, float* post_exp_tau, int algo,
                                         void* workspace, size_t workspace_bytes, cudaStream_t stream) {
    BATS_REQUIRE(batch >= 0 && n_post >= 0 && k_post > 0 && ld >= n_post && ld % 4 == 0, BATS_ERR_BAD_SHAPE,
                 "lif_forward_fc_queue: bad shape (ld must be >= n_post and a multiple of 4)");
    const int pad = (algo & BATS_FWD_NO_PAD) ? 0 : 1;
    const bool screen = (algo & BATS_FWD_STAGE_SCREEN) != 0;
    algo &= ~(BATS_FWD_NO_PAD | BATS_FWD_STAGE_SCREEN);
    BATS_REQUIRE(algo == BATS_FWD_AUTO || algo == BATS_FWD_TILE || algo == BATS_FWD_TILE64, BATS_ERR_BAD_SHAPE,
                 "lif_forward_fc_queue: algo must be BATS_FWD_AUTO, BATS_FWD_TILE or BATS_FWD_TILE64");
    if (batch == 0 || n_post == 0) return BATS_OK;
    BATS_REQUIRE(events && ev_count && weights_t && n_spikes && a && x && times && post_exp_tau && workspace,
                 BATS_ERR_NULL, "lif_forward_fc_queue: null pointer");
    BATS_REQUIRE(((uintptr_t)weights_t & 15) == 0 && ((uintptr_t)events & 15) == 0, BATS_ERR_BAD_SHAPE,
                 "lif_forward_fc_queue: weights_t and events must be 16-byte aligned");
    BATS_REQUIRE(((uintptr_t)workspace & 15) == 0 &&
                     workspace_bytes >= bats_lif_forward_fc_queue_workspace_bytes(batch),
                 BATS_ERR_WORKSPACE, "lif_forward_fc_queue: workspace too small or not 16-byte aligned");
    const bats::SolveConst sk = bats::make_solve_const(c, delta_theta_tau, tau, max_simulation);
    int* status = nullptr;
    BATS_CUDA((cudaError_t)bats::device_status(&status));
    int* head = reinterpret_cast<int*>(workspace);
    int* order = reinterpret_cast<int*>(reinterpret_cast<char*>(workspace) + 256);
    if (algo == BATS_FWD_TILE64 || (n_post > 32 && n_post <= 64))
        return bats::launch_queue<64, 16, 6>(screen, events, ev_count, ev_cap, weights_t, ld, batch, n_post, k_post,
                                                    sk, n_spikes, a, x, times, post_exp_tau, status, pad, order, head,
                                                    stream);
    if (n_post <= 32)
        return bats::launch_queue<32, 16, 8>(screen, events, ev_count, ev_cap, weights_t, ld, batch, n_post, k_post,
                                                    sk, n_spikes, a, x, times, post_exp_tau, status, pad, order, head,
                                                    stream);
    return bats::launch_queue<128, 8, 6>(screen, events, ev_count, ev_cap, weights_t, ld, batch, n_post, k_post, sk,
                                                n_spikes, a, x, times, post_exp_tau, status, pad, order, head, stream);
}
