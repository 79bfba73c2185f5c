// Convolutional LIF layer (valid convolution, stride 1) and 2x2 spike-union pooling.
//
// Neuron layouts follow the reference: a neuron (x, y, c) of a (X, Y, C) layer has index
// (x*Y + y)*C + c; filters are (C_out, fx, fy, C_in) (bats/Layers/ConvLIFLayer.py:20-37).
//
// Forward (replaces compute_spike_times_conv, bats/CudaKernels/CuFiles/Inference/compute_spike_times_conv.cu:93-174):
// the reference tests every event of the sample against every post neuron's receptive field and
// runs the crossing search after each event, relevant or not. Here a CTA owns a spatial tile of
// post positions x all output channels, keeps only the events inside the tile's receptive field,
// and each thread integrates only the events of its own receptive field, searching for crossings
// in (t_prev_relevant, t_this_relevant] before adding the next one. Because the neuron state does
// not change at an irrelevant event and the reference's windows between consecutive events tile
// that interval, this finds the same spikes with the same arithmetic. An event outside the field
// changes the reference's state only when one of its exponentials is not finite (an input later than
// about 88 tau_s overflows exp(t/tau_s)): its weight 0 times +inf is NaN, which the reference's solver
// turns into NaN spikes. Such events are therefore relevant to every neuron, with weight 0 outside the
// field, exactly as the reference adds them.
//
// Backward (replaces compute_weights_gradient_conv and propagate_errors_to_pre_spikes_conv,
// .../Backpropagation/compute_weights_gradient_conv.cu:11-61, propagate_errors_to_pre_spikes_conv.cu:11-89):
// per event and filter tap (c_out, dx, dy), the post neuron (x-dx, y-dy, c_out)'s first spike after the event gives a
// gradient term and a weighted error term. A cluster of eight CTAs per sample (group), each with a copy of the filter gradient
// in shared memory, added up in rank order; no atomics. With the events grouped by input position: a thread per tap
// (conv_backward_taps_kernel) or, where few neurons spike, a lane per event (conv_backward_grouped_kernel); without,
// conv_backward_cluster_kernel in time order. Filters too large for shared memory: one CTA per sample (conv_backward_kernel).
//
// Pooling (replaces aggregate_spikes_conv + argsort, .../Inference/aggregate_spikes_conv.cu:6-43,
// Wrappers/Inference/aggregate_spikes_conv.py:10-28; backward bats/Layers/PoolingLayer.py:55-66):
// a stable 4-way merge of the children's sorted spike lists, inf slots last in concatenation order.
#include <cooperative_groups.h>
#include <numeric>
#include <type_traits>
#include "common.cuh"
#include "async_copy.cuh"
#include "conv_form.cuh"
#include "abi_util.h"

namespace bats {

// An event inside the receptive field of a CTA's positions.
struct __align__(16) ConvEvent {
    float t, es, e;
    int xyc;  // x | y << 10 | c << 20; bit 31: an exponential is not finite (relevant to every neuron)
};

constexpr int CONV_GROUP = 8;              // list entries per pass of the screen
constexpr int CONV_POSITIONS = 16;         // positions per CTA at most (2.9 KB of list each)

// One position's list of relevant events, in time order: window constants (the window ends at the next relevant
// event), times and filter rows ((dx fy + dy) C + c, or -1: weight 0). SUB: kept events per round of the lists.
template <int SUB>
struct ConvList {
    CrossWindow win[SUB + CONV_GROUP];
    float t[SUB + CONV_GROUP + 1];
    int row[SUB + CONV_GROUP];
    int n;       // entries
    int groups;  // groups of CONV_GROUP entries that may be processed (the last entry waits for its window's end)
    int pad_[5];
};

// Appends the kept events sev[0 .. cnt) that are relevant to position (xo, yo) to its list (one warp): the entries not
// processed yet move to the front, the new ones follow, and the window constants are formed. last: no event follows,
// so the last window ends at +inf and the last group may be short.
template <int SUB>
__device__ __forceinline__ void conv_list_append(ConvList<SUB>& l, const ConvEvent* sev, int cnt, bool last, int xo, int yo,
                                                 int fx, int fy, int C, const SolveConst& sk, int lane) {
    int n = l.n;
    const int from = l.groups * CONV_GROUP;
    float t = 0.0f, es = 0.0f, e = 0.0f;
    int row = 0;
    n -= from;  // at most CONV_GROUP entries are left over
    if (lane < n) {
        t = l.t[from + lane];
        row = l.row[from + lane];
        es = l.win[from + lane].es;
        e = l.win[from + lane].e;
    }
    __syncwarp();
    if (lane < n) {
        l.t[lane] = t;
        l.row[lane] = row;
        l.win[lane].es = es;
        l.win[lane].e = e;
    }
    for (int q0 = 0; q0 < cnt; q0 += 32) {
        ConvEvent ev = {0.0f, 0.0f, 0.0f, 0};
        bool rel = false;
        if (q0 + lane < cnt) {
            ev = sev[q0 + lane];
            const int dx = (ev.xyc & 1023) - xo, dy = ((ev.xyc >> 10) & 1023) - yo;
            const bool in = dx >= 0 && dx < fx && dy >= 0 && dy < fy;
            row = in ? (dx * fy + dy) * C + ((ev.xyc >> 20) & 2047) : -1;
            rel = in || ev.xyc < 0;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, rel);
        if (rel) {
            const int at = n + __popc(bal & lanemask_lt());
            l.t[at] = ev.t;
            l.row[at] = row;
            l.win[at].es = ev.es;
            l.win[at].e = ev.e;
        }
        n += __popc(bal);
    }
    __syncwarp();
    for (int u = lane; u < n; u += 32) {
        const float e_u = l.win[u].e;
        const float e_next = u + 1 < n ? l.win[u + 1].e : BATS_INF;
        const CrossWindow w = cross_window(0.0f, 0.0f, e_u, e_next, sk);
        l.win[u].czz = w.czz;
        l.win[u].zw = w.zw;
        l.win[u].tcz = w.tcz;
        l.win[u].czzl = w.czzl;
        l.win[u].zl = w.zl;
        l.win[u].tczl = w.tczl;
    }
    const int groups = last ? (n + CONV_GROUP - 1) / CONV_GROUP : max(0, n - 1) / CONV_GROUP;
    // A short last group is filled up with events of weight and exponentials 0, which leave the state unchanged.
    for (int u = n + lane; u < groups * CONV_GROUP; u += 32) {
        l.row[u] = -1;
        l.win[u] = CrossWindow{0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    }
    if (lane == 0) {
        l.t[n] = BATS_INF;
        l.n = n;
        l.groups = groups;
    }
}

// CTA per (tile of TX x TY positions, sample), thread = (position, output channel). The sample's events inside the
// tile's receptive field are compacted into shared memory; SUB of them at a time, a warp per position builds the
// position's own list of relevant events, which its C_out threads then run through in groups of CONV_GROUP, as the
// fully-connected tile kernel runs through a stage: a branch-free pass with the screen of every event, and the exact
// loop from the first event after which a crossing cannot be ruled out. A warp's lanes may belong to two positions:
// they step through their own lists side by side.
// What bounds it: instruction issue. 12 x 12 x 15 -> 5 x 5 x 40, batch 128: 1.78 -> 0.76 ms; before, every thread tested
// every event of the tile for its own field and ran the screen one event at a time, lanes of two positions after one
// another. SUB 32: 0.90 ms (more barriers); it takes half the shared memory, see conv_narrow.
template <bool W_SMEM, int SUB>
__global__ void __launch_bounds__(1024)
conv_forward_kernel(const Event* __restrict__ ev, const int* __restrict__ ev_count, long long ev_cap,
                    const float* __restrict__ W, int X, int Y, int C, int fx, int fy, int C_out, int Xo, int Yo,
                    int TX, int TY, int tiles_y, int k_post, SolveConst sk, int* __restrict__ n_spikes,
                    float* __restrict__ a_out, float* __restrict__ x_out, float* __restrict__ t_out,
                    float* __restrict__ z_out) {
    pdl_prologue();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int swarp[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nwarps = blockDim.x >> 5;
    const int P = TX * TY;
    ConvList<SUB>* lists = reinterpret_cast<ConvList<SUB>*>(smem_raw);
    ConvEvent* sev = reinterpret_cast<ConvEvent*>(lists + P);  // SUB + blockDim entries
    float* sW = reinterpret_cast<float*>(sev + SUB + blockDim.x);
    const int s = blockIdx.y;
    const int tx0 = (blockIdx.x / tiles_y) * TX, ty0 = (blockIdx.x % tiles_y) * TY;
    const int R = fx * fy * C, ldw = W_SMEM ? (R | 1) : R;  // odd: a row's channels lie in different banks
    if (W_SMEM)
        for (int co = warp; co < C_out; co += nwarps)
            for (int q = lane; q < R; q += 32) cp_async4(sW + co * ldw + q, W + co * R + q);
    for (int p = tid; p < P; p += blockDim.x) lists[p].n = lists[p].groups = 0;
    const int co = tid % C_out, pl = tid / C_out;
    const int xo = tx0 + pl / TY, yo = ty0 + pl % TY;
    const bool active = pl < P && xo < Xo && yo < Yo;
    const int n_post = Xo * Yo * C_out;
    const int post = (xo * Yo + yo) * C_out + co;
    const long long obase = ((long long)s * n_post + (active ? post : 0)) * k_post;
    const ConvList<SUB>& l = lists[active ? pl : 0];
    const float* wrow = (W_SMEM ? sW : W) + (active ? co * ldw : 0);
    auto weight = [&](int row) { return row >= 0 ? wrow[row] : 0.0f; };
    // Receptive field of the whole tile.
    const int rx0 = tx0, rx1 = min(X, tx0 + TX + fx - 1), ry0 = ty0, ry1 = min(Y, ty0 + TY + fy - 1);

    float a = 0.0f, b = 0.0f;
    int n = 0;
    bool done = !active;
    const int E = ev_count[s];
    const Event* evs = ev + (long long)s * ev_cap;
    int kept = 0;  // events in sev
    for (int m0 = 0;; m0 += blockDim.x) {
        // Keep the events of this round that fall in the tile's receptive field, in time order.
        const bool last_round = m0 + (int)blockDim.x >= E;
        bool keep = false;
        ConvEvent ce = {0.0f, 0.0f, 0.0f, 0};
        if (m0 + tid < E) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(evs + m0 + tid));  // (t, j, es, e)
            const int j = __float_as_int(v.y);
            const int cc = j % C, xy = j / C, yy = xy % Y, xx = xy / Y;
            const bool finite = isfinite(v.z) && isfinite(v.w);
            // In the tile's receptive field, or relevant to every neuron (a non-finite exponential).
            keep = (xx >= rx0 && xx < rx1 && yy >= ry0 && yy < ry1) || !finite;
            ce = {v.x, v.z, v.w, xx | (yy << 10) | (cc << 20) | (finite ? 0 : (int)0x80000000u)};
        }
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) swarp[warp] = __popc(bal);
        if (W_SMEM && m0 == 0) cp_async_wait_all();
        __syncthreads();
        int off = kept, tot = 0;
        for (int w = 0; w < nwarps; ++w) {
            off += w < warp ? swarp[w] : 0;
            tot += swarp[w];
        }
        if (keep) sev[off + __popc(bal & lanemask_lt())] = ce;
        kept += tot;
        __syncthreads();
        int head = 0;
        while (kept - head >= SUB || (last_round && head < kept) || (last_round && kept == 0)) {
            const int cnt = min(SUB, kept - head);
            const bool last = last_round && head + cnt == kept;
            for (int p = warp; p < P; p += nwarps)
                conv_list_append(lists[p], sev + head, cnt, last, tx0 + p / TY, ty0 + p % TY, fx, fy, C, sk, lane);
            __syncthreads();
            if (!done) {
                const int groups = l.groups, total = l.n;
                for (int g = 0; g < groups && !done; ++g) {
                    const CrossWindow* win = l.win + g * CONV_GROUP;
                    const int* row = l.row + g * CONV_GROUP;
                    const float* tt = l.t + g * CONV_GROUP;
                    const int cnt_g = min(CONV_GROUP, total - g * CONV_GROUP);
                    float aa = a, bb = b;
                    unsigned cand = 0u;
#pragma unroll
                    for (int u = 0; u < CONV_GROUP; ++u) {
                        const CrossWindow c = win[u];
                        const float w = weight(row[u]);
                        aa = fmaf(w, c.es, aa);
                        bb = fmaf(w, c.e, bb);
                        cand |= cross_bit<true>(aa, bb, c, sk, 1u << u);
                    }
                    cand &= (2u << (cnt_g - 1)) - 1u;  // not the events that fill up the last group
                    if (cand) {
                        const int first = __ffs(cand) - 1;
                        aa = a;
                        bb = b;
                        for (int u = 0; u <= first; ++u) {
                            const float w = weight(row[u]);
                            aa = fmaf(w, win[u].es, aa);
                            bb = fmaf(w, win[u].e, bb);
                        }
                        bool cross = true;
                        for (int u = first;;) {
                            if (cross && solve_candidate<true>(aa, bb, tt[u], tt[u + 1], win[u], sk, n, k_post, obase,
                                                               a_out, x_out, t_out, z_out)) {
                                done = true;
                                break;
                            }
                            if (++u >= cnt_g) break;
                            const CrossWindow c = win[u];
                            const float w = weight(row[u]);
                            aa = fmaf(w, c.es, aa);
                            bb = fmaf(w, c.e, bb);
                            cross = may_cross<true>(aa, bb, c, sk);
                        }
                    }
                    a = aa;
                    b = bb;
                }
            }
            head += cnt;
            if (__syncthreads_and(done) || last) {  // every buffer full, or no event left
                kept = head = 0;
                m0 = E;
                break;
            }
        }
        if (m0 >= E || last_round) break;
        // The events not in a list yet move to the front (fewer than SUB).
        ConvEvent mv;
        const int rest = kept - head;
        if (tid < rest) mv = sev[head + tid];
        __syncthreads();
        if (tid < rest) sev[tid] = mv;
        kept = rest;
    }
    if (active) n_spikes[(long long)s * n_post + post] = n;
    // +inf past each neuron's spikes: the lanes run along the warp's 32 rows of k_post slots, most of which lie next to
    // one another (a store per lane and slot of its own row would touch 32 lines).
    const int free_from = active ? n : k_post;
    int r = lane / k_post, k = lane - r * k_post;  // the warp's row and slot of this lane
    const int dr = 32 / k_post, dk = 32 - dr * k_post;
    for (int q = 0; q < k_post; ++q) {
        const int nr = __shfl_sync(0xffffffffu, free_from, r & 31);
        const long long pr = (long long)s * n_post + __shfl_sync(0xffffffffu, post, r & 31);
        if (k >= nr) {
            t_out[pr * k_post + k] = BATS_INF;
            z_out[pr * k_post + k] = BATS_INF;
        }
        r += dr;
        k += dk;
        if (k >= k_post) {
            k -= k_post;
            ++r;
        }
    }
}

// One CTA per sample; thread q handles filter taps q, q + blockDim, ... of (C_out, fx, fy).
__global__ void conv_backward_kernel(const Event* __restrict__ ev, const int* __restrict__ ev_slot,
                                     const int* __restrict__ ev_count, long long ev_cap, const float* __restrict__ W,
                                     int Y, int C, int fx, int fy, int C_out, int Xo, int Yo,
                                     const float* __restrict__ post_t, const float2* __restrict__ tab,
                                     const int* __restrict__ nvalid, int k_post, float tau_s, float tau,
                                     long long pre_slots, float* __restrict__ grad, float* __restrict__ pre_err) {
    pdl_prologue();
    __shared__ float sred[32][33];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nwarps = blockDim.x >> 5;
    const int s = blockIdx.x;
    const int taps = C_out * fx * fy;
    const int n_post = Xo * Yo * C_out;
    const int E = ev_count[s];
    const Event* evs = ev + (long long)s * ev_cap;
    float* gs = grad + (long long)s * taps * C;
    for (int m0 = 0; m0 < E; m0 += 32) {
        const int cnt = min(32, E - m0);
        for (int q = 0; q < cnt; ++q) {
            const Event e = evs[m0 + q];
            const int cc = e.j % C, xy = e.j / C, yy = xy % Y, xx = xy / Y;
            float term = 0.0f;
            for (int tp = tid; tp < taps; tp += blockDim.x) {
                const int co = tp / (fx * fy), dx = (tp / fy) % fx, dy = tp % fy;
                const int xo = xx - dx, yo = yy - dy;
                if (xo < 0 || yo < 0 || xo >= Xo || yo >= Yo) continue;
                const long long pn = (long long)s * n_post + (xo * Yo + yo) * C_out + co;
                const int n = nvalid[pn];
                const float* tp_ = post_t + pn * k_post;
                int p = 0;
                while (p < n && tp_[p] <= e.t) ++p;
                if (p >= n) continue;
                const float2 AB = tab[pn * (k_post + 1) + p];
                gs[(long long)tp * C + cc] += fmaf(e.es, AB.x, -(e.e * AB.y));
                if (pre_err) term += W[(long long)tp * C + cc] * (AB.x * e.es / tau_s - AB.y * e.e / tau);
            }
            if (pre_err) {
#pragma unroll
                for (int o = 16; o >= 1; o >>= 1) term += __shfl_xor_sync(0xffffffffu, term, o);
                if (lane == 0) sred[q][warp] = term;
            }
        }
        if (pre_err) {
            __syncthreads();
            if (tid < cnt) {
                float acc = 0.0f;
                for (int w = 0; w < nwarps; ++w) acc += sred[tid][w];
                pre_err[(long long)s * pre_slots + ev_slot[(long long)s * ev_cap + m0 + tid]] = acc;
            }
            __syncthreads();
        }
    }
}

// Conv backward on a cluster of CONV_BWD_CLUSTER CTAs per sample (thread-block cluster, distributed
// shared memory). Thread = filter tap (co, dx, dy); the sample's events are dealt to the cluster's CTAs in
// groups of 32 (group g to CTA rank g % CONV_BWD_CLUSTER), so that eight times as many CTAs hide the
// latency of the post-spike lookups. Every CTA accumulates its events' gradient terms in a shared-memory
// copy of the per-sample filter gradient (taps x C), in event order; at the end each CTA sums one slice of
// the gradient over the cluster's copies in rank order (deterministic) and writes it. The pre-spike errors
// of a group of events are reduced over the taps inside the CTA that owns the group. Four events are
// processed at a time so that their lookups (binary searches over the post neuron's spike times, table
// entries) are in flight together.
constexpr int CONV_BWD_CLUSTER = 8;
constexpr int CONV_BWD_ILP = 4;

__global__ void __launch_bounds__(1024)
conv_backward_cluster_kernel(const Event* __restrict__ ev, const int* __restrict__ ev_slot,
                             const int* __restrict__ ev_count, long long ev_cap, const float* __restrict__ W, int Y,
                             int C, int fx, int fy, int C_out, int Xo, int Yo, const float* __restrict__ post_t,
                             const float2* __restrict__ tab, const int* __restrict__ nvalid, int k_post,
                             int search_top, float tau_s, float tau, long long pre_slots, float* __restrict__ grad,
                             float* __restrict__ pre_err, int batch, int group) {
    pdl_prologue();
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) float Gs[];  // taps * C
    __shared__ Event sev[32];
    __shared__ float sred[32][33];
    const unsigned rank = cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nwarps = blockDim.x >> 5;
    const int taps = C_out * fx * fy;
    const int total = taps * C;
    const int n_post = Xo * Yo * C_out;
    for (int q = tid; q < total; q += blockDim.x) Gs[q] = 0.0f;
    __syncthreads();
    // The cluster's samples (one with group == 1: the per-sample gradient), accumulated in order.
    const int s_end = min(batch, ((int)blockIdx.y + 1) * group);
    for (int s = (int)blockIdx.y * group; s < s_end; ++s) {
    const int E = ev_count[s];
    const Event* evs = ev + (long long)s * ev_cap;
    for (int g = (int)rank; g * 32 < E; g += CONV_BWD_CLUSTER) {
        const int m0 = g * 32;
        const int cnt = min(32, E - m0);
        if (tid < cnt) sev[tid] = evs[m0 + tid];
        __syncthreads();
        for (int q0 = 0; q0 < cnt; q0 += CONV_BWD_ILP) {
            float term[CONV_BWD_ILP];
#pragma unroll
            for (int u = 0; u < CONV_BWD_ILP; ++u) term[u] = 0.0f;
            for (int tp = tid; tp < taps; tp += blockDim.x) {
                const int co = tp / (fx * fy), dx = (tp / fy) % fx, dy = tp % fy;
                long long pn[CONV_BWD_ILP];
                int nv[CONV_BWD_ILP], pos[CONV_BWD_ILP], cc[CONV_BWD_ILP];
                float et[CONV_BWD_ILP];
#pragma unroll
                for (int u = 0; u < CONV_BWD_ILP; ++u) {
                    nv[u] = 0;
                    pos[u] = 0;
                    pn[u] = 0;
                    cc[u] = 0;
                    et[u] = 0.0f;
                    if (q0 + u < cnt) {
                        const Event e = sev[q0 + u];
                        cc[u] = e.j % C;
                        const int xy = e.j / C, yy = xy % Y, xx = xy / Y;
                        const int xo = xx - dx, yo = yy - dy;
                        et[u] = e.t;
                        if (xo >= 0 && yo >= 0 && xo < Xo && yo < Yo) {
                            pn[u] = (long long)s * n_post + (xo * Yo + yo) * C_out + co;
                            nv[u] = nvalid[pn[u]];
                        }
                    }
                }
                // Fixed-depth binary searches, the ILP searches interleaved: pos = #{k < n : t_k <= t}.
                for (int step = search_top; step > 0; step >>= 1) {
#pragma unroll
                    for (int u = 0; u < CONV_BWD_ILP; ++u) {
                        const int cand = pos[u] + step;
                        if (cand <= nv[u] && post_t[pn[u] * k_post + cand - 1] <= et[u]) pos[u] = cand;
                    }
                }
#pragma unroll
                for (int u = 0; u < CONV_BWD_ILP; ++u) {
                    if (pos[u] < nv[u]) {
                        const Event e = sev[q0 + u];
                        const float2 AB = tab[pn[u] * (k_post + 1) + pos[u]];
                        Gs[tp * C + cc[u]] += fmaf(e.es, AB.x, -(e.e * AB.y));
                        if (pre_err) term[u] += W[(long long)tp * C + cc[u]] * (AB.x * e.es / tau_s - AB.y * e.e / tau);
                    }
                }
            }
            if (pre_err) {
#pragma unroll
                for (int u = 0; u < CONV_BWD_ILP; ++u) {
                    float v = term[u];
#pragma unroll
                    for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                    if (lane == 0 && q0 + u < cnt) sred[q0 + u][warp] = v;
                }
            }
        }
        __syncthreads();
        if (pre_err && tid < cnt) {
            float acc = 0.0f;
            for (int w = 0; w < nwarps; ++w) acc += sred[tid][w];
            pre_err[(long long)s * pre_slots + ev_slot[(long long)s * ev_cap + m0 + tid]] = acc;
        }
        __syncthreads();
    }
    }
    cluster.sync();
    const int per = (total + CONV_BWD_CLUSTER - 1) / CONV_BWD_CLUSTER;
    const int q_end = min(total, ((int)rank + 1) * per);
    for (int q = (int)rank * per + tid; q < q_end; q += blockDim.x) {
        float acc = 0.0f;
        for (int r = 0; r < CONV_BWD_CLUSTER; ++r) acc += cluster.map_shared_rank(Gs, r)[q];
        grad[(long long)blockIdx.y * total + q] = acc;
    }
    cluster.sync();  // no CTA leaves while another still reads its shared memory
}

// Conv backward over events grouped by input position (the bucketed copy of the sort with
// bucket_width = C: one bucket per (x, y), time order inside), on a cluster of CONV_BWD_CLUSTER CTAs per sample group
// (position groups dealt to the ranks). Within a position group every filter tap sees one and the same post neuron
// (x - dx, y - dy, co). Two kernels, whose results are the same bit for bit, run one after the other: the first, the taps form,
// leaves the batch to the second, the events form, where few enough neurons spike (no host knows it).
struct ConvBwdShape {
    int Y, C, fx, fy, C_out, Xo, Yo, k_pre, k_post, n_pos;
};

// TAPS: the taps form alone; CHOOSE: both are launched, and the first decides.
enum class ConvForm { TAPS, CHOOSE };

// Where the events form takes the batch, the taps form leaves this in the first word of every group's gradient, which the events
// form overwrites: the decision is made in one kernel and read in the other. No gradient can look so: it is the result of an
// addition, whose NaN is 0x7fffffff.
constexpr unsigned CONV_LEFT = 0x7fc0b175u;

// The decision (conv_events_pays) is the batch's, so that the kernels do not run their longest samples one after the other
// (with pre-errors a choice per group took 0.917 of the taps form's time, one for the batch 0.885, mean of 2150 layers). Every CTA forms it from
// the same sample of the batch, with no word between them: every nv_step-th neuron and every s_step-th sample.
struct ConvVoteShape {
    int nv_step, nv_count, s_step, s_count;
};
constexpr int CONV_VOTE = 1024;  // neurons and samples looked at, at most

// In two halves around a barrier of the caller's, which the loads overlap with what else comes before it: the warps' counts,
// then their sum. The same in every thread of the grid.
struct ConvVote {
    int spiking[32];
    unsigned long long events[32];
};
__device__ __forceinline__ void conv_vote_count(ConvVote& v, const ConvVoteShape& vs, const int* __restrict__ boff,
                                                const int* __restrict__ nvalid, const ConvBwdShape& sh) {
    int spiking = 0;
    unsigned long long events = 0;
    for (int q = threadIdx.x; q < vs.s_count; q += blockDim.x)
        events += (unsigned)__ldg(boff + (long long)q * vs.s_step * (sh.n_pos + 1) + sh.n_pos);
#pragma unroll 8
    for (int q = threadIdx.x; q < vs.nv_count; q += blockDim.x)
        spiking += __ldg(nvalid + (long long)q * vs.nv_step) > 0 ? 1 : 0;
    spiking = __reduce_add_sync(0xffffffffu, spiking);
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) events += __shfl_xor_sync(0xffffffffu, events, o);
    if ((threadIdx.x & 31) == 0) {
        v.spiking[threadIdx.x >> 5] = spiking;
        v.events[threadIdx.x >> 5] = events;
    }
}
__device__ __forceinline__ bool conv_events_form(const ConvVote& v, const ConvVoteShape& vs, const ConvBwdShape& sh,
                                                 int batch) {
    const int lane = threadIdx.x & 31;
    const bool on = lane < (int)(blockDim.x >> 5);
    const unsigned spiking = __reduce_add_sync(0xffffffffu, on ? (unsigned)v.spiking[lane] : 0u);
    unsigned long long events = on ? v.events[lane] : 0;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) events += __shfl_xor_sync(0xffffffffu, events, o);
    return conv_events_pays((unsigned long long)spiking * (unsigned)vs.nv_step, events * (unsigned)vs.s_step, batch, sh.n_pos,
                            sh.C_out * sh.fx * sh.fy, sh.fx * sh.fy);
}

// The taps form: a thread per filter tap. A tap's post neuron has its spike data set up once per position and is followed by
// a forward-only cursor over the position's events. A spike's slot (neuron j, k-th spike of j) follows from the order of
// appearance of j in the group. The per-sample gradient copies are combined over the cluster as in
// conv_backward_cluster_kernel; pre errors are reduced over the taps in the CTA that owns the group.
template <bool PRE, bool W_SMEM>
__global__ void __launch_bounds__(1024)
conv_backward_taps_kernel(const Event* __restrict__ ev_b, const int* __restrict__ boff, long long ev_cap,
                          const float* __restrict__ W, ConvBwdShape sh, const float* __restrict__ post_t,
                          const float2* __restrict__ tab, const int* __restrict__ nvalid, float tau_s, float tau,
                          long long pre_slots, float* __restrict__ grad, float* __restrict__ pre_err, int batch,
                          int group, ConvForm form, ConvVoteShape vs) {
    pdl_prologue();
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) float4 cb_smem[];
    __shared__ Event sev[32];
    __shared__ float sred[32][33];
    __shared__ int sslot[32], scc[32];
    __shared__ ConvVote vote;
    const int s0 = (int)blockIdx.y * group, s_end = min(batch, s0 + group);
    const float inv_tau_s = 1.0f / tau_s, inv_tau = 1.0f / tau;  // the error terms' factors, as reciprocals
    const int rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nwarps = blockDim.x >> 5;
    const int C = sh.C, taps = sh.C_out * sh.fx * sh.fy;
    const int total = taps * C;
    const int n_post = sh.Xo * sh.Yo * sh.C_out;
    float* Gs = reinterpret_cast<float*>(cb_smem);          // [tap][channel]
    int* kcount = reinterpret_cast<int*>(Gs + total);       // per channel: earlier events of the position
    for (int q = tid; q < total; q += blockDim.x) Gs[q] = 0.0f;
    // The filters, for the pre-spike error terms: in shared memory when they fit (a thread's weight reads are C floats
    // apart, one cache sector per lane from global memory).
    const float* Wk = W;
    if (W_SMEM) {
        float* sWf = reinterpret_cast<float*>(kcount + C);
        for (int q = tid; q < total; q += blockDim.x) cp_async4(sWf + q, W + q);
        Wk = sWf;
    }
    if (form == ConvForm::CHOOSE) conv_vote_count(vote, vs, boff, nvalid, sh);
    const bool has_tap = tid < taps;
    const int co = has_tap ? tid / (sh.fx * sh.fy) : 0, dx = has_tap ? tid / sh.fy % sh.fx : 0;
    const int dy = has_tap ? tid % sh.fy : 0;
    if (W_SMEM) cp_async_wait_all();
    __syncthreads();
    if (form == ConvForm::CHOOSE && conv_events_form(vote, vs, sh, batch)) {  // uniform over the grid
        if (rank == 0 && tid == 0) grad[(long long)blockIdx.y * total] = __uint_as_float(CONV_LEFT);
        return;
    }
    // The cluster's samples (one with group == 1: the per-sample gradient), accumulated in order.
    for (int s = s0; s < s_end; ++s) {
        const int* bo = boff + (long long)s * (sh.n_pos + 1);
        const Event* evs = ev_b + (long long)s * ev_cap;
        for (int g = rank; g < sh.n_pos; g += CONV_BWD_CLUSTER) {
            const int beg = bo[g], end = bo[g + 1];
            if (beg >= end) continue;  // uniform over the CTA
            const int xo = g / sh.Y - dx, yo = g % sh.Y - dy;
            const bool in = has_tap && xo >= 0 && yo >= 0 && xo < sh.Xo && yo < sh.Yo;
            PostCursor cur;
            const long long pn = in ? (long long)s * n_post + (xo * sh.Yo + yo) * sh.C_out + co : 0;
            cur.init(post_t + pn * sh.k_post, tab + pn * (sh.k_post + 1), in ? nvalid[pn] : 0);
            // Two barriers per chunk: after warp 0 stages it (every thread reads it), and after the error terms are in
            // sred (every thread is done with the chunk's records; the chunk's events then sum the terms). The next
            // chunk's first barrier orders those sums' reads of sred and sslot before anything overwrites them (warp 0
            // sums, then stages; the other warps write sred only after that barrier).
            for (int m0 = beg; m0 < end; m0 += 32) {
                const int cnt = min(32, end - m0);
                if (warp == 0) {
                    if (m0 == beg) {  // the position's spike counters per channel: warp 0's alone
                        for (int q = lane; q < C; q += 32) kcount[q] = 0;
                        __syncwarp();
                    }
                    // Stage the chunk; the spikes' slots: j * k_pre + the order of appearance of j in the group (all
                    // events of a position share x and y, so j is fixed by the channel: earlier chunks' counts plus
                    // the rank among this chunk's events of the same channel).
                    Event e;
                    int c = -1;
                    if (lane < cnt) {
                        e = evs[m0 + lane];
                        c = e.j % C;
                        sev[lane] = e;
                        scc[lane] = c;
                    }
                    const unsigned peers = __match_any_sync(0xffffffffu, c);
                    const int before = __popc(peers & lanemask_lt());
                    int base = 0;
                    if (lane < cnt) base = kcount[c];
                    __syncwarp();
                    if (lane < cnt) {
                        sslot[lane] = e.j * sh.k_pre + base + before;
                        if (before == __popc(peers) - 1) kcount[c] = base + __popc(peers);
                    }
                }
                __syncthreads();
                float term[32];
#pragma unroll
                for (int q = 0; q < 32; ++q) {
                    term[q] = 0.0f;
                    if (q < cnt && in) {
                        const Event e = sev[q];
                        cur.advance_past(e.t);
                        if (cur.valid()) {
                            const int at = tid * C + scc[q];
                            Gs[at] += fmaf(e.es, cur.AB.x, -(e.e * cur.AB.y));
                            if (PRE) term[q] = Wk[at] * (cur.AB.x * e.es * inv_tau_s - cur.AB.y * e.e * inv_tau);
                        }
                    }
                }
                // The chunk's 32 error terms summed over the warp at once (lane q: event q), then over the warps.
                if (PRE) sred[lane][warp] = warp_transpose_reduce<32>(term);
                __syncthreads();  // every thread is done with the chunk's records (warp 0 may restage them next)
                if (PRE && tid < cnt) {
                    float acc = 0.0f;
                    for (int w = 0; w < nwarps; ++w) acc += sred[tid][w];
                    pre_err[(long long)s * pre_slots + sslot[tid]] = acc;
                }
            }
        }
    }
    cluster.sync();
    const int per = (total + CONV_BWD_CLUSTER - 1) / CONV_BWD_CLUSTER;
    const int q_end = min(total, (rank + 1) * per);
    for (int q = rank * per + tid; q < q_end; q += blockDim.x) {
        float acc = 0.0f;
        for (int r = 0; r < CONV_BWD_CLUSTER; ++r) acc += cluster.map_shared_rank(Gs, r)[q];
        grad[(long long)blockIdx.y * total + q] = acc;
    }
    cluster.sync();
}

// The events form: a warp's lanes are a position's events, 32 at a time, and it goes through those taps whose
// post neuron lies inside the output and spiked: the neuron's spike times and table rows lie on the lanes (K <= 32;
// loaded one neuron ahead), every lane finds its event's place among them by a binary search over shuffles and leaves its
// gradient term in shared memory. The events of a group are staged by (channel, time), so that a channel's terms are
// neighbours: its first lane adds them in time order to the CTA's gradient copy in shared memory ([tap][channel]).
// The pre-error of an event is its taps' terms summed as a balanced tree over each tile of 32 consecutive taps
// ((co fx + dx) fy + dy; pairs 16 apart first, as warp_transpose_reduce adds lanes), the tiles then in order: a warp walks
// the taps in the order of the tree's leaves and keeps the open subtrees' sums, so the errors do not depend on which taps
// take part. The work is dealt in units of CONV_BWD_UNIT taps that form a subtree of a tile, taken by the warps from a
// counter: output channels spike very unevenly, and with a tile per warp the warps waited for the busiest one 70 % of the
// time (units of 32 taps 3.28 ms, of 16 2.29, of 8 2.35 at the size below).
// The rank's events are taken in batches of whole positions (at most `batch_ev` events; a larger position in segments):
// staged once for all warps with their channel decoded and their slots ranked (slot k of neuron j: the k-th event of j in
// the group); the units' pre-error sums of the batch meet in sred and are added in order at its end. Three barriers per
// batch. The per-sample gradient copies are combined over the cluster as in conv_backward_cluster_kernel.
// What bounds it: instruction issue (4.7 M pairs of a spiking tap and up to 32 events, 8 rounds of a channel's terms each;
// 67 % of the issue slots of 128 CTAs). 40 filters 5 x 5 x 15 over 12 x 12, 128 samples: 2.65 -> 2.07 ms, the same
// sums.
constexpr int CONV_BWD_POS = (255 + CONV_BWD_CLUSTER - 1) / CONV_BWD_CLUSTER;  // positions per rank
constexpr int CONV_BWD_UNIT = 16;                                              // taps per unit: two units per tile

// ROWS: K <= 32, a neuron's rows fit the lanes; TOP: the largest power of two <= K (at most 16), the search's first step.
template <bool ROWS, int TOP, bool PRE, bool W_SMEM>
__global__ void __launch_bounds__(1024)
conv_backward_grouped_kernel(const Event* __restrict__ ev_b, const int* __restrict__ boff, long long ev_cap,
                             const float* __restrict__ W, ConvBwdShape sh, const float* __restrict__ post_t,
                             const float2* __restrict__ tab, const int* __restrict__ nvalid, float tau_s, float tau,
                             long long pre_slots, float* __restrict__ grad, float* __restrict__ pre_err, int batch,
                             int group, int batch_ev) {
    pdl_prologue();
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) float4 cb_smem[];
    __shared__ int s_beg[CONV_BWD_POS], s_len[CONV_BWD_POS], s_at[CONV_BWD_POS], s_next;
    const int s0 = (int)blockIdx.y * group, s_end = min(batch, s0 + group);
    // Every CTA reads the word before its first barrier of the cluster, and the gradient is written after it.
    if (__float_as_uint(grad[(long long)blockIdx.y * sh.C_out * sh.fx * sh.fy * sh.C]) != CONV_LEFT) return;
    const float inv_tau_s = 1.0f / tau_s, inv_tau = 1.0f / tau;  // the error terms' factors, as reciprocals
    const int rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nwarps = blockDim.x >> 5;
    const int C = sh.C, taps = sh.C_out * sh.fx * sh.fy, K = sh.k_post;
    constexpr int UNIT = CONV_BWD_UNIT, UNITS = 32 / UNIT;
    const int tiles = (taps + 31) / 32, units = tiles * UNITS, red_ld = units | 1;
    const int total = taps * C;
    const int n_post = sh.Xo * sh.Yo * sh.C_out;
    float4* sE = cb_smem;                                   // staged events: (t, es, e, channel)
    int* sslot = reinterpret_cast<int*>(sE + batch_ev);     // their slots
    int* schan = sslot + batch_ev;                          // channels in time order (staging)
    int* kcount = schan + batch_ev;                         // per channel: a split position's earlier events
    float* Gs = reinterpret_cast<float*>(kcount + C);       // [tap][channel]
    float* sWf = Gs + total;                                // W_SMEM: the filters, [tap][channel] as they lie
    float* sval = (W_SMEM ? sWf + total : sWf) + warp * 32;       // per warp: a chunk's gradient terms
    float* sred = (W_SMEM ? sWf + total : sWf) + nwarps * 32;     // PRE: [event][unit], 0 where no tap takes part
    for (int q = tid; q < total; q += blockDim.x) Gs[q] = 0.0f;
    if (W_SMEM)
        for (int q = tid; q < total; q += blockDim.x) sWf[q] = W[q];
    const float* Wk = W_SMEM ? sWf : W;
    const int n_mine = rank < sh.n_pos ? (sh.n_pos - 1 - rank) / CONV_BWD_CLUSTER + 1 : 0;
    // The cluster's samples (one with group == 1: the per-sample gradient), accumulated in order.
    for (int s = s0; s < s_end; ++s) {
        const int* bo = boff + (long long)s * (sh.n_pos + 1);
        const Event* evs = ev_b + (long long)s * ev_cap;
        const long long pn_s = (long long)s * n_post;
        const float* t_lane = post_t + pn_s * K + lane;
        const float2* tab_lane = tab + pn_s * (K + 1) + lane;
        __syncthreads();
        for (int i = tid; i < n_mine; i += blockDim.x) {
            const int g = rank + i * CONV_BWD_CLUSTER;
            s_beg[i] = bo[g];
            s_len[i] = bo[g + 1] - bo[g];
        }
        __syncthreads();
        // i0, off0: the first position of the batch and its first event not taken yet (uniform over the CTA).
        for (int i0 = 0, off0 = 0; i0 < n_mine;) {
            int i1 = i0, cnt = 0;  // positions i0 .. i1 - 1 whole, or one segment of position i0
            const bool split = off0 > 0 || s_len[i0] > batch_ev;
            if (split) {
                cnt = min(batch_ev, s_len[i0] - off0);
                i1 = i0 + 1;
            } else {
                while (i1 < n_mine && cnt + s_len[i1] <= batch_ev) cnt += s_len[i1++];
            }
            if (cnt > 0) {
                // Stage the batch by (channel, time) per position: a warp per position (a split one: all warps).
                auto channel = [&](int src) {
                    return __ldg(reinterpret_cast<const int*>(evs + src) + 1) % C;
                };
                auto place = [&](int at, int q, int len, int src, int base) {
                    const int c = schan[at + q];
                    int less = 0, earlier = 0;
                    for (int r = 0; r < len; ++r) {
                        const int cr = schan[at + r];
                        less += cr < c ? 1 : 0;
                        earlier += cr == c && r < q ? 1 : 0;
                    }
                    const float4 e = __ldg(reinterpret_cast<const float4*>(evs + src + q));  // (t, j, es, e)
                    const int to = at + less + earlier;
                    sE[to] = make_float4(e.x, e.z, e.w, __int_as_float(c));
                    sslot[to] = __float_as_int(e.y) * sh.k_pre + base + earlier;
                };
                if (split) {
                    const int src = s_beg[i0] + off0;
                    if (off0 == 0)
                        for (int q = tid; q < C; q += blockDim.x) kcount[q] = 0;
                    for (int q = tid; q < cnt; q += blockDim.x) schan[q] = channel(src + q);
                    __syncthreads();
                    for (int q = tid; q < cnt; q += blockDim.x) place(0, q, cnt, src, kcount[schan[q]]);
                    __syncthreads();
                    for (int c = tid; c < C; c += blockDim.x) {
                        int more = 0;
                        for (int r = 0; r < cnt; ++r) more += schan[r] == c ? 1 : 0;
                        kcount[c] += more;
                    }
                } else {
                    for (int w = warp; w < i1 - i0; w += nwarps) {
                        int at = 0;
                        for (int i = i0; i < i0 + w; ++i) at += s_len[i];
                        const int len = s_len[i0 + w], src = s_beg[i0 + w];
                        if (lane == 0) s_at[i0 + w] = at;
                        for (int q = lane; q < len; q += 32) schan[at + q] = channel(src + q);
                        __syncwarp();
                        for (int q = lane; q < len; q += 32) place(at, q, len, src, 0);
                    }
                }
                if (PRE)
                    for (int q = tid; q < cnt * red_ld; q += blockDim.x) sred[q] = 0.0f;
                if (tid == 0) s_next = 0;
                __syncthreads();
                // Units of taps from the counter, each through the batch's positions.
                for (;;) {
                    int u = 0;
                    if (lane == 0) u = atomicAdd(&s_next, 1);
                    u = __shfl_sync(0xffffffffu, u, 0);
                    if (u >= units) break;
                    // Leaf i of the unit is tap `leaf_tap(i)` of the tile: the bits of its place in the tree reversed.
                    const int tile0 = u / UNITS * 32, leaf0 = u % UNITS * UNIT;
                    auto leaf_tap = [&](int i) { return tile0 + (int)(__brev((unsigned)(leaf0 + i)) >> 27); };
                    const int tap = leaf_tap(lane % UNIT);
                    const bool has_tap = tap < taps;
                    const int co = tap / (sh.fx * sh.fy), dx = tap / sh.fy % sh.fx, dy = tap % sh.fy;
                    for (int i4 = i0; i4 < i1; i4 += UNITS) {
                        // Lane: one of the unit's taps (lane % UNIT) at one of 32 / UNIT positions, its post neuron
                        // (within the sample) and that neuron's spike count.
                        const int i = i4 + lane / UNIT, g = rank + i * CONV_BWD_CLUSTER;
                        const int xo = g / sh.Y - dx, yo = g % sh.Y - dy;
                        const bool in = has_tap && i < i1 && xo >= 0 && yo >= 0 && xo < sh.Xo && yo < sh.Yo &&
                                        s_len[min(i, i1 - 1)] > 0;
                        const int pn_l = in ? (xo * sh.Yo + yo) * sh.C_out + co : 0;
                        const int n_l = in ? __ldg(nvalid + pn_s + pn_l) : 0;
                        unsigned spiking = __ballot_sync(0xffffffffu, n_l > 0);
                        // Rows of the neuron at lane b: K spike times and table entries on the lanes, +inf and 0 past its
                        // spikes.
                        float t_row, a_row, b_row;
                        int n_row, pn_row;
                        auto load = [&](int b) {
                            n_row = __shfl_sync(0xffffffffu, n_l, b);
                            pn_row = __shfl_sync(0xffffffffu, pn_l, b);
                            t_row = BATS_INF;
                            a_row = b_row = 0.0f;
                            if (ROWS && lane < n_row) {
                                t_row = __ldg(t_lane + pn_row * K);
                                const float2 ab = __ldg(tab_lane + pn_row * (K + 1));
                                a_row = ab.x;
                                b_row = ab.y;
                            }
                        };
                        while (spiking) {  // the positions with a spike under the unit's taps
                            const int p = (__ffs(spiking) - 1) / UNIT;
                            const unsigned mine = (spiking >> (UNIT * p)) & 0xffffu;
                            spiking &= ~(0xffffu << (UNIT * p));
                            const bool few = __popc(mine) <= 2;
                            const int len = split ? cnt : s_len[i4 + p], at = split ? 0 : s_at[i4 + p];
                            for (int q0 = 0; q0 < len; q0 += 32) {
                                const bool on = q0 + lane < len;
                                const float4 e = on ? sE[at + q0 + lane]
                                                    : make_float4(-BATS_INF, 0.0f, 0.0f, __int_as_float(-1));
                                const int c = __float_as_int(e.w);
                                // A channel's events are neighbours: `run` of them from its first lane on.
                                const int c_before = __shfl_up_sync(0xffffffffu, c, 1);
                                const bool head = lane == 0 || c != c_before;
                                const unsigned later = __ballot_sync(0xffffffffu, head) & ~(lanemask_lt() * 2u + 1u);
                                const int run = head && on ? (later ? __ffs(later) - 1 : 32) - lane : 0;
                                const int longest = (int)__reduce_max_sync(0xffffffffu, (unsigned)run);
                                const int row = on ? c : 0;
                                float acc = 0.0f, open[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // open subtrees of 1, 2, 4 and 8 leaves
                                unsigned todo = mine;
                                int leaf = __ffs(todo) - 1;  // the leaf of acc
                                load(UNIT * p + leaf);
                                while (todo) {
                                    const int i_leaf = __ffs(todo) - 1;
                                    todo &= todo - 1u;
                                    const float t_cur = t_row, a_cur = a_row, b_cur = b_row;
                                    const int n = n_row, pn = pn_row, at_tap = leaf_tap(i_leaf) * C + row;
                                    if (todo) load(UNIT * p + __ffs(todo) - 1);
                                    // The event's place among the spikes: place = #{k : t_k <= t}.
                                    float A, B;
                                    bool valid;
                                    if (ROWS) {
                                        int last = -1;  // place - 1
#pragma unroll
                                        for (int step = TOP; step > 0; step >>= 1) {
                                            if (step > 2 && n < step) continue;  // uniform
                                            const float tk = __shfl_sync(0xffffffffu, t_cur, last + step);
                                            if (tk <= e.x) last += step;
                                        }
                                        if (TOP == 16 && K == 32) {  // the 32nd spike
                                            const float t31 = __shfl_sync(0xffffffffu, t_cur, 31);
                                            last += last == 30 && t31 <= e.x ? 1 : 0;
                                        }
                                        A = __shfl_sync(0xffffffffu, a_cur, last + 1);
                                        B = __shfl_sync(0xffffffffu, b_cur, last + 1);
                                        valid = on && last + 1 < n;
                                    } else {
                                        const long long r = pn_s + pn;
                                        const int place = post_position(post_t + r * K, n, e.x);
                                        const float2 ab =
                                            place < n ? __ldg(tab + r * (K + 1) + place) : make_float2(0.0f, 0.0f);
                                        A = ab.x;
                                        B = ab.y;
                                        valid = on && place < n;
                                    }
                                    sval[lane] = valid ? fmaf(e.y, A, -(e.z * B)) : 0.0f;
                                    if (PRE) {
                                        const float term =
                                            valid ? Wk[at_tap] * (A * e.y * inv_tau_s - B * e.z * inv_tau) : 0.0f;
                                        if (few) {  // one or two leaves: no order
                                            acc += term;
                                        } else {    // close the subtrees that end before this leaf
                                            const int up = 31 - __clz(leaf ^ i_leaf);
                                            if (up <= 0) {
                                                open[0] = acc;
                                            } else {
                                                acc += open[0];
                                                open[0] = 0.0f;
                                                if (up == 1) {
                                                    open[1] = acc;
                                                } else {
                                                    acc += open[1];
                                                    open[1] = 0.0f;
                                                    if (up == 2) {
                                                        open[2] = acc;
                                                    } else {
                                                        acc += open[2];
                                                        open[2] = 0.0f;
                                                        open[3] = acc;
                                                    }
                                                }
                                            }
                                            leaf = i_leaf;
                                            acc = term;
                                        }
                                    }
                                    __syncwarp();
                                    // The channels' terms in time order.
                                    float g_sum = run ? Gs[at_tap] : 0.0f;
#pragma unroll 4
                                    for (int r = 0; r < longest; ++r)
                                        if (r < run) g_sum += sval[lane + r];
                                    if (run) Gs[at_tap] = g_sum;
                                    __syncwarp();
                                }
                                if (PRE && !few) {
#pragma unroll
                                    for (int m = 0; m < 4; ++m) acc += open[m];
                                }
                                if (PRE && on) sred[(at + q0 + lane) * red_ld + u] = acc;
                            }
                        }
                    }
                }
                __syncthreads();
                if (PRE)
                    for (int q = tid; q < cnt; q += blockDim.x) {
                        const float* row = sred + q * red_ld;
                        float acc = 0.0f;
                        for (int w = 0; w < tiles; ++w, row += UNITS) acc += row[0] + row[1];
                        pre_err[(long long)s * pre_slots + sslot[q]] = acc;
                    }
                __syncthreads();  // the next batch's staging overwrites sE and sslot
            }
            if (split && off0 + cnt < s_len[i0]) {
                off0 += cnt;
            } else {
                i0 = i1;
                off0 = 0;
            }
        }
    }
    cluster.sync();
    const int per = (total + CONV_BWD_CLUSTER - 1) / CONV_BWD_CLUSTER;
    const int q_end = min(total, (rank + 1) * per);
    for (int q = rank * per + tid; q < q_end; q += blockDim.x) {
        float acc = 0.0f;
        for (int r = 0; r < CONV_BWD_CLUSTER; ++r) acc += cluster.map_shared_rank(Gs, r)[q];
        grad[(long long)blockIdx.y * total + q] = acc;
    }
    cluster.sync();
}

// Pool forward: one thread per (sample, pooled neuron).
__global__ void pool_forward_kernel(const int* __restrict__ n_spikes, const float* __restrict__ times, int batch, int X,
                                    int Y, int C, int K, int* __restrict__ out_n, float* __restrict__ out_t,
                                    int* __restrict__ out_idx) {
    pdl_prologue();
    const int Xo = X / 2, Yo = Y / 2;
    const long long n_out = (long long)Xo * Yo * C;
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (long long)batch * n_out) return;
    const int s = (int)(q / n_out);
    const int o = (int)(q % n_out);
    const int c = o % C, xy = o / C, yo = xy % Yo, xo = xy / Yo;
    long long src[4];
    int cnt[4], pos[4];
    int total = 0;
    for (int ch = 0; ch < 4; ++ch) {
        const int px = 2 * xo + (ch >> 1), py = 2 * yo + (ch & 1);
        const long long pidx = ((long long)s * X + px) * Y * C + (long long)py * C + c;
        src[ch] = pidx * K;
        // Spikes of a child are its leading finite slots.
        int nn = 0;
        while (nn < K && times[src[ch] + nn] < BATS_INF) ++nn;
        cnt[ch] = nn;
        pos[ch] = 0;
        total += n_spikes[pidx];
    }
    const long long obase = q * 4LL * K;
    int w = 0;
    while (true) {
        int best = -1;
        float bt = BATS_INF;
        for (int ch = 0; ch < 4; ++ch) {
            if (pos[ch] < cnt[ch]) {
                const float tt = times[src[ch] + pos[ch]];
                if (best < 0 || tt < bt) {
                    best = ch;
                    bt = tt;
                }
            }
        }
        if (best < 0) break;
        out_t[obase + w] = bt;
        out_idx[obase + w] = (int)(src[best] + pos[best]);
        ++pos[best];
        ++w;
    }
    for (int ch = 0; ch < 4; ++ch) {
        for (int k = cnt[ch]; k < K; ++k) {
            out_t[obase + w] = times[src[ch] + k];
            out_idx[obase + w] = (int)(src[ch] + k);
            ++w;
        }
    }
    out_n[q] = total;
}

// Pool forward with the trains in shared memory: `per` consecutive pooled neurons per CTA, a thread per (neuron, child). The
// children's slots are loaded, and the merged trains stored, as rows of consecutive slots. A slot's place in the merged train
// is counted: a spike comes after its child's earlier spikes and, of every other child, the earlier ones and
// the equal ones of children before its own (one pointer per other child, moved along the child's own spikes); the slots past
// a child's spikes follow in child order. That is the merge's result for trains in time order; a neuron with a child
// that is not is merged by one thread.
// What bounds it: instruction issue and the three barriers' latency, at 1.9 TB/s. A thread per pooled neuron that merged in global
// memory made every access of a warp a sector of its own: 24 x 24 x 15 channels, 128 samples, K 10: 165 -> 68 us; 8 x 8 x 40:
// 52 -> 27 us. (A warp per neuron with its 4 K slots on the lanes: 115 and 46 us.)
constexpr int POOL_NEURONS = 32;
constexpr int POOL_SMEM = 48 * 1024;
// Bytes per neuron: four child rows of an odd stride, the merged train, its indices, the first child.
__host__ __device__ constexpr int pool_neuron_bytes(int K) { return 4 * (4 * ((K | 1) + 2 * K) + 1); }

__global__ void __launch_bounds__(4 * POOL_NEURONS)
pool_forward_shared_kernel(const int* __restrict__ n_spikes, const float* __restrict__ times, int batch, int X, int Y, int C,
                           int K, unsigned inv_k, int* __restrict__ out_n, float* __restrict__ out_t,
                           int* __restrict__ out_idx, int per) {
    pdl_prologue();
    extern __shared__ float pool_smem[];
    const int tid = threadIdx.x, S = 4 * K, ld = K | 1;
    float* sT = pool_smem;                                // [neuron][child][slot], rows of `ld`
    float* sO = sT + per * 4 * ld;                        // the merged trains ...
    int* sI = reinterpret_cast<int*>(sO + per * S);       // ... and their indices
    int* s_first = sI + per * S;                          // the neurons' first children
    const int Xo = X / 2, Yo = Y / 2;
    const int n_out = Xo * Yo * C;
    const long long total = (long long)batch * n_out, q0 = (long long)blockIdx.x * per;
    const int n_here = (int)min((long long)per, total - q0);
    if (tid < n_here) {
        const long long q = q0 + tid;
        const int s = (int)(q / n_out), o = (int)(q % n_out);
        const int c = o % C, xy = o / C, yo = xy % Yo, xo = xy / Yo;
        s_first[tid] = ((s * X + 2 * xo) * Y + 2 * yo) * C + c;
    }
    __syncthreads();
    // Slot i of child ch over the CTA's neurons: consecutive in memory while the neurons are channels of one position.
    for (int ch = 0; ch < 4; ++ch) {
        const int step = ((ch >> 1) * Y + (ch & 1)) * C;
        for (int i = tid; i < n_here * K; i += blockDim.x) {
            const int g = K == 1 ? i : (int)__umulhi((unsigned)i, inv_k), k = i - g * K;
            sT[(g * 4 + ch) * ld + k] = times[(long long)(s_first[g] + step) * K + k];
        }
    }
    __syncthreads();
    const int g = tid >> 2, ch = tid & 3;
    if (g < per) {  // whole quads of lanes: per neurons of four threads
        const bool real = g < n_here;
        const unsigned quad = 15u << (tid & 28);
        const float* row = sT + (g * 4 + ch) * ld;
        const int first = real ? s_first[g] : 0;
        auto child = [&](int d) { return first + ((d >> 1) * Y + (d & 1)) * C; };
        // Spikes of a child are its leading finite slots.
        int cnt = 0;
        bool ordered = true;
        float before = -BATS_INF;
        for (; real && cnt < K; ++cnt) {
            const float t = row[cnt];
            if (!(t < BATS_INF)) break;
            ordered &= before <= t;
            before = t;
        }
        int n_sum = real ? n_spikes[child(ch)] : 0;
        n_sum += __shfl_xor_sync(quad, n_sum, 1);
        n_sum += __shfl_xor_sync(quad, n_sum, 2);
        if (real && ch == 0) out_n[q0 + g] = n_sum;
        ordered = __all_sync(quad, ordered);
        const float* other[3];
        int n_other[3], spikes = cnt, open_before = 0;
#pragma unroll
        for (int m = 1; m < 4; ++m) {  // the other children: ch ^ m
            const int d = ch ^ m, n_d = __shfl_xor_sync(quad, cnt, m);
            other[m - 1] = sT + (g * 4 + d) * ld;
            n_other[m - 1] = n_d;
            spikes += n_d;
            if (d < ch) open_before += K - n_d;
        }
        if (real) {
            float* o = sO + g * S;
            int* oi = sI + g * S;
            const int src = child(ch) * K;
            if (ordered) {
                int e[3] = {0, 0, 0};
                for (int k = 0; k < cnt; ++k) {
                    const float t = row[k];
                    int place = k;
#pragma unroll
                    for (int m = 0; m < 3; ++m) {
                        const bool ties = (ch ^ (m + 1)) < ch;
                        while (e[m] < n_other[m] && (other[m][e[m]] < t || (ties && other[m][e[m]] == t))) ++e[m];
                        place += e[m];
                    }
                    o[place] = t;
                    oi[place] = src + k;
                }
            } else if (ch == 0) {
                int pos[4] = {0, 0, 0, 0}, n[4] = {cnt, n_other[0], n_other[1], n_other[2]};  // child 0 ^ m is child m
                for (int w = 0; w < spikes; ++w) {
                    int best = -1;
                    float bt = BATS_INF;
                    for (int d = 0; d < 4; ++d) {
                        if (pos[d] >= n[d]) continue;
                        const float t = row[d * ld + pos[d]];
                        if (best < 0 || t < bt) {
                            best = d;
                            bt = t;
                        }
                    }
                    o[w] = bt;
                    oi[w] = child(best) * K + pos[best]++;
                }
            }
            for (int k = cnt; k < K; ++k) {
                o[spikes + open_before + k - cnt] = row[k];
                oi[spikes + open_before + k - cnt] = src + k;
            }
        }
    }
    __syncthreads();
    const long long base = q0 * S;
    for (int i = tid; i < n_here * S; i += blockDim.x) {
        out_t[base + i] = sO[i];
        out_idx[base + i] = sI[i];
    }
}

__global__ void pool_backward_kernel(const float* __restrict__ errors, const int* __restrict__ idx, long long count,
                                     float* __restrict__ pre_err) {
    pdl_prologue();
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < count;
         q += (long long)gridDim.x * blockDim.x)
        pre_err[idx[q]] = errors[q];
}

}  // namespace bats

// ---------------------------------------------------------------------------------------------
// C-ABI

// Positions per CTA: as many as give at most `threads` threads (at least one position; a layer of more output channels
// runs one position with C_out threads), in a tile close to a square (the smallest receptive field).
static void conv_tile(int C_out, int threads, int& TX, int& TY) {
    const int P = std::max(1, std::min(bats::CONV_POSITIONS, threads / C_out));
    TX = 1;
    while ((TX + 1) * (TX + 1) <= P) ++TX;
    TY = P / TX;
}

// A CTA has at least eight warps, which make the lists where few output channels use them, and at most 16 positions,
// whose lists leave room for other CTAs (2 filters 5 x 5 over 28 x 28, 128 samples: 117 us with two warps and 32
// positions, 57 so; 42 without lists; 3 filters 3 x 3 x 6 over 12 x 12: 115, 64 and 220). Larger tiles read the sample's
// events fewer times and share more of each receptive field; smaller ones give more CTAs and shorter waits at the
// barriers. 512 threads pay only where a sample can carry many events (12 x 12 x 15 x 40 slots, 768 CTAs: 0.76 ms, 256
// threads 0.87; 28 x 28 x 1 slots: 0.099 ms, 256 threads 0.087) and the grid still fills two CTAs on each of the 152 SMs;
// below that the tile is halved (42 CTAs of 512 threads: 0.142 ms, 168 of 128: 0.095).
static void conv_plan(int batch, int Xo, int Yo, int C_out, long long ev_cap, int& TX, int& TY) {
    for (int threads = ev_cap >= 8192 ? 512 : 256;; threads /= 2) {
        conv_tile(C_out, threads, TX, TY);
        const long long ctas = (long long)((Xo + TX - 1) / TX) * ((Yo + TY - 1) / TY) * batch;
        if (ctas >= 2 * 152 || threads <= 128) return;
    }
}

// Where the grid is past about a wave (eight CTAs on each of the 152 SMs), a tile has few neurons and a sample cannot carry many
// events, the CTAs take half the lists' length and half the warps, so that twice as many are resident: 1 filter 5 x 5 over 28 x
// 28, 128 samples of 10 / 74 / 400 events 37 / 44 / 58 -> 27 / 31 / 55 us (19 / 28 / 97 without lists), 2 filters 3 x 3 x 3 over
// 28 x 24, 186 samples 56 / 80 / 93 -> 38 / 57 / 74. With many events, or on smaller grids, it is slower: 9 filters 5 x 5 x 15 over
// 12 x 12, 1024 samples of 2000 events 767 -> 830 us, 2 filters, 128 samples 111 -> 144.
static bool conv_narrow(long long ctas, int neurons, long long ev_cap) {
    return ctas >= 8 * 152 && neurons <= 160 && ev_cap < 8192;
}

template <bool W_SMEM, int SUB, typename... Args>
static cudaError_t launch_conv_forward(dim3 grid, int threads, size_t smem, cudaStream_t stream, Args... args) {
    const cudaError_t e =
        (cudaError_t)bats::max_dynamic_smem_set((const void*)bats::conv_forward_kernel<W_SMEM, SUB>, (int)smem);
    if (e != cudaSuccess) return e;
    return bats::launch(bats::conv_forward_kernel<W_SMEM, SUB>, grid, threads, smem, stream, args...);
}

extern "C" int bats_conv_forward(const void* events, const int* ev_count, long long ev_cap, const float* weights,
                                 int batch, int X, int Y, int C, int fx, int fy, int C_out, int k_post, float c,
                                 float delta_theta_tau, float tau, float max_simulation, int* n_spikes, float* a,
                                 float* x, float* times, float* post_exp_tau, cudaStream_t stream) {
    BATS_REQUIRE(batch >= 0 && X >= fx && Y >= fy && fx > 0 && fy > 0 && C > 0 && C_out > 0 && k_post > 0 &&
                     X < 1024 && Y < 1024 && C < 2048 && C_out <= 1024,
                 BATS_ERR_BAD_SHAPE, "conv_forward: bad shape");
    if (batch == 0) return BATS_OK;
    BATS_REQUIRE(events && ev_count && weights && n_spikes && a && x && times && post_exp_tau, BATS_ERR_NULL,
                 "conv_forward: null pointer");
    const int Xo = X - fx + 1, Yo = Y - fy + 1;
    int TX, TY;
    conv_plan(batch, Xo, Yo, C_out, ev_cap, TX, TY);
    const int tiles_x = (Xo + TX - 1) / TX, tiles_y = (Yo + TY - 1) / TY;
    const bool narrow = conv_narrow((long long)tiles_x * tiles_y * batch, TX * TY * C_out, ev_cap);
    const int threads = std::max((TX * TY * C_out + 31) / 32 * 32, 32 * std::min(TX * TY, narrow ? 4 : 8));  // (they make lists)
    const size_t list = narrow ? sizeof(bats::ConvList<32>) : sizeof(bats::ConvList<64>);
    const size_t base_smem = TX * TY * list + ((narrow ? 32 : 64) + threads) * sizeof(bats::ConvEvent);
    const size_t w_smem = (size_t)C_out * ((fx * fy * C) | 1) * sizeof(float);
    const bool w_in_smem = base_smem + w_smem <= 200 * 1024;
    const size_t smem = base_smem + (w_in_smem ? w_smem : 0);
    dim3 grid(tiles_x * tiles_y, batch);
    const bats::SolveConst sk = bats::make_solve_const(c, delta_theta_tau, tau, max_simulation);
    const bats::Event* evs = reinterpret_cast<const bats::Event*>(events);
    auto launch = [&](auto w, auto sub) {
        return launch_conv_forward<w(), sub()>(grid, threads, smem, stream, evs, ev_count, ev_cap, weights, X, Y, C, fx, fy,
                                               C_out, Xo, Yo, TX, TY, tiles_y, k_post, sk, n_spikes, a, x, times, post_exp_tau);
    };
    using Yes = std::true_type;
    using No = std::false_type;
    using Half = std::integral_constant<int, 32>;
    using Full = std::integral_constant<int, 64>;
    BATS_CUDA(w_in_smem ? (narrow ? launch(Yes{}, Half{}) : launch(Yes{}, Full{}))
                        : (narrow ? launch(No{}, Half{}) : launch(No{}, Full{})));
    BATS_CUDA(cudaGetLastError());
    return BATS_OK;
}

extern "C" int bats_conv_backward(const void* events, const int* ev_slot, const int* ev_count, long long ev_cap,
                                  const float* weights, int batch, int X, int Y, int C, int fx, int fy, int C_out,
                                  int k_pre, const float* post_times, const void* tables, const int* nvalid,
                                  int k_post, float tau_s, float tau, float* grad_per_sample, float* pre_errors,
                                  cudaStream_t stream) {
    BATS_REQUIRE(batch >= 0 && X >= fx && Y >= fy && fx > 0 && fy > 0 && C > 0 && C_out > 0 && k_post > 0 &&
                     k_pre > 0,
                 BATS_ERR_BAD_SHAPE, "conv_backward: bad shape");
    if (batch == 0) return BATS_OK;
    BATS_REQUIRE(events && ev_slot && ev_count && weights && post_times && tables && nvalid && grad_per_sample,
                 BATS_ERR_NULL, "conv_backward: null pointer");
    const int Xo = X - fx + 1, Yo = Y - fy + 1;
    const long long taps = (long long)C_out * fx * fy;
    const long long pre_slots = (long long)X * Y * C * k_pre;
    BATS_CUDA(cudaMemsetAsync(grad_per_sample, 0, (size_t)batch * taps * C * sizeof(float), stream));
    if (pre_errors) BATS_CUDA(cudaMemsetAsync(pre_errors, 0, (size_t)batch * pre_slots * sizeof(float), stream));
    int threads = (int)std::min<long long>(1024, ((taps + 31) / 32) * 32);
    const size_t gbytes = (size_t)taps * C * sizeof(float);
    if (gbytes <= 160 * 1024) {
        // Cluster path: the per-sample filter gradient lives in shared memory of every CTA of the cluster.
        BATS_CUDA((cudaError_t)bats::max_dynamic_smem_set((const void*)bats::conv_backward_cluster_kernel, (int)gbytes));
        int top = 1;
        while (top * 2 <= k_post) top *= 2;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(bats::CONV_BWD_CLUSTER, batch);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = gbytes;
        cfg.stream = stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = bats::CONV_BWD_CLUSTER;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1 + (unsigned)bats::pdl_attribute(attr + 1);
        BATS_CUDA(cudaLaunchKernelEx(&cfg, bats::conv_backward_cluster_kernel,
                                     reinterpret_cast<const bats::Event*>(events), ev_slot, ev_count, ev_cap, weights,
                                     Y, C, fx, fy, C_out, Xo, Yo, post_times,
                                     reinterpret_cast<const float2*>(tables), nvalid, k_post, top, tau_s, tau,
                                     pre_slots, grad_per_sample, pre_errors, batch, 1));
        return BATS_OK;
    }
    BATS_CUDA(bats::launch(bats::conv_backward_kernel, batch, threads, 0, stream,
        reinterpret_cast<const bats::Event*>(events), ev_slot, ev_count, ev_cap, weights, Y, C, fx, fy, C_out, Xo, Yo,
        post_times, reinterpret_cast<const float2*>(tables), nvalid, k_post, tau_s, tau, pre_slots, grad_per_sample,
        pre_errors));
    BATS_CUDA(cudaGetLastError());
    return BATS_OK;
}

// Shared memory of conv_backward_grouped_kernel: the gradient copy always, the filters where they fit beside it, and the
// largest batch of events that the rest holds (at least 32).
static size_t conv_grouped_smem(long long taps, int C, int batch_ev, bool pre, bool w) {
    const size_t units = (size_t)(taps + 31) / 32 * (32 / bats::CONV_BWD_UNIT);
    return (size_t)batch_ev * (sizeof(float4) + 2 * sizeof(int) + (pre ? sizeof(float) * (units | 1) : 0)) +
           std::min<size_t>(32, units) * 32 * sizeof(float) + (size_t)C * sizeof(int) + (size_t)taps * C * sizeof(float) * (w ? 2 : 1);
}

template <bool PRE, bool W_SMEM>
static auto* conv_grouped_kernel(int k_post) {
    return k_post > 32    ? bats::conv_backward_grouped_kernel<false, 16, PRE, W_SMEM>
           : k_post >= 16 ? bats::conv_backward_grouped_kernel<true, 16, PRE, W_SMEM>
           : k_post >= 8  ? bats::conv_backward_grouped_kernel<true, 8, PRE, W_SMEM>
                          : bats::conv_backward_grouped_kernel<true, 4, PRE, W_SMEM>;
}

// From so many filter taps, and slots x tiles of 32 taps, on the events form is worth a second launch (a few us where no group
// takes it): 216 taps, 21 samples, few spiking 120 -> 62 us; 72 taps all spiking 44 us, and 81 in the events form. Below 10^4
// slots x tiles the times with it are 1.04 of those without (mean of 420 layers, 0.91 above).
constexpr long long CONV_EVENTS_TAPS = 192, CONV_EVENTS_WORK = 10000;

static cudaError_t launch_conv_grouped(const void* events_bucketed, const int* bucket_offsets, long long ev_cap,
                                       const float* weights, const bats::ConvBwdShape& sh, const float* post_times,
                                       const void* tables, const int* nvalid, float tau_s, float tau,
                                       long long pre_slots, float* grad, float* pre_errors, int batch, int group,
                                       cudaStream_t stream) {
    const long long taps = (long long)sh.C_out * sh.fx * sh.fy;
    const bool pre = pre_errors != nullptr;
    const bool choose = taps >= CONV_EVENTS_TAPS && ev_cap * ((taps + 31) / 32) >= CONV_EVENTS_WORK;
    const int groups = (batch + group - 1) / group;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(bats::CONV_BWD_CLUSTER, groups);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = bats::CONV_BWD_CLUSTER;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1 + (unsigned)bats::pdl_attribute(attr + 1);
    const auto* ev = reinterpret_cast<const bats::Event*>(events_bucketed);
    const auto* tab = reinterpret_cast<const float2*>(tables);
    {
        const size_t grad_bytes = (size_t)taps * sh.C * sizeof(float), small = grad_bytes + (size_t)sh.C * sizeof(int);
        const bool w = pre && small + grad_bytes <= 200 * 1024;
        const size_t smem = small + (w ? grad_bytes : 0);
        auto* kernel = !pre ? bats::conv_backward_taps_kernel<false, false>
                       : w  ? bats::conv_backward_taps_kernel<true, true>
                            : bats::conv_backward_taps_kernel<true, false>;
        cudaError_t e = (cudaError_t)bats::max_dynamic_smem_set((const void*)kernel, (int)smem);
        if (e != cudaSuccess) return e;
        cfg.blockDim = dim3((unsigned)((taps + 31) / 32 * 32));
        cfg.dynamicSmemBytes = smem;
        // Steps that share no factor with the neurons of a sample, so that every channel and position comes up.
        const long long neurons = (long long)batch * sh.Xo * sh.Yo * sh.C_out;
        bats::ConvVoteShape vs;
        vs.nv_step = (int)((neurons + bats::CONV_VOTE - 1) / bats::CONV_VOTE);
        while (std::gcd(vs.nv_step, sh.Xo * sh.Yo * sh.C_out) != 1) ++vs.nv_step;
        vs.nv_count = (int)((neurons + vs.nv_step - 1) / vs.nv_step);
        vs.s_step = (batch + bats::CONV_VOTE - 1) / bats::CONV_VOTE;
        vs.s_count = (batch + vs.s_step - 1) / vs.s_step;
        e = cudaLaunchKernelEx(&cfg, kernel, ev, bucket_offsets, ev_cap, weights, sh, post_times, tab, nvalid, tau_s, tau,
                               pre_slots, grad, pre_errors, batch, group,
                               choose ? bats::ConvForm::CHOOSE : bats::ConvForm::TAPS, vs);
        if (e != cudaSuccess || !choose) return e;
    }
    constexpr size_t LIMIT = 224 * 1024;
    const bool w = pre && conv_grouped_smem(taps, sh.C, 64, pre, true) <= LIMIT;
    int batch_ev = 512;
    while (batch_ev > 32 && conv_grouped_smem(taps, sh.C, batch_ev, pre, w) > LIMIT) batch_ev -= 32;
    const size_t smem = conv_grouped_smem(taps, sh.C, batch_ev, pre, w);
    auto* kernel = !pre ? conv_grouped_kernel<false, false>(sh.k_post)
                   : w  ? conv_grouped_kernel<true, true>(sh.k_post)
                        : conv_grouped_kernel<true, false>(sh.k_post);
    cudaError_t e = (cudaError_t)bats::max_dynamic_smem_set((const void*)kernel, (int)smem);
    if (e != cudaSuccess) return e;
    cfg.blockDim = dim3((unsigned)std::min<long long>(1024, (taps + 31) / 32 * (32 / bats::CONV_BWD_UNIT) * 32));
    cfg.dynamicSmemBytes = smem;
    return cudaLaunchKernelEx(&cfg, kernel, ev, bucket_offsets, ev_cap, weights, sh, post_times, tab, nvalid, tau_s, tau,
                              pre_slots, grad, pre_errors, batch, group, batch_ev);
}

extern "C" int bats_conv_backward_grouped(const void* events_bucketed, const int* bucket_offsets, long long ev_cap,
                                          const float* weights, int batch, int X, int Y, int C, int fx, int fy,
                                          int C_out, int k_pre, const float* post_times, const void* tables,
                                          const int* nvalid, int k_post, float tau_s, float tau,
                                          float* grad_per_sample, float* pre_errors, cudaStream_t stream) {
    BATS_REQUIRE(batch >= 0 && X >= fx && Y >= fy && fx > 0 && fy > 0 && C > 0 && C_out > 0 && k_post > 0 &&
                     k_pre > 0,
                 BATS_ERR_BAD_SHAPE, "conv_backward_grouped: bad shape");
    if (batch == 0) return BATS_OK;
    BATS_REQUIRE(events_bucketed && bucket_offsets && weights && post_times && tables && nvalid && grad_per_sample,
                 BATS_ERR_NULL, "conv_backward_grouped: null pointer");
    const long long taps = (long long)C_out * fx * fy;
    BATS_REQUIRE(taps <= 1024 && (long long)X * Y <= 255, BATS_ERR_BAD_SHAPE,
                 "conv_backward_grouped: needs at most 1024 taps and 255 input positions");
    const int Xo = X - fx + 1, Yo = Y - fy + 1;
    const long long pre_slots = (long long)X * Y * C * k_pre;
    const size_t gsmem = (size_t)taps * C * sizeof(float) + (size_t)C * sizeof(int);
    BATS_REQUIRE(gsmem <= 160 * 1024, BATS_ERR_BAD_SHAPE, "conv_backward_grouped: filter gradient too large");
    if (pre_errors) BATS_CUDA(cudaMemsetAsync(pre_errors, 0, (size_t)batch * pre_slots * sizeof(float), stream));
    const bats::ConvBwdShape sh = {Y, C, fx, fy, C_out, Xo, Yo, k_pre, k_post, X * Y};
    BATS_CUDA(launch_conv_grouped(events_bucketed, bucket_offsets, ev_cap, weights, sh, post_times, tables, nvalid,
                                  tau_s, tau, pre_slots, grad_per_sample, pre_errors, batch, 1, stream));
    return BATS_OK;
}

// Sum of per-group partial filter gradients (groups, total) in group order, divided by the batch.
namespace bats {
__global__ void conv_grad_reduce_kernel(const float* __restrict__ part, int groups, int total, float batch,
                                        float* __restrict__ grad) {
    pdl_prologue();
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= total) return;
    float acc = 0.0f;
    for (int g = 0; g < groups; ++g) acc += part[(long long)g * total + q];
    grad[q] = acc / batch;
}
}  // namespace bats

extern "C" size_t bats_conv_backward_adam_workspace_bytes(int batch, int C, int fx, int fy, int C_out, int group) {
    if (batch <= 0 || group <= 0) return 0;
    const long long groups = (batch + group - 1) / group;
    return ((size_t)groups * C_out * fx * fy * C * sizeof(float) + 255) & ~(size_t)255;
}

extern "C" int bats_conv_backward_adam(const void* events, const int* ev_slot, const int* ev_count,
                                       const void* events_bucketed, const int* bucket_offsets, long long ev_cap,
                                       float* weights, int batch, int X, int Y, int C, int fx, int fy, int C_out,
                                       int k_pre, const float* post_times, const void* tables, const int* nvalid,
                                       int k_post, float tau_s, float tau, float* pre_errors, int group, float* grad,
                                       float* m, float* v, float beta_1, float beta_2, float epsilon,
                                       float learning_rate, const double* powers, void* workspace,
                                       size_t workspace_bytes, cudaStream_t stream) {
    BATS_REQUIRE(batch >= 0 && X >= fx && Y >= fy && fx > 0 && fy > 0 && C > 0 && C_out > 0 && k_post > 0 &&
                     k_pre > 0 && group >= 1,
                 BATS_ERR_BAD_SHAPE, "conv_backward_adam: bad shape");
    if (batch == 0) return BATS_OK;
    BATS_REQUIRE(events && ev_slot && ev_count && weights && post_times && tables && nvalid && grad && m && v && powers,
                 BATS_ERR_NULL, "conv_backward_adam: null pointer");
    const int groups = (batch + group - 1) / group;
    BATS_REQUIRE(groups <= 65535, BATS_ERR_BAD_SHAPE, "conv_backward_adam: more than 65535 sample groups");
    BATS_REQUIRE(workspace && workspace_bytes >= bats_conv_backward_adam_workspace_bytes(batch, C, fx, fy, C_out, group),
                 BATS_ERR_WORKSPACE, "conv_backward_adam: workspace too small");
    const int Xo = X - fx + 1, Yo = Y - fy + 1;
    const long long taps = (long long)C_out * fx * fy;
    const int total = (int)(taps * C);
    const long long pre_slots = (long long)X * Y * C * k_pre;
    float* part = reinterpret_cast<float*>(workspace);
    if (pre_errors) BATS_CUDA(cudaMemsetAsync(pre_errors, 0, (size_t)batch * pre_slots * sizeof(float), stream));
    const bool grouped = events_bucketed && bucket_offsets && taps <= 1024 && (long long)X * Y <= 255 &&
                         (size_t)taps * C * sizeof(float) + (size_t)C * sizeof(int) <= 160 * 1024;
    const size_t gbytes = (size_t)taps * C * sizeof(float);
    BATS_REQUIRE(gbytes <= 160 * 1024, BATS_ERR_BAD_SHAPE, "conv_backward_adam: filter gradient too large");
    if (grouped) {
        const bats::ConvBwdShape sh = {Y, C, fx, fy, C_out, Xo, Yo, k_pre, k_post, X * Y};
        BATS_CUDA(launch_conv_grouped(events_bucketed, bucket_offsets, ev_cap, weights, sh, post_times, tables, nvalid,
                                      tau_s, tau, pre_slots, part, pre_errors, batch, group, stream));
    } else {
        const int threads = (int)std::min<long long>(1024, ((taps + 31) / 32) * 32);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(bats::CONV_BWD_CLUSTER, groups);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = gbytes;
        cfg.stream = stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = bats::CONV_BWD_CLUSTER;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1 + (unsigned)bats::pdl_attribute(attr + 1);
        BATS_CUDA((cudaError_t)bats::max_dynamic_smem_set((const void*)bats::conv_backward_cluster_kernel, (int)gbytes));
        int top = 1;
        while (top * 2 <= k_post) top *= 2;
        BATS_CUDA(cudaLaunchKernelEx(&cfg, bats::conv_backward_cluster_kernel,
                                     reinterpret_cast<const bats::Event*>(events), ev_slot, ev_count, ev_cap,
                                     (const float*)weights, Y, C, fx, fy, C_out, Xo, Yo, post_times,
                                     reinterpret_cast<const float2*>(tables), nvalid, k_post, top, tau_s, tau,
                                     pre_slots, part, pre_errors, batch, group));
    }
    BATS_CUDA(bats::launch(bats::conv_grad_reduce_kernel, (total + 255) / 256, 256, 0, stream, part, groups, total,
                           (float)batch, grad));
    BATS_CUDA(cudaGetLastError());
    return bats_adam_step_device(grad, m, v, total, beta_1, beta_2, epsilon, learning_rate, powers, weights, nullptr,
                                 0, 0, 0, stream);
}

extern "C" int bats_pool_forward(const int* n_spikes, const float* times, int batch, int X, int Y, int C, int K,
                                 int* out_n_spikes, float* out_times, int* out_indices, cudaStream_t stream) {
    BATS_REQUIRE(batch >= 0 && X >= 2 && Y >= 2 && C > 0 && K > 0, BATS_ERR_BAD_SHAPE, "pool_forward: bad shape");
    BATS_REQUIRE((long long)batch * X * Y * C * K < (1LL << 31), BATS_ERR_CAPACITY,
                 "pool_forward: indices exceed int32");
    if (batch == 0) return BATS_OK;
    BATS_REQUIRE(n_spikes && times && out_n_spikes && out_times && out_indices, BATS_ERR_NULL,
                 "pool_forward: null pointer");
    const long long total = (long long)batch * (X / 2) * (Y / 2) * C;
    const int per = std::min(bats::POOL_NEURONS, bats::POOL_SMEM / bats::pool_neuron_bytes(K));
    // The merge in shared memory where its rows leave room for enough neurons, or where there are few (thread per neuron / shared,
    // in us, a third of the slots filled; K 200: 3780 neurons 266 / 200, 7168 267 / 306, 23040 448 / 1065; K 64: 13440 88 / 83,
    // 45360 208 / 295; K 40: 45360 126 / 105). Rows of one slot lie next to one another as they are (K 1, 918 k neurons 33 / 49, 82 k
    // 8.4 / 9.3).
    const bool shared = K > 1 && per > 0 && (K <= 40 || total * K <= 1000000);
    if (shared) {
        // i / K for i < per * K as the high word of i * inv_k: exact while i * K < 2^32.
        const unsigned inv_k = K > 1 ? (unsigned)(((1ULL << 32) + K - 1) / K) : 0;
        BATS_CUDA(bats::launch(bats::pool_forward_shared_kernel, (unsigned)((total + per - 1) / per), (4 * per + 31) / 32 * 32,
            (size_t)per * bats::pool_neuron_bytes(K), stream, n_spikes, times, batch, X, Y, C, K, inv_k, out_n_spikes,
            out_times, out_indices, per));
        BATS_CUDA(cudaGetLastError());
        return BATS_OK;
    }
    BATS_CUDA(bats::launch(bats::pool_forward_kernel, (unsigned)((total + 127) / 128), 128, 0, stream, n_spikes, times,
        batch, X, Y, C, K, out_n_spikes, out_times, out_indices));
    BATS_CUDA(cudaGetLastError());
    return BATS_OK;
}

extern "C" int bats_pool_backward(const float* errors, const int* indices, long long count, float* pre_errors,
                                  long long pre_count, cudaStream_t stream) {
    BATS_REQUIRE(count >= 0 && pre_count >= 0, BATS_ERR_BAD_SHAPE, "pool_backward: bad shape");
    if (pre_count > 0) {
        BATS_REQUIRE(pre_errors, BATS_ERR_NULL, "pool_backward: null pointer");
        BATS_CUDA(cudaMemsetAsync(pre_errors, 0, (size_t)pre_count * sizeof(float), stream));
    }
    if (count == 0) return BATS_OK;
    BATS_REQUIRE(errors && indices, BATS_ERR_NULL, "pool_backward: null pointer");
    long long b = (count + 255) / 256;
    if (b > 152 * 16) b = 152 * 16;
    BATS_CUDA(bats::launch(bats::pool_backward_kernel, (unsigned)b, 256, 0, stream, errors, indices, count,
        pre_errors));
    BATS_CUDA(cudaGetLastError());
    return BATS_OK;
}
