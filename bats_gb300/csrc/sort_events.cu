// Per-sample time sort of all pre-synaptic spikes of a layer (one CTA per sample).
// The sort runs in shared memory whenever the sample's items fit (16448 items with 16-bit slot values for batches of at most
// 152 samples, 6720 for larger ones; 12320 and 4096 with 32-bit ones), else in a per-sample slice of the caller's workspace.
//
// Replaces get_sorted_spikes_indices + the three take_along_axis gathers + compute_pre_exps
// (bats/CudaKernels/Wrappers/Inference/get_sorted_spikes_indices.py:7-17,
//  bats/Layers/LIFLayer.py:66-84, bats/CudaKernels/CuFiles/Inference/compute_pre_exps.cu:2-22).
// The reference sorts every (neuron, slot) of the batch on the device with argpartition after a
// host sync on the largest spike count; here every sample's valid slots (time < +inf) are
// gathered into shared memory, dealt into equal spans of the sample's time and ranked inside their span by
// (time, slot) (samples of many equal times and very large ones by an LSD radix sort), so the event list needs no host sync and no
// padding to the batch maximum. Ties keep slot order, which makes the order deterministic.
//
// CTA b sorts sample b, or sample sample_order[b] when an order is given (the samples longest first: on a
// batch of uneven samples wider than the resident CTAs, the long samples then start in the first wave
// instead of setting the kernel's tail). The order changes the schedule only, never a result.
//
// For the backward pass the same kernel can also emit the events grouped by pre-neuron bucket
// (neuron / bucket_width), each bucket still in time order (one more stable counting pass), with
// the per-sample bucket offsets: the weight-gradient kernel then reads only its bucket's events.
#include "common.cuh"

namespace bats {

constexpr int SORT_BINS = 256;  // digit values of a counting pass; threads tid < SORT_BINS own one bin each
constexpr int SORT_MAX_BUCKETS = 255;
// Threads per CTA: 512 for layers of more than SORT_WIDE_CAP slots, 256 below (samples of a few hundred items, which a
// larger block only spreads thinner; the line was drawn with a radix sort: 0.88 -> 0.71 ms on the 4096-sample uneven
// batch's second sort, 0.093 -> 0.081 ms on 800 x 30 slots at batch 256).
constexpr int SORT_WIDE_CAP = 1024;
// Items held in shared memory (two key buffers and two value buffers): slot values are 16-bit when the
// layer has at most 65536 slots (cap = n_pre * k_pre), else 32-bit. Batches of at most SORT_SMALL_BATCH
// samples (no more CTAs than a GB300 has SMs: one CTA per SM costs no parallelism) get as many items as
// 227 KB holds beside the counters (SortShared: 34.9 KB at 512 threads); larger batches keep two CTAs per SM, at most
// 113 KB each. Samples with more valid slots than that sort in global scratch. (Layers of up to SORT_WIDE_CAP slots
// always fit.)
constexpr int SORT_SMALL_BATCH = 152;
constexpr int SORT_ROOM_MAX_U16 = 16448, SORT_ROOM_MAX_U32 = 12320, SORT_ROOM_U16 = 6720, SORT_ROOM_U32 = 4096;

template <int T>
struct SortShared {
    int hist[SORT_BINS];
    int base[SORT_BINS];
    int wcnt[T / 32][SORT_BINS];
    int wofs[T / 32][SORT_BINS];
    int warp_tot[T / 32];
    int appended;         // items found (gather_items)
    unsigned kmin, kmax;  // their smallest and largest key
    unsigned pairs;       // sum of the squares of the bucket sizes (bucket_sort); the items behind are read as uint4
};
static_assert(sizeof(SortShared<256>) % 16 == 0 && sizeof(SortShared<512>) % 16 == 0, "uint4 reads of the items");

// Exclusive scan of sh.hist (SORT_BINS bins, one per thread tid < SORT_BINS) into sh.base; clears sh.wcnt.
template <int T>
__device__ __forceinline__ void scan_bins(SortShared<T>& sh) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool bin = tid < SORT_BINS;
    const int v = bin ? sh.hist[tid] : 0;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31 && bin) sh.warp_tot[warp] = incl;
    __syncthreads();
    if (bin) {
        int woff = 0;
        for (int w = 0; w < warp; ++w) woff += sh.warp_tot[w];
        sh.base[tid] = woff + incl - v;
#pragma unroll
        for (int w = 0; w < T / 32; ++w) sh.wcnt[w][tid] = 0;
    }
    __syncthreads();
}

// One stable counting pass (digit < 256) of n (key, val) pairs from (ka, va) into (kb, vb), using the
// bin bases already in sh.base. Items are ranked in rounds of T in their current order; inside a warp,
// items of equal digit are ranked by their peer mask (the AND of nine ballots, one per bit of the digit or
// the out-of-range 256: faster here than __match_any_sync), across warps by a per-digit scan.
template <int T, typename V, typename DigitFn>
__device__ __forceinline__ void stable_pass(const uint32_t* ka, const V* va, uint32_t* kb, V* vb, int n,
                                            SortShared<T>& sh, DigitFn digit) {
    const int tid = threadIdx.x, warp = tid >> 5;
    for (int r0 = 0; r0 < n; r0 += T) {
        const int i = r0 + tid;
        const bool valid = i < n;
        uint32_t key = 0;
        V val = 0;
        int d = 256;
        if (valid) {
            key = ka[i];
            val = va[i];
            d = digit(key, (uint32_t)val);
        }
        unsigned peers = 0xffffffffu;
#pragma unroll
        for (int bit = 0; bit < 9; ++bit) {
            const bool on = (d >> bit) & 1;
            const unsigned bal = __ballot_sync(0xffffffffu, on);
            peers &= on ? bal : ~bal;
        }
        const int rank = __popc(peers & lanemask_lt());
        if (valid && rank == 0) sh.wcnt[warp][d] = __popc(peers);
        __syncthreads();
        if (tid < SORT_BINS) {
            int off = sh.base[tid];
#pragma unroll
            for (int w = 0; w < T / 32; ++w) {
                sh.wofs[w][tid] = off;
                off += sh.wcnt[w][tid];
                sh.wcnt[w][tid] = 0;
            }
            sh.base[tid] = off;
        }
        __syncthreads();
        if (valid) {
            const int pos = sh.wofs[warp][d] + rank;
            kb[pos] = key;
            vb[pos] = val;
        }
    }
    __syncthreads();
}

__device__ __forceinline__ Event make_event(uint32_t key, uint32_t slot, int k_pre, long long sample_off,
                                            const float* exp_s_in, const float* exp_in, float tau_s, float tau) {
    Event e;
    e.t = key_to_float(key);
    e.j = (int)slot / k_pre;
    if (exp_s_in) {
        e.es = exp_s_in[sample_off + slot];
        e.e = exp_in[sample_off + slot];
    } else {
        e.es = __expf(e.t / tau_s);
        e.e = __expf(e.t / tau);
    }
    return e;
}

struct TimeDigit {
    int shift;
    __device__ int operator()(uint32_t key, uint32_t) const { return (int)((key >> shift) & 255u); }
};
struct BucketDigit {
    int div;
    __device__ int operator()(uint32_t, uint32_t slot) const { return (int)slot / div; }
};

// Appends the calling warp's items (up to 8 per lane, those with t[u] < +inf and u < 8) to the list, in no particular
// order: one atomic per warp. Items past the room are only counted.
template <int T, typename V, int N>
__device__ __forceinline__ void append_items(const float (&t)[N], const uint32_t (&slot)[N], uint32_t* keys, V* vals,
                                             int room, SortShared<T>& sh, unsigned& kmin, unsigned& kmax) {
    const int lane = threadIdx.x & 31;
    int c = 0;
#pragma unroll
    for (int u = 0; u < N; ++u) c += t[u] < BATS_INF ? 1 : 0;
    int incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    int base = 0;
    if (lane == 31) base = atomicAdd(&sh.appended, incl);
    int pos = __shfl_sync(0xffffffffu, base, 31) + incl - c;
#pragma unroll
    for (int u = 0; u < N; ++u) {
        if (t[u] < BATS_INF) {
            const uint32_t key = float_to_key(t[u]);
            kmin = min(kmin, key);
            kmax = max(kmax, key);
            if (pos < room) {
                keys[pos] = key;
                vals[pos] = (V)slot[u];
            }
            ++pos;
        }
    }
}

// The sample's valid slots as an unordered list in shared memory (at most room items), with their number and their
// smallest and largest key in sh. One pass over the slots (with the pre layer's spike counts: over those below them),
// several loads in flight per thread.
template <int T, typename V>
__device__ __forceinline__ void gather_items(const float* __restrict__ tsrc, const int* __restrict__ cnt_src, int n_slots,
                                             int k_pre, uint32_t* keys, V* vals, int room, SortShared<T>& sh) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned kmin = 0xffffffffu, kmax = 0u;
    if (cnt_src) {
        const int n_pre = n_slots / k_pre;
        for (int r0 = warp * 32; r0 < n_pre; r0 += T) {
            const int j = r0 + lane;
            const int c = j < n_pre ? min(max(cnt_src[j], 0), k_pre) : 0;
            const int most = (int)__reduce_max_sync(0xffffffffu, (unsigned)c);
            for (int q0 = 0; q0 < most; q0 += 8) {
                float t[8];
                uint32_t slot[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    slot[u] = (uint32_t)(j * k_pre + q0 + u);
                    t[u] = q0 + u < c ? tsrc[slot[u]] : BATS_INF;
                }
                append_items<T, V, 8>(t, slot, keys, vals, room, sh, kmin, kmax);
            }
        }
    } else if ((n_slots & 3) == 0) {
        const float4* t4 = reinterpret_cast<const float4*>(tsrc);
        const int n4 = n_slots >> 2;
        for (int q0 = warp * 32; q0 < n4; q0 += 2 * T) {
            float t[8];
            uint32_t slot[8];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int q = q0 + h * T + lane;
                const float4 v = q < n4 ? t4[q] : make_float4(BATS_INF, BATS_INF, BATS_INF, BATS_INF);
                t[4 * h] = v.x;
                t[4 * h + 1] = v.y;
                t[4 * h + 2] = v.z;
                t[4 * h + 3] = v.w;
#pragma unroll
                for (int u = 0; u < 4; ++u) slot[4 * h + u] = (uint32_t)(4 * q + u);
            }
            append_items<T, V, 8>(t, slot, keys, vals, room, sh, kmin, kmax);
        }
    } else {
        for (int q0 = warp * 32; q0 < n_slots; q0 += 4 * T) {
            float t[4];
            uint32_t slot[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const int q = q0 + h * T + lane;
                slot[h] = (uint32_t)q;
                t[h] = q < n_slots ? tsrc[q] : BATS_INF;
            }
            append_items<T, V, 4>(t, slot, keys, vals, room, sh, kmin, kmax);
        }
    }
    kmin = __reduce_min_sync(0xffffffffu, kmin);
    kmax = __reduce_max_sync(0xffffffffu, kmax);
    if (lane == 0) {
        atomicMin(&sh.kmin, kmin);
        atomicMax(&sh.kmax, kmax);
    }
}

// A time's bucket among `buckets` equal parts of [t_min, t_max]: every step is monotone in t, so that the buckets are
// in time order whatever the roundings.
__device__ __forceinline__ int time_bucket(uint32_t key, float t_min, float scale, int buckets) {
    return (int)fminf((key_to_float(key) - t_min) * scale, (float)(buckets - 1));
}

// Comparisons per item up to which ranking inside the buckets is taken, against a radix sort of a second list in slot order. 54
// samples of 5500 items, times on a grid of 200 / 100 / 50 steps (27, 55 and 110 comparisons): 43, 58 and 86 us by
// comparison, 53 by radix; 8 samples of 11200 on 500 / 200 steps: 74 and 107, 104; 256 of 2400 on 50 / 20: 44 and 68, 58. (With up
// to 384 items in any bucket: 238 us on 20 steps, where the radix sort alone takes 72.)
constexpr unsigned SORT_COMPARISONS = 48;

// Sorts the n gathered items (ka, va) by (key, slot) with (kb, vb) as the second buffer, leaving them in (ka, va):
// the items are dealt into buckets of equal time spans, and each finds its place inside its bucket by counting the
// smaller ones. Six barriers whatever n, against three per 512 items and pass of a radix sort. False (nothing sorted)
// when that takes more than SORT_COMPARISONS comparisons per item (times on a coarse grid, or crowded by an outlier).
template <int T, typename V>
__device__ __forceinline__ bool bucket_sort(uint32_t* ka, V* va, uint32_t* kb, V* vb, int n, SortShared<T>& sh) {
    constexpr int NB = T / 32 * SORT_BINS;  // as many buckets as the counters of the counting passes hold
    constexpr int PER = NB / T;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int* count = &sh.wcnt[0][0];
    int* start = &sh.wofs[0][0];
    const float t_min = key_to_float(sh.kmin), span = key_to_float(sh.kmax) - t_min;
    const bool usable = span > 0.0f && span <= 3.0e38f;  // uniform; else all items are in one bucket
    const float scale = usable ? fminf((float)NB / span, 3.0e38f) : 0.0f;
    for (int q = tid; q < NB; q += T) count[q] = 0;
    if (tid == 0) sh.pairs = 0u;
    __syncthreads();
    for (int i = tid; i < n; i += T) atomicAdd(&count[time_bucket(ka[i], t_min, scale, NB)], 1);
    __syncthreads();
    // Exclusive scan: thread tid owns buckets PER * tid ..
    int own[PER], sum = 0;
    unsigned pairs = 0u;  // n^2 at most, below 2^32 for what fits in shared memory
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        own[u] = count[PER * tid + u];
        pairs += (unsigned)(own[u] * own[u]);
        sum += own[u];
    }
    pairs = __reduce_add_sync(0xffffffffu, pairs);
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) {
        sh.warp_tot[warp] = incl;
        atomicAdd(&sh.pairs, pairs);
    }
    __syncthreads();
    if (sh.pairs > SORT_COMPARISONS * (unsigned)n) return false;
    int base = incl - sum;
    for (int w = 0; w < warp; ++w) base += sh.warp_tot[w];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        start[PER * tid + u] = base;
        count[PER * tid + u] = base;  // the scatter's cursor; afterwards the bucket's end
        base += own[u];
    }
    __syncthreads();
    for (int i = tid; i < n; i += T) {
        const uint32_t key = ka[i];
        const int pos = atomicAdd(&count[time_bucket(key, t_min, scale, NB)], 1);
        kb[pos] = key;
        vb[pos] = va[i];
    }
    __syncthreads();
    for (int i = tid; i < n; i += T) {
        const uint32_t key = kb[i];
        const V val = vb[i];
        const int b = time_bucket(key, t_min, scale, NB);
        const int lo = start[b], hi = count[b];
        int r = lo;
        for (int q = lo; q < hi; ++q) {
            const uint32_t kq = kb[q];
            r += (kq < key || (kq == key && vb[q] < val)) ? 1 : 0;
        }
        ka[r] = key;
        va[r] = val;
    }
    __syncthreads();
    return true;
}

// The sample's valid slots as a list in slot order: a contiguous range of slots per warp, counted, then written. With the
// pre layer's spike counts the lanes are neurons and read the slots below their counts, else the lanes are slots; eight
// loads in flight per lane.
template <int T, typename V>
__device__ __forceinline__ void compact_slots(const float* __restrict__ tsrc, const int* __restrict__ cnt_src, int n_slots,
                                              int k_pre, uint32_t* keys, V* vals, SortShared<T>& sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rows = cnt_src ? n_slots / k_pre : n_slots;
    const int per = ((rows + 31) / 32 + T / 32 - 1) / (T / 32) * 32;
    const int lo = min(rows, warp * per), hi = min(rows, lo + per);
    auto put = [&](int pos, float t, int slot) {
        keys[pos] = float_to_key(t);
        vals[pos] = (V)slot;
    };
    // f(time, slot) for the valid slots of neuron j in order.
    auto each = [&](int j, auto f) {
        const int c = j < hi ? min(cnt_src[j], k_pre) : 0;
        for (int q0 = 0; q0 < c; q0 += 8) {
            float t[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) t[u] = q0 + u < c ? tsrc[j * k_pre + q0 + u] : BATS_INF;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (t[u] < BATS_INF) f(t[u], j * k_pre + q0 + u);
        }
    };
    int c = 0;
    if (cnt_src) {
        for (int r = lo; r < hi; r += 32) each(r + lane, [&](float, int) { ++c; });
    } else {
#pragma unroll 8
        for (int q = lo + lane; q < hi; q += 32) c += tsrc[q] < BATS_INF ? 1 : 0;
    }
    c = (int)__reduce_add_sync(0xffffffffu, (unsigned)c);
    if (lane == 0) sh.warp_tot[warp] = c;
    __syncthreads();
    int base = 0;
    for (int w = 0; w < warp; ++w) base += sh.warp_tot[w];
    if (cnt_src) {
        for (int r = lo; r < hi; r += 32) {
            int mine = 0;
            each(r + lane, [&](float, int) { ++mine; });
            int incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            int pos = base + incl - mine;
            each(r + lane, [&](float t, int slot) { put(pos++, t, slot); });
            base += __shfl_sync(0xffffffffu, incl, 31);
        }
    } else {
        for (int q0 = lo; q0 < hi; q0 += 8 * 32) {
            float t[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int q = q0 + 32 * u + lane;
                t[u] = q < hi ? tsrc[q] : BATS_INF;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const unsigned valid = __ballot_sync(0xffffffffu, t[u] < BATS_INF);
                if (t[u] < BATS_INF) put(base + __popc(valid & lanemask_lt()), t[u], q0 + 32 * u + lane);
                base += __popc(valid);
            }
        }
    }
    __syncthreads();
}

// LSD radix sort of the items by the time key, 8 bits a pass; passes whose digit is uniform are skipped. Ties keep their order.
template <int T, typename V>
__device__ __forceinline__ void radix_sort(uint32_t*& ka, V*& va, uint32_t*& kb, V*& vb, int n, SortShared<T>& sh) {
    const int tid = threadIdx.x;
    for (int shift = 0; shift < 32; shift += 8) {
        if (tid < SORT_BINS) sh.hist[tid] = 0;
        __syncthreads();
        for (int i = tid; i < n; i += T) atomicAdd(&sh.hist[(ka[i] >> shift) & 255u], 1);
        __syncthreads();
        if (__syncthreads_or(tid < SORT_BINS && sh.hist[tid] == n)) continue;
        scan_bins<T>(sh);
        stable_pass<T>(ka, va, kb, vb, n, sh, TimeDigit{shift});
        uint32_t* t0 = ka; ka = kb; kb = t0;
        V* t1 = va; va = vb; vb = t1;
    }
}

// V: type of the slot values (uint16_t when n_slots <= 65536). smem_cap: items held in shared memory.
// Samples of up to smem_cap valid slots: gathered into shared memory in any order, then bucket_sort. Where the times crowd too
// much for it, or in the global scratch where the sample is larger: compacted in slot order, then radix_sort. The order is by
// time, ties by slot, either way.
template <typename V>
struct __align__(4 * sizeof(V)) Quad {
    V x, y, z, w;
};

template <typename V, int T>
__global__ void __launch_bounds__(T)
sort_events_kernel(const float* __restrict__ times, const int* __restrict__ pre_counts, int n_slots, int k_pre,
                   float tau_s, float tau,
                   const float* __restrict__ exp_s_in, const float* __restrict__ exp_in, Event* __restrict__ ev_out,
                   int* __restrict__ slot_out, int* __restrict__ ev_count, Event* __restrict__ ev_bucketed,
                   int* __restrict__ bucket_off, int bucket_width, int n_buckets, long long cap, int smem_cap,
                   unsigned char* __restrict__ scratch, const int* __restrict__ sample_order) {
    pdl_prologue();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int SORT_THREADS = T;
    SortShared<T>& sh = *reinterpret_cast<SortShared<T>*>(smem_raw);
    unsigned char* smem_items = smem_raw + sizeof(SortShared<T>);

    const int s = sample_order ? __ldg(sample_order + blockIdx.x) : (int)blockIdx.x;
    if ((unsigned)s >= gridDim.x) return;  // not a sample of the batch: the order is not a permutation
    const int tid = threadIdx.x;
    const long long sample_off = (long long)s * n_slots;
    const float* tsrc = times + sample_off;
    const int n_pre = n_slots / k_pre;
    // With the pre layer's spike counts, neuron j's valid slots are among its first pre_counts[j] (the forward kernels
    // write +inf after them), so only those are read.
    const int* cnt_src = pre_counts ? pre_counts + (long long)s * n_pre : nullptr;

    uint32_t* ka = reinterpret_cast<uint32_t*>(smem_items);
    uint32_t* kb = ka + smem_cap;
    V* va = reinterpret_cast<V*>(kb + smem_cap);
    V* vb = va + smem_cap;
    if (tid == 0) {
        sh.appended = 0;
        sh.kmin = 0xffffffffu;
        sh.kmax = 0u;
    }
    __syncthreads();
    gather_items<T, V>(tsrc, cnt_src, n_slots, k_pre, ka, va, smem_cap, sh);
    __syncthreads();
    const int n = sh.appended;
    if (n == 0) {
        // No spike in this sample: empty event list (and empty buckets).
        if (tid == 0) ev_count[s] = 0;
        if (ev_bucketed)
            for (int q = tid; q <= n_buckets; q += SORT_THREADS) bucket_off[(long long)s * (n_buckets + 1) + q] = 0;
        return;
    }
    if (n <= 256) {
        // At most one item per thread: its rank is the number of smaller items, with one barrier.
        if (tid < ((4 - n) & 3)) ka[n + tid] = 0xffffffffu;  // up to a multiple of four
        __syncthreads();
        const uint32_t key = tid < n ? ka[tid] : 0u;
        const V val = tid < n ? va[tid] : V(0);
        if (tid < n) {
            // By time and slot as one 64-bit number (the keys past n are larger than any time's).
            const unsigned long long mine = (unsigned long long)key << 32 | val;
            auto before = [&](uint32_t k, V v) { return ((unsigned long long)k << 32 | v) < mine ? 1 : 0; };
            int rank = 0;
            const uint4* k4 = reinterpret_cast<const uint4*>(ka);
            const Quad<V>* v4 = reinterpret_cast<const Quad<V>*>(va);
#pragma unroll 2
            for (int q = 0; q < (n + 3) >> 2; ++q) {
                const uint4 k = k4[q];
                const Quad<V> v = v4[q];
                rank += before(k.x, v.x) + before(k.y, v.y) + before(k.z, v.z) + before(k.w, v.w);
            }
            kb[rank] = key;
            vb[rank] = val;
        }
        __syncthreads();
        uint32_t* t0 = ka; ka = kb; kb = t0;
        V* t1 = va; va = vb; vb = t1;
    } else if (n > smem_cap || !bucket_sort<T, V>(ka, va, kb, vb, n, sh)) {
        if (n > smem_cap) {  // two key and two value buffers in this sample's part of the global scratch (cap items each)
            ka = reinterpret_cast<uint32_t*>(scratch + (long long)s * cap * (8 + 2 * sizeof(V)));
            kb = ka + cap;
            va = reinterpret_cast<V*>(kb + cap);
            vb = va + cap;
        }
        compact_slots<T, V>(tsrc, cnt_src, n_slots, k_pre, ka, va, sh);
        radix_sort<T, V>(ka, va, kb, vb, n, sh);
    }

    Event* eo = ev_out + (long long)s * cap;
    int* so = slot_out ? slot_out + (long long)s * cap : nullptr;
    for (int m = tid; m < n; m += SORT_THREADS) {
        eo[m] = make_event(ka[m], (uint32_t)va[m], k_pre, sample_off, exp_s_in, exp_in, tau_s, tau);
        if (so) so[m] = (int)va[m];
    }
    if (tid == 0) ev_count[s] = n;

    if (ev_bucketed) {
        // Stable counting pass by pre-neuron bucket over the time-sorted items.
        const int div = k_pre * bucket_width;
        if (tid < SORT_BINS) sh.hist[tid] = 0;
        __syncthreads();
        for (int i = tid; i < n; i += SORT_THREADS) atomicAdd(&sh.hist[(int)va[i] / div], 1);
        __syncthreads();
        scan_bins<T>(sh);
        int* bo = bucket_off + (long long)s * (n_buckets + 1);
        if (tid < n_buckets) bo[tid] = sh.base[tid];
        if (tid == 0) bo[n_buckets] = n;
        __syncthreads();
        stable_pass<T>(ka, va, kb, vb, n, sh, BucketDigit{div});
        Event* be = ev_bucketed + (long long)s * cap;
        for (int m = tid; m < n; m += SORT_THREADS)
            be[m] = make_event(kb[m], (uint32_t)vb[m], k_pre, sample_off, exp_s_in, exp_in, tau_s, tau);
    }
}

}  // namespace bats

// ---------------------------------------------------------------------------------------------
// C-ABI launchers (declared in include/bats_gb300.h).
#include <algorithm>
#include "abi_util.h"

// Shared-memory items and value width for a batch of samples with cap slots each (see SORT_SMALL_BATCH).
static void sort_plan(int batch, long long cap, int* smem_cap, bool* u16) {
    *u16 = cap <= 65536;
    const bool small = batch <= bats::SORT_SMALL_BATCH;
    const int room = *u16 ? (small ? bats::SORT_ROOM_MAX_U16 : bats::SORT_ROOM_U16)
                          : (small ? bats::SORT_ROOM_MAX_U32 : bats::SORT_ROOM_U32);
    *smem_cap = (int)std::min<long long>(room, (cap + 31) / 32 * 32);
}

extern "C" size_t bats_sort_events_workspace_bytes(int batch, int n_pre, int k_pre) {
    const long long cap = (long long)n_pre * k_pre;
    int smem_cap;
    bool u16;
    sort_plan(batch, cap, &smem_cap, &u16);
    if (cap <= smem_cap) return 0;
    return (size_t)(batch > 0 ? batch : 0) * (size_t)cap * (u16 ? 12 : 16);
}

template <typename V, int T>
static cudaError_t launch_sort(const float* pre_times, const int* pre_counts, int batch, long long cap, int k_pre,
                               float tau_s, float tau, const float* exp_tau_s, const float* exp_tau, void* ev_out,
                               int* slot_out, int* ev_count, void* ev_bucketed, int* bucket_offsets, int bucket_width,
                               int n_buckets, int smem_cap, unsigned char* scratch, const int* sample_order,
                               cudaStream_t stream) {
    const size_t smem = sizeof(bats::SortShared<T>) + (size_t)smem_cap * (8 + 2 * sizeof(V));
    cudaError_t e = (cudaError_t)bats::max_dynamic_smem_set((const void*)bats::sort_events_kernel<V, T>, (int)smem);
    if (e != cudaSuccess) return e;
    return bats::launch(bats::sort_events_kernel<V, T>, batch, T, smem, stream, pre_times, pre_counts, (int)cap, k_pre,
                        tau_s, tau, exp_tau_s, exp_tau, reinterpret_cast<bats::Event*>(ev_out), slot_out, ev_count,
                        reinterpret_cast<bats::Event*>(ev_bucketed), bucket_offsets, bucket_width, n_buckets, cap,
                        smem_cap, scratch, sample_order);
}
#define SORT_ARGS pre_times, pre_counts, batch, cap, k_pre, tau_s, tau, exp_tau_s, exp_tau, ev_out, slot_out, \
                  ev_count, ev_bucketed, bucket_offsets, bucket_width, n_buckets, smem_cap, scratch, sample_order, \
                  stream

static int sort_events_impl(const float* pre_times, const int* pre_counts, int batch, int n_pre, int k_pre,
                            float tau_s, float tau, const float* exp_tau_s, const float* exp_tau, void* ev_out,
                            int* slot_out, int* ev_count, void* ev_bucketed, int* bucket_offsets, int bucket_width,
                            const int* sample_order, void* workspace, size_t workspace_bytes, cudaStream_t stream) {
    BATS_REQUIRE(batch >= 0 && n_pre >= 0 && k_pre > 0, BATS_ERR_BAD_SHAPE, "sort_events: bad shape");
    if (batch == 0) return BATS_OK;
    BATS_REQUIRE(pre_times && ev_out && ev_count, BATS_ERR_NULL, "sort_events: null pointer");
    BATS_REQUIRE((exp_tau_s == nullptr) == (exp_tau == nullptr), BATS_ERR_NULL, "sort_events: give both exps or none");
    const long long cap = (long long)n_pre * k_pre;
    BATS_REQUIRE(cap < (1LL << 30), BATS_ERR_CAPACITY, "sort_events: n_pre*k_pre too large");
    int n_buckets = 0;
    if (ev_bucketed) {
        BATS_REQUIRE(bucket_offsets && bucket_width > 0, BATS_ERR_NULL, "sort_events: bucket outputs");
        n_buckets = (n_pre + bucket_width - 1) / bucket_width;
        BATS_REQUIRE(n_buckets <= bats::SORT_MAX_BUCKETS, BATS_ERR_CAPACITY,
                     "sort_events: more than 255 pre-neuron buckets (n_pre > 255 * bucket_width)");
    }
    const size_t need = bats_sort_events_workspace_bytes(batch, n_pre, k_pre);
    BATS_REQUIRE(workspace_bytes >= need && (need == 0 || workspace), BATS_ERR_WORKSPACE,
                 "sort_events: workspace too small");
    int smem_cap;
    bool u16;
    sort_plan(batch, cap, &smem_cap, &u16);
    unsigned char* scratch = reinterpret_cast<unsigned char*>(workspace);
    cudaError_t err;
    if (!u16)  // (wide)
        err = launch_sort<uint32_t, 512>(SORT_ARGS);
    else
        err = cap > bats::SORT_WIDE_CAP ? launch_sort<uint16_t, 512>(SORT_ARGS) : launch_sort<uint16_t, 256>(SORT_ARGS);
    BATS_CUDA(err);
    return BATS_OK;
}

extern "C" int bats_sort_events(const float* pre_times, int batch, int n_pre, int k_pre, float tau_s,
                                float tau, const float* exp_tau_s, const float* exp_tau, void* ev_out, int* slot_out,
                                int* ev_count, void* ev_bucketed, int* bucket_offsets, int bucket_width,
                                void* workspace, size_t workspace_bytes, cudaStream_t stream) {
    return sort_events_impl(pre_times, nullptr, batch, n_pre, k_pre, tau_s, tau, exp_tau_s, exp_tau, ev_out, slot_out,
                            ev_count, ev_bucketed, bucket_offsets, bucket_width, nullptr, workspace, workspace_bytes,
                            stream);
}

extern "C" int bats_sort_events_counted(const float* pre_times, const int* pre_counts, int batch, int n_pre,
                                        int k_pre, float tau_s, float tau, const float* exp_tau_s,
                                        const float* exp_tau, void* ev_out, int* slot_out, int* ev_count,
                                        void* ev_bucketed, int* bucket_offsets, int bucket_width, void* workspace,
                                        size_t workspace_bytes, cudaStream_t stream) {
    BATS_REQUIRE(pre_counts || batch == 0, BATS_ERR_NULL, "sort_events_counted: null pre_counts");
    return sort_events_impl(pre_times, pre_counts, batch, n_pre, k_pre, tau_s, tau, exp_tau_s, exp_tau, ev_out,
                            slot_out, ev_count, ev_bucketed, bucket_offsets, bucket_width, nullptr, workspace,
                            workspace_bytes, stream);
}

extern "C" int bats_sort_events_counted_ordered(const float* pre_times, const int* pre_counts, int batch, int n_pre,
                                                int k_pre, float tau_s, float tau, const float* exp_tau_s,
                                                const float* exp_tau, void* ev_out, int* slot_out, int* ev_count,
                                                void* ev_bucketed, int* bucket_offsets, int bucket_width,
                                                const int* sample_order, void* workspace, size_t workspace_bytes,
                                                cudaStream_t stream) {
    BATS_REQUIRE(pre_counts || batch == 0, BATS_ERR_NULL, "sort_events_counted_ordered: null pre_counts");
    BATS_REQUIRE(sample_order || batch == 0, BATS_ERR_NULL, "sort_events_counted_ordered: null sample_order");
    return sort_events_impl(pre_times, pre_counts, batch, n_pre, k_pre, tau_s, tau, exp_tau_s, exp_tau, ev_out,
                            slot_out, ev_count, ev_bucketed, bucket_offsets, bucket_width, sample_order, workspace,
                            workspace_bytes, stream);
}
