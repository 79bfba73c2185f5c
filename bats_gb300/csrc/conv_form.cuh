// Which of the two forms of the position-grouped conv backward (conv_pool.cu) takes a batch, as a rule in whole
// numbers. Free of CUDA names, so that the host can be asked too.
#pragma once

#if defined(__CUDACC__)
#define BATS_FORM_HD __host__ __device__ __forceinline__
#else
#define BATS_FORM_HD inline
#endif

namespace bats {

// True for the events form: a batch of `samples` samples with `events` events over `n_pos` input positions and
// `spiking` post neurons that spike, filters of `taps` taps in all and `field` per output channel.
// The events form costs by the pairs of a spiking tap and up to 32 events (events / (32 n_pos samples) + 1/2 chunks of a
// position), the taps form by events and tiles of 32 taps, whatever spikes. The line is pairs <= 1/3 of events x tiles, from 256
// events x tiles a sample on (less does not repay the form's fixed cost). Measured on 2150 layers of 192 to 1024 taps, 1 to 256
// samples, K 4 to 32, every density, against the taps form alone (mean of the ratios, layers more than 1.2 times as long): with
// pre-errors 0.845, 34 (lines at 1/5 and 1/2: 0.850, 17 and 0.845, 60), without 0.804, 48 (0.812, 33 and 0.802, 64). Layers of
// convolutional networks lie near it: 24 filters 3 x 3 x 9, 21 samples, 0.24 pairs per event and tile, taps / events form 94 / 65 us;
// 40 filters 5 x 5 x 15, 128 samples, 0.19 pairs 2.65 / 2.07 ms; 16 filters 5 x 3 x 9, 114 samples, 0.59 pairs, no pre-errors
// 1.29 / 4.05 ms.
BATS_FORM_HD bool conv_events_pays(unsigned long long spiking, unsigned long long events, int samples, int n_pos,
                                   int taps, int field) {
    typedef unsigned __int128 wide;  // the products pass 64 bits for batches of many dense samples
    const unsigned long long work = events * (unsigned long long)((taps + 31) / 32);
    if (work < 256ull * (unsigned)samples) return false;
    const unsigned long long places = (unsigned long long)n_pos * (unsigned)samples;
    // pairs = spiking * field * (events + 16 places) / (32 places)
    const wide pairs32 = (wide)(spiking * (unsigned)field) * (events + 16ull * places);
    return pairs32 * 3u <= (wide)work * (32ull * places);
}

}  // namespace bats
