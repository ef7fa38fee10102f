// launch_rules.h -- which launches of the cell chain take the kernel of few cells
// (cell_chain_small.cu) and which the kernel of one thread a cell; the blocks an SM
// of the latter with outputs.
#pragma once
#include <cstdint>

namespace mhm {

// Waves of blocks of 128 threads, `blocks` of them an SM.
constexpr int64_t waves_of(int64_t cells, int sms, int blocks)
{
    return (cells + (int64_t)sms * blocks * 128 - 1) / ((int64_t)sms * blocks * 128);
}

// The blocks an SM that the registers of the one-thread-a-cell kernel are sized for
// with outputs or per-step fluxes.  With 3 blocks a thread holds what a step adds
// up, with 4 some of it goes through local memory, so a wave of 4 blocks takes
// about as much longer as it holds more cells: 4 where they save a third of the
// waves.  48 steps, 4 / 3 blocks: 57,840 cells, 1 / 3 / 5 / 8 horizons 0.59 / 0.57,
// 0.91 / 0.81, 1.27 / 1.21, 1.81 / 1.64 ms (one wave each); 62,500 cells 0.67 / 1.01,
// 1.03 / 1.44, 1.43 / 2.13, 2.02 / 3.03 (1 / 2 waves); 90,000 cells 1.20 / 1.09, 1.95 /
// 1.55, 2.71 / 2.27, 3.90 / 3.19 (2 / 2); 130,000 cells 1.31 / 1.60, 2.10 / 2.23, 2.97 /
// 3.38, 4.30 / 4.79 (2 / 3); 199,809 cells 1.96 / 2.15, 3.15 / 3.08, 4.46 / 4.65, 6.49 /
// 6.80 (3 / 4); 299,756 cells 2.67 / 3.14, 4.37 / 4.52, 6.15 / 6.80, 8.98 / 9.74 (4 / 6).
// With 2 blocks a large launch lacks warps (160,000 cells, 3 horizons, 240 steps:
// 10.3 ms with 3, 14.3 with 2).
constexpr int flux_blocks_per_sm(int64_t cells, int sms)
{
    return 3 * waves_of(cells, sms, 4) <= 2 * waves_of(cells, sms, 3) ? 4 : 3;
}

// Blocks of the kernel of few cells that an SM holds: H + 2 warps each, one more
// with outputs, at 64 registers a thread.
constexpr int small_blocks_per_sm(int H, bool flux) { return 32 / (H + 2 + (flux ? 1 : 0)); }

// `cells` counts members times cells; `lean` as the kernels' template argument.
//
// While its blocks (32 cells each) fit the GPU at once the kernel of few cells
// takes 0.4 to 0.8 of the other's time; every further wave repeats the latency of
// the steps, while the other kernel has one wave up to 77,824 cells.  So the line is drawn in waves, by horizon count: with few horizons the
// other kernel's step is short and a second wave loses, with many it still gains.
// Measured as this kernel's time over the other's, 48 hourly steps.
//   lean: 1 horizon 0.74 at 0.98 waves, 1.07 at 1.02 (49,506 cells 0.37 / 0.35 ms);
//     2 horizons 0.92 at 1.02, 1.00 at 1.35, 1.04 at 1.5; 3 horizons 0.84, 0.93 at
//     1.6, 1.01 at 1.85; 4 to 8 horizons 0.76-0.82, 0.86-1.00 at 1.98, 1.07-1.14 at
//     2.05.
//   general, where the other kernel is slower: 0.66-0.97 at 1.02, 0.73-0.98 at 1.98;
//     2 horizons 0.93 at 2.6, 5 horizons 0.95 at 2.5, 6 and 8 horizons 0.95 at 2.2.
//   outputs: 1 and 2 horizons 0.98-1.2 above one wave; 3 and 5 horizons 0.93 at 1.02,
//     1.00 at 1.2, 1.06 at 1.4; 4 horizons 0.84, 1.01 at 1.98; 6 horizons 0.93, 0.97
//     at 1.6, 1.03 at 1.75; 7 horizons 0.85, 0.88 at 1.98; 8 horizons 0.74, 0.94 at
//     2.5.
inline bool small_launch(int H, bool lean, bool flux, int64_t cells, int sms)
{
    constexpr int kWaves[3][8] = {{200, 260, 200, 200, 250, 225, 205, 225},  // hundredths: general,
                                  {100, 135, 185, 200, 200, 200, 200, 200},  // lean,
                                  {100, 100, 120, 200, 120, 165, 200, 250}}; // outputs
    if (H < 1 || H > 8) return false;
    const int64_t wave = (int64_t)sms * small_blocks_per_sm(H, flux) * 32;
    if (cells * 100 <= kWaves[flux ? 2 : lean ? 1 : 0][H - 1] * wave) return true;
    // With outputs and up to 4 horizons it also beats a second wave of the other
    // kernel's 4 blocks an SM that is not much more than begun.  1 / 2 / 3 / 4 horizons:
    // 79,800 cells 0.87 / 0.78 / 0.95 / 0.92 of its time, 90,000 cells 0.95 / 0.94 / 0.99 /
    // 0.98, 105,000 cells 1.00 / 1.00 / 1.17 / 1.12.
    const int64_t one = (int64_t)sms * 4 * 128;
    return flux && H <= 4 && cells > one && cells * 100 <= 116 * one;
}

} // namespace mhm
