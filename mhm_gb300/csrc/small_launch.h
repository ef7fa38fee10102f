// small_launch.h -- which launches of the cell chain take the kernel of few cells
// (cell_chain_small.cu) and which the kernel of one thread a cell.
#pragma once
#include <cstdint>

namespace mhm {

// Blocks of the kernel of few cells that an SM holds: H + 2 warps each, one more
// with outputs, at 64 registers a thread.
constexpr int small_blocks_per_sm(int H, bool flux) { return 32 / (H + 2 + (flux ? 1 : 0)); }

// `cells` counts members times cells; `lean` as the kernels' template argument.
//
// While its blocks (32 cells each) fit the GPU at once the kernel of few cells
// takes 0.4 to 0.8 of the other's time; every further wave repeats the latency of
// the steps, while the other kernel has one wave up to 77,824 cells (58,368 with
// outputs).  So the line is drawn in waves, by horizon count: with few horizons the
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
    // With outputs the other kernel holds 3 blocks an SM, and a further wave, nearly
    // empty at first, takes as long as the first.  1 / 2 / 3 / 4 horizons: 62,500
    // cells 0.70 / 0.75 / 0.78 / 0.79 of its time, 90,000 cells 0.95 / 0.94 / 0.99 /
    // 0.98, 105,000 cells 1.00 / 1.00 / 1.17 / 1.12; its third wave 118,000 cells 0.87 /
    // 0.86 / 0.93 / 0.96, 130,000 cells 0.93 / 0.88 / 1.01 / 0.94; its fourth 178,000
    // cells 0.90 / 0.90 / 1.03 / 1.03.
    const int64_t one = (int64_t)sms * 3 * 128;
    return flux && H <= 4 && cells > one && cells <= (H <= 2 ? 4 : 2) * one && cells % one * 100 <= 55 * one;
}

} // namespace mhm
