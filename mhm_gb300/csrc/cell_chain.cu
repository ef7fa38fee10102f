// cell_chain.cu -- launchers of the cell-chain kernel (register variant for
// 4 resident blocks per SM) and of the step-calendar kernel.  Variants sized
// for 6 and 8 resident blocks per SM live in cell_chain_o6.cu / _o8.cu, the
// kernel of small launches in cell_chain_small.cu.
#include "cell_chain_impl.cuh"
#include "launch_rules.h"

namespace mhm {

cudaError_t launch_cell_chain_o6(const CellArgs &a, int H, cudaStream_t s);
cudaError_t launch_cell_chain_o8(const CellArgs &a, int H, cudaStream_t s);
bool cell_chain_fits_small(const CellArgs &a);
cudaError_t launch_cell_chain_small(const CellArgs &a, cudaStream_t s);

// Calendar of steps tt0 .. tt0+n-1: forcing row, month, day flags, day of year.
__global__ void steps_fill_kernel(StepInfo *steps, int64_t tt0, int32_t n, int32_t jul_start, int32_t timestep,
                                  int32_t stride, int32_t lai_mode)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t tt = tt0 + i;
    const StepDate sd = step_date(jul_start, timestep, tt);
    StepInfo si;
    si.row = (int32_t)((tt + stride - 1) / stride); // iMeteoTS, mo_meteo_handler.f90:575-620
    si.month = (int8_t)sd.month;
    si.dflags = (int8_t)step_dflags(jul_start, timestep, tt);
    si.doy = (int16_t)sd.doy;
    si.hour = (int8_t)sd.hour;
    si.lai = (int16_t)step_lai(jul_start, timestep, tt, lai_mode);
    steps[i] = si;
}

cudaError_t launch_steps_fill(StepInfo *steps, int64_t tt0, int32_t n, int32_t jul_start, int32_t timestep,
                              int32_t stride, int32_t lai_mode, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    steps_fill_kernel<<<(n + 255) / 256, 256, 0, s>>>(steps, tt0, n, jul_start, timestep, stride, lai_mode);
    return cudaGetLastError();
}

// Initial states of one member: a value a state plane, zero routing states.
// Only writes, (5 + H) N + 4 L numbers; a call for 40,000 cells with 3 horizons
// 19 us, where building the planes on the host and copying them took 150 us.
__global__ void __launch_bounds__(256) init_states_kernel(const InitArgs a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, pl = blockIdx.y;
    if (pl < a.n_planes) {
        if (i < a.n_cells) a.states[(size_t)pl * a.n_cells + i] = a.value[pl];
    } else if (i < a.n_nodes) {
        a.routing[pl - a.n_planes][i] = 0.0;
    }
}

cudaError_t launch_init_states(const InitArgs &a, cudaStream_t s)
{
    const int n = max(a.n_cells, a.n_nodes);
    init_states_kernel<<<dim3((n + 255) / 256, a.n_planes + (a.n_nodes > 0 ? 4 : 0)), 256, 0, s>>>(a);
    return cudaGetLastError();
}

// The persistent multi-context launch: hl = horizon planes of the shared
// layout (6 or 8, at least every context's horizon count), `lean` as the
// contexts' common code path, occ = resident blocks per SM the registers are
// sized for (4 or 8).  One resident wave of blocks takes the tiles.
cudaError_t launch_cell_chain_fused(const FusedCellArgs &f, int hl, bool lean, int occ, cudaStream_t s)
{
    if (f.n_tiles <= 0) return cudaSuccess;
    const int block = 128;
    const size_t smem = hs_bytes(hl, block);
    void (*k)(const FusedCellArgs) = nullptr;
    const bool o8 = occ >= 8;
    if (hl == 6)
        k = lean ? (o8 ? cell_chain_fused_kernel<6, true, 8> : cell_chain_fused_kernel<6, true, 4>)
                 : (o8 ? cell_chain_fused_kernel<6, false, 8> : cell_chain_fused_kernel<6, false, 4>);
    else if (hl == 8)
        k = lean ? (o8 ? cell_chain_fused_kernel<8, true, 8> : cell_chain_fused_kernel<8, true, 4>)
                 : (o8 ? cell_chain_fused_kernel<8, false, 8> : cell_chain_fused_kernel<8, false, 4>);
    else
        return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int nb = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, block, smem)) != cudaSuccess) return e;
    const int64_t wave = (int64_t)(nb < 1 ? 1 : nb) * device_sms();
    const unsigned grid = (unsigned)(f.n_tiles < wave ? f.n_tiles : wave);
    k<<<grid, block, smem, s>>>(f);
    return cudaGetLastError();
}

// The register variant of a launch nobody chose one for: the fewest waves of
// blocks, then the fewest blocks an SM -- more registers shorten a step, another
// wave repeats all of them.  With 7 or 8 horizons 8 blocks' planes do not fit an
// SM's shared memory.  3 horizons, 48 steps, 4 / 6 / 8 blocks: 62,500 cells 0.51 /
// 0.61 / 0.68 ms, 99,856 cells 0.90 / 0.71 / 0.79, 160,000 cells 1.31 / 1.23 /
// 1.42, 250,000 cells 1.83 / 1.78 / 1.71; 6 horizons, 24 steps: 144,400 cells
// 0.75 / 0.88 / 0.68, 640,000 cells 3.10 / 2.83 / 2.86, 1e6 cells 4.65 / 4.24 /
// 4.21; 8 horizons 1e6 cells 5.57 / 5.07 / 5.56.
static int cell_chain_occ(const CellArgs &a, int H)
{
    const int64_t n = (int64_t)a.n_cells * a.n_members;
    const int sms = device_sms();
    int best = 4;
    int64_t best_waves = INT64_MAX;
    for (int occ = 4; occ <= (H <= 6 ? 8 : 6); occ += 2) {
        const int64_t waves = waves_of(n, sms, occ);
        if (waves < best_waves) best = occ, best_waves = waves;
    }
    return best;
}

// occ = resident blocks per SM the kernel's registers are sized for (4, 6, 8; 0:
// by the rule above)
cudaError_t launch_cell_chain(const CellArgs &a, int H, int occ, cudaStream_t s)
{
    if (H < 1 || H > kMaxHorizons) return cudaErrorInvalidValue;
    if (cell_chain_fits_small(a)) return launch_cell_chain_small(a, s);
    if (a.flux_aet || a.out.n_planes > 0) // per-step fluxes or aggregated outputs
        return flux_blocks_per_sm((int64_t)a.n_cells * a.n_members, device_sms()) == 4
                   ? launch_cell_chain_variant<4, true>(a, H, s)
                   : launch_cell_chain_variant<3, true>(a, H, s);
    if (occ == 0) occ = cell_chain_occ(a, H);
    switch (occ) {
    case 6: return launch_cell_chain_o6(a, H, s);
    case 8: return launch_cell_chain_o8(a, H, s);
    default: return launch_cell_chain_variant<4>(a, H, s);
    }
}

} // namespace mhm

MHM_BC_ACCESSOR(bc_take_cell_chain)
