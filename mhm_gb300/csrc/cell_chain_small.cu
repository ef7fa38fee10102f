// cell_chain_small.cu -- the cell chain of launches that leave the GPU mostly
// idle: few cells, so that the time of a call is the latency of a step, not the
// throughput of the SMs.
#include "cell_chain_impl.cuh"

namespace mhm {

namespace {

__device__ __forceinline__ void bar_sync(int id, int threads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// A block of H + 2 warps holds 32 cells, a lane of every warp belonging to a
// cell, and each warp does one part of every step:
//   surface  meteo, canopy, snow and the sealed bucket, one step ahead -- it
//            depends on the forcing and its own states only;
//   soil     the water's way down the horizons, the actual evapotranspiration,
//            and the zones below the soil;
//   H more   one horizon each, its parameters in registers: the runoff fraction
//            from the soil moisture a step leaves, the stress factor from the
//            soil moisture after infiltration.
// The operations, operands and their order within a cell are those of
// cell_chain_item, so the results are its bits.
//
// What bounds it: the latency of a step's longest chain.  One thread a cell
// runs a step's 2,100-3,500 dependent instructions and ~35 dependent FP64
// operations (64 cycles each) one after another, 14,000-18,000 cycles; here the
// chain is infiltration, one stress factor, the uptakes and one fraction,
// 5,000-10,000.  96 hourly steps of 9,216 cells: 1 horizon 0.51 -> 0.24 ms, 3
// horizons 0.68 -> 0.32, 6 horizons 0.96 -> 0.49; 36 cells, 2,160 steps of daily
// forcing 14.6 -> 5.0 ms.
//
// 64 registers a thread, so that as many blocks as possible are resident.
template <int H, bool LEAN>
__global__ void __launch_bounds__(32 * (H + 2), 1024 / (32 * (H + 2))) cell_chain_small_kernel(const CellArgs a)
{
    __shared__ double s_sm[H][32], s_fr[H][32], s_st[H][32], s_sms[H][32];
    __shared__ double s_pe[2][32], s_demand[2][32], s_rsealed[2][32]; // by parity of the step
    constexpr int n_warps = H + 2;
    const int lane = threadIdx.x & 31;
    // parts start at another warp in each block of an SM, so that the
    // schedulers share them
    const int part = (int)((threadIdx.x >> 5) + blockIdx.x / 152) % n_warps;
    const int64_t N = a.n_cells, gid = (int64_t)blockIdx.x * 32 + lane;
    bool active = gid < N * a.n_members;
    const int m = active ? (int)(gid / N) : 0, k = active ? (int)(gid - (int64_t)m * N) : 0;
    const StepInfo *steps = a.steps;
    bool reset_sm = a.reset_sm != 0;
    const size_t out_stride = (size_t)a.n_members * N;
    double *tro = a.tro + (size_t)m * N + k;
    if (a.member_step0) {
        const int32_t b = a.member_step0[m];
        if (b < 0) { // idle member slot: no state update, zero runoff
            if (active && part == 0)
                for (int t = 0; t < a.n_steps; ++t) tro[(size_t)t * out_stride] = 0.0;
            active = false;
        } else if (!bc_ok(BC_STEP_ROW, (long long)b + a.step_shift + a.n_steps - 1, a.n_step_rows)) {
            active = false;
        } else {
            steps += b + a.step_shift;
        }
        reset_sm = a.reset_ok && (b + a.step_shift == 0);
    }
    const double *P = a.params + (size_t)m * n_param_planes(H) * N + k;
    double *S = a.states + (size_t)m * n_state_planes(H) * N + k;
    auto par = [&](int plane) { return __ldg(P + (size_t)plane * N); };
    const bool feddes = LEAN || (a.proc_sm == 1 || a.proc_sm == 4);
    constexpr int all = 32 * n_warps, below = all - 32; // below: without the surface
    constexpr uint64_t kExpOne = 0x0010000000000000ull; // as in cell_chain_item
    uint64_t nonfin = 0;
    auto chk = [&](double x) { nonfin |= hm_abs_bits(hm_d2b(x)) + kExpOne; };

    if (part == 1) { // surface
        Surface<LEAN, true> sf;
        sf.load(a, P, S, par(P_FSEALED), k);
        bool on = active;
        for (int t = 0; t < a.n_steps; ++t) {
            if (on) {
                const StepInfo si = steps[t];
                const int32_t row = a.member_step0 ? a.step_shift + t : si.row - a.row_base;
                on = bc_ok(BC_FORCING_ROW, row, a.n_forc_rows) && sf.step(a, P, si, (size_t)row * N + k, m, k);
            }
            if (on) {
                sf.sealed_step();
                s_pe[t & 1][lane] = sf.prec_effect;
                s_demand[t & 1][lane] = sf.pet - sf.aet_can;
                s_rsealed[t & 1][lane] = sf.runoff_sealed;
            }
            bar_sync(1, all); // step t above the soil; the soil has taken step t - 1 from the other buffer
        }
        if (active) {
            S[(size_t)S_INTERC * N] = sf.interc;
            S[(size_t)S_SNOW * N] = sf.snow;
            S[(size_t)S_SEAL * N] = sf.seal;
            chk(sf.interc);
            chk(sf.snow);
            chk(sf.seal);
        }
    } else if (part == 0) { // soil
        Ground gd;
        gd.load(a, P, S);
        const double fsealed = par(P_FSEALED), fnotsealed = 1.0 - fsealed;
        bool frac_bounded = true; // every horizon's runoff fraction is in [0, 1]
        for (int h = 0; h < H; ++h) {
            const double sms = par(P_HORIZON + H + h);
            s_sms[h][lane] = sms;
            frac_bounded = frac_bounded && sm_frac_bounded(sms, par(P_HORIZON + 4 * H + h));
        }
        for (int t = 0; t < a.n_steps; ++t) {
            bar_sync(1, all); // the surface's step, the fractions
            double infil = 0.0, demand = 0.0;
            if (active) {
                const double pe = s_pe[t & 1][lane];
                demand = s_demand[t & 1][lane];
                // mo_soil_moisture.f90:230-252; +0 changes nothing (cell_chain_item)
                if (hm_d2b(pe) != 0 || !frac_bounded) {
                    infil = pe;
                    double sms[H], sm[H], fr[H];
#pragma unroll
                    for (int h = 0; h < H; ++h) sms[h] = s_sms[h][lane], sm[h] = s_sm[h][lane], fr[h] = s_fr[h][lane];
#pragma unroll
                    for (int h = 0; h < H; ++h) {
                        if (!hm_gt(sm[h], sms[h])) { // else the horizon passes its input on
                            const double tmp = infil * fr[h];
                            const double filled = sm[h] + tmp, rest = infil + hm_neg(tmp);
                            if (hm_unlikely(hm_gt(filled, sms[h]))) {
                                infil = infil + (sm[h] - sms[h]);
                                s_sm[h][lane] = sms[h];
                            } else {
                                infil = rest;
                                s_sm[h][lane] = filled;
                            }
                        }
                    }
                }
            }
            bar_sync(2, below); // the soil moisture after infiltration
            bar_sync(2, below); // the stress factors
            if (active) {
                double sm[H], st[H];
#pragma unroll
                for (int h = 0; h < H; ++h) sm[h] = s_sm[h][lane], st[h] = s_st[h][lane];
                double aet_above = 0.0; // masked running sum of positive aet above
#pragma unroll
                for (int h = 0; h < H; ++h) {
                    double aet = demand;
                    if (h > 0) aet = aet - aet_above;
                    aet = aet * st[h];
                    aet = hm_sel(hm_lt0(aet), 0.0, aet);
                    const bool enough = hm_gt(sm[h], aet);
                    const double d = sm[h] - hm_sel(enough, aet, kEps);
                    aet = hm_sel(enough, aet, d);
                    double left = hm_sel(enough, d, kEps);
                    left = hm_sel(hm_lt(left, kEps), kEps, left);
                    s_sm[h][lane] = left;
                    if (h == 0) {
                        aet_above = hm_sel(hm_gt0(aet), aet, 0.0);
                    } else if (h + 1 < H) {
                        aet_above = hm_sel(hm_gt0(aet), aet_above + aet, aet_above);
                    }
                }
            }
            bar_sync(2, below); // the soil moisture of the step
            if (active) {
                gd.step(infil);
                const double q_total = gd.total(fnotsealed, s_rsealed[t & 1][lane], fsealed);
                tro[(size_t)t * out_stride] = q_total;
                chk(q_total);
            }
        }
        if (active) {
            S[(size_t)S_UNSAT * N] = gd.unsat;
            S[(size_t)S_SAT * N] = gd.sat;
            chk(gd.unsat);
            chk(gd.sat);
        }
    } else { // horizon h
        const int h = part - 2;
        const double froots = par(P_HORIZON + h), sms = par(P_HORIZON + H + h), fc = par(P_HORIZON + 2 * H + h),
                     pw = par(P_HORIZON + 3 * H + h), beta = par(P_HORIZON + 4 * H + h);
        const double den = feddes ? fc - pw : sms - pw; // mo_soil_moisture.f90:358, :435
        const double jarvis = LEAN ? 0.0 : par(P_JARVIS);
        const uint64_t r_sms = hm_recip_of(sms), r_den = hm_recip_of(den), r_jarvis = LEAN ? 0 : hm_recip_of(jarvis);
        s_sm[h][lane] = reset_sm ? 0.5 * fc : S[(size_t)(S_SM + h) * N];
        for (int t = 0; t < a.n_steps; ++t) {
            if (active) { // 1 - the runoff fraction, mo_soil_moisture.f90:230-234
                const double smh = s_sm[h][lane];
                double fr = 0.0;
                if (hm_gt(smh, kEps) && !hm_gt(smh, sms)) fr = hm_exp(beta * hm_log(hm_div_r(smh, sms, r_sms)));
                s_fr[h][lane] = 1.0 - fr;
            }
            bar_sync(1, all);
            bar_sync(2, below);
            if (active) s_st[h][lane] = stress_factor(feddes, s_sm[h][lane], fc, pw, froots, den, r_den, jarvis, r_jarvis);
            bar_sync(2, below);
            bar_sync(2, below);
        }
        if (active) {
            const double smh = s_sm[h][lane];
            S[(size_t)(S_SM + h) * N] = smh;
            chk(smh);
        }
    }
    if (active && a.nonfinite && (nonfin >> 63)) atomicOr(a.nonfinite + m, 1);
}

} // namespace

template <bool LEAN> static cudaError_t launch_small(const CellArgs &a, cudaStream_t s)
{
    const int64_t n = (int64_t)a.n_cells * a.n_members;
    const unsigned grid = (unsigned)((n + 31) / 32);
    switch (a.n_horizons) {
#define MHM_CASE(HH)                                                                                               \
    case HH:                                                                                                       \
        cell_chain_small_kernel<HH, LEAN><<<grid, 32 * (HH + 2), 0, s>>>(a);                                       \
        return cudaGetLastError();
        MHM_CASE(1) MHM_CASE(2) MHM_CASE(3) MHM_CASE(4) MHM_CASE(5) MHM_CASE(6) MHM_CASE(7) MHM_CASE(8)
#undef MHM_CASE
    default:
        return cudaErrorInvalidValue;
    }
}

// Up to 180,000 warps' lanes (cells times H + 2): where the blocks no longer fit
// the GPU at once (96 steps, this kernel / one thread a cell: 1 horizon, 40,000
// cells 0.45 / 0.67 ms, 62,500 cells 0.80 / 0.76; 3 horizons, 25,600 cells 0.51 /
// 0.78, 40,000 cells 0.81 / 0.88, 62,500 cells 1.25 / 0.99; 6 horizons, 16,384
// cells 0.61 / 0.96, 25,600 cells 1.01 / 1.10, 40,000 cells 1.48 / 1.25).
bool cell_chain_fits_small(const CellArgs &a)
{
    return a.small_ok && (int64_t)a.n_cells * a.n_members * (a.n_horizons + 2) <= 180000;
}

cudaError_t launch_cell_chain_small(const CellArgs &a, cudaStream_t s)
{
    return cell_chain_lean(a) ? launch_small<true>(a, s) : launch_small<false>(a, s);
}

} // namespace mhm

MHM_BC_ACCESSOR(bc_take_cell_chain_small)
