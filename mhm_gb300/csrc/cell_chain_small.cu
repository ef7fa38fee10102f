// cell_chain_small.cu -- the cell chain of launches that leave the GPU mostly
// idle: few cells, so that the time of a call is the latency of a step, not the
// throughput of the SMs.
#include "cell_chain_impl.cuh"
#include "launch_rules.h"

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
//
// FLUX, aggregated outputs or per-step fluxes: one more warp adds up what the
// others post of a step while they work on the next.
template <int H, bool LEAN, bool FLUX>
__global__ void __launch_bounds__(32 * (H + 2 + FLUX), small_blocks_per_sm(H, FLUX))
    cell_chain_small_kernel(const CellArgs a)
{
    __shared__ double s_sm[H][32], s_fr[H][32], s_st[H][32], s_sms[H][32];
    __shared__ double s_pe[2][32], s_demand[2][32], s_rsealed[2][32]; // by parity of the step
    // posted for the outputs, by step: the surface's values (the surface is two
    // steps ahead of the reader), the values below
    constexpr int kSurf = 9, kBelow = 7, kPost = FLUX ? 32 : 1;
    __shared__ double s_surf[3][kSurf][kPost], s_below[2][kBelow][kPost], s_out[2][3][H][kPost]; // SM, aET, infiltration
    constexpr int n_warps = H + 2 + FLUX;
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
    constexpr int all = 32 * n_warps, below = 32 * (H + 1); // below: the soil and the horizons
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
                if constexpr (FLUX) {
                    const double v[kSurf] = {sf.interc, sf.snow, sf.seal, sf.pet, sf.aet_can, sf.aet_sealed_act,
                                             sf.runoff_sealed, sf.prec_effect, sf.melt};
#pragma unroll
                    for (int i = 0; i < kSurf; ++i) s_surf[t % 3][i][lane] = v[i];
                }
            }
            bar_sync(1, all); // step t above the soil; the soil has taken step t - 1 from the other buffer
        }
        if (FLUX) bar_sync(1, all);
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
        const double fsealed = par(P_FSEALED), share = Ground::share(fsealed);
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
                        if constexpr (FLUX) s_out[t & 1][2][h][lane] = infil;
                    }
                } else if constexpr (FLUX) {
#pragma unroll
                    for (int h = 0; h < H; ++h) s_out[t & 1][2][h][lane] = 0.0;
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
                    if constexpr (FLUX) s_out[t & 1][0][h][lane] = left, s_out[t & 1][1][h][lane] = aet;
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
                const double q_total = gd.total(share, s_rsealed[t & 1][lane], fsealed);
                tro[(size_t)t * out_stride] = q_total;
                chk(q_total);
                if constexpr (FLUX) {
                    const double v[kBelow] = {gd.unsat, gd.sat, gd.fast, gd.slow, gd.base, gd.perc, q_total};
#pragma unroll
                    for (int i = 0; i < kBelow; ++i) s_below[t & 1][i][lane] = v[i];
                }
            }
        }
        if (FLUX) bar_sync(1, all);
        if (active) {
            S[(size_t)S_UNSAT * N] = gd.unsat;
            S[(size_t)S_SAT * N] = gd.sat;
            chk(gd.unsat);
            chk(gd.sat);
        }
    } else if (FLUX && part == H + 2) { // outputs
        extern __shared__ double s_acc[]; // the running sums, [plane][32]
        const OutArgs &o = a.out;
        const size_t at = (size_t)m * N + k;
        const double fsealed = par(P_FSEALED), fnotsealed = 1.0 - fsealed, karst = par(P_KARST);
        double osat = 0.0;
        for (int h = 0; h < H; ++h) osat = osat + par(P_HORIZON + H + h);
        const uint64_t r_osat = hm_recip_of(osat);
        int cnt = o.cnt0, slot = o.slot0;
        const int64_t tt_w = o.n_planes > 0 && o.tt_w ? o.tt_w[m] : -1;
        if (active)
            for (int v = 0; v < o.n_planes; ++v) s_acc[v * 32 + lane] = o.acc[(size_t)v * out_stride + at];
        auto add = [&](int plane, double x) { s_acc[plane * 32 + lane] = s_acc[plane * 32 + lane] + x; };
        bar_sync(1, all);
        for (int t = 0; t < a.n_steps; ++t) {
            bar_sync(1, all); // step t below the soil, step t + 1 above it
            if (active) {
                const auto &u = s_surf[t % 3];
                const auto &d = s_below[t & 1];
                const auto &q = s_out[t & 1];
                double aet_soil = 0.0;
#pragma unroll
                for (int h = 0; h < H; ++h) aet_soil = aet_soil + q[1][h][lane];
                const OutStep v{u[0][lane], u[1][lane], u[2][lane], u[3][lane], u[4][lane], u[5][lane],
                                u[6][lane], u[7][lane], u[8][lane], d[0][lane], d[1][lane], d[2][lane],
                                d[3][lane], d[4][lane], d[5][lane], d[6][lane], aet_soil};
                if (a.flux_aet) {
                    const size_t fo = (size_t)t * out_stride + at;
                    a.flux_aet[fo] = v.aet_can + fsealed * v.aet_sealed + fnotsealed * aet_soil;
                    a.flux_loss[fo] = fnotsealed * (v.perc - v.perc * karst);
                }
                const int64_t tt = o.tt_base + t;
                if (o.n_planes > 0 && tt > o.warm_steps) {
                    // the weights of cell_chain_item
                    const bool ow = tt == tt_w;
                    double ofs = fsealed, ofns = fnotsealed;
                    if (ow) {
                        ofs = o.w_fsealed[at];
                        ofns = 1.0 - ofs;
                    }
                    for (int h = 0; h < H; ++h) {
                        if (o.plane[OF_INFIL] >= 0) add(o.plane[OF_INFIL] + h, q[2][h][lane] * ofns);
                        if (o.plane[OF_AET_L] >= 0) add(o.plane[OF_AET_L] + h, q[1][h][lane] * ofns);
                    }
                    out_add(
                        o, H, v, ow, ofs, ofns, osat, r_osat, add, [&](int h) { return q[0][h][lane]; },
                        [&](int h) { return ow ? o.w_sms[((size_t)m * H + h) * N + k] : par(P_HORIZON + H + h); });
                    out_close(o, s_acc + lane, 32, out_stride, at, tt, steps[t].dflags, cnt, slot);
                }
            }
        }
        if (active)
            for (int v = 0; v < o.n_planes; ++v) o.acc[(size_t)v * out_stride + at] = s_acc[v * 32 + lane];
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
        if (FLUX) bar_sync(1, all);
        if (active) {
            const double smh = s_sm[h][lane];
            S[(size_t)(S_SM + h) * N] = smh;
            chk(smh);
        }
    }
    if (active && a.nonfinite && (nonfin >> 63)) atomicOr(a.nonfinite + m, 1);
}

} // namespace

template <bool LEAN, bool FLUX> static cudaError_t launch_small(const CellArgs &a, cudaStream_t s)
{
    const size_t smem = FLUX ? (size_t)a.out.n_planes * 32 * sizeof(double) : 0;
    const int64_t n = (int64_t)a.n_cells * a.n_members;
    const unsigned grid = (unsigned)((n + 31) / 32);
    switch (a.n_horizons) {
#define MHM_CASE(HH)                                                                                               \
    case HH:                                                                                                       \
        cell_chain_small_kernel<HH, LEAN, FLUX><<<grid, 32 * (HH + 2 + FLUX), smem, s>>>(a);                                     \
        return cudaGetLastError();
        MHM_CASE(1) MHM_CASE(2) MHM_CASE(3) MHM_CASE(4) MHM_CASE(5) MHM_CASE(6) MHM_CASE(7) MHM_CASE(8)
#undef MHM_CASE
    default:
        return cudaErrorInvalidValue;
    }
}

bool cell_chain_fits_small(const CellArgs &a)
{
    const bool flux = a.flux_aet || a.out.n_planes > 0;
    return a.small_ok && small_launch(a.n_horizons, cell_chain_lean(a), flux, (int64_t)a.n_cells * a.n_members, device_sms());
}

cudaError_t launch_cell_chain_small(const CellArgs &a, cudaStream_t s)
{
    if (a.flux_aet || a.out.n_planes > 0) return launch_small<false, true>(a, s);
    return cell_chain_lean(a) ? launch_small<true, false>(a, s) : launch_small<false, false>(a, s);
}

} // namespace mhm

MHM_BC_ACCESSOR(bc_take_cell_chain_small)
