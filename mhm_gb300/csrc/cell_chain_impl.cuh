// cell_chain_impl.cuh -- the mHM L1 cell chain as one time-looping kernel
// (included by the translation units that instantiate its register/occupancy
// variants).
//
// One thread advances one (member, cell) through a chunk of time steps with
// all states and effective parameters in registers; forcing is read once per
// step as coalesced [step][cell] rows and the step's total runoff is written
// as a coalesced [step][member][cell] row.  The arithmetic of every step is
// the reference's, in the reference's order (compiled with --fmad=false;
// log/exp/pow from hmath.h), so a step here equals a step of
//   mHM() cell loop              src/mHM/mo_mhm.f90:458-517
//   get_corrected_pet/temp/prec  src/meteo/mo_meteo_handler.f90:915-1285
// bit for bit.  Expressions that depend on parameters only (c2TSTu/k, the
// degree-day threshold, FC-PW, ...) are evaluated once per chunk: the same
// operands give the same bits as the reference's per-step evaluation.
#pragma once
#include <cfloat>
#include <cmath>

#include "bounds.cuh"
#include "calendar.h"
#include "fp64i.h"
#include "hmath.h"
#include "mhm_kernels.cuh"

namespace mhm {

namespace {

constexpr double kEps = DBL_EPSILON; // src/common/mo_common_constants.f90:25
constexpr double kTwoThird = 2.0 / 3.0;
constexpr uint32_t kDenExp = 1023 - 4; // FC - PW of 2^-4 .. 2^11 mm takes hm_uptake
constexpr double kPiD = 3.141592653589793238462643383279502884197;
constexpr double kTwoPiD = 6.283185307179586476925286766559005768394;
constexpr double kDaySecs = 86400.0, kYearDays = 365.0, kSolarConst = 1367.0, kSpecHeatET = 2.45e06;
constexpr double kDeg2Rad = 3.141592653589793238462643383279502884197 / 180.0;
constexpr double kHarSamConst = 17.800;
// src/common/mo_constants.f90 (Psychro_dp) and src/mHM/mo_mhm_constants.f90 (tetens_c*, satpressureslope1)
constexpr double kPsychro = 0.0646, kTetensC1 = 0.6108, kTetensC2 = 17.270, kTetensC3 = 237.30;
constexpr double kSatPressureSlope1 = 4098.0;
constexpr double kT0 = 273.15; // FORCES mo_constants T0_dp (Celsius <-> Kelvin)
constexpr double kRho0 = 1.225, kCp0 = 1005.0; // air density, heat capacity (FORCES mo_constants)

// src/mHM/mo_pet.f90:314-355 (CUDA's sin/cos/tan/acos; only the daily-forcing
// Hargreaves variant uses it)
__device__ double extraterr_rad_approx(int doy, double latitude)
{
    double dr = 1.0 + 0.0330 * cos(kTwoPiD * doy / kYearDays);
    double delta = 0.4090 * sin(kTwoPiD * doy / kYearDays - 1.3900);
    double arg = -tan(latitude) * tan(delta);
    if (arg < -1.0) arg = -1.0;
    if (arg > 1.0) arg = 1.0;
    double omega = acos(arg);
    return kDaySecs / kPiD / kSpecHeatET * kSolarConst * dr *
           (omega * sin(latitude) * sin(delta) + cos(latitude) * cos(delta) * sin(omega));
}

// FORCES mo_utils LE (in-tree copy pre-proc/mtCLIM/mo_utils.f90 lesserequal_dp)
__device__ __forceinline__ bool le_dp(double a, double b)
{
    return !(((kEps * fabs(b) - fabs(a - b)) < 0.0) && (a > b));
}

// src/mHM/mo_pet.f90:73-116
__device__ double pet_hargreaves(double coeff, double tavg, double tmax, double tmin, double rad)
{
    double delta_temp = tmax - tmin;
    if (le_dp(delta_temp, 0.0) || le_dp(tavg, -kHarSamConst)) return 0.0;
    return coeff * rad * (tavg + kHarSamConst) * sqrt(delta_temp);
}

// src/mHM/mo_pet.f90:149-174 (pet_priestly), with slope_satpressure (:384-399)
// and sat_vap_pressure written as the reference does: exp(2 log(T + c3)) for
// the square, divisions in the same order
__device__ double pet_priestly(double alpha, double rn, double tavg)
{
    const double svp = kTetensC1 * hm_exp(kTetensC2 * tavg / (tavg + kTetensC3));
    const double delta = kSatPressureSlope1 * svp / hm_exp(2.0 * hm_log(tavg + kTetensC3));
    return alpha * delta / (kPsychro + delta) * (rn * kDaySecs / kSpecHeatET);
}

// src/mHM/mo_pet.f90:235-272 (pet_penman) with a_s = a_sh = 1, as the meteo
// handler calls it (mo_meteo_handler.f90:1087-1095); the same operation order
__device__ double pet_penman(double net_rad, double tavg, double act_vap, double ra, double rs)
{
    const double svp = kTetensC1 * hm_exp(kTetensC2 * tavg / (tavg + kTetensC3));
    const double slope = kSatPressureSlope1 * svp / hm_exp(2.0 * hm_log(tavg + kTetensC3));
    return kDaySecs / kSpecHeatET * (slope * net_rad + kRho0 * kCp0 * (svp - act_vap) * 1.0 / ra) /
           (slope + kPsychro * 1.0 / 1.0 * (1.0 + rs / ra));
}

// A thread's scalars live in registers (Surface, Ground); the soil moisture of
// each horizon and two reciprocals per horizon live in shared memory,
// [plane][H][blockDim] (consecutive threads -> consecutive words), so the
// horizon loop stays rolled: fewer registers (more warps per SM) and a smaller
// instruction footprint.
//
// Every division of the step divides by a value that is fixed over the chunk
// (SMs, the stress denominator FC - PW or SMs - PW, sealedThresh, the Jarvis
// threshold) or over a month (interception capacity, pan-evaporation
// coefficient): their fixed-point reciprocals (hm_recip_of) are computed once
// and each division runs hm_div_r -- the same correctly rounded quotient as
// hm_div at about half its integer instructions.  HS_RSMS / HS_RDEN hold the
// reciprocals' bits.
//
// The read-only per-horizon parameters are copied to shared memory too when
// that costs no occupancy -- SMs, FC, PW and beta up to 3 horizons, where 8
// planes of 8 blocks fit the SM -- and are read from the parameter planes in
// global memory (L1/L2-cached, coalesced) otherwise: with 6 horizons they would
// take 48 KB per block and cap the SM at 4 blocks.
//
// HS_FR holds 1 - the step's runoff fractions, which the block evaluates packed
// at the top of each step's soil moisture (with flux outputs, afterwards what
// each horizon passes on); with the parameters in global memory a plane of one
// pointer per thread (each thread's parameter planes) follows the horizon
// planes, so that a thread can read another's SMs and beta.  Then, per thread,
// the water that enters the soil and leaves its last horizon, and the list of
// the threads it is evaluated for.
enum HorizonPlane : int { HS_SM = 0, HS_RSMS, HS_RDEN, HS_FR, HS_PAR0, HS_PLANES_ALL = HS_PAR0 + 4 };
__host__ __device__ constexpr bool hs_params_shared(int HL) { return HL <= 3; }
__host__ __device__ constexpr int hs_planes(int HL) { return hs_params_shared(HL) ? HS_PLANES_ALL : HS_PAR0; }
// dynamic shared memory of a block of B threads
__host__ __device__ constexpr size_t hs_bytes(int HL, int B)
{
    return (size_t)hs_planes(HL) * HL * B * sizeof(double) + (hs_params_shared(HL) ? 0 : (size_t)B * sizeof(void *)) +
           (size_t)B * (sizeof(double) + sizeof(uint16_t));
}

// The running sums of the output variables lie behind the horizon planes where
// 4 blocks with them still fit an SM.
__host__ __device__ constexpr bool flux_sums_shared(int HL, int B, int n_planes)
{
    return hs_bytes(HL, B) % sizeof(double) == 0 && hs_bytes(HL, B) + (size_t)n_planes * B * sizeof(double) <= 56 * 1024;
}

// exp(beta * log(smh / SMs)) lies in [0, 1] for eps < smh <= SMs when SMs is
// finite and beta is finite and > 0 (integer tests on the bits)
__device__ __forceinline__ bool sm_frac_bounded(double sms, double beta)
{
    return hm_abs_bits(hm_d2b(sms)) < 0x7ff0000000000000ULL && hm_d2b(beta) - 1 < 0x7fefffffffffffffULL;
}

// The stress factor of one horizon, mo_soil_moisture.f90:340-365 (Feddes) and
// :415-450 (Jarvis); den = FC - PW or SMs - PW.
__device__ __forceinline__ double stress_factor(bool feddes, double smh, double fc, double pw, double froots,
                                                double den, uint64_t r_den, double jarvis, uint64_t r_jarvis)
{
    double stress;
    if (feddes) {
        const bool wet = hm_ge(smh, fc);
        stress = hm_sel(wet, froots, 0.0);
        // mo_soil_moisture.f90:358
        if (!wet && hm_gt(smh, pw)) stress = hm_div_r(froots * (smh - pw), den, r_den);
    } else {
        // with SMs == PW the quotient can be NaN (0 / 0): IEEE
        // comparisons then leave the stress at 0 as the oracle does
        double th = hm_div_r(smh - pw, den, r_den);
        th = hm_sel(hm_lt_ieee(th, 0.0), 0.0, th);
        th = hm_sel(hm_gt_ieee(th, 1.0), 1.0, th);
        const bool wet = hm_ge_ieee(th, jarvis);
        stress = hm_sel(wet, froots, 0.0);
        if (!wet && hm_lt_ieee(th, jarvis)) stress = froots * hm_div_r(th, jarvis, r_jarvis);
    }
    return stress;
}

// The uptake of one horizon for the operands hm_uptake leaves: the actual
// evapotranspiration and the storage left, in FP64 (mo_soil_moisture.f90:
// 254-286).  Out of line: a block takes it for few lanes, and its instructions
// stay out of the loop.
struct Uptake {
    double aet, smh;
};
__device__ __noinline__ Uptake uptake_general(bool feddes, double aet, double smh, double sms, double fc, double pw,
                                              double froots, uint64_t r_den, double jarvis, uint64_t r_jarvis)
{
    const double stress = stress_factor(feddes, smh, fc, pw, froots, feddes ? fc - pw : sms - pw, r_den, jarvis, r_jarvis);
    aet = aet * stress;
    aet = hm_sel(hm_lt0(aet), 0.0, aet);
    // enough: storage smh - aet, aet kept; else aet = smh - eps and
    // storage eps -- one subtraction serves both cases
    const bool enough = hm_gt(smh, aet);
    const double d = smh - hm_sel(enough, aet, kEps);
    Uptake u;
    u.aet = hm_sel(enough, aet, d);
    u.smh = hm_sel(enough, d, kEps);
    u.smh = hm_sel(hm_lt(u.smh, kEps), kEps, u.smh);
    return u;
}

// The part of a cell's step above the soil -- meteo, canopy, snow and the sealed
// bucket -- which depends on the forcing and on its own states only.  KEEP keeps
// the meteo of a daily forcing row from step to step (it changes with the row,
// the month and day or night, Hargreaves-Samani PET with the day too: a row is
// 24 steps, and above one hour a step several days) at the price of registers.
template <bool LEAN, bool KEEP = false> struct Surface {
    // states
    double interc, snow, seal;
    // parameters (and parameter-only derived values)
    double ddinc, ddmax_s, ddnopre_s, dd_thr, tthresh, sthresh, fasp, harsam, lat_rad;
    uint64_t r_sthresh, r_nd; // reciprocals of chunk-fixed divisors
    bool sealed, sthresh_pos, dd_thr_ok;
    // of the month and LAI entry, and of the day
    int cur_key = -1, cur_doy = -1;
    double imax = 0.0, petlai = 0.0, petsurf = 0.0, evap = 0.0, rad = 0.0;
    uint64_t r_imax = 0, r_evap = 0;
    size_t cur_f = ~(size_t)0;
    int cur_day = -1;
    // of the step
    double temp, prec;
    double pet, aet_can, prec_effect, melt, runoff_sealed, aet_sealed_act;

    __device__ __forceinline__ void load(const CellArgs &a, const double *P, const double *S, double fsealed, int k)
    {
        const int64_t N = a.n_cells;
        auto par = [&](int plane) { return __ldg(P + (size_t)plane * N); };
        const double c2 = a.c2TSTu;
        ddinc = par(P_DDINC);
        ddmax_s = par(P_DDMAX) * c2;     // mo_mhm.f90:463
        ddnopre_s = par(P_DDNOPRE) * c2; // mo_mhm.f90:464
        dd_thr = (ddmax_s - ddnopre_s) / ddinc; // mo_snow_accum_melt.f90:137
        tthresh = par(P_TTHRESH);
        sthresh = par(P_STHRESH);
        fasp = par(P_FASP);
        harsam = par(P_HARSAM);
        lat_rad = (a.proc_pet == 1) ? kDeg2Rad * __ldg(a.latitude + k) : 0.0;
        r_sthresh = hm_recip_of(sthresh);
        r_nd = hm_recip_of(a.nTstepDay);
        interc = S[(size_t)S_INTERC * N];
        snow = S[(size_t)S_SNOW * N] + 0.0; // a -0 ends with the first step's sum or zero
        seal = S[(size_t)S_SEAL * N];
        sealed = fsealed > 0.0;           // frac_sealed > 0
        sthresh_pos = sthresh > kEps;     // water_thresh_sealed > eps
        dd_thr_ok = !hm_isnan_i(dd_thr);  // prec <= NaN is false
    }

    // pet, temp and prec of the step (mo_meteo_handler.f90:915-1285)
    __device__ __forceinline__ void meteo(const CellArgs &a, const StepInfo si, const size_t f, const int k)
    {
        const int64_t N = a.n_cells;
        const int month = si.month;
        double pv = 0.0;
        if (a.proc_pet == 0) {
            pv = fasp * __ldg(a.pet + f);
        } else if (a.proc_pet == -1) {
            pv = petlai * __ldg(a.pet + f);
        } else if constexpr (LEAN) {
        } else if (a.proc_pet == 2) { // Rn = max(L1_netrad, 0), src/meteo/mo_meteo_handler.f90:1080-1085
            const double rn = __ldg(a.netrad + f);
            pv = pet_priestly(petlai, rn > 0.0 ? rn : 0.0, __ldg(a.temp + f));
        } else if (a.proc_pet == 3) { // aeroResist / wind speed, eabs in kPa, :1087-1095
            const double rn = __ldg(a.netrad + f);
            pv = pet_penman(rn > 0.0 ? rn : 0.0, __ldg(a.temp + f), __ldg(a.eabs + f) / 1000.0,
                            petlai / __ldg(a.wind + f), petsurf);
        } else {
            if (si.doy != cur_doy) {
                cur_doy = si.doy;
                rad = extraterr_rad_approx(cur_doy, lat_rad);
            }
            pv = fasp * pet_hargreaves(harsam, __ldg(a.temp + f), __ldg(a.tmax + f), __ldg(a.tmin + f), rad);
        }
        if (a.is_hourly) {
            pet = pv;
            temp = __ldg(a.temp + f);
            prec = __ldg(a.pre + f);
        } else if (a.w_pet) {
            // temporal_disagg_meteo_weights (mo_meteo_temporal_tools.f90:32-50) with
            // L1_*_weights(k, month, hour + 1), mo_meteo_handler.f90:1102-1107, 1183-1189,
            // 1265-1270; temperature corrected by T0 = 273.15 K
            const size_t wi = ((size_t)si.hour * 12 + (size_t)(month - 1)) * N + k;
            pet = (pv + 0.0) * __ldg(a.w_pet + wi) - 0.0;
            temp = (__ldg(a.temp + f) + kT0) * __ldg(a.w_temp + wi) - kT0;
            prec = (__ldg(a.pre + f) + 0.0) * __ldg(a.w_pre + wi) - 0.0;
        } else { // temporal_disagg_*_daynight, mo_meteo_temporal_tools.f90:66-161
            const int mi = month - 1;
            const double nd = a.nTstepDay;
            if (nd > 1.0) {
                const bool isday = (si.dflags & SF_ISDAY) != 0;
                pet = hm_div_r(2.0 * pv * (isday ? a.tab.fday_pet[mi] : a.tab.fnight_pet[mi]), nd, r_nd);
                temp = __ldg(a.temp + f) + (isday ? a.tab.fday_temp[mi] : a.tab.fnight_temp[mi]);
                prec = hm_div_r(2.0 * __ldg(a.pre + f) * (isday ? a.tab.fday_prec[mi] : a.tab.fnight_prec[mi]), nd, r_nd);
            } else {
                pet = pv;
                temp = __ldg(a.temp + f);
                prec = __ldg(a.pre + f);
            }
        }
    }

    // the step `si` of cell k of member m, forcing row `f` (an index); false:
    // the step's LAI entry is out of range (bounds-checked build)
    __device__ __forceinline__ bool step(const CellArgs &a, const double *P, const StepInfo si, const size_t f,
                                         const int m, const int k)
    {
        const int64_t N = a.n_cells;
        bool ok = true;
        // the month (evap_coeff) and the LAI entry (iLAI: the month, or the
        // step's entry of a gridded LAI series) as one key: their parameters
        // are reloaded together when either changes
        const int key = ((int)si.lai << 4) | si.month;
        if (hm_unlikely(key != cur_key)) {
            cur_key = key;
            evap = a.tab.evap[si.month - 1]; // evap_coeff of the calendar month
            r_evap = hm_recip_of(evap);
            if (!a.lai_series) { // iLAI = month: the monthly LAI slots
                imax = __ldg(P + (size_t)(P_MAXINTER + si.month - 1) * N);
                // petLAIcorFactor (proc_pet -1) or PrieTayAlpha (proc_pet 2) of the LAI month
                if (a.proc_pet == -1 || a.proc_pet >= 2) petlai = __ldg(P + (size_t)(P_PETLAI + si.month - 1) * N);
                // surfResist of the LAI month
                if (!LEAN && a.proc_pet == 3) petsurf = __ldg(P + (size_t)(P_PET2 + si.month - 1) * N);
            } else if (bc_ok(BC_LAI_STEP, si.lai - 1, a.n_lai)) { // a gridded LAI series: its entry iLAI
                const size_t NL = (size_t)a.n_lai * N;
                const double *ls =
                    a.lai_series + (size_t)m * lai_groups(a.proc_pet) * NL + (size_t)(si.lai - 1) * N + k;
                imax = __ldg(ls);
                if (a.proc_pet == -1 || a.proc_pet >= 2) petlai = __ldg(ls + NL);
                if (!LEAN && a.proc_pet == 3) petsurf = __ldg(ls + 2 * NL);
            } else {
                ok = false;
            }
            r_imax = hm_recip_of(imax);
        }
        bool fresh = true;
        if constexpr (KEEP) {
            const int day = key << 1 | (si.dflags & SF_ISDAY);
            fresh = a.is_hourly || a.w_pet || f != cur_f || day != cur_day ||
                    (!LEAN && a.proc_pet == 1 && si.doy != cur_doy);
            cur_f = f;
            cur_day = day;
        }
        if (fresh) meteo(a, si, f, k);
        // ---- canopy_interc, mo_canopy_interc.f90:75-133 ----
        // Branches that only pick between values are written as hm_sel (an
        // integer select of the bits): a double select or a merge of doubles
        // after a short if/else is issued on the FP64 pipe, the bottleneck.
        double throughfall;
        {
            const double aux = interc + prec;
            const bool full = hm_ge(aux, imax);
            throughfall = 0.0;
            if (full) throughfall = aux - imax;
            interc = hm_sel(full, imax, aux);
            aet_can = 0.0;
            if (hm_gt(imax, kEps)) aet_can = pet * hm_pow(hm_div_r(interc, imax, r_imax), kTwoThird);
            // a negative storage gives pow() = NaN: these two tests keep IEEE NaN semantics
            aet_can = hm_sel(hm_lt_ieee(aet_can, 0.0), 0.0, aet_can);
            const bool keep = hm_gt_ieee(interc, aet_can);
            const double rest = interc - aet_can;
            aet_can = hm_sel(keep, aet_can, interc);
            interc = hm_sel(keep, rest, 0.0);
        }
        // ---- snow_accum_melt, mo_snow_accum_melt.f90:70-158 ----
        {
            const bool warm = hm_gt(temp, tthresh);
            const double rain = hm_sel(warm, throughfall, 0.0);
            const double snowf = hm_sel(warm, 0.0, throughfall);
            melt = 0.0;
            prec_effect = rain; // 0 + rain
            if (warm) {
                double snow_left = 0.0;
                if (hm_gt0(snow)) { // the degree-day factor only matters here
                    const bool low = dd_thr_ok && hm_le(prec, dd_thr);
                    const double dd = hm_sel(low, ddnopre_s + ddinc * prec, ddmax_s);
                    const double aux = dd * (temp - tthresh);
                    const bool all = hm_gt(aux, snow);
                    melt = hm_sel(all, snow, aux);
                    snow_left = hm_sel(all, 0.0, snow - aux);
                    prec_effect = melt + rain;
                }
                snow = snow_left;
            } else if (hm_d2b(snowf) != 0) {
                snow = snow + snowf;
            }
        }
        return ok;
    }

    // the sealed bucket's step, mo_soil_moisture.f90:190-222
    __device__ __forceinline__ void sealed_step()
    {
        runoff_sealed = 0.0;
        aet_sealed_act = 0.0;
        if (sealed) {
            const double tmp = seal + prec_effect;
            const bool over = hm_gt(tmp, sthresh);
            if (over) runoff_sealed = tmp - sthresh;
            seal = hm_sel(over, sthresh, tmp);
            double aet_sealed = DBL_MAX;
            if (sthresh_pos) {
                aet_sealed = (hm_div_r(pet, evap, r_evap) - aet_can) * hm_div_r(seal, sthresh, r_sthresh);
                aet_sealed = hm_sel(hm_lt0(aet_sealed), 0.0, aet_sealed);
            }
            const bool keep = hm_gt(seal, aet_sealed);
            const double rest = seal - aet_sealed;
            aet_sealed_act = hm_sel(keep, aet_sealed, seal);
            seal = hm_sel(keep, rest, 0.0);
        }
    }
};

// Below the soil: the unsaturated and the saturated zone.
struct Ground {
    double unsat, sat;                                   // states
    double k0s, k1s, k2s, kps, uthresh, karst, alpha1; // c2TSTu / k and parameters
    bool karst_one;
    double fast, slow, base, perc; // of the step

    __device__ __forceinline__ void load(const CellArgs &a, const double *P, const double *S)
    {
        const int64_t N = a.n_cells;
        auto par = [&](int plane) { return __ldg(P + (size_t)plane * N); };
        const double c2 = a.c2TSTu;
        uthresh = par(P_UTHRESH);
        karst = par(P_KARST);
        karst_one = hm_d2b(karst) == 0x3ff0000000000000ULL;
        alpha1 = 1.0 + par(P_ALPHA); // mo_runoff.f90:139
        k1s = c2 / par(P_K1);        // mo_mhm.f90:484
        kps = c2 / par(P_KP);
        k0s = c2 / par(P_K0);
        k2s = c2 / par(P_K2);        // mo_mhm.f90:488
        unsat = S[(size_t)S_UNSAT * N];
        sat = S[(size_t)S_SAT * N];
    }

    __device__ __forceinline__ void step(const double infil_last)
    {
        // ---- runoff_unsat_zone, mo_runoff.f90:74-154 ----
        fast = slow = 0.0;
        unsat = unsat + infil_last;
        if (hm_unlikely(hm_gt(unsat, uthresh))) {
            fast = hm_min_sel(k0s * (unsat - uthresh), unsat - kEps);
            unsat = unsat - fast;
        }
        if (hm_gt(unsat, kEps)) {
            slow = k1s * hm_pow(unsat, alpha1);
            // not above a quarter of the store, of 2^-50 or more: below unsat - eps
            const uint32_t us = hm_hi(hm_d2b(unsat));
            if (hm_unlikely(hm_hi(hm_d2b(slow)) + 0x00200000u > us || us < 0x3cd00000u))
                slow = hm_min_sel(slow, unsat - kEps);
            unsat = unsat - slow;
        }
        perc = kps * unsat;
        // if the store cannot supply kp * unsat, perc = unsat: both branches of
        // the reference add perc * karstLoss to the saturated store
        const bool rest = hm_gt(unsat, perc);
        perc = hm_sel(rest, perc, unsat);
        double recharge = perc;
        if (hm_unlikely(!karst_one)) recharge = perc * karst; // perc * 1
        sat = sat + recharge;
        unsat = hm_sel(rest, unsat - perc, 0.0);
        // ---- runoff_sat_zone, mo_runoff.f90:191-212 ----
        {
            const bool pos = hm_gt0(sat);
            const double b0 = k2s * sat;
            base = hm_sel(pos, b0, 0.0);
            sat = hm_sel(pos, sat - b0, 0.0);
        }
    }

    // The unsealed share as total() takes it: NaN for an infinite sealed fraction,
    // whose product with a sealed runoff of +0, left out there, is NaN, as is that
    // of a positive one less the infinite unsealed part.
    static __device__ __forceinline__ double share(double fsealed)
    {
        const bool finite = (hm_hi(hm_d2b(fsealed)) & 0x7ff00000u) != 0x7ff00000u;
        return hm_sel(finite, 1.0 - fsealed, hm_b2d(0x7ff8000000000000ULL));
    }

    // L1_total_runoff, mo_runoff.f90:248-274; `fnotsealed` from share()
    __device__ __forceinline__ double total(double fnotsealed, double runoff_sealed, double fsealed) const
    {
        double q = base + slow;
        if (hm_d2b(fast) != 0) q = q + fast;
        q = q * fnotsealed;
        if (hm_d2b(runoff_sealed) != 0) q = q + runoff_sealed * fsealed;
        return q;
    }
};

// What the aggregated outputs take from a step.
struct OutStep {
    double interc, snow, seal, pet, aet_can, aet_sealed, runoff_sealed, prec_effect, melt; // surface
    double unsat, sat, fast, slow, base, perc, q_total, aet_soil;
};

// mHM_updateDataset, src/mHM/mo_write_fluxes_states.f90:283-438, but for the
// horizons' infiltration and aET: `add` adds to an output variable's plane; sm
// and sat_h give a horizon's soil moisture and its saturation; `osat` their sum
// over the column unless this step has its own weights (ow).
template <class Add, class Sm, class Sat>
__device__ __forceinline__ void out_add(const OutArgs &o, int H, const OutStep &v, bool ow, double ofs, double ofns,
                                        double osat, uint64_t r_osat, Add add, Sm sm, Sat sat_h)
{
    const int8_t *pl = o.plane;
    if (pl[OF_INTERC] >= 0) add(pl[OF_INTERC], v.interc);
    if (pl[OF_SNOW] >= 0) add(pl[OF_SNOW], v.snow);
    if (pl[OF_SWC] >= 0)
        for (int h = 0; h < H; ++h) add(pl[OF_SWC] + h, sm(h));
    if (pl[OF_SM] >= 0 || pl[OF_SM_ALL] >= 0) {
        double ssm = 0.0, ssat = ow ? 0.0 : osat;
        for (int h = 0; h < H; ++h) {
            if (pl[OF_SM] >= 0) add(pl[OF_SM] + h, hm_div(sm(h), sat_h(h)));
            ssm = ssm + sm(h);
            if (ow) ssat = ssat + sat_h(h);
        }
        if (pl[OF_SM_ALL] >= 0) add(pl[OF_SM_ALL], hm_div_r(ssm, ssat, ow ? hm_recip_of(ssat) : r_osat));
    }
    if (pl[OF_SEAL] >= 0) add(pl[OF_SEAL], v.seal);
    if (pl[OF_UNSAT] >= 0) add(pl[OF_UNSAT], v.unsat);
    if (pl[OF_SAT] >= 0) add(pl[OF_SAT], v.sat);
    if (pl[OF_PET] >= 0) add(pl[OF_PET], v.pet);
    if (pl[OF_AET] >= 0) add(pl[OF_AET], v.aet_soil * ofns + v.aet_can + v.aet_sealed * ofs);
    if (pl[OF_Q] >= 0) add(pl[OF_Q], v.q_total);
    if (pl[OF_QD] >= 0) add(pl[OF_QD], v.runoff_sealed * ofs);
    if (pl[OF_QIF] >= 0) add(pl[OF_QIF], v.fast * ofns);
    if (pl[OF_QIS] >= 0) add(pl[OF_QIS], v.slow * ofns);
    if (pl[OF_QB] >= 0) add(pl[OF_QB], v.base * ofns);
    if (pl[OF_RECHARGE] >= 0) add(pl[OF_RECHARGE], v.perc * ofns);
    if (pl[OF_PRE_EFFECT] >= 0) add(pl[OF_PRE_EFFECT], v.prec_effect);
    if (pl[OF_QSM] >= 0) add(pl[OF_QSM], v.melt);
}

// The step is counted; where an output interval ends with it, the sums or means
// go out and the sums start anew (writeVariableTimestep,
// src/common/mo_nc_output.f90:158-175).
__device__ __forceinline__ void out_close(const OutArgs &o, double *acc, size_t stride, size_t out_stride, size_t at,
                                          int64_t tt, int dflags, int &cnt, int &slot)
{
    ++cnt; // OutputVariable%counter
    if (!out_writeout(o.interval, tt - o.warm_steps, tt, o.n_tt, dflags)) return;
    double *dst = o.out + (size_t)slot * o.n_planes * out_stride + at;
    const uint64_t r_cnt = hm_recip_of((double)cnt);
    for (int v = 0; v < o.n_planes; ++v) {
        double *q = acc + (size_t)v * stride;
        const double x = *q;
        if (slot < o.max_slots)
            dst[(size_t)v * out_stride] = ((o.avg_mask >> v) & 1) ? hm_div_r(x, (double)cnt, r_cnt) : x;
        *q = 0.0;
    }
    ++slot;
    cnt = 0;
}

// SMs of the current device: the launch rules count in waves of blocks.  152 (a
// GB300's), should the runtime not say.
__host__ inline int device_sms()
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
        return 152;
    return sms;
}

__host__ inline bool cell_chain_lean(const CellArgs &a)
{
    return (a.proc_pet == 0 || a.proc_pet == -1) && (a.proc_sm == 1 || a.proc_sm == 4);
}

// LEAN: compiled for PET input (cases -1, 0) and the Feddes stress (soil-moisture
// cases 1, 4) only -- the configurations of the throughput workloads -- so that
// the Hargreaves / Priestley-Taylor / Penman-Monteith and Jarvis code is not in
// the instruction stream and the register allocation.
//
// cell_chain_item advances cell k of member m of the launch described by `a`;
// all B threads of the block call it, those without an item with active =
// false (and any cell and member in range).  HL sizes the shared-memory horizon
// planes; DYN takes the horizon count from a.n_horizons (<= HL) at run time, so
// that one launch can serve contexts with different horizon counts (the fused
// multi-context launch); otherwise it is HL.
template <int HL, bool FLUX, bool LEAN, bool DYN, int B>
__device__ __forceinline__ void cell_chain_item(const CellArgs &a, const int m, const int k, bool active)
{
    __shared__ int s_wet[3]; // threads in the list, by step modulo 3
    const int H = DYN ? a.n_horizons : HL;
    const int64_t N = a.n_cells;
    const StepInfo *steps = a.steps;
    bool reset_sm = a.reset_sm != 0;
    if (a.member_step0) {
        const int32_t b = a.member_step0[m];
        if (b < 0) { // idle member slot: no state update, zero runoff
            if (active)
                for (int t = 0; t < a.n_steps; ++t) a.tro[(size_t)t * a.n_members * N + (size_t)m * N + k] = 0.0;
            active = false;
        } else if (!bc_ok(BC_STEP_ROW, (long long)b + a.step_shift + a.n_steps - 1, a.n_step_rows)) {
            active = false;
        } else {
            steps += b + a.step_shift;
        }
        reset_sm = a.reset_ok && (b + a.step_shift == 0);
    }
    const int np = n_param_planes(H);
    const int ns = n_state_planes(H);
    const double *P = a.params + (size_t)m * np * N + k;
    double *S = a.states + (size_t)m * ns * N + k;
    auto par = [&](int plane) { return __ldg(P + (size_t)plane * N); };

    extern __shared__ double hsm[];
    const int tb = threadIdx.x;
    auto hs = [&](int plane, int h) -> double & { return hsm[(plane * HL + h) * B + tb]; };
    // the per-horizon parameters, groups 0..4 = fRoots, SMs, FC, PW, beta
    auto hp = [&](int g, int h) -> double {
        if (hs_params_shared(HL) && g > 0) return hs(HS_PAR0 + g - 1, h);
        return __ldg(P + (size_t)(P_HORIZON + g * H + h) * N);
    };
    const double **hptr = reinterpret_cast<const double **>(hsm + (size_t)hs_planes(HL) * HL * B);
    if constexpr (!hs_params_shared(HL)) hptr[tb] = P;
    double *soil_in = hsm + (size_t)hs_planes(HL) * HL * B + (hs_params_shared(HL) ? 0 : B);
    uint16_t *wet_list = reinterpret_cast<uint16_t *>(soil_in + B);
    if (tb < 3) s_wet[tb] = 0;
    __syncthreads();
    const bool feddes = LEAN || (a.proc_sm == 1 || a.proc_sm == 4);
    const double fsealed = par(P_FSEALED), fnotsealed = 1.0 - fsealed, share = Ground::share(fsealed);
    const double jarvis = LEAN ? 0.0 : par(P_JARVIS);
    const uint64_t r_jarvis = LEAN ? 0 : hm_recip_of(jarvis);
    Surface<LEAN> sf;
    Ground gd;
    sf.load(a, P, S, fsealed, k);
    gd.load(a, P, S);
    bool frac_bounded = true; // every horizon's runoff fraction is in [0, 1]
    uint32_t den_exp = 0;     // by horizon: the exponent of FC - PW less kDenExp, or 15: no hm_uptake
#pragma unroll 1
    for (int h = 0; h < H; ++h) {
        if constexpr (hs_params_shared(HL)) {
            for (int g = 1; g < 5; ++g) hs(HS_PAR0 + g - 1, h) = __ldg(P + (size_t)(P_HORIZON + g * H + h) * N);
        }
        const double sms = hp(1, h), fc = hp(2, h), pw = hp(3, h);
        hs(HS_RSMS, h) = hm_b2d(hm_recip_of(sms));
        hs(HS_RDEN, h) = hm_b2d(hm_recip_of(feddes ? fc - pw : sms - pw)); // mo_soil_moisture.f90:358, :435
        hs(HS_SM, h) = reset_sm ? 0.5 * fc : S[(size_t)(S_SM + h) * N];
        frac_bounded = frac_bounded && sm_frac_bounded(sms, hp(4, h));
        const uint32_t de = hm_hi(hm_d2b(fc - pw)) >> 20; // with the sign bit: at least 2048 if negative
        const bool up = feddes && hm_uptake_var(hp(0, h)) && hm_uptake_var(fc) && hm_uptake_var(pw) && de - kDenExp < 15u;
        den_exp |= (up ? de - kDenExp : 15u) << (4 * h);
    }
    const size_t out_stride = (size_t)a.n_members * N;
    double *tro = a.tro + (size_t)m * N + k;
    // aggregated flux/state outputs (flux variant): running sums, a plane per
    // output variable, in the block's shared memory for the launch.  A step adds
    // to every plane, one after another; in device memory each of these read,
    // add, write was a trip to the L2 (40,000 cells, 3 horizons, 14
    // planes, 240 steps: 3.91 ms, 3.62 with the sums on the chip).
    const OutArgs &o = a.out;
    double *oacc = nullptr, *const oacc_g = o.acc + (size_t)m * N + k;
    size_t ostr = out_stride;
    int ocnt = 0, oslot = 0;
    int64_t ott_w = -1;
    double osat = 0.0; // saturated soil moisture of the column, and its reciprocal
    uint64_t r_osat = 0;
    if constexpr (FLUX) {
        if (o.n_planes > 0 && active) {
            oacc = oacc_g;
            if (flux_sums_shared(HL, B, o.n_planes)) {
                oacc = hsm + hs_bytes(HL, B) / sizeof(double) + tb;
                ostr = B;
                for (int v = 0; v < o.n_planes; ++v) oacc[v * ostr] = oacc_g[v * out_stride];
            }
            ocnt = o.cnt0;
            oslot = o.slot0;
            if (o.tt_w) ott_w = o.tt_w[m];
            for (int h = 0; h < H; ++h) osat = osat + hp(1, h);
            r_osat = hm_recip_of(osat);
        }
    }
    // non-finite detection, integer operations only: a double is NaN or Inf
    // iff its sign-cleared bits are >= 0x7ff0...0, i.e. iff adding 2^52 to
    // them carries into bit 63; the OR over the steps keeps any such carry
    constexpr uint64_t kExpOne = 0x0010000000000000ull;
    uint64_t nonfin = 0;
    auto oadd = [&](int plane, double x) {
        double *q = oacc + (size_t)plane * ostr;
        *q = *q + x; // OutputVariable%data = data + value, src/common/mo_nc_output.f90:140-149
    };

    const bool store = active; // a failed index test ends the item's steps, not its states
    for (int t = 0, wet_slot = 0; t < a.n_steps; ++t) {
        StepInfo si{};
        // output weights: write_output runs after the calendar has advanced, so
        // it reads fSealed / soilMoistSat of the NEXT step's land-cover scene
        // (src/mHM/mo_mhm_interface_run.f90:621-629, 698-727)
        bool oon = false, ow = false;
        double ofs = 0.0, ofns = 0.0;
        bool need_frac = false;
        if (active) {
            si = steps[t];
            const int32_t row = a.member_step0 ? a.step_shift + t : si.row - a.row_base;
            active = bc_ok(BC_FORCING_ROW, row, a.n_forc_rows) && sf.step(a, P, si, (size_t)row * N + k, m, k);
        }
        if (active) {
            if constexpr (FLUX) {
                const int64_t tt = o.tt_base + t;
                oon = oacc != nullptr && tt > o.warm_steps;
                ow = oon && tt == ott_w;
                ofs = fsealed;
                ofns = fnotsealed; // run_cfg%L1_fNotSealed = 1 - L1_fSealed (:239)
                if (ow) {
                    ofs = o.w_fsealed[(size_t)m * N + k];
                    ofns = 1.0 - ofs;
                }
            }
            need_frac = hm_d2b(sf.prec_effect) != 0 || !frac_bounded;
        }
        // ---- the water's way through the horizons, mo_soil_moisture.f90:
        // 230-252 ----
        // A cell whose effective precipitation is +0 -- and whose runoff fractions
        // exp(beta log(SM / SMs)) are known to lie in [0, 1] -- needs none of
        // this: every horizon's input is then +0, pin * (1 - frac) is +0 for every
        // such fraction, and storage and input stay as they are.  The cells that
        // do are few in most hours and scattered over the warps, so the block
        // lists them and evaluates them packed: first all their fractions, a
        // thread per (cell, horizon) -- each depends on its horizon's
        // start-of-step soil moisture and on parameters only -- then the
        // horizons' chain, a thread per cell.  The same functions of the same
        // operands give the same bits on any thread.
        {
            const unsigned nm = __ballot_sync(~0u, need_frac);
            if (tb == 0) s_wet[wet_slot == 2 ? 0 : wet_slot + 1] = 0; // read last two barriers ago
            if (nm != 0) {
                int base = 0;
                if ((tb & 31) == 0) base = atomicAdd(&s_wet[wet_slot], __popc(nm));
                base = __shfl_sync(~0u, base, 0);
                if (need_frac) {
                    unsigned lt;
                    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
                    wet_list[base + __popc(nm & lt)] = (uint16_t)tb;
                    soil_in[tb] = sf.prec_effect;
                }
            }
            __syncthreads(); // the list, and the soil moisture of the last step
            const int n_wet = s_wet[wet_slot];
            wet_slot = wet_slot == 2 ? 0 : wet_slot + 1;
            if (n_wet > 0) {
                const int n_tasks = n_wet * H;
#pragma unroll 1
                for (int i = tb; i < n_tasks; i += B) {
                    const int h = (int)__fdividef((float)i + 0.5f, (float)n_wet); // i / n_wet
                    const int ow_ = wet_list[i - h * n_wet];                       // the thread the pair belongs to
                    const double smh = hsm[(HS_SM * HL + h) * B + ow_];
                    double sms, beta;
                    if constexpr (hs_params_shared(HL)) {
                        sms = hsm[(HS_PAR0 * HL + h) * B + ow_];
                        beta = hsm[((HS_PAR0 + 3) * HL + h) * B + ow_];
                    } else {
                        const double *Po = hptr[ow_];
                        sms = __ldg(Po + (size_t)(P_HORIZON + H + h) * N);
                        beta = __ldg(Po + (size_t)(P_HORIZON + 4 * H + h) * N);
                    }
                    double fr = 0.0;
                    if (hm_gt(smh, kEps) && !hm_gt(smh, sms))
                        fr = hm_exp(beta * hm_log(hm_div_r(smh, sms, hm_d2b(hsm[(HS_RSMS * HL + h) * B + ow_]))));
                    hsm[(HS_FR * HL + h) * B + ow_] = 1.0 - fr;
                }
                __syncthreads(); // the fractions
                // another warp each step, so that the SM's schedulers take turns
                const int wi = (tb + 32 * t) & (B - 1);
                if (wi < n_wet) {
                    const int ow_ = wet_list[wi];
                    const double *Po = nullptr;
                    if constexpr (!hs_params_shared(HL)) Po = hptr[ow_];
                    double infil = soil_in[ow_]; // prec_effec_soil of horizon 1
#pragma unroll 1
                    for (int h = 0; h < H; ++h) {
                        double sms;
                        if constexpr (hs_params_shared(HL)) sms = hsm[(HS_PAR0 * HL + h) * B + ow_];
                        else sms = __ldg(Po + (size_t)(P_HORIZON + H + h) * N);
                        double &sm = hsm[(HS_SM * HL + h) * B + ow_];
                        const double smh = sm;
                        if (!hm_gt(smh, sms)) { // else the horizon passes its input on
                            // frac_runoff = 0 when smh <= eps
                            const double tmp = infil * hsm[(HS_FR * HL + h) * B + ow_];
                            const double filled = smh + tmp;
                            const bool over = hm_gt(filled, sms);
                            // infil + (smh - sms) or infil - tmp, as one addition:
                            // infil - tmp is infil + (-tmp) exactly
                            double add = hm_neg(tmp);
                            if (hm_unlikely(over)) add = smh - sms;
                            infil = infil + add;
                            sm = hm_sel(over, sms, filled);
                        }
                        if constexpr (FLUX) hsm[(HS_FR * HL + h) * B + ow_] = infil;
                    }
                    soil_in[ow_] = infil;
                }
            }
            if (active) sf.sealed_step(); // the threads without a chain have it behind them when the chains end
            if (n_wet > 0) __syncthreads(); // what the horizons hold and pass on
        }
        if (!active) continue;
        // ---- soil_moisture, mo_soil_moisture.f90:176-286 ----
        const double infil_last = need_frac ? soil_in[tb] : 0.0;
        double aet_soil = 0.0; // for the optional flux outputs
        {
            double aet_above = 0.0; // masked running sum of positive aet above
            const double demand = sf.pet - sf.aet_can;
            // a horizon's parameters are read while the one above is worked on (but
            // for the fused launch, which has no registers left for it)
            constexpr bool ahead = !DYN;
            double nx_froots = 0.0, nx_fc = 0.0, nx_pw = 0.0;
            if (ahead) nx_froots = hp(0, 0), nx_fc = hp(2, 0), nx_pw = hp(3, 0);
#pragma unroll 1
            for (int h = 0; h < H; ++h) {
                double smh = hs(HS_SM, h);
                // demand minus the positive aet above (none above the first)
                double aet = demand;
                if (h > 0) aet = aet - aet_above;
                const double froots = ahead ? nx_froots : hp(0, h);
                const double fc = ahead ? nx_fc : hp(2, h), pw = ahead ? nx_pw : hp(3, h);
                if (ahead && h + 1 < H) nx_froots = hp(0, h + 1), nx_fc = hp(2, h + 1), nx_pw = hp(3, h + 1);
                const uint32_t de = (den_exp >> (4 * h)) & 15u;
                const uint64_t sb = hm_d2b(smh), ab = hm_d2b(aet);
                bool todo = true;
                if (de < 15u && hm_hi(sb) - 0x3cd00000u < 0x4c700000u - 0x3cd00000u) { // SM of 2^-50 .. 2^200 mm
                    if (ab == 0 || hm_hi(ab) - 0x80000000u < 0x7ff00000u || sb <= hm_d2b(pw)) {
                        // no demand left, or no water above the wilting point: none taken
                        if (hm_hi(ab) < 0x7ff00000u || hm_hi(ab) - 0x80000000u < 0x7ff00000u) {
                            aet = 0.0;
                            todo = false;
                        }
                    } else if (hm_uptake_var(aet)) {
                        // what is left is at least half of SM: above eps
                        todo = !hm_uptake(smh, pw, froots, aet, sb >= hm_d2b(fc), hm_d2b(hs(HS_RDEN, h)),
                                          (int)(de + kDenExp), &aet, &smh);
                    }
                }
                if (hm_unlikely(todo)) {
                    const Uptake u = uptake_general(feddes, aet, smh, hp(1, h), fc, pw, froots, hm_d2b(hs(HS_RDEN, h)),
                                                    jarvis, r_jarvis);
                    aet = u.aet;
                    smh = u.smh;
                }
                hs(HS_SM, h) = smh;
                if (h == 0) {
                    aet_above = hm_sel(hm_gt0(aet), aet, 0.0);
                } else if (h + 1 < H) { // nothing below reads the last horizon's
                    aet_above = hm_sel(hm_gt0(aet), aet_above + aet, aet_above);
                }
                if constexpr (FLUX) {
                    aet_soil = aet_soil + aet;
                    if (oon) { // soil_infil_L<h>, aET_L<h> (mo_write_fluxes_states.f90:414-426)
                        const double infil = need_frac ? hs(HS_FR, h) : 0.0;
                        if (o.plane[OF_INFIL] >= 0) oadd(o.plane[OF_INFIL] + h, infil * ofns);
                        if (o.plane[OF_AET_L] >= 0) oadd(o.plane[OF_AET_L] + h, aet * ofns);
                    }
                }
            }
        }
        gd.step(infil_last);
        if constexpr (FLUX) {
            if (a.flux_aet) {
                const size_t fo = (size_t)t * out_stride + (size_t)m * N + k;
                a.flux_aet[fo] = sf.aet_can + fsealed * sf.aet_sealed_act + fnotsealed * aet_soil;
                a.flux_loss[fo] = fnotsealed * (gd.perc - gd.perc * gd.karst);
            }
        }
        const double q_total = gd.total(share, sf.runoff_sealed, fsealed);
        tro[(size_t)t * out_stride] = q_total;
        nonfin |= hm_abs_bits(hm_d2b(q_total)) + kExpOne;
        if constexpr (FLUX) {
            if (oon) {
                const OutStep v{sf.interc, sf.snow, sf.seal, sf.pet, sf.aet_can, sf.aet_sealed_act, sf.runoff_sealed,
                                sf.prec_effect, sf.melt, gd.unsat, gd.sat, gd.fast, gd.slow, gd.base, gd.perc, q_total,
                                aet_soil};
                out_add(
                    o, H, v, ow, ofs, ofns, osat, r_osat, oadd, [&](int h) { return hs(HS_SM, h); },
                    [&](int h) { return ow ? o.w_sms[((size_t)m * H + h) * N + k] : hp(1, h); });
                out_close(o, oacc, ostr, out_stride, (size_t)m * N + k, o.tt_base + t, si.dflags, ocnt, oslot);
            }
        }
    }

    if (!store) return;
    if constexpr (FLUX) {
        if (oacc && oacc != oacc_g)
            for (int v = 0; v < o.n_planes; ++v) oacc_g[v * out_stride] = oacc[v * ostr];
    }
    S[(size_t)S_INTERC * N] = sf.interc;
    S[(size_t)S_SNOW * N] = sf.snow;
    S[(size_t)S_SEAL * N] = sf.seal;
    S[(size_t)S_UNSAT * N] = gd.unsat;
    S[(size_t)S_SAT * N] = gd.sat;
    auto chk = [&](double x) { nonfin |= hm_abs_bits(hm_d2b(x)) + kExpOne; };
    chk(sf.interc);
    chk(sf.snow);
    chk(sf.seal);
    chk(gd.unsat);
    chk(gd.sat);
#pragma unroll 1
    for (int h = 0; h < H; ++h) {
        const double smh = hs(HS_SM, h);
        S[(size_t)(S_SM + h) * N] = smh;
        chk(smh);
    }
    if (a.nonfinite && (nonfin >> 63)) atomicOr(a.nonfinite + m, 1);
}

// Work items of a launch, by 128 threads of a block: one member's 128
// consecutive cells, or -- when the members come in groups of 4 -- 32
// consecutive cells of 4 members (one member per warp, so a warp still walks 32
// neighbouring cells of one parameter set).  The blocks of one cell tile are
// consecutive in launch order and start together, so the forcing rows every
// member reads come from L1/L2 after the first member group instead of from
// DRAM once per member.
__host__ __device__ constexpr bool member_tiles(int64_t n_members) { return n_members > 1 && n_members % 4 == 0; }

// Blocks of 256 threads for up to 3 horizons when they fill the GPU several
// times over: the block's barriers keep two warps of each scheduler at the same
// instructions, which are then fetched once -- with few horizons a step is
// mostly straight-line code and waits for instructions (256 members of 40,000
// cells, 96 steps: 144 ms with 128 threads, 130 with 256, 131 with 512).  With
// 6 horizons the horizon loop is most of the step, and smaller blocks wait less
// at the barriers (1e6 cells, 96 steps: 16.5 / 17.1 / 18.0 ms).
inline int64_t wide_items(int sms) { return (int64_t)sms * 8 * 128 * 4; }
constexpr bool wide_blocks(int H, int MINB, bool FLUX) { return H <= 3 && MINB >= 6 && !FLUX; }

template <int H, int MINB, bool FLUX, bool LEAN, int B>
__global__ void __launch_bounds__(B, MINB * 128 / B) cell_chain_kernel(const CellArgs a)
{
    const int64_t N = a.n_cells;
    int m, k;
    bool active;
    if (member_tiles(a.n_members)) {
        const int64_t n_groups = a.n_members / 4;
        const int64_t tile = blockIdx.x / n_groups;
        m = (int)(blockIdx.x - tile * n_groups) * 4 + (int)((threadIdx.x >> 5) & 3);
        const int64_t kk = tile * (B / 4) + (threadIdx.x >> 7) * 32 + (threadIdx.x & 31);
        active = kk < N;
        k = active ? (int)kk : 0;
    } else {
        const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
        active = gid < N * a.n_members;
        m = active ? (int)(gid / N) : 0;
        k = active ? (int)(gid - (int64_t)m * N) : 0;
    }
    cell_chain_item<H, FLUX, LEAN, false, B>(a, m, k, active);
}

// The cell chain of several contexts in one persistent launch: a work queue
// of tiles (128 consecutive work items of one context), taken in queue order
// by the resident blocks with one atomic increment per tile.  Each block
// copies the tile's context description into shared memory and runs the same
// per-item code as cell_chain_kernel, so every item's arithmetic -- and
// result -- is that of the context's own launch.  No block waits on another:
// a block returns when the queue is empty.
template <int HL, bool LEAN, int MINB>
__global__ void __launch_bounds__(128, MINB) cell_chain_fused_kernel(const FusedCellArgs f)
{
    __shared__ CellArgs sa;
    __shared__ int32_t tile;
    for (;;) {
        if (threadIdx.x == 0) tile = atomicAdd(f.queue, 1);
        __syncthreads();
        const int32_t t = tile;
        if (t >= f.n_tiles) return;
        const uint32_t *src = reinterpret_cast<const uint32_t *>(f.args + __ldg(f.tile_ctx + t));
        uint32_t *dst = reinterpret_cast<uint32_t *>(&sa);
        for (int w = threadIdx.x; w < (int)(sizeof(CellArgs) / 4); w += blockDim.x) dst[w] = __ldg(src + w);
        __syncthreads();
        const int64_t gid = __ldg(f.tile_item0 + t) + threadIdx.x;
        const int64_t N = sa.n_cells;
        const bool active = gid < N * sa.n_members;
        const int m = active ? (int)(gid / N) : 0;
        cell_chain_item<HL, false, LEAN, true, 128>(sa, m, active ? (int)(gid - (int64_t)m * N) : 0, active);
        __syncthreads(); // the next tile may overwrite sa and the horizon planes
    }
}

// Launch with H as a template parameter (shared-memory size, loop bounds);
// MINB = resident blocks per SM the register allocation is sized for.
template <int H, int MINB, bool FLUX, bool LEAN, int B>
cudaError_t launch_cell_chain_b(const CellArgs &a, cudaStream_t s)
{
    const int64_t n = (int64_t)a.n_cells * a.n_members;
    const unsigned grid = member_tiles(a.n_members)
                              ? (unsigned)(((int64_t)a.n_cells + B / 4 - 1) / (B / 4) * (a.n_members / 4))
                              : (unsigned)((n + B - 1) / B);
    size_t smem = hs_bytes(H, B);
    if (FLUX && a.out.n_planes > 0 && flux_sums_shared(H, B, a.out.n_planes))
        smem += (size_t)a.out.n_planes * B * sizeof(double);
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(cell_chain_kernel<H, MINB, FLUX, LEAN, B>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    cell_chain_kernel<H, MINB, FLUX, LEAN, B><<<grid, B, smem, s>>>(a);
    return cudaGetLastError();
}

template <int MINB, bool FLUX, bool LEAN>
cudaError_t launch_cell_chain_h(const CellArgs &a, int H, cudaStream_t s)
{
    const bool wide = wide_blocks(H, MINB, FLUX) && (int64_t)a.n_cells * a.n_members >= wide_items(device_sms());
    switch (H) {
#define MHM_CASE(HH)                                                                                               \
    case HH:                                                                                                       \
        if constexpr (wide_blocks(HH, MINB, FLUX)) {                                                               \
            if (wide) return launch_cell_chain_b<HH, MINB, FLUX, LEAN, 256>(a, s);                                 \
        }                                                                                                          \
        return launch_cell_chain_b<HH, MINB, FLUX, LEAN, 128>(a, s);
        MHM_CASE(1) MHM_CASE(2) MHM_CASE(3) MHM_CASE(4) MHM_CASE(5) MHM_CASE(6) MHM_CASE(7) MHM_CASE(8)
#undef MHM_CASE
    default:
        return cudaErrorInvalidValue;
    }
}

template <int MINB, bool FLUX = false>
cudaError_t launch_cell_chain_variant(const CellArgs &a, int H, cudaStream_t s)
{
    if constexpr (!FLUX) {
        if (cell_chain_lean(a)) return launch_cell_chain_h<MINB, false, true>(a, H, s);
    }
    return launch_cell_chain_h<MINB, FLUX, false>(a, H, s);
}

} // namespace
} // namespace mhm
