// mpr.cu -- the multiscale parameter regionalisation (mpr(),
// src/MPR/mo_multi_param_reg.f90:67-654) on the device, per member.
//
// Everything the reference evaluates per L0 cell from the soil database is a
// function of the cell's (soil type, land cover) pair alone: the transfer
// functions, the depth-weighted horizon properties, the root fractions and
// the Ks variabilities.  So the first kernel evaluates them once per pair and
// member into a small table (tens of rows instead of millions of L0 cells);
// the second kernel gives every L1 cell a lane in each of H + 4 warps that
// walk its L0 sub-cells in the reference's column-major block order and forms the
// arithmetic and harmonic means from table rows and the few per-cell inputs
// (slope rank, aspect, LAI, geology), writing the member's effective
// parameters in place.  The per-cell values are the same IEEE operations on
// the same operands as the reference's per-cell loop, and every block sum
// keeps the reference's order, so results are bit-identical.
#include <cfloat>
#include <cmath>

#include "hmath.h"
#include "bounds.cuh"
#include "fp64i.h"
#include "mhm_kernels.cuh"
#include "mpr_host.h"

namespace mhm {

namespace {

// src/MPR/mo_mpr_constants.f90:34-62
constexpr double kBulkDensOrgMatter = 0.224, kFieldCapC1 = -0.60, kFieldCapC2 = 2.0, kVGSandThresh = 66.5;
__device__ constexpr double kVGN[18] = {1.392, 0.418, -0.024, 1.212, -0.704, -0.648, 0.023, 0.044, 3.168,
                             -2.562, 7.0E-9, 4.004, 3.750, -0.016, -4.197, 0.013, 0.076, 0.276};
constexpr double kKsC = 10.0, kPwpC = 1.0, kPwpMatPot = 15000.0;

// hydro_cond, src/MPR/mo_mpr_soilmoist.f90:736-772
__device__ double hydro_cond(const double *p, double sand, double clay)
{
    const double x = p[0] + p[1] * sand - p[2] * clay;
    double ks = p[3] * hm_exp(x * hm_log(kKsC));
    return (ks < 1.10) ? 1.10 : ks;
}

// Genuchten, :626-698
__device__ void genuchten(const double *p, double sand, double clay, double db, double &ths, double &n,
                          double &alpha)
{
    double x;
    if (sand < kVGSandThresh) {
        ths = p[0] + p[1] * clay + p[2] * db;
        n = kVGN[0] - kVGN[1] * hm_pow(sand, kVGN[2]) + kVGN[3] * hm_pow(clay, kVGN[4]);
        x = kVGN[5] + kVGN[6] * sand + kVGN[7] * clay - kVGN[8] * db;
    } else {
        ths = p[3] + p[4] * clay + p[5] * db;
        n = kVGN[9] + kVGN[10] * hm_pow(sand, kVGN[11]) + kVGN[12] * hm_pow(clay, kVGN[13]);
        x = kVGN[14] + kVGN[15] * sand + kVGN[16] * clay - kVGN[17] * db;
    }
    alpha = hm_exp(x);
    if (ths < 0.01) ths = 0.01;
    if (ths > 1.0) ths = 1.0;
    if (n < 1.01000) n = 1.01000;
    if (alpha < 0.00001) alpha = 0.00001;
}

// field_cap, :560-584
__device__ double field_cap(double ks, double ths, double n)
{
    const double x = (kFieldCapC1) * (kFieldCapC2 + hm_log10(ks));
    return ths * hm_exp(x * hm_log(n));
}

// PWP, :489-520
__device__ double pwp(double n, double alpha, double ths)
{
    const double m = kPwpC - (kPwpC / n);
    double x = kPwpC + hm_exp(n * hm_log(alpha * kPwpMatPot));
    x = hm_exp(m * hm_log(x));
    if (x < 1.0) x = 1.0;
    return ths / x;
}

// One table row: soil type s, land cover l (0 forest, 1 sealed, 2 pervious).
// mpr_sm (src/MPR/mo_mpr_soilmoist.f90:264-392) for the soil's horizons and
// the pair's L0 quantities, then mpr_SMhorizons (src/MPR/mo_mpr_smhorizons.f90:
// 340-582) for each model horizon; harmonic-mean operands are stored as the
// reciprocals the upscaling sums.
//
// What bounds it: one lane's chain of eleven elementary functions, then two
// powers and five divisions (9,000-12,000 cycles).  So a row has 16 lanes: a
// lane per soil horizon, then a lane per model horizon and one for the
// column's quantities.  30 rows, cold: 89 us with one thread a row, 41 us here (one
// copy of each function instead of the inlined ones changed nothing).
constexpr int kRowLanes = kMprMaxSoilHor, kTableRows = 4;
static_assert(kRowLanes == 16 && kMaxHorizons < kRowLanes, "a row's lanes are half a warp, the last for the column");
struct SoilRow {
    double ths[kMprMaxSoilHor], thfc[kMprMaxSoilHor], thpw[kMprMaxSoilHor], ks[kMprMaxSoilHor], db[kMprMaxSoilHor];
};

__device__ void soil_row(const MprArgs &a, const double *g, int s, int l, int lane, SoilRow &w, double *row)
{
    const int H = a.H, mh = a.max_hor, nh = a.n_hor[s], nt = a.n_till[s];
    const double *ps = g + a.off.soil;
    if (lane < nh) {
        const int j = lane;
        const double om_forest = (a.proc_sm <= 2) ? ps[2] + ps[0] : ps[0];
        const double pom = (l == 0) ? om_forest : (l == 1) ? ps[1] : ps[2];
        const double sand = a.sand[s * mh + j], clay = a.clay[s * mh + j], dbm = a.dbm[s * mh + j];
        double k = hydro_cond(ps + 9, sand, clay), n, alpha, db = dbm, ths;
        if (j < nt) {
            const double pm = 100.0 - pom;
            db = hm_div(100.0, hm_div(pom, kBulkDensOrgMatter) + hm_div(pm, dbm));
            k = k * hm_div(dbm, db);
        }
        genuchten(ps + 3, sand, clay, db, ths, n, alpha);
        w.db[j] = db;
        w.ks[j] = k;
        w.ths[j] = ths;
        w.thfc[j] = field_cap(k, ths, n);
        w.thpw[j] = pwp(n, alpha, ths);
    }
    __syncwarp();
    if (lane == kRowLanes - 1) {
        // Ks variabilities over the column (:330-352)
        double kh = 0.0, kv = 0.0, fc = 0.0, tot = 0.0;
        for (int j = 0; j < nh; ++j) {
            kh = kh + w.ths[j] * w.ks[j];
            kv = kv + hm_div(w.ths[j], w.ks[j]);
            fc = fc + w.thfc[j];
            tot = tot + w.ths[j];
        }
        const double sms_fc = hm_div(tot - fc, tot);
        const double ksvar_h = hm_div(hm_div(kh, tot), ps[12]);
        const double ksvar_v = hm_div(hm_div(tot, kv), ps[12]);
        const double *pi = g + a.off.interflow, *pp = g + a.off.perc;
        row[5 * H + 0] = pi[0] * sms_fc;                                                   // mpr_runoff HL1 operand
        row[5 * H + 1] = pi[3] * (1.0 + ksvar_h);                                          // K1 soil term
        row[5 * H + 2] = pi[4] * hm_div(1.0, ksvar_h) * hm_div(1.0, 1.0 + sms_fc);         // alpha operand
        row[5 * H + 3] = hm_div(pp[0] * (1.0 + sms_fc), 1.0 + ksvar_v);                    // karstic_layer Kp operand
    }
    if (lane >= H) return;

    // horizons (mpr_SMhorizons); its 4 or 8 parameters follow the first 13
    const int h = lane;
    const double *p2 = ps + 13;
    const double *wd = a.Wd + ((size_t)s * H + h) * mh;
    double a1 = 0.0, b1 = 0.0;
    for (int j = 0; j < nt; ++j)
        if (wd[j] > 0.0) a1 = a1 + w.db[j] * wd[j];
    for (int j = nt; j < nh; ++j)
        if (wd[j] >= 0.0) b1 = b1 + w.db[j] * wd[j];
    const double bd = a1 + b1;
    double sums[3];
    const double *th[3] = {w.ths, w.thfc, w.thpw};
    for (int q = 0; q < 3; ++q) {
        double x = 0.0, y = 0.0;
        for (int j = 0; j < nt; ++j)
            if (wd[j] > 0.0) x = x + th[q][j] * wd[j];
        for (int j = nt; j < nh; ++j)
            if (wd[j] > 0.0) y = y + th[q][j] * wd[j];
        sums[q] = x + y;
    }
    double dpth_f = 0.0, dpth_t = a.hd[h];
    if (h > 0 && h < H - 1) dpth_f = a.hd[h - 1];
    double dpth_t_roots = dpth_t;
    if (h == H - 1) {
        dpth_f = a.hd[H - 2];
        dpth_t = a.rz[s];               // this cell's own soil
        dpth_t_roots = a.dpth_t_last;   // what the root loop sees afterwards
    }
    const double sms = sums[0] * (dpth_t - dpth_f);
    const double fcv = sums[1] * (dpth_t - dpth_f);
    const double pwv = sums[2] * (dpth_t - dpth_f);
    double c;
    if (l == 0) {
        c = p2[0];
    } else if (l == 1) {
        c = p2[1];
    } else if (a.proc_sm <= 2) {
        c = p2[0] - p2[2];
    } else {
        const double rc_sand = p2[5] - p2[4], rc_clay = p2[5], fcmin = p2[6], fcmax = p2[6] + p2[7];
        double fcn = hm_div(hm_div(fcv, dpth_t_roots - dpth_f) - fcmin, fcmax - fcmin);
        if (fcn < 0.0)
            fcn = 0.0;
        else if (fcn > 1.0)
            fcn = 1.0;
        c = (fcn * rc_clay) + ((1.0 - fcn) * rc_sand);
    }
    const double fr = (1.0 - hm_pow(c, dpth_t_roots * 0.1)) - (1.0 - hm_pow(c, dpth_f * 0.1));
    row[MT_INV_SMS * H + h] = hm_div(1.0, sms);
    row[MT_INV_BETA * H + h] = hm_div(1.0, bd * p2[3]);
    row[MT_INV_PW * H + h] = hm_div(1.0, pwv);
    row[MT_INV_FC * H + h] = hm_div(1.0, fcv);
    row[MT_INV_FROOTS * H + h] = hm_div(1.0, fr);
}

// grid (ceil(n_keys / 4) + ceil(LAI entries / 64), members): soil rows, then
// (proc_pet = -1 with class LAI) the reciprocal LAI correction factors of
// pet_correctbyLAI (src/MPR/mo_mpr_pet.f90:60-140) per (land cover, LAI class,
// month)
__global__ void __launch_bounds__(kTableRows * kRowLanes) mpr_table_kernel(MprArgs a)
{
    __shared__ SoilRow rows[kTableRows];
    const int m = blockIdx.y, r = threadIdx.x / kRowLanes;
    const int row_blocks = (a.n_keys + kTableRows - 1) / kTableRows;
    const double *g = a.gamma + (size_t)m * a.n_gamma;
    const int ts = mpr_table_stride(a.H);
    if ((int)blockIdx.x < row_blocks) {
        const int t = (int)blockIdx.x * kTableRows + r;
        if (t >= a.n_keys) return;
        soil_row(a, g, t / 3, t % 3, threadIdx.x % kRowLanes, rows[r], a.table + ((size_t)m * a.n_keys + t) * ts);
        return;
    }
    const int u = ((int)blockIdx.x - row_blocks) * blockDim.x + threadIdx.x;
    if (a.proc_pet != -1 || u >= 3 * a.n_lai_classes * 12) return;
    const int l = u / (a.n_lai_classes * 12), c = (u / 12) % a.n_lai_classes, mo = u % 12;
    const double *p = g + a.off.pet;
    const double base = (l == 0) ? p[0] : (l == 1) ? p[1] : p[2];
    const double f = base + (p[3] * (1.0 - hm_exp(p[4] * a.lai_lut[c * 12 + mo])));
    a.petlai[(size_t)m * 3 * a.n_lai_classes * 12 + u] = hm_div(1.0, f);
}

// The arithmetic mean's division by the number of sub-cells, the same for all
// of a cell's means
struct Mean {
    double dn;
    uint64_t inv;
    __device__ explicit Mean(double n) : dn(n), inv(hm_recip_of(n)) {}
    __device__ double operator()(double sum) const { return hm_div_r(sum, dn, inv); }
};

// One soil horizon of a cell: harmonic means (upscale_harmonic_mean,
// src/MPR/mo_upscaling_operators.f90:369-432), then the limits of
// mpr_SMhorizons (src/MPR/mo_mpr_smhorizons.f90:712-737).  Returns the root
// fraction before its normalisation.
__device__ double upscale_horizon(const MprArgs &a, int h, int k, int ns, const double *tab, double *out)
{
    const int H = a.H, ts = mpr_table_stride(H);
    const size_t N = a.n1;
    const uint32_t *code = a.code + k;
    const double dn = (double)ns;
    double s_sms = 0.0, s_beta = 0.0, s_pw = 0.0, s_fc = 0.0, s_fr = 0.0;
    for (int j = 0; j < ns; ++j) {
        const uint32_t key = __ldg(code + (size_t)j * N) & kMprKeyMask;
        if (!bc_ok(BC_MPR_KEY, key, a.n_keys)) continue;
        const double *row = tab + (size_t)key * ts;
        s_sms = s_sms + __ldg(row + MT_INV_SMS * H + h);
        s_beta = s_beta + __ldg(row + MT_INV_BETA * H + h);
        s_pw = s_pw + __ldg(row + MT_INV_PW * H + h);
        s_fc = s_fc + __ldg(row + MT_INV_FC * H + h);
        s_fr = s_fr + __ldg(row + MT_INV_FROOTS * H + h);
    }
    double sms = hm_div(dn, s_sms), fc = hm_div(dn, s_fc), pw = hm_div(dn, s_pw);
    if (fc > sms) fc = sms - 0.01 * sms;
    if (pw > fc) pw = fc - 0.01 * fc;
    if (sms < 0.0) sms = 0.0001;
    if (fc < 0.0) fc = 0.0001;
    if (pw < 0.0) pw = 0.0001;
    out[(size_t)(P_HORIZON + 1 * H + h) * N + k] = sms;
    out[(size_t)(P_HORIZON + 2 * H + h) * N + k] = fc;
    out[(size_t)(P_HORIZON + 3 * H + h) * N + k] = pw;
    out[(size_t)(P_HORIZON + 4 * H + h) * N + k] = hm_div(dn, s_beta);
    return hm_div(dn, s_fr);
}

// Arithmetic means (upscale_arithmetic_mean, :266-329): the thresholds and
// recession constants of mpr_runoff (src/MPR/mo_mpr_runoff.f90:141-191) and
// baseflow_param; then the values that need no sub-cells: snow
// (snow_acc_melt_param, src/MPR/mo_multi_param_reg.f90:800-852), sealed
// threshold, karst loss (karstic_layer, :1032) and Jarvis threshold
__device__ void upscale_recession(const MprArgs &a, const double *g, int k, int ns, const double *tab, double *out)
{
    const int H = a.H, ts = mpr_table_stride(H);
    const size_t N = a.n1;
    const double *pi = g + a.off.interflow, *geo = g + a.off.geo;
    const double p1 = pi[1], p2 = pi[2];
    double s_k0 = 0.0, s_k1 = 0.0, s_k2 = 0.0;
    for (int j = 0; j < ns; ++j) {
        const uint32_t c = __ldg(a.code + k + (size_t)j * N);
        if (!bc_ok(BC_MPR_KEY, c & kMprKeyMask, a.n_keys) ||
            !bc_ok(BC_MPR_GEO, (long long)(c >> 24), (long long)a.n_gamma - a.off.geo))
            continue;
        const double t1 = p1 * (2.0 - __ldg(a.se + k + (size_t)j * N));
        double t0 = t1;
        if (c & kMprForest) t0 = t0 * p2;
        s_k0 = s_k0 + t0;
        s_k1 = s_k1 + (t1 + __ldg(tab + (size_t)(c & kMprKeyMask) * ts + 5 * H + 1));
        s_k2 = s_k2 + __ldg(geo + (c >> 24));
    }
    const Mean mean((double)ns);
    double k0 = mean(s_k0), k1 = mean(s_k1), k2 = mean(s_k2);
    if (k0 < 1.0) k0 = 1.0;
    if (k1 < 2.0) k1 = 2.0;
    if (k0 > k1) k0 = k1;
    if (k2 < k1) k2 = k1; // src/MPR/mo_multi_param_reg.f90:618
    out[(size_t)P_K0 * N + k] = k0;
    out[(size_t)P_K1 * N + k] = k1;
    out[(size_t)P_K2 * N + k] = k2;
    const double *psn = g + a.off.snow;
    const double ff = a.f_forest[k], fs = a.f_sealed[k], fp = a.f_perm[k];
    const double ddf_f = psn[1], ddf_i = psn[1] + psn[3] + psn[2], ddf_p = psn[1] + psn[3];
    const double mdf_f = psn[1] + psn[5], mdf_i = psn[1] + psn[3] + psn[2] + psn[6], mdf_p = psn[1] + psn[3] + psn[7];
    out[(size_t)P_FSEALED * N + k] = fs;
    out[(size_t)P_TTHRESH * N + k] = psn[0];
    out[(size_t)P_DDINC * N + k] = psn[4];
    out[(size_t)P_DDNOPRE * N + k] = (ddf_f * ff + ddf_i * fs + ddf_p * fp);
    out[(size_t)P_DDMAX * N + k] = (mdf_f * ff + mdf_i * fs + mdf_p * fp);
    out[(size_t)P_STHRESH * N + k] = g[a.off.runoff];
    out[(size_t)P_KARST * N + k] = 1.0 - (a.f_kar[k] * g[a.off.perc + 1]);
    out[(size_t)P_JARVIS * N + k] =
        (a.proc_sm == 2 || a.proc_sm == 3) ? g[a.off.soil + a.off.n_soil_params - 1] : 0.0;
}

// ... interflow threshold and exponent, percolation (karstic_layer), and
// pet_correctbyASP (src/MPR/mo_mpr_pet.f90:236-272)
__device__ void upscale_aspect(const MprArgs &a, const double *g, int k, int ns, const double *tab, double *out)
{
    const int H = a.H, ts = mpr_table_stride(H);
    const size_t N = a.n1;
    const double *pp = g + a.off.pet;
    const bool asp_on = (a.proc_pet == 0 || a.proc_pet == 1);
    const double tmax = pp[0] + pp[1];
    const double slope_lo = asp_on ? (tmax - pp[0]) / pp[2] : 0.0;
    const double slope_hi = asp_on ? (tmax - pp[0]) / (360.0 - pp[2]) : 0.0;
    double s_hl1 = 0.0, s_alpha = 0.0, s_kp = 0.0, s_asp = 0.0;
    for (int j = 0; j < ns; ++j) {
        const uint32_t c = __ldg(a.code + k + (size_t)j * N);
        if (!bc_ok(BC_MPR_KEY, c & kMprKeyMask, a.n_keys) ||
            !bc_ok(BC_MPR_GEO, (long long)(c >> 24), (long long)a.n_gamma - a.off.geo))
            continue;
        const double *row = tab + (size_t)(c & kMprKeyMask) * ts + 5 * H;
        s_hl1 = s_hl1 + __ldg(row);
        s_alpha = s_alpha + __ldg(row + 2);
        s_kp = s_kp + __ldg(row + 3);
        if (asp_on) {
            const double x = __ldg(a.asp + k + (size_t)j * N);
            // northern cells: the low branch below the threshold aspect;
            // southern cells: the mirrored assignment
            const bool low = ((c & kMprNorth) != 0) == (x < pp[2]);
            s_asp = s_asp + (pp[0] + hm_sel(low, slope_lo, slope_hi) * hm_sel(low, x, 360.0 - x));
        }
    }
    const Mean mean((double)ns);
    double kp = mean(s_kp);
    if (kp < 2.0) kp = 2.0;
    out[(size_t)P_UTHRESH * N + k] = mean(s_hl1);
    out[(size_t)P_ALPHA * N + k] = mean(s_alpha);
    out[(size_t)P_KP * N + k] = kp;
    out[(size_t)P_FASP * N + k] = asp_on ? mean(s_asp) : 0.0;
    out[(size_t)P_HARSAM * N + k] = (a.proc_pet == 1) ? pp[3] : 0.0;
}

// One LAI entry's means into their planes (a gridded series:
// [member][lai_groups][n_lai][N])
__device__ void put_lai(const MprArgs &a, int m, int mo, int k, double v_int, double v_pet, double v_pet2, double *out)
{
    const size_t N = a.n1;
    if (a.lai_out) {
        const int ng = lai_groups(a.proc_pet), n_lai = a.n_lai_steps;
        double *lo = a.lai_out + (size_t)m * ng * n_lai * N + (size_t)mo * N + k;
        lo[0] = v_int;
        if (ng > 1) lo[(size_t)n_lai * N] = v_pet;
        if (ng > 2) lo[(size_t)2 * n_lai * N] = v_pet2;
    } else {
        out[(size_t)(P_MAXINTER + mo) * N + k] = v_int;
        out[(size_t)(P_PETLAI + mo) * N + k] = v_pet;
        out[(size_t)(P_PET2 + mo) * N + k] = v_pet2;
    }
}

// LAI entries part, part + n_parts, ... of a cell: canopy_intercept_param
// (src/MPR/mo_multi_param_reg.f90:1132-1152) and pet_correctbyLAI, per LAI
// entry (12 monthly slots or a gridded series: the reference loops over
// size(LAI0, 2), :1142)
template <int PET>
__device__ void upscale_lai(const MprArgs &a, const double *g, int part, int n_parts, int k, int m, int ns, double *out)
{
    const size_t N = a.n1, slots = (size_t)a.max_sub * N;
    const double *pp = g + a.off.pet, gi = g[a.off.interc];
    const double *plai = a.petlai + (size_t)m * 3 * a.n_lai_classes * 12;
    const int n_lai = a.n_lai_steps;
    const Mean mean((double)ns);
    for (int mo = part; mo < n_lai; mo += n_parts) {
        double s_int = 0.0, s_pet = 0.0, s_pet2 = 0.0;
        for (int j = 0; j < ns; ++j) {
            const uint32_t c = __ldg(a.code + k + (size_t)j * N);
            if (!a.lai && !bc_ok(BC_MPR_LAI, (c >> 16) & 0xFFu, a.n_lai_classes)) continue;
            const double lai = a.lai ? __ldg(a.lai + mo * slots + (size_t)j * N + k)
                                     : __ldg(a.lai_lut + ((c >> 16) & 0xFFu) * 12 + mo);
            const int l = (int)((c & kMprKeyMask) % 3u); // 0 forest, 1 impervious, 2 pervious
            s_int = s_int + lai * gi;
            // priestley_taylor_alpha, src/MPR/mo_mpr_pet.f90:311-369: alpha0 = p1 + p2 LAI0
            if constexpr (PET == 2) s_pet = s_pet + (pp[0] + pp[1] * lai);
            if constexpr (PET == 3) {
                // aerodynamical_resistance, src/MPR/mo_multi_param_reg.f90:1165-1262: canopy
                // height by land cover (pervious: p3 LAI / max over the months), measurement
                // height 10 m raised above the canopy, log profile with karman = 0.41
                double hc = (l == 0) ? pp[0] : pp[1];
                if (l == 2) {
                    double mx = -1.0e300;
                    for (int t = 0; t < n_lai; ++t) { // MAXVAL(LAI0, dim=2) over every entry
                        const double x = a.lai ? __ldg(a.lai + t * slots + (size_t)j * N + k)
                                               : __ldg(a.lai_lut + ((c >> 16) & 0xFFu) * 12 + t);
                        mx = (t == 0 || x > mx) ? x : mx;
                    }
                    hc = pp[2] * lai / mx;
                }
                double zm = 10.0;
                if (zm < hc) zm = hc + zm;
                const double disp = pp[3] * hc, z0m = pp[4] * hc, z0h = pp[5] * z0m;
                s_pet = s_pet + hm_log((zm - disp) / z0m) * hm_log((zm - disp) / z0h) / (0.41 * 0.41);
                // bulksurface_resistance, src/MPR/mo_mpr_pet.f90:407-475, capped at 250 s m-1
                const double rs = pp[6] / (lai / (0.3 * lai + 1.2));
                s_pet2 = s_pet2 + (rs > 250.0 ? 250.0 : rs);
            }
            if constexpr (PET == -1) {
                double inv;
                if (a.lai) {
                    const double base = (l == 0) ? pp[0] : (l == 1) ? pp[1] : pp[2];
                    inv = 1.0 / (base + (pp[3] * (1.0 - hm_exp(pp[4] * lai))));
                } else {
                    inv = __ldg(plai + ((size_t)l * a.n_lai_classes + ((c >> 16) & 0xFFu)) * 12 + mo);
                }
                s_pet = s_pet + inv;
            }
        }
        put_lai(a, m, mo, k, mean(s_int), PET == -1 ? hm_div(mean.dn, s_pet) : PET >= 2 ? mean(s_pet) : 0.0,
                PET == 3 ? mean(s_pet2) : 0.0, out);
    }
}

// The same for the 12 months of class LAI where only canopy interception and
// the LAI correction depend on it: `lg`, the classes' LAI times the canopy
// factor, was multiplied once for the block
constexpr int kLaiParts = 2, kPartMonths = 12 / kLaiParts;
template <int PET>
__device__ void upscale_lai_classes(const MprArgs &a, const double *lg, int part, int k, int m, int ns, double *out)
{
    const size_t N = a.n1;
    const double *plai = a.petlai + (size_t)m * 3 * a.n_lai_classes * 12;
    const int mo0 = part * kPartMonths;
    double s_int[kPartMonths] = {}, s_pet[kPartMonths] = {};
    for (int j = 0; j < ns; ++j) {
        const uint32_t c = __ldg(a.code + k + (size_t)j * N), cls = (c >> 16) & 0xFFu;
        if (!bc_ok(BC_MPR_LAI, cls, a.n_lai_classes)) continue;
#pragma unroll
        for (int i = 0; i < kPartMonths; ++i) s_int[i] = s_int[i] + lg[cls * 12 + mo0 + i];
        if constexpr (PET == -1) {
            const double *p = plai + ((size_t)((c & kMprKeyMask) % 3u) * a.n_lai_classes + cls) * 12 + mo0;
#pragma unroll
            for (int i = 0; i < kPartMonths; ++i) s_pet[i] = s_pet[i] + __ldg(p + i);
        }
    }
    const Mean mean((double)ns);
#pragma unroll
    for (int i = 0; i < kPartMonths; ++i)
        put_lai(a, m, mo0 + i, k, mean(s_int[i]), PET == -1 ? hm_div(mean.dn, s_pet[i]) : 0.0, 0.0, out);
}

// grid (ceil(n1 / 32), members), block 32 cells x (H + 4) warps: a warp per
// soil horizon, two for the other means, two for the LAI entries.
//
// What bounds it: the FP64 pipe (19 cycles of an SM an instruction), so sums
// of table entries are all that is left on it -- about 40 additions a sub-cell
// with 3 horizons; divisions run on the integer pipe, and what belongs to
// another PET process or repeats over the cells is not issued.  One thread a
// cell issued 143 a sub-cell: 64 members of 9,216 cells with 16 sub-cells each
// 2.55 ms, 0.98 ms here.  The warps of a cell also shorten its chain where a
// launch has few cells: mhm_mpr of one member with 9,216 cells 0.24 -> 0.10 ms.
__global__ void __launch_bounds__(32 * (kMaxHorizons + 4)) mpr_upscale_kernel(MprArgs a)
{
    extern __shared__ double s_mpr[]; // [H][32] root fractions, then the classes' LAI times the canopy factor
    const int lane = threadIdx.x % 32, part = threadIdx.x / 32, H = a.H;
    const int k = blockIdx.x * 32 + lane, m = blockIdx.y;
    const double *g = a.gamma + (size_t)m * a.n_gamma;
    const double *tab = a.table + (size_t)m * a.n_keys * mpr_table_stride(H);
    double *out = a.params + (size_t)m * a.member_stride;
    double *lg = s_mpr + H * 32;
    const bool here = k < a.n1;
    const int ns = here ? a.nsub[k] : 0;
    if (!a.lai)
        for (int i = threadIdx.x; i < a.n_lai_classes * 12; i += blockDim.x) lg[i] = a.lai_lut[i] * g[a.off.interc];
    double froots = 0.0;
    if (here && part < H) froots = upscale_horizon(a, part, k, ns, tab, out);
    if (part < H) s_mpr[part * 32 + lane] = froots;
    __syncthreads();
    if (!here) return;
    if (part < H) { // the root normalisation of mpr_SMhorizons
        double ftot = 0.0;
        for (int h = 0; h < H; ++h) {
            const double f = s_mpr[h * 32 + lane];
            if (f > 0.0) ftot = ftot + f;
        }
        out[(size_t)(P_HORIZON + part) * a.n1 + k] = (ftot > 0.0) ? hm_div(froots, ftot) : 0.0;
    } else if (part == H) {
        upscale_recession(a, g, k, ns, tab, out);
    } else if (part == H + 1) {
        upscale_aspect(a, g, k, ns, tab, out);
    } else {
        const int p = part - H - 2;
        if (a.proc_pet == 2) upscale_lai<2>(a, g, p, kLaiParts, k, m, ns, out);
        else if (a.proc_pet == 3) upscale_lai<3>(a, g, p, kLaiParts, k, m, ns, out);
        else if (a.proc_pet == -1 && !a.lai) upscale_lai_classes<-1>(a, lg, p, k, m, ns, out);
        else if (a.proc_pet == -1) upscale_lai<-1>(a, g, p, kLaiParts, k, m, ns, out);
        else if (!a.lai) upscale_lai_classes<0>(a, lg, p, k, m, ns, out);
        else upscale_lai<0>(a, g, p, kLaiParts, k, m, ns, out);
    }
}

} // namespace

cudaError_t launch_mpr(const MprArgs &a, cudaStream_t s)
{
    if (a.n_members <= 0) return cudaSuccess;
    const int row_blocks = (a.n_keys + kTableRows - 1) / kTableRows, bs = kTableRows * kRowLanes;
    const int lai_blocks = a.proc_pet == -1 ? (3 * a.n_lai_classes * 12 + bs - 1) / bs : 0;
    mpr_table_kernel<<<dim3(row_blocks + lai_blocks, a.n_members), bs, 0, s>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const size_t smem = ((size_t)a.H * 32 + (a.lai ? 0 : (size_t)a.n_lai_classes * 12)) * sizeof(double);
    mpr_upscale_kernel<<<dim3((a.n1 + 31) / 32, a.n_members), 32 * (a.H + 4), smem, s>>>(a);
    return cudaGetLastError();
}

} // namespace mhm

MHM_BC_ACCESSOR(bc_take_mpr)
