// routing.cu -- mRM L1->L11 runoff accumulation and Muskingum link routing.
//
// The reference advances every link one step at a time in netPerm order
// (L11_routing, src/mRM/mo_mrm_routing.f90:380-481).  The per-link recurrence
// only reads the link's own previous step and the same-step outflow of its
// upstream links, so a chunk of steps runs through the river network as a
// pipeline, each node one step behind the node upstream.  Inflow sums at
// confluences keep the reference's order (upstream links in netPerm rank
// order, then the node's own qOUT), so results are bit-identical.
#include <cstdint>
#include <type_traits>

#include "bounds.cuh"
#include "calendar.h"
#include "fp64i.h"
#include "mhm_kernels.cuh"
#include "network.h"

namespace mhm {

// L11_runoff_acc, src/mRM/mo_mrm_pre_routing.f90:77-143: per (step, member,
// node) the area-weighted sum of its L1 cells in ascending cell order, then
// *1000/TST.  Output indexed by routing position.
__global__ void __launch_bounds__(256) runoff_acc_kernel(const AccArgs a)
{
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t L = a.n_nodes;
    const int64_t total = (int64_t)a.n_steps * a.n_members * L;
    if (gid >= total) return;
    const int pos = (int)(gid % L);
    const int64_t tm = gid / L; // t * M + m
    const int m = (int)(tm % a.n_members);
    const int t = (int)(tm / a.n_members);
    if (a.member_step0 && a.member_step0[m] < 0) return; // idle member
    // runoff of cell k for routing step t: the model step's value, or with a
    // routing step of `win` model steps their sum from 0 in step order
    // (RunToRout, src/mHM/mo_mhm_interface_run.f90:489-490)
    const size_t row_stride = (size_t)a.n_members * a.n_cells;
    const double *row = a.tro + ((size_t)t * a.win * a.n_members + m) * a.n_cells;
    auto run = [&](int k) -> double {
        if (a.win == 1) return __ldg(row + k);
        double r = 0.0;
        for (int j = 0; j < a.win; ++j) r = r + __ldg(row + j * row_stride + k);
        return r;
    };
    double q;
    if (a.map_flag) {
        double acc = 0.0;
        const int b = __ldg(a.node_cell_ptr + pos), e = __ldg(a.node_cell_ptr + pos + 1);
        for (int j = b; j < e; ++j) {
            const int k = __ldg(a.node_cells + j);
            if (!bc_ok(BC_ACC_CELL, k, a.n_cells)) continue;
            acc = acc + run(k) * __ldg(a.l1_area + k);
        }
        q = acc * 1000.0 / a.TST;
    } else {
        const int k = __ldg(a.pos_l11_l1 + pos);
        q = bc_ok(BC_ACC_L1, k, a.n_cells) ? run(k) * __ldg(a.pos_area + pos) * 1000.0 / a.TST : 0.0;
    }
    a.qout[((size_t)m * a.n_steps + t) * L + pos] = q;
}

// A step of an exported outflow series: the value and the number of the step,
// counted on through all launches, in one 16-byte word that is read and
// written whole.  A reader that finds the number it expects has the value; no
// other ordering is needed, and a word left by an earlier launch never matches.
__device__ __forceinline__ void put_step(longlong2 *p, double v, uint64_t id)
{
    asm volatile("{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"(id)
                 : "memory");
}
__device__ __forceinline__ void get_step(const longlong2 *p, uint64_t &v, uint64_t &id)
{
    asm volatile("{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}"
                 : "=l"(v), "=l"(id)
                 : "l"(p)
                 : "memory");
}

// Reads a step until it is there.  The wait has a limit: when it runs out, or
// another block's did, the launch is marked and false comes back.
__device__ bool wait_step(const RouteArgs &a, const longlong2 *p, uint64_t id, uint64_t &v)
{
    uint64_t got = ~id;
    for (int polls = 0; got != id; ++polls) {
        volatile uint32_t *ab = a.abort;
        if (polls > a.max_polls || ((polls & 63) == 63 && *ab == a.launch)) {
            *ab = a.launch;
            *reinterpret_cast<volatile int32_t *>(a.timed_out) = 1;
            return false;
        }
        get_step(p, v, got);
    }
    return true;
}

// The upstream links of a node with more of them than a thread keeps (none on a D8
// grid), by the lanes that are in this tick together: for each such node among them
// (`hub` >= 0) every lane reads the step of one link, and the next link's while these
// are added to the node's sum q one after another in their order.  Read by the node's
// own thread, each link was a trip to the L2 (a node with 2,000 of them, 240 steps:
// 161 ms; 56 ms where all blocks met after each step; 34 so).
__device__ __forceinline__ double add_hubs(const RouteArgs &a, const longlong2 *qx, int hub, int t, double q, bool &bad)
{
    const unsigned act = __activemask();
    const int lane = threadIdx.x & 31, n_act = __popc(act), rank = __popc(act & ((1u << lane) - 1));
    for (unsigned hubs = __ballot_sync(act, hub >= 0); hubs != 0; hubs &= hubs - 1) {
        const int src = __ffs((int)hubs) - 1, h = __shfl_sync(act, hub, src), th = __shfl_sync(act, t, src);
        const int u0 = __ldg(a.hub_ptr + h), u1 = __ldg(a.hub_ptr + h + 1);
        const uint64_t id = a.done0 + (uint64_t)th;
        const longlong2 *p = nullptr;
        uint64_t v = 0, got = id; // a lane without a link: adding +0 changes nothing
        auto fetch = [&](int u) {
            const int x = u < u1 ? __ldg(a.hub_ups + u) : -1;
            p = x >= 0 && bc_ok(BC_ROUTE_UP, x, a.n_exports) ? qx + (size_t)x * a.qx_stride + th : nullptr;
            v = 0;
            got = id;
            if (p) get_step(p, v, got);
        };
        double sum = __shfl_sync(act, q, src);
        fetch(u0 + rank);
        for (int u = u0; u < u1; u += n_act) {
            if (got != id && !bad) bad = !wait_step(a, p, id, v);
            const double mine = __longlong_as_double((long long)v);
            __syncwarp(act);
            fetch(u + n_act + rank);
            for (unsigned m = act; m != 0; m &= m - 1) sum = sum + __shfl_sync(act, mine, __ffs((int)m) - 1);
        }
        if (lane == src) q = sum;
    }
    return q;
}

// One block of the network for one member: a thread per node, a step per tick,
// each node `lag` ticks behind the block's first.  L11_routing body,
// src/mRM/mo_mrm_routing.f90:435-478: ((0 + qTR(up_1)) + qTR(up_2) + ...) +
// qOUT, then the Muskingum recurrence.
//
// What bounds it: the tick, a chain of dependent FP64 operations (64 cycles
// each on this GPU, three plus one per upstream link), of the instructions
// around them -- two warps wait for each in turn, so addresses move with the
// step instead of being computed from it, and what few networks need is an
// instantiation of its own (107 -> 75 a tick: 36 nodes, 2,160 steps 1.35 -> 0.93 ms) -- and a block barrier; a chunk of T steps takes T
// ticks plus the length of the river.  So everything a
// tick reads is already on the chip: outflows pass from node to node through a
// ring in shared memory, a node's own runoff and the outflows of other blocks
// are fetched a round of S ticks ahead.  A block exports the outflow of its
// pieces' last nodes to device memory, step by step.  Measured (one chunk of
// 240 steps): 62,500 nodes, 1,478 deep, 1.9 ms; the same on a 1,458-deep grid
// 1.9 ms; 576 nodes 0.17 ms.  A launch (or a cluster barrier) per wavefront
// of all nodes, whose loads all came from device memory, took 16.1, 27.9 and
// 0.69 ms.  64 nodes a block: with 32 a 576-node network takes 0.24 ms (more
// hand-overs), with 128 the deep one gains nothing (the FP64 pipe of the SM is
// shared by more warps a tick).  Two threads a node, one for
// the sum and one for the recurrence, take 7-14 % longer: the hand-over costs
// more than it takes off the chain.  S = 8 covers a device-memory load; S = 4 hands
// over sooner, 15-17 % faster where the river is longer than the chunk and up to
// 5 % slower where it is not.
//
// Blocks take (network block, member) pairs from a counter, in an order in
// which a pair waits only on pairs taken before it.  So whatever the number of
// resident blocks, the oldest running one waits on nothing unfinished and the
// launch ends; the limit in wait_step only guards against a defect.
//
// HUB: the network has nodes whose upstream links are read by add_hubs; another
// instantiation, so that its registers are not every network's.
template <int S, bool HUB>
__global__ void __launch_bounds__(kRouteBlock) route_flow_kernel(const RouteArgs a)
{
    // by tick: the outflows of the block's nodes, then of the series it takes,
    // then a slot that stays +0 (the upstream link of a node without one)
    constexpr int kSlots = 2 * kRouteBlock + 1, kZero = 2 * kRouteBlock;
    __shared__ double ring[2 * S][kSlots];
    __shared__ double own_q[2 * S][kRouteBlock]; // the nodes' own runoff by tick
    __shared__ uint32_t s_pair;
    const int tid = threadIdx.x;
    if (tid == 0) s_pair = atomicAdd(a.ticket, 1u) - a.ticket0;
    __syncthreads();
    const int b = (int)(s_pair / (uint32_t)a.n_members), m = (int)(s_pair - (uint32_t)b * a.n_members);
    if (a.member_step0 && a.member_step0[m] < 0) return; // idle member: routing states untouched
    const int p0 = __ldg(a.blk_ptr + b), n = __ldg(a.blk_ptr + b + 1) - p0;
    const int e0 = __ldg(a.ext_ptr + b), ne = __ldg(a.ext_ptr + b + 1) - e0;
    const int nT = a.n_steps;
    const int rounds = (nT + __ldg(a.blk_lag + b) + S - 1) / S;
    const int64_t L = a.n_nodes;
    const size_t ms = (size_t)m * L;
    longlong2 *const qx = a.qx + (size_t)m * a.n_exports * a.qx_stride;

    const bool own = tid < n;
    const int pos = p0 + tid;
    int lag = 0, flags = 0, ex = -1, nu = 0, hub = -1;
    int up[kRouteUps]; // the upstream links' slots
#pragma unroll
    for (int j = 0; j < kRouteUps; ++j) up[j] = kZero;
    double qtin1 = 0.0, qtr1 = 0.0, c1 = 0.0, c2 = 0.0;
    if (own) {
        lag = __ldg(a.pos_lag + pos);
        flags = __ldg(a.pos_flags + pos);
        ex = __ldg(a.pos_export + pos);
        const int4 w = __ldg(reinterpret_cast<const int4 *>(a.pos_ups) + pos);
        const int v[kRouteUps] = {(int16_t)w.x, w.x >> 16, (int16_t)w.y, w.y >> 16,
                                  (int16_t)w.z, w.z >> 16, (int16_t)w.w, w.w >> 16};
        if (HUB && v[0] == -2) {
            hub = v[1] + (v[2] << 15);
        } else {
#pragma unroll
            for (int j = 0; j < kRouteUps; ++j)
                if (v[j] >= 0 && bc_ok(BC_ROUTE_UP, v[j], kZero)) {
                    up[j] = v[j];
                    nu = j + 1;
                }
        }
        qtin1 = a.qtin1[ms + pos];
        qtr1 = a.qtr1[ms + pos];
        c1 = __ldg(a.C1 + ms + pos);
        c2 = __ldg(a.C2 + ms + pos);
    }
    const bool is_link = flags & 1, add_qout = flags & 2, cut = flags & 4; // cut: mo_mrm_routing.f90:447-452
    const bool keep_qmod = own && (a.qmod_all || (flags & 16));
    const double *qo = a.qout + (size_t)m * a.n_qsteps * L + pos;
    double *qm = a.qmod + (size_t)m * nT * L + pos;
    longlong2 *const out = ex >= 0 ? qx + (size_t)ex * a.qx_stride : nullptr;
    // warp-wide facts, so that a tick branches on them without divergence.
    // Adding the +0 of a link a node does not have changes nothing (its sum is
    // never -0), so all lanes of a warp add as many links as the longest list;
    // likewise the +0 runoff of a node that adds none.
    const int nu_warp = (int)__reduce_max_sync(~0u, (unsigned)nu);
    const bool hub_warp = HUB && __any_sync(~0u, hub >= 0), cut_warp = __any_sync(~0u, cut);
    const bool out_warp = __any_sync(~0u, ex >= 0), qmod_warp = __any_sync(~0u, keep_qmod);
    const int lag_hi = (int)__reduce_max_sync(~0u, (unsigned)lag);
    const int lag_lo = (int)__reduce_min_sync(~0u, own ? (unsigned)lag : 0xffffu);

    // series tid of the block's list
    const int x_in = tid < ne ? __ldg(a.ext_export + e0 + tid) : 0;
    const bool take = tid < ne && bc_ok(BC_ROUTE_UP, x_in, a.n_exports);
    const longlong2 *in = take ? qx + (size_t)x_in * a.qx_stride : nullptr;
    const int in_lag = take ? __ldg(a.ext_lag + e0 + tid) : 0;
    bool bad = false;
    uint64_t xv[S], xi[S];

    // what round r reads, S ticks from S * r
    auto fetch = [&](int r) {
        if (add_qout) {
            const int t0 = r * S - lag, h0 = (r & 1) * S;
            const unsigned dst = (unsigned)__cvta_generic_to_shared(&own_q[h0][tid]);
            auto get = [&](int j, const double *src) {
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + j * kRouteBlock * 8), "l"(src) : "memory");
            };
            if (t0 >= 0 && t0 + S <= nT && a.rdiv == 1) {
                if (bc_ok(BC_ROUTE_QOUT, t0 + S - 1, a.n_qsteps)) {
                    const double *src = qo + (size_t)t0 * L;
#pragma unroll
                    for (int j = 0; j < S; ++j, src += L) get(j, src);
                }
            } else if (t0 >= 0 && t0 + S <= nT) {
                const int row = t0 / a.rdiv;
                int left = (row + 1) * a.rdiv - t0; // steps that take this row
                if (bc_ok(BC_ROUTE_QOUT, (t0 + S - 1) / a.rdiv, a.n_qsteps)) {
                    const double *src = qo + (size_t)row * L;
#pragma unroll
                    for (int j = 0; j < S; ++j) {
                        get(j, src);
                        if (--left == 0) src += L, left = a.rdiv;
                    }
                }
            } else {
#pragma unroll 1
                for (int j = 0; j < S; ++j) {
                    const int t = t0 + j;
                    if ((unsigned)t >= (unsigned)nT) continue;
                    const int row = a.rdiv == 1 ? t : t / a.rdiv;
                    if (bc_ok(BC_ROUTE_QOUT, row, a.n_qsteps)) get(j, qo + (size_t)row * L);
                }
            }
        }
        if (take) {
            const int t0 = r * S - in_lag;
#pragma unroll
            for (int j = 0; j < S; ++j) {
                xv[j] = xi[j] = 0;
                if ((unsigned)(t0 + j) < (unsigned)nT) get_step(in + t0 + j, xv[j], xi[j]);
            }
        }
    };
    auto land = [&](int r) { // ... into shared memory: a tick reads the row of the tick before it
        if (take) {
            const int t0 = r * S - in_lag, h0 = (r & 1) * S;
#pragma unroll
            for (int j = 0; j < S; ++j) {
                const uint64_t id = a.done0 + (uint64_t)(t0 + j);
                if ((unsigned)(t0 + j) < (unsigned)nT && xi[j] != id && !bad)
                    bad = !wait_step(a, in + t0 + j, id, xv[j]);
                ring[(h0 + j - 1) & (2 * S - 1)][kRouteBlock + tid] = __longlong_as_double((long long)xv[j]);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    };
    // a node's steps follow one another from 0, so its pointers move with them
    longlong2 *out_t = out;
    uint64_t id_t = a.done0;
    // one tick; `k` its number, `i` its row of the ring
    auto tick = [&](int k, int i) {
        const double *row = ring[(i - 1) & (2 * S - 1)];
        const int t = k - lag;
        const double qo_t = own_q[i][tid];
        double q = row[up[0]];
        if (nu_warp > 1) {
            const double v1 = row[up[1]], v2 = row[up[2]];
            q = q + v1;
            if (nu_warp > 2) q = q + v2;
            if (nu_warp > 3) {
                q = q + row[up[3]];
                if (nu_warp > 4) {
                    q = q + row[up[4]];
                    if (nu_warp > 5) {
#pragma unroll
                        for (int u = 5; u < kRouteUps; ++u) q = q + row[up[u]];
                    }
                }
            }
        }
        if constexpr (HUB) {
            if (hub_warp) q = add_hubs(a, qx, hub, t, q, bad);
        }
        q = q + qo_t;
        // 0 + (-0) is +0: the sum starts at netNode_qTIN(:, IT) = 0
        q = hm_sel(hm_d2b(q) == 0x8000000000000000ULL, 0.0, q);
        const double keep = qtr1 + c1 * (qtin1 - qtr1);
        double qtr = keep + c2 * (q - qtin1);
        if (cut_warp) qtr = hm_sel(cut, 0.0, qtr);
        ring[i][tid] = qtr;
        if (out_warp && out) put_step(out_t, qtr, id_t);
        ++out_t;
        ++id_t;
        qtr1 = qtr;
        qtin1 = q;
        if (qmod_warp && keep_qmod) *qm = q; // L11_qMod = (0 + Qmod) / real(rout_loop = 1)
        qm += L;
    };
    if (tid < 2 * S) ring[tid][kZero] = 0.0;
#pragma unroll
    for (int i = 0; i < 2 * S; ++i) own_q[i][tid] = 0.0;
    fetch(0);
    land(0);
    if (__syncthreads_or(bad)) return;

    auto round = [&](int r, auto half) {
        constexpr int h0 = decltype(half)::value * S;
        if (r + 1 < rounds) fetch(r + 1);
        if (r * S >= lag_hi && (r + 1) * S - lag_lo <= nT) { // every node of the warp has a step in every tick
#pragma unroll
            for (int j = 0; j < S; ++j) {
                tick(r * S + j, h0 + j);
                if (j + 1 < S) __syncthreads();
            }
        } else {
#pragma unroll 1
            for (int j = 0; j < S; ++j) {
                const int k = r * S + j;
                if ((unsigned)(k - lag) < (unsigned)nT) tick(k, h0 + j);
                if (j + 1 < S) __syncthreads();
            }
        }
        if (r + 1 < rounds) land(r + 1);
        return __syncthreads_or(bad) != 0;
    };
    for (int r = 0; r < rounds; r += 2) {
        if (round(r, std::integral_constant<int, 0>())) return;
        if (r + 1 < rounds && round(r + 1, std::integral_constant<int, 1>())) return;
    }
    if (own) {
        a.qtin1[ms + pos] = qtin1;
        if (is_link) a.qtr1[ms + pos] = qtr1;
        if (a.qmod_last) a.qmod_last[ms + pos] = qtin1;
        if (a.qout_last) a.qout_last[ms + pos] = __ldg(qo + (size_t)(a.n_qsteps - 1) * L);
    }
}

__global__ void inflow_kernel(const InflowArgs a)
{
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= (int64_t)a.n_members * a.n_qsteps) return;
    const int m = (int)(gid / a.n_qsteps), s = (int)(gid - (int64_t)m * a.n_qsteps);
    int64_t tt0 = a.tt_base;
    if (a.member_step0) {
        const int32_t b = a.member_step0[m];
        if (b < 0) return; // idle member
        tt0 = (int64_t)b + a.step_shift + 1;
    }
    tt0 += (int64_t)s * a.win; // first model step of routing step s
    double *row = a.qout + ((size_t)m * a.n_qsteps + s) * a.n_nodes;
    // the days of this routing step (the host checks that the series covers the run)
    const int64_t d_first = (tt0 + a.steps_day - 1) / a.steps_day - a.day0;
    const int64_t d_last = (tt0 + (a.mean ? a.win - 1 : 0) + a.steps_day - 1) / a.steps_day - a.day0;
    if (!bc_ok(BC_INFLOW_DAY, d_first, a.n_days) || !bc_ok(BC_INFLOW_DAY, d_last, a.n_days)) return;
    for (int g = 0; g < a.n_inflow; ++g) {
        double Q;
        if (a.mean) {
            double acc = 0.0;
            for (int j = 0; j < a.win; ++j) {
                const int64_t day = (tt0 + j + a.steps_day - 1) / a.steps_day;
                acc = acc + __ldg(a.q + (size_t)(day - a.day0) * a.n_inflow + g);
            }
            Q = acc / a.tsf;
        } else {
            const int64_t day = (tt0 + a.steps_day - 1) / a.steps_day;
            Q = __ldg(a.q + (size_t)(day - a.day0) * a.n_inflow + g);
        }
        const int p = __ldg(a.pos + g);
        if (!bc_ok(BC_INFLOW_POS, p, a.n_nodes)) continue;
        double *v = row + p;
        *v = a.headwater[g] ? *v + Q : Q;
    }
}

// mhm_bounds_selftest: one failing test (index == extent) with no access
// behind it, so that the status path can be checked without any bad access
__global__ void bc_selftest_kernel(int n) { bc_ok(BC_SELFTEST, n, n); }

cudaError_t launch_bc_selftest(cudaStream_t s)
{
    bc_selftest_kernel<<<1, 1, 0, s>>>(7);
    return cudaGetLastError();
}

cudaError_t launch_inflow(const InflowArgs &a, cudaStream_t s)
{
    const int64_t n = (int64_t)a.n_members * a.n_qsteps;
    if (n == 0 || a.n_inflow == 0) return cudaSuccess;
    inflow_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(a);
    return cudaGetLastError();
}

__global__ void qmod_step_kernel(const QmodStepArgs a)
{
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t L = a.n_nodes;
    if (gid >= (int64_t)a.n_members * a.n_steps * L) return;
    const int pos = (int)(gid % L);
    const int64_t mt = gid / L;
    const int t = (int)(mt % a.n_steps), m = (int)(mt / a.n_steps);
    if (a.member_step0 && a.member_step0[m] < 0) return;
    const int64_t n_sub = (int64_t)a.n_steps * a.rdiv / a.win;
    const double *q = a.qmod_sub + (size_t)m * n_sub * L + pos;
    double v;
    if (a.rdiv > 1) {
        double acc = 0.0;
        for (int r = 0; r < a.rdiv; ++r) acc = acc + q[(size_t)(t * a.rdiv + r) * L];
        v = acc / (double)a.rdiv;
    } else {
        v = q[(size_t)(t / a.win) * L];
    }
    a.qmod[((size_t)m * a.n_steps + t) * L + pos] = v;
}

// mRM's Qrouted output (mRM_updateDataset / writeTimestep, called every model
// step after the warm-up: src/mHM/mo_mhm_interface_run.f90:651-668).  One
// thread per (member, node) walks the chunk's steps; with a routing step of
// `win` model steps the discharge state changes only at a window's last step.
__global__ void qrouted_kernel(const QroutArgs a)
{
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t L = a.n_nodes;
    if (gid >= (int64_t)a.n_members * L) return;
    const int pos = (int)(gid % L);
    const int m = (int)(gid / L);
    const size_t ML = (size_t)a.n_members * L;
    const double *q = a.qmod + (size_t)m * a.n_steps * L + pos;
    double acc = a.acc[(size_t)m * L + pos];
    int cnt = a.cnt0, slot = a.slot0;
    for (int t = 0; t < a.n_steps; ++t) {
        const int64_t tt = a.tt_base + t;
        if (tt <= a.warm_steps) continue;
        double v;
        if (a.win == 1 || (t + 1) % a.win == 0) v = q[(size_t)t * L];
        else if (t >= a.win) v = q[(size_t)((t / a.win) * a.win - 1) * L];
        else v = a.qmod_prev[(size_t)m * L + pos];
        acc = acc + v;
        ++cnt;
        if (out_writeout(a.interval, tt - a.warm_steps, tt, a.n_tt, step_dflags(a.jul_start, a.timestep, tt))) {
            if (slot < a.max_slots) a.out[(size_t)slot * ML + (size_t)m * L + pos] = acc / (double)cnt; // a mean
            acc = 0.0;
            cnt = 0;
            ++slot;
        }
    }
    a.acc[(size_t)m * L + pos] = acc;
}

// GaugeDischarge(gaugeIndexList) = L11_Qmod(gaugeNodeList), mo_mrm_routing.f90:299-301
__global__ void gauge_gather_kernel(const GaugeArgs a)
{
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t total = (int64_t)a.n_members * a.n_gauges * a.n_steps;
    if (gid >= total) return;
    const int t = (int)(gid % a.n_steps);
    const int64_t mg = gid / a.n_steps;
    const int g = (int)(mg % a.n_gauges);
    const int m = (int)(mg / a.n_gauges);
    const int gp = __ldg(a.gauge_pos + g);
    const double v = (a.member_step0 && a.member_step0[m] < 0) || !bc_ok(BC_GAUGE_POS, gp, a.n_nodes)
                         ? 0.0
                         : a.qmod[((size_t)m * a.n_steps + t) * a.n_nodes + gp];
    a.q_gauge[((size_t)m * a.n_gauges + g) * a.total_steps + a.step_offset + t] = v;
}

// reg_rout, src/mRM/mo_mrm_mpr.f90:61-119, one thread per link and member (the
// grid's second dimension; its parameters p5_stride after the previous one's);
// ss_max is the basin's max slope (parameter independent, computed on the host
// once).
__global__ void reg_rout_kernel(int n_links, int n_nodes, const double *p5, int p5_stride, double ss_max, double TS,
                                const double *length, const double *slope, const double *ffp,
                                const int32_t *link_pos, double *C1, double *C2)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_links) return;
    p5 += (size_t)blockIdx.y * p5_stride;
    const double p0 = p5[0], p1 = p5[1], p2 = p5[2], p3 = p5[3], p4 = p5[4];
    double K = p0 + p1 * (length[i] * 0.001) + p2 * slope[i] + p3 * ffp[i];
    double xi = p4 * (1.0 + slope[i] / ss_max);
    if (xi > 0.5) xi = 0.5;
    if (xi < 0.005) xi = 0.005;
    if (K > 0.5 * TS / xi) K = 0.5 * TS / xi;
    if (K < 0.5 * TS / (1.0 - xi)) K = 0.5 * TS / (1.0 - xi);
    const double c1 = TS / (K * (1.0 - xi) + 0.5 * TS);
    const size_t pos = (size_t)blockIdx.y * n_nodes + link_pos[i];
    C1[pos] = c1;
    C2[pos] = 1.0 - c1 * K / TS;
}

cudaError_t launch_runoff_acc(const AccArgs &a, cudaStream_t s)
{
    const int64_t n = (int64_t)a.n_steps * a.n_members * a.n_nodes;
    if (n == 0) return cudaSuccess;
    runoff_acc_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a);
    return cudaGetLastError();
}

// `round`: steps fetched ahead at a time, 1..16
cudaError_t launch_route_flow(const RouteArgs &a, int round, cudaStream_t s)
{
    if (a.n_members < 1 || a.n_steps < 1) return cudaSuccess;
    const unsigned grid = (unsigned)(a.n_blocks * a.n_members);
    if (round > 16) return cudaErrorInvalidValue;
    const auto kernel = a.n_hubs > 0 ? (round <= 4 ? route_flow_kernel<4, true> : route_flow_kernel<8, true>)
                                     : (round <= 4 ? route_flow_kernel<4, false> : route_flow_kernel<8, false>);
    kernel<<<grid, kRouteBlock, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_qmod_step(const QmodStepArgs &a, cudaStream_t s)
{
    const int64_t n = (int64_t)a.n_members * a.n_steps * a.n_nodes;
    if (n == 0) return cudaSuccess;
    qmod_step_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_qrouted(const QroutArgs &a, cudaStream_t s)
{
    const int64_t n = (int64_t)a.n_members * a.n_nodes;
    if (n == 0 || a.n_steps == 0) return cudaSuccess;
    qrouted_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_gauge_gather(const GaugeArgs &a, cudaStream_t s)
{
    const int64_t n = (int64_t)a.n_members * a.n_gauges * a.n_steps;
    if (n == 0) return cudaSuccess;
    gauge_gather_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_reg_rout(int n_members, int n_links, int n_nodes, const double *p5, int p5_stride, double ss_max,
                            double TS, const double *length, const double *slope, const double *ffp,
                            const int32_t *link_pos, double *C1, double *C2, cudaStream_t s)
{
    if (n_links <= 0 || n_members <= 0) return cudaSuccess;
    reg_rout_kernel<<<dim3((n_links + 127) / 128, n_members), 128, 0, s>>>(n_links, n_nodes, p5, p5_stride, ss_max, TS,
                                                                           length, slope, ffp, link_pos, C1, C2);
    return cudaGetLastError();
}

} // namespace mhm

MHM_BC_ACCESSOR(bc_take_routing)
