// integrate_fp64.cu -- the FP64 integrator and the FP64 collection of final states.
//
// Replaces, per electron, the ensemble solve
//   solve(EnsembleProblem(...), Tsit5(), EnsembleSerial(), reltol=traj_rtol)
// (src/TrajectorySimulation.jl:334-342, 3D :429-437) and the collection loop
// body (:344-397, 3D :439-497): retcode check, E_inf, SCTS post-pulse
// phase, Kepler asymptote, bin index and the deposit contribution.
//
// Tsit5 with OrdinaryDiffEq's defaults for `solve(prob, Tsit5(), reltol)`:
// abstol 1e-6, RMS error norm, PI controller (beta1 = 7/50, beta2 = 2/25,
// qmin = 1/5, qmax = 10, gamma = 9/10, qoldinit = 1e-4), Hairer's starting
// step, FSAL, t_final hit exactly.  Compiled with --fmad=false: every
// fused multiply-add is an explicit fma(), so the results are bit-identical
// to the CPU oracle's, and an electron's arithmetic does not depend on the lane,
// warp or kernel that carries it.
//
// What bounds it.  An FP64 warp instruction holds a sub-partition's issue port for 64
// to 76 cycles, whether one lane or 32 take part.  So the work is counted in FP64 warp
// instructions (fpint.h keeps divisions, roots, series and comparisons off that pipe;
// the laser is evaluated once for stages 6 and 7, which share their time), and there
// are two kernels for two loads:
//  * k_integrate_fp64, many electrons: one per lane, so a warp instruction serves 32.
//    Persistent; a lane that finishes takes the next electron from a queue, so step
//    counts that differ within a warp do not idle it.  FP64 operations per
//    attempt, so warp instructions of a full warp: 470 to 500 (hydrogen-like, 2D), 750 (an
//    SAE atom with a phase, 2D), 920 (3D).
//  * k_integrate_fp64_few, few electrons: eight lanes each.  The laser at an attempt's
//    five stage times (it does not depend on the state), the components' stage and
//    error sums and the controller's two powers run in parallel lanes: ~180 FP64
//    instructions per attempt, for 4 electrons per warp, and a third of the latency.
// The first kernel hands its last electrons to the second (kFewPerSm).
// Against one lane per electron in a static grid, with the same arithmetic: 1.9e5 Ar
// trajectories 20.7 -> 14.3 ms, 1.7e5 of H2 13.2 -> 7.6 ms, 1.1e5 H 18.6 -> 8.4 ms (their
// slowest takes 326 attempts), 1.2e3 H 14.8 -> 4.7 ms.

#include <algorithm>

#include "physics.cuh"

namespace etraj {
namespace {

constexpr double C2 = 0.161, C3 = 0.327, C4 = 0.9, C5 = 0.9800255409045097;
constexpr double A21 = 0.161;
constexpr double A31 = -0.008480655492356989, A32 = 0.335480655492357;
constexpr double A41 = 2.897153057105493, A42 = -6.359448489975075, A43 = 4.3622954328695815;
constexpr double A51 = 5.325864828439257, A52 = -11.748883564062828, A53 = 7.4955393428898365,
                 A54 = -0.09249506636175525;
constexpr double A61 = 5.86145544294642, A62 = -12.92096931784711, A63 = 8.159367898576159,
                 A64 = -0.071584973281401, A65 = -0.028269050394068383;
constexpr double A71 = 0.09646076681806523, A72 = 0.01, A73 = 0.4798896504144996,
                 A74 = 1.379008574103742, A75 = -3.290069515436081, A76 = 2.324710524099774;
constexpr double BT1 = -0.00178001105222577714, BT2 = -0.0008164344596567469,
                 BT3 = 0.007880878010261995, BT4 = -0.1447110071732629, BT5 = 0.5823571654525552,
                 BT6 = -0.45808210592918697, BT7 = 0.015151515151515152;
constexpr double ABSTOL = 1e-6, BETA1 = 0.14, BETA2 = 0.08, QMIN_INV = 5.0, QMAX_INV = 0.1,
                 GAMMA = 0.9, QOLDINIT = 1e-4;
constexpr long MAXITERS = 1000000L;

__device__ __forceinline__ double d_ulp(double x) {
    double a = fabs(x);
    uint64_t u = dm_d2u(a);
    int e = (int)(u >> 52);
    if (e == 0) return dm_u2d(1);
    if (e >= 2046) return dm_inf();
    int p = e - 1023 - 52;
    if (p >= -1022) return dm_pow2i(p);
    return dm_u2d(1ull << (p + 1074));
}
// Julia's min and max (NaN in, NaN out), compared on the integer pipe
__device__ __forceinline__ double jmin(double a, double b) {
    return (fi_isnan(a) || fi_isnan(b)) ? a + b : (fi_lt(a, b) ? a : b);
}
__device__ __forceinline__ double jmax(double a, double b) {
    return (fi_isnan(a) || fi_isnan(b)) ? a + b : (fi_lt(b, a) ? a : b);
}
// max(|a|, |b|), NaN if either is
__device__ __forceinline__ double max_abs(double a, double b) {
    const uint64_t m = 0x7fffffffffffffffull, i = fi_bits(a) & m, j = fi_bits(b) & m;
    return fi_real(i > j ? i : j);
}

__constant__ double cA[7][6] = {{0, 0, 0, 0, 0, 0},
                                {A21, 0, 0, 0, 0, 0},
                                {A31, A32, 0, 0, 0, 0},
                                {A41, A42, A43, 0, 0, 0},
                                {A51, A52, A53, A54, 0, 0},
                                {A61, A62, A63, A64, A65, 0},
                                {A71, A72, A73, A74, A75, A76}};
__constant__ double cC[5] = {0.0, C2, C3, C4, C5};
__constant__ double cBT[7] = {BT1, BT2, BT3, BT4, BT5, BT6, BT7};

// sum_j (v_j / sk_j)^2, j in order, to its root mean square
template <int N>
__device__ __forceinline__ double rms_of(double acc) {
    return DM_SQRT(N == 4 ? 0.25 * acc : DM_DIV(acc, (double)N));
}

// r^2 of a state, summed left to right
template <int DIM>
__device__ __forceinline__ double radius2(const double* u) {
    double r2 = u[0] * u[0] + u[1] * u[1];
    if (DIM == 3) r2 = r2 + u[2] * u[2];
    return r2;
}

// The clock and controller of one electron's solve.
struct Clock {
    double t, dt, dtpropose, lq, q11, dtmax, dtmin;  // lq: log(qold)
    int iter;   // attempts begun
    bool accept;
};

__device__ __forceinline__ void clock_start(Clock& c, double t0, double tf, double lq0) {
    c.t = t0;
    c.dtmax = tf - t0;
    c.dtmin = jmax(d_ulp(t0), d_ulp(tf));
    c.lq = lq0;
    c.q11 = 1.0;
    c.iter = 0;
    c.accept = false;
}

// The step size the next attempt starts from (the loop head's first lines).
__device__ __forceinline__ double next_dt(const Clock& c) {
    if (c.iter == 0) return c.dt;
    return c.accept ? c.dtpropose : DM_DIV(c.dt, jmin(QMIN_INV, DM_DIV(c.q11, GAMMA)));
}

// t < t_final (false for NaN)
__device__ __forceinline__ bool before(double t, double tf) { return !fi_isnan(t) && fi_lt(t, tf); }

// Start of an attempt with step c.dt = next_dt: a status above 0 ends the solve.
__device__ __forceinline__ int attempt_begin(Clock& c, double tf) {
    ++c.iter;
    c.dt = jmin(c.dtmax, c.dt);
    c.dt = jmax(c.dt, jmax(c.dtmin, d_ulp(c.t)));
    c.dt = jmin(c.dt, tf - c.t);
    if (fi_isnan(c.dt)) return 4;
    if (c.iter > MAXITERS) return 1;
    if (!fi_lt(c.dtmin, c.dt) && (!c.accept || fi_lt(c.t + c.dt, tf))) return 2;
    return 0;
}

// The two powers of the PI controller, EEst^beta1 and qold^beta2 = exp(beta2 log qold);
// the log of EEst serves as the next attempt's log qold.
struct Powers {
    double lE, x1, x2;
};
__device__ __forceinline__ Powers power_args(const Clock& c, double EEst) {
    Powers p;
    p.lE = dm_log(EEst);
    p.x1 = BETA1 * p.lE;
    p.x2 = BETA2 * c.lq;
    return p;
}
// End of an attempt that reached t1 = t + dt: acceptance and the next step proposed.
// snap: 100 ulp of t_final, within which the solve ends.
__device__ __forceinline__ void attempt_end(Clock& c, double EEst, double lE, double e1, double e2, double t1, double tf,
                                            double snap, double lq0) {
    double q = QMAX_INV;
    if (!fi_iszero(EEst)) {
        c.q11 = e1;
        q = jmax(QMAX_INV, jmin(QMIN_INV, DM_DIV(DM_DIV(e1, e2), GAMMA)));
    }
    c.accept = fi_bits(EEst) <= 0x3ff0000000000000ull;  // EEst <= 1 (EEst >= 0 or NaN)
    if (c.accept) {
        c.lq = fi_lt(QOLDINIT, EEst) ? lE : lq0;
        c.t = (fi_bits(fabs(t1 - tf)) < fi_bits(snap)) ? tf : t1;
        c.dtpropose = jmax(jmin(c.dtmax, DM_DIV(c.dt, q)), c.dtmin);
    }
}

// Hairer's starting step: dt0 from d0, d1, then dt from d1 and d2.
__device__ __forceinline__ double start_dt0(double d0, double d1, double dtmax) {
    const double dt0 = (d0 < 1e-5 || d1 < 1e-5) ? 1e-6 : DM_DIV(DM_DIV(d0, d1), 100.0);
    return jmin(dt0, dtmax);
}
__device__ __forceinline__ double start_dt(double d1, double d2, double dt0, double dtmax, double dtmin) {
    const double md = jmax(d1, d2);
    double dt1;
    if (md <= 1e-15) dt1 = jmax(1e-6, dt0 * 1e-3);
    else dt1 = dm_pow_pos(10.0, DM_DIV(-(2.0 + DM_DIV(dm_log(md), DM_LN10)), 5.0));
    return jmax(dtmin, jmin(jmin(100.0 * dt0, dt1), dtmax));
}

// An electron's initial state, or the state it was handed over with (below).
template <int DIM, int PHASE>
__device__ __forceinline__ double load_component(const InitSoA& soa, const TrajOut& out, int64_t g, int64_t s, int j,
                                                 bool resume) {
    if (j == 0) return soa.x[g];
    if (j == 1) return soa.y[g];
    if (DIM == 3 && j == 2) return resume ? out.c_im[s] : 0.0;
    const int k = j - DIM;
    if (k == 0) return soa.kx[g];
    if (k == 1) return soa.ky[g];
    if (DIM == 3 && k == 2) return soa.kz[g];
    return (PHASE != ETRAJ_PHASE_CTMC) ? soa.phase[g] : 0.0;
}
// The same places hold the final state where out.final_state is not asked for: the
// initial state is not read again, and the collection writes c_im afterwards.
template <int DIM, int PHASE>
__device__ __forceinline__ void store_component(const InitSoA& soa, const TrajOut& out, int64_t g, int64_t s, int j,
                                                double v) {
    const int k = j - DIM;
    if (j == 0) soa.x[g] = v;
    else if (j == 1) soa.y[g] = v;
    else if (DIM == 3 && j == 2) out.c_im[s] = v;
    else if (k == 0) soa.kx[g] = v;
    else if (k == 1) soa.ky[g] = v;
    else if (DIM == 3 && k == 2) soa.kz[g] = v;
    else if (PHASE != ETRAJ_PHASE_CTMC) soa.phase[g] = v;
}

// An electron between two attempts that goes to the second kernel: its state where the
// final state would go, its clock in the outputs the collection has yet to write, its
// index in the list (out.key).  FSAL's derivative is evaluated again there, with the
// same bits.
__device__ __forceinline__ void hand_over(const Clock& c, const TrajOut& out, int64_t s, double r2min) {
    // (the attempt just begun has not been made: its head runs again, on the step as it stands)
    out.c_re[s] = c.t;
    out.w_ion[s] = c.dt;
    out.w_unc[s] = c.lq;
    out.steps[s] = c.iter - 1;
    out.status[s] = c.accept ? 1 : 0;
    if (out.rmin) out.rmin[s] = r2min;
}
__device__ __forceinline__ void take_over(Clock& c, const TrajOut& out, int64_t s, double t0, double tf) {
    clock_start(c, t0, tf, 0.0);
    c.t = out.c_re[s];
    c.dt = out.w_ion[s];
    c.lq = out.w_unc[s];
    c.iter = out.steps[s];
    c.accept = out.status[s] != 0;
}

// Counters of the two kernels in `work`: the first's queue, electrons it has finished,
// electrons handed over, the second's queue.
enum { kQueue = 0, kFinished = 1, kHanded = 2, kQueueFew = 3 };

__device__ __forceinline__ void cross3(const double* a, const double* b, double* c) {
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
}

// Collection of one electron (TrajectorySimulation.jl:356-393, 3D :451-493).
// Returns true when the electron is finally ionized (E_inf >= 0).
template <int DIM, int PHASE, int N>
__device__ __forceinline__ bool collect(const DJob& J, int status, const double* f, double tr,
                                        double prob, const TrajOut& out, int64_t s) {
    uint32_t key = (uint32_t)J.grid;
    double cre = 0.0, cim = 0.0, wion = 0.0, wunc = 0.0;
    double pin[3] = {0.0, 0.0, 0.0};
    double phase_out = 0.0;
    bool ionized = false;
    if (status == 0) {
        double x, y, z, px, py, pz, K;
        if (DIM == 2) {
            x = f[0]; y = f[1]; z = 0.0; px = f[2]; py = f[3]; pz = 0.0;
            K = (px * px + py * py) / 2.0;
        } else {
            x = f[0]; y = f[1]; z = f[2]; px = f[3]; py = f[4]; pz = f[5];
            K = ((px * px + py * py) + pz * pz) / 2.0;
        }
        double phase = (PHASE == ETRAJ_PHASE_CTMC) ? 0.0 : f[N - 1];
        double E = K + target_V(J.target, x, y, z);
        double rv[3] = {x, y, z}, pv[3] = {px, py, pz}, L[3];
        cross3(rv, pv, L);
        double L2 = (L[0] * L[0] + L[1] * L[1]) + L[2] * L[2];
        const double Z = J.target.Z;
        if (PHASE == ETRAJ_PHASE_SCTS && E > 0.0) {
            phase = phase + J.target.Ip * tr;
            double sqrtb = DM_DIV(1.0, DM_SQRT(2.0 * E));
            double g = DM_SQRT(1.0 + (2.0 * E) * L2);
            // the 3D reference uses x*py where x*px is meant (TrajectorySimulation.jl:463)
            double rp = (DIM == 2) ? (x * px + y * py) : ((x * py + y * py) + z * pz);
            phase = phase - (Z * sqrtb) * (dm_log(g) + dm_asinh(DM_DIV(rp, g * sqrtb)));
        }
        phase_out = phase;
        if (E >= 0.0) {
            ionized = true;
            wion = prob;
            double pinf = DM_SQRT(2.0 * E);
            double nr = DM_SQRT((x * x + y * y) + z * z);
            double pL[3], a[3], La[3];
            cross3(pv, L, pL);
#pragma unroll
            for (int i = 0; i < 3; ++i) a[i] = pL[i] - DM_DIV(Z * rv[i], nr);
            cross3(L, a, La);
            double fac = DM_DIV(pinf, 1.0 + (pinf * pinf) * L2);
#pragma unroll
            for (int i = 0; i < 3; ++i) pin[i] = fac * (pinf * La[i] - a[i]);
            int64_t lin = 0, stride = 1;
            bool ok = true;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                int64_t num = J.pnum[d], ix = 1;
                if (num > 1) {
                    double pm = J.pmax[d];
                    double v = rint(DM_DIV(pin[d] + pm, J.binw[d]));
                    if (!(v >= 1.0 && v <= (double)num)) ok = false;
                    else ix = (int64_t)v;
                }
                lin += (ix - 1) * stride;
                stride *= num;
            }
            if (ok) {
                key = (uint32_t)lin;
                if (PHASE == ETRAJ_PHASE_CTMC) {
                    cre = prob;
                } else {
                    double sp = DM_SQRT(prob), sn, cs;
                    dm_sincos(phase, &sn, &cs);
                    cre = sp * cs;
                    cim = sp * sn;
                }
            } else {
                wunc = prob;
            }
        }
    }
    out.key[s] = key;
    out.c_re[s] = cre;
    out.c_im[s] = cim;
    out.w_ion[s] = wion;
    out.w_unc[s] = wunc;
    if (out.p_inf) {
        out.p_inf[3 * s] = pin[0];
        out.p_inf[3 * s + 1] = pin[1];
        out.p_inf[3 * s + 2] = pin[2];
    }
    if (out.fphase) out.fphase[s] = phase_out;
    return ionized;
}

constexpr int kThreads = 128;
constexpr int kRefill = 4;  // free lanes a warp waits for before it takes new electrons

template <int DIM, int PHASE>
constexpr int state_size() {
    return 2 * DIM + (PHASE != ETRAJ_PHASE_CTMC ? 1 : 0);
}

// One electron per lane.  A warp goes through the stages in step: stage st = 1..6 of
// every stepping lane, one evaluation of the right-hand side per turn; new electrons
// use the first two turns of an attempt for their starting step.  The stage
// derivatives are in shared memory (7 N doubles per lane).
// The loop body is larger than the instruction cache: with four and five warps per
// sub-partition a third of the time between a warp's instructions went to fetching.  So
// above two a block's warps go through the turns in step, a barrier at each, and share what
// they fetch: 15.0 -> 14.3 ms on 1.9e5 Ar, 7.9 -> 7.6 on 1.7e5 H2.  With two (3.0e4 Ne) the
// barrier costs more than it saves (a call 4.0 -> 4.2 ms).
// Blocks per SM, which sets the register budget (102 a thread for 5): with 4 the warps waited
// for instructions and results more of the time.  5 against 4:
// 17.2 -> 15.4 ms on 1.9e5 Ar (N = 5), 8.45 -> 8.07 on 1.7e5 H2 (N = 4); 6 spills: 17.6 and 9.0.
// At N = 7 the stage derivatives (7 N doubles per thread) leave room for 4.
template <int N>
constexpr int resident_blocks() {
    return N <= 6 ? 5 : 4;
}
template <int DIM, int PHASE, int TGT>
__global__ void __launch_bounds__(kThreads, resident_blocks<state_size<DIM, PHASE>()>())
k_integrate_fp64(const __grid_constant__ DJob J, InitSoA soa, const double* __restrict__ tsamp,
                 const int64_t* __restrict__ idx, const unsigned long long* __restrict__ count,
                 unsigned long long* __restrict__ work, TrajOut out, long long few, int one_per_warp) {
    constexpr int N = state_size<DIM, PHASE>();
    const long long n = (long long)(*count);
    if (n <= few) return;  // all of them go to the other kernel
    // as many warps per sub-partition, the same on all, as the electrons fill, and an even
    // share of the electrons for each
    const long long all = (long long)gridDim.x * (kThreads / 32);
    const long long used = min(all, one_per_warp * ((n + 32ll * one_per_warp - 1) / (32ll * one_per_warp)));
    if ((long long)blockIdx.x * (kThreads / 32) >= used) return;
    const int lanes = (int)min(32ll, (n + used - 1) / used);
    const bool in_step = used > 2ll * one_per_warp;
    extern __shared__ double s_K[];
    double* const K = s_K + threadIdx.x;
    auto slot = [&](int l, int j) -> double& { return K[(l * N + j) * kThreads]; };
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    const double tf = J.t_final, snap = 100.0 * d_ulp(tf), lq0 = dm_log(QOLDINIT);

    enum { kFree, kBase, kInit, kWait, kStep };
    int mode = kFree;
    bool drained = (long long)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5) >= used;
    long long s = 0, g = 0;
    double u[N], w[N];  // accepted state; state to evaluate (at st = 6: the new state)
    double Fx = 0.0, Fy = 0.0, tl = 0.0, d1 = 0.0, r2min = 0.0;
    Clock c = {};

    auto finish = [&](int status) {
        out.status[s] = status;
        out.steps[s] = c.iter - (status ? 1 : 0);  // (a failed solve ends at the head of an attempt)
        if (out.rmin) out.rmin[s] = DM_SQRT(r2min);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            if (out.final_state) out.final_state[s * N + j] = u[j];
            else store_component<DIM, PHASE>(soa, out, g, s, j, u[j]);
        }
        mode = kFree;
    };

    for (int st = 1;; st = (st == 6) ? 1 : st + 1) {
        if (in_step && st != 1) {
            __syncwarp();  // (lanes without an evaluation left the turn early)
            __syncthreads();
        }
        if (st == 1) {
            const bool had = mode != kFree;
            if (mode == kWait) mode = kStep;
            if (mode == kStep) {
                // the electron just advanced may be done (t = t_final) or not a number
                if (!before(c.t, tf)) {
                    finish(0);
                } else {
                    bool bad = false;
#pragma unroll
                    for (int j = 0; j < N; ++j) bad |= fi_isnan(u[j]) != 0;
                    c.dt = next_dt(c);
                    const int status = attempt_begin(c, tf);
                    if (status) finish(status);
                    else if (c.accept && bad) finish(3);
                }
            }
            const unsigned done = __ballot_sync(FULL, had && mode == kFree);
            if (done && lane == 0) atomicAdd(work + kFinished, (unsigned long long)__popc(done));
            const unsigned freem = __ballot_sync(FULL, mode == kFree && lane < lanes);
            if (!drained && (__popc(freem) >= kRefill || __popc(freem) == lanes)) {
                const int leader = __ffs(freem) - 1;
                unsigned long long base = 0ull;
                if (lane == leader) base = atomicAdd(work + kQueue, (unsigned long long)__popc(freem));
                base = __shfl_sync(FULL, base, leader);
                drained = (long long)base + __popc(freem) >= n;
                if (mode == kFree && lane < lanes) {
                    s = (long long)base + __popc(freem & lt_mask);
                    if (s < n) {
                        g = idx ? idx[s] : s;
                        clock_start(c, tsamp[soa.batch[g]], tf, lq0);
#pragma unroll
                        for (int j = 0; j < N; ++j) u[j] = w[j] = load_component<DIM, PHASE>(soa, out, g, s, j, false);
                        if (out.rmin) r2min = radius2<DIM>(u);
                        mode = kBase;
                    }
                }
            } else if (!drained) {
                // a warp with too few free lanes to ask the queue looks at it, so that its last
                // electrons can leave too (31 of 32 slow ones: a call of 177 -> 79 ms)
                unsigned long long taken = 0ull;
                if (lane == 0) taken = *(volatile unsigned long long*)(work + kQueue);
                drained = (long long)__shfl_sync(FULL, taken, 0) >= n;
            }
            if (drained && __ballot_sync(FULL, mode != kFree) != 0u) {
                // the queue is empty: once few electrons are left in all, the others go to
                // the second kernel, which has no use for full warps
                unsigned long long fin = 0ull;
                if (lane == 0) fin = *(volatile unsigned long long*)(work + kFinished);
                fin = __shfl_sync(FULL, fin, 0);
                if (n - (long long)fin <= few) {
                    const bool leave = mode == kStep;
                    const unsigned lm = __ballot_sync(FULL, leave);
                    unsigned long long k0 = 0ull;
                    if (lane == 0 && lm) k0 = atomicAdd(work + kHanded, (unsigned long long)__popc(lm));
                    k0 = __shfl_sync(FULL, k0, 0);
                    if (leave) {
                        hand_over(c, out, s, r2min);
                        out.key[k0 + __popc(lm & lt_mask)] = (uint32_t)s;
#pragma unroll
                        for (int j = 0; j < N; ++j) store_component<DIM, PHASE>(soa, out, g, s, j, u[j]);
                        mode = kFree;
                    }
                }
            }
            __syncwarp();  // (some lanes just handed an electron over, or took one)
            // (in step, the block leaves together)
            if (!(in_step ? __syncthreads_or(mode != kFree) != 0 : __ballot_sync(FULL, mode != kFree) != 0u)) break;
        }
        // ---- this turn's evaluation -----------------------------------------------------------
        if (mode == kStep) {
#pragma unroll
            for (int j = 0; j < 2 * DIM; ++j) w[j] = cA[st][0] * slot(0, j);
#pragma unroll 1
            for (int l = 1; l < st; ++l) {
                const double a = cA[st][l];
#pragma unroll
                for (int j = 0; j < 2 * DIM; ++j) w[j] = fma(a, slot(l, j), w[j]);
            }
#pragma unroll
            for (int j = 0; j < 2 * DIM; ++j) w[j] = fma(c.dt, w[j], u[j]);
            if (N > 2 * DIM && st == 6) {  // the phase enters no derivative: its sum is needed here only
                double a = A71 * slot(0, N - 1);
#pragma unroll
                for (int l = 1; l < 6; ++l) a = fma(cA[6][l], slot(l, N - 1), a);
                w[N - 1] = fma(c.dt, a, u[N - 1]);
            }
            tl = (st < 5) ? fma(cC[st], c.dt, c.t) : c.t + c.dt;
        } else {
            tl = (mode == kInit) ? c.t + c.dt : c.t;
        }
        if (mode == kFree || mode == kWait) continue;  // (to the barrier)
        if (!(mode == kStep && st == 6)) laser_F<false>(J.laser, tl, Fx, Fy);  // stage 7 is at stage 6's time
        double du[N];
        rhs_at<DIM, PHASE, TGT>(J, Fx, Fy, w, du);
        if (mode == kStep) {
#pragma unroll
            for (int j = 0; j < N; ++j) slot(st, j) = du[j];
            if (st == 6) {
                double acc = 0.0;
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    double e = BT1 * slot(0, j);
#pragma unroll
                    for (int l = 1; l < 6; ++l) e = fma(cBT[l], slot(l, j), e);
                    e = fma(BT7, du[j], e);
                    const double r = DM_DIV(c.dt * e, fma(max_abs(u[j], w[j]), J.rtol, ABSTOL));
                    acc = fma(r, r, acc);
                }
                const double EEst = rms_of<N>(acc);
                const Powers p = power_args(c, EEst);
                attempt_end(c, EEst, p.lE, dm_exp(p.x1), dm_exp(p.x2), tl, tf, snap, lq0);
                if (c.accept) {
#pragma unroll
                    for (int j = 0; j < N; ++j) {
                        u[j] = w[j];
                        slot(0, j) = du[j];
                    }
                    if (out.rmin) r2min = jmin(r2min, radius2<DIM>(u));
                }
            }
        } else {
            double a0 = 0.0, a1 = 0.0;
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const double sk = fma(fabs(u[j]), J.rtol, ABSTOL);
                if (mode == kBase) {
                    slot(0, j) = du[j];
                    const double q = DM_DIV(u[j], sk), r = DM_DIV(du[j], sk);
                    a0 = fma(q, q, a0);
                    a1 = fma(r, r, a1);
                } else {
                    const double r = DM_DIV(du[j] - slot(0, j), sk);
                    a1 = fma(r, r, a1);
                }
            }
            if (mode == kBase) {
                d1 = rms_of<N>(a1);
                c.dt = start_dt0(rms_of<N>(a0), d1, c.dtmax);
                if (c.dt < 10.0 * 2.220446049250313e-16) {
                    c.dt = 1e-6;
                    mode = kWait;
                } else {
#pragma unroll
                    for (int j = 0; j < N; ++j) w[j] = fma(c.dt, du[j], u[j]);
                    mode = kInit;
                }
            } else {
                c.dt = start_dt(d1, DM_DIV(rms_of<N>(a1), c.dt), c.dt, c.dtmax, c.dtmin);
                mode = kWait;
            }
        }
    }
}

// Eight lanes per electron, four electrons per warp: lane j of a group holds component j
// of the state and its seven stage derivatives; every lane of a group evaluates the
// target, the same values in all of them.
template <int DIM, int PHASE, int TGT>
__global__ void __launch_bounds__(kThreads, 4)
k_integrate_fp64_few(const __grid_constant__ DJob J, InitSoA soa, const double* __restrict__ tsamp,
                     const int64_t* __restrict__ idx, const unsigned long long* __restrict__ count,
                     unsigned long long* __restrict__ work, TrajOut out, long long few, int one_per_warp) {
    constexpr int N = state_size<DIM, PHASE>();
    const long long n_all = (long long)(*count);
    const bool resume = n_all > few;  // electrons handed over, else all of them
    const long long n = resume ? (long long)work[kHanded] : n_all;
    const int lane = threadIdx.x & 31, base = lane & 24, j = (lane & 7) < N ? (lane & 7) : N - 1;
    const unsigned gm = 0xffu << base;
    // while electrons are fewer than one per sub-partition and group, spread them over warps
    const int groups = (int)min((n + one_per_warp - 1) / one_per_warp, 4ll);
    const long long gid = ((long long)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5)) * groups + (base >> 3);
    const long long n_groups = (long long)gridDim.x * (kThreads / 32) * groups;
    if ((base >> 3) >= groups) return;
    const double tf = J.t_final, snap = 100.0 * d_ulp(tf), lq0 = dm_log(QOLDINIT);
    auto from = [&](double v, int lane_in_group) { return __shfl_sync(gm, v, base + lane_in_group); };
    auto sum_squares = [&](double q) {
        double acc = 0.0;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const double v = from(q, i);
            acc = fma(v, v, acc);
        }
        return acc;
    };
    // Derivative of component j at the state whose components the group's lanes hold: rhs_at
    // (physics.cuh) with its exponentials, and its divisions, in parallel lanes.
    auto rhs_of = [&](double Fx, double Fy, double v) {
        const DTarget& Tg = J.target;
        const int m = lane & 7;
        double w[N];
#pragma unroll
        for (int i = 0; i < N; ++i) w[i] = from(v, i);
        double r2 = w[0] * w[0] + w[1] * w[1];
        if (DIM == 3) r2 = r2 + w[2] * w[2];
        double coef, Vphase = 0.0;
        if (TGT == ETRAJ_TARGET_HYDROGEN_LIKE) {
            const double q = r2 + Tg.sc, rs = DM_SQRT(q);
            const double inv = DM_DIV(1.0, (m == 1) ? rs : q * rs);
            coef = (-Tg.Z) * from(inv, 0);
            if (PHASE != ETRAJ_PHASE_CTMC) Vphase = Tg.Z * from(inv, 1);
        } else {
            const double r = DM_SQRT(r2);
            const double q = r * r + Tg.sc, rs = DM_SQRT(q);
            const double ex = sae_exp(Tg, m == 0 ? Tg.b1 : m == 1 ? Tg.b2 : Tg.b3, r);
            const double e1 = from(ex, 0), e2 = from(ex, 1), e3 = from(ex, 2);
            const double br = (Tg.Z + (Tg.a1 * (1.0 + Tg.b1 * r)) * e1) + (Tg.a3 * (1.0 + Tg.b3 * r)) * e3;
            const double num = ((Tg.Z + Tg.a1 * e1) + (Tg.a2 * r) * e2) + Tg.a3 * e3;
            const double top = m == 0 ? 1.0 : m == 1 ? Tg.a2 * Tg.b2 : num;
            const double bot = m == 0 ? q * rs : (m == 2 && DIM == 2 && PHASE == ETRAJ_PHASE_SCTS) ? q : rs;
            const double quot = DM_DIV(top, bot);
            coef = -(from(quot, 0) * br + from(quot, 1) * e2);
            if (PHASE != ETRAJ_PHASE_CTMC) Vphase = from(quot, 2);
        }
        // a position's derivative is its momentum, a momentum's the force
        double x = w[0], p = w[DIM];
#pragma unroll
        for (int i = 1; i < DIM; ++i) {
            x = (j == DIM + i) ? w[i] : x;
            p = (j == i) ? w[DIM + i] : p;
        }
        double d = coef * x;
        if (j == DIM) d = d - Fx;
        if (j == DIM + 1) d = d - Fy;
        if (j < DIM) d = p;
        if (PHASE != ETRAJ_PHASE_CTMC) {
            const double tFx = coef * w[0], tFy = coef * w[1];
            double K = w[DIM] * w[DIM] + w[DIM + 1] * w[DIM + 1], W = w[0] * tFx + w[1] * tFy;
            if (DIM == 3) {
                K = K + w[5] * w[5];
                W = W + w[2] * (coef * w[2]);
            }
            K = K / 2.0;
            if (j == 2 * DIM) d = (PHASE == ETRAJ_PHASE_QTMC) ? -((Tg.Ip + K) - Vphase) : -((K - Vphase) + W);
        }
        return d;
    };

    long long e = gid, s = 0, g = 0;
    bool active = false, first = true;
    double u = 0.0, K0 = 0.0, r2min = 0.0, Fx, Fy;
    Clock c = {};
    auto r2_of = [&](double v) {
        const double x[3] = {from(v, 0), from(v, 1), DIM == 3 ? from(v, 2) : 0.0};
        return radius2<DIM>(x);
    };
    for (;;) {
        if (!active) {
            if (e >= n) break;
            s = resume ? (long long)out.key[e] : e;
            g = idx ? idx[s] : s;
            const double t0 = tsamp[soa.batch[g]];
            u = load_component<DIM, PHASE>(soa, out, g, s, j, resume);
            if (resume) {
                take_over(c, out, s, t0, tf);
                if (out.rmin) r2min = out.rmin[s];
            } else {
                clock_start(c, t0, tf, lq0);
                if (out.rmin) r2min = r2_of(u);
            }
            laser_F<false>(J.laser, c.t, Fx, Fy);
            K0 = rhs_of(Fx, Fy, u);
            if (!resume) {
                const double sk = fma(fabs(u), J.rtol, ABSTOL);
                const double d0 = rms_of<N>(sum_squares(DM_DIV(u, sk))), d1 = rms_of<N>(sum_squares(DM_DIV(K0, sk)));
                const double dt0 = start_dt0(d0, d1, c.dtmax);
                if (dt0 < 10.0 * 2.220446049250313e-16) {
                    c.dt = 1e-6;
                } else {
                    laser_F<false>(J.laser, t0 + dt0, Fx, Fy);
                    const double f1 = rhs_of(Fx, Fy, fma(dt0, K0, u));
                    c.dt = start_dt(d1, DM_DIV(rms_of<N>(sum_squares(DM_DIV(f1 - K0, sk))), dt0), dt0, c.dtmax, c.dtmin);
                }
            }
            active = first = true;
        }
        int status = -1;  // -1: at t_final
        if (before(c.t, tf)) {
            if (!first) c.dt = next_dt(c);
            first = false;
            status = attempt_begin(c, tf);
            const bool bad = __any_sync(gm, fi_isnan(u) != 0);
            if (status == 0 && c.accept && bad) status = 3;
        }
        if (status != 0) {
            if ((lane & 7) < N) {
                if (out.final_state) out.final_state[s * N + j] = u;
                else store_component<DIM, PHASE>(soa, out, g, s, j, u);
            }
            unsigned long long q = 0ull;
            if ((lane & 7) == 0) {
                out.status[s] = status < 0 ? 0 : status;
                out.steps[s] = c.iter - (status > 0 ? 1 : 0);
                if (out.rmin) out.rmin[s] = DM_SQRT(r2min);
                q = atomicAdd(work + kQueueFew, 1ull);
            }
            e = n_groups + (long long)__shfl_sync(gm, q, base);
            active = false;
            continue;
        }
        // the laser at the five stage times, one per lane
        const int m = lane & 7;
        double fx, fy;
        laser_F<false>(J.laser, (m < 4) ? fma(cC[m + 1], c.dt, c.t) : c.t + c.dt, fx, fy);
        // (a loop over the stages, its derivatives selected by index, is smaller code and was
        // slower: 5.4 against 5.0 ms on 1248 electrons)
        double K1, K2, K3, K4, K5, K6, w, a;
        w = fma(c.dt, A21 * K0, u);
        K1 = rhs_of(from(fx, 0), from(fy, 0), w);
        a = fma(A32, K1, A31 * K0);
        w = fma(c.dt, a, u);
        K2 = rhs_of(from(fx, 1), from(fy, 1), w);
        a = fma(A43, K2, fma(A42, K1, A41 * K0));
        w = fma(c.dt, a, u);
        K3 = rhs_of(from(fx, 2), from(fy, 2), w);
        a = fma(A54, K3, fma(A53, K2, fma(A52, K1, A51 * K0)));
        w = fma(c.dt, a, u);
        K4 = rhs_of(from(fx, 3), from(fy, 3), w);
        a = fma(A65, K4, fma(A64, K3, fma(A63, K2, fma(A62, K1, A61 * K0))));
        w = fma(c.dt, a, u);
        Fx = from(fx, 4);  // stage 7 is at stage 6's time
        Fy = from(fy, 4);
        K5 = rhs_of(Fx, Fy, w);
        a = fma(A76, K5, fma(A75, K4, fma(A74, K3, fma(A73, K2, fma(A72, K1, A71 * K0)))));
        w = fma(c.dt, a, u);
        K6 = rhs_of(Fx, Fy, w);
        a = fma(BT7, K6, fma(BT6, K5, fma(BT5, K4, fma(BT4, K3, fma(BT3, K2, fma(BT2, K1, BT1 * K0))))));
        const double r = DM_DIV(c.dt * a, fma(max_abs(u, w), J.rtol, ABSTOL));
        const double EEst = rms_of<N>(sum_squares(r));
        const Powers p = power_args(c, EEst);
        const double ex = dm_exp((lane & 1) ? p.x2 : p.x1);  // both powers in one pass
        attempt_end(c, EEst, p.lE, from(ex, 0), from(ex, 1), c.t + c.dt, tf, snap, lq0);
        if (c.accept) {
            u = w;
            K0 = K6;
            if (out.rmin) r2min = jmin(r2min, r2_of(u));
        }
    }
}

// The collection of the final states (out.final_state, or where the FP64 kernels leave
// them).
template <int DIM, int PHASE>
__global__ void __launch_bounds__(128)
k_collect_fp64(const __grid_constant__ DJob J, InitSoA soa, const double* __restrict__ tsamp,
               const int64_t* __restrict__ idx, const unsigned long long* __restrict__ count,
               TrajOut out) {
    constexpr int N = state_size<DIM, PHASE>();
    const int64_t n = (int64_t)(*count);
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n;
         s += (int64_t)gridDim.x * blockDim.x) {
        const int64_t g = idx ? idx[s] : s;
        double f[N];
#pragma unroll
        for (int j = 0; j < N; ++j)
            f[j] = out.final_state ? out.final_state[s * N + j] : load_component<DIM, PHASE>(soa, out, g, s, j, true);
        const int st = out.status[s] & 0xff;
        const bool ion = collect<DIM, PHASE, N>(J, st, f, tsamp[soa.batch[g]], soa.rate[g], out, s);
        out.status[s] = st | (ion ? 0x100 : 0);
    }
}

// Electrons per SM below which the second kernel takes over (7,296 on 152 SMs).  The second costs 3 to 4 times the pipe time per electron:
// with all 30,011 electrons of a Ne job in it, 14.7 ms against 4.0; at 1,248 hydrogen
// electrons with up to 347 attempts, 5.0 ms against 14.8 in the first.  16, 32, 48 and 80 measured
// the same on jobs of 3e4 to 2e5 electrons, 160 5 % more.
constexpr int kFewPerSm = 48;

template <int DIM, int PHASE, int TGT>
int launch_t(const DJob& J, InitSoA soa, const double* t, const int64_t* idx,
             const unsigned long long* count, unsigned long long* work, TrajOut out, int64_t max_n, int sm_count,
             cudaStream_t s) {
    constexpr size_t smem = (size_t)7 * state_size<DIM, PHASE>() * kThreads * sizeof(double);
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(k_integrate_fp64<DIM, PHASE, TGT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    constexpr int warps = kThreads / 32;
    const int64_t grid = (int64_t)sm_count * resident_blocks<state_size<DIM, PHASE>()>(), grid_few = (int64_t)sm_count * 4;
    const long long few = (long long)sm_count * kFewPerSm;
    cudaMemsetAsync(work, 0, 4 * sizeof(unsigned long long), s);
    int launches = 1;
    if (max_n > few) {
        const int64_t want = (max_n + kThreads - 1) / kThreads;
        k_integrate_fp64<DIM, PHASE, TGT><<<(unsigned)std::min(want, grid), kThreads, smem, s>>>(
            J, soa, t, idx, count, work, out, few, sm_count * warps);
        ++launches;
    }
    const int64_t want = (max_n + warps - 1) / warps;  // as many warps as electrons at most
    k_integrate_fp64_few<DIM, PHASE, TGT><<<(unsigned)std::max<int64_t>(1, std::min(want, grid_few)), kThreads, 0, s>>>(
        J, soa, t, idx, count, work, out, few, sm_count * warps);
    return launches;
}

}  // namespace

int launch_integrate_fp64(const DJob& J, InitSoA soa, const double* t, const int64_t* idx,
                          const unsigned long long* count, unsigned long long* work, TrajOut out, int64_t max_n,
                          int sm_count, cudaStream_t s) {
#define ETRAJ_DISPATCH_TGT(D, P)                                                               \
    return (J.target.kind == ETRAJ_TARGET_HYDROGEN_LIKE)                                       \
               ? launch_t<D, P, ETRAJ_TARGET_HYDROGEN_LIKE>(J, soa, t, idx, count, work, out, max_n, \
                                                            sm_count, s)                       \
               : launch_t<D, P, ETRAJ_TARGET_SAE>(J, soa, t, idx, count, work, out, max_n, sm_count, s);
    if (J.dim == 2) {
        if (J.phase == ETRAJ_PHASE_CTMC) { ETRAJ_DISPATCH_TGT(2, ETRAJ_PHASE_CTMC) }
        if (J.phase == ETRAJ_PHASE_QTMC) { ETRAJ_DISPATCH_TGT(2, ETRAJ_PHASE_QTMC) }
        ETRAJ_DISPATCH_TGT(2, ETRAJ_PHASE_SCTS)
    } else {
        if (J.phase == ETRAJ_PHASE_CTMC) { ETRAJ_DISPATCH_TGT(3, ETRAJ_PHASE_CTMC) }
        if (J.phase == ETRAJ_PHASE_QTMC) { ETRAJ_DISPATCH_TGT(3, ETRAJ_PHASE_QTMC) }
        ETRAJ_DISPATCH_TGT(3, ETRAJ_PHASE_SCTS)
    }
#undef ETRAJ_DISPATCH_TGT
}

int launch_collect_fp64(const DJob& J, InitSoA soa, const double* t, const int64_t* idx,
                        const unsigned long long* count, TrajOut out, int64_t max_n, int sm_count,
                        cudaStream_t s) {
    const int threads = 128;
    int64_t want = (max_n + threads - 1) / threads;
    int64_t cap = (int64_t)sm_count * 16;
    int blocks = (int)(want < cap ? (want > 0 ? want : 1) : cap);
#define ETRAJ_COLLECT(D, P) k_collect_fp64<D, P><<<blocks, threads, 0, s>>>(J, soa, t, idx, count, out)
    if (J.dim == 2) {
        if (J.phase == ETRAJ_PHASE_CTMC) ETRAJ_COLLECT(2, ETRAJ_PHASE_CTMC);
        else if (J.phase == ETRAJ_PHASE_QTMC) ETRAJ_COLLECT(2, ETRAJ_PHASE_QTMC);
        else ETRAJ_COLLECT(2, ETRAJ_PHASE_SCTS);
    } else {
        if (J.phase == ETRAJ_PHASE_CTMC) ETRAJ_COLLECT(3, ETRAJ_PHASE_CTMC);
        else if (J.phase == ETRAJ_PHASE_QTMC) ETRAJ_COLLECT(3, ETRAJ_PHASE_QTMC);
        else ETRAJ_COLLECT(3, ETRAJ_PHASE_SCTS);
    }
#undef ETRAJ_COLLECT
    return 1;
}

}  // namespace etraj
