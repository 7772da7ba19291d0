// The specialised fused kernel (fused.cuh): path, payoff and FP64 sums for baskets whose names share one kind.
#include <algorithm>
#include <cmath>
#include <numeric>
#include <type_traits>
#include <vector>

#include "mc.cuh"
#include "qe64.cuh"
#include "table_upload.cuh"

namespace ob {

namespace {

constexpr int gcd4(int c) { return c % 4 == 0 ? 4 : c % 2 == 0 ? 2 : 1; }

// Product bookkeeping of one leg, kept small: the ladder's extremes or the autocall's state.
template <typename R>
struct Leg {
    R hi, lo;       // ladder: extremes of ln perf; autocall: lo is the lowest ln perf
    double pv;      // autocall: discounted cash flows
    float coupons;  // autocall: coupons paid
    int flags;      // autocall: missed coupons (bits 0-15), alive (16), called (17), knocked (18)
};

constexpr int kAlive = 1 << 16, kCalled = 1 << 17, kKnocked = 1 << 18;

template <typename R, int PRODUCT>
__device__ __forceinline__ void leg_init(Leg<R>& l) {
    l.hi = R(-1e30), l.lo = PRODUCT == OB_PRODUCT_LADDER ? R(1e30) : R(0);
    l.pv = 0.0, l.coupons = 0.0f, l.flags = kAlive;
}

// Observation j of one leg (autocall): coupon with memory, then the call, or the redemption on the last date
// (packages/structured/src/optlab/structured/compiler.py:114-127,141-161,271-280).
template <typename R>
__device__ __forceinline__ void leg_observe(const FusedArgs<R>& a, const R* ln_trig, const double* disc, Leg<R>& l,
                                            R lp, int j) {
    if (!(l.flags & kAlive)) return;
    const double D = disc[j];
    if (a.has_coupon) {
        if (lp >= a.ln_cb) {
            const int k = a.memory ? 1 + (l.flags & 0xFFFF) : 1;
            l.pv += D * a.coupon * k, l.coupons += static_cast<float>(k), l.flags &= ~0xFFFF;
        } else {
            l.flags += 1;
        }
    }
    if (j < a.n_obs - 1) {
        if (lp >= ln_trig[j]) l.pv += D, l.flags = (l.flags & ~kAlive) | kCalled;
    } else {
        const bool ki = a.ki_daily ? l.lo < a.ln_ki : lp < a.ln_ki;
        const double perf = static_cast<double>(m_exp(lp));
        const double put = a.put_strike - perf > 0.0 ? a.put_strike - perf : 0.0;
        l.pv += D * (ki ? 1.0 - put : 1.0);
        l.flags = (l.flags & ~kAlive) | (ki ? kKnocked : 0);
    }
}

template <typename R, int PRODUCT>
__device__ __forceinline__ double leg_output(const FusedArgs<R>& a, const int* leg_type, const R* leg_strike,
                                             const int* leg_barrier, const R* ln_level, const Leg<R>& l, R lp_T,
                                             int k) {
    if (PRODUCT == OB_PRODUCT_AUTOCALL) {
        return k == 0 ? l.pv : k == 1 ? ((l.flags & kCalled) ? 1.0 : 0.0)
                                      : k == 2 ? ((l.flags & kKnocked) ? 1.0 : 0.0) : static_cast<double>(l.coupons);
    }
    const R U = a.spot0 * m_exp(lp_T);
    if (k == a.n_legs) return static_cast<double>(U);
    const int type = leg_type[k];
    const R K = leg_strike[k];
    R pay = type == 1 ? m_max(U - K, R(0)) : type == 2 ? m_max(K - U, R(0)) : type == 3 ? U - K : R(0);
    const int bt = leg_barrier[k];
    const R H = ln_level[k];
    const bool up = l.hi >= H, down = l.lo <= H;
    if ((bt == OB_BARRIER_UP_OUT && up) || (bt == OB_BARRIER_DOWN_OUT && down) || (bt == OB_BARRIER_UP_IN && !up) ||
        (bt == OB_BARRIER_DOWN_IN && !down))
        pay = R(0);
    return a.discount * static_cast<double>(pay);
}

template <typename R>
constexpr int min_blocks() {
    return sizeof(R) == 4 ? 2 : 1;
}

// KIND: 1 local vol (table), 2 Heston (Euler), 3 SLV (table x Heston, residuals on the aux stream), 4 Heston QE-M.
// TM: where the table is read (kTabStaged, kTabGlobal, kTabStreamed).
// Blocks of 512 an SM the register budget allows: two in float (64 registers), one in double; one for the mixer's
// 4- and 5-name baskets in float too, whose two legs' normals would spill at 64.
template <typename R, int N, bool MIX>
constexpr int fused_min_blocks() {
    return MIX && N >= 4 ? 1 : min_blocks<R>();
}

// Steps per batch of whole Philox blocks. One or two local-vol names draw two blocks a batch (8 or 4 steps), whose two
// independent multiply chains interleave (one name 1.317 -> 1.300 ms for the 2^20-path Phoenix, two 1150 -> 1045 us for
// 500k paths x 756 steps; one SLV name would draw four and spill in FP64).
constexpr int batch_steps(int n, int kind, bool mix) {
    const int c = kind == 4 ? 2 : kind == 2 ? 2 * n : n + (mix ? 1 : 0);
    return kind == 1 && c <= 2 ? 8 / c : 4 / gcd4(c);
}

// MIX (local vol, 2 to 5 names): the local-correlation mixer, one more normal a step after the names'.
template <typename R, int N, int KIND, int PRODUCT, int TM = kTabStaged, bool MIX = false>
__global__ void __launch_bounds__(TM == kTabStreamed ? 1024 : 512, TM == kTabStreamed ? 1 : fused_min_blocks<R, N, MIX>())
    fused_kernel(FusedArgs<R> a, long long n_pairs, long long first_pair, uint32_t k0, uint32_t k1,
                 double* __restrict__ partial) {
    constexpr bool QE = KIND == 4;
    constexpr bool VAR = KIND == 2 || KIND == 3;
    constexpr bool TABLE = KIND == 1 || KIND == 3;
    static_assert(!MIX || (KIND == 1 && N >= 2), "the mixer runs local-vol baskets");
    constexpr int C = QE ? 2 : (KIND == 2 ? 2 * N : N + (MIX ? 1 : 0));  // normals per step, stream 0
    constexpr int CA = KIND == 3 ? N : 0;                // normals per step, aux stream
    constexpr int G = batch_steps(N, KIND, MIX);
    constexpr int NB = C * G / 4, NBA = CA * G / 4;

    extern __shared__ __align__(16) unsigned char sm[];
    stage_blob(sm, a.blob, a.smem_blob);
    const int n_warps = blockDim.x >> 5, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n_acc = 2 * a.n_out;
    double* wacc = reinterpret_cast<double*>(sm + a.smem_acc);
    for (int t = threadIdx.x; t < n_warps * n_acc; t += blockDim.x) wacc[t] = 0.0;
    __syncthreads();
    const StepRec<R>* s_step = reinterpret_cast<const StepRec<R>*>(sm + a.off.step);
    const NameStep<R>* s_ns = reinterpret_cast<const NameStep<R>*>(sm + a.off.name_step);
    const R* s_root = reinterpret_cast<const R*>(sm + a.off.root);
    const R* s_hes = reinterpret_cast<const R*>(sm + a.off.hes);
    const Pair2<R>* s_tab = TM == kTabStaged ? reinterpret_cast<const Pair2<R>*>(sm + a.off.table2) : a.tab;
    const uint32_t tab_s = TM == kTabStreamed ? static_cast<uint32_t>(a.rs.off)
                                              : shared_address<TABLE && TM == kTabStaged>(s_tab);
    RowStream<R, G> rows(a.rs, a.tab, s_ns, sm, a.n_steps);
    if (TM == kTabStreamed) rows.first();
    const R* s_trig = reinterpret_cast<const R*>(sm + a.off.ln_trig);
    const double* s_disc = reinterpret_cast<const double*>(sm + a.off.obs_disc);
    const int S = a.n_steps;
    // the correlation root: in registers for up to three names, read from shared memory for more (registers spill)
    constexpr bool kRootRegs = N <= 3;
    R rt[kRootRegs ? N * N : 1];
#pragma unroll
    for (int k = 0; k < (kRootRegs ? N * N : 0); ++k) rt[k] = s_root[k];

    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    for (long long block0 = static_cast<long long>(blockIdx.x) * blockDim.x; block0 < n_pairs; block0 += stride) {
        const long long base = block0 + (threadIdx.x & ~31);
        if (TM != kTabStreamed && base >= n_pairs) break;  // (a streaming block's warps keep together)
        const bool active = base + lane < n_pairs;
        const uint64_t pair = static_cast<uint64_t>(first_pair + (active ? base + lane : n_pairs - 1));
        R x0[N], x1[N], v0[N], v1[N];
#pragma unroll
        for (int n = 0; n < N; ++n) {
            x0[n] = x1[n] = R(0);
            v0[n] = v1[n] = QE ? a.qe.v0 : (VAR ? s_hes[8 * n] : R(0));
        }
        Leg<R> l0, l1;
        leg_init<R, PRODUCT>(l0), leg_init<R, PRODUCT>(l1);
        R lp0 = R(0), lp1 = R(0);
        // One batch of G steps from step i0, its normals drawn first. For one local-vol name the full batches run
        // without testing for the last step and only the tail batch (CHECK) may stop inside, and an autocall's batches
        // without an observation run without testing each step for one (OBS false).
        auto run_batch = [&](int i0, int batch, auto check, auto observe) {
            constexpr bool CHECK = decltype(check)::value, OBS = decltype(observe)::value;
            if (TM == kTabStreamed && rows.opens(batch)) rows.turn(batch, block0 + stride < n_pairs);
            R z[C * G];
            R za[CA > 0 ? CA * G : 1];
            R q0 = R(0), q1 = R(0);
#pragma unroll
            for (int k = 0; k < NB; ++k)
                normals4<R>(pair, static_cast<uint64_t>(batch) * NB + k, 0u, k0, k1, z[4 * k], z[4 * k + 1],
                            z[4 * k + 2], z[4 * k + 3]);
#pragma unroll
            for (int k = 0; k < NBA; ++k)
                normals4<R>(pair, static_cast<uint64_t>(batch) * NBA + k, kAuxStream, k0, k1, za[4 * k],
                            za[4 * k + 1], za[4 * k + 2], za[4 * k + 3]);
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int i = i0 + g;
                if constexpr (CHECK && G > 1) {
                    if (i > S) break;
                }
                if (QE) {
                    const R zv = z[2 * g], zx = z[2 * g + 1];
                    qe_step(a.qe, x0[0], v0[0], zv, zx);
                    qe_step(a.qe, x1[0], v1[0], -zv, -zx);
                    lp0 = x0[0], lp1 = x1[0];
                } else {
                    const StepRec<R> st = s_step[i - 1];
                    const R* zs = &z[g * C];
                    R zc[N], wc[N];
                    R zm0[MIX ? N : 1], zm1[MIX ? N : 1];  // with the mixer each leg's own normals (signs in)
                    if (MIX) {
                        // paths.hpp:219-237: a common factor whose weight moves with the level of the basket (the
                        // log of the mean of S / F at the step's start), per leg
                        const R* s_low = reinterpret_cast<const R*>(sm + a.off.low_root);
                        const R den = reinterpret_cast<const R*>(sm + a.off.mix_den)[i - 1];
#pragma unroll
                        for (int leg = 0; leg < 2; ++leg) {
                            const R sg = leg ? R(-1) : R(1);
                            R mm = R(0);
#pragma unroll
                            for (int n = 0; n < N; ++n) mm += m_exp(leg ? x1[n] : x0[n]);
                            const R u = m_log(mm / static_cast<R>(N)) / den;
                            R wt = a.mix_base + a.mix_down * m_max(-u, R(0)) - a.mix_up * m_max(u, R(0));
                            wt = m_min(m_max(wt, R(0)), R(1));
                            const R market = a.mix_sign * sg * zs[N - 1], fr = sg * zs[N];
                            const R common = a.mix_cos * market + a.mix_sin * fr;
                            R other[N];
#pragma unroll
                            for (int n = 0; n < N - 1; ++n) other[n] = sg * zs[n];
                            other[N - 1] = a.mix_sin * market - a.mix_cos * fr;
                            const R sw = m_sqrt(wt), sl = m_sqrt(R(1) - wt);
#pragma unroll
                            for (int n = 0; n < N; ++n) {
                                R acc = R(0);
#pragma unroll
                                for (int b = 0; b < N; ++b) acc += s_low[n * N + b] * other[b];
                                (leg ? zm1 : zm0)[n] = sw * common + sl * acc;
                            }
                        }
                    }
#pragma unroll
                    for (int n = 0; n < N; ++n) {
                        R acc = R(0);
                        if (!MIX) {
#pragma unroll
                            for (int b = 0; b < N; ++b)
                                acc += (kRootRegs ? rt[n * N + b] : s_root[n * N + b]) * zs[b];
                        }
                        zc[n] = acc;
                    }
                    if (VAR) {
                        const R* zr = KIND == 3 ? &za[g * CA] : &z[g * C + N];
#pragma unroll
                        for (int n = 0; n < N; ++n) {
                            if (a.same) {
                                R acc = R(0);
#pragma unroll
                                for (int b = 0; b < N; ++b) acc += (kRootRegs ? rt[n * N + b] : s_root[n * N + b]) * zr[b];
                                wc[n] = acc;
                            } else {
                                wc[n] = zr[n];
                            }
                        }
                    }
                    R w0 = R(0), w1 = R(0);  // the worst log performance: the first name's, then the minimum
#pragma unroll
                    for (int n = 0; n < N; ++n) {
                        const NameStep<R> ns = s_ns[(i - 1) * N + n];
                        R var0, var1, vp0 = R(0), vp1 = R(0);
                        if (VAR) vp0 = m_max(v0[n], R(0)), vp1 = m_max(v1[n], R(0));
                        if (TABLE) {
                            R t0, t1;
                            table_vars<TM>(s_tab, sm, tab_s, ns.org, ns.inv_dx, TM == kTabStreamed ? rows.row(i) : ns.row,
                                           a.top, x0[n], x1[n], t0, t1);
                            var0 = KIND == 1 ? t0 : t0 * vp0, var1 = KIND == 1 ? t1 : t1 * vp1;
                        } else if (VAR) {
                            var0 = vp0, var1 = vp1;
                        } else {
                            var0 = var1 = s_hes[8 * n + 6];  // Black-Scholes: the name's constant variance
                        }
                        if (VAR) {
                            const R* h = s_hes + 8 * n;  // v0, kappa, theta, xi, rho, sqrt(1 - rho^2)
                            const R zv = h[4] * zc[n] + h[5] * wc[n];
                            v0[n] += h[1] * (h[2] - vp0) * st.dt + h[3] * (m_sqrt(vp0) * st.sdt) * zv;
                            v1[n] += h[1] * (h[2] - vp1) * st.dt + h[3] * (m_sqrt(vp1) * st.sdt) * (-zv);
                        }
                        if (MIX) {
                            x0[n] = lv_advance(x0[n], var0, st.hdt, st.sdt * zm0[n]);
                            x1[n] = lv_advance(x1[n], var1, st.hdt, st.sdt * zm1[n]);
                        } else {
                            const R zd = st.sdt * zc[n];  // sqrt(dt) z, the legs' +-
                            lv_advance_legs(x0[n], x1[n], var0, var1, st.hdt, zd);
                        }
                        if (n == 0) w0 = x0[n] + ns.lf, w1 = x1[n] + ns.lf;
                        else w0 = m_min(w0, x0[n] + ns.lf), w1 = m_min(w1, x1[n] + ns.lf);
                    }
                    lp0 = w0, lp1 = w1;
                }
                if (PRODUCT == OB_PRODUCT_LADDER) {
                    l0.hi = run_max(l0.hi, lp0), l0.lo = run_min(l0.lo, lp0);
                    l1.hi = run_max(l1.hi, lp1), l1.lo = run_min(l1.lo, lp1);
                } else if (!OBS && G % 2 == 0) {  // no one reads the low within the batch: two steps at a time
                    if (g % 2) l0.lo = run_min(l0.lo, q0, lp0), l1.lo = run_min(l1.lo, q1, lp1);
                    else q0 = lp0, q1 = lp1;
                } else {
                    l0.lo = run_min(l0.lo, lp0), l1.lo = run_min(l1.lo, lp1);
                    const int j = OBS ? s_step[i - 1].obs : -1;
                    if (j >= 0) {
                        leg_observe(a, s_trig, s_disc, l0, lp0, j);
                        leg_observe(a, s_trig, s_disc, l1, lp1, j);
                    }
                }
            }
        };
        if constexpr (N == 1 && KIND == 1) {  // (a second copy of the loop costs the wider kernels registers)
            // a step without an observation holds minus the steps to the next one: none in steps i0 .. i0 + G - 1
            // when step i0's entry is at most -G
            constexpr bool kSplitObs = PRODUCT == OB_PRODUCT_AUTOCALL;
            const int n_full = S / G;
            int i0 = 1, batch = 0;
            for (; batch < n_full; i0 += G, ++batch) {
                if (!kSplitObs || s_step[i0 - 1].obs <= -G)
                    run_batch(i0, batch, std::false_type{}, std::false_type{});
                else
                    run_batch(i0, batch, std::false_type{}, std::true_type{});
            }
            if (i0 <= S) run_batch(i0, batch, std::true_type{}, std::true_type{});
        } else {
            for (int i0 = 1, batch = 0; i0 <= S; i0 += G, ++batch)
                run_batch(i0, batch, std::true_type{}, std::true_type{});
        }
        const int* leg_type = reinterpret_cast<const int*>(sm + a.off.leg_type);
        const R* leg_strike = reinterpret_cast<const R*>(sm + a.off.leg_strike);
        const int* leg_barrier = reinterpret_cast<const int*>(sm + a.off.leg_barrier);
        const R* ln_level = reinterpret_cast<const R*>(sm + a.off.ln_level);
        for (int k = 0; k < a.n_out; ++k) {
            const double y =
                active ? 0.5 * (leg_output<R, PRODUCT>(a, leg_type, leg_strike, leg_barrier, ln_level, l0, lp0, k) +
                                leg_output<R, PRODUCT>(a, leg_type, leg_strike, leg_barrier, ln_level, l1, lp1, k))
                       : 0.0;
            const double s1 = warp_sum(y), s2 = warp_sum(y * y);
            if (lane == 0) wacc[warp * n_acc + k] += s1, wacc[warp * n_acc + a.n_out + k] += s2;
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < n_acc; t += blockDim.x) {
        double s = 0.0;
        for (int w = 0; w < n_warps; ++w) s += wacc[w * n_acc + t];
        partial[static_cast<long long>(blockIdx.x) * n_acc + t] = s;
    }
}

// Heston QE-M with the two legs of an antithetic pair on neighbouring lanes (lane 2k: +z, lane 2k+1: -z): twice the
// threads of fused_kernel for the same pairs, for the small path counts of QE books (2^15 pairs are 7 warps an SM at
// one pair a thread; the FP64 step is a long dependent chain and needs the warps to hide its latency). Philox block b
// of a pair holds (zv, zx) of steps 2b + 1 and 2b + 2; the two lanes draw alternate blocks (lane 2k block 2m, lane
// 2k + 1 block 2m + 1) and swap them, so each lane draws half the normals and steps one leg. The pair's value is
// the average of the lanes' payoffs, added once (by the even lane).
template <typename R, int PRODUCT>
__global__ void __launch_bounds__(512, min_blocks<R>())
    qe_pair_kernel(FusedArgs<R> a, long long n_pairs, long long first_pair, uint32_t k0, uint32_t k1,
                   double* __restrict__ partial) {
    extern __shared__ __align__(16) unsigned char sm[];
    stage_blob(sm, a.blob, a.smem_blob);
    const int n_warps = blockDim.x >> 5, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n_acc = 2 * a.n_out;
    double* wacc = reinterpret_cast<double*>(sm + a.smem_acc);
    for (int t = threadIdx.x; t < n_warps * n_acc; t += blockDim.x) wacc[t] = 0.0;
    __syncthreads();
    const int* s_obs = reinterpret_cast<const int*>(sm + a.off.step);  // the observation at each step's end, or negative
    const R* s_trig = reinterpret_cast<const R*>(sm + a.off.ln_trig);
    const double* s_disc = reinterpret_cast<const double*>(sm + a.off.obs_disc);
    const int* leg_type = reinterpret_cast<const int*>(sm + a.off.leg_type);
    const R* leg_strike = reinterpret_cast<const R*>(sm + a.off.leg_strike);
    const int* leg_barrier = reinterpret_cast<const int*>(sm + a.off.leg_barrier);
    const R* ln_level = reinterpret_cast<const R*>(sm + a.off.ln_level);
    const int S = a.n_steps;
    const int odd = lane & 1;
    const R sgn = odd ? R(-1) : R(1);
    constexpr unsigned kFull = 0xffffffffu;

    const long long stride = (static_cast<long long>(gridDim.x) * blockDim.x) >> 1;
    for (long long base = (static_cast<long long>(blockIdx.x) * blockDim.x + (threadIdx.x & ~31)) >> 1;
         base < n_pairs; base += stride) {
        const long long p = base + (lane >> 1);
        const bool active = p < n_pairs;
        const uint64_t pair = static_cast<uint64_t>(first_pair + (active ? p : n_pairs - 1));
        R x = R(0), v = a.qe.v0, lp = R(0);
        Leg<R> l;
        leg_init<R, PRODUCT>(l);
        auto keep = [&](int i) {  // the leg's books at step end i
            lp = x;
            if (PRODUCT == OB_PRODUCT_LADDER) {
                l.hi = run_max(l.hi, lp), l.lo = run_min(l.lo, lp);
            } else {
                l.lo = run_min(l.lo, lp);
                const int j = s_obs[i - 1];
                if (j >= 0) leg_observe(a, s_trig, s_disc, l, lp, j);
            }
        };
        // the lane's own block of the two of batch m, and both lanes' normals of its four steps
        auto swap = [&](const R (&z)[4], R (&e)[8]) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const R o = __shfl_xor_sync(kFull, z[k], 1);
                e[k] = odd ? o : z[k];      // block 2m: steps i0, i0 + 1
                e[4 + k] = odd ? z[k] : o;  // block 2m + 1: steps i0 + 2, i0 + 3
            }
        };
        if constexpr (sizeof(R) == 8) {
            // the steps of a batch and the next batch's draws and tails in one straight line: they do not wait for
            // each other
            const Qe64Tables& t = *reinterpret_cast<const Qe64Tables*>(sm + a.off.qe_tables);
            R e[8], tail[4];
            auto draw = [&](int m) {
                uint32_t c[4] = {static_cast<uint32_t>(pair), static_cast<uint32_t>(pair >> 32),
                                 static_cast<uint32_t>(2 * m + odd), 0u};
                philox4x32_10(c[0], c[1], c[2], c[3], k0, k1);
                R z[4];
                box_muller64(t, c[0], c[1], z[0], z[1]);
                box_muller64(t, c[2], c[3], z[2], z[3]);
                // the legs' tails add up to one: a lane takes those of its own block's two steps, of |z|, and swaps them
                const double t0 = tail64(t, fabs(z[0])), t1 = tail64(t, fabs(z[2]));
                const double o0 = __shfl_xor_sync(kFull, t0, 1), o1 = __shfl_xor_sync(kFull, t1, 1);
                tail[0] = odd ? o0 : t0, tail[1] = odd ? o1 : t1;
                tail[2] = odd ? t0 : o0, tail[3] = odd ? t1 : o1;
                swap(z, e);
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    e[2 * g] *= sgn, e[2 * g + 1] *= sgn;
                    tail[g] = e[2 * g] < 0.0 ? 1.0 - tail[g] : tail[g];
                }
            };
            draw(0);
            int i = 1, m = 0;
            for (; i + 3 <= S; i += 4) {
                R ce[8], ct[4];
#pragma unroll
                for (int k = 0; k < 8; ++k) ce[k] = e[k];
#pragma unroll
                for (int k = 0; k < 4; ++k) ct[k] = tail[k];
                draw(++m);
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    qe64_step(a.qe, t, x, v, ce[2 * g], ce[2 * g + 1], ct[g]);
                    keep(i + g);
                }
            }
#pragma unroll
            for (int g = 0; g < 3; ++g)
                if (i + g <= S) {
                    qe64_step(a.qe, t, x, v, e[2 * g], e[2 * g + 1], tail[g]);
                    keep(i + g);
                }
        } else {
            for (int i0 = 1, m = 0; i0 <= S; i0 += 4, ++m) {
                R z[4], e[8];
                normals4<R>(pair, static_cast<uint64_t>(2 * m + odd), 0u, k0, k1, z[0], z[1], z[2], z[3]);
                swap(z, e);
                // one copy of the step in the loop body: the four steps rotate the normals through e[0..1]
#pragma unroll 1
                for (int g = 0; g < 4; ++g) {
                    const int i = i0 + g;
                    if (i > S) break;
                    qe_step_warp(a.qe, x, v, sgn * e[0], sgn * e[1]);  // (all 32 lanes step together)
                    e[0] = e[2], e[1] = e[3], e[2] = e[4], e[3] = e[5], e[4] = e[6], e[5] = e[7];
                    keep(i);
                }
            }
        }
        for (int k = 0; k < a.n_out; ++k) {
            const double mine = leg_output<R, PRODUCT>(a, leg_type, leg_strike, leg_barrier, ln_level, l, lp, k);
            const double other = __shfl_xor_sync(kFull, mine, 1);
            const double y = active && !odd ? 0.5 * (mine + other) : 0.0;
            const double s1 = warp_sum(y), s2 = warp_sum(y * y);
            if (lane == 0) wacc[warp * n_acc + k] += s1, wacc[warp * n_acc + a.n_out + k] += s2;
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < n_acc; t += blockDim.x) {
        double s = 0.0;
        for (int w = 0; w < n_warps; ++w) s += wacc[w * n_acc + t];
        partial[static_cast<long long>(blockIdx.x) * n_acc + t] = s;
    }
}

// One to three local-vol names with the two legs of a pair on neighbouring lanes (as in qe_pair_kernel), for launches
// of few pairs: a warp then carries 16 pairs through half the instructions a step, and a launch that leaves the schedulers
// a warp or two each lasts as long as one warp's walk (fused_legs_apart has the sizes). The lanes draw alternate batches of
// Philox blocks and swap them. Each leg's arithmetic is fused_kernel's, so a pair's value is the same bit for bit.
template <typename R, int N, int PRODUCT, int TM>
__global__ void __launch_bounds__(512, 1)
    fused_legs_kernel(FusedArgs<R> a, long long n_pairs, long long first_pair, uint32_t k0, uint32_t k1,
                      double* __restrict__ partial) {
    constexpr int G = 4 / gcd4(N), NB = N * G / 4, Z = N * G;  // steps, blocks and normals of one lane's batch
    extern __shared__ __align__(16) unsigned char sm[];
    stage_blob(sm, a.blob, a.smem_blob);
    const int n_warps = blockDim.x >> 5, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n_acc = 2 * a.n_out;
    double* wacc = reinterpret_cast<double*>(sm + a.smem_acc);
    for (int t = threadIdx.x; t < n_warps * n_acc; t += blockDim.x) wacc[t] = 0.0;
    __syncthreads();
    const StepRec<R>* s_step = reinterpret_cast<const StepRec<R>*>(sm + a.off.step);
    const NameStep<R>* s_ns = reinterpret_cast<const NameStep<R>*>(sm + a.off.name_step);
    const R* s_root = reinterpret_cast<const R*>(sm + a.off.root);
    const Pair2<R>* s_tab = TM == kTabStaged ? reinterpret_cast<const Pair2<R>*>(sm + a.off.table2) : a.tab;
    const R* s_trig = reinterpret_cast<const R*>(sm + a.off.ln_trig);
    const double* s_disc = reinterpret_cast<const double*>(sm + a.off.obs_disc);
    const int* leg_type = reinterpret_cast<const int*>(sm + a.off.leg_type);
    const R* leg_strike = reinterpret_cast<const R*>(sm + a.off.leg_strike);
    const int* leg_barrier = reinterpret_cast<const int*>(sm + a.off.leg_barrier);
    const R* ln_level = reinterpret_cast<const R*>(sm + a.off.ln_level);
    const int S = a.n_steps, odd = lane & 1;
    constexpr unsigned kFull = 0xffffffffu;
    R rt[N * N];
#pragma unroll
    for (int k = 0; k < N * N; ++k) rt[k] = s_root[k];
    const long long stride = (static_cast<long long>(gridDim.x) * blockDim.x) >> 1;
    for (long long base = (static_cast<long long>(blockIdx.x) * blockDim.x + (threadIdx.x & ~31)) >> 1;
         base < n_pairs; base += stride) {
        const long long p = base + (lane >> 1);
        const bool active = p < n_pairs;
        const uint64_t pair = static_cast<uint64_t>(first_pair + (active ? p : n_pairs - 1));
        R x[N], lp = R(0);
#pragma unroll
        for (int n = 0; n < N; ++n) x[n] = R(0);
        Leg<R> l;
        leg_init<R, PRODUCT>(l);
        // The normals of the lanes' two batches (2 G steps). Each is drawn beside the steps of the one before, which do
        // not wait for it: a warp alone on its scheduler fills the one chain's waits with the other.
        R e[2 * Z];
        auto draw = [&](int m) {
            R z[Z];
#pragma unroll
            for (int k = 0; k < NB; ++k)
                normals4<R>(pair, static_cast<uint64_t>(2 * m + odd) * NB + k, 0u, k0, k1, z[4 * k], z[4 * k + 1],
                            z[4 * k + 2], z[4 * k + 3]);
#pragma unroll
            for (int k = 0; k < Z; ++k) {
                const R o = __shfl_xor_sync(kFull, z[k], 1);
                e[k] = odd ? o : z[k], e[Z + k] = odd ? z[k] : o;
            }
        };
        // 2 G steps from step i0; only the tail (CHECK) may stop inside
        auto run_batches = [&](int i0, int m, auto check, auto observe) {
            constexpr bool CHECK = decltype(check)::value, OBS = decltype(observe)::value;
            R c[2 * Z];
#pragma unroll
            for (int k = 0; k < 2 * Z; ++k) c[k] = e[k];
            if (!CHECK) draw(m + 1);
#pragma unroll
            for (int g = 0; g < 2 * G; ++g) {
                const int i = i0 + g;
                if constexpr (CHECK) {
                    if (i > S) break;
                }
                const StepRec<R> st = s_step[i - 1];
                R w = R(0);
#pragma unroll
                for (int n = 0; n < N; ++n) {
                    R acc = R(0);
#pragma unroll
                    for (int b = 0; b < N; ++b) acc += rt[n * N + b] * c[g * N + b];
                    const NameStep<R> ns = s_ns[(i - 1) * N + n];
                    int j;
                    R f;
                    table_cell(ns, a.top, x[n], j, f);
                    const Pair2<R> y = TM == kTabGlobal ? ldg_pair(s_tab + ns.row + j) : s_tab[ns.row + j];
                    const R zd = st.sdt * acc;  // sqrt(dt) z, the legs' +-
                    x[n] = lv_advance(x[n], m_fma(f, y.b, y.a), st.hdt, odd ? -zd : zd);
                    w = n == 0 ? x[n] + ns.lf : m_min(w, x[n] + ns.lf);
                }
                lp = w;
                if (PRODUCT == OB_PRODUCT_LADDER) {
                    l.hi = run_max(l.hi, lp), l.lo = run_min(l.lo, lp);
                } else {
                    l.lo = run_min(l.lo, lp);
                    const int j = OBS ? st.obs : -1;
                    if (j >= 0) leg_observe(a, s_trig, s_disc, l, lp, j);
                }
            }
        };
        draw(0);
        int i0 = 1, m = 0;
        for (; i0 + 2 * G - 1 <= S; i0 += 2 * G, ++m) {
            // (a step without an observation holds minus the steps to the next one)
            if (PRODUCT == OB_PRODUCT_LADDER || s_step[i0 - 1].obs <= -2 * G)
                run_batches(i0, m, std::false_type{}, std::false_type{});
            else
                run_batches(i0, m, std::false_type{}, std::true_type{});
        }
        if (i0 <= S) run_batches(i0, m, std::true_type{}, std::true_type{});
        for (int k = 0; k < a.n_out; ++k) {
            const double mine = leg_output<R, PRODUCT>(a, leg_type, leg_strike, leg_barrier, ln_level, l, lp, k);
            const double other = __shfl_xor_sync(kFull, mine, 1);
            const double y = active && !odd ? 0.5 * (mine + other) : 0.0;
            const double s1 = warp_sum(y), s2 = warp_sum(y * y);
            if (lane == 0) wacc[warp * n_acc + k] += s1, wacc[warp * n_acc + a.n_out + k] += s2;
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < n_acc; t += blockDim.x) {
        double s = 0.0;
        for (int w = 0; w < n_warps; ++w) s += wacc[w * n_acc + t];
        partial[static_cast<long long>(blockIdx.x) * n_acc + t] = s;
    }
}

template <typename R>
using FusedFn = void (*)(FusedArgs<R>, long long, long long, uint32_t, uint32_t, double*);

template <typename R, int KIND, int PRODUCT, int TM>
FusedFn<R> pick_n(int n) {
    if (n == 1) return fused_kernel<R, 1, KIND, PRODUCT, TM>;
    if (n == 2) return fused_kernel<R, 2, KIND, PRODUCT, TM>;
    if (n == 3) return fused_kernel<R, 3, KIND, PRODUCT, TM>;
    if constexpr (KIND == 1 || KIND == 0) {
        if (n == 4) return fused_kernel<R, 4, KIND, PRODUCT, TM>;
        if (n == 5) return fused_kernel<R, 5, KIND, PRODUCT, TM>;
    }
    return nullptr;
}

// Local-vol baskets of 2 to 5 names with the local-correlation mixer.
template <typename R, int PRODUCT, int TM>
FusedFn<R> pick_mix(int n) {
    switch (n) {
        case 2: return fused_kernel<R, 2, 1, PRODUCT, TM, true>;
        case 3: return fused_kernel<R, 3, 1, PRODUCT, TM, true>;
        case 4: return fused_kernel<R, 4, 1, PRODUCT, TM, true>;
        case 5: return fused_kernel<R, 5, 1, PRODUCT, TM, true>;
        default: return nullptr;
    }
}

// tm: where the kinds with a table (local vol, SLV) read it; rows are streamed for one local-vol name in float (in double
// the arithmetic bounds the step, not the table's reads).
template <typename R, int PRODUCT>
FusedFn<R> pick_fused(int kind, int n, int tm, bool mix) {
    if (tm == kTabStreamed) {
        if constexpr (sizeof(R) == 4)
            if (kind == 1 && n == 1 && !mix) return fused_kernel<R, 1, 1, PRODUCT, kTabStreamed>;
        return nullptr;
    }
    const bool global = tm == kTabGlobal;
    if (mix)
        return kind != 1 ? nullptr : global ? pick_mix<R, PRODUCT, kTabGlobal>(n) : pick_mix<R, PRODUCT, kTabStaged>(n);
    switch (kind) {
        case 0: return global ? nullptr : pick_n<R, 0, PRODUCT, kTabStaged>(n);
        case 1: return global ? pick_n<R, 1, PRODUCT, kTabGlobal>(n) : pick_n<R, 1, PRODUCT, kTabStaged>(n);
        case 2: return pick_n<R, 2, PRODUCT, kTabStaged>(n);
        case 3: return global ? pick_n<R, 3, PRODUCT, kTabGlobal>(n) : pick_n<R, 3, PRODUCT, kTabStaged>(n);
        case 4: return n == 1 ? qe_pair_kernel<R, PRODUCT> : nullptr;
        default: return nullptr;
    }
}

template <typename R, int PRODUCT, int TM>
FusedFn<R> pick_legs_n(int n) {
    if (n == 1) return fused_legs_kernel<R, 1, PRODUCT, TM>;
    if (n == 2) return fused_legs_kernel<R, 2, PRODUCT, TM>;
    if (n == 3) return fused_legs_kernel<R, 3, PRODUCT, TM>;
    return nullptr;
}

// The kernel with a pair's legs on two lanes for the same stage, or null.
template <typename R, int PRODUCT>
FusedFn<R> pick_legs(int kind, int n, int tm, bool mix) {
    if constexpr (sizeof(R) == 4)
        if (kind == 1 && !mix)
            return tm == kTabStaged ? pick_legs_n<R, PRODUCT, kTabStaged>(n) : pick_legs_n<R, PRODUCT, kTabGlobal>(n);
    return nullptr;
}

struct Blob {
    std::vector<unsigned char> bytes;
    template <typename T>
    int put(const T* src, size_t count) {
        const size_t at = (bytes.size() + 15) & ~static_cast<size_t>(15);
        const size_t n = count * sizeof(T);
        bytes.resize(at + ((n + 15) & ~static_cast<size_t>(15)), 0);
        if (src && n) std::memcpy(bytes.data() + at, src, n);
        return static_cast<int>(at);
    }
    template <typename T>
    int put(const std::vector<T>& v) {
        return put(v.data(), v.size());
    }
};

}  // namespace

// Packs the request for the specialised kernel; false when it does not apply (mixed kinds, a basket size without an
// instantiation, or inputs that would not fit the shared-memory budget), and the generic kernel then runs. The
// table goes into the stage when it fits beside the rest, else into global memory (the reference plan's rows: 801
// points for every step, megabytes), where it stays in L2 and is read through the read-only cache.
template <typename R>
bool fused_build(McPlan& plan, const ob_mc_request& rq) {
    const int n = rq.n_names, S = rq.n_steps;
    int kind = -1;
    if (rq.model == OB_MODEL_HESTON_QE) {
        kind = 4;
    } else {
        kind = rq.kind[0];
        for (int a = 1; a < n; ++a)
            if (rq.kind[a] != kind) return false;
    }
    if (rq.mixer && kind != 1) return false;  // the mixer beside other kinds: the generic kernel
    auto pick = [&](int tm) -> FusedFn<R> {
        return rq.product == OB_PRODUCT_LADDER ? pick_fused<R, OB_PRODUCT_LADDER>(kind, n, tm, rq.mixer != 0)
                                               : pick_fused<R, OB_PRODUCT_AUTOCALL>(kind, n, tm, rq.mixer != 0);
    };
    if (!pick(kTabStaged)) return false;
    FusedArgs<R> a{};
    a.n_steps = S, a.n_x = rq.n_x, a.same = rq.same;
    a.n_obs = rq.product == OB_PRODUCT_AUTOCALL ? rq.n_obs : 0;
    a.n_legs = rq.product == OB_PRODUCT_LADDER ? rq.n_legs : 0;
    a.n_out = rq.product == OB_PRODUCT_LADDER ? rq.n_legs + 1 : 4;
    a.top = static_cast<R>(rq.n_x - 1) - static_cast<R>(1e-4);
    a.spot0 = static_cast<R>(rq.spot[0]);
    Blob blob;
    std::vector<StepRec<R>> steps(S);
    for (int i = 0; i < S; ++i) {
        std::memset(&steps[i], 0, sizeof steps[i]);
        steps[i].dt = static_cast<R>(rq.dt[i]);
        steps[i].hdt = static_cast<R>(-0.5 * rq.dt[i]);
        steps[i].sdt = static_cast<R>(std::sqrt(rq.dt[i]));
        steps[i].obs = -1;
    }
    if (rq.product == OB_PRODUCT_AUTOCALL) {
        for (int j = 0; j < rq.n_obs; ++j) steps[rq.obs_step[j] - 1].obs = j;
        // steps without an observation: minus the number of steps to the next one (past the last, more than any
        // batch)
        int next = S + (1 << 20);
        for (int i = S; i >= 1; --i) {
            if (steps[i - 1].obs >= 0) next = i;
            else steps[i - 1].obs = i - next;
        }
    }
    if (kind == 4) {  // (its steps are all alike: the kernel reads an autocall's observations alone)
        std::vector<int> obs(rq.product == OB_PRODUCT_AUTOCALL ? S : 0);
        for (size_t i = 0; i < obs.size(); ++i) obs[i] = steps[i].obs;
        a.off.step = blob.put(obs);
    } else {
        a.off.step = blob.put(steps);
    }
    const bool table = kind == 1 || kind == 3;
    if (kind == 4) {
        a.qe = make_qe_consts<R>(rq.heston, rq.r, rq.q, rq.dt[0]);
        if (sizeof(R) == 8) a.off.qe_tables = blob.put(&qe64_tables(), 1);
    } else {
        std::vector<NameStep<R>> ns(static_cast<size_t>(S) * n);
        for (int i = 1; i <= S; ++i)
            for (int k = 0; k < n; ++k) {
                NameStep<R>& r = ns[static_cast<size_t>(i - 1) * n + k];
                std::memset(&r, 0, sizeof r);
                r.lf = static_cast<R>(rq.log_fwd[static_cast<size_t>(k) * (S + 1) + i]);
                if (table) {
                    const int row = rq.step_row[static_cast<size_t>(k) * S + (i - 1)];
                    set_cell_row(r, rq.row_lo[row], rq.row_inv_dx[row], a.top);
                    r.row = row;  // (the row's first cell, once it is known where the table goes)
                }
            }
        a.off.name_step = blob.put(ns);
        std::vector<R> root(static_cast<size_t>(n) * n);
        for (size_t k = 0; k < root.size(); ++k) root[k] = static_cast<R>(rq.root[k]);
        a.off.root = blob.put(root);
        std::vector<R> hes(8 * static_cast<size_t>(n), R(0));
        for (int k = 0; k < n; ++k) {
            for (int f = 0; f < 5; ++f) hes[8 * k + f] = static_cast<R>(rq.heston[5 * k + f]);
            const R rho = hes[8 * k + 4];
            hes[8 * k + 5] = static_cast<R>(std::sqrt(R(1) - rho * rho));
            hes[8 * k + 6] = static_cast<R>(rq.cvar[k]);  // Black-Scholes
        }
        a.off.hes = blob.put(hes);
        if (rq.mixer) {
            std::vector<R> den(S), low(static_cast<size_t>(n) * n);
            for (int i = 0; i < S; ++i)  // R arithmetic as the generic step: sigma sqrt(max(t0, 1/12))
                den[i] = static_cast<R>(rq.mix[4]) * std::sqrt(std::max(static_cast<R>(rq.t0[i]), R(1.0 / 12)));
            for (size_t k = 0; k < low.size(); ++k) low[k] = static_cast<R>(rq.low_root[k]);
            a.off.mix_den = blob.put(den), a.off.low_root = blob.put(low);
            a.mix_base = static_cast<R>(rq.mix[0]) + static_cast<R>(rq.mix[1]);
            a.mix_down = static_cast<R>(rq.mix[2]), a.mix_up = static_cast<R>(rq.mix[3]);
            a.mix_sign = static_cast<R>(rq.mix[5]), a.mix_cos = static_cast<R>(rq.mix[6]);
            a.mix_sin = static_cast<R>(rq.mix[7]);
        }
    }
    if (rq.product == OB_PRODUCT_LADDER) {
        std::vector<int> type(rq.n_legs), bar(rq.n_legs);
        std::vector<R> strike(rq.n_legs), lvl(rq.n_legs);
        for (int k = 0; k < rq.n_legs; ++k) {
            type[k] = rq.leg_type[k];
            strike[k] = static_cast<R>(rq.leg_strike[k]);
            bar[k] = rq.leg_barrier ? rq.leg_barrier[k] : 0;
            lvl[k] = bar[k] ? static_cast<R>(std::log(rq.leg_level[k] / rq.spot[0])) : R(0);
        }
        a.off.leg_type = blob.put(type), a.off.leg_strike = blob.put(strike);
        a.off.leg_barrier = blob.put(bar), a.off.ln_level = blob.put(lvl);
        a.discount = rq.discount;
    } else {
        std::vector<R> trig(rq.n_obs);
        for (int j = 0; j < rq.n_obs; ++j)
            trig[j] = rq.trigger[j] > 0 ? static_cast<R>(std::log(rq.trigger[j])) : R(1e30);
        a.off.ln_trig = blob.put(trig);
        a.off.obs_disc = blob.put(rq.obs_discount, rq.n_obs);
        a.has_coupon = rq.coupon > 0.0 || rq.coupon_barrier > 0.0;
        a.ln_cb = rq.coupon_barrier > 0 ? static_cast<R>(std::log(rq.coupon_barrier)) : R(-1e30);
        a.ln_ki = rq.ki_barrier > 0 ? static_cast<R>(std::log(rq.ki_barrier)) : R(-1e30);
        a.coupon = rq.coupon, a.put_strike = rq.put_strike, a.memory = rq.memory, a.ki_daily = rq.ki_daily;
    }
    const int block = 512;
    auto acc_bytes = [&](int b) { return static_cast<size_t>(b / 32) * 2 * a.n_out * sizeof(double); };
    const size_t budget = sizeof(R) == 4 ? (110u << 10) : (220u << 10);  // two blocks a SM in float, one in double
    auto aligned = [&] { return (blob.bytes.size() + 15) & ~static_cast<size_t>(15); };
    int tm = kTabStaged;
    if (table) {
        const size_t cells = static_cast<size_t>(rq.n_rows) * (rq.n_x - 1);
        if (aligned() + cells * sizeof(Pair2<R>) + acc_bytes(block) > budget) {
            tm = kTabGlobal;
            a.tab = upload_table<R>(plan.arena, rq.table, rq.n_rows, rq.n_x, nullptr);
        } else {
            a.off.table2 = blob.put<Pair2<R>>(nullptr, cells);
            pack_table<R>(rq.table, rq.n_x, rq.n_x - 1, 0, cells,
                          reinterpret_cast<Pair2<R>*>(blob.bytes.data() + a.off.table2));
        }
        NameStep<R>* ns = reinterpret_cast<NameStep<R>*>(blob.bytes.data() + a.off.name_step);
        for (size_t k = 0; k < static_cast<size_t>(S) * n; ++k)
            ns[k].row *= tm == kTabStaged ? rq.n_x - 1 : table_pitch<R>(rq.n_x);
    }
    a.smem_blob = a.smem_acc = static_cast<int>(aligned());
    const size_t smem = a.smem_acc + acc_bytes(block);
    if (smem > budget) return false;
    unsigned char* d = plan.arena.alloc<unsigned char>(std::max<size_t>(16, blob.bytes.size()));
    check_cuda(cudaMemcpy(d, blob.bytes.data(), blob.bytes.size(), cudaMemcpyHostToDevice), "copy blob");
    a.blob = d;
    const void* k = reinterpret_cast<const void*>(pick(tm));
    allow_smem(k, smem);
    if (occupancy(k, block, smem) < 1) return false;
    plan.n_names = n;
    // beside the kernel for many pairs those for fewer (McPlan::run chooses by each run's count)
    plan.kernel_legs = reinterpret_cast<const void*>(rq.product == OB_PRODUCT_LADDER
                                                         ? pick_legs<R, OB_PRODUCT_LADDER>(kind, n, tm, rq.mixer != 0)
                                                         : pick_legs<R, OB_PRODUCT_AUTOCALL>(kind, n, tm, rq.mixer != 0));
    if (plan.kernel_legs) allow_smem(plan.kernel_legs, smem);
    if (tm == kTabGlobal && pick(kTabStreamed)) {
        constexpr size_t kStreamBudget = 220u << 10;  // one block an SM
        const size_t acc = acc_bytes(kStreamedBlock);
        const int G = batch_steps(n, kind, false);
        if (plan_row_stream<R>(a.rs, rq.n_x, G, aligned(), kStreamBudget - acc)) {
            plan.kernel_rows = reinterpret_cast<const void*>(pick(kTabStreamed));
            plan.acc_rows = static_cast<int>(a.rs.off + row_stream_bytes(a.rs, G));
            plan.smem_rows = plan.acc_rows + acc;
            allow_smem(plan.kernel_rows, plan.smem_rows);
            if (occupancy(plan.kernel_rows, kStreamedBlock, plan.smem_rows) < 1) plan.kernel_rows = nullptr;
        }
    }
    plan.fused = true;
    plan.threads_per_pair = kind == 4 ? 2 : 1;
    plan.kernel = k;
    plan.block = block;
    plan.smem_bytes = smem;
    plan.n_out = a.n_out;
    plan.fused_args<R>() = a;
    return true;
}

// Whether a run of n_pairs on n names puts a pair's legs on two lanes: while an SM gets few warps of whole pairs.
// Kernel times, whole pairs against legs apart, 504 steps: one name (staged) 2^9 pairs 57 / 50 us, 2^13 60 / 53, 2^14.5 71 /
// 63, 2^15 72 / 71, 2^16 99 / 110; two names of 40 x 200 points 2^13 207 / 109, 2^15 194 / 135, 2^15.5 211 / 212; three
// 250 / 137, 237 / 202, 269 / 317; three of 801-point rows 398 / 190, 394 / 252, 410 / 432.
bool fused_legs_apart(int n, long long n_pairs, int sms) {
    return static_cast<double>(n_pairs) / (32.0 * sms) < (n == 1 ? 5.5 : 7.5);
}

// Whether a run of n_pairs streams its rows where the plan has that kernel (streams_rows has the times).
bool fused_streams_rows(long long n_pairs, int sms) { return streams_rows(n_pairs, sms, 12.0); }

template bool fused_build<float>(McPlan&, const ob_mc_request&);
template bool fused_build<double>(McPlan&, const ob_mc_request&);

}  // namespace ob
