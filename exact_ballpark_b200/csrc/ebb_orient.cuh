// SPDX-License-Identifier: MIT
// Dynamical orientation for a warp of 32 ships at once (EvolveBehaviorForBall's orientation branch, full.py:2459;
// GotoTorqueBreaks full.py:2155, GotoRollBreaks full.py:2224, ApplyTorque full.py:2292), warp-cooperative.
//
// Each torque search tries n1 = 1, 2, ... 99 accelerating ticks and keeps the first whose torque is within the
// maximum, in up to five rounds (each round re-derives the braking ticks n2): seven searches a ship and tick in the first
// ticks of the flight benchmark's worlds (their n1 a median of 10 and a mean of 16), 2.4 by the 200th. What bounds it is
// the issue of instructions, so the searches avoid most candidates, and every lane searches for its own ship
// (warp_search): it guesses n1 by bisection on the laws without their roundings, computes that candidate as the serial
// loop does (its kappa1 = tf^n1 by the serial loop's own float products, every eighth of them kept), and shows that every
// candidate before it fails by one comparison with bounds on what the serial loop's rounded operations can give
// (none_before). Where that does not settle a ship the neighbouring candidate is computed. What is left overshoots: the law
// passes long after num's nearest (the rolls at a mean n1 of 13 in the first ticks, 38 to 44 late in a flight). Eight lanes
// walk these ones' candidates, four ships at a time, from the last one shown to fail (of 96 to 99 in 100 every one up to
// the guess is), each told by bounds without a division, only those too near the maximum to be told computed (warp_walk).
// So the n1, alpha1 and kappa1 are the serial loop's, bit for bit.
// Of the searches 1 in 100 are walked at the 4th tick from rest, 14 at the 16th, 22 and 25 at the 32nd and 64th, 19 at the
// 128th and 200th. 65,536 worlds of 4 ships, us a tick at the 4th, 16th, 64th and 200th: 216, 313, 383 and 369; walked from
// the first candidate on 224, 344, 438 and 437; with 32 lanes on one ship and block of 32 candidates, all computed, 570,
// 506, 410 and 417. Over the first 8 ticks a second bisection past num's nearest in place of the walk was slower (312 us
// and 286), so were a scan of the law from there (401), the walk alone (636) and no neighbour (347). The set-up, the
// braking rounds (logf, pow) and ApplyTorque are one lane a ship too.
#pragma once

#include "ebb_flight.cuh"

namespace ebb {
namespace flight {

constexpr unsigned FULL_WARP = 0xffffffffu;
constexpr int GROUP = 8;                    // lanes that search one ship
constexpr int KAPPAS = 12;                  // a ship's kept kappas: kappa_8, kappa_16, ... kappa_96
constexpr int FOUND_FLOATS = 64;            // a warp's shared memory: each ship's found n1 and kappa1,
constexpr int ORIENT_FLOATS = FOUND_FLOATS + 32 * KAPPAS;      // and its kept kappas ([KAPPAS][32])

// One lane's ship for the warp's orientation step
struct DoLane {
    bool on;                 // live, and dynamical orientation applies
    D3 a;                    // in: the behaviour's thrust; out: the thrust after orientation
    float fmass, agility, sf, max_vel, max_ang_vel, rot_agility;
    bool warping;            // in warp proper: coasting, it turns toward its exit point
    F3 to_exit;              // (exit point - position) as floats
    F4 r0;
    F3 w0;
    F3 torque;               // out: GotoTorqueBreaks, GotoRollBreaks, ApplyTorque's rotation and angular velocity
    float roll;
    F4 rot1;
    F3 w1;
};

__device__ __forceinline__ float wbc(float v, int src) { return __shfl_sync(FULL_WARP, v, src); }
__device__ __forceinline__ int wbc(int v, int src) { return __shfl_sync(FULL_WARP, v, src); }
__device__ __forceinline__ F3 wbc(F3 v, int src) { return F3{wbc(v.x, src), wbc(v.y, src), wbc(v.z, src)}; }

// Bounds on a candidate without its divisions. Write A = n2dt kappa2 / (1 - kappa2) (tau without braking ticks) and
// u = 1 - kappa1: search_terms' num is tau - A kappa1 and its den tau (n1dt - A u) but for rounding. With each float
// operation's relative error at most 2^-24, num as the serial loop rounds it and as computed here (one fused operation,
// A's two) differ by less than 16 2^-24 (tau + |A| kappa1), the product by omega0 and the difference included; den by less
// than tau 8 2^-24 (n1dt + |A| u) beside its own last rounding; and the quotient, its square and its length add less than
// 2^-20 relatively, well inside the factors 0.998 and 1.002. Squared, (x + e)^2 <= 1.002 x^2 + 501 e^2 and
// (x - e)^2 >= 0.998 x^2 - 500 e^2. All of it in ranges where what underflows is far below the bounds and nothing overflows
// that the serial loop keeps (`plain` says where the bounds are not used: every candidate is then computed); a NaN decides
// nothing.
constexpr float NUM_ERROR = 1.0e-6f, DEN_ERROR = 5.0e-7f;      // above 16 2^-24 and 8 2^-24
struct Bounds {
    float A, tau, absA;
};
__device__ __forceinline__ bool in_range(float x, float lo, float hi) { return x >= lo && x <= hi; }

// the candidate's num and den as computed here, and what the serial loop's may differ by
__device__ __forceinline__ void candidate_terms(const Bounds& q, float k1, float n1dt, float* num, float* den, float* en,
                                                float* ed) {
    const float u = 1.0f - k1;
    *num = __fmaf_rn(-q.A, k1, q.tau);
    *den = q.tau * __fmaf_rn(-q.A, u, n1dt);
    *en = NUM_ERROR * __fmaf_rn(q.absA, k1, q.tau);
    *ed = DEN_ERROR * q.tau * __fmaf_rn(q.absA, u, n1dt);
}
// -1 the heading candidate fails, 1 it passes, 0 not told: |target - omega0 num|^2 against limit2 den^2
__device__ __forceinline__ int tell_heading(const Bounds& q, F3 target, F3 omega0, float omega2, float limit2, float k1,
                                            float n1dt) {
    float num, den, en, ed;
    candidate_terms(q, k1, n1dt, &num, &den, &en, &ed);
    const float x = __fmaf_rn(-omega0.x, num, target.x), y = __fmaf_rn(-omega0.y, num, target.y),
                z = __fmaf_rn(-omega0.z, num, target.z);
    const float v2 = __fmaf_rn(x, x, __fmaf_rn(y, y, z * z)), d2 = den * den;
    const float e2 = 520.0f * omega2 * en * en, f2 = 520.0f * ed * ed;
    const float low = __fmaf_rn(0.998f, v2, -e2), room = limit2 * __fmaf_rn(0.998f, d2, -f2);
    if (low > limit2 * __fmaf_rn(1.002f, d2, f2) && low > 1e-30f) return -1;
    if (__fmaf_rn(1.002f, v2, e2) < room && room > 1e-30f) return 1;
    return 0;
}
// the same of a roll candidate: |desired - omega num| against max |den|
__device__ __forceinline__ int tell_roll(const Bounds& q, float desired, float omega, float max_alpha, float k1, float n1dt) {
    float num, den, en, ed;
    candidate_terms(q, k1, n1dt, &num, &den, &en, &ed);
    const float v = fabs_(__fmaf_rn(-omega, num, desired)), d = fabs_(den), e = fabs_(omega) * en;
    const float low = __fmaf_rn(0.998f, v, -e), room = max_alpha * __fmaf_rn(0.998f, d, -ed);
    if (low > max_alpha * __fmaf_rn(1.002f, d, ed) && low > 1e-20f) return -1;
    if (__fmaf_rn(1.002f, v, e) < room && room > 1e-20f) return 1;
    return 0;
}

// One ship's search as its lane sets it up
struct Quest {
    Search q;
    float tf, max_alpha, limit2;
    bool squared;
    F3 target, omega0;                      // the heading's; a roll's desired angle and turning rate in x
};
// alpha1 and whether it is within the maximum, as the serial loop computes them (full.py:2189-2201, 2264-2276; the roll's
// by a true division)
template <bool ROLL>
__device__ __forceinline__ bool candidate(const Quest& s, float k1, float n1dt, F3* a1) {
    float num, den;
    search_terms(s.q, k1, n1dt, &num, &den);
    if (ROLL) {
        a1->x = fdiv(fsub(s.target.x, fmul(s.omega0.x, num)), den);
        return fabs_(a1->x) < s.max_alpha;
    }
    *a1 = f3_div(f3_sub(s.target, f3_mul(s.omega0, num)), den);
    return s.squared ? f3_dot(*a1, *a1) < s.limit2 : f3_len(*a1) < s.max_alpha;
}

// The searches of the lanes in `want` candidate by candidate, four ships at a time, eight lanes a ship: each lane's n1 and
// kappa1 (n1 = 100 with the 99th candidate's kappa1 when none passes), and its alpha1, left in that lane. `fail`: every
// candidate up to it is known to fail, so a ship's walk starts with the block of GROUP that holds the next one.
template <bool ROLL>
__device__ __forceinline__ void warp_walk(unsigned want, const Quest& mine, const Bounds& mine_bd, float o2, bool plain,
                                          int fail, const float* ndt_tab, float* found, int* n1_out, F3* a1_out,
                                          float* k1_out) {
    const int lane = threadIdx.x & 31, sub = lane & (GROUP - 1), first = lane & ~(GROUP - 1);
    const unsigned group = ((1u << GROUP) - 1u) << first;
    const bool searching = (want >> lane) & 1;
    while (want) {
        unsigned m = want;                                   // the next four ships, one a group
        int src = -1;
#pragma unroll
        for (int g = 0; g < 32 / GROUP; ++g) {
            const int k = __ffs(m) - 1;
            if (g == (lane / GROUP)) src = k;
            m &= m - 1;
        }
        want = m;
        const int from = src < 0 ? lane : src;
        Bounds bd;
        bd.A = wbc(mine_bd.A, from);
        bd.tau = wbc(mine.q.tau, from);
        bd.absA = fabs_(bd.A);
        const float tf = wbc(mine.tf, from), max_alpha = wbc(mine.max_alpha, from);
        float limit2 = 0.0f, omega2 = 0.0f;
        F3 target, omega0;
        if (ROLL) {
            target.x = wbc(mine.target.x, from);
            omega0.x = wbc(mine.omega0.x, from);
        } else {
            target = wbc(mine.target, from);
            omega0 = wbc(mine.omega0, from);
            limit2 = wbc(mine.limit2, from);
            omega2 = wbc(o2, from);
        }
        const bool untold = wbc((int)plain, from) != 0;
        const int failed = wbc(fail, from);
        int b = failed & ~(GROUP - 1);
        float k1 = b ? fmul(found[FOUND_FLOATS + (b / GROUP - 1) * 32 + from], tf) : tf;
#pragma unroll
        for (int i = 1; i < GROUP; ++i)                      // kappa_{b + sub + 1}
            if (i <= sub) k1 = fmul(k1, tf);
        bool open = src >= 0;
        for (;; b += GROUP) {
            const int n = b + sub + 1;
            const float n1dt = ndt_tab[n < TORQUE_STEPS ? n : TORQUE_STEPS - 1];
            int told = 0;
            if (!untold)
                told = ROLL ? tell_roll(bd, target.x, omega0.x, max_alpha, k1, n1dt)
                            : tell_heading(bd, target, omega0, omega2, limit2, k1, n1dt);
            if (n >= TORQUE_STEPS || n <= failed) told = -1;
            unsigned maybe = __ballot_sync(FULL_WARP, open && told >= 0) & group;
            const bool doubt = maybe != 0 && lane == __ffs(maybe) - 1 && told == 0;
            if (__any_sync(FULL_WARP, doubt)) {              // a group's first is not told: its candidates are computed
                Quest s;
                s.q.tau = bd.tau;
                s.q.n2 = wbc(mine.q.n2, from);
                s.q.kappa2 = wbc(mine.q.kappa2, from);
                s.q.n2dt = wbc(mine.q.n2dt, from);
                s.q.one_k2 = wbc(mine.q.one_k2, from);
                s.tf = tf;
                s.max_alpha = max_alpha;
                s.limit2 = limit2;
                s.squared = wbc((int)mine.squared, from) != 0;
                s.target = target;
                s.omega0 = omega0;
                F3 a1;
                if (told == 0) told = candidate<ROLL>(s, k1, n1dt, &a1) ? 1 : -1;
                maybe = __ballot_sync(FULL_WARP, open && told > 0) & group;
            }
            const bool last = b + GROUP >= TORQUE_STEPS - 1;
            if (open && (maybe || last)) {
                // the first that passes (every one before it fails), or the 99th
                const int w = maybe ? __ffs(maybe) - 1 : first + (TORQUE_STEPS - 2 - b);
                if (lane == w) {
                    found[2 * src] = __int_as_float(maybe ? n : TORQUE_STEPS);
                    found[2 * src + 1] = k1;
                }
                open = false;
            }
            if (!__any_sync(FULL_WARP, open)) break;
#pragma unroll
            for (int i = 0; i < GROUP; ++i) k1 = fmul(k1, tf);
        }
    }
    __syncwarp();
    if (searching) {
        const int n1 = __float_as_int(found[2 * lane]);
        const float k1 = found[2 * lane + 1];
        candidate<ROLL>(mine, k1, ndt_tab[n1 < TORQUE_STEPS ? n1 : TORQUE_STEPS - 1], a1_out);
        *n1_out = n1;
        *k1_out = k1;
    }
    __syncwarp();
}

__device__ __forceinline__ float exp2_near(float x) {
    float y;
    asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// kappa_n exactly, n < 100: the kept one below it and the products from there
__device__ __forceinline__ float kappa_at(const float* kept, int n, float tf) {
    const int b = n / GROUP, r = n % GROUP;
    float k = b ? kept[(b - 1) * 32] : 1.0f;
#pragma unroll
    for (int i = 1; i < GROUP; ++i)
        if (i <= r) k = fmul(k, tf);
    return k;
}
// Whether every candidate 1 .. n fails, told at once: num rises with n (kappa1 falls) from `first`, so the least
// |target - omega0 num| is at num's nearest to the line's foot (the same roll: where the coast ends on the target); den
// rises with n but for what the kappas' own rounding takes back, at most |A| (1 - tf + 2^-23) - dt a candidate.
template <bool ROLL>
__device__ __forceinline__ bool none_before(const Bounds& q, const Quest& s, float o2, float first, float foot, float kn,
                                            int n, float ndt_n, float dt) {
    const float num = fminf(fmaxf(foot, first), __fmaf_rn(-q.A, kn, q.tau));
    const float en = NUM_ERROR * (q.tau + q.absA);
    const float back = fmaxf(0.0f, __fmaf_rn(q.absA, (1.0f - s.tf) + 1.3e-7f, -dt)) * (float)n * 1.01f;
    const float u = 1.0f - kn;
    const float d = q.tau * (fabs_(__fmaf_rn(-q.A, u, ndt_n)) + back), ed = DEN_ERROR * q.tau * __fmaf_rn(q.absA, u, ndt_n);
    if (ROLL) {
        const float v = fabs_(__fmaf_rn(-s.omega0.x, num, s.target.x)), e = fabs_(s.omega0.x) * en;
        const float low = __fmaf_rn(0.998f, v, -e);
        return low > s.max_alpha * __fmaf_rn(1.002f, d, ed) && low > 1e-20f;
    }
    const float x = __fmaf_rn(-s.omega0.x, num, s.target.x), y = __fmaf_rn(-s.omega0.y, num, s.target.y),
                z = __fmaf_rn(-s.omega0.z, num, s.target.z);
    const float v2 = __fmaf_rn(x, x, __fmaf_rn(y, y, z * z));
    const float low = __fmaf_rn(0.998f, v2, -520.0f * o2 * en * en);
    return low > s.limit2 * __fmaf_rn(1.002f, d * d, 520.0f * ed * ed) && low > 1e-30f;
}

// The round's searches of the lanes in `want`: each searching lane's n1, kappa1 and alpha1. A lane guesses its own ship's
// n1 by bisection on the laws without their roundings, num's best so far in place of num, so that a passing candidate is
// followed by passing ones alone; computes that candidate as the serial loop does, and tells by bounds whether every one
// before it fails; where the two don't settle it, the one before a guess that passes or after one that fails is computed,
// and the ships still open walked from what was shown to fail.
template <bool ROLL>
__device__ __forceinline__ void warp_search(unsigned want, const Quest& mine, const float* ndt_tab, float* found, float dt,
                                            int* n1_out, F3* a1_out, float* k1_out) {
    const int lane = threadIdx.x & 31;
    const float* kept = found + FOUND_FLOATS + lane;
    bool settled = true, near = false, pass1 = false;
    Bounds bd;
    float first = 0.0f, foot = 0.0f, kb = 0.0f, k1 = 0.0f;
    int n = 0, fail = 0;                                     // every candidate up to `fail` fails
    float o2 = 0.0f;
    bool plain = false;
    if ((want >> lane) & 1) {
        bd.tau = bd.A = mine.q.tau;
        if (mine.q.n2 != 0) bd.A = fdiv(fmul(mine.q.n2dt, mine.q.kappa2), mine.q.one_k2);
        bd.absA = fabs_(bd.A);
        o2 = f3_dot(mine.omega0, mine.omega0);
        const float t2 = f3_dot(mine.target, mine.target), to = f3_dot(mine.target, mine.omega0);
        plain = !(in_range(mine.q.tau, 1e-8f, 1e8f) && bd.absA <= 1e8f && in_range(mine.tf, 0.0f, 1.0f) &&
                  (ROLL ? in_range(mine.max_alpha, 1e-8f, 1e8f) : mine.squared && in_range(mine.limit2, 1e-16f, 1e16f)) &&
                  t2 < 1e8f && o2 < 1e8f && in_range(dt, 1e-4f, 1e4f));
        settled = false;
        if (!plain) {
            const float l2 = __log2f(mine.tf), m2 = ROLL ? mine.max_alpha * mine.max_alpha : mine.limit2;
            first = __fmaf_rn(-bd.A, mine.tf, bd.tau);
            foot = __fdividef(to, o2);
            int below = 0;
            n = TORQUE_STEPS;
#pragma unroll 1
            while (n - below > 1) {
                const int mid = (below + n) >> 1;
                const float nf = (float)mid, k = exp2_near(nf * l2), u = 1.0f - k;
                const float num = __fmaf_rn(-bd.A, k, bd.tau), den = bd.tau * __fmaf_rn(-bd.A, u, nf * dt);
                const float best = fminf(fmaxf(foot, first), num);   // (num's best up to there: so a pass stays one)
                const bool pass = __fmaf_rn(__fmaf_rn(o2, best, -2.0f * to), best, t2) < m2 * den * den;
                below = pass ? below : mid;
                n = pass ? mid : n;
            }
            kb = kappa_at(kept, n - 1, mine.tf);
            const bool none = n == TORQUE_STEPS;             // (then the 99th's values)
            k1 = none ? kb : fmul(kb, mine.tf);
            pass1 = candidate<ROLL>(mine, k1, ndt_tab[none ? n - 1 : n], a1_out);
            near = n < TORQUE_STEPS - 1;
            if (n > 1 && none_before<ROLL>(bd, mine, o2, first, foot, kb, n - 1, ndt_tab[n - 1], dt)) fail = n - 1;
            settled = (none ? !pass1 : pass1) && fail == n - 1;
            *n1_out = n;
            *k1_out = k1;
        }
    }
    if (!settled && near) {
        const int q = pass1 ? n - 1 : n + 1;                 // (a passing guess of 1 is settled)
        const float kq = pass1 ? kb : fmul(k1, mine.tf);
        F3 a1;
        const bool pass = candidate<ROLL>(mine, kq, ndt_tab[q], &a1);
        if (pass1) {                                         // the candidates before the one before
            const int m = n - 2;
            settled = m == 0 || none_before<ROLL>(bd, mine, o2, first, foot, kappa_at(kept, m, mine.tf), m, ndt_tab[m], dt);
            fail = settled ? m : 0;
        } else if (fail == n - 1) {
            settled = pass;
            fail = q;                                        // (or it passes)
        }
        if (pass) {
            *a1_out = a1;
            *n1_out = q;
            *k1_out = kq;
        }
    }
    const unsigned open = __ballot_sync(FULL_WARP, !settled);
    if (open) warp_walk<ROLL>(open, mine, bd, o2, plain, fail, ndt_tab, found, n1_out, a1_out, k1_out);
}

// The warp's orientation step: every lane calls it together (lanes whose ship is off pass through). `found` is the
// warp's ORIENT_FLOATS floats of shared memory; `ndt_tab` the block's table float(n dt).
__device__ __forceinline__ void orient_warp(DoLane& d, const Cfg& c, const float* ndt_tab, float* found) {
    const F3 zero = F3{0.0f, 0.0f, 0.0f};
    d.torque = zero;
    d.roll = 0.0f;
    d.rot1 = d.r0;
    d.w1 = d.w0;
    PowCache pc;
    pow_cache_clear(pc);
    Turn t;
    float accel = 0.0f, inertia = 1.0f;
    bool thrust = false;
    F3 a32 = zero;
    if (d.on) {                                                       // full.py:2463-2465, 2115-2124
        accel = tof(d3_len(d.a));
        const float fmag = fmul(d.fmass, d.agility);
        const float max_accel = fdiv(fmul(fmul(c.ffriction, d.sf), d.max_vel), fmag);
        thrust = tod(accel) > dmul(DO_THRUST, tod(max_accel));
        t.max_ang_vel = d.max_ang_vel;
        inertia = fmul(fmag, d.rot_agility);
        t.t_scale = fdiv(c.ffriction, inertia);
        t.tf = lm::expf(fmul(fneg(c.fdt), t.t_scale));
        t.tau_s = fdiv(1.0f, t.t_scale);
        t.dt = c.dt;
        t.fdt = c.fdt;
        t.ndt_tab = ndt_tab;
        a32 = f3_of(d.a);
        float k = 1.0f;                                               // the kept kappas, as the loops form them
        float* kept = found + FOUND_FLOATS + (threadIdx.x & 31);
        for (int b = 0; b < KAPPAS; ++b) {
#pragma unroll
            for (int i = 0; i < GROUP; ++i) k = fmul(k, t.tf);
            kept[b * 32] = k;
        }
    }
    __syncwarp();

    // ---- GotoTorqueBreaks: the heading torque (toward the thrust, or a coasting warper's exit point)
    bool h_active = false;
    F3 h_target = zero, h_omega0 = zero, h_alpha1 = zero, h_alpha2 = zero;
    float h_max = 0.0f, h_limit2 = 0.0f, h_kappa1 = 1.0f, h_kappa2 = 1.0f, h_g = 0.0f;
    int h_n1 = 0, h_n2 = 0;
    bool h_sq = false;
    if (d.on && (thrust || d.warping)) {
        const F3 dir = thrust ? a32 : d.to_exit;
        h_max = fmul(t.max_ang_vel, t.t_scale);
        const float len_dir = f3_len(dir);
        if (!(h_max <= 0.0f) && !(len_dir == 0.0f)) {
            const F3 heading = f3_unit(m_apply(F3{0.0f, 0.0f, 1.0f}, m_of_q(d.r0)));
            F3 target = f3_div(f3_cross(heading, dir), len_dir);
            const float rot_len = f3_len(target);
            const float rot_angle = lm::acosf(fmax_(-1.0f, fmin_(1.0f, fdiv(f3_dot(dir, heading), len_dir))));
            if (tod(rot_len) > 1e-12) target = f3_mul(target, fdiv(rot_angle, rot_len));
            else if (rot_angle > 1.0f) target = F3{fneg(rot_angle), 0.0f, 0.0f};
            const F3 omega0 = f3_sub(d.w0, f3_mul(heading, f3_dot(heading, d.w0)));
            const float len_omega0 = f3_len(omega0);
            if (!(dmul(tod(len_omega0), t.dt) < 1e-4 && tod(rot_angle) < 1e-4)) {
                h_active = true;
                h_target = target;
                h_omega0 = omega0;
                h_sq = sqrt_threshold(h_max, &h_limit2);
                if (braking(t, len_omega0, &h_n2, &h_kappa2, &h_g, pc))
                    h_alpha2 = f3_mul(F3{fneg(omega0.x), fneg(omega0.y), fneg(omega0.z)}, h_g);
            }
        }
    }
    const bool h_ran = h_active;
    for (int round = 0; round < TORQUE_ROUNDS; ++round) {
        Search q;
        q.tau = t.tau_s;
        q.n2 = h_n2;
        q.kappa2 = h_kappa2;
        q.n2dt = 0.0f;
        q.one_k2 = 0.0f;
        if (h_active) {
            q.n2dt = ndt(h_n2, t.dt);
            q.one_k2 = fsub(1.0f, h_kappa2);
            if (h_n2 > 0) {
                const F3 theta2 = f3_add(f3_mul(f3_mul(h_alpha2, q.tau), fsub(q.n2dt, fmul(q.tau, q.one_k2))),
                                         f3_mul(f3_mul(h_omega0, q.tau), q.one_k2));
                if (tod(f3_len(f3_sub(h_target, theta2))) < 1e-3) {    // braking alone gets there
                    h_n1 = 0;
                    h_active = false;
                }
            }
        }
        const unsigned want = __ballot_sync(FULL_WARP, h_active);
        if (!want) break;
        const Quest mine{q, t.tf, h_max, h_limit2, h_sq, h_target, h_omega0};
        warp_search<false>(want, mine, ndt_tab, found, c.fdt, &h_n1, &h_alpha1, &h_kappa1);
        if (h_active) {
            const F3 omega1 = f3_add(f3_mul(h_alpha1, fmul(t.tau_s, fsub(1.0f, h_kappa1))), f3_mul(h_omega0, h_kappa1));
            const int n2_old = h_n2;
            h_alpha2 = zero;
            if (braking(t, f3_len(omega1), &h_n2, &h_kappa2, &h_g, pc))
                h_alpha2 = f3_mul(F3{fneg(omega1.x), fneg(omega1.y), fneg(omega1.z)}, h_g);
            if (h_n2 == n2_old) h_active = false;
        }
    }
    if (h_ran) {
        if (h_n1 > 0) d.torque = h_n1 > 1 ? f3_mul(f3_unit(h_alpha1), h_max) : h_alpha1;
        else if (h_n2 > 0) d.torque = h_alpha2;
    }

    // ---- GotoRollBreaks: the roll torque, rolling into strong turns, otherwise upright
    bool r_active = false;
    float r_max = 0.0f, r_desired = 0.0f, r_omega = 0.0f, r_alpha1 = 0.0f, r_alpha2 = 0.0f, r_kappa1 = 1.0f;
    float r_kappa2 = 1.0f, r_g = 0.0f;
    int r_n1 = 0, r_n2 = 0;
    if (d.on) {
        r_max = fmul(t.t_scale, t.max_ang_vel);
        if (!(r_max <= 0.0f)) {
            const M3 mat = m_of_q(q_conj(d.r0));
            const F3 ship_omega = m_apply(d.w0, mat);
            r_omega = ship_omega.z;
            const float len_torque = f3_len(d.torque);
            float turn_roll = 0.0f, weight = 0.0f;
            if (tod(len_torque) > dmul(0.05, tod(r_max))) {
                const F3 ship_torque = m_apply(d.torque, mat);
                const F3 flat = F3{ship_omega.x, ship_omega.y, 0.0f};
                if (f3_dot(flat, ship_torque) >= 0.0f || f3_len(flat) < fmul(tof(0.01), t.max_ang_vel)) {
                    turn_roll = lm::atan2f(fneg(ship_torque.y), fneg(ship_torque.x));
                    weight = fdiv(len_torque, t.t_scale);
                    if (weight > 1.0f) weight = 1.0f;
                }
            }
            const F3 up = m_apply(F3{0.0f, 1.0f, 0.0f}, mat);
            const float up_roll = up.z < tof(0.95) ? lm::atan2f(fneg(up.x), up.y) : 0.0f;
            r_desired = weight < tof(0.05) ? up_roll : fmul(weight, turn_roll);
            if (!(tod(fabs_(r_omega)) < 1e-4 && tod(fabs_(r_desired)) < 1e-4)) {
                r_active = true;
                if (braking(t, fabs_(r_omega), &r_n2, &r_kappa2, &r_g, pc)) r_alpha2 = fmul(fneg(r_omega), r_g);
            }
        }
    }
    const bool r_ran = r_active;
    for (int round = 0; round < TORQUE_ROUNDS; ++round) {
        Search q;
        q.tau = t.tau_s;
        q.n2 = r_n2;
        q.kappa2 = r_kappa2;
        q.n2dt = 0.0f;
        q.one_k2 = 0.0f;
        if (r_active) {
            q.n2dt = ndt(r_n2, t.dt);
            q.one_k2 = fsub(1.0f, r_kappa2);
            if (r_n2 > 0) {
                const float theta2 = fadd(fmul(fmul(q.tau, r_alpha2), fsub(q.n2dt, fmul(q.tau, q.one_k2))),
                                          fmul(fmul(q.tau, r_omega), q.one_k2));
                if (tod(fabs_(fsub(r_desired, theta2))) < 1e-3) {
                    r_n1 = 0;
                    r_active = false;
                }
            }
        }
        const unsigned want = __ballot_sync(FULL_WARP, r_active);
        if (!want) break;
        const Quest mine{q, t.tf, r_max, 0.0f, false, F3{r_desired, 0.0f, 0.0f}, F3{r_omega, 0.0f, 0.0f}};
        F3 a1 = zero;
        warp_search<true>(want, mine, ndt_tab, found, c.fdt, &r_n1, &a1, &r_kappa1);
        if (r_active) r_alpha1 = a1.x;
        if (r_active) {
            const float omega1 = fadd(fmul(fmul(r_alpha1, t.tau_s), fsub(1.0f, r_kappa1)), fmul(r_omega, r_kappa1));
            const int n2_old = r_n2;
            r_alpha2 = 0.0f;
            if (braking(t, fabs_(omega1), &r_n2, &r_kappa2, &r_g, pc)) r_alpha2 = fmul(fneg(omega1), r_g);
            if (r_n2 == n2_old) r_active = false;
        }
    }
    if (r_ran) {
        if (r_n1 > 0) d.roll = r_n1 > 1 ? fmul(r_alpha1 >= 0.0f ? 1.0f : -1.0f, r_max) : r_alpha1;
        else if (r_n2 > 0) d.roll = r_alpha2;
    }

    // ---- ApplyTorque (the tick's rotation, the commit's too) and the thrust along the heading a tick on
    if (d.on) {
        const float tau = fdiv(inertia, c.ffriction);
        const Turned tr = apply_torque(d.r0, d.w0, d.torque, d.roll, tau, c.fdt);
        d.rot1 = tr.rot;
        d.w1 = tr.w;
        if (thrust) {
            const F3 heading = m_apply(F3{0.0f, 0.0f, 1.0f}, m_of_q(d.rot1));
            const float cosangle = fmin_(1.0f, fdiv(f3_dot(heading, a32), accel));
            d.a = (cosangle <= 0.0f) ? D3{0.0, 0.0, 0.0} : d3_of(f3_mul(heading, fmul(fmul(cosangle, cosangle), accel)));
        }
    }
    __syncwarp();
}

}  // namespace flight
}  // namespace ebb
