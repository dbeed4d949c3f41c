// force_device.cuh -- device code of the i-block x j-particle direct sum,
// shared by the launch-per-call kernels (force.cu) and the resident serving
// kernel (resident.cu): per-i register state, the pair terms, one j-tile's
// consumption, and one task (an i-tile against a j-split) with its bulk-copy
// pipeline and its epilogue.  The pair terms' reference and the work
// decomposition are described at the top of force.cu.
#pragma once
#include <cfloat>
#include "common.cuh"
#include "kernels.h"
#include "predict_device.cuh"

namespace g6 {

constexpr uint64_t kWaitLimitNs = 1000000000ull;  // 1 s per tile wait
#ifndef G6B200_FOLD_TERMS
#define G6B200_FOLD_TERMS 64
#endif
constexpr int kFlush = G6B200_FOLD_TERMS;         // FP32 terms per FP64 fold
constexpr int kMaxWarps = 8;

// Variant bits of the mixed kernels: 2 = inner j-loop of the scalar layout
// unrolled by 4 (else 2): 1.3% faster.  (The paired layout's loop is
// unrolled by 16 with the indicators on, by 4 otherwise.)
constexpr int kVarUnroll4 = 2;
// 4 = GRAPE-4 pipeline (FP64 kernel only; see the file header).
constexpr int kVarG4 = 4;
// 8 = potential only (paired mixed and FP64 layouts): the energy sweeps.
constexpr int kVarPot = 8;
// 16 = paired mixed layout: also track the refinement's error indicators
// (the largest single acc and jerk terms: one FP32x2 multiply and two
// three-input integer maxima per pair of j).
constexpr int kVarStats = 16;

// T j per shared-memory tile, held as U records of JPU j each.
template <int K> struct Traits;
template <> struct Traits<kKernMixedDS> {
    using JRec = JRecMixed;
    static constexpr int T = 256, JPU = 1, U = T;
};
template <> struct Traits<kKernMixedP> {
    using JRec = JPairMixed;
    static constexpr int T = 256, JPU = 2, U = T / 2;
};
template <> struct Traits<kKernF64> {
    using JRec = JRecF64;
    static constexpr int T = 128, JPU = 1, U = T;
};

constexpr unsigned kHiInf = 0x7ff00000u;  // upper word of the FP64 +inf

// Per-i register state.

struct StateMixedBase {
    float vx, vy, vz, h2;
    float ax, ay, az, jx, jy, jz, pt;   // FP32 sums since the last fold
    double Ax, Ay, Az, Jx, Jy, Jz, Pt;  // FP64 totals
    float nr2;                          // best r^2 so far
    int nj, idx, i;
};

struct StateMixed : StateMixedBase {
    float xh, yh, zh, xl, yl, zl;
};

struct StateF64 {
    double x, y, z, vx, vy, vz, h2;
    double eps2;  // softening: the call's, or (GRAPE-4 variant) this i's
    double Ax, Ay, Az, Jx, Jy, Jz, Pt;  // acc, jerk x 3 sqrt(3), pot x sqrt(3): see inv_dist_s3
    unsigned nhi;  // smallest upper word of r^2 so far
    int nk;        // first j of the run that first reached it (-1: none)
    int nties;     // further runs that reached it: their first j are in process_task's ties[]
    double nr2;
    int nj, idx, i;
};

template <int K> struct StateOf;
template <> struct StateOf<kKernMixedDS> { using type = StateMixed; };
template <> struct StateOf<kKernF64> { using type = StateF64; };

__device__ __forceinline__ void nb_push(const ForceParams &p, int i, int j) {
    int k = atomicAdd(&p.nb_count[i], 1);
    if (k < p.nb_cap) p.nb_list[(size_t)i * p.nb_cap + k] = j;
}

__device__ __forceinline__ void init_mixed(StateMixedBase &s, const IRec &q) {
    s.vx = (float)q.v[0];
    s.vy = (float)q.v[1];
    s.vz = (float)q.v[2];
    s.h2 = (float)q.h2;
    s.idx = q.index;
    s.ax = s.ay = s.az = s.jx = s.jy = s.jz = s.pt = 0.f;
    s.Ax = s.Ay = s.Az = s.Jx = s.Jy = s.Jz = s.Pt = 0.0;
    s.nr2 = FLT_MAX;
    s.nj = -1;
}

__device__ __forceinline__ void load_i(StateMixed &s, const IRec &q, const ForceParams &p, bool &range_ok) {
    range_ok &= to_fixed_split(q.x[0], p.fs, s.xh, s.xl);
    range_ok &= to_fixed_split(q.x[1], p.fs, s.yh, s.yl);
    range_ok &= to_fixed_split(q.x[2], p.fs, s.zh, s.zl);
    init_mixed(s, q);
}

__device__ __forceinline__ void load_i(StateF64 &s, const IRec &q, const ForceParams &p, bool &) {
    s.x = q.x[0];
    s.y = q.x[1];
    s.z = q.x[2];
    s.vx = q.v[0];
    s.vy = q.v[1];
    s.vz = q.v[2];
    s.h2 = q.h2;
    s.idx = q.index;
    s.eps2 = p.eps2;
    s.Ax = s.Ay = s.Az = s.Jx = s.Jy = s.Jz = s.Pt = 0.0;
    s.nhi = kHiInf;
    s.nk = -1;
    s.nties = 0;
    s.nr2 = DBL_MAX;
    s.nj = -1;
}

// A j-particle as the mixed kernels see it after the shared-memory load.
struct JMixed {
    float dx, dy, dz;  // exact position difference rounded to FP32
    float vx, vy, vz, m;
    int index;
};

__device__ __forceinline__ void diff(const StateMixed &s, const JRecMixed &J, JMixed &o) {
    const float4 hi = J.hi, lo = J.lo, ve = J.vel;
    o.dx = (hi.x - s.xh) + (lo.x - s.xl);
    o.dy = (hi.y - s.yh) + (lo.y - s.yl);
    o.dz = (hi.z - s.zh) + (lo.z - s.zl);
    o.vx = ve.x;
    o.vy = ve.y;
    o.vz = ve.z;
    o.m = hi.w;
    o.index = __float_as_int(lo.w);
}

template <bool CHK, bool NB, bool IDENT, class S>
__device__ __forceinline__ void interact_mixed(S &s, const JMixed &J, int jg, float eps2, const ForceParams &p) {
    const float dvx = J.vx - s.vx;
    const float dvy = J.vy - s.vy;
    const float dvz = J.vz - s.vz;
    const float r2n = fmaf(J.dz, J.dz, fmaf(J.dy, J.dy, J.dx * J.dx));
    const float rv = fmaf(J.dz, dvz, fmaf(J.dy, dvy, J.dx * dvx));
    float r2 = r2n + eps2;
    float mj = J.m;
    float r2nn = r2n;
    bool self = false;
    if (CHK) {
        self = IDENT ? (jg == s.idx) : (J.index == s.idx);
        r2 = self ? 1.f : r2;
        mj = self ? 0.f : mj;
        r2nn = self ? FLT_MAX : r2nn;
    }
    float y = rsqrt_approx(r2);
    // One Newton-Raphson step: y <- y (1.5 - 0.5 r2 y^2).
    const float hy = (0.5f * r2) * y;
    y = y * fmaf(-hy, y, 1.5f);
    const float r2inv = y * y;
    const float mr = mj * y;
    const float mr3 = mr * r2inv;
    const float a3 = -3.f * rv * r2inv;
    s.pt -= mr;
    s.ax = fmaf(mr3, J.dx, s.ax);
    s.ay = fmaf(mr3, J.dy, s.ay);
    s.az = fmaf(mr3, J.dz, s.az);
    s.jx = fmaf(mr3, fmaf(a3, J.dx, dvx), s.jx);
    s.jy = fmaf(mr3, fmaf(a3, J.dy, dvy), s.jy);
    s.jz = fmaf(mr3, fmaf(a3, J.dz, dvz), s.jz);
    if (r2nn < s.nr2) {
        s.nr2 = r2nn;
        s.nj = jg;
    }
    if (NB) {
        bool hit = CHK && self ? (p.include_self && s.h2 > 0.f) : (r2n < s.h2);
        if (hit) nb_push(p, s.i, jg);
    }
}

// ---- FP64 layout.
//
// What bounds this loop is the register ports: a scheduler reads one 64-bit
// register operand per cycle for its warp, so an FP64 instruction with three
// different register operands takes 3 cycles, one with two takes the FP64
// pipe's 2 (measured: 3.04 and 2.04; an operand shared with the previous
// instruction, or a literal one, is free).  The loop below is written
// against that count -- about 72 cycles per j and warp:
//   * the inverse distance is the PTX approximation and one third-order step
//     in line (11 cycles; rsqrt() measured 26, with a branch for the special
//     values that keeps the pair terms of neighbouring j apart);
//   * it is scaled by sqrt(3), so that 3 (dr.dv) / r^2 needs no product of
//     its own;
//   * the nearest neighbour is kept as the upper word of r^2 (one integer
//     minimum per j instead of an FP64 compare and three selects).
// 16384 x 262144: 10.55 -> 9.40 ms; potential only, 65536 x 65536: 5.39 ->
// 3.69 ms.
constexpr double kThird = 1.0 / 3.0;

// sqrt(3) / r (r^2 finite, normal, positive) from x = r^2 / 3 and q = c x.
// The approximation y is taken of x; the residual e = c - q y^2 is that of q.
// With q = x, one instruction less, the result is off by what 1/3 is no
// double, 2.8e-17: enough for the potential, whose sum is scaled back by it
// (to_partial).  But every 3 (dr.dv) / r^2 then is 5.5e-17 too large, and the
// jerk's error against long doubles above the one with rsqrt() (1500 x 1500
// over eight clusters, rms: 5.21e-16 against 4.80e-16); the forces take q =
// r^2 itself: 4.64e-16, for 2 % of a 65536 x 65536 sweep.
// y's low word is zero, so that y^2 is exact.  Its relative error e / 2c,
// below 2^-19, goes to 5/16 (e/c)^3 by Householder's third-order step for
// x^(-1/2) (A. S. Householder, "The Numerical Treatment of a Single
// Nonlinear Equation", 1970), y (1 + (e/c)/2 + 3/8 (e/c)^2): below FP64's
// rounding.
template <int C>
__device__ __forceinline__ double inv_dist_s3(double x, double q) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-q, y * y, (double)C);
    return fma(y * e, fma(e, 0.375 / (C * C), 0.5 / C), y);
}

__device__ __forceinline__ double r2_f64(double dx, double dy, double dz) {
    return __fma_rn(dz, dz, __fma_rn(dy, dy, dx * dx));
}

template <bool IDENT>
__device__ __forceinline__ bool is_self(const StateF64 &s, const double4 &vel, int jg) {
    return IDENT ? jg == s.idx : vel.w == (double)s.idx;
}

// One pair term for any r^2 (zero, subnormal and infinite ones too) and of any
// size: not scaled.
template <bool CHK, bool IDENT, bool G4, bool PO>
__device__ __forceinline__ void interact_any(StateF64 &s, const double4 &pos, const double4 &vel, int jg) {
    const double dx = pos.x - s.x, dy = pos.y - s.y, dz = pos.z - s.z;
    double r2 = G4 ? g4_r2(dx, dy, dz, s.eps2) : r2_f64(dx, dy, dz) + s.eps2;
    double mj = pos.w;
    if (G4 ? !(r2 > 0.0) : (CHK && is_self<IDENT>(s, vel, jg))) {
        r2 = 1.0;
        mj = 0.0;
    }
    const double rinv = rsqrt(r2);
    const double mr = mj * rinv;
    s.Pt -= mr;
    if constexpr (!PO) {
        const double dvx = vel.x - s.vx, dvy = vel.y - s.vy, dvz = vel.z - s.vz;
        const double rv = dx * dvx + dy * dvy + dz * dvz;
        const double r2inv = rinv * rinv;
        const double mr3 = mr * r2inv;
        const double a3 = -3.0 * rv * r2inv;
        s.Ax += mr3 * dx;
        s.Ay += mr3 * dy;
        s.Az += mr3 * dz;
        s.Jx += mr3 * (dvx + a3 * dx);
        s.Jy += mr3 * (dvy + a3 * dy);
        s.Jz += mr3 * (dvz + a3 * dz);
    }
}

// One pair term, r^2 / 3 taken as finite, normal and positive (the caller
// sums again with interact_any when it was not: the sums then are not
// finite).  Returns the upper word of the unsoftened r^2 (all ones for the
// particle itself).
template <bool CHK, bool NB, bool IDENT, bool G4, bool PO>
__device__ __forceinline__ unsigned interact(StateF64 &s, const JRecF64 &J, int jg, const ForceParams &p) {
    const double dx = J.pos.x - s.x, dy = J.pos.y - s.y, dz = J.pos.z - s.z;
    double r2 = G4 ? g4_r2(dx, dy, dz, s.eps2) : r2_f64(dx, dy, dz);
    double m = J.pos.w;
    unsigned hi = (unsigned)__double2hiint(r2);
    bool self = false;
    if (CHK && !G4) self = is_self<IDENT>(s, J.vel, jg);
    if (NB) {
        const bool hit = CHK && self ? (p.include_self && s.h2 > 0.0) : (r2 < s.h2);
        if (hit) nb_push(p, s.i, jg);
    }
    if (CHK || G4) {
        // left out: m = 0 at r = 1 (GRAPE-4: r^2 = 0)
        const bool out = G4 ? (hi | (unsigned)__double2loint(r2)) == 0u : self;
        m = out ? 0.0 : m;
        r2 = out ? 1.0 : r2;
        hi = out ? 0xffffffffu : hi;
    }
    if constexpr (PO) {
        const double x = __fma_rn(r2, kThird, s.eps2 * kThird);
        const double y = inv_dist_s3<1>(x, x);
        s.Pt = __fma_rn(-m, y, s.Pt);
        return hi;
    }
    if (!G4) r2 += s.eps2;
    const double y = inv_dist_s3<3>(r2 * kThird, r2);
    const double dvx = J.vel.x - s.vx, dvy = J.vel.y - s.vy, dvz = J.vel.z - s.vz;
    const double rv = __fma_rn(dz, dvz, __fma_rn(dy, dvy, dx * dvx));
    const double q3 = y * y;  // 3 / r^2
    const double mr = m * y;
    const double mr3 = mr * q3;
    const double a3 = rv * q3;
    s.Pt -= mr;
    s.Ax = __fma_rn(mr3, dx, s.Ax);
    s.Ay = __fma_rn(mr3, dy, s.Ay);
    s.Az = __fma_rn(mr3, dz, s.Az);
    s.Jx = __fma_rn(mr3, __fma_rn(-a3, dx, dvx), s.Jx);
    s.Jy = __fma_rn(mr3, __fma_rn(-a3, dy, dvy), s.Jy);
    s.Jz = __fma_rn(mr3, __fma_rn(-a3, dz, dvz), s.Jz);
    return hi;
}

// Nearest neighbour of the FP64 kernels: of a run of RUN j from j0 in steps
// of JL (addresses), the one with the smallest unsoftened r^2, the first on
// a tie.  Up to eight records are loaded before the first is used.
template <int JL, bool IDENT>
__device__ __forceinline__ void nn_scan_one(StateF64 &s, const double4 &pos, double w, int jg) {
    const double r2 = r2_f64(pos.x - s.x, pos.y - s.y, pos.z - s.z);
    const bool self = IDENT ? jg == s.idx : w == (double)s.idx;
    if (!self && r2 < s.nr2) {
        s.nr2 = r2;
        s.nj = jg;
    }
}

template <int JL, int RUN, bool IDENT>
__device__ __forceinline__ void nn_scan_run(StateF64 &s, const JRecF64 *src, int j0) {
    constexpr int B = RUN < 8 ? RUN : 8;
#pragma unroll 1
    for (int b = 0; b < RUN; b += B) {
        double4 pos[B];
        double w[B];
#pragma unroll
        for (int u = 0; u < B; ++u) {
            pos[u] = src[j0 + (b + u) * JL].pos;
            w[u] = IDENT ? 0.0 : src[j0 + (b + u) * JL].vel.w;
        }
#pragma unroll
        for (int u = 0; u < B; ++u) nn_scan_one<JL, IDENT>(s, pos[u], w[u], j0 + (b + u) * JL);
    }
}

// ---- paired layout: one FP32x2 instruction evaluates i against two j.
// i-side values are held negated and duplicated in both halves, so every
// difference is an FP32x2 add of a j-pair and a loop-invariant register pair.
struct StateMixedP {
    float2 nxh, nyh, nzh, nxl, nyl, nzl, nvx, nvy, nvz;
    float h2;
    float2 ax, ay, az, jx, jy, jz, pm;  // FP32 sums since the last fold; pm = sum m/(4r)
    unsigned qa;                        // error indicators (kVarStats): bits of max m/(2r^2) (unsigned max)
    int qj;                             // and of max m/r^3 (signed max: the self term's -0.0 never wins)
    double Ax, Ay, Az, Jx, Jy, Jz, Pt;
    float nr2;
    int nk;  // first pair record of the run of records that first reached nr2 (-1: none)
    int nj, idx, i;
};
template <> struct StateOf<kKernMixedP> { using type = StateMixedP; };

__device__ __forceinline__ float2 dup(float v) { return make_float2(v, v); }

__device__ __forceinline__ void load_i(StateMixedP &s, const IRec &q, const ForceParams &p, bool &range_ok) {
    float h, l;
    range_ok &= to_fixed_split(q.x[0], p.fs, h, l);
    s.nxh = dup(-h);
    s.nxl = dup(-l);
    range_ok &= to_fixed_split(q.x[1], p.fs, h, l);
    s.nyh = dup(-h);
    s.nyl = dup(-l);
    range_ok &= to_fixed_split(q.x[2], p.fs, h, l);
    s.nzh = dup(-h);
    s.nzl = dup(-l);
    s.nvx = dup(-(float)q.v[0]);
    s.nvy = dup(-(float)q.v[1]);
    s.nvz = dup(-(float)q.v[2]);
    s.h2 = (float)q.h2;
    s.idx = q.index;
    s.ax = s.ay = s.az = s.jx = s.jy = s.jz = s.pm = make_float2(0.f, 0.f);
    s.qa = 0u;
    s.qj = 0;
    s.Ax = s.Ay = s.Az = s.Jx = s.Jy = s.Jz = s.Pt = 0.0;
    s.nr2 = FLT_MAX;
    s.nk = -1;
    s.nj = -1;
}

// Unsoftened squared distances of i to the two j of a record (the pair
// terms' own operations in their order), FLT_MAX for the particle itself.
template <bool IDENT>
__device__ __forceinline__ float2 pair_nn_r2(const StateMixedP &s, const JPairMixed &rec, int jg0) {
    const float4 hxy = rec.hxy, hzm = rec.hzm, lxy = rec.lxy, lzi = rec.lzi;
    const float2 dx = __fadd2_rn(__fadd2_rn(make_float2(hxy.x, hxy.y), s.nxh),
                                 __fadd2_rn(make_float2(lxy.x, lxy.y), s.nxl));
    const float2 dy = __fadd2_rn(__fadd2_rn(make_float2(hxy.z, hxy.w), s.nyh),
                                 __fadd2_rn(make_float2(lxy.z, lxy.w), s.nyl));
    const float2 dz = __fadd2_rn(__fadd2_rn(make_float2(hzm.x, hzm.y), s.nzh),
                                 __fadd2_rn(make_float2(lzi.x, lzi.y), s.nzl));
    float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
    if (IDENT ? (jg0 == s.idx) : (__float_as_int(lzi.z) == s.idx)) r2.x = FLT_MAX;
    if (IDENT ? (jg0 + 1 == s.idx) : (__float_as_int(lzi.w) == s.idx)) r2.y = FLT_MAX;
    return r2;
}

template <bool CHK, bool NB, bool IDENT, bool PO = false, bool STATS = false>
__device__ __forceinline__ void interact_pair(StateMixedP &s, const JPairMixed &J, int jg0, float2 eps2,
                                              const ForceParams &p) {
    if constexpr (PO) {
        // Potential only: the exact position difference, r^2, the refined
        // inverse distance and m/r -- the pot terms of the full form below,
        // rounded identically.
        const float2 dx = __fadd2_rn(__fadd2_rn(make_float2(J.hxy.x, J.hxy.y), s.nxh),
                                     __fadd2_rn(make_float2(J.lxy.x, J.lxy.y), s.nxl));
        const float2 dy = __fadd2_rn(__fadd2_rn(make_float2(J.hxy.z, J.hxy.w), s.nyh),
                                     __fadd2_rn(make_float2(J.lxy.z, J.lxy.w), s.nyl));
        const float2 dz = __fadd2_rn(__fadd2_rn(make_float2(J.hzm.x, J.hzm.y), s.nzh),
                                     __fadd2_rn(make_float2(J.lzi.x, J.lzi.y), s.nzl));
        float2 r2 = __fadd2_rn(__ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx))), eps2);
        float2 m = make_float2(J.hzm.z, J.hzm.w);
        if (CHK) {
            const bool self0 = IDENT ? (jg0 == s.idx) : (__float_as_int(J.lzi.z) == s.idx);
            const bool self1 = IDENT ? (jg0 + 1 == s.idx) : (__float_as_int(J.lzi.w) == s.idx);
            r2.x = self0 ? 1.f : r2.x;
            r2.y = self1 ? 1.f : r2.y;
            m.x = self0 ? 0.f : m.x;
            m.y = self1 ? 0.f : m.y;
        }
        float2 y = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
        const float2 ry = __fmul2_rn(r2, y);
        y = __fmul2_rn(y, __ffma2_rn(ry, y, dup(-3.f)));
        s.pm = __fadd2_rn(s.pm, __fmul2_rn(m, y));
        return;
    }
    const float2 dx = __fadd2_rn(__fadd2_rn(make_float2(J.hxy.x, J.hxy.y), s.nxh),
                                 __fadd2_rn(make_float2(J.lxy.x, J.lxy.y), s.nxl));
    const float2 dy = __fadd2_rn(__fadd2_rn(make_float2(J.hxy.z, J.hxy.w), s.nyh),
                                 __fadd2_rn(make_float2(J.lxy.z, J.lxy.w), s.nyl));
    const float2 dz = __fadd2_rn(__fadd2_rn(make_float2(J.hzm.x, J.hzm.y), s.nzh),
                                 __fadd2_rn(make_float2(J.lzi.x, J.lzi.y), s.nzl));
    const float2 dvx = __fadd2_rn(make_float2(J.vxy.x, J.vxy.y), s.nvx);
    const float2 dvy = __fadd2_rn(make_float2(J.vxy.z, J.vxy.w), s.nvy);
    const float2 dvz = __fadd2_rn(make_float2(J.vz.x, J.vz.y), s.nvz);
    const float2 r2n = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
    const float2 rv = __ffma2_rn(dz, dvz, __ffma2_rn(dy, dvy, __fmul2_rn(dx, dvx)));
    float2 r2 = __fadd2_rn(r2n, eps2);
    float2 m = make_float2(J.hzm.z, J.hzm.w);
    float2 r2nn = r2n;
    bool self0 = false, self1 = false;
    if (CHK) {
        self0 = IDENT ? (jg0 == s.idx) : (__float_as_int(J.lzi.z) == s.idx);
        self1 = IDENT ? (jg0 + 1 == s.idx) : (__float_as_int(J.lzi.w) == s.idx);
        r2.x = self0 ? 1.f : r2.x;
        r2.y = self1 ? 1.f : r2.y;
        m.x = self0 ? 0.f : m.x;
        m.y = self1 ? 0.f : m.y;
        r2nn.x = self0 ? FLT_MAX : r2nn.x;
        r2nn.y = self1 ? FLT_MAX : r2nn.y;
    }
    float2 y = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
    // One Newton-Raphson step, kept at -2 times its value:
    // y' = y (r2 y^2 - 3) = -2 y (1.5 - 0.5 r2 y^2), one instruction fewer
    // than the textbook form.  Every product below is the scalar kernel's
    // scaled by a power of two (exact), and the record's mass is -m/8, so
    // mr3 = (-m/8)(-2y)(4 y^2) and a3 = (-0.75 rv)(4 y^2) come out
    // bit-identical to the textbook form; pm sums m/(4r).
    const float2 ry = __fmul2_rn(r2, y);
    y = __fmul2_rn(y, __ffma2_rn(ry, y, dup(-3.f)));
    const float2 r2inv = __fmul2_rn(y, y);
    const float2 mr = __fmul2_rn(m, y);
    const float2 mr3 = __fmul2_rn(mr, r2inv);
    const float2 a3 = __fmul2_rn(__fmul2_rn(rv, dup(-0.75f)), r2inv);
    if (STATS) {
        // The refinement's error indicators, the largest single terms:
        // mr y = -m/(2 r^2) (y is -2/r, see above) and mr3 = m/r^3.  The
        // maxima are integer maxima of the bit patterns, off the FMA pipe:
        // non-positive floats order like their bits read as unsigned (t),
        // non-negative ones like their bits read as signed (mr3).  The self
        // term (m = +0, y < 0) gives mr3 = -0.0, whose bits 0x80000000 would
        // win an unsigned maximum over every positive float; as a signed
        // int it is the smallest value.
        // Both halves of the pair go into one register per indicator with a
        // three-input maximum.
        const float2 t = __fmul2_rn(mr, y);
        s.qa = __vimax3_u32(s.qa, __float_as_uint(t.x), __float_as_uint(t.y));
        s.qj = __vimax3_s32(s.qj, __float_as_int(mr3.x), __float_as_int(mr3.y));
    }
    s.pm = __fadd2_rn(s.pm, mr);
    s.ax = __ffma2_rn(mr3, dx, s.ax);
    s.ay = __ffma2_rn(mr3, dy, s.ay);
    s.az = __ffma2_rn(mr3, dz, s.az);
    s.jx = __ffma2_rn(mr3, __ffma2_rn(a3, dx, dvx), s.jx);
    s.jy = __ffma2_rn(mr3, __ffma2_rn(a3, dy, dvy), s.jy);
    s.jz = __ffma2_rn(mr3, __ffma2_rn(a3, dz, dvz), s.jz);
    if (STATS) {
        s.nr2 = fminf(fminf(s.nr2, r2nn.x), r2nn.y);  // which j it was: nn_of_run
    } else {
        if (r2nn.x < s.nr2) {
            s.nr2 = r2nn.x;
            s.nj = jg0;
        }
        if (r2nn.y < s.nr2) {
            s.nr2 = r2nn.y;
            s.nj = jg0 + 1;
        }
    }
    if (NB) {
        const bool hit0 = CHK && self0 ? (p.include_self && s.h2 > 0.f) : (r2n.x < s.h2);
        const bool hit1 = CHK && self1 ? (p.include_self && s.h2 > 0.f) : (r2n.y < s.h2);
        if (hit0) nb_push(p, s.i, jg0);
        if (hit1) nb_push(p, s.i, jg0 + 1);
    }
}

__device__ __forceinline__ void fold(StateMixedP &s) {
    s.Ax += (double)s.ax.x; s.Ax += (double)s.ax.y;
    s.Ay += (double)s.ay.x; s.Ay += (double)s.ay.y;
    s.Az += (double)s.az.x; s.Az += (double)s.az.y;
    s.Jx += (double)s.jx.x; s.Jx += (double)s.jx.y;
    s.Jy += (double)s.jy.x; s.Jy += (double)s.jy.y;
    s.Jz += (double)s.jz.x; s.Jz += (double)s.jz.y;
    s.Pt -= 4.0 * (double)s.pm.x; s.Pt -= 4.0 * (double)s.pm.y;  // pm sums m/(4r)
    s.ax = s.ay = s.az = s.jx = s.jy = s.jz = s.pm = make_float2(0.f, 0.f);
}

__device__ __forceinline__ void fold_pot(StateMixedP &s) {
    s.Pt -= 4.0 * (double)s.pm.x; s.Pt -= 4.0 * (double)s.pm.y;  // pm sums m/(4r)
    s.pm = make_float2(0.f, 0.f);
}

template <bool PO>
__device__ __forceinline__ void fold_any(StateMixedP &s) {
    if constexpr (PO)
        fold_pot(s);
    else
        fold(s);
}

__device__ __forceinline__ void fold(StateMixedBase &s) {
    s.Ax += (double)s.ax;
    s.Ay += (double)s.ay;
    s.Az += (double)s.az;
    s.Jx += (double)s.jx;
    s.Jy += (double)s.jy;
    s.Jz += (double)s.jz;
    s.Pt += (double)s.pt;
    s.ax = s.ay = s.az = s.jx = s.jy = s.jz = s.pt = 0.f;
}

// The nearest neighbour in two steps (single-call paired kernel, FP64
// kernels): the pair loop keeps a minimum alone, and after every run of
// NnRun records it is compared with its value before the run, so the run
// that first reached the minimum is known.  At the end of the task that
// run's records are looked through again (nn_of_run, nn_scan_run): the same
// j as a compare and select in every pair term.  The FP64 minimum is of the
// upper words alone, so runs that tie with it are listed and looked through
// too; past kTies of them (a particle so far out that all its r^2 agree in
// 20 bits) the thread's whole share is.  With two runs listed a lattice, where
// most particles have more, took 13.26 ms for 64000 x 64000 and 0.49 ms for
// 2000 x 64000; with eight 9.78 and 0.378 (distances without ties 9.74 and
// 0.371).  The far particles: 2000 of them 0.51 ms, 64000 x 64000 with 4096
// 10.6 ms.  Looking a tied run through at once instead cost 2000 x 64000 1.7 %
// without any ties.  A run divides a thread's
// share of a tile (a multiple of 16 records at 32 i-lanes, 4 at 8 i-lanes,
// any number at 1).
constexpr int kTies = 8;
template <int K, int JL, int R, int V> struct NnRun {
    static constexpr int value =
        JL == 1 ? (K == kKernF64 && (R == 2 || (V & (kVarG4 | kVarPot)) != 0) ? 16 : 8) : (JL == 4 ? 4 : 1);
};

template <int JL, int RUN, bool IDENT>
__device__ __forceinline__ void nn_of_run(StateMixedP &s, const JPairMixed *jrec) {
#pragma unroll 1
    for (int u = 0; u < RUN; ++u) {
        const int k = s.nk + u * JL;
        const float2 r2 = pair_nn_r2<IDENT>(s, jrec[k], 2 * k);
        if (r2.x == s.nr2 || r2.y == s.nr2) {
            s.nj = 2 * k + (r2.x == s.nr2 ? 0 : 1);
            return;
        }
    }
}

// Consume one shared-memory tile: this thread's j are kbase + m*JL.
template <int K, int R, int JL, bool CHK, bool NB, bool IDENT, int V>
__device__ __forceinline__ void consume_tile(typename StateOf<K>::type (&st)[R],
                                             const typename Traits<K>::JRec *S, int kbase,
                                             int per, int tb, const ForceParams &p, int (&ties)[R][kTies]) {
    if constexpr (K == kKernMixedP) {
        constexpr bool PO = (V & kVarPot) != 0;
        constexpr bool ST = (V & kVarStats) != 0;
        const float2 eps2 = dup((float)p.eps2);
        constexpr int kFlushPairs = kFlush / 2;
        if constexpr (ST) {
            constexpr int RUN = NnRun<K, JL, R, V>::value;
            // Unrolled by two runs, 16 records: 65536 x 262144 in 23.07 ms
            // (one run 23.38, a compare and select per term 23.78).
#pragma unroll 2
            for (int m0 = 0; m0 < per; m0 += RUN) {
                float before[R];
#pragma unroll
                for (int r = 0; r < R; ++r) before[r] = st[r].nr2;
#pragma unroll
                for (int u = 0; u < RUN; ++u) {
                    const int k = kbase + (m0 + u) * JL;
                    const JPairMixed J = S[k];
#pragma unroll
                    for (int r = 0; r < R; ++r) interact_pair<CHK, NB, IDENT, PO, ST>(st[r], J, tb + 2 * k, eps2, p);
                    if (kFlushPairs < RUN && (u + 1) % kFlushPairs == 0) {
#pragma unroll
                        for (int r = 0; r < R; ++r) fold(st[r]);
                    }
                }
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (st[r].nr2 < before[r]) st[r].nk = tb / 2 + kbase + m0 * JL;
                if (kFlushPairs >= RUN && ((m0 + RUN) % kFlushPairs == 0 || m0 + RUN >= per)) {
#pragma unroll
                    for (int r = 0; r < R; ++r) fold(st[r]);
                }
            }
            return;
        }
        // The batched and resident kernels, which hold three lane shapes in
        // one body, unroll by 4 (at 16 they spill).
        for (int m0 = 0; m0 < per; m0 += kFlushPairs) {
            const int m1 = min(m0 + kFlushPairs, per);
#pragma unroll (PO ? 8 : 4)
            for (int m = m0; m < m1; ++m) {
                const int k = kbase + m * JL;
                const JPairMixed J = S[k];
#pragma unroll
                for (int r = 0; r < R; ++r) interact_pair<CHK, NB, IDENT, PO, ST>(st[r], J, tb + 2 * k, eps2, p);
            }
#pragma unroll
            for (int r = 0; r < R; ++r) fold_any<PO>(st[r]);
        }
    } else if constexpr (K == kKernF64) {
        constexpr bool G4 = (V & kVarG4) != 0, PO = (V & kVarPot) != 0;
        constexpr int RUN = NnRun<K, JL, R, V>::value;
        for (int m0 = 0; m0 < per; m0 += RUN) {
            unsigned lo[R];
#pragma unroll
            for (int r = 0; r < R; ++r) lo[r] = 0xffffffffu;
#pragma unroll
            for (int u = 0; u < RUN; ++u) {
                const int k = kbase + (m0 + u) * JL;
                const JRecF64 J = S[k];
#pragma unroll
                for (int r = 0; r < R; ++r)
                    lo[r] = min(lo[r], interact<CHK, NB, IDENT, G4, PO>(st[r], J, tb + k, p));
            }
            // the GRAPE-4 pipeline returns no neighbour index
            if constexpr (!G4 && !PO) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int run = tb + kbase + m0 * JL;
                    // one branch, rarely taken: 2000 x 64000 0.371 ms, with selects
                    // for the smaller word and a branch for the tie 0.378
                    if (__builtin_expect(lo[r] <= st[r].nhi, 0)) {
                        if (lo[r] < st[r].nhi) {
                            st[r].nhi = lo[r];
                            st[r].nk = run;
                            st[r].nties = 0;
                        } else {
                            if (st[r].nties < kTies) ties[r][st[r].nties] = run;
                            if (st[r].nties <= kTies) ++st[r].nties;
                        }
                    }
                }
            }
        }
    } else {
        const float eps2 = (float)p.eps2;
        for (int m0 = 0; m0 < per; m0 += kFlush) {
            const int m1 = min(m0 + kFlush, per);
            if (V & kVarUnroll4) {
#pragma unroll 4
                for (int m = m0; m < m1; ++m) {
                    const int k = kbase + m * JL;
                    const auto J = S[k];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        JMixed d;
                        diff(st[r], J, d);
                        interact_mixed<CHK, NB, IDENT>(st[r], d, tb + k, eps2, p);
                    }
                }
            } else {
#pragma unroll 2
                for (int m = m0; m < m1; ++m) {
                    const int k = kbase + m * JL;
                    const auto J = S[k];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        JMixed d;
                        diff(st[r], J, d);
                        interact_mixed<CHK, NB, IDENT>(st[r], d, tb + k, eps2, p);
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < R; ++r) fold(st[r]);
        }
    }
}

__device__ __forceinline__ void take_min(double &r2, int &j, double o_r2, int o_j) {
    if (o_r2 < r2 || (o_r2 == r2 && (unsigned)o_j < (unsigned)j)) {
        r2 = o_r2;
        j = o_j;
    }
}

template <bool PO>
__device__ __forceinline__ void to_partial(const StateMixedBase &s, Partial &q, bool) {
    q.acc[0] = s.Ax; q.acc[1] = s.Ay; q.acc[2] = s.Az;
    q.jerk[0] = s.Jx; q.jerk[1] = s.Jy; q.jerk[2] = s.Jz;
    q.pot = s.Pt;
    q.nn_r2 = (double)s.nr2;
    q.nn_j = s.nj;
    q.qa = q.qj = 0.f;
}
template <bool PO>
__device__ __forceinline__ void to_partial(const StateMixedP &s, Partial &q, bool) {
    q.acc[0] = s.Ax; q.acc[1] = s.Ay; q.acc[2] = s.Az;
    q.jerk[0] = s.Jx; q.jerk[1] = s.Jy; q.jerk[2] = s.Jz;
    q.pot = s.Pt;
    q.nn_r2 = (double)s.nr2;
    q.nn_j = s.nj;
    q.qa = -2.f * __uint_as_float(s.qa);  // max m / r^2
    q.qj = __int_as_float(s.qj);          // max m / r^3
}
template <bool PO>
__device__ __forceinline__ void to_partial(const StateF64 &s, Partial &q, bool unscaled) {
    // 1/sqrt(3) and its cube (potential only: sqrt(kThird) as that is
    // rounded), in two doubles each: rounded to one they shift every sum the
    // same way, by as much as all its terms' roundings together.
    const auto scaled = [unscaled](double v, double hi, double lo) { return unscaled ? v : fma(v, hi, v * lo); };
    constexpr double h1 = 0.5773502691896257, l1 = PO ? 1.7425591686159977e-17 : 3.3450280739356345e-17;
    constexpr double h3 = 0.19245008972987526, l3 = -7.353623497300496e-18;
    for (int c = 0; c < 3; ++c) {
        q.acc[c] = scaled(c == 0 ? s.Ax : c == 1 ? s.Ay : s.Az, h3, l3);
        q.jerk[c] = scaled(c == 0 ? s.Jx : c == 1 ? s.Jy : s.Jz, h3, l3);
    }
    q.pot = scaled(s.Pt, h1, l1);
    q.nn_r2 = s.nr2;
    q.nn_j = s.nj;
    q.qa = q.qj = 0.f;
}

__device__ __forceinline__ void add_partial(Partial &a, const Partial &b) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
        a.acc[c] += b.acc[c];
        a.jerk[c] += b.jerk[c];
    }
    a.pot += b.pot;
    take_min(a.nn_r2, a.nn_j, b.nn_r2, b.nn_j);
    a.qa = fmaxf(a.qa, b.qa);
    a.qj = fmaxf(a.qj, b.qj);
}

// Sum over the lanes of a warp that share an i (lane bits >= log2(IL)).
template <int IL>
__device__ __forceinline__ void warp_reduce(Partial &q) {
#pragma unroll
    for (int off = IL; off < 32; off <<= 1) {
        Partial o;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            o.acc[c] = __shfl_xor_sync(0xffffffffu, q.acc[c], off);
            o.jerk[c] = __shfl_xor_sync(0xffffffffu, q.jerk[c], off);
        }
        o.pot = __shfl_xor_sync(0xffffffffu, q.pot, off);
        o.nn_r2 = __shfl_xor_sync(0xffffffffu, q.nn_r2, off);
        o.nn_j = __shfl_xor_sync(0xffffffffu, q.nn_j, off);
        o.qa = __shfl_xor_sync(0xffffffffu, q.qa, off);
        o.qj = __shfl_xor_sync(0xffffffffu, q.qj, off);
        add_partial(q, o);
    }
}

// Partial written by another CTA of the same launch: read around L1, in
// five 16-byte loads.
__device__ __forceinline__ Partial load_partial_cg(const Partial *src) {
    static_assert(sizeof(Partial) == 80, "five 16-byte words");
    const double2 *s = reinterpret_cast<const double2 *>(src);
    const double2 w0 = __ldcg(s), w1 = __ldcg(s + 1), w2 = __ldcg(s + 2), w3 = __ldcg(s + 3);
    const int4 w4 = __ldcg(reinterpret_cast<const int4 *>(src) + 4);
    Partial a;
    a.acc[0] = w0.x; a.acc[1] = w0.y; a.acc[2] = w1.x;
    a.jerk[0] = w1.y; a.jerk[1] = w2.x; a.jerk[2] = w2.y;
    a.pot = w3.x;
    a.nn_r2 = w3.y;
    a.nn_j = w4.x;
    a.qa = __int_as_float(w4.y);
    a.qj = __int_as_float(w4.z);
    return a;
}

__device__ __forceinline__ void store_partial(Partial *dst, const Partial &a) {
    double2 *d = reinterpret_cast<double2 *>(dst);
    d[0] = make_double2(a.acc[0], a.acc[1]);
    d[1] = make_double2(a.acc[2], a.jerk[0]);
    d[2] = make_double2(a.jerk[1], a.jerk[2]);
    d[3] = make_double2(a.pot, a.nn_r2);
    reinterpret_cast<int4 *>(dst)[4] = make_int4(a.nn_j, __float_as_int(a.qa), __float_as_int(a.qj), 0);
}

// One more arrival at an i-tile's counter: everything the CTA wrote before
// (the caller has synchronised it) is visible to whoever sees the count.
__device__ __forceinline__ int arrive_count(int *counter) {
    int old;
    asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;" : "=r"(old) : "l"(counter) : "memory");
    return old;
}

// MAPPED: honour p.out_map (only the FP64 layout's kernels, which run the
// refinement's pass, and the generic reduction kernels compile it in: in
// the paired mixed batch kernel it cost 100 bytes of spills).
template <bool MAPPED = true>
__device__ __forceinline__ void write_final(const ForceParams &p, int i, const Partial &q) {
    const size_t o = MAPPED && p.out_map ? (size_t)p.out_map[i] : (size_t)i;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        p.out_acc[3 * o + c] = q.acc[c];
        p.out_jerk[3 * o + c] = q.jerk[c];
    }
    p.out_pot[o] = q.pot;
    p.out_nn[o] = (q.nn_j < 0 || q.nn_j >= p.nj) ? 0 : q.nn_j;
    if (p.out_q) {
        p.out_q[2 * o] = q.qa;
        p.out_q[2 * o + 1] = q.qj;
    }
}

// The last CTA of an i-tile adds the splits' partial sums of its i
// (ib + 0 .. itile - 1).  The fold is a chain of loads from L2, so it is cut
// into as many segments of splits as the CTA has threads per i (at most
// `slots` partials in shared memory): each thread adds its segment's splits
// in order with four loads in flight, then the segments are added pairwise.
// 64 x 40192 in 63 splits: 26.7 us with one thread per i over all splits (and
// a __threadfence in every thread before the count), 20.5 now; 1 x 65536 in
// 64 splits 16.4 -> 12.3; 4096 x 65536 in 37, one segment, 0.636 -> 0.622 ms
// (the 16-byte loads and the single release).
// In the batched and FP64 kernels a function of its own, with the fields it
// needs passed by value: in line in each lane shape's task it made the
// batched kernels spill.  In line in the single-call paired kernel, whose
// pair loop a call costs 0.6 %.
struct FoldArgs {
    const Partial *part;
    int ni, nj, nsplit;
    double *out_acc, *out_jerk, *out_pot;
    int *out_nn;
    float *out_q;
    const int *out_map;
};
__device__ __forceinline__ void fold_splits_inline(FoldArgs f, int ib, int itile, int slots, Partial *red) {
    ForceParams p{};  // what write_final reads
    p.nj = f.nj;
    p.out_acc = f.out_acc;
    p.out_jerk = f.out_jerk;
    p.out_pot = f.out_pot;
    p.out_nn = f.out_nn;
    p.out_q = f.out_q;
    p.out_map = f.out_map;
    int it2 = 1;  // threads per segment: itile rounded up to a power of two
    while (it2 < itile) it2 <<= 1;
    int segs = 1;
    while (2 * segs * it2 <= slots && 8 * segs < f.nsplit) segs <<= 1;  // more than four splits each
    const int step = segs > 1 ? it2 : (int)blockDim.x;  // one segment: any itile, in rounds of the CTA
    const int g = segs > 1 ? (int)threadIdx.x / it2 : 0;
    const int s0 = (int)((long long)f.nsplit * g / segs), s1 = (int)((long long)f.nsplit * (g + 1) / segs);
    for (int k = segs > 1 ? (int)threadIdx.x & (it2 - 1) : (int)threadIdx.x; k < itile; k += step) {
        const int i = ib + k;
        if (i >= f.ni || g >= segs) break;
        const Partial *src = f.part + i;
        Partial a = load_partial_cg(src + (size_t)s0 * f.ni);
        int sp = s0 + 1;
        for (; sp + 4 <= s1; sp += 4) {
            Partial b[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) b[u] = load_partial_cg(src + (size_t)(sp + u) * f.ni);
#pragma unroll
            for (int u = 0; u < 4; ++u) add_partial(a, b[u]);
        }
        for (; sp < s1; ++sp) add_partial(a, load_partial_cg(src + (size_t)sp * f.ni));
        if (segs > 1)
            red[g * it2 + k] = a;
        else
            write_final<true>(p, i, a);
    }
    if (segs == 1) return;
    const int k = (int)threadIdx.x & (it2 - 1), i = ib + k;
    const bool mine = k < itile && i < f.ni;
    for (int w = segs >> 1; w > 0; w >>= 1) {
        __syncthreads();
        if (mine && g < w) add_partial(red[g * it2 + k], red[(g + w) * it2 + k]);
    }
    if (mine && g == 0) write_final<true>(p, i, red[k]);
}

static __device__ __noinline__ void fold_splits(FoldArgs f, int ib, int itile, int slots, Partial *red) {
    fold_splits_inline(f, ib, itile, slots, red);
}

// Resident CTAs per SM the register budget is sized for (3 for the paired
// kernel measured 1.7% slower: 80 registers with spills).
template <int K, int R> struct MinBlocks {
    static constexpr int value = R >= 4 ? 1 : 2;
};

// Where a task's j come from: predicted records in device memory, copied
// tile by tile,
struct JRecords {
    static constexpr bool kInPlace = false;
};
// or a small FP64 call's raw j-state and updates, predicted by the CTA that
// needs them: its whole j-range, into shared memory in one pass (so the
// loads' latency is paid once) and, by the first i-tile's CTAs, into the
// record array too, which then holds the prediction for later calls.
struct JFromCall {
    static constexpr bool kInPlace = true;
    const SmallCall *sc;
    double *jraw;
    int *jindex;
    int *s_addr;  // [kSmallMax] in shared memory
};

__device__ __forceinline__ void predict_range(const JFromCall &src, const ForceParams &p, int jb, int n, bool store,
                                              bool last, JRecF64 *tiles) {
    const SmallCall &sc = *src.sc;
    JRecF64 *out = static_cast<JRecF64 *>(const_cast<void *>(p.jrec));
    constexpr int B = 2;  // records per thread whose loads are issued together
    for (int r0 = threadIdx.x; r0 < n; r0 += B * blockDim.x) {
        double raw[B][JF_K18];
        int id[B];
#pragma unroll
        for (int u = 0; u < B; ++u) {
            const int j = jb + r0 + u * (int)blockDim.x;
            if (r0 + u * (int)blockDim.x < n && j < sc.nj) {
#pragma unroll
                for (int f = 0; f < JF_K18; ++f) raw[u][f] = src.jraw[(size_t)f * sc.cap + j];
                id[u] = src.jindex[j];
            }
        }
#pragma unroll
        for (int u = 0; u < B; ++u) {
            const int r = r0 + u * (int)blockDim.x, j = jb + r;
            if (r >= n) break;
            JRecF64 rec;
            if (j < sc.nj) {
                // an updated particle's raw state is being rewritten: its
                // values are the update's
                const int k = find_update(src.s_addr, sc.n_upd, j);
                double xp[3], vp[3], m;
                if (k >= 0) {
                    predict_vals(sc.vals[k], sc.ti, xp, vp, m);
                    id[u] = sc.index[k];
                } else {
                    predict_vals(raw[u], sc.ti, xp, vp, m);
                }
                rec.pos = make_double4(xp[0], xp[1], xp[2], m);
                rec.vel = make_double4(vp[0], vp[1], vp[2], (double)id[u]);
            } else {
                rec.pos = make_double4(kDummyPos, kDummyPos, kDummyPos, 0.0);
                rec.vel = make_double4(0.0, 0.0, 0.0, -1.0);
            }
            tiles[r] = rec;
            if (store) out[j] = rec;
        }
    }
    // the record array's padding may be wider than this kernel's tiles
    if (store && last) {
        JRecF64 rec;
        rec.pos = make_double4(kDummyPos, kDummyPos, kDummyPos, 0.0);
        rec.vel = make_double4(0.0, 0.0, 0.0, -1.0);
        for (int j = p.nj_pad + threadIdx.x; j < sc.nj_pad; j += blockDim.x) out[j] = rec;
    }
}

// One task: the i-tile `itile_idx` of item p against its j-split `split`.
// Shared memory holds the two mbarriers (initialised by the caller) and the
// tile ring; `gt` counts the tiles this CTA consumed before (it sets the
// ring stage and the mbarrier phase, so a persistent CTA can run many
// tasks back to back).
template <int K, int IL, int R, bool NB, bool IDENT, int V, class Src = JRecords>
__device__ __forceinline__ bool process_task(const ForceParams &p, int itile_idx, int split, unsigned char *smem,
                                             int &gt, const Src &src = Src{}) {
    using Tr = Traits<K>;
    using JRec = typename Tr::JRec;
    using State = typename StateOf<K>::type;
    constexpr int T = Tr::T;     // j per tile
    constexpr int U = Tr::U;     // records per tile
    constexpr int JPU = Tr::JPU; // j per record
    constexpr int JL = 32 / IL;
    constexpr unsigned kTileBytes = U * sizeof(JRec);

    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);          // [2], never reused
    JRec *tiles = reinterpret_cast<JRec *>(smem + 128);           // [2][U]
    Partial *red = reinterpret_cast<Partial *>(smem + 128);       // epilogue reuse

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int NW = blockDim.x >> 5;
    const int H = p.H;
    const int G = NW / H;
    const int g = warp % G, h = warp / G;
    const int il = lane % IL, jl = lane / IL;
    const int itile = G * IL * R;
    const int islot = g * IL * R + il;  // slot of r = 0 inside the i-tile
    const int i0 = itile_idx * itile + islot;

    State st[R];
    int ties[R][kTies];  // FP64: runs whose smallest upper word ties with the least (NnRun)
    bool range_ok = true;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = i0 + r * IL;
        const bool valid = i < p.ni;
        load_i(st[r], p.irec[valid ? i : p.ni - 1], p, range_ok);
        if constexpr (K == kKernF64 && (V & kVarG4) != 0) st[r].eps2 = p.ieps2[valid ? i : p.ni - 1];
        st[r].i = i;
        if (!valid) st[r].h2 = 0;
    }
    if (!range_ok) atomicOr(p.status, ST_RANGE);

    const int jb = split * p.jper;
    const int je = min(jb + p.jper, p.nj_pad);
    const int ntiles = max(0, (je - jb) / T);
    const JRec *jrec = reinterpret_cast<const JRec *>(p.jrec);
    const int g0 = gt;

    const int per = U / (H * JL);
    const int kbase = h * (U / H) + jl;
    auto consume = [&](const JRec *S, int tb) {
        bool chk = true;
        if (IDENT) {
            bool mine = false;
#pragma unroll
            for (int r = 0; r < R; ++r) mine |= (unsigned)(st[r].idx - tb) < (unsigned)T;
            chk = __any_sync(0xffffffffu, mine);
        }
        if (chk)
            consume_tile<K, R, JL, true, NB, IDENT, V>(st, S, kbase, per, tb, p, ties);
        else
            consume_tile<K, R, JL, false, NB, IDENT, V>(st, S, kbase, per, tb, p, ties);
    };
    bool ok = true;
    int t = 0;
    if constexpr (Src::kInPlace) {
        predict_range(src, p, jb, ntiles * T, itile_idx == 0, je == p.nj_pad, tiles);
        __syncthreads();
        for (; t < ntiles; ++t) consume(tiles + t * U, jb + t * T);
    } else {
        // The previous task's epilogue may still read the tile area, and has
        // written its reductions there: ordinary stores, ordered before the
        // copies by the proxy fence.
        __syncthreads();
        if (threadIdx.x == 0 && ntiles > 0) {
            if (g0 != 0) fence_proxy_async();
            const int b = g0 & 1;
            mbar_arrive_expect_tx(&bars[b], kTileBytes);
            bulk_g2s(tiles + b * U, jrec + jb / JPU, kTileBytes, &bars[b]);
        }

        for (; t < ntiles; ++t) {
            const int gg = g0 + t;
            const int b = gg & 1;
            if (threadIdx.x == 0 && t + 1 < ntiles) {
                mbar_arrive_expect_tx(&bars[b ^ 1], kTileBytes);
                bulk_g2s(tiles + (b ^ 1) * U, jrec + (jb + (t + 1) * T) / JPU, kTileBytes, &bars[b ^ 1]);
            }
            const bool arrived = mbar_wait_bounded(&bars[b], (gg >> 1) & 1, kWaitLimitNs);
            consume(tiles + b * U, jb + t * T);
            // The barrier that frees the tile buffer for the next copy also makes
            // a timed-out wait (on any thread) the whole CTA's decision.
            if (__syncthreads_or(!arrived)) {
                ok = false;
                break;
            }
        }
    }
    gt = g0 + ntiles;
    if (!ok) {
        // A tile copy did not arrive within its bound: no further copy is
        // issued and the remaining tiles are skipped.  Before the epilogue
        // reuses the tile area, wait (bounded again) for this CTA's copies
        // still in flight -- tile t and, when it was issued, tile t + 1.
        if (threadIdx.x == 0) {
            const int gg = g0 + t;
            mbar_wait_bounded(&bars[gg & 1], (gg >> 1) & 1, kWaitLimitNs);
            if (t + 1 < ntiles) mbar_wait_bounded(&bars[(gg + 1) & 1], ((gg + 1) >> 1) & 1, kWaitLimitNs);
            atomicOr(p.status, ST_TMA_TIMEOUT);
        }
        __syncthreads();
    }

    // ---- epilogue: lanes -> warps -> (output | split partial)
    // Records of the last two tiles are still in shared memory (all of them
    // when they were predicted here), the others are read where they came
    // from.
    constexpr int RUN = NnRun<K, JL, R, V>::value;
    constexpr bool kRunNn = (K == kKernMixedP && (V & kVarStats) != 0) ||
                            (K == kKernF64 && (V & (kVarG4 | kVarPot)) == 0);
    const JRec *all = Src::kInPlace ? tiles - jb / JPU : jrec;
    auto records_of = [&](int unit) -> const JRec * {
        if (Src::kInPlace) return all;
        const int t2 = (unit * JPU - jb) / T;
        return t2 >= ntiles - 2 ? tiles + ((g0 + t2) & 1) * U - (jb + t2 * T) / JPU : jrec;
    };
    Partial q[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        bool unscaled = false;
        if constexpr (K == kKernMixedP && kRunNn) {
            if (st[r].nk >= 0) nn_of_run<JL, RUN, IDENT>(st[r], all);
        }
        if constexpr (K == kKernF64) {
            const int first = jb + kbase;
            // A sum that is not finite: some r^2 overflowed, vanished, or is
            // negative or NaN, or a sum is too large for the scale.  Summed
            // again, unscaled, with the pair term for any r^2.
            double zero = 0.0 * st[r].Pt;  // NaN when a sum is not finite
            if constexpr ((V & kVarPot) == 0)
                zero += 0.0 * st[r].Ax + 0.0 * st[r].Ay + 0.0 * st[r].Az + 0.0 * st[r].Jx + 0.0 * st[r].Jy +
                        0.0 * st[r].Jz;
            unscaled = !(zero == 0.0);
            if (unscaled) {
                st[r].Ax = st[r].Ay = st[r].Az = st[r].Jx = st[r].Jy = st[r].Jz = st[r].Pt = 0.0;
#pragma unroll 1
                for (int t2 = 0; t2 < ntiles; ++t2)
#pragma unroll 1
                    for (int m = 0; m < per; ++m) {
                        const int jg = first + t2 * T + m * JL;
                        interact_any<true, IDENT, (V & kVarG4) != 0, (V & kVarPot) != 0>(st[r], all[jg].pos,
                                                                                        all[jg].vel, jg);
                    }
            }
            if constexpr (kRunNn) {
                if (st[r].nties > kTies) {
#pragma unroll 1
                    for (int t2 = 0; t2 < ntiles; ++t2)
#pragma unroll 1
                        for (int m = 0; m < per; m += RUN) nn_scan_run<JL, RUN, IDENT>(st[r], all, first + t2 * T + m * JL);
                } else if (st[r].nk >= 0) {
#pragma unroll 1
                    for (int u = -1; u < st[r].nties; ++u) {
                        const int k = u < 0 ? st[r].nk : ties[r][u];
                        nn_scan_run<JL, RUN, IDENT>(st[r], records_of(k), k);
                    }
                }
            }
        }
        to_partial<(V & kVarPot) != 0>(st[r], q[r], unscaled);
        if (JL > 1) warp_reduce<IL>(q[r]);
    }
    if (H > 1) {
        if (Src::kInPlace || (K == kKernF64 && kRunNn)) __syncthreads();  // the tile area was read above
        if (jl == 0) {
#pragma unroll
            for (int r = 0; r < R; ++r) red[h * itile + islot + r * IL] = q[r];
        }
        __syncthreads();
        if (h == 0 && jl == 0) {
            for (int hh = 1; hh < H; ++hh) {
#pragma unroll
                for (int r = 0; r < R; ++r) add_partial(q[r], red[hh * itile + islot + r * IL]);
            }
        }
    }
    if (h == 0 && jl == 0) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = i0 + r * IL;
            if (i >= p.ni) continue;
            if (p.nsplit == 1 && !p.keep_partials)
                write_final<K == kKernF64>(p, i, q[r]);
            else
                store_partial(&p.part[(size_t)split * p.ni + i], q[r]);
        }
    }
    if (p.nsplit > 1 && p.tile_counter && !p.keep_partials) {
        // Last CTA of this i-tile folds the splits.  One thread releases the
        // CTA's partials and acquires the others' (a __threadfence in every
        // thread took 1-2 us of a small call).
        __shared__ int s_last;
        __syncthreads();
        if (threadIdx.x == 0) s_last = arrive_count(&p.tile_counter[itile_idx]) == p.nsplit - 1;
        __syncthreads();
        if (s_last) {
            const FoldArgs f{p.part,     p.ni,      p.nj,     p.nsplit, p.out_acc, p.out_jerk,
                             p.out_pot,  p.out_nn,  p.out_q,  K == kKernF64 ? p.out_map : nullptr};
            const int slots = IL == 32 ? (int)blockDim.x : (int)blockDim.x / 2;
            if constexpr ((V & kVarStats) != 0)
                fold_splits_inline(f, itile_idx * itile, itile, slots, red);
            else
                fold_splits(f, itile_idx * itile, itile, slots, red);
            if (threadIdx.x == 0) p.tile_counter[itile_idx] = 0;
        }
    }
    return ok;
}

__device__ __forceinline__ void init_bars(unsigned char *smem) {
    if (threadIdx.x == 0) {
        uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_barrier_init();
    }
}

}  // namespace g6
