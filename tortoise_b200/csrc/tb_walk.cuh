// tb_walk.cuh -- the candidate walk of precalculateIndices and its tests, shared
// by the streamed collision operator (tb_stream.cu) and the tuple enumeration
// (tb_enumerate.cu).
#pragma once

#include "tb_geom.cuh"
#include "tb_stream.cuh"

namespace tb {

constexpr int ST_QUEUE = 64;   // candidate slots per warp (31 left over + 32 pushed at most)
constexpr int ST_SPAN = 16;    // steps of 32 consecutive items per run of a warp

struct WBox {
    double l[2], h[2];
};

// One section's box, shrunk by 1e-8 section units (MeshSubset.cpp:62-66),
// in absolute coordinates.
__device__ __forceinline__ WBox walk_section_box(const WalkLeg& m, int sx, int sy) {
    WBox b;
    const double lo0 = xa(double(sx), 0.00000001), lo1 = xa(double(sy), 0.00000001);
    const double hi0 = xs(double(sx + 1), 0.00000001), hi1 = xs(double(sy + 1), 0.00000001);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        b.l[i] = xa(m.origin[i], xa(xm(m.dG[i][0], lo0), xm(m.dG[i][1], lo1)));
        b.h[i] = xa(m.origin[i], xa(xm(m.dG[i][0], hi0), xm(m.dG[i][1], hi1)));
    }
    return b;
}

__device__ __forceinline__ WBox walk_box_scale(WBox b, double s) {
    if (s >= 0.0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) { b.l[i] = xm(b.l[i], s); b.h[i] = xm(b.h[i], s); }
    } else {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const double t = b.l[i];
            b.l[i] = xm(b.h[i], s);
            b.h[i] = xm(t, s);
        }
    }
    return b;
}

// A lane's place in the work-item numbering, as digits (least significant
// first): the element choice, then for legs L-2 .. 0 the section's x and y,
// then the umklapp column.  A warp walks runs of consecutive items, so most
// steps change the last digits only: the box sums of the legs in front
// (legs 0..L-3) and their energies are kept from the previous item.
template <int L>
struct WalkPos {
    int comb, u;
    int sx[TB_MAX_LEGS], sy[TB_MAX_LEGS];
};

template <int L>
__device__ __forceinline__ void walk_decode(const StreamDev& sd, int64_t item, WalkPos<L>& p) {
    constexpr int C = 1 << (L - 1);
    p.comb = int(item % C);
    int64_t r = item / C;
#pragma unroll
    for (int l = L - 2; l >= 0; --l) {
        const int sec = int(r % sd.nsec[l]);
        r /= sd.nsec[l];
        p.sx[l] = sec % sd.leg[l].nx;
        p.sy[l] = sec / sd.leg[l].nx;
    }
    p.u = int(r);
}

// p += 32 items.  Returns true when a digit of legs 0..L-3 or the umklapp
// column changed (the kept box sums are stale).
template <int L>
__device__ __forceinline__ bool walk_advance(const StreamDev& sd, WalkPos<L>& p) {
    constexpr int C = 1 << (L - 1);
    int carry = 32 / C;
    bool front = false;
#pragma unroll
    for (int l = L - 2; l >= 0; --l) {
        if (carry) {
            if (l < L - 2) front = true;
            int x = p.sx[l] + carry;
            carry = 0;
            if (x >= sd.leg[l].nx) { carry = x / sd.leg[l].nx; x -= carry * sd.leg[l].nx; }
            int y = p.sy[l] + carry;
            carry = 0;
            if (y >= sd.leg[l].ny) { carry = y / sd.leg[l].ny; y -= carry * sd.leg[l].ny; }
            p.sx[l] = x;
            p.sy[l] = y;
        }
    }
    if (carry) { p.u += carry; front = true; }
    return front;
}

// What the legs in front contribute to an item: their box sum (legs 0..L-3),
// the umklapp shift and the energy-window partial sums of legs 0..L-3.
struct WalkFront {
    WBox box;
    double gu[2];
    double mn, mx;
};

// The item at p: elements of legs 0..L-2, the last leg's section range
// [lo, hi) and the energy-window sums of legs 0..L-2 (pmn, pmx; the last
// leg's term is added per candidate).  The decoding and box arithmetic of
// k_enumerate, term for term and in the same order (the kept front sums are
// its partial sums); fr is refreshed when ok is false.
template <int L>
__device__ __forceinline__ void walk_at(const ChanDev& c, const StreamDev& sd, const WalkPos<L>& p, WalkFront& fr,
                                        bool& ok, int (&e)[L], int (&lo)[2], int (&hi)[2], double& pmn,
                                        double& pmx) {
#pragma unroll
    for (int l = 0; l < L - 1; ++l) e[l] = 2 * (p.sy[l] * sd.leg[l].nx + p.sx[l]) + ((p.comb >> (L - 2 - l)) & 1);
    if (!ok) {
        const double ux = c.umk[2 * p.u], uy = c.umk[2 * p.u + 1];
        fr.gu[0] = xa(xm(c.gvec[0], ux), xm(c.gvec[2], uy));
        fr.gu[1] = xa(xm(c.gvec[1], ux), xm(c.gvec[3], uy));
        fr.mn = 0.0;
        fr.mx = 0.0;
#pragma unroll
        for (int l = 0; l < L - 2; ++l) {
            const WBox b = walk_box_scale(walk_section_box(sd.leg[l], p.sx[l], p.sy[l]), c.leg[l].dir);
            if (l == 0) fr.box = b;
            else {
#pragma unroll
                for (int i = 0; i < 2; ++i) { fr.box.l[i] = xa(fr.box.l[i], b.l[i]); fr.box.h[i] = xa(fr.box.h[i], b.h[i]); }
            }
            const double emin = __ldg(sd.leg[l].minE + e[l]), emax = __ldg(sd.leg[l].maxE + e[l]);
            fr.mn += (c.leg[l].dir > 0) ? emin : -emax;
            fr.mx += (c.leg[l].dir > 0) ? emax : -emin;
        }
        ok = true;
    }
    constexpr int K = L - 2;   // the leg whose section changes from item to item
    WBox acc = walk_box_scale(walk_section_box(sd.leg[K], p.sx[K], p.sy[K]), c.leg[K].dir);
    if (K > 0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) { acc.l[i] = xa(fr.box.l[i], acc.l[i]); acc.h[i] = xa(fr.box.h[i], acc.h[i]); }
    }
    acc.l[0] = xa(acc.l[0], fr.gu[0]); acc.h[0] = xa(acc.h[0], fr.gu[0]);
    acc.l[1] = xa(acc.l[1], fr.gu[1]); acc.h[1] = xa(acc.h[1], fr.gu[1]);
    acc = walk_box_scale(acc, -c.leg[L - 1].dir);
    const WalkLeg& ml = sd.leg[L - 1];
    const int ns[2] = {ml.nx, ml.ny};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const double tl = xa(xm(ml.invdG[i][0], xs(acc.l[0], ml.origin[0])), xm(ml.invdG[i][1], xs(acc.l[1], ml.origin[1])));
        const double th = xa(xm(ml.invdG[i][0], xs(acc.h[0], ml.origin[0])), xm(ml.invdG[i][1], xs(acc.h[1], ml.origin[1])));
        const int aa = int(floor(tl));
        const int bb = int(xa(floor(th), 1.0));
        lo[i] = min(max(aa, 0), ns[i]);
        hi[i] = min(max(bb, 0), ns[i]);
    }
    pmn = fr.mn;
    pmx = fr.mx;
    if (lo[0] != hi[0] && lo[1] != hi[1]) {
        const double emin = __ldg(sd.leg[K].minE + e[K]), emax = __ldg(sd.leg[K].maxE + e[K]);
        pmn += (c.leg[K].dir > 0) ? emin : -emax;
        pmx += (c.leg[K].dir > 0) ? emax : -emin;
    }
}

// Per-tuple thresholds of a cheaper "clearly outside" test than
// theta_decide's: T[0] for kp0 + al0, T[1] for al1 + al2.  Over the whole
// Monte-Carlo domain (every coordinate of q in [0, 1]) the fused
// coordinates obey |al_r| <= B_r = |a0_r| + sum_j |G_rj| (up to a factor
// 1 + 1e-15, covered by the 1.000001 below), so theta_decide's per-point
// bounds mg0 + tiny (2 + |al0|) and mg1 + mg2 + tiny (1 + |al1| + |al2|) are
// at most X = mg0 + tiny (2 + B0) and Y = mg1 + mg2 + tiny (1 + B1 + B2).
// A point with fl(kp0 + al0) > fl(1 + 4 X) has fl(fl(kp0 + al0) - 1) > 3.8 X
// (X >= 2 tiny, so the roundings of 1 + 4 X and of the difference cost less
// than 0.2 X), above theta_decide's computed bound: theta_decide also calls
// it outside.  Likewise for al1 + al2 against fl(1 + 4 Y).  The faster test
// therefore only sends a few more points to the exact evaluation, and every
// decision stays the reference-order one.
template <int L>
__device__ __forceinline__ void outside_thresholds(const AlphaMap<L>& am, double (&T)[2]) {
    constexpr int R = AlphaMap<L>::R;
    const double tiny = 8.0 * 1.1102230246251565e-16;
    double B[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        double t = fabs(am.a0[r]);
#pragma unroll
        for (int j = 0; j < R; ++j) t += fabs(am.G[r][j]);
        B[r] = 1.000001 * t;
    }
    const double X = am.mg[0] + tiny * (2.0 + B[0]);
    const double Y = (am.mg[1] + am.mg[2]) + tiny * ((1.0 + B[1]) + B[2]);
    T[0] = 1.0 + 4.0 * X;
    T[1] = 1.0 + 4.0 * Y;
}

// theta_decide with the per-tuple thresholds above: the same decision.
template <int L>
__device__ __forceinline__ bool theta_decide_t(const TupleGeom<L>& g, const double (&Ci)[3][3], const AlphaMap<L>& am,
                                               const double (&T)[2], const double* qv) {
    constexpr int R = AlphaMap<L>::R;
    double al[3];
    alpha_fast<L>(am, qv, al);
    const double kp0 = qv[R - 1];
    const bool out = (al[0] < -am.mg[0]) || (al[1] < -am.mg[1]) || (al[2] < -am.mg[2]) ||
                     (__dadd_rn(kp0, al[0]) > T[0]) || (__dadd_rn(al[1], al[2]) > T[1]);
    if (out) return false;
    return alpha_theta<L>(g, Ci, am, qv, al);
}

// The Monte-Carlo table in FP32, FT floats a point (built by the block).
template <int L>
struct FloatTable {
    static constexpr int R = 2 * (L - 2) + 1;
    static constexpr int FT = R <= 1 ? 1 : R <= 4 ? 4 : 8;
};
__device__ __forceinline__ float float_point(const StreamDev& sd, double q) {
    return sd.wide ? __int_as_float(0x7fc00000) : float(q);
}

// The points that FP32 arithmetic cannot place clearly outside: bit m is clear
// only where theta_decide is false.  Most points of most tuples are far outside,
// and FP32 runs beside the FP64 pipe at twice its rate, so the FP64 decisions
// are left to the set bits (12x10 e-e, streamed: 13.0 -> 10.3 ms; enumeration of
// 16x16 e-e: 91 -> 62 ms).  With u = 2^-24, B_r = |a0_r| + sum_j |G_rj| and |q_j|
// <= 1.5, the FP32 value of alpha_r (operands rounded to FP32, at most R + 1 fused
// steps) is within 1.5 (R + 4) u B_r of the real map, R <= 5, and so within E_r =
// 16 u B_r: a value below -(E_r + 4 mg_r) leaves the FP64 one below -mg_r, and
// kp0 + alpha_0 or alpha_1 + alpha_2 above their threshold T (outside_thresholds)
// by those E and 16 u of the operands leaves the FP64 sum above T.  Comparisons
// with NaN are false, and an infinite bound keeps every point: a table with larger
// coordinates is NaN in FP32 (float_point).
template <int L>
__device__ __forceinline__ uint64_t maybe_inside(const AlphaMap<L>& am, const double (&T)[2], const float* tab, int nmc) {
    constexpr int R = AlphaMap<L>::R, FT = FloatTable<L>::FT;
    const double u = 5.9604644775390625e-8;
    float a[3], G[3][R], lo[3], B[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        double b = fabs(am.a0[r]);
        a[r] = float(am.a0[r]);
#pragma unroll
        for (int j = 0; j < R; ++j) {
            b += fabs(am.G[r][j]);
            G[r][j] = float(am.G[r][j]);
        }
        B[r] = __double2float_ru(16.0 * u * b);
        lo[r] = -__double2float_ru(16.0 * u * b + 4.0 * am.mg[r]);
    }
    const float hi0 = __double2float_ru(T[0] + 32.0 * u) + 2.0f * B[0];
    const float hi1 = __double2float_ru(T[1] + 32.0 * u) + 2.0f * (B[1] + B[2]);
    uint32_t word[2] = {0u, 0u};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int m0 = 32 * h, m1 = min(nmc, m0 + 32);
        uint32_t bit = 1u;
#pragma unroll 1   // more points a step cost registers (a 12x10 e-e evaluation: 2 11.2 ms, 4 12.2, against 10.3)
        for (int m = m0; m < m1; ++m, bit += bit) {
            float q[R];
#pragma unroll
            for (int j = 0; j < R; ++j) q[j] = tab[m * FT + j];
            float al[3];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                al[r] = a[r];
#pragma unroll
                for (int j = 0; j < R; ++j) al[r] = fmaf(G[r][j], q[j], al[r]);
            }
            const bool out = (al[0] < lo[0]) || (al[1] < lo[1]) || (al[2] < lo[2]) || (q[R - 1] + al[0] > hi0) ||
                             (al[1] + al[2] > hi1);
            word[h] |= out ? 0u : bit;
        }
    }
    const uint64_t mask = uint64_t(word[1]) << 32 | word[0];
    return mask;
}

}  // namespace tb
