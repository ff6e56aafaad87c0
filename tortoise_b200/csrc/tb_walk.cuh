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

// True when no point of the Monte-Carlo domain -- every free leg's point in
// its reference triangle, the partially constrained leg's coordinate in
// [0, 1] -- can pass the simplex tests ThetapC * ThetaFC
// (IntegratorCore.hpp:318-320), whatever the order the constrained
// coordinates are evaluated in: over the whole domain one of al0, al1, al2
// stays below 0, or kp0 + al0 or al1 + al2 stays above 1, by more than four
// times the rounding bound am.mg (which already covers the distance between
// the fused map and the reference-order evaluation).  Then neither table has
// a point inside: the survival sum is 0 and the tuple does not survive.
template <int L>
__device__ __forceinline__ bool domain_excludes(const AlphaMap<L>& am) {
    constexpr int R = AlphaMap<L>::R;
    const double eps = 2.220446049250313e-16;
    double hi[3];
    double plo = am.a0[0];                 // min of kp0 + al0
    double slo = am.a0[1] + am.a0[2];      // min of al1 + al2
#pragma unroll
    for (int r = 0; r < 3; ++r) hi[r] = am.a0[r];
#pragma unroll
    for (int b = 0; b < L - 2; ++b) {      // free legs: vertices (0,0), (1,0), (0,1)
#pragma unroll
        for (int r = 0; r < 3; ++r) hi[r] += fmax(0.0, fmax(am.G[r][2 * b], am.G[r][2 * b + 1]));
        plo += fmin(0.0, fmin(am.G[0][2 * b], am.G[0][2 * b + 1]));
        slo += fmin(0.0, fmin(am.G[1][2 * b] + am.G[2][2 * b], am.G[1][2 * b + 1] + am.G[2][2 * b + 1]));
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) hi[r] += fmax(0.0, am.G[r][R - 1]);   // kp0 in [0, 1]
    plo += fmin(0.0, am.G[0][R - 1] + 1.0);
    slo += fmin(0.0, am.G[1][R - 1] + am.G[2][R - 1]);
    const double m0 = 4.0 * am.mg[0], m1 = 4.0 * am.mg[1], m2 = 4.0 * am.mg[2];
    if (hi[0] < -m0 || hi[1] < -m1 || hi[2] < -m2) return true;
    if (plo - m0 > 1.0 + 8.0 * eps * (1.0 + fabs(plo))) return true;
    if (slo - (m1 + m2) > 1.0 + 8.0 * eps * (1.0 + fabs(slo))) return true;
    return false;
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

}  // namespace tb
