// tb_stream.cu -- the Monte-Carlo collision operator with its tuples
// enumerated on the fly, for channels whose tuple list does not fit in
// device memory (four-leg electron-electron channels on fine meshes: about
// 2e9 surviving tuples at 32x32, 3e10 at 64x64).
//
// Every evaluation walks the reference's candidate space again and keeps
// nothing between evaluations:
//   * work items (umklapp, sections of legs 0..L-2, element choice in those
//     sections) and, per item, the element box of the last leg: the nested
//     loops of nestedForSections / nestedForElements (include/Physics/
//     Scattering/ScatteringChannel.hpp:205-255) with the TrapezoidalSubset
//     box arithmetic (src/Geometry/Structured/DirectSpace/MeshSubset.cpp);
//   * the energy window, the determinant filter and the survival test of
//     precalculateIndices (src/Physics/Scattering/ScatteringChannel.cpp:
//     476-504) on the survival table;
//   * for the survivors, which points of the quadrature table lie inside the
//     simplices, and TypeB's sums over those points only
//     (include/Physics/Scattering/IntegratorCore.hpp:260-357).
// Every decision uses the same explicitly rounded operations as the stored
// enumeration (k_enumerate, compiled unfused) and the mask builder
// (k_theta_mask), and the sums use the stored-list kernel's code
// (tb_mcpoint.cuh), so a streamed evaluation adds the same per-tuple values
// as the stored-list path.
//
// Work distribution: a warp walks runs of consecutive work items, 32 at a
// time (one per lane); the lanes step through their boxes in lock step and
// push the candidates that pass the energy window into a per-warp queue in
// shared memory.  Three stages drain the queues, each on 32 entries at a
// time, one per lane: the determinant filter and an FP32 pass over the survival
// points, which ends most candidates (queue 0 -> 1); the FP64 survival test at
// the points it left (queue 1 -> 2); then the points inside, the sums and the
// scatter for the surviving tuples.  So every stage runs on full warps
// whatever the box sizes and the pass rate of the stage before.
#include "tb_dp45.cuh"
#include "tb_mcpoint.cuh"
#include "tb_scatter.cuh"
#include "tb_stream.cuh"
#include "tb_walk.cuh"

namespace tb {

// 4 warps per block, 3 blocks per SM: the register cap of 168 per thread
// spills a little, but 12 resident warps per SM instead of 8 hide more of the
// FP64 latency (a 16x16 e-e evaluation: 306 ms against 387 ms with blocks of
// 8 warps at 221 registers, one block per SM)
constexpr int ST_WARPS = 4;    // warps per block
#ifndef TB_STREAM_MIN_BLOCKS
#define TB_STREAM_MIN_BLOCKS 3
#endif

// MODE: ST_PROPAGATE (the collision terms), ST_RATE (rate_leg's scattering
// rate) or ST_VJP (acc = grad_f += the transposed terms for the co-state co,
// grad_amp[k] += <co, dC/d amplitude_k>; the stored-list VJP's arithmetic).
enum { ST_PROPAGATE = 0, ST_RATE = 1, ST_VJP = 2 };

template <int L, int MODE>
__global__ void __launch_bounds__(ST_WARPS * 32, TB_STREAM_MIN_BLOCKS)
    k_collision_stream(ChanDev c, StreamDev sd, int64_t it0, int64_t it1, const InstDev* __restrict__ insts,
                       int n_insts, const double* __restrict__ f, double* __restrict__ acc,
                       const DPCtl* __restrict__ ctl, int rate_leg, FxAcc fx, const double* __restrict__ co,
                       double* __restrict__ grad_amp, FxAcc fx_amp) {
    constexpr bool RATE = MODE == ST_RATE;
    {
        // every instance off or its run finished: nothing to add
        bool any = false;
        for (int k = 0; k < n_insts && !any; ++k)
            any = insts[k].amp_full != 0.0 && !(ctl && ctl[insts[k].run].done);
        if (!any) return;
    }
    constexpr int R = 2 * (L - 2) + 1;
    extern __shared__ __align__(16) double s_tab[];   // [nmc R] quadrature table, then [nmc R] survival table
    // per-warp candidate queues: [0] inside the energy window, [1] past the
    // determinant filter and with points that may be inside, [2] surviving tuples
    __shared__ int32_t s_q[3][ST_WARPS][L + 1][ST_QUEUE];
    __shared__ uint64_t s_may[ST_WARPS][ST_QUEUE];   // queue 1: survival points that may be inside
    double* s_mc = s_tab;
    double* s_pre = s_tab + c.nmc * R;
    float* s_fmc = reinterpret_cast<float*>(s_tab + (2 * c.nmc * R + 1) / 2 * 2);   // their FP32 copies
    float* s_fpre = s_fmc + c.nmc * FloatTable<L>::FT;
    for (int i = threadIdx.x; i < c.nmc * R; i += blockDim.x) {
        s_mc[i] = c.mc[i];
        s_pre[i] = sd.mc_pre[i];
        s_fmc[i / R * FloatTable<L>::FT + i % R] = float_point(sd, c.mc[i]);
        s_fpre[i / R * FloatTable<L>::FT + i % R] = float_point(sd, sd.mc_pre[i]);
    }
    __syncthreads();
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double sqrt2 = 1.4142135623730951;   // sqrt(2.0), correctly rounded
    double prodc = 1.0;
#pragma unroll
    for (int l = 0; l < L; ++l) prodc *= sqrt2;
    // s_cnt[k]: prodc added k times to 0.0, in sequence
    __shared__ double s_cnt[65];
    if (threadIdx.x == 0) {
        double t = 0.0;
        s_cnt[0] = t;
        for (int k = 1; k <= 64; ++k) s_cnt[k] = (t += prodc);
    }
    __syncthreads();
    const double inv_fact_nmc = c.fact * double(c.nmc);
    unsigned long long n_pre = 0, n_det = 0, n_surv = 0, n_pts = 0, n_tin = 0;

    int q1n = 0;   // candidates in queue 1 (warp-uniform)
    int q2n = 0;   // surviving tuples in queue 2 (warp-uniform)

    // Stage 1 for `take` candidates of queue 0 from slot `first` on, one per
    // lane: the determinant filter, then the points of the survival table that
    // FP32 cannot place outside; the candidates with such a point go to queue 1.
    // Most candidates of the energy window end here.
    auto stage1 = [&](int first, int take) {
        const bool valid = lane < take;
        int e[L];
        int u = 0;
#pragma unroll
        for (int l = 0; l < L; ++l) e[l] = valid ? s_q[0][warp][l][first + lane] : 0;
        if (valid) u = s_q[0][warp][L][first + lane];
        TupleGeom<L> g;
        tuple_geometry<L>(c, e, u, g);
        bool ok = valid && (fabs(g.det) >= c.min_det);
        n_pre += valid ? 1 : 0;
        n_det += ok ? 1 : 0;
        uint64_t may = 0;
        if (ok) {
            double Ci[3][3];
            dc_inverse<L>(g, Ci);
            AlphaMap<L> am;
            alpha_map<L>(g, Ci, am);
            double T[2];
            outside_thresholds<L>(am, T);
            may = maybe_inside<L>(am, T, s_fpre, c.nmc);
            ok = may != 0ull || c.threshold < 0.0;
        }
        const unsigned bal = __ballot_sync(full, ok);
        if (ok) {
            const int pos = q1n + __popc(bal & ((1u << lane) - 1u));
#pragma unroll
            for (int l = 0; l <= L; ++l) s_q[1][warp][l][pos] = l < L ? e[l] : u;
            s_may[warp][pos] = may;
        }
        q1n += __popc(bal);
        __syncwarp();
    };

    // Stage 2 for `take` candidates of queue 1 from slot `first` on, one per
    // lane: the survival test; the surviving tuples go to queue 2.
    auto survive = [&](int first, int take) {
        const bool valid = lane < take;
        int e[L];
        int u = 0;
#pragma unroll
        for (int l = 0; l < L; ++l) e[l] = valid ? s_q[1][warp][l][first + lane] : 0;
        if (valid) u = s_q[1][warp][L][first + lane];
        TupleGeom<L> g;
        tuple_geometry<L>(c, e, u, g);
        const double adet = fabs(g.det);
        bool ok = valid && (adet >= c.min_det);
        double Ci[3][3];
        dc_inverse<L>(g, Ci);
        AlphaMap<L> am;
        alpha_map<L>(g, Ci, am);
        // survival test of precalculateIndices on the survival table: the
        // count of k_enumerate's, with each point's simplex decision taken
        // the way k_theta_mask takes it (the fused map, re-evaluated in the
        // reference's order near a face: the same decisions, at a fraction of
        // the cost of evaluating every point in that order)
        // (the reference adds prodc for every point inside: the sum of cnt
        // such terms is s_cnt[cnt], the same additions in the same order)
        double T[2];
        outside_thresholds<L>(am, T);
        const double per = 1.0 / (c.fact * double(c.nmc) * adet);
        // res grows with the count: where one point inside is enough, the first one ends the search
        const bool one = fabs(per * s_cnt[1] * c.amp_vol) > c.threshold;
        int cnt = 0;
        for (uint64_t mk = valid ? s_may[warp][first + lane] : 0ull; mk; mk &= mk - 1)
            if (theta_decide_t<L>(g, Ci, am, T, s_pre + (__ffsll((long long)mk) - 1) * R)) {
                ++cnt;
                if (one) break;
            }
        double res = per * s_cnt[cnt];
        res *= c.amp_vol;
        ok = ok && (fabs(res) > c.threshold);
        n_surv += ok ? 1 : 0;
        const unsigned bal = __ballot_sync(full, ok);
        if (ok) {
            const int pos = q2n + __popc(bal & ((1u << lane) - 1u));
#pragma unroll
            for (int l = 0; l <= L; ++l) s_q[2][warp][l][pos] = l < L ? e[l] : u;
        }
        q2n += __popc(bal);
        __syncwarp();
    };

    // Stage 3 for `take` surviving tuples of queue 2 from slot `first` on,
    // one per lane: the points inside, the sums, the scatter.  (The survivors
    // are a fifth of the candidates that reach stage 2; gathered into full
    // warps, the quadrature runs on every lane.)
    auto evaluate = [&](int first, int take) {
        const bool valid = lane < take;
        int e[L];
        int u = 0;
#pragma unroll
        for (int l = 0; l < L; ++l) e[l] = valid ? s_q[2][warp][l][first + lane] : 0;
        if (valid) u = s_q[2][warp][L][first + lane];
        TupleGeom<L> g;
        tuple_geometry<L>(c, e, u, g);
        const double adet = fabs(g.det);
        double Ci[3][3];
        dc_inverse<L>(g, Ci);
        AlphaMap<L> am;
        alpha_map<L>(g, Ci, am);
        // the points inside the simplices on the quadrature table (k_theta_mask's)
        uint64_t mk = 0;
        if (valid) {
            double T[2];
            outside_thresholds<L>(am, T);
            for (uint64_t w = maybe_inside<L>(am, T, s_fmc, c.nmc); w; w &= w - 1) {
                const int m = __ffsll((long long)w) - 1;
                if (theta_decide_t<L>(g, Ci, am, T, s_mc + m * R)) mk |= 1ull << m;
            }
        }
        n_pts += __popcll(mk);
        n_tin += mk ? 1 : 0;
        if (!__any_sync(full, mk != 0ull)) return;
        const bool live = mk != 0ull;
        if (MODE == ST_VJP) {
            // k_vjp_mc's terms for the tuples of the list (tf = 1: no functAmplitude)
            const double scale = live ? 1.0 / (c.fact * double(c.nmc) * fabs(g.det)) : 0.0;
            for (int k = 0; k < n_insts; ++k) {
                const InstDev in = insts[k];
                double gA[L][3], gB[L][3], gamp, sa[L], sb[L];
                vjp_point_sums<L, true>(c, in, f, co, e, g, Ci, s_mc, mk, live, gA, gB, gamp, sa, sb);
                if (live) {
                    const double sc = scale * (in.amp_full * 1.0);
#pragma unroll
                    for (int l = 0; l < L; ++l) {
                        const int64_t key = in.foff[l] + 3 * (int64_t)e[l];
#pragma unroll
                        for (int j = 0; j < 3; ++j) {
                            const double gv = __dmul_rn(sc, fma(sb[l], gB[l][j], __dmul_rn(sa[l], gA[l][j])));
                            if (fx.w) fx_add(fx, key + j, gv);
                            else atomicAdd(acc + key + j, gv);
                        }
                    }
                }
                block_atomic_sum(live ? scale * (c.amp_vol * 1.0) * gamp : 0.0, grad_amp + k, fx_amp, k);
            }
            return;
        }
        const double scale = live ? 1.0 / (inv_fact_nmc * adet) : 0.0;
        for (int k = 0; k < n_insts; ++k) {
            const InstDev in = insts[k];
            if (in.amp_full == 0.0) continue;
            if (ctl && ctl[in.run].done) continue;
            const double ampt = in.amp_full;
            double s0 = 0.0, sx[L], sy[L];
#pragma unroll
            for (int l = 0; l < L; ++l) { sx[l] = 0.0; sy[l] = 0.0; }
            if (live) {
                double fv[L][3];
                leg_values<L, RATE>(c, in, f, e, rate_leg, fv);
                inside_point_sums<L, RATE>(c, am, s_mc, mk, fv, rate_leg, s0, sx, sy);
            }
#pragma unroll
            for (int l = 0; l < L; ++l) {
                if (RATE && l != rate_leg) continue;   // uniform: the rate keeps one leg
                const double d = RATE ? -c.leg[l].dir : c.leg[l].dir;
                const int64_t key = in.foff[l] + 3 * (int64_t)e[l];
                const double v0 = d * ((scale * s0) * ampt), v1 = d * ((scale * sx[l]) * ampt),
                             v2 = d * ((scale * sy[l]) * ampt);
                if (fx.w) {
                    if (live) fx_add3(fx, key, v0, v1, v2);
                } else if (l < L - 1) {
                    warp_scatter3(live ? key : -1, acc + key, v0, v1, v2);
                } else if (live) {
                    atomicAdd(acc + key + 0, v0);
                    atomicAdd(acc + key + 1, v1);
                    atomicAdd(acc + key + 2, v2);
                }
            }
        }
    };

    int qn = 0;   // queued candidates (warp-uniform)
    // Each warp takes runs of ST_SPAN x 32 consecutive items, interleaved
    // over the grid; the lanes hold consecutive items and step by 32.
    const int64_t n_warps = int64_t(gridDim.x) * ST_WARPS;
    const int64_t run = int64_t(ST_SPAN) * 32;
    const WalkLeg& ml = sd.leg[L - 1];
    for (int64_t rb = it0 + (int64_t(blockIdx.x) * ST_WARPS + warp) * run; rb < it1; rb += n_warps * run) {
        WalkPos<L> p;
        walk_decode<L>(sd, rb + lane, p);
        WalkFront fr;
        bool front_ok = false;
        for (int st = 0; st < ST_SPAN; ++st) {
            const int64_t base = rb + int64_t(st) * 32;
            if (base >= it1) break;
            const int64_t item = base + lane;
            int e[L];
            int lo[2] = {0, 0}, hi[2] = {0, 0};
            double pmn = 0.0, pmx = 0.0;   // energy window of legs 0..L-2, summed in leg order
            int ncand = 0;
            if (item < it1) {
                walk_at<L>(c, sd, p, fr, front_ok, e, lo, hi, pmn, pmx);
                if (lo[0] != hi[0] && lo[1] != hi[1]) ncand = 2 * (hi[0] - lo[0]) * (hi[1] - lo[1]);
            }
            const int u = p.u;
            const int maxc = __reduce_max_sync(full, unsigned(ncand));
            // candidate k of the box: element 2 (cx + cy nx) + ie with
            // cx = lo0 + (k / 2) % nbx, cy = lo1 + (k / 2) / nbx, ie = k % 2
            int cx = lo[0], cy = lo[1], ie = 0;
            for (int k = 0; k < maxc; ++k) {
                bool pass = false;
                int el = 0;
                if (k < ncand) {
                    el = 2 * (cx + cy * ml.nx) + ie;
                    const double emin = __ldg(ml.minE + el), emax = __ldg(ml.maxE + el);
                    const double minE = pmn + ((c.leg[L - 1].dir > 0) ? emin : -emax);
                    const double maxE = pmx + ((c.leg[L - 1].dir > 0) ? emax : -emin);
                    pass = (minE <= 0.0) && (maxE >= 0.0);
                }
                if (ie) {
                    ie = 0;
                    if (++cx == hi[0]) { cx = lo[0]; ++cy; }
                } else {
                    ie = 1;
                }
                const unsigned bal = __ballot_sync(full, pass);
                if (pass) {
                    const int pos = qn + __popc(bal & ((1u << lane) - 1u));
#pragma unroll
                    for (int l = 0; l < L - 1; ++l) s_q[0][warp][l][pos] = e[l];
                    s_q[0][warp][L - 1][pos] = el;
                    s_q[0][warp][L][pos] = u;
                }
                qn += __popc(bal);
                __syncwarp();
                if (qn >= 32) {
                    stage1(qn - 32, 32);
                    qn -= 32;
                    if (q1n >= 32) {
                        survive(q1n - 32, 32);
                        q1n -= 32;
                        if (q2n >= 32) {
                            evaluate(q2n - 32, 32);
                            q2n -= 32;
                        }
                    }
                    __syncwarp();   // the slots are reused
                }
            }
            if (walk_advance<L>(sd, p)) front_ok = false;
        }
    }
    // the queues' remainders, survivors first once queue 1 is empty
    if (qn > 0) stage1(0, qn);
    for (;;) {
        if (q2n >= 32 || (q1n == 0 && q2n > 0)) {
            const int t = min(q2n, 32);
            evaluate(q2n - t, t);
            q2n -= t;
        } else if (q1n > 0) {
            const int t = min(q1n, 32);
            survive(q1n - t, t);
            q1n -= t;
        } else {
            break;
        }
        __syncwarp();
    }
    if (sd.counts) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            n_pre += __shfl_down_sync(full, n_pre, o);
            n_det += __shfl_down_sync(full, n_det, o);
            n_surv += __shfl_down_sync(full, n_surv, o);
            n_pts += __shfl_down_sync(full, n_pts, o);
            n_tin += __shfl_down_sync(full, n_tin, o);
        }
        if (lane == 0 && (n_pre | n_det | n_surv | n_pts | n_tin)) {
            atomicAdd(sd.counts + 0, n_pre);
            atomicAdd(sd.counts + 1, n_det);
            atomicAdd(sd.counts + 2, n_surv);
            atomicAdd(sd.counts + 3, n_pts);
            atomicAdd(sd.counts + 4, n_tin);
        }
    }
}

template <int L, int MODE>
static int launch_stream(const ChanDev& c, const StreamDev& sd, int64_t it0, int64_t it1, const InstDev* insts,
                         int n_insts, const double* f, double* acc, const DPCtl* ctl, cudaStream_t s, int rate_leg,
                         const FxAcc& fx, const double* co = nullptr, double* grad_amp = nullptr,
                         const FxAcc& fx_amp = FxAcc{}) {
    auto kern = k_collision_stream<L, MODE>;
    const int threads = ST_WARPS * 32;
    const size_t smem = 2 * sizeof(double) * size_t(c.nmc) * c.R + 16 + 2 * sizeof(float) * size_t(c.nmc) * FloatTable<L>::FT;
    int dev = 0, nsm = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
    if (per_sm < 1) per_sm = 1;
    const int64_t batches = (it1 - it0 + ST_SPAN * 32 - 1) / (ST_SPAN * 32);
    int64_t blocks = (batches + ST_WARPS - 1) / ST_WARPS;
    // several waves of resident blocks: the work per item varies a lot
    const int64_t cap = int64_t(nsm) * per_sm * 8;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) return TB_OK;
    kern<<<unsigned(blocks), threads, smem, s>>>(c, sd, it0, it1, insts, n_insts, f, acc, ctl,
                                                 MODE == ST_RATE ? rate_leg : -1, fx, co, grad_amp, fx_amp);
    TB_CUDA(cudaGetLastError());
    return TB_OK;
}

int launch_collision_stream(const ChanDev& c, const StreamDev& sd, int64_t item_begin, int64_t item_end,
                            const InstDev* insts, int n_insts, const double* f, double* acc, const DPCtl* ctl,
                            cudaStream_t s, int rate_leg, const FxAcc& fx) {
    if (item_end <= item_begin || n_insts <= 0) return TB_OK;
    if (c.nmc > 64) { set_error("streamed channels take at most 64 Monte-Carlo points"); return TB_ERR_ARG; }
#define TB_ST(LL)                                                                                             \
    (rate_leg >= 0                                                                                            \
         ? launch_stream<LL, ST_RATE>(c, sd, item_begin, item_end, insts, n_insts, f, acc, ctl, s, rate_leg, fx) \
         : launch_stream<LL, ST_PROPAGATE>(c, sd, item_begin, item_end, insts, n_insts, f, acc, ctl, s, -1, fx))
    switch (c.L) {
        case 2: return TB_ST(2);
        case 3: return TB_ST(3);
        case 4: return TB_ST(4);
    }
#undef TB_ST
    set_error("nlegs must be 2..4");
    return TB_ERR_ARG;
}

int launch_vjp_stream(const ChanDev& c, const StreamDev& sd, int64_t item_begin, int64_t item_end,
                      const InstDev* insts, int n_insts, const double* f, const double* u, double* grad_f,
                      double* grad_amp, cudaStream_t s, const FxAcc& fx, const FxAcc& fx_amp) {
    if (item_end <= item_begin || n_insts <= 0) return TB_OK;
    if (c.nmc > 64) { set_error("streamed channels take at most 64 Monte-Carlo points"); return TB_ERR_ARG; }
    StreamDev q = sd;
    q.counts = nullptr;
#define TB_SV(LL) launch_stream<LL, ST_VJP>(c, q, item_begin, item_end, insts, n_insts, f, grad_f, nullptr, s, -1, \
                                            fx, u, grad_amp, fx_amp)
    switch (c.L) {
        case 2: return TB_SV(2);
        case 3: return TB_SV(3);
        case 4: return TB_SV(4);
    }
#undef TB_SV
    set_error("nlegs must be 2..4");
    return TB_ERR_ARG;
}

}  // namespace tb
