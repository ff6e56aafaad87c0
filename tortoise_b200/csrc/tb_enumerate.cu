// tb_enumerate.cu -- on-device tuple enumeration (the "precalculateIndices"
// step of the reference), compiled with --fmad=false so that every
// floating-point decision (box floors, energy window, determinant filter,
// survival threshold) rounds exactly like the reference's unfused C++.
//
// Reference loop structure (followed one-to-one):
//   deterministicIteration / nestedForSections / nestedForElements
//       include/Physics/Scattering/ScatteringChannel.hpp:205-255
//   survival test inside precalculateIndices
//       src/Physics/Scattering/ScatteringChannel.cpp:476-504
//   TrapezoidalSubset box arithmetic
//       src/Geometry/Structured/DirectSpace/MeshSubset.cpp:62-66, 82-87, 121-125, 169-194
//
// Design: the work items are (umklapp, section of legs 0..L-2, element choice
// of legs 0..L-2) flattened so that increasing item index is the reference's
// loop order; each item scans the element box of the last leg in increasing
// element id (which is the reference's MeshSubsetElementIterator order).  A
// count pass, an exclusive scan and a write pass then emit the surviving
// tuples in exactly the reference's order, deterministically, with no sort.
//
// Two count passes.  k_enumerate scans an item per thread and evaluates every
// point of a candidate in the reference's order, and the write pass does all of
// it again.  k_enum_walk is the streamed operator's walk (tb_walk.cuh): it
// gathers the candidates of each stage into full warps, drops those that FP32
// places outside at every point, decides the others on the fused map where the
// rounding bound allows (the same decisions), and leaves one bit per surviving candidate of an
// item, so that k_enum_write has no test to repeat.  It takes tables of at most
// 64 points inside the reference domain, and boxes of at most 64 candidates;
// a channel that does not fit goes through k_enumerate.  Measured, whole
// tb_create: 64x64 two-band e-ph 97 -> 37 ms (enumeration 72 -> 14), 16x16 e-e
// 410 -> 105 ms (367 -> 64).
#include <cub/cub.cuh>

#include <algorithm>

#include "tb_enumerate.cuh"
#include "tb_geom.cuh"
#include "tb_walk.cuh"

namespace tb {

struct EnumLeg {
    const double* minE;
    const double* maxE;
    int nx, ny;
    double origin[2];
    double dG[2][2];
    double invdG[2][2];
};

struct EnumArgs {
    ChanDev c;
    EnumLeg leg[TB_MAX_LEGS];
    int64_t nsec[TB_MAX_LEGS];   // sections of legs 0..L-2 (1 for unused)
    const double* mc_pre;        // [nmc*R] device
};

struct Box { double l[2], h[2]; };

__device__ __forceinline__ Box section_box(const EnumLeg& m, int sx, int sy) {
    Box b;
    const double lo0 = double(sx) + 0.00000001, lo1 = double(sy) + 0.00000001;
    const double hi0 = double(sx + 1) - 0.00000001, hi1 = double(sy + 1) - 0.00000001;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        b.l[i] = m.origin[i] + (m.dG[i][0] * lo0 + m.dG[i][1] * lo1);
        b.h[i] = m.origin[i] + (m.dG[i][0] * hi0 + m.dG[i][1] * hi1);
    }
    return b;
}

__device__ __forceinline__ Box box_scale(Box b, double s) {
    if (s >= 0.0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) { b.l[i] *= s; b.h[i] *= s; }
    } else {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const double t = b.l[i];
            b.l[i] = b.h[i] * s;
            b.h[i] = t * s;
        }
    }
    return b;
}

template <int L>
__global__ void __launch_bounds__(256) k_enumerate(EnumArgs a, int64_t item0, int64_t count, uint32_t* counts,
                                                   const uint32_t* offsets, int32_t* out, int64_t stride,
                                                   int64_t base, unsigned long long* diag) {
    extern __shared__ double s_mc[];
    const ChanDev& c = a.c;
    constexpr int R = 2 * (L - 2) + 1;
    for (int i = threadIdx.x; i < c.nmc * R; i += blockDim.x) s_mc[i] = a.mc_pre[i];
    __syncthreads();
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t n_pre = 0, n_det = 0, n_surv = 0;
    if (t < count) {
        const int64_t item = item0 + t;
        constexpr int C = 1 << (L - 1);
        const int comb = int(item % C);
        int64_t r = item / C;
        int sec[TB_MAX_LEGS] = {0, 0, 0, 0};
#pragma unroll
        for (int l = L - 2; l >= 0; --l) {
            sec[l] = int(r % a.nsec[l]);
            r /= a.nsec[l];
        }
        const int u = int(r);
        // box of the last leg: -dir[L-1] * (sum_l dir[l] * box_l + gVec * u)
        const double ux = c.umk[2 * u], uy = c.umk[2 * u + 1];
        const double gu0 = c.gvec[0] * ux + c.gvec[2] * uy;
        const double gu1 = c.gvec[1] * ux + c.gvec[3] * uy;
        Box acc;
#pragma unroll
        for (int l = 0; l < L - 1; ++l) {
            const EnumLeg& m = a.leg[l];
            Box b = box_scale(section_box(m, sec[l] % m.nx, sec[l] / m.nx), c.leg[l].dir);
            if (l == 0) acc = b;
            else {
#pragma unroll
                for (int i = 0; i < 2; ++i) { acc.l[i] += b.l[i]; acc.h[i] += b.h[i]; }
            }
        }
        acc.l[0] += gu0; acc.h[0] += gu0;
        acc.l[1] += gu1; acc.h[1] += gu1;
        acc = box_scale(acc, -c.leg[L - 1].dir);
        const EnumLeg& ml = a.leg[L - 1];
        int lo[2], hi[2];
        const int ns[2] = {ml.nx, ml.ny};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const double tl = ml.invdG[i][0] * (acc.l[0] - ml.origin[0]) + ml.invdG[i][1] * (acc.l[1] - ml.origin[1]);
            const double th = ml.invdG[i][0] * (acc.h[0] - ml.origin[0]) + ml.invdG[i][1] * (acc.h[1] - ml.origin[1]);
            const int aa = int(floor(tl));
            const int bb = int(floor(th) + 1.0);
            lo[i] = min(max(aa, 0), ns[i]);
            hi[i] = min(max(bb, 0), ns[i]);
        }
        if (lo[0] != hi[0] && lo[1] != hi[1]) {
            int e[L];
            double mn[L], mx[L];
#pragma unroll
            for (int l = 0; l < L - 1; ++l) {
                const int bit = (comb >> (L - 2 - l)) & 1;
                e[l] = 2 * sec[l] + bit;
                const double emin = __ldg(a.leg[l].minE + e[l]), emax = __ldg(a.leg[l].maxE + e[l]);
                mn[l] = (c.leg[l].dir > 0) ? emin : -emax;
                mx[l] = (c.leg[l].dir > 0) ? emax : -emin;
            }
            const double sqrt2 = 1.4142135623730951;  // sqrt(2.0) correctly rounded
            double prodc = 1.0;
#pragma unroll
            for (int l = 0; l < L; ++l) prodc *= sqrt2;
            uint32_t local = 0;
            for (int sy = lo[1]; sy < hi[1]; ++sy)
                for (int sx = lo[0]; sx < hi[0]; ++sx)
                    for (int ie = 0; ie < 2; ++ie) {
                        const int el = 2 * (sx + sy * ml.nx) + ie;
                        e[L - 1] = el;
                        const double emin = __ldg(ml.minE + el), emax = __ldg(ml.maxE + el);
                        mn[L - 1] = (c.leg[L - 1].dir > 0) ? emin : -emax;
                        mx[L - 1] = (c.leg[L - 1].dir > 0) ? emax : -emin;
                        double minE = 0.0, maxE = 0.0;
#pragma unroll
                        for (int k = 0; k < L; ++k) { minE += mn[k]; maxE += mx[k]; }
                        if (!((minE <= 0.0) && (maxE >= 0.0))) continue;
                        ++n_pre;
                        TupleGeom<L> g;
                        tuple_geometry<L>(c, e, u, g);
                        if (!(fabs(g.det) >= c.min_det)) continue;
                        ++n_det;
                        double Ci[3][3];
                        dc_inverse<L>(g, Ci);
                        double sum = 0.0;
                        double p[L][2];
                        for (int m = 0; m < c.nmc; ++m) {
                            const bool th = mc_point_exact<L>(g, Ci, s_mc + m * R, p);
                            sum += th ? prodc : 0.0;
                        }
                        double res = (1.0 / (c.fact * double(c.nmc) * fabs(g.det))) * sum;
                        res *= c.amp_vol;
                        if (!(fabs(res) > c.threshold)) continue;
                        if (offsets) {
                            const int64_t pos = base + (int64_t)offsets[t] + local;
#pragma unroll
                            for (int l = 0; l < L; ++l) out[l * stride + pos] = e[l];
                            out[L * stride + pos] = u;
                        }
                        ++local;
                    }
            n_surv = local;
        }
        if (counts) counts[t] = n_surv;
    }
    if (diag && !offsets) {
        unsigned long long v0 = n_pre, v1 = n_det, v2 = n_surv;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v0 += __shfl_down_sync(0xffffffffu, v0, o);
            v1 += __shfl_down_sync(0xffffffffu, v1, o);
            v2 += __shfl_down_sync(0xffffffffu, v2, o);
        }
        if ((threadIdx.x & 31) == 0 && (v0 | v1 | v2)) {
            atomicAdd(diag + 0, v0);
            atomicAdd(diag + 1, v1);
            atomicAdd(diag + 2, v2);
        }
    }
}

constexpr int EW_WARPS = 8;

// bits[item - item0]: bit k set when candidate k of the item's box survives;
// diag += candidates inside the energy window, with a valid determinant;
// *overflow is set when a box holds more than 64 candidates.
template <int L>
__global__ void __launch_bounds__(EW_WARPS * 32, 2) k_enum_walk(ChanDev c, StreamDev sd, int64_t item0, int64_t count, int span,
                                                                unsigned long long* __restrict__ bits,
                                                                unsigned long long* __restrict__ diag,
                                                                int* __restrict__ overflow) {
    constexpr int R = 2 * (L - 2) + 1;
    extern __shared__ __align__(16) double s_pre[];   // the table, then its FP32 copy
    // per-warp queues: [0] inside the energy window, [1] with a
    // valid determinant and points that may be inside.  Row L: the umklapp column, row L + 1: the
    // item (relative) and the candidate's bit
    __shared__ int32_t s_q[2][EW_WARPS][L + 2][ST_QUEUE];
    __shared__ uint64_t s_may[EW_WARPS][ST_QUEUE];   // queue 1: points that may be inside
    __shared__ double s_cnt[65];   // prodc added k times to 0.0, in sequence
    float* s_fl = reinterpret_cast<float*>(s_pre + (c.nmc * R + 1) / 2 * 2);
    for (int i = threadIdx.x; i < c.nmc * R; i += blockDim.x) {
        s_pre[i] = sd.mc_pre[i];
        s_fl[i / R * FloatTable<L>::FT + i % R] = float_point(sd, sd.mc_pre[i]);   // not wide: in_domain
    }
    if (threadIdx.x == 0) {
        const double sqrt2 = 1.4142135623730951;   // sqrt(2.0) correctly rounded
        double prodc = 1.0, t = 0.0;
        for (int l = 0; l < L; ++l) prodc *= sqrt2;
        s_cnt[0] = t;
        for (int k = 1; k <= 64; ++k) s_cnt[k] = (t += prodc);
    }
    __syncthreads();
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long n_pre = 0, n_det = 0;
    int q1n = 0;   // candidates in queue 1 (warp-uniform)

    auto take = [&](int q, int first, int n, int (&e)[L], int& u, int& code) {
        const bool valid = lane < n;
#pragma unroll
        for (int l = 0; l < L; ++l) e[l] = valid ? s_q[q][warp][l][first + lane] : 0;
        u = valid ? s_q[q][warp][L][first + lane] : 0;
        code = valid ? s_q[q][warp][L + 1][first + lane] : 0;
        return valid;
    };
    auto filter = [&](int first, int n) {
        int e[L], u, code;
        const bool valid = take(0, first, n, e, u, code);
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
            may = maybe_inside<L>(am, T, s_fl, c.nmc);
            ok = may != 0ull || c.threshold < 0.0;
        }
        const unsigned bal = __ballot_sync(full, ok);
        if (ok) {
            const int pos = q1n + __popc(bal & ((1u << lane) - 1u));
#pragma unroll
            for (int l = 0; l < L; ++l) s_q[1][warp][l][pos] = e[l];
            s_q[1][warp][L][pos] = u;
            s_q[1][warp][L + 1][pos] = code;
            s_may[warp][pos] = may;
        }
        q1n += __popc(bal);
        __syncwarp();
    };
    auto survive = [&](int first, int n) {
        int e[L], u, code;
        const bool valid = take(1, first, n, e, u, code);
        TupleGeom<L> g;
        tuple_geometry<L>(c, e, u, g);
        const double adet = fabs(g.det);
        double Ci[3][3];
        dc_inverse<L>(g, Ci);
        AlphaMap<L> am;
        alpha_map<L>(g, Ci, am);
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
        if (valid && (adet >= c.min_det) && (fabs(res) > c.threshold)) atomicOr(bits + (code >> 6), 1ull << (code & 63));
        __syncwarp();
    };

    int qn = 0;   // queued candidates (warp-uniform)
    const int64_t n_warps = int64_t(gridDim.x) * EW_WARPS;
    const int64_t run = int64_t(span) * 32;
    const WalkLeg& ml = sd.leg[L - 1];
    const int64_t it1 = item0 + count;
    for (int64_t rb = item0 + (int64_t(blockIdx.x) * EW_WARPS + warp) * run; rb < it1; rb += n_warps * run) {
        WalkPos<L> p;
        walk_decode<L>(sd, rb + lane, p);
        WalkFront fr;
        bool front_ok = false;
        for (int st = 0; st < span; ++st) {
            const int64_t base = rb + int64_t(st) * 32;
            if (base >= it1) break;
            const int64_t item = base + lane;
            int e[L];
            int lo[2] = {0, 0}, hi[2] = {0, 0};
            double pmn = 0.0, pmx = 0.0;
            int ncand = 0;
            if (item < it1) {
                walk_at<L>(c, sd, p, fr, front_ok, e, lo, hi, pmn, pmx);
                if (lo[0] != hi[0] && lo[1] != hi[1]) ncand = 2 * (hi[0] - lo[0]) * (hi[1] - lo[1]);
            }
            if (ncand > 64) {
                *overflow = 1;
                ncand = 0;
            }
            const int maxc = __reduce_max_sync(full, unsigned(ncand));
            int cx = lo[0], cy = lo[1];
            for (int k = 0; k < maxc; ++k) {
                const int ie = k & 1;
                bool pass = false;
                int el = 0;
                if (k < ncand) {
                    el = 2 * (cx + cy * ml.nx) + ie;
                    const double emin = __ldg(ml.minE + el), emax = __ldg(ml.maxE + el);
                    const double minE = pmn + ((c.leg[L - 1].dir > 0) ? emin : -emax);
                    const double maxE = pmx + ((c.leg[L - 1].dir > 0) ? emax : -emin);
                    pass = (minE <= 0.0) && (maxE >= 0.0);
                }
                if (ie && ++cx == hi[0]) { cx = lo[0]; ++cy; }
                const unsigned bal = __ballot_sync(full, pass);
                if (pass) {
                    const int pos = qn + __popc(bal & ((1u << lane) - 1u));
#pragma unroll
                    for (int l = 0; l < L - 1; ++l) s_q[0][warp][l][pos] = e[l];
                    s_q[0][warp][L - 1][pos] = el;
                    s_q[0][warp][L][pos] = p.u;
                    s_q[0][warp][L + 1][pos] = int32_t(item - item0) << 6 | k;
                }
                qn += __popc(bal);
                __syncwarp();
                if (qn >= 32) {
                    filter(qn - 32, 32);
                    qn -= 32;
                    if (q1n >= 32) {
                        survive(q1n - 32, 32);
                        q1n -= 32;
                    }
                    __syncwarp();   // the slots are reused
                }
            }
            if (walk_advance<L>(sd, p)) front_ok = false;
        }
    }
    if (qn > 0) filter(0, qn);
    while (q1n > 0) {
        const int t = min(q1n, 32);
        survive(q1n - t, t);
        q1n -= t;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        n_pre += __shfl_down_sync(full, n_pre, o);
        n_det += __shfl_down_sync(full, n_det, o);
    }
    if (lane == 0 && (n_pre | n_det)) {
        atomicAdd(diag + 0, n_pre);
        atomicAdd(diag + 1, n_det);
    }
}

// The surviving candidates of each item at base + offsets[item - item0] on.
template <int L>
__global__ void __launch_bounds__(256) k_enum_write(ChanDev c, StreamDev sd, int64_t item0, int64_t count,
                                                    const unsigned long long* __restrict__ bits,
                                                    const uint32_t* __restrict__ offsets, int32_t* __restrict__ out,
                                                    int64_t stride, int64_t base) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long b = t < count ? bits[t] : 0ull;
    if (!b) return;
    WalkPos<L> p;
    walk_decode<L>(sd, item0 + t, p);
    WalkFront fr;
    bool front_ok = false;
    int e[L], lo[2], hi[2];
    double pmn, pmx;
    walk_at<L>(c, sd, p, fr, front_ok, e, lo, hi, pmn, pmx);
    const int nbx = hi[0] - lo[0];
    for (int64_t pos = base + offsets[t]; b; b &= b - 1, ++pos) {
        const int k = __ffsll((long long)b) - 1, cell = k >> 1;
        e[L - 1] = 2 * (lo[0] + cell % nbx + (lo[1] + cell / nbx) * sd.leg[L - 1].nx) + (k & 1);
#pragma unroll
        for (int l = 0; l < L; ++l) out[l * stride + pos] = e[l];
        out[L * stride + pos] = p.u;
    }
}

struct BitCount {
    __host__ __device__ uint32_t operator()(unsigned long long b) const {
#ifdef __CUDA_ARCH__
        return uint32_t(__popcll((long long)b));
#else
        return uint32_t(__builtin_popcountll(b));
#endif
    }
};

// Free points in the reference triangle, the last coordinate in [0, 1]: what
// outside_thresholds and maybe_inside assume of a table.
static bool in_domain(const double* q, int nmc, int L) {
    const int R = 2 * (L - 2) + 1;
    for (int m = 0; m < nmc; ++m) {
        const double* p = q + size_t(m) * R;
        for (int b = 0; b < L - 2; ++b)
            if (!(p[2 * b] >= 0.0 && p[2 * b + 1] >= 0.0 && p[2 * b] + p[2 * b + 1] <= 1.0)) return false;
        if (!(p[R - 1] >= 0.0 && p[R - 1] <= 1.0)) return false;
    }
    return true;
}

// Host driver: chunked count / scan / write.  Output is SoA with L+1 rows
// (L element-id rows, then the umklapp row) of length `cap`.
int enumerate_channel(const ChanDev& c, const HostMesh* meshes, const HostBand* bands, const int* leg_band,
                      const double* h_mc_pre, const double* d_mc_pre, const double* const* d_minE, const double* const* d_maxE,
                      cudaStream_t stream, DeviceTuples& outT, int64_t diag[3]) {
    const int L = c.L;
    EnumArgs a;
    a.c = c;
    for (int l = 0; l < TB_MAX_LEGS; ++l) a.nsec[l] = 1;
    for (int l = 0; l < L; ++l) {
        const HostMesh& m = meshes[bands[leg_band[l]].mesh];
        EnumLeg& el = a.leg[l];
        el.minE = d_minE[l];
        el.maxE = d_maxE[l];
        el.nx = m.nx;
        el.ny = m.ny;
        for (int i = 0; i < 2; ++i) {
            el.origin[i] = m.origin[i];
            for (int j = 0; j < 2; ++j) { el.dG[i][j] = m.dG[i][j]; el.invdG[i][j] = m.invdG[i][j]; }
        }
        if (l < L - 1) a.nsec[l] = int64_t(m.nx) * m.ny;
    }
    a.mc_pre = d_mc_pre;
    int64_t total = c.n_umk;
    for (int l = 0; l < L - 1; ++l) total *= a.nsec[l];
    total *= (int64_t(1) << (L - 1));

    const int64_t CH = int64_t(1) << 24;
    const int64_t chunk = total < CH ? total : CH;
    uint32_t *d_counts = nullptr, *d_offsets = nullptr;
    unsigned long long *d_diag = nullptr, *bits = nullptr;
    void* d_tmp = nullptr;
    char* base = nullptr;
    size_t tmp_bytes = 0, scan_bytes = 0;
    int rc = TB_OK;
    auto fail = [&](int code, const char* what) {
        set_error(std::string("enumerate: ") + what);
        rc = code;
    };
    // one allocation: a 64-bit word per item (the walk's bits; the other pass
    // keeps its counts there), the walk's overflow flag, the totals, the offsets
    // and the scan's scratch
    const size_t items = size_t(chunk > 0 ? chunk : 1);
    cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, d_counts, d_offsets, int(items), stream);
    {
        cub::TransformInputIterator<uint32_t, BitCount, const unsigned long long*> p0(bits, BitCount{});
        cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, p0, d_offsets, int(items), stream);
    }
    tmp_bytes = std::max(tmp_bytes, scan_bytes);
    const size_t offs = sizeof(unsigned long long) * (items + 4), tmps = (offs + sizeof(uint32_t) * items + 255) / 256 * 256;
    if (cudaMalloc(&base, tmps + tmp_bytes) != cudaSuccess) {
        fail(TB_ERR_OOM, "scratch allocation failed");
    } else {
        bits = reinterpret_cast<unsigned long long*>(base);
        d_counts = reinterpret_cast<uint32_t*>(base);
        d_diag = bits + items + 1;
        d_offsets = reinterpret_cast<uint32_t*>(base + offs);
        d_tmp = base + tmps;
    }
    if (rc == TB_OK) cudaMemsetAsync(d_diag, 0, sizeof(unsigned long long) * 3, stream);
    const size_t smem = sizeof(double) * size_t(c.nmc) * c.R;
    int64_t n = 0;
    if (outT.cap == 0 && rc == TB_OK) rc = outT.reserve(L, int64_t(1) << 20, stream);
    // room for `add` more tuples behind the first n
    auto room = [&](uint64_t add) {
        int64_t want = outT.cap;
        while (want < n + int64_t(add)) want *= 2;
        return want > outT.cap ? outT.grow(L, want, n, stream) : int(TB_OK);
    };
    bool walked = false;
    if (rc == TB_OK && c.nmc <= 64 && in_domain(h_mc_pre, c.nmc, L)) {
        StreamDev sd{};
        for (int l = 0; l < L; ++l) {
            const EnumLeg& el = a.leg[l];
            WalkLeg& w = sd.leg[l];
            w.minE = el.minE;
            w.maxE = el.maxE;
            w.nx = el.nx;
            w.ny = el.ny;
            for (int i = 0; i < 2; ++i) {
                w.origin[i] = el.origin[i];
                for (int j = 0; j < 2; ++j) { w.dG[i][j] = el.dG[i][j]; w.invdG[i][j] = el.invdG[i][j]; }
            }
        }
        for (int l = 0; l < TB_MAX_LEGS; ++l) sd.nsec[l] = a.nsec[l];
        sd.n_items = total;
        sd.mc_pre = d_mc_pre;
        int overflow = 0;
        walked = true;
        cub::TransformInputIterator<uint32_t, BitCount, const unsigned long long*> pops(bits, BitCount{});
        cudaMemsetAsync(bits + items, 0, sizeof(unsigned long long), stream);
        int* d_over = reinterpret_cast<int*>(bits + items);
        for (int64_t s = 0; s < total && walked && rc == TB_OK && !overflow; s += chunk) {
            const int64_t cnt = (total - s) < chunk ? (total - s) : chunk;
            // shorter runs of items where there are few: a warp's run is serial (8x8 e-ph: 170 us a channel at 16)
            const int span = int(std::max<int64_t>(1, std::min<int64_t>(ST_SPAN, cnt / (32 * 148 * 2 * EW_WARPS))));
            const int64_t runs = (cnt + span * 32 - 1) / (span * 32);
            const unsigned grid = unsigned(std::min<int64_t>((runs + EW_WARPS - 1) / EW_WARPS, 148 * 2 * 8));
            const unsigned wgrid = unsigned((cnt + 255) / 256);
            const size_t wsmem = smem + 16 + sizeof(float) * 8 * size_t(c.nmc);
            cudaMemsetAsync(bits, 0, sizeof(unsigned long long) * size_t(cnt), stream);
            switch (L) {
                case 2: k_enum_walk<2><<<grid, EW_WARPS * 32, wsmem, stream>>>(c, sd, s, cnt, span, bits, d_diag, d_over); break;
                case 3: k_enum_walk<3><<<grid, EW_WARPS * 32, wsmem, stream>>>(c, sd, s, cnt, span, bits, d_diag, d_over); break;
                default: k_enum_walk<4><<<grid, EW_WARPS * 32, wsmem, stream>>>(c, sd, s, cnt, span, bits, d_diag, d_over); break;
            }
            if (cudaGetLastError() != cudaSuccess) { fail(TB_ERR_CUDA, "walk launch failed"); break; }
            cub::DeviceScan::ExclusiveSum(d_tmp, tmp_bytes, pops, d_offsets, int(cnt), stream);
            uint32_t last = 0;
            unsigned long long last_bits = 0;
            cudaMemcpyAsync(&last, d_offsets + cnt - 1, sizeof(last), cudaMemcpyDeviceToHost, stream);
            cudaMemcpyAsync(&last_bits, bits + cnt - 1, sizeof(last_bits), cudaMemcpyDeviceToHost, stream);
            cudaMemcpyAsync(&overflow, d_over, sizeof(overflow), cudaMemcpyDeviceToHost, stream);
            if (cudaStreamSynchronize(stream) != cudaSuccess) { fail(TB_ERR_CUDA, "count pass failed"); break; }
            const uint64_t add = uint64_t(last) + BitCount{}(last_bits);
            if (overflow || add == 0) continue;
            if (add >= (uint64_t(1) << 31)) { fail(TB_ERR_CAPACITY, "more than 2^31 survivors in one chunk"); break; }
            rc = room(add);
            if (rc != TB_OK) break;
            switch (L) {
                case 2: k_enum_write<2><<<wgrid, 256, 0, stream>>>(c, sd, s, cnt, bits, d_offsets, outT.d, outT.cap, n); break;
                case 3: k_enum_write<3><<<wgrid, 256, 0, stream>>>(c, sd, s, cnt, bits, d_offsets, outT.d, outT.cap, n); break;
                default: k_enum_write<4><<<wgrid, 256, 0, stream>>>(c, sd, s, cnt, bits, d_offsets, outT.d, outT.cap, n); break;
            }
            if (cudaGetLastError() != cudaSuccess) { fail(TB_ERR_CUDA, "write launch failed"); break; }
            n += int64_t(add);
        }
        if (rc == TB_OK && walked && cudaStreamSynchronize(stream) != cudaSuccess) fail(TB_ERR_CUDA, "write pass failed");
        if (overflow && rc == TB_OK) {   // a box beyond the bits: from the start with the other pass
            walked = false;
            n = 0;
            cudaMemsetAsync(d_diag, 0, sizeof(unsigned long long) * 3, stream);
        }
        if (rc == TB_OK && walked) {
            const unsigned long long ns = (unsigned long long)n;
            cudaMemcpyAsync(d_diag + 2, &ns, sizeof(ns), cudaMemcpyHostToDevice, stream);
            cudaStreamSynchronize(stream);
        }
    }
    for (int64_t s = 0; s < total && rc == TB_OK && !walked; s += chunk) {
        const int64_t cnt = (total - s) < chunk ? (total - s) : chunk;
        const unsigned grid = unsigned((cnt + 255) / 256);
        switch (L) {
            case 2: k_enumerate<2><<<grid, 256, smem, stream>>>(a, s, cnt, d_counts, nullptr, nullptr, 0, 0, d_diag); break;
            case 3: k_enumerate<3><<<grid, 256, smem, stream>>>(a, s, cnt, d_counts, nullptr, nullptr, 0, 0, d_diag); break;
            default: k_enumerate<4><<<grid, 256, smem, stream>>>(a, s, cnt, d_counts, nullptr, nullptr, 0, 0, d_diag); break;
        }
        if (cudaGetLastError() != cudaSuccess) { fail(TB_ERR_CUDA, "count launch failed"); break; }
        cub::DeviceScan::ExclusiveSum(d_tmp, tmp_bytes, d_counts, d_offsets, int(cnt), stream);
        uint32_t last[2];
        cudaMemcpyAsync(&last[0], d_offsets + cnt - 1, sizeof(uint32_t), cudaMemcpyDeviceToHost, stream);
        cudaMemcpyAsync(&last[1], d_counts + cnt - 1, sizeof(uint32_t), cudaMemcpyDeviceToHost, stream);
        if (cudaStreamSynchronize(stream) != cudaSuccess) { fail(TB_ERR_CUDA, "count pass failed"); break; }
        const uint64_t add = uint64_t(last[0]) + uint64_t(last[1]);
        if (add >= (uint64_t(1) << 31)) { fail(TB_ERR_CAPACITY, "more than 2^31 survivors in one chunk"); break; }
        if (add == 0) continue;
        rc = room(add);
        if (rc != TB_OK) break;
        switch (L) {
            case 2: k_enumerate<2><<<grid, 256, smem, stream>>>(a, s, cnt, nullptr, d_offsets, outT.d, outT.cap, n, nullptr); break;
            case 3: k_enumerate<3><<<grid, 256, smem, stream>>>(a, s, cnt, nullptr, d_offsets, outT.d, outT.cap, n, nullptr); break;
            default: k_enumerate<4><<<grid, 256, smem, stream>>>(a, s, cnt, nullptr, d_offsets, outT.d, outT.cap, n, nullptr); break;
        }
        if (cudaGetLastError() != cudaSuccess) { fail(TB_ERR_CUDA, "write launch failed"); break; }
        n += int64_t(add);
    }
    if (rc == TB_OK) {
        unsigned long long h[3];
        cudaMemcpyAsync(h, d_diag, sizeof(h), cudaMemcpyDeviceToHost, stream);
        if (cudaStreamSynchronize(stream) != cudaSuccess) fail(TB_ERR_CUDA, "enumeration failed");
        diag[0] = int64_t(h[0]); diag[1] = int64_t(h[1]); diag[2] = int64_t(h[2]);
        outT.n = n;
    }
    cudaFree(base);
    return rc;
}

int DeviceTuples::reserve(int L, int64_t cap_, cudaStream_t stream) {
    release();
    if (cudaMalloc(&d, sizeof(int32_t) * size_t(L + 1) * size_t(cap_)) != cudaSuccess) {
        d = nullptr;
        set_error("tuple list allocation failed");
        return TB_ERR_OOM;
    }
    cap = cap_;
    n = 0;
    return TB_OK;
}

int DeviceTuples::grow(int L, int64_t cap_, int64_t keep, cudaStream_t stream) {
    int32_t* nd = nullptr;
    if (cudaMalloc(&nd, sizeof(int32_t) * size_t(L + 1) * size_t(cap_)) != cudaSuccess) {
        set_error("tuple list allocation failed while growing");
        return TB_ERR_OOM;
    }
    for (int r = 0; r <= L; ++r)
        if (keep > 0)
            cudaMemcpyAsync(nd + size_t(r) * cap_, d + size_t(r) * cap, sizeof(int32_t) * size_t(keep),
                            cudaMemcpyDeviceToDevice, stream);
    cudaStreamSynchronize(stream);
    cudaFree(d);
    d = nd;
    cap = cap_;
    return TB_OK;
}

void DeviceTuples::release() {
    if (d) cudaFree(d);
    d = nullptr;
    cap = 0;
    n = 0;
}

}  // namespace tb
