// tb_rows.cu -- the collision operator over packed rows of tuples.
//
// In scatteringIntegrationTypeB (include/Physics/Scattering/IntegratorCore.hpp:
// 260-357) a tuple contributes through its Monte-Carlo points inside the
// simplices only (tb_theta.cu), and everything but the legs' f is fixed for the
// life of a handle.  A row keeps, for 32 tuples that share their leg-0 element,
// the affine map of the constrained coordinates, the weight and the mask of
// points inside, so an evaluation reads 120 bytes per three-leg tuple (172 with
// four legs), in whole lines, instead of the 864 bytes of its moments or the
// element tables of three legs.
//
//   * One warp takes consecutive rows, one lane per tuple.  Rows of one leg-0
//     element follow one another and their tuples are sorted by point count,
//     so the lanes of a warp run nearly the same number of points, and leg 0's
//     three sums stay in registers until the element changes.
//   * A point's coordinates q are read from a shared-memory table that holds
//     16 copies side by side, one per lane of a half warp: the lanes visit
//     different points, and with one copy their 64-bit reads would collide.
//   * The legs' linear forms and the test functions are affine in q, so the
//     tuple's map is folded into the forms' coefficients once and the loop over
//     the points accumulates 1 + R sums (of the integrand times 1 and q);
//     the constrained legs' moments follow from those after the loop.
//   * A warp's rows come by bulk copies into its own shared-memory stages, one
//     row ahead.
//   * Legs 1 and 2 are staged in shared memory and added by consecutive lanes,
//     so the three adds of an element fall into one or two sectors (added lane
//     by lane they bound the kernel: 587 against 336 us at 64x64 e-ph).
//   * All channels of a handle run in one launch; blocks are dealt out by cost.
//
// Measured (64x64 two-band e-ph, 8.7 M tuples, 50 M points, whole right-hand
// side): 306-328 us against 1516-1596 us through the FP64 moment tensor; three bands and
// two phonons at 72x56: 640 against 3128 us; the rates of every leg at 40x24
// with umklapp: 178 against 1792 us; 16x16 e-e (40.8 M tuples of 172 bytes, 156 M
// points): 1.56 ms against 3.58 ms of the list kernel (k_collision_mc), of which
// the adds take 0.2 and the reads could take 1.07 at the copy rate; an 8x8 e-e
// integration 21 against 32 ms.  The 64x64 kernel reads 3.4 TB/s and issues half
// of the time, with 27 % of the FP64 pipe: fixed-latency dependencies of the
// 16 warps on an SM bound it, then the shared-memory pipe (65 %).
//
// The deterministic mode keeps the arithmetic of the streamed and list kernels
// (tb_mcpoint.cuh), operation for operation, and adds exactly (tb_exact.cuh);
// there leg 0's sums are kept as exact integers in registers.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <memory>
#include <utility>

#include "tb_bulk.cuh"
#include "tb_dp45.cuh"
#include "tb_drift.cuh"
#include "tb_geom.cuh"
#include "tb_rows.cuh"

namespace tb {

// Shares of rows that a block takes, one per warp.  16 warps leave 128 registers
// a thread, which the three-leg propagation and its exact variant fit; 20 spill
// (a 64x64 e-ph right-hand side: 421 us against 336), 12 hide less latency
// (350).  Four legs need 168 registers and 11 KB of stages a warp: 12 warps.
__host__ __device__ constexpr int row_shares(int L) { return L == 4 ? 12 : 16; }
// What a launch computes: the collision terms, scattering rates, or the
// transposed operator.
enum { ROW_PROPAGATE = 0, ROW_RATE = 1, ROW_VJP = 2 };
// Warps of a block: the rates and the transpose accumulate sums for every leg
// and take fewer (rates: 184 us against 210 with 16 at 40x24 e-ph with umklapp).
__host__ __device__ constexpr int row_shares_few(int L) { return L == 4 ? 8 : 12; }
template <int L, int MODE> struct RowCap {
    static constexpr bool FEW = MODE != ROW_PROPAGATE;
    static constexpr int W = FEW ? row_shares_few(L) : row_shares(L);
};
constexpr int ROW_STAGES = 2;    // rows of a warp in shared memory
constexpr int ROW_COPIES = 16;   // copies of the point table, one per lane of a half warp

// row_form of {fermion in, fermion out}, {fermion in, boson in, fermion out} and
// {two fermions in, two fermions out}
constexpr int FORM_2 = 0x01, FORM_3 = 0x23, FORM_4 = 0x03;

int row_form(const ChanDev& c) {
    int d = 0;
    for (int l = 0; l < c.L; ++l) d |= (c.leg[l].dir > 0.0 ? 1 << l : 0) | (c.leg[l].stat > 0.0 ? 16 << l : 0);
    return d;
}

template <int L>
struct RowDim {
    static constexpr int R = 2 * (L - 2) + 1;
    static constexpr int ND = 3 * (R + 1) + 1;   // doubles per tuple: a0, G, w
    static constexpr int BYTES = 32 * (8 * ND + 8 + 4 * (L - 1));
};

size_t row_bytes(int L) { return L == 2 ? RowDim<2>::BYTES : L == 3 ? RowDim<3>::BYTES : RowDim<4>::BYTES; }

void PointRows::release() {
    if (blk) cudaFree(blk);   // the allocation's base: rows, perm, row_e0
    blk = nullptr;
    row_e0 = nullptr;
    perm = nullptr;
    nrows = n = points = bytes = 0;
    cost.clear();
    run_cost.clear();
}

void RowSet::release() {
    if (d_chan) cudaFree(d_chan);   // the allocation's base: channels, work, bounds
    d_chan = nullptr;
    d_work = nullptr;
    d_bounds[0] = d_bounds[1] = nullptr;
    nblocks = 0;
}

// ------------------------------------------------------------------ build
// first[e] = the first tuple whose leg-0 element is e or above (e0 ascending)
__global__ void k_rows_first(const int32_t* __restrict__ e0, int64_t n, int ne, int64_t* __restrict__ first) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e > ne) return;
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t m = (lo + hi) / 2;
        if (e0[m] < e) lo = m + 1;
        else hi = m;
    }
    first[e] = lo;
}

// The lanes of an element's last row that hold no tuple: no points, element 0.
template <int L>
__global__ void __launch_bounds__(256) k_rows_pad(const int64_t* __restrict__ first, const int64_t* __restrict__ row0,
                                                  int ne, unsigned char* __restrict__ blk, int32_t* __restrict__ perm) {
    constexpr int ND = RowDim<L>::ND;
    const int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (e >= ne) return;
    const int64_t count = first[e + 1] - first[e];
    if (count % 32 == 0 || lane < count % 32) return;
    const int64_t row = row0[e] + count / 32;
    unsigned char* b = blk + row * RowDim<L>::BYTES;
    for (int k = 0; k < ND; ++k) reinterpret_cast<double*>(b)[32 * k + lane] = 0.0;
    reinterpret_cast<uint64_t*>(b + 256 * ND)[lane] = 0ull;
    for (int l = 1; l < L; ++l) reinterpret_cast<int32_t*>(b + 256 * (ND + 1))[32 * (l - 1) + lane] = 0;
    perm[row * 32 + lane] = -1;
}

// Tuple j of the sorted list goes to lane (j - first[e0]) % 32 of row
// row0[e0] + (j - first[e0]) / 32.
template <int L>
__global__ void __launch_bounds__(256) k_rows_fill(ChanDev c, const int32_t* __restrict__ ids,
                                                   const uint64_t* __restrict__ mask, const int32_t* __restrict__ perm,
                                                   int64_t n, const int64_t* __restrict__ first,
                                                   const int64_t* __restrict__ row0, unsigned char* __restrict__ blk,
                                                   int32_t* __restrict__ row_e0, int32_t* __restrict__ row_perm,
                                                   int32_t* __restrict__ row_pts) {
    constexpr int R = RowDim<L>::R, ND = RowDim<L>::ND;
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
        int e[L];
#pragma unroll
        for (int l = 0; l < L; ++l) e[l] = ids[l * n + j];
        const int u = ids[L * n + j];
        TupleGeom<L> g;
        tuple_geometry<L>(c, e, u, g);
        double Ci[3][3];
        dc_inverse<L>(g, Ci);
        AlphaMap<L> am;
        alpha_map<L>(g, Ci, am);
        const int64_t k = j - first[e[0]];
        const int64_t row = row0[e[0]] + k / 32;
        const int lane = int(k % 32);
        unsigned char* b = blk + row * RowDim<L>::BYTES;
        double* d = reinterpret_cast<double*>(b) + lane;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            d[32 * r] = am.a0[r];
#pragma unroll
            for (int q = 0; q < R; ++q) d[32 * (3 + r * R + q)] = am.G[r][q];
        }
        d[32 * (ND - 1)] = 1.0 / (c.fact * double(c.nmc) * fabs(g.det));
        reinterpret_cast<uint64_t*>(b + 256 * ND)[lane] = mask[j];
        int32_t* ei = reinterpret_cast<int32_t*>(b + 256 * (ND + 1));
#pragma unroll
        for (int l = 1; l < L; ++l) ei[32 * (l - 1) + lane] = e[l];
        row_perm[row * 32 + lane] = perm[j];
        atomicMax(row_pts + 2 * row, __popcll(mask[j]));
        atomicAdd(row_pts + 2 * row + 1, 7 + __popcll(mask[j]));
        if (lane == 0) row_e0[row] = e[0];
    }
}

int build_rows(const ChanDev& c, const ThetaList& th, PointRows& rows, int64_t max_bytes, cudaStream_t s) {
    rows.release();
    const int64_t n = th.n;
    if (n <= 0) return TB_OK;
    const int ne = c.leg[0].ne;
    // an element's tuples fill (count + 31) / 32 rows
    const int64_t most = n / 32 + ne + 1;
    const size_t elem = sizeof(int64_t) * size_t(ne + 1);
    char* base = nullptr;
    if (cudaMalloc(&base, 2 * elem + 2 * sizeof(int32_t) * size_t(most)) != cudaSuccess) {
        cudaGetLastError();
        return TB_OK;
    }
    std::unique_ptr<char, cudaError_t (*)(char*)> tmp(base, [](char* p) { return cudaFree(p); });
    int64_t* d_first = reinterpret_cast<int64_t*>(base);
    int64_t* d_row0 = reinterpret_cast<int64_t*>(base + elem);
    int32_t* d_pts = reinterpret_cast<int32_t*>(base + 2 * elem);
    const unsigned blocks = unsigned(std::min<int64_t>((n + 255) / 256, 148 * 16));
    k_rows_first<<<unsigned(ne / 256 + 1), 256, 0, s>>>(th.ids, n, ne, d_first);
    TB_CUDA(cudaGetLastError());
    std::vector<int64_t> first(size_t(ne) + 1, 0), row0(size_t(ne) + 1, 0);
    TB_CUDA(cudaMemcpyAsync(first.data(), d_first, elem, cudaMemcpyDeviceToHost, s));
    TB_CUDA(cudaStreamSynchronize(s));
    for (size_t e = 0; e < size_t(ne); ++e) row0[e + 1] = row0[e] + (first[e + 1] - first[e] + 31) / 32;
    const int64_t nrows = row0[size_t(ne)];
    const size_t bytes = row_bytes(c.L) * size_t(nrows), words = 33 * sizeof(int32_t) * size_t(nrows);
    if (int64_t(bytes + words) > max_bytes || cudaMalloc(&rows.blk, bytes + words) != cudaSuccess) {
        cudaGetLastError();
        rows.blk = nullptr;
        return TB_OK;
    }
    rows.perm = reinterpret_cast<int32_t*>(rows.blk + bytes);
    rows.row_e0 = rows.perm + 32 * nrows;
    TB_CUDA(cudaMemsetAsync(d_pts, 0, 2 * sizeof(int32_t) * size_t(nrows), s));
    TB_CUDA(cudaMemcpyAsync(d_row0, row0.data(), elem, cudaMemcpyHostToDevice, s));
#define TB_FILL(LL)                                                                                                    \
    k_rows_pad<LL><<<unsigned((int64_t(ne) * 32 + 255) / 256), 256, 0, s>>>(d_first, d_row0, ne, rows.blk, rows.perm); \
    k_rows_fill<LL><<<blocks, 256, 0, s>>>(c, th.ids, th.mask, th.perm, n, d_first, d_row0, rows.blk, rows.row_e0,     \
                                           rows.perm, d_pts)
    switch (c.L) {
        case 2: TB_FILL(2); break;
        case 3: TB_FILL(3); break;
        default: TB_FILL(4); break;
    }
#undef TB_FILL
    TB_CUDA(cudaGetLastError());
    std::vector<int32_t> pts(2 * size_t(nrows), 0);
    TB_CUDA(cudaMemcpyAsync(pts.data(), d_pts, sizeof(int32_t) * pts.size(), cudaMemcpyDeviceToHost, s));
    TB_CUDA(cudaStreamSynchronize(s));
    // a row costs its longest lane beside a fixed part; run-minor, its tuples
    // one after another
    rows.cost.assign(size_t(nrows) + 1, 0);
    rows.run_cost.assign(size_t(nrows) + 1, 0);
    for (size_t r = 0; r < size_t(nrows); ++r) {
        rows.cost[r + 1] = rows.cost[r] + 8 + pts[2 * r];
        rows.run_cost[r + 1] = rows.run_cost[r] + pts[2 * r + 1];
    }
    rows.nrows = nrows;
    rows.bytes = int64_t(bytes + words);
    rows.n = n;
    rows.points = th.points;
    return TB_OK;
}

// ----------------------------------------------------------------- prepare
__global__ void __launch_bounds__(256) k_rows_prepare(ElemDev ed, const double* __restrict__ f, double4* __restrict__ f4,
                                                      const double* __restrict__ u, double4* __restrict__ u4,
                                                      int* __restrict__ nf, double* __restrict__ drift_acc,
                                                      const DPCtl* __restrict__ ctl) {
    const int band = ed.blk_band[blockIdx.x];
    const BandDev& bd = ed.bands[band];
    bool bad = false;
    const int e = (blockIdx.x - ed.blk_first[band]) * blockDim.x + threadIdx.x;
    auto pad = [&](const double* src, double4* dst) {
        const int64_t o = bd.off + 3 * (int64_t)e;
        const double x = src[o], y = src[o + 1], z = src[o + 2];
        dst[bd.off / 3 + e] = make_double4(x, y, z, 0.0);
        bad = bad || !(isfinite(x) && isfinite(y) && isfinite(z));
    };
    if (e < bd.ne && !(ctl && ctl[ed.band_run[band]].done)) {
        pad(f, f4);
        if (u) pad(u, u4);
        if (drift_acc && (bd.vel[0] != 0.0 || bd.vel[1] != 0.0)) drift_element(bd, f, e, drift_acc);
    }
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0) nf[blockIdx.x] = bad ? 1 : 0;
}

int launch_rows_prepare(const ElemDev& ed, const double* f, double4* f4, int* nf, const DPCtl* ctl, cudaStream_t s,
                        const double* u, double4* u4, double* drift_acc) {
    k_rows_prepare<<<ed.nblk, 256, 0, s>>>(ed, f, f4, u, u4, nf, drift_acc, ctl);
    TB_CUDA(cudaGetLastError());
    return TB_OK;
}

// -------------------------------------------------------------- evaluation
// The point table of one lane: entry j of point m at q[(m R + j) ROW_COPIES].
struct RowTable {
    const double* q;
    __device__ __forceinline__ double operator()(int i) const { return q[i * ROW_COPIES]; }
};

// The same with one copy, for lanes that visit the same point.
struct FlatTable {
    const double* q;
    __device__ __forceinline__ double operator()(int i) const { return q[i]; }
};

// One tuple's map, from this lane's column of the staged row.
template <int L>
struct RowMap {
    static constexpr int R = RowDim<L>::R;
    double a0_[3], G_[3][R];
    __device__ __forceinline__ explicit RowMap(const double* d) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            a0_[k] = d[32 * k];
#pragma unroll
            for (int j = 0; j < R; ++j) G_[k][j] = d[32 * (3 + k * R + j)];
        }
    }
    __device__ __forceinline__ double a0(int k) const { return a0_[k]; }
    __device__ __forceinline__ double G(int k, int j) const { return G_[k][j]; }
};

// The same, read from the stage at each use: for lanes that share a tuple a
// read is one broadcast, and the registers go to more warps.
template <int L>
struct StageMap {
    static constexpr int R = RowDim<L>::R;
    const double* d;
    __device__ __forceinline__ double a0(int k) const { return d[32 * k]; }
    __device__ __forceinline__ double G(int k, int j) const { return d[32 * (3 + k * R + j)]; }
};

// The values a tuple adds to its legs' elements: v[l] = (1, x_l, y_l)
// moments of the integrand, scaled.
template <int L>
struct RowOut {
    double v[L][3];
};

// Whether leg l is ingoing, and 1 + s t with its statistics s = +-1: from the
// template's FORM (row_form), or (FORM < 0) from the channel.
template <int FORM>
__device__ __forceinline__ bool leg_in(const RowChan& c, int l) {
    return FORM >= 0 ? ((FORM >> l) & 1) != 0 : c.leg[l].dir > 0.0;
}
template <int FORM>
__device__ __forceinline__ double leg_stat(const RowChan& c, int l) {
    return FORM >= 0 ? (((FORM >> (4 + l)) & 1) ? 1.0 : -1.0) : c.leg[l].stat;
}

// The legs' linear forms as affine functions of q.  Free leg l < L - 2 lies
// at (q[2l], q[2l+1]), leg L - 2 at (q[R-1], al0), leg L - 1 at (al1, al2)
// with al = a0 + G q (IntegratorCore.hpp:298-320).
template <int L>
struct RowForms {
    static constexpr int R = RowDim<L>::R;
    double fr[L > 2 ? L - 2 : 1][3];   // free legs
    double p0, p[R], c0, c[R];
    template <class Map>
    __device__ __forceinline__ void set(const Map& m, const double4 (&f)[L]) {
#pragma unroll
        for (int l = 0; l < L - 2; ++l) { fr[l][0] = f[l].x; fr[l][1] = f[l].y; fr[l][2] = f[l].z; }
        const double4 P = f[L - 2], C = f[L - 1];
        p0 = fma(P.z, m.a0(0), P.x);
        c0 = fma(C.z, m.a0(2), fma(C.y, m.a0(1), C.x));
#pragma unroll
        for (int j = 0; j < R; ++j) {
            p[j] = j == R - 1 ? fma(P.z, m.G(0, j), P.y) : P.z * m.G(0, j);
            c[j] = fma(C.z, m.G(2, j), C.y * m.G(1, j));
        }
    }
    __device__ __forceinline__ void at(const double (&q)[R], double (&t)[L]) const {
#pragma unroll
        for (int l = 0; l < L - 2; ++l) t[l] = fma(fr[l][2], q[2 * l + 1], fma(fr[l][1], q[2 * l], fr[l][0]));
        double a = p0, b = c0;
#pragma unroll
        for (int j = 0; j < R; ++j) { a = fma(p[j], q[j], a); b = fma(c[j], q[j], b); }
        t[L - 2] = a;
        t[L - 1] = b;
    }
};

// Propagation of one tuple: the loss and gain forms of a leg
// (ScatteringChannel.cpp:633-641) are t and 1 + s t (s the statistics), in
// this order for an ingoing leg and swapped for an outgoing one; the loss
// product carries leg 0's minus sign.
template <int L, int FORM, class Map, class Table>
__device__ __forceinline__ void row_tuple(const RowChan& c, const Map& m, uint64_t mk, const double4 (&f)[L],
                                          const Table& tab, double scale, RowOut<L>& o) {
    constexpr int R = RowDim<L>::R;
    RowForms<L> F;
    F.set(m, f);
    double s0 = 0.0, sq[R];
#pragma unroll
    for (int j = 0; j < R; ++j) sq[j] = 0.0;
    double st[L];
#pragma unroll
    for (int l = 0; l < L; ++l) st[l] = leg_stat<FORM>(c, l);
    auto product = [&](const double (&t)[L]) {
        double pa = 1.0, pb = 1.0;
#pragma unroll
        for (int l = 0; l < L; ++l) {
            const double u = fma(st[l], t[l], 1.0);
            const bool in = leg_in<FORM>(c, l);
            const double a = in ? t[l] : u, b = in ? u : t[l];
            pb = l ? pb * b : b;
            if (l < L - 1) pa = l ? pa * a : a;
            else pb = fma(-pa, a, pb);
        }
        return pb;
    };
    for (; mk; mk &= mk - 1) {
        const int i = (__ffsll((long long)mk) - 1) * R;
        double q[R], t[L];
#pragma unroll
        for (int j = 0; j < R; ++j) q[j] = tab(i + j);
        F.at(q, t);
        const double v = product(t);
        s0 += v;
#pragma unroll
        for (int j = 0; j < R; ++j) sq[j] = fma(q[j], v, sq[j]);
    }
    s0 *= scale;
#pragma unroll
    for (int j = 0; j < R; ++j) sq[j] *= scale;
    double y = m.a0(0) * s0, cx = m.a0(1) * s0, cy = m.a0(2) * s0;
#pragma unroll
    for (int j = 0; j < R; ++j) {
        y = fma(m.G(0, j), sq[j], y);
        cx = fma(m.G(1, j), sq[j], cx);
        cy = fma(m.G(2, j), sq[j], cy);
    }
#pragma unroll
    for (int l = 0; l < L; ++l) {
        const bool in = leg_in<FORM>(c, l);
        const double x = l < L - 2 ? sq[l < L - 2 ? 2 * l : 0] : l == L - 2 ? sq[R - 1] : cx;
        const double z = l < L - 2 ? sq[l < L - 2 ? 2 * l + 1 : 0] : l == L - 2 ? y : cy;
        o.v[l][0] = in ? s0 : -s0;
        o.v[l][1] = in ? x : -x;
        o.v[l][2] = in ? z : -z;
    }
}

// Scattering rates of one tuple: leg r's forms become the unit forms
// (ScatteringChannel.cpp:562-564), for every leg r in one pass over the points.
template <int L, int FORM>
__device__ __forceinline__ void row_tuple_rate(const RowChan& c, const RowMap<L>& m, uint64_t mk,
                                               const double4 (&f)[L], const RowTable& tab, double scale,
                                               RowOut<L>& o) {
    constexpr int R = RowDim<L>::R;
    RowForms<L> F;
    F.set(m, f);
    double s0[L], sq[L][R];
#pragma unroll
    for (int l = 0; l < L; ++l) {
        s0[l] = 0.0;
#pragma unroll
        for (int j = 0; j < R; ++j) sq[l][j] = 0.0;
    }
    double st[L];
#pragma unroll
    for (int l = 0; l < L; ++l) st[l] = leg_stat<FORM>(c, l);
    for (; mk; mk &= mk - 1) {
        const int i = (__ffsll((long long)mk) - 1) * R;
        double q[R], t[L], a[L], b[L];
#pragma unroll
        for (int j = 0; j < R; ++j) q[j] = tab(i + j);
        F.at(q, t);
#pragma unroll
        for (int l = 0; l < L; ++l) {
            const double u = fma(st[l], t[l], 1.0);
            const bool in = leg_in<FORM>(c, l);
            a[l] = in ? t[l] : u;
            b[l] = in ? u : t[l];
        }
#pragma unroll
        for (int r = 0; r < L; ++r) {
            const bool in = leg_in<FORM>(c, r);
            double pa = in ? -2.0 : -2.0 * st[r], pb = in ? 2.0 * st[r] : 2.0;
#pragma unroll
            for (int l = 0; l < L; ++l)
                if (l != r) { pa *= a[l]; pb *= b[l]; }
            const double v = pa + pb;
            s0[r] += v;
#pragma unroll
            for (int j = 0; j < R; ++j)
                if (r >= L - 2 || j / 2 == r) sq[r][j] = fma(q[j], v, sq[r][j]);   // a free leg needs its own two
        }
    }
#pragma unroll
    for (int r = 0; r < L; ++r) {
        double x, z;
        if (r < L - 2) {
            x = sq[r][r < L - 2 ? 2 * r : 0];
            z = sq[r][r < L - 2 ? 2 * r + 1 : 0];
        } else {
            const int y = r == L - 2 ? 0 : 2;
            x = r == L - 2 ? sq[r][R - 1] : m.a0(1) * s0[r];
            z = m.a0(y) * s0[r];
#pragma unroll
            for (int j = 0; j < R; ++j) {
                if (r == L - 1) x = fma(m.G(1, j), sq[r][j], x);
                z = fma(m.G(y, j), sq[r][j], z);
            }
        }
        const double d = leg_in<FORM>(c, r) ? -scale : scale;
        o.v[r][0] = d * s0[r];
        o.v[r][1] = d * x;
        o.v[r][2] = d * z;
    }
}

// The transposed operator of one tuple: the u-weighted test functions of all
// legs are one affine function of q; at every point it multiplies, for each leg,
// the derivative of the gain-minus-loss product with respect to that leg's form.
// Returns the sum of the u-weighted integrand (times the amplitude gradient's
// scale: the caller's).  About 42 FP64 instructions a point with three legs; at
// 24x24 e-ph a transposed evaluation fell from 174 us (k_vjp_mc, four launches,
// nine FP64 atomics a tuple and lane) to 70 with what surrounds it.
template <int L, int FORM>
__device__ __forceinline__ double row_tuple_vjp(const RowChan& c, const RowMap<L>& m, uint64_t mk,
                                                const double4 (&f)[L], const double4 (&u)[L], const RowTable& tab,
                                                double scale, RowOut<L>& o) {
    constexpr int R = RowDim<L>::R;
    RowForms<L> F;
    F.set(m, f);
    double w0 = 0.0, wq[R];
    {
        RowForms<L> U;
        U.set(m, u);
#pragma unroll
        for (int j = 0; j < R; ++j)
            wq[j] = (leg_in<FORM>(c, L - 2) ? U.p[j] : -U.p[j]) + (leg_in<FORM>(c, L - 1) ? U.c[j] : -U.c[j]);
        w0 = (leg_in<FORM>(c, L - 2) ? U.p0 : -U.p0) + (leg_in<FORM>(c, L - 1) ? U.c0 : -U.c0);
#pragma unroll
        for (int l = 0; l < L - 2; ++l) {
            const double d = leg_in<FORM>(c, l) ? 1.0 : -1.0;
            w0 = fma(d, U.fr[l][0], w0);
            wq[2 * l] = fma(d, U.fr[l][1], wq[2 * l]);
            wq[2 * l + 1] = fma(d, U.fr[l][2], wq[2 * l + 1]);
        }
    }
    double s0[L], sq[L][R], total = 0.0;
#pragma unroll
    for (int l = 0; l < L; ++l) {
        s0[l] = 0.0;
#pragma unroll
        for (int j = 0; j < R; ++j) sq[l][j] = 0.0;
    }
    double st[L];
#pragma unroll
    for (int l = 0; l < L; ++l) st[l] = leg_stat<FORM>(c, l);
    for (; mk; mk &= mk - 1) {
        const int i = (__ffsll((long long)mk) - 1) * R;
        double q[R], t[L], a[L], b[L];
#pragma unroll
        for (int j = 0; j < R; ++j) q[j] = tab(i + j);
        F.at(q, t);
        double om = w0;
#pragma unroll
        for (int j = 0; j < R; ++j) om = fma(wq[j], q[j], om);
#pragma unroll
        for (int l = 0; l < L; ++l) {
            const double v = fma(st[l], t[l], 1.0);
            const bool in = leg_in<FORM>(c, l);
            a[l] = in ? t[l] : v;
            b[l] = in ? v : t[l];
        }
#pragma unroll
        for (int r = 0; r < L; ++r) {
            // d / dt_r of (product of b) - (product of a)
            const bool in = leg_in<FORM>(c, r);
            double pa = om, pb = om;
#pragma unroll
            for (int l = 0; l < L; ++l)
                if (l != r) { pa *= a[l]; pb *= b[l]; }
            if (r == L - 1) total = fma(pb, b[r], fma(-pa, a[r], total));
            const double v = in ? fma(st[r], pb, -pa) : fma(-st[r], pa, pb);
            s0[r] += v;
#pragma unroll
            for (int j = 0; j < R; ++j)
                if (r >= L - 2 || j / 2 == r) sq[r][j] = fma(q[j], v, sq[r][j]);   // a free leg needs its own two
        }
    }
#pragma unroll
    for (int r = 0; r < L; ++r) {
        double x, z;
        if (r < L - 2) {
            x = sq[r][r < L - 2 ? 2 * r : 0];
            z = sq[r][r < L - 2 ? 2 * r + 1 : 0];
        } else {
            const int y = r == L - 2 ? 0 : 2;
            x = r == L - 2 ? sq[r][R - 1] : m.a0(1) * s0[r];
            z = m.a0(y) * s0[r];
#pragma unroll
            for (int j = 0; j < R; ++j) {
                if (r == L - 1) x = fma(m.G(1, j), sq[r][j], x);
                z = fma(m.G(y, j), sq[r][j], z);
            }
        }
        o.v[r][0] = scale * s0[r];
        o.v[r][1] = scale * x;
        o.v[r][2] = scale * z;
    }
    return total;
}

// Propagation and rates with the list and streamed kernels' operations in their order
// (inside_point_sums, tb_mcpoint.cuh): the deterministic mode's bits.
template <int L, bool RATE>
__device__ __forceinline__ void row_tuple_listed(const RowChan& c, const RowMap<L>& m, uint64_t mk,
                                                 const double4 (&f)[L], const RowTable& tab, double w, double ampt,
                                                 RowOut<L>& o) {
    constexpr int R = RowDim<L>::R;
    constexpr int NR = RATE ? L : 1;
    double s0[NR], sx[L], sy[L];
#pragma unroll
    for (int r = 0; r < NR; ++r) s0[r] = 0.0;
#pragma unroll
    for (int l = 0; l < L; ++l) { sx[l] = 0.0; sy[l] = 0.0; }
    for (; mk; mk &= mk - 1) {
        const int i = (__ffsll((long long)mk) - 1) * R;
        double q[R], al[3], px[L], py[L], a[L], b[L];
#pragma unroll
        for (int j = 0; j < R; ++j) q[j] = tab(i + j);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            double t = m.a0(r);
#pragma unroll
            for (int j = 0; j < R; ++j) t = fma(m.G(r, j), q[j], t);
            al[r] = t;
        }
#pragma unroll
        for (int l = 0; l < L - 2; ++l) { px[l] = q[2 * l]; py[l] = q[2 * l + 1]; }
        px[L - 2] = q[R - 1]; py[L - 2] = al[0];
        px[L - 1] = al[1]; py[L - 1] = al[2];
#pragma unroll
        for (int l = 0; l < L; ++l) {
            const double t = fma(f[l].z, py[l], fma(f[l].y, px[l], f[l].x));
            a[l] = fma(c.leg[l].fa, t, c.leg[l].fa0);
            b[l] = fma(c.leg[l].fb, t, c.leg[l].fb0);
        }
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            double pa = 1.0, pb = 1.0;
#pragma unroll
            for (int l = 0; l < L; ++l) {
                double x = a[l], y = b[l];
                if (RATE && l == r) {
                    const double d = c.leg[l].dir, s = c.leg[l].stat;
                    x = (l == 0 ? -1.0 : 1.0) * __dadd_rn(__dmul_rn(1. - d, s), 1. + d);
                    y = __dadd_rn(__dmul_rn(1. + d, s), 1. - d);
                }
                pa = __dmul_rn(pa, x);
                pb = __dmul_rn(pb, y);
            }
            const double v = __dadd_rn(pa, pb);
            s0[r] += v;
#pragma unroll
            for (int l = 0; l < L; ++l)
                if (!RATE || l == r) { sx[l] = fma(px[l], v, sx[l]); sy[l] = fma(py[l], v, sy[l]); }
        }
    }
#pragma unroll
    for (int l = 0; l < L; ++l) {
        const double d = RATE ? -c.leg[l].dir : c.leg[l].dir;
        o.v[l][0] = d * ((w * s0[RATE ? l : 0]) * ampt);
        o.v[l][1] = d * ((w * sx[l]) * ampt);
        o.v[l][2] = d * ((w * sy[l]) * ampt);
    }
}

// v on the exact grid, as fx_add takes it; false: nothing to add.
__device__ __forceinline__ bool fx_grid(const FxAcc& a, double v, Fx& x) {
    if (!fx_of(v, x)) {
        if (!isfinite(v) || !a.sat) {
            atomicOr(a.poison, 1u);
            return false;
        }
        atomicOr(a.sat, 1u);
        fx_of(v < 0.0 ? -FX_CLAMP : FX_CLAMP, x);
    }
    return true;
}

// Leg 0's sums of one warp, kept until the element changes.
template <bool DET>
struct LegZero {
    double v[3] = {0.0, 0.0, 0.0};
    __device__ __forceinline__ void add(const double (&x)[3], const FxAcc&) {
#pragma unroll
        for (int j = 0; j < 3; ++j) v[j] += x[j];
    }
    __device__ __forceinline__ void flush(double* acc, int64_t key, const FxAcc&) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int j = 0; j < 3; ++j) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
        const int lane = threadIdx.x & 31;
        if (lane < 3) atomicAdd(acc + key + lane, lane == 0 ? v[0] : lane == 1 ? v[1] : v[2]);
        v[0] = v[1] = v[2] = 0.0;
    }
};

template <>
struct LegZero<true> {
    unsigned long long w[3][3] = {};
    __device__ __forceinline__ void add(const double (&x)[3], const FxAcc& fx) {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            Fx g;
            if (fx_grid(fx, x[j], g)) fx_add_plain(w[j], g);
        }
    }
    __device__ __forceinline__ void flush(double*, int64_t key, const FxAcc& fx) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                Fx g;
                g.w0 = __shfl_xor_sync(0xffffffffu, w[j][0], o);
                g.w1 = __shfl_xor_sync(0xffffffffu, w[j][1], o);
                g.w2 = __shfl_xor_sync(0xffffffffu, w[j][2], o);
                fx_add_plain(w[j], g);
            }
        const int lane = threadIdx.x & 31;
        if (lane < 3) {
            Fx g;
            g.w0 = lane == 0 ? w[0][0] : lane == 1 ? w[1][0] : w[2][0];
            g.w1 = lane == 0 ? w[0][1] : lane == 1 ? w[1][1] : w[2][1];
            g.w2 = lane == 0 ? w[0][2] : lane == 1 ? w[1][2] : w[2][2];
            if (g.w0 | g.w1 | g.w2) fx_atomic_add(fx.w + 3 * (key + lane), g);
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) w[j][0] = w[j][1] = w[j][2] = 0ull;
    }
};

__device__ __forceinline__ bool finite3(const double* v) { return isfinite(v[0]) && isfinite(v[1]) && isfinite(v[2]); }

// A state with non-finite coefficients: the full quadrature multiplies the
// integrand of every tuple by its Theta, also by 0, so each tuple that touches
// such an element makes its legs NaN, also one without a point inside.  Tuples
// [t0, t1) of the whole list.
template <int L>
__device__ __noinline__ void spread_nonfinite(const RowChan& c, const InstDev* insts, int n_insts, int64_t t0,
                                              int64_t t1, const double* f, double* acc, const DPCtl* ctl, bool rate,
                                              int rate_leg, const FxAcc& fx, const double* u = nullptr,
                                              double* gamp = nullptr, unsigned int* gamp_poison = nullptr) {
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    for (int64_t i = t0 + threadIdx.x; i < t1; i += blockDim.x) {
        int e[L];
#pragma unroll
        for (int l = 0; l < L; ++l) e[l] = __ldg(c.tup + l * c.stride + i);
        for (int k = 0; k < n_insts; ++k) {
            const InstDev& in = insts[k];
            if (!u && (in.amp_full == 0.0 || (ctl && ctl[in.run].done))) continue;
            bool bad[L], all = false;
            int nbad = 0;
#pragma unroll
            for (int l = 0; l < L; ++l) {
                bad[l] = !finite3(f + in.foff[l] + 3 * (int64_t)e[l]);
                nbad += bad[l] ? 1 : 0;
                if (u) all = all || !finite3(u + in.foff[l] + 3 * (int64_t)e[l]);
            }
            if (nbad == 0 && !all) continue;
            if (u && gamp_poison) atomicOr(gamp_poison, 1u);
            else if (u) atomicAdd(gamp + k, nan);
#pragma unroll
            for (int l = 0; l < L; ++l) {
                // a leg's rate and derivative do not depend on its own f
                if (rate && rate_leg >= 0 && l != rate_leg) continue;
                if ((rate || u) && !all && nbad == (bad[l] ? 1 : 0)) continue;
                if (fx.w) atomicOr(fx.poison, 1u);
                else
                    for (int j = 0; j < 3; ++j) atomicAdd(acc + in.foff[l] + 3 * (int64_t)e[l] + j, nan);
            }
        }
    }
}

template <int L, int FORM, int MODE, bool DET, bool MULTI>
__global__ void __launch_bounds__(RowCap<L, MODE>::W * 32, 1) k_rows(const RowChan* __restrict__ chans,
                                                            const RowWork* __restrict__ work,
                                                            const int32_t* __restrict__ bounds,
                                                            const InstDev* __restrict__ one,
                                                            const double* __restrict__ f,
                                                            const double4* __restrict__ f4,
                                                            const int* __restrict__ nf, int n_nf,
                                                            double* __restrict__ acc, double* __restrict__ accr,
                                                            int copies, int64_t ndofs, const DPCtl* __restrict__ ctl,
                                                            int rate_leg, FxAcc fx, int* __restrict__ err_flag,
                                                            int wait_polls, const double* __restrict__ u,
                                                            const double4* __restrict__ u4,
                                                            double* __restrict__ gamp) {
    constexpr bool RATE = MODE == ROW_RATE, VJP = MODE == ROW_VJP;
    constexpr int R = RowDim<L>::R, ND = RowDim<L>::ND;
    constexpr uint32_t BYTES = RowDim<L>::BYTES;
    extern __shared__ __align__(128) unsigned char s_raw[];
    __shared__ RowChan c;
    __shared__ __align__(8) uint64_t s_bar[RowCap<L, MODE>::W][ROW_STAGES];
    const RowWork w = work[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_warps = blockDim.x >> 5;
    if (accr && blockIdx.x % copies) acc = accr + int64_t(blockIdx.x % copies - 1) * ndofs;
    for (int i = tid; i < int(sizeof(RowChan) / sizeof(int)); i += blockDim.x)
        reinterpret_cast<int*>(&c)[i] = reinterpret_cast<const int*>(chans + w.chan)[i];
    __syncthreads();
    const InstDev* insts = one ? one : c.insts + (MULTI ? w.i0 : 0);
    const int n_insts = MULTI ? w.i1 - w.i0 : 1;
    if (!VJP) {
        // every instance off or its run finished: nothing to add (an amplitude
        // of 0 still has a gradient)
        bool any = false;
        for (int k = 0; k < n_insts && !any; ++k)
            any = insts[k].amp_full != 0.0 && !(ctl && ctl[insts[k].run].done);
        if (!any) return;
    }
    // this warp's rows, and the copies of its first ones
    bounds += blockIdx.x * (n_warps + 1) + warp;   // one share a warp
    const int r0 = bounds[0], r1 = bounds[1];
    unsigned char* const stage = s_raw + size_t(warp) * ROW_STAGES * BYTES;
    uint64_t* const bar = s_bar[warp];
    auto fetch = [&](int r, int s) {
        mbar_expect_tx_arrive(&bar[s], BYTES);
        bulk_g2s(stage + s * BYTES, c.blk + int64_t(r) * BYTES, BYTES, &bar[s]);
    };
    if (lane == 0) {
        for (int s = 0; s < ROW_STAGES; ++s) mbar_init(&bar[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int s = 0; s < ROW_STAGES; ++s)
            if (r0 + s < r1) fetch(r0 + s, s);
    }
    double* const s_v = reinterpret_cast<double*>(s_raw + size_t(n_warps) * ROW_STAGES * BYTES) + warp * 96 * (L - 1);
    double* const s_q = reinterpret_cast<double*>(s_raw + size_t(n_warps) * (ROW_STAGES * BYTES + 768 * (L - 1)));
    for (int i = tid; i < c.nmc * R * ROW_COPIES; i += blockDim.x) s_q[i] = __ldg(c.mc + i / ROW_COPIES);
    __syncthreads();
    const RowTable tab{s_q + (lane & (ROW_COPIES - 1))};
    LegZero<DET> z;
    int e0 = -1;
    double4 f0 = make_double4(0., 0., 0., 0.), u0 = f0;
    int64_t off[L], el[L];
    double amp = 0.0, ga = 0.0;   // ga: this lane's part of the amplitude gradient
    if (VJP) gamp += c.gamp0 + (MULTI ? w.i0 : 0);
    if (!MULTI) {
#pragma unroll
        for (int l = 0; l < L; ++l) { off[l] = insts[0].foff[l]; el[l] = off[l] / 3; }
        amp = insts[0].amp_full;
    }
    int e0_next = r0 < r1 ? __ldg(c.row_e0 + r0) : 0;   // the next row's leg-0 element
    for (int r = r0; r < r1; ++r) {
        const int used = r - r0;
        const int s = used % ROW_STAGES;
        const int e0_row = e0_next;
        if (r + 1 < r1) e0_next = __ldg(c.row_e0 + r + 1);
        // one verdict for the warp: what follows assumes all of its lanes
        if (!__all_sync(0xffffffffu, mbar_wait(&bar[s], uint32_t(used / ROW_STAGES) & 1u, wait_polls))) {
            // record the failure and give the copies in flight a bounded
            // chance to land before the block releases its shared memory
            if (lane == 0) atomicExch(err_flag, 1);
            for (int k = 0; k < ROW_STAGES && r + k < r1; ++k)
                mbar_wait(&bar[(used + k) % ROW_STAGES], uint32_t((used + k) / ROW_STAGES) & 1u, 1 << 16);
            break;
        }
        const unsigned char* b = stage + s * BYTES;
        const RowMap<L> m(reinterpret_cast<const double*>(b) + lane);
        const uint64_t mk = reinterpret_cast<const uint64_t*>(b + 256 * ND)[lane];
        int e[L];
        e[0] = e0_row;
#pragma unroll
        for (int l = 1; l < L; ++l) e[l] = reinterpret_cast<const int32_t*>(b + 256 * (ND + 1))[32 * (l - 1) + lane];
        double tf = 1.0;
        if (c.tamp && mk) tf = __ldg(c.tamp + __ldg(c.perm + int64_t(r) * 32 + lane));
        const unsigned live = __ballot_sync(0xffffffffu, mk != 0ull);
        if (!MULTI && e[0] != e0) {
            if (e0 >= 0 && (!RATE || rate_leg <= 0)) z.flush(acc, off[0] + 3 * (int64_t)e0, fx);
            e0 = e[0];
            f0 = load_32(f4 + el[0] + e0);
            if (VJP) u0 = load_32(u4 + el[0] + e0);
        }
        for (int k = 0; k < (MULTI ? n_insts : 1); ++k) {
            if (MULTI) {
                const InstDev& in = insts[k];
                amp = in.amp_full;
                if (!VJP && (amp == 0.0 || (ctl && ctl[in.run].done))) continue;
#pragma unroll
                for (int l = 0; l < L; ++l) { off[l] = in.foff[l]; el[l] = off[l] / 3; }
                f0 = load_32(f4 + el[0] + e[0]);
                if (VJP) u0 = load_32(u4 + el[0] + e[0]);
            }
            double4 f[L];
            f[0] = f0;
#pragma unroll
            for (int l = 1; l < L; ++l) f[l] = load_32(f4 + el[l] + e[l]);
            RowOut<L> o;
            const double wt = reinterpret_cast<const double*>(b)[32 * (ND - 1) + lane];
            if constexpr (VJP) {
                double4 u[L];
                u[0] = u0;
#pragma unroll
                for (int l = 1; l < L; ++l) u[l] = load_32(u4 + el[l] + e[l]);
                const double g = row_tuple_vjp<L, FORM>(c, m, mk, f, u, tab, wt * (amp * tf), o);
                ga = fma(wt * (c.amp_vol * tf), g, ga);
                if (MULTI) {
                    for (int d = 16; d > 0; d >>= 1) ga += __shfl_xor_sync(0xffffffffu, ga, d);
                    if (lane == 0 && ga != 0.0) atomicAdd(gamp + k, ga);
                    ga = 0.0;
                }
            } else if (DET) row_tuple_listed<L, RATE>(c, m, mk, f, tab, wt, amp * tf, o);
            else if (RATE) row_tuple_rate<L, FORM>(c, m, mk, f, tab, wt * (amp * tf), o);
            else row_tuple<L, FORM>(c, m, mk, f, tab, wt * (amp * tf), o);
            if (!RATE || rate_leg <= 0) {
                z.add(o.v[0], fx);
                if (MULTI) z.flush(acc, off[0] + 3 * (int64_t)e[0], fx);
            }
            if (DET) {
#pragma unroll
                for (int l = 1; l < L; ++l)
                    if (mk && (!RATE || rate_leg < 0 || rate_leg == l))
                        fx_add3(fx, off[l] + 3 * (int64_t)e[l], o.v[l][0], o.v[l][1], o.v[l][2]);
            } else {
                // entry 96 (l - 1) + 3 t + j: moment j of leg l of lane t's tuple
                __syncwarp();
#pragma unroll
                for (int l = 1; l < L; ++l)
#pragma unroll
                    for (int j = 0; j < 3; ++j) s_v[96 * (l - 1) + 3 * lane + j] = o.v[l][j];
                __syncwarp();
#pragma unroll
                for (int l = 1; l < L; ++l) {
                    if (RATE && rate_leg >= 0 && rate_leg != l) continue;   // uniform
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        const int x = 32 * p + lane, t = x / 3;
                        const int et = __shfl_sync(0xffffffffu, e[l], t);
                        if ((live >> t) & 1u)
                            atomicAdd(acc + off[l] + 3 * (int64_t)et + (x - 3 * t), s_v[96 * (l - 1) + x]);
                    }
                }
            }
        }
        __syncwarp();   // every lane is done with the stage
        if (lane == 0 && r + ROW_STAGES < r1) fetch(r + ROW_STAGES, s);
    }
    if (!MULTI && e0 >= 0 && (!RATE || rate_leg <= 0)) z.flush(acc, off[0] + 3 * (int64_t)e0, fx);
    if (VJP && !MULTI) {
        for (int d = 16; d > 0; d >>= 1) ga += __shfl_xor_sync(0xffffffffu, ga, d);
        if (lane == 0 && ga != 0.0) atomicAdd(gamp, ga);
    }
    int bad = 0;
    for (int i = tid; i < n_nf; i += blockDim.x) bad |= nf[i];
    if (__syncthreads_or(bad))
        spread_nonfinite<L>(c, insts, n_insts, w.t0, w.t1, f, acc, ctl, RATE, rate_leg, fx, VJP ? u : nullptr, gamp);
}

// spread_nonfinite of a transposed evaluation alone, for handles whose
// transpose is evaluated by another kernel.
template <int L>
__global__ void __launch_bounds__(256) k_rows_spread(const RowChan* __restrict__ chans, const RowWork* __restrict__ work,
                                                     const double* __restrict__ f, const int* __restrict__ nf, int n_nf,
                                                     FxAcc fx, const double* __restrict__ u, unsigned int* gamp_poison) {
    int bad = 0;
    for (int i = threadIdx.x; i < n_nf; i += blockDim.x) bad |= nf[i];
    if (!__syncthreads_or(bad)) return;
    const RowWork w = work[blockIdx.x];
    const RowChan& c = chans[w.chan];
    spread_nonfinite<L>(c, c.insts + w.i0, w.i1 - w.i0, w.t0, w.t1, f, nullptr, nullptr, false, -1, fx, u, nullptr,
                        gamp_poison);
}

// acc += the further accumulators, which are cleared.  A latency chain on the
// small meshes that have them: FOLD_LOADS loads of a thread are in flight before
// the first is cleared, and a block's 32 warps cover up to 160 accumulators at
// once (147 of 96 dofs: 7.9 us with 8 warps and one load at a time, 4.4 now; a
// 5x5 e-e right-hand side 32.8 us and 28.7, an 8x8 integration 21.0 ms and 20.6).
constexpr int FOLD_LOADS = 5;
__global__ void __launch_bounds__(1024) k_rows_fold(double* __restrict__ acc, double* __restrict__ accr, int n,
                                                    int64_t ndofs) {
    __shared__ double s[32][33];
    const int64_t d = int64_t(blockIdx.x) * 32 + threadIdx.x;
    double v = 0.0;
    if (d < ndofs)
        for (int k = threadIdx.y; k < n; k += 32 * FOLD_LOADS) {
            double x[FOLD_LOADS];
#pragma unroll
            for (int i = 0; i < FOLD_LOADS; ++i) x[i] = k + 32 * i < n ? accr[(k + 32 * i) * ndofs + d] : 0.0;
#pragma unroll
            for (int i = 0; i < FOLD_LOADS; ++i) {
                v += x[i];
                if (k + 32 * i < n) accr[(k + 32 * i) * ndofs + d] = 0.0;
            }
        }
    s[threadIdx.y][threadIdx.x] = v;
    __syncthreads();
    v = s[threadIdx.x][threadIdx.y];   // warp y: the sums of dof y
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int64_t t = int64_t(blockIdx.x) * 32 + threadIdx.y;
    if (threadIdx.x == 0 && t < ndofs) acc[t] += v;
}

// Accumulators for a set of nblocks blocks: the adds of small meshes fall on so
// few sectors that the L2 serialises them.  Where an element takes more than
// ROW_ADDS of them every block has its own copy, within ROW_COPY_BYTES for all.
// Measured: 16x16 e-e (239,000 adds an element) 6.6 ms with one copy, 1.79 with
// 32, 1.71 with 64, 1.58 with 148; an 8x8 e-e integration (29,000) 165 ms with
// one, 54 with 4, 29 with 16, 23 with 64 and with 148; 64x64 e-ph (900) 324 us
// with one, 335 with 2, 340 with 8.  Around the line, a right-hand side in us with
// one and with a copy a block: e-ph 40x40 with umklapp (1200 adds) 176 / 160, 96x96
// (1500) 941 / 1029, 64x64 with umklapp (1900) 537 / 560; e-e 3x3 (1200) 33 / 29, 4x3
// (2100) 43 / 29, 5x4 (4900) 115 / 27, 6x6 (11,900) 277 / 38; four legs with bosons
// 8x6 (17,000) 263 / 51.
constexpr int64_t ROW_ADDS = 2000, ROW_COPY_BYTES = int64_t(64) << 20;
static int row_copies(int64_t adds_per_element, int nblocks, int64_t ndofs) {
    if (adds_per_element <= ROW_ADDS) return 1;
    return int(std::max<int64_t>(1, std::min<int64_t>(nblocks, ROW_COPY_BYTES / (8 * std::max<int64_t>(ndofs, 1)))));
}

static size_t rows_smem(int L, int nmc, int warps) {
    return size_t(warps) * (ROW_STAGES * row_bytes(L) + 768 * size_t(L - 1)) +
           sizeof(double) * size_t(nmc) * size_t(2 * (L - 2) + 1) * ROW_COPIES;
}

template <int L, int FORM, int MODE, bool DET, bool MULTI>
static int launch_k_rows(const RowSet& rs, const RowArgs& A, cudaStream_t s) {
    auto kern = k_rows<L, FORM, MODE, DET, MULTI>;
    // the shared-memory limit, set once on each device the kernel runs on
    static std::atomic<unsigned long long> attr_devices{0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !((attr_devices.load() >> dev) & 1ull)) {
        TB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     int(rows_smem(L, 64, RowCap<L, MODE>::W))));
        if (dev >= 0 && dev < 64) attr_devices.fetch_or(1ull << dev);
    }
    const int warps = rs.shares[RowCap<L, MODE>::FEW];
    kern<<<unsigned(rs.nblocks), unsigned(32 * warps), rows_smem(L, rs.nmc_max, warps), s>>>(
        rs.d_chan, rs.d_work, rs.d_bounds[RowCap<L, MODE>::FEW], A.one, A.f, A.f4, A.nf, A.ed->nblk, A.acc, A.accr, rs.copies,
        A.ed->ndofs, A.ctl, A.rate_leg, A.fx, A.err_flag, A.polls, A.u, A.u4, A.gamp);
    TB_CUDA(cudaGetLastError());
    if (A.accr && rs.copies > 1) {
        k_rows_fold<<<unsigned((A.ed->ndofs + 31) / 32), dim3(32, 32), 0, s>>>(A.acc, A.accr, rs.copies - 1, A.ed->ndofs);
        TB_CUDA(cudaGetLastError());
    }
    return TB_OK;
}

template <int L, int FORM, int MODE, bool DET>
static int launch_rows_m(const RowSet& rs, const RowArgs& A, cudaStream_t s) {
    if (rs.multi && !A.one) return launch_k_rows<L, FORM, MODE, DET, true>(rs, A, s);
    return launch_k_rows<L, FORM, MODE, DET, false>(rs, A, s);
}

// The channels that addScatteringChannelsWildcards builds in the reference's
// examples are compiled in (FORM_2, FORM_3, FORM_4); others select their forms
// at run time.
template <int L>
static int launch_rows_l(const RowSet& rs, const RowArgs& A, cudaStream_t s) {
    constexpr int CANON = L == 2 ? FORM_2 : L == 3 ? FORM_3 : FORM_4;
    const bool canon = rs.form == CANON;
    if (A.u) return canon ? launch_rows_m<L, CANON, ROW_VJP, false>(rs, A, s) : launch_rows_m<L, -1, ROW_VJP, false>(rs, A, s);
    if (A.fx.w) return A.rate ? launch_rows_m<L, -1, ROW_RATE, true>(rs, A, s) : launch_rows_m<L, -1, ROW_PROPAGATE, true>(rs, A, s);
    if (A.rate) return canon ? launch_rows_m<L, CANON, ROW_RATE, false>(rs, A, s) : launch_rows_m<L, -1, ROW_RATE, false>(rs, A, s);
    return canon ? launch_rows_m<L, CANON, ROW_PROPAGATE, false>(rs, A, s)
                 : launch_rows_m<L, -1, ROW_PROPAGATE, false>(rs, A, s);
}

int launch_rows(const RowSet& rs, const RowArgs& A, cudaStream_t s) {
    if (rs.nblocks <= 0) return TB_OK;
    if (rs.L == 2) return launch_rows_l<2>(rs, A, s);
    if (rs.L == 3) return launch_rows_l<3>(rs, A, s);
    return launch_rows_l<4>(rs, A, s);
}

int launch_rows_spread(const RowSet& rs, const RowArgs& A, const FxAcc& fx_amp, cudaStream_t s) {
    if (rs.nblocks <= 0) return TB_OK;
    auto kern = rs.L == 2 ? k_rows_spread<2> : rs.L == 3 ? k_rows_spread<3> : k_rows_spread<4>;
    kern<<<unsigned(rs.nblocks), 256, 0, s>>>(rs.d_chan, rs.d_work, A.f, A.nf, A.ed->nblk, A.fx, A.u, fx_amp.poison);
    TB_CUDA(cudaGetLastError());
    return TB_OK;
}

int build_row_set(int L, int form, const std::vector<RowChan>& chan, const std::vector<const PointRows*>& rows,
                  int64_t ndofs, RowSet& out, cudaStream_t s, int S, bool whole) {
    out.release();
    out.L = L;
    out.form = form;
    out.S = S;
    out.nmc_max = 0;
    out.multi = false;
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    int64_t nrows = 0;
    for (const PointRows* r : rows) nrows += r->nrows;
    if (nrows <= 0) return TB_OK;
    // a warp takes the instances of a row one after another; where the rows do
    // not fill the chip's warps, parts of the instances go to blocks of their
    // own.  Deterministic 8x8 e-ph right-hand sides, us, without and with: 16 runs
    // 361 / 160, 48 runs 1037 / 368, 128 runs 2732 / 953 (the run-minor
    // contraction of exact sums took 243, 587 and 1370); FP64 atomics, 7 runs
    // 55 / 35; from 16x16 on the rows fill the chip.
    const int64_t parts = whole ? 1 : std::max<int64_t>(1, int64_t(nsm) * row_shares(L) / nrows);
    nrows = 0;
    // what blocks are dealt out to: (channel, part of its instances)
    struct Item { int chan, chunk, i0, i1; };
    std::vector<Item> item;
    for (size_t i = 0; i < chan.size(); ++i) {
        const int n = chan[i].n_insts;
        const int chunks = S ? (n + S - 1) / S : int(std::min<int64_t>(n, parts));
        for (int k = 0; k < chunks; ++k)
            item.push_back({int(i), k, int(int64_t(n) * k / chunks), int(int64_t(n) * (k + 1) / chunks)});
        nrows += rows[i]->nrows * chunks;
        out.nmc_max = std::max(out.nmc_max, chan[i].nmc);
        out.multi = out.multi || n > 1;
    }
    // one block per SM; fewer warps in each where there are fewer rows than
    // warps.  Every item gets a block of its own at least, the others go one
    // by one to the item with the largest cost per block.
    const int64_t per_sm = std::max<int64_t>(4, (nrows + nsm - 1) / nsm);
    out.shares[0] = int(std::min<int64_t>(row_shares(L), per_sm));
    out.shares[1] = int(std::min<int64_t>(row_shares_few(L), per_sm));
    std::vector<int64_t> nb(item.size(), 1);
    auto cost_of = [&](size_t i) -> const std::vector<int64_t>& {
        const PointRows& r = *rows[size_t(item[i].chan)];
        return S ? r.run_cost : r.cost;
    };
    auto load = [&](size_t i) {
        return double(cost_of(i).back()) * (S ? 1 : item[i].i1 - item[i].i0) / double(nb[i]);
    };
    for (int64_t left = std::min<int64_t>(nsm, (nrows + out.shares[0] - 1) / out.shares[0]) - int64_t(item.size()); left > 0;
         --left) {
        size_t best = 0;
        for (size_t i = 1; i < item.size(); ++i)
            if (load(i) > load(best)) best = i;
        nb[best] += 1;
    }
    std::vector<RowWork> work;
    std::vector<int32_t> bounds[2];
    for (size_t i = 0; i < item.size(); ++i) {
        const RowChan& c = chan[size_t(item[i].chan)];
        const std::vector<int64_t>& cost = cost_of(i);
        for (int64_t b = 0; b < nb[i]; ++b) {
            RowWork w{};
            w.chan = item[i].chan;
            w.chunk = item[i].chunk;
            w.i0 = item[i].i0;
            w.i1 = item[i].i1;
            w.t0 = c.n * b / nb[i];
            w.t1 = c.n * (b + 1) / nb[i];
            work.push_back(w);
            for (int k = 0; k < 2; ++k)
                for (int64_t p = b * out.shares[k]; p <= (b + 1) * out.shares[k]; ++p)   // rows up to the p-th share
                    bounds[k].push_back(int32_t(std::lower_bound(cost.begin(), cost.end(),
                                                                 cost.back() * p / (nb[i] * out.shares[k])) -
                                                cost.begin()));
        }
    }
    const size_t cb = (sizeof(RowChan) * chan.size() + 255) / 256 * 256, wb = (sizeof(RowWork) * work.size() + 255) / 256 * 256;
    const size_t bb = sizeof(int32_t) * bounds[0].size();
    std::vector<char> all(cb + wb + bb + sizeof(int32_t) * bounds[1].size());
    std::memcpy(all.data(), chan.data(), sizeof(RowChan) * chan.size());
    std::memcpy(all.data() + cb, work.data(), sizeof(RowWork) * work.size());
    std::memcpy(all.data() + cb + wb, bounds[0].data(), bb);
    std::memcpy(all.data() + cb + wb + bb, bounds[1].data(), sizeof(int32_t) * bounds[1].size());
    char* base = nullptr;
    if (cudaMalloc(&base, all.size()) != cudaSuccess) {
        cudaGetLastError();
        set_error("row set allocation failed");
        return TB_ERR_OOM;
    }
    out.d_chan = reinterpret_cast<RowChan*>(base);
    out.bytes = all.size();
    out.d_work = reinterpret_cast<RowWork*>(base + cb);
    out.d_bounds[0] = reinterpret_cast<int32_t*>(base + cb + wb);
    out.d_bounds[1] = reinterpret_cast<int32_t*>(base + cb + wb + bb);
    TB_CUDA(cudaMemcpyAsync(base, all.data(), all.size(), cudaMemcpyHostToDevice, s));
    TB_CUDA(cudaStreamSynchronize(s));
    out.nblocks = int(work.size());
    int64_t adds = 0;   // of the channel whose smallest band takes the most for each element
    for (size_t i = 0; i < chan.size(); ++i) {
        int64_t ne = chan[i].leg[1].ne;
        for (int l = 2; l < L; ++l) ne = std::min<int64_t>(ne, chan[i].leg[l].ne);
        adds = std::max(adds, rows[i]->n * (L - 1) / std::max<int64_t>(ne, 1));
    }
    out.copies = S ? 1 : row_copies(adds, out.nblocks, ndofs);
    return TB_OK;
}

// --------------------------------------------------------------- many runs
int rows_lane_group(int n) {
    int best = 32;
    for (int S : {16, 8})
        if ((n + S - 1) / S * S < (n + best - 1) / best * best) best = S;
    return best;
}

__device__ __forceinline__ const RunState& tile_state(const RunState* st, int n_st, int tile) {
    int k = 0;
    while (k + 1 < n_st && tile >= st[k + 1].tile0) ++k;
    return st[k];
}

__device__ __forceinline__ int64_t run_slot(const RunState& st, int64_t d, int i) {
    return (int64_t(i / st.S) * st.ndof + d) * st.S + i % st.S;
}

// fT[i / S][d][i % S] = f[dof_off[i] + d], 32 dofs x 32 runs a tile
__global__ void __launch_bounds__(256) k_runs_state_gather(const RunState* __restrict__ st, int n_st,
                                                           const double* __restrict__ f, int* __restrict__ nf,
                                                           const DPCtl* __restrict__ ctl) {
    __shared__ double tile[32][33];
    const RunState& S = tile_state(st, n_st, blockIdx.x);
    const int k = blockIdx.x - S.tile0, tx = threadIdx.x, ty = threadIdx.y;
    const int i0 = (k % S.tiles_i) * 32;
    const int64_t d0 = int64_t(k / S.tiles_i) * 32;
    bool bad = false;
    for (int y = ty; y < 32; y += 8) {
        const int i = i0 + y;
        double v = 0.0;
        if (i < S.n && d0 + tx < S.ndof && !(ctl && ctl[S.run[i]].done)) {
            v = __ldg(f + S.dof_off[i] + d0 + tx);
            bad = bad || !isfinite(v);
        }
        tile[y][tx] = v;
    }
    bad = __syncthreads_or(bad);
    if (tx == 0 && ty == 0) nf[blockIdx.x] = bad ? 1 : 0;
    for (int y = ty; y < 32; y += 8)
        if (d0 + y < S.ndof && i0 + tx < S.np) S.fT[run_slot(S, d0 + y, i0 + tx)] = tile[tx][y];
}

// acc[dof_off[i] + d] += accT[i / S][d][i % S], which is cleared.  Every coefficient of
// the state belongs to one run of one structure, so the adds need no atomics.
__global__ void __launch_bounds__(256) k_runs_state_scatter(const RunState* __restrict__ st, int n_st,
                                                            double* __restrict__ acc, const DPCtl* __restrict__ ctl) {
    __shared__ double tile[32][33];
    const RunState& S = tile_state(st, n_st, blockIdx.x);
    const int k = blockIdx.x - S.tile0, tx = threadIdx.x, ty = threadIdx.y;
    const int i0 = (k % S.tiles_i) * 32;
    const int64_t d0 = int64_t(k / S.tiles_i) * 32;
    for (int y = ty; y < 32; y += 8) {
        double v = 0.0;
        if (d0 + y < S.ndof && i0 + tx < S.np) {
            double* p = S.accT + run_slot(S, d0 + y, i0 + tx);
            v = *p;
            *p = 0.0;
        }
        tile[y][tx] = v;
    }
    __syncthreads();
    for (int y = ty; y < 32; y += 8) {
        const int i = i0 + y;
        if (i < S.n && d0 + tx < S.ndof && !(ctl && ctl[S.run[i]].done)) acc[S.dof_off[i] + d0 + tx] += tile[tx][y];
    }
}

// The rows for S runs at a time: lane = (tuple of a group of 32 / S, run).  A
// tuple's map, mask and points are the same for its S lanes (broadcast reads);
// the legs' f and their adds are coalesced pieces of run-minor rows; leg 0's f
// and sums stay in registers while the element does.  Per tuple and run it does
// 19 FP64 instructions a point and 45 more, against 320 of the contraction over
// 27 moments; it issues 46 % of the time, bound by fixed-latency dependencies.
// 48 runs on three meshes (32x32, 24x24, 16x16) to t = 0.5: 152 ms against 334 ms
// through k_collision_runs.  16 warps a block at 126 registers: 12 warps take
// 182 ms, 20 (spilled) 165; two points a step 158.
template <int L, int FORM, int S>
__global__ void __launch_bounds__(row_shares(L) * 32, 1) k_rows_runs(const RowChan* __restrict__ chans,
                                                                 const RowWork* __restrict__ work,
                                                                 const int32_t* __restrict__ bounds,
                                                                 const double* __restrict__ f,
                                                                 const int* __restrict__ nf, int n_nf,
                                                                 double* __restrict__ acc,
                                                                 const DPCtl* __restrict__ ctl,
                                                                 int* __restrict__ err_flag, int wait_polls) {
    constexpr int R = RowDim<L>::R, ND = RowDim<L>::ND, G = 32 / S;
    constexpr uint32_t BYTES = RowDim<L>::BYTES;
    extern __shared__ __align__(128) unsigned char s_raw[];
    __shared__ RowChan c;
    __shared__ __align__(8) uint64_t s_bar[row_shares(L)][ROW_STAGES];
    const RowWork w = work[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_warps = blockDim.x >> 5;
    for (int i = tid; i < int(sizeof(RowChan) / sizeof(int)); i += blockDim.x)
        reinterpret_cast<int*>(&c)[i] = reinterpret_cast<const int*>(chans + w.chan)[i];
    __syncthreads();
    const int g = lane / S, run = w.chunk * S + lane % S;
    double amp = 0.0;   // 0: padding, switched off or finished
    if (run < c.n_insts) {
        const InstDev& in = c.insts[run];
        if (in.amp_full != 0.0 && !(ctl && ctl[in.run].done)) amp = in.amp_full;
    }
    if (__all_sync(0xffffffffu, amp == 0.0)) return;   // uniform in the block
    bounds += blockIdx.x * (n_warps + 1) + warp;   // one share a warp
    const int r0 = bounds[0], r1 = bounds[1];
    unsigned char* const stage = s_raw + size_t(warp) * ROW_STAGES * BYTES;
    uint64_t* const bar = s_bar[warp];
    auto fetch = [&](int r, int s) {
        mbar_expect_tx_arrive(&bar[s], BYTES);
        bulk_g2s(stage + s * BYTES, c.blk + int64_t(r) * BYTES, BYTES, &bar[s]);
    };
    if (lane == 0) {
        for (int s = 0; s < ROW_STAGES; ++s) mbar_init(&bar[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int s = 0; s < ROW_STAGES; ++s)
            if (r0 + s < r1) fetch(r0 + s, s);
    }
    double* const s_q = reinterpret_cast<double*>(s_raw + size_t(n_warps) * ROW_STAGES * BYTES);
    for (int i = tid; i < c.nmc * R; i += blockDim.x) s_q[i] = __ldg(c.mc + i);
    __syncthreads();
    const FlatTable tab{s_q};
    // element e of leg l: coefficient j at [3 e S + j S]
    const double* fl[L];
    double* al[L];
#pragma unroll
    for (int l = 0; l < L; ++l) {
        const int64_t o = (w.chunk * c.ndof + c.loff[l]) * S + lane % S;
        fl[l] = c.fT + o;
        al[l] = c.accT + o;
    }
    double z[3] = {0.0, 0.0, 0.0};
    int e0 = -1;
    double4 f0 = make_double4(0., 0., 0., 0.);
    auto flush = [&]() {
#pragma unroll
        for (int o = S; o < 32; o *= 2)
#pragma unroll
            for (int j = 0; j < 3; ++j) z[j] += __shfl_xor_sync(0xffffffffu, z[j], o);
        if (g == 0 && amp != 0.0) {
            double* o = al[0] + 3 * S * e0;
#pragma unroll
            for (int j = 0; j < 3; ++j) atomicAdd(o + j * S, z[j]);
        }
        z[0] = z[1] = z[2] = 0.0;
    };
    for (int r = r0; r < r1; ++r) {
        const int s = (r - r0) % ROW_STAGES;
        const int e0_row = __ldg(c.row_e0 + r);
        if (e0_row != e0) {
            if (e0 >= 0) flush();
            e0 = e0_row;
            const double* p = fl[0] + 3 * S * e0;
            f0 = make_double4(__ldg(p), __ldg(p + S), __ldg(p + 2 * S), 0.0);
        }
        // one verdict for the warp, as in k_rows
        if (!__all_sync(0xffffffffu, mbar_wait(&bar[s], uint32_t((r - r0) / ROW_STAGES) & 1u, wait_polls))) {
            // record the failure and give the copies in flight a bounded
            // chance to land before the block releases its shared memory
            if (lane == 0) atomicExch(err_flag, 1);
            for (int k = 0; k < ROW_STAGES && r + k < r1; ++k)
                mbar_wait(&bar[(r + k - r0) % ROW_STAGES], uint32_t((r + k - r0) / ROW_STAGES) & 1u, 1 << 16);
            break;
        }
        const unsigned char* b = stage + s * BYTES;
#pragma unroll 1
        for (int t0 = 0; t0 < 32; t0 += G) {
            const int t = t0 + g;
            const uint64_t mk = reinterpret_cast<const uint64_t*>(b + 256 * ND)[t];
            if (__all_sync(0xffffffffu, mk == 0ull)) break;   // the padding of the element's last row
            double4 fv[L];
            double* o[L];
            fv[0] = f0;
#pragma unroll
            for (int l = 1; l < L; ++l) {
                const int k = 3 * S * reinterpret_cast<const int32_t*>(b + 256 * (ND + 1))[32 * (l - 1) + t];
                const double* p = fl[l] + k;
                o[l] = al[l] + k;
                fv[l] = make_double4(__ldg(p), __ldg(p + S), __ldg(p + 2 * S), 0.0);
            }
            const StageMap<L> m{reinterpret_cast<const double*>(b) + t};
            double scale = reinterpret_cast<const double*>(b)[32 * (ND - 1) + t] * amp;
            if (c.tamp && mk) scale *= __ldg(c.tamp + __ldg(c.perm + int64_t(r) * 32 + t));
            RowOut<L> v;
            row_tuple<L, FORM>(c, m, mk, fv, tab, scale, v);
#pragma unroll
            for (int j = 0; j < 3; ++j) z[j] += v.v[0][j];
            if (mk && amp != 0.0) {
#pragma unroll
                for (int l = 1; l < L; ++l)
#pragma unroll
                    for (int j = 0; j < 3; ++j) atomicAdd(o[l] + j * S, v.v[l][j]);
            }
        }
        __syncwarp();   // every lane is done with the stage
        if (lane == 0 && r + ROW_STAGES < r1) fetch(r + ROW_STAGES, s);
    }
    if (e0 >= 0) flush();
    int bad = 0;
    for (int i = tid; i < n_nf; i += blockDim.x) bad |= nf[i];
    if (__syncthreads_or(bad)) {
        const int i0 = w.chunk * S;
        FxAcc none;
        spread_nonfinite<L>(c, c.insts + i0, min(S, c.n_insts - i0), w.t0, w.t1, f, acc, ctl, false, -1, none);
    }
}

template <int L, int FORM, int S>
static int launch_k_rows_runs(const RowSet& rs, int n_tiles, const double* f, const int* nf, double* acc,
                              const DPCtl* ctl, cudaStream_t s, int* err_flag, int polls) {
    auto kern = k_rows_runs<L, FORM, S>;
    auto bytes = [](int nmc, int warps) {
        return size_t(warps) * ROW_STAGES * row_bytes(L) + sizeof(double) * size_t(nmc) * RowDim<L>::R;
    };
    static std::atomic<unsigned long long> attr_devices{0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !((attr_devices.load() >> dev) & 1ull)) {
        TB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes(64, row_shares(L)))));
        if (dev >= 0 && dev < 64) attr_devices.fetch_or(1ull << dev);
    }
    kern<<<unsigned(rs.nblocks), unsigned(32 * rs.shares[0]), bytes(rs.nmc_max, rs.shares[0]), s>>>(
        rs.d_chan, rs.d_work, rs.d_bounds[0], f, nf, n_tiles, acc, ctl, err_flag, polls);
    TB_CUDA(cudaGetLastError());
    return TB_OK;
}

template <int L, int FORM>
static int launch_rows_runs_s(const RowSet& rs, int n_tiles, const double* f, const int* nf, double* acc,
                              const DPCtl* ctl, cudaStream_t s, int* err_flag, int polls) {
    if (rs.S == 8) return launch_k_rows_runs<L, FORM, 8>(rs, n_tiles, f, nf, acc, ctl, s, err_flag, polls);
    if (rs.S == 16) return launch_k_rows_runs<L, FORM, 16>(rs, n_tiles, f, nf, acc, ctl, s, err_flag, polls);
    return launch_k_rows_runs<L, FORM, 32>(rs, n_tiles, f, nf, acc, ctl, s, err_flag, polls);
}

int launch_run_rows(const std::vector<RowSet>& sets, const RunState* st, int n_st, int n_tiles, const double* f,
                    int* nf, double* acc, const DPCtl* ctl, cudaStream_t s, int* err_flag, int polls) {
    if (sets.empty()) return TB_OK;
    k_runs_state_gather<<<unsigned(n_tiles), dim3(32, 8), 0, s>>>(st, n_st, f, nf, ctl);
    TB_CUDA(cudaGetLastError());
    for (const RowSet& rs : sets) {
        if (rs.nblocks <= 0) continue;
        int rc;
        if (rs.L == 2)
            rc = rs.form == FORM_2 ? launch_rows_runs_s<2, FORM_2>(rs, n_tiles, f, nf, acc, ctl, s, err_flag, polls)
                              : launch_rows_runs_s<2, -1>(rs, n_tiles, f, nf, acc, ctl, s, err_flag, polls);
        else if (rs.L == 4)
            rc = rs.form == FORM_4 ? launch_rows_runs_s<4, FORM_4>(rs, n_tiles, f, nf, acc, ctl, s, err_flag, polls)
                                   : launch_rows_runs_s<4, -1>(rs, n_tiles, f, nf, acc, ctl, s, err_flag, polls);
        else
            rc = rs.form == FORM_3 ? launch_rows_runs_s<3, FORM_3>(rs, n_tiles, f, nf, acc, ctl, s, err_flag, polls)
                              : launch_rows_runs_s<3, -1>(rs, n_tiles, f, nf, acc, ctl, s, err_flag, polls);
        TB_TRY(rc);
    }
    k_runs_state_scatter<<<unsigned(n_tiles), dim3(32, 8), 0, s>>>(st, n_st, acc, ctl);
    TB_CUDA(cudaGetLastError());
    return TB_OK;
}

}  // namespace tb
