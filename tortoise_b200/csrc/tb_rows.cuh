// tb_rows.cuh -- packed rows of tuples: the Monte-Carlo quadrature over the
// points inside the simplices.
#pragma once

#include <vector>

#include "tb_kernels.cuh"
#include "tb_theta.cuh"

namespace tb {

// The tuples of one channel that have a point inside the simplices, 32 to a
// row; all tuples of a row share their leg-0 element (the last row of an
// element is padded with tuples without points).  A row is one contiguous
// block (row_bytes), each field 32 wide:
//   double   a0[3], G[3][R]   the affine map of the constrained coordinates
//   double   w                1 / (fact nmc |det|)
//   uint64_t mask             the points inside
//   int32_t  e[L - 1]         element ids of legs 1 .. L-1
struct PointRows {
    unsigned char* blk = nullptr;
    int32_t* row_e0 = nullptr;      // [nrows]
    int32_t* perm = nullptr;        // [nrows][32] index in the channel's list (padding: -1)
    int64_t nrows = 0;
    int64_t n = 0, points = 0;      // tuples and points inside
    int64_t bytes = 0;              // device memory of the rows
    std::vector<int64_t> cost;      // [nrows + 1] running cost of the rows (host)
    std::vector<int64_t> run_cost;  // the same, run-minor
    void release();
};

size_t row_bytes(int L);

// Directions and statistics of a channel's legs: bit l: leg l is ingoing, bit
// 4 + l: it is a boson.
int row_form(const ChanDev& c);

// Builds the rows from a ThetaList.  rows.blk stays null when they would take
// more than max_bytes (the caller then keeps another path).
int build_rows(const ChanDev& c, const ThetaList& th, PointRows& rows, int64_t max_bytes, cudaStream_t s);

// What the kernel needs of one channel, in device memory.
struct RowChan {
    const unsigned char* blk;
    const int32_t* row_e0;
    const int32_t* perm;
    const double* mc;
    const double* tamp;             // functAmplitude per tuple, or null
    const InstDev* insts;
    int n_insts;
    int nmc;
    int gamp0;                      // its first slot among the amplitude gradients
    double amp_vol;
    LegDev leg[4];
    // shared by many runs: the structure's run-minor state and accumulator
    // (RunState), the legs' band offsets within a run
    const double* fT;
    double* accT;
    int64_t ndof;
    int64_t loff[4];
    // the whole list, for states with non-finite coefficients
    const int32_t* tup;
    int64_t stride, n;
};

// One block's work: rows of channel chan, in shares that RowSet's bounds
// delimit, and the part [t0, t1) of its whole list.
struct RowWork {
    int chan;
    int chunk;       // run-minor sets: which S runs
    int i0, i1;      // other sets: instances [i0, i1) of the channel
    int64_t t0, t1;
};

// A set of channels of equal leg count and form that one launch
// evaluates.
struct RowSet {
    int L = 0;
    int form = 0;                   // row_form
    RowChan* d_chan = nullptr;
    RowWork* d_work = nullptr;
    // per block the bounds of its shares (shares + 1), one share a warp: for
    // propagation, and for the kernels that take fewer warps
    int32_t* d_bounds[2] = {nullptr, nullptr};
    int shares[2] = {0, 0};
    size_t bytes = 0;               // of the allocation behind d_chan
    int nblocks = 0;
    int nmc_max = 0;
    int copies = 1;                 // accumulators that its blocks share out (row_copies)
    bool multi = false;             // some channel has several instances
    int S = 0;                      // run-minor: runs per lane group (8, 16 or 32), else 0
    void release();
};

// A structure whose runs share its rows: the state of its n runs, run-minor
// in groups of S ([i / S][dof][i % S]).
// Run i of the structure starts at dof_off[i] of the handle's state.
struct RunState {
    double* fT;
    double* accT;                   // all zero between evaluations
    const int64_t* dof_off;         // [n]
    const int* run;                 // [n] run numbers (DPCtl index)
    int n, np, S;                   // np: n padded to whole groups
    int64_t ndof;                   // dofs of one run
    int tile0, tiles_i;             // first tile of the structure, tiles across runs
};

// Runs per lane group for n runs: the widest of 32, 16 and 8 that pads n least.
int rows_lane_group(int n);

// Uploads the set (on s, which it waits for) for the given channels (rows of channel i in rows[i]) of a
// handle with ndofs coefficients;
// blocks are dealt out by the rows' cost.  whole: every block takes all
// instances of its channel (a set that is also launched for one instance).
int build_row_set(int L, int form, const std::vector<RowChan>& chan, const std::vector<const PointRows*>& rows,
                  int64_t ndofs, RowSet& out, cudaStream_t s, int S = 0, bool whole = false);

// f4[e] = (f0, f1, f2, 0) of every element of the state, u4 of u likewise when
// it is given; nf[b] != 0 marks an element block with a non-finite coefficient.
// drift_acc non-null: the drift term is added there too (launch_drift's; the
// same pass over the elements saves its launch, 5 us).
int launch_rows_prepare(const ElemDev& ed, const double* f, double4* f4, int* nf, const DPCtl* ctl, cudaStream_t s,
                        const double* u = nullptr, double4* u4 = nullptr, double* drift_acc = nullptr);

// One evaluation of a set.
struct RowArgs {
    const ElemDev* ed = nullptr;
    const double* f = nullptr;      // the state, and what launch_rows_prepare made of it
    const double4* f4 = nullptr;
    const int* nf = nullptr;
    double* acc = nullptr;          // or fx: the collision terms are added here
    double* accr = nullptr;         // the set's copies - 1 further accumulators of ed->ndofs doubles,
                                    // all zero between launches (null: one for all blocks)
    FxAcc fx{};
    const DPCtl* ctl = nullptr;
    const InstDev* one = nullptr;   // this instance in place of the channels' instances
    bool rate = false;              // scattering rate of leg rate_leg (of every leg when negative)
    int rate_leg = -1;
    // non-null: the transposed operator for the co-state u instead, acc +=
    // C'(f)^T u and gamp[gamp0 + k] += <u, dC / d amplitude_k>
    const double* u = nullptr;
    const double4* u4 = nullptr;
    double* gamp = nullptr;
    int* err_flag = nullptr;        // set when a bounded wait (polls) for a staged row runs out
    int polls = 0;
};
int launch_rows(const RowSet& rs, const RowArgs& a, cudaStream_t s);

// What the tuples without a point inside add to the exact sums of a transposed
// evaluation (a.u) when a.nf marks non-finite coefficients.
int launch_rows_spread(const RowSet& rs, const RowArgs& a, const FxAcc& fx_amp, cudaStream_t s);

// The run-minor sets: the structures' states gathered, each set evaluated,
// their accumulators added to acc and cleared.  st: device copy of the n_st
// structures (n_tiles tiles in all); nf as above, one flag per tile.
int launch_run_rows(const std::vector<RowSet>& sets, const RunState* st, int n_st, int n_tiles, const double* f,
                    int* nf, double* acc, const DPCtl* ctl, cudaStream_t s, int* err_flag, int polls);

}  // namespace tb
