// tb_drift.cu -- field-driven drift: the DG upwind Vlasov operator of the
// reference (include/Physics/Transport/Vlasov.hpp:69-118), as a block-sparse
// operator with 3x3 blocks (self plus up to three face neighbours) evaluated
// matrix-free: one thread per element reads its own 3 coefficients and those
// of the upwind neighbours, and adds (volume - surface) into the pre-M^-1
// accumulator (M^-1 is applied with the collision terms).
//
// Geometry follows Mesh<2>: periodic adjacency and faces (src/Geometry/
// Structured/DirectSpace/Mesh.cpp:573-660); basis derivatives evaluated on
// calculate_verticesCoord (Mesh.cpp:147-163, 222-241), which places vertices
// at relativeOrigin + dGVec * (section + vertex).
#include "tb_dp45.cuh"
#include "tb_drift.cuh"
#include "tb_kernels.cuh"

namespace tb {

__global__ void __launch_bounds__(256) k_drift(ElemDev ed, const double* __restrict__ f, double* __restrict__ acc,
                                               const DPCtl* __restrict__ ctl) {
    const int band = ed.blk_band[blockIdx.x];
    const BandDev& bd = ed.bands[band];
    if (bd.vel[0] == 0.0 && bd.vel[1] == 0.0) return;
    if (ctl && ctl[ed.band_run[band]].done) return;
    const int e = (blockIdx.x - ed.blk_first[band]) * blockDim.x + threadIdx.x;
    if (e >= bd.ne) return;
    drift_element(bd, f, e, acc);
}

int launch_drift(const ElemDev& ed, const double* f, double* acc, const DPCtl* ctl, cudaStream_t s) {
    k_drift<<<ed.nblk, 256, 0, s>>>(ed, f, acc, ctl);
    TB_CUDA(cudaGetLastError());
    return TB_OK;
}

}  // namespace tb
