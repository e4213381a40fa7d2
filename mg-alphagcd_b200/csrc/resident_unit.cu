// resident_unit.cu -- the resident level kernels for weight kind WK_UNIT.
#include "resident.cuh"

namespace mg {
namespace lmr {

bool launch_resident_unit(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s) {
    return launch_resident_kind<WK_UNIT>(A, prec, ver, grid, s);
}

bool launch_batch_unit(const ResidentBatchArgs &A, int prec, int ver, int ctas, unsigned most, cudaStream_t s) {
    return launch_batch_kind<WK_UNIT>(A, prec, ver, ctas, most, s);
}

}  // namespace lmr
}  // namespace mg
