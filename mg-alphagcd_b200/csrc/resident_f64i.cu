// resident_f64i.cu -- the resident level kernels for weight kind WK_F64I.
#include "resident.cuh"

namespace mg {
namespace lmr {

bool launch_resident_f64i(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s) {
    return launch_resident_kind<WK_F64I>(A, prec, ver, grid, s);
}

bool launch_batch_f64i(const ResidentBatchArgs &A, int prec, int ver, int ctas, unsigned most, cudaStream_t s) {
    return launch_batch_kind<WK_F64I>(A, prec, ver, ctas, most, s);
}

}  // namespace lmr
}  // namespace mg
