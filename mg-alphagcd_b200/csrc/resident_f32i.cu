// resident_f32i.cu -- the resident level kernels for weight kind WK_F32I.
#include "resident.cuh"

namespace mg {
namespace lmr {

bool launch_resident_f32i(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s) {
    return launch_resident_kind<WK_F32I>(A, prec, ver, grid, s);
}

bool launch_batch_f32i(const ResidentBatchArgs &A, int prec, int ver, int ctas, unsigned most, cudaStream_t s) {
    return launch_batch_kind<WK_F32I>(A, prec, ver, ctas, most, s);
}

}  // namespace lmr
}  // namespace mg
