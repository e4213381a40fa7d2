// resident_f32.cu -- the resident level kernels for weight kind WK_F32.
#include "resident.cuh"

namespace mg {
namespace lmr {

bool launch_resident_f32(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s) {
    return launch_resident_kind<WK_F32>(A, prec, ver, grid, s);
}

bool launch_batch_f32(const ResidentBatchArgs &A, int prec, int ver, int ctas, unsigned most, cudaStream_t s) {
    return launch_batch_kind<WK_F32>(A, prec, ver, ctas, most, s);
}

}  // namespace lmr
}  // namespace mg
