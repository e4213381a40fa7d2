// resident_u32.cu -- the resident level kernel for weight kind WK_U32.
#include "resident.cuh"

namespace mg {
namespace lmr {

void launch_resident_u32(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s) {
    launch_resident_kind<WK_U32>(A, prec, ver, grid, s);
}

}  // namespace lmr
}  // namespace mg
