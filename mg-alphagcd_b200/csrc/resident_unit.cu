// resident_unit.cu -- the resident level kernel for weight kind WK_UNIT.
#include "resident.cuh"

namespace mg {
namespace lmr {

void launch_resident_unit(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s) {
    launch_resident_kind<WK_UNIT>(A, prec, ver, grid, s);
}

}  // namespace lmr
}  // namespace mg
