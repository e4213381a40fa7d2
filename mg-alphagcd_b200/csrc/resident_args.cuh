// resident_args.cuh -- arguments of the resident level kernel (resident.cuh)
// and its launchers, one per weight kind (resident_*.cu).
#pragma once

#include "engine.cuh"

namespace mg {
namespace lmr {

constexpr int kResidentThreads = 1024;
constexpr int kResidentIters = 48;     // iterations of one launch (the host launches again while a level goes on)
constexpr int kResidentMaxBits = 14;   // slots of a CTA's table: 2^14 (9 or 13 bytes each)
constexpr unsigned kBarrierSpins = 1u << 24;
// warp steps of a tile task in flight at once: SBM runs of 4.0 M entries took
// 9.6 ms of kernel time with 1, 6.2 ms with 2 and 6.2 ms with 4 (spills)
constexpr int kTileU = 2;
// largest number of distinct communities a vertex may see: 2/3 of the CTA's table
constexpr uint32_t kResidentCapacity = (1u << kResidentMaxBits) / 3 * 2;

// The loop's state, kept between launches: the assignment buffers (base: last
// accepted, p: swept next, nx: written next), the direction, Q of the base.
struct ResidentState {
    int base, p, nx, up, first, done, err, iters;
    double curQ;
    unsigned long long distinct;  // candidates of the last sweep
};

struct ResidentArgs {
    const uint32_t *col;
    const void *w;
    const uint32_t *perm;  // vertices by degree class
    const uint2 *rows;     // their row ranges
    const double *k;
    double *sigma;
    uint32_t *C[3];
    GainK K;
    double mass, thr;
    uint32_t n;
    unsigned long long nnz;
    int integral;
    int bits;  // log2 of the CTA's table slots
    // class-list ranges: [cut[1], cut[2]) 128 threads per vertex, [cut[2],
    // cut[3]) 256, [cut[3], cut[4]) the CTA
    uint32_t cut[5];
    // tasks of a warp: kind 0 a warp vertex, kinds 1..5 tiles of 32, 16, 8, 4
    // and 2 lanes (kTileU steps each); task_end is cumulative
    uint32_t kind_off[6], kind_size[6], task_end[6], tasks;
    ResidentState *state;
    SweepAcc *acc;       // one per iteration, zeroed; pad receives Q
    uint32_t *task_ctr;  // one per iteration, zeroed
    unsigned *barrier;   // zeroed
};

void launch_resident_unit(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s);
void launch_resident_u32(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s);
void launch_resident_f32i(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s);
void launch_resident_f64i(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s);
void launch_resident_f32(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s);
void launch_resident_f64(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s);

}  // namespace lmr
}  // namespace mg
