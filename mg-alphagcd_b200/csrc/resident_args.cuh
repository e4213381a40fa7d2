// resident_args.cuh -- arguments of the resident level kernel (resident.cuh)
// and its launchers, one per weight kind (resident_*.cu).
#pragma once

#include "engine.cuh"

namespace mg {
namespace lmr {

constexpr int kResidentThreads = 1024;
constexpr int kResidentIters = 48;     // iterations of one launch (the host launches again while a level goes on)
constexpr int kResidentMaxBits = 14;   // slots of a CTA's table: 2^14 (9 or 13 bytes each)
constexpr unsigned kBarrierPolls = 1u << 24;
// warp steps of a tile task in flight at once: SBM runs of 4.0 M entries took
// 5.8 ms of kernel time with 1, 5.0 ms with 2, 5.6 ms with 3 and 5.3 ms with 4
// (spills)
constexpr int kTileU = 2;
// largest number of distinct communities a vertex may see: 7/8 of the CTA's table (few vertices
// are that large; the probes of a table filled so far cost less than leaving the level)
constexpr uint32_t kResidentCapacity = (1u << kResidentMaxBits) / 8 * 7;

// log2 of the slots of a CTA's table for a level of that largest degree (or
// number of communities a vertex can see): as small as the level allows, since
// what the table does not take stays L1 for the community and sigma gathers
inline int resident_bits(uint32_t most) {
    return most <= 32 ? 10 : most <= 64 ? 12 : most <= 128 ? 13 : kResidentMaxBits;
}

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
    int sweeps;      // iterations of this launch, at most kResidentIters
    unsigned polls;  // of a barrier before a block gives up
    int sms;         // (launcher) SMs of the device
    uint32_t cls[kSweepClasses + 1];  // start of every degree class in the class list; n
    ResidentState *state;
    SweepAcc *acc;       // one per iteration, zeroed; pad receives Q
    uint32_t *task_ctr;  // one per iteration, zeroed
    unsigned *barrier;   // zeroed
};

// The batched form (lm_resident_batch_kernel): a graph per cluster of CTAs.
constexpr int kResidentBatchIters = 1024;  // iterations of a graph in one launch
struct ResidentTotals {
    unsigned long long edges;   // entries swept by the graphs that finished
    unsigned long long sweeps;  // most sweeps of one graph
    uint32_t open, pad;         // graphs that need another launch
};
struct ResidentBatchArgs {
    const uint32_t *col;
    const void *w;
    const uint32_t *perm;
    const uint2 *rows;
    const double *k;
    double *sigma;
    uint32_t *C[3];
    double thr;
    int integral, bits;
    int sweeps;             // iterations of a graph in this launch
    const uint32_t *cls;    // per graph: start of its part of every degree class (graphs + 1 rows)
    const uint32_t *goff;   // first vertex of each graph
    const uint32_t *gnnz;
    const GainK *gk;
    const double *mass;
    const uint32_t *order;  // graphs to run, largest first
    uint32_t count;
    uint32_t *queue;        // zeroed
    ResidentState *state;   // per graph
    uint32_t *gword;
    double *curQ;
    unsigned long long *iters, *distinct;
    ResidentTotals *totals;  // zeroed
};

#define MG_RESIDENT_KINDS(X) X(unit) X(u32) X(f32i) X(f64i) X(f32) X(f64)
// The launchers return false, with nothing launched, when the device holds no
// block (no cluster) of the kernel.
#define MG_RESIDENT_BATCH(k) \
    bool launch_batch_##k(const ResidentBatchArgs &A, int prec, int ver, int ctas, unsigned most, cudaStream_t s);
MG_RESIDENT_KINDS(MG_RESIDENT_BATCH)
#undef MG_RESIDENT_BATCH

bool launch_resident_unit(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s);
bool launch_resident_u32(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s);
bool launch_resident_f32i(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s);
bool launch_resident_f64i(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s);
bool launch_resident_f32(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s);
bool launch_resident_f64(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s);

}  // namespace lmr
}  // namespace mg
