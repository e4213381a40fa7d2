// resident.cu -- host side of the resident level kernel (resident.cuh): which
// levels take it, its work split, and the loop that launches it.
#include <algorithm>
#include <cstring>

#include "handles.cuh"
#include "resident_args.cuh"

namespace mg {

namespace {

using namespace lmr;

// One transfer each way per launch: the state and the zeroed sums, counters
// and barrier of the launch go up, the state and the sums come back.
struct ResidentBlock {
    ResidentState state;
    SweepAcc acc[kResidentIters];
    uint32_t task_ctr[kResidentIters];
    unsigned barrier;
};

}  // namespace

bool resident_size(uint32_t n, uint64_t nnz, uint32_t max_degree, int integral) {
    if (n == 0 || nnz > (integral ? kResidentMaxEntries : kResidentMaxEntriesReal)) return false;
    return std::min(max_degree, n) <= kResidentCapacity;
}

bool resident_level(const GraphView &g, const MoveLevel &lvl, const MoveWorkspace &ws, int integral) {
    return resident_allowed(ws) && resident_size(g.n, g.nnz, lvl.bins.max_degree, integral);
}

bool resident_run(mg_ctx *ctx, const GraphView &g, const MoveLevel &lvl, const SweepParams &p, double thr,
                  ResidentResult &out, cudaStream_t s) {
    MoveWorkspace &ws = ctx->mws;
    const Bins &B = lvl.bins;
    ResidentBlock *hb = (ResidentBlock *)ws.h_resident;
    if (!hb) {
        MG_CUDA(cudaMallocHost(&ws.h_resident, sizeof(ResidentBlock)));
        hb = (ResidentBlock *)ws.h_resident;
    }
    ResidentBlock *db = (ResidentBlock *)ws.res_block.ensure(sizeof(ResidentBlock));
    ResidentArgs A = {};
    A.col = g.col;
    A.w = g.w;
    A.perm = ws.perm.get();
    A.rows = ws.rows.get();
    A.k = ctx->k.get();
    A.sigma = ctx->sigma.get();
    for (int i = 0; i < 3; i++) A.C[i] = ctx->C[i].get();
    A.K = gain_constants(p.mass);
    A.mass = p.mass;
    A.thr = thr;
    A.n = g.n;
    A.nnz = g.nnz;
    A.integral = p.integral;
    A.bits = resident_bits(std::min(B.max_degree, g.n));
    for (int c = 0; c < kSweepClasses; c++) A.cls[c] = B.offset[c];
    A.cls[kSweepClasses] = g.n;
    A.sweeps = ws.test_sweeps > 0 ? std::min(ws.test_sweeps, kResidentIters) : kResidentIters;
    A.polls = ws.test_polls ? ws.test_polls : kBarrierPolls;
    A.sms = ws.resident_sms();
    // CTAs: work for half of a CTA's warps, or as many as the device holds
    uint64_t warps = 0;
    for (int c = 0; c < kSweepClasses; c++)
        warps += c > 5 ? B.size[c] * ceil_div(1ull << c, 1ull << (A.bits - 6)) : ceil_div(B.size[c], kTileU * (32u >> c));
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(warps, 16), 0xffffu));
    A.state = &db->state;
    A.acc = db->acc;
    A.task_ctr = db->task_ctr;
    A.barrier = &db->barrier;
    const int wk = p.integral ? (g.wk == WK_F32 ? (int)WK_F32I : g.wk == WK_F64 ? (int)WK_F64I : g.wk) : g.wk;
    if (p.precision == MG_PREC_INT64)
        MG_CHECK(p.integral && p.mass < 2147483648.0, MG_ERR_UNSUPPORTED,
                 "int64 precision needs integral weights with total below 2^31");
    memset(hb, 0, sizeof *hb);
    hb->state.nx = 1;
    hb->state.up = 1;
    hb->state.first = 1;
    out = ResidentResult();
    do {
        const ResidentState st = hb->state;
        memset(hb, 0, sizeof *hb);
        hb->state = st;
        hb->state.iters = 0;
        MG_CUDA(cudaMemcpyAsync(db, hb, sizeof *hb, cudaMemcpyHostToDevice, s));
        const auto launch = wk == WK_UNIT ? launch_resident_unit : wk == WK_U32 ? launch_resident_u32
                          : wk == WK_F32I ? launch_resident_f32i : wk == WK_F64I ? launch_resident_f64i
                          : wk == WK_F32 ? launch_resident_f32 : launch_resident_f64;
        if (!launch(A, p.precision, p.version, grid, s)) return false;
        MG_CUDA(cudaMemcpyAsync(hb, db, sizeof(ResidentState) + sizeof(SweepAcc) * kResidentIters,
                                cudaMemcpyDeviceToHost, s));
        MG_CUDA(cudaStreamSynchronize(s));
        if (hb->state.err) return false;
        for (int i = 0; i < hb->state.iters; i++) {
            out.Q.push_back(hb->acc[i].pad);
            out.distinct.push_back(hb->acc[i].distinct);
        }
    } while (!hb->state.done);
    out.base = hb->state.base;
    return true;
}

}  // namespace mg
