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

bool resident_level(const GraphView &g, const MoveLevel &lvl, const MoveWorkspace &ws) {
    if (ws.forced_policy || g.n == 0 || g.nnz > kResidentMaxEntries) return false;
    return std::min(lvl.bins.max_degree, g.n) <= kResidentCapacity;
}

void resident_run(mg_ctx *ctx, const GraphView &g, const MoveLevel &lvl, const SweepParams &p, double thr,
                  ResidentResult &out, cudaStream_t s) {
    MoveWorkspace &ws = ctx->mws;
    const Bins &B = lvl.bins;
    ResidentBlock *hb = (ResidentBlock *)ws.h_resident;
    if (!hb) {
        MG_CUDA(cudaMallocHost(&ws.h_resident, sizeof(ResidentBlock)));
        hb = (ResidentBlock *)ws.h_resident;
    }
    ResidentBlock *db = (ResidentBlock *)ws.resident.ensure(sizeof(ResidentBlock));
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
    // The table: as small as the level allows, since what it does not take
    // stays L1 for the community and sigma gathers.
    const uint32_t most = std::min(B.max_degree, g.n);
    A.bits = most <= 32 ? 10 : most <= 64 ? 12 : most <= 128 ? 13 : kResidentMaxBits;
    const uint32_t S = 1u << A.bits;
    auto class_of = [](uint32_t deg) {  // last class of degrees <= deg (a power of two)
        int c = 0;
        while ((1u << c) < deg) c++;
        return c;
    };
    const int cw = std::max(5, class_of(S / 64)), c128 = std::max(cw, class_of(S / 16)),
              c256 = std::max(c128, class_of(S / 8));
    auto start = [&](int c) { return c < kSweepClasses ? B.offset[c] : g.n; };
    A.cut[1] = start(cw + 1);
    A.cut[2] = start(c128 + 1);
    A.cut[3] = start(c256 + 1);
    A.cut[4] = g.n;
    A.kind_off[0] = start(6);
    A.kind_size[0] = A.cut[1] - start(6);
    for (int kd = 1; kd <= 5; kd++) {
        const int c = 6 - kd;  // classes 5, 4, 3, 2 and (one kind) 1 with 0
        const uint32_t o = kd == 5 ? 0 : start(c);
        A.kind_off[kd] = o;
        A.kind_size[kd] = start(c + 1) - o;
    }
    uint32_t tasks = 0;
    for (int kd = 0; kd < 6; kd++) {
        const uint32_t per = kd == 0 ? 1 : kTileU << (kd - 1);
        tasks += (uint32_t)ceil_div(A.kind_size[kd], per);
        A.task_end[kd] = tasks;
    }
    A.tasks = tasks;
    // CTAs: half a CTA's warps busy with a task each, or one per large vertex
    const uint64_t want = ceil_div(tasks, kResidentThreads / 64) + (A.cut[2] - A.cut[1] + 7) / 8 +
                          (A.cut[3] - A.cut[2] + 3) / 4 + (A.cut[4] - A.cut[3]);
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(want, kNumSMs));
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
        if (wk == WK_UNIT) launch_resident_unit(A, p.precision, p.version, grid, s);
        else if (wk == WK_U32) launch_resident_u32(A, p.precision, p.version, grid, s);
        else if (wk == WK_F32I) launch_resident_f32i(A, p.precision, p.version, grid, s);
        else if (wk == WK_F64I) launch_resident_f64i(A, p.precision, p.version, grid, s);
        else if (wk == WK_F32) launch_resident_f32(A, p.precision, p.version, grid, s);
        else launch_resident_f64(A, p.precision, p.version, grid, s);
        MG_CUDA(cudaMemcpyAsync(hb, db, sizeof(ResidentState) + sizeof(SweepAcc) * kResidentIters,
                                cudaMemcpyDeviceToHost, s));
        MG_CUDA(cudaStreamSynchronize(s));
        MG_CHECK(!hb->state.err, MG_ERR_TIMEOUT, "resident level: a grid barrier was not reached by every block");
        for (int i = 0; i < hb->state.iters; i++) {
            out.Q.push_back(hb->acc[i].pad);
            out.distinct.push_back(hb->acc[i].distinct);
        }
    } while (!hb->state.done);
    out.base = hb->state.base;
}

}  // namespace mg
