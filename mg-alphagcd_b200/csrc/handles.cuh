// handles.cuh -- the opaque handles behind the C ABI (mg_ctx, mg_graph,
// mg_result) and the engine entry points the ABI calls.
#pragma once

#include <cstdlib>
#include <functional>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <algorithm>
#include <vector>

#include "engine.cuh"

namespace mg {
// Host memory of a result's assignment.  A context keeps one page-locked buffer
// (at most kPinnedIds ids) that the result it is lent to gives back when it
// ends, also after the context: a copy of 64 MB into it runs at the link's
// speed, where fresh pageable memory costs its page faults and a staged copy
// (R-MAT-24: 25 of 45 ms of host time beside a run).  While it is lent out,
// further results take plain memory.
constexpr size_t kPinnedIds = 64u << 20;
struct PinnedSpare {
    std::mutex mu;
    uint32_t *p = nullptr;
    size_t cap = 0;
    // frees the buffer (unless a result holds it); returns its bytes
    size_t trim() {
        std::lock_guard<std::mutex> lk(mu);
        if (!p) return 0;
        const size_t bytes = cap * sizeof(uint32_t);
        cudaFreeHost(p);
        p = nullptr;
        cap = 0;
        return bytes;
    }
    ~PinnedSpare() { trim(); }
};
class HostIds {
public:
    HostIds() = default;
    HostIds(const HostIds &) = delete;
    HostIds &operator=(const HostIds &) = delete;
    HostIds(HostIds &&o) noexcept { swap(o); }
    HostIds &operator=(HostIds &&o) noexcept {
        swap(o);
        return *this;
    }
    ~HostIds() { release(); }
    // n uninitialised ids (plain memory without a spare buffer); does nothing
    // when they are there already
    void ensure(size_t n, const std::shared_ptr<PinnedSpare> &spare) {
        if (p_ && n_ == n) return;
        release();
        if (spare && n >= kPinnedFrom && n <= kPinnedIds) {
            std::lock_guard<std::mutex> lk(spare->mu);
            if (!lent_ok(*spare, n)) return plain(n);
            p_ = spare->p;
            cap_ = spare->cap;
            spare->p = nullptr;
            spare->cap = kLent;
            spare_ = spare;
            n_ = n;
            return;
        }
        plain(n);
    }
    uint32_t *data() { return p_; }
    const uint32_t *data() const { return p_; }
    uint32_t &operator[](size_t i) { return p_[i]; }

private:
    static constexpr size_t kPinnedFrom = 1u << 18;  // smaller copies cost less than the lending
    uint32_t *p_ = nullptr;
    size_t n_ = 0, cap_ = 0;
    std::shared_ptr<PinnedSpare> spare_;  // set: p_ is its buffer
    void swap(HostIds &o) {
        std::swap(p_, o.p_);
        std::swap(n_, o.n_);
        std::swap(cap_, o.cap_);
        spare_.swap(o.spare_);
    }
    // the spare buffer is there and large enough (made or grown here unless lent)
    static bool lent_ok(PinnedSpare &s, size_t n) {
        if (s.p && s.cap >= n) return true;
        if (!s.p && s.cap == kLent) return false;
        if (s.p) cudaFreeHost(s.p);
        s.p = nullptr;
        s.cap = 0;
        if (cudaMallocHost(&s.p, n * sizeof(uint32_t)) != cudaSuccess) {
            cudaGetLastError();  // no page-locked memory: plain memory serves
            s.p = nullptr;
            return false;
        }
        s.cap = n;
        return true;
    }
    void plain(size_t n) {
        p_ = (uint32_t *)malloc(std::max<size_t>(n, 1) * sizeof(uint32_t));
        if (!p_) throw std::bad_alloc();
        n_ = n;
    }
    void release() {
        if (spare_) {
            std::lock_guard<std::mutex> lk(spare_->mu);
            spare_->p = p_;
            spare_->cap = cap_;
        } else {
            free(p_);
        }
        spare_.reset();
        p_ = nullptr;
        n_ = cap_ = 0;
    }
    static constexpr size_t kLent = ~(size_t)0;  // PinnedSpare::cap while a result holds the buffer
};
}  // namespace mg

struct mg_ctx {
    int device = 0;
    int verbose = 0;
    size_t budget = 0;
    std::string last_error;
    mg::BufPool pool;  // (before the buffers that return to it)
    cudaStream_t stream = nullptr;
    mg::MoveWorkspace mws;
    mg::CoarsenWorkspace cws;
    // Louvain run state (grow-only, reused across runs)
    mg::DBuf<uint32_t> C[3], Cd, assign, tmp32;
    mg::DBuf<double> k, sigma;
    mg::LevelGraph lv[2];
    mg::SweepAcc *h_acc = nullptr;  // pinned
    std::shared_ptr<mg::PinnedSpare> spare = std::make_shared<mg::PinnedSpare>();
    cudaEvent_t ev[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    ~mg_ctx();
};

struct mg_graph {
    mg_ctx *ctx = nullptr;
    uint32_t n = 0;
    uint64_t nnz = 0;
    mg::DBuf<uint32_t> off, col;
    mg::DBuf<float> w32;
    mg::DBuf<double> w64;
    int wk = mg::WK_UNIT;
    double mass = 0;
    int integral = 1;
    int sorted_rows = 0;  // every row strictly increasing (no repeated neighbour)
    void attach(mg_ctx *c) {  // the context and its buffer pool
        ctx = c;
        off.pool = col.pool = &c->pool;
        w32.pool = &c->pool;
        w64.pool = &c->pool;
    }
    int symmetric = 0;    // integral and symmetric as a multiset of entries (GraphView::symmetric)
    mg::GraphView view() const {
        mg::GraphView v;
        v.n = n;
        v.nnz = nnz;
        v.off = off.get();
        v.col = col.get();
        v.wk = wk;
        v.sorted_rows = sorted_rows != 0;
        v.symmetric = symmetric != 0;
        v.w = wk == mg::WK_F32 ? (const void *)w32.get() : wk == mg::WK_F64 ? (const void *)w64.get() : nullptr;
        return v;
    }
};

struct mg_result {
    uint32_t n0 = 0;
    mg_summary sum{};
    mg::HostIds assignment;
    std::vector<uint32_t> level_sizes;
    std::vector<double> trace;  // rows of 4
    std::vector<std::vector<uint32_t>> level_maps;  // dendrogram (keep_levels)
    // the graph every level worked on (keep_levels >= 2): offsets, columns,
    // weights as double
    struct LevelCsr {
        std::vector<uint32_t> off, col;
        std::vector<double> w;
    };
    std::vector<LevelCsr> level_csr;
};

namespace mg {
// per-graph sums of one batched sweep
struct GSum {
    unsigned long long sin_u, s2_u;
    double sin_f, s2_f;
};
// device-side control block of a batched run
struct BatchCtrl {
    int up;                     // direction of the next sweep
    int active;                 // graphs taking part in the next sweep
    unsigned long long sweeps;  // sweeps run
    unsigned long long edges;   // entries of the graphs that took part in them
    long long budget;           // sweeps left in this launch (CUDA-graph loop)
    unsigned long long active_vertices;  // vertices of the graphs active in the next sweep
    unsigned long long listed;  // vertices on the active lists (set by the host)
    unsigned long long pad[2];  // pad[0]: blocks done in the decision kernel
};
// Device state of a batch, resident between runs.
struct BatchWork {
    DBuf<uint32_t> gid, goff, goff_new, goff0, gword, gnnz, loops, Cf;
    // active lists: light-class entries (class order) and vertices (id order), each
    // with the graph of every entry; double-buffered for compaction
    DBuf<uint32_t> lperm[2], lpgid[2], lvert[2], lvgid[2], flags, pos;
    DBuf<double> sinv, curQ, gmass;
    DBuf<GainK> gk;
    DBuf<unsigned long long> iters;
    DBuf<GSum> sums;
    DBuf<BatchCtrl> ctrl;
    BatchCtrl *h_ctrl = nullptr;  // pinned
    // construction and run scratch, kept so that a batch object reused for
    // the next set of graphs allocates (and frees) nothing once warm
    DBuf<uint32_t> pu, pv, small;
    DBuf<uint64_t> off64, pbase;
    DBuf<unsigned char> gen;
    DBuf<int> bad;
    DBuf<uint8_t> alive;
    // resident batch kernel: class ranges and queue order of the graphs; their
    // loop states, then totals and queue
    DBuf<uint32_t> rcls, rorder;
    DBuf<unsigned char> rstate;
    LevelGraph built;  // swapped with the union's buffers by the generator
    ~BatchWork();
};
}  // namespace mg

struct mg_batch {
    mg_ctx *ctx = nullptr;
    uint32_t graphs = 0;
    mg_graph u;                     // the packed union: rows and columns in union ids
    std::vector<uint32_t> voff;     // first vertex of each graph (graphs + 1)
    std::vector<uint64_t> eoff;     // first entry of each graph (graphs + 1)
    std::vector<double> mass;       // per graph
    std::vector<int> integral;      // per graph
    mg::BatchWork work;
};

struct mg_batch_result {
    uint32_t graphs = 0;
    mg_summary sum{};
    std::vector<mg_batch_graph_summary> per;
    std::vector<uint32_t> voff;        // first vertex of each graph
    mg::HostIds assignment;            // graph-local community of every packed vertex
};

namespace mg {

void ctx_prepare(mg_ctx *ctx);
// After a call that failed: waits for what it had queued (copies from the caller's
// page-locked arrays, kernels on buffers that are back in the pool) and forgets the
// error, which the call reports, so that no later launch check finds it.
void ctx_quiesce(mg_ctx *ctx);
// error text for entry points that run without a context (mg_last_error(NULL))
void set_orphan_error(const std::string &msg);
// graph construction
void graph_from_host_csr(mg_graph *g, uint32_t n, const uint64_t *offsets, const uint32_t *cols, const void *w,
                         int weight_type);
void graph_from_device_csr(mg_graph *g, uint32_t n, uint64_t nnz, const uint32_t *d_off, const uint32_t *d_cols,
                           const void *d_w, int weight_type);
void graph_from_level(mg_graph *g, LevelGraph &lv, int integral, double mass);
void graph_generate_rmat(mg_graph *g, int scale, int edge_factor, double a, double b, double c, uint64_t seed);
void graph_generate_sbm(mg_graph *g, uint32_t n, uint32_t blocks, double mean_degree, double intra_frac,
                        uint64_t seed);
void graph_generate_chunglu(mg_graph *g, uint32_t n, double exponent, double mean_degree, double max_degree,
                            int lognormal, uint64_t seed);
// Louvain
void louvain_run(mg_ctx *ctx, const mg_graph *g, const mg_run_opts &o, mg_result &res);
// batched form
void batch_generate(mg_batch *b, const mg_gen_params *params);
void batch_from_host_csr(mg_batch *b, const uint64_t *voff, const uint64_t *offsets, const uint32_t *cols,
                         const void *w, int weight_type);
// Called by batch_run, on its thread, as soon as graph g's result is final:
// its summary and its graph-local assignment (n_g entries).
using GraphDoneFn = std::function<void(uint32_t g, const mg_batch_graph_summary &sum, const uint32_t *assignment)>;
void batch_run(mg_batch *b, const mg_run_opts &o, int flags, mg_batch_result &res, const GraphDoneFn *done = nullptr);

}  // namespace mg
