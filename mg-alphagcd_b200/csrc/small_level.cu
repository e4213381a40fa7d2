// small_level.cu -- from one small level to the next in one block.
//
// Between two levels of a run lie the relabelling, the coarsening, the vertex
// weights and the degree classes of the new level: about 25 launches and four
// read-backs (coarsen.cu, bins.cu), 150 us however small the level is.  A level
// of at most kSmallEntries entries fits one block's shared memory and
// registers, so small_level_kernel does all of it and the host reads one block
// of counts back.  The new level is the one coarsen_level gives (rows sorted by
// neighbour community, exact integer weights of integral graphs).
#include "handles.cuh"
#include "lm_kernels.cuh"

namespace mg {

namespace {

using namespace lmk;

constexpr int kT = 1024, kWarpsS = kT / 32, kPer = 8;
constexpr uint32_t kS = kSmallEntries;
static_assert(kS == kT * kPer, "eight entries per thread");
constexpr int kRow = kWarpsS + 1;  // counters by digit and warp, padded (bank conflicts)

// shared memory: [newid | counters] [row of an entry | first entry of a run] [keys] [values | sums]
constexpr size_t kBytesA = 256 * kRow * sizeof(uint32_t), kBytesB = kS * sizeof(uint32_t);
static_assert(kBytesA >= kS * sizeof(uint32_t), "the new ids fit the counters' place");
template <class V>
constexpr size_t small_smem() {
    return kBytesA + 2 * kBytesB + (kS + 1) * sizeof(V);
}

// exclusive prefix over the block's threads; *total: the sum
template <class T>
__device__ __forceinline__ T block_prefix(T v, T *wsum, T *total) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    T incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)lane >= o) incl += y;
    }
    __syncthreads();
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    T before = 0, all = 0;
    for (uint32_t w = 0; w < kWarpsS; w++) {
        if (w < warp) before += wsum[w];
        all += wsum[w];
    }
    *total = all;
    return before + incl - v;
}

struct SmallArgs {
    uint32_t n, m;
    const uint32_t *off, *col;
    const void *w;
    const uint32_t *C;
    uint32_t *Cd;
    int coarsen;  // 0: relabel only (the run's last phase)
    uint32_t *noff, *ncol;
    void *nw;  // u32 (integral) or f64
    double *k, *sigma;
    uint32_t *C0, *perm;
    uint2 *rows;
    SmallInfo *info;
};

template <int WK>
__global__ void __launch_bounds__(kT) small_level_kernel(SmallArgs A) {
    using V = typename ValT<WK>::type;
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t *newid = (uint32_t *)smem, *cnt = newid;
    uint32_t *rowat = (uint32_t *)(smem + kBytesA);
    uint32_t *sk = (uint32_t *)(smem + kBytesA + kBytesB);
    V *sv = (V *)(smem + kBytesA + 2 * kBytesB);
    __shared__ uint32_t wsum[kWarpsS];
    __shared__ uint32_t csize[kSweepClasses], cpos[kSweepClasses], maxdeg;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    // dense ids of the used communities, in order
    for (uint32_t i = t; i < kS; i += kT) {
        newid[i] = 0;
        rowat[i] = 0;
    }
    if (t < kSweepClasses) csize[t] = 0;
    if (t == 0) maxdeg = 0;
    __syncthreads();
    for (uint32_t v = t; v < A.n; v += kT) newid[A.C[v]] = 1;
    // non-empty rows at their first entry
    for (uint32_t v = t; v < A.n; v += kT) {
        const uint32_t lo = A.off[v];
        if (lo < A.off[v + 1]) rowat[lo] = v;
    }
    __syncthreads();
    uint32_t f[kPer], sum = 0, nn;
#pragma unroll
    for (int q = 0; q < kPer; q++) {
        f[q] = newid[t * kPer + q];
        sum += f[q];
    }
    uint32_t id = block_prefix<uint32_t>(sum, wsum, &nn);
#pragma unroll
    for (int q = 0; q < kPer; q++) {
        newid[t * kPer + q] = id;
        id += f[q];
    }
    __syncthreads();
    for (uint32_t v = t; v < A.n; v += kT) A.Cd[v] = newid[A.C[v]];
    if (t == 0) {
        A.info->n = nn;
        A.info->nnz = 0;
    }
    if (!A.coarsen) return;
    // the row of every entry: prefix maximum of the marks
    uint32_t run = 0;
#pragma unroll
    for (int q = 0; q < kPer; q++) {
        run = max(run, rowat[t * kPer + q]);
        rowat[t * kPer + q] = run;
    }
    uint32_t inc = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if ((int)lane >= o) inc = max(inc, y);
    }
    if (lane == 31) wsum[warp] = inc;
    uint32_t pre = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) pre = 0;
    __syncthreads();
    for (uint32_t w = 0; w < warp; w++) pre = max(pre, wsum[w]);
#pragma unroll
    for (int q = 0; q < kPer; q++) rowat[t * kPer + q] = max(rowat[t * kPer + q], pre);
    __syncthreads();
    // keys (row community, column community) and weights; a warp holds 256
    // consecutive entries, in lane order
    const int bc = nn > 1 ? 32 - __clz(nn - 1) : 1;
    const uint32_t wbase = warp * (kPer * 32), lt = (1u << lane) - 1u;
    uint32_t key[kPer];
    V val[kPer];
#pragma unroll
    for (int r = 0; r < kPer; r++) {
        const uint32_t e = wbase + r * 32 + lane;
        key[r] = 0xffffffffu;
        val[r] = V(0);
        if (e < A.m) {
            key[r] = newid[A.C[rowat[e]]] << bc | newid[A.C[A.col[e]]];
            val[r] = wget<WK>(A.w, e);
        }
    }
    // stable sort, eight bits a pass (as the one-block sort of primitives.cu)
    for (int shift = 0; shift < 2 * bc; shift += 8) {
        __syncthreads();
        for (uint32_t d = t; d < 256 * kRow; d += kT) cnt[d] = 0;
        __syncthreads();
        uint32_t rank[kPer];
#pragma unroll
        for (int r = 0; r < kPer; r++) {
            const uint32_t e = wbase + r * 32 + lane;
            const uint32_t d = e < A.m ? (key[r] >> shift) & 0xFFu : 0x100u;
            const uint32_t peers = __match_any_sync(0xffffffffu, d);
            const uint32_t before = __popc(peers & lt);
            const uint32_t base = d < 256 ? cnt[d * kRow + warp] : 0u;
            rank[r] = base + before;
            __syncwarp();
            if (d < 256 && before == 0) cnt[d * kRow + warp] = base + __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        uint32_t *mine = cnt + (t >> 2) * kRow + (t & 3u) * 8;
        uint32_t c[8], acc = 0, all;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            c[q] = acc;
            acc += mine[q];
        }
        const uint32_t before = block_prefix<uint32_t>(acc, wsum, &all);
#pragma unroll
        for (int q = 0; q < 8; q++) mine[q] = before + c[q];
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kPer; r++) {
            const uint32_t e = wbase + r * 32 + lane;
            if (e < A.m) {
                const uint32_t pos = cnt[((key[r] >> shift) & 0xFFu) * kRow + warp] + rank[r];
                sk[pos] = key[r];
                sv[pos] = val[r];
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kPer; r++) {
            const uint32_t e = wbase + r * 32 + lane;
            if (e < A.m) {
                key[r] = sk[e];
                val[r] = sv[e];
            }
        }
    }
    __syncthreads();
    // runs of equal keys: eight consecutive entries per thread
    uint32_t prev = t ? sk[t * kPer - 1] : 0xffffffffu;
    uint32_t heads = 0;
#pragma unroll
    for (int q = 0; q < kPer; q++) {
        const uint32_t e = t * kPer + q;
        key[q] = e < A.m ? sk[e] : 0xffffffffu;
        val[q] = e < A.m ? sv[e] : V(0);
        if (e < A.m && (e == 0 || key[q] != (q ? key[q - 1] : prev))) heads++;
    }
    uint32_t nnz;
    uint32_t at = block_prefix<uint32_t>(heads, wsum, &nnz);
    __syncthreads();  // sv becomes the runs' sums
    for (uint32_t i = t; i <= kS; i += kT) sv[i] = V(0);
    __syncthreads();
    {
        // a thread adds its pieces of runs; only the first and last are shared
        uint32_t cur = at - 1u;
        V part = V(0);
        for (int q = 0; q < kPer; q++) {
            const uint32_t e = t * kPer + q;
            if (e >= A.m) break;
            const uint32_t before = q ? key[q - 1] : prev;
            if (e == 0 || key[q] != before) {
                if (q) atomicAdd(&sv[cur], part);
                cur = at++;
                part = V(0);
                A.ncol[cur] = key[q] & ((1u << bc) - 1u);
                // rows (previous entry's row, this row] start here
                const uint32_t row = key[q] >> bc;
                for (uint32_t r = e == 0 ? 0u : (before >> bc) + 1u; r <= row; r++) A.noff[r] = cur;
            }
            part += val[q];
            if (e + 1 == A.m || q + 1 == kPer) atomicAdd(&sv[cur], part);
            if (e + 1 == A.m)
                for (uint32_t r = (key[q] >> bc) + 1u; r <= nn; r++) A.noff[r] = nnz;
        }
        if (A.m == 0)
            for (uint32_t r = t; r <= nn; r += kT) A.noff[r] = 0;
    }
    __syncthreads();
    for (uint32_t i = t; i < nnz; i += kT) {
        if constexpr (kIntg<WK>) ((uint32_t *)A.nw)[i] = sv[i];
        else ((double *)A.nw)[i] = sv[i];
    }
    // the new level's start: weights, singletons, degree classes (rows of a
    // class in any order)
    for (uint32_t r = warp; r < nn; r += kWarpsS) {
        const uint32_t lo = A.noff[r], hi = A.noff[r + 1];
        V s = V(0);
        for (uint32_t i = lo + lane; i < hi; i += 32) s += sv[i];
        s = value_sum(s);
        if (lane == 0) {
            const double x = v2d(s);
            A.k[r] = x;
            A.sigma[r] = x;
            A.C0[r] = r;
            const uint32_t d = hi - lo;
            atomicAdd(&csize[d <= 1 ? 0 : 32 - __clz(d - 1)], 1u);
            atomicMax(&maxdeg, d);
        }
    }
    __syncthreads();
    if (t == 0) {
        uint32_t o = 0;
        for (int c = 0; c < kSweepClasses; c++) {
            A.info->offset[c] = cpos[c] = o;
            A.info->size[c] = csize[c];
            o += csize[c];
        }
        A.info->nnz = nnz;
        A.info->max_degree = maxdeg;
    }
    __syncthreads();
    for (uint32_t r = t; r < nn; r += kT) {
        const uint32_t lo = A.noff[r], hi = A.noff[r + 1], d = hi - lo;
        const uint32_t q = atomicAdd(&cpos[d <= 1 ? 0 : 32 - __clz(d - 1)], 1u);
        A.perm[q] = r;
        A.rows[q] = make_uint2(lo, hi);
    }
}

template <int WK>
void launch_small(const SmallArgs &A, cudaStream_t s) {
    constexpr size_t smem = small_smem<typename ValT<WK>::type>();
    raise_smem_limit((const void *)small_level_kernel<WK>, smem);
    small_level_kernel<WK><<<1, kT, smem, s>>>(A);
    MG_LAUNCH_CHECK();
}

}  // namespace

void small_level(mg_ctx *ctx, const GraphView &g, const uint32_t *C, uint32_t *Cd, bool coarsen, int integral,
                 LevelGraph &out, MoveLevel &lvl, uint32_t &n_new, cudaStream_t s) {
    MoveWorkspace &ws = ctx->mws;
    SmallInfo *d = ws.small.ensure(1);
    SmallInfo *h = (SmallInfo *)ws.prim.pinned();
    static_assert(sizeof(SmallInfo) <= kPinnedWords * sizeof(uint32_t), "the counts fit the pinned words");
    SmallArgs A = {};
    A.n = g.n;
    A.m = (uint32_t)g.nnz;
    A.off = g.off;
    A.col = g.col;
    A.w = g.w;
    A.C = C;
    A.Cd = Cd;
    A.coarsen = coarsen;
    A.info = d;
    if (coarsen) {
        A.noff = out.off.ensure((size_t)g.n + 1);
        A.ncol = out.col.ensure(g.nnz + 1);
        A.nw = integral ? (void *)out.wi.ensure(g.nnz + 1) : (void *)out.w.ensure(g.nnz + 1);
        A.k = ctx->k.get();
        A.sigma = ctx->sigma.get();
        A.C0 = ctx->C[0].get();
        A.perm = ws.perm.ensure((size_t)g.n + 1);
        A.rows = ws.rows.ensure((size_t)g.n + 1);
    }
    const int wk = integral ? (g.wk == WK_F32 ? (int)WK_F32I : g.wk == WK_F64 ? (int)WK_F64I : g.wk) : g.wk;
    if (wk == WK_UNIT) launch_small<WK_UNIT>(A, s);
    else if (wk == WK_U32) launch_small<WK_U32>(A, s);
    else if (wk == WK_F32I) launch_small<WK_F32I>(A, s);
    else if (wk == WK_F64I) launch_small<WK_F64I>(A, s);
    else if (wk == WK_F32) launch_small<WK_F32>(A, s);
    else launch_small<WK_F64>(A, s);
    MG_CUDA(cudaMemcpyAsync(h, d, sizeof *h, cudaMemcpyDeviceToHost, s));
    MG_CUDA(cudaStreamSynchronize(s));
    n_new = h->n;
    if (!coarsen) return;
    out.n = h->n;
    out.nnz = h->nnz;
    out.wk = integral ? WK_U32 : WK_F64;
    out.symmetric = g.symmetric && integral;
    lvl = MoveLevel();
    lvl.bins.scheme = kSweepScheme;
    lvl.bins.count = kSweepClasses;
    lvl.bins.max_degree = h->max_degree;
    for (int c = 0; c < kSweepClasses; c++) {
        lvl.bins.size[c] = h->size[c];
        lvl.bins.offset[c] = h->offset[c];
    }
}

}  // namespace mg
