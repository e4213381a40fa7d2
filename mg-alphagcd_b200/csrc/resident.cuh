// resident.cuh -- all iterations of a small level in one cooperative kernel.
//
// A level whose sweep takes a few tens of microseconds is bound by what lies
// between its kernels: a sweep by degree class is about ten launches on two
// streams, a read-back of the sums and a host decision, and the sigma update
// (an SBM of 65,536 vertices: 107 us per iteration, of which the edges need
// about 15).  lm_resident_kernel keeps the whole accept / reject loop of a
// level (louvain::run, src/louvain/louvain.cu:1401-1715) on the device: one
// 1,024-thread CTA per SM, a sweep over all degree classes, a grid barrier,
// the decision (taken by every CTA from the same sums), the sigma update, a
// second barrier.  The per-vertex arithmetic is the sweep kernels'
// (lm_kernels.cuh): the same candidates, the same gain expression and the
// same total order, so results are equal bit for bit on integral weights.
//
// Work split inside a sweep, by the level's degree classes (bins.cu):
//   degree <= 32         T-lane tiles, two steps in flight per warp
//   degree <= S/64       a warp per vertex, table of S/32 slots
//   degree <= S/16       128 threads per vertex, table of S/8 slots
//   degree <= S/8        256 threads per vertex, table of S/4 slots
//   larger               the CTA per vertex, table of S slots at load <= 2/3
// The tables are nested slices of one shared-memory region (a warp's slice
// lies in its group's, a group's in the CTA's) and every vertex leaves its
// slots empty, so a group moves on to the next kind of work without a CTA
// barrier.  Tiles and warp vertices are taken from a counter (the next task is
// fetched while the current one runs), so CTAs that hold large vertices do
// not hold up the rest.
#pragma once

#include "lm_kernels.cuh"
#include "resident_args.cuh"

namespace mg {
namespace lmr {

using namespace lmk;

constexpr int kThreads = kResidentThreads;
constexpr int kWarps = kThreads / 32;

template <int GT>
__device__ __forceinline__ void bar_group() {
    if constexpr (GT == 32) {
        __syncwarp();
    } else if constexpr (GT == kThreads) {
        __syncthreads();
    } else {
        // named barriers 1..8 (groups of 128) and 9..12 (groups of 256)
        const int id = (GT == 128 ? 1 : 9) + (int)(threadIdx.x / GT);
        asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(GT) : "memory");
    }
}

template <class V, class G>
struct Shared {
    // sums of a group's vertex, double-buffered by the parity of the vertex
    V acc_e[2][8], acc_s[2][8];
    uint32_t cnt[2][8];
    G red_g[kWarps];
    uint32_t red_c[kWarps];
    V wbuf[kWarps][32];
    double red_sin[kWarps];
    unsigned long long red_d[kWarps], red_u[kWarps];
    double red_f[kWarps];
    ResidentState st;  // the loop's state, the same in every CTA
    int ok;
};

// ---- degree <= 32: T lanes per vertex, U warp steps in flight ----------------
template <int T, int U, int WK, int PREC, int VER, class SH>
__device__ __forceinline__ void tile_task(const ResidentArgs &A, const uint32_t *P, uint32_t *N, uint32_t q0,
                                          uint32_t q1, int up, double &sin, unsigned &dcnt, SH &sh) {
    using G = typename Prec<PREC>::G;
    using V = typename ValT<WK>::type;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t gl = lane & (T - 1), gbase = lane & ~(uint32_t)(T - 1);
    const uint32_t gmask = T == 32 ? 0xffffffffu : (((1u << T) - 1u) << gbase);
    constexpr uint32_t GPW = 32 / T;
    uint32_t i[U], src[U], j[U], c[U];
    V w[U];
    double ki[U], a[U];
    bool act[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        const uint32_t q = q0 + u * GPW + lane / T;
        act[u] = q < q1;
        i[u] = act[u] ? A.perm[q] : 0u;
        const uint2 r = act[u] ? A.rows[q] : make_uint2(0, 0);
        const uint32_t e = r.x + gl;
        const bool has = act[u] && e < r.y;
        j[u] = has ? __ldg(A.col + e) : kEmpty;
        w[u] = has ? wget<WK>(A.w, e) : V(0);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        src[u] = act[u] ? P[i[u]] : 0u;
        c[u] = j[u] != kEmpty ? P[j[u]] : kEmpty;
        ki[u] = act[u] ? A.k[i[u]] : 0.0;
    }
    double sc[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        a[u] = act[u] ? A.sigma[src[u]] - ki[u] : 0.0;
        const bool cand = j[u] != kEmpty && c[u] != src[u] && is_candidate<VER>(c[u], src[u], up);
        sc[u] = cand ? A.sigma[c[u]] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const bool has = j[u] != kEmpty;
        const bool self = has && j[u] == i[u];
        const bool inner = has && !self && c[u] == src[u];
        const bool cand = has && c[u] != src[u] && is_candidate<VER>(c[u], src[u], up);
        const uint32_t peers = __match_any_sync(0xffffffffu, cand ? c[u] : kEmpty) & gmask;
        const bool leader = cand && (uint32_t)(__ffs(peers) - 1) == lane;
        double kic, e_src, selfw;
        if constexpr (WK == WK_UNIT) {
            kic = u2d(__popc(peers));
            e_src = u2d(__popc(__ballot_sync(0xffffffffu, inner) & gmask));
            selfw = u2d(__popc(__ballot_sync(0xffffffffu, self) & gmask));
        } else {
            sh.wbuf[warp][lane] = w[u];
            __syncwarp();
            V ks = V(0);
            if (leader)
                for (uint32_t mset = peers; mset; mset &= mset - 1) ks += sh.wbuf[warp][__ffs(mset) - 1];
            __syncwarp();
            V es = inner ? w[u] : V(0), ss = self ? w[u] : V(0);
            if constexpr (T == 32) {
                es = value_sum(es);
                ss = value_sum(ss);
            } else {
#pragma unroll
                for (int o = T / 2; o > 0; o >>= 1) {
                    es += __shfl_xor_sync(0xffffffffu, es, o);
                    ss += __shfl_xor_sync(0xffffffffu, ss, o);
                }
            }
            kic = v2d(ks);
            e_src = v2d(es);
            selfw = v2d(ss);
        }
        G best = G(0);
        uint32_t dst = src[u];
        if (leader) {
            const G g = Prec<PREC>::gain(kic, e_src, ki[u], a[u], sc[u], A.K);
            if (better(g, c[u], best, dst, up)) {
                best = g;
                dst = c[u];
            }
            dcnt++;
        }
        tile_argmax<T>(best, dst, up);
        if (act[u] && gl == 0) {
            N[i[u]] = final_choice<VER>(dst, src[u], up);
            sin += e_src + selfw;
        }
    }
}

// ---- GT threads per vertex, shared-memory table of at most 2^bits slots ------
// DENSE (the CTA's table): no insertion list, the evaluation scans the slots.
template <int GT, int WK, int PREC, int VER, bool DENSE, class SH>
__device__ __forceinline__ void hash_vertex(const ResidentArgs &A, const uint32_t *P, uint32_t *N, uint32_t q, int up,
                                            int agg, uint32_t *keys, typename ValT<WK>::type *vals, uint16_t *used,
                                            int max_bits, int &par, double &sin, unsigned &dcnt, SH &sh) {
    using G = typename Prec<PREC>::G;
    using V = typename ValT<WK>::type;
    constexpr int BATCH = 4, EB = 4;
    const uint32_t lane = threadIdx.x & 31u, t = threadIdx.x % GT;
    const int g = threadIdx.x / GT;
    const uint32_t i = A.perm[q];
    const uint2 row = A.rows[q];
    const uint32_t lo = row.x, hi = row.y;
    const uint32_t src = P[i];
    const double ki = A.k[i];
    const int tb = table_bits(hi - lo, max_bits);
    const uint32_t mask = (1u << tb) - 1u;
    V e_part = V(0), s_part = V(0);
    uint32_t nw = 0;  // GT == 32: candidates listed so far (uniform in the warp)
    auto insert = [&](uint32_t key, V val) {
        uint32_t hnew = kEmpty;
        if (key != kEmpty) {
            uint32_t h = hash_slot(key, tb);
            for (uint32_t p = 0; p <= mask; p++) {
                const uint32_t prev = atomicCAS(keys + h, kEmpty, key);
                if (prev == kEmpty) {
                    hnew = h;
                    break;
                }
                if (prev == key) break;
                h = (h + 1) & mask;
            }
            atomicAdd(vals + h, val);
        }
        if constexpr (!DENSE) {
            const uint32_t m = __ballot_sync(0xffffffffu, hnew != kEmpty);
            if (m) {
                uint32_t pos;
                if constexpr (GT == 32) {
                    pos = nw;
                    nw += __popc(m);
                } else {
                    const uint32_t leader = __ffs(m) - 1;
                    pos = 0;
                    if (lane == leader) pos = atomicAdd(&sh.cnt[par][g], (uint32_t)__popc(m));
                    pos = __shfl_sync(0xffffffffu, pos, leader);
                }
                if (hnew != kEmpty) used[pos + __popc(m & ((1u << lane) - 1u))] = (uint16_t)hnew;
            }
        }
    };
    uint32_t rk = kEmpty;  // run combining, as in the sweep kernels
    V rs = V(0);
    for (uint32_t wbase = lo + (t & ~31u); wbase < hi; wbase += GT * BATCH) {  // warp-uniform
        const uint32_t base = wbase + lane;
        uint32_t jj[BATCH], cc[BATCH];
        V ww[BATCH];
#pragma unroll
        for (int b = 0; b < BATCH; b++) {
            const uint32_t e = base + b * GT;
            jj[b] = e < hi ? __ldg(A.col + e) : kEmpty;
            ww[b] = e < hi ? wget<WK>(A.w, e) : V(0);
        }
#pragma unroll
        for (int b = 0; b < BATCH; b++) cc[b] = jj[b] != kEmpty ? P[jj[b]] : kEmpty;
#pragma unroll
        for (int b = 0; b < BATCH; b++) {
            if (wbase + b * GT >= hi) break;
            const uint32_t c = cc[b];
            const bool cand = jj[b] != kEmpty && c != src && is_candidate<VER>(c, src, up);
            if (agg) {
                const bool same = cand && c == rk;
                const uint32_t fk = cand && !same ? rk : kEmpty;
                const V fv = rs;
                if (cand) {
                    rs = same ? rs + ww[b] : ww[b];
                    rk = c;
                }
                insert(fk, fv);
            } else {
                insert(cand ? c : kEmpty, ww[b]);
            }
            if (jj[b] != kEmpty && c == src) {
                if (jj[b] != i) e_part += ww[b];
                else s_part += ww[b];
            }
        }
    }
    if (agg) insert(rk, rs);
    e_part = value_sum(e_part);
    s_part = value_sum(s_part);
    if constexpr (GT > 32) {
        if (lane == 0) {
            if (e_part != V(0)) atomicAdd(&sh.acc_e[par][g], e_part);
            if (s_part != V(0)) atomicAdd(&sh.acc_s[par][g], s_part);
        }
    }
    bar_group<GT>();
    const double a = A.sigma[src] - ki;
    double e_src, selfw;
    uint32_t nd;
    if constexpr (GT == 32) {
        e_src = v2d(e_part);
        selfw = v2d(s_part);
        nd = nw;
    } else {
        e_src = v2d(sh.acc_e[par][g]);
        selfw = v2d(sh.acc_s[par][g]);
        nd = DENSE ? mask + 1u : sh.cnt[par][g];
    }
    G best = G(0);
    uint32_t dst = src;
    for (uint32_t ub = t & ~31u; ub < nd; ub += GT * EB) {  // warp-uniform
        uint32_t kk[EB];
        double sc[EB], kv[EB];
#pragma unroll
        for (int b = 0; b < EB; b++) {
            kk[b] = kEmpty;
            if (ub + b * GT >= nd) break;
            const uint32_t u = ub + lane + b * GT;
            if (u < nd) {
                const uint32_t h = DENSE ? u : used[u];
                kk[b] = keys[h];
                if (!DENSE || kk[b] != kEmpty) {
                    kv[b] = v2d(vals[h]);
                    keys[h] = kEmpty;
                    vals[h] = V(0);
                    if (DENSE) dcnt++;
                }
            }
        }
#pragma unroll
        for (int b = 0; b < EB; b++) {
            if (ub + b * GT >= nd) break;
            if (kk[b] != kEmpty) sc[b] = A.sigma[kk[b]];
        }
#pragma unroll
        for (int b = 0; b < EB; b++) {
            if (ub + b * GT >= nd) break;
            if (kk[b] != kEmpty) {
                const G gn = Prec<PREC>::gain(kv[b], e_src, ki, a, sc[b], A.K);
                if (better(gn, kk[b], best, dst, up)) {
                    best = gn;
                    dst = kk[b];
                }
            }
        }
    }
    warp_argmax(best, dst, up);
    if constexpr (GT > 32) {
        const int warp = threadIdx.x >> 5;
        if (lane == 0) {
            sh.red_g[warp] = best;
            sh.red_c[warp] = dst;
        }
        bar_group<GT>();
        if (t == 0) {
            for (int w2 = 1; w2 < GT / 32; w2++)
                if (better(sh.red_g[warp + w2], sh.red_c[warp + w2], best, dst, up)) {
                    best = sh.red_g[warp + w2];
                    dst = sh.red_c[warp + w2];
                }
        }
    }
    if (t == 0) {
        N[i] = final_choice<VER>(dst, src, up);
        sin += e_src + selfw;
        if (!DENSE) dcnt += nd;
        if constexpr (GT > 32) {
            // used again two vertices on, after at least one more barrier
            sh.cnt[par][g] = 0;
            sh.acc_e[par][g] = V(0);
            sh.acc_s[par][g] = V(0);
        }
    }
    if constexpr (GT == 32) __syncwarp();
    par ^= 1;
}

// Grid barrier (cooperative launch: all CTAs are resident).  The counter only
// grows; `target` is the count that completes this barrier.  Thread 0 gives up
// after kBarrierSpins polls (seconds), which ends the kernel with an error.
__device__ __forceinline__ bool grid_wait(unsigned *ctr, unsigned target) {
    __threadfence();
    atomicAdd(ctr, 1u);
    for (unsigned spin = 0; spin < kBarrierSpins; spin++) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
        if (v >= target) {
            __threadfence();
            return true;
        }
    }
    return false;
}

template <int WK, int PREC, int VER>
__global__ void __launch_bounds__(kThreads, 1) lm_resident_kernel(ResidentArgs A) {
    using G = typename Prec<PREC>::G;
    using V = typename ValT<WK>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ Shared<V, G> sh;
    const uint32_t S = 1u << A.bits;
    V *vals = (V *)smem_raw;
    uint32_t *keys = (uint32_t *)(smem_raw + sizeof(V) * S);
    uint16_t *used = (uint16_t *)(smem_raw + (sizeof(V) + sizeof(uint32_t)) * S);
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    for (uint32_t s = t; s < S; s += kThreads) {
        keys[s] = kEmpty;
        vals[s] = V(0);
    }
    if (t < 16) {
        (&sh.cnt[0][0])[t] = 0;
        (&sh.acc_e[0][0])[t] = V(0);
        (&sh.acc_s[0][0])[t] = V(0);
    }
    if (t == 0) sh.st = *A.state;
    __syncthreads();
    unsigned bar = 0;  // barriers passed
    const uint32_t gthreads = gridDim.x * kThreads, gt = blockIdx.x * kThreads + t;
    const uint32_t gwarps = gridDim.x * kWarps;
    for (int it = 0; it < kResidentIters; it++) {
        SweepAcc *acc = A.acc + it;
        const uint32_t *P = A.C[sh.st.p];
        uint32_t *N = A.C[sh.st.nx];
        const int up = sh.st.up;
        const int agg = !sh.st.first && 2 * sh.st.distinct < A.nnz;
        double sin = 0;
        unsigned dcnt = 0;
        int par = 0;
        // the CTA per vertex, largest degrees first
        for (uint32_t q = A.cut[3] + blockIdx.x; q < A.cut[4]; q += gridDim.x)
            hash_vertex<kThreads, WK, PREC, VER, true>(A, P, N, A.cut[4] - 1 - (q - A.cut[3]), up, agg, keys, vals,
                                                       used, A.bits, par, sin, dcnt, sh);
        __syncthreads();  // the groups below reuse the sums of group 0
        {
            const uint32_t g = t / 256;
            const uint32_t sl = S / 4 * g;
            par = 0;
            for (uint32_t q = A.cut[2] + blockIdx.x * 4 + g; q < A.cut[3]; q += gridDim.x * 4)
                hash_vertex<256, WK, PREC, VER, false>(A, P, N, A.cut[3] - 1 - (q - A.cut[2]), up, agg, keys + sl,
                                                       vals + sl, used + sl / 2, A.bits - 2, par, sin, dcnt, sh);
        }
        __syncthreads();
        {
            const uint32_t g = t / 128;
            const uint32_t sl = S / 8 * g;
            par = 0;
            for (uint32_t q = A.cut[1] + blockIdx.x * 8 + g; q < A.cut[2]; q += gridDim.x * 8)
                hash_vertex<128, WK, PREC, VER, false>(A, P, N, A.cut[2] - 1 - (q - A.cut[1]), up, agg, keys + sl,
                                                       vals + sl, used + sl / 2, A.bits - 3, par, sin, dcnt, sh);
        }
        // warp vertices and tiles, by task
        {
            const uint32_t sl = S / 32 * warp;
            uint32_t task = blockIdx.x * kWarps + warp;
            while (task < A.tasks) {
                uint32_t nxt = 0;
                if (lane == 0) nxt = gwarps + atomicAdd(A.task_ctr + it, 1u);
                int kind = 0;  // 0: warp vertices, 1..5: tiles of 32, 16, 8, 4, 2 lanes
                while (kind < 5 && task >= A.task_end[kind]) kind++;
                const uint32_t k0 = task - (kind ? A.task_end[kind - 1] : 0u);
                const uint32_t q0 = A.kind_off[kind], q1 = A.kind_off[kind] + A.kind_size[kind];
                if (kind == 0)
                    hash_vertex<32, WK, PREC, VER, false>(A, P, N, q1 - 1 - k0, up, agg, keys + sl, vals + sl,
                                                          used + sl / 2, A.bits - 5, par, sin, dcnt, sh);
                else if (kind == 1)
                    tile_task<32, kTileU, WK, PREC, VER>(A, P, N, q0 + k0 * kTileU, q1, up, sin, dcnt, sh);
                else if (kind == 2)
                    tile_task<16, kTileU, WK, PREC, VER>(A, P, N, q0 + k0 * 2 * kTileU, q1, up, sin, dcnt, sh);
                else if (kind == 3)
                    tile_task<8, kTileU, WK, PREC, VER>(A, P, N, q0 + k0 * 4 * kTileU, q1, up, sin, dcnt, sh);
                else if (kind == 4)
                    tile_task<4, kTileU, WK, PREC, VER>(A, P, N, q0 + k0 * 8 * kTileU, q1, up, sin, dcnt, sh);
                else
                    tile_task<2, kTileU, WK, PREC, VER>(A, P, N, q0 + k0 * 16 * kTileU, q1, up, sin, dcnt, sh);
                task = __shfl_sync(0xffffffffu, nxt, 0);
            }
        }
        // sum of sigma^2 of P's communities
        unsigned long long su = 0;
        double sf = 0;
        for (uint32_t c = gt; c < A.n; c += gthreads) {
            const double s = A.sigma[c];
            if (A.integral) {
                const unsigned long long u = (unsigned long long)s;
                su += u * u;
            } else {
                sf += s * s;
            }
        }
        sin = warp_sum(sin);
        const unsigned long long dw = warp_sum((unsigned long long)dcnt);
        su = warp_sum(su);
        sf = warp_sum(sf);
        if (lane == 0) {
            sh.red_sin[warp] = sin;
            sh.red_d[warp] = dw;
            sh.red_u[warp] = su;
            sh.red_f[warp] = sf;
        }
        __syncthreads();
        if (warp == 0) {
            const double bs = warp_sum(lane < kWarps ? sh.red_sin[lane] : 0.0);
            const unsigned long long bd = warp_sum(lane < kWarps ? sh.red_d[lane] : 0ull);
            const unsigned long long bu = warp_sum(lane < kWarps ? sh.red_u[lane] : 0ull);
            const double bf = warp_sum(lane < kWarps ? sh.red_f[lane] : 0.0);
            if (lane == 0) {
                if (A.integral) {
                    if (bs != 0) atomicAdd(&acc->sin_u, (unsigned long long)bs);
                    if (bu) atomicAdd(&acc->s2_u, bu);
                } else {
                    if (bs != 0) atomicAdd(&acc->sin_f, bs);
                    if (bf != 0) atomicAdd(&acc->s2_f, bf);
                }
                if (bd) atomicAdd(&acc->distinct, bd);
                bar++;
                const bool ok = grid_wait(A.barrier, bar * gridDim.x);
                sh.ok = ok;
                // Q(P), the host's operations each rounded as written
                const double x = A.integral ? __ull2double_rn(__ldcg(&acc->sin_u)) : __ldcg(&acc->sin_f);
                const double y = A.integral ? __ull2double_rn(__ldcg(&acc->s2_u)) : __ldcg(&acc->s2_f);
                const double Q = __dsub_rn(__ddiv_rn(x, A.mass), __ddiv_rn(y, __dmul_rn(A.mass, A.mass)));
                if (blockIdx.x == 0) acc->pad = Q;
                ResidentState st = sh.st;
                st.distinct = __ldcg(&acc->distinct);
                st.iters++;
                if (st.first || __dsub_rn(Q, st.curQ) > A.thr) {
                    // the move P -> N is taken; N is swept next
                    const int after = 3 - st.p - st.nx;
                    st.curQ = Q;
                    st.base = st.p;
                    st.p = st.nx;
                    st.nx = after;
                    st.up ^= 1;
                    st.first = 0;
                } else {
                    st.done = 1;
                }
                sh.st = st;
            }
        }
        __syncthreads();
        if (!sh.ok) {
            if (t == 0) A.state->err = 1;
            return;
        }
        if (sh.st.done) break;
        for (uint32_t v = gt; v < A.n; v += gthreads) {
            const uint32_t x = P[v], y = N[v];
            if (x != y) {
                const double kv = A.k[v];
                atomicAdd(A.sigma + x, -kv);
                atomicAdd(A.sigma + y, kv);
            }
        }
        __syncthreads();
        if (t == 0) {
            bar++;
            sh.ok = grid_wait(A.barrier, bar * gridDim.x);
        }
        __syncthreads();
        if (!sh.ok) {
            if (t == 0) A.state->err = 1;
            return;
        }
    }
    // every CTA holds the same state; all read theirs before the first barrier
    if (blockIdx.x == 0 && t == 0) *A.state = sh.st;
}

template <int WK>
size_t resident_smem(int bits) {
    return ((size_t)1 << bits) * (sizeof(typename ValT<WK>::type) + sizeof(uint32_t) + 1);
}

template <int WK, int PREC, int VER>
void launch_resident(const ResidentArgs &A, unsigned grid, cudaStream_t s) {
    auto kern = lm_resident_kernel<WK, PREC, VER>;
    raise_smem_limit((const void *)kern, resident_smem<WK>(kResidentMaxBits));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = resident_smem<WK>(A.bits);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    MG_CUDA(cudaLaunchKernelEx(&cfg, kern, A));
    MG_LAUNCH_CHECK();
}

template <int WK>
void launch_resident_kind(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s) {
    auto version = [&](auto precc) {
        constexpr int PREC = decltype(precc)::value;
        if (ver == 1) launch_resident<WK, PREC, 1>(A, grid, s);
        else launch_resident<WK, PREC, 2>(A, grid, s);
    };
    if (prec == MG_PREC_FP64) {
        version(std::integral_constant<int, MG_PREC_FP64>());
        return;
    }
    if (prec == MG_PREC_FP32) {
        version(std::integral_constant<int, MG_PREC_FP32>());
        return;
    }
    if constexpr (kIntg<WK>) {
        if (prec == MG_PREC_INT64) {
            version(std::integral_constant<int, MG_PREC_INT64>());
            return;
        }
    }
    throw Error(MG_ERR_INVALID, "unknown weight kind or precision");
}

}  // namespace lmr
}  // namespace mg
