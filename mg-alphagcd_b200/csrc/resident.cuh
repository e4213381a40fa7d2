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
//   larger               the CTA per vertex, table of S slots at load <= 7/8
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
    ResidentState st;  // the loop's state, the same in every CTA of the team
    int ok;
    // the graph's part of the class list: vertices [beg[c], end[c]) per degree
    // class, and the warp tasks of classes cw .. 0, cumulative
    uint32_t beg[kSweepClasses], end[kSweepClasses];
    uint32_t task_end[kSweepClasses];
    uint32_t chunk;  // tasks taken at a time
};

// Last classes whose vertices fit a warp's, 128 threads' and 256 threads' part
// of a table of 2^bits slots (2 * degree slots); tiles serve classes 0-5.
__device__ __forceinline__ int class_warp(int bits) { return max(5, bits - 6); }
__device__ __forceinline__ int class_128(int bits) { return max(class_warp(bits), bits - 4); }
__device__ __forceinline__ int class_256(int bits) { return max(class_warp(bits), bits - 3); }

// Task counts of the warp stage from the class ranges (one thread), for a team
// of `size` CTAs.  A warp takes up to 16 tasks with one atomic, an eighth of its
// share: with one task each, the counter's address was the limit of a sweep
// (1.5 atomics per ns; SBM of 4.0 M entries 72 us a sweep, 60 us with chunks).
template <class SH>
__device__ __forceinline__ void count_tasks(SH &sh, int bits, uint32_t size) {
    uint32_t sum = 0;
    const int cw = class_warp(bits);
    for (int i = 0; i <= cw; i++) {
        const int c = cw - i;
        const uint32_t m = sh.end[c] - sh.beg[c];
        const uint32_t per = c > 5 ? 1u : kTileU << (c == 0 ? 4 : 5 - c);
        sum += (m + per - 1) / per;
        sh.task_end[i] = sum;
    }
    sh.chunk = max(1u, min(16u, sum / (size * kWarps * 8)));
}


// ---- degree <= 32: T lanes per vertex, U warp steps in flight ----------------
template <int T, int U, int WK, int PREC, int VER, class AV, class SH>
__device__ __forceinline__ void tile_task(const AV &A, const uint32_t *P, uint32_t *N, uint32_t q0,
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
template <int GT, int WK, int PREC, int VER, bool DENSE, class AV, class SH>
__device__ __forceinline__ void hash_vertex(const AV &A, const uint32_t *P, uint32_t *N, uint32_t q, int up,
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
// after `polls` polls (seconds), which ends the kernel with an error: blocks of
// the launch may not have started, held back by other work on the device.
__device__ __forceinline__ bool grid_wait(unsigned *ctr, unsigned target, unsigned polls) {
    __threadfence();
    atomicAdd(ctr, 1u);
    for (unsigned spin = 0; spin < polls; spin++) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
        if (v >= target) {
            __threadfence();
            return true;
        }
    }
    return false;
}

// The vertices of classes [c0, c1], largest first, that fall to group `x` of
// `groups`; f(q) works entry q of the class list.
template <class SH, class F>
__device__ __forceinline__ void each_vertex(const SH &sh, int c0, int c1, uint32_t x, uint32_t groups, F f) {
    for (int c = c1; c >= c0; c--) {
        const uint32_t m = sh.end[c] - sh.beg[c];
        for (; x < m; x += groups) f(sh.end[c] - 1 - x);
        x -= m;
    }
}

// One sweep of a graph by a team of CTAs (this one is `rank` of `size`): the
// vertices of its class ranges, P -> N.  grab() hands out the next warp task.
template <int WK, int PREC, int VER, class AV, class SH, class Grab>
__device__ __forceinline__ void team_sweep(const AV &A, const uint32_t *P, uint32_t *N, int up, int agg, int bits,
                                           uint32_t rank, uint32_t size, uint32_t *keys,
                                           typename ValT<WK>::type *vals, uint16_t *used, double &sin, unsigned &dcnt,
                                           SH &sh, Grab grab) {
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    const uint32_t S = 1u << bits;
    const int cw = class_warp(bits), c128 = class_128(bits), c256 = class_256(bits);
    int par = 0;
    // the CTA per vertex
    each_vertex(sh, c256 + 1, kSweepClasses - 1, rank, size, [&](uint32_t q) {
        hash_vertex<kThreads, WK, PREC, VER, true>(A, P, N, q, up, agg, keys, vals, used, bits, par, sin, dcnt, sh);
    });
    __syncthreads();  // the groups below reuse the sums of group 0
    {
        const uint32_t g = t / 256, sl = S / 4 * g;
        par = 0;
        each_vertex(sh, c128 + 1, c256, rank * 4 + g, size * 4, [&](uint32_t q) {
            hash_vertex<256, WK, PREC, VER, false>(A, P, N, q, up, agg, keys + sl, vals + sl, used + sl / 2, bits - 2,
                                                   par, sin, dcnt, sh);
        });
    }
    __syncthreads();
    {
        const uint32_t g = t / 128, sl = S / 8 * g;
        par = 0;
        each_vertex(sh, cw + 1, c128, rank * 8 + g, size * 8, [&](uint32_t q) {
            hash_vertex<128, WK, PREC, VER, false>(A, P, N, q, up, agg, keys + sl, vals + sl, used + sl / 2, bits - 3,
                                                   par, sin, dcnt, sh);
        });
    }
    // warp vertices and tiles, by task
    const uint32_t sl = S / 32 * warp, tasks = sh.task_end[cw];
    const uint32_t ch = sh.chunk;
    uint32_t k = rank * kWarps + warp;  // chunk of tasks
    while (k * ch < tasks) {
        uint32_t nxt = 0;
        if (lane == 0) nxt = size * kWarps + grab();
        const uint32_t t1 = min(tasks, (k + 1) * ch);
        for (uint32_t task = k * ch; task < t1; task++) {
            int i = 0;
            while (task >= sh.task_end[i]) i++;
            const int c = cw - i;
            const uint32_t k0 = task - (i ? sh.task_end[i - 1] : 0u);
            const uint32_t q0 = sh.beg[c], q1 = sh.end[c];
            if (c > 5)
                hash_vertex<32, WK, PREC, VER, false>(A, P, N, q1 - 1 - k0, up, agg, keys + sl, vals + sl,
                                                      used + sl / 2, bits - 5, par, sin, dcnt, sh);
            else if (c == 5)
                tile_task<32, kTileU, WK, PREC, VER>(A, P, N, q0 + k0 * kTileU, q1, up, sin, dcnt, sh);
            else if (c == 4)
                tile_task<16, kTileU, WK, PREC, VER>(A, P, N, q0 + k0 * 2 * kTileU, q1, up, sin, dcnt, sh);
            else if (c == 3)
                tile_task<8, kTileU, WK, PREC, VER>(A, P, N, q0 + k0 * 4 * kTileU, q1, up, sin, dcnt, sh);
            else if (c == 2)
                tile_task<4, kTileU, WK, PREC, VER>(A, P, N, q0 + k0 * 8 * kTileU, q1, up, sin, dcnt, sh);
            else
                tile_task<2, kTileU, WK, PREC, VER>(A, P, N, q0 + k0 * 16 * kTileU, q1, up, sin, dcnt, sh);
        }
        k = __shfl_sync(0xffffffffu, nxt, 0);
    }
}

// sum of sigma^2 over the communities [c0, c1), a thread's part
__device__ __forceinline__ void sigma_sq(const double *sigma, uint32_t c0, uint32_t c1, uint32_t step, int integral,
                                         unsigned long long &su, double &sf) {
    for (uint64_t c = c0; c < c1; c += step) {
        const double s = sigma[c];
        if (integral) {
            const unsigned long long u = (unsigned long long)s;
            su += u * u;
        } else {
            sf += s * s;
        }
    }
}

// A thread's parts of a sweep's sums, added up over the CTA: valid in thread 0.
struct SweepSums {
    double sin;
    unsigned long long distinct, s2_u;
    double s2_f;
};
template <class SH>
__device__ __forceinline__ SweepSums cta_sums(double sin, unsigned dcnt, unsigned long long su, double sf, SH &sh) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
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
    SweepSums r = {0, 0, 0, 0};
    if (warp == 0) {
        r.sin = warp_sum(sh.red_sin[lane]);
        r.distinct = warp_sum(sh.red_d[lane]);
        r.s2_u = warp_sum(sh.red_u[lane]);
        r.s2_f = warp_sum(sh.red_f[lane]);
    }
    return r;
}

// Q of a sweep's input assignment, the host's operations each rounded as written
__device__ __forceinline__ double sweep_q(double sin, double s2, double mass) {
    return __dsub_rn(__ddiv_rn(sin, mass), __ddiv_rn(s2, __dmul_rn(mass, mass)));
}

// The accept / reject step after a sweep with Q(P) = Q.
__device__ __forceinline__ void next_state(ResidentState &st, double Q, unsigned long long distinct, double thr) {
    st.distinct = distinct;
    st.iters++;
    if (st.first || __dsub_rn(Q, st.curQ) > thr) {
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
}

// sigma follows the move P -> N of the vertices [v0, v1)
template <class AV>
__device__ __forceinline__ void move_sigma(const AV &A, const uint32_t *P, const uint32_t *N, uint32_t v0, uint32_t v1,
                                           uint32_t step) {
    for (uint64_t v = v0; v < v1; v += step) {
        const uint32_t x = P[v], y = N[v];
        if (x != y) {
            const double kv = A.k[v];
            atomicAdd(A.sigma + x, -kv);
            atomicAdd(A.sigma + y, kv);
        }
    }
}

// empty table, zero sums
template <class V, class SH>
__device__ __forceinline__ void clear_tables(uint32_t *keys, V *vals, uint32_t S, SH &sh) {
    for (uint32_t s = threadIdx.x; s < S; s += kThreads) {
        keys[s] = kEmpty;
        vals[s] = V(0);
    }
    if (threadIdx.x < 16) {
        (&sh.cnt[0][0])[threadIdx.x] = 0;
        (&sh.acc_e[0][0])[threadIdx.x] = V(0);
        (&sh.acc_s[0][0])[threadIdx.x] = V(0);
    }
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
    const uint32_t t = threadIdx.x;
    clear_tables(keys, vals, S, sh);
    if (t < kSweepClasses) {
        sh.beg[t] = A.cls[t];
        sh.end[t] = A.cls[t + 1];
    }
    if (t == 0) sh.st = *A.state;
    __syncthreads();
    if (t == 0) count_tasks(sh, A.bits, gridDim.x);
    __syncthreads();
    unsigned bar = 0;  // barriers passed (thread 0)
    const uint32_t gthreads = gridDim.x * kThreads, gt = blockIdx.x * kThreads + t;
    for (int it = 0; it < A.sweeps; it++) {
        SweepAcc *acc = A.acc + it;
        const uint32_t *P = A.C[sh.st.p];
        uint32_t *N = A.C[sh.st.nx];
        double sin = 0, sf = 0;
        unsigned dcnt = 0;
        unsigned long long su = 0;
        team_sweep<WK, PREC, VER>(A, P, N, sh.st.up, !sh.st.first && 2 * sh.st.distinct < A.nnz, A.bits, blockIdx.x,
                                  gridDim.x, keys, vals, used, sin, dcnt, sh,
                                  [&] { return atomicAdd(A.task_ctr + it, 1u); });
        sigma_sq(A.sigma, gt, A.n, gthreads, A.integral, su, sf);
        const SweepSums r = cta_sums(sin, dcnt, su, sf, sh);
        if (t == 0) {
            if (A.integral) {
                if (r.sin != 0) atomicAdd(&acc->sin_u, (unsigned long long)r.sin);
                if (r.s2_u) atomicAdd(&acc->s2_u, r.s2_u);
            } else {
                if (r.sin != 0) atomicAdd(&acc->sin_f, r.sin);
                if (r.s2_f != 0) atomicAdd(&acc->s2_f, r.s2_f);
            }
            if (r.distinct) atomicAdd(&acc->distinct, r.distinct);
            bar++;
            sh.ok = grid_wait(A.barrier, bar * gridDim.x, A.polls);
            const double x = A.integral ? __ull2double_rn(__ldcg(&acc->sin_u)) : __ldcg(&acc->sin_f);
            const double y = A.integral ? __ull2double_rn(__ldcg(&acc->s2_u)) : __ldcg(&acc->s2_f);
            const double Q = sweep_q(x, y, A.mass);
            if (blockIdx.x == 0) acc->pad = Q;
            next_state(sh.st, Q, __ldcg(&acc->distinct), A.thr);
        }
        __syncthreads();
        if (!sh.ok) {
            if (t == 0) A.state->err = 1;
            return;
        }
        if (sh.st.done) break;
        move_sigma(A, P, N, gt, A.n, gthreads);
        __syncthreads();
        if (t == 0) {
            bar++;
            sh.ok = grid_wait(A.barrier, bar * gridDim.x, A.polls);
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

// Many graphs packed as one union: a cluster of CTAs takes a graph through all
// iterations of its phase, then the next one from the queue (largest first).
// Graphs share nothing, so the clusters never wait for one another: the
// barriers of an iteration are cluster barriers, the sums of a sweep are read
// from the cluster's CTAs through distributed shared memory.
template <int WK, int PREC, int VER>
__global__ void __launch_bounds__(kThreads, 1) lm_resident_batch_kernel(ResidentBatchArgs A) {
    using G = typename Prec<PREC>::G;
    using V = typename ValT<WK>::type;
    namespace cg = cooperative_groups;
    struct View {
        const uint32_t *col;
        const void *w;
        const uint32_t *perm;
        const uint2 *rows;
        const double *k;
        double *sigma;
        const GainK &K;
    };
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ Shared<V, G> sh;
    __shared__ GainK gk;
    __shared__ SweepSums part[2];   // this CTA's sums, by the parity of the sweep
    __shared__ uint32_t ctr[2];     // warp tasks handed out (rank 0's is the cluster's)
    __shared__ uint32_t next, v0, v1;
    __shared__ unsigned long long nnz;
    __shared__ double mass;
    cg::cluster_group cl = cg::this_cluster();
    const uint32_t rank = cl.block_rank(), size = cl.num_blocks();
    const uint32_t S = 1u << A.bits;
    V *vals = (V *)smem_raw;
    uint32_t *keys = (uint32_t *)(smem_raw + sizeof(V) * S);
    uint16_t *used = (uint16_t *)(smem_raw + (sizeof(V) + sizeof(uint32_t)) * S);
    const uint32_t t = threadIdx.x, lane = t & 31u;
    const uint32_t tt = rank * kThreads + t, tn = size * kThreads;
    clear_tables(keys, vals, S, sh);
    if (t < 2) ctr[t] = 0;
    const View view = {A.col, A.w, A.perm, A.rows, A.k, A.sigma, gk};
    uint32_t *const ctr0 = cl.map_shared_rank(&ctr[0], 0);
    while (true) {
        if (rank == 0 && t == 0) next = atomicAdd(A.queue, 1u);
        cl.sync();
        const uint32_t qi = *cl.map_shared_rank(&next, 0);
        if (qi >= A.count) break;
        const uint32_t g = A.order[qi];
        if (t < kSweepClasses) {
            sh.beg[t] = A.cls[(size_t)g * kSweepClasses + t];
            sh.end[t] = A.cls[(size_t)(g + 1) * kSweepClasses + t];
        }
        if (t == 0) {
            gk = A.gk[g];
            mass = A.mass[g];
            nnz = A.gnnz[g];
            v0 = A.goff[g];
            v1 = A.goff[g + 1];
            sh.st = A.state[g];
        }
        __syncthreads();
        if (t == 0) count_tasks(sh, A.bits, size);
        __syncthreads();
        // (iterations of a launch are bounded; the host launches again)
        for (int it = 0; it < A.sweeps && !sh.st.done; it++) {
            const int par = it & 1;
            const uint32_t *P = A.C[sh.st.p];
            uint32_t *N = A.C[sh.st.nx];
            double sin = 0, sf = 0;
            unsigned dcnt = 0;
            unsigned long long su = 0;
            team_sweep<WK, PREC, VER>(view, P, N, sh.st.up, !sh.st.first && 2 * sh.st.distinct < nnz, A.bits, rank,
                                      size, keys, vals, used, sin, dcnt, sh,
                                      [&] { return atomicAdd(ctr0 + par, 1u); });
            sigma_sq(A.sigma, v0 + tt, v1, tn, A.integral, su, sf);
            const SweepSums r = cta_sums(sin, dcnt, su, sf, sh);
            if (t == 0) part[par] = r;
            cl.sync();  // every CTA's sums, and the new assignment, are there
            if (t < 32) {
                SweepSums x = {0, 0, 0, 0};
                if (lane < size) x = *cl.map_shared_rank(&part[par], lane);
                x.sin = warp_sum(x.sin);
                x.distinct = warp_sum(x.distinct);
                x.s2_u = warp_sum(x.s2_u);
                x.s2_f = warp_sum(x.s2_f);
                if (lane == 0) {
                    const double a = A.integral ? __ull2double_rn((unsigned long long)x.sin) : x.sin;
                    const double b = A.integral ? __ull2double_rn(x.s2_u) : x.s2_f;
                    next_state(sh.st, sweep_q(a, b, mass), x.distinct, A.thr);
                    if (rank == 0) {
                        ctr[par] = 0;  // every CTA is past this sweep's tasks
                        atomicAdd(A.distinct, x.distinct);
                    }
                }
            }
            __syncthreads();
            if (!sh.st.done) move_sigma(view, P, N, v0 + tt, v1, tn);
            cl.sync();
        }
        if (rank == 0 && t == 0) {
            A.state[g] = sh.st;
            if (sh.st.done) {
                A.gword[g] = gw_make(false, sh.st.p, sh.st.nx, sh.st.base, false, false, 0, 0);
                A.curQ[g] = sh.st.curQ;
                A.iters[g] += (unsigned long long)(sh.st.iters - 1);
                atomicAdd(&A.totals->edges, nnz * (unsigned long long)sh.st.iters);
                atomicMax(&A.totals->sweeps, (unsigned long long)sh.st.iters);
            } else {
                atomicAdd(&A.totals->open, 1u);
            }
        }
    }
    cl.sync();  // no CTA leaves while others may still read its memory
}

template <int WK>
size_t resident_smem(int bits) {
    return ((size_t)1 << bits) * (sizeof(typename ValT<WK>::type) + sizeof(uint32_t) + 1);
}

// At most `grid` CTAs, and as many as run at once.
template <int WK, int PREC, int VER>
bool launch_resident(const ResidentArgs &A, unsigned grid, cudaStream_t s) {
    auto kern = lm_resident_kernel<WK, PREC, VER>;
    raise_smem_limit((const void *)kern, resident_smem<WK>(kResidentMaxBits));
    const unsigned fit = (unsigned)(blocks_per_sm((const void *)kern, kThreads, resident_smem<WK>(A.bits)) * A.sms);
    if (fit == 0) return false;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(std::min(grid, fit));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = resident_smem<WK>(A.bits);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, A);
    if (e == cudaErrorCooperativeLaunchTooLarge) {  // fewer SMs than the device reports
        cudaGetLastError();
        return false;
    }
    MG_CUDA(e);
    MG_LAUNCH_CHECK();
    return true;
}

template <int WK, int PREC, int VER>
cudaLaunchConfig_t batch_config(const ResidentBatchArgs &A, int ctas, unsigned grid, cudaStream_t s,
                                cudaLaunchAttribute *at) {
    raise_smem_limit((const void *)lm_resident_batch_kernel<WK, PREC, VER>, resident_smem<WK>(kResidentMaxBits));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = resident_smem<WK>(A.bits);
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

// As many clusters of `ctas` CTAs as the device holds, at most `most`.
template <int WK, int PREC, int VER>
bool launch_batch(const ResidentBatchArgs &A, int ctas, unsigned most, cudaStream_t s) {
    auto kern = lm_resident_batch_kernel<WK, PREC, VER>;
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t cfg = batch_config<WK, PREC, VER>(A, ctas, (unsigned)ctas, s, at);
    int fit = 0;
    MG_CUDA(cudaOccupancyMaxActiveClusters(&fit, (void *)kern, &cfg));
    if (fit == 0) return false;
    cfg.gridDim = dim3(std::min((unsigned)fit, most) * (unsigned)ctas);
    MG_CUDA(cudaLaunchKernelEx(&cfg, kern, A));
    MG_LAUNCH_CHECK();
    return true;
}

template <int WK>
bool launch_batch_kind(const ResidentBatchArgs &A, int prec, int ver, int ctas, unsigned most, cudaStream_t s) {
    auto version = [&](auto precc) {
        constexpr int PREC = decltype(precc)::value;
        return ver == 1 ? launch_batch<WK, PREC, 1>(A, ctas, most, s)
                        : launch_batch<WK, PREC, 2>(A, ctas, most, s);
    };
    if (prec == MG_PREC_FP64) return version(std::integral_constant<int, MG_PREC_FP64>());
    if (prec == MG_PREC_FP32) return version(std::integral_constant<int, MG_PREC_FP32>());
    if constexpr (kIntg<WK>) {
        if (prec == MG_PREC_INT64) return version(std::integral_constant<int, MG_PREC_INT64>());
    }
    throw Error(MG_ERR_INVALID, "unknown weight kind or precision");
}

template <int WK>
bool launch_resident_kind(const ResidentArgs &A, int prec, int ver, unsigned grid, cudaStream_t s) {
    auto version = [&](auto precc) {
        constexpr int PREC = decltype(precc)::value;
        return ver == 1 ? launch_resident<WK, PREC, 1>(A, grid, s)
                        : launch_resident<WK, PREC, 2>(A, grid, s);
    };
    if (prec == MG_PREC_FP64) return version(std::integral_constant<int, MG_PREC_FP64>());
    if (prec == MG_PREC_FP32) return version(std::integral_constant<int, MG_PREC_FP32>());
    if constexpr (kIntg<WK>) {
        if (prec == MG_PREC_INT64) return version(std::integral_constant<int, MG_PREC_INT64>());
    }
    throw Error(MG_ERR_INVALID, "unknown weight kind or precision");
}

}  // namespace lmr
}  // namespace mg
