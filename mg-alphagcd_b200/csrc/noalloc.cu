// noalloc.cu -- a local-move sweep that allocates nothing.
//
// Some callers cannot call cudaMalloc: a serving process that has handed its
// whole HBM budget to its own pool, or code that must not enter the CUDA
// allocator at all.  mg_local_move_noalloc gives them one local-move sweep on
// a graph they already hold in device memory.  There is no room for lists of
// vertices by degree, so every kernel walks all vertices and takes those of
// its degrees:
//   <= 32       8 lanes per vertex, <= 256 a warp: tables in shared memory
//   <= 2,048    256 threads per vertex, <= 10,922 a 1,024-thread CTA: the same
//   larger      a CTA per vertex, tables in a fixed file-scope device array of
//               kNoAllocScratchBytes (room for pow2(2 * max degree + 2) slots
//               per CTA)
// The kernels of degrees that the graph does not have are not launched.  A
// vertex uses only the first pow2 >= 2 * its degree slots of its table and
// leaves them empty, so the work per vertex follows its own degree.  Threads
// per vertex follow the degree because most vertices have few edges: 256
// threads for each vertex took 29.8 ms on 500,009 vertices with 9.9 M entries
// (integer weights, degrees up to 1.4e4).
// The arithmetic is the engine's FP64 gain (same tie-break, same version 1 / 2
// rules), so for integral weights the result equals mg_local_move exactly.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "handles.cuh"

namespace mg {
void set_orphan_error(const std::string &msg);
}

namespace {

using namespace mg;

constexpr size_t kNoAllocScratchBytes = 16u << 20;  // 16 MiB held by every GPU that loads the library
constexpr int kNoAllocThreads = 256;
constexpr int kMaxDevices = 64;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

struct NoAllocArgs {
    const uint32_t *off, *col;
    const double *w;
    const uint32_t *C;
    const double *sigma, *k;
    uint32_t *C_new;
    uint32_t n;
    double m, two_m, r_m, r_two_m;
    int version, up;
};

// word 0 of the scratch: max degree (written by the first kernel)
__global__ void noalloc_maxdeg_kernel(const uint32_t *off, uint32_t n, uint32_t *out) {
    uint32_t mx = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        mx = max(mx, off[i + 1] - off[i]);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if ((threadIdx.x & 31) == 0) atomicMax(out, mx);
}

__global__ void noalloc_clear_kernel(uint32_t *keys, double *vals, size_t slots) {
    for (size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x; s < slots; s += (size_t)gridDim.x * blockDim.x) {
        keys[s] = kEmpty;
        vals[s] = 0.0;
    }
}

__device__ __forceinline__ bool nb_better(double g2, uint32_t c2, double g1, uint32_t c1, int up) {
    return g2 > g1 || (g2 == g1 && (up ? c2 < c1 : c2 > c1));
}

// table value: unit weights count in 32 bits, others add in double
template <bool UNIT>
using NbVal = typename std::conditional<UNIT, uint32_t, double>::type;
template <bool UNIT>
__device__ __forceinline__ NbVal<UNIT> nb_weight(const NoAllocArgs &A, uint32_t e) {
    if constexpr (UNIT) return 1u;
    else return A.w[e];
}
__device__ __forceinline__ double nb_double(uint32_t x) { return u2d(x); }
__device__ __forceinline__ double nb_double(double x) { return x; }

// log2 of the slots of a vertex of degree d: at least 2 * d and 16, at most 2^most
__device__ __forceinline__ int nb_bits(uint32_t d, int most) {
    const int want = d <= 8 ? 4 : 32 - __clz(2 * d - 1);
    return want < most ? want : most;
}

__device__ __forceinline__ double nb_gain(const NoAllocArgs &A, double kic, double e_src, double ki, double a,
                                          double sc) {
    double t = __dmul_rn(ki, __dsub_rn(a, sc));
    t = div_by(t, A.two_m, A.r_two_m);
    t = __dsub_rn(e_src, t);
    return div_by(__dsub_rn(kic, t), A.m, A.r_m);
}

__device__ __forceinline__ uint32_t nb_final(const NoAllocArgs &A, uint32_t dst, uint32_t src) {
    if (A.version == 1) return dst;
    return A.up ? (dst < src ? dst : src) : (dst > src ? dst : src);
}

// The edges t, t + GT, ... of vertex v into its table; returns the thread's
// part of e.  Four edges in flight per thread.
template <int GT, bool UNIT>
__device__ __forceinline__ NbVal<UNIT> nb_insert(const NoAllocArgs &A, uint32_t v, uint32_t lo, uint32_t hi,
                                                 uint32_t src, uint32_t t, uint32_t *keys, NbVal<UNIT> *vals,
                                                 int bits) {
    using V = NbVal<UNIT>;
    const uint32_t mask = (1u << bits) - 1u;
    V e_part = V(0);
    for (uint32_t base = lo + t; base < hi; base += 4 * GT) {
        uint32_t j[4], c[4];
        V w[4];
#pragma unroll
        for (int b = 0; b < 4; b++) {
            const uint32_t e = base + b * GT;
            j[b] = e < hi ? A.col[e] : kEmpty;
            w[b] = e < hi ? nb_weight<UNIT>(A, e) : V(0);
        }
#pragma unroll
        for (int b = 0; b < 4; b++) c[b] = j[b] != kEmpty ? A.C[j[b]] : kEmpty;
#pragma unroll
        for (int b = 0; b < 4; b++) {
            if (j[b] == kEmpty) continue;
            if (c[b] == src) {
                if (j[b] != v) e_part += w[b];  // self-loops (j == v) stay out of e_src
                continue;
            }
            if (A.version == 1 && !(A.up ? c[b] < src : c[b] > src)) continue;
            uint32_t s = hash_slot(c[b], bits);
            for (uint32_t p = 0; p <= mask; p++) {
                const uint32_t prev = atomicCAS(keys + s, kEmpty, c[b]);
                if (prev == kEmpty || prev == c[b]) break;
                s = (s + 1) & mask;
            }
            atomicAdd(vals + s, w[b]);
        }
    }
    return e_part;
}

// The thread's best of the table's slots t, t + GT, ..., which it empties.
template <int GT, bool UNIT>
__device__ __forceinline__ void nb_evaluate(const NoAllocArgs &A, double e_src, double ki, double a, uint32_t t,
                                            uint32_t *keys, NbVal<UNIT> *vals, int bits, double &best, uint32_t &dst) {
    const uint32_t ts = 1u << bits;
    for (uint32_t s0 = t; s0 < ts; s0 += 4 * GT) {
        uint32_t c[4];
        double kic[4], sc[4];
#pragma unroll
        for (int b = 0; b < 4; b++) {
            const uint32_t s = s0 + b * GT;
            c[b] = s < ts ? keys[s] : kEmpty;
            if (c[b] != kEmpty) {
                kic[b] = nb_double(vals[s]);
                keys[s] = kEmpty;
                vals[s] = 0;
            }
        }
#pragma unroll
        for (int b = 0; b < 4; b++)
            if (c[b] != kEmpty) sc[b] = A.sigma[c[b]];
#pragma unroll
        for (int b = 0; b < 4; b++) {
            if (c[b] == kEmpty) continue;
            const double g = nb_gain(A, kic[b], e_src, ki, a, sc[b]);
            if (nb_better(g, c[b], best, dst, A.up)) {
                best = g;
                dst = c[b];
            }
        }
    }
}

// One vertex by GT <= 32 lanes of a warp (mask: those lanes).
template <int GT, bool UNIT>
__device__ __forceinline__ void nb_vertex(const NoAllocArgs &A, uint32_t v, uint32_t lo, uint32_t hi, uint32_t lanes,
                                          uint32_t *keys, NbVal<UNIT> *vals, int most) {
    const uint32_t t = threadIdx.x & (GT - 1);
    const uint32_t src = A.C[v];
    const double ki = A.k[v];
    const int bits = nb_bits(hi - lo, most);
    NbVal<UNIT> e = nb_insert<GT, UNIT>(A, v, lo, hi, src, t, keys, vals, bits);
    __syncwarp(lanes);
#pragma unroll
    for (int o = GT / 2; o > 0; o >>= 1) e += __shfl_xor_sync(lanes, e, o);
    const double a = A.sigma[src] - ki;
    double best = 0.0;
    uint32_t dst = src;
    nb_evaluate<GT, UNIT>(A, nb_double(e), ki, a, t, keys, vals, bits, best, dst);
#pragma unroll
    for (int o = GT / 2; o > 0; o >>= 1) {
        const double g2 = __shfl_xor_sync(lanes, best, o);
        const uint32_t c2 = __shfl_xor_sync(lanes, dst, o);
        if (nb_better(g2, c2, best, dst, A.up)) {
            best = g2;
            dst = c2;
        }
    }
    if (t == 0) A.C_new[v] = nb_final(A, dst, src);
    __syncwarp(lanes);  // the table is empty before the next vertex
}

// Degrees up to kWarpDeg: a warp takes `per` consecutive vertices (4 to 32: as
// many as leave every warp of the device some), first those of at most kLaneDeg
// edges, four at a time by 8 lanes, then the others.
// 4 blocks of 256 threads per SM (48 KB of tables each).
constexpr uint32_t kLaneDeg = 32, kWarpDeg = 256, kGroupDeg = 2048, kCtaDeg = 10922;
constexpr int kWarpBits = 9, kGroupBits = 12, kCtaBits = 14;
constexpr int kCtaThreads = 1024;

template <bool UNIT>
__global__ void __launch_bounds__(kNoAllocThreads, 4) noalloc_warp_kernel(NoAllocArgs A, uint32_t per) {
    using V = NbVal<UNIT>;
    constexpr uint32_t S = 1u << kWarpBits;
    extern __shared__ __align__(16) unsigned char nb_smem[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    V *vals = (V *)nb_smem + warp * S;
    uint32_t *keys = (uint32_t *)(nb_smem + sizeof(V) * S * (kNoAllocThreads / 32)) + warp * S;
    for (uint32_t s = lane; s < S; s += 32) {
        keys[s] = kEmpty;
        vals[s] = V(0);
    }
    __syncwarp();
    const uint32_t tile = lane / 8, lanes = 0xffu << (8 * tile);
    constexpr uint32_t kWarps = kNoAllocThreads / 32;
    const uint64_t step = (uint64_t)gridDim.x * kWarps * per;
    for (uint64_t v0 = ((uint64_t)blockIdx.x * kWarps + warp) * per; v0 < A.n; v0 += step) {
        const uint64_t v = v0 + lane;
        const bool mine = lane < per && v < A.n;
        const uint32_t lo = mine ? A.off[v] : 0u, hi = mine ? A.off[v + 1] : 0u;
        const uint32_t d = hi - lo;
        // one tile's slice: a quarter of the warp's
        for (uint32_t r = 0; r < per; r += 4) {
            const uint32_t q = r + tile;
            const uint32_t vd = __shfl_sync(0xffffffffu, d, q), vlo = __shfl_sync(0xffffffffu, lo, q);
            if (v0 + q < A.n && vd <= kLaneDeg)
                nb_vertex<8, UNIT>(A, (uint32_t)v0 + q, vlo, vlo + vd, lanes, keys + tile * (S / 4),
                                   vals + tile * (S / 4), kWarpBits - 2);
            __syncwarp();
        }
        uint32_t rest = __ballot_sync(0xffffffffu, mine && d > kLaneDeg && d <= kWarpDeg);
        for (; rest; rest &= rest - 1) {
            const uint32_t q = __ffs(rest) - 1;
            const uint32_t vd = __shfl_sync(0xffffffffu, d, q), vlo = __shfl_sync(0xffffffffu, lo, q);
            nb_vertex<32, UNIT>(A, (uint32_t)v0 + q, vlo, vlo + vd, 0xffffffffu, keys, vals, kWarpBits);
        }
    }
}

// One vertex by a CTA of NT threads.
template <int NT, bool UNIT>
__device__ __forceinline__ void nb_cta_vertex(const NoAllocArgs &A, uint32_t v, uint32_t *keys, NbVal<UNIT> *vals,
                                              int most, double *red_g, uint32_t *red_c) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t lo = A.off[v], hi = A.off[v + 1], src = A.C[v];
    const double ki = A.k[v];
    const int bits = nb_bits(hi - lo, most);
    const double ep = warp_sum(
        nb_double(nb_insert<NT, UNIT>(A, v, lo, hi, src, threadIdx.x, keys, vals, bits)));
    if (lane == 0) red_g[warp] = ep;
    __syncthreads();
    double e_src = 0;
    for (int i = 0; i < NT / 32; i++) e_src += red_g[i];
    const double a = A.sigma[src] - ki;
    double best = 0.0;
    uint32_t dst = src;
    nb_evaluate<NT, UNIT>(A, e_src, ki, a, threadIdx.x, keys, vals, bits, best, dst);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double g2 = __shfl_xor_sync(0xffffffffu, best, o);
        const uint32_t c2 = __shfl_xor_sync(0xffffffffu, dst, o);
        if (nb_better(g2, c2, best, dst, A.up)) {
            best = g2;
            dst = c2;
        }
    }
    __syncthreads();  // everyone has read red_g
    if (lane == 0) {
        red_g[warp] = best;
        red_c[warp] = dst;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < NT / 32; i++)
            if (nb_better(red_g[i], red_c[i], best, dst, A.up)) {
                best = red_g[i];
                dst = red_c[i];
            }
        A.C_new[v] = nb_final(A, dst, src);
    }
    __syncthreads();  // the table is empty, red_* are read
}

// The vertices of degrees in (dmin, dmax], a CTA each.  A CTA looks at `span`
// vertices at a time (at most NT), eight consecutive ones (a sector of offsets)
// from each of span / 8 places spread over the ids, so that hubs with
// neighbouring ids fall to different CTAs.  GLOBAL: the tables are the CTA's part of the scratch
// array (cleared by the host), else shared memory.
template <int NT, bool UNIT, bool GLOBAL>
__global__ void __launch_bounds__(NT) noalloc_cta_kernel(NoAllocArgs A, uint32_t dmin, uint32_t dmax, int most,
                                                         uint32_t span, uint32_t *tkeys, double *tvals) {
    using V = NbVal<UNIT>;
    extern __shared__ __align__(16) unsigned char nb_smem[];
    __shared__ double red_g[NT / 32];
    __shared__ uint32_t red_c[NT / 32];
    __shared__ uint32_t list[NT], count;
    const uint32_t S = 1u << most;
    V *vals = GLOBAL ? (V *)(tvals + (size_t)blockIdx.x * S) : (V *)nb_smem;
    uint32_t *keys = GLOBAL ? tkeys + (size_t)blockIdx.x * S : (uint32_t *)(nb_smem + sizeof(V) * S);
    if constexpr (!GLOBAL) {
        for (uint32_t s = threadIdx.x; s < S; s += NT) {
            keys[s] = kEmpty;
            vals[s] = V(0);
        }
    }
    const uint32_t eights = (uint32_t)(((uint64_t)A.n + 7) / 8), rounds = (eights + span / 8 - 1) / (span / 8);
    for (uint32_t r = blockIdx.x; r < rounds; r += gridDim.x) {
        if (threadIdx.x == 0) count = 0;
        __syncthreads();
        const uint64_t v = ((uint64_t)r + (uint64_t)(threadIdx.x / 8) * rounds) * 8 + threadIdx.x % 8;
        if (threadIdx.x < span && v < A.n) {
            const uint32_t d = A.off[v + 1] - A.off[v];
            if (d > dmin && d <= dmax) list[atomicAdd(&count, 1u)] = (uint32_t)v;
        }
        __syncthreads();
        const uint32_t cnt = count;
        for (uint32_t i = 0; i < cnt; i++) nb_cta_vertex<NT, UNIT>(A, list[i], keys, vals, most, red_g, red_c);
        __syncthreads();
    }
}

std::mutex g_noalloc_mu;
void *g_noalloc_addr[kMaxDevices] = {nullptr};

template <bool UNIT>
constexpr size_t nb_smem_bytes(int bits, int tables) {
    return ((sizeof(NbVal<UNIT>) + sizeof(uint32_t)) * (size_t)tables) << bits;
}

// shared-memory limits of the kernels, per device
template <bool UNIT>
cudaError_t nb_set_limits() {
    cudaError_t e = cudaFuncSetAttribute(noalloc_warp_kernel<UNIT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)nb_smem_bytes<UNIT>(kWarpBits, kNoAllocThreads / 32));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(noalloc_cta_kernel<kNoAllocThreads, UNIT, false>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)nb_smem_bytes<UNIT>(kGroupBits, 1));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(noalloc_cta_kernel<kCtaThreads, UNIT, false>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)nb_smem_bytes<UNIT>(kCtaBits, 1));
    return e;
}

template <bool UNIT>
void nb_launch(const NoAllocArgs &A, uint32_t maxdeg, uint32_t blocks, uint32_t tsize, uint32_t *tkeys, double *tvals,
               cudaStream_t s) {
    // vertices per CTA and round: as many as leave `ctas` CTAs some
    auto span_for = [&](uint32_t nt, uint64_t ctas) {
        uint32_t span = nt;
        while (span > 8 && A.n / span < ctas) span /= 2;
        return span;
    };
    auto grid_for = [&](uint32_t span, uint64_t ctas) {
        return (unsigned)std::min<uint64_t>(ctas, ceil_div(ceil_div(A.n, 8), span / 8));
    };
    if (maxdeg > kCtaDeg) {
        // the scratch keeps the previous call's contents: clear the tables
        noalloc_clear_kernel<<<148 * 4, 256, 0, s>>>(tkeys, tvals, (size_t)blocks * tsize);
        noalloc_cta_kernel<kCtaThreads, UNIT, true><<<blocks, kCtaThreads, 0, s>>>(
            A, kCtaDeg, 0xFFFFFFFFu, 31 - __builtin_clz(tsize), span_for(kCtaThreads, blocks), tkeys, tvals);
    }
    if (maxdeg > kGroupDeg) {
        const uint32_t span = span_for(kCtaThreads, 148);
        noalloc_cta_kernel<kCtaThreads, UNIT, false>
            <<<grid_for(span, 148), kCtaThreads, nb_smem_bytes<UNIT>(kCtaBits, 1), s>>>(A, kGroupDeg, kCtaDeg, kCtaBits,
                                                                                        span, nullptr, nullptr);
    }
    if (maxdeg > kWarpDeg) {
        const uint32_t span = span_for(kNoAllocThreads, 148 * 4);
        noalloc_cta_kernel<kNoAllocThreads, UNIT, false>
            <<<grid_for(span, 148 * 4), kNoAllocThreads, nb_smem_bytes<UNIT>(kGroupBits, 1), s>>>(
                A, kWarpDeg, kGroupDeg, kGroupBits, span, nullptr, nullptr);
    }
    constexpr uint64_t kWarps = kNoAllocThreads / 32;
    uint32_t per = 32;
    while (per > 4 && A.n / per < 148 * 4 * kWarps) per /= 2;
    noalloc_warp_kernel<UNIT><<<(unsigned)std::min<uint64_t>(148 * 4, ceil_div(A.n, per * kWarps)), kNoAllocThreads,
                                nb_smem_bytes<UNIT>(kWarpBits, kNoAllocThreads / 32), s>>>(A, per);
}

mg_status noalloc_fail(mg_status st, const std::string &msg) {
    set_orphan_error("mg_local_move_noalloc: " + msg);
    return st;
}

}  // namespace

extern "C" mg_status mg_local_move_noalloc(uint32_t n, const uint32_t *d_offsets, const uint32_t *d_cols,
                                           const double *d_weights, double mass, const uint32_t *d_C,
                                           const double *d_sigma, const double *d_k, uint32_t *d_C_new,
                                           int version, int up, void *stream) {
    if (!d_offsets || !d_cols || !d_C || !d_sigma || !d_k || !d_C_new)
        return noalloc_fail(MG_ERR_INVALID, "NULL argument");
    if (version < 0 || version > 2) return noalloc_fail(MG_ERR_INVALID, "version must be 0, 1 or 2");
    if (n == 0) return MG_OK;
    if (!(mass > 0)) return noalloc_fail(MG_ERR_INVALID, "mass must be positive");
    cudaStream_t s = (cudaStream_t)stream;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
        return noalloc_fail(MG_ERR_CUDA, "no current CUDA device");
    void *base = nullptr;
    {
        // once per device, with that device current: the device address of the
        // static array (its host-side name is only a stand-in)
        std::lock_guard<std::mutex> lock(g_noalloc_mu);
        if (!g_noalloc_addr[dev]) {
            cudaError_t e = nb_set_limits<true>();
            if (e == cudaSuccess) e = nb_set_limits<false>();
            if (e == cudaSuccess) e = cudaGetSymbolAddress(&g_noalloc_addr[dev], g_noalloc_scratch);
            if (e != cudaSuccess) {
                g_noalloc_addr[dev] = nullptr;
                return noalloc_fail(MG_ERR_CUDA, std::string("device set-up: ") + cudaGetErrorString(e));
            }
        }
        base = g_noalloc_addr[dev];
    }
    // word 0: max degree; tables start at byte 256
    uint32_t *d_maxdeg = (uint32_t *)base;
    if (cudaMemsetAsync(d_maxdeg, 0, sizeof(uint32_t), s) != cudaSuccess)
        return noalloc_fail(MG_ERR_CUDA, "memset failed");
    noalloc_maxdeg_kernel<<<148, 256, 0, s>>>(d_offsets, n, d_maxdeg);
    uint32_t maxdeg = 0;
    if (cudaMemcpyAsync(&maxdeg, d_maxdeg, sizeof maxdeg, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return noalloc_fail(MG_ERR_CUDA, cudaGetErrorString(cudaGetLastError()));
    const uint32_t tsize = pow2_at_least(2ull * maxdeg + 2, 32);
    const size_t table_bytes = (size_t)tsize * (sizeof(uint32_t) + sizeof(double));
    const size_t room = kNoAllocScratchBytes - 512;  // 256-byte header + alignment of the value array
    if (table_bytes > room)
        return noalloc_fail(MG_ERR_UNSUPPORTED, "max degree " + std::to_string(maxdeg) +
                                                    " needs a table larger than the static scratch (16 MiB)");
    // CTAs of the degrees above kCtaDeg
    const uint32_t blocks = (uint32_t)std::min<size_t>({room / table_bytes, (size_t)148, (size_t)n});
    uint32_t *tkeys = (uint32_t *)((unsigned char *)base + 256);
    double *tvals = (double *)((unsigned char *)base + 256 + (((size_t)blocks * tsize * sizeof(uint32_t) + 255) & ~(size_t)255));
    NoAllocArgs A;
    A.off = d_offsets;
    A.col = d_cols;
    A.w = d_weights;
    A.C = d_C;
    A.sigma = d_sigma;
    A.k = d_k;
    A.C_new = d_C_new;
    A.n = n;
    A.m = mass / 2.0;
    A.two_m = 2.0 * A.m;
    A.r_m = 1.0 / A.m;
    A.r_two_m = 1.0 / A.two_m;
    A.version = version;
    A.up = up ? 1 : 0;
    if (d_weights) nb_launch<false>(A, maxdeg, blocks, tsize, tkeys, tvals, s);
    else nb_launch<true>(A, maxdeg, blocks, tsize, tkeys, tvals, s);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return noalloc_fail(MG_ERR_CUDA, cudaGetErrorString(e));
    return MG_OK;
}
