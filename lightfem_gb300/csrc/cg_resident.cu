// Resident PCG: the whole Krylov loop of the pointwise preconditioners (Jacobi, 2x2
// nodal blocks) in one kernel whose CTAs stay on their SMs from the first product
// to convergence (pcg_solve, src/solver.cpp:532-627, and the FP32-inner /
// FP64-refinement scheme of cg_graph.cu, with the same stop rules and error codes).
//
// What it removes.  As a graph of kernels an iteration cost 20 us (mixed) to 28 us
// (FP64) on a mesh of 81 nodes, where there is nothing to compute: launches, a
// last-CTA tail per dot product, the conditional node.  Here an iteration crosses
// the grid twice, 0.8 us for p.q and 1.4 us for r.r and r.z with z published.
//
// Layout.  K's 2x2 blocks lie in slices of 32 nodes, a thread per node: for each of
// a node's eight off-diagonal blocks the slice holds 32 consecutive values, so a
// warp's loads are whole lines, no lane is idle at a nine-block row, and no
// shuffles are needed (on GB300 an FP64 instruction holds an SM's FP64 pipe for 19
// cycles whatever its active lanes: the quarter-warp rows of cg64_product spent 72
// of them a node, this form 36).  Neighbours are 16-bit offsets from the node.
//
// p in shared memory.  A CTA owns consecutive slices; the columns of its rows span
// a window of nodes, and the CTA keeps p of the whole window in shared memory.
// z is what the CTAs exchange (through L2): each forms p = z + beta p for its
// window, its neighbours' nodes included, with the same operation, so every copy
// of a p is the same bit for bit and no third crossing publishes p.
//
// Sums.  A dot product's CTA totals are added as integers: with the previous
// iteration's total as the scale, a total becomes an 88-bit fixed-point number
// (2^-70 of the scale), whose two words are added to two counters in L2 by
// red.add.  The top byte of a word counts the arrivals, so the poll that sees the
// last CTA also has the sum, and the order of arrival does not matter.  A total
// out of range, or a sum that lost more than ten bits of the scale, sends all CTAs
// to a plain sum of the FP64 totals behind a counter.  152 CTAs, GB300: 0.83 us
// without and 1.40 us with the release and acquire that publish z, against 2.6 us
// for a counter and 152 FP64 partials.
//
// Small meshes run in one thread-block cluster, whose CTAs exchange their totals
// through distributed shared memory and a cluster barrier (0.2 us).
//
// Measured, us an iteration as a graph of kernels and here (n x n plane-strain
// cantilevers, log-normal moduli, RCM, Jacobi; GB300):
//   n            8     50    100   200   400   640   800   1000
//   FP64  graph  28.5  29.8  32.1  36.1  57.7  ~97         200
//         here    6.3   7.8   8.4  11.2  23.9  50.2  74.3  106
//   mixed graph  20.9  20.0  20.1  21.5  24.5  ~33         58
//         here    3.9   6.0   7.3   7.6  10.5  13.3  34.1  49.3
// FP64 is bound by the FP64 pipe from 300 on (50 instructions a node, 39 us at 640);
// mixed by the crossings up to 640 and by HBM from 800 on, where K leaves L2.
#include "cg_math.cuh"
#include "common.cuh"
#include "kernels.hpp"

#include <algorithm>
#include <cmath>
#include <vector>

namespace lfgpu {
namespace {

using u64 = unsigned long long;

constexpr int kSlice = 32;       // nodes per slice, a thread each
constexpr int kGroup = 8;        // off-diagonal blocks per node and group
constexpr int kMaxCluster = 16;
constexpr int kWords = 8;        // words of one packed sum (two per quantity)
constexpr int kScaleBits = 70;   // fixed-point bits below the previous total's leading bit
constexpr int kRangeBits = 87;   // |total| < 2^87 units

struct ResArgs {
    int nb, slices, grid;
    const int* group_ptr;        // first group of each slice, or nullptr: one group a slice
    const int2* window;          // per CTA: first and end node of its rows' columns
    const uint4* off;            // per group and lane: eight 16-bit column offsets
    const float4* v32;           // [group][8][32]
    const float4* d32;           // per node: compensated diagonal's high parts and the block's off-diagonal
    const float2* dlo;           // per node: the diagonal's low parts
    const double2* v64;          // [group][8][2][32]: top and bottom rows
    const double2* d64;          // [2][padded nodes]
    const int* rowptr;
    const int* col;
    const double* K;
    const double* f;
    const double* x0;
    double* x;
    const void* pc;              // inverse diagonal or 2x2 factors, in the working precision
    void* z;                     // published M^-1 r
    void* r;                     // residual and product, where shared memory has no room for them
    void* q;
    float2* xhi;
    float2* xlo;
    int window_cap;              // nodes of the window in shared memory
    int own_cap;                 // nodes whose r and q are in shared memory (0: in global memory)
    int keep;                    // slices below this stay in L2, later ones stream
    u64* words;
    double* partials;
    u64* bar;
    DeviceStatus* status;
    PcgResult* result;
    double target, target2;      // sqrt(s) <= target exactly when s <= target2
    double reduction;
    long long maxit, max_ref;
    int restart;
};

// ------------------------------------------------------------------ loads
__device__ __forceinline__ u64 policy_keep() {
    u64 p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
// Matrix data: cached in L1 (CACHED: the CTA's share fits) or past it, with an L2 policy.
template <bool CACHED>
__device__ __forceinline__ float4 ld_matrix(const float4* p, u64 pol) {
    if constexpr (CACHED) return __ldg(p);
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p), "l"(pol));
    return v;
}
template <bool CACHED>
__device__ __forceinline__ double2 ld_matrix(const double2* p, u64 pol) {
    if constexpr (CACHED) return __ldg(p);
    double2 v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;"
                 : "=d"(v.x), "=d"(v.y)
                 : "l"(p), "l"(pol));
    return v;
}
template <bool CACHED>
__device__ __forceinline__ uint4 ld_matrix(const uint4* p, u64 pol) {
    if constexpr (CACHED) return __ldg(p);
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p), "l"(pol));
    return v;
}
__device__ __forceinline__ int offset_of(const uint4& o, int k) {
    const unsigned w = k < 2 ? o.x : k < 4 ? o.y : k < 6 ? o.z : o.w;
    return (k & 1) ? static_cast<int>(w) >> 16 : static_cast<int>(w << 16) >> 16;
}

// ------------------------------------------------------------------ sums
struct ResShared {
    double total[3];             // last totals: p.q, r.r, r.z
    double alpha64, beta64;
    float alpha, alpha_lo, beta;
    int next;                    // kGo, kStop, kRefine
    int ok;
    double xch[2][2][kMaxCluster];  // cluster: the peers' totals
};
enum { kGo = 0, kStop = 1, kRefine = 2 };

__device__ __forceinline__ u64 ld_relaxed(const u64* p) {
    u64 v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ u64 ld_acquire(const u64* p) {
    u64 v;
    asm volatile("ld.acquire.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
template <bool PUBLISH>
__device__ __forceinline__ void red_add(u64* p, u64 v) {
    if constexpr (PUBLISH) asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
    else asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Spin until done(value) holds; bounded by the handle's wait limit, and ended by
// another CTA's abort.
template <bool PUBLISH, typename Done>
__device__ __forceinline__ bool spin(const u64* p, u64& v, DeviceStatus* status, u64 limit, Done&& done) {
    v = PUBLISH ? ld_acquire(p) : ld_relaxed(p);
    if (done(v)) return true;
    const u64 t0 = global_ns();
    for (unsigned it = 1;; ++it) {
        v = PUBLISH ? ld_acquire(p) : ld_relaxed(p);
        if (done(v)) return true;
        if (global_ns() - t0 > limit) {
            atomicExch(&status->abort, 1u);
            record_failure(status, LFGPU_ERR_TIMEOUT, static_cast<int>(blockIdx.x));
            return false;
        }
        if ((it & 31u) == 0u && ld_relaxed_gpu(&status->abort) != 0u) return false;
    }
}

// The grid's sum of K values, one per CTA, by warp 0 of every CTA (v: in all its
// lanes, totals on return).  `prev`: the scale, last sums of the same quantities;
// buf: the packed sum's words, next: words that CTA 0 clears for later sums when
// this one publishes (their last readers arrived before this CTA got here).
struct GridSync {
    u64* words;
    double* partials;
    u64* bar;
    DeviceStatus* status;
    u64 limit;
    int grid;
    u64 arrivals;                // of the counter, so far

    template <int K>
    __device__ __forceinline__ bool plain(double (&v)[K]) {
        const int lane = threadIdx.x & 31;
        double* slot = partials + ((arrivals / grid) & 1) * static_cast<size_t>(grid) * kMaxReduce;
        arrivals += grid;
        int ok = 1;
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < K; ++k) __stcg(slot + blockIdx.x * kMaxReduce + k, v[k]);
            red_add<true>(bar, 1ull);
            u64 seen;
            const u64 want = arrivals;
            ok = spin<true>(bar, seen, status, limit, [&](u64 s) { return s >= want; });
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        __syncwarp();
        if (!ok) return false;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            double t = 0.0;
            for (int b = lane; b < grid; b += 32) t += __ldcg(slot + b * kMaxReduce + k);
            v[k] = warp_sum(t);
        }
        return true;
    }

    template <int K, bool PUBLISH>
    __device__ __forceinline__ bool sum(double (&v)[K], const double* prev, u64* buf, u64* next_a, u64* next_b) {
        const int lane = threadIdx.x & 31;
        if (PUBLISH && blockIdx.x == 0 && lane < kWords) {
            asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(next_a + lane), "l"(0ull) : "memory");
            asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(next_b + lane), "l"(0ull) : "memory");
        }
        __syncwarp();
        // The scale's exponent; the same in every CTA.
        bool usable = true;
        int e[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const u64 b = static_cast<u64>(__double_as_longlong(prev[k]));
            e[k] = static_cast<int>(b >> 52) - 1023;  // a negative value or NaN gives a large exponent
            usable = usable && e[k] > -900 && e[k] < 900;
        }
        if (usable) {
            const int k = min(lane >> 1, K - 1);
            double mine = v[0];
            int scale = e[0];
            if (K > 1 && k == 1) {
                mine = v[K - 1];
                scale = e[K - 1];
            }
            const u64 b = static_cast<u64>(__double_as_longlong(mine));
            const int ex = static_cast<int>((b >> 52) & 0x7ff);
            const u64 m = (b & 0xfffffffffffffull) | (ex ? 1ull << 52 : 0ull);
            const int sh = (ex ? ex : 1) - 1075 + kScaleBits - scale;
            const bool bad = ex == 0x7ff || (m != 0 && sh > kRangeBits - 53);
            unsigned __int128 u = 0;
            if (!bad) {
                if (sh >= 0) u = static_cast<unsigned __int128>(m) << min(sh, kRangeBits - 53);
                else if (sh > -54) u = (m + (1ull << (-sh - 1))) >> -sh;
                if (b >> 63) u = static_cast<unsigned __int128>(0) - u;
                u += static_cast<unsigned __int128>(1) << kRangeBits;
            }
            const u64 low = static_cast<u64>(u) & 0xffffffffffffull;
            const u64 high = static_cast<u64>(u >> 48) & 0xffffffffffull;
            const bool is_high = lane & 1;
            u64 got = 0;
            int ok = 1;
            if (lane < 2 * K) {
                red_add<PUBLISH>(buf + lane, (1ull << 56) | (is_high ? (bad ? 1ull << 48 : 0ull) | high : low));
                const u64 n = static_cast<u64>(grid);
                ok = spin<PUBLISH>(buf + lane, got, status, limit, [&](u64 s) { return (s >> 56) == n; });
            }
            if (!__all_sync(0xffffffffu, ok)) return false;
            got &= (1ull << 56) - 1;
            bool lost = false;
            double t[K];
#pragma unroll
            for (int j = 0; j < K; ++j) {
                const u64 lo = __shfl_sync(0xffffffffu, got, 2 * j), hi = __shfl_sync(0xffffffffu, got, 2 * j + 1);
                const unsigned __int128 all = (static_cast<unsigned __int128>(hi & 0xffffffffffffull) << 48) + lo;
                const __int128 s = static_cast<__int128>(
                    all - (static_cast<unsigned __int128>(static_cast<unsigned>(grid)) << kRangeBits));
                // Positive, and within ten bits of the scale: else the plain sum.
                lost = lost || (hi >> 48) != 0 || s < (static_cast<__int128>(1) << (kScaleBits - 10));
                const u64 top = static_cast<u64>(s >> 32);  // at least 28 bits, at most 64
                const u64 rest = static_cast<u64>(s) & 0xffffffffull;
                const int lead = __clzll(static_cast<long long>(top));
                const u64 w = (top << lead) | (lead >= 32 ? rest << (lead - 32) : rest >> (32 - lead));
                const double d = __ull2double_rn(w);  // s = w 2^(32 - lead), to 64 bits
                t[j] = d * __longlong_as_double(static_cast<long long>(1023 + 32 - lead + e[j] - kScaleBits) << 52);
            }
            if (!lost) {
#pragma unroll
                for (int j = 0; j < K; ++j) v[j] = t[j];
                return true;
            }
        }
        return plain<K>(v);
    }
};

// Per-thread values to the CTA's totals, in all lanes of warp 0.
template <int K>
__device__ __forceinline__ void block_total(const double (&t)[K], double (&v)[K], double* s_red) {
    const int T = blockDim.x, tid = threadIdx.x, lane = tid & 31;
    if (T > 32) {
        // Through shared memory: shuffles in every warp would hold the FP64 pipe
        // 19 cycles per warp and step.
#pragma unroll
        for (int k = 0; k < K; ++k) s_red[k * T + tid] = t[k];
        __syncthreads();
    } else {
        __syncwarp();
    }
    if (tid < 32) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            double a = t[k], b = 0.0;
            if (T > 32) {
                a = s_red[k * T + lane];
                int w = lane + 32;
                for (; w + 32 < T; w += 64) {
                    b += s_red[k * T + w];
                    a += s_red[k * T + w + 32];
                }
                if (w < T) b += s_red[k * T + w];
            }
            v[k] = a + b;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
            for (int k = 0; k < K; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
        }
    }
}
template <int K>
__device__ __forceinline__ void block_total(FloatPair (&t)[K], double (&v)[K], double*) {
    FloatPair w[K];
    block_pair_reduce<K>(t, w);
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = static_cast<double>(w[k].hi) + static_cast<double>(w[k].lo);
}

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void store_peer(const double* slot, unsigned rank, double v) {
    unsigned addr;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(smem_u32(slot)), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

// The sum over all CTAs of K per-thread values, then fin(totals) on thread 0 of
// every CTA; false when a wait ran out.  PUBLISH: the CTAs' earlier global writes
// are visible to all after it.  FAST: the packed sum, scaled by prev.
template <bool CLUSTER, int K, bool PUBLISH, bool FAST, typename V, typename Fin>
__device__ __forceinline__ bool reduce(const ResArgs& a, ResShared& sh, GridSync& g, double* s_red, V (&t)[K],
                                       const double* prev, unsigned parity, Fin&& fin) {
    double v[K];
    block_total<K>(t, v, s_red);
    bool ok = true;
    if constexpr (CLUSTER) {
        const int lane = threadIdx.x & 31;
        if (a.grid > 1) {
            const unsigned rank = cluster_rank();
            if (threadIdx.x < 32 && lane < a.grid) {
#pragma unroll
                for (int k = 0; k < K; ++k) store_peer(&sh.xch[parity & 1][k][rank], lane, v[k]);
            }
            cluster_barrier();
            if (threadIdx.x < 32) {
#pragma unroll
                for (int k = 0; k < K; ++k) v[k] = lane < a.grid ? sh.xch[parity & 1][k][lane] : 0.0;
#pragma unroll
                for (int o = kMaxCluster / 2; o > 0; o >>= 1) {
#pragma unroll
                    for (int k = 0; k < K; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
                }
            }
        }
    } else {
        if (threadIdx.x < 32) {
            // Two sets of words for the p.q sums (parity 0, 1), two for the others.
            u64* base = a.words;
            const unsigned it = parity >> 1;
            u64* mine = base + (2 * (parity & 1) + (it & 1)) * 16;
            if constexpr (FAST)
                ok = g.sum<K, PUBLISH>(v, prev, mine, base + ((it + 1) & 1) * 16, base + (2 + ((it + 1) & 1)) * 16);
            else
                ok = g.plain<K>(v);
        }
    }
    if (threadIdx.x == 0) {
        if (ok) fin(v);
        sh.ok = ok;
    }
    __syncthreads();
    return sh.ok != 0;
}

// ------------------------------------------------------------------ rows
// y = K p of one node of slice s (FP32: without the compensated diagonal's rounding
// of p, as mx_product), p of the window in shared memory, wi the node's own place.
template <bool CACHED>
__device__ __forceinline__ float2 slice_row(const ResArgs& a, int s, int node, const float2* win, int wi, u64 pol) {
    const int lane = threadIdx.x & 31;
    int g = s, end = s + 1;
    if (a.group_ptr) {
        g = __ldg(a.group_ptr + s);
        end = __ldg(a.group_ptr + s + 1);
    }
    const float4 d = ld_matrix<CACHED>(a.d32 + node, pol);
    const float2 x = win[wi], lo = __ldg(a.dlo + node);
    float s0 = d.y * x.y, s1 = d.z * x.x;
    for (; g < end; ++g) {
        const uint4 o = ld_matrix<CACHED>(a.off + g * kSlice + lane, pol);
        const float4* v = a.v32 + static_cast<size_t>(g) * (kGroup * kSlice) + lane;
        float4 w[kGroup];
#pragma unroll
        for (int k = 0; k < kGroup; ++k) w[k] = ld_matrix<CACHED>(v + k * kSlice, pol);
#pragma unroll
        for (int k = 0; k < kGroup; ++k) {
            const float2 p = win[wi + offset_of(o, k)];
            s0 = fmaf(w[k].x, p.x, s0);
            s1 = fmaf(w[k].z, p.x, s1);
            s0 = fmaf(w[k].y, p.y, s0);
            s1 = fmaf(w[k].w, p.y, s1);
        }
    }
    return make_float2(with_diag(s0, d.x, lo.x, x.x), with_diag(s1, d.w, lo.y, x.y));
}
template <bool CACHED>
__device__ __forceinline__ double2 slice_row(const ResArgs& a, int s, int node, const double2* win, int wi, u64 pol) {
    const int lane = threadIdx.x & 31;
    int g = s, end = s + 1;
    if (a.group_ptr) {
        g = __ldg(a.group_ptr + s);
        end = __ldg(a.group_ptr + s + 1);
    }
    const double2 x = win[wi];
    const double2 d0 = ld_matrix<CACHED>(a.d64 + node, pol);
    const double2 d1 = ld_matrix<CACHED>(a.d64 + static_cast<size_t>(a.slices) * kSlice + node, pol);
    double s0 = d0.x * x.x, s1 = d1.x * x.x;
    s0 = fma(d0.y, x.y, s0);
    s1 = fma(d1.y, x.y, s1);
    for (; g < end; ++g) {
        const uint4 o = ld_matrix<CACHED>(a.off + g * kSlice + lane, pol);
        const double2* v = a.v64 + static_cast<size_t>(g) * (2 * kGroup * kSlice) + lane;
        double2 w[2 * kGroup];
#pragma unroll
        for (int k = 0; k < 2 * kGroup; ++k) w[k] = ld_matrix<CACHED>(v + k * kSlice, pol);
#pragma unroll
        for (int k = 0; k < kGroup; ++k) {
            const double2 p = win[wi + offset_of(o, k)];
            s0 = fma(w[2 * k].x, p.x, s0);
            s1 = fma(w[2 * k + 1].x, p.x, s1);
            s0 = fma(w[2 * k].y, p.y, s0);
            s1 = fma(w[2 * k + 1].y, p.y, s1);
        }
    }
    return make_double2(s0, s1);
}

// (f - K x) of one node in FP64 from the CSR values of a paired pattern (rows 2i and
// 2i + 1 share their columns); x as other CTAs wrote it.
__device__ __forceinline__ double2 residual_row(const ResArgs& a, int node, const double* x) {
    const int b = __ldg(a.rowptr + 2 * node), len = __ldg(a.rowptr + 2 * node + 1) - b;
    const double2* k0 = reinterpret_cast<const double2*>(a.K + b);
    const double2* k1 = reinterpret_cast<const double2*>(a.K + b + len);
    double s0 = 0.0, s1 = 0.0;
    const int m = len / 2;
#pragma unroll 3
    for (int k = 0; k < m; ++k) {
        const double2 xv = __ldcg(reinterpret_cast<const double2*>(x + __ldg(a.col + b + 2 * k)));
        const double2 u = __ldg(k0 + k), w = __ldg(k1 + k);
        s0 = fma(u.x, xv.x, s0);
        s0 = fma(u.y, xv.y, s0);
        s1 = fma(w.x, xv.x, s1);
        s1 = fma(w.y, xv.y, s1);
    }
    const double2 fv = __ldg(reinterpret_cast<const double2*>(a.f) + node);
    return make_double2(fv.x - s0, fv.y - s1);
}

template <int PRECOND>
__device__ __forceinline__ double2 precond_at(const ResArgs& a, int node, double2 r) {
    const double* pc = static_cast<const double*>(a.pc);
    if (PRECOND == LFGPU_PRECOND_JACOBI) {
        const double2 d = __ldg(reinterpret_cast<const double2*>(pc) + node);
        return make_double2(d.x * r.x, d.y * r.y);
    }
    return block2_apply(pc, node, r.x, r.y);
}
template <int PRECOND>
__device__ __forceinline__ float2 precond_at(const ResArgs& a, int node, float2 r) {
    return precond32_at<PRECOND>(static_cast<const float*>(a.pc), node, r);
}

__device__ __forceinline__ float2 to_working(double2 v, float2) {
    return make_float2(static_cast<float>(v.x), static_cast<float>(v.y));
}
__device__ __forceinline__ double2 to_working(double2 v, double2) { return v; }

// ------------------------------------------------------------------ the solver
template <bool MIXED, int PRECOND, bool CLUSTER, bool CACHED>
__global__ void __launch_bounds__(MIXED ? 1024 : 512, 1) resident_pcg(ResArgs a) {
    using V = typename std::conditional<MIXED, float2, double2>::type;
    using Sum = typename std::conditional<MIXED, FloatPair, double>::type;
    extern __shared__ __align__(16) unsigned char res_smem[];
    __shared__ ResShared sh;
    __shared__ double s_red[MIXED ? 2 * 1024 : 2 * 512];
    const int tid = threadIdx.x, T = blockDim.x, warp = tid >> 5, W = T >> 5;
    const int cta = blockIdx.x;
    const int sb = static_cast<int>(static_cast<long long>(a.slices) * cta / a.grid);
    const int se = static_cast<int>(static_cast<long long>(a.slices) * (cta + 1) / a.grid);
    const int2 wnd = a.window[cta];
    const int w0 = wnd.x, wn = wnd.y - wnd.x;
    V* win = reinterpret_cast<V*>(res_smem);
    V* const z = static_cast<V*>(a.z);
    // r and q of the CTA's nodes, by place in the CTA.
    V* const r = a.own_cap ? win + a.window_cap : static_cast<V*>(a.r) + sb * kSlice;
    V* const q = a.own_cap ? r + a.own_cap : static_cast<V*>(a.q) + sb * kSlice;
    const u64 pol_keep = policy_keep(), pol_stream = l2_evict_first_policy();
    GridSync g{a.words, a.partials, a.bar, a.status, a.status->wait_limit_ns, a.grid, 0ull};
    unsigned parity = 0;  // 2 * iterations + sums of this one: consecutive sums differ in the last bit
    long long it = 0, refs = 0;
    int status = 0, converged = 0, stagnated = 0;
    double r0 = 0.0, rho = 0.0, rr_last = 0.0;  // kept by thread 0
    double rmax = 0.0, rtrue = 0.0, rtrue_prev = 0.0;
    int no_progress = 0;
    if constexpr (CLUSTER) {
        if (a.grid > 1) cluster_barrier();  // every CTA runs before a peer stores into it
    }
    auto each_node = [&](auto&& body) {  // this thread's nodes: body(slice, node, place)
        for (int s = sb + warp; s < se; s += W) {
            const int node = s * kSlice + (tid & 31);
            if (node < a.nb) body(s, node, node - sb * kSlice);
        }
    };

    // ---- start: x, r, z; r.r (FP64) and r.z
    {
        double t[2] = {0.0, 0.0};
        each_node([&](int, int node, int at) {
            double2 xv = make_double2(0.0, 0.0), rv;
            if (a.x0) {
                xv = reinterpret_cast<const double2*>(a.x0)[node];
                rv = residual_row(a, node, a.x0);
            } else {
                rv = __ldg(reinterpret_cast<const double2*>(a.f) + node);
            }
            reinterpret_cast<double2*>(a.x)[node] = xv;
            const V rw = to_working(rv, V{});
            const V zv = precond_at<PRECOND>(a, node, rw);
            r[at] = rw;
            __stcg(z + node, zv);
            if constexpr (MIXED) {
                a.xhi[node] = make_float2(0.f, 0.f);
                a.xlo[node] = make_float2(0.f, 0.f);
            }
            t[0] += rv.x * rv.x + rv.y * rv.y;
            t[1] += static_cast<double>(rw.x * zv.x + rw.y * zv.y);
        });
        for (int j = tid; j < wn; j += T) win[j] = V{};
        const bool ok = reduce<CLUSTER, 2, true, false>(a, sh, g, s_red, t, nullptr, 1u, [&](const double* s) {
            r0 = sqrt(fmax(0.0, s[0]));
            rho = s[1];
            rmax = rtrue = rtrue_prev = r0;
            rr_last = s[0];
            sh.total[0] = 0.0;
            sh.total[1] = s[0];
            sh.total[2] = s[1];
            sh.beta = 0.f;
            sh.beta64 = 0.0;
            sh.next = kGo;
            if (r0 <= a.target) {
                converged = 1;
                sh.next = kStop;
            } else if (!(s[1] > 0.0) || !isfinite(s[1])) {
                status = LFGPU_ERR_RHO_INITIAL;
                sh.next = kStop;
            }
        });
        if (!ok) return;
    }

    while (sh.next != kStop) {
        // ---- p = z + beta p over the window
        if constexpr (MIXED) {
            const float beta = sh.beta;
            for (int j = tid; j < wn; j += T) {
                const float2 zv = __ldcg(z + w0 + j), pv = win[j];
                win[j] = make_float2(pnew(zv.x, pv.x, beta), pnew(zv.y, pv.y, beta));
            }
        } else {
            const double beta = sh.beta64;
            for (int j = tid; j < wn; j += T) {
                const double2 zv = __ldcg(z + w0 + j), pv = win[j];
                win[j] = make_double2(fma(beta, pv.x, zv.x), fma(beta, pv.y, zv.y));
            }
        }
        __syncthreads();
        // ---- q = K p, p.q
        {
            Sum t[1] = {};
            each_node([&](int s, int node, int at) {
                const int wi = node - w0;
                const V y = slice_row<CACHED>(a, s, node, win, wi, s < a.keep ? pol_keep : pol_stream);
                const V p = win[wi];
                q[at] = y;
                if constexpr (MIXED) t[0].add(p.x * y.x + p.y * y.y);
                else t[0] += p.x * y.x + p.y * y.y;
            });
            const bool ok =
                reduce<CLUSTER, 1, false, true>(a, sh, g, s_red, t, sh.total, parity++, [&](const double* s) {
                    sh.total[0] = s[0];
                    if (!(s[0] > 0.0) || !isfinite(s[0])) {
                        status = LFGPU_ERR_NOT_SPD;
                        sh.next = kStop;
                    } else if constexpr (MIXED) {
                        pair_quotient(rho, s[0], sh.alpha, sh.alpha_lo);
                    } else {
                        sh.alpha64 = rho / s[0];
                    }
                });
            if (!ok) return;
        }
        if (sh.next == kStop) break;
        // ---- x += alpha p, r -= alpha q, z = M^-1 r; r.r and r.z
        {
            Sum t[2] = {};
            if constexpr (MIXED) {
                const float alpha = sh.alpha, alpha_lo = sh.alpha_lo;
                each_node([&](int, int node, int at) {
                    const float2 p = win[node - w0], qv = q[at];
                    float2 rv = r[at], hv = a.xhi[node], lv = a.xlo[node];
                    pair_axpy(hv.x, lv.x, alpha, alpha_lo, p.x);
                    pair_axpy(hv.y, lv.y, alpha, alpha_lo, p.y);
                    rv.x -= alpha * qv.x;
                    rv.y -= alpha * qv.y;
                    const float2 zv = precond_at<PRECOND>(a, node, rv);
                    a.xhi[node] = hv;
                    a.xlo[node] = lv;
                    r[at] = rv;
                    __stcg(z + node, zv);
                    t[0].add(rv.x * rv.x + rv.y * rv.y);
                    t[1].add(rv.x * zv.x + rv.y * zv.y);
                });
            } else {
                const double alpha = sh.alpha64;
                double2* x2 = reinterpret_cast<double2*>(a.x);
                each_node([&](int, int node, int at) {
                    const double2 p = win[node - w0], qv = q[at];
                    double2 rv = r[at], xv = x2[node];
                    xv.x += alpha * p.x;
                    xv.y += alpha * p.y;
                    rv.x -= alpha * qv.x;
                    rv.y -= alpha * qv.y;
                    const double2 zv = precond_at<PRECOND>(a, node, rv);
                    x2[node] = xv;
                    r[at] = rv;
                    __stcg(z + node, zv);
                    t[0] += rv.x * rv.x + rv.y * rv.y;
                    t[1] += rv.x * zv.x + rv.y * zv.y;
                });
            }
            const bool ok =
                reduce<CLUSTER, 2, true, true>(a, sh, g, s_red, t, sh.total + 1, parity++, [&](const double* s) {
                    sh.total[1] = s[0];
                    sh.total[2] = s[1];
                    it += 1;
                    if constexpr (MIXED) {
                        // Only decides when to replace the residual: FP32 is enough.
                        const double rn = static_cast<double>(__fsqrt_rn(static_cast<float>(fmax(0.0, s[0]))));
                        rmax = fmax(rmax, rn);
                        if (rn <= a.reduction * rmax || rn <= a.target || it >= a.maxit) {
                            sh.next = kRefine;
                        } else if (!(s[1] > 0.0) || !isfinite(s[1])) {
                            status = LFGPU_ERR_RHO;
                            sh.next = kStop;
                        } else {
                            float lo;
                            pair_quotient(s[1], rho, sh.beta, lo);
                            rho = s[1];
                        }
                    } else {
                        rr_last = s[0];
                        if (fmax(0.0, s[0]) <= a.target2) {
                            converged = 1;
                            sh.next = kStop;
                        } else if (!(s[1] > 0.0) || !isfinite(s[1])) {
                            status = LFGPU_ERR_RHO;
                            sh.next = kStop;
                        } else {
                            sh.beta64 = s[1] / rho;
                            rho = s[1];
                            if (it >= a.maxit) sh.next = kStop;
                        }
                    }
                });
            if (!ok) return;
        }
        // ---- residual replacement: x += correction, r = f - K x in FP64, z, beta
        if constexpr (MIXED) {
            if (sh.next != kRefine) continue;
            double2* x2 = reinterpret_cast<double2*>(a.x);
            each_node([&](int, int node, int) {
                const float2 hv = a.xhi[node], lv = a.xlo[node];
                double2 xv = x2[node];
                xv.x += static_cast<double>(hv.x) + static_cast<double>(lv.x);
                xv.y += static_cast<double>(hv.y) + static_cast<double>(lv.y);
                x2[node] = xv;
                a.xhi[node] = make_float2(0.f, 0.f);
                a.xlo[node] = make_float2(0.f, 0.f);
            });
            double none[1] = {0.0};
            unsigned swap = parity;
            if (!reduce<CLUSTER, 1, true, false>(a, sh, g, s_red, none, nullptr, swap++, [](const double*) {})) return;
            double t[2] = {0.0, 0.0};
            each_node([&](int, int node, int at) {
                const double2 rv = residual_row(a, node, a.x);
                const float2 rw = to_working(rv, float2{});
                const float2 zv = precond_at<PRECOND>(a, node, rw);
                r[at] = rw;
                __stcg(z + node, zv);
                t[0] += rv.x * rv.x + rv.y * rv.y;
                t[1] += static_cast<double>(rw.x * zv.x + rw.y * zv.y);
            });
            const bool ok = reduce<CLUSTER, 2, true, false>(a, sh, g, s_red, t, nullptr, swap++, [&](const double* s) {
                refs += 1;
                sh.next = kGo;
                const double rt = sqrt(fmax(0.0, s[0]));
                rtrue = rt;
                if (rt <= a.target) {
                    converged = 1;
                    sh.next = kStop;
                } else if (refs >= a.max_ref || it >= a.maxit) {
                    sh.next = kStop;
                } else {
                    no_progress = rt >= rtrue_prev ? no_progress + 1 : 0;
                    if (no_progress >= 3) {
                        stagnated = 1;
                        sh.next = kStop;
                    }
                    rtrue_prev = fmin(rtrue_prev, rt);
                    rmax = rt;
                }
                if (sh.next == kGo) {
                    if (!(s[1] > 0.0) || !isfinite(s[1])) {
                        status = LFGPU_ERR_RHO;
                        sh.next = kStop;
                    } else {
                        sh.beta = a.restart ? 0.f : static_cast<float>(s[1] / rho);
                        rho = s[1];
                        sh.total[1] = s[0];
                        sh.total[2] = s[1];
                    }
                }
            });
            if (!ok) return;
        }
    }
    if constexpr (MIXED) {
        double2* x2 = reinterpret_cast<double2*>(a.x);
        each_node([&](int, int node, int) {
            const float2 hv = a.xhi[node], lv = a.xlo[node];
            double2 xv = x2[node];
            xv.x += static_cast<double>(hv.x) + static_cast<double>(lv.x);
            xv.y += static_cast<double>(hv.y) + static_cast<double>(lv.y);
            x2[node] = xv;
        });
    }
    if (cta == 0 && tid == 0) {
        PcgResult res{};
        res.iterations = it;
        res.refinements = refs;
        res.initial_residual = r0;
        res.final_residual = MIXED ? rtrue : sqrt(fmax(0.0, rr_last));
        res.status = status;
        res.converged = converged;
        res.stagnated = stagnated;
        *a.result = res;
    }
}

// ------------------------------------------------------------------ setup kernels
// Per CTA of a grid: the nodes its rows' columns span.  info: [0] widest window,
// [1] most blocks in a row, [2] farthest column (in nodes).
__global__ void __launch_bounds__(256) resident_windows(int nb, int slices, int grid, const int* __restrict__ rowptr,
                                                        const int* __restrict__ col, int2* __restrict__ window,
                                                        int* __restrict__ info) {
    __shared__ int s_lo, s_hi, s_deg, s_far;
    const int c = blockIdx.x;
    const int n0 = min(nb, static_cast<int>(static_cast<long long>(slices) * c / grid) * kSlice);
    const int n1 = min(nb, static_cast<int>(static_cast<long long>(slices) * (c + 1) / grid) * kSlice);
    if (threadIdx.x == 0) {
        s_lo = n0;
        s_hi = n1;
        s_deg = s_far = 0;
    }
    __syncthreads();
    int lo = n0, hi = n1, deg = 0, far = 0;
    for (int i = n0 + threadIdx.x; i < n1; i += blockDim.x) {
        const int b = rowptr[2 * i], e = rowptr[2 * i + 1];
        const int first = col[b] >> 1, last = col[e - 1] >> 1;  // columns ascend
        lo = min(lo, first);
        hi = max(hi, last + 1);
        deg = max(deg, (e - b) / 2);
        far = max(far, max(i - first, last - i));
    }
    atomicMin(&s_lo, lo);
    atomicMax(&s_hi, hi);
    atomicMax(&s_deg, deg);
    atomicMax(&s_far, far);
    __syncthreads();
    if (threadIdx.x == 0) {
        window[c] = make_int2(s_lo, s_hi);
        atomicMax(info + 0, s_hi - s_lo);
        atomicMax(info + 1, s_deg);
        atomicMax(info + 2, s_far);
    }
}

// Groups of kGroup off-diagonal blocks each slice needs.
__global__ void resident_groups(int nb, int slices, const int* __restrict__ rowptr, int* __restrict__ groups) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= slices) return;
    int most = 0;
    for (int i = s * kSlice; i < min(nb, (s + 1) * kSlice); ++i)
        most = max(most, (rowptr[2 * i + 1] - rowptr[2 * i]) / 2 - 1);
    groups[s] = max(1, (most + kGroup - 1) / kGroup);
}

// Column offsets of every slice: a node's off-diagonal blocks in column order; unused
// places point at the node itself (their values are zero).
__global__ void resident_offsets(int nb, int slices, const int* __restrict__ group_ptr,
                                 const int* __restrict__ rowptr, const int* __restrict__ col,
                                 uint4* __restrict__ off) {
    const int node = blockIdx.x * blockDim.x + threadIdx.x;
    const int s = node / kSlice, lane = node % kSlice;
    if (s >= slices) return;
    int k = 0, e = 0;
    if (node < nb) {
        k = rowptr[2 * node];
        e = rowptr[2 * node + 1];
    }
    const int g0 = group_ptr ? group_ptr[s] : s, g1 = group_ptr ? group_ptr[s + 1] : s + 1;
    for (int g = g0; g < g1; ++g) {
        unsigned w[kGroup / 2] = {};
#pragma unroll
        for (int j = 0; j < kGroup; ++j) {
            while (k < e && (col[k] >> 1) == node) k += 2;
            int d = 0;
            if (k < e) {
                d = (col[k] >> 1) - node;
                k += 2;
            }
            w[j / 2] |= (static_cast<unsigned>(d) & 0xffffu) << (16 * (j & 1));
        }
        off[g * kSlice + lane] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// Values of every slice from the CSR values of a paired pattern.  FP32: rounded, with
// the compensated diagonal of sparse.cu's compensated_diag_kernel (same operations
// in the same order), its high parts beside the diagonal block's off-diagonal.
template <bool FP32>
__global__ void resident_values(int nb, int slices, const int* __restrict__ group_ptr, const int* __restrict__ rowptr,
                                const int* __restrict__ col, const double* __restrict__ K, float4* __restrict__ v32,
                                float4* __restrict__ d32, float2* __restrict__ dlo, double2* __restrict__ v64,
                                double2* __restrict__ d64) {
    const int node = blockIdx.x * blockDim.x + threadIdx.x;
    const int s = node / kSlice, lane = node % kSlice;
    if (s >= slices) return;
    int b = 0, len = 0;
    if (node < nb) {
        b = rowptr[2 * node];
        len = (rowptr[2 * node + 1] - b) / 2;
    }
    const double2* k0 = reinterpret_cast<const double2*>(K + b);
    const double2* k1 = reinterpret_cast<const double2*>(K + b + 2 * len);
    const int g0 = group_ptr ? group_ptr[s] : s, g1 = group_ptr ? group_ptr[s + 1] : s + 1;
    double err0 = 0.0, err1 = 0.0;
    double2 dia0 = make_double2(0.0, 0.0), dia1 = make_double2(0.0, 0.0);
    int k = 0;
    auto diagonal = [&] {  // passes over the diagonal block
        if (k < len && (col[b + 2 * k] >> 1) == node) {
            dia0 = k0[k];
            dia1 = k1[k];
            ++k;
        }
    };
    for (int g = g0; g < g1; ++g) {
#pragma unroll
        for (int j = 0; j < kGroup; ++j) {
            diagonal();
            double2 u = make_double2(0.0, 0.0), w = u;
            if (k < len) {
                u = k0[k];
                w = k1[k];
                ++k;
            }
            if (FP32) {
                const float4 v = make_float4(static_cast<float>(u.x), static_cast<float>(u.y), static_cast<float>(w.x),
                                             static_cast<float>(w.y));
                err0 += u.x - static_cast<double>(v.x);
                err1 += w.y - static_cast<double>(v.w);
                v32[(static_cast<size_t>(g) * kGroup + j) * kSlice + lane] = v;
            } else {
                v64[(static_cast<size_t>(g) * kGroup + j) * 2 * kSlice + lane] = u;
                v64[((static_cast<size_t>(g) * kGroup + j) * 2 + 1) * kSlice + lane] = w;
            }
        }
    }
    diagonal();
    if (FP32) {
        const double c0 = dia0.x + err0, c1 = dia1.y + err1;
        const float h0 = static_cast<float>(c0), h1 = static_cast<float>(c1);
        d32[node] = make_float4(h0, static_cast<float>(dia0.y), static_cast<float>(dia1.x), h1);
        dlo[node] = make_float2(static_cast<float>(c0 - static_cast<double>(h0)),
                                static_cast<float>(c1 - static_cast<double>(h1)));
    } else {
        d64[node] = dia0;
        d64[static_cast<size_t>(slices) * kSlice + node] = dia1;
    }
}

// ------------------------------------------------------------------ launch shapes
struct Shape {
    bool cluster = false;
    int grid = 0, threads = 0, smem = 0;
    int window_cap = 0, own_cap = 0;
    bool cached = false;
};

// Meshes up to these many nodes run in one cluster.
constexpr int kClusterNodes64 = 3600, kClusterNodes32 = 8192;
constexpr int kStaticSmem64 = 12 * 1024, kStaticSmem32 = 20 * 1024;

int slices_of(const Context& c) { return static_cast<int>((c.n / 2 + kSlice - 1) / kSlice); }

Shape launch_shape(const Context& c, bool mixed) {
    const int nodes = static_cast<int>(c.n / 2), slices = slices_of(c);
    const int max_warps = mixed ? 32 : 16;
    Shape s;
    s.cluster = nodes <= (mixed ? kClusterNodes32 : kClusterNodes64);
    if (s.cluster) {
        s.grid = 1;
        while (s.grid < kMaxCluster && s.grid * (mixed ? 4 : 1) < slices) s.grid *= 2;
    } else {
        s.grid = c.num_sms;
    }
    const int per = (slices + s.grid - 1) / s.grid;
    s.threads = 32 * std::max(1, std::min(max_warps, per));
    return s;
}

}  // namespace

// The slices and windows of the current pattern; false when the resident kernel does
// not take it.
static bool resident_structure(Context& c, bool mixed, Shape& s) {
    Context::Resident& res = c.resident;
    const int nb = static_cast<int>(c.n / 2), slices = slices_of(c);
    s = launch_shape(c, mixed);
    Context::Resident::Grid& grid = res.grid[mixed ? 1 : 0];
    if (grid.version != c.pattern_version) {
        grid.window.ensure(s.grid);
        res.info.ensure(4);
        LF_CUDA(cudaMemsetAsync(res.info.p, 0, 4 * sizeof(int), c.stream));
        resident_windows<<<s.grid, 256, 0, c.stream>>>(nb, slices, s.grid, c.rowptr, c.col, grid.window, res.info);
        LF_CUDA(cudaGetLastError());
        c.launches += 1;
        LF_CUDA(cudaMemcpyAsync(grid.info, res.info.p, 3 * sizeof(int), cudaMemcpyDeviceToHost, c.stream));
        LF_CUDA(cudaStreamSynchronize(c.stream));
        grid.version = c.pattern_version;
    }
    if (grid.info[2] > 32767) return false;
    const int vec = mixed ? 8 : 16;
    int optin = 0;
    LF_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c.device));
    const int room = optin - (mixed ? kStaticSmem32 : kStaticSmem64);
    s.window_cap = (grid.info[0] + 1) & ~1;
    const int own = (slices + s.grid - 1) / s.grid * kSlice;
    if (s.window_cap > room / vec) return false;
    s.own_cap = (s.window_cap + 2 * own) <= room / vec ? own : 0;
    s.smem = vec * (s.window_cap + 2 * s.own_cap);
    // The CTA's matrix share fits L1 beside its shared memory.
    const int row_bytes = mixed ? 8 * 16 + 16 + 16 + 8 + 24 : 8 * 32 + 32 + 16 + 48;
    s.cached = s.cluster || own * row_bytes + s.smem < optin - 40 * 1024;
    if (res.pattern_version != c.pattern_version) {
        int groups = slices;
        res.uniform = grid.info[1] <= kGroup + 1;
        if (!res.uniform) {
            std::vector<int> ptr(static_cast<size_t>(slices) + 1, 0);
            res.group_ptr.ensure(static_cast<size_t>(slices) + 1);
            resident_groups<<<grid_for(slices, 256), 256, 0, c.stream>>>(nb, slices, c.rowptr, res.group_ptr);
            LF_CUDA(cudaGetLastError());
            c.launches += 1;
            LF_CUDA(cudaMemcpyAsync(ptr.data() + 1, res.group_ptr.p, sizeof(int) * slices, cudaMemcpyDeviceToHost,
                                    c.stream));
            LF_CUDA(cudaStreamSynchronize(c.stream));
            for (int k = 0; k < slices; ++k) ptr[k + 1] += ptr[k];
            groups = ptr[slices];
            LF_CUDA(cudaMemcpyAsync(res.group_ptr.p, ptr.data(), sizeof(int) * ptr.size(), cudaMemcpyHostToDevice,
                                    c.stream));
            LF_CUDA(cudaStreamSynchronize(c.stream));
        }
        res.groups = groups;
        res.off.ensure(static_cast<size_t>(groups) * kSlice);
        resident_offsets<<<slices, kSlice, 0, c.stream>>>(nb, slices, res.uniform ? nullptr : res.group_ptr.p,
                                                          c.rowptr, c.col, res.off);
        LF_CUDA(cudaGetLastError());
        c.launches += 1;
        res.pattern_version = c.pattern_version;
        res.k_version[0] = res.k_version[1] = ~0ull;
    }
    return true;
}

bool run_resident(Context& c, const SolveSetup& s, PcgResult* out, float* kernel_ms) {
    if (!c.paired || c.num_sms > 255 || c.n < 2) return false;
    const bool mixed = s.mixed != 0;
    Shape sh;
    if (!resident_structure(c, mixed, sh)) return false;
    Context::Resident& res = c.resident;
    const int nb = static_cast<int>(c.n / 2), slices = slices_of(c);
    const size_t padded = static_cast<size_t>(slices) * kSlice;
    if (res.k_version[mixed] != c.k_version) {
        const size_t blocks = static_cast<size_t>(res.groups) * kGroup * kSlice;
        const int* ptr = res.uniform ? nullptr : res.group_ptr.p;
        if (mixed) {
            res.v32.ensure(blocks);
            res.d32.ensure(padded);
            res.dlo.ensure(padded);
            resident_values<true><<<grid_for(padded, 128), 128, 0, c.stream>>>(
                nb, slices, ptr, c.rowptr, c.col, c.K, res.v32, res.d32, res.dlo, nullptr, nullptr);
        } else {
            res.v64.ensure(2 * blocks);
            res.d64.ensure(2 * padded);
            resident_values<false><<<grid_for(padded, 128), 128, 0, c.stream>>>(
                nb, slices, ptr, c.rowptr, c.col, c.K, nullptr, nullptr, nullptr, res.v64, res.d64);
        }
        LF_CUDA(cudaGetLastError());
        c.launches += 1;
        res.k_version[mixed] = c.k_version;
    }
    ResArgs a{};
    a.nb = nb;
    a.slices = slices;
    a.grid = sh.grid;
    a.group_ptr = res.uniform ? nullptr : res.group_ptr.p;
    a.window = res.grid[mixed].window;
    a.off = res.off;
    a.v32 = res.v32;
    a.d32 = res.d32;
    a.dlo = res.dlo;
    a.v64 = res.v64;
    a.d64 = res.d64;
    a.rowptr = c.rowptr;
    a.col = c.col;
    a.K = c.K;
    a.f = s.rhs;
    a.x0 = s.x0;
    a.x = s.x;
    const bool jac = s.precond == LFGPU_PRECOND_JACOBI;
    if (mixed) {
        a.pc = jac ? static_cast<const void*>(c.inv_diag32.p) : static_cast<const void*>(c.blk32.p);
        for (int k : {1, 0, 4}) c.v32[k].ensure(2 * padded);
        a.z = c.v32[1].p;
        a.r = c.v32[0].p;
        a.q = c.v32[4].p;
        c.xhi.ensure(c.n);
        c.xlo.ensure(c.n);
        a.xhi = reinterpret_cast<float2*>(c.xhi.p);
        a.xlo = reinterpret_cast<float2*>(c.xlo.p);
    } else {
        a.pc = jac ? static_cast<const void*>(c.inv_diag64.p) : static_cast<const void*>(c.blk64.p);
        for (int k : {1, 0, 3}) c.v64[k].ensure(2 * padded);
        a.z = c.v64[1].p;
        a.r = c.v64[0].p;
        a.q = c.v64[3].p;
    }
    a.window_cap = sh.window_cap;
    a.own_cap = sh.own_cap;
    a.keep = slices;
    res.words.ensure(64);
    c.bar.ensure(1);
    c.partials.ensure(static_cast<size_t>(2) * sh.grid * kMaxReduce);
    c.pcg_result.ensure(1);
    LF_CUDA(cudaMemsetAsync(res.words.p, 0, 64 * sizeof(u64), c.stream));
    LF_CUDA(cudaMemsetAsync(c.bar.p, 0, sizeof(u64), c.stream));
    LF_CUDA(cudaMemsetAsync(c.pcg_result.p, 0, sizeof(PcgResult), c.stream));
    a.words = res.words;
    a.partials = c.partials;
    a.bar = c.bar;
    a.status = c.status;
    a.result = c.pcg_result;
    a.target = s.tolerance;
    // The largest s with sqrt(s) <= target (sqrt is monotone and correctly rounded).
    a.target2 = s.tolerance * s.tolerance;
    while (a.target2 > 0.0 && std::sqrt(a.target2) > s.tolerance) a.target2 = std::nextafter(a.target2, 0.0);
    while (std::sqrt(std::nextafter(a.target2, HUGE_VAL)) <= s.tolerance && std::isfinite(a.target2))
        a.target2 = std::nextafter(a.target2, HUGE_VAL);
    a.reduction = s.inner_reduction;
    a.maxit = s.max_iterations;
    a.max_ref = s.max_refinements;
    a.restart = s.restart;
    auto launch = [&](auto kernel) {
        LF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sh.smem));
        if (sh.cluster && sh.grid > 8)
            LF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(sh.grid);
        cfg.blockDim = dim3(sh.threads);
        cfg.dynamicSmemBytes = sh.smem;
        cfg.stream = c.stream;
        cudaLaunchAttribute attr[1] = {};
        if (sh.cluster) {
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = sh.grid;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        } else {  // every CTA resident at once, or the launch fails
            attr[0].id = cudaLaunchAttributeCooperative;
            attr[0].val.cooperative = 1;
        }
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        LF_CUDA(cudaEventRecord(c.ev_a, c.stream));
        LF_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
        LF_CUDA(cudaEventRecord(c.ev_b, c.stream));
        c.launches += 1;
    };
    constexpr int J = LFGPU_PRECOND_JACOBI, B = LFGPU_PRECOND_BLOCK2;
    if (mixed && sh.cluster) jac ? launch(resident_pcg<true, J, true, true>) : launch(resident_pcg<true, B, true, true>);
    else if (mixed && sh.cached) jac ? launch(resident_pcg<true, J, false, true>) : launch(resident_pcg<true, B, false, true>);
    else if (mixed) jac ? launch(resident_pcg<true, J, false, false>) : launch(resident_pcg<true, B, false, false>);
    else if (sh.cluster) jac ? launch(resident_pcg<false, J, true, true>) : launch(resident_pcg<false, B, true, true>);
    else if (sh.cached) jac ? launch(resident_pcg<false, J, false, true>) : launch(resident_pcg<false, B, false, true>);
    else jac ? launch(resident_pcg<false, J, false, false>) : launch(resident_pcg<false, B, false, false>);
    LF_CUDA(cudaMemcpyAsync(out, c.pcg_result.p, sizeof(PcgResult), cudaMemcpyDeviceToHost, c.stream));
    *kernel_ms = elapsed_ms(c);
    check_status(c);
    c.resident_ran = true;
    return true;
}

}  // namespace lfgpu
