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
// shuffles are needed.  On GB300 an FP64 instruction holds its quarter of the SM for
// 64 cycles (19 an SM over the four quarters) whatever its active lanes: the
// quarter-warp rows of cg64_product spent 72 of them a node, this form 36.
// Neighbours are 16-bit offsets from the node.
//
// p in shared memory.  A CTA owns consecutive slices; the columns of its rows span
// a window of nodes, and the CTA keeps p of the whole window in shared memory.
// z is what the CTAs exchange: each forms p = z + beta p for its window, its
// neighbours' nodes included, with the same operation, so every copy of a p is the
// same bit for bit and no third crossing publishes p.
//
// Sums.  A thread's share of a dot product becomes a fixed-point number, scaled by the
// previous iteration's total, in limbs that a warp adds with one instruction each and
// a CTA in shared memory; a CTA's sum then travels in two words, added to two
// counters in L2 by red.add.  The top byte of a word counts the arrivals, so the poll
// that sees the last CTA also has the sum.  Integers: the order of arrival does not
// matter, and the total is that of the shares to 2^-56 (FP32 pairs) or 2^-70 (FP64) of
// the scale.  A share out of range, or a total that lost more than ten bits of the
// scale, sends all CTAs to a plain sum of FP64 totals behind a counter.  A crossing of
// 152 CTAs takes 0.83 us this way (1.40 us with a release and acquire that publish z),
// against 2.6 us for a counter and 152 FP64 partials.
//
// Three ways to meet.  kCluster, small meshes: one thread-block cluster; z and the
// words go to the peers' shared memory with st.async and red.async, which count their
// bytes on the receiver's mbarrier (0.25 us a crossing).  kTagged: the grid; z goes to
// L2 in words that carry the iteration's number, so that it needs no fence and the
// warps past the first fetch it while warp 0 waits for the sums.  kPublished, large
// meshes: plain z behind release and acquire, half the bytes.
//
// Measured, us an iteration as a graph of kernels and here (n x n plane-strain
// cantilevers, log-normal moduli, RCM, Jacobi; GB300):
//   n            8     20    50    80    100   200   300   400   500   640   800   1000
//   FP64  graph  28.5        29.8        32.1  36.1  44.9  57.7        ~97         200
//         here    4.8   4.9   5.6   6.0   7.2   8.5  13.7  20.3  29.4  45.2  68.1  103
//   mixed graph  20.9        20.0        20.1  21.5  24.2  24.5   28   ~33         58
//         here    2.3   2.6   2.7   3.1   4.1   3.9   5.1   6.6   7.6  11.5  21.8  34.4
// FP64 is bound by the FP64 pipe from 200 on (52 instructions a node; at 640 ncu counts it
// busy for 79 % of the time, 36 us); mixed by the crossings up to 400 and by HBM from 800
// on, where K leaves L2.  With FP64 shuffles and FP64 scalars in the sums a mixed iteration
// took 3.9 us at 8, 6.0 at 50 and 7.6 at 200, an FP64 one 6.3, 7.8 and 11.2.
#include "cg_fixed.hpp"
#include "cg_math.cuh"
#include "common.cuh"
#include "kernels.hpp"

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <type_traits>
#include <vector>

namespace lfgpu {
namespace {

using u64 = unsigned long long;

constexpr int kSlice = 32;       // nodes per slice, a thread each
constexpr int kGroup = 8;        // off-diagonal blocks per node and group
constexpr int kMaxCluster = 16;
constexpr int kStaticSmem64 = 12 * 1024, kStaticSmem32 = 20 * 1024;  // beside the dynamic shared memory

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
    void* z;                     // published M^-1 r (kTagged: as tagged words)
    void* r;                     // residual and product, where shared memory has no room for them
    void* q;
    float2* xhi;
    float2* xlo;
    int window_cap;              // nodes of the window in shared memory
    int halo_cap;                // nodes of the arriving halo
    int own_cap;                 // nodes whose r and q are in shared memory (0: in global memory)
    int x_cap;                   // the same for the solution or its correction pair
    int keep;                    // of 16 slices this many stay in L2, the others stream
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
// Volatile: a row's loads are issued together, before its arithmetic.
template <bool CACHED>
__device__ __forceinline__ float4 ld_matrix(const float4* p, u64 pol) {
    float4 v;
    if constexpr (CACHED)
        asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    else
        asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                     : "l"(p), "l"(pol));
    return v;
}
template <bool CACHED>
__device__ __forceinline__ double2 ld_matrix(const double2* p, u64 pol) {
    double2 v;
    if constexpr (CACHED)
        asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    else
        asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;"
                     : "=d"(v.x), "=d"(v.y)
                     : "l"(p), "l"(pol));
    return v;
}
template <bool CACHED>
__device__ __forceinline__ uint4 ld_matrix(const uint4* p, u64 pol) {
    uint4 v;
    if constexpr (CACHED)
        asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    else
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
enum { kCluster = 0, kTagged = 1, kPublished = 2 };  // how the CTAs meet and exchange z
enum { kGo = 0, kStop = 1, kRefine = 2 };
enum { kPq = 0, kRr = 1, kRz = 2 };

// A dot product's total: FP64, or an unevaluated FP32 pair in the mixed loop, whose
// scalars then need no FP64 arithmetic.
struct PairTotal {
    float hi, lo;
};
template <bool MIXED>
using Total = typename std::conditional<MIXED, PairTotal, double>::type;
// Comparisons on the bits: an FP64 instruction takes 64 cycles.
__device__ __forceinline__ long long bits_of(double v) { return __double_as_longlong(v); }
__device__ __forceinline__ bool positive(double v) { return bits_of(v) > 0 && bits_of(v) < 0x7ff0000000000000ll; }
__device__ __forceinline__ bool positive(PairTotal v) { return v.hi > 0.f && v.hi < INFINITY; }
__device__ __forceinline__ void assign(double& t, double v) { t = v; }
__device__ __forceinline__ void assign(PairTotal& t, double v) {
    t.hi = static_cast<float>(v);
    t.lo = static_cast<float>(v - static_cast<double>(t.hi));
}
// num / den of positive pairs as a pair of about 44 bits: a quotient by the
// approximate reciprocal, its exact remainder, and a correction.
__device__ __forceinline__ void quotient(PairTotal num, PairTotal den, float& hi, float& lo) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(den.hi));
    if (!(den.hi > 0x1p-120f && den.hi < 0x1p120f)) {  // the approximate reciprocal's range
        pair_quotient(num.hi, num.lo, den.hi, den.lo, hi, lo);
        return;
    }
    const float q1 = __fmul_rn(num.hi, y);
    const float r = __fadd_rn(__fmaf_rn(-q1, den.hi, num.hi), __fmaf_rn(-q1, den.lo, num.lo));
    const float q2 = __fmul_rn(r, y);
    hi = __fadd_rn(q1, q2);
    lo = __fsub_rn(q2, __fsub_rn(hi, q1));
}

struct ResShared {
    int e[3];                    // scales of the sums: exponents of the last totals (p.q, r.r, r.z)
    float up[3], down[3][2];     // mixed: 2^-e, and 2^(e - 36) as a product of two floats
    int limb[2][4];              // the CTA's sums being formed
    int bad;                     // a thread's share was out of range
    int next;                    // kGo, kStop, kRefine
    int state;                   // of the last sum: 0 a wait ran out, 1 done, 2 to be formed in FP64
    int fail;                    // a wait for a neighbour's z ran out
    int peers;
    double alpha64, beta64;
    float alpha, alpha_lo, beta;
    u64 acc[2][4];               // cluster: the totals' words, added by the peers
    double xch[2][2][kMaxCluster];  // cluster: the peers' FP64 totals
    u64 mbar[4];                 // cluster: fixed-point sums 0 and 1, FP64 sums 0 and 1
    int4 peer[kMaxCluster];      // cluster: first and end of this CTA's nodes in a peer's window, place there, rank
};

__device__ __forceinline__ void set_scale(ResShared& sh, int k, double t) { sh.e[k] = exponent_of(t); }
__device__ __forceinline__ void set_scale(ResShared& sh, int k, PairTotal t) {
    const int e = exponent_of_pair(t.hi);
    sh.e[k] = e;
    if (e != kNoScale) pair_scale(e, sh.up[k], sh.down[k]);
}

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

// Spin until read() returns true; bounded by the handle's wait limit, and ended by
// another CTA's abort.
template <typename Read>
__device__ __forceinline__ bool spin(DeviceStatus* status, u64 limit, Read&& read) {
    if (read()) return true;
    const u64 t0 = global_ns();
    for (unsigned it = 1;; ++it) {
        if (read()) return true;
        if (global_ns() - t0 > limit) {
            atomicExch(&status->abort, 1u);
            record_failure(status, LFGPU_ERR_TIMEOUT, static_cast<int>(blockIdx.x));
            return false;
        }
        if ((it & 31u) == 0u && ld_relaxed_gpu(&status->abort) != 0u) return false;
    }
}

// A thread's share in limbs, and a total from the words' sums over n CTAs (low in even
// lanes, high in odd ones), in both lanes; false out of range (cg_fixed.hpp).
__device__ __forceinline__ bool to_limbs(const ResShared& sh, int k, const FloatPair& v, int (&l)[3]) {
    return pair_limbs(sh.up[k], v.hi, v.lo, l);
}
__device__ __forceinline__ bool to_limbs(const ResShared& sh, int k, double v, int (&l)[4]) {
    return fp64_limbs(sh.e[k], v, l);
}
__device__ __forceinline__ bool from_words(const ResShared& sh, int k, u64 word, int n, PairTotal& out) {
    const u64 other = __shfl_xor_sync(0xffffffffu, word, 1);
    const bool odd = threadIdx.x & 1;
    return pair_total(sh.down[k], odd ? other : word, odd ? word : other, n, out.hi, out.lo);
}
__device__ __forceinline__ bool from_words(const ResShared& sh, int k, u64 word, int n, double& out) {
    const u64 other = __shfl_xor_sync(0xffffffffu, word, 1);
    const bool odd = threadIdx.x & 1;
    return fp64_total(sh.e[k], odd ? other : word, odd ? word : other, n, out);
}

// Per-thread values to the CTA's totals in FP64, in all lanes of warp 0.
template <int K>
__device__ __forceinline__ void block_total(const double (&t)[K], double (&v)[K], double* s_red) {
    const int T = blockDim.x, tid = threadIdx.x, lane = tid & 31;
#pragma unroll
    for (int k = 0; k < K; ++k) s_red[k * T + tid] = t[k];
    __syncthreads();
    if (tid < 32) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            v[k] = 0.0;
            for (int w = lane; w < T; w += 32) v[k] += s_red[k * T + w];
            v[k] = warp_sum(v[k]);
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

// ------------------------------------------------------------------ cluster
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of a shared-memory variable in CTA `rank` of the cluster.
__device__ __forceinline__ unsigned peer_address(const void* p, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}
// Stores and additions to a peer's shared memory that count their bytes on its mbarrier.
__device__ __forceinline__ void send(unsigned addr, double v, unsigned bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(addr), "d"(v), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void send(unsigned addr, float2 v, unsigned bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "f"(v.x), "f"(v.y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void send(unsigned addr, double2 v, unsigned bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "d"(v.x), "d"(v.y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void send_add(unsigned addr, u64 v, unsigned bar) {
    asm volatile("red.async.relaxed.cluster.shared::cluster.mbarrier::complete_tx::bytes.add.u64 [%0], %1, [%2];" ::"r"(addr),
                 "l"(v), "r"(bar)
                 : "memory");
}

// What a CTA needs to form sums with the others: the words of the packed sums (kSets
// sets for p.q, as many for r.r and r.z), the FP64 sum's slots and counter; in a
// cluster the phases of its mbarriers.
constexpr int kSets = 4, kSetStride = 16;
struct GridSync {
    u64* words;
    double* partials;
    u64* bar;
    DeviceStatus* status;
    u64 limit;
    int grid;
    u64 arrivals;                // of the counter, so far
    unsigned phase;              // bit b: parity of the phase mbarrier b is in

    // The grid's sums of K FP64 values by warp 0 of every CTA (v: in all its lanes).
    // The CTAs' earlier writes are visible to all after it.
    template <int K>
    __device__ __forceinline__ bool plain(double (&v)[K]) {
        const int lane = threadIdx.x & 31;
        double* slot = partials + ((arrivals / grid) & 1) * static_cast<size_t>(grid) * kMaxReduce;
        arrivals += grid;
        int ok = 1;
        __syncwarp();
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < K; ++k) __stcg(slot + blockIdx.x * kMaxReduce + k, v[k]);
            red_add<true>(bar, 1ull);
            const u64 want = arrivals;
            ok = spin(status, limit, [&] { return ld_acquire(bar) >= want; });
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

    // CTA 0, warp 0: clears the words of the sets two iterations on, in every iteration and
    // whichever way its r.r and r.z sum is formed.  Their last readers are past them, and CTA
    // 0 sees the old values (answered()) before it arrives at another sum, so nobody adds to
    // a word before it is cleared.
    __device__ __forceinline__ u64 clear_ahead(unsigned it) {
        const int lane = threadIdx.x & 31;
        u64 old = 0;
        if (blockIdx.x == 0 && lane >= 8 && lane < 14) {
            // Two words of a p.q set, four of an r.r and r.z set.
            u64* w = words + ((it + 2) & (kSets - 1)) * kSetStride +
                     (lane < 10 ? lane - 8 : kSets * kSetStride + lane - 10);
            asm volatile("atom.relaxed.gpu.global.exch.b64 %0, [%1], %2;" : "=l"(old) : "l"(w), "l"(0ull) : "memory");
        }
        return old;
    }
    // Waits for the exchange's answer, here and not before (CTA 0 would hold up the others);
    // always true: no word counts 255 arrivals.
    static __device__ __forceinline__ bool answered(u64 old) {
        asm volatile("" : "+l"(old)::"memory");
        return (old >> 56) != 255ull;
    }

    // A lane's word added over the CTAs (live lanes: 2 k and 2 k + 1).
    template <bool PUBLISH>
    __device__ __forceinline__ bool packed(u64& word, bool live, u64* set) {
        const int lane = threadIdx.x & 31;
        int ok = 1;
        const u64 n = static_cast<u64>(grid);
        if (live) {
            red_add<PUBLISH>(set + lane, word);
            ok = spin(status, limit, [&] {
                word = PUBLISH ? ld_acquire(set + lane) : ld_relaxed(set + lane);
                return (word >> 56) == n;
            });
        }
        return __all_sync(0xffffffffu, ok) != 0;
    }

    // Cluster: wait for mbarrier b's phase, in which `bytes` arrive.
    __device__ __forceinline__ bool arrive_and_wait(ResShared& sh, int b, unsigned bytes) {
        if ((threadIdx.x & 31) == 0) mbar_expect_tx(sh.mbar + b, bytes);
        __syncwarp();
        const unsigned parity = (phase >> b) & 1u;
        const bool ok = spin(status, limit, [&] { return mbar_try_wait(sh.mbar + b, parity); });
        phase ^= 1u << b;
        return __all_sync(0xffffffffu, ok) != 0;
    }
};

// The sum over all CTAs of K per-thread values of quantities FIRST.., then
// fin(totals) on thread 0 of every CTA; false when a wait ran out.  FAST: in fixed
// point at the scales of the last totals, where they allow it.  PUBLISH: on the grid the
// CTAs' earlier global writes are visible to all after it; in a cluster only what the
// peers sent here is (meet() orders global memory there).  halo_bytes (cluster): z
// that the peers send for this sum.  it: the iteration, for the words' set.
// meanwhile(): work of the warps past the first while warp 0 waits.  Consecutive sums
// use different slots: a peer that is one sum ahead then cannot reach this one's.
template <int SYNC, bool MIXED, int FIRST, int K, bool PUBLISH, bool FAST, typename V, typename Meanwhile, typename Fin>
__device__ __forceinline__ bool reduce(const ResArgs& a, ResShared& sh, GridSync& g, double* s_red, V (&t)[K],
                                       unsigned it, [[maybe_unused]] unsigned halo_bytes, Meanwhile&& meanwhile, Fin&& fin) {
    const int lane = threadIdx.x & 31;
    constexpr int kSlot = FIRST == kPq ? 0 : 1;
    bool fast = FAST;
    if (FAST) {
#pragma unroll
        for (int k = 0; k < K; ++k) fast = fast && sh.e[FIRST + k] != kNoScale;
    }
    Total<MIXED> tot[K];
    if (FAST && fast) {
        constexpr int L = kLimbs<MIXED>;
        int l[K][L];
        bool in_range = true;
#pragma unroll
        for (int k = 0; k < K; ++k) in_range = to_limbs(sh, FIRST + k, t[k], l[k]) && in_range;
        if (!in_range) sh.bad = 1;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            int mine = 0;
#pragma unroll
            for (int j = 0; j < L; ++j) {
                const int s = __reduce_add_sync(0xffffffffu, l[k][j]);
                if (lane == j) mine = s;
            }
            if (lane < L) atomicAdd(&sh.limb[k][lane], mine);
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            const bool live = lane < 2 * K;
            const int k = K > 1 ? (lane >> 1) & 1 : 0;
            const bool bad = sh.bad != 0;
            u64 word = sum_word<MIXED>(sh.limb[k], lane & 1, bad);
            __syncwarp();
            if (lane < 8) (&sh.limb[0][0])[lane] = 0;
            if (lane == 8) sh.bad = 0;
            bool ok = true;
            if constexpr (SYNC == kCluster) {
                if (a.grid > 1) {
                    // Lane: word lane & 3 to peers lane / 4, lane / 4 + 8.
                    if ((lane & 3) < 2 * K)
                        for (int p = lane >> 2; p < a.grid; p += 8)
                            send_add(peer_address(&sh.acc[kSlot][lane & 3], p), word, peer_address(sh.mbar + kSlot, p));
                    ok = g.arrive_and_wait(sh, kSlot, static_cast<unsigned>(a.grid * 2 * K * 8) + halo_bytes);
                    word = sh.acc[kSlot][lane & 3];
                    __syncwarp();
                    if (live) sh.acc[kSlot][lane] = 0;
                }
            } else {
                u64* set = a.words + ((FIRST == kPq ? 0 : kSets) + (it & (kSets - 1))) * kSetStride;
                const u64 old = FIRST == kRr ? g.clear_ahead(it) : 0ull;
                ok = g.packed<PUBLISH>(word, live, set);
                ok = __all_sync(0xffffffffu, ok && GridSync::answered(old)) != 0;
            }
            Total<MIXED> mt;
            bool good = from_words(sh, FIRST + k, word, a.grid, mt);
            good = good && ((word >> 48) & 0xff) == 0;
            good = __all_sync(0xffffffffu, good || !live) != 0;
            tot[0] = mt;
            if constexpr (K > 1) {
                if constexpr (MIXED) {
                    tot[1].hi = __shfl_sync(0xffffffffu, mt.hi, 2);
                    tot[1].lo = __shfl_sync(0xffffffffu, mt.lo, 2);
                } else {
                    tot[1] = __shfl_sync(0xffffffffu, mt, 2);
                }
            }
            if (lane == 0) {
                if (ok && good) fin(tot);
                sh.state = !ok ? 0 : good ? 1 : 2;
            }
        } else {
            if constexpr (SYNC != kCluster) meanwhile();
        }
        __syncthreads();
        const int state = sh.state;
        if (state != 2) return state != 0 && sh.fail == 0;
        if constexpr (SYNC == kCluster) halo_bytes = 0;  // z has arrived
    }
    // In FP64, CTA by CTA.
    double v[K];
    bool ok = true;
    block_total<K>(t, v, s_red);
    if (threadIdx.x < 32) {
        if constexpr (SYNC == kCluster) {
            if (a.grid > 1) {
                const unsigned rank = cluster_rank();
                if (lane < a.grid) {
                    const unsigned bar = peer_address(sh.mbar + 2 + kSlot, lane);
#pragma unroll
                    for (int k = 0; k < K; ++k) send(peer_address(&sh.xch[kSlot][k][rank], lane), v[k], bar);
                }
                ok = g.arrive_and_wait(sh, 2 + kSlot, static_cast<unsigned>(a.grid * K * 8) + halo_bytes);
#pragma unroll
                for (int k = 0; k < K; ++k) v[k] = warp_sum(lane < a.grid ? sh.xch[kSlot][k][lane] : 0.0);
            }
        } else {
            if constexpr (FAST && FIRST == kRr) {
                if (!fast) ok = __all_sync(0xffffffffu, GridSync::answered(g.clear_ahead(it))) != 0;  // not yet done above
            }
            ok = g.plain<K>(v) && ok;
        }
        if (lane == 0) {
            if (ok) {
#pragma unroll
                for (int k = 0; k < K; ++k) assign(tot[k], v[k]);
                fin(tot);
            }
            sh.state = ok;
        }
    }
    __syncthreads();
    if constexpr (SYNC == kTagged) {
        if (!(FAST && fast)) {  // not yet done above
            if (threadIdx.x >= 32 && sh.state) meanwhile();
            __syncthreads();
        }
    }
    return sh.state != 0 && sh.fail == 0;
}

// All CTAs' earlier global writes are visible to all after it (reads past L1); false when
// a wait ran out.  Through the counter in L2 in a cluster too: what its sums send to an
// mbarrier orders the peers' shared memory and nothing else.
__device__ __forceinline__ bool meet(const ResArgs& a, ResShared& sh, GridSync& g) {
    __syncthreads();
    if (threadIdx.x < 32) {
        g.arrivals += a.grid;
        if (threadIdx.x == 0) {
            red_add<true>(a.bar, 1ull);
            const u64 want = g.arrivals;
            sh.state = spin(a.status, g.limit, [&] { return ld_acquire(a.bar) >= want; });
        }
    }
    __syncthreads();
    return sh.state != 0;
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
// 2i + 1 share their columns); x as other CTAs wrote it.  A row's terms go to four sums by
// their place modulo four, as in the CSR product: those with u and those with v cancel
// apart from one another, and in one sum they leave a residual whose rounding is up to
// twice as large.  It bounds what a mixed solve can reach: of 800 solves at
// tolerances of 1e-9 to 1e-12 with moduli over four decades 363 converged within 20,000
// iterations with one sum a row, 408 with four, 404 in the graph of kernels.  WIDE:
// both rows and all sums at once; else, with 64 registers a thread, a row and two sums at a
// time (all at once spills, and costs the loop around it 4 to 14 %).
template <bool WIDE>
__device__ __forceinline__ double2 residual_row(const ResArgs& a, int node, const double* x) {
    const int b = __ldg(a.rowptr + 2 * node), len = __ldg(a.rowptr + 2 * node + 1) - b;
    const double2* k0 = reinterpret_cast<const double2*>(a.K + b);
    const int m = len / 2;
    double sum[2] = {0.0, 0.0};
    if constexpr (WIDE) {
        const double2* k1 = reinterpret_cast<const double2*>(a.K + b + len);
        double s0[4] = {}, s1[4] = {};
#pragma unroll 1
        for (int k = 0; k < m; k += 2) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (k + j >= m) break;
                const double2 xv = __ldcg(reinterpret_cast<const double2*>(x + __ldg(a.col + b + 2 * (k + j))));
                const double2 u = __ldg(k0 + k + j), w = __ldg(k1 + k + j);
                s0[2 * j] = fma(u.x, xv.x, s0[2 * j]);
                s0[2 * j + 1] = fma(u.y, xv.y, s0[2 * j + 1]);
                s1[2 * j] = fma(w.x, xv.x, s1[2 * j]);
                s1[2 * j + 1] = fma(w.y, xv.y, s1[2 * j + 1]);
            }
        }
        sum[0] = (s0[0] + s0[1]) + (s0[2] + s0[3]);
        sum[1] = (s1[0] + s1[1]) + (s1[2] + s1[3]);
    } else {
#pragma unroll 2
        for (int row = 0; row < 2; ++row) {
            double t = 0.0;
#pragma unroll 1
            for (int j = 0; j < 2; ++j) {
                double su = 0.0, sv = 0.0;
#pragma unroll 1
                for (int k = j; k < m; k += 2) {
                    const double2 xv = __ldcg(reinterpret_cast<const double2*>(x + __ldg(a.col + b + 2 * k)));
                    const double2 u = __ldg(k0 + row * m + k);
                    su = fma(u.x, xv.x, su);
                    sv = fma(u.y, xv.y, sv);
                }
                t += su + sv;
            }
            if (row) sum[1] = t;
            else sum[0] = t;
        }
    }
    const double2 fv = __ldg(reinterpret_cast<const double2*>(a.f) + node);
    return make_double2(fv.x - sum[0], fv.y - sum[1]);
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
// A published z: two 64-bit words a value pair in FP32, four in FP64, each a 32-bit
// part of a value over the publication's number, so that a reader sees from the
// word itself whether it has arrived: no fence, and the wait for a neighbour's z
// overlaps the wait for the sums.
template <typename V>
constexpr int kTagWords = sizeof(V) / 4;
__device__ __forceinline__ void publish_tagged(u64* w, float2 v, unsigned tag) {
    const u64 t = static_cast<u64>(tag) << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(w), "l"(t | __float_as_uint(v.x)),
                 "l"(t | __float_as_uint(v.y))
                 : "memory");
}
__device__ __forceinline__ void publish_tagged(u64* w, double2 v, unsigned tag) {
    const u64 t = static_cast<u64>(tag) << 32;
    const u64 x = static_cast<u64>(__double_as_longlong(v.x)), y = static_cast<u64>(__double_as_longlong(v.y));
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(w), "l"(t | (x >> 32)), "l"(t | (x & 0xffffffffull))
                 : "memory");
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(w + 2), "l"(t | (y >> 32)), "l"(t | (y & 0xffffffffull))
                 : "memory");
}
__device__ __forceinline__ void ld_two(const u64* w, u64& a, u64& b) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(w) : "memory");
}
__device__ __forceinline__ bool read_tagged(const u64* w, unsigned tag, float2& v) {
    u64 a, b;
    ld_two(w, a, b);
    v = make_float2(__uint_as_float(static_cast<unsigned>(a)), __uint_as_float(static_cast<unsigned>(b)));
    return static_cast<unsigned>(a >> 32) == tag && static_cast<unsigned>(b >> 32) == tag;
}
__device__ __forceinline__ bool read_tagged(const u64* w, unsigned tag, double2& v) {
    u64 a, b, c, d;
    ld_two(w, a, b);
    ld_two(w + 2, c, d);
    v.x = __longlong_as_double(static_cast<long long>((a << 32) | (b & 0xffffffffull)));
    v.y = __longlong_as_double(static_cast<long long>((c << 32) | (d & 0xffffffffull)));
    return static_cast<unsigned>(a >> 32) == tag && static_cast<unsigned>(b >> 32) == tag &&
           static_cast<unsigned>(c >> 32) == tag && static_cast<unsigned>(d >> 32) == tag;
}

// Threads of a CTA: 64 registers a thread let 32 warps stream the FP32 matrix; where it
// sits in L1, and in FP64, which the FP64 pipe bounds, 16 warps with 128 registers do.
constexpr int max_threads(bool mixed, bool cached) { return mixed && !cached ? 1024 : 512; }

template <bool MIXED, int PRECOND, int SYNC, bool CACHED>
__global__ void __launch_bounds__(max_threads(MIXED, CACHED), 1) resident_pcg(ResArgs a) {
    using V = typename std::conditional<MIXED, float2, double2>::type;
    using Sum = typename std::conditional<MIXED, FloatPair, double>::type;
    using Tot = Total<MIXED>;
    constexpr bool kPublish = SYNC == kPublished;
    constexpr bool kWide = max_threads(MIXED, CACHED) < 1024;
    static_assert(max_threads(MIXED, CACHED) <= kLimbThreads<MIXED>, "the CTA's limb sums would overflow");
    extern __shared__ __align__(16) unsigned char res_smem[];
    __shared__ ResShared sh;
    __shared__ double s_red[2 * max_threads(MIXED, CACHED)];
    const int tid = threadIdx.x, T = blockDim.x, warp = tid >> 5, W = T >> 5;
    const int cta = blockIdx.x;
    const int sb = static_cast<int>(static_cast<long long>(a.slices) * cta / a.grid);
    const int se = static_cast<int>(static_cast<long long>(a.slices) * (cta + 1) / a.grid);
    const int n0 = min(a.nb, sb * kSlice), n1 = min(a.nb, se * kSlice);  // the CTA's nodes
    const int2 wnd = a.window[cta];
    const int w0 = wnd.x, left = n0 - wnd.x, halo = left + (wnd.y - n1);  // the window's other nodes
    V* const win = reinterpret_cast<V*>(res_smem);
    V* const own = win + left;                       // p of the CTA's nodes
    V* const zh = win + a.window_cap;                // z of the halo as it arrives (not kPublished)
    V* const state = zh + a.halo_cap;
    // By place in the CTA: r; q, then z from the update to the next direction.
    V* const r = a.own_cap ? state : static_cast<V*>(a.r) + sb * kSlice;
    V* const q = a.own_cap ? state + a.own_cap : static_cast<V*>(a.q) + sb * kSlice;
    // The solution: x (FP64) or the correction pair (mixed).
    V* const xs = a.x_cap ? state + 2 * a.own_cap
                          : MIXED ? reinterpret_cast<V*>(a.xhi) + sb * kSlice : reinterpret_cast<V*>(a.x) + sb * kSlice;
    V* const xl = MIXED ? (a.x_cap ? xs + a.x_cap : reinterpret_cast<V*>(a.xlo) + sb * kSlice) : nullptr;
    const u64 pol_keep = policy_keep(), pol_stream = l2_evict_first_policy();
    GridSync g{a.words, a.partials, a.bar, a.status, a.status->wait_limit_ns, a.grid, 0ull, 0u};
    unsigned it32 = 0;  // iterations, in every thread
    unsigned tag = 0;   // publications of z
    long long it = 0, refs = 0;  // from here on: kept by thread 0
    int status = 0, converged = 0, stagnated = 0, no_progress = 0;
    double r0 = 0.0, rtrue = 0.0, rtrue_prev = 0.0;
    Tot rho{}, rr_last{};
    // Mixed: squares of the inner residual norm, of its largest since the last replacement,
    // and of the bounds on it.
    float rr_max = 0.f;
    const float refine_below = static_cast<float>(a.reduction * a.reduction);
    const float stop_below = static_cast<float>(a.target * a.target);
    // This thread's nodes: body(slice, node, place).
    auto each_node = [&](auto&& body) {
        for (int s = sb + warp; s < se; s += W) {
            const int node = s * kSlice + (tid & 31);
            if (node < a.nb) body(s, node, node - sb * kSlice);
        }
    };
    int reach_lo = 0, reach_hi = a.nb;  // nodes below reach_lo or from reach_hi on: in other CTAs' windows
    if (tid == 0) {
        sh.bad = sh.fail = 0;
        sh.next = kGo;
        for (int k = 0; k < 3; ++k) sh.e[k] = kNoScale;
    }
    if (tid < 8) {
        (&sh.limb[0][0])[tid] = 0;
        (&sh.acc[0][0])[tid] = 0;
    }
    if constexpr (SYNC == kCluster) {
        if (tid == 0) {
            for (int b = 0; b < 4; ++b) mbar_init(sh.mbar + b, 1);
            mbar_init_fence();
            // This CTA's nodes in the peers' windows: a peer's left halo starts its window,
            // its right halo follows the left one.
            int n = 0;
            for (int p = 0; p < a.grid; ++p) {
                const int2 pw = a.window[p];
                const int p0 = min(a.nb, static_cast<int>(static_cast<long long>(a.slices) * p / a.grid) * kSlice);
                const int p1 = min(a.nb, static_cast<int>(static_cast<long long>(a.slices) * (p + 1) / a.grid) * kSlice);
                int4 e = make_int4(0, 0, 0, p);
                if (p > cta) e = make_int4(max(n0, pw.x), min(n1, p0), -pw.x, p);
                if (p < cta) e = make_int4(max(n0, p1), min(n1, pw.y), p0 - pw.x - p1, p);
                if (e.x < e.y) sh.peer[n++] = e;
            }
            sh.peers = n;
        }
        __syncthreads();
        if (a.grid > 1) cluster_barrier();  // every CTA runs, its mbarriers ready, before a peer sends to it
    } else {
        __shared__ int s_reach[2];
        if (tid == 0) {
            s_reach[0] = 0;
            s_reach[1] = a.nb;
        }
        __syncthreads();
        for (int c = tid; c < a.grid; c += T) {
            const int2 pw = a.window[c];
            if (c < cta) atomicMax(&s_reach[0], pw.y);
            if (c > cta) atomicMin(&s_reach[1], pw.x);
        }
        __syncthreads();
        reach_lo = s_reach[0];
        reach_hi = s_reach[1];
    }
    // Of the CTA's matrix, what stays in L2 (keep_share).  FP32 waits for HBM and reads it
    // last: interleaved 24.2 and 34.5 us an iteration at 840x840 and 1000x1000, last 23.0-24.3
    // and 33.7 (by s mod 16 alone, always the same warps', 24.9 and 35.2).  FP64 shares its
    // time with the pipe and has it interleaved: 45.2 us at 640x640, last 46.2.
    auto keep_slice = [&](int s) {
        if constexpr (MIXED) return (se - s) * 16 <= (se - sb) * a.keep;
        else return ((s + 5 * (s >> 5)) & 15) < a.keep;
    };
    // z of a node to whoever has it in a window; cluster: for the r.r and r.z sum in fixed
    // point (mbarrier 1) or in FP64 (3).
    int z_bar = 3;
    const unsigned halo_bytes = static_cast<unsigned>(halo * static_cast<int>(sizeof(V)));
    auto publish = [&](int node, V zv) {
        if constexpr (SYNC == kCluster) {
            const int peers = sh.peers;
            for (int p = 0; p < peers; ++p) {
                const int4 e = sh.peer[p];
                if (node >= e.x && node < e.y)
                    send(peer_address(zh + (node + e.z), e.w), zv, peer_address(sh.mbar + z_bar, e.w));
            }
        } else if (node < reach_lo || node >= reach_hi) {
            if constexpr (SYNC == kTagged)
                publish_tagged(static_cast<u64*>(a.z) + static_cast<size_t>(node) * kTagWords<V>, zv, tag);
            else
                __stcg(static_cast<V*>(a.z) + node, zv);
        }
    };
    // z of the halo, by the warps past the first, while warp 0 waits for the sums.
    auto fetch = [&] {
        if constexpr (SYNC == kTagged) {
            bool ok = true;
            for (int j = tid - 32; j < halo && ok; j += T - 32) {
                const int node = j < left ? w0 + j : n1 + (j - left);
                const u64* w = static_cast<const u64*>(a.z) + static_cast<size_t>(node) * kTagWords<V>;
                V zv;
                ok = spin(a.status, g.limit, [&] { return read_tagged(w, tag, zv); });
                zh[j] = zv;
            }
            if (!ok) sh.fail = 1;
        }
    };
    auto nothing = [] {};

    auto solve = [&]() -> bool {
    // ---- start: x, r, z; r.r (FP64) and r.z
    {
        double t[2] = {0.0, 0.0};
        tag += 1;
        each_node([&](int, int node, int at) {
            double2 xv = make_double2(0.0, 0.0), rv;
            if (a.x0) {
                xv = reinterpret_cast<const double2*>(a.x0)[node];
                rv = residual_row<kWide>(a, node, a.x0);
            } else {
                rv = __ldg(reinterpret_cast<const double2*>(a.f) + node);
            }
            const V rw = to_working(rv, V{});
            const V zv = precond_at<PRECOND>(a, node, rw);
            r[at] = rw;
            q[at] = zv;
            own[at] = V{};
            if constexpr (MIXED) {
                reinterpret_cast<double2*>(a.x)[node] = xv;
                xs[at] = V{};
                xl[at] = V{};
            } else {
                xs[at] = xv;
            }
            publish(node, zv);
            t[0] += rv.x * rv.x + rv.y * rv.y;
            t[1] += static_cast<double>(rw.x * zv.x + rw.y * zv.y);
        });
        for (int j = tid; j < halo; j += T) win[j < left ? j : j + (n1 - n0)] = V{};
        const bool ok = reduce<SYNC, false, kRr, 2, true, false>(
            a, sh, g, s_red, t, 0u, halo_bytes, fetch, [&](const double* s) {
                r0 = sqrt(fmax(0.0, s[0]));
                assign(rho, s[1]);
                assign(rr_last, s[0]);
                rr_max = static_cast<float>(s[0]);
                rtrue = rtrue_prev = r0;
                Tot t0;
                assign(t0, s[0]);
                set_scale(sh, kRr, t0);
                set_scale(sh, kRz, rho);
                sh.beta = 0.f;
                sh.beta64 = 0.0;
                if (r0 <= a.target) {
                    converged = 1;
                    sh.next = kStop;
                } else if (!(s[1] > 0.0) || !isfinite(s[1])) {
                    status = LFGPU_ERR_RHO_INITIAL;
                    sh.next = kStop;
                }
            });
        if (!ok) return false;
    }

    while (sh.next != kStop) {
        // ---- p = z + beta p over the window
        if constexpr (MIXED) {
            const float beta = sh.beta;
            auto turn = [&](float2& p, float2 zv) { p = make_float2(pnew(zv.x, p.x, beta), pnew(zv.y, p.y, beta)); };
            each_node([&](int, int, int at) { turn(own[at], q[at]); });
            for (int j = tid; j < halo; j += T) {
                const int place = j < left ? j : j + (n1 - n0);
                turn(win[place], kPublish ? __ldcg(static_cast<const V*>(a.z) + w0 + place) : zh[j]);
            }
        } else {
            const double beta = sh.beta64;
            auto turn = [&](double2& p, double2 zv) { p = make_double2(fma(beta, p.x, zv.x), fma(beta, p.y, zv.y)); };
            each_node([&](int, int, int at) { turn(own[at], q[at]); });
            for (int j = tid; j < halo; j += T) {
                const int place = j < left ? j : j + (n1 - n0);
                turn(win[place], kPublish ? __ldcg(static_cast<const V*>(a.z) + w0 + place) : zh[j]);
            }
        }
        __syncthreads();
        // ---- q = K p, p.q
        {
            Sum t[1] = {};
            each_node([&](int s, int node, int at) {
                const V y = slice_row<CACHED>(a, s, node, win, node - w0, keep_slice(s) ? pol_keep : pol_stream);
                const V p = own[at];
                q[at] = y;
                if constexpr (MIXED) t[0].add(p.x * y.x + p.y * y.y);
                else t[0] += p.x * y.x + p.y * y.y;
            });
            const bool ok = reduce<SYNC, MIXED, kPq, 1, false, true>(
                a, sh, g, s_red, t, it32, 0u, nothing, [&](const Tot* s) {
                    set_scale(sh, kPq, s[0]);
                    if (!positive(s[0])) {
                        status = LFGPU_ERR_NOT_SPD;
                        sh.next = kStop;
                    } else if constexpr (MIXED) {
                        quotient(rho, s[0], sh.alpha, sh.alpha_lo);
                    } else {
                        sh.alpha64 = rho / s[0];
                    }
                });
            if (!ok) return false;
        }
        if (sh.next == kStop) break;
        // ---- x += alpha p, r -= alpha q, z = M^-1 r; r.r and r.z
        {
            Sum t[2] = {};
            tag += 1;
            z_bar = sh.e[kRr] != kNoScale && sh.e[kRz] != kNoScale ? 1 : 3;
            if constexpr (MIXED) {
                const float alpha = sh.alpha, alpha_lo = sh.alpha_lo;
                each_node([&](int, int node, int at) {
                    const float2 p = own[at], qv = q[at];
                    float2 rv = r[at], hv = xs[at], lv = xl[at];
                    rv.x -= alpha * qv.x;
                    rv.y -= alpha * qv.y;
                    const float2 zv = precond_at<PRECOND>(a, node, rv);
                    publish(node, zv);
                    r[at] = rv;
                    q[at] = zv;
                    pair_axpy(hv.x, lv.x, alpha, alpha_lo, p.x);
                    pair_axpy(hv.y, lv.y, alpha, alpha_lo, p.y);
                    xs[at] = hv;
                    xl[at] = lv;
                    t[0].add(rv.x * rv.x + rv.y * rv.y);
                    t[1].add(rv.x * zv.x + rv.y * zv.y);
                });
            } else {
                const double alpha = sh.alpha64;
                each_node([&](int, int node, int at) {
                    const double2 p = own[at], qv = q[at];
                    double2 rv = r[at], xv = xs[at];
                    rv.x -= alpha * qv.x;
                    rv.y -= alpha * qv.y;
                    const double2 zv = precond_at<PRECOND>(a, node, rv);
                    publish(node, zv);
                    r[at] = rv;
                    q[at] = zv;
                    xv.x += alpha * p.x;
                    xv.y += alpha * p.y;
                    xs[at] = xv;
                    t[0] += rv.x * rv.x + rv.y * rv.y;
                    t[1] += rv.x * zv.x + rv.y * zv.y;
                });
            }
            const bool ok = reduce<SYNC, MIXED, kRr, 2, kPublish, true>(
                a, sh, g, s_red, t, it32, halo_bytes, fetch, [&](const Tot* s) {
                    set_scale(sh, kRr, s[0]);
                    set_scale(sh, kRz, s[1]);
                    it += 1;
                    if constexpr (MIXED) {
                        // Only decides when to replace the residual: FP32 is enough.
                        const float rr = fmaxf(0.f, s[0].hi);
                        rr_max = fmaxf(rr_max, rr);
                        if (rr <= refine_below * rr_max || rr <= stop_below || it >= a.maxit) {
                            sh.next = kRefine;
                        } else if (!positive(s[1])) {
                            status = LFGPU_ERR_RHO;
                            sh.next = kStop;
                        } else {
                            float lo;
                            quotient(s[1], rho, sh.beta, lo);
                            rho = s[1];
                        }
                    } else {
                        rr_last = s[0];
                        if (!(s[0] > a.target2)) {  // NaN counts as zero, as in the reference
                            converged = 1;
                            sh.next = kStop;
                        } else if (!positive(s[1])) {
                            status = LFGPU_ERR_RHO;
                            sh.next = kStop;
                        } else {
                            sh.beta64 = s[1] / rho;
                            rho = s[1];
                            if (it >= a.maxit) sh.next = kStop;
                        }
                    }
                });
            if (!ok) return false;
            it32 += 1;
        }
        // ---- residual replacement: x += correction, r = f - K x in FP64, z, beta
        if constexpr (MIXED) {
            if (sh.next != kRefine) continue;
            double2* x2 = reinterpret_cast<double2*>(a.x);
            each_node([&](int, int node, int at) {
                const float2 hv = xs[at], lv = xl[at];
                double2 xv = x2[node];
                xv.x += static_cast<double>(hv.x) + static_cast<double>(lv.x);
                xv.y += static_cast<double>(hv.y) + static_cast<double>(lv.y);
                x2[node] = xv;
                xs[at] = V{};
                xl[at] = V{};
            });
            // The residual reads x of the other CTAs' nodes.
            if (!meet(a, sh, g)) return false;
            double t[2] = {0.0, 0.0};
            tag += 1;
            z_bar = 3;
            each_node([&](int, int node, int at) {
                const double2 rv = residual_row<kWide>(a, node, a.x);
                const float2 rw = to_working(rv, float2{});
                const float2 zv = precond_at<PRECOND>(a, node, rw);
                publish(node, zv);
                r[at] = rw;
                q[at] = zv;
                t[0] += rv.x * rv.x + rv.y * rv.y;
                t[1] += static_cast<double>(rw.x * zv.x + rw.y * zv.y);
            });
            const bool ok = reduce<SYNC, false, kRr, 2, true, false>(
                a, sh, g, s_red, t, 0u, halo_bytes, fetch, [&](const double* s) {
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
                        rr_max = static_cast<float>(s[0]);
                    }
                    if (sh.next == kGo) {
                        if (!(s[1] > 0.0) || !isfinite(s[1])) {
                            status = LFGPU_ERR_RHO;
                            sh.next = kStop;
                        } else {
                            const double last = static_cast<double>(rho.hi) + static_cast<double>(rho.lo);
                            sh.beta = a.restart ? 0.f : static_cast<float>(s[1] / last);
                            assign(rho, s[1]);
                            Tot t0;
                            assign(t0, s[0]);
                            set_scale(sh, kRr, t0);
                            set_scale(sh, kRz, rho);
                        }
                    }
                });
            if (!ok) return false;
        }
    }
    return true;
    };
    const bool solved = solve();
    if constexpr (SYNC == kCluster) {
        if (a.grid > 1) {
            // No CTA leaves while a peer may still send to it.  After a wait that ran out
            // sends may be on their way that no phase here tracks: 100 us for them.
            cluster_barrier();
            if (!solved) {
                const u64 t0 = global_ns();
                while (global_ns() - t0 < 100000ull) {
                }
            }
        }
    }
    if (!solved) return;
    {
        double2* x2 = reinterpret_cast<double2*>(a.x);
        each_node([&](int, int node, int at) {
            if constexpr (MIXED) {
                const float2 hv = xs[at], lv = xl[at];
                double2 xv = x2[node];
                xv.x += static_cast<double>(hv.x) + static_cast<double>(lv.x);
                xv.y += static_cast<double>(hv.y) + static_cast<double>(lv.y);
                x2[node] = xv;
            } else {
                x2[node] = xs[at];
            }
        });
    }
    if (cta == 0 && tid == 0) {
        PcgResult res{};
        res.iterations = it;
        res.refinements = refs;
        res.initial_residual = r0;
        if constexpr (MIXED) res.final_residual = rtrue;
        else res.final_residual = sqrt(fmax(0.0, rr_last));
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
        atomicMax(info + 3, s_hi - s_lo - (n1 - n0));
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
    int sync = kPublished;
    int grid = 0, threads = 0, smem = 0;
    int window_cap = 0, halo_cap = 0, own_cap = 0, x_cap = 0;
    bool cached = false;
};

// Meshes up to these many nodes run in one cluster, up to these with tagged z.
constexpr int kClusterNodes64 = 3600, kClusterNodes32 = 8192;
constexpr int kTaggedNodes64 = 300000, kTaggedNodes32 = 400000;

int slices_of(const Context& c) { return static_cast<int>((c.n / 2 + kSlice - 1) / kSlice); }

Shape launch_shape(const Context& c, bool mixed) {
    const int nodes = static_cast<int>(c.n / 2), slices = slices_of(c);
    Shape s;
    if (nodes <= (mixed ? kClusterNodes32 : kClusterNodes64)) {
        s.sync = kCluster;
        s.grid = 1;
        while (s.grid < kMaxCluster && s.grid * (mixed ? 4 : 1) < slices) s.grid *= 2;
    } else {
        s.sync = nodes <= (mixed ? kTaggedNodes32 : kTaggedNodes64) ? kTagged : kPublished;
        s.grid = c.num_sms;
    }
    return s;
}

}  // namespace

// Of 16 slices, how many are to stay in L2 between iterations: all while the matrix is
// up to 3/4 of it, beyond that 3/10 of it, the rest of the L2 being the vectors' and the
// stream's.  us an iteration on GB300 (135 MB of L2), all kept / 3/10 of L2 / none:
// FP32 700x700 (83 MB) 14.1 / 18.9 / 20.3, 760x760 (97 MB) 19.3 / 19.8 / 21.4, 800x800
// (108 MB) 27.4 / 21.8 / -, 840x840 (119 MB) 32.4 / 24.3 / 25.4, 1000x1000 (169 MB)
// 44.1 / 33.7 / 34.9; FP64 560x560
// (96 MB) 38.1 / 37.5 / 38.4, 640x640 (125 MB) 49.0 / 45.4 / 47.0.
int keep_share(const Context& c, bool mixed) {
    const size_t padded = static_cast<size_t>(slices_of(c)) * kSlice;
    const size_t rows = static_cast<size_t>(c.resident.groups) * kSlice;
    const double bytes = mixed ? 144.0 * rows + 24.0 * padded : 272.0 * rows + 32.0 * padded;
    int l2 = 0;
    LF_CUDA(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, c.device));
    if (bytes <= 0.75 * l2) return 16;
    return static_cast<int>(16.0 * 0.3 * l2 / bytes + 0.5);
}

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
        LF_CUDA(cudaMemcpyAsync(grid.info, res.info.p, 4 * sizeof(int), cudaMemcpyDeviceToHost, c.stream));
        LF_CUDA(cudaStreamSynchronize(c.stream));
        grid.version = c.pattern_version;
    }
    if (grid.info[2] > 32767) return false;
    const int vec = mixed ? 8 : 16;
    int optin = 0;
    LF_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c.device));
    const int room = (optin - (mixed ? kStaticSmem32 : kStaticSmem64)) / vec;
    s.window_cap = (grid.info[0] + 1) & ~1;
    s.halo_cap = s.sync == kPublished ? 0 : (grid.info[3] + 1) & ~1;
    const int own = (slices + s.grid - 1) / s.grid * kSlice;
    int used = s.window_cap + s.halo_cap;
    if (used > room) return false;
    if (used + 2 * own <= room) {
        s.own_cap = own;
        used += 2 * own;
        const int x = (mixed ? 2 : 1) * own;
        if (used + x <= room) {
            s.x_cap = own;
            used += x;
        }
    }
    s.smem = vec * used;
    // The CTA's matrix share fits L1 beside its shared memory.
    const int row_bytes = mixed ? 8 * 16 + 16 + 16 + 8 + 12 : 8 * 32 + 32 + 16 + 24;
    s.cached = s.sync == kCluster || own * row_bytes + s.smem < optin - 24 * 1024;
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
    // Warps take the CTA's slices in rounds: no more warps than the rounds can use evenly,
    // in pairs (400x400, 33 slices: 18 warps twice rather than 32 and one).  us an iteration
    // on GB300 with as many as fit and so: mixed 300x300 5.8, 5.1; 400x400 7.9, 7.1; 560x560
    // 10.1, 9.05; FP64 300x300 14.4, 13.6; 400x400 21.9, 20.3; 560x560 38.2, 36.9.  A mixed
    // solve that waits for HBM wants the loads of all: 840x840 24.1, 24.7; 1000x1000 33.8, 34.9.
    int warps = std::min(max_threads(mixed, s.cached) / 32, own / kSlice);
    if (!(mixed && keep_share(c, mixed) < 16)) {
        const int rounds = (own / kSlice + warps - 1) / warps;
        warps = std::min(warps, ((own / kSlice + rounds - 1) / rounds + 1) & ~1);
    }
    s.threads = 32 * std::max(s.sync == kCluster ? 1 : 4, warps);
    return true;
}

// Everything a solve needs on the device, and the kernel's arguments; false when the
// resident kernel does not take the pattern.
static bool resident_setup(Context& c, const SolveSetup& s, Shape& sh, ResArgs& a) {
    if (!c.paired || c.num_sms >= 255 || c.n < 2) return false;  // a word counts arrivals in a byte (answered())
    const bool mixed = s.mixed != 0;
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
    a.halo_cap = sh.halo_cap;
    a.own_cap = sh.own_cap;
    a.x_cap = sh.x_cap;
    a.keep = keep_share(c, mixed);
    if (sh.sync == kTagged) {
        const size_t words = padded * (mixed ? kTagWords<float2> : kTagWords<double2>);
        res.tagged.ensure(words);
        LF_CUDA(cudaMemsetAsync(res.tagged.p, 0, words * sizeof(u64), c.stream));  // no tag of an earlier solve
        a.z = res.tagged.p;
    }
    constexpr int kWordCount = 2 * kSets * kSetStride;
    res.words.ensure(kWordCount);
    c.bar.ensure(1);
    c.partials.ensure(static_cast<size_t>(2) * sh.grid * kMaxReduce);
    c.pcg_result.ensure(1);
    LF_CUDA(cudaMemsetAsync(res.words.p, 0, kWordCount * sizeof(u64), c.stream));
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
    return true;
}

bool run_resident(Context& c, const SolveSetup& s, PcgResult* out, float* kernel_ms) {
    Shape sh;
    ResArgs a{};
    try {
        if (!resident_setup(c, s, sh, a)) return false;
    } catch (const Error& e) {
        if (e.code != LFGPU_ERR_NOMEM) throw;
        // No room for the slices beside K: the graph of kernels reads K as it is.
        c.resident.release();
        return false;
    }
    const bool mixed = s.mixed != 0, jac = s.precond == LFGPU_PRECOND_JACOBI;
    auto launch = [&](auto kernel) {
        allow_dynamic_smem(kernel, s.mixed ? kStaticSmem32 : kStaticSmem64);
        if (sh.sync == kCluster && sh.grid > 8)
            LF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(sh.grid);
        cfg.blockDim = dim3(sh.threads);
        cfg.dynamicSmemBytes = sh.smem;
        cfg.stream = c.stream;
        cudaLaunchAttribute attr[2] = {};
        attr[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;  // the rest of the SM's memory is L1
        attr[1].val.sharedMemCarveout = std::min(100, (sh.smem + kStaticSmem32) * 100 / (228 * 1024) + 1);
        if (sh.sync == kCluster) {
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = sh.grid;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        } else {  // every CTA resident at once, or the launch fails
            attr[0].id = cudaLaunchAttributeCooperative;
            attr[0].val.cooperative = 1;
        }
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        LF_CUDA(cudaEventRecord(c.ev_a, c.stream));
        LF_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
        LF_CUDA(cudaEventRecord(c.ev_b, c.stream));
        c.launches += 1;
    };
    auto by_sync = [&](auto m, auto p) {
        constexpr bool M = decltype(m)::value;
        constexpr int P = decltype(p)::value;
        if (sh.sync == kCluster) launch(resident_pcg<M, P, kCluster, true>);
        else if (sh.sync == kTagged && sh.cached) launch(resident_pcg<M, P, kTagged, true>);
        else if (sh.sync == kTagged) launch(resident_pcg<M, P, kTagged, false>);
        else launch(resident_pcg<M, P, kPublished, false>);
    };
    using J = std::integral_constant<int, LFGPU_PRECOND_JACOBI>;
    using B = std::integral_constant<int, LFGPU_PRECOND_BLOCK2>;
    if (mixed) jac ? by_sync(std::true_type{}, J{}) : by_sync(std::true_type{}, B{});
    else jac ? by_sync(std::false_type{}, J{}) : by_sync(std::false_type{}, B{});
    LF_CUDA(cudaMemcpyAsync(out, c.pcg_result.p, sizeof(PcgResult), cudaMemcpyDeviceToHost, c.stream));
    *kernel_ms = elapsed_ms(c);
    check_status(c);
    c.resident_ran = true;
    return true;
}

}  // namespace lfgpu
