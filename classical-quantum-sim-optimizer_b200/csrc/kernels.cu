// Per-gate statevector kernels for sm_100a (one HBM pass per operation).
//
// Each kernel restates one loop of src/engine.rs as a flat, coalesced pass:
// a thread owns IPT work items spaced one block-width apart, issues all of its
// 16-byte (c128) or 8-byte (c64) loads before any arithmetic, and touches only
// the amplitudes the operation changes (controls and fixed diagonal patterns
// are folded into the index map, so a CX moves half of the state, a CZ a quarter).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <type_traits>

#include "common.hpp"
#include "kernels.hpp"

namespace dq {
namespace k {
namespace {

using dev::CondList;
using dev::InsertSet;

constexpr int kThreads = 256;
constexpr int kIPT = 4;

inline void check_launch(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) fail(kCudaError, std::string(what) + ": " + cudaGetErrorString(e));
}

inline unsigned blocks_for(uint64_t items, int per_block) {
    uint64_t b = (items + per_block - 1) / per_block;
    if (b == 0) b = 1;
    if (b > 0x7fffffffULL) fail(kValueError, "launch too large");
    return unsigned(b);
}

InsertSet make_insert(std::vector<int> pos) {
    std::sort(pos.begin(), pos.end());
    if (pos.size() > 8) fail(kValueError, "too many fixed qubits in one operation");
    InsertSet s{};
    s.k = int(pos.size());
    for (size_t i = 0; i < pos.size(); i++) s.pos[i] = pos[i];
    return s;
}

// ---------------------------------------------------------------------------
// 1q gate / X on pairs
// ---------------------------------------------------------------------------
template <typename V>
__global__ void __launch_bounds__(kThreads) k_gate1q(V* __restrict__ s, int n, int nfree, uint64_t items, InsertSet ins,
                                                     uint64_t fixed, uint64_t tbit, double2 u00, double2 u01,
                                                     double2 u10, double2 u11, int is_x, CondList cond,
                                                     const uint64_t* __restrict__ cbits, int cwords) {
    const uint64_t start = uint64_t(blockIdx.x) * (kThreads * kIPT) + threadIdx.x;
    const uint64_t fmask = (uint64_t(1) << nfree) - 1;
    uint64_t idx[kIPT];
    bool act[kIPT];
    V a[kIPT], b[kIPT];
#pragma unroll
    for (int t = 0; t < kIPT; t++) {
        uint64_t g = start + uint64_t(t) * kThreads;
        act[t] = g < items;
        idx[t] = 0;
        if (act[t]) {
            uint64_t st = g >> nfree;
            idx[t] = (st << n) | dev::expand(g & fmask, ins) | fixed;
            if (cond.n && !dev::cond_ok(cond, cbits, cwords, st)) act[t] = false;
        }
        if (act[t]) {
            a[t] = s[idx[t]];
            b[t] = s[idx[t] + tbit];
        }
    }
    const V m00 = dev::from_d2<V>(u00), m01 = dev::from_d2<V>(u01);
    const V m10 = dev::from_d2<V>(u10), m11 = dev::from_d2<V>(u11);
#pragma unroll
    for (int t = 0; t < kIPT; t++) {
        if (!act[t]) continue;
        if (is_x) {
            s[idx[t]] = b[t];
            s[idx[t] + tbit] = a[t];
        } else {
            s[idx[t]] = dev::cadd(dev::cmul(m00, a[t]), dev::cmul(m01, b[t]));
            s[idx[t] + tbit] = dev::cadd(dev::cmul(m10, a[t]), dev::cmul(m11, b[t]));
        }
    }
}

// ---------------------------------------------------------------------------
// SWAP on (01, 10) pairs
// ---------------------------------------------------------------------------
template <typename V>
__global__ void __launch_bounds__(kThreads) k_swap(V* __restrict__ s, int n, int nfree, uint64_t items, InsertSet ins,
                                                   uint64_t fixed, uint64_t lowbit, uint64_t highbit, CondList cond,
                                                   const uint64_t* __restrict__ cbits, int cwords) {
    const uint64_t start = uint64_t(blockIdx.x) * (kThreads * kIPT) + threadIdx.x;
    const uint64_t fmask = (uint64_t(1) << nfree) - 1;
    uint64_t idx[kIPT];
    bool act[kIPT];
    V a[kIPT], b[kIPT];
#pragma unroll
    for (int t = 0; t < kIPT; t++) {
        uint64_t g = start + uint64_t(t) * kThreads;
        act[t] = g < items;
        idx[t] = 0;
        if (act[t]) {
            uint64_t st = g >> nfree;
            idx[t] = (st << n) | dev::expand(g & fmask, ins) | fixed;
            if (cond.n && !dev::cond_ok(cond, cbits, cwords, st)) act[t] = false;
        }
        if (act[t]) {
            a[t] = s[idx[t] | lowbit];
            b[t] = s[idx[t] | highbit];
        }
    }
#pragma unroll
    for (int t = 0; t < kIPT; t++) {
        if (!act[t]) continue;
        s[idx[t] | lowbit] = b[t];
        s[idx[t] | highbit] = a[t];
    }
}

// ---------------------------------------------------------------------------
// Diagonal gates
// ---------------------------------------------------------------------------
struct DiagTable {
    int k;
    int q[5];
    double2 d[32];
};

template <typename V>
__global__ void __launch_bounds__(kThreads) k_diag_full(V* __restrict__ s, int n, uint64_t items, DiagTable tab,
                                                        CondList cond, const uint64_t* __restrict__ cbits, int cwords) {
    const uint64_t start = uint64_t(blockIdx.x) * (kThreads * kIPT) + threadIdx.x;
    const uint64_t lmask = (uint64_t(1) << n) - 1;
#pragma unroll
    for (int t = 0; t < kIPT; t++) {
        uint64_t g = start + uint64_t(t) * kThreads;
        if (g >= items) continue;
        if (cond.n && !dev::cond_ok(cond, cbits, cwords, g >> n)) continue;
        uint64_t i = g & lmask;
        int j = 0;
        for (int q = 0; q < tab.k; q++) j = (j << 1) | int((i >> tab.q[q]) & 1);
        s[g] = dev::cmul(s[g], dev::from_d2<V>(tab.d[j]));
    }
}

template <typename V>
__global__ void __launch_bounds__(kThreads) k_diag_entry(V* __restrict__ s, int n, int nfree, uint64_t items,
                                                         InsertSet ins, uint64_t fixed, double2 val, CondList cond,
                                                         const uint64_t* __restrict__ cbits, int cwords) {
    const uint64_t start = uint64_t(blockIdx.x) * (kThreads * kIPT) + threadIdx.x;
    const uint64_t fmask = (uint64_t(1) << nfree) - 1;
    const V v = dev::from_d2<V>(val);
    uint64_t idx[kIPT];
    bool act[kIPT];
    V a[kIPT];
#pragma unroll
    for (int t = 0; t < kIPT; t++) {
        uint64_t g = start + uint64_t(t) * kThreads;
        act[t] = g < items;
        idx[t] = 0;
        if (act[t]) {
            uint64_t st = g >> nfree;
            idx[t] = (st << n) | dev::expand(g & fmask, ins) | fixed;
            if (cond.n && !dev::cond_ok(cond, cbits, cwords, st)) act[t] = false;
        }
        if (act[t]) a[t] = s[idx[t]];
    }
#pragma unroll
    for (int t = 0; t < kIPT; t++)
        if (act[t]) s[idx[t]] = dev::cmul(a[t], v);
}

// ---------------------------------------------------------------------------
// Dense k-qubit gates (k <= 5): gather 2^k amplitudes, multiply, scatter.
// ---------------------------------------------------------------------------
struct Offsets {
    uint64_t o[32];
};

template <typename V, int K>
__global__ void __launch_bounds__(kThreads) k_dense(V* __restrict__ s, int n, int nfree, uint64_t items, InsertSet ins,
                                                    Offsets off, const double2* __restrict__ m, CondList cond,
                                                    const uint64_t* __restrict__ cbits, int cwords) {
    constexpr int D = 1 << K;
    __shared__ double2 sm[D * D];
    for (int i = threadIdx.x; i < D * D; i += blockDim.x) sm[i] = m[i];
    __syncthreads();
    const uint64_t g = uint64_t(blockIdx.x) * kThreads + threadIdx.x;
    if (g >= items) return;
    const uint64_t st = g >> nfree;
    if (cond.n && !dev::cond_ok(cond, cbits, cwords, st)) return;
    const uint64_t base = (st << n) | dev::expand(g & ((uint64_t(1) << nfree) - 1), ins);
    V v[D];
#pragma unroll
    for (int j = 0; j < D; j++) v[j] = s[base | off.o[j]];
#pragma unroll 1
    for (int row = 0; row < D; row++) {
        V acc = dev::czero<V>();
#pragma unroll
        for (int col = 0; col < D; col++) acc = dev::cadd(acc, dev::cmul(dev::from_d2<V>(sm[row * D + col]), v[col]));
        s[base | off.o[row]] = acc;
    }
}

// ---------------------------------------------------------------------------
// Measurement: branch sums, per-state draw, collapse
// ---------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Deterministic block sum of two values; result valid in thread 0.
__device__ __forceinline__ void block_sum2(double& a, double& b) {
    __shared__ double sa[32], sb[32];
    a = warp_sum(a);
    b = warp_sum(b);
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) {
        sa[w] = a;
        sb[w] = b;
    }
    __syncthreads();
    if (w == 0) {
        int nw = (blockDim.x + 31) >> 5;
        a = lane < nw ? sa[lane] : 0.0;
        b = lane < nw ? sb[lane] : 0.0;
        a = warp_sum(a);
        b = warp_sum(b);
    }
}

template <typename V>
__global__ void __launch_bounds__(kThreads) k_prob2(const V* __restrict__ s, int n, int chunk_bits, int P, uint64_t qbit,
                                                    double* __restrict__ partial, CondList cond,
                                                    const uint64_t* __restrict__ cbits, int cwords) {
    const uint64_t st = blockIdx.x / P;
    const uint64_t c = blockIdx.x % P;
    if (cond.n && !dev::cond_ok(cond, cbits, cwords, st)) return;
    const uint64_t off = c << chunk_bits;
    const uint64_t base = (st << n) + off;
    const uint64_t len = uint64_t(1) << chunk_bits;
    double p0 = 0.0, p1 = 0.0;
    for (uint64_t i = threadIdx.x; i < len; i += blockDim.x) {
        double v = dev::norm2(s[base + i]);
        if ((off + i) & qbit)
            p1 += v;
        else
            p0 += v;
    }
    block_sum2(p0, p1);
    if (threadIdx.x == 0) {
        partial[(st * P + c) * 2] = p0;
        partial[(st * P + c) * 2 + 1] = p1;
    }
}

__global__ void k_measure_finalize(uint64_t W, int P, const double* __restrict__ partial,
                                   const uint64_t* __restrict__ rng_seed, uint64_t* __restrict__ draws,
                                   int* __restrict__ outcome, double* __restrict__ scale, uint64_t* __restrict__ cbits,
                                   int cwords, int64_t cbit, CondList cond, int* __restrict__ err) {
    const uint64_t st = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (st >= W) return;
    if (cond.n && !dev::cond_ok(cond, cbits, cwords, st)) {
        outcome[st] = -1;
        return;
    }
    double p0 = 0.0, p1 = 0.0;
    for (int c = 0; c < P; c++) {
        p0 += partial[(st * P + c) * 2];
        p1 += partial[(st * P + c) * 2 + 1];
    }
    double total = p0 + p1;
    if (!(isfinite(total) && total > 0.0)) {
        *err = 1;
        outcome[st] = -1;
        return;
    }
    uint64_t k = draws[st];
    draws[st] = k + 1;
    double r = dev::u64_to_unit(dev::chacha8_u64(rng_seed[st], k));
    int o = r < p1 / total ? 1 : 0;
    outcome[st] = o;
    scale[st] = 1.0 / sqrt(o ? p1 : p0);
    if (cbit >= 0) {
        uint64_t* w = cbits + st * uint64_t(cwords) + (uint64_t(cbit) >> 6);
        uint64_t bit = uint64_t(1) << (uint64_t(cbit) & 63);
        *w = o ? (*w | bit) : (*w & ~bit);
    }
}

template <typename V>
__global__ void __launch_bounds__(kThreads) k_collapse(V* __restrict__ s, int n, uint64_t items, int q,
                                                       const int* __restrict__ outcome,
                                                       const double* __restrict__ scale, int reset) {
    const uint64_t start = uint64_t(blockIdx.x) * (kThreads * kIPT) + threadIdx.x;
    const int nf = n - 1;
    const uint64_t fmask = (uint64_t(1) << nf) - 1;
    const uint64_t qb = uint64_t(1) << q;
#pragma unroll
    for (int t = 0; t < kIPT; t++) {
        uint64_t g = start + uint64_t(t) * kThreads;
        if (g >= items) continue;
        uint64_t st = g >> nf;
        int o = outcome[st];
        if (o < 0) continue;
        double sc = scale[st];
        uint64_t j = g & fmask;
        uint64_t low = qb - 1;
        uint64_t i0 = (st << n) | (j & low) | ((j & ~low) << 1);
        uint64_t i1 = i0 | qb;
        if (o == 0) {
            s[i0] = dev::cscale(s[i0], sc);
            s[i1] = dev::czero<V>();
        } else if (reset) {
            s[i0] = dev::cscale(s[i1], sc);
            s[i1] = dev::czero<V>();
        } else {
            s[i0] = dev::czero<V>();
            s[i1] = dev::cscale(s[i1], sc);
        }
    }
}

// A run of measurements, one CTA per state.  Each outcome fixes a qubit, and the
// next branch sums run over the amplitudes that agree with the outcomes so far,
// so the sums read two states' worth in all and nothing is written until the
// run ends: then the state is collapsed once (mode kChainKeep), reset (a run of
// one, kChainReset) or left as it is when nothing follows that reads it
// (kChainDiscard).  Separate measurements read and write 2.5 states each in
// three launches.  States of up to 12 qubits keep their squared magnitudes in
// shared memory.  Bound by L2 and HBM; 300 states of 15 qubits (157 MB): 89 us a
// run of one, 168 us one of all 15 qubits with the histogram's bits; the 15-qubit dynamic
// circuit of three rounds 3.7 -> 2.65 ms with it.
constexpr int kChainMax = 64;
constexpr int kChainCached = 12;
enum ChainMode : int { kChainDiscard = 0, kChainKeep = 1, kChainReset = 2 };

struct MeasureList {
    int count;
    uint8_t q[kChainMax];
    int64_t cbit[kChainMax];
};

__device__ __forceinline__ uint64_t deposit_mask(uint64_t x, uint64_t mask) {
    uint64_t out = 0;
    while (mask) {
        const uint64_t low = mask & (~mask + 1);
        if (x & 1) out |= low;
        x >>= 1;
        mask ^= low;
    }
    return out;
}

template <typename V>
__global__ void k_measure_chain(V* __restrict__ s, int n, const __grid_constant__ MeasureList ml, int mode,
                                CondList cond, const uint64_t* __restrict__ rng_seed, uint64_t* __restrict__ draws,
                                uint64_t* __restrict__ cbits, int cwords, int* __restrict__ err) {
    extern __shared__ double norms[];
    __shared__ double branch;
    __shared__ int result;
    const uint64_t st = blockIdx.x;
    if (cond.n && !dev::cond_ok(cond, cbits, cwords, st)) return;
    V* __restrict__ a = s + (st << n);
    const uint64_t len = uint64_t(1) << n;
    const bool cached = n <= kChainCached;
    if (cached) {
        for (uint64_t i = threadIdx.x; i < len; i += blockDim.x) norms[i] = dev::norm2(a[i]);
        __syncthreads();
    }
    uint64_t fixed = 0, value = 0;
    uint64_t drawn = threadIdx.x == 0 ? draws[st] : 0;
    for (int t = 0; t < ml.count; t++) {
        const uint64_t bit = uint64_t(1) << ml.q[t];
        double p0 = 0.0, p1 = 0.0;
        if (!(fixed & bit)) {
            const uint64_t free = (len - 1) ^ fixed;
            const uint64_t count = uint64_t(1) << __popcll(free);
            const uint64_t step = deposit_mask(blockDim.x, free);
            uint64_t i = deposit_mask(threadIdx.x, free);
            uint64_t k = threadIdx.x;
            // Four loads in flight: a CTA alone has to keep its state's reads going.
            for (; !cached && k + 3 * uint64_t(blockDim.x) < count; k += 4 * uint64_t(blockDim.x)) {
                V v[4];
                uint64_t at[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    at[u] = i;
                    v[u] = a[i | value];
                    i = ((i | ~free) + step) & free;
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const double x = dev::norm2(v[u]);
                    if (at[u] & bit)
                        p1 += x;
                    else
                        p0 += x;
                }
            }
            for (; k < count; k += blockDim.x) {
                const double v = cached ? norms[i | value] : dev::norm2(a[i | value]);
                if (i & bit)
                    p1 += v;
                else
                    p0 += v;
                i = ((i | ~free) + step) & free;
            }
            block_sum2(p0, p1);
        }
        if (threadIdx.x == 0) {
            if (fixed & bit) {  // measured before in this run: its branch holds everything
                p0 = value & bit ? 0.0 : branch;
                p1 = value & bit ? branch : 0.0;
            }
            const double total = p0 + p1;
            if (!(isfinite(total) && total > 0.0)) {
                *err = 1;
                result = -1;
            } else {
                const double r = dev::u64_to_unit(dev::chacha8_u64(rng_seed[st], drawn++));
                const int o = r < p1 / total ? 1 : 0;
                result = o;
                branch = o ? p1 : p0;
                const int64_t c = ml.cbit[t];
                if (c >= 0) {
                    uint64_t* w = cbits + st * uint64_t(cwords) + (uint64_t(c) >> 6);
                    const uint64_t cb = uint64_t(1) << (uint64_t(c) & 63);
                    *w = o ? (*w | cb) : (*w & ~cb);
                }
            }
        }
        __syncthreads();
        const int o = result;
        if (o < 0) break;
        fixed |= bit;
        if (o) value |= bit;
        __syncthreads();  // `result` is read before the next round writes it
    }
    if (threadIdx.x == 0) draws[st] = drawn;
    if (mode == kChainDiscard || fixed == 0) return;
    const double sc = 1.0 / sqrt(branch);
    if (mode == kChainReset) {
        for (uint64_t j = threadIdx.x; j < len / 2; j += blockDim.x) {
            const uint64_t i0 = (j & (fixed - 1)) | ((j & ~(fixed - 1)) << 1), i1 = i0 | fixed;
            a[i0] = dev::cscale(a[value ? i1 : i0], sc);
            a[i1] = dev::czero<V>();
        }
        return;
    }
    for (uint64_t i = threadIdx.x; i < len; i += 4 * uint64_t(blockDim.x)) {
        V v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint64_t at = i + u * uint64_t(blockDim.x);
            v[u] = at < len && (at & fixed) == value ? a[at] : dev::czero<V>();
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint64_t at = i + u * uint64_t(blockDim.x);
            if (at < len) a[at] = (at & fixed) == value ? dev::cscale(v[u], sc) : dev::czero<V>();
        }
    }
}

// ---------------------------------------------------------------------------
// State initialisation
// ---------------------------------------------------------------------------
template <typename V>
__global__ void k_set_first(V* s, int n, uint64_t W) {
    uint64_t st = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (st < W) {
        V one = dev::czero<V>();
        one.x = 1;
        s[st << n] = one;
    }
}

template <typename V>
__global__ void k_broadcast(V* __restrict__ dst, const V* __restrict__ src, int n, uint64_t items) {
    for (uint64_t g = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; g < items; g += uint64_t(gridDim.x) * blockDim.x)
        dst[g] = src[g & ((uint64_t(1) << n) - 1)];
}

// ---------------------------------------------------------------------------
// Probabilities, CDF, sampling
// ---------------------------------------------------------------------------
template <typename V>
__global__ void k_norm2(const V* __restrict__ s, double* __restrict__ out, uint64_t len) {
    for (uint64_t g = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; g < len; g += uint64_t(gridDim.x) * blockDim.x)
        out[g] = dev::norm2(s[g]);
}

// Marginal probabilities.  The state is read once, in index order: a CTA takes
// chunks of 2^c amplitudes (c <= 12), each thread the 2^c / 256 elements t + 256 j
// of a chunk, and adds the squared magnitudes of every chunk that only differs in
// unselected high qubits into its own 16 sums.  The sums then meet in shared
// memory, where those of one local output are added.  One CTA per value of the
// selected high qubits and per part of the unselected ones; the parts' tables
// are added by k_marginal_parts in order, so the result does not depend on
// scheduling.  Bound by HBM: 1.28 ms at 30 qubits of complex64 (6.7 TB/s), 88 us at 25
// of complex128 (6.1 TB/s); with one atomic add per amplitude it took 42 ms at 30 qubits.
constexpr int kMargBits = 12;  // local qubits of a chunk
constexpr int kMargThreads = 256;

struct MarginalPlan {
    int c;                     // local qubits
    int kl, kh;                // selected qubits below c, and from c up
    int parts_bits;
    uint64_t high_free;        // chunk-index bits of the unselected high qubits
    uint8_t local_q[kMargBits], local_out[kMargBits];  // selected local qubit -> output bit (ascending)
    uint8_t local_free[kMargBits];                     // unselected local qubits, ascending
    uint8_t high_q[64], high_out[64];                  // selected high qubit (chunk-index bit) -> output bit
};

__device__ __forceinline__ uint64_t deposit_bits(uint64_t x, const uint8_t* to, int n) {
    uint64_t r = 0;
    for (int i = 0; i < n; i++) r |= ((x >> i) & 1) << to[i];
    return r;
}

template <typename V>
__global__ void __launch_bounds__(kMargThreads, 2)
    k_marginal(const V* __restrict__ s, const __grid_constant__ MarginalPlan p, double* __restrict__ out,
               uint64_t nout) {
    constexpr int E = (1 << kMargBits) / kMargThreads;
    __shared__ double sums[1 << kMargBits];
    const uint32_t size = 1u << p.c;
    const uint64_t part = blockIdx.x & ((uint64_t(1) << p.parts_bits) - 1);
    const uint64_t h = blockIdx.x >> p.parts_bits;
    const uint64_t fixed = deposit_bits(h, p.high_q, p.kh);
    // Unselected high qubits: the part fixes the lowest of them, the loop runs over the others.
    uint64_t mine = 0, loop = p.high_free;
    for (int i = 0; i < p.parts_bits; i++) {
        const uint64_t low = loop & (~loop + 1);
        if ((part >> i) & 1) mine |= low;
        loop ^= low;
    }
    double acc[E];
#pragma unroll
    for (int j = 0; j < E; j++) acc[j] = 0.0;
    uint64_t at = 0;
    do {
        const V* __restrict__ chunk = s + ((fixed | mine | at) << p.c);
        V v[E];
#pragma unroll
        for (int j = 0; j < E; j++) {
            const uint32_t e = threadIdx.x + j * kMargThreads;
            v[j] = e < size ? chunk[e] : dev::czero<V>();
        }
#pragma unroll
        for (int j = 0; j < E; j++) acc[j] += dev::norm2(v[j]);
        at = ((at | ~loop) + 1) & loop;
    } while (at != 0);
#pragma unroll
    for (int j = 0; j < E; j++) {
        const uint32_t e = threadIdx.x + j * kMargThreads;
        if (e < size) sums[e] = acc[j];
    }
    __syncthreads();
    // Local output x: the sum over the 2^(c - kl) elements with its selected
    // bits, by G threads each and then by halves.
    const int fb = p.c - p.kl;
    const int gb = p.kl >= 8 ? 0 : (8 - p.kl < fb ? 8 - p.kl : fb);
    const uint32_t G = 1u << gb, lane = threadIdx.x & (G - 1);
    double* __restrict__ o = out + part * nout;
    const uint64_t high_out = deposit_bits(h, p.high_out, p.kh);
    const uint32_t step = kMargThreads >> gb;
    for (uint32_t x0 = 0; x0 < (1u << p.kl); x0 += step) {
        const uint32_t x = x0 + (threadIdx.x >> gb);
        double sum = 0.0;
        if (x < (1u << p.kl)) {
            const uint32_t base = uint32_t(deposit_bits(x, p.local_q, p.kl));
            for (uint32_t r = lane; r < (1u << fb); r += G)
                sum += sums[base | uint32_t(deposit_bits(r, p.local_free, fb))];
        }
        for (uint32_t w = G >> 1; w >= 32; w >>= 1) {  // G > 32 only where one round covers every output
            __syncthreads();
            sums[threadIdx.x] = sum;
            __syncthreads();
            if (lane < w) sum += sums[threadIdx.x + w];
        }
        for (uint32_t w = G >= 32 ? 16 : G >> 1; w > 0; w >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, w);
        if (lane == 0 && x < (1u << p.kl)) o[high_out | deposit_bits(x, p.local_out, p.kl)] = sum;
    }
}

// Small states, which L2 holds and which few CTAs would read by chunks: a group of
// 2^G_bits threads per output gathers its terms, then adds them in a fixed order.
// A query of 8 of 16 qubits takes 45 us, 55 by chunks, of 2 of 12 qubits 35 and 42, of 10 of
// 20 qubits 96 and 105. Up to four terms a thread; with eight (1 of 12 qubits, 4 of 15) the
// chunks are 1 to 3 us quicker, and from 21 qubits on they are for nearly all selections.
constexpr int kGatherQubits = 20, kGatherBits = 8;
constexpr uint64_t kGatherTerms = 4;

struct GatherPlan {
    int k, G_bits;
    uint8_t q[64];   // selected qubits, output bit k - 1 first
    uint64_t rest;   // the others
};

template <typename V>
__global__ void __launch_bounds__(256) k_marginal_gather(const V* __restrict__ s, int n, const __grid_constant__ GatherPlan p,
                                                        double* __restrict__ out, uint64_t nout) {
    __shared__ double sm[256];
    const int G = 1 << p.G_bits, lane = threadIdx.x & (G - 1);
    const uint64_t j = (uint64_t(blockIdx.x) * 256 + threadIdx.x) >> p.G_bits;
    double acc = 0.0;
    if (j < nout) {
        uint64_t base = 0;
        for (int t = 0; t < p.k; t++) base |= ((j >> (p.k - 1 - t)) & 1) << p.q[t];
        const uint64_t terms = uint64_t(1) << (n - p.k);
        for (uint64_t r = lane; r < terms; r += G) acc += dev::norm2(s[base | deposit_mask(r, p.rest)]);
    }
    sm[threadIdx.x] = acc;
    __syncthreads();
    for (int w = G >> 1; w > 0; w >>= 1) {
        if (lane < w) sm[threadIdx.x] += sm[threadIdx.x + w];
        __syncthreads();
    }
    if (lane == 0 && j < nout) out[j] = sm[threadIdx.x];
}

// A CTA adds 32 outputs, eight threads each: thread y the parts y, y + 8, ...,
// then the eight in order (one thread each took 17 us for 256 outputs of 1,024 parts).
__global__ void __launch_bounds__(256) k_marginal_parts(const double* __restrict__ parts, uint64_t nout, int count,
                                                        double* __restrict__ out) {
    __shared__ double sm[8][32];
    const uint64_t j = uint64_t(blockIdx.x) * 32 + threadIdx.x;
    double sum = 0.0;
    if (j < nout) {
#pragma unroll 8
        for (int i = int(threadIdx.y); i < count; i += 8) sum += parts[uint64_t(i) * nout + j];
    }
    sm[threadIdx.y][threadIdx.x] = sum;
    __syncthreads();
    if (threadIdx.y == 0 && j < nout) {
        for (int y = 1; y < 8; y++) sum += sm[y][threadIdx.x];
        out[j] = sum;
    }
}

constexpr int kScanItems = 8;
constexpr int kScanTile = 256 * kScanItems;
static_assert(kScanTile == kScanTileEntries, "the tile that callers index by");

// Tile-local inclusive scan of `in` into x (V = double: in == x, in place;
// V = float2 / double2: the squared magnitudes of a state, as k_norm2 computes
// them, so the probability table is never written and re-read).
template <typename V>
__global__ void __launch_bounds__(256) k_scan_tiles(const V* __restrict__ in, double* __restrict__ x, uint64_t len,
                                                    double* __restrict__ sums) {
    __shared__ double warp_tot[8];
    const uint64_t base = uint64_t(blockIdx.x) * kScanTile + uint64_t(threadIdx.x) * kScanItems;
    double v[kScanItems];
    double run = 0.0;
    // A whole run of complex64 amplitudes is read as 16-byte vectors (two
    // amplitudes each); the sums are the same, in the same order.
    const bool full = base + kScanItems <= len;
    bool done = false;
    if constexpr (std::is_same<V, float2>::value) {
        if (full && (reinterpret_cast<uintptr_t>(in) & 15) == 0) {
            const float4* p = reinterpret_cast<const float4*>(in + base);
            float4 f[kScanItems / 2];
#pragma unroll
            for (int i = 0; i < kScanItems / 2; i++) f[i] = p[i];
#pragma unroll
            for (int i = 0; i < kScanItems / 2; i++) {
                run += dev::norm2(make_float2(f[i].x, f[i].y));
                v[2 * i] = run;
                run += dev::norm2(make_float2(f[i].z, f[i].w));
                v[2 * i + 1] = run;
            }
            done = true;
        }
    }
    if (!done) {
#pragma unroll
        for (int i = 0; i < kScanItems; i++) {
            double e = 0.0;
            if (base + i < len) {
                if constexpr (std::is_same<V, double>::value)
                    e = in[base + i];
                else
                    e = dev::norm2(in[base + i]);
            }
            run += e;
            v[i] = run;
        }
    }
    // inclusive warp scan of thread totals
    double t = run;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        double y = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += y;
    }
    if (lane == 31) warp_tot[w] = t;
    __syncthreads();
    double wprefix = 0.0;
    for (int i = 0; i < w; i++) wprefix += warp_tot[i];
    double excl = wprefix + t - run;
    if (full && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        double2* px = reinterpret_cast<double2*>(x + base);
#pragma unroll
        for (int i = 0; i < kScanItems / 2; i++) px[i] = make_double2(v[2 * i] + excl, v[2 * i + 1] + excl);
    } else {
#pragma unroll
        for (int i = 0; i < kScanItems; i++)
            if (base + i < len) x[base + i] = v[i] + excl;
    }
    if (threadIdx.x == 255) {
        double tot = 0.0;
        for (int i = 0; i < 8; i++) tot += warp_tot[i];
        sums[blockIdx.x] = tot;
    }
}

__global__ void k_scan_add(double* __restrict__ x, uint64_t len, const double* __restrict__ sums) {
    const uint64_t blk = blockIdx.x + 1;  // tile 0 needs no offset
    const double add = sums[blk - 1];
    for (uint64_t i = threadIdx.x; i < kScanTile; i += blockDim.x) {
        uint64_t g = blk * kScanTile + i;
        if (g < len) x[g] += add;
    }
}

// Entry i of running sums kept in two levels: tile-local sums x plus the
// inclusive sums of whole tiles before it (the same addition k_scan_add makes).
__device__ __forceinline__ double two_level(const double* __restrict__ x, const double* __restrict__ tiles,
                                            uint64_t i) {
    double v = x[i];
    if (tiles && i >= uint64_t(kScanTile)) v = v + tiles[i / uint64_t(kScanTile) - 1];
    return v;
}

__global__ void k_take_total(const double* __restrict__ cdf, uint64_t len, const double* __restrict__ tiles,
                             double* scalar, int* err) {
    double t = two_level(cdf, tiles, len - 1);
    *scalar = t;
    if (!(isfinite(t) && t > 0.0)) *err = 1;
}

// The table holds unnormalised running sums; each probe normalises the entry it
// reads (by the total, clamped to 1 when clamp, the last entry 1).
__global__ void k_sample(const double* __restrict__ cdf, uint64_t len, uint64_t seed, uint64_t shots, int per_shot,
                         const double* __restrict__ tiles, const double* __restrict__ total_dev, int clamp,
                         uint64_t* __restrict__ out) {
    uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= shots) return;
    const double total = *total_dev;
    uint64_t v = per_shot ? dev::chacha8_u64(seed + t, 0) : dev::chacha8_u64(seed, t);
    double draw = dev::u64_to_unit(v);
    uint64_t lo = 0, hi = len;
    while (lo < hi) {
        uint64_t mid = lo + (hi - lo) / 2;
        double c = two_level(cdf, tiles, mid) / total;
        if (clamp) c = fmin(c, 1.0);
        if (mid == len - 1) c = 1.0;
        if (c <= draw)
            lo = mid + 1;
        else
            hi = mid;
    }
    out[t] = lo < len - 1 ? lo : len - 1;
}

template <typename V>
__global__ void __launch_bounds__(256) k_dot(const V* __restrict__ a, const double2* __restrict__ b, uint64_t len,
                                            double2* __restrict__ partial) {
    double re = 0.0, im = 0.0;
    for (uint64_t g = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; g < len; g += uint64_t(gridDim.x) * blockDim.x) {
        V x = a[g];
        double2 y = b[g];
        double xr = x.x, xi = -double(x.y);
        re += xr * y.x - xi * y.y;
        im += xr * y.y + xi * y.x;
    }
    block_sum2(re, im);
    if (threadIdx.x == 0) partial[blockIdx.x] = make_double2(re, im);
}

template <typename VA, typename VB>
__global__ void __launch_bounds__(256) k_compare(const VA* __restrict__ a, const VB* __restrict__ b, uint64_t len,
                                                double* __restrict__ partial) {
    double re = 0.0, im = 0.0, mx = 0.0, na = 0.0, nb = 0.0;
    for (uint64_t g = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; g < len; g += uint64_t(gridDim.x) * blockDim.x) {
        VA x = a[g];
        VB y = b[g];
        double xr = x.x, xi = x.y, yr = y.x, yi = y.y;
        re += xr * yr + xi * yi;
        im += xr * yi - xi * yr;
        na += xr * xr + xi * xi;
        nb += yr * yr + yi * yi;
        double dr = xr - yr, di = xi - yi;
        mx = fmax(mx, sqrt(dr * dr + di * di));
    }
    block_sum2(re, im);
    __syncthreads();  // block_sum2's shared partials are reused below
    block_sum2(na, nb);
    __shared__ double smx[32];
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) smx[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = 0.0;
        for (int w = 0; w < int(blockDim.x >> 5); w++) m = fmax(m, smx[w]);
        partial[blockIdx.x * 5] = re;
        partial[blockIdx.x * 5 + 1] = im;
        partial[blockIdx.x * 5 + 2] = m;
        partial[blockIdx.x * 5 + 3] = na;
        partial[blockIdx.x * 5 + 4] = nb;
    }
}

template <typename V>
__global__ void k_gather(const V* __restrict__ s, const uint64_t* __restrict__ idx, uint64_t count,
                         double2* __restrict__ out) {
    for (uint64_t g = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; g < count; g += uint64_t(gridDim.x) * blockDim.x) {
        const V v = s[idx[g]];
        out[g] = make_double2(v.x, v.y);
    }
}

// Partials of sum_i (-1)^popcount((i ^ x) & z) conj(a_i) a_(i ^ x): <a|X^x Z^z|a>.
template <typename V>
__global__ void __launch_bounds__(256) k_pauli(const V* __restrict__ a, uint64_t len, uint64_t x, uint64_t z,
                                              double2* __restrict__ partial) {
    double re = 0.0, im = 0.0;
    for (uint64_t g = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; g < len; g += uint64_t(gridDim.x) * blockDim.x) {
        const V u = a[g];
        const V w = a[g ^ x];
        const double sgn = (__popcll((g ^ x) & z) & 1) ? -1.0 : 1.0;
        const double ur = u.x, ui = -double(u.y);
        re += sgn * (ur * w.x - ui * w.y);
        im += sgn * (ur * w.y + ui * w.x);
    }
    block_sum2(re, im);
    if (threadIdx.x == 0) partial[blockIdx.x] = make_double2(re, im);
}

__global__ void k_widen(const float2* __restrict__ s, double2* __restrict__ out, uint64_t len) {
    for (uint64_t g = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; g < len; g += uint64_t(gridDim.x) * blockDim.x)
        out[g] = make_double2(s[g].x, s[g].y);
}

uint64_t control_fixed(const std::vector<Ctl>& controls) {
    uint64_t v = 0;
    for (auto& c : controls)
        if (c.value) v |= uint64_t(1) << c.qubit;
    return v;
}

template <typename V>
void gate1q_t(const Batch& b, int target, const std::vector<Ctl>& controls, const double2 u[4], bool is_x,
              const CondList& cond) {
    std::vector<int> pos{target};
    for (auto& c : controls) pos.push_back(c.qubit);
    InsertSet ins = make_insert(pos);
    int nfree = b.n - ins.k;
    uint64_t items = b.W << nfree;
    k_gate1q<V><<<blocks_for(items, kThreads * kIPT), kThreads, 0, b.stream>>>(
        static_cast<V*>(b.amps), b.n, nfree, items, ins, control_fixed(controls), uint64_t(1) << target, u[0], u[1],
        u[2], u[3], is_x ? 1 : 0, cond, b.cbits, b.cwords);
    check_launch("gate1q");
}

template <typename V>
void swap_t(const Batch& b, int qa, int qb, const std::vector<Ctl>& controls, const CondList& cond) {
    std::vector<int> pos{qa, qb};
    for (auto& c : controls) pos.push_back(c.qubit);
    InsertSet ins = make_insert(pos);
    int nfree = b.n - ins.k;
    uint64_t items = b.W << nfree;
    int lo = std::min(qa, qb), hi = std::max(qa, qb);
    k_swap<V><<<blocks_for(items, kThreads * kIPT), kThreads, 0, b.stream>>>(
        static_cast<V*>(b.amps), b.n, nfree, items, ins, control_fixed(controls), uint64_t(1) << lo, uint64_t(1) << hi,
        cond, b.cbits, b.cwords);
    check_launch("swap");
}

template <typename V>
void diagonal_t(const Batch& b, const std::vector<int>& qubits, const std::vector<double2>& diag,
                const CondList& cond) {
    const int kq = int(qubits.size());
    std::vector<int> nontrivial;
    for (int j = 0; j < (1 << kq); j++)
        if (!(diag[j].x == 1.0 && diag[j].y == 0.0)) nontrivial.push_back(j);
    if (nontrivial.empty()) return;
    if (int(nontrivial.size()) * 2 <= (1 << kq)) {
        InsertSet ins = make_insert(qubits);
        int nfree = b.n - kq;
        uint64_t items = b.W << nfree;
        for (int j : nontrivial) {
            uint64_t fixed = 0;
            for (int t = 0; t < kq; t++)
                if ((j >> (kq - 1 - t)) & 1) fixed |= uint64_t(1) << qubits[t];
            k_diag_entry<V><<<blocks_for(items, kThreads * kIPT), kThreads, 0, b.stream>>>(
                static_cast<V*>(b.amps), b.n, nfree, items, ins, fixed, diag[j], cond, b.cbits, b.cwords);
            check_launch("diag_entry");
        }
        return;
    }
    DiagTable tab{};
    tab.k = kq;
    for (int t = 0; t < kq; t++) tab.q[t] = qubits[t];
    for (int j = 0; j < (1 << kq); j++) tab.d[j] = diag[j];
    uint64_t items = b.W << b.n;
    k_diag_full<V><<<blocks_for(items, kThreads * kIPT), kThreads, 0, b.stream>>>(static_cast<V*>(b.amps), b.n, items,
                                                                                   tab, cond, b.cbits, b.cwords);
    check_launch("diag_full");
}

template <typename V, int K>
void dense_k(const Batch& b, const std::vector<int>& qubits, const double2* dm, const CondList& cond) {
    Offsets off{};
    for (int j = 0; j < (1 << K); j++) {
        uint64_t o = 0;
        for (int bit = 0; bit < K; bit++) o |= uint64_t((j >> (K - 1 - bit)) & 1) << qubits[bit];
        off.o[j] = o;
    }
    InsertSet ins = make_insert(qubits);
    int nfree = b.n - K;
    uint64_t items = b.W << nfree;
    k_dense<V, K><<<blocks_for(items, kThreads), kThreads, 0, b.stream>>>(static_cast<V*>(b.amps), b.n, nfree, items,
                                                                          ins, off, dm, cond, b.cbits, b.cwords);
    check_launch("dense");
}

template <typename V>
void dense_t(const Batch& b, const std::vector<int>& qubits, const double2* dm, const CondList& cond) {
    switch (qubits.size()) {
        case 1: dense_k<V, 1>(b, qubits, dm, cond); break;
        case 2: dense_k<V, 2>(b, qubits, dm, cond); break;
        case 3: dense_k<V, 3>(b, qubits, dm, cond); break;
        case 4: dense_k<V, 4>(b, qubits, dm, cond); break;
        case 5: dense_k<V, 5>(b, qubits, dm, cond); break;
        default: fail(kValueError, "Dense gate arity exceeds supported maximum");
    }
}

template <typename V>
void measure_t(const Batch& b, int qubit, int64_t cbit, bool reset, const CondList& cond) {
    int pbits = std::max(0, std::min(10, b.n - 12));
    int P = 1 << pbits;
    int chunk_bits = b.n - pbits;
    uint64_t grid = b.W * uint64_t(P);
    k_prob2<V><<<blocks_for(grid, 1), kThreads, 0, b.stream>>>(static_cast<const V*>(b.amps), b.n, chunk_bits, P,
                                                              uint64_t(1) << qubit, b.partial, cond, b.cbits, b.cwords);
    check_launch("prob2");
    k_measure_finalize<<<blocks_for(b.W, 128), 128, 0, b.stream>>>(b.W, P, b.partial, b.rng_seed, b.draws, b.outcome,
                                                                  b.scale, b.cbits, b.cwords, cbit, cond, b.err);
    check_launch("measure_finalize");
    uint64_t items = b.W << (b.n - 1);
    k_collapse<V><<<blocks_for(items, kThreads * kIPT), kThreads, 0, b.stream>>>(
        static_cast<V*>(b.amps), b.n, items, qubit, b.outcome, b.scale, reset ? 1 : 0);
    check_launch("collapse");
}

template <typename V>
void measure_draw_t(const Batch& b, int qubit, double draw, int* outcome_host) {
    const int pbits = std::max(0, std::min(10, b.n - 12));
    const int P = 1 << pbits;
    k_prob2<V><<<P, kThreads, 0, b.stream>>>(static_cast<const V*>(b.amps), b.n, b.n - pbits, P, uint64_t(1) << qubit,
                                            b.partial, CondList{}, b.cbits, b.cwords);
    check_launch("prob2");
    std::vector<double> part(size_t(P) * 2);
    cudaError_t e = cudaMemcpyAsync(part.data(), b.partial, part.size() * 8, cudaMemcpyDeviceToHost, b.stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(b.stream);
    if (e != cudaSuccess) fail(kCudaError, std::string("branch sums: ") + cudaGetErrorString(e));
    // The branch sums in the order k_measure_finalize adds them.
    double p0 = 0.0, p1 = 0.0;
    for (int c = 0; c < P; c++) {
        p0 += part[size_t(c) * 2];
        p1 += part[size_t(c) * 2 + 1];
    }
    const double total = p0 + p1;
    if (!(std::isfinite(total) && total > 0.0)) fail(kRuntimeError, "Cannot measure a state with nonfinite or zero norm");
    const int o = draw < p1 / total ? 1 : 0;  // engine.rs:405
    const double scale = 1.0 / std::sqrt(o ? p1 : p0);
    e = cudaMemcpyAsync(b.outcome, &o, sizeof(int), cudaMemcpyHostToDevice, b.stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(b.scale, &scale, sizeof(double), cudaMemcpyHostToDevice, b.stream);
    if (e != cudaSuccess) fail(kCudaError, std::string("measurement upload: ") + cudaGetErrorString(e));
    const uint64_t items = uint64_t(1) << (b.n - 1);
    k_collapse<V><<<blocks_for(items, kThreads * kIPT), kThreads, 0, b.stream>>>(static_cast<V*>(b.amps), b.n, items,
                                                                                  qubit, b.outcome, b.scale, 0);
    check_launch("collapse");
    // The host values above must not change before the copies read them.
    e = cudaStreamSynchronize(b.stream);
    if (e != cudaSuccess) fail(kCudaError, std::string("collapse: ") + cudaGetErrorString(e));
    *outcome_host = o;
}

// out[i * 2^nl + j] = left[j] * right[i]: the state of the merged block whose
// low nl qubits are the left block's (src/distributed/pblock/model.rs:216-230).
template <typename V>
__global__ void k_kron(const V* __restrict__ left, int nl, const V* __restrict__ right, uint64_t len,
                       V* __restrict__ out) {
    for (uint64_t g = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; g < len; g += uint64_t(gridDim.x) * blockDim.x)
        out[g] = dev::cmul(left[g & ((uint64_t(1) << nl) - 1)], right[g >> nl]);
}

unsigned stream_grid(uint64_t len) {
    uint64_t b = (len + 255) / 256;
    return unsigned(std::max<uint64_t>(1, std::min<uint64_t>(b, 148 * 32)));
}

}  // namespace

void gate1q(const Batch& b, int target, const std::vector<Ctl>& controls, const double2 u[4], bool is_x,
            const CondList& cond) {
    if (b.c64)
        gate1q_t<float2>(b, target, controls, u, is_x, cond);
    else
        gate1q_t<double2>(b, target, controls, u, is_x, cond);
}

void swap(const Batch& b, int qa, int qb, const std::vector<Ctl>& controls, const CondList& cond) {
    if (b.c64)
        swap_t<float2>(b, qa, qb, controls, cond);
    else
        swap_t<double2>(b, qa, qb, controls, cond);
}

void diagonal(const Batch& b, const std::vector<int>& qubits, const std::vector<double2>& diag, const CondList& cond) {
    if (b.c64)
        diagonal_t<float2>(b, qubits, diag, cond);
    else
        diagonal_t<double2>(b, qubits, diag, cond);
}

void dense(const Batch& b, const std::vector<int>& qubits, const double2* dm, const CondList& cond) {
    if (b.c64)
        dense_t<float2>(b, qubits, dm, cond);
    else
        dense_t<double2>(b, qubits, dm, cond);
}

void measure(const Batch& b, int qubit, int64_t cbit, bool reset, const CondList& cond) {
    if (b.c64)
        measure_t<float2>(b, qubit, cbit, reset, cond);
    else
        measure_t<double2>(b, qubit, cbit, reset, cond);
}

int sm_count() {
    int dev = 0, c = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev);
    return c > 0 ? c : 148;
}

int measure_chain_max() { return kChainMax; }

bool measure_chain_applies(const Batch& b, int count) {
    // Microseconds of both forms, fitted on one B200: a CTA streams its state
    // at about 60 GB/s, up to four a SM at a time; separate measurements take three
    // launches and 2.5 passes at 5.5 TB/s.
    const double bytes = double(uint64_t(1) << b.n) * (b.c64 ? 8.0 : 16.0);
    const double rounds = std::ceil(double(b.W) / (4.0 * sm_count()));
    const double chain = 4.0 + 1.5 * count + rounds * 3.0 * bytes / 60e3;
    const double separate = count * (12.0 + 2.5 * bytes * double(b.W) / 5.5e6);
    return chain < separate && b.W <= 0x7fffffffULL;
}

void measure_chain(const Batch& b, const std::vector<int>& qubits, const std::vector<int64_t>& cbits, bool keep,
                   bool reset, const dev::CondList& cond) {
    if (qubits.empty() || qubits.size() > size_t(kChainMax) || (reset && qubits.size() != 1))
        fail(kValueError, "a run of measurements holds 1 to 64 qubits");
    MeasureList ml{};
    ml.count = int(qubits.size());
    for (size_t i = 0; i < qubits.size(); i++) {
        ml.q[i] = uint8_t(qubits[i]);
        ml.cbit[i] = cbits[i];
    }
    const int threads = 1 << std::min(9, std::max(5, b.n - 2));
    const size_t smem = b.n <= kChainCached ? sizeof(double) << b.n : 0;
    const int mode = reset ? kChainReset : keep ? kChainKeep : kChainDiscard;
    if (b.c64)
        k_measure_chain<float2><<<blocks_for(b.W, 1), threads, smem, b.stream>>>(
            static_cast<float2*>(b.amps), b.n, ml, mode, cond, b.rng_seed, b.draws, b.cbits, b.cwords, b.err);
    else
        k_measure_chain<double2><<<blocks_for(b.W, 1), threads, smem, b.stream>>>(
            static_cast<double2*>(b.amps), b.n, ml, mode, cond, b.rng_seed, b.draws, b.cbits, b.cwords, b.err);
    check_launch("measure_chain");
}

void measure_draw(const Batch& b, int qubit, double draw, int* outcome) {
    if (b.W != 1) fail(kValueError, "a measurement with a given draw takes one state");
    if (b.c64)
        measure_draw_t<float2>(b, qubit, draw, outcome);
    else
        measure_draw_t<double2>(b, qubit, draw, outcome);
}

void kron(cudaStream_t s, bool c64, const void* left, int nl, const void* right, int nr, void* out) {
    const uint64_t len = uint64_t(1) << (nl + nr);
    if (c64)
        k_kron<float2><<<stream_grid(len), 256, 0, s>>>(static_cast<const float2*>(left), nl,
                                                         static_cast<const float2*>(right), len, static_cast<float2*>(out));
    else
        k_kron<double2><<<stream_grid(len), 256, 0, s>>>(static_cast<const double2*>(left), nl,
                                                          static_cast<const double2*>(right), len,
                                                          static_cast<double2*>(out));
    check_launch("kron");
}

void init_basis(const Batch& b) {
    size_t bytes = size_t(b.W << b.n) * (b.c64 ? 8 : 16);
    cudaMemsetAsync(b.amps, 0, bytes, b.stream);
    if (b.c64)
        k_set_first<float2><<<blocks_for(b.W, 128), 128, 0, b.stream>>>(static_cast<float2*>(b.amps), b.n, b.W);
    else
        k_set_first<double2><<<blocks_for(b.W, 128), 128, 0, b.stream>>>(static_cast<double2*>(b.amps), b.n, b.W);
    check_launch("init_basis");
}

void broadcast(const Batch& b, const void* src) {
    uint64_t items = b.W << b.n;
    if (b.c64)
        k_broadcast<float2><<<stream_grid(items), 256, 0, b.stream>>>(static_cast<float2*>(b.amps),
                                                                       static_cast<const float2*>(src), b.n, items);
    else
        k_broadcast<double2><<<stream_grid(items), 256, 0, b.stream>>>(static_cast<double2*>(b.amps),
                                                                        static_cast<const double2*>(src), b.n, items);
    check_launch("broadcast");
}

void norm2(const Batch& b, double* out) {
    uint64_t len = uint64_t(1) << b.n;
    if (b.c64)
        k_norm2<float2><<<stream_grid(len), 256, 0, b.stream>>>(static_cast<const float2*>(b.amps), out, len);
    else
        k_norm2<double2><<<stream_grid(len), 256, 0, b.stream>>>(static_cast<const double2*>(b.amps), out, len);
    check_launch("norm2");
}

namespace {
MarginalPlan marginal_plan(int n, const std::vector<int>& qubits) {
    MarginalPlan p{};
    p.c = std::min(n, kMargBits);
    const int k = int(qubits.size());
    std::vector<char> selected(size_t(n), 0);
    for (int b = 0; b < k; b++) {  // output bit b
        const int q = qubits[size_t(k - 1 - b)];
        selected[size_t(q)] = 1;
        if (q < p.c) {
            p.local_q[p.kl] = uint8_t(q);
            p.local_out[p.kl++] = uint8_t(b);
        } else {
            p.high_q[p.kh] = uint8_t(q - p.c);
            p.high_out[p.kh++] = uint8_t(b);
        }
    }
    int free = 0, high_free = 0;
    for (int q = 0; q < n; q++) {
        if (selected[size_t(q)]) continue;
        if (q < p.c) {
            p.local_free[free++] = uint8_t(q);
        } else {
            p.high_free |= uint64_t(1) << (q - p.c);
            high_free++;
        }
    }
    // About 8 CTAs to an SM, a part taking at least one chunk; up to four chunks
    // take less time in one CTA than a second launch.
    while (high_free > 2 && p.parts_bits < high_free && p.kh + p.parts_bits < 10) p.parts_bits++;
    return p;
}
}  // namespace

namespace {
bool gathers(int n, const std::vector<int>& qubits) {
    const int free = n - int(qubits.size());
    return n <= kGatherQubits && (uint64_t(1) << std::max(0, free - kGatherBits)) <= kGatherTerms;
}
}  // namespace

size_t marginal_scratch(int n, const std::vector<int>& qubits) {
    if (gathers(n, qubits)) return 0;
    const MarginalPlan p = marginal_plan(n, qubits);
    return p.parts_bits ? size_t(1) << (p.parts_bits + int(qubits.size())) : 0;
}

void marginal(const Batch& b, const std::vector<int>& qubits, double* out, double* scratch) {
    const uint64_t nout = uint64_t(1) << qubits.size();
    if (gathers(b.n, qubits)) {
        GatherPlan g{};
        g.k = int(qubits.size());
        g.G_bits = std::min(kGatherBits, b.n - g.k);
        g.rest = (uint64_t(1) << b.n) - 1;
        for (int t = 0; t < g.k; t++) {
            g.q[t] = uint8_t(qubits[size_t(t)]);
            g.rest &= ~(uint64_t(1) << qubits[size_t(t)]);
        }
        const unsigned grid = blocks_for(nout << g.G_bits, 256);
        if (b.c64)
            k_marginal_gather<float2><<<grid, 256, 0, b.stream>>>(static_cast<const float2*>(b.amps), b.n, g, out, nout);
        else
            k_marginal_gather<double2><<<grid, 256, 0, b.stream>>>(static_cast<const double2*>(b.amps), b.n, g, out, nout);
        check_launch("marginal");
        return;
    }
    const MarginalPlan p = marginal_plan(b.n, qubits);
    const unsigned grid = blocks_for(uint64_t(1) << (p.kh + p.parts_bits), 1);
    double* to = p.parts_bits ? scratch : out;
    if (b.c64)
        k_marginal<float2><<<grid, kMargThreads, 0, b.stream>>>(static_cast<const float2*>(b.amps), p, to, nout);
    else
        k_marginal<double2><<<grid, kMargThreads, 0, b.stream>>>(static_cast<const double2*>(b.amps), p, to, nout);
    check_launch("marginal");
    if (p.parts_bits) {
        k_marginal_parts<<<blocks_for(nout, 32), dim3(32, 8), 0, b.stream>>>(scratch, nout, 1 << p.parts_bits, out);
        check_launch("marginal_parts");
    }
}

size_t scan_tmp_size(uint64_t len) {
    size_t total = 0;
    while (len > uint64_t(kScanTile)) {
        len = (len + kScanTile - 1) / kScanTile;
        total += len;
    }
    return total + 1;
}

int scan_launches(uint64_t len) {
    const uint64_t nb = (len + kScanTile - 1) / kScanTile;
    return nb > 1 ? 2 + scan_launches(nb) : 1;
}

void scan(cudaStream_t s, double* x, uint64_t len, double* tmp) {
    uint64_t nb = (len + kScanTile - 1) / kScanTile;
    k_scan_tiles<double><<<blocks_for(nb, 1), 256, 0, s>>>(x, x, len, tmp);
    check_launch("scan_tiles");
    if (nb > 1) {
        scan(s, tmp, nb, tmp + nb);
        k_scan_add<<<blocks_for(nb - 1, 1), 256, 0, s>>>(x, len, tmp);
        check_launch("scan_add");
    }
}

void scan_probs(const Batch& b, double* x, double* tmp, bool add_tiles) {
    const uint64_t len = uint64_t(1) << b.n;
    const uint64_t nb = (len + kScanTile - 1) / kScanTile;
    if (b.c64)
        k_scan_tiles<float2><<<blocks_for(nb, 1), 256, 0, b.stream>>>(static_cast<const float2*>(b.amps), x, len, tmp);
    else
        k_scan_tiles<double2>
            <<<blocks_for(nb, 1), 256, 0, b.stream>>>(static_cast<const double2*>(b.amps), x, len, tmp);
    check_launch("scan_probs");
    if (nb > 1) {
        scan(b.stream, tmp, nb, tmp + nb);
        if (add_tiles) {
            k_scan_add<<<blocks_for(nb - 1, 1), 256, 0, b.stream>>>(x, len, tmp);
            check_launch("scan_add");
        }
    }
}

void scan_local(cudaStream_t s, double* x, uint64_t len, double* tmp) {
    uint64_t nb = (len + kScanTile - 1) / kScanTile;
    k_scan_tiles<double><<<blocks_for(nb, 1), 256, 0, s>>>(x, x, len, tmp);
    check_launch("scan_tiles");
    if (nb > 1) scan(s, tmp, nb, tmp + nb);
}

void scan_states(cudaStream_t s, bool c64, const void* amps, uint64_t len, double* x, double* tmp) {
    const uint64_t nb = (len + kScanTile - 1) / kScanTile;
    if (c64)
        k_scan_tiles<float2><<<blocks_for(nb, 1), 256, 0, s>>>(static_cast<const float2*>(amps), x, len, tmp);
    else
        k_scan_tiles<double2><<<blocks_for(nb, 1), 256, 0, s>>>(static_cast<const double2*>(amps), x, len, tmp);
    check_launch("scan_states");
    if (nb > 1) scan(s, tmp, nb, tmp + nb);
}

void take_total(cudaStream_t s, const double* cdf, uint64_t len, const double* tiles, double* scalar, int* err) {
    k_take_total<<<1, 1, 0, s>>>(cdf, len, tiles, scalar, err);
    check_launch("take_total");
}

void sample_sums(cudaStream_t s, const double* sums, const double* tiles, uint64_t len, const double* total_dev,
                 bool clamp, uint64_t seed, uint64_t shots, bool per_shot_seed, uint64_t* out) {
    if (shots == 0) return;
    k_sample<<<blocks_for(shots, 128), 128, 0, s>>>(sums, len, seed, shots, per_shot_seed ? 1 : 0, tiles, total_dev,
                                                     clamp ? 1 : 0, out);
    check_launch("sample");
}

int dot_partials(const Batch& b, const double2* other, double2* partial) {
    uint64_t len = uint64_t(1) << b.n;
    if (b.c64)
        k_dot<float2><<<kDotBlocks, 256, 0, b.stream>>>(static_cast<const float2*>(b.amps), other, len, partial);
    else
        k_dot<double2><<<kDotBlocks, 256, 0, b.stream>>>(static_cast<const double2*>(b.amps), other, len, partial);
    check_launch("dot");
    return kDotBlocks;
}

void gather(const Batch& b, const uint64_t* idx, uint64_t count, double2* out) {
    if (count == 0) return;
    const unsigned grid = unsigned(std::min<uint64_t>((count + 255) / 256, 1184));
    if (b.c64)
        k_gather<float2><<<grid, 256, 0, b.stream>>>(static_cast<const float2*>(b.amps), idx, count, out);
    else
        k_gather<double2><<<grid, 256, 0, b.stream>>>(static_cast<const double2*>(b.amps), idx, count, out);
    check_launch("gather");
}

int pauli_partials(const Batch& b, uint64_t x, uint64_t z, double2* partial) {
    const uint64_t len = uint64_t(1) << b.n;
    if (b.c64)
        k_pauli<float2><<<kDotBlocks, 256, 0, b.stream>>>(static_cast<const float2*>(b.amps), len, x, z, partial);
    else
        k_pauli<double2><<<kDotBlocks, 256, 0, b.stream>>>(static_cast<const double2*>(b.amps), len, x, z, partial);
    check_launch("pauli expectation");
    return kDotBlocks;
}

void compare(cudaStream_t s, const void* a, bool a64, const void* b, bool b64, uint64_t len, double* partial) {
    if (!a64 && !b64)
        k_compare<double2, double2><<<kDotBlocks, 256, 0, s>>>(static_cast<const double2*>(a),
                                                               static_cast<const double2*>(b), len, partial);
    else if (!a64 && b64)
        k_compare<double2, float2><<<kDotBlocks, 256, 0, s>>>(static_cast<const double2*>(a),
                                                              static_cast<const float2*>(b), len, partial);
    else if (a64 && !b64)
        k_compare<float2, double2><<<kDotBlocks, 256, 0, s>>>(static_cast<const float2*>(a),
                                                              static_cast<const double2*>(b), len, partial);
    else
        k_compare<float2, float2><<<kDotBlocks, 256, 0, s>>>(static_cast<const float2*>(a),
                                                             static_cast<const float2*>(b), len, partial);
    check_launch("compare");
}

void widen(const Batch& b, double2* out) {
    uint64_t len = uint64_t(1) << b.n;
    k_widen<<<stream_grid(len), 256, 0, b.stream>>>(static_cast<const float2*>(b.amps), out, len);
    check_launch("widen");
}

}  // namespace k
}  // namespace dq
