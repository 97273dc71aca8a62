// Tile passes as Pauli rotations: the sm_100a kernel (complex128).
#include <algorithm>
#include <cstring>
#include <string>

#include <cuda_pipeline.h>

#include "common.hpp"
#include "rotations.hpp"

namespace dq {
namespace k {
namespace {

constexpr int E = kRotEntries;

// A pass as a launch argument.
struct RotPass {
    int m, nphases;
    int data, ndata;  // words of the steps' data
    int tell;
    uint8_t q[kRotMaxTile];  // tile qubits, ascending
    uint16_t out_dir[kRotMaxTile];
    uint16_t out_outer[kRotMaxOuter];
    uint16_t out_const;
    uint32_t sign_local, sign_outer;
    int sign_const, outer_moves;
    // Tile index bits from m - 4 up, by their value k: offset in the state,
    // place on entry and on exit, and (bit k) sign.
    uint64_t reg_off[E];
    uint16_t reg_in[E], reg_out[E];
    uint32_t reg_sign;
};

struct RotWords {
    uint4 w[kRotParamWords];
};

// Programs: steps from the launch argument (uniform loads from the constant
// bank) and their data from shared memory.
struct ArgWords {
    const RotWords* a;
    const uint4* table;
    __device__ __forceinline__ uint4 operator()(uint32_t i) const { return a->w[i]; }
    __device__ __forceinline__ uint4 data(uint32_t i) const { return table[i]; }
    // (as doubles: taken apart from a uint4, each factor cost two register moves, a quarter of a table's instructions)
    __device__ __forceinline__ double2 factor(uint32_t i) const { return reinterpret_cast<const double2*>(table)[i]; }
};

__device__ __forceinline__ double lo_hi(uint32_t lo, uint32_t hi) { return __hiloint2double(int(hi), int(lo)); }
__device__ __forceinline__ double2 pair_of(uint4 u) { return make_double2(lo_hi(u.x, u.y), lo_hi(u.z, u.w)); }

__device__ __forceinline__ double2 cmul_fma(double2 a, double2 b) {
    return make_double2(fma(-a.y, b.y, a.x * b.x), fma(a.y, b.x, a.x * b.y));
}

// a <- a b in place: one temporary.
__device__ __forceinline__ void cmul_in_place(double2& a, double2 b) {
    const double t = a.y * b.y;
    a.y *= b.x;
    a.y = fma(a.x, b.y, a.y);
    a.x = fma(a.x, b.x, -t);
}

// x <- x - s t y, y <- y + s w x (kRotKept: y <- w y + s t x; kRotImag: x - i s t y, y - i s w x) on the pairs of
// entries that differ by D, x the one whose lowest bit of D is clear; s = -1
// where `signs` has the entry's bit.
template <int D, int KIND>
__device__ __forceinline__ void rotate(double2 (&a)[E], double t, double w, uint32_t signs) {
    constexpr int L = D & -D;
#pragma unroll
    for (int v = 0; v < E; v++) {
        if (v & L) continue;
        const int u = v ^ D;
        double tv = t, wv = w;
        if (KIND != int(kRotPlain)) {
            const int flip = int((signs << (31 - v)) & 0x80000000u);
            tv = __hiloint2double(__double2hiint(t) ^ flip, __double2loint(t));
            if (KIND != int(kRotKept)) wv = __hiloint2double(__double2hiint(w) ^ flip, __double2loint(w));
        }
        if (KIND == int(kRotKept)) {
            a[v].x = fma(-tv, a[u].x, a[v].x);
            a[v].y = fma(-tv, a[u].y, a[v].y);
            a[u].x = fma(tv, a[v].x, w * a[u].x);
            a[u].y = fma(tv, a[v].y, w * a[u].y);
        } else if (KIND == int(kRotImag)) {
            a[v].x = fma(tv, a[u].y, a[v].x);
            a[v].y = fma(-tv, a[u].x, a[v].y);
            a[u].x = fma(wv, a[v].y, a[u].x);
            a[u].y = fma(-wv, a[v].x, a[u].y);
        } else {
            a[v].x = fma(-tv, a[u].x, a[v].x);
            a[v].y = fma(-tv, a[u].y, a[v].y);
            a[u].x = fma(wv, a[v].x, a[u].x);
            a[u].y = fma(wv, a[v].y, a[u].y);
        }
    }
}

__device__ __forceinline__ uint32_t odd(uint32_t x) { return __popc(x) & 1u; }

// The rotations of a phase, fetched one ahead.
template <class W>
struct RotStream {
    const W& words;
    uint32_t at, index;
    uint4 w, d;
    __device__ __forceinline__ RotStream(const W& words_, uint32_t first, uint32_t index_)
        : words(words_), at(first), index(index_), w(words_(first)), d(words_(first + 1)) {}
    __device__ __forceinline__ void advance(uint32_t n) {
        at += n;
        w = words(at);
        d = words(at + 1);
    }
    __device__ __forceinline__ void plain(double& t, double& u) {
        t = lo_hi(w.x, w.y);
        u = lo_hi(w.z, w.w);
        advance(1);
    }
    // With the sign of this thread's slot.
    __device__ __forceinline__ void with_signs(double& t, double& u, uint32_t& signs, bool kept) {
        const uint32_t flip = odd(d.y & index) << 31;
        t = lo_hi(w.x, w.y ^ flip);
        u = lo_hi(w.z, kept ? w.w : w.w ^ flip);
        signs = d.x;
        advance(2);
    }
};

template <int J, class W>
__device__ __forceinline__ void unit_rotation(double2 (&a)[E], uint32_t what, RotStream<W>& rots) {
    const uint32_t kind = (what >> (2 * J)) & 3u;
    if (kind == 0) return;
    double t, u;
    uint32_t signs = 0;
    if (kind == kRotPlain + 1) {
        rots.plain(t, u);
        rotate<1 << J, int(kRotPlain)>(a, t, u, signs);
        return;
    }
    rots.with_signs(t, u, signs, kind == kRotKept + 1);
    if (kind == kRotSigned + 1)
        rotate<1 << J, int(kRotSigned)>(a, t, u, signs);
    else
        rotate<1 << J, int(kRotKept)>(a, t, u, signs);
}

__device__ __forceinline__ uint32_t mask_of(uint4 four, uint32_t i) {
    return i & 2 ? (i & 1 ? four.w : four.z) : (i & 1 ? four.y : four.x);
}

template <class W>
__device__ __forceinline__ void apply_step(double2 (&a)[E], const W& words, uint4 s, uint32_t index, RotStream<W>& rots) {
    if (s.x & 0xFFu) {
        unit_rotation<0>(a, s.x, rots);
        unit_rotation<1>(a, s.x, rots);
        unit_rotation<2>(a, s.x, rots);
        unit_rotation<3>(a, s.x, rots);
    }
    if (s.x & 0xF00u) {
        double t, u;
        uint32_t signs;
        rots.with_signs(t, u, signs, ((s.x >> 12) & 3u) == kRotKept);
        switch ((s.x >> 8) & 63u) {
#define DQ_ROT(D)                                                                        \
    case kRotSigned << 4 | D: rotate<D, int(kRotSigned)>(a, t, u, signs); break;         \
    case kRotKept << 4 | D: rotate<D, int(kRotKept)>(a, t, u, signs); break;             \
    case kRotImag << 4 | D: rotate<D, int(kRotImag)>(a, t, u, signs); break;
#define DQ_IMAG(D) \
    case kRotImag << 4 | D: rotate<D, int(kRotImag)>(a, t, u, signs); break;
            DQ_IMAG(1) DQ_IMAG(2) DQ_ROT(3) DQ_IMAG(4) DQ_ROT(5) DQ_ROT(6) DQ_ROT(7) DQ_IMAG(8)
            DQ_ROT(9) DQ_ROT(10) DQ_ROT(11) DQ_ROT(12) DQ_ROT(13) DQ_ROT(14) DQ_ROT(15)
#undef DQ_IMAG
#undef DQ_ROT
            default: break;
        }
    }
    if (s.x & kRotTable) {
#pragma unroll
        for (int v = 0; v < E; v++) cmul_in_place(a[v], words.factor(s.y + v));
    }
    if (s.x & kRotSlots) {
        const uint32_t n = s.w & 0xFFFFu, data = s.z + ((n + 3) >> 2);
        double2 z = make_double2(1.0, 0.0);
        for (uint32_t i = 0; i < n; i++) {
            uint4 c = words.data(data + i);
            c.w ^= odd(mask_of(words.data(s.z + (i >> 2)), i) & index) << 31;
            z = i ? cmul_fma(z, pair_of(c)) : pair_of(c);
        }
#pragma unroll
        for (int v = 0; v < E; v++) {
            const int hi = __double2hiint(z.y) ^ int((s.w << (15 - v)) & 0x80000000u);
            cmul_in_place(a[v], make_double2(z.x, __hiloint2double(hi, __double2loint(z.y))));
        }
    }
    if (s.x & kRotSlotModuli) {
        const uint32_t n = s.w & 0xFFFFu, data = s.z + ((n + 3) >> 2);
        double g = 1.0, h = 1.0;
        for (uint32_t i = 0; i < n; i++) {
            const double2 c = pair_of(words.data(data + i));
            const bool o = odd(mask_of(words.data(s.z + (i >> 2)), i) & index);
            g *= o ? c.y : c.x;
            h *= o ? c.x : c.y;
        }
#pragma unroll
        for (int v = 0; v < E; v++) {
            const double f = (s.w >> (16 + v)) & 1u ? h : g;
            a[v].x *= f;
            a[v].y *= f;
        }
    }
}

__device__ __forceinline__ uint32_t swz(uint32_t e) {
    const uint32_t f = (e >> 3) ^ (e >> 6) ^ (e >> 9) ^ (e >> 12);
    return e ^ (f & 7u);
}

// One phase of a tile: this thread's 16 amplitudes through the steps.
template <class W>
__device__ __forceinline__ void rotation_phase(double2* tile, const W& words, int ph, uint32_t slot, uint32_t index) {
    const uint4 h0 = words(3 * ph), h1 = words(3 * ph + 1), h2 = words(3 * ph + 2);
    const uint32_t ub[9] = {h1.x & 0xFFFFu, h1.x >> 16, h1.y & 0xFFFFu, h1.y >> 16, h1.z & 0xFFFFu,
                            h1.z >> 16,     h1.w & 0xFFFFu, h1.w >> 16, h2.x & 0xFFFFu};
    uint32_t place = 0;
#pragma unroll
    for (int b = 0; b < 9; b++) place ^= (slot >> b) & 1u ? ub[b] : 0u;
    const uint32_t vb[4] = {h0.z & 0xFFFFu, h0.z >> 16, h0.w & 0xFFFFu, h0.w >> 16};
    uint32_t vv[E];
#pragma unroll
    for (int v = 0; v < E; v++)
        vv[v] = (v & 1 ? vb[0] : 0u) ^ (v & 2 ? vb[1] : 0u) ^ (v & 4 ? vb[2] : 0u) ^ (v & 8 ? vb[3] : 0u);
    double2 a[E];
#pragma unroll
    for (int v = 0; v < E; v++) a[v] = tile[place ^ vv[v]];
    RotStream<W> rots(words, h2.y, index);
    uint4 next = words(h0.x);
    for (uint32_t o = 1; o <= h0.y; o++) {
        const uint4 st = next;
        next = words(h0.x + o);
        apply_step(a, words, st, index, rots);
    }
#pragma unroll
    for (int v = 0; v < E; v++) tile[place ^ vv[v]] = a[v];
}

// The last sweep: out of the frame, with its signs, to the state.
__device__ __forceinline__ void store_tile(const double2* tile, double2* __restrict__ gp, const RotPass& p, int rest,
                                           uint64_t outer, uint32_t slot, uint32_t place) {
    uint32_t c = p.out_const ^ place;
    uint32_t sg = uint32_t(p.sign_const) ^ odd(p.sign_outer & uint32_t(outer)) ^ odd(p.sign_local & slot);
    if (p.outer_moves)
        for (int j = 0; j < rest; j++)
            if ((outer >> j) & 1) c ^= p.out_outer[j];
#pragma unroll
    for (int k = 0; k < E; k++) {
        double2 x = tile[c ^ p.reg_out[k]];
        const int flip = int((sg ^ (uint32_t(p.reg_sign) >> k)) << 31);
        x.x = __hiloint2double(__double2hiint(x.x) ^ flip, __double2loint(x.x));
        x.y = __hiloint2double(__double2hiint(x.y) ^ flip, __double2loint(x.y));
        gp[p.reg_off[k]] = x;
    }
}

// Few or small tiles.  Persistent; a CTA holds `1 << pack` tiles of 2^m amplitudes at
// a time, 2^(m-4) threads each.
template <class W>
__device__ __forceinline__ void rotation_body(double2* __restrict__ s, int n, const RotPass& p, int pack,
                                              uint64_t total_tiles, int basis, const W& words) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int m = p.m, tbits = m - kRotRegBits;
    double2* all = reinterpret_cast<double2*>(smem_raw);
    // Per slot (tile index bits below tbits): its offset in the state and its
    // place in the last sweep.  The register part of both is in the pass.
    uint64_t* slot_off = reinterpret_cast<uint64_t*>(smem_raw + (sizeof(double2) << (m + pack)));
    uint16_t* slot_out = reinterpret_cast<uint16_t*>(slot_off + (1 << tbits));
    for (int e = threadIdx.x; e < (1 << tbits); e += blockDim.x) {
        uint64_t off = 0;
        uint32_t pl = 0;
        for (int b = 0; b < tbits; b++)
            if ((e >> b) & 1) {
                off |= uint64_t(1) << p.q[b];
                pl ^= p.out_dir[b];
            }
        slot_off[e] = off;
        slot_out[e] = uint16_t(pl);
    }
    __syncthreads();
    const int rest = n - m;
    const uint32_t slot = threadIdx.x & ((1u << tbits) - 1), sub = threadIdx.x >> tbits;
    double2* tile = all + (size_t(sub) << m);
    for (uint64_t t0 = uint64_t(blockIdx.x) << pack; t0 < total_tiles; t0 += uint64_t(gridDim.x) << pack) {
        const uint64_t t = t0 + sub;
        const bool live = t < total_tiles;  // the barriers below are taken by every thread all the same
        const uint64_t outer = t & ((uint64_t(1) << rest) - 1);
        uint64_t at = outer;
        for (int b = 0; b < m; b++) {
            const uint64_t low = (uint64_t(1) << p.q[b]) - 1;
            at = (at & low) | ((at & ~low) << 1);
        }
        double2* __restrict__ gp = s + (((t >> rest) << n) | at | slot_off[slot]);
        const uint32_t in_place = swz(slot);
        if (basis) {
#pragma unroll
            for (int k = 0; k < E; k++)
                tile[in_place ^ p.reg_in[k]] = make_double2(outer == 0 && slot == 0 && k == 0 ? 1.0 : 0.0, 0.0);
        } else if (live) {
#pragma unroll
            for (int k = 0; k < E; k++)
                __pipeline_memcpy_async(&tile[in_place ^ p.reg_in[k]], gp + p.reg_off[k], sizeof(double2));
        }
        __pipeline_commit();
        __pipeline_wait_prior(0);
        __syncthreads();
        const uint32_t index = slot | uint32_t(outer) << kRotSlotBits;
        for (int ph = 0; ph < p.nphases; ph++) {
            rotation_phase(tile, words, ph, slot, index);
            __syncthreads();
        }
        if (live) store_tile(tile, gp, p, rest, outer, slot, slot_out[slot]);
        __syncthreads();
    }
}

// Shared memory of the tiles and the offset and place tables, a multiple of 16 bytes.
__host__ __device__ inline size_t rotation_tile_smem(int m, int pack) {
    const size_t tables = (size_t(1) << (m - kRotRegBits)) * (sizeof(uint64_t) + sizeof(uint16_t));
    return (sizeof(double2) << (m + pack)) + ((tables + 15) & ~size_t(15));
}

constexpr int kRotThreads = 512;  // of the largest tile; 128 registers a thread, 16 warps to an SM

__global__ void __launch_bounds__(kRotThreads, 1)
    k_rotations_arg(double2* __restrict__ s, int n, int pack, uint64_t total_tiles, int basis,
                    const __grid_constant__ RotPass p, const __grid_constant__ RotWords w) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint4* table = reinterpret_cast<uint4*>(smem_raw + rotation_tile_smem(p.m, pack));
    for (int i = threadIdx.x; i < p.ndata; i += blockDim.x) table[i] = w.w[p.data + i];
    // (the body synchronises before the first step)
    rotation_body(s, n, p, pack, total_tiles, basis, ArgWords{&w, table});
}

constexpr int kTeamTile = 12;      // qubits of a team's tile
constexpr int kTeamThreads = 256;  // one thread per 16 amplitudes
constexpr int kTeamBuffers = 3;
// Tiles to an SM from which the teams are used.  With few, the rounds are what
// counts and the teams start behind (one B200, 20 layers of brickwork: 512 tiles,
// 3.5 to an SM, 0.738 ms against 0.755 in teams; 1,024 tiles 1.386 against 1.376).
constexpr uint64_t kTeamTiles = 6;

__device__ __forceinline__ void bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Two teams of 256 threads take a CTA's tiles in turn, from three buffers.
// Tile j lies in buffer j % 3 and is worked on by team j % 2; the other team
// fetches it, when it has stored tile j - 3, and says so (barrier 3 + j % 3)
// while it works on tile j - 1, so that neither team waits for memory and each
// starts its tile in the middle of the other's.  Two CTAs of one tile each left an SM
// with half its warps while a tile was fetched: 27-qubit brickwork of 40 layers 97.0 -> 91.5 ms,
// 25-qubit QFT 2.70 -> 2.60, 24-qubit ansatz of 8 layers 2.17 -> 2.05.  (With
// an mbarrier for a tile's arrival the teams drift together: 97.0 ms.)
// Phase `tell` is the second of the pass (the first of two): after the first, the
// teller waits for its own fetch (92.6 ms for the 91.5), in the pass's middle the
// other team for the teller (95.7).  Past the middle the teams would take turns
// for good: passes with most of their work in the first phase run without teams.
template <class W>
__device__ __forceinline__ void team_body(double2* __restrict__ s, int n, const RotPass& p, uint64_t total_tiles, int basis,
                                          const W& words) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int m = kTeamTile;
    double2* all = reinterpret_cast<double2*>(smem_raw);
    uint64_t* slot_off = reinterpret_cast<uint64_t*>(all + (size_t(kTeamBuffers) << m));
    uint16_t* slot_out = reinterpret_cast<uint16_t*>(slot_off + kTeamThreads);
    uint16_t* outer_bit = slot_out + kTeamThreads;
    const uint32_t slot = threadIdx.x & (kTeamThreads - 1);
    // (the shuffle tells the compiler that a warp's threads agree; without it the
    // program's words leave the uniform registers: 105 ms for the 91.5 above)
    const int team = __shfl_sync(~0u, int(threadIdx.x / kTeamThreads), 0);
    const int rest = n - m;
    if (team == 0) {
        uint64_t off = 0;
        uint32_t pl = 0;
        for (int b = 0; b < m - kRotRegBits; b++)
            if ((slot >> b) & 1u) {
                off |= uint64_t(1) << p.q[b];
                pl ^= p.out_dir[b];
            }
        slot_off[slot] = off;
        slot_out[slot] = uint16_t(pl);
    } else if (slot < 32) {
        int bit = int(slot);
        for (int b = 0; b < m; b++) bit += int(p.q[b]) <= bit;
        outer_bit[slot] = uint16_t(bit);
    }
    __syncthreads();  // (the steps' data too)
    const int tiles = int((total_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x);
    auto outer_of = [&](int j) { return (blockIdx.x + uint64_t(j) * gridDim.x) & ((uint64_t(1) << rest) - 1); };
    auto state_of = [&](int j) {
        const uint64_t t = blockIdx.x + uint64_t(j) * gridDim.x;
        const uint32_t lane = threadIdx.x & 31u;
        const uint64_t mine = ((t >> lane) & 1u & uint32_t(int(lane) < rest)) << outer_bit[lane];
        const uint64_t at = uint64_t(__reduce_or_sync(~0u, uint32_t(mine >> 32))) << 32 | __reduce_or_sync(~0u, uint32_t(mine));
        return s + (((t >> rest) << n) | at | slot_off[slot]);
    };
    auto fetch = [&](int j, int buffer) {
        double2* tile = all + (size_t(buffer) << m);
        const uint32_t in_place = swz(slot);
        const double2* gp = state_of(j);
        const bool one = outer_of(j) == 0 && slot == 0;
#pragma unroll
        for (int k = 0; k < E; k++) {
            double2* to = &tile[in_place ^ p.reg_in[k]];
            if (basis)
                *to = make_double2(one && k == 0 ? 1.0 : 0.0, 0.0);
            else
                __pipeline_memcpy_async(to, gp + p.reg_off[k], sizeof(double2));
        }
        __pipeline_commit();
    };
    if (team < tiles) fetch(team, team);
    if (team == 1 && tiles > 2) fetch(2, 2);
    int buffer = team;
    // Both teams take the same number of turns (uniform control flow); the
    // second's last one may be idle and touches no buffer: the other team may
    // still be at work there.
    for (int i = 0; i < (tiles + 1) / 2; i++) {
        const int j = 2 * i + team;
        if (i == 0) {
            if (team == 1 && tiles > 2)
                __pipeline_wait_prior(1);
            else
                __pipeline_wait_prior(0);
            bar_sync(1 + team, kTeamThreads);
        } else if (j < tiles) {
            bar_sync(3 + buffer, 2 * kTeamThreads);
        }
        double2* tile = all + (size_t(buffer) << m);
        const uint32_t index = slot | uint32_t(outer_of(j)) << kRotSlotBits;
        const int phases = j < tiles ? p.nphases : 0;
        for (int ph = 0; ph < phases; ph++) {
            rotation_phase(tile, words, ph, slot, index);
            if (ph == p.tell && j >= 1 && j + 1 < tiles) {
                __pipeline_wait_prior(0);
                __threadfence_block();
                bar_arrive(3 + (buffer == kTeamBuffers - 1 ? 0 : buffer + 1), 2 * kTeamThreads);
            }
            bar_sync(1 + team, kTeamThreads);
        }
        if (j < tiles) store_tile(tile, state_of(j), p, rest, outer_of(j), slot, slot_out[slot]);
        if (j + 3 < tiles) {
            bar_sync(1 + team, kTeamThreads);
            fetch(j + 3, buffer);
        }
        buffer = buffer == 0 ? kTeamBuffers - 1 : buffer - 1;  // (j + 2) % 3
    }
}

__host__ __device__ constexpr size_t team_tile_smem() {
    return (sizeof(double2) * kTeamBuffers << kTeamTile) + kTeamThreads * (sizeof(uint64_t) + sizeof(uint16_t)) +
           32 * sizeof(uint16_t);
}

__global__ void __launch_bounds__(2 * kTeamThreads, 1)
    k_rotations_team(double2* __restrict__ s, int n, uint64_t total_tiles, int basis, const __grid_constant__ RotPass p,
                     const __grid_constant__ RotWords w) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint4* table = reinterpret_cast<uint4*>(smem_raw + team_tile_smem());
    for (int i = threadIdx.x; i < p.ndata; i += blockDim.x) table[i] = w.w[p.data + i];
    team_body(s, n, p, total_tiles, basis, ArgWords{&w, table});
}

constexpr int kSwapThreads = 256, kSwapEach = 8;
constexpr uint64_t kSwapStates = uint64_t(1) << 19;  // amplitudes, 8 MB

// A permutation of the state: amplitude x becomes -+ the one at y = const ^ the XOR of to[b] over x's bits.
struct StateMap {
    uint64_t to[64], to_const, sign;
    int sign_const;
};

// Passes of relabellings that are their own inverse (swap networks) and leave
// qubit 0 in place: pairs (x, y) change places where they are.  Bound by HBM or L2.
// A tile kernel without qubit 0 moves 16 bytes at a time, half a sector; this one
// moves whole rows (25-qubit QFT without pinned qubits: last pass 0.43 -> 0.24 ms).
// With qubit 0 in the tile it is the faster one while the state stays in L2
// (QFT of 16 qubits 0.076 -> 0.069 ms; 13 and 19 qubits equal); from 22 qubits on the
// tile kernel reads its rows in better order (25 qubits 2.12 ms against 2.28).
__global__ void __launch_bounds__(kSwapThreads) k_swap_places(double2* __restrict__ s, int n, uint64_t states,
                                                              const __grid_constant__ StateMap map) {
    constexpr uint64_t chunk = uint64_t(kSwapThreads) * kSwapEach;
    const uint64_t len = uint64_t(1) << n, chunks = (len + chunk - 1) / chunk;
    uint64_t low = map.to_const;
    for (int b = 0; b < 8 && b < n; b++)
        if ((threadIdx.x >> b) & 1u) low ^= map.to[b];
    for (uint64_t c = blockIdx.x; c < chunks * states; c += gridDim.x) {
        double2* __restrict__ a = s + c / chunks * len;
        const uint64_t base = c % chunks * chunk;
        uint64_t high = low;
        for (int b = 0; (base >> b) != 0; b++)
            if ((base >> b) & 1u) high ^= map.to[b];
        double2 p[kSwapEach], q[kSwapEach];
        uint64_t y[kSwapEach];
#pragma unroll
        for (int k = 0; k < kSwapEach; k++) {
            const uint64_t x = base | uint64_t(k) * kSwapThreads | threadIdx.x;
            y[k] = high ^ (k & 1 ? map.to[8] : 0) ^ (k & 2 ? map.to[9] : 0) ^ (k & 4 ? map.to[10] : 0);
            if (x >= len) y[k] = 0;
            if (x < y[k]) q[k] = __ldcg(a + y[k]);
            if (x <= y[k]) p[k] = __ldcg(a + x);
        }
#pragma unroll
        for (int k = 0; k < kSwapEach; k++) {
            const uint64_t x = base | uint64_t(k) * kSwapThreads | threadIdx.x;
            const int sx = int(uint32_t(__popcll(map.sign & x) + map.sign_const) << 31);
            const int sy = int(uint32_t(__popcll(map.sign & y[k]) + map.sign_const) << 31);
            auto flip = [](double2 z, int f) {
                return make_double2(__hiloint2double(__double2hiint(z.x) ^ f, __double2loint(z.x)),
                                    __hiloint2double(__double2hiint(z.y) ^ f, __double2loint(z.y)));
            };
            if (x < y[k]) {
                a[x] = flip(q[k], sx);
                a[y[k]] = flip(p[k], sy);
            } else if (x == y[k] && sx) {
                a[x] = flip(p[k], sx);
            }
        }
    }
}

// The pass as a map of the state's indices; false if it is not its own inverse.
bool own_inverse(const RotProgram& r, const std::vector<int>& tile_qubits, int n, StateMap& map) {
    auto deposit = [&](uint32_t e) {
        uint64_t x = 0;
        for (int b = 0; b < r.m; b++)
            if ((e >> b) & 1u) x |= uint64_t(1) << tile_qubits[size_t(b)];
        return x;
    };
    // Places are swizzled tile indices; the swizzle is its own inverse.
    map = StateMap{};
    map.to_const = deposit(rot_swizzle(r.out_const));
    map.sign_const = r.sign_const;
    for (int q = 0, b = 0, j = 0; q < n; q++) {
        if (b < r.m && tile_qubits[size_t(b)] == q) {
            map.to[q] = deposit(rot_swizzle(r.out_dir[b]));
            if ((r.sign_local >> b) & 1u) map.sign |= uint64_t(1) << q;
            b++;
        } else {
            map.to[q] = uint64_t(1) << q;
            if (j < kRotMaxOuter) {
                map.to[q] ^= deposit(rot_swizzle(r.out_outer[j]));
                if ((r.sign_outer >> j) & 1u) map.sign |= uint64_t(1) << q;
            }
            j++;
        }
    }
    auto image = [&](uint64_t x) {
        uint64_t y = 0;
        for (int q = 0; q < n; q++)
            if ((x >> q) & 1u) y ^= map.to[q];
        return y;
    };
    for (int q = 0; q < n; q++)
        if (image(map.to[q]) != uint64_t(1) << q) return false;
    return image(map.to_const) == map.to_const;
}

// CTAs of the kernel that are resident at once on the current device, asked of
// the runtime when the shape differs from this thread's last launch.
template <typename Kernel>
uint64_t resident_ctas(Kernel kernel, int threads, size_t smem) {
    struct Shape {
        const void* kernel = nullptr;
        int dev = -1, threads = 0;
        size_t smem = 0;
        uint64_t ctas = 0;
    };
    static thread_local Shape last;
    int dev = 0;
    cudaGetDevice(&dev);
    const void* id = reinterpret_cast<const void*>(kernel);
    if (last.kernel == id && last.dev == dev && last.threads == threads && last.smem >= smem) return last.ctas;
    // The limit is the device's, not this launch's: it holds for every thread's launches of the kernel.
    int most = 0;
    cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, int(cudaSharedmemCarveoutMaxShared));
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
    last = {id, dev, threads, smem, uint64_t(std::max(sms, 1)) * uint64_t(std::max(per_sm, 1))};
    return last.ctas;
}

}  // namespace

void rotation_pass(const Batch& b, const std::vector<int>& tile_qubits, const RotProgram& r, bool basis) {
    if (b.c64) fail(kValueError, "rotation passes run on complex128 states");
    const bool swaps = r.nphases == 0 && !basis && (tile_qubits[0] > 0 || (b.W << b.n) <= kSwapStates);
    if (StateMap map; swaps && own_inverse(r, tile_qubits, b.n, map) && map.to[0] == 1) {
        const uint64_t chunks = ((uint64_t(1) << b.n) + kSwapThreads * kSwapEach - 1) / (kSwapThreads * kSwapEach) * b.W;
        k_swap_places<<<unsigned(std::min(chunks, resident_ctas(k_swap_places, kSwapThreads, 0))), kSwapThreads, 0, b.stream>>>(
            static_cast<double2*>(b.amps), b.n, b.W, map);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) fail(kCudaError, std::string("rotation pass: ") + cudaGetErrorString(e));
        return;
    }
    RotPass p{};
    p.m = r.m;
    p.nphases = r.nphases;
    p.tell = r.tell;
    for (int i = 0; i < r.m; i++) {
        p.q[i] = uint8_t(tile_qubits[size_t(i)]);
        p.out_dir[i] = r.out_dir[i];
    }
    std::memcpy(p.out_outer, r.out_outer, sizeof p.out_outer);
    p.out_const = r.out_const;
    p.sign_local = r.sign_local;
    p.sign_outer = r.sign_outer;
    p.sign_const = r.sign_const;
    for (uint16_t x : r.out_outer) p.outer_moves |= x != 0;
    const int tb = r.m - kRotRegBits;
    for (int k = 0; k < E; k++) {
        p.reg_in[k] = uint16_t(rot_swizzle(uint32_t(k) << tb));
        for (int j = 0; j < kRotRegBits; j++)
            if ((k >> j) & 1) {
                p.reg_off[k] |= uint64_t(1) << p.q[tb + j];
                p.reg_out[k] = uint16_t(p.reg_out[k] ^ r.out_dir[tb + j]);
            }
        if (__builtin_parity(r.sign_local & (uint32_t(k) << tb))) p.reg_sign |= 1u << k;
    }
    // Small tiles share a CTA, up to 64 threads.
    const int tbits = r.m - kRotRegBits;
    const uint64_t total = b.W << (b.n - r.m);
    int pack = 0;
    while (tbits + pack < 6 && (uint64_t(2) << pack) <= total) pack++;
    const int threads = 1 << (tbits + pack);
    if (r.words.size() > size_t(kRotParamWords)) fail(kValueError, "rotation program larger than a launch argument");
    p.data = r.data;
    p.ndata = int(r.words.size()) - r.data;
    const size_t smem = rotation_tile_smem(r.m, pack) + size_t(p.ndata) * sizeof(uint4);
    const uint64_t ctas = (total + (uint64_t(1) << pack) - 1) >> pack;
    static thread_local RotWords args;
    std::memcpy(args.w, r.words.data(), r.words.size() * sizeof(uint4));
    const size_t team_smem = team_tile_smem() + size_t(p.ndata) * sizeof(uint4);
    const bool teams = r.m == kTeamTile && r.tell >= 0;
    const uint64_t sms = teams ? resident_ctas(k_rotations_team, 2 * kTeamThreads, team_smem) : 0;
    if (teams && total >= kTeamTiles * sms)
        k_rotations_team<<<unsigned(sms), 2 * kTeamThreads, team_smem, b.stream>>>(static_cast<double2*>(b.amps), b.n, total, basis ? 1 : 0, p, args);
    else
        k_rotations_arg<<<unsigned(std::min(ctas, resident_ctas(k_rotations_arg, threads, smem))), unsigned(threads), smem,
                          b.stream>>>(
            static_cast<double2*>(b.amps), b.n, pack, total, basis ? 1 : 0, p, args);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) fail(kCudaError, std::string("rotation pass: ") + cudaGetErrorString(e));
}

}  // namespace k
}  // namespace dq
