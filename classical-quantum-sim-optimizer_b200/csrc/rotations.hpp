// Tile passes as Pauli rotations (rotations.cpp plans them, rotation_pass.cu runs them).
//
// Gates other than dense matrices are products of three things, and a pass of
// such gates is rewritten in them on the host:
//   * relabellings of the basis: X, CX, SWAP.  They never move an amplitude.
//     The planner keeps, for every qubit q, the mask and constant that read its
//     value off the place p an amplitude is stored at (q = parity(mask_q & p) ^
//     const_q) and the direction v_q in which the place changes when q flips.
//     The pass's last sweep writes every amplitude to the index it then has.
//   * phases exp(i a Z^mu): a factor e^(+-ia) by the parity of mu & p.  Phases
//     of equal mu merge, also across the CX and CZ gates between them.
//   * rotations exp(-i theta/2 P), P = X^v Z^mu (times i where mu & v is odd),
//     which mix the amplitudes at p and p ^ v.  With t = tan(theta/2) and s =
//     +-1 by the parity of mu & p, the pair becomes
//       x <- x - s t y, then y <- y + s t/(1 + t^2) x,
//     which is the rotation but for factors cos and 1/cos of the two: two
//     fused multiply-adds per amplitude, in place (no copy of x), instead of
//     the eight of a complex 2x2 matrix.  The factors are the moduli of a
//     phase and go into the next table.  Where no table follows soon enough,
//     both are formed from the old pair and one cosine is owed by the whole state.  Angles are reduced so that |t| <= 1
//     (the quarter turns taken out are Pauli matrices: relabellings and signs).
// A one-qubit unitary is a phase, a Y rotation and a phase. With one control the
// rotation becomes one about Y and one about Z Y, without phases between (12-qubit
// CU3 circuits of 10 layers 0.106 -> 0.085 ms, CRX and H 0.204 -> 0.100); with
// more, as in Toffolis, Y rotations around controlled-Z phases.
//
// Rotations and phases are scheduled into phases of four directions (a
// subspace V of the 2^m places): a thread holds the 16 amplitudes of one coset
// of V in registers, applies every rotation whose direction lies in V and
// whose predecessors (earlier ones it does not commute with) are done, and
// stores them back.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "compile.hpp"
#include "kernels.hpp"

namespace dq {

constexpr int kRotRegBits = 4;
constexpr int kRotEntries = 1 << kRotRegBits;
constexpr int kRotMinTile = 5, kRotMaxTile = 13;  // tile qubits a pass may have
constexpr int kRotSlotBits = kRotMaxTile - kRotRegBits;
// Parity masks of the kernel hold the slot (thread) bits below bit kRotSlotBits
// and the bits of the tile's index above.
constexpr int kRotMaxOuter = 32 - kRotSlotBits;
constexpr int kRotParamWords = 1980;  // largest program, a launch argument (31,680 bytes)

// A pass's program, in 16-byte words:
//   phase p at 3p: {first step word, steps, v0 | v1 << 16, v2 | v3 << 16}, then the
//     slot bits' places b0..b7 two to a register, then {b8, first rotation
//     word, 0, 0}; all places swizzled (rot_swizzle);
//   steps, one word each: {what | flags, table, slot data, slot terms | signs << 16}.
//     A step applies, in this order and where present, a rotation on each
//     register bit j (what: kind + 1 at bits 2j), one on another direction
//     (its 4 bits on V's basis at bits 8-11, kind at 12-13), a table of phases
//     and either slot phases or slot moduli;
//   rotations in the order applied: {t, t / (1 + t^2)} ({t, 1 + t^2} for kRotKept)
//     and, except kRotPlain, {signs, parity mask, 0, 0};
//   data: a table's 16 factors; slot terms' ceil(terms / 4) words of parity
//     masks, then for each its (cos, sin) or (modulus, 1 / modulus), conjugated
//     or inverted by its parity and by the register signs.
// `signs` is one bit per register entry.
constexpr uint32_t kRotPlain = 0;    // no signs among its first entries and no parity mask; register bits only
constexpr uint32_t kRotSigned = 1;
constexpr uint32_t kRotKept = 2;     // x - s t y and y + s t x, both owed the same cosine; signed
constexpr uint32_t kRotImag = 3;     // P without the factor i; signed, never on its own place
constexpr uint32_t kRotTable = 1u << 16, kRotSlots = 1u << 17, kRotSlotModuli = 1u << 18;

struct RotProgram {
    int m = 0;                       // tile qubits
    int nphases = 0;
    std::vector<uint4> words;
    int data = 0;                    // first word of the steps' data
    std::vector<int> phase_data;     // where each phase's data begin among them
    int tell = -1;                   // phase after which a team's fetch counts as done (rotation_pass.cu); -1: no teams
    // Where the last sweep finds the amplitude of tile index e: XOR of
    // out_dir[q] over e's set bits, out_outer[j] over the set bits of the
    // tile's index, and out_const (all swizzled).
    uint16_t out_dir[kRotMaxTile] = {};
    uint16_t out_outer[kRotMaxOuter] = {};
    uint16_t out_const = 0;
    // ... and the sign it takes: parity(sign_local & e) ^ parity(sign_outer & tile index) ^ sign_const.
    uint32_t sign_local = 0, sign_outer = 0;
    int sign_const = 0;
    double flops_per_amp = 0.0;      // real operations per amplitude
    int rotations = 0, tables = 0, slot_phases = 0;
};

// Swizzled place: the low 3 bits XOR every higher 3-bit chunk (GF(2)-linear).
inline uint32_t rot_swizzle(uint32_t p) {
    uint32_t f = 0;
    for (uint32_t x = p >> 3; x; x >>= 3) f ^= x;
    return p ^ (f & 7u);
}

// Whether ops[begin, end) are planned with the target qubits of a pass in its
// tile only (TilePlanOptions::targets_only): all of them have a rotation form
// (a pass that had to run in register phases would need every qubit) and some
// are diagonal on several qubits.  Those reach out of the tile for a slot
// phase each, and passes then hold far more of them (25-qubit QFT 9 -> 4
// passes, 24-qubit ansatz 5 -> 4, both faster); with CX alone the phases lost
// to slots outweigh the passes saved (27-qubit brickwork 13 -> 12, 3 % slower).
bool rotation_targets_only(const std::vector<Operation>& ops, size_t begin, size_t end, int n, int m);

// Lowest qubits that every tile of ops[begin, end) holds
// (TilePlanOptions::pinned_low).  A tile without them is fetched and stored 16
// bytes at a time, half a sector and an L1 lookup each: some 8,000 cycles on the
// 35,000 to 45,000 of a pass.  Two give up a sixth of a tile's qubits for runs of 64
// bytes.  20 to 26 qubits, brickwork, QFT, ansatz and layers: 13 % faster at 24 qubits,
// 7 to 10 % at the others (one pinned qubit 5 to 9 %, three 2 to 9 %); 27-qubit
// brickwork 89.0 -> 84.8 ms, 25-qubit QFT 2.39 -> 2.12, 28-qubit ansatz 22.5 -> 17.2.  Below 20 qubits a pass is one
// wave of tiles and their number counts: 18 qubits 7 % slower.  None
// where an operation has no rotation form or touches more than the tile has left.
int rotation_pinned_low(const std::vector<Operation>& ops, size_t begin, size_t end, int n, int m);

// Whether register phases (phased.hpp) are expected to take less time than rotation
// passes for ops[begin, end) on one state of n qubits that is a single tile. One or
// two warps then run all of it, and what counts is the number of rotations and
// tables in their chain against the number of fused two-qubit matrices. Register
// phases and rotations on 9 qubits in 30 layers: CU3 0.074 and 0.133 ms, C4X and RY 0.092
// and 0.194, CX and U3 0.150 and 0.124, CZ and RY RZ 0.278 and 0.102. From 12 qubits on, and where
// several states fill the device, rotations are quicker or within 3 % (12-qubit CU3 of
// 30 layers excepted, 0.178 and 0.209).
bool register_phases_quicker(const std::vector<Operation>& ops, size_t begin, size_t end, int n);

// Plans the pass `ops` over `tile_qubits` (ascending) of an n-qubit state.
// Targets and swapped qubits are tile qubits; controls and diagonal qubits may
// lie outside, where the tile's index gives their value.  False when an
// operation has no such form (a dense matrix that is no Pauli rotation, a matrix
// further from a unitary one than its entries' rounding) or the tile is too small or large.
bool build_rotation_pass(const std::vector<Operation>& ops, const std::vector<int>& tile_qubits, int n,
                         RotProgram& out);

// A program as programs of at most `most` words, to be run one after another: cut
// between phases.  A launch argument's steps and rotations come through the constant
// bank.  Read from device memory instead, 40 layers of 8-qubit brickwork (2,686
// words) took 0.222 ms, as two launches 0.159; 60 layers on 12 of 26 qubits (4
// launches, each a sweep of the state) 41.1 and 26.3.
std::vector<RotProgram> split_rotation_pass(RotProgram&& p, size_t most = kRotParamWords);

namespace k {
// One pass over every tile of every state (complex128), of at most kRotParamWords words.
// `basis`: every state is |0...0> on entry; the pass builds its input tiles
// itself and reads nothing of the state.
void rotation_pass(const Batch& b, const std::vector<int>& tile_qubits, const RotProgram& p, bool basis);
}  // namespace k

}  // namespace dq
