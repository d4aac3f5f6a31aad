// Stage programs of the tiled passes: what the tile kernels execute.
//
// The planner's stage ops are compiled, per register stage, into a stream of
// 16-byte words (plain C++, no CUDA headers, so the CPU tests can interpret it).
// One instruction is a header word and its operands:
//
//   header.x   code | arg << 8 | words << 16 (words of the instruction, header
//              included); A = a set of register bits, b = one of them
//   R          real rotations on the register bits of header.y, each as three
//              shears (t = tan(phi / 2), s = sin(phi), |phi| <= pi/2): t, s per bit
//              at a fixed place, bit 0 in header.z, .w and two bits per word
//              after it (complex64) or one bit per word (complex128)
//   X          the same with the imaginary off-diagonal of RX
//   G b        any complex 2x2: header.y = virtual-index mask that must be set; the
//              entries m00, m01, m10, m11 follow
//   T          one constant phase per register amplitude: 2^(register bits) entries
//   TS         the same as shears (t, s of every phase, all within a quarter turn
//              either way): three operations per amplitude instead of four, and
//              no drift of the norm (a shear has determinant 1 whatever its
//              rounding; a rounded (cos, sin) scales what it turns, the same way
//              in every step of an evolution)
//   PS A       constant phase as a shear on the register amplitudes whose bits A
//              are all set (complex64; t, s in header.z, .w)
//   PU A       constant phase on the register amplitudes whose bits A are all set
//              (re, im in header.z, .w or the next word)
//   SG A       sign flip of those amplitudes
//   PH A       phase on those amplitudes that is a product over a list of (mask,
//              phase): an entry counts when the thread's virtual index has all
//              bits of mask set.  header.y = entries.  complex64: angles in
//              2^-32 turns, header.z = constant part, two (mask, angle) per word.
//              complex128: complex factors, one word constant part, two words
//              (mask) (re, im) each.
//   D b        PH on all amplitudes and PH on those with bit b, one multiplication
//              per amplitude: header.y = entries of the first | of the second
//              << 16; constant parts in header.z, .w (complex64) or two words
//   SL A       sign flips: header.y = masks, header.z = constant parity; four
//              masks per word
//   OP A       any other op of kind A (X also for a 2x2 without a diagonal):
//              header.y = register target bits, the second in the second byte, and
//              register controls in the third, header.z = its controls elsewhere;
//              the matrix of a 1q or 2q gate follows
//
// Why a program and not the ops themselves: the tile kernels are bound by
// instructions (every one costs a warp about seven cycles at any occupancy the
// register block allows) and, for complex128, by the FP64 pipe.  Diagonal gates
// commute, so all phases of a stage that multiply the same register amplitudes are
// one multiplication whose factor a thread works out once; a controlled phase
// costs a list entry (4 instructions) where it took 16 complex products.  Every
// unitary 2x2 is phase x real rotation x phase: the rotation takes three fused
// multiply-adds per pair and component in place (a complex 2x2 takes eight and
// the re / im swaps), and the phases before and after the rotations of a layer
// join in one T.
#pragma once
#include <cstdint>
#include <vector>
#include "planner.h"

namespace nqpu {

// Per-stage constants of the register block's addressing, kStageTabWords words per
// stage, in front of the pass's instructions.  The host works them out once per
// plan (a CTA used to, one thread per stage: about 4 us at the head of every
// pass):
//   S..S+3     slot offsets swz(vector bit of free register bit i)
//   CW..CW+3   slot offsets of the write-back images of the free register bits
//   HB         bit i: the image of free register bit i flips amplitude bit 0 (complex64)
//   MZ         image of register bit 0 (complex64; 1 = bit 0 stays bit 0)
//   CZ, HZ     slot offset and bit 0 of MZ's image
//   WS, WH     slot offset and bit 0 of the constant translation sbx
//   NC, OB, OE conditional translations, program range (words behind the tables)
//   CC, CS, CH per conditional translation: control mask, slot offset, bit 0
//   UL, UH     deposit of thread-index bits 0..3 / 4..7 into the vector index
//   SL, SH     the same deposits through the swizzle (swz is linear over XOR)
struct StageTab {
  enum : int { S = 0, CW = 4, HB = 8, MZ = 9, CZ = 10, HZ = 11, WS = 12, WH = 13, NC = 14, OB = 15, OE = 16,
               CC = 17, CS = 21, CH = 25, UL = 32, UH = 48, SL = 64, SH = 80 };
};
static_assert(StageTab::SH + 16 <= kStageTabWords && kStageTabWords % 4 == 0, "stage table layout");

enum TileCode : uint32_t { TC_R, TC_X, TC_TS, TC_T, TC_PS, TC_PH, TC_PU, TC_SG, TC_SL, TC_D, TC_G, TC_OP };

// The op list with every complex 2x2 reduced to rotation x phase where a later 2x2
// on its qubit can take the rest: a phase passes through controls and diagonal
// ops, an RX through X targets, so before a CNOT each of the two qubits hands one
// of its three Euler angles on.  A layer's gates then need one phase table per
// stage instead of two.  Same length, same qubits per op.
std::vector<Op> carry_phases(std::vector<Op> ops);

// Compile every stage of `plan` (built from `ops`) into plan->prog and set the
// word ranges in its pass and stage records: per pass the stage tables, then the
// instructions (prog_begin .. prog_end of a stage count from the first of them).
void build_tile_prog(const std::vector<Op>& ops, TilePlan* plan);

}  // namespace nqpu
