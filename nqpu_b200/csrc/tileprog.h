// Stage programs of the tiled passes: what the tile kernels execute.
//
// The planner's stage ops are compiled, per register stage, into a stream of
// 16-byte words (plain C++, no CUDA headers, so the CPU tests can interpret it).
// One instruction is a header word and its operands:
//
//   header.x   code | words << 16 (words of the instruction, header included)
//   R + b      real 2x2 on register bit b: header.y = virtual-index mask that must
//   X + b      be set; the matrix entries (m00, m01, m10, m11) follow, real for R,
//              real diagonal and imaginary off-diagonal for X, complex for G
//   G + b
//   PH + A     phase on the register amplitudes whose bits A are all set.  The
//              phase is a product over a list of (mask, phase): an entry counts
//              when the thread's virtual index has all bits of mask set.
//              header.y = entries.  complex64: angles in 2^-32 turns, header.z =
//              constant part, two (mask, angle) per word.  complex128: complex
//              factors, one word constant part, two words (mask) (re, im) each.
//   PU + A     the same with a constant phase (complex64: re, im in header.z, .w)
//   D + b      PH on all amplitudes and PH on those with bit b, one multiplication
//              per amplitude: header.y = entries of the first | of the second
//              << 16; constant parts in header.z, .w (complex64) or two words
//   SG + A     sign flips on the amplitudes with bits A: header.y = masks, header.z
//              = constant parity; four masks per word
//   LEG        any other op: its TileOp record follows
//
// Why a program and not the ops themselves: the tile kernels are bound by issue
// (FP32) and by the FP64 pipe, and diagonal gates commute, so all phases of a
// stage that multiply the same register amplitudes are one multiplication whose
// factor a thread works out once instead of once per amplitude and gate.  A
// controlled phase costs a list entry (4 instructions) where it took 16 complex
// products; RY, H and RX need half or less of a complex 2x2 product.
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

enum TileCode : uint32_t {
  TC_R = 0, TC_X = 8, TC_G = 16, TC_D = 24, TC_PH = 32, TC_PU = 64, TC_SG = 96, TC_LEG = 128,
};

// Compile every stage of `plan` (built from `ops`) into plan->prog and set the
// word ranges in its pass and stage records: per pass the stage tables, then the
// instructions (prog_begin .. prog_end of a stage count from the first of them).
void build_tile_prog(const std::vector<Op>& ops, TilePlan* plan);

}  // namespace nqpu
