// Shapes of the fused 1x1 pair (kb_conv_fused.cu): how a pair Cm -> Ct -> Cn is divided, and which pairs can be.  Host-only code (no
// CUDA).
#pragma once

#include <initializer_list>

namespace kb {

constexpr int PP_CG = 3;        // epilogue warps per TMEM lane quarter
constexpr int PP_NUM_A2 = 4;    // operand chunks of GEMM2 in tensor memory
constexpr int PP_A2_COLS = 32;  // 64 channels of 16 bits, two per column

// Accumulators of GEMM1 that fit next to GEMM2's and its operand chunks: two if possible.
inline int postPreAccumulators(int NP, int Cn) { return 2 * NP + Cn + PP_NUM_A2 * PP_A2_COLS <= 512 ? 2 : 1; }

// A warp of the first epilogue takes units cg, cg + PP_CG, ... of every tile, and waits for the accumulator of a unit's part by the
// parity of the part's turn.  That says "this turn" only to a warp that knows the accumulator's turn before to be over, which it
// does where the part it waited for last is no more than one round of the accumulators back (parts complete in order).
// Parts of 64 channels hold two units for three warps, so that a warp skips some: at 448 channels (seven parts) one goes from part
// 5 of a tile to part 1 of the next, number 8.  Parts 4, 6 and 8 share an accumulator; until 6 is done the barrier is in the
// phase that follows 4, and the wait for 8 passes at once.
inline bool postPreWarpsKeepUp(int Ct, int NP, int Cn) {
  const int units = Ct / 32, perPart = NP / 32, parts = Ct / NP, D = postPreAccumulators(NP, Cn);
  for(int cg = 0; cg < PP_CG && cg < units; cg++) {
    int before = cg / perPart;
    for(int u = cg + PP_CG; u < units; u += PP_CG) {
      if(u / perPart - before > D) return false;
      before = u / perPart;
    }
    if(parts + cg / perPart - before > D) return false;  // its first unit of the next tile
  }
  return true;
}

// Output channels of GEMM1 per part: whole K chunks of GEMM2, one accumulator next to GEMM2's and its operand chunks, and no part
// skipped by a warp that counts on it.  0: no such width.
inline int postPrePartWidth(int Ct, int Cn) {
  for(int np : {192, 128, 64})
    if(Ct % np == 0 && np + Cn + PP_NUM_A2 * PP_A2_COLS <= 512 && postPreWarpsKeepUp(Ct, np, Cn)) return np;
  return 0;
}
// A weight slot holds a 64-channel chunk for one part of GEMM1 or as many output channels of GEMM2.
inline int postPrePieces(int Ct, int Cn) {
  const int np = postPrePartWidth(Ct, Cn);
  for(int i = 1; i <= 4; i++)
    if(Cn % (16 * i) == 0 && Cn / i <= np) return i;
  return 0;
}

}  // namespace kb
