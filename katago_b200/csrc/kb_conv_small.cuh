// Tensor-core convolution for small batches (kb_conv_small.cu): what kb_conv_tc.cu needs to dispatch to it.
#pragma once

#include "kb_kernels.cuh"
#include "kb_tc_ptx.cuh"

namespace kb {

// Tile widths the kernel is launched with.
constexpr int CONV_SMALL_WIDTHS[] = {16, 32, 48, 64, 96, 128, 192, 256};
constexpr int CONV_SMALL_NUM_WIDTHS = sizeof(CONV_SMALL_WIDTHS) / sizeof(int);
inline int convSmallMapIndex(int BN) {
  for(int i = 0; i < CONV_SMALL_NUM_WIDTHS; i++)
    if(CONV_SMALL_WIDTHS[i] == BN) return i;
  return -1;
}

struct ConvSmallShape {
  int dt, inC, outC, taps;      // taps: 1 or 9
  int haloPad, aRows;           // of the activation box for 128-row tiles, as in the convolution's plan; 64 rows less for 64-row tiles
  const CUtensorMap* tmA;       // activations, box of 64 channels x aRows rows
  CUtensorMap tmA64;            // the same, box of aRows - 64 rows
  // weights [taps][outC][inC], boxes of 64 channels x CONV_SMALL_WIDTHS[i] rows x 1 tap and (3x3 only) x 3 taps
  CUtensorMap tmB[CONV_SMALL_NUM_WIDTHS], tmB3[CONV_SMALL_NUM_WIDTHS];
};

// A CTA's tile: BM rows (64 or 128) x BN output channels (the last tile of a row may have fewer), tapGroup taps per weight slot,
// smem bytes of shared memory.  BM = 0: the wide-tile kernels are the better choice.
struct ConvSmallTile {
  int BM = 0, BN = 0, tapGroup = 1, smem = 0;
};

// True if the kernel has a variant for this epilogue (of a convolution whose wide-tile form has the staged epilogue).
bool convSmallSupports(const Epilogue& ep);
ConvSmallTile convSmallTile(const ConvSmallShape& s, const Epilogue& ep, int rows, int numSMs);
cudaError_t launchConvSmall(cudaStream_t st, const ConvSmallShape& s, const ConvSmallTile& tile, Geom g, const Epilogue& ep, int* statusWord);

}  // namespace kb
