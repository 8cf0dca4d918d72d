// Tensor-core convolution for small batches (kb_conv_small.cu): what kb_conv_tc.cu needs to dispatch to it.
#pragma once

#include "kb_kernels.cuh"
#include "kb_tc_ptx.cuh"

namespace kb {

// Tile widths the kernel is launched with.
constexpr int CONV_SMALL_WIDTHS[4] = {16, 32, 64, 96};
inline int convSmallMapIndex(int BN) { return BN <= 32 ? BN / 16 - 1 : BN / 32; }

struct ConvSmallShape {
  int dt, inC, outC, taps;      // taps: 1 or 9
  int haloPad, aRows;           // of the activation box, as in the convolution's plan
  const CUtensorMap* tmA;       // activations, box of 64 channels x aRows rows
  CUtensorMap tmB[4];           // weights [taps][outC][inC], boxes of 64 channels x CONV_SMALL_WIDTHS[i] rows x 1 or 3 taps
};

// True if the kernel has a variant for this epilogue (staged-epilogue convolutions without row sums).
bool convSmallSupports(const Epilogue& ep);
// Output channels per CTA for this many 128-row tiles, or 0 where the wide-tile kernels are the better choice.
int convSmallTileWidth(int outC, int rowTiles, int numSMs);
cudaError_t launchConvSmall(cudaStream_t st, const ConvSmallShape& s, int BN, int numSMs, Geom g, const Epilogue& ep, int* statusWord);

}  // namespace kb
