// fp32 convolution on the CUDA cores for 1x1 and 3x3 kernels over 4-channel-aligned tensors.
//
// convSimtKernel (kb_kernels.cu) takes any shape, one 16-channel slice of one tap at a time with two block barriers each and
// scalar loads; a 3x3 96->96 layer of eight boards ran at 6.5 of the 72 TFLOP/s the FMA units give, its 100 blocks spending
// their time on the load latency between the barriers.  Here a block stages ALL taps of a 16-channel slice at once: its
// output rows with their halo (every tap reads the same staged rows at another offset, the padded-rows layout makes that a
// constant) and the nine weight slices, double-buffered with cp.async, so that there are inC/16 steps per tile instead of
// 9*inC/16.  A tile is 32 to 80 rows x 32 channels; eight warps share each half of its rows, each computes all of them over two
// channels of every slice, up to 5 x 8 outputs per thread, and the eight sums are added in warp order at the end.  Measured
// per 96->96 layer of eight boards (event overhead of 4.5 us included): 72 us before; 37 us with 4 x 4 outputs per thread, whose
// shared-memory loads took twice the time of the FMAs; 35 us with 8 x 8 from eight warps (two per scheduler, 41 % FMA
// utilisation, and 156 tiles of 64 rows on 148 SMs); 27 us with up to 5 x 8 from sixteen.  The issue slots (62 % taken) were then
// nearer their limit than the FMA units (43 %): packed FMAs on pairs of channels take half of them, same bits.  Device time of the
// net before and after: b6c96 at 1 / 8 / 33 / 64 boards 232 / 342 / 1011 / 1796 -> 229 / 311 / 954 / 1691 us, b18 at 1 / 4 / 8
// 3439 / 3891 / 6887 -> 3351 / 3512 / 6450.  The order of the additions is the same in every batch size.
#include "kb_kernels.cuh"
#include "kb_act.cuh"
#include "kb_tc_ptx.cuh"

#include <algorithm>

namespace kb {

namespace {

constexpr int CF_BN = 32, CF_BK = 16;
constexpr int CF_AS = CF_BK + 4;      // floats per staged row: cp.async writes 16-byte pieces; the 8-byte loads of the eight rows a warp reads start 20 floats apart
constexpr int CF_KG = 8;               // warps that share a tile's channels
constexpr int CF_THREADS = 512;        // two halves of a tile's rows, CF_KG warps each
constexpr int cfRows(int nr) { return 16 * nr; }  // rows of a tile whose threads hold nr x 8 outputs

__device__ __forceinline__ void cpAsync16(float* dst, const float* src, bool valid) {
  // zero-filled where there is nothing to read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smemU32(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

template <int TAPS, int NR>
__global__ void __launch_bounds__(CF_THREADS) convF32Kernel(
  const float* in, int inStride, int inC, const float* __restrict__ w, int outC, int halo, Geom g, Epilogue ep) {
  extern __shared__ float4 smem4[];
  float* sm = reinterpret_cast<float*>(smem4);
  constexpr int BM = cfRows(NR);
  const int aRows = BM + 2 * halo;
  const int aFloats = aRows * CF_AS, bFloats = TAPS * CF_BK * CF_BN;
  const int stage = aFloats + bFloats;
  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int kg = warp & (CF_KG - 1);         // this warp takes channels 2*kg, 2*kg+1 of every slice
  const int r0 = (warp / CF_KG) * (BM / 2);  // of this half of the rows
  const int tx = lane & 3, ty = lane >> 2;   // 8 channels (4 from tx*4, 4 from 16+tx*4); rows r0 + ty, r0 + ty+8, ...
  const int m0 = (int)blockIdx.x * BM, n0 = (int)blockIdx.y * CF_BN;
  const int slices = (inC + CF_BK - 1) / CF_BK;

  auto loadB = [&](int s) {
    float* dst = sm + (s & 1) * stage + aFloats;
    for(int i = tid; i < TAPS * CF_BK * (CF_BN / 4); i += CF_THREADS) {
      const int c = (i & 7) * 4, kt = i >> 3;  // kt = tap * 16 + channel of the slice
      const int k = s * CF_BK + (kt & 15), tap = kt >> 4;
      const bool ok = k < inC && n0 + c < outC;
      cpAsync16(dst + kt * CF_BN + c, ok ? w + ((size_t)tap * inC + k) * outC + n0 + c : w, ok);
    }
  };
  auto loadA = [&](int s) {
    float* dst = sm + (s & 1) * stage;
    for(int i = tid; i < aRows * (CF_BK / 4); i += CF_THREADS) {
      const int c = (i & 3) * 4, r = i >> 2;
      const int row = m0 - halo + r, k = s * CF_BK + c;
      const bool ok = row >= 0 && row < g.rowsPad && k < inC;
      cpAsync16(dst + r * CF_AS + c, ok ? in + (size_t)row * inStride + k : in, ok);
    }
  };

  gridDepLaunch();
  loadB(0);        // weights: nothing in the stream produces them
  gridDepWait();
  loadA(0);
  asm volatile("cp.async.commit_group;" ::: "memory");

  // pairs of neighbouring channels: the packed fp32 instructions do two IEEE operations in one issue slot
  float2 acc[NR][4];
#pragma unroll
  for(int i = 0; i < NR; i++)
#pragma unroll
    for(int j = 0; j < 4; j++) acc[i][j] = make_float2(0.0f, 0.0f);

  for(int s = 0; s < slices; s++) {
    if(s + 1 < slices) { loadB(s + 1); loadA(s + 1); }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const float* sA = sm + (s & 1) * stage + 2 * kg;
    const float* sB = sm + (s & 1) * stage + aFloats + 2 * kg * CF_BN + tx * 4;
#pragma unroll(TAPS == 9 ? 3 : 1)
    for(int tap = 0; tap < TAPS; tap++) {
      const int shift = TAPS == 9 ? (tap / 3 - 1) * g.RW + tap % 3 - 1 : 0;
      const float* a = sA + (r0 + ty + halo + shift) * CF_AS;
      const float* b = sB + tap * CF_BK * CF_BN;
      float2 av[NR];
#pragma unroll
      for(int i = 0; i < NR; i++) av[i] = *reinterpret_cast<const float2*>(a + 8 * i * CF_AS);
#pragma unroll
      for(int k = 0; k < 2; k++) {
        const float4 b0 = *reinterpret_cast<const float4*>(b + k * CF_BN), b1 = *reinterpret_cast<const float4*>(b + k * CF_BN + 16);
#pragma unroll
        for(int i = 0; i < NR; i++) {
          const float x1 = k == 0 ? av[i].x : av[i].y;
          const float2 x = make_float2(x1, x1);
          acc[i][0] = __ffma2_rn(x, make_float2(b0.x, b0.y), acc[i][0]); acc[i][1] = __ffma2_rn(x, make_float2(b0.z, b0.w), acc[i][1]);
          acc[i][2] = __ffma2_rn(x, make_float2(b1.x, b1.y), acc[i][2]); acc[i][3] = __ffma2_rn(x, make_float2(b1.z, b1.w), acc[i][3]);
        }
      }
    }
    __syncthreads();  // the buffer is free for the slice after next
  }

  // The warps' partial sums of the tile, added in warp order by the thread that finishes 4 channels of a row.
#pragma unroll
  for(int i = 0; i < NR; i++) {
    float4* o = reinterpret_cast<float4*>(sm + (kg * BM + r0 + ty + 8 * i) * CF_BN);
    o[tx] = make_float4(acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y);
    o[4 + tx] = make_float4(acc[i][2].x, acc[i][2].y, acc[i][3].x, acc[i][3].y);
  }
  __syncthreads();
  for(int i = tid; i < BM * (CF_BN / 4); i += CF_THREADS) {
    const int r = i >> 3, cl = (i & 7) * 4, c = n0 + cl;
    const int m = m0 + r;
    if(m >= g.rowsPad || c >= outC) continue;
    const int br = m % g.PB, y = br / g.RW, x = br - y * g.RW;
    const bool point = m < g.rows && y < g.Y && x < g.X;
    const float mk = ep.mask ? ep.mask[m] : 1.0f;
    const int bIdx = min(m / g.PB, g.n - 1);
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // stays 0 on rows of the layout that are not board points, as in the general kernel
    if(point) {
#pragma unroll
      for(int k = 0; k < CF_KG; k++) {
        const float4 t = *reinterpret_cast<const float4*>(sm + (k * BM + r) * CF_BN + cl);
        v[0] += t.x; v[1] += t.y; v[2] += t.z; v[3] += t.w;
      }
    }
#pragma unroll
    for(int j = 0; j < 4; j++) {
      if(ep.biasNC) v[j] += ep.biasNC[(size_t)bIdx * outC + c + j];
      if(ep.residual) v[j] = (ep.resMask ? v[j] * mk : v[j]) + reinterpret_cast<const float*>(ep.residual)[(size_t)m * ep.resStride + c + j];
    }
    if(ep.outRaw) {
      float* o = reinterpret_cast<float*>(ep.outRaw) + (size_t)m * ep.rawStride + (c - ep.rawC0);
      if(c >= ep.rawC0 && c + 4 <= ep.rawC1 && (reinterpret_cast<uintptr_t>(o) & 15) == 0) *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
      else {
#pragma unroll
        for(int j = 0; j < 4; j++)
          if(c + j >= ep.rawC0 && c + j < ep.rawC1) o[j] = v[j];
      }
    }
    if(ep.outAct) {
      float* o = reinterpret_cast<float*>(ep.outAct) + (size_t)m * ep.actStride + (c - ep.actC0);
      float q[4];
#pragma unroll
      for(int j = 0; j < 4; j++) {
        const int ca = c + j - ep.actC0;
        const bool in4 = c + j >= ep.actC0 && c + j < ep.actC1;
        q[j] = (in4 && mk == 1.0f) ? applyActF(v[j] * ep.scale[ca] + ep.bias[ca], ep.act) : 0.0f;
      }
      if(c >= ep.actC0 && c + 4 <= ep.actC1 && (reinterpret_cast<uintptr_t>(o) & 15) == 0) *reinterpret_cast<float4*>(o) = make_float4(q[0], q[1], q[2], q[3]);
      else {
#pragma unroll
        for(int j = 0; j < 4; j++)
          if(c + j >= ep.actC0 && c + j < ep.actC1) o[j] = q[j];
      }
    }
  }
}

size_t smemBytes(int taps, int nr, int halo) {
  const size_t stages = 2 * ((size_t)(cfRows(nr) + 2 * halo) * CF_AS + (size_t)taps * CF_BK * CF_BN);
  return std::max(stages, (size_t)CF_KG * cfRows(nr) * CF_BN) * sizeof(float);
}

typedef void (*ConvF32Fn)(const float*, int, int, const float*, int, int, Geom, Epilogue);
constexpr int CF_MAX_NR = 5;
constexpr int CF_MAX_SMEM = 200 * 1024;
ConvF32Fn kernelOf(int taps, int nr) {
  static const ConvF32Fn k1[] = {convF32Kernel<1, 2>, convF32Kernel<1, 3>, convF32Kernel<1, 4>, convF32Kernel<1, 5>};
  static const ConvF32Fn k9[] = {convF32Kernel<9, 2>, convF32Kernel<9, 3>, convF32Kernel<9, 4>, convF32Kernel<9, 5>};
  return (taps == 9 ? k9 : k1)[nr - 2];
}

}  // namespace

// 16-byte rows of activations and weights; wider kernels reach past the one column of padding of the layout.
bool convF32Eligible(const void* in, int inStride, int inC, const void* w, int outC, int kY, int kX, const Geom& g) {
  return ((kY == 1 && kX == 1) || (kY == 3 && kX == 3)) && (inC % 4) == 0 && (outC % 4) == 0 && (inStride % 4) == 0 &&
         (reinterpret_cast<uintptr_t>(in) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 &&
         smemBytes(kY * kX, CF_MAX_NR, kY == 3 ? g.RW + 1 : 0) <= CF_MAX_SMEM;
}

cudaError_t launchConvF32(
  cudaStream_t st, const void* in, int inStride, int inC, const void* w, int outC, int kY, Geom g, const Epilogue& ep) {
  const int halo = kY == 3 ? g.RW + 1 : 0;
  const int sms = smCount();
  // Rows per tile: what counts is the SM with the most tiles, times their height (b6c96, eight boards: 150 tiles of 64 rows are
  // two on some SM, 120 of 80 rows one everywhere).
  const int nTiles = (outC + CF_BN - 1) / CF_BN;
  int nr = 2;
  long long best = 0;
  for(int c = 2; c <= CF_MAX_NR; c++) {
    const long long tiles = (long long)((g.rows + cfRows(c) - 1) / cfRows(c)) * nTiles;
    const long long cost = (tiles + sms - 1) / sms * c;
    if(c == 2 || cost <= best) { best = cost; nr = c; }
  }
  const ConvF32Fn fn = kernelOf(kY * kY, nr);
  if(const cudaError_t e = allowSharedMemory((const void*)fn, CF_MAX_SMEM)) return e;
  return launchDependent(fn, dim3((g.rows + cfRows(nr) - 1) / cfRows(nr), nTiles), dim3(CF_THREADS), smemBytes(kY * kY, nr, halo), st, (const float*)in,
                         inStride, inC, (const float*)w, outC, halo, g, ep);
}

}  // namespace kb
