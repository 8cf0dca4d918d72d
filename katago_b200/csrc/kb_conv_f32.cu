// fp32 convolution on the CUDA cores for 1x1 and 3x3 kernels over 4-channel-aligned tensors.
//
// convSimtKernel (kb_kernels.cu) takes any shape, one 16-channel slice of one tap at a time with two block barriers each and
// scalar loads; a 3x3 96->96 layer of eight boards ran at 6.5 of the 72 TFLOP/s the FMA units give, its 100 blocks spending
// their time on the load latency between the barriers.  Here a block stages ALL taps of a 16-channel slice at once: the 64
// output rows with their halo (every tap reads the same staged rows at another offset, the padded-rows layout makes that a
// constant) and the nine weight slices, double-buffered with cp.async, so that there are inC/16 steps per tile instead of
// 9*inC/16.  Tiles of 64 x 32 keep small batches on many SMs (eight boards: 150 blocks).  Each of the eight warps computes
// the whole tile over two channels of every slice, 8 x 8 outputs per thread, and the eight sums are added in warp order at
// the end: with 4 x 4 outputs per thread and two halves of a slice the shared-memory loads took twice the time of the FMAs
// (32 us per layer).  The order of the additions is the same in every batch size.
#include "kb_kernels.cuh"
#include "kb_act.cuh"
#include "kb_tc_ptx.cuh"

#include <mutex>
#include <vector>
#include <algorithm>

namespace kb {

namespace {

constexpr int CF_BM = 64, CF_BN = 32, CF_BK = 16;
constexpr int CF_AS = CF_BK + 4;      // floats per staged row: 16-byte loads of rows 20 floats apart meet no bank twice
constexpr int CF_THREADS = 256;

__device__ __forceinline__ void cpAsync16(float* dst, const float* src, bool valid) {
  // zero-filled where there is nothing to read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smemU32(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

template <int TAPS>
__global__ void __launch_bounds__(CF_THREADS) convF32Kernel(
  const float* __restrict__ in, int inStride, int inC, const float* __restrict__ w, int outC, int halo, Geom g, Epilogue ep) {
  extern __shared__ float4 smem4[];
  float* sm = reinterpret_cast<float*>(smem4);
  const int aRows = CF_BM + 2 * halo;
  const int aFloats = aRows * CF_AS, bFloats = TAPS * CF_BK * CF_BN;
  const int stage = aFloats + bFloats;
  const int tid = threadIdx.x;
  const int kg = tid >> 5, lane = tid & 31;  // this warp takes channels 2*kg, 2*kg+1 of every slice
  const int tx = lane & 3, ty = lane >> 2;   // 8 channels (4 from tx*4, 4 from 16+tx*4); rows ty, ty+8, ..., ty+56
  const int m0 = (int)blockIdx.x * CF_BM, n0 = (int)blockIdx.y * CF_BN;
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

  float acc[8][8];
#pragma unroll
  for(int i = 0; i < 8; i++)
#pragma unroll
    for(int j = 0; j < 8; j++) acc[i][j] = 0.0f;

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
      const float* a = sA + (ty + halo + shift) * CF_AS;
      const float* b = sB + tap * CF_BK * CF_BN;
      float2 av[8];
#pragma unroll
      for(int i = 0; i < 8; i++) av[i] = *reinterpret_cast<const float2*>(a + 8 * i * CF_AS);
#pragma unroll
      for(int k = 0; k < 2; k++) {
        const float4 b0 = *reinterpret_cast<const float4*>(b + k * CF_BN), b1 = *reinterpret_cast<const float4*>(b + k * CF_BN + 16);
#pragma unroll
        for(int i = 0; i < 8; i++) {
          const float x = k == 0 ? av[i].x : av[i].y;
          acc[i][0] = fmaf(x, b0.x, acc[i][0]); acc[i][1] = fmaf(x, b0.y, acc[i][1]);
          acc[i][2] = fmaf(x, b0.z, acc[i][2]); acc[i][3] = fmaf(x, b0.w, acc[i][3]);
          acc[i][4] = fmaf(x, b1.x, acc[i][4]); acc[i][5] = fmaf(x, b1.y, acc[i][5]);
          acc[i][6] = fmaf(x, b1.z, acc[i][6]); acc[i][7] = fmaf(x, b1.w, acc[i][7]);
        }
      }
    }
    __syncthreads();  // the buffer is free for the slice after next
  }

  // The warps' partial sums of the 64 x 32 tile, added in warp order by the thread that finishes 8 channels of a row.
#pragma unroll
  for(int i = 0; i < 8; i++) {
    float4* o = reinterpret_cast<float4*>(sm + kg * CF_BM * CF_BN + (ty + 8 * i) * CF_BN);
    o[tx] = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    o[4 + tx] = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
  }
  __syncthreads();
  const int r = tid >> 2, m = m0 + r;
  if(m >= g.rowsPad) return;
  const int br = m % g.PB, y = br / g.RW, x = br - y * g.RW;
  const bool point = m < g.rows && y < g.Y && x < g.X;
  const float mk = ep.mask ? ep.mask[m] : 1.0f;
  const int bIdx = min(m / g.PB, g.n - 1);
#pragma unroll
  for(int h = 0; h < 2; h++) {
    const int cl = h * 16 + (tid & 3) * 4, c = n0 + cl;
    if(c >= outC) continue;
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // stays 0 on rows of the layout that are not board points, as in the general kernel
    if(point) {
#pragma unroll
      for(int k = 0; k < CF_THREADS / 32; k++) {
        const float4 t = *reinterpret_cast<const float4*>(sm + k * CF_BM * CF_BN + r * CF_BN + cl);
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

size_t smemBytes(int taps, int halo) {
  const size_t stages = 2 * ((size_t)(CF_BM + 2 * halo) * CF_AS + (size_t)taps * CF_BK * CF_BN);
  return std::max(stages, (size_t)(CF_THREADS / 32) * CF_BM * CF_BN) * sizeof(float);
}

}  // namespace

// 16-byte rows of activations and weights; wider kernels reach past the one column of padding of the layout.
bool convF32Eligible(const void* in, int inStride, int inC, const void* w, int outC, int kY, int kX, const Geom& g) {
  return ((kY == 1 && kX == 1) || (kY == 3 && kX == 3)) && (inC % 4) == 0 && (outC % 4) == 0 && (inStride % 4) == 0 &&
         (reinterpret_cast<uintptr_t>(in) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 &&
         smemBytes(kY * kX, kY == 3 ? g.RW + 1 : 0) <= 200 * 1024;
}

cudaError_t launchConvF32(
  cudaStream_t st, const void* in, int inStride, int inC, const void* w, int outC, int kY, Geom g, const Epilogue& ep) {
  const int halo = kY == 3 ? g.RW + 1 : 0;
  const size_t smem = smemBytes(kY * kY, halo);
  void (*fn)(const float*, int, int, const float*, int, int, Geom, Epilogue) = kY == 3 ? convF32Kernel<9> : convF32Kernel<1>;
  {
    // opt in to the large dynamic shared memory once per device
    static std::mutex mu;
    static std::vector<int> done;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    if(std::find(done.begin(), done.end(), dev) == done.end()) {
      cudaError_t e = cudaFuncSetAttribute((const void*)convF32Kernel<9>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
      if(e == cudaSuccess) e = cudaFuncSetAttribute((const void*)convF32Kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
      if(e != cudaSuccess) return e;
      done.push_back(dev);
    }
  }
  return launchDependent(fn, dim3(g.rowsPad / CF_BM, (outC + CF_BN - 1) / CF_BN), dim3(CF_THREADS), smem, st, (const float*)in, inStride, inC,
                         (const float*)w, outC, halo, g, ep);
}

}  // namespace kb
