// Tensor-core convolution for small batches: one CTA per tile of 128 rows x 16 to 64 output channels.
//
// convTcKernel (kb_conv_tc.cu) gives every CTA a wide tile and a deep pipeline, which is right when there are more tiles
// than SMs.  A batch of a few positions has 4 to 40 row tiles: with 192- or 256-wide tiles most SMs idle, and a layer
// takes as long as ONE tile, i.e. 108 MMAs in a row (3x3 192->192), a weight stream of 663 KB into one SM, an epilogue of
// six 32-channel units and the start-up of a kernel.  Everything here shortens that chain:
//
// * narrow tiles: the same MMAs per tile, but 41 to 49 cycles each (M=128, N=32 to 64) instead of 96, a third to a twelfth of
//   the weights per SM, and an epilogue of one 16- or 32-channel piece per warp.  The order of the additions inside an
//   accumulator does not depend on N, so a position's results stay the same bit for bit in every batch size;
// * a weight load and its barriers cover three taps (twelve MMAs): a tcgen05.commit costs as much as two narrow MMAs;
// * about half of the shared memory of an SM and at most 64 TMEM columns per CTA, so that the CTAs of the next launch
//   (programmatic dependent launch) are resident, have their barriers, their TMEM and their first weights, when the last
//   tile of this launch is done;
// * the epilogue goes straight from registers to global memory (whole 32-byte sectors per thread).
//
// Each CTA computes one tile and leaves.  Every wait is bounded; see kb_conv_tc.cu.
#include "kb_conv_dev.cuh"
#include "kb_conv_small.cuh"

#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <vector>
#include <utility>

namespace kb {

namespace {

constexpr int CS_BM = 128;
constexpr int CS_BK = 64;
constexpr int CS_EPI_WARPS = 8;                    // two per TMEM lane quarter, each over half of the tile's channels
constexpr int CS_THREADS = 64 + 32 * CS_EPI_WARPS;  // producer warp, MMA warp, epilogue warps
constexpr int CS_MAX_SLOTS = 32;
constexpr int CS_MAX_BN = 64;
// barriers (full and empty of both rings, accumulator), the TMEM slot and flags, the norm parameters of the tile, and the
// slack of the 1024-byte alignment
constexpr int CS_FIXED_SMEM = (4 * CS_MAX_SLOTS + 1) * 8 + 64 + 2 * CS_MAX_BN * 4 + 1024;
// Shared memory of a CTA: half an SM (228 KB, 1 KB of it reserved per CTA), or all of one where two launches together have
// no more CTAs than the device has SMs
constexpr int CS_SMEM_HALF = 112 * 1024, CS_SMEM_FULL = 226 * 1024;

enum { CS_ERR_PRODUCER_TIMEOUT = 121, CS_ERR_MMA_TIMEOUT = 122, CS_ERR_EPILOGUE_TIMEOUT = 123 };

struct ConvSmallArgs {
  Geom g;
  Epilogue ep;
  int outC, BN;
  int taps;        // 1 or 9
  int tapGroup;    // taps per weight slot: 1 (1x1) or 3 (3x3)
  int kChunks;     // 64-channel chunks of the input
  int lastSteps;   // 16-channel MMA steps of the last chunk
  int haloPad;     // rows loaded above the tile
  int aSlotBytes, bSlotBytes;
  int numA, numB;  // ring depths
  uint32_t idesc, tmemCols;
  int* status;
};

template <typename T, int ACT>
__global__ void __launch_bounds__(CS_THREADS, 2) convSmallKernel(
  const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const ConvSmallArgs a) {
  extern __shared__ uint8_t smemRaw[];
  uint8_t* smemA = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~(uintptr_t)1023);
  uint8_t* smemB = smemA + (size_t)a.numA * a.aSlotBytes;
  float* sScale = reinterpret_cast<float*>(smemB + (size_t)a.numB * a.bSlotBytes);
  float* sBias = sScale + CS_MAX_BN;
  uint64_t* fullA = reinterpret_cast<uint64_t*>(sBias + CS_MAX_BN);
  uint64_t* emptyA = fullA + a.numA;
  uint64_t* fullB = emptyA + a.numA;
  uint64_t* emptyB = fullB + a.numB;
  uint64_t* accFull = emptyB + a.numB;
  uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(accFull + 1);
  volatile int* abortFlag = reinterpret_cast<volatile int*>(tmemSlot + 1);

  const int warp = warpIndex(), lane = threadIdx.x & 31;
  const int n0 = (int)blockIdx.x * a.BN, m0 = (int)blockIdx.y * CS_BM;
  const Epilogue& ep = a.ep;
  const int groupsPerChunk = a.taps / a.tapGroup;
  const int totalB = a.kChunks * groupsPerChunk;

  gridDepLaunch();
  if(warp == 0 && electOne()) {
    for(int s = 0; s < a.numA; s++) { mbarInit(smemU32(&fullA[s]), 1); mbarInit(smemU32(&emptyA[s]), 1); }
    for(int s = 0; s < a.numB; s++) { mbarInit(smemU32(&fullB[s]), 1); mbarInit(smemU32(&emptyB[s]), 1); }
    mbarInit(smemU32(accFull), 1);
    *abortFlag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fenceProxyAsync();
    // The first weights: nothing before this launch produces them, and the ring is empty.
    const int pre = a.numB < totalB ? a.numB : totalB;
    for(int i = 0; i < pre; i++) {
      const uint32_t bar = smemU32(&fullB[i]);
      mbarExpectTx(bar, (uint32_t)a.bSlotBytes);
      tmaLoad3d(smemU32(smemB + (size_t)i * a.bSlotBytes), &tmB, (i / groupsPerChunk) * CS_BK, n0, (i % groupsPerChunk) * a.tapGroup, bar);
    }
  }
  if(warp == 1) { tmemAlloc(smemU32(tmemSlot), a.tmemCols); tmemRelinquish(); }
  if(warp >= 2 && ep.outAct && ep.scale) {
    // norm parameters of this tile's channels (weights as well)
    for(int i = (int)threadIdx.x - 64; i < a.BN; i += CS_THREADS - 64) {
      const int ca = n0 + i - ep.actC0;
      const bool in = n0 + i >= ep.actC0 && n0 + i < ep.actC1;
      sScale[i] = in ? ep.scale[ca] : 0.0f;
      sBias[i] = in ? ep.bias[ca] : 0.0f;
    }
  }
  tcFenceBefore();
  __syncthreads();
  tcFenceAfter();
  const uint32_t tmemBase = *tmemSlot;

  if(warp == 0) {
    // ---------------- TMA producer ----------------
    if(electOne()) {
      bool ok = true;
      int ib = a.numB < totalB ? a.numB : totalB;  // next weight slot to request
      gridDepWait();  // activations belong to the kernels before this one
      // they may have been written with ordinary stores
      asm volatile("fence.proxy.async.global;" ::: "memory");
      auto loadB = [&]() {
        const uint32_t s = (uint32_t)(ib % a.numB);
        if(!mbarWait(smemU32(&emptyB[s]), (uint32_t)(ib / a.numB - 1) & 1u, abortFlag)) { ok = false; return; }
        const uint32_t bar = smemU32(&fullB[s]);
        mbarExpectTx(bar, (uint32_t)a.bSlotBytes);
        tmaLoad3d(smemU32(smemB + (size_t)s * a.bSlotBytes), &tmB, (ib / groupsPerChunk) * CS_BK, n0, (ib % groupsPerChunk) * a.tapGroup, bar);
        ib++;
      };
      for(int kc = 0; kc < a.kChunks && ok; kc++) {
        const uint32_t s = (uint32_t)(kc % a.numA);
        if(kc >= a.numA) {
          // weight slots that come free before this activation slot does are refilled first
          while(ok && ib < totalB && ib < a.numB + (kc - a.numA + 1) * groupsPerChunk) loadB();
          if(ok && !mbarWait(smemU32(&emptyA[s]), (uint32_t)(kc / a.numA - 1) & 1u, abortFlag)) ok = false;
          if(!ok) break;
        }
        const uint32_t bar = smemU32(&fullA[s]);
        mbarExpectTx(bar, (uint32_t)a.aSlotBytes);
        tmaLoad2d(smemU32(smemA + (size_t)s * a.aSlotBytes), &tmA, kc * CS_BK, m0 - a.haloPad, bar);
      }
      while(ok && ib < totalB) loadB();
      if(!ok && !*abortFlag) { *abortFlag = 1; atomicCAS(a.status, 0, CS_ERR_PRODUCER_TIMEOUT); }
    }
  }
  else if(warp == 1) {
    // ---------------- MMA issuer ----------------
    if(electOne()) {
      const uint32_t descHi = (uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29);  // stride offset | version | SWIZZLE_128B
      const uint32_t aLoBase = ((smemU32(smemA) & 0x3FFFFu) >> 4) | (1u << 16);
      const uint32_t bLoBase = ((smemU32(smemB) & 0x3FFFFu) >> 4) | (1u << 16);
      const uint32_t aSlot16 = (uint32_t)a.aSlotBytes >> 4, bSlot16 = (uint32_t)a.bSlotBytes >> 4, bTap16 = (uint32_t)a.BN * 8u;
      const bool freeA = a.kChunks > a.numA, freeB = totalB > a.numB;
      uint32_t sa = 0, phA = 0, sb = 0, phB = 0, accumulate = 0;
      bool ok = true;
      for(int kc = 0; kc < a.kChunks && ok; kc++) {
        if(!mbarWait(smemU32(&fullA[sa]), phA, abortFlag)) { ok = false; break; }
        const uint32_t aLo = aLoBase + sa * aSlot16;
        const int steps = kc + 1 < a.kChunks ? CS_BK / 16 : a.lastSteps;
        for(int grp = 0; grp < groupsPerChunk; grp++) {
          if(!mbarWait(smemU32(&fullB[sb]), phB, abortFlag)) { ok = false; break; }
          tcFenceAfter();
          const uint32_t bLo = bLoBase + sb * bSlot16;
          if(a.taps == 9) {
            // the three taps of board line dy = grp - 1: one row (128 bytes, 8 units) apart in the halo tile
            const uint32_t aT = aLo + (uint32_t)(a.haloPad + (grp - 1) * a.g.RW - 1) * 8u;
            if(steps == CS_BK / 16) {
#pragma unroll
              for(int t = 0; t < 3; t++) {
#pragma unroll
                for(int k = 0; k < CS_BK / 16; k++) {
                  ummaLoHi(tmemBase, aT + 8u * t + 2 * k, bLo + t * bTap16 + 2 * k, descHi, a.idesc, accumulate);
                  accumulate = 1;
                }
              }
            }
            else {
              for(int t = 0; t < 3; t++)
                for(int k = 0; k < steps; k++) {
                  ummaLoHi(tmemBase, aT + 8u * t + 2 * k, bLo + t * bTap16 + 2 * k, descHi, a.idesc, accumulate);
                  accumulate = 1;
                }
            }
          }
          else {
            for(int k = 0; k < steps; k++) {
              ummaLoHi(tmemBase, aLo + 2 * k, bLo + 2 * k, descHi, a.idesc, accumulate);
              accumulate = 1;
            }
          }
          if(freeB) ummaCommit(smemU32(&emptyB[sb]));
          if(++sb == (uint32_t)a.numB) { sb = 0; phB ^= 1u; }
        }
        if(freeA && ok) ummaCommit(smemU32(&emptyA[sa]));
        if(++sa == (uint32_t)a.numA) { sa = 0; phA ^= 1u; }
      }
      if(ok) ummaCommit(smemU32(accFull));
      else if(!*abortFlag) { *abortFlag = 1; atomicCAS(a.status, 0, CS_ERR_MMA_TIMEOUT); }
    }
  }
  else {
    // ---------------- Epilogue: TMEM lane quarter = warp % 4; two warps per quarter take the 16-channel groups in turn ----------------
    const int q = warp & 3, half = (warp - 2) >> 2;
    const int m = m0 + q * 32 + lane;
    const int groups = a.BN / 16;
    gridDepWait();
    const float mk = ep.mask ? ep.mask[m] : 1.0f;
    const bool on = mk == 1.0f;
    const int bIdx = min(m / a.g.PB, a.g.n - 1);
    const float* biasRow = ep.biasNC ? ep.biasNC + (size_t)bIdx * a.outC : nullptr;
    const T* resRow = ep.residual ? reinterpret_cast<const T*>(ep.residual) + (size_t)m * ep.resStride : nullptr;
    // The residual and the board's bias of the first group are on their way while the MMAs run.
    uint4 res[2];
    float4 bias[4];
    auto fetch = [&](int gi) {
      const int c = n0 + gi * 16;
      if(resRow) {
        res[0] = reinterpret_cast<const uint4*>(resRow + c)[0];
        res[1] = reinterpret_cast<const uint4*>(resRow + c)[1];
      }
      if(biasRow) {
#pragma unroll
        for(int j = 0; j < 4; j++) bias[j] = reinterpret_cast<const float4*>(biasRow + c)[j];
      }
    };
    if(half < groups) fetch(half);
    bool ok = mbarWait(smemU32(accFull), 0u, abortFlag);
    ok = __all_sync(0xffffffffu, ok);
    if(!ok) {
      if(lane == 0 && !*abortFlag) { *abortFlag = 1; atomicCAS(a.status, 0, CS_ERR_EPILOGUE_TIMEOUT); }
    }
    else {
      tcFenceAfter();
      for(int gi = half; gi < groups; gi += 2) {
        const int c = n0 + gi * 16;
        uint32_t r[16];
        tmemLd16(tmemBase + ((uint32_t)(q * 32) << 16) + (uint32_t)(gi * 16), r);
        tmemLdWait();
        // from here on operation for operation what epilogueTileTma (kb_conv_tc.cu) computes
        float2 v[8];
#pragma unroll
        for(int k = 0; k < 8; k++) v[k] = make_float2(__uint_as_float(r[2 * k]), __uint_as_float(r[2 * k + 1]));
        if(biasRow) {
#pragma unroll
          for(int k = 0; k < 4; k++) {
            v[2 * k] = __fadd2_rn(v[2 * k], make_float2(bias[k].x, bias[k].y));
            v[2 * k + 1] = __fadd2_rn(v[2 * k + 1], make_float2(bias[k].z, bias[k].w));
          }
        }
        if(resRow) {
          if(ep.resMask) {
            const float2 mk2 = make_float2(mk, mk);
#pragma unroll
            for(int k = 0; k < 8; k++) v[k] = __fmul2_rn(v[k], mk2);
          }
          const uint32_t xu[8] = {res[0].x, res[0].y, res[0].z, res[0].w, res[1].x, res[1].y, res[1].z, res[1].w};
#pragma unroll
          for(int k = 0; k < 8; k++) v[k] = Pack2<T>::addTo(xu[k], v[k]);
        }
        if(gi + 2 < groups) fetch(gi + 2);
        if(ep.outRaw && c >= ep.rawC0 && c < ep.rawC1) {
          uint32_t pk[8];
#pragma unroll
          for(int k = 0; k < 8; k++) pk[k] = Pack2<T>::pack(v[k].x, v[k].y);
          uint4* o = reinterpret_cast<uint4*>(reinterpret_cast<T*>(ep.outRaw) + (size_t)m * ep.rawStride + (c - ep.rawC0));
          o[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          o[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
        if(ep.outAct && c >= ep.actC0 && c < ep.actC1) {
          const float4* sp = reinterpret_cast<const float4*>(sScale + gi * 16);
          const float4* bp = reinterpret_cast<const float4*>(sBias + gi * 16);
          float2 x[8];
#pragma unroll
          for(int k = 0; k < 4; k++) {
            const float4 s4 = sp[k], b4 = bp[k];
            x[2 * k] = __ffma2_rn(v[2 * k], make_float2(s4.x, s4.y), make_float2(b4.x, b4.y));
            x[2 * k + 1] = __ffma2_rn(v[2 * k + 1], make_float2(s4.z, s4.w), make_float2(b4.z, b4.w));
          }
          actStaged2<ACT, 8>(x);
          uint32_t pk[8];
#pragma unroll
          for(int k = 0; k < 8; k++) pk[k] = on ? Pack2<T>::pack(x[k].x, x[k].y) : 0u;
          uint4* o = reinterpret_cast<uint4*>(reinterpret_cast<T*>(ep.outAct) + (size_t)m * ep.actStride + (c - ep.actC0));
          o[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          o[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
      }
    }
  }

  // ---------------- common exit ----------------
  tcFenceBefore();
  __syncthreads();
  if(*abortFlag) {
    // give copies that may still be in flight time to land before the shared memory is released
    if(threadIdx.x == 0) {
      const uint64_t t0 = globalTimerNs();
      while(globalTimerNs() - t0 < 2000000ull) { __nanosleep(1000); }
    }
    __syncthreads();
  }
  if(warp == 1) {
    tcFenceAfter();
    tmemDealloc(tmemBase, a.tmemCols);
  }
}

typedef void (*ConvSmallKernelFn)(CUtensorMap, CUtensorMap, ConvSmallArgs);
template <typename T>
ConvSmallKernelFn smallKernelForT(int act) {
  switch(act) {
    case KB_ACT_IDENTITY: return convSmallKernel<T, KB_ACT_IDENTITY>;
    case KB_ACT_RELU: return convSmallKernel<T, KB_ACT_RELU>;
    case KB_ACT_MISH: return convSmallKernel<T, KB_ACT_MISH>;
    case KB_ACT_SILU: return convSmallKernel<T, KB_ACT_SILU>;
    case KB_ACT_MISH_SCALE8: return convSmallKernel<T, KB_ACT_MISH_SCALE8>;
    default: return nullptr;
  }
}

}  // namespace

bool convSmallSupports(const Epilogue& ep) {
  if(ep.sumsqOut || ep.rowSumsq || ep.act == KB_ACT_SWIGLU_PAIRS || ep.act == KB_ACT_ROPE_QK) return false;
  return !ep.outAct || smallKernelForT<__half>(ep.act) != nullptr;
}

// How wide the tiles of a launch are.  CTAs of one SM share its tensor pipe, but a narrow MMA leaves most of the pipe to
// the other CTA (N=32: 16 of 41 cycles), so the limit is the number of CTAs that are resident at once, two per SM; below
// it narrower tiles shorten each CTA's share of the weights and of the epilogue.
int convSmallTileWidth(int outC, int rowTiles, int numSMs) {
  static const int forced = getenv("KB_SMALL_BN") ? atoi(getenv("KB_SMALL_BN")) : 0;
  for(int bn : {32, 64}) {
    if(forced > 0 && bn != forced) continue;
    if(outC % bn == 0 && (long long)rowTiles * (outC / bn) <= 2LL * numSMs) return bn;
  }
  return 0;
}

cudaError_t launchConvSmall(cudaStream_t st, const ConvSmallShape& s, int BN, int numSMs, Geom g, const Epilogue& ep, int* statusWord) {
  if(BN % 16 != 0 || BN > CS_MAX_BN || BN < 16 || s.outC % BN != 0) return cudaErrorInvalidValue;
  ConvSmallArgs a;
  a.g = g; a.ep = ep;
  a.outC = s.outC; a.BN = BN;
  a.taps = s.taps; a.tapGroup = s.taps == 9 ? 3 : 1;
  a.kChunks = (s.inC + CS_BK - 1) / CS_BK;
  a.lastSteps = ((s.inC - 1) % CS_BK) / 16 + 1;
  a.haloPad = s.haloPad;
  a.aSlotBytes = s.aRows * 128;
  a.bSlotBytes = a.tapGroup * BN * 128;
  const int totalB = a.kChunks * (a.taps / a.tapGroup);
  const dim3 grid(s.outC / BN, (g.rows + CS_BM - 1) / CS_BM);
  const bool roomy = 2 * (int)(grid.x * grid.y) <= numSMs;
  const int budget = (roomy ? CS_SMEM_FULL : CS_SMEM_HALF) - CS_FIXED_SMEM;
  if(a.taps == 9) {
    // two activation slots (22.5 KB each on a 19x19 board; more where there is room), weights in the rest
    a.numA = std::min(roomy ? 4 : 2, a.kChunks);
    a.numB = std::min(std::min(totalB, CS_MAX_SLOTS), (budget - a.numA * a.aSlotBytes) / a.bSlotBytes);
  }
  else {
    a.numA = std::min(std::min(a.kChunks, CS_MAX_SLOTS), budget / (a.aSlotBytes + a.bSlotBytes));
    a.numB = a.numA;
  }
  if(a.numA < 1 || a.numB < 1) return cudaErrorInvalidValue;
  const size_t smem = (size_t)a.numA * a.aSlotBytes + (size_t)a.numB * a.bSlotBytes + CS_FIXED_SMEM;
  // instruction descriptor: D=f32, A/B format, both K-major, N>>3 at bit 17, M>>4 at bit 24
  const uint32_t fmt = s.dt == DT_F16 ? 0u : 1u;
  a.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(CS_BM >> 4) << 24);
  a.tmemCols = BN <= 32 ? 32u : 64u;
  a.status = statusWord;
  const int act = ep.outAct ? ep.act : KB_ACT_IDENTITY;
  ConvSmallKernelFn fn = s.dt == DT_F16 ? smallKernelForT<__half>(act) : smallKernelForT<__nv_bfloat16>(act);
  if(!fn) return cudaErrorInvalidValue;
  {
    // opt in to the large dynamic shared memory once per variant and device
    static std::mutex mu;
    static std::vector<std::pair<const void*, int>> done;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    const std::pair<const void*, int> key((const void*)fn, dev);
    if(std::find(done.begin(), done.end(), key) == done.end()) {
      cudaError_t e = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, CS_SMEM_FULL);
      if(e != cudaSuccess) return e;
      done.push_back(key);
    }
  }
  static const bool usePdl = getenv("KB_NO_PDL") == nullptr;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(CS_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[1];
  if(usePdl) {
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
  }
  return cudaLaunchKernelEx(&cfg, fn, *s.tmA, BN == 32 ? s.tmB32 : s.tmB64, a);
}

}  // namespace kb
