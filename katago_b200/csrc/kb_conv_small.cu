// Tensor-core convolution for small batches: one CTA per tile of 128 rows x 16 to 96 output channels.
//
// convTcKernel (kb_conv_tc.cu) gives every CTA a wide tile and a deep pipeline, which is right when there are more tiles
// than SMs.  A batch of a few positions has 4 to 40 row tiles: with 192- or 256-wide tiles most SMs idle, and a layer
// takes as long as ONE tile, i.e. 108 MMAs in a row (3x3 192->192), a weight stream of 663 KB into one SM, an epilogue of
// six 32-channel units and the start-up of a kernel.  Everything here shortens that chain:
//
// * narrow tiles: the same MMAs per tile, but about 50 cycles each (M=128, N=32, issued by this loop in isolation) instead of 96, a half
//   to a twelfth of the weights per SM, and an epilogue of one to three 8-channel pieces per warp.  The order of the additions
//   inside an accumulator does not depend on N, so a position's results stay the same bit for bit in every batch size;
// * all weights of a tile in shared memory where they fit, behind one barrier, else a ring whose slots hold three taps: a
//   wait costs the issuing warp as much as two narrow MMAs;
// * barriers, TMEM, weights and tensor maps are on their way before the wait for the launch before this one
//   (programmatic dependent launch); what is left after it is the activations, the MMAs and the epilogue;
// * the epilogue goes straight from registers to global memory.
//
// A 3x3 192->192 launch of one position takes 6.5 us (15 us per layer in the wide-tile chain), and nothing in it is busy: on the
// 48 SMs that have a tile the tensor pipe works 7 % of the cycles and 12 % of the issue slots are taken.  It is a chain of the
// launch boundary, the first activations, 108 MMAs in a row and the epilogue.
//
// Each CTA computes one tile and leaves.  Every wait is bounded; see kb_conv_tc.cu.
#include "kb_conv_dev.cuh"
#include "kb_conv_small.cuh"

#include <algorithm>

namespace kb {

namespace {

constexpr int CS_BM = 128;
constexpr int CS_BK = 64;
constexpr int CS_EPI_WARPS = 16;                   // four per TMEM lane quarter
constexpr int CS_THREADS = 64 + 32 * CS_EPI_WARPS;  // producer warp, MMA warp, epilogue warps
constexpr int CS_MAX_SLOTS = 32;
constexpr int CS_MAX_BN = 96;
// barriers (full and empty of both rings, accumulator), the TMEM slot and flags, the norm parameters of the tile, and the
// slack of the 1024-byte alignment
constexpr int CS_FIXED_SMEM = (4 * CS_MAX_SLOTS + 1) * 8 + 64 + 2 * CS_MAX_BN * 4 + 1024;
// Shared memory of a CTA: all of an SM where the tiles are no more than the SMs, else half of one (228 KB, 1 KB reserved per CTA)
constexpr int CS_SMEM_HALF = 113 * 1024, CS_SMEM_FULL = 226 * 1024;

enum { CS_ERR_PRODUCER_TIMEOUT = 121, CS_ERR_MMA_TIMEOUT = 122, CS_ERR_EPILOGUE_TIMEOUT = 123 };

struct ConvSmallArgs {
  Geom g;
  Epilogue ep;
  int outC, BN;
  int taps;        // 1 or 9
  int tapGroup;    // taps per weight slot: 1 (1x1) or 3 (3x3)
  int kChunks;     // 64-channel chunks of the input; the last one may reach past the last channel (zeros)
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
  const bool residentB = a.numB >= totalB;  // all weights of the tile fit: one barrier for all of them

  if(warp == 0 && electOne()) {
    for(int s = 0; s < a.numA; s++) { mbarInit(smemU32(&fullA[s]), 1); mbarInit(smemU32(&emptyA[s]), 1); }
    for(int s = 0; s < a.numB; s++) { mbarInit(smemU32(&fullB[s]), 1); mbarInit(smemU32(&emptyB[s]), 1); }
    mbarInit(smemU32(accFull), 1);
    *abortFlag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fenceProxyAsync();
    // The first weights: nothing before this launch produces them, and the ring is empty.
    if(residentB) mbarExpectTx(smemU32(&fullB[0]), (uint32_t)(totalB * a.bSlotBytes));
    const int pre = residentB ? totalB : a.numB;
    for(int i = 0; i < pre; i++) {
      const uint32_t bar = smemU32(&fullB[residentB ? 0 : i]);
      if(!residentB) mbarExpectTx(bar, (uint32_t)a.bSlotBytes);
      tmaLoad3d(smemU32(smemB + (size_t)i * a.bSlotBytes), &tmB, (i / groupsPerChunk) * CS_BK, n0, (i % groupsPerChunk) * a.tapGroup, bar);
    }
    prefetchTensorMap(&tmA);
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
  gridDepLaunch();  // only now that this CTA holds its tensor memory (see gridDepLaunch)
  const uint32_t tmemBase = *tmemSlot;

  if(warp == 0) {
    // ---------------- TMA producer: all lanes wait, an elected one issues ----------------
    // Behind a wait it asks the abort flag before it arms a slot.  The flag is raised before any slot can be given back
    // wrongly: by its own wait, or by one of the MMA issuer, which goes on after a time-out (its MMAs stay inside the CTA's
    // buffers, and each of its arrivals ends a phase of a barrier that counts one).
    auto wait = [&](uint64_t* bar, uint32_t parity) { (void)mbarWaitWarp(smemU32(bar), parity, abortFlag, a.status, CS_ERR_PRODUCER_TIMEOUT); };
    int ib = residentB ? totalB : a.numB;  // next weight slot to request
    gridDepWait();  // activations belong to the kernels before this one
    // they may have been written with ordinary stores
    asm volatile("fence.proxy.async.global;" ::: "memory");
    auto loadB = [&]() {
      const uint32_t s = (uint32_t)(ib % a.numB);
      wait(&emptyB[s], (uint32_t)(ib / a.numB - 1) & 1u);
      if(electOne() && !*abortFlag) {
        const uint32_t bar = smemU32(&fullB[s]);
        mbarExpectTx(bar, (uint32_t)a.bSlotBytes);
        tmaLoad3d(smemU32(smemB + (size_t)s * a.bSlotBytes), &tmB, (ib / groupsPerChunk) * CS_BK, n0, (ib % groupsPerChunk) * a.tapGroup, bar);
      }
      ib++;
    };
    auto loadA = [&](int kc, uint32_t s) {
      const uint32_t bar = smemU32(&fullA[s]);
      mbarExpectTx(bar, (uint32_t)a.aSlotBytes);
      tmaLoad2d(smemU32(smemA + (size_t)s * a.aSlotBytes), &tmA, kc * CS_BK, m0 - a.haloPad, bar);
    };
    const int first = min(a.numA, a.kChunks);
    if(electOne()) {
      for(int kc = 0; kc < first; kc++) loadA(kc, (uint32_t)kc);
    }
    for(int kc = first; kc < a.kChunks; kc++) {
      const uint32_t s = (uint32_t)(kc % a.numA);
      // weight slots that come free before this activation slot does are refilled first
      while(ib < totalB && ib < a.numB + (kc - a.numA + 1) * groupsPerChunk) loadB();
      wait(&emptyA[s], (uint32_t)(kc / a.numA - 1) & 1u);
      if(electOne() && !*abortFlag) loadA(kc, s);
    }
    while(ib < totalB) loadB();
  }
  else if(warp == 1) {
    // ---------------- MMA issuer: all lanes wait, an elected one issues ----------------
    auto wait = [&](uint64_t* bar, uint32_t parity) { (void)mbarWaitWarp(smemU32(bar), parity, abortFlag, a.status, CS_ERR_MMA_TIMEOUT); };
    const uint32_t descHi = (uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29);  // stride offset | version | SWIZZLE_128B
    const uint32_t aLoBase = ((smemU32(smemA) & 0x3FFFFu) >> 4) | (1u << 16);
    const uint32_t bLoBase = ((smemU32(smemB) & 0x3FFFFu) >> 4) | (1u << 16);
    const uint32_t aSlot16 = (uint32_t)a.aSlotBytes >> 4, bSlot16 = (uint32_t)a.bSlotBytes >> 4, bTap16 = (uint32_t)a.BN * 8u;
    const bool freeA = a.kChunks > a.numA;
    uint32_t sa = 0, phA = 0, sb = 0, phB = 0;
    if(residentB) wait(&fullB[0], 0u);
    for(int kc = 0; kc < a.kChunks; kc++) {
      wait(&fullA[sa], phA);
      const uint32_t aLo = aLoBase + sa * aSlot16;
      if(a.taps == 9) {
        for(int grp = 0; grp < 3; grp++) {
          if(!residentB) wait(&fullB[sb], phB);
          tcFenceAfter();
          if(electOne()) {
            // the three taps of board line dy = grp - 1: one row (128 bytes, 8 units) apart in the halo tile
            const uint32_t aT = aLo + (uint32_t)(a.haloPad + (grp - 1) * a.g.RW - 1) * 8u, bLo = bLoBase + sb * bSlot16;
#pragma unroll
            for(int t = 0; t < 3; t++) {
#pragma unroll
              for(int k = 0; k < CS_BK / 16; k++)
                ummaLoHi(tmemBase, aT + 8u * t + 2 * k, bLo + t * bTap16 + 2 * k, descHi, a.idesc, (t == 0 && k == 0) ? (uint32_t)(kc + grp) : 1u);
            }
            if(!residentB) ummaCommit(smemU32(&emptyB[sb]));
            if(freeA && grp == 2) ummaCommit(smemU32(&emptyA[sa]));
          }
          if(++sb == (uint32_t)a.numB) { sb = 0; phB ^= 1u; }
        }
      }
      else {
        if(!residentB) wait(&fullB[sb], phB);
        tcFenceAfter();
        if(electOne()) {
          const uint32_t bLo = bLoBase + sb * bSlot16;
#pragma unroll
          for(int k = 0; k < CS_BK / 16; k++) ummaLoHi(tmemBase, aLo + 2 * k, bLo + 2 * k, descHi, a.idesc, k == 0 ? (uint32_t)kc : 1u);
          if(!residentB) ummaCommit(smemU32(&emptyB[sb]));
          if(freeA) ummaCommit(smemU32(&emptyA[sa]));
        }
        if(++sb == (uint32_t)a.numB) { sb = 0; phB ^= 1u; }
      }
      if(++sa == (uint32_t)a.numA) { sa = 0; phA ^= 1u; }
    }
    if(electOne()) ummaCommit(smemU32(accFull));
  }
  else {
    // ---------------- Epilogue: TMEM lane quarter = warp % 4; four warps per quarter take the 8-channel groups in turn ----------------
    // Little code per thread on purpose: it runs one to three times per launch, so fetching it counts.
    const int q = warp & 3, part = (warp - 2) >> 2;
    const int m = m0 + q * 32 + lane;
    const int groups = a.BN / 8;
    gridDepWait();
    const float mk = ep.mask ? ep.mask[m] : 1.0f;
    const bool on = mk == 1.0f;
    const int bIdx = min(m / a.g.PB, a.g.n - 1);
    const float* biasRow = ep.biasNC ? ep.biasNC + (size_t)bIdx * a.outC + n0 : nullptr;
    const T* resRow = ep.residual ? reinterpret_cast<const T*>(ep.residual) + (size_t)m * ep.resStride + n0 : nullptr;
    // The residual and the board's bias of the first group are on their way while the MMAs run.
    uint4 res = make_uint4(0u, 0u, 0u, 0u);
    float4 bias[2];
    auto fetch = [&](int gi) {
      if(resRow) res = *reinterpret_cast<const uint4*>(resRow + gi * 8);
      if(biasRow) { bias[0] = reinterpret_cast<const float4*>(biasRow + gi * 8)[0]; bias[1] = reinterpret_cast<const float4*>(biasRow + gi * 8)[1]; }
    };
    if(part < groups) fetch(part);
    bool ok = mbarWait(smemU32(accFull), 0u, abortFlag);
    ok = __all_sync(0xffffffffu, ok);
    if(!ok) {
      if(lane == 0 && !*abortFlag) { *abortFlag = 1; atomicCAS(a.status, 0, CS_ERR_EPILOGUE_TIMEOUT); }
    }
    else {
      tcFenceAfter();
#pragma unroll 1
      for(int gi = part; gi < groups; gi += CS_EPI_WARPS / 4) {
        const int c = n0 + gi * 8;
        uint32_t r[8];
        tmemLd8(tmemBase + ((uint32_t)(q * 32) << 16) + (uint32_t)(gi * 8), r);
        tmemLdWait();
        // from here on operation for operation what epilogueTileTma (kb_conv_tc.cu) computes
        float2 v[4];
#pragma unroll
        for(int k = 0; k < 4; k++) v[k] = make_float2(__uint_as_float(r[2 * k]), __uint_as_float(r[2 * k + 1]));
        if(biasRow) {
#pragma unroll
          for(int k = 0; k < 2; k++) {
            v[2 * k] = __fadd2_rn(v[2 * k], make_float2(bias[k].x, bias[k].y));
            v[2 * k + 1] = __fadd2_rn(v[2 * k + 1], make_float2(bias[k].z, bias[k].w));
          }
        }
        if(resRow) {
          if(ep.resMask) {
            const float2 mk2 = make_float2(mk, mk);
#pragma unroll
            for(int k = 0; k < 4; k++) v[k] = __fmul2_rn(v[k], mk2);
          }
          const uint32_t xu[4] = {res.x, res.y, res.z, res.w};
#pragma unroll
          for(int k = 0; k < 4; k++) v[k] = Pack2<T>::addTo(xu[k], v[k]);
        }
        if(gi + CS_EPI_WARPS / 4 < groups) fetch(gi + CS_EPI_WARPS / 4);
        if(ep.outRaw && c >= ep.rawC0 && c < ep.rawC1) {
          uint4 o;
          o.x = Pack2<T>::pack(v[0].x, v[0].y); o.y = Pack2<T>::pack(v[1].x, v[1].y);
          o.z = Pack2<T>::pack(v[2].x, v[2].y); o.w = Pack2<T>::pack(v[3].x, v[3].y);
          *reinterpret_cast<uint4*>(reinterpret_cast<T*>(ep.outRaw) + (size_t)m * ep.rawStride + (c - ep.rawC0)) = o;
        }
        if(ep.outAct && c >= ep.actC0 && c < ep.actC1) {
          const float4* sp = reinterpret_cast<const float4*>(sScale + gi * 8);
          const float4* bp = reinterpret_cast<const float4*>(sBias + gi * 8);
          float2 x[4];
#pragma unroll
          for(int k = 0; k < 2; k++) {
            const float4 s4 = sp[k], b4 = bp[k];
            x[2 * k] = __ffma2_rn(v[2 * k], make_float2(s4.x, s4.y), make_float2(b4.x, b4.y));
            x[2 * k + 1] = __ffma2_rn(v[2 * k + 1], make_float2(s4.z, s4.w), make_float2(b4.z, b4.w));
          }
          actStaged2<ACT, 4>(x);
          uint4 o = make_uint4(0u, 0u, 0u, 0u);
          if(on) {
            o.x = Pack2<T>::pack(x[0].x, x[0].y); o.y = Pack2<T>::pack(x[1].x, x[1].y);
            o.z = Pack2<T>::pack(x[2].x, x[2].y); o.w = Pack2<T>::pack(x[3].x, x[3].y);
          }
          *reinterpret_cast<uint4*>(reinterpret_cast<T*>(ep.outAct) + (size_t)m * ep.actStride + (c - ep.actC0)) = o;
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

// How wide the tiles of a launch are.  While the tiles are no more than the SMs, each CTA has an SM to itself and the
// narrowest such tile is the best: its CTAs stream the fewest weights and have the shortest epilogue.  (b18, whole net, 16 /
// 32 / 64 / 96 wide: one position 714 / 774 / 958 / 1084 us, five 1277 / 836 / 1020 / 1184, eight - / 1426 / 1057 / 1205,
// twenty - / - / 1954 / 1328; the figures left of the smallest are past one CTA per SM with a full SM's memory each.)
// Past that, two CTAs share an SM with half of its memory each: with 152 64-wide tiles b28's twelve positions take 2411 us
// against 2536 in 128-wide tiles with an SM each and 3049 in the wide-tile kernels; with 228 32-wide ones b18's twelve
// take 1143 us against 1106 in 114 64-wide ones.  Over the whole range of this rule, against the wide-tile kernels: b18 with
// 24 to 31 boards (225 to 291 64-wide tiles) 1278 to 1299 us against 1426 to 1439, with 96 to 120 boards of 9x9 1290 to 1301
// against 1437 to 1441, b28 with 12 to 23 boards 2261 to 2359 against 2836 to 2947; one board past it both are the same.
int convSmallTileWidth(int outC, int rowTiles, int numSMs) {
  for(int bn : {16, 32, 64, 96})
    if(outC % bn == 0 && (long long)rowTiles * (outC / bn) <= numSMs) return bn;
  for(int bn : {32, 64})
    if(outC % bn == 0 && (long long)rowTiles * (outC / bn) <= 2LL * numSMs) return bn;
  return 0;
}

cudaError_t launchConvSmall(cudaStream_t st, const ConvSmallShape& s, int BN, int numSMs, Geom g, const Epilogue& ep, int* statusWord) {
  if(BN % 16 != 0 || BN > CS_MAX_BN || BN < 16 || s.outC % BN != 0) return cudaErrorInvalidValue;
  ConvSmallArgs a;
  a.g = g; a.ep = ep;
  a.outC = s.outC; a.BN = BN;
  a.taps = s.taps; a.tapGroup = s.taps == 9 ? 3 : 1;
  a.kChunks = (s.inC + CS_BK - 1) / CS_BK;
  a.haloPad = s.haloPad;
  a.aSlotBytes = s.aRows * 128;
  a.bSlotBytes = a.tapGroup * BN * 128;
  const int totalB = a.kChunks * (a.taps / a.tapGroup);
  const dim3 grid(s.outC / BN, (g.rows + CS_BM - 1) / CS_BM);
  const bool roomy = (int)(grid.x * grid.y) <= numSMs;
  const int budget = (roomy ? CS_SMEM_FULL : CS_SMEM_HALF) - CS_FIXED_SMEM;
  if(a.taps == 9) {
    // all weights of the tile if they fit next to at least two activation slots (22.5 KB each on a 19x19 board), which the
    // MMAs then never wait for; else a ring of them next to two slots (three where there is room)
    const int allB = totalB * a.bSlotBytes;
    a.numA = std::min(roomy ? 3 : 2, a.kChunks);
    a.numB = std::min(std::min(totalB, CS_MAX_SLOTS), (budget - a.numA * a.aSlotBytes) / a.bSlotBytes);
    if(a.numB < totalB && totalB <= CS_MAX_SLOTS && allB + 2 * a.aSlotBytes <= budget) { a.numA = 2; a.numB = totalB; }
    while(a.numB == totalB && a.numA < a.kChunks && a.numA < CS_MAX_SLOTS && allB + (a.numA + 1) * a.aSlotBytes <= budget) a.numA++;
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
  a.tmemCols = BN <= 32 ? 32u : BN <= 64 ? 64u : 128u;
  a.status = statusWord;
  const int act = ep.outAct ? ep.act : KB_ACT_IDENTITY;
  ConvSmallKernelFn fn = s.dt == DT_F16 ? smallKernelForT<__half>(act) : smallKernelForT<__nv_bfloat16>(act);
  if(!fn) return cudaErrorInvalidValue;
  if(const cudaError_t e = allowSharedMemory((const void*)fn, CS_SMEM_FULL)) return e;
  return launchDependent(fn, grid, dim3(CS_THREADS), smem, st, *s.tmA, s.tmB[convSmallMapIndex(BN)], a);
}

}  // namespace kb
