// Tensor-core convolution for small batches: one CTA per tile of 64 or 128 rows x 16 to 256 output channels.
//
// convTcKernel (kb_conv_tc.cu) gives every CTA a wide tile and a deep pipeline, which is right when there are more tiles
// than SMs.  A batch of a few positions has 4 to 40 row tiles: with 192- or 256-wide tiles most SMs idle, and a layer
// takes as long as ONE tile, i.e. 108 MMAs in a row (3x3 192->192), a weight stream of 663 KB into one SM, an epilogue of
// six 32-channel units and the start-up of a kernel.  Everything here shortens that chain:
//
// * small tiles: the same MMAs per tile, but cheaper ones, a part of the weights per SM and a short epilogue.  Cycles per MMA
//   (K=16, issued back to back): 128 rows 41 / 42 / 46 / 50 / 58 / 66 / 98 for N = 16 / 32 / 48 / 64 / 96 / 128 / 192, 64 rows
//   28 / 28 / 31 / 34 / 50 / 66 / 98: up to N = 64 the operand rows read from shared memory set the pace, so half the rows cost
//   two thirds.  The order of the additions inside an accumulator depends on neither, so a position's results stay the same
//   bit for bit in every batch size;
// * all weights of a tile in shared memory where they fit, behind one barrier, else a ring;
// * barriers, TMEM, weights and tensor maps are on their way before the wait for the launch before this one
//   (programmatic dependent launch); what is left after it is the activations, the MMAs and the epilogue;
// * the MMAs come from one elected thread whose loops are chosen once per launch and whose waits cost a single try: with a run-time
//   choice of the loop's form and a bounded wait spelled out inside it, every step cost 470 cycles beyond its MMAs
//   (3x3 192->192 of one position: 6.2 k cycles from the first MMA to the last, 1x1 384->192 3.7 k; now 3.5 k and 1.6 k);
// * the epilogue goes straight from registers to global memory, 32 bytes (a sector) per thread and access: with 16-byte accesses
//   the closing 1x1 of five positions took 1.5 to 4.5 us for its epilogue alone, every sector being written twice.
//
// What is left of a launch (5.6 us for a 3x3 layer of one position before these changes, 4.5 us now) is the launch boundary (about 1 us),
// the first activations (0.6 us), the MMAs and the epilogue (0.5 us).
//
// Each CTA computes one tile and leaves.  Every wait is bounded; see kb_conv_tc.cu.
#include "kb_conv_dev.cuh"
#include "kb_conv_small.cuh"

#include <algorithm>
#include <type_traits>

namespace kb {

namespace {

constexpr int CS_BK = 64;
constexpr int CS_EPI_WARPS = 12;                    // three per TMEM lane quarter
constexpr int CS_PARTS = CS_EPI_WARPS / 4;
constexpr int CS_THREADS = 64 + 32 * CS_EPI_WARPS;  // producer warp, MMA warp, epilogue warps
constexpr int CS_MAX_SLOTS = 32;
constexpr int CS_MAX_BN = 256;
// barriers (full and empty of both rings, accumulator), the TMEM slot and flags, the norm parameters of the tile, and the
// slack of the 1024-byte alignment
constexpr int CS_FIXED_SMEM = (4 * CS_MAX_SLOTS + 1) * 8 + 64 + 2 * CS_MAX_BN * 4 + 1024;
// Shared memory of a CTA: half of an SM's (228 KB, 1 KB reserved per CTA) or all of it
constexpr int CS_SMEM_HALF = 113 * 1024, CS_SMEM_FULL = 226 * 1024;

// Kernel variant that records the sums of squares of its raw output (Epilogue::sumsqOut) and has no activated one.
constexpr int CS_ACT_ROW_SUMS = 102;

enum { CS_ERR_PRODUCER_TIMEOUT = 121, CS_ERR_MMA_TIMEOUT = 122, CS_ERR_EPILOGUE_TIMEOUT = 123 };

// Sum of the partials that the small-batch kernel wrote for row m, twelve loads at a time (a 384-channel row).
__device__ __forceinline__ float rowSumOfUnits(const float* sums, int stride, int slots, uint32_t ends, int m) {
  float ss = 0.0f, part = 0.0f;
  for(int k0 = 0; k0 < slots; k0 += 12) {
    float t[12];
#pragma unroll
    for(int k = 0; k < 12; k++) t[k] = sums[(size_t)min(k0 + k, slots - 1) * stride + m];
#pragma unroll
    for(int k = 0; k < 12; k++) {
      // past the last slot no group ends
      part += t[k];
      const bool end = k0 + k < 32 && ((ends >> ((k0 + k) & 31)) & 1u);
      ss += end ? part : 0.0f;
      part = end ? 0.0f : part;
    }
  }
  return ss;
}
// The factor of a row-normalised convolution (Epilogue::rowSumsq) for row m, whose mask is mk; 1 without one.
__device__ __forceinline__ float rowNormScale(const Epilogue& ep, int m, float mk) {
  if(!ep.rowSumsq) return 1.0f;
  float ss = 0.0f;
  if(ep.rowSumsqEnds != 0u) ss = rowSumOfUnits(ep.rowSumsq, ep.sumsqRowStride, ep.rowSumsqSlots, ep.rowSumsqEnds, m);
  else
    for(int k = 0; k < ep.rowSumsqSlots; k++) ss += ep.rowSumsq[(size_t)k * ep.sumsqRowStride + m];
  return mk == 1.0f ? rsqrtf(fmaf(ss, ep.rowInvC, ep.rowEps)) : 0.0f;
}

struct ConvSmallArgs {
  Geom g;
  Epilogue ep;
  int outC, BN;
  int taps;        // 1 or 9
  int tapGroup;    // taps per weight slot: 1 or 3 (3x3)
  int kChunks;     // 64-channel chunks of the input; the last one may reach past the last channel (zeros)
  int haloPad;     // rows loaded above the tile
  int aSlotBytes, bSlotBytes;
  int numA, numB;  // ring depths
  uint32_t idesc, tmemCols;
  int* status;
  uint8_t sumRank[32];  // row sums: slot of each 32-channel unit (rowSumRank; a table, as its divisions took 0.5 us)
};

template <typename T, int ACT, int BM>
__global__ void __launch_bounds__(CS_THREADS, 2) convSmallKernel(
  const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ ConvSmallArgs a) {
  extern __shared__ uint8_t smemRaw[];
  uint8_t* smemA = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~(uintptr_t)1023);
  uint8_t* smemB = smemA + (size_t)a.numA * a.aSlotBytes;
  float* sScale = reinterpret_cast<float*>(smemB + (size_t)a.numB * a.bSlotBytes);
  float* sBias = sScale + CS_MAX_BN;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sBias + CS_MAX_BN);
  uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(bars + 2 * (a.numA + a.numB) + 1);
  volatile int* abortFlag = reinterpret_cast<volatile int*>(tmemSlot + 1);
  // barriers by shared-memory address: full and empty of the activation ring, full and empty of the weight ring, accumulator
  const uint32_t fullA = smemU32(bars), emptyA = fullA + 8u * (uint32_t)a.numA;
  const uint32_t fullB = emptyA + 8u * (uint32_t)a.numA, emptyB = fullB + 8u * (uint32_t)a.numB, accFull = emptyB + 8u * (uint32_t)a.numB;
  const uint32_t sA = smemU32(smemA), sB = smemU32(smemB);

  const int warp = warpIndex(), lane = threadIdx.x & 31;
  const int n0 = (int)blockIdx.x * a.BN, m0 = (int)blockIdx.y * BM;
  const Epilogue& ep = a.ep;
  const int groupsPerChunk = a.taps / a.tapGroup;
  const int totalB = a.kChunks * groupsPerChunk;
  const bool residentB = a.numB >= totalB;  // all weights of the tile fit: one barrier for all of them

  if(warp == 0 && electOne()) {
    for(int s = 0; s < 2 * (a.numA + a.numB) + 1; s++) mbarInit(fullA + 8u * (uint32_t)s, 1);
    *abortFlag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fenceProxyAsync();
    // The first weights: nothing before this launch produces them, and the ring is empty.
    if(residentB) mbarExpectTx(fullB, (uint32_t)(totalB * a.bSlotBytes));
    const int pre = residentB ? totalB : a.numB;
    for(int i = 0; i < pre; i++) {
      const uint32_t bar = residentB ? fullB : fullB + 8u * (uint32_t)i;
      if(!residentB) mbarExpectTx(bar, (uint32_t)a.bSlotBytes);
      tmaLoad3d(sB + (uint32_t)(i * a.bSlotBytes), &tmB, (i / groupsPerChunk) * CS_BK, n0, (i % groupsPerChunk) * a.tapGroup, bar);
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
  if(ACT == KB_ACT_ROPE_QK && warp >= 2) {
    // rotary frequencies of this tile's query and key channels
    for(int i = (int)threadIdx.x - 64; i < a.BN; i += CS_THREADS - 64) sScale[i] = n0 + i < ep.ropeC1 ? ep.ropeFreq[n0 + i] : 0.0f;
  }
  tcFenceBefore();
  __syncthreads();
  tcFenceAfter();
  gridDepLaunch();  // only now that this CTA holds its tensor memory (see gridDepLaunch)
  const uint32_t tmemBase = *tmemSlot;

  if(warp == 0) {
    // ---------------- TMA producer: one thread, which leaves behind a wait that ran out ----------------
    if(electOne()) {
      auto wait = [&](uint32_t bar, uint32_t parity) { return mbarWaitThread(bar, parity, abortFlag, a.status, CS_ERR_PRODUCER_TIMEOUT); };
      gridDepWait();  // activations belong to the kernels before this one
      // they may have been written with ordinary stores
      asm volatile("fence.proxy.async.global;" ::: "memory");
      auto loadA = [&](int kc, uint32_t s) {
        mbarExpectTx(fullA + 8u * s, (uint32_t)a.aSlotBytes);
        tmaLoad2d(sA + s * (uint32_t)a.aSlotBytes, &tmA, kc * CS_BK, m0 - a.haloPad, fullA + 8u * s);
      };
      const int first = min(a.numA, a.kChunks);
      for(int kc = 0; kc < first; kc++) loadA(kc, (uint32_t)kc);
      int ib = residentB ? totalB : a.numB;  // next weight slot to request
      uint32_t sb = 0, phB = 0;              // its place in the ring
      bool ok = true;
      auto loadB = [&](int upTo) {
        for(; ib < upTo && ok; ib++) {
          if(!wait(emptyB + 8u * sb, phB)) { ok = false; break; }
          mbarExpectTx(fullB + 8u * sb, (uint32_t)a.bSlotBytes);
          tmaLoad3d(sB + sb * (uint32_t)a.bSlotBytes, &tmB, (ib / groupsPerChunk) * CS_BK, n0, (ib % groupsPerChunk) * a.tapGroup, fullB + 8u * sb);
          if(++sb == (uint32_t)a.numB) { sb = 0; phB ^= 1u; }
        }
      };
      uint32_t s = 0, phA = 0;
      for(int kc = first; kc < a.kChunks && ok; kc++) {
        // weight slots that come free before this activation slot does are refilled first
        loadB(min(totalB, a.numB + (kc - a.numA + 1) * groupsPerChunk));
        if(!ok || !wait(emptyA + 8u * s, phA)) { ok = false; break; }
        loadA(kc, s);
        if(++s == (uint32_t)a.numA) { s = 0; phA ^= 1u; }
      }
      if(ok) loadB(totalB);
    }
  }
  else if(warp == 1) {
    // ---------------- MMA issuer: one thread; what a launch decides once is decided outside its loops ----------------
    if(electOne()) {
      auto wait = [&](uint32_t bar, uint32_t parity) { return mbarWaitThread(bar, parity, abortFlag, a.status, CS_ERR_MMA_TIMEOUT); };
      const uint32_t descHi = (uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29);  // stride offset | version | SWIZZLE_128B
      const uint32_t aLoBase = ((sA & 0x3FFFFu) >> 4) | (1u << 16), bLoBase = ((sB & 0x3FFFFu) >> 4) | (1u << 16);
      const uint32_t aSlot16 = (uint32_t)a.aSlotBytes >> 4, bSlot16 = (uint32_t)a.bSlotBytes >> 4, bTap16 = (uint32_t)a.BN * 8u;
      const uint32_t idesc = a.idesc, RW8 = (uint32_t)a.g.RW * 8u;
      const uint32_t tap0 = a.taps == 9 ? (uint32_t)(a.haloPad - a.g.RW - 1) * 8u : 0u;  // first row of the first tap in the halo tile
      const int kChunks = a.kChunks, numA = a.numA, numB = a.numB;
      const bool freeA = kChunks > numA;
      // LINES x TAPS taps: a weight slot holds SLOT of them
      auto issue = [&](auto lines, auto taps, auto slot, auto resident) {
        constexpr int LINES = decltype(lines)::value, TAPS = decltype(taps)::value, SLOT = decltype(slot)::value;
        constexpr bool RES = decltype(resident)::value;
        uint32_t sa = 0, phA = 0, sb = 0, phB = 0, accumulate = 0;
        if(RES && !wait(fullB, 0u)) return false;
        for(int kc = 0; kc < kChunks; kc++) {
          if(!wait(fullA + 8u * sa, phA)) return false;
          uint32_t aLo = aLoBase + sa * aSlot16 + tap0;
#pragma unroll 1
          for(int line = 0; line < LINES; line++, aLo += RW8) {
#pragma unroll
            for(int t = 0; t < TAPS; t++) {
              if(t % SLOT == 0) {
                if(!RES && !wait(fullB + 8u * sb, phB)) return false;
                tcFenceAfter();
              }
              const uint32_t bLo = bLoBase + sb * bSlot16 + (uint32_t)(t % SLOT) * bTap16;
#pragma unroll
              for(int k = 0; k < CS_BK / 16; k++) {
                ummaLoHi(tmemBase, aLo + 8u * t + 2 * k, bLo + 2 * k, descHi, idesc, accumulate);
                accumulate = 1;
              }
              if(t % SLOT == SLOT - 1) {
                if(!RES) ummaCommit(emptyB + 8u * sb);
                if(++sb == (uint32_t)numB) { sb = 0; phB ^= 1u; }
              }
            }
          }
          if(freeA) ummaCommit(emptyA + 8u * sa);
          if(++sa == (uint32_t)numA) { sa = 0; phA ^= 1u; }
        }
        return true;
      };
      constexpr std::integral_constant<int, 1> one{};
      constexpr std::integral_constant<int, 3> three{};
      bool ok;
      if(a.taps == 1) ok = residentB ? issue(one, one, one, std::true_type{}) : issue(one, one, one, std::false_type{});
      else if(residentB) ok = issue(three, three, three, std::true_type{});
      else if(a.tapGroup == 3) ok = issue(three, three, three, std::false_type{});
      else ok = issue(three, three, one, std::false_type{});
      if(ok) ummaCommit(accFull);
    }
  }
  else {
    // ---------------- Epilogue: TMEM lane quarter = warp % 4; three warps per quarter take the 16-channel units in turn ----------------
    // A thread owns 16 channels of a row: 32 bytes, a whole sector, in one access per tensor.  A 64-row accumulator lies in
    // the first 16 lanes of each quarter.
    // Row sums and SwiGLU go by 32 channels: a warp then takes both 16-channel halves in turn.
    constexpr int QROWS = BM / 4, HALVES = (ACT == CS_ACT_ROW_SUMS || ACT == KB_ACT_SWIGLU_PAIRS) ? 2 : 1;
    const int q = warp & 3, part = (warp - 2) >> 2;
    const bool row = lane < QROWS;
    const int m = m0 + q * QROWS + (lane & (QROWS - 1));
    const int units = min(a.BN, a.outC - n0) / (16 * HALVES);
    gridDepWait();
    const float mk = ep.mask ? ep.mask[m] : 1.0f;
    const bool on = mk == 1.0f;
    const int bIdx = min(m / a.g.PB, a.g.n - 1);
    const float* biasRow = ep.biasNC ? ep.biasNC + (size_t)bIdx * a.outC + n0 : nullptr;
    const T* resRow = ep.residual ? reinterpret_cast<const T*>(ep.residual) + (size_t)m * ep.resStride + n0 : nullptr;
    // This warp's 16-channel pieces in order: piece i is number (part + CS_PARTS * (i / HALVES)) * HALVES + i % HALVES of the tile.
    const int pieces = part < units ? ((units - 1 - part) / CS_PARTS + 1) * HALVES : 0;
    auto pieceAt = [&](int i) { return (part + CS_PARTS * (i / HALVES)) * HALVES + i % HALVES; };
    const float rowScale = rowNormScale(ep, m, mk);
    // rotary embedding: this thread's board point; rows that are not board points turn by the angle of (0,0), which is 0
    float ropePx = 0.0f, ropePy = 0.0f;
    if(ACT == KB_ACT_ROPE_QK) {
      const int br = m % a.g.PB, y = br / a.g.RW, x = br - y * a.g.RW;
      if(y < a.g.Y && x < a.g.X) { ropePx = (float)x; ropePy = (float)y; }
    }
    // slots of the row sums of this warp's first two units, read while the MMAs run
    const int slot0 = ACT == CS_ACT_ROW_SUMS ? a.sumRank[(n0 / 32 + part) & 31] : 0;
    const int slot1 = ACT == CS_ACT_ROW_SUMS ? a.sumRank[(n0 / 32 + part + CS_PARTS) & 31] : 0;
    float2 held[ACT == KB_ACT_SWIGLU_PAIRS ? 8 : 2];  // SwiGLU: silu of the unit's first half; row sums: the two running sums
    // The residual of the warp's first two pieces is on its way while the MMAs run (loads behind them wait their turn among the
    // operand copies of the SM's other CTA: b28 at twelve positions 1622 us with one piece ahead, 1599 with two), that of a third
    // while the first is computed.  64-row tiles are so narrow that a warp has one piece (two with row sums).
    constexpr bool AHEAD = BM == 128 || HALVES == 2;
    uint32_t res[8] = {0, 0, 0, 0, 0, 0, 0, 0}, resNext[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if(resRow && row && pieces > 0) ldGlobal32(resRow + pieceAt(0) * 16, res);
    if(AHEAD && resRow && row && pieces > 1) ldGlobal32(resRow + pieceAt(1) * 16, resNext);
    bool ok = mbarWait(accFull, 0u, abortFlag);
    ok = __all_sync(0xffffffffu, ok);
    if(!ok) {
      if(lane == 0 && !*abortFlag) { *abortFlag = 1; atomicCAS(a.status, 0, CS_ERR_EPILOGUE_TIMEOUT); }
    }
    else {
      tcFenceAfter();
#pragma unroll 1
      for(int i = 0; i < pieces; i++) {
        const int u = pieceAt(i), c = n0 + u * 16;
        uint32_t r[16];
        tmemLd16(tmemBase + ((uint32_t)(q * 32) << 16) + (uint32_t)(u * 16), r);
        tmemLdWait();
        // from here on operation for operation what epilogueTileTma (kb_conv_tc.cu) computes
        float2 v[8];
#pragma unroll
        for(int k = 0; k < 8; k++) v[k] = make_float2(__uint_as_float(r[2 * k]), __uint_as_float(r[2 * k + 1]));
        if(ep.rowSumsq) {
          const float2 rs = make_float2(rowScale, rowScale);
#pragma unroll
          for(int k = 0; k < 8; k++) v[k] = __fmul2_rn(v[k], rs);
        }
        if(biasRow) {
          const float4* bp = reinterpret_cast<const float4*>(biasRow + u * 16);
#pragma unroll
          for(int k = 0; k < 4; k++) {
            const float4 b4 = bp[k];
            v[2 * k] = __fadd2_rn(v[2 * k], make_float2(b4.x, b4.y));
            v[2 * k + 1] = __fadd2_rn(v[2 * k + 1], make_float2(b4.z, b4.w));
          }
        }
        if(resRow) {
          if(ep.resMask) {
            const float2 mk2 = make_float2(mk, mk);
#pragma unroll
            for(int k = 0; k < 8; k++) v[k] = __fmul2_rn(v[k], mk2);
          }
#pragma unroll
          for(int k = 0; k < 8; k++) v[k] = Pack2<T>::addTo(res[k], v[k]);
          if(AHEAD) {
#pragma unroll
            for(int k = 0; k < 8; k++) res[k] = resNext[k];
            if(row && i + 2 < pieces) ldGlobal32(resRow + pieceAt(i + 2) * 16, resNext);
          }
          else if(row && i + 1 < pieces) ldGlobal32(resRow + pieceAt(i + 1) * 16, res);
        }
        if(ACT == KB_ACT_ROPE_QK && c < ep.ropeC1) {
          const float4* fq = reinterpret_cast<const float4*>(sScale + u * 16);
#pragma unroll
          for(int k = 0; k < 4; k++) {
            const float4 f = fq[k];
            float sn0, cs0, sn1, cs1;
            __sincosf(fmaf(ropePy, f.y, ropePx * f.x), &sn0, &cs0);
            __sincosf(fmaf(ropePy, f.w, ropePx * f.z), &sn1, &cs1);
            const float2 t0 = v[2 * k], t1 = v[2 * k + 1];
            v[2 * k] = make_float2(t0.x * cs0 - t0.y * sn0, t0.x * sn0 + t0.y * cs0);
            v[2 * k + 1] = make_float2(t1.x * cs1 - t1.y * sn1, t1.x * sn1 + t1.y * cs1);
          }
        }
        uint32_t o[8];
        if(ACT == CS_ACT_ROW_SUMS && c >= ep.rawC0 && c < ep.rawC1) {
          if((i & 1) == 0) { held[0] = make_float2(0.0f, 0.0f); held[1] = make_float2(0.0f, 0.0f); }
#pragma unroll
          for(int k = 0; k < 8; k++) held[k & 1] = __ffma2_rn(v[k], v[k], held[k & 1]);
          if((i & 1) == 1 && row) ep.sumsqOut[(size_t)(i < 2 ? slot0 : i < 4 ? slot1 : a.sumRank[c / 32]) * ep.sumsqRowStride + m] = (held[0].x + held[0].y) + (held[1].x + held[1].y);
        }
        if(ep.outRaw && c >= ep.rawC0 && c < ep.rawC1) {
#pragma unroll
          for(int k = 0; k < 8; k++) o[k] = Pack2<T>::pack(v[k].x, v[k].y);
          if(row) stGlobal32(reinterpret_cast<T*>(ep.outRaw) + (size_t)m * ep.rawStride + (c - ep.rawC0), o);
        }
        if(ACT == KB_ACT_SWIGLU_PAIRS) {
          // pieces alternate between 16 "up" channels and their 16 "gate" channels: h = silu(up) * gate
          if(ep.outAct && c >= ep.actC0 && c < ep.actC1) {
            if((i & 1) == 0) {
              const float2 kk2 = make_float2(-1.4426950408889634f, -1.4426950408889634f), one2 = make_float2(1.0f, 1.0f);
#pragma unroll
              for(int k = 0; k < 8; k++) {
                float2 n = __fmul2_rn(v[k], kk2);
                n = __fadd2_rn(one2, make_float2(ex2Approx(n.x), ex2Approx(n.y)));
                held[k % (sizeof(held) / sizeof(float2))] = __fmul2_rn(v[k], make_float2(rcpApprox(n.x), rcpApprox(n.y)));
              }
            }
            else {
#pragma unroll
              for(int k = 0; k < 8; k++) { const float2 h = __fmul2_rn(held[k % (sizeof(held) / sizeof(float2))], v[k]); o[k] = Pack2<T>::pack(h.x, h.y); }
              if(row) stGlobal32(reinterpret_cast<T*>(ep.outAct) + (size_t)m * ep.actStride + (c - 16 - ep.actC0) / 2, o);
            }
          }
        }
        else if(ep.outAct && c >= ep.actC0 && c < ep.actC1) {
          const float4* sp = reinterpret_cast<const float4*>(sScale + u * 16);
          const float4* bp = reinterpret_cast<const float4*>(sBias + u * 16);
#pragma unroll
          for(int k = 0; k < 4; k++) {
            const float4 s4 = sp[k], b4 = bp[k];
            v[2 * k] = __ffma2_rn(v[2 * k], make_float2(s4.x, s4.y), make_float2(b4.x, b4.y));
            v[2 * k + 1] = __ffma2_rn(v[2 * k + 1], make_float2(s4.z, s4.w), make_float2(b4.z, b4.w));
          }
          actStaged2<ACT, 8>(v);
#pragma unroll
          for(int k = 0; k < 8; k++) o[k] = on ? Pack2<T>::pack(v[k].x, v[k].y) : 0u;
          if(row) stGlobal32(reinterpret_cast<T*>(ep.outAct) + (size_t)m * ep.actStride + (c - ep.actC0), o);
        }
      }
    }
  }

  // ---------------- common exit ----------------
  __syncwarp();
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
template <typename T, int BM>
ConvSmallKernelFn smallKernelForT(int act) {
  switch(act) {
    case KB_ACT_IDENTITY: return convSmallKernel<T, KB_ACT_IDENTITY, BM>;
    case KB_ACT_RELU: return convSmallKernel<T, KB_ACT_RELU, BM>;
    case KB_ACT_MISH: return convSmallKernel<T, KB_ACT_MISH, BM>;
    case KB_ACT_SILU: return convSmallKernel<T, KB_ACT_SILU, BM>;
    case KB_ACT_MISH_SCALE8: return convSmallKernel<T, KB_ACT_MISH_SCALE8, BM>;
    case KB_ACT_SWIGLU_PAIRS: return convSmallKernel<T, KB_ACT_SWIGLU_PAIRS, BM>;
    case KB_ACT_ROPE_QK: return convSmallKernel<T, KB_ACT_ROPE_QK, BM>;
    case CS_ACT_ROW_SUMS: return convSmallKernel<T, CS_ACT_ROW_SUMS, BM>;
    default: return nullptr;
  }
}
template <int BM>
ConvSmallKernelFn smallKernelFor(int dt, int act) {
  return dt == DT_F16 ? smallKernelForT<__half, BM>(act) : smallKernelForT<__nv_bfloat16, BM>(act);
}

// The kernel's variant for an epilogue, or -1.
int smallVariant(const Epilogue& ep) {
  if(ep.sumsqOut) return !ep.outAct && ep.act != KB_ACT_ROPE_QK ? CS_ACT_ROW_SUMS : -1;
  if(ep.act == KB_ACT_ROPE_QK) return !ep.outAct ? KB_ACT_ROPE_QK : -1;
  if(ep.act == KB_ACT_SWIGLU_PAIRS) return ep.outAct && !ep.outRaw ? KB_ACT_SWIGLU_PAIRS : -1;
  return ep.outAct ? ep.act : KB_ACT_IDENTITY;
}

}  // namespace

bool convSmallSupports(const Epilogue& ep) {
  // an epilogue thread moves 16 channels of a row in one 32-byte access
  auto sectors = [](const void* p, int stride) { return (reinterpret_cast<uintptr_t>(p) & 31) == 0 && stride % 16 == 0; };
  if(ep.outRaw && !sectors(ep.outRaw, ep.rawStride)) return false;
  if(ep.outAct && !sectors(ep.outAct, ep.actStride)) return false;
  if(ep.residual && !sectors(ep.residual, ep.resStride)) return false;
  const int variant = smallVariant(ep);
  return variant >= 0 && smallKernelFor<128>(DT_F16, variant) != nullptr;
}

// Which tile a launch takes.  Device time of the whole net, fp16, 19x19, in us; wide = the kernels of kb_conv_tc.cu / kb_conv_fused.cu.
//
// One CTA per SM with all of its shared memory, for layers whose MMAs outweigh the rest (3x3, and 1x1 with a long K loop): the
// first tile of the list, cheapest MMAs first, of which there are no more than SMs.  Varied for the 3x3 layers of b18: one
// position 64 x 32 516, 64 x 48 541, 64 x 16 and 128 x 16 553, 128 x 32 577; five 64 x 48 662, 128 x 32 663, 128 x 48 687;
// eight 128 x 48 774, 128 x 64 811, 64 x 96 838 (its weights do not stay resident); twelve 128 x 64 823, 128 x 96 861, twice as
// many half tiles on shared SMs 872; twenty 128 x 96 983, 128 x 48 on shared SMs 1034.  b28: twelve 128 x 96 (the last tile of a row 64
// wide) 1768, 128 x 128 1885, 128 x 64 on shared SMs 2050; twenty 128 x 128 1970, 128 x 64 on shared SMs 2101.
//
// Two CTAs per SM, which hide each other's start, loads and epilogue: 1x1 layers with a short K loop (the closing ones, whose
// epilogue reads a residual and writes two tensors) and whatever does not fit above.  Closing 1x1 of b18: one position 64 x 16
// 492, 128 x 16 504; five 128 x 32 639, 128 x 64 with an SM each 663; eight 128 x 48 725, 128 x 96 with an SM each 764; b28, twelve
// 128 x 96 1647, 128 x 192 with an SM each 1659.  3x3 layers past 148 tiles: b18 at 28 positions 128 x 64 1139, wide 1274; at 37
// 128 x 96 1305, wide 1441; b28 at 30 128 x 96 2728, wide 3283; at 40 128 x 128 3059, wide 3404.  192-wide 3x3 tiles with half an SM
// have two weight slots and are slower than the wide kernels (b18 at 48: 2353 against 1794).
//
// The projections of a transformer follow the same rules, with tiles of whole 32-channel units where row sums or SwiGLU pairs
// need them.  Producers of row sums keep to one CTA per SM (12-layer transformer, 32 boards: 1252 us with wide tiles, 1345 with
// 192-wide ones on shared SMs); the up|gate projection takes 256-wide tiles on shared SMs (11 boards, relative-position bias: 695
// us against 753 with 192-wide ones, wide 783) and, past those, up to one and a half rounds of 192-wide ones.  Of those batches, four
// layers, these / wide tiles: 384 channels with an FFN of 1024 at 12 boards 260 / 265, of 768 at 16 290 / 299 and 17 320 / 328, of 1536 at 8
// 233 / 253; 256 channels 219 / 229; 512 channels 340 / 341; 13x13 boards 25 281 / 286, 26 284 / 288; 9x9 49 262 / 265, 51 283 / 287.
// Plain transformer at 1 / 4 / 8 / 16 boards: 570 -> 367, 586 -> 417, 665 -> 519, 808 (wide).
//
// Weight slots of three taps where a wait is a good part of a slot's MMAs (b18, twelve positions, N = 64: 823 against 848 with one
// tap), of one tap for wide tiles with half an SM (b18, 37 positions, N = 96: 1340 against 1589 with three).
ConvSmallTile convSmallTile(const ConvSmallShape& s, const Epilogue& ep, int rows, int numSMs) {
  const int slot = s.taps == 9 ? 3 : 1;
  // row sums and SwiGLU go by 32 channels
  const int unit = ep.sumsqOut || ep.act == KB_ACT_SWIGLU_PAIRS ? 32 : 16;
  auto tiles = [&](int bm, int bn) { return bn % unit != 0 ? 1LL << 40 : (long long)((rows + bm - 1) / bm) * ((s.outC + bn - 1) / bn); };
  // one CTA per SM
  if(s.taps == 9 || s.inC > 256) {
    const int shapes[][2] = {{64, 32}, {64, 48}, {128, 32}, {128, 48}, {128, 64}, {128, 96}, {128, 128}};
    for(const auto& t : shapes)
      if(tiles(t[0], t[1]) <= numSMs) return ConvSmallTile{t[0], t[1], slot, CS_SMEM_FULL};
  }
  // two CTAs per SM
  if(ep.sumsqOut) return ConvSmallTile{};  // see above
  if(s.taps == 1 && tiles(64, 16) <= 2LL * numSMs) return ConvSmallTile{64, 16, 1, CS_SMEM_HALF};
  for(int bn : {16, 32, 48, 64, 96, 128, 192})
    if((s.taps == 1 || bn < 192) && tiles(128, bn) <= 2LL * numSMs) return ConvSmallTile{128, bn, s.taps == 9 && bn < 64 ? 3 : 1, CS_SMEM_HALF};
  if(ep.act == KB_ACT_SWIGLU_PAIRS && tiles(128, 256) <= 2LL * numSMs) return ConvSmallTile{128, 256, 1, CS_SMEM_HALF};
  if(ep.act == KB_ACT_SWIGLU_PAIRS && tiles(128, 192) <= 3LL * numSMs) return ConvSmallTile{128, 192, 1, CS_SMEM_HALF};
  return ConvSmallTile{};
}

cudaError_t launchConvSmall(cudaStream_t st, const ConvSmallShape& s, const ConvSmallTile& tile, Geom g, const Epilogue& ep, int* statusWord) {
  const int BM = tile.BM, BN = tile.BN, mi = convSmallMapIndex(BN);
  if((BM != 64 && BM != 128) || mi < 0 || (tile.tapGroup != 1 && (tile.tapGroup != 3 || s.taps != 9))) return cudaErrorInvalidValue;
  ConvSmallArgs a;
  a.g = g; a.ep = ep;
  a.outC = s.outC; a.BN = BN;
  a.taps = s.taps; a.tapGroup = tile.tapGroup;
  a.kChunks = (s.inC + CS_BK - 1) / CS_BK;
  a.haloPad = s.haloPad;
  a.aSlotBytes = (BM == 64 ? s.aRows - 64 : s.aRows) * 128;
  const dim3 grid((s.outC + BN - 1) / BN, (g.rows + BM - 1) / BM);
  const int budget = tile.smem - CS_FIXED_SMEM;
  // all weights of the tile (in slots of three taps) if they fit next to at least two activation slots (three in a full SM); the
  // MMAs then never wait for them.  Else a ring next to two or three activation slots.
  const int allB = a.kChunks * s.taps * BN * 128;
  const int minA = std::min(tile.smem == CS_SMEM_FULL ? 3 : 2, a.kChunks);
  if(a.kChunks * (s.taps == 9 ? 3 : 1) <= CS_MAX_SLOTS && allB + std::min(2, a.kChunks) * a.aSlotBytes <= budget) {
    a.tapGroup = s.taps == 9 ? 3 : 1;
    a.numB = a.kChunks * (s.taps / a.tapGroup);
    a.bSlotBytes = a.tapGroup * BN * 128;
    a.numA = std::min(std::min(a.kChunks, CS_MAX_SLOTS), (budget - allB) / a.aSlotBytes);
  }
  else if(s.taps == 9) {
    a.bSlotBytes = a.tapGroup * BN * 128;
    a.numA = minA;
    if(budget - a.numA * a.aSlotBytes < 2 * a.bSlotBytes) a.numA = std::min(2, a.kChunks);
    a.numB = std::min(std::min(a.kChunks * (9 / a.tapGroup), CS_MAX_SLOTS), (budget - a.numA * a.aSlotBytes) / a.bSlotBytes);
  }
  else {
    a.bSlotBytes = BN * 128;
    a.numA = std::min(std::min(a.kChunks, CS_MAX_SLOTS), budget / (a.aSlotBytes + a.bSlotBytes));
    a.numB = a.numA;
  }
  if(a.numA < 1 || a.numB < 1) return cudaErrorInvalidValue;
  const size_t smem = (size_t)a.numA * a.aSlotBytes + (size_t)a.numB * a.bSlotBytes + CS_FIXED_SMEM;
  // instruction descriptor: D=f32, A/B format, both K-major, N>>3 at bit 17, M>>4 at bit 24
  const uint32_t fmt = s.dt == DT_F16 ? 0u : 1u;
  a.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
  a.tmemCols = 32;
  while((int)a.tmemCols < BN) a.tmemCols *= 2;
  a.status = statusWord;
  for(int u = 0; u < 32; u++) a.sumRank[u] = ep.sumsqOut ? (uint8_t)rowSumRank(u, ep.sumsqTile, ep.sumsqWarps) : 0;
  const int act = smallVariant(ep);
  ConvSmallKernelFn fn = BM == 64 ? smallKernelFor<64>(s.dt, act) : smallKernelFor<128>(s.dt, act);
  if(!fn) return cudaErrorInvalidValue;
  if(const cudaError_t e = allowSharedMemory((const void*)fn, CS_SMEM_FULL)) return e;
  return launchDependent(fn, grid, dim3(CS_THREADS), smem, st, BM == 64 ? s.tmA64 : *s.tmA, a.tapGroup == 3 ? s.tmB3[mi] : s.tmB[mi], a);
}

}  // namespace kb
