// The 1x1 convolution that closes a nested bottleneck block and the 1x1 convolution that opens the next one, as one
// kernel (eigenbackend.cpp:1254-1303: trunk += postConv(act(postBN(mid))); nextMid = preConv(act(preBN(trunk)))).
//
// As two launches the pair is bound by memory: the first writes the activated trunk tensor (the widest tensor of the
// net) only for the second to read it back once.  Here the activated values never leave the SM: the epilogue of the
// first GEMM writes them into tensor memory, from where the second GEMM takes its A operand.  Per 128 rows the kernel reads
// the block's mid tensor and the residual stream and writes the stream, the next block's mid stream and its activated
// form: 7/12 of the bytes of the two separate kernels.
//
// One persistent CTA per SM; warp 0 issues TMA loads, warp 1 issues the MMAs, warps 2..13 are epilogue warps (three per
// TMEM lane quarter).  GEMM1 (rows x Cm -> Ct) runs in parts of 64 to 192 output channels; the epilogue of a part adds the
// residual, stores the updated stream (TMA), and writes act(norm(.)) * mask, two 16-bit channels per column, into one of four
// operand chunks of 64 channels; GEMM2 (rows x Ct -> Cn) multiplies the chunks in turn into an accumulator of its own, whose
// epilogue stores the next mid stream and its activated form.  Weights of both GEMMs stream through one ring of slots.
// Every wait is bounded.
#include "kb_conv_dev.cuh"
#include "kb_fused_shape.h"

#include <cuda.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>
#include <algorithm>
#include <utility>

namespace kb {

constexpr int PP_BM = 128;          // rows per tile
constexpr int PP_EPI_WARPS = 4 * PP_CG;
constexpr int PP_THREADS = 64 + 32 * PP_EPI_WARPS;
constexpr int PP_UNIT = 32 * 64;    // staging unit: 32 rows x 32 channels of the storage type (64-byte swizzle)
constexpr int PP_CHUNK = PP_BM * 128;  // one 64-channel K chunk of an A operand: 128 rows x 128 bytes
constexpr int PP_MAX_SLOTS = 8;     // weight ring
constexpr int PP_STAGE = 3;         // staging units per epilogue warp: two of the residual / updated stream, one more for GEMM2's outputs
constexpr int PP_FIXED = 512;       // barriers and the TMEM slot

// Optional timeline (build with -DKB_TC_TRACE): CTA 0 records SM cycle counts of its MMA warp and of its first epilogue
// warp for the first tiles; read back with kb_debug_trace_pp.
#ifdef KB_TC_TRACE
__device__ long long g_ppTrace[1024];
#define PPT(cond, slot) do { if(blockIdx.x == 0 && (cond) && (slot) < 1024) g_ppTrace[(slot)] = clock64(); } while(0)
#else
#define PPT(cond, slot) do { } while(0)
#endif

enum { PP_ERR_PRODUCER = 111, PP_ERR_MMA = 112, PP_ERR_EPILOGUE = 113, PP_ERR_ALIGNMENT = 114 };

struct PostPreArgs {
  Geom g;
  int Cm, Ct, Cn;          // GEMM1: Cm -> Ct (+ residual); GEMM2: Ct -> Cn
  int NP, parts;           // output channels of GEMM1 per part (64, 128 or 192), Ct / NP
  int N2, pieces;          // output channels of GEMM2 per weight slot, Cn / N2
  int kc1;                 // Cm / 64
  int numB, bSlot;         // weight ring: slots and bytes per slot
  int numD1;               // accumulators of GEMM1 (1 or 2)
  uint32_t idesc1, idesc2;
  const float* scale1; const float* bias1;   // norm + activation between the two convolutions (Ct channels)
  const float* scale2; const float* bias2;   // norm + activation after the second one (Cn channels)
  const float* mask;
  int* status;
};

// What bounds it: no unit alone.  b18 at batch 256 (profiles/conv_kernels_by_shape_ncu.md): special-function pipe busy for 50 % of
// the cycles (two operations per activated value), issue slots 40 %, L1 and shared memory 43 %, DRAM 37 %, tensor pipe 23 %; the 3.5 warps of
// a scheduler mostly wait for results of fixed latency and for tensor memory.  256 -> 512 -> 256 (bf16) stays lower: 39, 32, 35, 32 and
// 25 %, with twice the waits for tensor memory per instruction and one accumulator for GEMM1.
// With the operand chunks of GEMM2 in shared memory a tile of 128 rows moved 1.5 MB through it and took 18.5 k cycles, now 1.3 MB and 17 k.
// Tried on top of that and slower: parts of 128 channels with two accumulators of GEMM1 (A1 is read three times instead of
// twice; 97 us a launch at batch 256 against 86), 24 epilogue warps with units of 16 channels (97 us), outputs of GEMM2 from registers in
// 32-byte pieces (104 us), one reciprocal for two activations (no change).  batch 256: 89.4 -> 85.8 us; 256 -> 512 -> 256 (b28, batch
// 512, bf16) 254 us against 265 as two launches.
//
// The outputs of GEMM2 are read one tile late, after the warp's first unit of the next tile: nobody waits for GEMM2's last chunk
// (1.6 k cycles a tile).  Schedule over the CTA's tiles, parts numbered through, with D accumulators for GEMM1:
//   MMA warp:  G1(0) .. G1(D-1) | for each part P: G2(first chunk of P) | G1(P+D) | G2(other chunks of P)
//   epilogue:  for each tile: unit cg | outputs of GEMM2 of the tile before | units cg+3, cg+6, ...
// shared memory: [A1: kc1 chunks][weight ring][staging: 3 units per epilogue warp][barriers]
// tensor memory: [GEMM1: D x NP columns][GEMM2: Cn][operand chunks: 4 x 32]
template <typename T, int ACT>
__global__ void __launch_bounds__(PP_THREADS, 1) convPostPreKernel(
  const __grid_constant__ CUtensorMap tmA1, const __grid_constant__ CUtensorMap tmW1, const __grid_constant__ CUtensorMap tmW2,
  const __grid_constant__ CUtensorMap tmS, const __grid_constant__ CUtensorMap tmRaw2, const __grid_constant__ CUtensorMap tmAct2,
  const __grid_constant__ PostPreArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sA1 = smem;
  uint8_t* sB = sA1 + (size_t)a.kc1 * PP_CHUNK;
  uint8_t* sStage = sB + (size_t)a.numB * a.bSlot;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sStage + (size_t)PP_EPI_WARPS * PP_STAGE * PP_UNIT);
  uint64_t* a1Full = bars;
  uint64_t* a1Empty = a1Full + 1;
  uint64_t* bFull = a1Empty + 1;             // [PP_MAX_SLOTS]
  uint64_t* bEmpty = bFull + PP_MAX_SLOTS;   // [PP_MAX_SLOTS]
  uint64_t* d1Full = bEmpty + PP_MAX_SLOTS;  // [2]
  uint64_t* d1Empty = d1Full + 2;            // [2]
  uint64_t* a2Full = d1Empty + 2;            // [PP_NUM_A2]
  uint64_t* a2Empty = a2Full + PP_NUM_A2;    // [PP_NUM_A2]
  uint64_t* d2Full = a2Empty + PP_NUM_A2;
  uint64_t* d2Empty = d2Full + 1;
  uint64_t* resFull = d2Empty + 1;           // [PP_EPI_WARPS][2]
  uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(resFull + PP_EPI_WARPS * 2);
  volatile int* abortFlag = reinterpret_cast<volatile int*>(tmemSlot + 1);
  static_assert((2 + 2 * PP_MAX_SLOTS + 4 + 2 * PP_NUM_A2 + 2 + PP_EPI_WARPS * 2) * 8 + 8 <= PP_FIXED, "barriers");

  const int warp = warpIndex(), lane = threadIdx.x & 31;
  const int grid = (int)gridDim.x;
  const int allTiles = a.g.rowsPad / PP_BM;
  const int nTiles = (int)blockIdx.x < allTiles ? (allTiles - 1 - (int)blockIdx.x) / grid + 1 : 0;  // of this CTA
  const int cpp = a.NP / 64;   // K chunks of GEMM2 per part
  const int UP = a.NP / 32;    // 32-channel units per part

  if(threadIdx.x == 0) {
    mbarInit(smemU32(a1Full), 1); mbarInit(smemU32(a1Empty), 1);
    for(int s = 0; s < PP_MAX_SLOTS; s++) { mbarInit(smemU32(&bFull[s]), 1); mbarInit(smemU32(&bEmpty[s]), 1); }
    for(int s = 0; s < 2; s++) { mbarInit(smemU32(&d1Full[s]), 1); mbarInit(smemU32(&d1Empty[s]), 4 * UP); }  // a part's units x 4 quarters
    for(int s = 0; s < PP_NUM_A2; s++) { mbarInit(smemU32(&a2Full[s]), 8); mbarInit(smemU32(&a2Empty[s]), 1); }  // a chunk = 2 units x 4 quarters
    mbarInit(smemU32(d2Full), 1); mbarInit(smemU32(d2Empty), PP_EPI_WARPS);
    for(int s = 0; s < PP_EPI_WARPS * 2; s++) mbarInit(smemU32(&resFull[s]), 1);
    // the swizzled operand layouts assume a 1024-byte aligned base
    *abortFlag = (smemU32(smem) & 1023u) ? 1 : 0;
    if(*abortFlag) atomicCAS(a.status, 0, PP_ERR_ALIGNMENT);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if(warp == 1) { tmemAlloc(smemU32(tmemSlot), 512); tmemRelinquish(); }
  tcFenceBefore();
  __syncthreads();
  tcFenceAfter();
  gridDepLaunch();
  const uint32_t tmemBase = *tmemSlot;
  // tensor memory: accumulators of GEMM1, accumulator of GEMM2, operand chunks of GEMM2
  const uint32_t d2Col = (uint32_t)(a.numD1 * a.NP), a2Col = d2Col + (uint32_t)a.Cn;
  const bool bad = *abortFlag != 0;

  if(bad) {
    // misaligned shared memory: nothing runs
  }
  else if(warp == 0) {
    // ---------------- TMA producer: in the order in which the MMA warp consumes ----------------
    if(electOne()) {
      uint32_t sb = 0, ph = 0;
      bool ok = true;
      auto loadW = [&](const CUtensorMap* tm, int kc, int row, uint32_t bytes) {
        if(!ok) return;
        if(!mbarWait(smemU32(&bEmpty[sb]), ph ^ 1u, abortFlag)) { ok = false; return; }
        const uint32_t bar = smemU32(&bFull[sb]);
        mbarExpectTx(bar, bytes);
        tmaLoad2d(smemU32(sB + (size_t)sb * a.bSlot), tm, kc * 64, row, bar);
        if(++sb == (uint32_t)a.numB) { sb = 0; ph ^= 1u; }
      };
      int gTile = 0, gPart = 0;  // the next part of GEMM1
      int first = 0;             // its first K chunk whose weights have not been requested
      auto loadG1 = [&]() {
        if(gTile >= nTiles) return;
        if(gPart == 0 && ok) {
          // the buffer is free once the last part of the tile before has been multiplied
          if(!mbarWait(smemU32(a1Empty), ((uint32_t)gTile & 1u) ^ 1u, abortFlag)) { ok = false; return; }
          mbarExpectTx(smemU32(a1Full), (uint32_t)(a.kc1 * PP_CHUNK));
          const int row = ((int)blockIdx.x + gTile * grid) * PP_BM;
          for(int kc = 0; kc < a.kc1; kc++) tmaLoad2d(smemU32(sA1 + (size_t)kc * PP_CHUNK), &tmA1, kc * 64, row, smemU32(a1Full));
        }
        for(int kc = first; kc < a.kc1; kc++) loadW(&tmW1, kc, gPart * a.NP, (uint32_t)a.NP * 128u);
        first = 0;
        if(++gPart == a.parts) { gPart = 0; gTile++; }
      };
      auto loadG2 = [&](int chunk) {
        for(int i = 0; i < a.pieces; i++) loadW(&tmW2, chunk, i * a.N2, (uint32_t)a.N2 * 128u);
      };
      // the first weights do not wait for the kernels before this one
      if(nTiles > 0)
        for(; first < min(a.kc1, a.numB); first++) loadW(&tmW1, first, 0, (uint32_t)a.NP * 128u);
      gridDepWait();
      for(int i = 0; i < a.numD1; i++) loadG1();
      for(int t = 0; t < nTiles && ok; t++) {
        for(int p = 0; p < a.parts && ok; p++) {
          loadG2(p * cpp);
          loadG1();
          for(int c = 1; c < cpp; c++) loadG2(p * cpp + c);
        }
      }
      if(!ok && !*abortFlag) { *abortFlag = 1; atomicCAS(a.status, 0, PP_ERR_PRODUCER); }
    }
  }
  else if(warp == 1) {
    // ---------------- MMA issuer ----------------
    if(electOne()) {
      const uint32_t descHi = (uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29);
      const uint32_t a1Lo = ((smemU32(sA1) & 0x3FFFFu) >> 4) | (1u << 16);
      const uint32_t bLo = ((smemU32(sB) & 0x3FFFFu) >> 4) | (1u << 16);
      const uint32_t chunk16 = (uint32_t)PP_CHUNK >> 4, bSlot16 = (uint32_t)a.bSlot >> 4;
      uint32_t sb = 0, ph = 0;
      bool ok = true;
      // the four MMAs of a 64-channel step with the next weight slot
      // (A from shared memory: descriptor; from tensor memory: column, 8 per 16 channels)
      auto step = [&](auto fromTmem, uint32_t d, uint32_t aT, uint32_t idesc, uint32_t accumulate) {
        if(!mbarWait(smemU32(&bFull[sb]), ph, abortFlag)) { ok = false; return; }
        tcFenceAfter();
        const uint32_t bT = bLo + sb * bSlot16;
#pragma unroll
        for(int k = 0; k < 4; k++) {
          if(decltype(fromTmem)::value) ummaTmemA(d, aT + 8 * k, bT + 2 * k, descHi, idesc, k == 0 ? accumulate : 1u);
          else ummaLoHi(d, aT + 2 * k, bT + 2 * k, descHi, idesc, k == 0 ? accumulate : 1u);
        }
        ummaCommit(smemU32(&bEmpty[sb]));
        if(++sb == (uint32_t)a.numB) { sb = 0; ph ^= 1u; }
      };
      int gTile = 0, gPart = 0;  // the next part of GEMM1
      uint32_t G1n = 0;          // parts of GEMM1 issued so far: accumulator G1n & 1 and its barrier phases
      auto g1 = [&]() {
        if(gTile >= nTiles || !ok) return;
        if(gPart == 0 && !mbarWait(smemU32(a1Full), (uint32_t)gTile & 1u, abortFlag)) { ok = false; return; }
        const uint32_t buf = a.numD1 == 2 ? G1n & 1u : 0u, use = a.numD1 == 2 ? G1n >> 1 : G1n;
        PPT(true, G1n * 4);
        if(!mbarWait(smemU32(&d1Empty[buf]), (use & 1u) ^ 1u, abortFlag)) { ok = false; return; }
        PPT(true, G1n * 4 + 1);
        for(int kc = 0; kc < a.kc1 && ok; kc++) step(std::false_type{}, tmemBase + buf * (uint32_t)a.NP, a1Lo + (uint32_t)kc * chunk16, a.idesc1, kc > 0 ? 1u : 0u);
        if(!ok) return;
        ummaCommit(smemU32(&d1Full[buf]));
        PPT(true, G1n * 4 + 2);
        G1n++;
        if(++gPart == a.parts) { gPart = 0; gTile++; ummaCommit(smemU32(a1Empty)); }
      };
      uint32_t A = 0, phA = 0, GC = 0;  // operand chunk to multiply next, its phase, chunks issued so far
      (void)GC;
      auto g2 = [&](int tile, bool firstOfTile, bool lastOfTile) {
        if(!ok) return;
        PPT(true, 256 + GC * 4);
        if(!mbarWait(smemU32(&a2Full[A]), phA, abortFlag)) { ok = false; return; }
        PPT(true, 256 + GC * 4 + 1);
        if(firstOfTile && !mbarWait(smemU32(d2Empty), ((uint32_t)tile & 1u) ^ 1u, abortFlag)) { ok = false; return; }
        for(int i = 0; i < a.pieces && ok; i++)
          step(std::true_type{}, tmemBase + d2Col + (uint32_t)(i * a.N2), tmemBase + a2Col + A * PP_A2_COLS, a.idesc2, firstOfTile ? 0u : 1u);
        if(!ok) return;
        ummaCommit(smemU32(&a2Empty[A]));
        if(lastOfTile) ummaCommit(smemU32(d2Full));
        PPT(true, 256 + GC * 4 + 2);
        GC++;
        if(++A == (uint32_t)PP_NUM_A2) { A = 0; phA ^= 1u; }
      };
      for(int i = 0; i < a.numD1; i++) g1();
      for(int t = 0; t < nTiles && ok; t++) {
        for(int p = 0; p < a.parts && ok; p++) {
          g2(t, p == 0, p + 1 == a.parts && cpp == 1);
          g1();
          for(int c = 1; c < cpp; c++) g2(t, false, p + 1 == a.parts && c + 1 == cpp);
        }
      }
      if(!ok && !*abortFlag) { *abortFlag = 1; atomicCAS(a.status, 0, PP_ERR_MMA); }
    }
  }
  else {
    // ---------------- Epilogue: TMEM lane quarter = warp % 4 ----------------
    const int q = warp & 3;
    const int cg = (warp - 2) >> 2;
    const int ew = warp - 2;
    uint8_t* sR = sStage + (size_t)ew * PP_STAGE * PP_UNIT;  // residual units, from which the updated stream leaves again
    uint8_t* sO = sR + 2 * PP_UNIT;
    uint64_t* myRes = resFull + ew * 2;
    const int U1 = a.Ct / 32, U2 = a.Cn / 32;  // units of the two epilogues
    const int mine = (U1 - cg + PP_CG - 1) / PP_CG;  // of the first one, per tile
    const int sw64 = (lane >> 1) & 3;  // 64-byte swizzle of the staging units
    bool alive = true;
    uint32_t rs = 0;   // residual units consumed so far: ring slot rs % 2, phase (rs / 2) & 1
    // the sequence of this warp's residual units: (tile, unit)
    int nt = 0, nu = cg;
    auto fetchNext = [&](uint32_t slotSeq) {
      // an elected thread: request the residual of the next unit of this warp's sequence into ring slot slotSeq % 2
      if(nt >= nTiles || nu >= U1) return;
      const uint32_t b = slotSeq & 1u;
      mbarExpectTx(smemU32(&myRes[b]), (uint32_t)PP_UNIT);
      tmaLoad2d(smemU32(sR + (size_t)b * PP_UNIT), &tmS, nu * 32, ((int)blockIdx.x + nt * grid) * PP_BM + q * 32, smemU32(&myRes[b]));
      nu += PP_CG;
      if(nu >= U1) { nu = cg; nt++; }
    };
    uint32_t ppUnit = 0;
    (void)ppUnit;
    gridDepWait();
    if(electOne()) fetchNext(0);
    __syncwarp();
    bool on = false, onBefore = false;  // this row is a board point: in this tile, in the tile before
    for(int t = 0; t <= nTiles && alive; t++) {
      const int m0 = ((int)blockIdx.x + t * grid) * PP_BM;
      onBefore = on;
      if(t < nTiles) on = a.mask[m0 + q * 32 + lane] == 1.0f;
      for(int j = 0; alive && (j < mine || j < 2); j++) {
        if(j == 1 && t > 0) {
          // ---- second epilogue, of the tile before: the next block's mid stream and its activated form ----
          PPT(threadIdx.x == 64, 512 + ppUnit * 6);
          bool ok = mbarWait(smemU32(d2Full), (uint32_t)(t - 1) & 1u, abortFlag);
          if(!__all_sync(0xffffffffu, ok)) { alive = false; break; }
          PPT(threadIdx.x == 64, 512 + ppUnit * 6 + 1);
          tcFenceAfter();
          for(int u = cg; u < U2; u += PP_CG) {
            uint32_t r[32];
            tmemLd32(tmemBase + d2Col + (uint32_t)(u * 32) + ((uint32_t)(q * 32) << 16), r);
            tmemLdWait();
            if(u + PP_CG >= U2) {
              // this warp's last load: the next tile's GEMM2 may start
              tcFenceBefore();
              __syncwarp();
              if(electOne()) mbarArrive(smemU32(d2Empty));
            }
            const int c = u * 32;
            float2 v[16];
#pragma unroll
            for(int k = 0; k < 16; k++) v[k] = make_float2(__uint_as_float(r[2 * k]), __uint_as_float(r[2 * k + 1]));
            uint32_t rawP[16], actP[16];
#pragma unroll
            for(int k = 0; k < 16; k++) rawP[k] = Pack2<T>::pack(v[k].x, v[k].y);
            {
              const float4* sp = reinterpret_cast<const float4*>(a.scale2 + c);
              const float4* bp = reinterpret_cast<const float4*>(a.bias2 + c);
#pragma unroll
              for(int hh = 0; hh < 2; hh++) {
                float2 x[8];
#pragma unroll
                for(int k = 0; k < 4; k++) {
                  const float4 s4 = __ldg(sp + 4 * hh + k), b4 = __ldg(bp + 4 * hh + k);
                  x[2 * k] = __ffma2_rn(v[8 * hh + 2 * k], make_float2(s4.x, s4.y), make_float2(b4.x, b4.y));
                  x[2 * k + 1] = __ffma2_rn(v[8 * hh + 2 * k + 1], make_float2(s4.z, s4.w), make_float2(b4.z, b4.w));
                }
                actStaged2<ACT, 8>(x);
#pragma unroll
                for(int k = 0; k < 8; k++) actP[8 * hh + k] = onBefore ? Pack2<T>::pack(x[k].x, x[k].y) : 0u;
              }
            }
            // staging: the ring slot that does not hold the residual requested ahead, and the third unit
            if(electOne()) bulkWaitRead0();
            __syncwarp();
            uint8_t* sRaw = sR + (size_t)((rs + 1u) & 1u) * PP_UNIT;
#pragma unroll
            for(int jj = 0; jj < 4; jj++) {
              *reinterpret_cast<uint4*>(sRaw + lane * 64 + ((jj ^ sw64) << 4)) = make_uint4(rawP[4 * jj], rawP[4 * jj + 1], rawP[4 * jj + 2], rawP[4 * jj + 3]);
              *reinterpret_cast<uint4*>(sO + lane * 64 + ((jj ^ sw64) << 4)) = make_uint4(actP[4 * jj], actP[4 * jj + 1], actP[4 * jj + 2], actP[4 * jj + 3]);
            }
            fenceProxyAsync();
            __syncwarp();
            if(electOne()) {
              const int row = m0 - grid * PP_BM + q * 32;
              tmaStore2d(&tmRaw2, smemU32(sRaw), c, row);
              tmaStore2d(&tmAct2, smemU32(sO), c, row);
              bulkCommit();
            }
          }
          if(cg >= U2) {
            __syncwarp();
            if(electOne()) mbarArrive(smemU32(d2Empty));
          }
          PPT(threadIdx.x == 64, 512 + ppUnit * 6 + 4);
          ppUnit++;
        }
        if(t == nTiles || j >= mine) continue;
        // ---- first epilogue: unit u of GEMM1 ----
        const int u = cg + PP_CG * j;
        const uint32_t G = (uint32_t)(t * a.parts + u / UP);  // its part, counted over the CTA's tiles
        const uint32_t buf = a.numD1 == 2 ? G & 1u : 0u, use = a.numD1 == 2 ? G >> 1 : G;
        PPT(threadIdx.x == 64, 512 + ppUnit * 6);
        bool ok = mbarWait(smemU32(&d1Full[buf]), use & 1u, abortFlag);
        if(!__all_sync(0xffffffffu, ok)) { alive = false; break; }
        tcFenceAfter();
        const uint32_t slot = rs & 1u;
        uint32_t r[32];
        tmemLd32(tmemBase + buf * (uint32_t)a.NP + (uint32_t)((u % UP) * 32) + ((uint32_t)(q * 32) << 16), r);
        // the slot of the unit after this one held this warp's store before last: it must have been read; then the
        // next residual is requested, so that its latency hides behind this unit's arithmetic
        if(electOne()) { bulkWaitRead0(); fetchNext(rs + 1u); }
        __syncwarp();
        bool landed = mbarWait(smemU32(&myRes[slot]), (rs >> 1) & 1u, abortFlag);
        if(!__all_sync(0xffffffffu, landed)) { alive = false; break; }
        tmemLdWait();
        PPT(threadIdx.x == 64, 512 + ppUnit * 6 + 1);
        tcFenceBefore();
        __syncwarp();
        if(electOne()) mbarArrive(smemU32(&d1Empty[buf]));
        const int c = u * 32;  // first output channel of this unit
        float2 v[16];
#pragma unroll
        for(int k = 0; k < 16; k++) v[k] = make_float2(__uint_as_float(r[2 * k]), __uint_as_float(r[2 * k + 1]));
        uint8_t* rRow = sR + (size_t)slot * PP_UNIT + lane * 64;
#pragma unroll
        for(int jj = 0; jj < 4; jj++) {
          const uint4 x = *reinterpret_cast<const uint4*>(rRow + ((jj ^ sw64) << 4));
          const uint32_t xu[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for(int k = 0; k < 4; k++) v[4 * jj + k] = Pack2<T>::addTo(xu[k], v[4 * jj + k]);
        }
        // updated stream: in place of the residual, then out by TMA
#pragma unroll
        for(int jj = 0; jj < 4; jj++) {
          uint4 o;
          o.x = Pack2<T>::pack(v[4 * jj].x, v[4 * jj].y); o.y = Pack2<T>::pack(v[4 * jj + 1].x, v[4 * jj + 1].y);
          o.z = Pack2<T>::pack(v[4 * jj + 2].x, v[4 * jj + 2].y); o.w = Pack2<T>::pack(v[4 * jj + 3].x, v[4 * jj + 3].y);
          *reinterpret_cast<uint4*>(rRow + ((jj ^ sw64) << 4)) = o;
        }
        // norm + activation + mask of the layer between the two convolutions
        uint32_t actP[16];
        {
          const float4* sp = reinterpret_cast<const float4*>(a.scale1 + c);
          const float4* bp = reinterpret_cast<const float4*>(a.bias1 + c);
#pragma unroll
          for(int hh = 0; hh < 2; hh++) {
            float2 x[8];
#pragma unroll
            for(int k = 0; k < 4; k++) {
              const float4 s4 = __ldg(sp + 4 * hh + k), b4 = __ldg(bp + 4 * hh + k);
              x[2 * k] = __ffma2_rn(v[8 * hh + 2 * k], make_float2(s4.x, s4.y), make_float2(b4.x, b4.y));
              x[2 * k + 1] = __ffma2_rn(v[8 * hh + 2 * k + 1], make_float2(s4.z, s4.w), make_float2(b4.z, b4.w));
            }
            actStaged2<ACT, 8>(x);
#pragma unroll
            for(int k = 0; k < 8; k++) actP[8 * hh + k] = on ? Pack2<T>::pack(x[k].x, x[k].y) : 0u;
          }
        }
        // K chunk of GEMM2 this unit belongs to: its columns are free once the chunk PP_NUM_A2 before it has been multiplied
        const uint32_t gc = (uint32_t)(t * (U1 / 2) + u / 2), round = gc / (uint32_t)PP_NUM_A2, abuf = gc % (uint32_t)PP_NUM_A2;
        PPT(threadIdx.x == 64, 512 + ppUnit * 6 + 2);
        {
          bool e = mbarWait(smemU32(&a2Empty[abuf]), (round & 1u) ^ 1u, abortFlag);
          if(!__all_sync(0xffffffffu, e)) { alive = false; break; }
        }
        PPT(threadIdx.x == 64, 512 + ppUnit * 6 + 3);
        tcFenceAfter();
        tmemSt16(tmemBase + a2Col + abuf * PP_A2_COLS + (uint32_t)((u & 1) * 16) + ((uint32_t)(q * 32) << 16), actP);
        tmemStWait();
        tcFenceBefore();
        fenceProxyAsync();
        __syncwarp();
        if(electOne()) {
          mbarArrive(smemU32(&a2Full[abuf]));
          tmaStore2d(&tmS, smemU32(sR + (size_t)slot * PP_UNIT), c, m0 + q * 32);
          bulkCommit();
        }
        PPT(threadIdx.x == 64, 512 + ppUnit * 6 + 4);
        ppUnit++;
        rs++;
      }
    }
    if(!alive && lane == 0 && !*abortFlag) { *abortFlag = 1; atomicCAS(a.status, 0, PP_ERR_EPILOGUE); }
    if(electOne()) bulkWaitAll();
  }

  // ---------------- common exit ----------------
  tcFenceBefore();
  __syncthreads();
  if(*abortFlag && threadIdx.x == 0 && !bad) {
    const uint64_t t0 = globalTimerNs();
    while(globalTimerNs() - t0 < 2000000ull) { __nanosleep(1000); }
  }
  __syncthreads();
  if(warp == 1) {
    tcFenceAfter();
    tmemDealloc(tmemBase, 512);
  }
}

// ---------------------------------------------------------------------------------------------
// Host side

typedef CUresult (*EncodeTiledFn2)(
  CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn2 encodeFn() {
  static EncodeTiledFn2 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, []() {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn2>(p);
  });
  return fn;
}

static bool enc2d(CUtensorMap* tm, int dt, const void* base, uint64_t inner, uint64_t outer, uint64_t strideBytes, uint32_t boxInner, uint32_t boxOuter, CUtensorMapSwizzle sw) {
  EncodeTiledFn2 fn = encodeFn();
  if(!fn) return false;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {strideBytes};
  cuuint32_t box[2] = {boxInner, boxOuter};
  cuuint32_t estr[2] = {1, 1};
  return fn(tm, dt == DT_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct ConvPostPrePlan {
  CUtensorMap tmA1, tmW1, tmW2, tmS, tmRaw2, tmAct2;
  PostPreArgs a;
  int dt, act, numSMs;
  size_t smemBytes;
};

typedef void (*PostPreKernelFn)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, PostPreArgs);
template <typename T>
static PostPreKernelFn postPreKernelForT(int act) {
  switch(act) {
    case KB_ACT_RELU: return convPostPreKernel<T, KB_ACT_RELU>;
    case KB_ACT_MISH: return convPostPreKernel<T, KB_ACT_MISH>;
    case KB_ACT_SILU: return convPostPreKernel<T, KB_ACT_SILU>;
    case KB_ACT_MISH_SCALE8: return convPostPreKernel<T, KB_ACT_MISH_SCALE8>;
    default: return convPostPreKernel<T, KB_ACT_IDENTITY>;
  }
}

// Which widths: all that fit.  Whole nets of 18 blocks, fp16, in seconds of steady load (power-limited), two launches / fused in us, at 128
// and at 256 boards: 384 channels with 192 inside 3311 / 3114, 6608 / 6243; 320 with 192 3228 / 3096, 6473 / 6284; 256 with 192 3112 / 2982,
// 6244 / 6043; 384 with 256 5128 / 5003, 9783 / 9599; 256 with 256 4878 / 4746, 9340 / 9101; 512 with 192 3620 / 3425, 7204 / 6908; 192 with
// 256 4725 / 4621, 9053 / 8915; b28 (512 with 256) 8236 / 7986, 15706 / 15402, at 24 and 48 boards 2451 / 2457, 4521 / 4574.  Single calls behind
// idle gaps gain 1 to 6 % at 100 to 256 boards.  Narrow pairs gain more (six blocks at 256 boards: 256 with 128 1166 / 1100, 128 with 64
// 697 / 642, 64 with 64 624 / 578).  The exception found: bursts of some tens of milliseconds of six-block nets with unscaled random weights,
// in which pairs with 192 and more channels inside were up to 8 % slower fused at 256 boards.
bool convPostPreEligible(int dt, int Cm, int Ct, int Cn) {
  if(dt != DT_F16 && dt != DT_BF16) return false;
  if((Cm % 64) != 0 || (Ct % 64) != 0 || (Cn % 32) != 0 || Cn > 256 || Cn < 64) return false;
  const int NP = postPrePartWidth(Ct, Cn);
  if(NP == 0 || postPrePieces(Ct, Cn) == 0) return false;
  // shared memory: A1, the staging units of the epilogue warps, three weight slots
  const long fixed = (long)(Cm / 64) * PP_CHUNK + (long)PP_EPI_WARPS * PP_STAGE * PP_UNIT + PP_FIXED;
  return 227L * 1024 - fixed >= 3L * NP * 128;
}

// in1: [rows][Cm] activated mid tensor; w1: [Ct][Cm]; stream: [rows][Ct] residual stream, updated in place; w2: [Cn][Ct];
// raw2 / act2: [rows][Cn].  All tensors dense (row stride = channel count) and 16-byte aligned.
ConvPostPrePlan* convPostPreCreate(
  int dt, const void* in1, int Cm, const void* w1, void* stream, int Ct, const float* scale1, const float* bias1, int act1,
  const void* w2, void* raw2, void* act2, int Cn, const float* scale2, const float* bias2, int act2code, const float* mask,
  int rowsPadMax) {
  if(!convPostPreEligible(dt, Cm, Ct, Cn) || act1 != act2code) return nullptr;
  ConvPostPrePlan* p = new ConvPostPrePlan();
  std::memset(&p->a, 0, sizeof(p->a));
  p->dt = dt; p->act = act1;
  PostPreArgs& a = p->a;
  a.Cm = Cm; a.Ct = Ct; a.Cn = Cn; a.kc1 = Cm / 64;
  a.NP = postPrePartWidth(Ct, Cn); a.parts = Ct / a.NP;
  a.pieces = postPrePieces(Ct, Cn); a.N2 = Cn / a.pieces;
  a.numD1 = postPreAccumulators(a.NP, Cn);
  a.bSlot = a.NP * 128;
  const long fixed = (long)a.kc1 * PP_CHUNK + (long)PP_EPI_WARPS * PP_STAGE * PP_UNIT + PP_FIXED;
  a.numB = (int)std::min<long>((227L * 1024 - fixed) / a.bSlot, PP_MAX_SLOTS);
  p->smemBytes = (size_t)fixed + (size_t)a.numB * a.bSlot;
  const uint32_t fmt = dt == DT_F16 ? 0u : 1u;
  a.idesc1 = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(a.NP >> 3) << 17) | ((uint32_t)(PP_BM >> 4) << 24);
  a.idesc2 = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(a.N2 >> 3) << 17) | ((uint32_t)(PP_BM >> 4) << 24);
  a.scale1 = scale1; a.bias1 = bias1; a.scale2 = scale2; a.bias2 = bias2; a.mask = mask;
  const uint64_t rows = (uint64_t)rowsPadMax;
  bool ok = enc2d(&p->tmA1, dt, in1, (uint64_t)Cm, rows, (uint64_t)Cm * 2, 64, PP_BM, CU_TENSOR_MAP_SWIZZLE_128B) &&
            enc2d(&p->tmW1, dt, w1, (uint64_t)Cm, (uint64_t)Ct, (uint64_t)Cm * 2, 64, (uint32_t)a.NP, CU_TENSOR_MAP_SWIZZLE_128B) &&
            enc2d(&p->tmW2, dt, w2, (uint64_t)Ct, (uint64_t)Cn, (uint64_t)Ct * 2, 64, (uint32_t)a.N2, CU_TENSOR_MAP_SWIZZLE_128B) &&
            enc2d(&p->tmS, dt, stream, (uint64_t)Ct, rows, (uint64_t)Ct * 2, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B) &&
            enc2d(&p->tmRaw2, dt, raw2, (uint64_t)Cn, rows, (uint64_t)Cn * 2, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B) &&
            enc2d(&p->tmAct2, dt, act2, (uint64_t)Cn, rows, (uint64_t)Cn * 2, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B);
  if(!ok) { delete p; return nullptr; }
  int dev = 0, sms = 148;
  if(cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  p->numSMs = sms;
  return p;
}

void convPostPreDestroy(ConvPostPrePlan* p) { delete p; }

cudaError_t launchConvPostPre(cudaStream_t st, const ConvPostPrePlan* p, Geom g, int* statusWord) {
  PostPreArgs a = p->a;
  a.g = g;
  a.status = statusWord;
  const int numTiles = g.rowsPad / PP_BM;
  const int grid = numTiles < p->numSMs ? numTiles : p->numSMs;
  PostPreKernelFn fn = p->dt == DT_F16 ? postPreKernelForT<__half>(p->act) : postPreKernelForT<__nv_bfloat16>(p->act);
  {
    static std::mutex mu;
    static std::vector<std::pair<const void*, int>> done;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    const std::pair<const void*, int> key((const void*)fn, dev);
    if(std::find(done.begin(), done.end(), key) == done.end()) {
      cudaError_t e = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
      if(e != cudaSuccess) return e;
      done.push_back(key);
    }
  }
  static const bool usePdl = getenv("KB_NO_PDL") == nullptr;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid); cfg.blockDim = dim3(PP_THREADS); cfg.dynamicSmemBytes = p->smemBytes; cfg.stream = st;
  cudaLaunchAttribute attr[1];
  int numAttrs = 0;
  if(usePdl) {
    attr[numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[numAttrs].val.programmaticStreamSerializationAllowed = 1;
    numAttrs++;
  }
  cfg.attrs = attr; cfg.numAttrs = numAttrs;
  return cudaLaunchKernelEx(&cfg, fn, p->tmA1, p->tmW1, p->tmW2, p->tmS, p->tmRaw2, p->tmAct2, a);
}

}  // namespace kb

#ifdef KB_TC_TRACE
extern "C" int kb_debug_trace_pp(long long* out, int n) { return (int)cudaMemcpyFromSymbol(out, kb::g_ppTrace, sizeof(long long) * n); }
#endif
