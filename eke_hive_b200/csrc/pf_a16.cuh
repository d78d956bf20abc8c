// Grouped GEMM of the prefill operator with bf16 activations (W4A16, the reference's default prefill arithmetic,
// engine/src/qwen/fn_moe_pf.cu:118-437) on the 5th-generation tensor cores: tcgen05.mma kind::f16, bf16 × bf16 → fp32 in tensor memory.
//
// The NVFP4 weights are the A operand (M = 128 rows of the record's matrix), the activation rows of one expert's pairs the B operand
// (N ≤ 256 pairs, N a multiple of 16 chosen per tile), so one dequantised weight value serves up to 256 multiply-adds and the
// accumulator's lanes are weight rows — the epilogue thread of a lane owns one output row of the expert, as in the decode kernels.
// Dequantisation: e2m1 → bf16 by byte permutes, × the e4m3 block scale as bf16 — the product has ≤ 6 significant bits, exact in bf16 —
// written into the K-major 128-byte-swizzle operand tile by sixteen warps; every product of the MMA is therefore the exact product of
// the decode operators, sums are fp32.  Rounding points after the sums are the reference's (g, u → bf16 after the
// global scale, y → bf16, down → bf16 before the routing weight).
//
// A work item is 256 weight rows (two A tiles of 128) × one tile of pairs; with tiles of 256 pairs the two accumulators fill the CTA's
// tensor memory and the MMAs of the next item wait for the epilogue.  Per 64 k values an item moves 32 KB of activations and 8 KB of codes from L2 into
// shared memory (with one A tile per item the activation stream alone ran into what the SMs can pull out of L2).
//
// Per CTA (persistent, one per SM, 28 warps): warp 9 (one thread) streams by TMA the raw code boxes of the weights (128 bytes × 64
// rows, 256 k values per row, through the call's own weight maps, wmap.cuh), warp 26 the activation boxes (64 values × 64 rows of
// bf16) of the tile; warps 10-25 (eight per A tile) turn a raw box into four operand tiles, fetching their row's block scales from
// global memory a raw box ahead; warp 8 and warp 27 (one thread each) issue the MMAs of an A tile (128 × N × 16, four a step); warps 0-3 and 4-7 run
// the epilogues of the two accumulators.  Gate/up: an A tile holds 64 gate and 64 up rows arranged so that lanes l and l + 16 of a
// warp hold the gate and the up value of the same row of I — SwiGLU needs one exchange.  Every wait is bounded; a barrier gets one
// arrival per warp, not per thread (arrivals on one barrier are taken one after the other).
#pragma once
#include "wmap.cuh"

namespace hb {

// Shared memory and tensor memory by the pairs a tile may have (MMA N).  An expert's run decides what bounds the kernel: with 256 pairs the
// tensor pipe (an MMA of M = 128 takes max(47, N / 2) clocks, measured) and the activation stream; with a few dozen pairs — a prompt of a
// couple of thousand tokens over 512 experts — the weights: an activation stage is then a quarter of the size, so there is room for a
// deeper ring of raw codes (they come from HBM), and the sums leave room in tensor memory: the dequantised weights go there, as the A
// operand, without touching shared memory (writing them to it and reading them back was what bounded small tiles: 1050 of 1600 clocks a
// step with the MMAs waiting on it), and with ≤ 64 pairs the sums of two items, so the MMAs need not wait for the epilogue.  Measured for
// 1999 rows of 512 experts (hidden 2048, intermediate 512, top-10: 39 pairs an expert), tiles of ≤ 256 in shared memory → ≤ 64 in tensor
// memory, the issuing threads elected, two steps a hand-over: gate/up 440 → 240 µs, down 260 → 145 µs.  What bounds it now is the
// dequantisation (640 of 1030 clocks a step of 64 k values; the MMAs are busy for half of it).
template <int BN_>
struct A16Cfg {
  static constexpr int BN = BN_;                                     // pairs of a tile, at most
  static constexpr bool AT = BN <= 128;                              // the dequantised weights sit in tensor memory (else: swizzled tiles in shared memory)
  static constexpr int KA = AT ? 2 : 1;                              // steps of 64 k values a weight stage holds: the hand-over of a stage costs as much as its values
  static constexpr int STA = 2;                                      // operand rings: dequantised weight stages, activation tiles
  static constexpr int STB = BN <= 64 ? 8 : BN <= 128 ? 5 : 3;
  static constexpr int RAWS = AT ? 4 : 2;                            // raw code slots (256 k values each)
  static constexpr int NACC = BN <= 64 ? 2 : 1;                      // accumulator buffers of 2·BN columns
  static constexpr int A1 = 128 * 128;                               // one A tile: 128 rows × 64 bf16; raw codes of 256 k values take as much
  static constexpr int A = AT ? 0 : 2 * A1;                          // both A tiles of a step in shared memory
  static constexpr int B = BN * 128;                                 // BN rows × 64 bf16
  static constexpr int RAW = 2 * A1;                                 // raw codes of both A tiles: 128 rows × 128 bytes each (256 k values per row)
  static constexpr int ACOL = NACC * 2 * BN;                         // tensor memory: accumulators, then stages of two A tiles of 32 columns (bf16 pairs)
  static constexpr int SMEM = 1024 + STA * A + STB * B + RAWS * RAW + 1024;
  static_assert(SMEM <= 227 * 1024 && ACOL + (AT ? STA * KA * 64 : 0) <= 512, "shared memory, tensor memory");
};
constexpr int A16_BN_MIN = 64;
constexpr int A16_THREADS = 28 * 32;            // warps 0-3 and 4-7 epilogues of the two A tiles, 8 and 27 their MMAs, 9 raw codes, 10-17 and 18-25 dequantisation, 26 activations
constexpr int A16_W_MMA = 8, A16_W_TMA = 9, A16_W_DQ0 = 10, A16_W_ACT = 26, A16_W_MMA1 = 27, A16_DQ_THREADS = 512;
constexpr int A16_TMEM_COLS = 512;

struct A16Args {
  const TileRef* tiles; const int* n_tiles;     // tiles of ≤ BN consecutive slots of one expert's run of the sorted pairs
  const int* perm;                              // pair of a slot (the down pass writes its rows by pair)
  const uint8_t* const* tab;                    // expert records of the layer
  int down;                                     // 0: gate/up (out = y bf16 [slot, I]); 1: down (out = bf16 [pair, H])
  int K, n_out;                                 // inner dimension (H | I), output rows per expert (I | H)
  uint32_t off_w, off_s0, off_s1, off_g;        // record offsets: first matrix, scales of the matrix of lanes 0-15 / 16-31 of a warp (gate / up; down:
                                                // the same matrix twice), global scales
  int row2;                                     // matrix rows between the two 64-row boxes of an A tile
  WmArgs wm;                                    // the weight maps of this pass
  float limit;
  __nv_bfloat16* out;
  uint32_t* err;
};

__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

__device__ __forceinline__ void tc_mma_f16_at(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {   // A in tensor memory
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

// two f16 values (exactly representable in bf16) → bf16x2, element order kept
__device__ __forceinline__ uint32_t f16x2_to_bf16x2(uint32_t h2) {
  const __half2 h = *reinterpret_cast<const __half2*>(&h2);
  const float2 f = __half22float2(h);
  const __nv_bfloat162 b = __floats2bfloat162_rn(f.x, f.y);
  return *reinterpret_cast<const uint32_t*>(&b);
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ uint32_t bmul2_u32(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// Eight e2m1 codes (one word, element 0 in the low nibble) → eight bf16 values times the block scale `sv` (bf16x2, both halves the same), as
// four bf16x2 words in element order — on the integer pipe: the conversion unit is too slow for one conversion per element.  The bf16
// pattern of a magnitude code m is looked up bytewise with byte permutes (high bytes 00 3F 3F 3F 40 40 40 40, low bytes 00 00 80 C0 00 40
// 80 C0 for 0, .5, 1, 1.5, 2, 3, 4, 6), the sign bits come from a permute in sign-replication mode; the product of such a value and an
// e4m3 scale has at most 6 significant bits: exact in bf16.
__device__ __forceinline__ uint4 a16_dequant8(uint32_t w, uint32_t sv) {
  const uint32_t wa = w << 4;
  uint32_t o[4];
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const uint32_t sel = (half ? (w >> 16) : w) & 0x7777u;
    const uint32_t hi = prmt(0x3F3F3F00u, 0x40404040u, sel), lo = prmt(0xC0800000u, 0xC0804000u, sel);
    const uint32_t sg = prmt(wa, w, half ? 0xFBEAu : 0xD9C8u);            // byte i = 0xFF where element i is negative
    const uint32_t hs = hi | (sg & 0x80808080u);
    o[2 * half] = bmul2_u32(prmt(lo, hs, 0x5140u), sv);
    o[2 * half + 1] = bmul2_u32(prmt(lo, hs, 0x7362u), sv);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// The slot-ordered copy of the activation rows: row `slot` = x[perm[slot] / K].  One CTA per slot at a time; the first CTA stamps the weight
// maps of both GEMMs instead (the last one of a grid larger than the chip would start when the others are nearly done).
__global__ void __launch_bounds__(256) a16_gather_kernel(const __nv_bfloat16* __restrict__ x, const int* __restrict__ perm, const int* __restrict__ n_slots, int K,
                                                         int H, __nv_bfloat16* __restrict__ out, const __grid_constant__ WmStamp wm) {
  if (blockIdx.x == 0) { wm_stamp(wm); return; }
  const int n = *n_slots;
  for (int s = blockIdx.x - 1; s < n; s += gridDim.x - 1) {
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(perm[s] / K) * H);
    uint4* dst = reinterpret_cast<uint4*>(out + (size_t)s * H);
    for (int i = threadIdx.x; i < H / 8; i += 256) dst[i] = __ldg(src + i);
  }
}

// Optional in-kernel timing (compile with -DHB_A16_TRACE): the roles of every CTA sum the clocks they spend in each kind of wait.
#ifdef HB_A16_TRACE
__device__ long long g_a16_trace[2 * 256 * 16];   // gate/up launch, down launch
#define A16_TIMED(acc, stmt) do { const long long t_ = clock64(); stmt; acc += clock64() - t_; } while (0)
#define A16_PUT(slot, v) g_a16_trace[(a.down * 256 + blockIdx.x) * 16 + (slot)] = (v)
#else
#define A16_TIMED(acc, stmt) do { stmt; } while (0)
#define A16_PUT(slot, v) do { } while (0)
#endif

template <int BN>
__global__ void __launch_bounds__(A16_THREADS, 1) a16_gemm_kernel(const A16Args a, const __grid_constant__ CUtensorMap tmB) {
  using C = A16Cfg<BN>;
  extern __shared__ uint8_t a16_raw[];
  const uint32_t raw0 = smem_u32(a16_raw), base = (raw0 + 1023u) & ~1023u;
  uint8_t* sm = a16_raw + (base - raw0);
  uint8_t* smA = sm;                                   // [STA][2 A tiles][16 KB]
  uint8_t* smB = smA + C::STA * C::A;                // [STB][BN rows × 128 bytes]
  uint8_t* smR = smB + C::STB * C::B;                // [RAWS][2 A tiles][16 KB] raw codes
  uint64_t* fullA = reinterpret_cast<uint64_t*>(smR + C::RAWS * C::RAW);
  uint64_t* emptyA = fullA + C::STA;
  uint64_t* fullB = emptyA + C::STA;
  uint64_t* emptyB = fullB + C::STB;
  uint64_t* fullR = emptyB + C::STB;
  uint64_t* emptyR = fullR + C::RAWS;
  uint64_t* acc_full = emptyR + C::RAWS;                // [NACC]
  uint64_t* acc_empty = acc_full + C::NACC;             // [NACC]
  uint64_t* mma_done = acc_empty + C::NACC;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);
  const int warp = warp_uniform(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STA; ++s) { mbar_init(&fullA[s], A16_DQ_THREADS / 32); mbar_init(&emptyA[s], 2); }   // one arrival per dequantisation warp; one commit per issuing thread
    for (int s = 0; s < C::STB; ++s) { mbar_init(&fullB[s], 1); mbar_init(&emptyB[s], 2); }
    for (int s = 0; s < C::RAWS; ++s) { mbar_init(&fullR[s], 1); mbar_init(&emptyR[s], A16_DQ_THREADS / 32); }
    for (int s = 0; s < C::NACC; ++s) { mbar_init(&acc_full[s], 2); mbar_init(&acc_empty[s], 8); }
    mbar_init(mma_done, 2);
    mbar_fence_init();
  }
  if (warp == A16_W_MMA) { tmem_alloc(tmem_slot, A16_TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const int arows = a.down ? 128 : 64;                        // matrix rows an A tile advances (gate/up: 64 of each matrix)
  const int nT = a.n_out / (2 * arows);                       // items per tile: two A tiles each
  const int n_items_all = *a.n_tiles * nT;
  const int nk = a.K >> 6;                                    // steps per item (a multiple of 4)

  if (warp == A16_W_TMA) {
    // ------------------------------------------------------------------------------------------------ raw code boxes: one thread
    if (elect_one()) {
      uint32_t rit = 0;
      bool ok = true;
      [[maybe_unused]] long long tw = 0, t0 = clock64();
      WmReader wm;
      wm.init(a.wm);
      for (int item = blockIdx.x; item < n_items_all && ok; item += gridDim.x) {
        const int ti = item / nT, t = item - ti * nT;
        const TileRef tl = a.tiles[ti];
        const uint8_t* rec = a.tab[tl.expert];
        WmBox box;
        if (!rec || !wm.locate(rec + a.off_w, box, a.err)) break;
        const int r0 = 2 * t * arows;
        for (int rs = 0; rs < nk / 4 && ok; ++rs, ++rit) {
          const uint32_t sl = rit % C::RAWS;
          A16_TIMED(tw, ok = mbar_wait(&emptyR[sl], ((rit / C::RAWS) & 1u) ^ 1u, a.err, 0x1u));
          if (!ok) break;
          const uint32_t rb = smem_u32(smR + sl * C::RAW);
          mbar_expect_tx(&fullR[sl], C::RAW);
#pragma unroll
          for (int uu = 0; uu < 2; ++uu) {
            wm.load(rb + uu * C::A1, box, rs * 128, r0 + uu * arows, &fullR[sl]);
            wm.load(rb + uu * C::A1 + C::A1 / 2, box, rs * 128, r0 + uu * arows + a.row2, &fullR[sl]);
          }
        }
      }
      A16_PUT(0, tw); A16_PUT(1, clock64() - t0);
    }
  } else if (warp == A16_W_ACT) {
    // ------------------------------------------------------------------------------------------------ activation boxes: one thread (apart from the codes, whose ring
    // must run ahead whatever the activation ring does)
    if (elect_one()) {
      uint32_t kit = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < n_items_all && ok; item += gridDim.x) {
        const TileRef tl = a.tiles[item / nT];
        const int nbox = (tl.rows + 63) >> 6;
        for (int kb = 0; kb < nk; ++kb, ++kit) {
          const uint32_t sb = kit % C::STB;
          if (!(ok = mbar_wait(&emptyB[sb], ((kit / C::STB) & 1u) ^ 1u, a.err, 0x2u))) break;
          const uint32_t bb = smem_u32(smB + sb * C::B);
          mbar_expect_tx(&fullB[sb], (uint32_t)nbox * 8192u);
          for (int i = 0; i < nbox; ++i) tma_load_2d(bb + i * 8192, &tmB, kb * 64, tl.slot0 + i * 64, &fullB[sb]);
        }
      }
    }
  } else if (warp >= A16_W_DQ0 && warp < A16_W_DQ0 + A16_DQ_THREADS / 32) {
    // ------------------------------------------------------------------------------------------------ dequantisation: thread (u, r, h) owns half a row
    // of A tile u in every step: A row r, k values [32 h, 32 h + 32) of the step's 64
    // (A in tensor memory: a warp reaches the lanes of quarter (warp index mod 4), a thread's lane there is its row)
    const int dt = threadIdx.x - A16_W_DQ0 * 32, u = dt >> 8, r = C::AT ? (warp & 3) * 32 + lane : (dt & 255) >> 1, h = C::AT ? (dt >> 7) & 1 : dt & 1;
    const uint32_t acol = tmem + ((uint32_t)((warp & 3) * 32) << 16) + C::ACOL + u * 32 + h * 16;
    int rr, srow; uint32_t soff;                               // raw row, row of the scale matrix inside the A tile, which scale matrix
    if (a.down) { rr = r; srow = r; soff = a.off_s0; }
    else {
      const int q = r >> 5, j = r & 31;
      rr = j < 16 ? 16 * q + j : 64 + 16 * q + (j - 16);
      srow = 16 * q + (j & 15);
      soff = j < 16 ? a.off_s0 : a.off_s1;
    }
    const int sbytes = a.K >> 4;                               // scale bytes per matrix row
    uint32_t rit = 0, kit = 0;
    [[maybe_unused]] int pend = -1;                            // weight stage that is stored but not announced yet
    bool ok = true;
    [[maybe_unused]] long long tw = 0, tc = 0, t0 = clock64(), tl0 = 0;
    for (int item = blockIdx.x; item < n_items_all && ok; item += gridDim.x) {
      const int ti = item / nT, t = item - ti * nT;
      const uint8_t* rec = a.tab[a.tiles[ti].expert];
      if (!rec) break;
      const uint8_t* srowp = rec + soff + (size_t)((2 * t + u) * arows + srow) * sbytes;
      uint4 sc = __ldg(reinterpret_cast<const uint4*>(srowp));
      for (int rs = 0; rs < nk / 4 && ok; ++rs, ++rit) {
        uint4 sc_next = sc;
        if (rs + 1 < nk / 4) sc_next = __ldg(reinterpret_cast<const uint4*>(srowp + (size_t)(rs + 1) * 16));
        const uint32_t sl = rit % C::RAWS;
        if (lane == 0) A16_TIMED(tw, ok = mbar_wait(&fullR[sl], (rit / C::RAWS) & 1u, a.err, 0x4u));
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) break;
        const uint8_t* rawrow = smR + sl * C::RAW + u * C::A1 + rr * 128;
        const uint32_t scw[4] = {sc.x, sc.y, sc.z, sc.w};
        auto dequant = [&](int kq, uint4& o0, uint4& o1, uint4& o2, uint4& o3) {                             // 32 codes of this thread's row
          const uint4 cw = *reinterpret_cast<const uint4*>(rawrow + (((kq * 2 + h) ^ (rr & 7)) << 4));
          const uint32_t s2 = (scw[kq] >> (16 * h)) & 0xffffu;                                              // the two block scales
          const uint32_t sh = f16x2_to_bf16x2(cvt_e4m3x2_f16x2(s2));
          const uint32_t slo = __byte_perm(sh, sh, 0x1010), shi = __byte_perm(sh, sh, 0x3232);             // (s0, s0), (s1, s1) as bf16
          o0 = a16_dequant8(cw.x, slo); o1 = a16_dequant8(cw.y, slo); o2 = a16_dequant8(cw.z, shi); o3 = a16_dequant8(cw.w, shi);
        };
        if constexpr (C::AT) {
          // two steps a stage; the stage before is announced after this one's first values are worked out (its stores have landed by then)
#pragma unroll
          for (int kq = 0; kq < 4; ++kq) {
#ifdef HB_A16_TRACE
            tl0 = clock64();
#endif
            uint4 o0, o1, o2, o3;
            dequant(kq, o0, o1, o2, o3);
#ifdef HB_A16_TRACE
            if (o0.x == 0x12345u && o3.w == 0x54321u) tc += 1;
            tc += clock64() - tl0;
#endif
            const uint32_t sa = kit % C::STA;
            if (kq % C::KA == 0) {
              if (pend >= 0) { tc_wait_st(); tc_fence_before(); __syncwarp(); if (lane == 0) mbar_arrive(&fullA[pend]); }
              A16_TIMED(tw, ok = mbar_wait(&emptyA[sa], ((kit / C::STA) & 1u) ^ 1u, a.err, 0x8u));
              ok = __all_sync(0xffffffffu, ok);
              pend = -1;
              if (!ok) break;
              tc_fence_after();
            }
            const uint32_t w16[16] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y, o1.z, o1.w, o2.x, o2.y, o2.z, o2.w, o3.x, o3.y, o3.z, o3.w};
            tc_st16(acol + (sa * C::KA + kq % C::KA) * 64, w16);
            if (kq % C::KA == C::KA - 1) { pend = (int)sa; ++kit; }
          }
        } else {
#pragma unroll
          for (int kq = 0; kq < 4; ++kq, ++kit) {
#ifdef HB_A16_TRACE
            tl0 = clock64();
#endif
            uint4 o0, o1, o2, o3;
            dequant(kq, o0, o1, o2, o3);
#ifdef HB_A16_TRACE
            if (o0.x == 0x12345u && o3.w == 0x54321u) tc += 1;            // keeps the values' computation in front of the clock read
            tc += clock64() - tl0;
#endif
            // one lane waits for the slot and one lane announces the warp's rows
            const uint32_t sa = kit % C::STA;
            if (lane == 0) A16_TIMED(tw, ok = mbar_wait(&emptyA[sa], ((kit / C::STA) & 1u) ^ 1u, a.err, 0x8u));
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) break;
            uint8_t* arow = smA + sa * C::A + u * C::A1 + r * 128;
            *reinterpret_cast<uint4*>(arow + (((h * 4 + 0) ^ (r & 7)) << 4)) = o0;
            *reinterpret_cast<uint4*>(arow + (((h * 4 + 1) ^ (r & 7)) << 4)) = o1;
            *reinterpret_cast<uint4*>(arow + (((h * 4 + 2) ^ (r & 7)) << 4)) = o2;
            *reinterpret_cast<uint4*>(arow + (((h * 4 + 3) ^ (r & 7)) << 4)) = o3;
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&fullA[sa]);
          }
        }
        if (!ok) break;
        __syncwarp();
        if (lane == 0) mbar_arrive(&emptyR[sl]);
        sc = sc_next;
      }
    }
    if (C::AT && pend >= 0) { tc_wait_st(); tc_fence_before(); __syncwarp(); if (lane == 0) mbar_arrive(&fullA[pend]); }
    if (dt == 0) { A16_PUT(2, tw); A16_PUT(3, clock64() - t0); A16_PUT(4, tc); }
  } else if (warp == A16_W_MMA || warp == A16_W_MMA1) {
    // ------------------------------------------------------------------------------------------------ MMA issue: one thread per A tile (one thread for both spent a
    // thousand clocks a step on its instructions alone, in the shadow of sixteen dequantising warps)
    const uint32_t uu = warp == A16_W_MMA ? 0u : 1u;
    if (elect_one()) {
      // few instructions a step: they run one at a time, between those of four other warps
      uint32_t n_it = 0, sa = 0, pa = 0, sb = 0, pb = 0;
      bool ok = true;
      [[maybe_unused]] long long twa = 0, twb = 0, twe = 0, t0 = clock64(), kit = 0;
      const uint64_t ad0 = tc_desc_sw128(base + uu * C::A1), bd0 = tc_desc_sw128(base + C::STA * C::A);
      for (int item = blockIdx.x; item < n_items_all && ok; item += gridDim.x, ++n_it) {
        const int rows = a.tiles[item / nT].rows;
        const uint32_t N = (uint32_t)((rows + 15) & ~15);
        // kind::f16: D fp32 (bit 4), A and B bf16 (format 1 at bits 7 and 10), both K-major, N / 8 at bit 17, M / 16 at bit 24
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) | ((128u >> 4) << 24);
        const uint32_t buf = n_it % C::NACC, acc = tmem + buf * (2 * BN) + uu * BN;
        if (n_it >= C::NACC) A16_TIMED(twe, ok = mbar_wait(&acc_empty[buf], (n_it / C::NACC - 1u) & 1u, a.err, 0x10u));   // the epilogue has read the buffer's previous sums
        if (!ok) break;
        tc_fence_after();
        uint32_t more = 0u;                                       // 0 for the item's first MMA: it overwrites the accumulator
        for (int kb = 0; kb < nk; ++kb) {
          A16_TIMED(twb, ok = mbar_wait(&fullB[sb], pb, a.err, 0x40u));
          if (!ok) break;
          const int ka = kb % C::KA;                                // step within the weight stage (nk is a multiple of four)
          if (ka == 0) A16_TIMED(twa, ok = mbar_wait(&fullA[sa], pa, a.err, 0x20u));
          if (!ok) break;
          tc_fence_after();
          const uint64_t ad = ad0 + sa * (uint32_t)(C::A >> 4), bd = bd0 + sb * (uint32_t)(C::B >> 4);
          const uint32_t at = tmem + C::ACOL + (sa * C::KA + ka) * 64 + uu * 32;
#pragma unroll
          for (uint32_t j = 0; j < 4; ++j) {
            if constexpr (C::AT) tc_mma_f16_at(acc, at + 8 * j, bd + 2 * j, idesc, j ? 1u : more);
            else tc_mma_f16(acc, ad + 2 * j, bd + 2 * j, idesc, j ? 1u : more);
          }
          more = 1u;
          tc_commit(&emptyB[sb]);
          if (ka == C::KA - 1) {
            tc_commit(&emptyA[sa]);
            if (++sa == C::STA) { sa = 0; pa ^= 1u; }
          }
          if (++sb == C::STB) { sb = 0; pb ^= 1u; }
#ifdef HB_A16_TRACE
          ++kit;
#endif
        }
        if (ok) tc_commit(&acc_full[buf]);
      }
      tc_commit(mma_done);
      mbar_wait(mma_done, 0, a.err, 0x80u);
      A16_PUT(5, twa); A16_PUT(6, twb); A16_PUT(7, twe); A16_PUT(8, clock64() - t0); A16_PUT(9, kit);
    }
  } else {
    // ------------------------------------------------------------------------------------------------ epilogues: warp 4 u + q reads lanes [32 q, 32 q + 32) of accumulator u
    const int u = warp >> 2, q = warp & 3, tl_ = threadIdx.x & 127;   // tl_ = row of the A tile
    bool ok = true;
    uint32_t n_it = 0;
    [[maybe_unused]] long long tw = 0, t0 = clock64(), tld = 0;
    for (int item = blockIdx.x; item < n_items_all && ok; item += gridDim.x, ++n_it) {
      const int ti = item / nT, t = item - ti * nT;
      const TileRef tl = a.tiles[ti];
      const uint8_t* rec = a.tab[tl.expert];
      if (!rec) break;
      const float gsc = __ldg(reinterpret_cast<const float*>(rec + a.off_g) + (a.down ? 2 : lane < 16 ? 0 : 1));
      // down: the pairs (output rows) of the tile's columns, lane l those of columns 32 i + l — fetched while the MMAs run and handed
      // round by shuffles below
      int my_pair[C::BN / 32];
#pragma unroll
      for (int i = 0; i < C::BN / 32; ++i) my_pair[i] = a.down && 32 * i + lane < tl.rows ? __ldg(a.perm + tl.slot0 + 32 * i + lane) : 0;
      const uint32_t buf = n_it % C::NACC;
      A16_TIMED(tw, ok = mbar_wait(&acc_full[buf], (n_it / C::NACC) & 1u, a.err, 0x100u));
      if (!ok) break;
      tc_fence_after();
      const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16) + buf * (2 * BN) + u * BN;
#pragma unroll
      for (int ci = 0; ci < C::BN / 32; ++ci) {
        const int c0 = 32 * ci;
        if (c0 >= tl.rows) break;
        uint32_t rg[32];
        A16_TIMED(tld, tc_ld32(trow + c0, rg); tc_wait_ld());
        if (a.down) {
          unsigned short* orow = reinterpret_cast<unsigned short*>(a.out) + (size_t)(2 * t + u) * 128 + tl_;
#pragma unroll
          for (int c = 0; c < 32; c += 2) {                     // two columns per conversion
            const __nv_bfloat162 b2 = __floats2bfloat162_rn(__uint_as_float(rg[c]) * gsc, __uint_as_float(rg[c + 1]) * gsc);
            const uint32_t bw = *reinterpret_cast<const uint32_t*>(&b2);
            const int p0 = __shfl_sync(0xffffffffu, my_pair[ci], c), p1 = __shfl_sync(0xffffffffu, my_pair[ci], c + 1);
            if (c0 + c < tl.rows) orow[(size_t)p0 * a.n_out] = (unsigned short)(bw & 0xffffu);
            if (c0 + c + 1 < tl.rows) orow[(size_t)p1 * a.n_out] = (unsigned short)(bw >> 16);
          }
        } else {
          // lanes 0-15 hold the gate values of 16 rows of I, lanes 16-31 the up values of the same rows.  Of a pair of columns the low
          // half-warp finishes the even one and the high half-warp the odd one: one exchange per pair, every lane computes
          const bool hi = lane >= 16;
          __nv_bfloat16* orow = a.out + (size_t)(tl.slot0 + c0 + (hi ? 1 : 0)) * a.n_out + (2 * t + u) * 64 + 16 * q + (lane & 15);
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            const float v0 = bf16r(__uint_as_float(rg[c]) * gsc), v1 = bf16r(__uint_as_float(rg[c + 1]) * gsc);
            const float got = __shfl_xor_sync(0xffffffffu, hi ? v0 : v1, 16);      // low lanes get u of the even column, high lanes g of the odd one
            float gv = hi ? got : v0, uv = hi ? v1 : got;
            if (a.limit > 0.f) { uv = fminf(fmaxf(uv, -a.limit), a.limit); gv = fminf(gv, a.limit); }
            // silu by the fast reciprocal (the decode kernels divide exactly; the difference is below the bf16 rounding that follows in
            // all but a few cases in a thousand — with tiles of more than 64 pairs the accumulators are not double-buffered, and the exact
            // division's instructions were the longest part of the time the MMAs wait for this epilogue)
            if (c0 + c + (hi ? 1 : 0) < tl.rows) orow[(size_t)c * a.n_out] = __float2bfloat16(__fdividef(gv, 1.f + __expf(-gv)) * uv);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
    if (threadIdx.x == 0) { A16_PUT(10, tw); A16_PUT(11, clock64() - t0); A16_PUT(12, tld); A16_PUT(13, (long long)n_it); }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == A16_W_MMA) { tc_fence_after(); tmem_dealloc(tmem, A16_TMEM_COLS); }
}

}  // namespace hb
