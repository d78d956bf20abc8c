// Dense decode GEMV for one weight matrix (or a gate/up pair), M ≤ 16 activation rows: NVFP4 and the 3-/2-bit group-64 formats
// (hb_qmat).  HBM-bound: every weight byte is read once, decoded in registers and fed to m16n8k16 tensor-core tiles whose 8
// columns are activation rows (fp32 accumulation); more than 8 rows take two tiles per decoded weight, not a second pass.
//
//   unit      a strip of 16 matrix rows (gate/up pair: 8 gate rows + the same 8 up rows, so that one lane ends with both halves of an
//             activation) over the CTA's columns.  ONE warp owns a unit: it streams the strip's 16 rows through its own cp.async ring,
//             256 columns a stage, and keeps the sums in registers until the columns end.  No warp waits for another one on the way.
//   CTA       one per SM, 16 warps (8 with two column tiles).  It first turns its columns of the activation rows into f16 B fragments
//             in shared memory, in the order the tiles consume them; every (row, 256-column slice) gets its own power-of-two rescale
//             so bf16 outliers cannot overflow f16, undone in fp32 when the slice is accumulated.
//   cluster   up to 8 CTAs split K when one CTA's shared memory cannot hold the fragments of all columns (kMaxSlices) or the strips
//             alone do not fill the chip.  The partial sums of a strip cross once, through distributed shared memory (st.async): rank r
//             of the cluster adds up, in rank order, and finishes the r-th part of the tile.  No workspace, no second kernel.
//
// The form before this one put 8 warps on 8 slices of the same strip, a ninth warp summed their tiles strip by strip, K splits met in
// a workspace and a second kernel: per strip a round of waits on the slot ring, two CTAs of warps an SM (one for the 3-bit format, whose
// high-bit plane had its own fragments), and rows 9-16 streamed the weights a second time.  Measured per FFN of 5120 x 17408 (gate/up +
// down; before → now): NVFP4, 1 row 49.7 → 38.2 µs (3.9 TB/s); 3 bits, 8 rows 103 → 62.8; 2 bits, 3 rows 58.2 → 40.7; 3 bits, 13 rows of
// 2048 x 6144 79 → 47.  What bounds it now: NVFP4 the memory stream and 4 µs of start-up a launch; the low-bit formats the decode (110
// ALU instructions a tile at half rate) and one warp's latency over a tile where K is split and only 10 of 16 warps have a strip.
//
// Low-bit decode without subtractions per element: a field left at bit 4^j or 16^j of an f16 mantissa under exponent 0x64 reads as
// 1024 + q·4^j (2 bits) or 1024 + q·16^j (3 bits).  The B fragments carry the matching 4^-j / 16^-j factors (exact), and the
// 1024·Σx' offset is removed per group together with the zero-point:  y += s·(tile − zp·S0 − S1), S0 = Σ x, S1 = 1024·Σ x'.
// Scales and zero-points applied in fp32.  The 3-bit codes are put together from both planes before that (the high bits are spread
// to the low fields' spacing for 16 columns at a time), so they need no fragments and no tile of their own.
#include "moe_stream.cuh"

namespace hb {

constexpr int kDSlice = 256;            // columns per pipeline stage
constexpr int kMaxSlices = 20;          // of one CTA: 80 KB of fragments for 8 rows, 160 KB for 16
constexpr int kMaxCluster = 8;
__host__ __device__ constexpr int dense_warps(int nb) { return nb == 1 ? 16 : 8; }

// A stage = 16 rows of codes (first plane, second plane), then 16 bytes of scales (and zero-points) a row.  Rows are packed; 16-byte
// chunks are exchanged inside a row by the row's number so that the eight rows a load touches lie in different banks.
__host__ __device__ constexpr int dense_row_w(int fmt) { return fmt == HB_FMT_NVFP4 ? 128 : 64; }
__host__ __device__ constexpr int dense_row_h(int fmt) { return fmt == HB_FMT_LB3_G64 ? 32 : 0; }
__host__ __device__ constexpr int dense_stage_bytes(int fmt) { return 16 * (dense_row_w(fmt) + dense_row_h(fmt) + 16); }

// 4^(j·sign) as a pair of f16
__host__ __device__ constexpr uint32_t lowbit_factor(int j, int sign) { return (uint32_t)(0x3C00 + sign * j * 0x800) * 0x10001u; }

// Fragment order.  Quad q (registers 4q .. 4q + 3) of lane (tok, t) of a slice: registers r, halves =
//   NVFP4          columns 64t + 2r, 64t + 2r + 1
//   low-bit        with gq = r >> 3, pr = r & 7: columns 64gq + 16t + c and + 8;  2 bits: c = pr, times 4^-j, j = pr < 5 ? pr : pr - 5;
//                  3 bits: c = 0 2 4 6 1 3 5 7 [pr], times 16^-(pr & 1)
// One warp per (slice, row): v = the 8 columns [8·lane, 8·lane + 8) of the slice.  xb: quad (q, t) of this row goes to xb[q·qs + t].
template <int FMT>
__device__ __forceinline__ void dense_build_row_slice(uint4 v, int lane, uint4* xb, int qs, float* inv) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  const uint32_t m2 = __vmaxu2(__vmaxu2(w[0] & 0x7fff7fffu, w[1] & 0x7fff7fffu), __vmaxu2(w[2] & 0x7fff7fffu, w[3] & 0x7fff7fffu));
  const uint32_t am = __reduce_max_sync(0xffffffffu, max(m2 & 0xffffu, m2 >> 16));
  const int e = min(max((int)(am >> 7), 27), 254);                       // bf16 exponent field of the largest magnitude
  const float f = __int_as_float((uint32_t)(127 + 14 + 127 - e) << 23);  // the maximum lands in [2^14, 2^15)
  if (lane == 0) *inv = __int_as_float((uint32_t)(e - 14) << 23);
  uint32_t h[4];                                                         // columns (0 1) (2 3) (4 5) (6 7) as f16 pairs
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __half2 hh = __floats2half2_rn(__uint_as_float(w[j] << 16) * f, __uint_as_float(w[j] & 0xffff0000u) * f);
    h[j] = *reinterpret_cast<const uint32_t*>(&hh);
  }
  if (FMT == HB_FMT_NVFP4) {
    xb[(lane & 7) * qs + (lane >> 3)] = make_uint4(h[0], h[1], h[2], h[3]);
    return;
  }
  // even lanes put together registers 0-3 (their own columns the low halves), odd lanes registers 4-7 (their own the high halves)
  const bool hi = lane & 1;
  if (FMT == HB_FMT_LB3_G64) {                                           // → (0 2) (4 6) (1 3) (5 7)
    const uint32_t p0 = __byte_perm(h[0], h[1], 0x5410), p1 = __byte_perm(h[2], h[3], 0x5410);
    const uint32_t p2 = __byte_perm(h[0], h[1], 0x7632), p3 = __byte_perm(h[2], h[3], 0x7632);
    h[0] = p0; h[1] = p1; h[2] = p2; h[3] = p3;
  }
  const uint32_t g0 = __shfl_xor_sync(0xffffffffu, hi ? h[0] : h[2], 1), g1 = __shfl_xor_sync(0xffffffffu, hi ? h[1] : h[3], 1);
  const uint32_t a0 = hi ? g0 : h[0], b0 = hi ? h[2] : g0, a1 = hi ? g1 : h[1], b1 = hi ? h[3] : g1;
  const uint32_t o[4] = {__byte_perm(a0, b0, 0x5410), __byte_perm(a0, b0, 0x7632), __byte_perm(a1, b1, 0x5410), __byte_perm(a1, b1, 0x7632)};
  const uint32_t f0 = FMT == HB_FMT_LB2_G64 && hi ? lowbit_factor(4, -1) : lowbit_factor(0, -1);   // 4^-j of registers 0-3: j = 0 1 2 3, of 4-7: 4 0 1 2
  const uint32_t f1 = FMT == HB_FMT_LB3_G64 ? lowbit_factor(2, -1) : hi ? lowbit_factor(0, -1) : lowbit_factor(1, -1);   // 16^-1 = 4^-2
  const uint32_t f2 = FMT == HB_FMT_LB3_G64 ? lowbit_factor(0, -1) : hi ? lowbit_factor(1, -1) : lowbit_factor(2, -1);
  const uint32_t f3 = FMT == HB_FMT_LB3_G64 ? lowbit_factor(2, -1) : hi ? lowbit_factor(2, -1) : lowbit_factor(3, -1);
  xb[(2 * (lane >> 3) + (hi ? 1 : 0)) * qs + ((lane & 7) >> 1)] = make_uint4(hmul2_u32(o[0], f0), hmul2_u32(o[1], f1), hmul2_u32(o[2], f2), hmul2_u32(o[3], f3));
}

struct DenseMat { const uint8_t* w; const uint8_t* wh; const uint8_t* s; const uint8_t* zp; float g; };
struct DenseArgs {
  DenseMat mat[2]; int n_mats;
  uint32_t* err;                          // the context's error word (bounded waits)
  int N, K, M, ldx; uint32_t m_inv;        // m_inv: ceil(2^32 / M) for i / M (M > 1)
  int sl0, slices;                        // this launch covers slices [sl0, sl0 + slices) of K / 256
  const __nv_bfloat16* x;
  int mode; void* y; int ldy;             // 0: y fp32, 1: y bf16, 2: act = bf16( bf16(silu(bf16 gate)) · bf16 up )
  float4* acc; int acc_in, last;          // K beyond one launch: sums so far [strip][tile][lane], read if acc_in, written unless last
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N_>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N_) : "memory"); }
__device__ __forceinline__ uint32_t map_cluster(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_async4(uint32_t dst, float4 v, uint32_t bar) {   // into a CTA of the cluster, counted in bytes on that CTA's barrier
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
               ::"r"(dst), "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w)), "r"(bar) : "memory");
}

// (w & M) | base as one logic instruction: an instruction holds one constant, so the exponent bits have to sit in a register, and the
// compiler is kept from seeing that they are a constant (it made two instructions of it: 179 ALU instructions a tile instead of 110).
template <uint32_t M>
__device__ __forceinline__ uint32_t field_f16(uint32_t w, uint32_t base) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(w), "n"(M), "r"(base));
  return r;
}
// One lane's 16 three-bit codes of a group: w = low two bits (column c at bits 2c), h = high bits (column c at bit c).  p[pr]: columns
// c, c + 8 (c = 0 2 4 6 1 3 5 7 [pr]) as 1024 + q·16^(pr & 1).  The spread high bits sit at 2c, one bit above where a 4-bit field
// starting at an even column needs them and exactly where the odd columns (moved down by 2) do.
__device__ __forceinline__ void lb3_pairs(uint32_t w, uint32_t h, uint32_t base, uint32_t (&p)[8]) {
  uint32_t s = (h | (h << 8)) & 0x00ff00ffu;
  s = (s | (s << 4)) & 0x0f0f0f0fu;
  s = (s | (s << 2)) & 0x33333333u;
  s = (s | (s << 1)) & 0x55555555u;
  const uint32_t e = (w & 0x33333333u) | ((s << 2) & 0x44444444u), o = ((w >> 2) & 0x33333333u) | (s & 0x44444444u);
  const uint32_t e8 = e >> 8, o8 = o >> 8;
  p[0] = field_f16<0x00070007u>(e, base); p[1] = field_f16<0x00700070u>(e, base);
  p[2] = field_f16<0x00070007u>(e8, base); p[3] = field_f16<0x00700070u>(e8, base);
  p[4] = field_f16<0x00070007u>(o, base); p[5] = field_f16<0x00700070u>(o, base);
  p[6] = field_f16<0x00070007u>(o8, base); p[7] = field_f16<0x00700070u>(o8, base);
}
__device__ __forceinline__ void lb2_pairs(uint32_t w, uint32_t base, uint32_t (&p)[8]) {
  const uint32_t w2 = w >> 10;
  p[0] = field_f16<0x00030003u>(w, base); p[1] = field_f16<0x000C000Cu>(w, base); p[2] = field_f16<0x00300030u>(w, base);
  p[3] = field_f16<0x00C000C0u>(w, base); p[4] = field_f16<0x03000300u>(w, base);
  p[5] = field_f16<0x00030003u>(w2, base); p[6] = field_f16<0x000C000Cu>(w2, base); p[7] = field_f16<0x00300030u>(w2, base);
}

struct DenseSmem { size_t sums, inv, xch, bars, ring, total; };   // byte offsets; the fragments come first
__host__ __device__ constexpr DenseSmem dense_smem(int fmt, int nb, int mt, int slices, int cluster, int nst) {
  DenseSmem s{};
  size_t o = (size_t)slices * nb * mt * 512;
  s.sums = o; o += fmt == HB_FMT_NVFP4 ? 0 : (size_t)slices * nb * 256;
  s.inv = o; o += (size_t)slices * nb * 32;
  s.xch = o; o += cluster > 1 ? (size_t)dense_warps(nb) * 2 * nb * 512 : 0;
  s.bars = o; o += (size_t)dense_warps(nb) * 2 * 8;
  o = (o + 127) / 128 * 128;
  s.ring = o; o += (size_t)dense_warps(nb) * nst * dense_stage_bytes(fmt);
  s.total = o;
  return s;
}

template <int FMT, int NB, int NST>
__global__ void __launch_bounds__(dense_warps(NB) * 32, 1) dense_gemv_kernel(const DenseArgs a) {
  constexpr int WARPS = dense_warps(NB), STG = dense_stage_bytes(FMT), RW = dense_row_w(FMT), RH = dense_row_h(FMT);
  extern __shared__ __align__(128) uint8_t dsm[];
  uint32_t rank, C;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(C));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int ncl = gridDim.x / C, cl = blockIdx.x / C;
  const int s_lo = a.sl0 + (int)((long long)a.slices * rank / C), nsl = a.sl0 + (int)((long long)a.slices * (rank + 1) / C) - s_lo;
  const int mt = min(a.M, 8);                                            // rows a column tile holds in shared memory
  const DenseSmem L = dense_smem(FMT, NB, mt, (a.slices + (int)C - 1) / (int)C, (int)C, NST);
  uint4* xb_s = reinterpret_cast<uint4*>(dsm);                           // [slice][tile][8 quads][mt rows][4]
  float2* sums_s = reinterpret_cast<float2*>(dsm + L.sums);              // [slice][tile][4 groups][8 rows] (S0, -S1)
  float* inv_s = reinterpret_cast<float*>(dsm + L.inv);                  // [slice][tile][8 rows]
  uint64_t* bar = reinterpret_cast<uint64_t*>(dsm + L.bars) + warp * 2;  // [2 slots] the peers' parts of this warp's strip are here
  const uint32_t ring = smem_u32(dsm + L.ring) + warp * NST * STG;
  const uint32_t xch = smem_u32(dsm + L.xch) + warp * 2 * NB * 512;      // [slot][tile][source rank][lane of the part] float4
  const int K = a.K, rows_per = a.n_mats == 2 ? 8 : 16, strips = (a.N + rows_per - 1) / rows_per, step = ncl * WARPS;
  if (C > 1) {
    if (lane == 0) { mbar_init(&bar[0], 1); mbar_init(&bar[1], 1); mbar_fence_init(); }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  }
  // ---- the weight stream: (strip, slice) in order, NST - 1 stages ahead of the arithmetic.  Each lane keeps the addresses of its own
  // 16-byte pieces of a stage and moves them on by a slice.
  constexpr int NC = FMT == HB_FMT_NVFP4 ? 4 : 2, CW = FMT == HB_FMT_NVFP4 ? 8 : 4;   // code pieces a lane fetches; 16-byte pieces of a row
  int istrip = warp * ncl + cl, isl = 0, istage = 0;
  const uint8_t* pc[NC];
  const uint8_t *ph = nullptr, *ps = nullptr;
  auto point = [&]() {                                                   // at the first slice of strip istrip
    const int n0 = istrip * rows_per;
    auto row_of = [&](int r, bool& m1) { m1 = rows_per == 8 && r >= 8; return (size_t)min(n0 + (m1 ? r - 8 : r), a.N - 1); };
    bool m1;
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      const size_t n = row_of(lane / CW + 32 / CW * i, m1);
      pc[i] = (m1 ? a.mat[1].w : a.mat[0].w) + n * (K / (FMT == HB_FMT_NVFP4 ? 2 : 4)) + (size_t)s_lo * RW + (lane % CW) * 16;
    }
    if (FMT == HB_FMT_LB3_G64) { const size_t n = row_of(lane >> 1, m1); ph = (m1 ? a.mat[1].wh : a.mat[0].wh) + n * (K / 8) + (size_t)s_lo * 32 + (lane & 1) * 16; }
    const size_t n = row_of(lane & 15, m1);
    if (FMT == HB_FMT_NVFP4) ps = (m1 ? a.mat[1].s : a.mat[0].s) + n * (K / 16) + (size_t)s_lo * 16;
    else ps = (lane >> 4 ? (m1 ? a.mat[1].zp : a.mat[0].zp) : (m1 ? a.mat[1].s : a.mat[0].s)) + (n * (K / 64) + (size_t)s_lo * 4) * 2;
  };
  if (istrip < strips) point();
  uint32_t dc[NC];                                                       // where the pieces go inside a stage
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    const int r = lane / CW + 32 / CW * i, c = lane % CW;
    dc[i] = ring + r * RW + ((FMT == HB_FMT_NVFP4 ? c ^ (r & 1) : c ^ ((r >> 1) & 3)) << 4);
  }
  const uint32_t dh = ring + 16 * RW + (lane >> 1) * RH + (((lane & 1) ^ ((lane >> 3) & 1)) << 4);
  const uint32_t ds = ring + 16 * (RW + RH) + (lane & 15) * 16 + (FMT == HB_FMT_NVFP4 ? 0 : (lane >> 4) * 8);
  auto issue_next = [&]() {
    if (istrip < strips) {
      const uint32_t st = istage * STG;
#pragma unroll
      for (int i = 0; i < NC; ++i) { cp_async16(dc[i] + st, pc[i]); pc[i] += RW; }
      if (FMT == HB_FMT_LB3_G64) { cp_async16(dh + st, ph); ph += 32; }
      if (FMT == HB_FMT_NVFP4) { if (lane < 16) cp_async16(ds + st, ps); ps += 16; }
      else { cp_async8(ds + st, ps); ps += 8; }
      if (++isl == nsl) { isl = 0; istrip += step; if (istrip < strips) point(); }
    }
    if (++istage == NST) istage = 0;
    cp_async_commit();                                                   // always commit: the group count stays in step with the stages
  };
  if (nsl > 0) for (int i = 0; i < NST - 1; ++i) issue_next();           // weights do not depend on the previous kernel: fetch before waiting for it
  griddep_wait();
  griddep_launch();
  // ---- B fragments of this CTA's columns, one warp per (slice, row); five rows' loads in flight together
  {
    constexpr int UN = 5;
    const int todo = nsl * a.M;
    for (int i0 = warp; i0 < todo; i0 += WARPS * UN) {
      uint4 v[UN];
      int sl[UN], m[UN];
#pragma unroll
      for (int u = 0; u < UN; ++u) {
        const int i = i0 + u * WARPS;
        sl[u] = a.M == 1 ? i : (int)__umulhi((uint32_t)i, a.m_inv); m[u] = i - sl[u] * a.M;
        if (i < todo) v[u] = __ldcg(reinterpret_cast<const uint4*>(a.x + (size_t)m[u] * a.ldx + (size_t)(s_lo + sl[u]) * kDSlice) + lane);
      }
#pragma unroll
      for (int u = 0; u < UN; ++u) {
        if (i0 + u * WARPS < todo) {
          const int sb = sl[u] * NB + (m[u] >> 3), tok = m[u] & 7;
          dense_build_row_slice<FMT>(v[u], lane, xb_s + (size_t)sb * mt * 32 + tok * 4, mt * 4, inv_s + sb * 8 + tok);
        }
      }
    }
  }
  const int tokc = min(g, mt - 1);                                       // B fragments of rows that are not there: another row's, for columns nobody reads
  if (FMT != HB_FMT_NVFP4) {
    // the tile of a 64-column group sums (1024 + q·b^j)·x': S0 = Σ x removes the zero-point, S1 = 1024·Σ x' the offset — both as tiles
    // whose weights are constants
    __syncthreads();
    for (int i = warp; i < nsl * NB * 4; i += WARPS) {
      const int sb = i >> 2, gq = i & 3;
      const uint4* xb = xb_s + (size_t)sb * mt * 32 + tokc * 4 + t;
      const uint4 b0 = xb[2 * gq * mt * 4], b1 = xb[(2 * gq + 1) * mt * 4];
      const uint32_t b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
      float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int m4 = 0; m4 < 4; ++m4) {
        uint32_t one[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) { const int pr = 2 * m4 + h; one[h] = lowbit_factor(FMT == HB_FMT_LB3_G64 ? 2 * (pr & 1) : pr < 5 ? pr : pr - 5, 1); }
        const uint32_t a0[4] = {one[0], one[0], one[1], one[1]}, a1[4] = {0x64006400u, 0x64006400u, 0x64006400u, 0x64006400u};
        mma_f16_16816(s0, a0, b[2 * m4], b[2 * m4 + 1]);
        mma_f16_16816(s1, a1, b[2 * m4], b[2 * m4 + 1]);
      }
      if (g == 0) *reinterpret_cast<float4*>(sums_s + sb * 32 + gq * 8 + 2 * t) = make_float4(s0[0], -s1[0], s0[1], -s1[1]);
    }
  }
  if (C > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // every CTA's barriers are set up
  __syncthreads();

  // finishes the lane's four values of a tile: rows g, g + 8 of the strip (pair: gate and up of the same output), activation rows 2t, 2t + 1
  auto finish = [&](const float4& v, int strip, int nb) {
    const float c4[4] = {v.x, v.y, v.z, v.w};
    const float ga = FMT == HB_FMT_NVFP4 ? a.mat[0].g : 1.f, gb = FMT == HB_FMT_NVFP4 && a.n_mats == 2 ? a.mat[1].g : ga;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int m = nb * 8 + 2 * t + c, n = strip * rows_per + g;
      if (m >= a.M) continue;
      const float lo = c4[c] * ga, hi = c4[c + 2] * gb;
      if (a.mode == 2) {
        if (n < a.N) {
          const float gv = bf16r(lo), uv = bf16r(hi);
          reinterpret_cast<__nv_bfloat16*>(a.y)[(size_t)m * a.ldy + n] = __float2bfloat16(bf16r(gv / (1.f + __expf(-gv))) * uv);
        }
      } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int nn = n + 8 * h;
          const float r = h ? hi : lo;
          if (nn < a.N) {
            if (a.mode == 0) reinterpret_cast<float*>(a.y)[(size_t)m * a.ldy + nn] = r;
            else reinterpret_cast<__nv_bfloat16*>(a.y)[(size_t)m * a.ldy + nn] = __float2bfloat16(r);
          }
        }
      }
    }
  };
  auto emit = [&](float4 v, int strip, int nb) {                         // the strip's sums over this launch's columns
    if (a.acc) {
      float4* p = a.acc + ((size_t)strip * NB + nb) * 32 + lane;
      if (a.acc_in) { const float4 o = *p; v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w; }
      if (!a.last) { *p = v; return; }
    }
    finish(v, strip, nb);
  };
  // cluster: lane l's values are added up by rank l·C/32.  A warp finishes strip i after the arithmetic of strip i + 1 and before
  // it sends that: whoever has all parts of strip i + 1 knows that its peers are done with the slot of strip i.
  const int part = 32 / (int)C, owner = lane / part;
  float4 own[NB];                                                        // this lane's share of the strip that is on its way
  int pend = -1, pslot = 0;
  uint32_t pph = 0;
  bool ok = true;
  auto settle = [&]() {
    if (pend < 0) return;
    ok = mbar_wait(&bar[pslot], pph, a.err, 0x10000u) && ok;
    if (owner == (int)rank && ok) {
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int r = 0; r < (int)C; ++r) {                               // rank order: the same sum on every run
          float4 o = own[nb];
          if (r != (int)rank) {
            const uint32_t at = xch + (uint32_t)((pslot * NB + nb) * 512 + (r * part + lane - owner * part) * 16);
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(o.x), "=f"(o.y), "=f"(o.z), "=f"(o.w) : "r"(at) : "memory");
          }
          s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w;
        }
        emit(s, pend, nb);
      }
    }
    pend = -1;
    if (pslot) pph ^= 1u;
    pslot ^= 1;
    __syncwarp();
  };

  int cstage = 0;
  int sslot = 0;
  uint32_t base;                                                         // two f16 of 1024
  asm volatile("mov.b32 %0, 0x64006400;" : "=r"(base));
  for (int strip = warp * ncl + cl; strip < strips && ok; strip += step) {
    float tot[NB][4];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) { tot[nb][0] = 0.f; tot[nb][1] = 0.f; tot[nb][2] = 0.f; tot[nb][3] = 0.f; }
    for (int sl = 0; sl < nsl; ++sl) {
      cp_async_wait<NST - 2>();
      __syncwarp();                                                      // this stage has landed for all lanes, and all are through with the one before it
      issue_next();
      const uint8_t* st = dsm + L.ring + (size_t)(warp * NST + cstage) * STG;
      const uint4* xb = xb_s + (size_t)sl * NB * mt * 32 + tokc * 4 + t;
      if constexpr (FMT == HB_FMT_NVFP4) {
        const uint32_t s4a = *reinterpret_cast<const uint32_t*>(st + 16 * RW + g * 16 + 4 * t), s4b = *reinterpret_cast<const uint32_t*>(st + 16 * RW + (g + 8) * 16 + 4 * t);
        const uint32_t fa[2] = {cvt_e4m3x2_f16x2(s4a & 0xffffu), cvt_e4m3x2_f16x2(s4a >> 16)};
        const uint32_t fb[2] = {cvt_e4m3x2_f16x2(s4b & 0xffffu), cvt_e4m3x2_f16x2(s4b >> 16)};
        float c[NB][2][4];
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
          for (int i = 0; i < 8; ++i) c[nb][i >> 2][i & 3] = 0.f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int ch = ((2 * t + h) ^ (g & 1)) << 4;
          const uint4 qa = *reinterpret_cast<const uint4*>(st + g * RW + ch), qb = *reinterpret_cast<const uint4*>(st + (g + 8) * RW + ch);
          const uint32_t wqa[4] = {qa.x, qa.y, qa.z, qa.w}, wqb[4] = {qb.x, qb.y, qb.z, qb.w};
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            const int j = 4 * h + jj;
            const uint32_t sca = __byte_perm(fa[h], 0, (jj >> 1) ? 0x3232 : 0x1010), scb = __byte_perm(fb[h], 0, (jj >> 1) ? 0x3232 : 0x1010);
            uint32_t ha[4], hb_[4];
            cvt_e2m1x8_f16x2(wqa[jj], ha);
            cvt_e2m1x8_f16x2(wqb[jj], hb_);
#pragma unroll
            for (int i = 0; i < 4; ++i) { ha[i] = hmul2_u32(ha[i], sca); hb_[i] = hmul2_u32(hb_[i], scb); }
#pragma unroll
            for (int nb = 0; nb < NB; ++nb) {
              const uint4 b = xb[(nb * 8 + j) * mt * 4];
              { const uint32_t afr[4] = {ha[0], hb_[0], ha[1], hb_[1]}; mma_f16_16816(c[nb][0], afr, b.x, b.y); }
              { const uint32_t afr[4] = {ha[2], hb_[2], ha[3], hb_[3]}; mma_f16_16816(c[nb][1], afr, b.z, b.w); }
            }
          }
        }
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          const float2 iv = *reinterpret_cast<const float2*>(inv_s + (sl * NB + nb) * 8 + 2 * t);     // undo the slice factor of rows 2t, 2t+1
#pragma unroll
          for (int i = 0; i < 4; ++i) tot[nb][i] = fmaf(c[nb][0][i] + c[nb][1][i], (i & 1) ? iv.y : iv.x, tot[nb][i]);
        }
      } else {
        const uint8_t* sz = st + 16 * (RW + RH);
        const uint4 szA = *reinterpret_cast<const uint4*>(sz + g * 16), szB = *reinterpret_cast<const uint4*>(sz + (g + 8) * 16);
        const uint32_t szAw[4] = {szA.x, szA.y, szA.z, szA.w}, szBw[4] = {szB.x, szB.y, szB.z, szB.w};   // {s01, s23, zp01, zp23} as f16 pairs
        float sub[NB][4];
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) { sub[nb][0] = 0.f; sub[nb][1] = 0.f; sub[nb][2] = 0.f; sub[nb][3] = 0.f; }
#pragma unroll
        for (int gq = 0; gq < 4; ++gq) {
          const int ch = ((gq ^ ((g >> 1) & 3)) << 4) + 4 * t;           // rows g and g + 8 exchange their chunks alike
          const uint32_t wA = *reinterpret_cast<const uint32_t*>(st + g * RW + ch), wB = *reinterpret_cast<const uint32_t*>(st + (g + 8) * RW + ch);
          uint32_t pA[8], pB[8];
          if constexpr (FMT == HB_FMT_LB3_G64) {
            const uint8_t* hp = st + 16 * RW + (((gq >> 1) ^ ((g >> 2) & 1)) << 4) + (gq & 1) * 8 + 2 * t;
            lb3_pairs(wA, *reinterpret_cast<const uint16_t*>(hp + g * RH), base, pA);
            lb3_pairs(wB, *reinterpret_cast<const uint16_t*>(hp + (g + 8) * RH), base, pB);
          } else { lb2_pairs(wA, base, pA); lb2_pairs(wB, base, pB); }
          const __half2 sA2 = *reinterpret_cast<const __half2*>(&szAw[gq >> 1]), zA2 = *reinterpret_cast<const __half2*>(&szAw[2 + (gq >> 1)]);
          const __half2 sB2 = *reinterpret_cast<const __half2*>(&szBw[gq >> 1]), zB2 = *reinterpret_cast<const __half2*>(&szBw[2 + (gq >> 1)]);
          const float sA = (gq & 1) ? __high2float(sA2) : __low2float(sA2), zA = (gq & 1) ? __high2float(zA2) : __low2float(zA2);
          const float sB = (gq & 1) ? __high2float(sB2) : __low2float(sB2), zB = (gq & 1) ? __high2float(zB2) : __low2float(zB2);
#pragma unroll
          for (int nb = 0; nb < NB; ++nb) {
            const uint4 b0 = xb[(nb * 8 + 2 * gq) * mt * 4], b1 = xb[(nb * 8 + 2 * gq + 1) * mt * 4];
            const uint32_t b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
            // scale and zero-point in fp32: y += s·(tile − zp·S0 − S1); the tile starts from the two corrections
            const float4 su = *reinterpret_cast<const float4*>(sums_s + (sl * NB + nb) * 32 + gq * 8 + 2 * t);   // (S0, -S1) of rows 2t, 2t+1
            float tmp[4] = {fmaf(-zA, su.x, su.y), fmaf(-zA, su.z, su.w), fmaf(-zB, su.x, su.y), fmaf(-zB, su.z, su.w)};
#pragma unroll
            for (int m4 = 0; m4 < 4; ++m4) { const uint32_t afr[4] = {pA[2 * m4], pB[2 * m4], pA[2 * m4 + 1], pB[2 * m4 + 1]}; mma_f16_16816(tmp, afr, b[2 * m4], b[2 * m4 + 1]); }
            sub[nb][0] = fmaf(sA, tmp[0], sub[nb][0]);
            sub[nb][1] = fmaf(sA, tmp[1], sub[nb][1]);
            sub[nb][2] = fmaf(sB, tmp[2], sub[nb][2]);
            sub[nb][3] = fmaf(sB, tmp[3], sub[nb][3]);
          }
        }
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          const float2 iv = *reinterpret_cast<const float2*>(inv_s + (sl * NB + nb) * 8 + 2 * t);     // undo the slice factor of rows 2t, 2t+1
#pragma unroll
          for (int i = 0; i < 4; ++i) tot[nb][i] = fmaf(sub[nb][i], (i & 1) ? iv.y : iv.x, tot[nb][i]);
        }
      }
      if (++cstage == NST) cstage = 0;
    }
    if (C == 1) {
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) emit(make_float4(tot[nb][0], tot[nb][1], tot[nb][2], tot[nb][3]), strip, nb);
    } else {
      settle();                                                          // the strip before this one
      if (!ok) break;
      if (lane == 0) mbar_expect_tx(&bar[sslot], (C - 1) * (uint32_t)part * 16 * NB);
      const uint32_t rbar = map_cluster(smem_u32(&bar[sslot]), owner), rx = map_cluster(xch, owner);
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        own[nb] = make_float4(tot[nb][0], tot[nb][1], tot[nb][2], tot[nb][3]);
        if (owner != (int)rank) st_async4(rx + (uint32_t)((sslot * NB + nb) * 512 + ((int)rank * part + lane - owner * part) * 16), own[nb], rbar);
      }
      pend = strip;
      sslot ^= 1;
    }
  }
  if (C > 1) {
    settle();
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // a CTA's memory outlives its peers' stores
  }
  cp_async_wait<0>();
}

// ------------------------------------------------------------------------------------------------ low-bit dequant (bit-exact definition)
__global__ void lb_dequant_kernel(int bits, const uint8_t* __restrict__ w, const uint8_t* __restrict__ wh, const __half* __restrict__ s,
                                  const __half* __restrict__ zp, int N, int K, __nv_bfloat16* __restrict__ out) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < (size_t)N * K; i += (size_t)gridDim.x * blockDim.x) {
    const size_t n = i / K; const int k = (int)(i % K);
    int q = (w[n * (K / 4) + k / 4] >> (2 * (k & 3))) & 3;
    if (bits == 3) q |= ((wh[n * (K / 8) + k / 8] >> (k & 7)) & 1) << 2;
    const float sf = __half2float(s[n * (K / 64) + k / 64]), zf = __half2float(zp[n * (K / 64) + k / 64]);
    out[i] = __float2bfloat16(__fmul_rn(__fsub_rn((float)q, zf), sf));
  }
}

}  // namespace hb

using namespace hb;

namespace {
int check_mat(hb_ctx* ctx, const hb_qmat* W, const char* fn) {
  HB_REQUIRE(ctx, W && W->w && W->s, HB_ERR_INVALID, "%s: NULL matrix", fn);
  HB_REQUIRE(ctx, W->fmt == HB_FMT_NVFP4 || W->fmt == HB_FMT_LB3_G64 || W->fmt == HB_FMT_LB2_G64, HB_ERR_INVALID, "%s: unknown format %d", fn, W->fmt);
  HB_REQUIRE(ctx, W->N > 0 && W->K > 0 && W->K % kDSlice == 0, HB_ERR_UNSUPPORTED, "%s: N=%d K=%d (K must be a multiple of %d)", fn, W->N, W->K, kDSlice);
  HB_REQUIRE(ctx, W->fmt == HB_FMT_NVFP4 || W->zp, HB_ERR_INVALID, "%s: low-bit matrix without zero-points", fn);
  HB_REQUIRE(ctx, hb_aligned(W->w, 16) && hb_aligned(W->s, 16) && (W->fmt == HB_FMT_NVFP4 || hb_aligned(W->zp, 8)), HB_ERR_INVALID,
             "%s: weight / scale pointers must be 16-byte aligned", fn);
  return HB_OK;
}
DenseMat to_mat(const hb_qmat* W) {
  DenseMat m;
  m.w = W->w; m.s = reinterpret_cast<const uint8_t*>(W->s); m.zp = reinterpret_cast<const uint8_t*>(W->zp); m.g = W->g;
  m.wh = W->fmt == HB_FMT_LB3_G64 ? W->w + (size_t)W->N * (W->K / 4) : nullptr;
  return m;
}
// How many CTAs split K (1, 2, 4 or 8): a function of the matrix alone, so that a row's sums do not depend on the rows beside it.
// A CTA's work is ceil(strips per cluster) · slices tiles; one warp takes about 8 times as long over a tile as a full SM does (measured:
// 0.4 µs against 0.05), so the tiles one warp has to do in a row count 8-fold; handing the sums over costs about as much as 8 tiles.
int dense_cluster(const hb_ctx* ctx, int N, int n_mats, int slices) {
  const int strips = n_mats == 2 ? (N + 7) / 8 : (N + 15) / 16;
  int best = 0, best_cost = 0;
  for (int i = 0; i < 4; ++i) {
    const int c = 1 << i, ncl = ctx->dense_clusters[i], per = (slices + c - 1) / c;
    if (ncl < 1 || per > kMaxSlices || (c > slices && best)) continue;
    const int units = (strips + ncl - 1) / ncl, serial = (units + dense_warps(1) - 1) / dense_warps(1) * per;
    const int cost = (units * per > 8 * serial ? units * per : 8 * serial) + (c > 1 ? 8 : 0);
    if (!best || cost < best_cost) { best = c; best_cost = cost; }
  }
  return best ? best : kMaxCluster;
}
constexpr int kLaunchSlices = kMaxSlices * kMaxCluster;    // slices one launch covers at most (K = 40960)
int dense_launches(int K) { return (K / kDSlice + kLaunchSlices - 1) / kLaunchSlices; }

// Eight rows fit beside the shallower ring whatever share of the columns dense_cluster gives a CTA, so every call has a way to run.  Two column
// tiles do not: 20 slices of a 9-16 row call take 160 KB of fragments, and a cluster's exchange buffer leaves too little for three stages
// (NVFP4 236928 and 3 bits 234880 of 232448 bytes).
constexpr bool dense_eight_rows_fit() {
  for (int fmt = 0; fmt < 3; ++fmt)
    for (int c = 1; c <= kMaxCluster; c *= 2)
      if (dense_smem(fmt, 1, 8, kMaxSlices, c, 3).total > 227 * 1024) return false;
  return true;
}
static_assert(HB_FMT_NVFP4 < 3 && HB_FMT_LB3_G64 < 3 && HB_FMT_LB2_G64 < 3 && dense_eight_rows_fit(), "shared memory");

using DenseFn = void (*)(const DenseArgs);
struct DenseKernel { DenseFn fn; int nst; };
// The ring depths built for a format, deepest first.  An SM's rings hold, NVFP4 / 3 / 2 bits: one column tile (16 warps) 147 / 115 / 123 KB, shallow
// 111 / 86 / 61; two (8 warps) 74 / 57 / 41 KB, shallow 55 / 43 / 31; all stages but one are in flight.
template <int FMT>
void dense_kernels(int nb, DenseKernel (&k)[2]) {
  constexpr int D = FMT == HB_FMT_LB2_G64 ? 6 : 4;
  if (nb == 1) { k[0] = DenseKernel{dense_gemv_kernel<FMT, 1, D>, D}; k[1] = DenseKernel{dense_gemv_kernel<FMT, 1, 3>, 3}; }
  else { k[0] = DenseKernel{dense_gemv_kernel<FMT, 2, 4>, 4}; k[1] = DenseKernel{dense_gemv_kernel<FMT, 2, 3>, 3}; }
}
void dense_kernels(int fmt, int nb, DenseKernel (&k)[2]) {
  if (fmt == HB_FMT_NVFP4) dense_kernels<HB_FMT_NVFP4>(nb, k);
  else if (fmt == HB_FMT_LB2_G64) dense_kernels<HB_FMT_LB2_G64>(nb, k);
  else dense_kernels<HB_FMT_LB3_G64>(nb, k);
}

// the deepest of the built rings that fits with M rows and `per` slices a CTA, -1: none
int dense_depth(const hb_ctx* ctx, int fmt, int M, int per, int C, const DenseKernel (&k)[2], size_t* smem) {
  for (int v = 0; v < 2; ++v)
    if ((*smem = dense_smem(fmt, M > 8 ? 2 : 1, M < 8 ? M : 8, per, C, k[v].nst).total) <= (size_t)ctx->smem_optin) return v;
  return -1;
}

int dense_run(hb_ctx* ctx, const hb_qmat* A, const hb_qmat* B2, const void* x, int ldx, int M, int mode, void* y, int ldy, void* ws, cudaStream_t st) {
  const int fmt = A->fmt, slices = A->K / kDSlice, nb = M > 8 ? 2 : 1, launches = dense_launches(A->K);
  DenseArgs a{};
  a.mat[0] = to_mat(A); if (B2) a.mat[1] = to_mat(B2);
  a.n_mats = B2 ? 2 : 1; a.N = A->N; a.K = A->K; a.M = M; a.ldx = ldx; a.x = reinterpret_cast<const __nv_bfloat16*>(x);
  a.m_inv = M > 1 ? (uint32_t)(((1ull << 32) + M - 1) / M) : 0u;
  a.mode = mode; a.y = y; a.ldy = ldy; a.err = ctx->dev_err;
  DenseKernel k[2];
  dense_kernels(fmt, nb, k);
  auto split = [&](int i, int* sl0, int* n) { *sl0 = (int)((long long)slices * i / launches); *n = (int)((long long)slices * (i + 1) / launches) - *sl0; };
  for (int i = 0; i < launches; ++i) {                                       // before anything runs: does every launch fit?
    int sl0, n; size_t smem;
    split(i, &sl0, &n);
    const int C = dense_cluster(ctx, A->N, a.n_mats, n);
    if (dense_depth(ctx, fmt, M, (n + C - 1) / C, C, k, &smem) >= 0) continue;
    HB_REQUIRE(ctx, M > 8, HB_ERR_UNSUPPORTED, "dense_gemv: N=%d K=%d needs %zu bytes of shared memory", A->N, A->K, smem);
    // two column tiles do not fit: the first eight rows and the rest one after the other.  The split of the columns stays the matrix's, so
    // the sums are the same.
    const int r = dense_run(ctx, A, B2, x, ldx, 8, mode, y, ldy, ws, st);
    return r ? r : dense_run(ctx, A, B2, a.x + 8 * (size_t)ldx, ldx, M - 8, mode, static_cast<char*>(y) + 8 * (size_t)ldy * (mode == 0 ? 4 : 2), ldy, ws, st);
  }
  for (int i = 0; i < launches; ++i) {
    split(i, &a.sl0, &a.slices);
    a.acc = launches > 1 ? reinterpret_cast<float4*>(ws) : nullptr; a.acc_in = i > 0; a.last = i == launches - 1;
    const int C = dense_cluster(ctx, A->N, a.n_mats, a.slices), per = (a.slices + C - 1) / C;
    size_t smem;
    const int v = dense_depth(ctx, fmt, M, per, C, k, &smem);
    const int strips = B2 ? (A->N + 7) / 8 : (A->N + 15) / 16, most = ctx->dense_clusters[C == 1 ? 0 : C == 2 ? 1 : C == 4 ? 2 : 3];
    const int ncl = most < strips ? most : strips;
    const int r = hb_launch_cluster(ctx, fmt == HB_FMT_NVFP4 ? "dense_gemv_nvfp4" : fmt == HB_FMT_LB2_G64 ? "dense_gemv_lb2" : "dense_gemv_lb3", true, C, k[v].fn,
                                    dim3((unsigned)(ncl * C)), dim3(dense_warps(nb) * 32), smem, st, a);
    if (r) return r;
  }
  return HB_OK;
}
}  // namespace

int hbk_dense_setup(hb_ctx* ctx) {
  for (int fmt : {HB_FMT_NVFP4, HB_FMT_LB3_G64, HB_FMT_LB2_G64})
    for (int nb = 1; nb <= 2; ++nb) {
      DenseKernel k[2];
      dense_kernels(fmt, nb, k);
      for (auto& kk : k) HB_CUDA(ctx, cudaFuncSetAttribute(reinterpret_cast<const void*>(kk.fn), cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->smem_optin));
    }
  // how many clusters of each size run at once when every CTA takes an SM: a cluster stays inside one GPC
  DenseKernel k[2];
  dense_kernels(HB_FMT_NVFP4, 1, k);
  for (int i = 0; i < 4; ++i) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 1u << i; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(ctx->sm_count >> i << i)); cfg.blockDim = dim3(dense_warps(1) * 32); cfg.dynamicSmemBytes = (size_t)ctx->smem_optin;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    int n = 0;
    if (i) HB_CUDA(ctx, cudaOccupancyMaxActiveClusters(&n, k[0].fn, &cfg));
    ctx->dense_clusters[i] = i ? n : ctx->sm_count;
  }
  return HB_OK;
}

extern "C" {

size_t hb_dense_gemv_ws_bytes(int fmt, int N, int K, int n_mats) {
  if (K <= 0 || N <= 0 || K % kDSlice || n_mats < 1 || n_mats > 2) return 0;
  (void)fmt;
  return dense_launches(K) > 1 ? (size_t)(n_mats == 2 ? (N + 7) / 8 : (N + 15) / 16) * 2 * 512 : 256;   // sums between the launches of a very long K
}

int hb_dense_gemv(hb_ctx* ctx, const hb_qmat* W, const void* x, int ldx, int M, void* yb, float* yf, int ldy, void* ws, void* stream) {
  if (!ctx) return HB_ERR_INVALID;
  int r = check_mat(ctx, W, "dense_gemv");
  if (r) return r;
  HB_REQUIRE(ctx, x && ((yb != nullptr) != (yf != nullptr)), HB_ERR_INVALID, "dense_gemv: x NULL, or not exactly one of yb / yf given");
  HB_REQUIRE(ctx, hb_aligned(x, 16) && ldx % 8 == 0, HB_ERR_INVALID, "dense_gemv: x must be 16-byte aligned with ldx a multiple of 8");
  HB_REQUIRE(ctx, M >= 1 && M <= 16 && ldx >= W->K && ldy >= W->N, HB_ERR_UNSUPPORTED, "dense_gemv: M=%d (1..16) ldx=%d ldy=%d", M, ldx, ldy);
  HB_REQUIRE(ctx, ws && hb_aligned(ws, 256), HB_ERR_WORKSPACE, "dense_gemv: ws NULL or not 256-byte aligned");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return dense_run(ctx, W, nullptr, x, ldx, M, yf ? 0 : 1, yf ? static_cast<void*>(yf) : yb, ldy, ws, st);
}

int hb_dense_gemv_gu(hb_ctx* ctx, const hb_qmat* G, const hb_qmat* U, const void* x, int ldx, int M, void* act, int lda, void* ws, void* stream) {
  if (!ctx) return HB_ERR_INVALID;
  int r = check_mat(ctx, G, "dense_gemv_gu");
  if (!r) r = check_mat(ctx, U, "dense_gemv_gu");
  if (r) return r;
  HB_REQUIRE(ctx, G->fmt == U->fmt && G->N == U->N && G->K == U->K, HB_ERR_INVALID, "dense_gemv_gu: gate and up must share format and shape");
  HB_REQUIRE(ctx, x && hb_aligned(x, 16) && ldx % 8 == 0, HB_ERR_INVALID, "dense_gemv_gu: x must be 16-byte aligned with ldx a multiple of 8");
  HB_REQUIRE(ctx, x && act && M >= 1 && M <= 16 && ldx >= G->K && lda >= G->N, HB_ERR_UNSUPPORTED, "dense_gemv_gu: M=%d (1..16) ldx=%d lda=%d", M, ldx, lda);
  HB_REQUIRE(ctx, ws && hb_aligned(ws, 256), HB_ERR_WORKSPACE, "dense_gemv_gu: ws NULL or not 256-byte aligned");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return dense_run(ctx, G, U, x, ldx, M, 2, act, lda, ws, st);
}

int hb_lb_dequant(hb_ctx* ctx, const hb_qmat* W, void* out_bf16, void* stream) {
  if (!ctx) return HB_ERR_INVALID;
  HB_REQUIRE(ctx, W && W->w && W->s && W->zp && out_bf16, HB_ERR_INVALID, "lb_dequant: NULL argument");
  HB_REQUIRE(ctx, (W->fmt == HB_FMT_LB3_G64 || W->fmt == HB_FMT_LB2_G64) && W->N > 0 && W->K > 0 && W->K % 64 == 0, HB_ERR_UNSUPPORTED,
             "lb_dequant: format %d N=%d K=%d", W->fmt, W->N, W->K);
  const size_t n = (size_t)W->N * W->K;
  size_t blocks = (n + 255) / 256, cap = (size_t)ctx->sm_count * 16;
  if (blocks > cap) blocks = cap;
  return hb_launch(ctx, "lb_dequant", false, lb_dequant_kernel, dim3((unsigned)blocks), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream),
                   W->fmt == HB_FMT_LB3_G64 ? 3 : 2, W->w, W->fmt == HB_FMT_LB3_G64 ? W->w + (size_t)W->N * (W->K / 4) : (const uint8_t*)nullptr,
                   reinterpret_cast<const __half*>(W->s), reinterpret_cast<const __half*>(W->zp), W->N, W->K, reinterpret_cast<__nv_bfloat16*>(out_bf16));
}

}  // extern "C"
