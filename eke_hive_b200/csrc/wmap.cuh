// Weight boxes of expert records by TMA.  A record table lives in device memory and may change between calls, records sit wherever their
// owner put them (16-byte aligned), and the host knows none of the addresses, so no tensor map can be made per record.  Instead one
// byte matrix [2^31 rows][pitch] covers the records of a table: its base is the lowest record's address (the anchor), and a matrix whose
// distance from the anchor is not a whole number of rows goes through variant v of the map, based v·16 bytes higher (pitch / 16 variants
// cover every 16-byte aligned address).
//
// The maps belong to the call: a CTA of a kernel that runs ahead of the GEMM anyway reads the call's table, stamps the variants into the
// call's workspace (8 KB to 30 KB, some 2 µs beside the other CTAs), and the GEMM reads them from there.  Nothing about them is kept from
// one call to the next: a captured call stamps its own maps on every replay, and calls of other shapes and tables in between do not
// reach them.
#pragma once
#include "tc_common.cuh"

namespace hb {

constexpr int kWmHead = 256;                                           // bytes in front of the maps: the anchor
constexpr int kWmVariants = 32;                                        // residues of 4096-aligned records: pitch / gcd(pitch, 4096) at most
__host__ __device__ constexpr int wm_variants(int K) { return K / 32; }   // of a matrix of K columns: pitch K / 2 bytes, 16 bytes apart
__host__ __device__ constexpr size_t wm_bytes(int K) { return kWmHead + (size_t)wm_variants(K) * sizeof(CUtensorMap); }

// What a stamping CTA needs; kind 0: gate and up (K = H), 1: down (K = I).
struct WmStamp {
  CUtensorMap tpl[2];                                                  // the map with any base
  const uint8_t* const* tab; int n_tab; const uint8_t* extra;          // the call's records: a table and one more (or nullptr)
  uint8_t* dst[2]; int nv[2];                                          // where the maps go, how many
};
// The whole block takes part.  The maps are complete for kernels behind this one that acquire them (tmap_acquire).
__device__ __forceinline__ void wm_stamp(const WmStamp& s) {
  __shared__ unsigned long long lo;
  if (threadIdx.x == 0) lo = s.extra ? reinterpret_cast<unsigned long long>(s.extra) : ~0ull;
  __syncthreads();
  unsigned long long mn = ~0ull;
  for (int i = threadIdx.x; i < s.n_tab; i += blockDim.x) { const unsigned long long p = __ldcg(reinterpret_cast<const unsigned long long*>(s.tab) + i); if (p) mn = min(mn, p); }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
  if ((threadIdx.x & 31) == 0) atomicMin(&lo, mn);
  __syncthreads();
  const unsigned long long anchor = lo == ~0ull ? 1ull << 40 : lo & ~15ull;
  if (threadIdx.x < 2) *reinterpret_cast<unsigned long long*>(threadIdx.x ? s.dst[1] : s.dst[0]) = anchor;
  for (int i = threadIdx.x; i < s.nv[0] + s.nv[1]; i += blockDim.x) {
    const bool dn = i >= s.nv[0];
    const int v = dn ? i - s.nv[0] : i;
    const uint4* src = reinterpret_cast<const uint4*>(dn ? &s.tpl[1] : &s.tpl[0]);
    uint4* dst = reinterpret_cast<uint4*>((dn ? s.dst[1] : s.dst[0]) + kWmHead) + (size_t)v * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) dst[j] = src[j];
    asm volatile("tensormap.replace.tile.global_address.global.b1024.b64 [%0], %1;" ::"l"(dst), "l"(anchor + 16ull * (unsigned)v) : "memory");
    asm volatile("fence.proxy.tensormap::generic.release.gpu;" ::: "memory");
  }
}

// The reading side, for the one thread that issues the copies.
struct WmArgs { const uint8_t* base; int pitch, pshift, gshift; };     // pshift: log2(pitch), -1 where it is no power of two up to 4096; gshift: log2(gcd(pitch, 4096))
struct WmBox { const CUtensorMap* map; int row; const uint8_t* far; };
struct WmReader {
  WmArgs a;
  unsigned long long anchor;
  uint32_t seen;                                                       // variants of 4096-aligned records acquired so far
  __device__ __forceinline__ void init(const WmArgs& a_) { a = a_; anchor = *reinterpret_cast<const unsigned long long*>(a.base); seen = 0u; }
  // Where matrix `w` (16-byte aligned) is.  A matrix more than 2^31 rows above the anchor is out of a box's coordinates (256 GB at the shortest
  // rows, 2 TB at 2048 columns): no map, its boxes are put together from 16-byte copies.
  __device__ __forceinline__ bool locate(const uint8_t* w, WmBox& b, uint32_t* err) {
    const unsigned long long delta = reinterpret_cast<unsigned long long>(w) - anchor;
    const unsigned long long row = a.pshift >= 0 ? delta >> a.pshift : delta / (unsigned)a.pitch;
    const uint32_t rem = (uint32_t)(delta - row * (unsigned)a.pitch);
    if (rem & 15u) { atomicOr(err, 0x400000u); return false; }
    b.map = nullptr; b.row = 0; b.far = w;
    if (row + (1ull << 24) < (1ull << 31)) {
      b.map = reinterpret_cast<const CUtensorMap*>(a.base + kWmHead) + (rem >> 4); b.row = (int)row;
      const uint32_t bit = rem & ((1u << a.gshift) - 1u) ? 0u : 1u << (rem >> a.gshift);
      if (!(seen & bit)) { tmap_acquire(b.map); seen |= bit; }
    }
    return true;
  }
  // 64 rows from row r of the matrix, bytes [c, c + 128) of each → shared memory under the 128-byte swizzle
  __device__ __forceinline__ void load(uint32_t dst, const WmBox& b, int c, int r, uint64_t* bar) const {
    if (b.map) tma_load_2d(dst, b.map, c, b.row + r, bar);
    else far_box(dst, b.far + (size_t)r * a.pitch + c, a.pitch, bar);
  }
  static __device__ __forceinline__ void far_box(uint32_t dst, const uint8_t* src, int pitch, uint64_t* bar) {
#pragma unroll 1
    for (int r = 0; r < 64; ++r, src += pitch)
#pragma unroll 1
      for (int ch = 0; ch < 8; ++ch)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 16, [%2];"
                     ::"r"(dst + r * 128 + ((ch ^ (r & 7)) << 4)), "l"(src + ch * 16), "r"(smem_u32(bar)) : "memory");
  }
};

inline int wm_gcd4096(int pitch) { int g = 1; while (g < 4096 && pitch % (2 * g) == 0) g *= 2; return g; }
inline WmArgs wm_args(const uint8_t* base, int K) {
  WmArgs a{base, K / 2, -1, 0};
  const int g = wm_gcd4096(a.pitch);
  while ((1 << a.gshift) < g) ++a.gshift;
  if (a.pitch == g) a.pshift = a.gshift;
  return a;
}

}  // namespace hb

// What stamps the maps of a call whose matrices have H and I columns into `base` (wm_bytes(H) for gate and up, then wm_bytes(I) for down)
int hbk_wm_stamp_args(hb_ctx* ctx, const uint8_t* const* tab, int n_tab, const uint8_t* extra, int H, int I, uint8_t* base, hb::WmStamp* out);
