// utl_pack.cu -- the batched pack in two launches (utl_qpack.cuh).
//
// The first (pack_plan_kernel) reads the values and decides every block: its plan
// goes into the block's entry of the offset table, the packed lengths are
// summed per 32, 1024 and 32768 blocks.  The second (pack_write_kernel) knows the
// byte offset of its blocks from those sums, reads the values again, writes
// the blocks into an image with the output's alignment and sends it out by a
// bulk store.  No block waits for another, neither kernel holds values in
// shared memory while it waits, and each is small enough for the instruction
// cache, which the one-launch packs (a warp's plan and write code, and the
// wait for the offsets between them) are not.
//
// Measured on 2^26 uint64 values of three shapes: 489 us (903 in one launch),
// of which the first launch is about 130 (its read of 537 MB takes 82 at the
// copy rate) and the second the rest: at 14 warps on an SM it issues 35% of the
// time and waits for loads and for shared memory, about two cycles per issue
// each.  One warp writing the exceptions of the tile's
// 32 blocks, a lane each, executes fewer instructions but leaves three warps
// at a barrier: 577 us, and 695 against 627 on 2^28 outlier values.
#include <cuda_runtime.h>
#include <stdint.h>

#include "utl_launch.h"
#include "utl_qpack.cuh"
#include "utl_streams.cuh"

namespace utl {
namespace qp {

constexpr int kWarps = 4;
constexpr int kThreads = 32 * kWarps;
constexpr int kTile = 8 * kWarps;  // blocks of a CTA
static_assert(kTile == 32, "a lane per block of the tile");

// Packed bytes of the tiles, of 32 of them and of 1024 (the groups' start at
// zero).  Up to kDirectTiles tiles the second launch sums the tiles' own and
// there are no groups: nothing to clear, one operation less on the stream.
constexpr int kDirectTiles = 1024;
struct Sums {
  uint32_t* one;
  uint32_t* g32;
  unsigned long long* g1024;  // null: no groups
};
// In the pack's scratch: 4 1/8 bytes per 32 blocks, of its 16.
inline size_t sums_bytes(int64_t n_tiles) {
  return 8 * (size_t)((n_tiles + 1023) / 1024) + 4 * (size_t)n_tiles + 4 * (size_t)((n_tiles + 31) / 32);
}
inline Sums sums_in(void* scratch, int64_t n_tiles) {
  Sums s;
  s.g1024 = (unsigned long long*)scratch;
  s.one = (uint32_t*)(s.g1024 + (n_tiles + 1023) / 1024);
  s.g32 = s.one + n_tiles;
  if (n_tiles <= kDirectTiles) s.g1024 = nullptr;
  return s;
}

// First value and value count of the lane's block b (0: none); b0: the
// warp's first block.
__device__ __forceinline__ int block_of(const PackArgs& a, int64_t b0, int64_t b, int lane, uint64_t* first) {
  uint64_t f, e;
  if (a.n_streams == 1) {
    f = a.val_off[0] + (uint64_t)b * kBlock;
    e = a.val_off[1];
  } else {
    if (b0 >= a.n_blocks) return 0;
    const int s0 = warp_stream_of(a.block_start, a.n_streams, b0, lane);
    const int64_t bb = min(b, a.n_blocks - 1);
    const int s = stream_from(a.block_start, a.n_streams, s0, bb);
    f = a.val_off[s] + (uint64_t)(bb - (int64_t)a.block_start[s]) * kBlock;
    e = a.val_off[s + 1];
  }
  *first = f;
  return b < a.n_blocks ? (int)min((uint64_t)kBlock, e - f) : 0;
}

template <bool LAST>
__device__ __forceinline__ uint4 ld_chunk(const uint4* p) {
  return LAST ? __ldcs(p) : __ldg(p);
}

// The n values at v (zero past them).  lo, hi: the bytes the stream table
// describes.  LAST: not needed in the cache afterwards.  Whole warp.
template <bool LAST>
__device__ __forceinline__ void load_block(const uint32_t* v, int n, uintptr_t lo, uintptr_t hi, int j, int lane,
                                           uint32_t (&x)[8][4]) {
  const uintptr_t a = (uintptr_t)v;
  const int m = (int)(a >> 2) & 3;  // words past a 16-byte boundary
  if (__all_sync(kFull, n == kBlock && m == 0)) {
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const uint4 t = ld_chunk<LAST>((const uint4*)v + 4 * r + j);
      x[r][0] = t.x; x[r][1] = t.y; x[r][2] = t.z; x[r][3] = t.w;
    }
    return;
  }
  const uintptr_t a0 = a & ~(uintptr_t)15, a1 = (a + 4 * (uintptr_t)n + 15) & ~(uintptr_t)15;
  if (__all_sync(kFull, n == 0 || (a0 >= lo && a1 <= hi))) {
    // the aligned chunks that cover the block; a row's words past the lane's
    // own chunk come from the next lane (lane 0's next row for lane 3)
    const uint4* p = (const uint4*)a0;
    const int chunks = n > 0 ? (int)((a1 - a0) >> 4) : 0;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    const bool m2 = (m & 2) != 0, m1 = (m & 1) != 0;
    const int src = (lane & 28) | ((j + 1) & 3);
    uint4 t = j < chunks ? ld_chunk<LAST>(p + j) : zero;
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const int c = 4 * (r + 1) + j;
      const uint4 down = c < chunks && (r < 7 || j == 0) ? ld_chunk<LAST>(p + c) : zero;
      const uint4 give = j == 0 ? down : t;
      const uint32_t u0 = __shfl_sync(kFull, give.x, src), u1 = __shfl_sync(kFull, give.y, src),
                     u2 = __shfl_sync(kFull, give.z, src);
      const uint32_t w0 = m2 ? t.z : t.x, w1 = m2 ? t.w : t.y, w2 = m2 ? u0 : t.z, w3 = m2 ? u1 : t.w,
                     w4 = m2 ? u2 : u0;
      x[r][0] = m1 ? w1 : w0;
      x[r][1] = m1 ? w2 : w1;
      x[r][2] = m1 ? w3 : w2;
      x[r][3] = m1 ? w4 : w3;
      t = down;
    }
    if (__any_sync(kFull, n < kBlock)) zero_padding(x, n, j);
    return;
  }
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int k = 0; k < 4; k++) x[r][k] = pos_of(r, k, j) < n ? v[pos_of(r, k, j)] : 0u;
}
// uint64 values as low and high words.
template <bool LAST>
__device__ __forceinline__ void load_block64(const uint64_t* v, int n, int j, uint32_t (&x)[8][4],
                                             uint32_t (&h)[8][4]) {
  if (__all_sync(kFull, n == kBlock && ((uintptr_t)v & 15) == 0)) {
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const uint4 A = ld_chunk<LAST>((const uint4*)v + 8 * r + 2 * j);
      const uint4 B = ld_chunk<LAST>((const uint4*)v + 8 * r + 2 * j + 1);
      x[r][0] = A.x; x[r][1] = A.z; x[r][2] = B.x; x[r][3] = B.z;
      h[r][0] = A.y; h[r][1] = A.w; h[r][2] = B.y; h[r][3] = B.w;
    }
    return;
  }
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint2 t = pos_of(r, k, j) < n ? ((const uint2*)v)[pos_of(r, k, j)] : make_uint2(0u, 0u);
      x[r][k] = t.x;
      h[r][k] = t.y;
    }
}

// Minimum of a uint64 block and whether it is written as FOR64 or as two
// sub-blocks (packUint64Scalar, uint64.go:302-333): FOR64 when !NoFOR, min > 0
// and max - min < 2^32, else the low words alone when every value fits 32
// bits, else low words then high words.
struct Shape64 {
  uint32_t mnl, mnh;
  bool for64, two;
};
__device__ __forceinline__ Shape64 shape64(const uint32_t (&x)[8][4], const uint32_t (&h)[8][4], int n, int flag,
                                           bool part, int j) {
  Shape64 s;
  const uint32_t mxh = q_max(max32(h));
  s.mnh = block_min(h, n, part, j);
  // low words of the minimum and the maximum, where the high words leave the
  // difference a chance to be below 2^32
  uint32_t mnl = 0xFFFFFFFFu, mxl = 0;
  if (__any_sync(kFull, n > 0 && mxh - s.mnh <= 1u)) {
#pragma unroll
    for (int r = 0; r < 8; r++)
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (!part || pos_of(r, k, j) < n) {
          if (h[r][k] == s.mnh) mnl = min(mnl, x[r][k]);
          if (h[r][k] == mxh) mxl = max(mxl, x[r][k]);
        }
    mnl = q_min(mnl);
    mxl = q_max(mxl);
  }
  s.mnl = mnl;
  const uint64_t mn = ((uint64_t)s.mnh << 32) | mnl, mx = ((uint64_t)mxh << 32) | mxl;
  s.for64 = n > 0 && !(flag & kNoFOR) && mxh - s.mnh <= 1u && mn > 0 && mx - mn < (1ull << 32);
  s.two = n > 0 && !s.for64 && mxh != 0;
  return s;
}

constexpr int kFor64Bit = 2 * kPlanBits, kTwoBit = kFor64Bit + 1;

template <bool DELTA, bool U64>
__global__ void __launch_bounds__(kThreads, U64 ? 4 : 6) pack_plan_kernel(PackArgs a, Sums sums) {
  __shared__ uint32_t s_len;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q = lane >> 2, j = lane & 3;
  const int64_t t = blockIdx.x, b0 = t * kTile + warp * 8, b = b0 + q;
  if (tid == 0) s_len = 0;
  asm volatile("griddepcontrol.launch_dependents;");
  uint64_t first = 0;
  const int n = block_of(a, b0, b, lane, &first);
  const bool part = __any_sync(kFull, n > 0 && n < kBlock);
  uint64_t plan;
  uint32_t len;
  if constexpr (U64) {
    uint32_t x[8][4], h[8][4];
    load_block64<false>((const uint64_t*)a.values + first, n, j, x, h);
    const Shape64 s = shape64(x, h, n, a.flag, part, j);
    uint32_t p_hi = 0;
    if (__any_sync(kFull, s.two)) p_hi = plan_sub<DELTA>(h, s.two ? n : 0, a.flag, false, 0, part, j);
    if (__any_sync(kFull, s.for64)) sub_rows(x, s.for64 ? s.mnl : 0u, n, part, j);
    const uint32_t p_lo = plan_sub<DELTA>(x, n, a.flag, s.for64, s.for64 ? 8 : s.two ? 2 : 0, part, j);
    plan = (uint64_t)p_lo | ((uint64_t)p_hi << kPlanBits) | ((uint64_t)s.for64 << kFor64Bit) |
           ((uint64_t)s.two << kTwoBit);
    len = (p_lo & kPlanLen) + (p_hi & kPlanLen);
  } else {
    uint32_t x[8][4];
    const uintptr_t lo = (uintptr_t)a.values + 4 * a.val_off[0], hi = (uintptr_t)a.values + 4 * a.val_off[a.n_streams];
    load_block<false>((const uint32_t*)a.values + first, n, lo, hi, j, lane, x);
    plan = plan_sub<DELTA>(x, n, a.flag, false, 0, part, j);
    len = (uint32_t)plan & kPlanLen;
  }
  if (j == 0 && n > 0) a.block_off[b] = plan;
  len = __reduce_add_sync(kFull, j == 0 ? len : 0u);
  __syncthreads();
  if (lane == 0) atomicAdd(&s_len, len);
  __syncthreads();
  if (tid == 0) {
    sums.one[t] = s_len;
    if (sums.g1024) {
      atomicAdd(&sums.g32[t >> 5], s_len);
      atomicAdd(&sums.g1024[t >> 10], (unsigned long long)s_len);
    }
  }
}

template <bool U64>
struct __align__(16) WriteSmem {
  static constexpr int kMaxLen = U64 ? 1048 : 520;  // bound of a block's bytes
  uint4 img[kWarps][(8 * kMaxLen + 32) / 16];
  uint4 slot[kWarps][8 * 33];  // a chunk between the blocks: the quads on different banks
};

template <bool DELTA, bool U64>
__global__ void __launch_bounds__(kThreads, U64 ? 4 : 6) pack_write_kernel(PackArgs a, Sums sums) {
  extern __shared__ uint4 smem4[];
  WriteSmem<U64>& S = *(WriteSmem<U64>*)smem4;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q = lane >> 2, j = lane & 3;
  const int64_t t = blockIdx.x, b0 = t * kTile + warp * 8;
  uint64_t first = 0;
  const int n = block_of(a, b0, b0 + q, lane, &first);
  const bool part = __any_sync(kFull, n > 0 && n < kBlock);
  uint32_t x[8][4], h[U64 ? 8 : 1][4];
  if constexpr (U64) {
    load_block64<true>((const uint64_t*)a.values + first, n, j, x, h);
  } else {
    const uintptr_t lo = (uintptr_t)a.values + 4 * a.val_off[0], hi = (uintptr_t)a.values + 4 * a.val_off[a.n_streams];
    load_block<true>((const uint32_t*)a.values + first, n, lo, hi, j, lane, x);
  }
  // Up to here nothing of the first launch was needed: this one starts before
  // that has ended (programmatic dependent launch) and waits for it here.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // the plans of the tile's blocks, a lane each, and the bytes before the tile
  const int64_t bl = t * kTile + lane;
  const uint64_t pl = bl < a.n_blocks ? a.block_off[bl] : 0ull;
  uint64_t before = 0;
  if (sums.g1024) {
    const int64_t t32 = t & ~(int64_t)31, t1024 = t & ~(int64_t)1023;
    if (t32 + lane < t) before = sums.one[t32 + lane];
    if (t1024 + 32 * lane < t32) before += sums.g32[(t1024 >> 5) + lane];
    for (int64_t g = lane; g < (t1024 >> 10); g += 32) before += sums.g1024[g];
  } else {
#pragma unroll 4
    for (int i = lane; i < (int)t; i += 32) before += sums.one[i];
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) before += shfl_xor64(before, d);
  const uint32_t len = ((uint32_t)pl & kPlanLen) + (U64 ? (uint32_t)(pl >> kPlanBits) & kPlanLen : 0u);
  const uint32_t incl = (uint32_t)warp_incl_scan((int)len, lane), excl = incl - len;
  __syncthreads();  // every warp has read the tile's plans
  if (warp == 0 && bl < a.n_blocks) {
    a.block_off[bl] = before + excl;
    if (bl == a.n_blocks - 1) {
      a.block_off[a.n_blocks] = before + incl;
      if (!U64 && a.stats) {  // for the next batch's route
        a.stats[0] = before + incl;
        a.stats[1] = (uint64_t)a.n_blocks;
      }
    }
  }
  const uint32_t w0 = __shfl_sync(kFull, excl, warp * 8), w1 = __shfl_sync(kFull, incl, warp * 8 + 7);
  const uint64_t g = before + w0;
  if (w1 == w0) return;
  if (before + w1 > a.out_cap) {
    if (lane == 0 && a.err) atomicOr(a.err, 1u << 9);
    return;
  }
  const uint32_t p0 = __shfl_sync(kFull, (uint32_t)pl, warp * 8 + q), p1 = __shfl_sync(kFull, (uint32_t)(pl >> 32), warp * 8 + q);
  const uint32_t off = __shfl_sync(kFull, excl, warp * 8 + q) - w0;
  uint8_t* dst = a.out + g;
  const int lead = (int)((uintptr_t)dst & 15);
  uint8_t* o = (uint8_t*)S.img[warp] + lead + off;
  uint4* slot = S.slot[warp] + 33 * q;
  const uint32_t special = (uint32_t)(a.flag & kSpecial) << 14;
  if constexpr (U64) {
    const uint64_t p = ((uint64_t)p1 << 32) | p0;
    const bool for64 = (p >> kFor64Bit) & 1u, two = (p >> kTwoBit) & 1u;
    Sub s;
    s.plan = p0 & kPlanMask;
    s.n = n;
    s.for64 = for64;
    s.base64 = 0;
    s.blk2 = two ? (int)((uint32_t)(p >> kPlanBits) & kPlanLen) : -1;
    s.hflags = kTypeU64 | special | (two ? kHdrCombine : 0u);
    if (__any_sync(kFull, for64)) {
      const Shape64 sh = shape64(x, h, n, a.flag, part, j);
      if (for64) s.base64 = ((uint64_t)sh.mnh << 32) | sh.mnl;
      sub_rows(x, for64 ? sh.mnl : 0u, n, part, j);  // the low 32 bits of x - min
    }
    write_sub<DELTA>(x, s, a.flag, part, o, slot, j, lane);
    if (__any_sync(kFull, two)) {
      Sub u;
      u.plan = two ? (uint32_t)(p >> kPlanBits) & kPlanMask : 0u;
      u.n = n;
      u.for64 = false;
      u.base64 = 0;
      u.blk2 = -1;
      u.hflags = kTypeU64 | special;
      write_sub<DELTA>(h, u, a.flag, part, o + (s.plan & kPlanLen), slot, j, lane);
    }
  } else {
    Sub s;
    s.plan = p0 & kPlanMask;
    s.n = n;
    s.for64 = false;
    s.base64 = 0;
    s.blk2 = -1;
    s.hflags = kTypeU32 | special;
    write_sub<DELTA>(x, s, a.flag, part, o, slot, j, lane);
  }
  // [lead, end) of the image to dst: whole 16-byte chunks by a bulk store,
  // the ragged ends a byte per lane
  const int end = lead + (int)(w1 - w0), c0 = (lead + 15) & ~15, c1 = end & ~15;
  const uint8_t* img = (const uint8_t*)S.img[warp];
  uint8_t* base = dst - lead;
  tma::proxy_fence();
  __syncwarp();
  if (c1 > c0 && lane == 0) {
    tma::bulk_store(base + c0, img + c0, (uint32_t)(c1 - c0));
    tma::bulk_commit();
  }
  const int e = lane & 15;
  if (lane < 16) {
    if (e >= lead && e < min(c0, end)) base[e] = img[e];
  } else if (max(c0, c1) + e < end) {
    base[max(c0, c1) + e] = img[max(c0, c1) + e];
  }
  if (lane == 0) tma::bulk_wait_all();
}

}  // namespace qp

namespace launch {

template <bool DELTA, bool U64>
static cudaError_t pack_attr() {
  const auto k = qp::pack_write_kernel<DELTA, U64>;
  const cudaError_t e =
      cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(qp::WriteSmem<U64>));
  if (e == cudaSuccess) cudaFuncSetAttribute((const void*)k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  return e;
}
cudaError_t pack_two_setup() {
  cudaError_t e;
  if ((e = pack_attr<false, false>()) != cudaSuccess) return e;
  if ((e = pack_attr<true, false>()) != cudaSuccess) return e;
  if ((e = pack_attr<false, true>()) != cudaSuccess) return e;
  return pack_attr<true, true>();
}

template <bool DELTA, bool U64>
static cudaError_t pack_run(const PackArgs& a, const qp::Sums& s, cudaStream_t st) {
  qp::pack_plan_kernel<DELTA, U64><<<(unsigned)a.n_tiles, qp::kThreads, 0, st>>>(a, s);
  cudaLaunchConfig_t c = {};
  cudaLaunchAttribute early;
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  c.gridDim = dim3((unsigned)a.n_tiles);
  c.blockDim = dim3(qp::kThreads);
  c.dynamicSmemBytes = sizeof(qp::WriteSmem<U64>);
  c.stream = st;
  c.attrs = &early;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, qp::pack_write_kernel<DELTA, U64>, a, s);
}

// Which batches take the two launches: uint64 ones of any size (2^26 values of
// three shapes 903 -> 489 us), and all others up to kSmallBlocks blocks, where
// the one-launch pack's warps, a tile of 32 blocks each, leave SMs idle: 2^20
// outlier values 16.4 -> 13.1 us, as many postings in 128 lists 36 -> 25 us.
// (The host pays for the second launch: 2^12 aligned values issued back to back
// by one thread 10.3 -> 11.4 us, where the call alone takes 22.9 -> 19.6 us and a
// graph of them 10.4 -> 4.3 us each.)
// Above, the one-launch pack reads the values once: 2^22 outlier values 20.0
// against 22.5 us, 2^28 495 against 627.  But its image holds a tile of blocks
// of up to kRoundBlock bytes each; a tile of larger ones takes several rounds.
// Only NoPatch data has such blocks as a rule, and only then: 2^27 values under
// NoPatch, one launch against two, in blocks of 132 bytes 168 us : 240, 196
// bytes 192 : 259, 260 bytes 352 : 257, 438 bytes 532 : 301.  So a large NoPatch
// batch goes by the mean block of the one before it, and by one launch while
// that is not known.
constexpr int64_t kSmallBlocks = 16384;
bool pack_by_two(bool u64, int flag, int64_t n_blocks, uint64_t mean) {
  return u64 || n_blocks <= kSmallBlocks || ((flag & kNoPatch) && mean > kRoundBlock);
}
bool pack_two_clears(int64_t n_blocks) { return n_blocks > (int64_t)qp::kDirectTiles * qp::kTile; }

cudaError_t pack_two(bool u64, const PackArgs& a_in, cudaStream_t st) {
  cudaError_t e;
  PackArgs a = a_in;
  a.n_tiles = (a.n_blocks + qp::kTile - 1) / qp::kTile;
  if (a.n_tiles > INT32_MAX || qp::sums_bytes(a.n_tiles) > pack_scratch_bytes(a.n_blocks)) return cudaErrorInvalidValue;
  const qp::Sums s = qp::sums_in(a.counter, a.n_tiles);
  const bool d = (a.flag & kDelta) != 0;
  if (u64) e = d ? pack_run<true, true>(a, s, st) : pack_run<false, true>(a, s, st);
  else e = d ? pack_run<true, false>(a, s, st) : pack_run<false, false>(a, s, st);
  note_launch(2);
  const cudaError_t last = cudaGetLastError();
  return e != cudaSuccess ? e : last;
}

}  // namespace launch
}  // namespace utl
