// utl_qpack.cuh -- batched UTL-PFOR pack of uint32 and uint64 blocks in two
// launches, four lanes per block.
//
// A warp works on eight consecutive blocks at once, a quad of lanes 4q..4q+3
// per block: lane j of the quad holds UTL lanes 4j..4j+3 of every row, so
// row r of the block is the 16-byte chunk 4r + j of its values.  Row-wise
// work (FOR, delta, zigzag, bit packing) stays in the thread; block-wide
// results cross the quad by two shuffles.
//
// Every decision and byte follows PackUint32 / PackUint64 (pack.go:76-97,
// scalar.go:126-235, uint64.go:124-333) as cited at each step.
#pragma once
#include "utl_device.cuh"
#include "utl_quad.cuh"
#include "utl_unpack.cuh"

namespace utl {
namespace qp {

// ---- quad primitives (lanes 4q..4q+3), whole warp converged ----
__device__ __forceinline__ uint32_t q_add(uint32_t x) {
  x += __shfl_xor_sync(kFull, x, 1);
  return x + __shfl_xor_sync(kFull, x, 2);
}
__device__ __forceinline__ uint32_t q_or(uint32_t x) {
  x |= __shfl_xor_sync(kFull, x, 1);
  return x | __shfl_xor_sync(kFull, x, 2);
}
__device__ __forceinline__ uint32_t q_min(uint32_t x) {
  x = min(x, __shfl_xor_sync(kFull, x, 1));
  return min(x, __shfl_xor_sync(kFull, x, 2));
}
__device__ __forceinline__ uint32_t q_max(uint32_t x) {
  x = max(x, __shfl_xor_sync(kFull, x, 1));
  return max(x, __shfl_xor_sync(kFull, x, 2));
}
// exclusive prefix over the quad's lanes j = 0..3
__device__ __forceinline__ uint32_t q_excl(uint32_t x, int j) {
  uint32_t t = x;
  uint32_t y = __shfl_up_sync(kFull, t, 1);
  if (j >= 1) t += y;
  y = __shfl_up_sync(kFull, t, 2);
  if (j >= 2) t += y;
  return t - x;
}
__device__ __forceinline__ uint32_t min32(const uint32_t (&x)[8][4]) {
  uint32_t m = x[0][0];
#pragma unroll
  for (int r = 0; r < 8; r++) {
    m = __vimin3_u32(m, x[r][0], x[r][1]);
    m = __vimin3_u32(m, x[r][2], x[r][3]);
  }
  return m;
}
__device__ __forceinline__ uint32_t max32(const uint32_t (&x)[8][4]) {
  uint32_t m = x[0][0];
#pragma unroll
  for (int r = 0; r < 8; r++) {
    m = __vimax3_u32(m, x[r][0], x[r][1]);
    m = __vimax3_u32(m, x[r][2], x[r][3]);
  }
  return m;
}

// Counts of the block's values by bucket clz/4, quad-wide (bytes: E buckets
// 0,2,4,6, O buckets 1,3,5,7; zeros drop out), as bytes 0..3 / 4..7.
struct Counts {
  uint32_t b03, b47;
};
__device__ __forceinline__ Counts counts(const uint32_t (&x)[8][4]) {
  uint32_t E, O;
  quad::bucket_hist(x, E, O);
  E = q_add(E);
  O = q_add(O);
  return Counts{__byte_perm(E, O, 0x5140), __byte_perm(E, O, 0x7362)};
}
// exc[si] in byte si: values wider than 4*si bits (select_bitwidth.go:46-72).
__device__ __forceinline__ uint64_t exc_counts(const Counts& c) {
  const uint32_t p03 = c.b03 * 0x01010101u;
  const uint32_t p47 = c.b47 * 0x01010101u + (p03 >> 24) * 0x01010101u;
  return ((uint64_t)__byte_perm(p03, 0, 0x0123) << 32) | __byte_perm(p47, 0, 0x0123);
}
// Steps the widest value takes: the non-zero bytes of exc form a prefix.
__device__ __forceinline__ int max_step(uint64_t e) {
  const uint32_t lo = (uint32_t)e, hi = (uint32_t)(e >> 32);
  return hi ? 4 + ((39 - __clz(hi)) >> 3) : (39 - __clz(lo)) >> 3;
}
// Width choice of chooseBestFromExcCounts (select_bitwidth.go:56-121), two
// steps per quad lane: lane j costs steps j and j + 4, and the quad takes
// the least (cost, then the wider step: the reference walks down from the
// widest and replaces only on a strictly lower cost).  Returns the step.
__device__ __forceinline__ int choose_step(uint64_t e, int j) {
  const int ms = max_step(e);
  uint32_t key = ((uint32_t)(4 + 64 * ms) << 4) | (uint32_t)(8 - ms);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int si = j + 4 * h;
    const int c = (int)(((h ? (uint32_t)(e >> 32) : (uint32_t)e) >> (8 * j)) & 0xFFu);
    const int cost = 6 + 64 * si + min(c, 16) + ((c + 3) >> 2) + c * ((ms - si + 1) >> 1);
    const uint32_t k = ((uint32_t)cost << 4) | (uint32_t)(8 - si);
    if (si < ms) key = min(key, k);
  }
  return 8 - (int)(q_min(key) & 15u);
}
// StreamVByte data bytes at width 4*s: a value of bucket b has
// ceil((32 - 4b - 4s) / 8) high-part bytes, which is entry b + s of the
// table {4,4,3,3,2,2,1,1} (zero past it).
__device__ __forceinline__ int svb_bytes(const Counts& c, int s) {
  const uint64_t w = quad::shr64_clamp(0x0101020203030404ull, (uint32_t)(8 * s));
  return (int)__dp4a(c.b47, (uint32_t)(w >> 32), __dp4a(c.b03, (uint32_t)w, 0u));
}

// Position of x[r][k] in its block.
__device__ __forceinline__ int pos_of(int r, int k, int j) { return 16 * r + 4 * j + k; }

__device__ __forceinline__ void zero_padding(uint32_t (&x)[8][4], int n, int j) {
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (pos_of(r, k, j) >= n) x[r][k] = 0u;
}
// Minimum of the block's values (n of them when part).
__device__ __forceinline__ uint32_t block_min(const uint32_t (&x)[8][4], int n, bool part, int j) {
  uint32_t m = 0xFFFFFFFFu;
  if (part) {
#pragma unroll
    for (int r = 0; r < 8; r++)
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (pos_of(r, k, j) < n) m = min(m, x[r][k]);
  } else {
    m = min32(x);
  }
  return q_min(m);
}
__device__ __forceinline__ int for_width(uint32_t base) {  // width code of a FOR base (for.go:95-126)
  const int nb = (len32(base) + 7) >> 3;
  return nb >= 3 ? 3 : nb;
}

// Per-lane delta of the block's values down the rows (delta.go:23-48; the FOR
// base cancels below row 0); returns whether any difference borrowed.
// Padding deltas are zero (scalar.go:34-40).
__device__ __forceinline__ bool delta_rows(uint32_t (&x)[8][4], int n, uint32_t base, bool part, int j) {
  if (part) {  // repeat the value one row up
#pragma unroll
    for (int r = 0; r < 8; r++)
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (pos_of(r, k, j) >= n) x[r][k] = r > 0 ? x[r > 0 ? r - 1 : 0][k] : base;
  }
  bool borrow = false;
#pragma unroll
  for (int r = 7; r >= 1; r--)
#pragma unroll
    for (int k = 0; k < 4; k++) {
      borrow |= x[r][k] < x[r - 1][k];
      x[r][k] -= x[r - 1][k];
    }
#pragma unroll
  for (int k = 0; k < 4; k++) x[0][k] -= base;
  return borrow;
}
__device__ __forceinline__ void zigzag_rows(uint32_t (&x)[8][4], bool zz) {
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int k = 0; k < 4; k++) x[r][k] = zz ? zz_enc(x[r][k]) : x[r][k];
}
__device__ __forceinline__ void sub_rows(uint32_t (&x)[8][4], uint32_t base, int n, bool part, int j) {
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int k = 0; k < 4; k++) x[r][k] -= base;
  if (part) zero_padding(x, n, j);
}

// A planned sub-block in 25 bits: length (11), width step (4), exceptions
// (8), zigzag, FOR.  The FOR base is found again by the writer.
__device__ __forceinline__ uint32_t plan_word(int len, int step, int exc, bool zz, bool use_for) {
  return (uint32_t)len | ((uint32_t)step << 11) | ((uint32_t)exc << 15) | (zz ? 1u << 23 : 0u) |
         (use_for ? 1u << 24 : 0u);
}
constexpr int kPlanBits = 25;
constexpr uint32_t kPlanMask = (1u << kPlanBits) - 1u, kPlanLen = 2047u;

// Decide the sub-block in x (n values, zero past them; n = 0: nothing), in
// the steps of scalar.go:126-235: FOR (for.go:95-126), delta and zigzag
// (delta.go:23-48), width and exceptions (select_bitwidth.go:20-121),
// StreamVByte length (svb.go).  extra: header bytes beside the FOR base
// (block2Len, FOR64 base).  part: some quad's block is partial (warp-uniform).
// x is used up.  Whole warp; returns the plan word, quad-uniform.
template <bool DELTA>
__device__ __forceinline__ uint32_t plan_sub(uint32_t (&x)[8][4], int n, int flag, bool for_off, int extra, bool part,
                                             int j) {
  uint32_t base = 0, mx = 0;
  bool use_for = false, have = false;
  Counts c{0u, 0u};
  if (!DELTA) {
    c = counts(x);
    have = true;
  }
  const bool want_for = !(flag & kNoFOR) && !for_off && n > 0;
  if (__any_sync(kFull, want_for)) {
    const uint32_t mn = block_min(x, n, part, j);
    mx = q_max(max32(x));
    const int for_max = round_step(len32(mx - mn));
    const bool cand = want_for && mn != 0 && for_max < round_step(len32(mx));
    if (__any_sync(kFull, cand)) {
      if (!have) c = counts(x);
      const int std_w = 4 * choose_step(exc_counts(c), j);  // whole warp
      use_for = cand && for_max < std_w;
      base = use_for ? mn : 0u;
    }
  }
  // a constant block under FOR: every work value is zero
  const bool flat = !DELTA && use_for && mx == base;
  bool zz = false;
  if (DELTA) {
    zz = q_or(delta_rows(x, n, base, part, j) ? 1u : 0u) != 0;
    if (__any_sync(kFull, zz)) zigzag_rows(x, zz);
    c = counts(x);
  } else if (__any_sync(kFull, use_for && !flat)) {
    sub_rows(x, base, n, part, j);
    c = counts(x);
  }
  if (flat) c.b03 = c.b47 = 0u;
  const uint64_t e = exc_counts(c);
  int step, exc = 0;
  if (flag & kNoPatch) {
    step = max_step(e);
  } else {
    step = choose_step(e, j);
    exc = (int)(quad::shr64_clamp(e, (uint32_t)(8 * step)) & 0xFFu);
  }
  const int forb = use_for ? ((1 << for_width(base)) >> 1) : 0;
  int len = 4 + extra + forb + 64 * step;
  if (exc) len += 2 + min(exc, 16) + ((exc + 3) >> 2) + svb_bytes(c, step);
  return n > 0 ? plan_word(len, step, exc, zz, use_for) : 0u;
}

// ---- the writer ----
__device__ __forceinline__ void put4(uint8_t* p, uint32_t v, int nb) {
  if (nb > 0) p[0] = (uint8_t)v;
  if (nb > 1) p[1] = (uint8_t)(v >> 8);
  if (nb > 2) p[2] = (uint8_t)(v >> 16);
  if (nb > 3) p[3] = (uint8_t)(v >> 24);
}
// One word row of the payload: lane j's four words end the aligned words
// aw[16w + 4j ..]; the bytes in front of them come from the lane before
// (lane 3 of the previous row for j = 0; the header for row 0).
struct Row {
  uint32_t* aw;   // the aligned word the lane's first payload byte falls in
  int sh;         // 8 * (bytes of that word in front of it)
  uint32_t last;  // lane 3: its last word of the previous row
  int src;        // the lane before
  int j;
  unsigned qm;
};
__device__ __forceinline__ void put_row(Row& w, int i, uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3) {
  const uint32_t prev = __shfl_sync(w.qm, w.j == 3 ? w.last : c3, w.src);
  uint32_t* a = w.aw + 16 * i;
  a[0] = __funnelshift_l(prev, c0, w.sh);
  a[1] = __funnelshift_l(c0, c1, w.sh);
  a[2] = __funnelshift_l(c1, c2, w.sh);
  a[3] = __funnelshift_l(c2, c3, w.sh);
  w.last = c3;
}

// UTL payload (scalar.go:7-59) of the quad's block at width bw (quad-uniform).
__device__ __forceinline__ void put_payload(const uint32_t (&x)[8][4], int bw, Row w) {
  if (bw == 8) {
    // words are the low bytes of four consecutive rows
#pragma unroll
    for (int i = 0; i < 2; i++) {
      uint32_t c[4];
#pragma unroll
      for (int k = 0; k < 4; k++)
        c[k] = __byte_perm(__byte_perm(x[4 * i][k], x[4 * i + 1][k], 0x0040),
                           __byte_perm(x[4 * i + 2][k], x[4 * i + 3][k], 0x0040), 0x5410);
      put_row(w, i, c[0], c[1], c[2], c[3]);
    }
  } else if (bw == 16) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      uint32_t c[4];
#pragma unroll
      for (int k = 0; k < 4; k++) c[k] = __byte_perm(x[2 * i][k], x[2 * i + 1][k], 0x5410);
      put_row(w, i, c[0], c[1], c[2], c[3]);
    }
  } else if (bw > 0) {
    // any width: a word row is complete when a row of values reaches its end
    const uint32_t mask = bw >= 32 ? 0xFFFFFFFFu : ((1u << bw) - 1u);
    uint32_t acc[4] = {0, 0, 0, 0};
    int pos = 0, i = 0;
#pragma unroll
    for (int r = 0; r < 8; r++) {
      uint32_t m[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        m[k] = x[r][k] & mask;
        acc[k] |= m[k] << pos;
      }
      pos += bw;
      if (pos >= 32) {
        put_row(w, i, acc[0], acc[1], acc[2], acc[3]);
        i++;
        pos -= 32;
#pragma unroll
        for (int k = 0; k < 4; k++) acc[k] = pos ? m[k] >> (bw - pos) : 0u;
      }
    }
  }
  // the last word's bytes past the last aligned word
  if (bw > 0 && w.j == 3) put4((uint8_t*)(w.aw + 4 * bw + 4 - 16), w.last >> ((32 - w.sh) & 31), w.sh >> 3);
}

// Exceptions (exceptions.go:138-186): index and StreamVByte bytes at xi.
// Lane j codes the exceptions of rows 2j and 2j + 1 (positions 32j..32j+31),
// so the lanes' exceptions follow each other in position order.  slot: the
// block's work values.  Whole warp; exc = 0 for quads without any.
__device__ __forceinline__ void put_exceptions(const uint32_t (&x)[8][4], const uint32_t* slot, int bw, int exc,
                                               uint8_t* xi, int j, int lane) {
  const uint32_t mask = exc ? (1u << bw) - 1u : 0xFFFFFFFFu;  // bw < 32 with exceptions
  uint32_t m = 0;
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (x[r][k] > mask) m |= 1u << (4 * r + k);
  // rows 2p, 2p+1 of this lane as their bits of bitmap word p; lane j
  // collects word j from the quad
  uint32_t o[4];
#pragma unroll
  for (int p = 0; p < 4; p++) {
    const uint32_t u = m >> (8 * p);
    o[p] = ((u & 0xFu) | ((u & 0xF0u) << 12)) << (4 * j);
  }
  const bool b1 = (j & 2) != 0, b0 = (j & 1) != 0;
  uint32_t k0 = b1 ? o[2] : o[0], k1 = b1 ? o[3] : o[1];
  k0 |= __shfl_xor_sync(kFull, b1 ? o[0] : o[2], 2);
  k1 |= __shfl_xor_sync(kFull, b1 ? o[1] : o[3], 2);
  const uint32_t W = (b0 ? k1 : k0) | __shfl_xor_sync(kFull, b0 ? k0 : k1, 1);
  const int first = (int)q_excl((uint32_t)__popc(W), j);
  const bool list = exc <= 16;
  const int nc = (exc + 3) >> 2;
  uint8_t* svb = xi + min(exc, 16);
  if (!list) {
    put4(xi + 4 * j, W, 4);
    for (int g = j; g < nc; g += 4) svb[g] = 0;
  }
  __syncwarp();
  // The codes.  With more than 16 exceptions the lanes share control bytes and
  // OR their codes into the aligned word.  That word may reach into the bitmap
  // before and the data after (never out of the block's own bytes: there are 16
  // bytes of bitmap and at least 17 of data), so both are written on the other
  // side of a barrier: an atomic leaves no order between itself and a plain
  // store to its word.
  uint32_t ctrl = 0;
  int tot = 0, rank = first;
  for (uint32_t b = W; b; b &= b - 1, rank++) {
    const int pos = 32 * j + __ffs(b) - 1;
    const int code = (31 - __clz(slot[pos] >> bw)) >> 3;  // StreamVByte length - 1
    if (list) {
      xi[rank] = (uint8_t)pos;
      ctrl |= (uint32_t)code << (2 * rank);
    } else if (code) {
      const uintptr_t g = (uintptr_t)(svb + (rank >> 2));
      atomicOr((uint32_t*)(g & ~(uintptr_t)3), (uint32_t)code << (8 * (int)(g & 3) + 2 * (rank & 3)));
    }
    tot += code + 1;
  }
  int d = nc + (int)q_excl((uint32_t)tot, j);
  ctrl = q_or(ctrl);
  if (list && j < nc) svb[j] = (uint8_t)(ctrl >> (8 * j));
  __syncwarp();
  for (uint32_t b = W; b; b &= b - 1) {
    const uint32_t hv = slot[32 * j + __ffs(b) - 1] >> bw;
    const int code = (31 - __clz(hv)) >> 3;
    uint8_t* p = svb + d;
    p[0] = (uint8_t)hv;
    if (code > 0) p[1] = (uint8_t)(hv >> 8);
    if (code > 1) p[2] = (uint8_t)(hv >> 16);
    if (code > 2) p[3] = (uint8_t)(hv >> 24);
    d += code + 1;
  }
}

// A sub-block's place and shape for the writer (quad-uniform).
struct Sub {
  uint32_t plan;   // plan word (0: none)
  uint32_t hflags; // header bits beside count, width, exceptions, FOR and delta
  int n;
  int blk2;        // block2Len, -1: no such field
  bool for64;
  uint64_t base64;
};
// Write the sub-block whose values are in x at o (shared memory).  x becomes
// the work values.  slot4: 32 chunks of scratch, the block's own.
template <bool DELTA>
__device__ __forceinline__ void write_sub(uint32_t (&x)[8][4], const Sub& s, int flag, bool part, uint8_t* o,
                                          uint4* slot4, int j, int lane) {
  const int len = (int)(s.plan & kPlanLen), bw = 4 * (int)((s.plan >> 11) & 15u), exc = (int)((s.plan >> 15) & 0xFFu);
  const bool zz = (s.plan >> 23) & 1u, use_for = (s.plan >> 24) & 1u;
  uint32_t base = 0;
  if (__any_sync(kFull, use_for)) {
    const uint32_t m = block_min(x, s.n, part, j);
    base = use_for ? m : 0u;
  }
  if (DELTA) {
    delta_rows(x, s.n, base, part, j);
    if (__any_sync(kFull, zz)) zigzag_rows(x, zz);
  } else if (__any_sync(kFull, use_for && (bw || exc))) {
    sub_rows(x, base, s.n, part, j);
  }
  const int fw = for_width(base);
  const int forb = s.for64 ? 8 : (use_for ? ((1 << fw) >> 1) : 0);
  const int p_off = 4 + (exc ? 2 : 0) + forb + (s.blk2 >= 0 ? 2 : 0);
  // header bytes (header.go:102, uint64.go:124-157): the word, StreamVByte
  // length, FOR base, block2Len
  uint32_t h[4];
  {
    uint64_t t = s.for64 ? s.base64 : (uint64_t)base;
    if (s.blk2 >= 0) t |= (uint64_t)(uint32_t)s.blk2 << (8 * forb);
    h[0] = (uint32_t)s.n | ((uint32_t)bw << 6) | s.hflags | ((uint32_t)exc << 24) |
           ((uint32_t)(s.for64 ? 3 : use_for ? fw : 0) << 15) | (DELTA ? kHdrDelta | (zz ? kHdrZigZag : 0u) : 0u);
    h[1] = (uint32_t)t;
    h[2] = (uint32_t)(t >> 32);
    h[3] = 0;
    if (exc) {
      h[3] = h[2] >> 16;
      h[2] = __funnelshift_l(h[1], h[2], 16);
      h[1] = (h[1] << 16) | (uint32_t)(len - p_off - 16 * bw - min(exc, 16));
    }
  }
  const bool any_exc = __any_sync(kFull, exc > 0);
  if (any_exc) {
#pragma unroll
    for (int r = 0; r < 8; r++) slot4[4 * r + j] = make_uint4(x[r][0], x[r][1], x[r][2], x[r][3]);
    __syncwarp();
    put_exceptions(x, (const uint32_t*)slot4, bw, exc, o + p_off + 16 * bw, j, lane);
    __syncwarp();
  }
  if (len > 0) {
    put4(o + 4 * j, j == 0 ? h[0] : j == 1 ? h[1] : j == 2 ? h[2] : h[3], p_off - 4 * j);
    uint8_t* pay = o + p_off;
    const int b = p_off - 4;  // the four bytes in front of the payload
    const uint32_t lo = b < 4 ? h[0] : b < 8 ? h[1] : h[2], hi = b < 4 ? h[1] : b < 8 ? h[2] : h[3];
    Row w;
    const int d = (int)((uintptr_t)pay & 3);
    w.aw = (uint32_t*)(pay - d) + 4 * j;
    w.sh = 8 * d;
    w.last = __funnelshift_r(lo, hi, (b & 3) * 8);
    w.src = (lane & 28) | ((lane + 3) & 3);
    w.j = j;
    w.qm = 0xFu << (lane & 28);
    put_payload(x, bw, w);
  }
  __syncwarp();
}

}  // namespace qp
}  // namespace utl
