// utl_get.cu -- batched GetUint32 / GetUint64: a thread per query.
//
// A query is a chain of dependent loads (stream table, block offsets, header,
// payload) on a block that is rarely in a cache, so it is bound by latency and
// by the sectors it touches.  Nearly every query takes the direct path
// (direct_get): whole words of a block that lies inside the buffer, the header
// first, then at once all payload words of the position's lane it needs.  Blocks that fail a check and
// forms the direct path leaves out (deep positions of plain delta blocks and of
// delta blocks with exceptions) take the general path, which reads
// byte by byte within bounds and reports the reference's exact status; whole
// unpacks the reference makes there are done by the warp.
//
// Measured, 2^20 random queries: 1000 delta lists of 10^8 values 159 -> 76 us;
// uint64 streams of three shapes 130 -> 85 us (flag 0), 845 -> 711 us (Delta);
// 2^26 outlier values 51 -> 49 us; 2^20 11-bit values, all in L2, 20 us as
// before.  64 registers (four CTAs on an SM): at 48 the lists take 71 us but
// the spills cost the plain queries 10%.
#include <cuda_runtime.h>
#include <stdint.h>

#include "utl_get.cuh"
#include "utl_launch.h"
#include "utl_quad.cuh"

namespace utl {

constexpr int kGThreads = 256;

// The 32 bits at a, read as the one or two whole words that hold them: up to
// three bytes before a and three after its last are read with them.
__device__ __forceinline__ uint32_t ld_word(const uint8_t* a) {
  const uintptr_t x = (uintptr_t)a;
  const uint32_t* w = (const uint32_t*)(x & ~(uintptr_t)3);
  const int sh = (int)(x & 3) * 8;
  uint32_t hi = 0;
  if (sh) hi = __ldg(w + 1);
  return __funnelshift_r(__ldg(w), hi, sh);
}

// The nb (1..4) bytes at p + off of a block of len bytes; near its end byte by
// byte, so that nothing after the block is read.
__device__ __forceinline__ uint32_t ld_bytes(const uint8_t* p, int off, int nb, int len) {
  uint32_t v = 0;
  if (off + 7 <= len) {
    v = ld_word(p + off);
  } else {
    for (int i = 0; i < nb; i++) v |= (uint32_t)p[off + i] << (8 * i);
  }
  return nb >= 4 ? v : v & ((1u << (8 * nb)) - 1u);
}

// The StreamVByte values of a block's exceptions, asked for in ascending rank
// (svb.go:40-100): the control words (16 codes each) are read as they are
// reached.
struct Svb {
  const uint8_t* p;  // the block
  int ctl, nc, end;  // offset and number of control bytes, block end
  int word, acc;     // control word held, data bytes of the words before it
  uint32_t codes;
  __device__ __forceinline__ void open(const uint8_t* block, int at, int exc, int block_end) {
    p = block;
    ctl = at;
    nc = (exc + 3) >> 2;
    end = block_end;
    word = -1;
    acc = 0;
    codes = 0;
  }
  // The value of the given rank; false if its data runs past the block.
  __device__ __forceinline__ bool value(int rank, uint32_t& v) {
    while (word < (rank >> 4)) {
      if (word >= 0) acc += 16 + quad::sum2bit(codes);
      word++;
      codes = 0;
      if (4 * word < nc) codes = ld_bytes(p, ctl + 4 * word, min(4, nc - 4 * word), end);
    }
    const int k = rank & 15, code = (int)((codes >> (2 * k)) & 3u);
    const int at = ctl + nc + acc + k + quad::sum2bit(codes & ((1u << (2 * k)) - 1u));
    if (at + code + 1 > end) return false;
    v = ld_bytes(p, at, code + 1, end);
    return true;
  }
};

// The packed value of a row of the UTL lane whose word i is at w + 64 i
// (get.go:34-67).
__device__ __forceinline__ uint32_t row_value(const uint8_t* w, int row, int bw, uint32_t mask) {
  if (bw == 0) return 0u;
  const int bit = row * bw, s = bit & 31;
  const uint8_t* q = w + 64 * (bit >> 5);
  uint32_t hi = 0;
  if (s + bw > 32) hi = ld_word(q + 64);
  return __funnelshift_r(ld_word(q), hi, s) & mask;
}

// Whether the whole words of the bytes up to a reach past the buffer's end hi.
__device__ __forceinline__ bool past(uintptr_t a, uintptr_t hi) { return ((a + 3) & ~(uintptr_t)3) > hi; }

// getUint32Scalar (get.go:81-190) for position pos of the block at p (len
// bytes, inside the buffer) where it succeeds without a whole unpack; false
// otherwise.  lo, hi: the buffer's first whole word and its end.  Whole words
// can reach out of the buffer in its first block, by the header, and in its
// last one, by what ends it: the header or a base alone, or the last UTL lane's
// last word (`risk`).  (Leaving that block to the general path altogether made
// two thirds of the warps run both paths when a buffer holds 32 blocks: 2^20
// queries on 4096 uint32 values 23.3 us, 15.8 by the general path alone, 14.2
// so; the checks cost uint64 queries some 3%.)
struct Direct {
  uint32_t h, value;  // header, result
  int p_off, end;     // payload offset, block end
};
__device__ __forceinline__ bool direct_get(const uint8_t* p, int len, int pos, bool for_u64, uintptr_t lo, uintptr_t hi,
                                           Direct& d) {
  if (len < 4) return false;
  uint32_t h;
  if ((uintptr_t)p < lo || past((uintptr_t)p + 4, hi))
    h = (uint32_t)p[0] | ((uint32_t)p[1] << 8) | ((uint32_t)p[2] << 16) | ((uint32_t)p[3] << 24);
  else
    h = ld_word(p);
  d.h = h;
  const int count = (int)(h & 0xFFu), bwf = (int)((h >> 8) & 31u), type = (int)((h >> 13) & 3u);
  const int forw = (int)((h >> 15) & 3u), exc = (int)(h >> 24), bw = 4 * bwf;
  const bool delta = (h & kHdrDelta) != 0, zz = (h & kHdrZigZag) != 0;
  const bool combine = for_u64 && (h & kHdrCombine);
  if (for_u64 ? type != 3 : (type != 1 && type != 2)) return false;
  const int row = pos >> 4, lane = pos & 15;
  if (pos >= count || bwf > 8 || exc > count) return false;
  if (delta && (!zz || exc) && row > delta_full_unpack_threshold(bw)) return false;
  const bool u64s = for_u64 && forw == 3 && !combine;
  const int fo = 4 + (exc ? 2 : 0), forb = u64s ? 8 : ((1 << forw) >> 1), isz = min(exc, 16);
  const int p_off = fo + forb + (combine ? 2 : 0), xs = p_off + 16 * bw;
  int end = xs;
  if (len < end) return false;
  if (exc) {
    if (len < 6) return false;
    const int svb_len = (int)ld_bytes(p, 4, 2, len);
    if (svb_len < ((exc + 3) >> 2)) return false;
    end += isz + svb_len;
    if (len < end) return false;
  }
  const bool risk = lane == 15 && bw && past((uintptr_t)p + (uintptr_t)xs, hi);
  if (risk && (delta || for_u64)) return false;
  d.p_off = p_off;
  d.end = end;
  uint32_t base = 0;
  if (!u64s) {
    if (forw == 3) {
      if (past((uintptr_t)p + (uintptr_t)fo + 4, hi)) return false;
      base = ld_word(p + fo);
    }
    else if (forw) base = (uint32_t)p[fo] | (forw == 2 ? (uint32_t)p[fo + 1] << 8 : 0u);
  }
  const uint8_t* w = p + p_off + 4 * lane;  // word i of the lane at w + 64 i
  const uint32_t mask = bwf >= 8 ? 0xFFFFFFFFu : ((1u << bw) - 1u);
  const bool list = exc <= 16;
  Svb svb;
  svb.open(p, xs + isz, exc, end);
  uint32_t v = 0;
  if (!delta) {
    if (!for_u64 && risk) {
      const int bit = row * bw, s = bit & 31, at = p_off + 4 * lane + 64 * (bit >> 5);
      uint32_t up = 0;
      if (s + bw > 32) up = ld_bytes(p, at + 64, 4, end);
      v = __funnelshift_r(ld_bytes(p, at, 4, end), up, s) & mask;
    } else {
      v = row_value(w, row, bw, mask);
    }
    if (exc) {
      // findExceptionIndex, exceptions.go:293-325 (a list ends at the first
      // larger position)
      int ei = -1;
      if (list) {
        for (int i = 0; i < exc; i++) {
          const int x = (int)p[xs + i];
          if (x >= pos) {
            if (x == pos) ei = i;
            break;
          }
        }
      } else if ((p[xs + (pos >> 3)] >> (pos & 7)) & 1) {
        ei = bitmap_rank128(GlobalBytes{p, end}, xs, 16, pos >> 3, pos & 7);
      }
      if (ei >= exc) return false;
      uint32_t hv = 0;
      if (ei >= 0 && !svb.value(ei, hv)) return false;
      v |= shl32(hv, bw);
    }
  } else {
    // getValueWithDelta, get.go:250-285: the lane's words up to the row's
    // last bit, all loads out together
    const int nw = ((row + 1) * bw + 31) >> 5;
    uint32_t r[8];
#pragma unroll
    for (int i = 0; i < 8; i++) r[i] = i < nw ? ld_word(w + 64 * i) : 0u;
    // their values, word after word (a row's value starts in word i and may
    // end in the next)
    int k = 0, s = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint32_t next = i < 7 ? r[i < 7 ? i + 1 : 7] : 0u;
      for (; s < 32 && k <= row; s += bw, k++) {
        const uint32_t x = __funnelshift_r(r[i], next, s) & mask;
        v += zz ? zz_dec(x) : x;
        if (bw == 0) k = row;  // all rows are zero
      }
      s -= 32;
    }
    if (exc) {
      // applyLaneExceptions, get.go:297-334: the lane's exceptions up to the
      // row, each by what its high part changes in the sum.  A list out of
      // order, or data that runs past the block, is left to the general path.
      // First which exceptions those are (a list: bit i of m for entry i; a
      // bitmap: bit k for row k), then their values: the queries of a warp
      // run the costly part together.
      uint32_t e[4], m = 0;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int nb = list ? min(4, exc - 4 * i) : 4;
        e[i] = nb > 0 ? ld_bytes(p, xs + 4 * i, nb, end) : 0u;
        if (list) {
          // entries of this UTL lane: their low nibble is it
          const uint32_t t = (e[i] & 0x0F0F0F0Fu) ^ ((uint32_t)lane * 0x01010101u);
          uint32_t z = ~(t + 0x7F7F7F7Fu) & 0x80808080u;
          if (nb < 4) z &= nb > 0 ? (1u << (8 * nb)) - 1u : 0u;
          m |= (((z >> 7) * 0x10204080u) >> 28) << (4 * i);
        } else {
          m |= (((e[i] >> lane) & 1u) | (((e[i] >> (16 + lane)) & 1u) << 1)) << (2 * i);
        }
      }
      if (!list) m &= (2u << row) - 1u;
      int last = -1;
      for (; m; m &= m - 1) {
        const int i = __ffs(m) - 1;
        int at, rank = i;
        if (list) {
          const uint32_t q = i < 8 ? (i < 4 ? e[0] : e[1]) : (i < 12 ? e[2] : e[3]);
          const int x = (int)((q >> (8 * (i & 3))) & 0xFFu);
          if (x > pos) break;  // the reference looks no further
          if (x <= last) return false;
          last = x;
          at = x >> 4;
        } else {
          at = i;
          rank = i > 1 ? __popc(e[0]) : 0;
          if (i > 3) rank += __popc(e[1]);
          if (i > 5) rank += __popc(e[2]);
          const uint32_t q = i < 4 ? (i < 2 ? e[0] : e[1]) : (i < 6 ? e[2] : e[3]);
          rank += __popc(q & ((1u << (16 * (i & 1) + lane)) - 1u));
          if (rank >= exc) return false;
        }
        uint32_t hv;
        if (!svb.value(rank, hv)) return false;
        hv = shl32(hv, bw);
        if (zz) {
          const uint32_t x = row_value(w, at, bw, mask);
          hv = zz_dec(x | hv) - zz_dec(x);
        }
        v += hv;
      }
    }
  }
  d.value = v + base;
  return true;
}

// Where query q's position lies; false when it is outside its stream.
__device__ __forceinline__ bool locate(const GetArgs& a, int64_t q, SubGet& sg) {
  const uint32_t s = a.q_stream[q];
  const uint64_t p = a.q_pos[q];
  if (s >= (uint32_t)a.n_streams || p >= a.val_off[s + 1] - a.val_off[s]) return false;
  const int64_t b = (int64_t)a.block_start[s] + (int64_t)(p / kBlock);
  const uint64_t off = a.block_off[b], end = a.block_off[b + 1];
  const uint64_t e2 = min(end, a.packed_len);
  const int64_t rd = (e2 > off) ? (int64_t)(e2 - off) : 0;
  sg = SubGet{a.packed + off, rd, (end >= off) ? (int64_t)(end - off) : 0, (int)(p % kBlock)};
  return true;
}

template <bool U64>
__device__ __forceinline__ void answer(const GetArgs& a, int64_t q, int status, int ovf, uint64_t result) {
  if (U64) ((uint64_t*)a.out)[q] = status == kOK ? result : 0ull;
  else ((uint32_t*)a.out)[q] = status == kOK ? (uint32_t)result : 0u;
  if (a.status) a.status[q] = status | (ovf << 8);
  if (status != kOK && a.err) atomicOr(a.err, 1u << status);
}

// The general path, for the lanes of a warp that need it (whole warp).  It
// starts again from the query: nothing is kept across the direct path for it,
// where it would cost every query registers.  hb: 128 words of the warp's own.
template <bool U64>
__device__ __noinline__ void get_general(const GetArgs& a, bool live, uint32_t* hb) {
  const int lane = threadIdx.x & 31;
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  SubGet sg{nullptr, 0, 0, 0};
  if (live) locate(a, q, sg);
  int status = kOK, ovf = 0;
  uint64_t result = 0;
  if (!U64) {
    GetResult r{kOK, 0, 0u, false};
    if (live) r = thread_get_u32(GlobalBytes{sg.p, sg.rd}, sg.len, sg.pos, false);
    resolve_full<false>(live, sg, r, hb, lane);
    if (live) {
      status = r.status;
      ovf = r.ovf;
      result = r.value;
    }
  } else {
    // getUint64Scalar, uint64.go:372-436
    const GlobalBytes g{sg.p, sg.rd};
    uint32_t h = 0;
    bool go = live;
    if (go) {
      if (sg.len < 4) { status = kErrInvalidBuffer; go = false; }
      else {
        h = g.u32(0);
        if (((h >> 13) & 3) != 3) { status = kErrUnsupportedType; go = false; }
      }
    }
    GetResult r{kOK, 0, 0u, false};
    if (go) r = thread_get_u32(g, sg.len, sg.pos, true);
    resolve_full<true>(go, sg, r, hb, lane);
    if (go && r.status != kOK) { status = r.status; ovf = r.ovf; go = false; }
    const uint32_t lower = r.value;
    const int forw = (int)((h >> 15) & 3), exc = (int)(h >> 24);
    SubGet sg2{nullptr, 0, 0, sg.pos};
    bool second = false;
    if (go) {
      if (!(h & kHdrCombine)) {
        uint64_t base = 0;
        if (forw == 3) {
          const int off = 4 + (exc > 0 ? 2 : 0);
          if (sg.len < off + 8) { status = kErrInvalidBuffer; go = false; }
          else base = g.u64(off);
        }
        if (go) result = (uint64_t)lower + base;
      } else {
        const int64_t meta = 4 + (exc > 0 ? 2 : 0) + ((1 << forw) >> 1) + 2;
        if (sg.len < meta) { status = kErrInvalidBuffer; go = false; }
        else {
          const int64_t b2len = g.u16(meta - 2);
          int64_t b1 = meta + (int64_t)(((h >> 8) & 31) * 4) * 16;
          if (exc > 0) b1 += min(exc, 16) + (int64_t)g.u16(4);
          if (b1 + b2len > sg.len) { status = kErrInvalidBuffer; go = false; }
          else {
            const int64_t rd2 = max((int64_t)0, min(b2len, sg.rd - b1));
            sg2 = SubGet{sg.p + b1, rd2, b2len, sg.pos};
            second = true;
          }
        }
      }
    }
    GetResult r2{kOK, 0, 0u, false};
    if (second) r2 = thread_get_u32(GlobalBytes{sg2.p, sg2.rd}, sg2.len, sg2.pos, true);
    resolve_full<true>(second, sg2, r2, hb, lane);
    if (second) {
      if (r2.status != kOK) { status = r2.status; ovf = r2.ovf; }
      else result = ((uint64_t)r2.value << 32) | lower;
    }
  }
  if (live) answer<U64>(a, q, status, ovf, result);
}

template <bool U64>
__global__ void __launch_bounds__(kGThreads, 4) get_kernel(const __grid_constant__ GetArgs a) {
  __shared__ uint32_t hb[kGThreads / 32][kBlock];  // whole unpacks
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = q < a.n_queries;

  int status = kOK;
  uint64_t result = 0;
  bool slow = false;
  SubGet sg{nullptr, 0, 0, 0};
  if (act) {
    slow = locate(a, q, sg);
    if (!slow) status = kErrPositionOutOfRange;
  }
  __syncwarp();  // the warp's queries into the direct path together: 57.0 -> 56.7 us on the lists
  if (slow && sg.rd == sg.len && sg.len < (1 << 20)) {
    // the buffer's first whole word and its end
    const uintptr_t lo = ((uintptr_t)a.packed + 3) & ~(uintptr_t)3, hi = (uintptr_t)a.packed + (uintptr_t)a.packed_len;
    const uint8_t* p = sg.p;
    const int len = (int)sg.len;
    Direct d;
    if (direct_get(p, len, sg.pos, U64, lo, hi, d)) {
      result = d.value;
      slow = false;
      if (U64) {  // getUint64Scalar, uint64.go:372-436
        if (d.h & kHdrCombine) {
          const int b2 = (int)ld_bytes(p, d.p_off - 2, 2, len);
          Direct d2;
          slow = d.end + b2 > len || !direct_get(p + d.end, b2, sg.pos, true, lo, hi, d2);
          if (!slow) result |= (uint64_t)d2.value << 32;
        } else if (((d.h >> 15) & 3u) == 3u) {
          const uint8_t* f = p + d.p_off - 8;
          slow = past((uintptr_t)f + 8, hi);
          if (!slow) result += (uint64_t)ld_word(f) | ((uint64_t)ld_word(f + 4) << 32);
        }
      }
    }
  }
  if (act && !slow) answer<U64>(a, q, status, 0, result);
  if (__any_sync(kFull, slow)) get_general<U64>(a, slow, hb[threadIdx.x >> 5]);
}

namespace launch {

cudaError_t get(bool u64, const GetArgs& a, cudaStream_t st) {
  if (a.n_queries <= 0) return cudaSuccess;
  const int64_t grid = (a.n_queries + kGThreads - 1) / kGThreads;
  if (u64) get_kernel<true><<<(unsigned)grid, kGThreads, 0, st>>>(a);
  else get_kernel<false><<<(unsigned)grid, kGThreads, 0, st>>>(a);
  note_launch(1);
  return cudaGetLastError();
}

}  // namespace launch
}  // namespace utl
