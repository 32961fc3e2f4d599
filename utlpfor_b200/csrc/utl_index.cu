// utl_index.cu -- device stream indexer: the block offsets of a packed
// stream that carries no index, i.e. what a caller gets by walking the
// stream with BlockLength block after block (block_length.go:8-65, caller
// pattern example_test.go:171-186).
//
// The walk is a chain: each block's start follows from the previous one's
// header.  It is done speculatively in parallel (index_starts_kernel): a CTA
// stages a region of the stream in shared memory; each team of four threads
// guesses a block start in its own 1008 bytes and walks the chain to their
// end; then the teams take over the exits of the teams before them and walk
// again where a guess was wrong, until nothing changes.  The region's own
// entry is taken from the region before it, which tells it as soon as it has
// settled on its guesses; the starts are kept as bits and a second launch
// turns them into offsets.
//
// The first region whose chain stops at its true entry's bad block ends the
// walk: the second launch counts the blocks before it.  A region that told a
// wrong exit leaves the whole call to the second path, which handles
// everything: the stream is cut into partitions of kPart bytes; one thread per
// partition finds a position where kSync consecutive headers parse and stay
// inside the stream (a true block start lies within the first kMaxBlock bytes
// of every partition), walks from there to the partition's end and records
// where its chain leaves the partition.  A second pass checks, in parallel, that the
// chain entering each partition (the previous partition's exit) meets that
// partition's chain -- two chains that share one position share all later
// ones -- and derives the partition's true block count.  Partitions whose
// check fails (a false start, or a stream error) are walked again one after
// the other from the true entry, which also finds the first bad block.  A
// scan of the counts places each partition's blocks, and a last pass walks
// every partition from its true entry and writes the offsets.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "utl_launch.h"
#include "utl_unpack.cuh"

namespace utl {
namespace index {

constexpr int64_t kPart = 8192;      // partition bytes (>= kMaxBlock)
constexpr int64_t kMaxBlock = 2048;  // every block is at most MaxBlockLength64(0) = 2038 bytes
constexpr int kSync = 6;             // headers that must parse in a row to accept a start
constexpr int kThreads = 256;
constexpr int kErrCapacity = 9;  // UTL_ERR_CAPACITY

__device__ __forceinline__ uint32_t byte_at(const uint8_t* p, uint64_t len, uint64_t i) {
  return i < len ? (uint32_t)p[i] : 0u;
}

// BlockLength of the block at byte off (block_length.go:8-65); on success
// also requires the block to end inside the stream, as the caller's next
// Unpack would (ErrInvalidBuffer otherwise).  Returns a status code.
__device__ int block_length_at(const uint8_t* p, uint64_t len, uint64_t off, uint64_t* out) {
  if (off + 4 > len) return kErrInvalidBuffer;
  const uint32_t h = byte_at(p, len, off) | (byte_at(p, len, off + 1) << 8) | (byte_at(p, len, off + 2) << 16) |
                     (byte_at(p, len, off + 3) << 24);
  const int count = (int)(h & 0xFFu), bw = (int)((h >> 8) & 0x1Fu) * 4, type = (int)((h >> 13) & 3u);
  const int forw = (int)((h >> 15) & 3u), exc = (int)(h >> 24);
  if (count > kBlock) return kErrInvalidBlockLength;
  if (bw > 32) return kErrInvalidBuffer;
  const bool combine = (h & (1u << 19)) && type == 3;
  if (type == 3) {
    if (h & ((1u << 18) | (1u << 20))) return kErrInvalidFlags;
  } else if (h & ((1u << 18) | (1u << 19) | (1u << 20))) {
    return kErrInvalidFlags;
  }
  const int forb = (type == 3 && !combine && forw == 3) ? 8 : ((1 << forw) >> 1);
  const uint64_t p_off = 4 + (exc ? 2 : 0) + forb + (combine ? 2 : 0);
  uint64_t b1 = p_off + ((uint64_t)bw << 4);
  if (exc) {
    if (off + 6 > len) return kErrInvalidBuffer;
    b1 += (uint64_t)(exc <= 16 ? exc : 16) + (byte_at(p, len, off + 4) | (byte_at(p, len, off + 5) << 8));
  }
  if (combine) {
    if (off + p_off > len) return kErrInvalidBuffer;
    b1 += byte_at(p, len, off + p_off - 2) | (byte_at(p, len, off + p_off - 1) << 8);
  }
  if (off + b1 > len) return kErrInvalidBuffer;
  *out = b1;
  return kOK;
}

struct Part {
  int64_t entry;   // first block start of the thread's chain (-1: none found)
  int64_t exit;    // where the chain leaves the partition (-1: it hit an error)
  int64_t count;   // blocks of the chain that start in the partition
  int64_t tcount;  // true block count (after the check)
  int32_t ok;      // the partition's chain is the stream's chain
  int32_t pad;
};

// Walk from `pos` while the block start is below `end`; counts the blocks.
// Returns the first start at or past `end`, or -1 on an error (err/epos set).
__device__ int64_t walk(const uint8_t* p, uint64_t len, int64_t pos, int64_t end, int64_t* count, int* err,
                        int64_t* epos) {
  int64_t c = 0;
  while (pos < end && (uint64_t)pos < len) {
    uint64_t L;
    const int st = block_length_at(p, len, (uint64_t)pos, &L);
    if (st != kOK) {
      *err = st;
      *epos = pos;
      *count = c;
      return -1;
    }
    pos += (int64_t)L;
    c++;
  }
  *count = c;
  return pos;
}

// Walk the chains from x (the stream's) and y (a partition's) forward, the
// one behind each time, until they meet before `end`.  On a meeting
// returns true with hx/hy = blocks each chain took to get there.
__device__ bool meet(const uint8_t* p, uint64_t len, int64_t x, int64_t y, int64_t end, int64_t* hx, int64_t* hy) {
  int64_t cx = 0, cy = 0;
  while (x != y) {
    if (x >= end || y >= end) return false;
    uint64_t L;
    if (x < y) {
      if (block_length_at(p, len, (uint64_t)x, &L) != kOK) return false;
      x += (int64_t)L;
      cx++;
    } else {
      if (block_length_at(p, len, (uint64_t)y, &L) != kOK) return false;
      y += (int64_t)L;
      cy++;
    }
  }
  *hx = cx;
  *hy = cy;
  return x < end;
}

__global__ void __launch_bounds__(kThreads) speculate_kernel(const uint8_t* p, uint64_t len, int64_t n_parts,
                                                             Part* parts) {
  const int64_t k = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (k >= n_parts) return;
  const int64_t start = k * kPart, end = min((int64_t)len, start + kPart);
  int64_t entry = -1;
  if (k == 0) {
    entry = 0;
  } else {
    const int64_t stop = min(end, start + kMaxBlock);
    for (int64_t x = start; x < stop && entry < 0; x++) {
      int64_t q = x;
      int good = 0;
      for (; good < kSync && (uint64_t)q < len; good++) {
        uint64_t L;
        // a start is accepted only on blocks a packer can emit (no block is
        // longer than kMaxBlock); the walks keep BlockLength's own rules
        if (block_length_at(p, len, (uint64_t)q, &L) != kOK || L > (uint64_t)kMaxBlock) break;
        q += (int64_t)L;
      }
      if (good == kSync || (uint64_t)q == len) entry = x;
    }
  }
  Part r;
  r.entry = entry;
  r.count = 0;
  r.exit = -1;
  r.tcount = 0;
  r.ok = 0;
  r.pad = 0;
  if (entry >= 0) {
    int err = 0;
    int64_t epos = 0;
    r.exit = walk(p, len, entry, end, &r.count, &err, &epos);
  }
  parts[k] = r;
}

// Partition k's chain is the stream's chain when the chain entering it (the
// previous partition's exit, assumed true) meets it; the true count then
// differs from the chain's count by the blocks between the two positions.
__global__ void __launch_bounds__(kThreads) check_kernel(const uint8_t* p, uint64_t len, int64_t n_parts,
                                                         Part* parts, int64_t* first_bad) {
  const int64_t k = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (k >= n_parts) return;
  Part& r = parts[k];
  if (k == 0) {
    r.ok = r.exit >= 0;
    r.tcount = r.count;
  } else {
    const int64_t x = parts[k - 1].exit, y = r.entry;
    const int64_t end = min((int64_t)len, k * kPart + kPart);
    bool ok = false;
    int64_t tc = 0;
    if (x >= 0 && r.exit >= 0) {
      if (x >= end) {
        // no block starts here; the partition's own chain is not the stream's,
        // and where it leads to must not enter the next one
        ok = end == (int64_t)len;
      } else if (y >= 0) {
        int64_t hx, hy;
        if (meet(p, len, x, y, end, &hx, &hy)) {  // the chains share every block from the meeting on
          ok = true;
          tc = hx + r.count - hy;
        }
      }
    }
    r.ok = ok;
    r.tcount = tc;
  }
  if (!r.ok) atomicMin((unsigned long long*)first_bad, (unsigned long long)k);
}

// Walk one partition after another from the first unchecked one, whose
// entry is true, until a partition's own chain meets the true chain again
// (it and the partitions after it are then right) or the stream ends or
// fails.  err_info: code, partition, blocks of that partition before the
// bad block.
__global__ void fixup_kernel(const uint8_t* p, uint64_t len, int64_t n_parts, Part* parts, int64_t k0,
                             int64_t* err_info) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  int64_t k = k0;
  int64_t x = k == 0 ? 0 : parts[k - 1].exit;
  while (k < n_parts) {
    const int64_t end = min((int64_t)len, k * kPart + kPart);
    int64_t c;
    int err = 0;
    int64_t epos = 0;
    const int64_t e = walk(p, len, x, end, &c, &err, &epos);
    Part& r = parts[k];
    if (e < 0) {
      err_info[0] = err;
      err_info[1] = k;
      err_info[2] = c;
      r.tcount = c;
      r.exit = -1;
      for (int64_t j = k; j < n_parts; j++) parts[j].ok = 1;  // nothing past the error is used
      return;
    }
    r.tcount = c;
    r.exit = e;
    r.ok = 1;
    k++;
    if (k >= n_parts) return;
    Part& q = parts[k];
    const int64_t nend = min((int64_t)len, k * kPart + kPart);
    if (e < nend && q.entry >= 0 && q.exit >= 0) {  // a block that spans it leaves no meeting there
      int64_t hx, hy;
      if (meet(p, len, e, q.entry, nend, &hx, &hy)) {
        q.tcount = hx + q.count - hy;
        q.ok = 1;
        return;
      }
    }
    x = e;
  }
}

__global__ void __launch_bounds__(kThreads) unchecked_kernel(int64_t n_parts, const Part* parts, int64_t* first_bad) {
  const int64_t k = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (k < n_parts && !parts[k].ok) atomicMin((unsigned long long*)first_bad, (unsigned long long)k);
}

// Exclusive scan of the true counts into base[] (one CTA); base[n] = total.
__global__ void __launch_bounds__(1024) scan_kernel(int64_t n_parts, const Part* parts, int64_t* base) {
  __shared__ int64_t sums[1024];
  const int t = threadIdx.x;
  const int64_t per = (n_parts + 1023) / 1024;
  const int64_t lo = min(n_parts, per * t), hi = min(n_parts, lo + per);
  int64_t s = 0;
  for (int64_t k = lo; k < hi; k++) s += parts[k].tcount;
  sums[t] = s;
  __syncthreads();
  for (int d = 1; d < 1024; d <<= 1) {
    const int64_t v = t >= d ? sums[t - d] : 0;
    __syncthreads();
    sums[t] += v;
    __syncthreads();
  }
  int64_t run = sums[t] - s;
  for (int64_t k = lo; k < hi; k++) {
    base[k] = run;
    run += parts[k].tcount;
  }
  if (t == 1023) base[n_parts] = sums[1023];
}

// Each partition's true blocks, from its true entry: their offsets.
__global__ void __launch_bounds__(kThreads) write_kernel(const uint8_t* p, uint64_t len, int64_t n_parts,
                                                         const Part* parts, const int64_t* base, uint64_t* block_off) {
  const int64_t k = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (k >= n_parts) return;
  const int64_t end = min((int64_t)len, k * kPart + kPart);
  int64_t pos = k == 0 ? 0 : parts[k - 1].exit;
  int64_t i = base[k];
  const int64_t stop = base[k + 1];
  while (pos < end && i < stop) {
    uint64_t L;
    if (block_length_at(p, len, (uint64_t)pos, &L) != kOK) break;
    block_off[i++] = (uint64_t)pos;
    pos += (int64_t)L;
  }
  if (k == n_parts - 1) block_off[stop] = len;
}

// ---- the first path ----
// Bound by the latency of guessing and walking (dependent shared-memory loads
// and byte arithmetic) with 24 warps on an SM, not by its one read of the
// stream: 2^26 outlier values under NoFOR (75 MB, 2331 regions, 524 289 blocks)
// take 34 us here, 8 us in the second launch and 60 us for the whole call,
// against 397 us by the second path (a thread per 8 KB on global memory, and
// five round trips with the host).  A bad block half way: 44 us for 2^25 values
// (343 us when it was left to the second path as well, 309 by that alone).
// A team of four threads has 1008 bytes.  Finding a start takes about a block
// length of places to look at, so four threads share it; walking is serial
// and one does it.  252 words from team to team put the eight teams of a warp,
// four words each, on all 32 banks.
constexpr int kRT = 128;                  // threads of a CTA
constexpr int kTeam = 4;                  // threads of a team
constexpr int kTeams = kRT / kTeam;
constexpr int kSub = 1008;                // bytes of a team
constexpr int kBitWords = kSub / 32 + 1;  // their block starts as bits
constexpr int kRegion = kSub * kTeams;    // bytes of a CTA (32 KB: six CTAs, 24 warps, on an SM)
constexpr int kAhead = 32;                // staged bytes past the region (headers that start in it)
static_assert(kRegion % 16 == 0, "regions keep the stream's alignment");
constexpr uint32_t kDrainPolls = 1u << 22;  // for a copy that must land before the CTA ends, whatever the knob says

// Result of the first path: the block count, or the status and the index of
// the first bad block; open: neither is known.
struct __align__(16) FastResult {
  int64_t blocks;
  int32_t status;
  int32_t open;
};
// The first region that failed, and how: all regions before it are right, so
// its own entry is the stream's, and a chain that stops there stops at the
// stream's first bad block.  A region without an entry (the one before it
// failed, or a wait ran out) or whose exit is not what it told says nothing.
// Held as ~key, so that zero is none and the maximum the first region.
struct FastCtl {
  uint32_t ticket, pad;
  unsigned long long worst;
};
constexpr uint32_t kOpen = 0xFFFF;  // in place of the bad block's position
static_assert(kRegion < 0xFFFF, "positions in 16 bits");
__device__ __forceinline__ void fail_region(FastCtl* ctl, int32_t r, uint32_t pos) {
  atomicMax(&ctl->worst, ~(((unsigned long long)(uint32_t)r << 16) | pos));
}

// What the two launches share: block counts of the regions, of their groups
// of 32 and of 1024, and the block starts of each region as bits (a word row
// of 32 per team).
struct RegionTables {
  FastCtl* ctl;
  int64_t* exits;
  unsigned long long* g1024;
  uint32_t* one;
  uint32_t* g32;
  uint32_t* bits;
};
// Bytes of the tables in the scratch; those before `bits` start out zero.
inline size_t tables_zeroed(int64_t n) {
  const size_t z = sizeof(FastCtl) + 8 * (size_t)n + 8 * (size_t)((n + 1023) / 1024) + 4 * (size_t)n +
                   4 * (size_t)((n + 31) / 32);
  return (z + 15) / 16 * 16;
}
inline size_t tables_bytes(int64_t n) { return tables_zeroed(n) + (size_t)n * kTeams * kBitWords * 4; }
inline RegionTables tables(void* scratch, int64_t n) {
  RegionTables t;
  t.ctl = (FastCtl*)scratch;
  t.exits = (int64_t*)(t.ctl + 1);
  t.g1024 = (unsigned long long*)(t.exits + n);
  t.one = (uint32_t*)(t.g1024 + (n + 1023) / 1024);
  t.g32 = t.one + n;
  t.bits = (uint32_t*)((uint8_t*)scratch + tables_zeroed(n));
  return t;
}

// A staged region: byte x of it is byte x + mis of buf.
struct Staged {
  const uint32_t* buf;
  int mis;
  int end;  // bytes from the region's start to the stream's end (clamped)
  __device__ __forceinline__ uint32_t u32(int x) const {
    const int a = x + mis;
    return __funnelshift_r(buf[a >> 2], buf[(a >> 2) + 1], (a & 3) * 8);
  }
};

// BlockLength (block_length.go:8-65) of the block at x, which must also end
// inside the stream; 0 where it fails.  Fields past the stream's end read
// staged garbage that only makes the block longer: it fails all the same.
__device__ __forceinline__ int region_length(const Staged& s, int x) {
  const int a = x + s.mis, sh = (a & 3) * 8;
  const uint32_t* w = s.buf + (a >> 2);
  const uint32_t w1 = w[1], h = __funnelshift_r(w[0], w1, sh), h2 = __funnelshift_r(w1, w[2], sh);
  const uint32_t forw = (h >> 15) & 3u, exc = h >> 24;
  int n = 4 + (int)((h >> 2) & 0x7C0u) + (int)((1u << forw) >> 1);
  if (exc) n += 2 + (int)min(exc, 16u) + (int)(h2 & 0xFFFFu);
  uint32_t bad = h & (7u << 18);
  if ((h & (3u << 13)) == (3u << 13)) {  // uint64 (uint64.go:124-189)
    bad = h & (5u << 18);
    if (h & (1u << 19)) n += 2 + (int)(s.u32(x + 4 + (exc ? 2 : 0) + (int)((1u << forw) >> 1)) & 0xFFFFu);
    else if (forw == 3) n += 4;
  }
  return bad == 0 && (h & 0xFFu) <= (uint32_t)kBlock && (h & 0x1F00u) <= 0x800u && x + n <= s.end ? n : 0;
}
// Whether a packer may have put a block header h at a place, h2 the four bytes
// after it (guesses only): what the encoders write, the StreamVByte length
// within its bounds for the exception count among it (exceptions.go:122-130).
__device__ __forceinline__ bool plausible(uint32_t h, uint32_t h2) {
  const uint32_t count = h & 0xFFu, type = (h >> 13) & 3u, exc = h >> 24;
  const uint32_t data = (h2 & 0xFFFFu) - ((exc + 3) >> 2) - exc;
  return count - 1u < (uint32_t)kBlock && (h & 0x1F00u) <= 0x800u && type != 0u &&
         !(h & (type == 3u ? 5u << 18 : 7u << 18)) && exc <= count && (exc == 0 || data <= 3 * exc);
}
// The bytes (bit 8i + 7) of w, followed by wn, where a header may start, four
// at once and never missing one: count 1..128; width field at most 8, type not
// 0; header bits 18 and 20 clear; exceptions (but for the lowest bit) no more
// than values.
__device__ __forceinline__ uint32_t maybe_headers(uint32_t w, uint32_t wn) {
  const uint32_t w1 = __funnelshift_r(w, wn, 8), w2 = __funnelshift_r(w, wn, 16), w3 = __funnelshift_r(w, wn, 25);
  const uint32_t count = w ^ ((w | 0x80808080u) - 0x01010101u);
  const uint32_t wide = (w1 & 0x1F1F1F1Fu) + 0x77777777u, typed = (w1 & 0x60606060u) + 0x60606060u;
  const uint32_t bits = (w2 & 0x14141414u) + 0x7C7C7C7Cu;
  const uint32_t excs = ((w >> 1) | 0x80808080u) - (w3 & 0x7F7F7F7Fu);
  return count & ~wide & typed & ~bits & excs & 0x80808080u;
}
// Whether the block at x (a plausible header) is followed by another one, or
// leads out of the region or to the stream's end.
__device__ __forceinline__ bool followed(const Staged& s, int x) {
  const int n = region_length(s, x);
  if (n == 0 || n > (int)kMaxBlock) return false;
  x += n;
  if (x >= kRegion || x == s.end) return true;
  return x + 4 <= s.end && plausible(s.u32(x), s.u32(x + 4));
}

__global__ void __launch_bounds__(kRT) index_starts_kernel(const uint8_t* p, uint64_t len, int32_t n_regions,
                                                           RegionTables tab, uint32_t spin) {
  __shared__ __align__(16) uint32_t buf[(16 + kRegion + kAhead + 16) / 4];
  __shared__ uint32_t bits[kTeams][kBitWords | 1];  // block starts in each team's bytes
  __shared__ int X[kTeams];  // where each team's chain leaves its bytes (-1: not known, -2: it failed)
  __shared__ int s_region, s_entry, s_from, s_bad;
  __shared__ uint32_t s_total;
  __shared__ uint64_t bar;
  const int k = threadIdx.x, lane = k & 31;
  if (k == 0) {
    tma::mbar_init(&bar, 1);
    tma::mbar_init_fence();
    s_region = (int)atomicAdd(&tab.ctl->ticket, 1u);
    s_total = 0;
    s_bad = (int)kOpen;
  }
  __syncthreads();
  const int32_t r = s_region;
  const int64_t start = (int64_t)r * kRegion;
  // the 16-byte chunks that cover the region and what is ahead: those inside
  // the stream by one bulk copy, the bytes of the chunks at its ends singly
  const uintptr_t lo = (uintptr_t)p, hi = lo + len;
  const uintptr_t a0 = (lo + start) & ~(uintptr_t)15;
  const uintptr_t a1 = min((uint64_t)((hi + 15) & ~(uintptr_t)15), (uint64_t)(a0 + 16 + kRegion + kAhead));
  const uintptr_t t0 = max((uint64_t)a0, (uint64_t)((lo + 15) & ~(uintptr_t)15));
  const uintptr_t t1 = min((uint64_t)a1, (uint64_t)(hi & ~(uintptr_t)15));
  Staged s;
  s.buf = buf;
  s.mis = (int)(lo & 15);
  s.end = (int)min((uint64_t)(1 << 30), len - (uint64_t)start);
  const bool bulk = t1 > t0;
  if (bulk && k == 0) {
    tma::mbar_expect_tx(&bar, (uint32_t)(t1 - t0));
    tma::bulk_load((uint8_t*)buf + (t0 - a0), (const void*)t0, (uint32_t)(t1 - t0), &bar);
  }
  const uintptr_t e0 = bulk ? t0 : a1;  // [a0, e0) and [t1, a1) byte by byte
  for (uintptr_t a = a0 + k; a < e0; a += kRT) ((uint8_t*)buf)[a - a0] = a >= lo && a < hi ? *(const uint8_t*)a : 0;
  if (bulk)
    for (uintptr_t a = t1 + k; a < a1; a += kRT) ((uint8_t*)buf)[a - a0] = a < hi ? *(const uint8_t*)a : 0;
  if (__syncthreads_or(bulk && !tma::mbar_wait(&bar, 0, spin))) {
    // The copy did not land within the limit: nothing in buf is looked at.
    // The call is left to the second path, and the copy gets the full limit
    // to land before the CTA's shared memory goes to another one.
    if (k == 0) {
      *(volatile int64_t*)&tab.exits[r] = -1;
      fail_region(tab.ctl, r, kOpen);
    }
    tma::mbar_wait(&bar, 0, kDrainPolls);
    return;
  }

  // a start per team, guessed: the four threads look at alternate pairs of words
  const int team = k / kTeam, c4 = k % kTeam;
  const int own = kSub * team, own_end = own + kSub;
  const unsigned tm = 0xFu << (lane & 28);
  int t = -1;  // where the team's chain starts
  bool more = r > 0 || team > 0;
  if (!more) t = 0;
  const int stop = min(own_end, s.end - 3);
  int x0 = own - (s.mis & 3), from = own;  // the first byte of the team's next eight words, the next place
  while (__any_sync(kFull, more)) {
    // a place that may hold a header is looked at closely; the first that
    // passes is followed by all teams of the warp together (each on its own
    // way would repeat that part)
    int found = kRegion;
    if (more) {
      for (; x0 < stop; x0 += 8 * kTeam) {
        const int x = x0 + 8 * c4;
        if (x < stop) {
          const uint32_t* w = buf + ((x + s.mis) >> 2);
          const uint32_t w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3];
          // bit 7 of byte i: place x + i; bit 3: place x + 4 + i
          uint32_t m = maybe_headers(w0, w1) | maybe_headers(w1, w2) >> 4;
          while (m) {
            const int f = __ffs(m & 0x80808080u ? m & 0x80808080u : m) - 1;
            m &= ~(1u << f);
            const bool up = (f & 4) == 0;
            const int i = f >> 3, y = x + i + (up ? 4 : 0);
            const uint32_t a0 = up ? w1 : w0, a1 = up ? w2 : w1, a2 = up ? w3 : w2;
            if (y >= from && y < stop && plausible(__funnelshift_r(a0, a1, 8 * i), __funnelshift_r(a1, a2, 8 * i))) {
              found = y;
              break;
            }
          }
        }
        if (__any_sync(tm, found != kRegion)) break;
      }
      found = min(found, __shfl_xor_sync(tm, found, 1));
      found = min(found, __shfl_xor_sync(tm, found, 2));
    }
    __syncwarp();
    if (more) {
      if (found == kRegion) {
        more = false;
      } else if (followed(s, found)) {
        t = found;
        more = false;
      } else {
        from = found + 1;  // these words again
      }
    }
    __syncwarp();
  }
  __syncwarp();
  if (k == 0) s_entry = t;
  // walk from t through the team's bytes (its first thread); -2 at a bad block
  int stuck = 0;
  const auto walk = [&]() {
    int x = t;
    while (x < own_end && x < s.end) {
      const int n = region_length(s, x);
      if (n == 0) {
        stuck = x;
        return -2;
      }
      const int b = x - own;
      bits[team][b >> 5] |= 1u << (b & 31);
      x += n;
    }
    return x;
  };
  const bool first = c4 == 0;
#pragma unroll
  for (int i = 0; i < kBitWords / kTeam; i++) bits[team][kBitWords / kTeam * c4 + i] = 0;
  __syncwarp();
  int mine = -1;  // where the chain from t leaves
  if (first) {
    if (t >= 0) mine = walk();
    X[team] = mine;
  }
  __syncthreads();
  // every team's chain is the continuation of the one before it, the first
  // one's that from the region's entry: team i is right after at most i + 1
  // rounds (with right guesses, after one)
  const auto settle = [&]() {
    for (int round = 0; round <= kTeams; round++) {
      bool change = false;
      int now = 0;
      if (first) {
        // the last known exit before; it has to lead here, not into a team
        // between that knows nothing yet
        int before = team - 1;
        while (before > 0 && X[before] == -1) before--;
        int want = before < 0 ? s_entry : X[before];
        if (before < team - 1 && want >= 0 && want < min(own, s.end)) want = -1;
        if (want >= 0 && want != t) {
#pragma unroll 1
          for (int i = 0; i < kBitWords; i++) bits[team][i] = 0;
          t = want;
          mine = walk();
        }
        now = want == -2 ? -2 : mine;
        change = now != X[team];
      }
      __syncthreads();
      if (first) X[team] = now;
      if (!__syncthreads_or(change)) break;
    }
    return X[kTeams - 1];
  };
  int leave = settle();
  // The exit is told to the next region at once: guessed chains have met the
  // stream's long before.  Then the entry is taken from the region before,
  // and the teams settle again if it differs; the exit has to stay what was
  // told.  (exits: position + 1; 0 = not yet,
  // -1 = failed.)
  const int first_leave = leave;
  bool entered = true;
  if (k == 0 && leave >= 0) *(volatile int64_t*)&tab.exits[r] = start + leave + 1;
  if (r > 0) {
    if (k == 0) {
      int64_t e = 0;
      for (uint32_t it = 0; it <= spin && e == 0; it++) {
        if (it) __nanosleep(64);
        e = *(volatile int64_t*)&tab.exits[r - 1];
      }
      s_from = e > 0 ? (int)(e - 1 - start) : -2;
    }
    __syncthreads();
    const int from = s_from;
    entered = from >= 0;
    if (from != s_entry) {
      __syncthreads();
      if (k == 0) s_entry = from;
      __syncthreads();
      leave = entered ? settle() : -2;
    }
  }
  if (k == 0 && first_leave < 0) *(volatile int64_t*)&tab.exits[r] = leave >= 0 ? start + leave + 1 : -1;
  // The first team of a chain that stopped is the one that met the bad block
  // (the others only took that over).
  if (entered && leave < 0 && first && X[team] == -2 && (team == 0 || X[team - 1] != -2)) s_bad = stuck;
  const bool failed = leave < 0 || (first_leave >= 0 && leave != first_leave) ||
                      (r == n_regions - 1 && start + leave != (int64_t)len);

  // the starts and their counts, for the second launch
  int c = 0;
  uint32_t* out = tab.bits + (size_t)r * (kTeams * kBitWords);
#pragma unroll
  for (int i = 0; i < kTeams * kBitWords / kRT; i++) {
    const int e = i * kRT + k;
    const uint32_t w = bits[e / kBitWords][e % kBitWords];
    c += __popc(w);
    out[e] = w;
  }
  c = (int)__reduce_add_sync(kFull, (unsigned)c);
  if (lane == 0) atomicAdd(&s_total, (uint32_t)c);
  __syncthreads();
  if (k == 0) {
    tab.one[r] = s_total;
    atomicAdd(&tab.g32[r >> 5], s_total);
    atomicAdd(&tab.g1024[r >> 10], (unsigned long long)s_total);
    if (failed) fail_region(tab.ctl, r, (uint32_t)s_bad);
  }
}

// The stream's first bad block, at place bad of region r, by the thread whose
// eight words its start would be in: its index is the count of the starts
// before it, at of them in the words before.
__device__ __noinline__ void report_bad(const uint8_t* p, uint64_t len, int32_t r, int bad, int64_t at,
                                        const uint32_t* words, FastResult* result) {
  const int places = bad % kSub & 255;  // of these words before it
  for (int i = 0; 32 * i < places; i++)
    at += __popc(places - 32 * i >= 32 ? words[i] : words[i] & ((1u << (places - 32 * i)) - 1u));
  uint64_t n;
  const int status = block_length_at(p, len, (uint64_t)r * kRegion + (uint64_t)bad, &n);
  *result = FastResult{at, status, status == kOK ? 1 : 0};
}

// The offsets of a region's blocks from its starts: a thread per eight words
// of bits, after the blocks before the region.  (In the first launch a region
// would have to wait for all before it, which cost half as much again.)
__global__ void __launch_bounds__(kRT) index_write_kernel(const uint8_t* p, uint64_t len, int32_t n_regions,
                                                          RegionTables tab, uint64_t* block_off, int64_t max_blocks,
                                                          FastResult* result) {
  static_assert(kTeams * kBitWords == 8 * kRT, "eight words a thread");
  __shared__ int wsum[kRT / 32];
  const int k = threadIdx.x, lane = k & 31, warp = k >> 5;
  const int32_t r = blockIdx.x;
  const uint4* in = (const uint4*)(tab.bits + (size_t)r * (kTeams * kBitWords)) + 2 * k;
  const uint4 A = in[0], B = in[1];
  const unsigned long long worst = ~__ldg(&tab.ctl->worst);
  const int r32 = r & ~31, r1024 = r & ~1023;
  uint64_t sum = (r32 + lane < r ? tab.one[r32 + lane] : 0u);
  if (r1024 + 32 * lane < r32) sum += tab.g32[(r1024 >> 5) + lane];
  for (int g = lane; g < r1024 >> 10; g += 32) sum += tab.g1024[g];
  uint32_t w[8] = {A.x, A.y, A.z, A.w, B.x, B.y, B.z, B.w};
  int c = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) c += __popc(w[i]);
  const int incl = warp_incl_scan(c, lane);
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) sum += shfl_xor64(sum, d);
  int64_t at = (int64_t)sum + incl - c;
#pragma unroll
  for (int i = 0; i < kRT / 32; i++) at += i < warp ? wsum[i] : 0;
  const uint64_t first = (uint64_t)r * kRegion + (uint64_t)(kSub * (k / kTeam) + 256 * (k % kTeam));
#pragma unroll
  for (int i = 0; i < 8; i++)
    for (uint32_t b = w[i]; b; b &= b - 1, at++)
      if (at < max_blocks) block_off[at] = first + (uint64_t)(32 * i + __ffs(b) - 1);
  if (r == n_regions - 1 && k == kRT - 1) {
    if (at <= max_blocks) block_off[at] = len;
    if (worst == ~0ull || (worst & 0xFFFFu) == kOpen) *result = FastResult{at, kOK, worst == ~0ull ? 0 : 1};
  }
  if ((uint32_t)(worst >> 16) == (uint32_t)r && (worst & 0xFFFFu) != kOpen && worst != ~0ull) {
    const int bad = (int)(worst & 0xFFFFu);
    if (k == kTeam * (bad / kSub) + (bad % kSub >> 8)) report_bad(p, len, r, bad, at - c, (const uint32_t*)in, result);
  }
}

}  // namespace index

namespace launch {

size_t index_scratch_bytes(uint64_t len) {
  const int64_t n_parts = (int64_t)((len + index::kPart - 1) / index::kPart);
  const int64_t n_regions = (int64_t)((len + index::kRegion - 1) / index::kRegion);
  const size_t slow = (size_t)n_parts * sizeof(index::Part) + (size_t)(n_parts + 1) * 8 + 64;
  return std::max(slow, index::tables_bytes(n_regions));
}

// Block offsets of the packed stream p[0, len) into block_off (capacity
// max_blocks + 1).  Synchronizes st.  Returns a status; *n_blocks is the
// block count, or on an error the index of the bad block.  res_d / res_h: 16
// bytes of mapped host memory of this call's own.
int index_stream(const uint8_t* p, uint64_t len, uint64_t* block_off, int64_t max_blocks, int64_t* n_blocks,
                 void* scratch, void* res_d, const void* res_h, cudaStream_t st, cudaError_t* cerr) {
  using namespace index;
  *n_blocks = 0;
  *cerr = cudaSuccess;
  const int64_t n_parts = (int64_t)((len + kPart - 1) / kPart);
  int64_t* ctl = (int64_t*)scratch;  // first_bad, err code, err partition, err count
  Part* parts = (Part*)((uint8_t*)scratch + 64);
  int64_t* base = (int64_t*)(parts + n_parts);
  if (len == 0) {
    if (max_blocks < 0) return kErrCapacity;
    *cerr = cudaMemsetAsync(block_off, 0, 8, st);
    if (*cerr == cudaSuccess) *cerr = cudaStreamSynchronize(st);
    return *cerr == cudaSuccess ? kOK : -1;
  }
  const int64_t n_regions = (int64_t)((len + kRegion - 1) / kRegion);
  if (n_regions < INT32_MAX) {
    const RegionTables tab = tables(scratch, n_regions);
    if ((*cerr = cudaMemsetAsync(scratch, 0, tables_zeroed(n_regions), st)) != cudaSuccess) return -1;
    index_starts_kernel<<<(unsigned)n_regions, kRT, 0, st>>>(p, len, (int32_t)n_regions, tab, spin_limit());
    index_write_kernel<<<(unsigned)n_regions, kRT, 0, st>>>(p, len, (int32_t)n_regions, tab, block_off, max_blocks,
                                                            (FastResult*)res_d);
    note_launch(2);
    if ((*cerr = cudaGetLastError()) != cudaSuccess) return -1;
    if ((*cerr = cudaStreamSynchronize(st)) != cudaSuccess) return -1;
    const FastResult f = *(const FastResult*)res_h;
    if (!f.open) {
      *n_blocks = f.blocks;
      if (f.status != kOK) return f.status;
      return f.blocks > max_blocks ? kErrCapacity : kOK;
    }
  }
  const int64_t init[4] = {INT64_MAX, 0, -1, 0};
  if ((*cerr = cudaMemcpyAsync(ctl, init, sizeof(init), cudaMemcpyHostToDevice, st)) != cudaSuccess) return -1;
  const unsigned grid = (unsigned)((n_parts + kThreads - 1) / kThreads);
  speculate_kernel<<<grid, kThreads, 0, st>>>(p, len, n_parts, parts);
  check_kernel<<<grid, kThreads, 0, st>>>(p, len, n_parts, parts, ctl);
  note_launch(2);
  for (;;) {
    int64_t h[4];
    if ((*cerr = cudaMemcpyAsync(h, ctl, sizeof(h), cudaMemcpyDeviceToHost, st)) != cudaSuccess) return -1;
    if ((*cerr = cudaStreamSynchronize(st)) != cudaSuccess) return -1;
    if (h[1] != 0 || h[0] == INT64_MAX) break;  // an error found, or every partition checked
    const int64_t reset = INT64_MAX;
    if ((*cerr = cudaMemcpyAsync(ctl, &reset, 8, cudaMemcpyHostToDevice, st)) != cudaSuccess) return -1;
    fixup_kernel<<<1, 32, 0, st>>>(p, len, n_parts, parts, h[0], ctl + 1);
    unchecked_kernel<<<grid, kThreads, 0, st>>>(n_parts, parts, ctl);
    note_launch(2);
  }
  scan_kernel<<<1, 1024, 0, st>>>(n_parts, parts, base);
  note_launch(1);
  int64_t h[4], total = 0;
  if ((*cerr = cudaMemcpyAsync(h, ctl, sizeof(h), cudaMemcpyDeviceToHost, st)) != cudaSuccess) return -1;
  if ((*cerr = cudaMemcpyAsync(&total, base + n_parts, 8, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return -1;
  if ((*cerr = cudaStreamSynchronize(st)) != cudaSuccess) return -1;
  if (h[1] != 0) {  // the walk failed at block base[partition] + count
    int64_t b = 0;
    if ((*cerr = cudaMemcpyAsync(&b, base + h[2], 8, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return -1;
    if ((*cerr = cudaStreamSynchronize(st)) != cudaSuccess) return -1;
    *n_blocks = b + h[3];
    return (int)h[1];
  }
  *n_blocks = total;
  if (total > max_blocks) return kErrCapacity;
  write_kernel<<<grid, kThreads, 0, st>>>(p, len, n_parts, parts, base, block_off);
  note_launch(1);
  if ((*cerr = cudaGetLastError()) != cudaSuccess) return -1;
  if ((*cerr = cudaStreamSynchronize(st)) != cudaSuccess) return -1;
  return kOK;
}

}  // namespace launch
}  // namespace utl
