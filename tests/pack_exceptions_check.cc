// Runs utl::qp::put_exceptions (the exception writer of the two-launch pack) on
// the CPU, a thread for each lane of one warp, and checks its bytes against a
// serial writer.  Built with -fsanitize=thread, which ends the program with an
// error where two lanes touch the same bytes of the image, one of them writing,
// with no warp barrier between them: an atomic on a word and a plain store to a
// byte of it among others, which no memory model orders.
//
// Eight blocks lie back to back as in the kernel's image: exception counts
// around the list / bitmap border and the control bytes' ends, at every byte
// alignment of the StreamVByte region.  Prints "ok <warps>".
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <barrier>
#include <random>
#include <thread>
#include <vector>

#define __device__
#define __forceinline__ inline
#define __shared__ static
using std::max;
using std::min;
struct uint4 { uint32_t x, y, z, w; };
inline uint4 make_uint4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) { return {a, b, c, d}; }

// ---- one warp ----
static thread_local int t_lane;
static std::barrier<> g_bar(32);
static uint64_t g_box[32];
inline void __syncwarp(unsigned = 0xFFFFFFFFu) { g_bar.arrive_and_wait(); }
static uint32_t exchange(uint32_t v, int src) {
  g_box[t_lane] = v;
  __syncwarp();
  const uint32_t r = (uint32_t)g_box[src];
  __syncwarp();
  return r;
}
inline uint32_t __shfl_sync(unsigned, uint32_t v, int s) { return exchange(v, s & 31); }
inline uint32_t __shfl_xor_sync(unsigned, uint32_t v, int m) { return exchange(v, t_lane ^ m); }
inline uint32_t __shfl_up_sync(unsigned, uint32_t v, int d) { return exchange(v, t_lane >= d ? t_lane - d : t_lane); }
inline bool __any_sync(unsigned, bool p) {
  bool any = false;
  for (int i = 0; i < 32; i++) any |= exchange(p, i) != 0;
  return any;
}
inline uint32_t atomicOr(uint32_t* p, uint32_t v) { return __atomic_fetch_or(p, v, __ATOMIC_RELAXED); }
// ---- instructions ----
inline int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }
inline int __ffs(uint32_t x) { return __builtin_ffs((int)x); }
inline int __popc(uint32_t x) { return __builtin_popcount(x); }
inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, int s) {
  s &= 31;
  return s ? (hi << s) | (lo >> (32 - s)) : hi;
}
inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, int s) {
  s &= 31;
  return s ? (lo >> s) | (hi << (32 - s)) : lo;
}
inline uint32_t __byte_perm(uint32_t a, uint32_t b, uint32_t s) {
  const uint64_t v = ((uint64_t)b << 32) | a;
  uint32_t r = 0;
  for (int i = 0; i < 4; i++) r |= (uint32_t)((v >> (8 * ((s >> (4 * i)) & 7))) & 0xFF) << (8 * i);
  return r;
}
inline uint32_t __dp4a(uint32_t a, uint32_t b, uint32_t c) {
  for (int i = 0; i < 4; i++) c += ((a >> (8 * i)) & 255) * ((b >> (8 * i)) & 255);
  return c;
}
inline uint32_t __vimin3_u32(uint32_t a, uint32_t b, uint32_t c) { return min(a, min(b, c)); }
inline uint32_t __vimax3_u32(uint32_t a, uint32_t b, uint32_t c) { return max(a, max(b, c)); }
// ---- what utl_qpack.cuh takes from the headers it includes ----
namespace utl {
constexpr int kBlock = 128;
constexpr unsigned kFull = 0xFFFFFFFFu;
enum : int { kDelta = 1, kNoFOR = 2, kNoPatch = 4 };
constexpr uint32_t kHdrDelta = 1u << 22, kHdrZigZag = 1u << 23;
inline int len32(uint32_t x) { return 32 - __clz(x); }
inline int round_step(int bw) { return (bw + 3) & ~3; }
inline uint32_t zz_enc(uint32_t v) { return (v << 1) ^ (uint32_t)((int32_t)v >> 31); }
namespace quad {
inline uint64_t shr64_clamp(uint64_t x, uint32_t s) { return s >= 64 ? 0 : x >> s; }
inline uint32_t shl_clamp(uint32_t x, uint32_t s) { return s >= 32 ? 0 : x << s; }
inline void bucket_hist(const uint32_t (&)[8][4], uint32_t&, uint32_t&) {}
}  // namespace quad
}  // namespace utl
#include "qpack_host.h"  // utl_qpack.cuh without its #include lines

struct Block {
  uint32_t v[128];
  int bw, exc, at;  // width, exceptions, image offset of the exception bytes
};

// Index and StreamVByte bytes of a block (exceptions.go:138-186).
static std::vector<uint8_t> serial(const Block& b) {
  std::vector<uint8_t> pos, ctl((b.exc + 3) / 4, 0), data;
  uint8_t map[16] = {0};
  for (int i = 0; i < 128; i++) {
    const uint32_t hv = b.v[i] >> b.bw;
    if (!hv) continue;
    const int r = (int)pos.size(), code = (31 - __clz(hv)) >> 3;
    pos.push_back((uint8_t)i);
    map[i >> 3] |= (uint8_t)(1 << (i & 7));
    ctl[r >> 2] |= (uint8_t)(code << (2 * (r & 3)));
    for (int k = 0; k <= code; k++) data.push_back((uint8_t)(hv >> (8 * k)));
  }
  std::vector<uint8_t> out = pos;
  if (b.exc > 16) out.assign(map, map + 16);
  out.insert(out.end(), ctl.begin(), ctl.end());
  out.insert(out.end(), data.begin(), data.end());
  return out;
}

int main() {
  std::mt19937 rng(7);
  const int counts[] = {0, 1, 3, 4, 15, 16, 17, 18, 19, 20, 21, 24, 31, 33, 47, 64, 100, 128};
  const int n_counts = (int)(sizeof(counts) / sizeof(counts[0]));
  const int warps = 24;
  for (int w = 0; w < warps; w++) {
    std::vector<Block> blocks(8);
    std::vector<std::vector<uint8_t>> want;
    int at = w & 3;
    for (int q = 0; q < 8; q++) {
      Block& b = blocks[q];
      b.bw = 4 * (int)(rng() % 6);
      b.exc = counts[(5 * w + 7 * q) % n_counts];
      for (int i = 0; i < 128; i++) b.v[i] = b.bw ? rng() & ((1u << b.bw) - 1u) : 0u;
      std::vector<int> place(128);
      for (int i = 0; i < 128; i++) place[i] = i;
      std::shuffle(place.begin(), place.end(), rng);
      for (int e = 0; e < b.exc; e++) {
        const int len = 1 + (int)(rng() % (32 - b.bw));  // bits of the high part
        const uint32_t hv = (1u << (len - 1)) | (rng() & ((1u << (len - 1)) - 1u));
        b.v[place[e]] |= hv << b.bw;
      }
      b.at = at;
      want.push_back(serial(b));
      at += (int)want.back().size() + (int)(rng() % 4);
    }
    std::vector<uint32_t> image(at / 4 + 2, 0xA5A5A5A5u), slots(8 * 132);
    uint8_t* img = (uint8_t*)image.data();
    for (int q = 0; q < 8; q++) memcpy(&slots[132 * q], blocks[q].v, sizeof(blocks[q].v));
    std::vector<std::thread> lanes;
    for (int l = 0; l < 32; l++)
      lanes.emplace_back([&, l] {
        t_lane = l;
        const Block& b = blocks[l >> 2];
        const int j = l & 3;
        uint32_t x[8][4];
        for (int r = 0; r < 8; r++)
          for (int k = 0; k < 4; k++) x[r][k] = b.v[16 * r + 4 * j + k];
        utl::qp::put_exceptions(x, &slots[132 * (l >> 2)], b.bw, b.exc, img + b.at, j, l);
      });
    for (auto& t : lanes) t.join();
    for (int q = 0; q < 8; q++)
      if (memcmp(img + blocks[q].at, want[q].data(), want[q].size()) != 0) {
        printf("warp %d block %d: exceptions %d width %d differ\n", w, q, blocks[q].exc, blocks[q].bw);
        return 1;
      }
  }
  printf("ok %d\n", warps);
  return 0;
}
