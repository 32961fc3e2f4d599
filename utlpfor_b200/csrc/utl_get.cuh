// utl_get.cuh -- Get queries that need a whole-block unpack, resolved by the
// warp (batched Get and the per-call Get).
#pragma once
#include "utl_device.cuh"

namespace utl {

struct SubGet {
  const uint8_t* p;  // sub-block start
  int64_t rd;        // readable bytes
  int64_t len;       // the reference's len(src)
  int pos;
};

// Resolve every lane whose r.need_full is set with a warp-wide unpack of
// its block (getUint32FullUnpack / getFullUnpackViaBlock, get.go:198-218,
// 339-349), bounded by the block end the thread validated.
template <bool U64>
__device__ __forceinline__ void resolve_full(bool active, const SubGet& q, GetResult& r, uint32_t* hb, int lane) {
  unsigned m = __ballot_sync(kFull, active && r.need_full);
  while (m) {
    const int src = __ffs(m) - 1;
    m &= m - 1;
    const uint8_t* p = (const uint8_t*)__shfl_sync(kFull, (unsigned long long)q.p, src);
    const int64_t rd = (int64_t)__shfl_sync(kFull, (unsigned long long)q.rd, src);
    const int64_t len = (int64_t)__shfl_sync(kFull, (unsigned long long)r.end, src);
    const int pos = __shfl_sync(kFull, q.pos, src);
    uint32_t v[4];
    const GlobalBytes g{p, rd};
    const UnpackResult u = warp_unpack_block(g, 0, len, U64, v, hb, lane);
    const int slot = pos >> 5;
    uint32_t mine = slot == 0 ? v[0] : slot == 1 ? v[1] : slot == 2 ? v[2] : v[3];
    const uint32_t val = __shfl_sync(kFull, mine, pos & 31);
    if (lane == src) {
      r.need_full = false;
      r.status = u.status;
      r.ovf = u.ovf;
      r.value = val;
    }
  }
}

}  // namespace utl
