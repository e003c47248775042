// A warp of 32 lanes on the host, for code whose lanes vote and shuffle: every
// lane is a fibre that runs to its next warp operation and waits there for
// the others.  All lanes meet the same operations in the same order.
#pragma once
#include <ucontext.h>

#include <functional>
#include <vector>

#include "host_march_shim.h"

struct HostLane {
  int x;
};
inline HostLane threadIdx{0};

namespace host_warp {
constexpr int LANES = 32;
inline ucontext_t back, lane_ctx[LANES];
inline std::function<void()> body;
inline bool ended[LANES];
inline unsigned slot[2][LANES];
inline int turn[LANES];

inline void entry()
{
  body();
  ended[threadIdx.x] = true;
  swapcontext(&lane_ctx[threadIdx.x], &back);
}

// Posts v and waits for every lane's; the values of this operation.
inline const unsigned* meet(unsigned v)
{
  const int l = threadIdx.x, t = turn[l] ^= 1;
  slot[t][l] = v;
  swapcontext(&lane_ctx[l], &back);
  return slot[t];
}

inline void run(std::function<void()> f)
{
  static std::vector<std::vector<char>> stacks(LANES, std::vector<char>(1 << 17));
  body = f;
  for (int l = 0; l < LANES; ++l) {
    ended[l] = false;
    turn[l] = 0;
    getcontext(&lane_ctx[l]);
    lane_ctx[l].uc_stack.ss_sp = stacks[l].data();
    lane_ctx[l].uc_stack.ss_size = stacks[l].size();
    lane_ctx[l].uc_link = nullptr;
    makecontext(&lane_ctx[l], entry, 0);
  }
  for (bool any = true; any;) {
    any = false;
    for (int l = 0; l < LANES; ++l)
      if (!ended[l]) {
        threadIdx.x = l;
        swapcontext(&back, &lane_ctx[l]);
        any = any || !ended[l];
      }
  }
}

template <class T>
inline unsigned bits(T v)
{
  static_assert(sizeof(T) == 4, "a word");
  unsigned u;
  std::memcpy(&u, &v, 4);
  return u;
}
}  // namespace host_warp

template <class T>
inline T __shfl_sync(unsigned, T v, int src)
{
  const unsigned u = host_warp::meet(host_warp::bits(v))[src & 31];
  T r;
  std::memcpy(&r, &u, 4);
  return r;
}
inline unsigned __reduce_min_sync(unsigned, unsigned v)
{
  const unsigned* p = host_warp::meet(v);
  return *std::min_element(p, p + 32);
}
inline unsigned __reduce_max_sync(unsigned, unsigned v)
{
  const unsigned* p = host_warp::meet(v);
  return *std::max_element(p, p + 32);
}
inline unsigned __ballot_sync(unsigned, bool v)
{
  const unsigned* p = host_warp::meet(v);
  unsigned r = 0;
  for (int l = 0; l < 32; ++l) r |= p[l] << l;
  return r;
}
inline bool __any_sync(unsigned m, bool v) { return __ballot_sync(m, v) != 0; }
inline void __syncwarp() { host_warp::meet(0); }
inline int __clzll(long long v) { return v ? __builtin_clzll((unsigned long long)v) : 64; }
inline int __ffs(unsigned v) { return __builtin_ffs((int)v); }
inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }
