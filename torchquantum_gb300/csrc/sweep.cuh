// sweep.cuh -- tiles of amplitudes in shared memory, worked on from registers.
//
// A thread takes 2^b amplitudes of a tile: every value of b register bits, tile bit 0 always
// one of them (slot 0), the others (slots 1..b-1) chosen per sweep; the remaining tile bits
// come from the thread index.  Ops whose targets are register bits then need no
// exchange; between sweeps the tile is re-dealt through shared memory.
//
// Shared memory layout: amplitude l of the tile lives at l ^ (g(l) << 1), g(l) the XOR of
// the 3-bit fields of l >> 4: linear over XOR, keeps 16-byte pairs (bit 0) whole, and makes
// the 16-byte accesses of 8 lanes conflict free whenever the three lowest lane bits map
// to tile bits of different classes (bit - 1) mod 3, which the host picks where it can.
#pragma once

#include "bulk.cuh"
#include "common.cuh"
#include "f32x2.cuh"

namespace tqk {
namespace sweep {

__host__ __device__ __forceinline__ uint32_t swz(uint32_t l) {
  return l ^ ((((l >> 4) ^ (l >> 7) ^ (l >> 10)) & 7u) << 1);
}

// Compile-time loop: f(Const<0>) ... f(Const<N - 1>).
template <int I>
struct Const {
  static constexpr int value = I;
};
template <int N, int I = 0, typename F>
__device__ __forceinline__ void unroll(const F& f) {
  if constexpr (I < N) {
    f(Const<I>{});
    unroll<N, I + 1>(f);
  }
}

// A thread's amplitudes by register pattern (bit 0 = index bit 0, bit j = slot j), between
// a tile in shared memory and the named registers of A.  Pair q: the N other slots as its
// bits (rphys: their places).
template <int N>
__device__ __forceinline__ uint32_t piece(const uint16_t (&rphys)[N], int q) {
  uint32_t o = 0;
#pragma unroll
  for (int j = 0; j < N; ++j)
    if ((q >> j) & 1) o ^= rphys[j];
  return o;
}
template <typename A, int N>
__device__ __forceinline__ void load_regs(const uint16_t (&rphys)[N], const float2* tile, uint32_t tp) {
  const uint32_t at = bulk::smem_addr(tile);
  unroll<1 << N>([&](auto q) { A::template load<2 * q.value>(at + 8 * (tp ^ piece(rphys, q.value))); });
}
template <typename A, int N>
__device__ __forceinline__ void store_regs(const uint16_t (&rphys)[N], float2* tile, uint32_t tp) {
  const uint32_t at = bulk::smem_addr(tile);
  unroll<1 << N>([&](auto q) { A::template store<2 * q.value>(at + 8 * (tp ^ piece(rphys, q.value))); });
}

// The pairs of AMPS register patterns that differ in slot S; MASK: those in rmask only.
template <int S, bool MASK, int AMPS, typename F>
__device__ __forceinline__ void each_pair(uint32_t rmask, const F& f) {
  unroll<AMPS>([&](auto q) {
    if constexpr (!((q.value >> S) & 1))
      if (!MASK || ((rmask >> q.value) & 1u)) f(q, Const<q.value | (1 << S)>{});
  });
}

}  // namespace sweep
}  // namespace tqk
