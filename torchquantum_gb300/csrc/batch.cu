// batch.cu -- persistent runner for many independent circuits of different sizes.
//
// A circuit is a list of passes (tqk_batch_plan); a pass holds ops whose target bits lie
// in a tile of 2^tile_bits amplitudes (tile_mask, tile_bits 10..14 per launch), applied
// tile by tile in shared memory: gather the tile from the circuit's state, apply every op
// of the pass in register sweeps, scatter it back.  Circuits with n <= tile_bits are one tile
// and one pass: their whole life is in shared memory.  Diagonal ops (CZ, CZ ladders) and controls need
// no tile bit -- their signs split into per-tile constants and tile-local terms -- so the
// planner gives them to any pass.
//
// Work is one item per (circuit, pass, tile) (tqk_batch_items), handed out in waves of
// pass index by a global counter to persistent CTAs (1..8 per SM), so the tiles of a large
// circuit's pass run on many SMs at once.  An item of pass p > 0 waits (bounded) for the
// completion counter of pass p - 1; every item's dependencies are handed out before it,
// so the earliest unfinished item can always run (a CTA takes its next item while it stores
// the current one, never before).  A tile publishes its stores
// (__threadfence) before counting itself done; dependent tiles read through L2
// (cp.async.cg) since their SM's L1 may hold the previous pass's lines.  Last-pass tiles
// add their <Z> partial (float64 atomics) and the tile that completes a circuit stamps
// its completion time.
#include <stdint.h>

#include <vector>

#include "bulk.cuh"
#include "common.cuh"
#include "sweep.cuh"

namespace tqk {
namespace batch {

constexpr int kMaxTileBits = TQK_BATCH_TILE_BITS;
constexpr int kMinTileBits = 10;
constexpr int kLowReserve = 5;  // address bits 0-4 stay in every tile: warps read 256-byte runs
constexpr int kFirst = 1, kLast = 2;

struct Tabs {
  uint32_t lo[128];  // amplitude offset of tile index bits 0-6
  uint32_t hi[128];  // ... and bits 7-13
};

__device__ __forceinline__ uint32_t dep(const Tabs& t, uint32_t l) { return t.lo[l & 127] + t.hi[l >> 7]; }

__device__ __forceinline__ int local_pos(uint32_t tmask, int b) { return __popc(tmask & ((1u << b) - 1u)); }

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

constexpr long long kWaitCycles = 4000000000ll;  // ~2 s at 2 GHz

// ------------------------------------------------------------------ sweeps
// A pass's ops run from registers (sweep.cuh): the ops are taken in order, a sweep ending before
// the op whose target would be the fifth besides tile bit 0 (or after kSweepOps; with 16
// amplitudes a thread, the fourth).  A warp of its own reads the ops ahead of the others, cuts the
// next sweep and writes it out while they run the current one, so a sweep costs them one
// barrier, the one after its stores.  (Reading and cutting in every warp between the barriers:
// 13.3 ms below.)
// What bounds it: float32 multiply-adds (8 per amplitude and one-qubit op: 4.9 us of the 11 us a
// 2^13-amplitude item of 18 such ops takes an SM), the two shared-memory crossings of a sweep
// (2.5 us) and the latency of 12 warps an SM, all the registers allow.  256 circuits of n = 8..20
// and 2..40 layers, ms: one op per crossing and barrier 11.4 (13-bit tiles, 3 CTAs of 256);
// sweeps of 16 amplitudes a thread 8.9 (3 x 256), of 32 8.4 (3 x 128).  96 circuits of up to 13
// qubits, one tile each: 0.58 before, 0.38 now (256 threads, 32 amplitudes).  A row of fewer
// amplitudes than a thread holds works in a tile of that many, the rest zero: 119 circuits of 7
// qubits and 17 layers, launch included, 112 us op by op (each op's and matrix's read before it), 88 in
// sweeps.
constexpr int kMaxAmpBits = 5;  // 2^AB amplitudes per thread: AB = 5, or 4 where CTAs are many
constexpr int kSweepOps = 8;

// How a sweep's threads run an op.  Patterns: sets of a thread's registers.
// Below 16: a 2x2 matrix on slot (code & 7); with SW_SOME on the patterns `reg` only.
enum { SW_SOME = 8, SW_SIGN = 16, SW_NONE = 17 };
struct alignas(16) SweepOp {
  int code;
  uint32_t reg;    // matrix: patterns it acts on; signs: patterns negated in every thread
  uint32_t need;   // matrix: thread bits that must be set; signs: if not 0, all set negates ..
  uint32_t reg2;   // signs: .. these patterns
  uint32_t lin;    // signs: each of these thread bits negates every pattern
  uint32_t quad;   // signs: each pair of thread bits (b, b + 1), b in quad, negates every pattern
  uint16_t side[kMaxAmpBits];  // signs: by slot: thread bits that each negate the patterns with it set
};
struct SweepRec {
  int count;
  uint16_t rphys[kMaxAmpBits - 1];  // places of the register bits (slots 1 ..)
  uint32_t lane[32], high[32];   // a thread's tile offset (low half) and its place: by lane, by the bits above
  SweepOp op[kSweepOps];
  float4 m[kSweepOps][4];  // (re, re, im, -)
};

__device__ __forceinline__ uint32_t slot_patterns(int s) {
  constexpr uint32_t p[kMaxAmpBits] = {0xaaaaaaaau, 0xccccccccu, 0xf0f0f0f0u, 0xff00ff00u, 0xffff0000u};
  return p[s];
}

// Bits of v at the bits of mask, moved together.
__device__ __forceinline__ uint32_t gather_bits(uint32_t v, uint32_t mask) {
  uint32_t r = 0;
  for (int j = 0; mask != 0; mask &= mask - 1, ++j) r |= ((v >> (__ffs(mask) - 1)) & 1u) << j;
  return r;
}

// The warp that prepares the sweeps.  Lane l holds the op whose index is l modulo 32, of the
// 32 next ones: its reads were issued several sweeps before it is needed.
template <int AB>
struct SweepMaker {
  const tqk_batch_op* ops;
  const float2* mats;
  int num_ops, n, tb;
  uint32_t tmask, base;
  int at, mine;  // next op; this lane's
  tqk_batch_op op;
  float2 m[4];
  bool fresh;  // op read, its matrix not yet

  __device__ __forceinline__ void read_op() {
    if (mine < num_ops) {
      op = ops[mine];
      fresh = true;
    }
  }
  __device__ __forceinline__ void start(int lane) {
    at = 0;
    mine = lane;
    fresh = false;
    read_op();
  }

  // The ladder's or pair's signs: CZ on (b, b + 1), b in `pairs` (bits of the state).
  __device__ __forceinline__ void ladder(uint32_t pairs, uint32_t regs, const int (&r)[AB], SweepOp& so) const {
    const uint32_t in = tmask, out = base;  // base: bits outside the tile
    const uint32_t lin = gather_bits(in & (((out >> 1) & pairs) ^ ((out & pairs) << 1)), in);
    const uint32_t quad = gather_bits(in & (in >> 1) & pairs, in);
    signs((__popc(out & (out >> 1) & pairs) & 1) ? ~0u : 0u, lin, quad, regs, r, so);
  }
  // Signs from terms in tile bits: constant patterns, single bits and neighbours (b, b + 1).
  __device__ __forceinline__ void signs(uint32_t constant, uint32_t lin, uint32_t quad, uint32_t regs,
                                        const int (&r)[AB], SweepOp& so) const {
    so.code = SW_SIGN;
    so.reg = constant;
    so.need = so.reg2 = 0u;
    so.lin = lin & ~regs;
    so.quad = quad & ~regs & ~(regs >> 1);
    uint32_t side[AB];
#pragma unroll
    for (int s = 0; s < AB; ++s) {
      const uint32_t own = slot_patterns(s), bit = 1u << r[s];
      if (lin & bit) so.reg ^= own;
      side[s] = 0;
      if (quad & bit) {  // (r, r + 1)
        const uint32_t up = bit << 1;
        if (regs & up) {
#pragma unroll
          for (int t = 0; t < AB; ++t)
            if (r[t] == r[s] + 1) so.reg ^= own & slot_patterns(t);
        } else {
          side[s] |= up;
        }
      }
      if (r[s] > 0 && (quad & (bit >> 1)) && !(regs & (bit >> 1))) side[s] ^= bit >> 1;  // (r - 1, r)
    }
#pragma unroll
    for (int s = 0; s < kMaxAmpBits; ++s) so.side[s] = static_cast<uint16_t>(s < AB ? side[s < AB ? s : 0] : 0u);
  }

  // CZ of two bits of the state.
  __device__ __forceinline__ void cz(int b0, int b1, uint32_t regs, const int (&r)[AB], SweepOp& so) const {
    const bool in0 = (tmask >> b0) & 1u, in1 = (tmask >> b1) & 1u;
    if ((!in0 && !((base >> b0) & 1u)) || (!in1 && !((base >> b1) & 1u))) {  // never set
      so.code = SW_NONE;
      return;
    }
    uint32_t pat = ~0u, need = 0;
    auto take = [&](bool in, int b) {
      if (!in) return;
      const int l = local_pos(tmask, b);
      if (!((regs >> l) & 1u)) need |= 1u << l;
#pragma unroll
      for (int s = 0; s < AB; ++s)
        if (r[s] == l) pat &= slot_patterns(s);
    };
    take(in0, b0);
    take(in1, b1);
    so.code = SW_SIGN;
    so.lin = so.quad = 0u;
#pragma unroll
    for (int s = 0; s < kMaxAmpBits; ++s) so.side[s] = 0;
    so.need = need;
    so.reg = need ? 0u : pat;
    so.reg2 = pat;
  }

  __device__ __forceinline__ void make(SweepRec& rec) {
    const int lane = threadIdx.x & 31;
    if (fresh) {
      if (op.kind == TQK_B_DENSE1 || op.kind == TQK_B_CTRL1) {
#pragma unroll
        for (int e = 0; e < 4; ++e) m[e] = __ldg(mats + 4 * static_cast<int64_t>(op.mat) + e);
      }
      fresh = false;
    }
    int target = 0;  // a tile bit; 0 (always a register) for the others
    if (mine < num_ops && op.kind <= TQK_B_CTRL1)
      target = local_pos(tmask, n - 1 - (op.kind == TQK_B_DENSE1 ? op.w0 : op.w1));
    // by position from `at`: the targets of the ops up to each
    uint32_t tg = __shfl_sync(0xffffffffu, target > 0 ? 1u << target : 0u, (at + lane) & 31);
    if (at + lane >= num_ops) tg = 0u;
#pragma unroll
    for (int d = 1; d < kSweepOps; d <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, tg, d);
      if (lane >= d) tg |= v;
    }
    const bool fit = lane < kSweepOps && at + lane < num_ops && __popc(tg) <= AB - 1;
    const int count = __ffs(~__ballot_sync(0xffffffffu, fit)) - 1;  // leading ops that fit
    uint32_t regs = __shfl_sync(0xffffffffu, tg, count > 0 ? count - 1 : 0);
    if (count == 0) regs = 0u;
    for (int b = tb - 1; __popc(regs) < AB - 1; --b) regs |= 1u << b;  // tb >= AB: never bit 0
    regs |= 1u;
    int r[AB];
    {
      uint32_t left = regs;
#pragma unroll
      for (int s = 0; s < AB; ++s, left &= left - 1) r[s] = __ffs(left) - 1;
    }
    const int pos = (lane - at) & 31;
    if (pos < count) {
      SweepOp so;
      if (op.kind <= TQK_B_CTRL1) {
        so.code = __popc(regs & ((1u << target) - 1u));
        so.reg = ~0u;
        so.need = 0u;
        if (op.kind == TQK_B_CTRL1) {
          const int cb = n - 1 - op.w0;
          if (!((tmask >> cb) & 1u)) {
            if (!((base >> cb) & 1u)) so.code = SW_NONE;  // control outside the tile and clear
          } else {
            const int lc = local_pos(tmask, cb);
            if ((regs >> lc) & 1u) {
              so.code |= SW_SOME;
#pragma unroll
              for (int s = 0; s < AB; ++s)
                if (r[s] == lc) so.reg = slot_patterns(s);
            } else {
              so.need = 1u << lc;
            }
          }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) rec.m[pos][e] = make_float4(m[e].x, m[e].x, m[e].y, 0.f);
      } else if (op.kind == TQK_B_CZ) {
        cz(n - 1 - op.w0, n - 1 - op.w1, regs, r, so);
      } else {  // ladder: bits n - 1 - w1 .. n - 1 - w0
        ladder(((1u << (op.w1 - op.w0)) - 1u) << (n - 1 - op.w1), regs, r, so);
      }
      rec.op[pos] = so;
      mine += 32;
      read_op();
    }
    // The thread bits: of the lowest three lane bits one in each class (bit - 1) mod 3 (the 16-byte
    // pieces of 8 lanes then lie in different banks), the others ascending.
    uint32_t free = ((1u << tb) - 1u) & ~regs, v = 0, hv = 0;
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      const uint32_t cls = j < 3 ? free & (0x2492u << j) : 0u, bit = cls ? cls & (~cls + 1u) : free & (~free + 1u);
      if ((lane >> j) & 1) v |= bit;
      free ^= bit;
    }
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      const uint32_t bit = free & (~free + 1u);
      if ((lane >> j) & 1) hv |= bit;
      free ^= bit;
    }
    rec.lane[lane] = v | sweep::swz(v) << 16;
    rec.high[lane] = hv | sweep::swz(hv) << 16;
    if (lane == 0) {
      rec.count = count;
#pragma unroll
      for (int s = 1; s < AB; ++s) rec.rphys[s - 1] = static_cast<uint16_t>(sweep::swz(1u << r[s]));
    }
    at += count;
  }
};

// Negate the register patterns of mask.
template <int AB>
__device__ __forceinline__ void flip_patterns(uint32_t mask) {
  if (mask == 0) return;
  sweep::unroll<1 << AB>([&](auto q) {
    const uint32_t s = (mask << (31 - q.value)) & 0x80000000u;
    f2::Psi::flip<q.value>((static_cast<f2::pair>(s) << 32) | s);
  });
}

template <int AB, int S, bool MASK>
__device__ __forceinline__ void dense_rows(const float4* m4, uint32_t rmask) {
  f2::Factor m[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(m4 + e);
    m[e] = {v.x, __uint_as_float(static_cast<uint32_t>(v.y))};
  }
  if constexpr (S < AB)
    sweep::each_pair<S, MASK, 1 << AB>(rmask, [&](auto q, auto u) { f2::Psi::dense2<q.value, u.value>(m); });
}

// Run a sweep on the tile (all threads but the preparing warp).
template <int THREADS, int AB>
__device__ __forceinline__ void run_sweep(const SweepRec& rec, float2* amp, int tb) {
  const int count = rec.count;
  // read again at each use: kept, the 16 places are registers that the amplitudes need
  auto places = [&](uint16_t (&rphys)[AB - 1]) {
#pragma unroll
    for (int j = 0; j < AB - 1; ++j) rphys[j] = *const_cast<const volatile uint16_t*>(rec.rphys + j);
  };
  const uint32_t slots = 1u << (tb - AB);  // threads' worth of amplitudes
#pragma unroll 1
  for (uint32_t vt = threadIdx.x; vt < slots; vt += THREADS) {  // (part of a warp in the smallest tiles)
    const uint32_t e = rec.lane[threadIdx.x & 31] ^ rec.high[vt >> 5], tl = e & 0xffffu;
    {
      uint16_t rphys[AB - 1];
      places(rphys);
      sweep::load_regs<f2::Psi>(rphys, amp, e >> 16);
    }
#pragma unroll 1
    for (int j = 0; j < count; ++j) {
      const SweepOp& so = rec.op[j];
      const int4 head = *reinterpret_cast<const int4*>(&so);
      const int code = head.x;
      const uint32_t need = static_cast<uint32_t>(head.z);
      if (code < SW_SIGN) {
        if ((tl & need) == need) {
          const float4* m4 = rec.m[j];
          switch (code) {
            case 0: dense_rows<AB, 0, false>(m4, 0u); break;
            case 1: dense_rows<AB, 1, false>(m4, 0u); break;
            case 2: dense_rows<AB, 2, false>(m4, 0u); break;
            case 3: dense_rows<AB, 3, false>(m4, 0u); break;
            case 4: dense_rows<AB, 4, false>(m4, 0u); break;
            case SW_SOME | 0: dense_rows<AB, 0, true>(m4, so.reg); break;
            case SW_SOME | 1: dense_rows<AB, 1, true>(m4, so.reg); break;
            case SW_SOME | 2: dense_rows<AB, 2, true>(m4, so.reg); break;
            case SW_SOME | 3: dense_rows<AB, 3, true>(m4, so.reg); break;
            default: dense_rows<AB, 4, true>(m4, so.reg); break;
          }
        }
      } else if (code == SW_SIGN) {
        uint32_t mask = so.reg;
        if ((__popc(tl & so.lin) + __popc(tl & (tl >> 1) & so.quad)) & 1) mask = ~mask;
        if (so.need != 0u && (tl & so.need) == so.need) mask ^= so.reg2;
#pragma unroll
        for (int s = 0; s < AB; ++s)
          if (__popc(tl & so.side[s]) & 1) mask ^= slot_patterns(s);
        flip_patterns<AB>(mask);
      }
    }
    uint16_t rphys[AB - 1];
    places(rphys);
    sweep::store_regs<f2::Psi>(rphys, amp, e >> 16);
  }
}

// The two sides of an item's sweeps, from before the barrier that ends the tile's load.  Calls,
// not inlined: each side has the registers to itself.
template <int AB>
__device__ __noinline__ void make_sweeps(SweepRec* rec, const tqk_batch_op* ops, int num_ops, const float2* mats,
                                         int n, uint32_t tmask, uint32_t base) {
  SweepMaker<AB> s;
  s.ops = ops;
  s.mats = mats;
  s.num_ops = num_ops;
  s.n = n;
  s.tb = max(__popc(tmask), AB);
  s.tmask = tmask;
  s.base = base;
  s.start(threadIdx.x & 31);
  s.make(rec[0]);
  __syncthreads();
#pragma unroll 1
  for (int sw = 0; rec[sw & 1].count != 0; ++sw) {
    s.make(rec[(sw + 1) & 1]);
    __syncthreads();
  }
}

template <int THREADS, int AB>
__device__ __noinline__ void run_sweeps(const SweepRec* rec, float2* amp, int tb) {
  TQK_AMPLITUDE_REGISTERS_32;
  __syncthreads();
#pragma unroll 1
  for (int sw = 0; rec[sw & 1].count != 0; ++sw) {
    run_sweep<THREADS, AB>(rec[sw & 1], amp, tb);
    __syncthreads();
  }
}

// An item as its CTA works on it.
struct Work {
  int valid;  // 0: no more items; -1: a plan made for a larger tile
  int circuit, pass, flags, num_ops, n, z_wire, prev_tiles, ntiles;
  uint32_t tmask, base;  // bits of the tile; value of the others
  const tqk_batch_op* ops;
  float2* state;  // NULL: the circuit has none
};

// The next item into w and its tables into tabs (one warp).
__device__ __noinline__ void fetch_item(Work& w, Tabs& tabs, const tqk_batch_circuit* circ, const tqk_batch_op* ops,
                                        const tqk_batch_pass* passes, const tqk_batch_item* items, long long n_items,
                                        float2* states, int* counter, int max_tb) {
  const int lane = threadIdx.x & 31;
  int i = lane == 0 ? atomicAdd(counter, 1) : 0;
  i = __shfl_sync(0xffffffffu, i, 0);
  if (i >= n_items) {
    if (lane == 0) w.valid = 0;
    return;
  }
  const tqk_batch_item it = items[i];
  const tqk_batch_pass P = passes[it.pass];
  const tqk_batch_circuit C = circ[it.circuit];
  const int n = C.n, tb = __popc(P.tile_mask);
  const uint32_t omask = (n >= 32 ? 0xffffffffu : ((1u << n) - 1u)) & ~P.tile_mask;
  uint32_t base = 0;
  for (int b = 0, j = 0; b < n; ++b) {
    if (!((omask >> b) & 1u)) continue;
    if ((it.tile >> j) & 1) base |= 1u << b;
    ++j;
  }
  // deposit tables of the tile bits: lo[x] from the first 7, hi[x] from the others (lane: x's
  // low 5 bits)
  uint32_t low = 0, add[4] = {0u, 0u, 0u, 0u}, low2 = 0;
  uint32_t left = P.tile_mask;
  for (int j = 0; j < 14 && left != 0; ++j, left &= left - 1) {
    const uint32_t bit = left & (~left + 1u);
    const int k = j % 7;
    if (k < 5) {
      if ((lane >> k) & 1) (j < 7 ? low : low2) |= bit;
    } else {
      add[(j < 7 ? 0 : 2) + k - 5] = bit;
    }
  }
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    tabs.lo[32 * x + lane] = low | (x & 1 ? add[0] : 0u) | (x & 2 ? add[1] : 0u);
    tabs.hi[32 * x + lane] = low2 | (x & 1 ? add[2] : 0u) | (x & 2 ? add[3] : 0u);
  }
  if (lane == 0) {
    w.valid = tb > max_tb || tb < 1 ? -1 : 1;
    w.circuit = it.circuit;
    w.pass = it.pass;
    w.flags = P.flags;
    w.num_ops = P.num_ops;
    w.n = n;
    w.z_wire = C.z_wire;
    w.prev_tiles = (P.flags & kFirst) ? 0 : 1 << (n - __popc(passes[it.pass - 1].tile_mask));
    w.ntiles = 1 << (n - tb);
    w.tmask = P.tile_mask;
    w.base = base;
    w.ops = ops + P.first_op;
    w.state = C.state_off >= 0 ? states + C.state_off : nullptr;
  }
}

// THREADS threads per CTA and a warp that prepares (the next item, its sweeps), MINB CTAs per
// SM for the register budget; the tile holds up to 2^max_tb amplitudes (dynamic shared
// memory).
template <int THREADS, int MINB, int AB>
__global__ void __launch_bounds__(THREADS + 32, MINB)
    k_batch(const tqk_batch_circuit* circ, int ncirc, const tqk_batch_op* ops, const tqk_batch_pass* passes,
            const tqk_batch_item* items, long long n_items, const float2* mats, float2* states, int write_states,
            double* z_out, int* pass_done, unsigned long long* t_done, int* counter, int* status, int max_tb) {
  extern __shared__ float4 amp_raw[];  // 16-byte aligned: ops use float4 accesses
  float2* amp = reinterpret_cast<float2*>(amp_raw);
  __shared__ Tabs tab_buf[2];
  __shared__ Work work[2];
  __shared__ SweepRec rec[2];
  __shared__ double red[THREADS / 32];
  const bool maker = threadIdx.x >= THREADS;  // the warp that prepares
  const uint32_t tid = threadIdx.x;
  if (t_done != nullptr && blockIdx.x == 0 && threadIdx.x == 0) t_done[ncirc] = global_ns();
  if (maker) fetch_item(work[0], tab_buf[0], circ, ops, passes, items, n_items, states, counter, max_tb);
  __syncthreads();
  for (int cur = 0;; cur ^= 1) {
    const Work& W = work[cur];
    const Tabs& tabs = tab_buf[cur];
    if (W.valid == 0) break;
    if (W.valid < 0) {  // record and skip the item
      if (threadIdx.x == 0) {
        atomicExch(status, TQK_BAD_SHAPE);
        atomicAdd(pass_done + W.pass, 1);
      }
      __syncthreads();  // the other slot's item is done with
      if (maker)
        fetch_item(work[cur ^ 1], tab_buf[cur ^ 1], circ, ops, passes, items, n_items, states, counter, max_tb);
      __syncthreads();
      continue;
    }
    const int tb = __popc(W.tmask);
    const uint32_t tsz = 1u << tb;
    if (W.prev_tiles > 0) {  // every tile of the previous pass must be stored
      if (threadIdx.x == 0) {
        const volatile int* d = pass_done + W.pass - 1;
        const long long t0 = clock64();
        while (*d < W.prev_tiles) {
          if (clock64() - t0 > kWaitCycles) {
            atomicExch(status, TQK_TIMEOUT);
            break;
          }
        }
        __threadfence();
      }
      __syncthreads();
    }
    if (maker) {
      make_sweeps<AB>(rec, W.ops, W.num_ops, mats, W.n, W.tmask, W.base);
      fetch_item(work[cur ^ 1], tab_buf[cur ^ 1], circ, ops, passes, items, n_items, states, counter, max_tb);
    } else {
      if (W.flags & kFirst) {
        for (uint32_t l = tid; l < max(tsz, 1u << AB); l += THREADS)
          amp[sweep::swz(l)] = make_float2((W.base == 0u && l == 0) ? 1.f : 0.f, 0.f);
      } else if (2u * tid < tsz) {
        // 16-byte pieces through L2 (another SM may have stored them: .cg skips this SM's L1);
        // tile bits 0-4 are address bits 0-4, so a warp's pieces are 256-byte runs
        // (both places are linear: that of tile index l + k is the sum or XOR of theirs)
        const float2* src = W.state + W.base + dep(tabs, 2u * tid);
        const uint32_t dst = sweep::swz(2u * tid);
        for (uint32_t k = 0; k < tsz; k += 2u * THREADS)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(bulk::smem_addr(amp + (dst ^ sweep::swz(k)))),
                       "l"(src + dep(tabs, k))
                       : "memory");
        asm volatile("cp.async.wait_all;" ::: "memory");
      }
      run_sweeps<THREADS, AB>(rec, amp, max(tb, AB));
      if (W.flags & kLast) {
        const int zbit = W.n - 1 - W.z_wire;
        const bool in = (W.tmask >> zbit) & 1u;
        const int zl = local_pos(W.tmask, zbit);
        const uint32_t out = (W.base >> zbit) & 1u;
        double zacc = 0.0;
        for (uint32_t l = tid; l < tsz; l += THREADS) {
          const float2 a = amp[sweep::swz(l)];
          const bool minus = in ? (l >> zl) & 1u : out;
          zacc = fma(static_cast<double>(a.x), static_cast<double>(minus ? -a.x : a.x), zacc);
          zacc = fma(static_cast<double>(a.y), static_cast<double>(minus ? -a.y : a.y), zacc);
        }
        for (int o = 16; o > 0; o >>= 1) zacc += __shfl_xor_sync(0xffffffffu, zacc, o);
        if ((tid & 31) == 0) red[tid >> 5] = zacc;
      }
      if (((W.flags & kLast) == 0 || write_states) && W.state != nullptr && 2u * tid < tsz) {
        float2* dst = W.state + W.base + dep(tabs, 2u * tid);
        const uint32_t src = sweep::swz(2u * tid);
        for (uint32_t k = 0; k < tsz; k += 2u * THREADS)
          *reinterpret_cast<float4*>(dst + dep(tabs, k)) =
              *reinterpret_cast<const float4*>(amp + (src ^ sweep::swz(k)));
      }
      __threadfence();  // stored before the tile counts as done
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      if (W.flags & kLast) {
        double sum = 0.0;
        for (int w = 0; w < THREADS / 32; ++w) sum += red[w];
        atomicAdd(z_out + W.circuit, sum);
        __threadfence();
      }
      const int old = atomicAdd(pass_done + W.pass, 1);
      if ((W.flags & kLast) && old == W.ntiles - 1 && t_done != nullptr) t_done[W.circuit] = global_ns();
    }
  }
}

// Bits of an op's wires (all of them) and of its targets (the bits that must be in the tile).
void op_bits(const tqk_batch_op& op, int n, uint32_t* wires, uint32_t* targets) {
  auto bit = [n](int w) { return 1u << (n - 1 - w); };
  switch (op.kind) {
    case TQK_B_DENSE1:
      *wires = *targets = bit(op.w0);
      break;
    case TQK_B_CTRL1:
      *wires = bit(op.w0) | bit(op.w1);
      *targets = bit(op.w1);
      break;
    case TQK_B_CZ:
      *wires = bit(op.w0) | bit(op.w1);
      *targets = 0;
      break;
    default: {  // ladder
      uint32_t m = 0;
      for (int w = op.w0; w <= op.w1; ++w) m |= bit(w);
      *wires = m;
      *targets = 0;
    }
  }
}

}  // namespace batch
}  // namespace tqk

using namespace tqk;

extern "C" int tqk_batch_plan(tqk_batch_circuit* circuits, int ncirc, const tqk_batch_op* ops_in, int n_mats,
                              tqk_batch_op* ops_out, tqk_batch_pass* passes, int max_passes, int tile_bits) {
  const char* what = "tqk_batch_plan";
  if (ncirc < 0) return -fail(TQK_BAD_SHAPE, "%s: ncirc %d", what, ncirc);
  if (ncirc > 0 && (!circuits || !passes || !ops_out)) return -fail(TQK_BAD_POINTER, "%s: null pointer", what);
  if (tile_bits < batch::kMinTileBits || tile_bits > batch::kMaxTileBits)
    return -fail(TQK_BAD_SHAPE, "%s: tile_bits %d outside %d..%d", what, tile_bits, batch::kMinTileBits,
                 batch::kMaxTileBits);
  const int T = tile_bits;
  int np = 0;
  for (int ci = 0; ci < ncirc; ++ci) {
    tqk_batch_circuit& c = circuits[ci];
    const int n = c.n;
    if (n < 1 || n > TQK_BATCH_MAX_QUBITS) return -fail(TQK_TOO_MANY_QUBITS, "%s: circuit %d has n=%d", what, ci, n);
    if (c.z_wire < 0 || c.z_wire >= n) return -fail(TQK_BAD_WIRES, "%s: circuit %d z_wire %d", what, ci, c.z_wire);
    if (c.num_ops < 0 || c.first_op < 0 || (c.num_ops > 0 && !ops_in))
      return -fail(TQK_BAD_SHAPE, "%s: circuit %d op range", what, ci);
    for (int k = 0; k < c.num_ops; ++k) {
      const tqk_batch_op& op = ops_in[c.first_op + k];
      const bool two = op.kind == TQK_B_CTRL1 || op.kind == TQK_B_CZ || op.kind == TQK_B_CZ_LADDER;
      if (op.kind < TQK_B_DENSE1 || op.kind > TQK_B_CZ_LADDER)
        return -fail(TQK_BAD_SHAPE, "%s: circuit %d op %d kind %d", what, ci, k, op.kind);
      if (op.w0 < 0 || op.w0 >= n || (two && (op.w1 < 0 || op.w1 >= n)))
        return -fail(TQK_BAD_WIRES, "%s: circuit %d op %d wires out of range", what, ci, k);
      if ((op.kind == TQK_B_CTRL1 || op.kind == TQK_B_CZ) && op.w0 == op.w1)
        return -fail(TQK_BAD_WIRES, "%s: circuit %d op %d uses a wire twice", what, ci, k);
      if (op.kind == TQK_B_CZ_LADDER && op.w1 <= op.w0)
        return -fail(TQK_BAD_WIRES, "%s: circuit %d op %d ladder needs w0 < w1", what, ci, k);
      if ((op.kind == TQK_B_DENSE1 || op.kind == TQK_B_CTRL1) && (op.mat < 0 || op.mat >= n_mats))
        return -fail(TQK_BAD_SHAPE, "%s: circuit %d op %d matrix index %d (have %d)", what, ci, k, op.mat, n_mats);
    }
    c.first_pass = np;
    const uint32_t full = (n >= 32) ? 0xffffffffu : ((1u << n) - 1u);
    if (n <= T) {  // one tile, one pass
      if (np >= max_passes) return -fail(TQK_SCRATCH_TOO_SMALL, "%s: more than %d passes", what, max_passes);
      for (int k = 0; k < c.num_ops; ++k) ops_out[c.first_op + k] = ops_in[c.first_op + k];
      passes[np++] = {c.first_op, c.num_ops, full, batch::kFirst | batch::kLast};
    } else {
      if (c.state_off < 0) return -fail(TQK_BAD_POINTER, "%s: circuit %d (n=%d) needs a state buffer", what, ci, n);
      const uint32_t low = (1u << batch::kLowReserve) - 1u;
      std::vector<int> pending(c.num_ops), rest;
      for (int k = 0; k < c.num_ops; ++k) pending[k] = c.first_op + k;
      int out = c.first_op;
      do {
        uint32_t tile = low, blocked = 0;
        const int start = out;
        rest.clear();
        for (int idx : pending) {
          uint32_t wb, tg;
          batch::op_bits(ops_in[idx], n, &wb, &tg);
          if ((wb & blocked) == 0u && __builtin_popcount(tile | tg) <= T) {
            tile |= tg;
            ops_out[out++] = ops_in[idx];
          } else {  // stays for a later pass; later ops on these wires must wait too
            blocked |= wb;
            rest.push_back(idx);
          }
        }
        for (int b = 0; b < n && __builtin_popcount(tile) < T; ++b) tile |= 1u << b;  // fill with low bits
        if (np >= max_passes) return -fail(TQK_SCRATCH_TOO_SMALL, "%s: more than %d passes", what, max_passes);
        passes[np++] = {start, out - start, tile & full, 0};
        pending.swap(rest);
      } while (!pending.empty());
      passes[c.first_pass].flags |= batch::kFirst;
      passes[np - 1].flags |= batch::kLast;
    }
    c.num_passes = np - c.first_pass;
  }
  return np;
}

extern "C" int64_t tqk_batch_items(const tqk_batch_circuit* circuits, int ncirc, const tqk_batch_pass* passes,
                                   tqk_batch_item* items, int64_t max_items) {
  const char* what = "tqk_batch_items";
  if (ncirc < 0) return -fail(TQK_BAD_SHAPE, "%s: ncirc %d", what, ncirc);
  if (ncirc > 0 && (!circuits || !passes || !items)) return -fail(TQK_BAD_POINTER, "%s: null pointer", what);
  int max_np = 0;
  for (int c = 0; c < ncirc; ++c) max_np = circuits[c].num_passes > max_np ? circuits[c].num_passes : max_np;
  int64_t k = 0;
  for (int w = 0; w < max_np; ++w) {
    for (int c = 0; c < ncirc; ++c) {
      if (w >= circuits[c].num_passes) continue;
      const int pi = circuits[c].first_pass + w;
      const int ntiles = 1 << (circuits[c].n - __builtin_popcount(passes[pi].tile_mask));
      for (int t = 0; t < ntiles; ++t) {
        if (k >= max_items) return -fail(TQK_SCRATCH_TOO_SMALL, "%s: more than %lld items", what, (long long)max_items);
        items[k++] = {c, pi, t, 0};
      }
    }
  }
  return k;
}

namespace {
// Kernel variants: (threads per CTA, CTAs per SM the register budget is sized for, amplitudes
// per thread as a power of two).
template <int THREADS, int MINB, int AB>
int launch_batch(const tqk_batch_circuit* circuits, int ncirc, const tqk_batch_op* ops, const tqk_batch_pass* passes,
                 const tqk_batch_item* items, int64_t n_items, const void* mats, void* states, int write_states,
                 double* z_out, int* pass_done, uint64_t* t_done, int* counter, int* status, int tile_bits,
                 int ctas_per_sm, cudaStream_t stream) {
  auto kern = batch::k_batch<THREADS, MINB, AB>;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const size_t smem = sizeof(float2) << tile_bits;
  // attributes are set once per device and variant (before any stream capture: the
  // first launch of a variant on a device must not be captured)
  static int attr_set[64] = {0};
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         static_cast<int>(sizeof(float2) << batch::kMaxTileBits));
    attr_set[dev] = 1;
  }
  int fit = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kern, THREADS + 32, smem) != cudaSuccess || fit < 1) fit = 1;
  const int per_sm = ctas_per_sm < fit ? ctas_per_sm : fit;
  const int64_t slots = static_cast<int64_t>(sms) * per_sm;
  const int grid = static_cast<int>(n_items < slots ? n_items : slots);
  kern<<<grid, THREADS + 32, smem, stream>>>(circuits, ncirc, ops, passes, items, n_items,
                                        static_cast<const float2*>(mats), static_cast<float2*>(states), write_states,
                                        z_out, pass_done, reinterpret_cast<unsigned long long*>(t_done), counter,
                                        status, tile_bits);
  return launch_status("tqk_batch_run");
}
}  // namespace

extern "C" int tqk_batch_run(const tqk_batch_circuit* circuits, int ncirc, const tqk_batch_op* ops,
                             const tqk_batch_pass* passes, const tqk_batch_item* items, int64_t n_items,
                             const void* mats, void* states, int write_states, double* z_out, int* pass_done,
                             uint64_t* t_done, int* counter, int* status, const tqk_batch_config* config,
                             void* stream) {
  const char* what = "tqk_batch_run";
  if (ncirc <= 0 || n_items <= 0) return TQK_OK;
  if (!circuits || !passes || !items || !z_out || !pass_done || !counter || !status)
    return fail(TQK_BAD_POINTER, "%s: null pointer", what);
  if (n_items > 0x7fffffff) return fail(TQK_BAD_SHAPE, "%s: too many items", what);
  tqk_batch_config cfg = {TQK_BATCH_TILE_BITS, 512, 1, 0};
  if (config) cfg = *config;
  if (cfg.tile_bits < batch::kMinTileBits || cfg.tile_bits > batch::kMaxTileBits)
    return fail(TQK_BAD_SHAPE, "%s: tile_bits %d outside %d..%d", what, cfg.tile_bits, batch::kMinTileBits,
                batch::kMaxTileBits);
  if (cfg.ctas_per_sm < 1 || cfg.ctas_per_sm > 8)
    return fail(TQK_BAD_SHAPE, "%s: ctas_per_sm %d outside 1..8", what, cfg.ctas_per_sm);
  cudaStream_t s = as_stream(stream);
#define TQK_BATCH_ARGS circuits, ncirc, ops, passes, items, n_items, mats, states, write_states, z_out, pass_done, \
                       t_done, counter, status, cfg.tile_bits, cfg.ctas_per_sm, s
  // 32 amplitudes a thread where the CTAs asked for leave it the registers (8.4 ms against 8.9 with
  // 16 for 256 circuits of 8 to 20 qubits), else 16
  switch (cfg.threads) {
    case 512:
      return launch_batch<512, 1, 4>(TQK_BATCH_ARGS);
    case 256:
      return cfg.ctas_per_sm >= 2 ? launch_batch<256, 3, 4>(TQK_BATCH_ARGS) : launch_batch<256, 1, 5>(TQK_BATCH_ARGS);
    case 128:
      // many CTAs of small tiles: a tile of 2^9 amplitudes is 32 threads' worth, and more threads a CTA only
      // keep CTAs off the SM (us, 128 threads of 32 amplitudes and 3 CTAs / of 16 and 6 / these 8: 2000
      // circuits of 5 qubits 184 / 137 / 106; 1000 of 10 378 / - / 215)
      if (cfg.ctas_per_sm >= 4 && cfg.tile_bits == 10) return launch_batch<32, 8, 4>(TQK_BATCH_ARGS);
      if (cfg.ctas_per_sm >= 4 && cfg.tile_bits == 11) return launch_batch<64, 8, 4>(TQK_BATCH_ARGS);
      return launch_batch<128, 3, 5>(TQK_BATCH_ARGS);
    default:
      return fail(TQK_BAD_SHAPE, "%s: threads %d (128, 256 or 512)", what, cfg.threads);
  }
#undef TQK_BATCH_ARGS
}
