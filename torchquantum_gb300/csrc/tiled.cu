// tiled.cu -- runs of gates on any qubits applied in one pass over the state.
//
// Gate by gate, the plain method streams the touched amplitudes through HBM once per gate:
// 40 gates on a 268 MB state (n = 22, bsz = 8) took 40 forward passes and as many reverse
// steps, each near the copy rate, 7.0 ms together.  A run of gates whose targets all lie in
// a set of 12 index bits (the tile bits) shares one pass instead: a CTA takes the 2^12
// amplitudes of a tile (every value of the tile bits, the other index bits fixed), applies
// every op of the run there, and writes the tile back.  Controls and the wires of diagonal
// ops may be anywhere: bits outside the tile are constants of the tile.  The same 40 gates
// are two passes each way, 2.1 ms together.
//
// Sweeps.  Inside a tile the ops run from registers.  A thread holds 16 amplitudes: every
// value of four "register bits", index bit 0 always one of them; the other tile bits come
// from the thread index.  An op whose target is a register bit needs no exchange at all.
// The host cuts the run into sweeps of ops with at most three targets besides bit 0 (ops on
// disjoint wires commute, so a sweep also takes later ops whose wires no earlier left-out
// op touches); between sweeps the tile crosses shared memory once, re-dealt to the next
// sweep's register bits.
//   What bounds it: issue slots, then the float32 pipe.  A dense op is 8 multiply-adds per
//   amplitude forward (6 issue slots, f32x2.cuh) and 24 in reverse with its cotangent; its
//   factors are read once per thread from a table in shared memory, and a crossing (2
//   instructions per amplitude) is shared by all ops of a sweep.  Measured per op of 120
//   RX, RY and RZ at n = 22, bsz = 8: 11.9 us forward and 39 us in reverse (36.5 with plain
//   float32 sums over the warp; float32 pipe alone: 7.2 and 22 a dense op); one op per
//   shared-memory crossing (staged.cu): 24 and 70 us.
//   Registers: 16 amplitudes are 32 registers forward, 64 for the reverse pass's psi and
//   lam, so 256 threads fit 3 and 2 CTAs per SM, whose loads, sweeps and stores overlap.
//   (32 amplitudes per thread: 3 % faster forward, 10 % slower in reverse; 4 CTAs of 64
//   registers: 10 % slower forward.)
//
// The reverse pass holds the psi and lam tiles of the same amplitudes and walks the run
// backwards: psi <- U^H psi, lam <- U^H lam and, for ops with a cotangent slot,
// sum lam_in conj(psi_out): float32 over a thread's amplitudes and eight threads (64 terms, as in
// the kernels of one gate), pairs of float32 (sum and error) over the warps and tiles, float64
// where the CTAs' sums meet.
#include <stdint.h>

#include <atomic>

#include "bulk.cuh"
#include "common.cuh"
#include "sweep.cuh"

namespace tqk {
namespace tiled {

using namespace sweep;

constexpr int kAmpBits = 4;  // 2^4 amplitudes per thread
constexpr int kAmps = 1 << kAmpBits;
constexpr int kMinBits = 9;  // a tile fills at least one warp
constexpr int kMaxBits = TQK_STAGED_MAX_TILE_BITS;
constexpr int kMaxThreads = 1 << (kMaxBits - kAmpBits);
constexpr int kMaxWarps = kMaxThreads / 32;
constexpr int kTabEntries = 32 + kMaxWarps;  // lane and warp parts of a sweep's thread mapping

// The code path an op takes, chosen on the host: one straight-line body per register slot
// for the common forms, so that the registers are updated in place.
enum {
  GO_DENSE = 0,    // + slot: 2x2, no condition on register bits
  GO_REAL = 4,     // + slot: the same with a real matrix (half the products)
  GO_MASK = 8,     // + slot: 2x2 where the register pattern satisfies the condition
  GO_X = 12,       // + slot: flip
  GO_XMASK = 16,   // + slot
  GO_SPLIT = 20,   // + slot: one factor where the register bit is clear, another where it is set
  GO_SCALE = 24,   // one factor for all registers
  GO_SCALEMASK = 25,
  GO_DIAG = 26     // two-bit diagonal with bits in registers
};

struct SOp {
  int32_t go;             // GO_*
  uint32_t rmask;         // register patterns whose bits satisfy the condition (bit p = pattern p)
  uint32_t tmask, tval;   // condition on the thread's tile-local bits
  uint64_t omask, oval;   // condition on the index bits outside the tile
  // diagonal ops: the entry index takes nd bits (most significant first), each from one place
  int32_t nd;
  int32_t dslot[2];       // register slot of the bit, or -1
  int32_t dbit[2];        // tile-local bit given by the thread, or -1
  int32_t obit[2];        // index bit outside the tile, or -1
  int32_t nent;           // operand entries (complex)
  int32_t matrix;         // the operand is a 2x2 matrix
  int32_t gidx;           // adjoint: index of the op's accumulator, or -1
  const float2* operand;  // [batch][nent]: 2x2 matrix, phase or diagonal
  int64_t op_stride;      // float2 per row (0 when shared by every row)
  double* grad;           // complex128 cotangent (interleaved), or null
  int64_t grad_stride;    // doubles per row (0 when shared)
};

struct Sweep {
  int16_t first, count;         // its ops
  uint16_t rphys[kAmpBits - 1]; // shared-memory offset of register slots 1..3
  uint8_t pos[8];               // local bit of each thread-index bit
};

struct Params {
  float2* psi;            // tiles are stored here ..
  float2* lam;
  const float2* psi_in;   // .. and loaded from here (in place: the same)
  const float2* lam_in;
  int n, m;               // qubits; tile bits
  int tiles_log;          // tiles per row: 2^tiles_log
  int per_row;            // some op has an operand for each row
  uint32_t items;         // tiles of all rows
  uint32_t row_ctas;      // CTAs of each row, or 0: an even share of the items each
  uint64_t outer;         // index bits outside the tile
  int nsweeps, nops, ngrad;
  uint8_t grad_op[TQK_STAGED_MAX_OPS];  // op of each accumulator
  uint8_t tb[kMaxBits];   // index bit of tile-local bit j (ascending)
  int64_t ioff[kAmps / 2];  // offset within the tile of copy piece group i
  Sweep sweeps[TQK_STAGED_MAX_OPS];
  SOp ops[TQK_STAGED_MAX_OPS];
};

// t deposited into the bits of mask
__device__ __forceinline__ uint64_t deposit(uint64_t t, uint64_t mask) {
  uint64_t r = 0;
  while (mask) {
    const uint64_t low = mask & (~mask + 1);
    if (t & 1) r |= low;
    t >>= 1;
    mask ^= low;
  }
  return r;
}

// Work: the tiles of all rows.  With operands that all rows share the CTAs take them in turn.  Else a
// CTA should work out its tables for few rows: while whole CTAs a row leave at most a sixteenth of the
// places empty, each row's CTAs take its tiles in turn; at more rows a CTA gets an even share of
// neighbouring tiles.  (Whole CTAs a row at any number of rows: 14 wires, 305 rows, two U3 22 us forward
// and 63 in reverse, now 18 and 52; shares at any number: 40 gates at 22 wires and 8 rows 2477 us a
// step, 2453 so.)
struct Items {
  uint32_t it, end, step;
};
__device__ __forceinline__ Items items_of(const Params& p) {
  const uint32_t c = blockIdx.x;
  if (!p.per_row) return {c, p.items, gridDim.x};
  if (p.row_ctas > 0) {
    const uint32_t row = c / p.row_ctas;
    return {(row << p.tiles_log) + c % p.row_ctas, (row + 1) << p.tiles_log, p.row_ctas};
  }
  const uint64_t n = p.items;
  return {static_cast<uint32_t>(n * c / gridDim.x), static_cast<uint32_t>(n * (c + 1) / gridDim.x), 1u};
}
__device__ __forceinline__ uint32_t tile_of(const Params& p, uint32_t it) { return it & ((1u << p.tiles_log) - 1u); }

// A thread's part of the tile copies, worked out anew for each copy: held across the op
// loop its addresses would take registers from the amplitudes.
struct Frame {
  int64_t off;     // state offset of the thread's first 16-byte piece
  uint32_t lphys;  // its offset in the tile
};

__device__ __forceinline__ Frame frame(const Params& p, uint32_t row, uint64_t base) {
  uint32_t l = threadIdx.x << 1;
  asm volatile("" : "+r"(l));  // not a loop invariant to the compiler
  Frame f;
  f.off = (static_cast<int64_t>(row) << p.n) + static_cast<int64_t>(base);
  for (int j = 1; j < p.m; ++j)
    if ((l >> j) & 1u) f.off += 1ll << p.tb[j];
  f.lphys = swz(l);
  return f;
}

// Issue the copies of one tile: 16-byte pieces at local 2 (tid + i threads).
__device__ __forceinline__ void load_tile(const Params& p, const Frame& f, const float2* state, float2* tile) {
#pragma unroll
  for (int i = 0; i < kAmps / 2; ++i) {
    const uint32_t dst = bulk::smem_addr(tile + (f.lphys ^ swz(static_cast<uint32_t>(i) * 2u * blockDim.x)));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(state + f.off + p.ioff[i]) : "memory");
  }
}

__device__ __forceinline__ void store_tile(const Params& p, const Frame& f, float2* state, const float2* tile) {
#pragma unroll
  for (int i = 0; i < kAmps / 2; ++i)
    *reinterpret_cast<float4*>(state + f.off + p.ioff[i]) =
        *reinterpret_cast<const float4*>(tile + (f.lphys ^ swz(static_cast<uint32_t>(i) * 2u * blockDim.x)));
}

__device__ __forceinline__ void wait_loads() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
}

// Thread mapping of every sweep: entry = logical offset | (shared-memory offset << 16).
__device__ __forceinline__ void build_tables(const Params& p, uint32_t* tab) {
  for (int i = threadIdx.x; i < p.nsweeps * kTabEntries; i += blockDim.x) {
    const Sweep& s = p.sweeps[i / kTabEntries];
    const int e = i % kTabEntries;
    uint32_t l = 0;
    if (e < 32)
      for (int j = 0; j < 5; ++j) l |= ((static_cast<uint32_t>(e) >> j) & 1u) << s.pos[j];
    else
      for (int j = 0; j < 3; ++j) l |= ((static_cast<uint32_t>(e - 32) >> j) & 1u) << s.pos[5 + j];
    tab[i] = l | (swz(l) << 16);
  }
}

// The thread's entry of a sweep; read where it is used, not kept.
__device__ __forceinline__ uint32_t thread_offset(const volatile uint32_t* tab, int s) {
  return tab[s * kTabEntries + (threadIdx.x & 31)] ^ tab[s * kTabEntries + 32 + (threadIdx.x >> 5)];
}

// ------------------------------------------------------------------ op tables
// What the op loop reads of an op, in shared memory.
struct Decoded {
  int32_t go, gidx;
  uint32_t tmask, tval;
  uint64_t omask, oval;
};

// Decoded ops and their factors for a row: fac[op][entry] = (re, re, im, -), of U
// or (ADJ) of U^H.
template <bool ADJ>
__device__ __forceinline__ void build_ops(const Params& p, int64_t row, float4* fac, Decoded* dec) {
  for (int j = threadIdx.x; j < p.nops; j += blockDim.x) {
    const SOp& o = p.ops[j];
    int go = o.go;
    if (go < GO_REAL) {
      bool real = true;
      for (int f = 0; f < 4; ++f) real &= __ldg(o.operand + row * o.op_stride + f).y == 0.f;
      if (real) go += GO_REAL - GO_DENSE;
    }
    dec[j] = {go, o.gidx, o.tmask, o.tval, o.omask, o.oval};
  }
  for (int i = threadIdx.x; i < p.nops * 4; i += blockDim.x) {
    const SOp& o = p.ops[i >> 2];
    int f = i & 3;
    if (f >= o.nent) continue;  // a flip has no entries and no operand
    if (ADJ && o.matrix) f = (f & 1) << 1 | f >> 1;
    const float2 v = __ldg(o.operand + row * o.op_stride + f);
    fac[i] = make_float4(v.x, v.x, ADJ ? -v.y : v.y, 0.f);
  }
}

struct Source {
  const Params& p;
  const float4* fac;
  __device__ __forceinline__ f2::Factor get(int j, int f) const {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(fac + 4 * j + f);
    return {v.x, __uint_as_float(static_cast<uint32_t>(v.y))};
  }
  __device__ __forceinline__ void matrix(int j, f2::Factor (&m)[4]) const {
#pragma unroll
    for (int f = 0; f < 4; ++f) m[f] = get(j, f);
  }
};

// ------------------------------------------------------------------ ops on one state
template <int S, bool MASK, typename A>
__device__ __forceinline__ void x_slot(uint32_t rmask) {
  each_pair<S, MASK, kAmps>(rmask, [&](auto q, auto u) { A::template swap<q.value, u.value>(); });
}

// Diagonal ops: entry-index bits that do not vary over the thread's registers, the bits
// that do, and the register patterns of each value of those.
__device__ __forceinline__ int diag_const(const SOp& o, uint32_t tl, uint64_t base) {
  int d = 0;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    if (j >= o.nd) break;
    const int place = o.nd - 1 - j;
    if (o.dbit[j] >= 0) d |= static_cast<int>((tl >> o.dbit[j]) & 1u) << place;
    else if (o.obit[j] >= 0) d |= static_cast<int>((base >> o.obit[j]) & 1u) << place;
  }
  return d;
}
__device__ __forceinline__ int diag_reg_bits(const SOp& o) {
  int v = 0;
  if (o.nd > 0 && o.dslot[0] >= 0) v |= 1 << (o.nd - 1);
  if (o.nd > 1 && o.dslot[1] >= 0) v |= 1;
  return v;
}
__device__ __forceinline__ uint32_t diag_patterns(const SOp& o, int e) {
  uint32_t m = 0xffffu;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    if (j >= o.nd || o.dslot[j] < 0) continue;
    const uint32_t sm = o.dslot[j] == 0 ? 0xaaaau : (o.dslot[j] == 1 ? 0xccccu : (o.dslot[j] == 2 ? 0xf0f0u : 0xff00u));
    m &= ((e >> (o.nd - 1 - j)) & 1) ? sm : ~sm;
  }
  return m;
}

template <bool MASK, typename A>
__device__ __forceinline__ void scale_regs(const f2::Factor& m, uint32_t mask) {
  unroll<kAmps>([&](auto q) {
    if (!MASK || ((mask >> q.value) & 1u)) A::template scale<q.value>(m);
  });
}

template <int S, typename A>
__device__ __forceinline__ void split_regs(const f2::Factor& m0, const f2::Factor& m1) {
  unroll<kAmps>([&](auto q) { A::template scale<q.value>(((q.value >> S) & 1) ? m1 : m0); });
}

// ------------------------------------------------------------------ forward
template <int S, bool REAL, bool MASK>
__device__ __forceinline__ void fwd_dense(int j, const Source& src) {
  f2::Factor m[4];
  src.matrix(j, m);
  each_pair<S, MASK, kAmps>(MASK ? src.p.ops[j].rmask : 0u, [&](auto q, auto u) {
    if constexpr (REAL) f2::Psi::real2<q.value, u.value>(m);
    else f2::Psi::dense2<q.value, u.value>(m);
  });
}

__device__ __forceinline__ void apply_fwd(int j, int go, const Source& src, uint32_t tl, uint64_t base) {
  const SOp& o = src.p.ops[j];
  switch (go) {
    case GO_DENSE: fwd_dense<0, false, false>(j, src); break;
    case GO_DENSE + 1: fwd_dense<1, false, false>(j, src); break;
    case GO_DENSE + 2: fwd_dense<2, false, false>(j, src); break;
    case GO_DENSE + 3: fwd_dense<3, false, false>(j, src); break;
    case GO_REAL: fwd_dense<0, true, false>(j, src); break;
    case GO_REAL + 1: fwd_dense<1, true, false>(j, src); break;
    case GO_REAL + 2: fwd_dense<2, true, false>(j, src); break;
    case GO_REAL + 3: fwd_dense<3, true, false>(j, src); break;
    case GO_MASK: fwd_dense<0, false, true>(j, src); break;
    case GO_MASK + 1: fwd_dense<1, false, true>(j, src); break;
    case GO_MASK + 2: fwd_dense<2, false, true>(j, src); break;
    case GO_MASK + 3: fwd_dense<3, false, true>(j, src); break;
    case GO_X: x_slot<0, false, f2::Psi>(0u); break;
    case GO_X + 1: x_slot<1, false, f2::Psi>(0u); break;
    case GO_X + 2: x_slot<2, false, f2::Psi>(0u); break;
    case GO_X + 3: x_slot<3, false, f2::Psi>(0u); break;
    case GO_XMASK: x_slot<0, true, f2::Psi>(o.rmask); break;
    case GO_XMASK + 1: x_slot<1, true, f2::Psi>(o.rmask); break;
    case GO_XMASK + 2: x_slot<2, true, f2::Psi>(o.rmask); break;
    case GO_XMASK + 3: x_slot<3, true, f2::Psi>(o.rmask); break;
    case GO_SPLIT: split_regs<0, f2::Psi>(src.get(j, 0), src.get(j, 1)); break;
    case GO_SPLIT + 1: split_regs<1, f2::Psi>(src.get(j, 0), src.get(j, 1)); break;
    case GO_SPLIT + 2: split_regs<2, f2::Psi>(src.get(j, 0), src.get(j, 1)); break;
    case GO_SPLIT + 3: split_regs<3, f2::Psi>(src.get(j, 0), src.get(j, 1)); break;
    case GO_SCALE: scale_regs<false, f2::Psi>(src.get(j, diag_const(o, tl, base)), 0u); break;
    case GO_SCALEMASK: scale_regs<true, f2::Psi>(src.get(j, 0), o.rmask); break;
    default: {
      const int dc = diag_const(o, tl, base), rb = diag_reg_bits(o);
      for (int e = rb;; e = (e - 1) & rb) {  // every value of the register-held bits
        scale_regs<true, f2::Psi>(src.get(j, dc | e), diag_patterns(o, e));
        if (e == 0) break;
      }
    }
  }
}

__global__ void __launch_bounds__(kMaxThreads, 3) k_tiled(const __grid_constant__ Params p) {
  TQK_AMPLITUDE_REGISTERS;
  extern __shared__ float4 sm4[];
  float2* tile = reinterpret_cast<float2*>(sm4);
  float4* fac = reinterpret_cast<float4*>(tile + (1u << p.m));
  Decoded* dec = reinterpret_cast<Decoded*>(fac + p.nops * 4);
  uint32_t* tab = reinterpret_cast<uint32_t*>(dec + p.nops);
  build_tables(p, tab);
  const Source src{p, fac};
  bool fresh = true;
  for (Items w = items_of(p); w.it < w.end; w.it += w.step) {
    const uint32_t row = w.it >> p.tiles_log;
    const uint64_t base = deposit(tile_of(p, w.it), p.outer);
    if (fresh) build_ops<false>(p, row, fac, dec);
    fresh = p.per_row && (w.it + w.step) >> p.tiles_log != row;
    load_tile(p, frame(p, row, base), p.psi_in, tile);
    wait_loads();  // also orders the tables
#pragma unroll 1
    for (int s = 0; s < p.nsweeps; ++s) {
      const Sweep& sw = p.sweeps[s];
      const uint32_t e = thread_offset(tab, s);
      const uint32_t tl = e & 0xffffu;
      load_regs<f2::Psi>(sw.rphys, tile, e >> 16);
#pragma unroll 1
      for (int j = sw.first; j < sw.first + sw.count; ++j) {
        const Decoded d = dec[j];
        if ((base & d.omask) != d.oval || (tl & d.tmask) != d.tval) continue;
        apply_fwd(j, d.go, src, tl, base);
      }
      store_regs<f2::Psi>(sw.rphys, tile, thread_offset(tab, s) >> 16);
      __syncthreads();
    }
    store_tile(p, frame(p, row, base), p.psi, tile);
    __syncthreads();
  }
}

// ------------------------------------------------------------------ reverse
// Reverse step of a dense 2x2 (the factors of U^H): psi, lam <- U^H, and the cotangent sums
// g[r][c] += lam_in_r conj(psi_out_c).
template <int S, bool GRAD, bool REAL, bool MASK>
__device__ __forceinline__ void adj_dense(int j, const Source& src) {
  f2::Factor m[4];
  src.matrix(j, m);
  each_pair<S, MASK, kAmps>(MASK ? src.p.ops[j].rmask : 0u, [&](auto q, auto u) {
    constexpr int Q = q.value, U = u.value;
    if constexpr (REAL) f2::Psi::real2<Q, U>(m);
    else f2::Psi::dense2<Q, U>(m);
    if constexpr (GRAD) {
      f2::sum_add<0, Q, Q>();
      f2::sum_add<1, Q, U>();
      f2::sum_add<2, U, Q>();
      f2::sum_add<3, U, U>();
    }
    if constexpr (REAL) f2::Lam::real2<Q, U>(m);
    else f2::Lam::dense2<Q, U>(m);
  });
}

// Entry f of a diagonal op on the patterns of mask.
template <bool GRAD, bool MASK>
__device__ __forceinline__ void adj_factor(int j, int f, uint32_t mask, const Source& src) {
  const f2::Factor m = src.get(j, f);
  if (GRAD) f2::side_zero();
  unroll<kAmps>([&](auto q) {
    if (!MASK || ((mask >> q.value) & 1u)) {
      f2::Psi::scale<q.value>(m);
      if constexpr (GRAD) f2::side_add<q.value>();
      f2::Lam::scale<q.value>(m);
    }
  });
  if (GRAD)
    unroll<4>([&](auto e) {
      if (f == e.value) f2::side_put<e.value>();
    });
}

template <int S, bool GRAD>
__device__ __forceinline__ void adj_split(int j, const Source& src) {
  const f2::Factor m0 = src.get(j, 0), m1 = src.get(j, 1);
  unroll<kAmps>([&](auto q) {
    constexpr int E = (q.value >> S) & 1;
    f2::Psi::scale<q.value>(E ? m1 : m0);
    if constexpr (GRAD) f2::sum_add<E, q.value, q.value>();
    f2::Lam::scale<q.value>(E ? m1 : m0);
  });
}

template <int S, bool MASK>
__device__ __forceinline__ void adj_x(uint32_t rmask) {
  x_slot<S, MASK, f2::Psi>(rmask);
  x_slot<S, MASK, f2::Lam>(rmask);
}

// One reverse step of op j; GRAD: adds the thread's cotangent to the sums.
template <bool GRAD>
__device__ __forceinline__ void apply_adj(int j, int go, const Source& src, uint32_t tl, uint64_t base) {
  const SOp& o = src.p.ops[j];
  switch (go) {
    case GO_DENSE: adj_dense<0, GRAD, false, false>(j, src); break;
    case GO_DENSE + 1: adj_dense<1, GRAD, false, false>(j, src); break;
    case GO_DENSE + 2: adj_dense<2, GRAD, false, false>(j, src); break;
    case GO_DENSE + 3: adj_dense<3, GRAD, false, false>(j, src); break;
    case GO_REAL: adj_dense<0, GRAD, true, false>(j, src); break;
    case GO_REAL + 1: adj_dense<1, GRAD, true, false>(j, src); break;
    case GO_REAL + 2: adj_dense<2, GRAD, true, false>(j, src); break;
    case GO_REAL + 3: adj_dense<3, GRAD, true, false>(j, src); break;
    case GO_MASK: adj_dense<0, GRAD, false, true>(j, src); break;
    case GO_MASK + 1: adj_dense<1, GRAD, false, true>(j, src); break;
    case GO_MASK + 2: adj_dense<2, GRAD, false, true>(j, src); break;
    case GO_MASK + 3: adj_dense<3, GRAD, false, true>(j, src); break;
    case GO_X: adj_x<0, false>(0u); break;
    case GO_X + 1: adj_x<1, false>(0u); break;
    case GO_X + 2: adj_x<2, false>(0u); break;
    case GO_X + 3: adj_x<3, false>(0u); break;
    case GO_XMASK: adj_x<0, true>(o.rmask); break;
    case GO_XMASK + 1: adj_x<1, true>(o.rmask); break;
    case GO_XMASK + 2: adj_x<2, true>(o.rmask); break;
    case GO_XMASK + 3: adj_x<3, true>(o.rmask); break;
    case GO_SPLIT: adj_split<0, GRAD>(j, src); break;
    case GO_SPLIT + 1: adj_split<1, GRAD>(j, src); break;
    case GO_SPLIT + 2: adj_split<2, GRAD>(j, src); break;
    case GO_SPLIT + 3: adj_split<3, GRAD>(j, src); break;
    case GO_SCALE: adj_factor<GRAD, false>(j, diag_const(o, tl, base), 0u, src); break;
    case GO_SCALEMASK: adj_factor<GRAD, true>(j, 0, o.rmask, src); break;
    default: {
      const int dc = diag_const(o, tl, base), rb = diag_reg_bits(o);
      for (int e = rb;; e = (e - 1) & rb) {
        adj_factor<GRAD, true>(j, dc | e, diag_patterns(o, e), src);
        if (e == 0) break;
      }
    }
  }
}

// Sum v[0..8) over the warp: afterwards lane L holds the sum of value (L >> 2) as a pair (sum, error):
// plain float32 over eight threads, exact beyond (16: a thread's part is of 16 terms, not 8: over four).
__device__ __forceinline__ float warp_sum8(float (&v)[8], bool of16, int lane, float& err) {
#pragma unroll
  for (int h = 4, o = 16; h >= 2; h >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const float send = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  const bool up = (lane & 4) != 0;
  float s = up ? v[1] : v[0], r = __shfl_xor_sync(0xffffffffu, up ? v[0] : v[1], 4), e;
  if (of16) {  // uniform
    s = two_sum(s, r, err);
    err += __shfl_xor_sync(0xffffffffu, err, 2);
    s = two_sum(s, __shfl_xor_sync(0xffffffffu, s, 2), e);
    err += e;
  } else {
    s += r;
    s = two_sum(s, __shfl_xor_sync(0xffffffffu, s, 2), err);
  }
  s = two_sum(s, __shfl_xor_sync(0xffffffffu, s, 1), e);
  err += __shfl_xor_sync(0xffffffffu, err, 1) + e;
  return s;
}

__global__ void __launch_bounds__(kMaxThreads, 2) k_tiled_adj(const __grid_constant__ Params p) {
  TQK_AMPLITUDE_REGISTERS;
  extern __shared__ float4 sm4[];
  float2* ps = reinterpret_cast<float2*>(sm4);
  float2* ls = ps + (1u << p.m);
  float4* fac = reinterpret_cast<float4*>(ls + (1u << p.m));
  // a tile's warp sums in gtile [ngrad][warps][8 sums, 8 errors], their sums over warps and tiles
  // in gacc [ngrad][8], pairs too
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int nacc = p.ngrad * 8;
  float2* gacc = reinterpret_cast<float2*>(fac + p.nops * 4);
  float* gtile = reinterpret_cast<float*>(gacc + nacc);
  Decoded* dec = reinterpret_cast<Decoded*>(gtile + 2 * nacc * warps);
  uint32_t* tab = reinterpret_cast<uint32_t*>(dec + p.nops);
  build_tables(p, tab);
  for (int i = threadIdx.x; i < nacc; i += blockDim.x) gacc[i] = make_float2(0.f, 0.f);
  const Source src{p, fac};
  bool fresh = true;
  for (Items w = items_of(p); w.it < w.end; w.it += w.step) {
    const uint32_t row = w.it >> p.tiles_log;
    const uint64_t base = deposit(tile_of(p, w.it), p.outer);
    if (fresh) build_ops<true>(p, row, fac, dec);
    fresh = p.per_row && (w.it + w.step) >> p.tiles_log != row;  // the next item is another row's
    {
      const Frame f = frame(p, row, base);
      load_tile(p, f, p.psi_in, ps);
      load_tile(p, f, p.lam_in, ls);
    }
    wait_loads();
#pragma unroll 1
    for (int s = p.nsweeps - 1; s >= 0; --s) {
      const Sweep& sw = p.sweeps[s];
      const uint32_t e = thread_offset(tab, s);
      const uint32_t tl = e & 0xffffu;
      load_regs<f2::Psi>(sw.rphys, ps, e >> 16);
      load_regs<f2::Lam>(sw.rphys, ls, e >> 16);
#pragma unroll 1
      for (int j = sw.first + sw.count - 1; j >= sw.first; --j) {
        const Decoded d = dec[j];
        float* gw = gtile + (d.gidx * warps + warp) * 16;
        if ((base & d.omask) != d.oval) {  // uniform for the tile
          if (d.gidx >= 0 && lane < 16) gw[lane] = 0.f;
          continue;
        }
        const bool on = (tl & d.tmask) == d.tval;
        if (d.gidx < 0) {  // uniform
          if (on) apply_adj<false>(j, d.go, src, tl, base);
          continue;
        }
        unroll<4>([&](auto k) { f2::sum_zero<k.value>(); });
        if (on) apply_adj<true>(j, d.go, src, tl, base);
        float v[8];
        unroll<4>([&](auto k) {
          const float2 g = f2::sum_get<k.value>();
          v[2 * k.value] = g.x;
          v[2 * k.value + 1] = g.y;
        });
        __syncwarp();
        float err;
        const float sum = warp_sum8(v, d.go >= GO_SCALE, lane, err);
        if ((lane & 3) == 0) {
          gw[lane >> 2] = sum;
          gw[8 + (lane >> 2)] = err;
        }
      }
      const uint32_t tp = thread_offset(tab, s) >> 16;
      store_regs<f2::Psi>(sw.rphys, ps, tp);
      store_regs<f2::Lam>(sw.rphys, ls, tp);
      __syncthreads();
    }
    {
      const Frame f = frame(p, row, base);
      store_tile(p, f, p.psi, ps);
      store_tile(p, f, p.lam, ls);
    }
    for (int i = threadIdx.x; i < nacc; i += blockDim.x) {
      float2 g = gacc[i];
      for (int w = 0; w < warps; ++w) {
        const float* gw = gtile + ((i >> 3) * warps + w) * 16 + (i & 7);
        float e;
        g.x = two_sum(g.x, gw[0], e);
        g.y += gw[8] + e;
      }
      if (fresh || w.it + w.step >= w.end) {  // the sums so far, one atomic per value
        const SOp& o = p.ops[p.grad_op[i >> 3]];
        if ((i & 7) < 2 * o.nent) atomicAdd(o.grad + row * o.grad_stride + (i & 7), pair_value(g.x, g.y));
        g = make_float2(0.f, 0.f);
      }
      gacc[i] = g;
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ host: plan and launch
// Cut the ops (in order) into sweeps of at most three targets besides bit 0: a sweep takes
// every op whose wires no earlier left-out op touches and whose target fits.  Fills the
// order of the ops, the sweeps' op ranges and their register bits; returns the sweeps.
struct HostOp {
  uint64_t wires;  // every index bit the op touches
  int target;      // tile-local bit of the target, or -1 (diagonal)
};

int plan_sweeps(const HostOp* ops, int nops, int m, int* order, Sweep* sweeps, int (*regs)[kAmpBits - 1]) {
  bool done[TQK_STAGED_MAX_OPS] = {false};
  int ns = 0, out = 0;
  while (out < nops) {
    uint64_t blocked = 0;
    uint32_t tgt = 0;
    int nt = 0;
    Sweep& s = sweeps[ns];
    s.first = static_cast<int16_t>(out);
    for (int j = 0; j < nops; ++j) {
      if (done[j]) continue;
      const int t = ops[j].target;
      const bool fits = t <= 0 || ((tgt >> t) & 1u) || nt < kAmpBits - 1;
      if ((ops[j].wires & blocked) || !fits) {
        blocked |= ops[j].wires;
        continue;
      }
      if (t > 0 && !((tgt >> t) & 1u)) {
        tgt |= 1u << t;
        ++nt;
      }
      done[j] = true;
      order[out++] = j;
    }
    s.count = static_cast<int16_t>(out - s.first);
    for (int b = m - 1; b > 0 && nt < kAmpBits - 1; --b)  // fill with the highest free bits
      if (!((tgt >> b) & 1u)) {
        tgt |= 1u << b;
        ++nt;
      }
    for (int b = 1, k = 0; b < m; ++b)
      if ((tgt >> b) & 1u) regs[ns][k++] = b;
    ++ns;
  }
  return ns;
}

}  // namespace tiled
}  // namespace tqk

using namespace tqk;

namespace {

int fill_tiled(tiled::Params& p, int64_t bsz, int n, const tqk_staged_op* ops, int nops, uint64_t tile_mask,
               bool adjoint, const char* what) {
  const int m = __builtin_popcountll(tile_mask);
  if (nops < 0 || nops > TQK_STAGED_MAX_OPS)
    return fail(TQK_BAD_SHAPE, "%s: %d ops (at most %d per pass)", what, nops, TQK_STAGED_MAX_OPS);
  if (nops > 0 && ops == nullptr) return fail(TQK_BAD_POINTER, "%s: null op list", what);
  p.n = n;
  p.m = m;
  p.nops = nops;
  p.tiles_log = n - m;
  p.items = static_cast<uint32_t>(bsz << (n - m));
  p.per_row = 0;
  p.outer = ((1ull << n) - 1ull) & ~tile_mask;
  int local[64];  // tile-local bit of an index bit, or -1
  for (int b = 0, j = 0; b < 64; ++b) {
    local[b] = -1;
    if (b < n && ((tile_mask >> b) & 1ull)) {
      p.tb[j] = static_cast<uint8_t>(b);
      local[b] = j++;
    }
  }
  tiled::HostOp h[TQK_STAGED_MAX_OPS];
  int hbits[TQK_STAGED_MAX_OPS][TQK_STAGED_MAX_WIRES];
  for (int j = 0; j < nops; ++j) {
    const tqk_staged_op& s = ops[j];
    if (s.nwires < 1 || s.nwires > TQK_STAGED_MAX_WIRES)
      return fail(TQK_BAD_WIRES, "%s: op %d has %d wires", what, j, s.nwires);
    uint64_t used = 0;
    for (int w = 0; w < s.nwires; ++w) {
      if (s.wires[w] < 0 || s.wires[w] >= n)
        return fail(TQK_BAD_WIRES, "%s: op %d wire %d out of range", what, j, s.wires[w]);
      hbits[j][w] = n - 1 - s.wires[w];
      if (used & (1ull << hbits[j][w])) return fail(TQK_BAD_WIRES, "%s: op %d repeats wire %d", what, j, s.wires[w]);
      used |= 1ull << hbits[j][w];
    }
    if (s.batch != 1 && s.batch != bsz && s.kind != TQK_S_X)
      return fail(TQK_BAD_SHAPE, "%s: op %d operand batch %lld (1 or bsz)", what, j, (long long)s.batch);
    if (s.kind != TQK_S_X && s.operand == nullptr) return fail(TQK_BAD_POINTER, "%s: op %d null operand", what, j);
    h[j].wires = used;
    h[j].target = -1;
    if (s.kind == TQK_S_DENSE1 || s.kind == TQK_S_X) {  // wires[0 .. nwires-1) controls, wires[nwires-1] target
      const int tb = hbits[j][s.nwires - 1];
      if (local[tb] < 0)
        return fail(TQK_BAD_WIRES, "%s: op %d target wire %d is outside the tile (bit %d)", what, j,
                    s.wires[s.nwires - 1], tb);
      h[j].target = local[tb];
    } else if (s.kind == TQK_S_DIAG) {
      if (s.nwires > 2) return fail(TQK_UNSUPPORTED, "%s: op %d diagonal on %d wires (1 or 2)", what, j, s.nwires);
    } else if (s.kind != TQK_S_PHASE) {
      return fail(TQK_BAD_SHAPE, "%s: op %d kind %d", what, j, s.kind);
    }
  }
  int order[TQK_STAGED_MAX_OPS], regs[TQK_STAGED_MAX_OPS][tiled::kAmpBits - 1];
  p.nsweeps = tiled::plan_sweeps(h, nops, m, order, p.sweeps, regs);
  p.ngrad = 0;
  for (int si = 0; si < p.nsweeps; ++si) {
    tiled::Sweep& s = p.sweeps[si];
    int slot_of[TQK_STAGED_MAX_TILE_BITS];  // register slot of a tile-local bit, or -1
    for (int b = 0; b < m; ++b) slot_of[b] = b == 0 ? 0 : -1;
    for (int k = 0; k < tiled::kAmpBits - 1; ++k) {
      slot_of[regs[si][k]] = k + 1;
      s.rphys[k] = static_cast<uint16_t>(tiled::swz(1u << regs[si][k]));
    }
    // thread bits: the three lowest lanes from different bank classes where possible, then
    // the other tile bits ascending
    int cnt = 0;
    uint32_t used = 0;
    for (int cls = 0; cls < 3; ++cls)
      for (int b = 1; b < m; ++b)
        if (slot_of[b] < 0 && (b - 1) % 3 == cls) {
          s.pos[cnt++] = static_cast<uint8_t>(b);
          used |= 1u << b;
          break;
        }
    for (int b = 1; b < m; ++b)
      if (slot_of[b] < 0 && !((used >> b) & 1u)) s.pos[cnt++] = static_cast<uint8_t>(b);
    for (; cnt < 8; ++cnt) s.pos[cnt] = 0;  // no such thread bit
    for (int i = s.first; i < s.first + s.count; ++i) {
      const int j = order[i];
      const tqk_staged_op& src = ops[j];
      tiled::SOp& o = p.ops[i];
      o = tiled::SOp{};
      o.operand = static_cast<const float2*>(src.operand);
      o.grad = adjoint && src.kind != TQK_S_X ? src.grad : nullptr;
      o.gidx = o.grad ? p.ngrad : -1;
      if (o.grad) p.grad_op[p.ngrad++] = static_cast<uint8_t>(i);
      const bool per_row = src.batch > 1 && src.kind != TQK_S_X;
      p.per_row |= per_row;
      const bool targeted = src.kind == TQK_S_DENSE1 || src.kind == TQK_S_X;
      for (int w = 0; w < 2; ++w) o.dslot[w] = o.dbit[w] = o.obit[w] = -1;
      if (src.kind == TQK_S_DIAG) {
        o.nd = src.nwires;
        o.nent = 1 << src.nwires;
        int held = 0;
        for (int w = 0; w < src.nwires; ++w) {
          const int lb = local[hbits[j][w]];
          if (lb < 0) o.obit[w] = hbits[j][w];
          else if (slot_of[lb] >= 0) o.dslot[w] = slot_of[lb], ++held;
          else o.dbit[w] = lb;
        }
        o.go = held == 0 ? tiled::GO_SCALE : (o.nd == 1 ? tiled::GO_SPLIT + o.dslot[0] : tiled::GO_DIAG);
      } else {
        const int nc = targeted ? src.nwires - 1 : src.nwires;
        const bool want = src.kind != TQK_S_X || src.ctrl_val;
        uint32_t rc = 0, rv = 0;  // condition on the register bits
        for (int w = 0; w < nc; ++w) {
          const int b = hbits[j][w], lb = local[b];
          if (lb < 0) {
            o.omask |= 1ull << b;
            if (want) o.oval |= 1ull << b;
          } else if (slot_of[lb] >= 0) {
            rc |= 1u << slot_of[lb];
            if (want) rv |= 1u << slot_of[lb];
          } else {
            o.tmask |= 1u << lb;
            if (want) o.tval |= 1u << lb;
          }
        }
        for (uint32_t q = 0; q < tiled::kAmps; ++q)
          if ((q & rc) == rv) o.rmask |= 1u << q;
        const int slot = targeted ? slot_of[h[j].target] : 0;
        if (src.kind == TQK_S_DENSE1) o.go = (rc ? tiled::GO_MASK : tiled::GO_DENSE) + slot;
        else if (src.kind == TQK_S_X) o.go = (rc ? tiled::GO_XMASK : tiled::GO_X) + slot;
        else o.go = rc ? tiled::GO_SCALEMASK : tiled::GO_SCALE;
        o.matrix = src.kind == TQK_S_DENSE1;
        o.nent = o.matrix ? 4 : (src.kind == TQK_S_PHASE ? 1 : 0);
      }
      o.op_stride = per_row ? o.nent : 0;
      o.grad_stride = per_row ? 2 * o.nent : 0;
    }
  }
  const int threads = 1 << (m - tiled::kAmpBits);
  for (int i = 0; i < tiled::kAmps / 2; ++i) {
    p.ioff[i] = 0;
    for (int b = 1; b < m; ++b)
      if (((i * 2 * threads) >> b) & 1) p.ioff[i] += 1ll << p.tb[b];
  }
  return TQK_OK;
}

int tiled_entry(const void* psi_in, const void* lam_in, void* psi, void* lam, int64_t bsz, int n, const tqk_staged_op* ops, int nops, uint64_t tile_mask,
                int* status, bool adjoint, void* stream, const char* what) {
  int rc = check_state(psi, bsz, n, what);
  if (rc) return rc;
  if (adjoint && (rc = check_state(lam, bsz, n, what))) return rc;
  if ((rc = check_state(psi_in, bsz, n, what))) return rc;
  if (adjoint && (rc = check_state(lam_in, bsz, n, what))) return rc;
  const int m = __builtin_popcountll(tile_mask);
  if (n < tiled::kMinBits || (tile_mask >> n) != 0 || m != (n < tiled::kMaxBits ? n : tiled::kMaxBits) ||
      (tile_mask & 1ull) == 0)
    return fail(TQK_BAD_SHAPE, "%s: a tile holds min(n, %d) of n = %d >= %d index bits, bit 0 among them (mask %llx)",
                what, tiled::kMaxBits, n, tiled::kMinBits, (unsigned long long)tile_mask);
  tiled::Params p;
  if ((rc = fill_tiled(p, bsz, n, ops, nops, tile_mask, adjoint, what))) return rc;
  if (nops == 0) return TQK_OK;
  if (status == nullptr) return fail(TQK_BAD_POINTER, "%s: null status word", what);
  p.psi = static_cast<float2*>(psi);
  p.lam = static_cast<float2*>(lam);
  p.psi_in = static_cast<const float2*>(psi_in);
  p.lam_in = static_cast<const float2*>(lam_in);
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int threads = 1 << (m - tiled::kAmpBits);
  const size_t tile = sizeof(float2) << m;
  const size_t tables = nops * (4 * sizeof(float4) + sizeof(tiled::Decoded)) +
                        static_cast<size_t>(p.nsweeps) * tiled::kTabEntries * sizeof(uint32_t);
  const size_t acc = static_cast<size_t>(p.ngrad) * 8 * (sizeof(float2) + threads / 32 * 2 * sizeof(float));
  const size_t smem = adjoint ? 2 * tile + acc + tables : tile + tables;
  auto kern = adjoint ? tiled::k_tiled_adj : tiled::k_tiled;
  static std::atomic<uint64_t> configured[2];  // devices whose attribute is set
  const uint64_t bit = 1ull << (dev & 63);
  if (!(configured[adjoint].load() & bit)) {
    constexpr size_t top = 2 * (sizeof(float2) << tiled::kMaxBits) +
                           TQK_STAGED_MAX_OPS * (8 * (sizeof(float2) + tiled::kMaxWarps * 2 * sizeof(float)) +
                                                 4 * sizeof(float4) + sizeof(tiled::Decoded) +
                                                 tiled::kTabEntries * sizeof(uint32_t));
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(top)) != cudaSuccess)
      return fail(TQK_CUDA_ERROR, "%s: cannot reserve %d bytes of shared memory", what, static_cast<int>(top));
    configured[adjoint].fetch_or(bit);
  }
  int fit = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kern, threads, smem) != cudaSuccess || fit < 1) fit = 1;
  const uint32_t slots = static_cast<uint32_t>(sms) * fit;  // CTAs that fill the GPU once
  uint32_t grid = slots < p.items ? slots : p.items;
  p.row_ctas = grid / static_cast<uint32_t>(bsz);
  if (grid - p.row_ctas * static_cast<uint32_t>(bsz) > grid / 16) p.row_ctas = 0;
  if (p.per_row && p.row_ctas > 0) grid = p.row_ctas * static_cast<uint32_t>(bsz);
  kern<<<grid, threads, smem, as_stream(stream)>>>(p);
  return launch_status(what);
}

}  // namespace

extern "C" int tqk_tiled_apply(void* state, int64_t bsz, int n, const tqk_staged_op* ops, int nops, uint64_t tile_mask,
                               int* status, void* stream) {
  return tiled_entry(state, nullptr, state, nullptr, bsz, n, ops, nops, tile_mask, status, false, stream, "tqk_tiled_apply");
}

extern "C" int tqk_tiled_adjoint(void* psi, void* lam, int64_t bsz, int n, const tqk_staged_op* ops, int nops,
                                 uint64_t tile_mask, int* status, void* stream) {
  return tiled_entry(psi, lam, psi, lam, bsz, n, ops, nops, tile_mask, status, true, stream, "tqk_tiled_adjoint");
}

extern "C" int tqk_tiled_adjoint_to(const void* psi_in, const void* lam_in, void* psi, void* lam, int64_t bsz, int n,
                                    const tqk_staged_op* ops, int nops, uint64_t tile_mask, int* status,
                                    void* stream) {
  const char* what = "tqk_tiled_adjoint_to";
  const char* a[2] = {static_cast<const char*>(psi_in), static_cast<const char*>(lam_in)};
  const char* o[2] = {static_cast<const char*>(psi), static_cast<const char*>(lam)};
  const int64_t bytes = n >= 0 && n < 48 && bsz > 0 ? bsz * (int64_t(8) << n) : 0;
  for (int i = 0; i < 2; ++i)
    for (int j = 0; j < 2; ++j)
      if ((i != j || a[i] != o[j]) && a[i] < o[j] + bytes && o[j] < a[i] + bytes)
        return fail(TQK_BAD_POINTER, "%s: an input overlaps an output other than its own buffer", what);
  if (o[0] < o[1] + bytes && o[1] < o[0] + bytes) return fail(TQK_BAD_POINTER, "%s: psi and lam overlap", what);
  return tiled_entry(psi_in, lam_in, psi, lam, bsz, n, ops, nops, tile_mask, status, true, stream, what);
}
