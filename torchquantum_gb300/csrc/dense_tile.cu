// dense_tile.cu -- dense gates on 3 to 6 wires, forward and reverse, on the CUDA cores.
//
// The gate is a small complex matrix product Y = U X: rows are the 2^k values of the target
// bits, columns the assignments of the other bits.  A CTA takes a tile of up to 2^12
// amplitudes (2^k rows by 2^(12-k) columns, the columns over the lowest other index bits),
// holds it and U in shared memory, and each of its 256 threads forms a 4 x 4 block of Y: per
// column index c two 16-byte loads of U and two of X feed 64 float32 multiply-adds, so the
// float32 pipe is the bound, and HBM where k is small.  With one output per thread and step
// (k_dense_k, k_dense_k_adj in apply.cu) every complex multiply-add takes two shared loads, in
// reverse one from global memory.  n = 22, bsz = 8 (S = 268 MB), k = 3 / 4 / 5 / 6, us: forward
// 707 / 677 / 783 / 1100 before, 146 / 178 / 251 / 397 here (float32 pipe alone 29 / 58 / 116 /
// 232, 2 S of HBM 79); reverse with cotangent 2091 / 2096 / 1525 / 2635 before, 589 / 773 / 902 /
// 1563 here.
// Each output's sum runs over c in ascending order with one fused multiply-add per product,
// so states are the same bit for bit as there.
//
// Tiles are copied in address order whatever the target bits are (coalesced), by maps from
// the tile's address bits to (row, column).  The reverse step holds the psi and lam tiles:
// psi <- U^H psi (or U^-1 psi, or the gate's kept input as it is), the cotangent
// sum lam_in psi_out^H, lam <- U^H lam.  A thread's part of the cotangent is 4 x 4 entries
// over a share of the columns: float32 sums of at most 32 columns, as in the kernels above, then
// pairs of float32 values (sum and error) over the warp's threads and the CTA's tiles, and a
// float64 atomic per entry at the end.  (Plain float32 over 256 columns and the warp took 614 / 735 /
// 964 / 1409 us, with the errors of that many additions.)
#include <stdint.h>

#include <atomic>

#include "dense_tile.cuh"

namespace tqk {
namespace dtile {

constexpr int kMaxThreads = 256;
constexpr int kTileBits = 12;
constexpr int kChunk = 32;   // columns a thread's cotangent sums take before they go to pairs of float32
constexpr int kCopies = 16;  // amplitudes a thread copies at most (a tile of 16 per thread)

struct Params {
  const float2* in;
  float2* state;
  const float2* lam_in;
  float2* lam;
  int n, m;                  // qubits; column bits of a tile
  int ld;                    // row stride of a tile in shared memory (even: 16-byte pairs)
  int tiles_log;             // tiles per row: 2^tiles_log
  int64_t items;             // tiles of all rows (below 2^31)
  uint64_t outer;            // index bits outside the tile
  int bits;                  // address bits of a tile: k + m
  uint8_t pos[kTileBits];    // index bit of the tile's address bit j (ascending)
  int32_t step[kTileBits];   // its step in shared memory: a column, or a row
  int64_t coff[kCopies];     // state offset and shared-memory offset of a thread's i-th copy,
  int32_t cstep[kCopies];    // relative to its first
  const float2* mat;
  const float2* uinv;
  int64_t mat_stride;
  double* grad;
  int64_t grad_stride;
};

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

// A thread's part of the tile copies: elements threadIdx.x + i * blockDim.x in address order.
struct Copy {
  uint64_t off;
  int at, count;
  __device__ __forceinline__ explicit Copy(const Params& p) : off(0), at(0) {
    for (int j = 0; j < p.bits; ++j)
      if ((threadIdx.x >> j) & 1u) {
        off |= 1ull << p.pos[j];
        at += p.step[j];
      }
    const int total = 1 << p.bits, tid = static_cast<int>(threadIdx.x), nt = static_cast<int>(blockDim.x);
    count = tid < total ? (total - tid + nt - 1) / nt : 0;
  }
  __device__ __forceinline__ void load(const Params& p, const float2* src, float2* tile) const {
#pragma unroll
    for (int i = 0; i < kCopies; ++i)
      if (i < count) tile[at + p.cstep[i]] = src[off + p.coff[i]];
  }
  __device__ __forceinline__ void store(const Params& p, float2* dst, const float2* tile) const {
#pragma unroll
    for (int i = 0; i < kCopies; ++i)
      if (i < count) dst[off + p.coff[i]] = tile[at + p.cstep[i]];
  }
};

// Work: the tiles of all rows.  With one matrix for all rows the CTAs take them in turn (neighbouring
// tiles at the same time), with a matrix a row an even share of neighbouring ones each.
// (CTAs of one row each, rounded down to whole rows, left up to half of the places for CTAs empty:
// n = 16, k = 5 reverse with cotangent, 153 / 305 rows 513 / 829 us, now 296 / 535.)
// I: 32 bits forward, 64 in reverse, as the registers come out (n = 22, bsz = 8: k = 6 forward 394
// us, 417 with 64; kept input, k = 3 reverse 299 us, 341 with 32).
template <typename I>
struct Items {
  I it, end;
  uint32_t step;
};
template <typename I>
__device__ __forceinline__ Items<I> items_of(const Params& p) {
  if (p.mat_stride == 0) return {static_cast<I>(blockIdx.x), static_cast<I>(p.items), gridDim.x};
  return {static_cast<I>(p.items * blockIdx.x / gridDim.x), static_cast<I>(p.items * (blockIdx.x + 1) / gridDim.x), 1u};
}
template <typename I>
__device__ __forceinline__ uint64_t item_base(const Params& p, I it) {
  return (static_cast<uint64_t>(it >> p.tiles_log) << p.n) + deposit(it & ((I(1) << p.tiles_log) - I(1)), p.outer);
}

// mt[c * D + r] = M[r][c]
template <int K>
__device__ __forceinline__ void load_transposed(const float2* src, float2* mt) {
  constexpr int D = 1 << K;
  for (int i = threadIdx.x; i < D * D; i += blockDim.x) mt[(i % D) * D + i / D] = src[i];
}
template <int K>
__device__ __forceinline__ void load_plain(const float2* src, float2* mt) {
  for (int i = threadIdx.x; i < (1 << (2 * K)); i += blockDim.x) mt[i] = src[i];
}

// The thread's 4 x 4 block: rows 4 tr .. + 3, columns 2 tc, 2 tc + 1 and the same in the
// tile's upper half (of at least four columns).
struct Block {
  int r0, c0, c1;
  bool active;
};
template <int K>
__device__ __forceinline__ Block block_of(const Params& p) {
  const int tcs = p.m < 2 ? 1 : 1 << (p.m - 2);
  const int tr = static_cast<int>(threadIdx.x) / tcs, tc = static_cast<int>(threadIdx.x) % tcs;
  return {4 * tr, 2 * tc, 2 * tc + 2 * tcs, tr < (1 << K) / 4};
}

// acc[i][j] = sum_c w(c, r0 + i) x(c, column j); CONJ: w conjugated.  w[c * D + r].
template <int K, bool CONJ>
__device__ __forceinline__ void product(int ld, const Block& b, const float2* w, const float2* x,
                                        float2 (&acc)[4][4]) {
  constexpr int D = 1 << K;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int c = 0; c < D; ++c) {
    const float4 w0 = ld4(w + c * D + b.r0), w1 = ld4(w + c * D + b.r0 + 2);
    const float4 x0 = ld4(x + c * ld + b.c0), x1 = ld4(x + c * ld + b.c1);
    const float2 wr[4] = {lo2(w0), hi2(w0), lo2(w1), hi2(w1)};
    const float2 xc[4] = {lo2(x0), hi2(x0), lo2(x1), hi2(x1)};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        acc[i][j] = CONJ ? cfma_conj(wr[i], xc[j], acc[i][j]) : cfma(wr[i], xc[j], acc[i][j]);
  }
}

__device__ __forceinline__ void put_block(int ld, const Block& b, const float2 (&acc)[4][4], float2* tile) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    st4(tile + (b.r0 + i) * ld + b.c0, pack4(acc[i][0], acc[i][1]));
    st4(tile + (b.r0 + i) * ld + b.c1, pack4(acc[i][2], acc[i][3]));
  }
}

// Shared memory (float2): the matrix, then the tile (even row strides: 16-byte aligned rows).
template <int K>
__global__ void __launch_bounds__(kMaxThreads, 3) k_fwd(const __grid_constant__ Params p) {
  extern __shared__ float4 sm4[];
  constexpr int D = 1 << K;
  float2* w = reinterpret_cast<float2*>(sm4);
  float2* x = w + D * D;
  const Copy cp(p);
  const Block b = block_of<K>(p);
  auto todo = items_of<uint32_t>(p);
  while (todo.it < todo.end) {
    // the items that share a matrix
    const uint32_t end = p.mat_stride == 0 ? todo.end : min(todo.end, ((todo.it >> p.tiles_log) + 1u) << p.tiles_log);
    load_transposed<K>(p.mat + (todo.it >> p.tiles_log) * p.mat_stride, w);
    for (; todo.it < end; todo.it += todo.step) {
      const uint64_t base = item_base(p, todo.it);
      cp.load(p, p.in + base, x);
      __syncthreads();
      float2 acc[4][4];
      if (b.active) product<K, false>(p.ld, b, w, x, acc);
      __syncthreads();
      if (b.active) put_block(p.ld, b, acc, x);
      __syncthreads();
      cp.store(p, p.state + base, x);
      __syncthreads();
    }
  }
}

// ------------------------------------------------------------------ cotangent sums
// Halving steps of a fold: 2^H threads of a warp share a block of entries.
template <int K>
constexpr int kHalvings = K == 3 ? 5 : (K == 4 ? 4 : (K == 5 ? 2 : 0));

// tot summed over the 2^H threads by halves (each step hands half of the values over) and added to
// the thread's 32 >> H pairs; tot becomes zero.
template <int H>
__device__ __forceinline__ void fold(float (&tot)[32], float (&hi)[32 >> H], float (&lo)[32 >> H], int gs) {
  float e[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) e[i] = 0.f;
#pragma unroll
  for (int h = 16, o = (1 << H) >> 1; o > 0; h >>= 1, o >>= 1) {
    const bool up = (gs & o) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const float send = up ? tot[i] : tot[i + h], keep = up ? tot[i + h] : tot[i];
      float err;
      tot[i] = two_sum(keep, __shfl_xor_sync(0xffffffffu, send, o), err);
      if (h < 16) {
        const float es = up ? e[i] : e[i + h], ek = up ? e[i + h] : e[i];
        err += ek + __shfl_xor_sync(0xffffffffu, es, o);
      }
      e[i] = err;
    }
  }
#pragma unroll
  for (int i = 0; i < (32 >> H); ++i) {
    float err;
    hi[i] = two_sum(hi[i], tot[i], err);
    lo[i] += err + e[i];
  }
#pragma unroll
  for (int i = 0; i < 32; ++i) tot[i] = 0.f;
}

enum { PSI_UH = 0, PSI_INV = 1, PSI_KEPT = 2 };

template <int K, int PSI, bool GRAD>
__global__ void __launch_bounds__(kMaxThreads, 2) k_adj(const __grid_constant__ Params p) {
  extern __shared__ float4 sm4[];
  constexpr int D = 1 << K;
  float2* w = reinterpret_cast<float2*>(sm4);
  float2* wi = w + D * D;                             // PSI_INV only
  float2* ps = wi + (PSI == PSI_INV ? D * D : 0);
  float2* ls = ps + D * p.ld;
  const Copy cp(p);
  const Block b = block_of<K>(p);
  // cotangent blocks of 4 x 4 entries, the columns shared out over `split` threads per block
  constexpr int kBlocks = D * D / 16, H = kHalvings<K>, NV = GRAD ? 32 >> H : 1;
  const int split = static_cast<int>(blockDim.x) / kBlocks;  // a power of two, 2^H at least with a cotangent
  const int gb = static_cast<int>(threadIdx.x) / split, gs = static_cast<int>(threadIdx.x) % split;
  float tot[GRAD ? 32 : 1], hi[NV], lo[NV];
#pragma unroll
  for (int e = 0; e < (GRAD ? 32 : 1); ++e) tot[e] = 0.f;
#pragma unroll
  for (int e = 0; e < NV; ++e) hi[e] = lo[e] = 0.f;
  int summed = 0;  // columns in tot
  // entries (gr + D/4 i, gc + D/4 j): neighbouring threads read neighbouring rows
  constexpr int Q = D / 4;
  const int gr = gb / Q, gc = gb % Q;
  auto todo = items_of<int64_t>(p);
  // one loop over items and matrices (a loop of its own for each matrix's items spills: kept input,
  // k = 3, n = 22, bsz = 8 373 us, this 299)
  int64_t row = -1;
  for (; todo.it < todo.end; todo.it += todo.step) {
    const int64_t was = row;
    row = todo.it >> p.tiles_log;
    if (was < 0 || (row != was && p.mat_stride != 0)) {
      load_plain<K>(p.mat + row * p.mat_stride, w);  // (U^H)[r][c] = conj U[c][r]
      if (PSI == PSI_INV) load_transposed<K>(p.uinv + row * p.mat_stride, wi);
    }
    // the last item of its matrix
    const bool last = todo.it + todo.step >= todo.end || (p.grad_stride != 0 && (todo.it + 1) >> p.tiles_log != row);
    const uint64_t base = item_base(p, todo.it);
    if (PSI != PSI_KEPT || GRAD) cp.load(p, (PSI == PSI_KEPT ? p.in : p.state) + base, ps);
    cp.load(p, p.lam_in + base, ls);
    __syncthreads();
    if (PSI != PSI_KEPT) {
      float2 acc[4][4];
      if (b.active) {
        if (PSI == PSI_INV) product<K, false>(p.ld, b, wi, ps, acc);
        else product<K, true>(p.ld, b, w, ps, acc);
      }
      __syncthreads();
      if (b.active) put_block(p.ld, b, acc, ps);
      __syncthreads();
      cp.store(p, p.state + base, ps);
    }
    if constexpr (GRAD) {  // += sum over the thread's columns (pairs 2 gs, 2 gs + 2 split, ...) of lam conj(psi)
      const int cols = 1 << p.m;
#pragma unroll 1
      for (int cb = 0; cb < cols; cb += kChunk * split) {
        const int ce = min(cols, cb + kChunk * split);
#pragma unroll 1
        for (int c = cb + 2 * gs; c < ce; c += 2 * split) {
          float4 l[4], y[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            l[i] = ld4(ls + (gr + Q * i) * p.ld + c);
            y[i] = ld4(ps + (gc + Q * i) * p.ld + c);
            if (cols == 1) l[i].z = l[i].w = y[i].z = y[i].w = 0.f;  // no second column
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float2 v = make_float2(tot[2 * (4 * i + j)], tot[2 * (4 * i + j) + 1]);
              v = cfma_bconj(hi2(l[i]), hi2(y[j]), cfma_bconj(lo2(l[i]), lo2(y[j]), v));
              tot[2 * (4 * i + j)] = v.x;
              tot[2 * (4 * i + j) + 1] = v.y;
            }
        }
        // the same for every thread: a thread's columns of a tile are 2^k or fewer
        summed += max(2, (ce - cb) / split);
        if (K >= 5 || summed >= kChunk || last) {
          fold<H>(tot, hi, lo, gs);
          summed = 0;
        }
      }
    }
    float2 acc[4][4];
    if (b.active) product<K, true>(p.ld, b, w, ls, acc);
    __syncthreads();
    if (b.active) put_block(p.ld, b, acc, ls);
    __syncthreads();
    cp.store(p, p.lam + base, ls);
    if constexpr (GRAD) {
      if (last) {  // one atomic per value of the thread's
        double* gd = p.grad + row * p.grad_stride + 2 * (gr * D + gc);
        int first = 0;
#pragma unroll
        for (int h = 16, o = (1 << H) >> 1; o > 0; h >>= 1, o >>= 1)
          if (gs & o) first += h;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          const int e = (first + i) >> 1;
          atomicAdd(gd + 2 * (Q * (e >> 2) * D + Q * (e & 3)) + ((first + i) & 1), pair_value(hi[i], lo[i]));
          hi[i] = lo[i] = 0.f;
        }
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ host
// Column bits of a tile: as many as its 2^12 amplitudes hold, fewer while the state has fewer
// tiles than twice the SMs; with a cotangent, whose atomics on one matrix meet, fewer than
// the SMs, and 32 columns at least (n = 13, bsz = 4, k = 3: 20 us with 8 columns, 512 CTAs).
int column_bits(const DenseTileArgs& a, bool grad) {
  int m = a.n - a.k < kTileBits - a.k ? a.n - a.k : kTileBits - a.k;
  while (m > (grad ? 5 : 3) && (a.bsz << (a.n - a.k - m)) < (grad ? 152 : 2 * 152)) --m;
  return m;
}

// Threads of a CTA: 16 amplitudes each, at least a warp; the cotangent needs 2^H per 4 x 4 block of
// its entries.
int threads_of(int k, int m, bool grad) {
  int t = 1 << (k + m < 9 ? 5 : k + m - 4);
  const int least = k == 3 ? 4 << kHalvings<3> : (k == 4 ? 16 << kHalvings<4> : kMaxThreads);
  return grad && t < least ? least : t;
}

// Row stride of a tile: padded so that the rows that neighbouring threads read start in
// different banks (five wires: four threads read 64 bytes of each row).
int row_stride(int k, int m) { return (m < 2 ? 4 : 1 << m) + (k == 5 ? 8 : 2); }

size_t tile_bytes(int k, int m) { return sizeof(float2) * (static_cast<size_t>(1) << k) * row_stride(k, m); }

void fill(Params& p, const DenseTileArgs& a, int m, int threads) {
  const int D = 1 << a.k;
  p.in = a.in;
  p.state = a.state;
  p.lam_in = a.lam_in;
  p.lam = a.lam;
  p.n = a.n;
  p.m = m;
  p.ld = row_stride(a.k, p.m);
  p.bits = a.k + p.m;
  p.tiles_log = a.n - p.bits;
  p.items = a.bsz << p.tiles_log;
  uint64_t tgt = 0, used = 0;
  for (int j = 0; j < a.k; ++j) tgt |= 1ull << a.tbits[j];
  int bit = 0, cols = 0;
  for (int q = 0; q < a.n; ++q) {
    const bool target = (tgt >> q) & 1ull;
    if (!target && cols == p.m) continue;
    int j = 0;
    while (target && a.tbits[j] != q) ++j;
    p.pos[bit] = static_cast<uint8_t>(q);
    p.step[bit++] = target ? p.ld << (a.k - 1 - j) : 1 << cols++;
    used |= 1ull << q;
  }
  p.outer = ((1ull << a.n) - 1ull) & ~used;
  for (int i = 0; i < kCopies; ++i) {
    p.coff[i] = 0;
    p.cstep[i] = 0;
    for (int j = 0; j < p.bits; ++j)
      if (((i * threads) >> j) & 1) {
        p.coff[i] += 1ll << p.pos[j];
        p.cstep[i] += p.step[j];
      }
  }
  p.mat = a.mat;
  p.uinv = a.uinv;
  p.mat_stride = a.mat_batch > 1 ? static_cast<int64_t>(D) * D : 0;
  p.grad = a.grad;
  p.grad_stride = a.mat_batch > 1 ? 2ll * D * D : 0;
}

// Largest dynamic request of a kernel, reserved once per device.
int reserve(const void* kern, std::atomic<uint64_t>& done, int dev, size_t bytes) {
  const uint64_t bit = 1ull << (dev & 63);
  if (done.load() & bit) return TQK_OK;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)) != cudaSuccess)
    return fail(TQK_CUDA_ERROR, "dense k-wire gate: cannot reserve %d bytes of shared memory", static_cast<int>(bytes));
  done.fetch_or(bit);
  return TQK_OK;
}

template <typename Kernel>
int launch(Kernel kern, std::atomic<uint64_t>& done, const Params& p, int threads, size_t smem, size_t top,
           const char* what, cudaStream_t st) {
  int dev = 0, sms = 0, fit = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int rc = reserve(reinterpret_cast<const void*>(kern), done, dev, top);
  if (rc) return rc;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kern, threads, smem) != cudaSuccess || fit < 1) fit = 1;
  // resident CTAs only: each loads its matrices (and flushes their cotangents) once
  const int64_t slots = static_cast<int64_t>(sms) * fit;
  kern<<<static_cast<unsigned>(slots < p.items ? slots : p.items), threads, smem, st>>>(p);
  return launch_status(what);
}

template <int K>
int launch_fwd(const DenseTileArgs& a, cudaStream_t st) {
  static std::atomic<uint64_t> done{0};
  const int m = column_bits(a, false), threads = threads_of(K, m, false);
  Params p;
  fill(p, a, m, threads);
  constexpr size_t mat = sizeof(float2) << (2 * K);
  return launch(k_fwd<K>, done, p, threads, mat + tile_bytes(K, p.m), mat + tile_bytes(K, kTileBits - K),
                "dense k-wire gate", st);
}

template <int K, int PSI, bool GRAD>
int launch_adj(const DenseTileArgs& a, cudaStream_t st) {
  static std::atomic<uint64_t> done{0};
  const int m = column_bits(a, GRAD), threads = threads_of(K, m, GRAD);
  Params p;
  fill(p, a, m, threads);
  constexpr size_t mat = (PSI == PSI_INV ? 2 : 1) * (sizeof(float2) << (2 * K));
  return launch(k_adj<K, PSI, GRAD>, done, p, threads, mat + 2 * tile_bytes(K, p.m),
                mat + 2 * tile_bytes(K, kTileBits - K), "adjoint dense k-wire gate", st);
}

template <int K>
int launch_adj_k(const DenseTileArgs& a, cudaStream_t st) {
  if (a.stored) return a.grad ? launch_adj<K, PSI_KEPT, true>(a, st) : launch_adj<K, PSI_KEPT, false>(a, st);
  if (a.uinv) return a.grad ? launch_adj<K, PSI_INV, true>(a, st) : launch_adj<K, PSI_INV, false>(a, st);
  return a.grad ? launch_adj<K, PSI_UH, true>(a, st) : launch_adj<K, PSI_UH, false>(a, st);
}

}  // namespace dtile

int launch_dense_tile(const DenseTileArgs& a, cudaStream_t st) {
  switch (a.k) {
    case 3: return dtile::launch_fwd<3>(a, st);
    case 4: return dtile::launch_fwd<4>(a, st);
    case 5: return dtile::launch_fwd<5>(a, st);
    case 6: return dtile::launch_fwd<6>(a, st);
    default: return fail(TQK_TOO_MANY_QUBITS, "dense k-wire gate: k=%d", a.k);
  }
}

int launch_dense_tile_adj(const DenseTileArgs& a, cudaStream_t st) {
  switch (a.k) {
    case 3: return dtile::launch_adj_k<3>(a, st);
    case 4: return dtile::launch_adj_k<4>(a, st);
    case 5: return dtile::launch_adj_k<5>(a, st);
    case 6: return dtile::launch_adj_k<6>(a, st);
    default: return fail(TQK_TOO_MANY_QUBITS, "adjoint dense k-wire gate: k=%d", a.k);
  }
}

}  // namespace tqk
