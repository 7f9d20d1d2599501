// sample.cu -- computational-basis sampling of a statevector on the GPU.
//
// Upstream's tq.measure copies |psi|^2 to the host and draws shots with
// random.choices (measurement/measurements.py:37-74).  Here each shot is an inverse-CDF
// draw on the device: given a uniform u in [0, 1), the outcome is the first index i
// whose running sum of |psi_j|^2 (j <= i) exceeds u * sum_j |psi_j|^2.  Kernels:
//   k_tile_sums  one warp per tile of 2^tb amplitudes: the tile's probability (float64);
//   k_tile_scan  one block per row: inclusive prefix sums of the tile probabilities;
//   k_draw       one warp per (row, shot): search over the tile prefixes, then the running
//                sum over the chosen tile's amplitudes (rows of less than a tile: k_draw_row);
//   k_parity     one block per (row, string): the share of even minus odd parities of the
//                outcomes on a string's sites.
// Uniforms come from the caller (a seeded torch generator), so draws are reproducible.
//
// What bounds them: float64 (one warp operation in 16 cycles) in the sums and the scan; reads
// of one tile per shot in the draw.
#include <stdint.h>

#include "common.cuh"

namespace tqk {
namespace sample {

constexpr int kTileBits = 8;
constexpr int kDrawWarps = 8;  // warps of a k_draw block
constexpr int kParityStrings = 32;  // strings a launch
struct ParityMasks {
  unsigned long long m[kParityStrings];
};

__device__ __forceinline__ double prob(float2 a) { return (double)a.x * a.x + (double)a.y * a.y; }

// grid (ceil(ntiles / 8), bsz), 256 threads: warp w of the block sums tile 8 * blockIdx.x + w
__global__ void __launch_bounds__(256) k_tile_sums(const float2* state, int n, int tb, int64_t ntiles,
                                                   double* tile_sum) {
  const int64_t b = blockIdx.y;
  const int64_t tile = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (tile >= ntiles) return;
  const float2* src = state + (b << n) + (tile << tb);
  double s = 0.0;
  for (int j = lane; j < (1 << tb); j += 32) {
    const double x = src[j].x, y = src[j].y;
    s = fma(x, x, fma(y, y, s));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) tile_sum[b * ntiles + tile] = s;
}

// One block (1024 threads) per row: in-place inclusive scan in chunks of 8192: a thread's 8
// values, the warp's threads, the block's warps.  (Ten additions a value and 80
// barriers took 21 us for 4 rows of 4096 tiles, this takes 9.)
constexpr int kScanPer = 8;
__global__ void __launch_bounds__(1024) k_tile_scan(double* tile_sum, int64_t ntiles) {
  __shared__ double warp_sum[32];
  double* row = tile_sum + (int64_t)blockIdx.x * ntiles;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double carry = 0.0;
  for (int64_t base = 0; base < ntiles; base += 1024 * kScanPer) {
    const int64_t i0 = base + (int64_t)threadIdx.x * kScanPer;
    double v[kScanPer];
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
      v[k] = i0 + k < ntiles ? row[i0 + k] : 0.0;
      if (k > 0) v[k] += v[k - 1];
    }
    double incl = v[kScanPer - 1];  // of the warp's threads up to this one
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      double w = warp_sum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += u;
      }
      warp_sum[lane] = w;
    }
    __syncthreads();
    const double up = __shfl_up_sync(0xffffffffu, incl, 1);
    const double before = carry + ((warp > 0 ? warp_sum[warp - 1] : 0.0) + (lane > 0 ? up : 0.0));
#pragma unroll
    for (int k = 0; k < kScanPer; ++k)
      if (i0 + k < ntiles) row[i0 + k] = before + v[k];
    carry += warp_sum[31];
    __syncthreads();
  }
}

// The draw within a tile of 2^kTileBits amplitudes, amplitude by amplitude in float64: each lane
// squares 8 of them, the additions go through all lanes in order.
__device__ __noinline__ int draw_in_tile(const float2* src, double before, double target) {
  const int lane = threadIdx.x & 31;
  double p[8];
  uint32_t some = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    p[k] = prob(src[8 * lane + k]);
    if (p[k] > 0.0) some = 8 * lane + k;
  }
  double acc = before;
  for (int l = 0; l < 32; ++l) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      acc += __shfl_sync(0xffffffffu, p[k], l);
      if (acc > target) return 8 * l + k;  // the same for every lane
    }
  }
  return __reduce_max_sync(0xffffffffu, some);  // rounding left target at the tile's end: the last one not zero
}

// The outcome from sums in R (a lane's 8 neighbouring amplitudes, then the warp's), or -1 where
// the target t (from the tile's start) is not farther than the margin from both of the
// outcome's ends.  float32: at most 16 roundings of sums up to the tile's and t's own; `walk`
// covers the float64 walk's 256 additions on sums up to the row's.
template <typename R>
__device__ __forceinline__ int sure_draw(const float4 (&v)[4], R t, R walk) {
  const int lane = threadIdx.x & 31;
  R c[8];  // running sums over the lane's amplitudes
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const R x0 = v[k].x, y0 = v[k].y, x1 = v[k].z, y1 = v[k].w;
    c[2 * k] = fma(x0, x0, y0 * y0) + (k > 0 ? c[2 * k - (k > 0)] : R(0));
    c[2 * k + 1] = fma(x1, x1, y1 * y1) + c[2 * k];
  }
  R incl = c[7];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const R u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  const R all = __shfl_sync(0xffffffffu, incl, 31), start = incl - c[7];
  const R margin = (sizeof(R) == 4 ? R(32 * 5.9604645e-8) * (all + fabs(t)) + R(1e-37) : R(0)) + walk;
  int j = 8;  // the lane's first amplitude whose sum exceeds t
#pragma unroll
  for (int k = 7; k >= 0; --k)
    if (start + c[k] > t) j = k;
  const uint32_t who = __ballot_sync(0xffffffffu, j < 8);
  if (who == 0) return -1;
  R below = start, above = start;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (k == j) above = start + c[k];
    if (k == j - 1) below = start + c[k];
  }
  const int mine = above - t > margin && t - below > margin ? 8 * lane + j : -1;
  return __shfl_sync(0xffffffffu, mine, __ffs(who) - 1);
}

// One warp per shot.  The tile: the first whose inclusive prefix exceeds the target, 32 places
// at a time.  Within it float32 sums settle all but about one shot in 500, float64 ones all but
// the odd one of the others, and those go through the tile in order: outcomes are the ordered
// walk's either way.  n = 20, 4 rows, 8192 shots: 118 -> 29 us (a thread per shot walked its tile
// alone).
__global__ void __launch_bounds__(256) k_draw(const float2* state, int n, int tb, int64_t ntiles,
                                              const double* prefix, const double* uniforms, int64_t shots,
                                              int64_t* out) {
  const int64_t b = blockIdx.y;
  const int lane = threadIdx.x & 31;
  const double* pre = prefix + b * ntiles;
  const double total = pre[ntiles - 1];
  for (int64_t s = (int64_t)blockIdx.x * kDrawWarps + (threadIdx.x >> 5); s < shots;
       s += (int64_t)gridDim.x * kDrawWarps) {
    const double target = uniforms[b * shots + s] * total;
    int64_t lo = 0, hi = ntiles - 1;  // the tile lies in [lo, hi]
    while (lo < hi) {
      const int64_t step = (hi - lo + 32) >> 5;  // pieces of `step` tiles, a lane each: their last tiles
      const int64_t at = min(lo + (lane + 1) * step - 1, hi);
      const uint32_t over = __ballot_sync(0xffffffffu, pre[at] > target);
      const int first = over ? __ffs(over) - 1 : 31;
      const int64_t l2 = lo + first * step;
      hi = min(l2 + step - 1, hi);
      lo = min(l2, hi);
    }
    const double before = lo > 0 ? pre[lo - 1] : 0.0;
    const float2* src = state + (b << n) + (lo << tb);
    float4 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = ld4(src + 8 * lane + 2 * k);
    const double t = target - before, walk = 1e-12 * total;
    int pick = sure_draw<float>(v, static_cast<float>(t), static_cast<float>(walk));
    if (pick < 0) pick = sure_draw<double>(v, t, walk);
    if (pick < 0) pick = draw_in_tile(src, before, target);
    if (lane == 0) out[b * shots + s] = (lo << tb) + pick;
  }
}

// Rows of less than a tile: a block walks its row once, amplitude by amplitude in float64, and its
// threads search the running sums, a shot each (the sums do not decrease, so the first that
// exceeds the target is the walk's stop; where they end in NaN the walk itself decides).
// What bounds it: the walk's chain of additions, paid once a block.  6 qubits, 32 rows, 65536
// shots: 1722 us with a walk a thread, 28212 with a warp per shot, which leaves 31 lanes without
// work, 66 here.
__global__ void __launch_bounds__(256) k_draw_row(const float2* state, int n, const double* total_of,
                                                  const double* uniforms, int64_t shots, int64_t* out) {
  __shared__ double p[1 << (kTileBits - 1)], sum[1 << (kTileBits - 1)];
  __shared__ int last_nonzero;
  const int64_t b = blockIdx.y;
  const int count = 1 << n, tid = threadIdx.x;
  if (tid < count) p[tid] = prob(state[(b << n) + tid]);
  __syncthreads();
  if (tid == 0) {
    double acc = 0.0;
    int last = 0;
    for (int j = 0; j < count; ++j) {
      if (p[j] > 0.0) last = j;
      acc += p[j];
      sum[j] = acc;
    }
    last_nonzero = last;
  }
  __syncthreads();
  const double total = total_of[b];
  const bool whole = sum[count - 1] == sum[count - 1];
  for (int64_t s = (int64_t)blockIdx.x * 256 + tid; s < shots; s += (int64_t)gridDim.x * 256) {
    const double target = uniforms[b * shots + s] * total;
    int lo = 0, hi = count;
    if (whole) {
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (sum[mid] > target) hi = mid;
        else lo = mid + 1;
      }
    } else {
      while (lo < count && !(sum[lo] > target)) ++lo;
    }
    out[b * shots + s] = lo < count ? lo : last_nonzero;  // rounding left target at the end: the last one not zero
  }
}

// out[string][row] = mean over the shots of (-1)^popcount(outcome & mask)
__global__ void __launch_bounds__(1024) k_parity(const int64_t* outcomes, int64_t shots, const ParityMasks masks,
                                                 int64_t bsz, float* out) {
  __shared__ unsigned long long odd;
  const int64_t b = blockIdx.x;
  const unsigned long long mask = masks.m[blockIdx.y];
  const int64_t* row = outcomes + b * shots;
  if (threadIdx.x == 0) odd = 0;
  __syncthreads();
  unsigned long long mine = 0;
#pragma unroll 4
  for (int64_t s = threadIdx.x; s < shots; s += 1024)
    mine += __popcll(static_cast<unsigned long long>(row[s]) & mask) & 1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(&odd, mine);
  __syncthreads();
  if (threadIdx.x == 0)
    out[blockIdx.y * bsz + b] = static_cast<float>(
        static_cast<double>(shots - 2 * static_cast<int64_t>(odd)) * (1.0 / static_cast<double>(shots)));
}

}  // namespace sample
}  // namespace tqk

using namespace tqk;

extern "C" int64_t tqk_sample_scratch_bytes(int64_t bsz, int n) {
  if (bsz < 1 || n < 1 || n > TQK_MAX_QUBITS) return 0;
  const int tb = n < sample::kTileBits ? n : sample::kTileBits;
  return bsz * (1ll << (n - tb)) * (int64_t)sizeof(double);
}

extern "C" int tqk_sample(const void* state, int64_t bsz, int n, const double* uniforms, int64_t shots,
                          int64_t* out, void* scratch, int64_t scratch_bytes, void* stream) {
  const char* what = "tqk_sample";
  int rc = check_state(state, bsz, n, what);
  if (rc) return rc;
  if (shots < 0) return fail(TQK_BAD_SHAPE, "%s: shots %lld", what, (long long)shots);
  if (shots == 0) return TQK_OK;
  if (!uniforms || !out || !scratch) return fail(TQK_BAD_POINTER, "%s: null pointer", what);
  if (bsz > 65535) return fail(TQK_BAD_SHAPE, "%s: bsz %lld > 65535", what, (long long)bsz);
  if (shots > (1ll << 31) * 256) return fail(TQK_BAD_SHAPE, "%s: too many shots", what);
  if (scratch_bytes < tqk_sample_scratch_bytes(bsz, n))
    return fail(TQK_SCRATCH_TOO_SMALL, "%s: scratch %lld < %lld bytes", what, (long long)scratch_bytes,
                (long long)tqk_sample_scratch_bytes(bsz, n));
  const int tb = n < sample::kTileBits ? n : sample::kTileBits;
  const int64_t ntiles = 1ll << (n - tb);
  auto* st = static_cast<const float2*>(state);
  auto* pre = static_cast<double*>(scratch);
  cudaStream_t s = as_stream(stream);
  sample::k_tile_sums<<<dim3((unsigned)((ntiles + 7) / 8), (unsigned)bsz), 256, 0, s>>>(st, n, tb, ntiles, pre);
  sample::k_tile_scan<<<(unsigned)bsz, 1024, 0, s>>>(pre, ntiles);
  if (tb < sample::kTileBits) {
    int64_t blocks = (shots + 255) / 256, most = 8 * 152 / bsz;  // several shots a thread once the GPU is full
    if (most < 1) most = 1;
    if (blocks > most) blocks = most;
    sample::k_draw_row<<<dim3((unsigned)blocks, (unsigned)bsz), 256, 0, s>>>(st, n, pre, uniforms, shots, out);
    return launch_status(what);
  }
  const int64_t blocks = (shots + sample::kDrawWarps - 1) / sample::kDrawWarps;
  sample::k_draw<<<dim3((unsigned)(blocks < (1 << 20) ? blocks : (1 << 20)), (unsigned)bsz),
                   32 * sample::kDrawWarps, 0, s>>>(st, n, tb, ntiles, pre,
                                                                                      uniforms, shots, out);
  return launch_status(what);
}

extern "C" int tqk_sample_parity(const int64_t* outcomes, int64_t bsz, int64_t shots, const uint64_t* masks, int m,
                                 float* out, void* stream) {
  const char* what = "tqk_sample_parity";
  if (bsz < 1 || bsz > 0x7fffffffll) return fail(TQK_BAD_SHAPE, "%s: bsz %lld", what, (long long)bsz);
  if (shots < 1) return fail(TQK_BAD_SHAPE, "%s: shots %lld", what, (long long)shots);
  if (m <= 0) return TQK_OK;
  if (!outcomes || !masks || !out) return fail(TQK_BAD_POINTER, "%s: null pointer", what);
  for (int j0 = 0; j0 < m; j0 += sample::kParityStrings) {
    const int cnt = m - j0 < sample::kParityStrings ? m - j0 : sample::kParityStrings;
    sample::ParityMasks pm;
    for (int j = 0; j < sample::kParityStrings; ++j) pm.m[j] = j < cnt ? masks[j0 + j] : 0ull;
    sample::k_parity<<<dim3((unsigned)bsz, (unsigned)cnt), 1024, 0, as_stream(stream)>>>(outcomes, shots, pm, bsz,
                                                                                       out + (int64_t)j0 * bsz);
    const int rc = launch_status(what);
    if (rc) return rc;
  }
  return TQK_OK;
}
