// program.cu -- gate operands from parameters, fused-block unitaries, and their
// backward, all on the GPU in float64.
//
// A recorded circuit is described by plain arrays (include/tqk.h):
//   tqk_gate_desc  one parameterised gate: its type, where its parameters live (any
//                  strided float32/float64 tensor, read in place), where its operand goes;
//   tqk_block_op   one op inside a fused block (kind, bit positions in the block);
//   tqk_block_desc one fused block (its ops, width, batch, where U goes).
// Kernels:
//   k_gate_operands  params -> operands (complex128 and complex64), one gate per block;
//   k_param_grads    operand cotangents -> d loss / d params (analytic derivatives,
//                    atomically added into a float64 buffer laid out like the params);
//   k_block_build    U = G_m ... G_1 for every (block, batch row), 2^k x 2^k in shared memory;
//   k_block_unbuild  the reverse: from dL/dU, every op's operand cotangent
//                    (W <- G_j^H W, X <- G_j^H X, grad_j = sum over the other bits of X W^H).
#include <math.h>
#include <type_traits>

#include "common.cuh"

namespace tqk {
namespace prog {

// Complex scalars: float64 (C2) for operands and block unitaries; float32 (F2) for the
// block unbuild sweeps, whose input cotangent carries complex64 accuracy (partial sums
// go to float64 before any atomic).
template <typename R>
struct CT {
  R x, y;
  using real = R;
};
using C2 = CT<double>;
using F2 = CT<float>;
__device__ __forceinline__ C2 mk(double a, double b) { return C2{a, b}; }
template <typename C>
__device__ __forceinline__ C mkc(double a, double b) {
  return C{static_cast<typename C::real>(a), static_cast<typename C::real>(b)};
}
template <typename C>
__device__ __forceinline__ C cmul2(C a, C b) {
  return C{a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
template <typename C>
__device__ __forceinline__ C conj2(C a) {
  return C{a.x, -a.y};
}
template <typename C>
__device__ __forceinline__ C cadd2(C a, C b) {
  return C{a.x + b.x, a.y + b.y};
}
__device__ __forceinline__ C2 expi(double t) {
  double s, c;
  sincos(t, &s, &c);
  return C2{c, s};
}
__device__ __forceinline__ C2 scale(C2 a, double s) { return C2{a.x * s, a.y * s}; }
__device__ __forceinline__ C2 mul_i(C2 a) { return C2{-a.y, a.x}; }  // i * a

// Operand size (complex entries) per operand shape.
__host__ __device__ inline int operand_size(int type) {
  switch (type) {
    case TQK_G_RZ: return 2;
    case TQK_G_PHASE: case TQK_G_CU1: return 1;
    case TQK_G_CRZ: case TQK_G_RZZ: return 4;
    case TQK_G_RXX: case TQK_G_RYY: case TQK_G_RZX: case TQK_G_SINGLEEXC: return 16;
    default: return 4;  // 2x2 dense / controlled block
  }
}

__host__ __device__ inline int operand_is_diag(int type) {
  return type == TQK_G_RZ || type == TQK_G_PHASE || type == TQK_G_CU1 || type == TQK_G_CRZ || type == TQK_G_RZZ;
}

// Operand of gate `type` (or its derivative w.r.t. parameter `dk`, dk >= 0) at params p.
__device__ void operand(int type, const double* p, int dk, C2* m) {
  const bool d = dk >= 0;
  switch (type) {
    case TQK_G_U3:
    case TQK_G_CU3:
    case TQK_G_CU: {  // [[c, -e^{il} s], [e^{if} s, e^{i(f+l)} c]] (x e^{ig} for cu)
      const double th = p[0], ph = p[1], la = p[2];
      double s, c;
      sincos(th / 2, &s, &c);
      double a00 = c, a01 = s, a10 = s, a11 = c;  // magnitudes before phases
      if (d && dk == 0) { a00 = -s / 2; a01 = c / 2; a10 = c / 2; a11 = -s / 2; }
      m[0] = mk(a00, 0);
      m[1] = scale(expi(la), -a01);
      m[2] = scale(expi(ph), a10);
      m[3] = scale(expi(ph + la), a11);
      if (d && dk == 1) { m[0] = mk(0, 0); m[1] = mk(0, 0); m[2] = mul_i(m[2]); m[3] = mul_i(m[3]); }
      if (d && dk == 2) { m[0] = mk(0, 0); m[2] = mk(0, 0); m[1] = mul_i(m[1]); m[3] = mul_i(m[3]); }
      if (type == TQK_G_CU) {
        const C2 g = expi(p[3]);
        if (d && dk == 3) {  // d/dgamma of e^{ig} U3 = i e^{ig} U3
          double s2, c2;
          sincos(th / 2, &s2, &c2);
          m[0] = mk(c2, 0);
          m[1] = scale(expi(la), -s2);
          m[2] = scale(expi(ph), s2);
          m[3] = scale(expi(ph + la), c2);
          for (int e = 0; e < 4; ++e) m[e] = mul_i(m[e]);
        }
        for (int e = 0; e < 4; ++e) m[e] = cmul2(m[e], g);
      }
      return;
    }
    case TQK_G_RX:
    case TQK_G_CRX: {
      double s, c;
      sincos(p[0] / 2, &s, &c);
      if (d) { const double t = c; c = -s / 2; s = t / 2; }
      m[0] = mk(c, 0); m[1] = mk(0, -s); m[2] = mk(0, -s); m[3] = mk(c, 0);
      return;
    }
    case TQK_G_RY:
    case TQK_G_CRY: {
      double s, c;
      sincos(p[0] / 2, &s, &c);
      if (d) { const double t = c; c = -s / 2; s = t / 2; }
      m[0] = mk(c, 0); m[1] = mk(-s, 0); m[2] = mk(s, 0); m[3] = mk(c, 0);
      return;
    }
    case TQK_G_RZ: {  // diag(e^{-it/2}, e^{it/2})
      m[0] = expi(-p[0] / 2);
      m[1] = expi(p[0] / 2);
      if (d) { m[0] = scale(mul_i(m[0]), -0.5); m[1] = scale(mul_i(m[1]), 0.5); }
      return;
    }
    case TQK_G_CRZ: {  // diag(1, 1, e^{-it/2}, e^{it/2})
      m[0] = mk(d ? 0 : 1, 0);
      m[1] = mk(d ? 0 : 1, 0);
      m[2] = expi(-p[0] / 2);
      m[3] = expi(p[0] / 2);
      if (d) { m[2] = scale(mul_i(m[2]), -0.5); m[3] = scale(mul_i(m[3]), 0.5); }
      return;
    }
    case TQK_G_RZZ: {  // diag(e^{-it/2}, e^{it/2}, e^{it/2}, e^{-it/2})
      const C2 a = expi(-p[0] / 2), b = expi(p[0] / 2);
      m[0] = a; m[1] = b; m[2] = b; m[3] = a;
      if (d) {
        m[0] = scale(mul_i(a), -0.5); m[3] = m[0];
        m[1] = scale(mul_i(b), 0.5); m[2] = m[1];
      }
      return;
    }
    case TQK_G_PHASE:
    case TQK_G_CU1: {
      m[0] = expi(p[0]);
      if (d) m[0] = mul_i(m[0]);
      return;
    }
    case TQK_G_ROT:
    case TQK_G_CROT: {  // RZ(om) RY(th) RZ(ph): a = (ph+om)/2, dd = (ph-om)/2
      const double ph = p[0], th = p[1], om = p[2];
      double s, c;
      sincos(th / 2, &s, &c);
      const double a = (ph + om) / 2, dd = (ph - om) / 2;
      double c0 = c, s0 = s;
      if (d && dk == 1) { c0 = -s / 2; s0 = c / 2; }
      m[0] = scale(expi(-a), c0);
      m[1] = scale(expi(dd), -s0);
      m[2] = scale(expi(-dd), s0);
      m[3] = scale(expi(a), c0);
      if (d && dk == 0) {
        m[0] = scale(mul_i(m[0]), -0.5); m[1] = scale(mul_i(m[1]), 0.5);
        m[2] = scale(mul_i(m[2]), -0.5); m[3] = scale(mul_i(m[3]), 0.5);
      }
      if (d && dk == 2) {
        m[0] = scale(mul_i(m[0]), -0.5); m[1] = scale(mul_i(m[1]), -0.5);
        m[2] = scale(mul_i(m[2]), 0.5); m[3] = scale(mul_i(m[3]), 0.5);
      }
      return;
    }
    case TQK_G_U2: {  // (1/sqrt2)[[1, -e^{il}], [e^{if}, e^{i(f+l)}]]
      const double r = 0.70710678118654752440;
      m[0] = mk(r, 0);
      m[1] = scale(expi(p[1]), -r);
      m[2] = scale(expi(p[0]), r);
      m[3] = scale(expi(p[0] + p[1]), r);
      if (d && dk == 0) { m[0] = mk(0, 0); m[1] = mk(0, 0); m[2] = mul_i(m[2]); m[3] = mul_i(m[3]); }
      if (d && dk == 1) { m[0] = mk(0, 0); m[2] = mk(0, 0); m[1] = mul_i(m[1]); m[3] = mul_i(m[3]); }
      return;
    }
    case TQK_G_R: {  // [[c, -i e^{-if} s], [-i e^{if} s, c]]
      double s, c;
      sincos(p[0] / 2, &s, &c);
      const C2 em = expi(-p[1]), ep = expi(p[1]);
      if (d && dk == 1) {
        m[0] = mk(0, 0); m[3] = mk(0, 0);
        m[1] = scale(em, -s);
        m[2] = scale(ep, s);
        return;
      }
      if (d) { const double t = c; c = -s / 2; s = t / 2; }
      m[0] = mk(c, 0); m[3] = mk(c, 0);
      m[1] = cmul2(mk(0, -s), em);
      m[2] = cmul2(mk(0, -s), ep);
      return;
    }
    case TQK_G_RXX:
    case TQK_G_RYY:
    case TQK_G_RZX:
    case TQK_G_SINGLEEXC: {
      double s, c;
      sincos(p[0] / 2, &s, &c);
      if (d) { const double t = c; c = -s / 2; s = t / 2; }
      for (int e = 0; e < 16; ++e) m[e] = mk(0, 0);
      const double one = d ? 0.0 : 1.0;
      if (type == TQK_G_RXX) {
        m[0] = m[5] = m[10] = m[15] = mk(c, 0);
        m[3] = m[6] = m[9] = m[12] = mk(0, -s);
      } else if (type == TQK_G_RYY) {
        m[0] = m[5] = m[10] = m[15] = mk(c, 0);
        m[3] = m[12] = mk(0, s);
        m[6] = m[9] = mk(0, -s);
      } else if (type == TQK_G_RZX) {
        m[0] = m[5] = m[10] = m[15] = mk(c, 0);
        m[1] = m[4] = mk(0, -s);
        m[11] = m[14] = mk(0, s);
      } else {
        m[0] = m[15] = mk(one, 0);
        m[5] = m[10] = mk(c, 0);
        m[6] = mk(-s, 0);
        m[9] = mk(s, 0);
      }
      return;
    }
    default:
      return;
  }
}

__device__ __forceinline__ void operand_inverse(int type, C2* m) {
  const int sz = operand_size(type);
  if (operand_is_diag(type)) {
    for (int e = 0; e < sz; ++e) m[e] = conj2(m[e]);
    return;
  }
  const int dim = sz == 16 ? 4 : 2;
  C2 t[16];
  for (int r = 0; r < dim; ++r)
    for (int c = 0; c < dim; ++c) t[r * dim + c] = conj2(m[c * dim + r]);
  for (int e = 0; e < sz; ++e) m[e] = t[e];
}

__device__ __forceinline__ double load_param(const tqk_gate_desc& g, int64_t b, int k) {
  const int64_t idx = b * g.p_row_stride + k * g.p_col_stride;
  return g.p_is_double ? static_cast<const double*>(g.p)[idx] : static_cast<double>(static_cast<const float*>(g.p)[idx]);
}

__global__ void k_gate_operands(const tqk_gate_desc* gates, int ngates) {
  const int gi = blockIdx.x;
  if (gi >= ngates) return;
  const tqk_gate_desc g = gates[gi];
  const int sz = operand_size(g.type);
  for (int64_t b = threadIdx.x; b < g.batch; b += blockDim.x) {
    double p[4];
    for (int k = 0; k < g.nparam && k < 4; ++k) p[k] = load_param(g, b, k);
    C2 m[16];
    operand(g.type, p, -1, m);
    if (g.inverse) operand_inverse(g.type, m);
    double2* o128 = static_cast<double2*>(g.op128) + b * sz;
    float2* o64 = static_cast<float2*>(g.op64) + b * sz;
    for (int e = 0; e < sz; ++e) {
      if (g.op128) o128[e] = make_double2(m[e].x, m[e].y);
      if (g.op64) o64[e] = make_float2(static_cast<float>(m[e].x), static_cast<float>(m[e].y));
    }
  }
}

// dL/dp_k = Re sum_e conj(G_e) dOp_e / dp_k, accumulated into grad buffers shaped like params.
__global__ void k_param_grads(const tqk_gate_desc* gates, int ngates) {
  const int gi = blockIdx.x;
  if (gi >= ngates) return;
  const tqk_gate_desc g = gates[gi];
  if (g.grad == nullptr || g.op_grad == nullptr) return;
  const double2* op_grad = static_cast<const double2*>(g.op_grad);
  const int sz = operand_size(g.type);
  for (int64_t b = threadIdx.x; b < g.batch; b += blockDim.x) {
    double p[4];
    for (int k = 0; k < g.nparam && k < 4; ++k) p[k] = load_param(g, b, k);
    const int64_t o = b * sz;
    for (int k = 0; k < g.nparam; ++k) {
      C2 dm[16];
      operand(g.type, p, k, dm);
      if (g.inverse) operand_inverse(g.type, dm);
      double acc = 0.0;
      for (int e = 0; e < sz; ++e) {
        const double2 G = op_grad[o + e];
        acc += G.x * dm[e].x + G.y * dm[e].y;  // Re(conj(G) dm)
      }
      atomicAdd(g.grad + b * g.p_row_stride + k * g.p_col_stride, acc);
    }
  }
}

// ------------------------------------------------------------------ block build / unbuild
// A 2^k x 2^k product in shared memory.  Float64 products of a few blocks bound the build
// (the pipe does 2 FMAs a clock per SM) and chains of small sweeps the reverse, so the work
// per op is cut and spread:
//  * Columns are independent (each op multiplies from the left): 2^split CTAs share a block,
//    each with the columns whose last `split` bits have its value.
//  * Bits count in the order the ops reach them.  Before an op reaches bit t the product is
//    the identity on it, so ops work on the 2^t x 2^t entries of the bits reached so far
//    (join); in reverse the cotangent's partial trace over a bit is all that the ops before
//    it see (drop).
//  * Ops and operands are read 32 at a time, one op per lane, ahead of the sweeps; a sweep of
//    the reverse updates W and X and takes the operand's cotangent together: one barrier an op.
// Measured (20 wires, 320 gates in 20 blocks, one of 61 ops; 24 wires, 400 gates in 34 blocks for
// each of 16 rows): build 915 -> 154 us and 937 -> 259 us (of which half is the pipe), reverse
// 793 -> 147 us and 648 -> 156 us.

// Descriptor limits the block kernels rely on (shared memory holds a 64 x 64 block; an op
// touches at most 6 wires, a dense part at most 2 targets): a block or op outside them is
// skipped, never indexed (the host checks them before upload).
__device__ __forceinline__ bool block_ok(const tqk_block_desc& bl) { return bl.k >= 1 && bl.k <= 6 && bl.num_ops >= 0; }

__device__ __forceinline__ bool op_ok(const tqk_block_op& op, int k) {
  if (op.nw < 1 || op.nw > 6 || op.nctrl < 0 || op.nctrl > op.nw) return false;
  for (int j = 0; j < op.nw; ++j)
    if (op.pos[j] < 0 || op.pos[j] >= k) return false;
  const int kt = op.nw - op.nctrl;
  switch (op.kind) {
    case TQK_K_DENSE:
    case TQK_K_CTRL: return kt >= 1 && kt <= 2 && op.op_size >= (1 << kt) * (1 << kt);
    case TQK_K_X: return kt == 1;
    case TQK_K_SWAP: return kt == 2;
    case TQK_K_PHASE: return op.op_size >= 1;
    case TQK_K_DIAG: return op.op_size >= (1 << op.nw);
    default: return false;
  }
}

constexpr int kChunk = 32;  // ops read at a time
constexpr int kBuildPlaces = 152;
constexpr int kBuildEntryBits = 9;  // entries of a block that a CTA of the build holds

struct ShOp {
  const double2* opnd;
  double* grad;
  int16_t kind, nw, nctrl, reach;  // reach: bits reached with this op; kind -1: skipped
  uint16_t fixed;                  // rows' control bits (PHASE: all bits)
  uint8_t pos[6], asc[6];          // the op's bits in its own and in ascending order
};

template <typename C>
struct Stage {
  ShOp op[kChunk];
  C m[kChunk][16];
  int first[6];     // op that first touches a bit (num_ops: none)
  uint8_t rank[6];  // bit -> its place in that order
  uint8_t at[64];   // row in that order -> row of the block
};

// Order of the bits and the row table; ends with the block synchronised.
template <typename C>
__device__ void order_bits(Stage<C>& sh, const tqk_block_desc& bl, const tqk_block_op* ops) {
  const int tid = threadIdx.x;
  if (tid < 32) {
    int first[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) first[q] = bl.num_ops;
    for (int i0 = 0; i0 < bl.num_ops; i0 += 32) {
      uint32_t mask = 0;
      if (i0 + tid < bl.num_ops) {
        const tqk_block_op& op = ops[bl.first_op + i0 + tid];
        if (op_ok(op, bl.k))
          for (int j = 0; j < op.nw; ++j) mask |= 1u << op.pos[j];
      }
      bool open = false;
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        const uint32_t who = __ballot_sync(0xffffffffu, (mask >> q) & 1u);
        if (first[q] == bl.num_ops && who != 0) first[q] = i0 + __ffs(who) - 1;
        open |= q < bl.k && first[q] == bl.num_ops;
      }
      if (!open) break;
    }
    int rank[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      rank[q] = 0;
#pragma unroll
      for (int p = 0; p < 6; ++p)
        if (p < bl.k && (first[p] < first[q] || (first[p] == first[q] && p < q))) ++rank[q];
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t r = 0;
#pragma unroll
      for (int q = 0; q < 6; ++q)
        if (q < bl.k) r |= (((tid + 32 * h) >> rank[q]) & 1u) << q;
      sh.at[tid + 32 * h] = static_cast<uint8_t>(r);
    }
#pragma unroll
    for (int q = 0; q < 6; ++q)
      if (tid == q) {
        sh.first[q] = first[q];
        sh.rank[q] = static_cast<uint8_t>(rank[q]);
      }
  }
  __syncthreads();
}

template <typename C>
__device__ __forceinline__ C from_d2(const double2& v) {
  return mkc<C>(v.x, v.y);
}

// Ops i0 .. i0 + 31 of the block into shared memory; ends with the block synchronised.
template <typename C>
__device__ void stage_ops(Stage<C>& sh, const tqk_block_desc& bl, const tqk_block_op* ops, int i0, int64_t b) {
  const int tid = threadIdx.x;
  if (tid < kChunk && i0 + tid < bl.num_ops) {
    const tqk_block_op& op = ops[bl.first_op + i0 + tid];
    ShOp o;
    o.kind = -1;
    uint32_t bits = 0;
    for (int j = 0; j < 6; ++j) bits |= j < op.nw && op.pos[j] >= 0 ? 1u << (op.pos[j] & 31) : 0u;
    if (op_ok(op, bl.k) && __popc(bits) == op.nw) {  // (a bit named twice: no row has it clear once)
      const int64_t row = (op.batch > 1 ? b : 0) * op.op_size;
      o.kind = static_cast<int16_t>(op.kind);
      o.nw = static_cast<int16_t>(op.nw);
      o.nctrl = static_cast<int16_t>(op.nctrl);
      o.opnd = static_cast<const double2*>(op.operand) + row;
      o.grad = op.grad == nullptr ? nullptr : static_cast<double*>(op.grad) + 2 * row;
      uint32_t mask = 0, fixed = 0;
      for (int j = 0; j < op.nw; ++j) {
        o.pos[j] = sh.rank[op.pos[j]];
        mask |= 1u << o.pos[j];
        if (op.kind == TQK_K_PHASE || (op.kind != TQK_K_DIAG && j < op.nctrl)) fixed |= 1u << o.pos[j];
      }
      if (op.kind == TQK_K_X && !op.ctrl_val) fixed = 0;  // a flip under open controls
      o.fixed = static_cast<uint16_t>(fixed);
      int n = 0, reach = 0;
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        if ((mask >> q) & 1u) o.asc[n++] = static_cast<uint8_t>(q);
        reach += q < bl.k && sh.first[q] <= i0 + tid;
      }
      o.reach = static_cast<int16_t>(reach);
    }
    sh.op[tid] = o;
  }
  __syncthreads();
  for (int e = tid; e < kChunk * 16; e += blockDim.x) {
    const int i = e >> 4, q = e & 15;
    if (i0 + i >= bl.num_ops) break;
    const ShOp& o = sh.op[i];
    int n = 0;
    if (o.kind == TQK_K_PHASE) n = 1;
    else if (o.kind == TQK_K_DIAG) n = 1 << min(static_cast<int>(o.nw), 4);
    else if (o.kind == TQK_K_DENSE || o.kind == TQK_K_CTRL) n = 1 << 2 * (o.nw - o.nctrl);
    if (q < n) sh.m[i][q] = from_d2<C>(o.opnd[q]);
  }
  __syncthreads();
}

// Row g of those with the op's bits clear.
__device__ __forceinline__ int clear_row(int g, const ShOp& op) {
  for (int j = 0; j < op.nw; ++j) {
    const int p = op.asc[j];
    g = ((g >> p) << (p + 1)) | (g & ((1 << p) - 1));
  }
  return g;
}

// Rows of the patterns over op bits pos[from], .., pos[from + N - 1] (the first is the pattern's
// most significant bit).
template <int N>
__device__ __forceinline__ void pattern_rows(const ShOp& op, int from, int (&pat)[1 << N]) {
#pragma unroll
  for (int a = 0; a < (1 << N); ++a) {
    pat[a] = 0;
#pragma unroll
    for (int j = 0; j < N; ++j)
      if ((a >> (N - 1 - j)) & 1) pat[a] |= 1 << op.pos[from + j];
  }
}

template <typename C>
__device__ __forceinline__ C fma2(C a, C b, C c) {  // a b + c
  return C{fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y))};
}

// A matrix of one CTA: 2^reach rows (leading dimension ld) by 2^lc columns.
struct Part {
  int ld, lc;
  int reach;
};

// The rows an exchange op (flip, swap) swaps within the rows of one clear_row.
__device__ __forceinline__ void exchange_rows(const ShOp& op, int& r0, int& r1) {
  r0 = op.kind == TQK_K_X ? 0 : 1 << op.pos[op.nctrl];
  r1 = 1 << op.pos[op.kind == TQK_K_X ? op.nw - 1 : op.nctrl + 1];
}

// One target whose matrix has real diagonal and real (RY, H) or imaginary (RX) off-diagonal
// entries: half the float64 products.
__device__ __forceinline__ bool half_real(const C2* m) {
  return m[0].y == 0.0 && m[3].y == 0.0 && ((m[1].y == 0.0 && m[2].y == 0.0) || (m[1].x == 0.0 && m[2].x == 0.0));
}

__device__ __forceinline__ void build_half_real(C2* U, const Part& p, const ShOp& op, const C2* m) {
  const bool real = m[1].y == 0.0 && m[2].y == 0.0;
  const double d0 = m[0].x, d1 = m[3].x, o0 = real ? m[1].x : m[1].y, o1 = real ? m[2].x : m[2].y;
  const int items = 1 << (p.reach - op.nw + p.lc), high = p.ld << op.pos[op.nctrl];
  for (int w = threadIdx.x; w < items; w += blockDim.x) {
    C2* u = U + (clear_row(w >> p.lc, op) | op.fixed) * p.ld + (w & ((1 << p.lc) - 1));
    const C2 a = u[0], b = u[high];
    const C2 ta = real ? a : mul_i(a), tb = real ? b : mul_i(b);
    u[0] = C2{fma(o0, tb.x, d0 * a.x), fma(o0, tb.y, d0 * a.y)};
    u[high] = C2{fma(d1, b.x, o1 * ta.x), fma(d1, b.y, o1 * ta.y)};
  }
}

template <int KT>
__device__ __forceinline__ void build_dense(C2* U, const Part& p, const ShOp& op, const C2* m) {
  constexpr int DT = 1 << KT;
  int pat[DT];
  pattern_rows<KT>(op, op.nctrl, pat);
  C2 M[DT * DT];
#pragma unroll
  for (int e = 0; e < DT * DT; ++e) M[e] = m[e];
  const int items = 1 << (p.reach - op.nw + p.lc);
  for (int w = threadIdx.x; w < items; w += blockDim.x) {
    C2* u = U + (clear_row(w >> p.lc, op) | op.fixed) * p.ld + (w & ((1 << p.lc) - 1));
    C2 x[DT];
#pragma unroll
    for (int a = 0; a < DT; ++a) x[a] = u[pat[a] * p.ld];
#pragma unroll
    for (int a = 0; a < DT; ++a) {
      C2 y = cmul2(M[a * DT], x[0]);
#pragma unroll
      for (int c = 1; c < DT; ++c) y = fma2(M[a * DT + c], x[c], y);
      u[pat[a] * p.ld] = y;
    }
  }
}

__device__ void build_op(C2* U, const Part& p, const ShOp& op, const C2* m) {
  const int cols = 1 << p.lc, items = 1 << (p.reach - op.nw + p.lc);
  if (op.kind == TQK_K_PHASE) {
    const C2 ph = m[0];
    for (int w = threadIdx.x; w < items; w += blockDim.x) {
      C2& u = U[(clear_row(w >> p.lc, op) | op.fixed) * p.ld + (w & (cols - 1))];
      u = cmul2(ph, u);
    }
  } else if (op.kind == TQK_K_DIAG) {
    for (int w = threadIdx.x; w < 1 << (p.reach + p.lc); w += blockDim.x) {
      const int r = w >> p.lc;
      int di = 0;
      for (int j = 0; j < op.nw; ++j) di = (di << 1) | ((r >> op.pos[j]) & 1);
      C2& u = U[r * p.ld + (w & (cols - 1))];
      u = cmul2(op.nw <= 4 ? m[di] : from_d2<C2>(op.opnd[di]), u);
    }
  } else if (op.kind == TQK_K_X || op.kind == TQK_K_SWAP) {
    int r0, r1;
    exchange_rows(op, r0, r1);
    for (int w = threadIdx.x; w < items; w += blockDim.x) {
      C2* u = U + (clear_row(w >> p.lc, op) | op.fixed) * p.ld + (w & (cols - 1));
      const C2 v = u[r0 * p.ld];
      u[r0 * p.ld] = u[r1 * p.ld];
      u[r1 * p.ld] = v;
    }
  } else if (op.nw - op.nctrl == 1 && half_real(m)) {
    build_half_real(U, p, op, m);
  } else if (op.nw - op.nctrl == 1) {
    build_dense<1>(U, p, op, m);
  } else {
    build_dense<2>(U, p, op, m);
  }
}

// Column bits that the CTAs of a block share out: all that are offered while the blocks (and rows of those
// with a batch) are fewer than the SMs; beyond, a CTA keeps as many columns as its shared memory holds (2^9
// entries), since the reading and ordering of the ops is paid in each CTA.  (Always 8 CTAs a block: 100 blocks
// of 64 rows, 6 ops, k = 3 / 4 / 5 / 6 847 / 844 / 870 / 1023 us, so 132 / 140 / 286 / 1008; one CTA of 256 threads and
// all columns, whatever the width: 321 / 349 / 778 / 3000.)
__device__ __forceinline__ int columns_shared(const tqk_block_desc& bl) {
  const int64_t ctas = static_cast<int64_t>(gridDim.x) * (bl.batch > 1 ? bl.batch : 1);
  return ctas < kBuildPlaces ? bl.k : max(0, bl.k - min(4, kBuildEntryBits - bl.k));
}

__global__ void k_block_build(const tqk_block_desc* blocks, const tqk_block_op* ops, int split) {
  extern __shared__ double2 smem_u[];
  __shared__ Stage<C2> sh;
  C2* U = reinterpret_cast<C2*>(smem_u);
  const tqk_block_desc bl = blocks[blockIdx.x];
  const int64_t b = blockIdx.y;
  const int z = blockIdx.z;
  if (b >= bl.batch || !block_ok(bl)) return;
  split = min(split, columns_shared(bl));
  if (z >> split) return;
  const int tid = threadIdx.x, nth = blockDim.x, whole = bl.k - split;  // bits with all columns
  Part p{1 << whole, 0, 0};
  order_bits(sh, bl, ops);
  if (tid == 0) U[0] = mk(1.0, 0.0);
  __syncthreads();
  for (int i = 0; i <= bl.num_ops; ++i) {
    const bool last = i == bl.num_ops;  // then only the bits that no op touches are left
    const int q = i % kChunk;
    if (!last && q == 0) {
      __syncthreads();  // a skipped op at the end of the chunk before has no barrier after its kind is read
      stage_ops(sh, bl, ops, i, b);
    }
    if (!last && sh.op[q].kind < 0) continue;  // uniform for the CTA
    const int reach = last ? bl.k : sh.op[q].reach;
    while (p.reach < reach) {  // join: U <- U (x) identity on the next bit
      const int d = 1 << p.reach, cols = 1 << p.lc, v = (z >> max(p.reach - whole, 0)) & 1;
      const bool both = p.reach < whole;
      for (int w = tid; w < d << p.lc; w += nth) {
        C2* u = U + (w >> p.lc) * p.ld + (w & (cols - 1));
        const C2 val = *u, none = mk(0.0, 0.0);
        if (both) {
          u[cols] = none;
          u[d * p.ld] = none;
          u[d * p.ld + cols] = val;
        } else {
          *u = v ? none : val;
          u[d * p.ld] = v ? val : none;
        }
      }
      p.lc += both;
      ++p.reach;
      __syncthreads();
    }
    if (last) break;
    build_op(U, p, sh.op[q], sh.m[q]);
    __syncthreads();
  }
  const int D = 1 << bl.k;
  double2* dst = static_cast<double2*>(bl.u) + b * D * D;
  for (int e = tid; e < D << whole; e += nth) {
    const C2 v = U[e];
    dst[sh.at[e >> whole] * D + sh.at[(e & ((1 << whole) - 1)) | (z << whole)]] = make_double2(v.x, v.y);
  }
}

// ---- reverse.  With W the product of the ops before an op and X = (ops after)^H dL/dU, the
// operand's cotangent is the sum, over the rows with the op's control bits set and over the
// columns, of X[row with target pattern a] conj(W[row with target pattern b]) at entry (a, b)
// (diagonal ops: a = b over all op bits; phase ops: the single all-ones pattern).  Threads sum
// their items in float32 (diagonals on more than two bits in float64), warps and CTAs in float64.

struct Sums {
  double v[2][8][32];  // by op parity: a warp's sums, written before the barrier that ends the op
};

// Sums of v over the warp by halves (each step hands half of the values over: NV - 1 + log2(32/NV)
// float64 additions instead of 5 NV) into out[0 .. NV).
template <int NV, typename R>
__device__ __forceinline__ void warp_sums(const R (&v)[NV], double* out) {
  const int lane = threadIdx.x & 31;
  double s[NV];
#pragma unroll
  for (int h = NV / 2, o = 16; h >= 1; h >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      if (h == NV / 2) {  // the first hand-over in the type of the terms
        const R send = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
        s[i] = static_cast<double>(keep) + static_cast<double>(__shfl_xor_sync(0xffffffffu, send, o));
      } else {
        const double send = up ? s[i] : s[i + h], keep = up ? s[i + h] : s[i];
        s[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
  }
#pragma unroll
  for (int o = 16 / NV; o >= 1; o >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
  if (lane % (32 / NV) == 0) out[lane / (32 / NV)] = s[0];
}

// X (cotangent) and W to before a dense op; its cotangent's warp sums into out.  Warps without
// items add nothing (active_warps leaves them out).
template <int KT>
__device__ __forceinline__ void unbuild_dense(F2* X, F2* W, const Part& p, const ShOp& op, const F2* m, double* out) {
  constexpr int DT = 1 << KT, NE = DT * DT;
  int pat[DT];
  pattern_rows<KT>(op, op.nctrl, pat);
  F2 M[NE];
#pragma unroll
  for (int e = 0; e < NE; ++e) M[e] = m[e];
  float acc[2 * NE];
#pragma unroll
  for (int q = 0; q < 2 * NE; ++q) acc[q] = 0.f;
  const int items = 1 << (p.reach - op.nw + p.lc);
  if (static_cast<int>(threadIdx.x & ~31u) >= items) return;
  for (int w = threadIdx.x; w < items; w += blockDim.x) {
    const int at = (clear_row(w >> p.lc, op) | op.fixed) * p.ld + (w & ((1 << p.lc) - 1));
    F2 xs[DT], ws[DT], wn[DT];
#pragma unroll
    for (int a = 0; a < DT; ++a) {
      xs[a] = X[at + pat[a] * p.ld];
      ws[a] = W[at + pat[a] * p.ld];
    }
#pragma unroll
    for (int a = 0; a < DT; ++a) {
      F2 y = cmul2(conj2(M[a]), ws[0]), g = cmul2(conj2(M[a]), xs[0]);
#pragma unroll
      for (int c = 1; c < DT; ++c) {
        y = fma2(conj2(M[c * DT + a]), ws[c], y);
        g = fma2(conj2(M[c * DT + a]), xs[c], g);
      }
      wn[a] = y;
      W[at + pat[a] * p.ld] = y;
      X[at + pat[a] * p.ld] = g;
    }
#pragma unroll
    for (int a = 0; a < DT; ++a)
#pragma unroll
      for (int c = 0; c < DT; ++c) {
        acc[2 * (a * DT + c)] += xs[a].x * wn[c].x + xs[a].y * wn[c].y;  // x * conj(w)
        acc[2 * (a * DT + c) + 1] += xs[a].y * wn[c].x - xs[a].x * wn[c].y;
      }
  }
  if (op.grad != nullptr) warp_sums(acc, out);
}

// The same for the 2^NW patterns over the op's last NW bits with its other bits at `fixed`
// (diagonals of up to 4 bits, parts of larger ones, phases: NW = 0).
template <int NW>
__device__ __forceinline__ void unbuild_diag(F2* X, F2* W, const Part& p, const ShOp& op, int fixed, const F2* m,
                                             double* out) {
  constexpr int DT = 1 << NW;
  int pat[DT];
  pattern_rows<NW>(op, op.nw - NW, pat);
  typename std::conditional<(NW > 2), double, float>::type acc[2 * DT];
#pragma unroll
  for (int q = 0; q < 2 * DT; ++q) acc[q] = 0;
  const int items = 1 << (p.reach - op.nw + p.lc);
  if (static_cast<int>(threadIdx.x & ~31u) >= items) return;
  for (int w = threadIdx.x; w < items; w += blockDim.x) {
    const int at = (clear_row(w >> p.lc, op) | fixed) * p.ld + (w & ((1 << p.lc) - 1));
#pragma unroll
    for (int a = 0; a < DT; ++a) {
      const int i = at + pat[a] * p.ld;
      const F2 d = conj2(m[a]), x = X[i], w2 = cmul2(d, W[i]);
      acc[2 * a] += x.x * w2.x + x.y * w2.y;
      acc[2 * a + 1] += x.y * w2.x - x.x * w2.y;
      W[i] = w2;
      X[i] = cmul2(d, x);
    }
  }
  if (op.grad != nullptr) warp_sums(acc, out);
}

// After a barrier: the CTA's sums added to the operand's cotangent.
__device__ __forceinline__ void add_sums(const double (*v)[32], const Part& p, const ShOp& op, double* grad, int count) {
  if (static_cast<int>(threadIdx.x) >= count) return;
  const int warps = min(static_cast<int>(blockDim.x >> 5), max(1, (1 << (p.reach - op.nw + p.lc)) >> 5));
  double t = 0.0;
  for (int w = 0; w < warps; ++w) t += v[w][threadIdx.x];
  atomicAdd(grad + threadIdx.x, t);
}

// Returns the number of sums.
__device__ int unbuild_op(F2* X, F2* W, const Part& p, const ShOp& op, F2* m, Sums& sums, int par) {
  double* out = sums.v[par][threadIdx.x >> 5];
  if (op.kind == TQK_K_X || op.kind == TQK_K_SWAP) {
    int r0, r1;
    exchange_rows(op, r0, r1);
    const int items = 1 << (p.reach - op.nw + p.lc);
    for (int w = threadIdx.x; w < items; w += blockDim.x) {
      const int at = (clear_row(w >> p.lc, op) | op.fixed) * p.ld + (w & ((1 << p.lc) - 1));
      const int i0 = at + r0 * p.ld, i1 = at + r1 * p.ld;
      const F2 w0 = W[i0], x0 = X[i0];
      W[i0] = W[i1];
      W[i1] = w0;
      X[i0] = X[i1];
      X[i1] = x0;
    }
    return 0;
  }
  if (op.kind == TQK_K_PHASE) {
    unbuild_diag<0>(X, W, p, op, op.fixed, m, out);
    return 2;
  }
  if (op.kind == TQK_K_DIAG) {
    if (op.nw == 1) unbuild_diag<1>(X, W, p, op, 0, m, out);
    else if (op.nw == 2) unbuild_diag<2>(X, W, p, op, 0, m, out);
    else if (op.nw == 3) unbuild_diag<3>(X, W, p, op, 0, m, out);
    else {
      // one part of 16 patterns for each value of the bits before the last four; all but the
      // last are added here, the last by the caller
      const int high = op.nw - 4;
      for (int h = 0;; ++h) {
        int fixed = 0;
        for (int j = 0; j < high; ++j)
          if ((h >> (high - 1 - j)) & 1) fixed |= 1 << op.pos[j];
        unbuild_diag<4>(X, W, p, op, fixed, m, out);
        if (h == (1 << high) - 1) break;
        __syncthreads();
        if (op.grad != nullptr) add_sums(sums.v[par], p, op, op.grad + 32 * h, 32);
        if (threadIdx.x < 16) m[threadIdx.x] = from_d2<F2>(op.opnd[16 * (h + 1) + threadIdx.x]);
        __syncthreads();
      }
    }
    return 2 << min(static_cast<int>(op.nw), 4);
  }
  if (op.nw - op.nctrl == 1) {
    unbuild_dense<1>(X, W, p, op, m, out);
    return 8;
  }
  unbuild_dense<2>(X, W, p, op, m, out);
  return 32;
}

__global__ void k_block_unbuild(const tqk_block_desc* blocks, const tqk_block_op* ops, int split) {
  extern __shared__ double2 smem_u[];
  __shared__ Stage<F2> sh;
  __shared__ Sums sums;
  const tqk_block_desc bl = blocks[blockIdx.x];
  const int64_t b = blockIdx.y;
  const int z = blockIdx.z;
  if (b >= bl.batch || bl.gu == nullptr || !block_ok(bl)) return;
  split = min(split, bl.k);
  if (z >> split) return;
  const int tid = threadIdx.x, nth = blockDim.x, whole = bl.k - split;
  const int D = 1 << bl.k;
  Part p{1 << whole, whole, bl.k};
  F2* W = reinterpret_cast<F2*>(smem_u);
  F2* X = W + (D << whole);
  order_bits(sh, bl, ops);
  const double2* us = static_cast<const double2*>(bl.u) + b * D * D;
  const double2* gs = static_cast<const double2*>(bl.gu) + b * D * D;
  for (int e = tid; e < D << whole; e += nth) {
    const int i = sh.at[e >> whole] * D + sh.at[(e & ((1 << whole) - 1)) | (z << whole)];
    W[e] = from_d2<F2>(us[i]);
    X[e] = from_d2<F2>(gs[i]);
  }
  int par = 0;
  for (int i = bl.num_ops - 1; i >= 0; --i) {
    const int q = i % kChunk;
    if (q == kChunk - 1 || i == bl.num_ops - 1) {
      __syncthreads();  // the sums of the chunk after read its table
      stage_ops(sh, bl, ops, i - q, b);
    }
    const ShOp& op = sh.op[q];
    if (op.kind < 0) continue;  // uniform for the CTA
    while (p.reach > op.reach) {  // drop: X <- its partial trace over the last bit
      --p.reach;
      const bool both = p.reach < whole;
      p.lc -= both;
      const int d = 1 << p.reach, cols = 1 << p.lc;
      if (both || ((z >> (p.reach - whole)) & 1)) {
        for (int w = tid; w < d << p.lc; w += nth) {
          const int e = (w >> p.lc) * p.ld + (w & (cols - 1)), o = e + d * p.ld;
          if (both) {
            X[e] = cadd2(X[e], X[o + cols]);
          } else {  // this CTA's columns have the bit set: so have the rows that meet W's
            X[e] = X[o];
            W[e] = W[o];
          }
        }
        __syncthreads();
      }
    }
    const int count = unbuild_op(X, W, p, op, sh.m[q], sums, par);
    __syncthreads();
    if (op.grad != nullptr && count > 0) {
      const int skip = op.kind == TQK_K_DIAG && op.nw > 4 ? 32 * ((1 << (op.nw - 4)) - 1) : 0;
      add_sums(sums.v[par], p, op, op.grad + skip, count);
    }
    par ^= 1;
  }
}

}  // namespace prog
}  // namespace tqk

using namespace tqk;

extern "C" int tqk_gate_operand_size(int type) { return prog::operand_size(type); }

extern "C" int tqk_gate_operands(const tqk_gate_desc* gates, int ngates, void* stream) {
  if (ngates <= 0) return TQK_OK;
  if (!gates) return fail(TQK_BAD_POINTER, "tqk_gate_operands: null gate table");
  prog::k_gate_operands<<<ngates, 32, 0, as_stream(stream)>>>(gates, ngates);
  return launch_status("tqk_gate_operands");
}

extern "C" int tqk_param_grads(const tqk_gate_desc* gates, int ngates, void* stream) {
  if (ngates <= 0) return TQK_OK;
  if (!gates) return fail(TQK_BAD_POINTER, "tqk_param_grads: null gate table");
  prog::k_param_grads<<<ngates, 32, 0, as_stream(stream)>>>(gates, ngates);
  return launch_status("tqk_param_grads");
}

// Column bits that a block's CTAs share out, and threads: best of splits 0 to 3 with 64 to 256
// threads on the circuits named at the kernels (build 154 + 259 us against 299 + 299 without a
// split; reverse 147 + 156 against 152 + 206).  The reverse sums at most 8
// float32 terms a thread (64 rows x 16 columns over 64 threads, one target).  Idle CTAs (rows
// of a block without a batch, narrow blocks) leave at once.
constexpr int kBuildSplit = 3, kBuildThreads = 128;  // (6-wire blocks: 2^12 entries)
static_assert(12 - kBuildSplit == prog::kBuildEntryBits, "a CTA's share of a 6-wire block");
constexpr int kUnbuildSplit = 2, kUnbuildThreads = 64;

extern "C" int tqk_block_build(const tqk_block_desc* blocks, int nblocks, int max_batch, const tqk_block_op* ops,
                               void* stream) {
  if (nblocks <= 0) return TQK_OK;
  if (!blocks || !ops) return fail(TQK_BAD_POINTER, "tqk_block_build: null pointer");
  if (max_batch < 1 || max_batch > 65535) return fail(TQK_BAD_SHAPE, "tqk_block_build: batch %d", max_batch);
  const size_t smem = sizeof(double2) << prog::kBuildEntryBits;
  dim3 grid(nblocks, max_batch, 1 << kBuildSplit);
  prog::k_block_build<<<grid, kBuildThreads, smem, as_stream(stream)>>>(blocks, ops, kBuildSplit);
  return launch_status("tqk_block_build");
}

extern "C" int tqk_block_unbuild(const tqk_block_desc* blocks, int nblocks, int max_batch, const tqk_block_op* ops,
                                 void* stream) {
  if (nblocks <= 0) return TQK_OK;
  if (!blocks || !ops) return fail(TQK_BAD_POINTER, "tqk_block_unbuild: null pointer");
  if (max_batch < 1 || max_batch > 65535) return fail(TQK_BAD_SHAPE, "tqk_block_unbuild: batch %d", max_batch);
  const size_t smem = 2 * (64 * 64 >> kUnbuildSplit) * sizeof(float2);
  dim3 grid(nblocks, max_batch, 1 << kUnbuildSplit);
  prog::k_block_unbuild<<<grid, kUnbuildThreads, smem, as_stream(stream)>>>(blocks, ops, kUnbuildSplit);
  return launch_status("tqk_block_unbuild");
}
