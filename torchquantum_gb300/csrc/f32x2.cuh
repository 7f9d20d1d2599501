// f32x2.cuh -- amplitudes in named registers, for loops that apply ops chosen at run time.
//
// A thread keeps its amplitudes across a loop whose body is a switch over op kinds and
// register slots.  As a C++ array they become values that every case redefines, and the
// code behind the switch fills with moves and spills that bring them back to one place
// (measured: ~500 issue cycles for a flip of 16 psi and lam amplitudes, a pure renaming).
// So they live in registers declared once per kernel in PTX and every op updates them by
// name: ta<q> (psi), tb<q> (lam), and the cotangent sums gr<e>, gi<e>, hr, hi.
//
// An amplitude (re, im) is one 64-bit register.  A product with a complex factor m is one
// packed FMA (fma.rn.f32x2, two multiply-adds per issue slot) by (mr, mr) and two scalar
// FMAs by -+mi, whose signs are operand modifiers: three slots for four multiply-adds and
// no moves.  (The float32 pipe does as many multiply-adds a cycle packed as scalar; a
// second packed FMA would need a swap or a negation on the half-rate integer pipe.)
#pragma once

#include <stdint.h>

namespace tqk {
namespace f2 {

using pair = unsigned long long;  // low word, high word

// A complex factor: (mr, mr) and mi.
struct Factor {
  pair r;
  float i;
};
__device__ __forceinline__ pair make(float lo, float hi) {
  pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}

// Once per kernel, before any other use: for 16 amplitudes of two states and sums, or for
// 32 of one state.
#define TQK_AMPLITUDE_REGISTERS asm volatile(".reg .b64 ta<16>, tb<16>, gr<4>, hr;\n .reg .f32 gi<4>, hi;")
#define TQK_AMPLITUDE_REGISTERS_32 asm volatile(".reg .b64 ta<32>;")

// P: 'a' or 'b'.  Load / store the amplitudes Q, Q + 1 (16 bytes of shared memory).
#define TQK_DEFINE_REGS(NAME, P)                                                                                  \
  struct NAME {                                                                                                   \
    template <int Q>                                                                                              \
    static __device__ __forceinline__ void load(uint32_t addr) {                                                  \
      asm volatile("ld.shared.v2.b64 {t" P "%1, t" P "%2}, [%0];" ::"r"(addr), "n"(Q), "n"(Q + 1) : "memory");    \
    }                                                                                                             \
    template <int Q>                                                                                              \
    static __device__ __forceinline__ void store(uint32_t addr) {                                                 \
      asm volatile("st.shared.v2.b64 [%0], {t" P "%1, t" P "%2};" ::"r"(addr), "n"(Q), "n"(Q + 1) : "memory");    \
    }                                                                                                             \
    template <int Q, int U>                                                                                       \
    static __device__ __forceinline__ void swap() {                                                               \
      asm volatile(                                                                                               \
          "{\n .reg .b64 t;\n mov.b64 t, t" P "%0;\n mov.b64 t" P "%0, t" P "%1;\n mov.b64 t" P "%1, t;\n}" ::"n"(Q), \
          "n"(U));                                                                                                \
    }                                                                                                             \
    /* exclusive or with a sign pattern */                                                                        \
    template <int Q>                                                                                              \
    static __device__ __forceinline__ void flip(pair s) {                                                         \
      asm volatile("xor.b64 t" P "%0, t" P "%0, %1;" ::"n"(Q), "l"(s));                                            \
    }                                                                                                             \
    /* (Q, U) <- real 2x2.  Here and below an output's products with its own input come last: in gates near  \
       the identity they are the large ones, and only the last addition rounds at their size */                 \
    template <int Q, int U>                                                                                       \
    static __device__ __forceinline__ void real2(const Factor (&m)[4]) {                                          \
      asm volatile(                                                                                               \
          "{\n .reg .b64 t, u;\n"                                                                                 \
          " mul.rn.f32x2 t, %3, t" P "%1;\n mul.rn.f32x2 u, %4, t" P "%0;\n"                                       \
          " fma.rn.f32x2 t" P "%0, %2, t" P "%0, t;\n fma.rn.f32x2 t" P "%1, %5, t" P "%1, u;\n}" ::"n"(Q),       \
          "n"(U), "l"(m[0].r), "l"(m[1].r), "l"(m[2].r), "l"(m[3].r));                                            \
    }                                                                                                             \
    /* (Q, U) <- complex 2x2: the imaginary products of both inputs first */                                      \
    template <int Q, int U>                                                                                       \
    static __device__ __forceinline__ void dense2(const Factor (&m)[4]) {                                         \
      asm volatile(                                                                                               \
          "{\n .reg .f32 x, y, z, w, ny, nw, p, q;\n .reg .b64 t, u;\n"                                            \
          " mov.b64 {x, y}, t" P "%0;\n mov.b64 {z, w}, t" P "%1;\n neg.f32 ny, y;\n neg.f32 nw, w;\n"             \
          " mul.rn.f32 p, %7, nw;\n mul.rn.f32 q, %7, z;\n"                                                        \
          " fma.rn.f32 p, %6, ny, p;\n fma.rn.f32 q, %6, x, q;\n mov.b64 t, {p, q};\n"                             \
          " mul.rn.f32 p, %8, ny;\n mul.rn.f32 q, %8, x;\n"                                                        \
          " fma.rn.f32 p, %9, nw, p;\n fma.rn.f32 q, %9, z, q;\n mov.b64 u, {p, q};\n"                             \
          " fma.rn.f32x2 u, %4, t" P "%0, u;\n fma.rn.f32x2 t, %3, t" P "%1, t;\n"                                 \
          " fma.rn.f32x2 t" P "%1, %5, t" P "%1, u;\n fma.rn.f32x2 t" P "%0, %2, t" P "%0, t;\n}" ::"n"(Q),       \
          "n"(U), "l"(m[0].r), "l"(m[1].r), "l"(m[2].r), "l"(m[3].r), "f"(m[0].i), "f"(m[1].i), "f"(m[2].i),      \
          "f"(m[3].i));                                                                                           \
    }                                                                                                             \
    template <int Q>                                                                                              \
    static __device__ __forceinline__ void scale(const Factor& m) {                                               \
      asm volatile(                                                                                               \
          "{\n .reg .f32 x, y, p, q;\n .reg .b64 t;\n"                                                             \
          " mov.b64 {x, y}, t" P "%0;\n neg.f32 y, y;\n mul.rn.f32 p, %2, y;\n mul.rn.f32 q, %2, x;\n"            \
          " mov.b64 t, {p, q};\n fma.rn.f32x2 t" P "%0, %1, t" P "%0, t;\n}" ::"n"(Q), "l"(m.r), "f"(m.i));        \
    }                                                                                                             \
  }
TQK_DEFINE_REGS(Psi, "a");
TQK_DEFINE_REGS(Lam, "b");
#undef TQK_DEFINE_REGS

// Cotangent sums: sum E += lam_L conj(psi_Y).  gr holds lam.re psi.re and lam.im psi.im in
// its halves, gi lam.im psi.re - lam.re psi.im.
template <int E>
__device__ __forceinline__ void sum_zero() {
  asm volatile("mov.b64 gr%0, 0;\n mov.f32 gi%0, 0f00000000;" ::"n"(E));
}
template <int E, int L, int Y>
__device__ __forceinline__ void sum_add() {
  asm volatile(
      "{\n .reg .f32 x, y, z, w, nx;\n mov.b64 {x, y}, tb%1;\n mov.b64 {z, w}, ta%2;\n neg.f32 nx, x;\n"
      " fma.rn.f32x2 gr%0, tb%1, ta%2, gr%0;\n fma.rn.f32 gi%0, y, z, gi%0;\n fma.rn.f32 gi%0, nx, w, gi%0;\n}" ::"n"(E),
      "n"(L), "n"(Y));
}
template <int E>
__device__ __forceinline__ float2 sum_get() {
  float2 v;
  asm volatile("{\n .reg .f32 x, y;\n mov.b64 {x, y}, gr%2;\n add.rn.f32 %0, x, y;\n mov.f32 %1, gi%2;\n}"
               : "=f"(v.x), "=f"(v.y)
               : "n"(E));
  return v;
}
// A sum whose entry is known at run time only: gathered in hr, hi, then put in its place.
__device__ __forceinline__ void side_zero() { asm volatile("mov.b64 hr, 0;\n mov.f32 hi, 0f00000000;"); }
template <int Q>
__device__ __forceinline__ void side_add() {
  asm volatile(
      "{\n .reg .f32 x, y, z, w, nx;\n mov.b64 {x, y}, tb%0;\n mov.b64 {z, w}, ta%0;\n neg.f32 nx, x;\n"
      " fma.rn.f32x2 hr, tb%0, ta%0, hr;\n fma.rn.f32 hi, y, z, hi;\n fma.rn.f32 hi, nx, w, hi;\n}" ::"n"(Q));
}
template <int E>
__device__ __forceinline__ void side_put() {
  asm volatile("mov.b64 gr%0, hr;\n mov.f32 gi%0, hi;" ::"n"(E));
}

}  // namespace f2
}  // namespace tqk
