// carry_chain.cuh -- multi-word add-with-carry chains in inline PTX
// (internal header).
//
// All compute the N-word sum s[0..N) = a[0..N) + b[0..N) + carry in, the carry
// rippling from word 0 upward through the hardware carry flag (add.cc /
// addc.cc), one instruction per word.
//   add_chain8_cc(s, a, b, cin, cout) : carry in if cin != 0 (cin + 0xFFFFFFFF
//     sets the flag), cout = carry out of word 7 (0 or 1)
//   add_chainN_pp and its halves : carries popped from and pushed to words
//   add_runN : no carry in or out
#pragma once
#include <cstdint>

namespace ngia {

__device__ __forceinline__ void add_chain8_cc(uint32_t *s, const uint32_t *a, const uint32_t *b, uint32_t cin, uint32_t &cout) {
  asm("{\n\t.reg .u32 t;\n\t"
      "add.cc.u32 t, %25, 0xFFFFFFFF;\n\t"
      "addc.cc.u32 %0, %9, %17;\n\t"
      "addc.cc.u32 %1, %10, %18;\n\t"
      "addc.cc.u32 %2, %11, %19;\n\t"
      "addc.cc.u32 %3, %12, %20;\n\t"
      "addc.cc.u32 %4, %13, %21;\n\t"
      "addc.cc.u32 %5, %14, %22;\n\t"
      "addc.cc.u32 %6, %15, %23;\n\t"
      "addc.cc.u32 %7, %16, %24;\n\t"
      "addc.u32 %8, 0, 0;\n\t"
      "}"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]), "=r"(cout)
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(cin));
}

// ---- carry words ---------------------------------------------------------------
// Chains whose carry in is popped from the top bit of a word (add.cc x, x, x:
// the flag takes bit 31, x shifts left) and whose carry out is appended at
// the bottom of another (addc x, x, x: x = 2x + flag).  32 calls in column
// order fill `cout` with column 0's carry in bit 31, which is the order the
// next chain pops them in.
//   add_chainN_pp : pop in, push out
//   add_chain8_pc : pop in, carry out as 0/1 in c (first half of 16 words)
//   add_chain8_cp : carry in from c != 0, push out (second half)
__device__ __forceinline__ void add_chain3_pp(uint32_t *s, const uint32_t *a, const uint32_t *b,
                                              uint32_t &cin, uint32_t &cout) {
  asm("add.cc.u32 %3, %3, %3;\n\t"
      "addc.cc.u32 %0, %5, %8;\n\t"
      "addc.cc.u32 %1, %6, %9;\n\t"
      "addc.cc.u32 %2, %7, %10;\n\t"
      "addc.u32 %4, %4, %4;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "+r"(cin), "+r"(cout)
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(b[0]), "r"(b[1]), "r"(b[2]));
}

__device__ __forceinline__ void add_chain4_pp(uint32_t *s, const uint32_t *a, const uint32_t *b,
                                              uint32_t &cin, uint32_t &cout) {
  asm("add.cc.u32 %4, %4, %4;\n\t"
      "addc.cc.u32 %0, %6, %10;\n\t"
      "addc.cc.u32 %1, %7, %11;\n\t"
      "addc.cc.u32 %2, %8, %12;\n\t"
      "addc.cc.u32 %3, %9, %13;\n\t"
      "addc.u32 %5, %5, %5;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "+r"(cin), "+r"(cout)
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]));
}

__device__ __forceinline__ void add_chain6_pp(uint32_t *s, const uint32_t *a, const uint32_t *b,
                                              uint32_t &cin, uint32_t &cout) {
  asm("add.cc.u32 %6, %6, %6;\n\t"
      "addc.cc.u32 %0, %8, %14;\n\t"
      "addc.cc.u32 %1, %9, %15;\n\t"
      "addc.cc.u32 %2, %10, %16;\n\t"
      "addc.cc.u32 %3, %11, %17;\n\t"
      "addc.cc.u32 %4, %12, %18;\n\t"
      "addc.cc.u32 %5, %13, %19;\n\t"
      "addc.u32 %7, %7, %7;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "+r"(cin), "+r"(cout)
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]),
        "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]));
}

__device__ __forceinline__ void add_chain8_pp(uint32_t *s, const uint32_t *a, const uint32_t *b,
                                              uint32_t &cin, uint32_t &cout) {
  asm("add.cc.u32 %8, %8, %8;\n\t"
      "addc.cc.u32 %0, %10, %18;\n\t"
      "addc.cc.u32 %1, %11, %19;\n\t"
      "addc.cc.u32 %2, %12, %20;\n\t"
      "addc.cc.u32 %3, %13, %21;\n\t"
      "addc.cc.u32 %4, %14, %22;\n\t"
      "addc.cc.u32 %5, %15, %23;\n\t"
      "addc.cc.u32 %6, %16, %24;\n\t"
      "addc.cc.u32 %7, %17, %25;\n\t"
      "addc.u32 %9, %9, %9;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]), "+r"(cin), "+r"(cout)
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
}

__device__ __forceinline__ void add_chain8_pc(uint32_t *s, const uint32_t *a, const uint32_t *b,
                                              uint32_t &cin, uint32_t &c) {
  asm("add.cc.u32 %8, %8, %8;\n\t"
      "addc.cc.u32 %0, %10, %18;\n\t"
      "addc.cc.u32 %1, %11, %19;\n\t"
      "addc.cc.u32 %2, %12, %20;\n\t"
      "addc.cc.u32 %3, %13, %21;\n\t"
      "addc.cc.u32 %4, %14, %22;\n\t"
      "addc.cc.u32 %5, %15, %23;\n\t"
      "addc.cc.u32 %6, %16, %24;\n\t"
      "addc.cc.u32 %7, %17, %25;\n\t"
      "addc.u32 %9, 0, 0;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]), "+r"(cin), "=r"(c)
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
}

__device__ __forceinline__ void add_chain8_cp(uint32_t *s, const uint32_t *a, const uint32_t *b,
                                              uint32_t c, uint32_t &cout) {
  asm("{\n\t.reg .u32 t;\n\t"
      "add.cc.u32 t, %25, 0xFFFFFFFF;\n\t"
      "addc.cc.u32 %0, %9, %17;\n\t"
      "addc.cc.u32 %1, %10, %18;\n\t"
      "addc.cc.u32 %2, %11, %19;\n\t"
      "addc.cc.u32 %3, %12, %20;\n\t"
      "addc.cc.u32 %4, %13, %21;\n\t"
      "addc.cc.u32 %5, %14, %22;\n\t"
      "addc.cc.u32 %6, %15, %23;\n\t"
      "addc.cc.u32 %7, %16, %24;\n\t"
      "addc.u32 %8, %8, %8;\n\t"
      "}"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]), "+r"(cout)
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(c));
}

// s[0..K) = a + b + (carry popped from cin), carry out pushed into cout.
template <int K>
__device__ __forceinline__ void add_words_pp(uint32_t *s, const uint32_t *a, const uint32_t *b,
                                             uint32_t &cin, uint32_t &cout) {
  if constexpr (K == 3) add_chain3_pp(s, a, b, cin, cout);
  else if constexpr (K == 4) add_chain4_pp(s, a, b, cin, cout);
  else if constexpr (K == 6) add_chain6_pp(s, a, b, cin, cout);
  else if constexpr (K == 8) add_chain8_pp(s, a, b, cin, cout);
  else {
    static_assert(K == 16, "carry-word chains of 3, 4, 6, 8 or 16 words");
    uint32_t c;
    add_chain8_pc(s, a, b, cin, c);
    add_chain8_cp(s + 8, a + 8, b + 8, c, cout);
  }
}


// ---- one chain of a window's words, no carry in or out -------------------------
// add_run<N>(s, a, b): s[0..N) = a[0..N) + b[0..N) as one N-word number, the
// carry rippling through the flag across the whole run (no carry value
// materialised between words).  Written out for each window width.
__device__ __forceinline__ void add_run4(uint32_t *s, const uint32_t *a, const uint32_t *b) {
  asm(
      "add.cc.u32 %0, %4, %8;\n\t"
      "addc.cc.u32 %1, %5, %9;\n\t"
      "addc.cc.u32 %2, %6, %10;\n\t"
      "addc.u32 %3, %7, %11;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]));
}
__device__ __forceinline__ void add_run5(uint32_t *s, const uint32_t *a, const uint32_t *b) {
  asm(
      "add.cc.u32 %0, %5, %10;\n\t"
      "addc.cc.u32 %1, %6, %11;\n\t"
      "addc.cc.u32 %2, %7, %12;\n\t"
      "addc.cc.u32 %3, %8, %13;\n\t"
      "addc.u32 %4, %9, %14;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]));
}
__device__ __forceinline__ void add_run6(uint32_t *s, const uint32_t *a, const uint32_t *b) {
  asm(
      "add.cc.u32 %0, %6, %12;\n\t"
      "addc.cc.u32 %1, %7, %13;\n\t"
      "addc.cc.u32 %2, %8, %14;\n\t"
      "addc.cc.u32 %3, %9, %15;\n\t"
      "addc.cc.u32 %4, %10, %16;\n\t"
      "addc.u32 %5, %11, %17;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]));
}
__device__ __forceinline__ void add_run7(uint32_t *s, const uint32_t *a, const uint32_t *b) {
  asm(
      "add.cc.u32 %0, %7, %14;\n\t"
      "addc.cc.u32 %1, %8, %15;\n\t"
      "addc.cc.u32 %2, %9, %16;\n\t"
      "addc.cc.u32 %3, %10, %17;\n\t"
      "addc.cc.u32 %4, %11, %18;\n\t"
      "addc.cc.u32 %5, %12, %19;\n\t"
      "addc.u32 %6, %13, %20;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]));
}
__device__ __forceinline__ void add_run8(uint32_t *s, const uint32_t *a, const uint32_t *b) {
  asm(
      "add.cc.u32 %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32 %7, %15, %23;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
}
__device__ __forceinline__ void add_run9(uint32_t *s, const uint32_t *a, const uint32_t *b) {
  asm(
      "add.cc.u32 %0, %9, %18;\n\t"
      "addc.cc.u32 %1, %10, %19;\n\t"
      "addc.cc.u32 %2, %11, %20;\n\t"
      "addc.cc.u32 %3, %12, %21;\n\t"
      "addc.cc.u32 %4, %13, %22;\n\t"
      "addc.cc.u32 %5, %14, %23;\n\t"
      "addc.cc.u32 %6, %15, %24;\n\t"
      "addc.cc.u32 %7, %16, %25;\n\t"
      "addc.u32 %8, %17, %26;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]), "=r"(s[8])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(a[8]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(b[8]));
}
__device__ __forceinline__ void add_run10(uint32_t *s, const uint32_t *a, const uint32_t *b) {
  asm(
      "add.cc.u32 %0, %10, %20;\n\t"
      "addc.cc.u32 %1, %11, %21;\n\t"
      "addc.cc.u32 %2, %12, %22;\n\t"
      "addc.cc.u32 %3, %13, %23;\n\t"
      "addc.cc.u32 %4, %14, %24;\n\t"
      "addc.cc.u32 %5, %15, %25;\n\t"
      "addc.cc.u32 %6, %16, %26;\n\t"
      "addc.cc.u32 %7, %17, %27;\n\t"
      "addc.cc.u32 %8, %18, %28;\n\t"
      "addc.u32 %9, %19, %29;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]), "=r"(s[8]), "=r"(s[9])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(a[8]), "r"(a[9]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(b[8]), "r"(b[9]));
}
__device__ __forceinline__ void add_run11(uint32_t *s, const uint32_t *a, const uint32_t *b) {
  asm(
      "add.cc.u32 %0, %11, %22;\n\t"
      "addc.cc.u32 %1, %12, %23;\n\t"
      "addc.cc.u32 %2, %13, %24;\n\t"
      "addc.cc.u32 %3, %14, %25;\n\t"
      "addc.cc.u32 %4, %15, %26;\n\t"
      "addc.cc.u32 %5, %16, %27;\n\t"
      "addc.cc.u32 %6, %17, %28;\n\t"
      "addc.cc.u32 %7, %18, %29;\n\t"
      "addc.cc.u32 %8, %19, %30;\n\t"
      "addc.cc.u32 %9, %20, %31;\n\t"
      "addc.u32 %10, %21, %32;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]), "=r"(s[8]), "=r"(s[9]), "=r"(s[10])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(a[8]), "r"(a[9]), "r"(a[10]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(b[8]), "r"(b[9]), "r"(b[10]));
}
__device__ __forceinline__ void add_run12(uint32_t *s, const uint32_t *a, const uint32_t *b) {
  asm(
      "add.cc.u32 %0, %12, %24;\n\t"
      "addc.cc.u32 %1, %13, %25;\n\t"
      "addc.cc.u32 %2, %14, %26;\n\t"
      "addc.cc.u32 %3, %15, %27;\n\t"
      "addc.cc.u32 %4, %16, %28;\n\t"
      "addc.cc.u32 %5, %17, %29;\n\t"
      "addc.cc.u32 %6, %18, %30;\n\t"
      "addc.cc.u32 %7, %19, %31;\n\t"
      "addc.cc.u32 %8, %20, %32;\n\t"
      "addc.cc.u32 %9, %21, %33;\n\t"
      "addc.cc.u32 %10, %22, %34;\n\t"
      "addc.u32 %11, %23, %35;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]), "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(a[8]), "r"(a[9]), "r"(a[10]), "r"(a[11]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(b[8]), "r"(b[9]), "r"(b[10]), "r"(b[11]));
}
__device__ __forceinline__ void add_run14(uint32_t *s, const uint32_t *a, const uint32_t *b) {
  asm(
      "add.cc.u32 %0, %14, %28;\n\t"
      "addc.cc.u32 %1, %15, %29;\n\t"
      "addc.cc.u32 %2, %16, %30;\n\t"
      "addc.cc.u32 %3, %17, %31;\n\t"
      "addc.cc.u32 %4, %18, %32;\n\t"
      "addc.cc.u32 %5, %19, %33;\n\t"
      "addc.cc.u32 %6, %20, %34;\n\t"
      "addc.cc.u32 %7, %21, %35;\n\t"
      "addc.cc.u32 %8, %22, %36;\n\t"
      "addc.cc.u32 %9, %23, %37;\n\t"
      "addc.cc.u32 %10, %24, %38;\n\t"
      "addc.cc.u32 %11, %25, %39;\n\t"
      "addc.cc.u32 %12, %26, %40;\n\t"
      "addc.u32 %13, %27, %41;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]), "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11]), "=r"(s[12]), "=r"(s[13])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(a[8]), "r"(a[9]), "r"(a[10]), "r"(a[11]), "r"(a[12]), "r"(a[13]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(b[8]), "r"(b[9]), "r"(b[10]), "r"(b[11]), "r"(b[12]), "r"(b[13]));
}
__device__ __forceinline__ void add_run16(uint32_t *s, const uint32_t *a, const uint32_t *b) {
  asm(
      "add.cc.u32 %0, %16, %32;\n\t"
      "addc.cc.u32 %1, %17, %33;\n\t"
      "addc.cc.u32 %2, %18, %34;\n\t"
      "addc.cc.u32 %3, %19, %35;\n\t"
      "addc.cc.u32 %4, %20, %36;\n\t"
      "addc.cc.u32 %5, %21, %37;\n\t"
      "addc.cc.u32 %6, %22, %38;\n\t"
      "addc.cc.u32 %7, %23, %39;\n\t"
      "addc.cc.u32 %8, %24, %40;\n\t"
      "addc.cc.u32 %9, %25, %41;\n\t"
      "addc.cc.u32 %10, %26, %42;\n\t"
      "addc.cc.u32 %11, %27, %43;\n\t"
      "addc.cc.u32 %12, %28, %44;\n\t"
      "addc.cc.u32 %13, %29, %45;\n\t"
      "addc.cc.u32 %14, %30, %46;\n\t"
      "addc.u32 %15, %31, %47;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]), "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11]), "=r"(s[12]), "=r"(s[13]), "=r"(s[14]), "=r"(s[15])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(a[8]), "r"(a[9]), "r"(a[10]), "r"(a[11]), "r"(a[12]), "r"(a[13]), "r"(a[14]), "r"(a[15]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(b[8]), "r"(b[9]), "r"(b[10]), "r"(b[11]), "r"(b[12]), "r"(b[13]), "r"(b[14]), "r"(b[15]));
}
__device__ __forceinline__ void add_run18(uint32_t *s, const uint32_t *a, const uint32_t *b) {
  asm("add.cc.u32 %0, %18, %36;\n\t"
      "addc.cc.u32 %1, %19, %37;\n\t"
      "addc.cc.u32 %2, %20, %38;\n\t"
      "addc.cc.u32 %3, %21, %39;\n\t"
      "addc.cc.u32 %4, %22, %40;\n\t"
      "addc.cc.u32 %5, %23, %41;\n\t"
      "addc.cc.u32 %6, %24, %42;\n\t"
      "addc.cc.u32 %7, %25, %43;\n\t"
      "addc.cc.u32 %8, %26, %44;\n\t"
      "addc.cc.u32 %9, %27, %45;\n\t"
      "addc.cc.u32 %10, %28, %46;\n\t"
      "addc.cc.u32 %11, %29, %47;\n\t"
      "addc.cc.u32 %12, %30, %48;\n\t"
      "addc.cc.u32 %13, %31, %49;\n\t"
      "addc.cc.u32 %14, %32, %50;\n\t"
      "addc.cc.u32 %15, %33, %51;\n\t"
      "addc.cc.u32 %16, %34, %52;\n\t"
      "addc.u32 %17, %35, %53;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]),
        "=r"(s[7]), "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11]), "=r"(s[12]), "=r"(s[13]),
        "=r"(s[14]), "=r"(s[15]), "=r"(s[16]), "=r"(s[17])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]),
        "r"(a[8]), "r"(a[9]), "r"(a[10]), "r"(a[11]), "r"(a[12]), "r"(a[13]), "r"(a[14]),
        "r"(a[15]), "r"(a[16]), "r"(a[17]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]),
        "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(b[8]), "r"(b[9]), "r"(b[10]), "r"(b[11]), "r"(b[12]),
        "r"(b[13]), "r"(b[14]), "r"(b[15]), "r"(b[16]), "r"(b[17]));
}
__device__ __forceinline__ void add_run20(uint32_t *s, const uint32_t *a, const uint32_t *b) {
  asm("add.cc.u32 %0, %20, %40;\n\t"
      "addc.cc.u32 %1, %21, %41;\n\t"
      "addc.cc.u32 %2, %22, %42;\n\t"
      "addc.cc.u32 %3, %23, %43;\n\t"
      "addc.cc.u32 %4, %24, %44;\n\t"
      "addc.cc.u32 %5, %25, %45;\n\t"
      "addc.cc.u32 %6, %26, %46;\n\t"
      "addc.cc.u32 %7, %27, %47;\n\t"
      "addc.cc.u32 %8, %28, %48;\n\t"
      "addc.cc.u32 %9, %29, %49;\n\t"
      "addc.cc.u32 %10, %30, %50;\n\t"
      "addc.cc.u32 %11, %31, %51;\n\t"
      "addc.cc.u32 %12, %32, %52;\n\t"
      "addc.cc.u32 %13, %33, %53;\n\t"
      "addc.cc.u32 %14, %34, %54;\n\t"
      "addc.cc.u32 %15, %35, %55;\n\t"
      "addc.cc.u32 %16, %36, %56;\n\t"
      "addc.cc.u32 %17, %37, %57;\n\t"
      "addc.cc.u32 %18, %38, %58;\n\t"
      "addc.u32 %19, %39, %59;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]),
        "=r"(s[7]), "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11]), "=r"(s[12]), "=r"(s[13]),
        "=r"(s[14]), "=r"(s[15]), "=r"(s[16]), "=r"(s[17]), "=r"(s[18]), "=r"(s[19])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]),
        "r"(a[8]), "r"(a[9]), "r"(a[10]), "r"(a[11]), "r"(a[12]), "r"(a[13]), "r"(a[14]),
        "r"(a[15]), "r"(a[16]), "r"(a[17]), "r"(a[18]), "r"(a[19]), "r"(b[0]), "r"(b[1]),
        "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(b[8]), "r"(b[9]),
        "r"(b[10]), "r"(b[11]), "r"(b[12]), "r"(b[13]), "r"(b[14]), "r"(b[15]), "r"(b[16]),
        "r"(b[17]), "r"(b[18]), "r"(b[19]));
}
__device__ __forceinline__ void add_run24(uint32_t *s, const uint32_t *a, const uint32_t *b) {
  asm("add.cc.u32 %0, %24, %48;\n\t"
      "addc.cc.u32 %1, %25, %49;\n\t"
      "addc.cc.u32 %2, %26, %50;\n\t"
      "addc.cc.u32 %3, %27, %51;\n\t"
      "addc.cc.u32 %4, %28, %52;\n\t"
      "addc.cc.u32 %5, %29, %53;\n\t"
      "addc.cc.u32 %6, %30, %54;\n\t"
      "addc.cc.u32 %7, %31, %55;\n\t"
      "addc.cc.u32 %8, %32, %56;\n\t"
      "addc.cc.u32 %9, %33, %57;\n\t"
      "addc.cc.u32 %10, %34, %58;\n\t"
      "addc.cc.u32 %11, %35, %59;\n\t"
      "addc.cc.u32 %12, %36, %60;\n\t"
      "addc.cc.u32 %13, %37, %61;\n\t"
      "addc.cc.u32 %14, %38, %62;\n\t"
      "addc.cc.u32 %15, %39, %63;\n\t"
      "addc.cc.u32 %16, %40, %64;\n\t"
      "addc.cc.u32 %17, %41, %65;\n\t"
      "addc.cc.u32 %18, %42, %66;\n\t"
      "addc.cc.u32 %19, %43, %67;\n\t"
      "addc.cc.u32 %20, %44, %68;\n\t"
      "addc.cc.u32 %21, %45, %69;\n\t"
      "addc.cc.u32 %22, %46, %70;\n\t"
      "addc.u32 %23, %47, %71;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]),
        "=r"(s[7]), "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11]), "=r"(s[12]), "=r"(s[13]),
        "=r"(s[14]), "=r"(s[15]), "=r"(s[16]), "=r"(s[17]), "=r"(s[18]), "=r"(s[19]), "=r"(s[20]),
        "=r"(s[21]), "=r"(s[22]), "=r"(s[23])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]),
        "r"(a[8]), "r"(a[9]), "r"(a[10]), "r"(a[11]), "r"(a[12]), "r"(a[13]), "r"(a[14]),
        "r"(a[15]), "r"(a[16]), "r"(a[17]), "r"(a[18]), "r"(a[19]), "r"(a[20]), "r"(a[21]),
        "r"(a[22]), "r"(a[23]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]),
        "r"(b[6]), "r"(b[7]), "r"(b[8]), "r"(b[9]), "r"(b[10]), "r"(b[11]), "r"(b[12]),
        "r"(b[13]), "r"(b[14]), "r"(b[15]), "r"(b[16]), "r"(b[17]), "r"(b[18]), "r"(b[19]),
        "r"(b[20]), "r"(b[21]), "r"(b[22]), "r"(b[23]));
}
__device__ __forceinline__ void add_run28(uint32_t *s, const uint32_t *a, const uint32_t *b) {
  asm("add.cc.u32 %0, %28, %56;\n\t"
      "addc.cc.u32 %1, %29, %57;\n\t"
      "addc.cc.u32 %2, %30, %58;\n\t"
      "addc.cc.u32 %3, %31, %59;\n\t"
      "addc.cc.u32 %4, %32, %60;\n\t"
      "addc.cc.u32 %5, %33, %61;\n\t"
      "addc.cc.u32 %6, %34, %62;\n\t"
      "addc.cc.u32 %7, %35, %63;\n\t"
      "addc.cc.u32 %8, %36, %64;\n\t"
      "addc.cc.u32 %9, %37, %65;\n\t"
      "addc.cc.u32 %10, %38, %66;\n\t"
      "addc.cc.u32 %11, %39, %67;\n\t"
      "addc.cc.u32 %12, %40, %68;\n\t"
      "addc.cc.u32 %13, %41, %69;\n\t"
      "addc.cc.u32 %14, %42, %70;\n\t"
      "addc.cc.u32 %15, %43, %71;\n\t"
      "addc.cc.u32 %16, %44, %72;\n\t"
      "addc.cc.u32 %17, %45, %73;\n\t"
      "addc.cc.u32 %18, %46, %74;\n\t"
      "addc.cc.u32 %19, %47, %75;\n\t"
      "addc.cc.u32 %20, %48, %76;\n\t"
      "addc.cc.u32 %21, %49, %77;\n\t"
      "addc.cc.u32 %22, %50, %78;\n\t"
      "addc.cc.u32 %23, %51, %79;\n\t"
      "addc.cc.u32 %24, %52, %80;\n\t"
      "addc.cc.u32 %25, %53, %81;\n\t"
      "addc.cc.u32 %26, %54, %82;\n\t"
      "addc.u32 %27, %55, %83;\n\t"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]),
        "=r"(s[7]), "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11]), "=r"(s[12]), "=r"(s[13]),
        "=r"(s[14]), "=r"(s[15]), "=r"(s[16]), "=r"(s[17]), "=r"(s[18]), "=r"(s[19]), "=r"(s[20]),
        "=r"(s[21]), "=r"(s[22]), "=r"(s[23]), "=r"(s[24]), "=r"(s[25]), "=r"(s[26]), "=r"(s[27])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]),
        "r"(a[8]), "r"(a[9]), "r"(a[10]), "r"(a[11]), "r"(a[12]), "r"(a[13]), "r"(a[14]),
        "r"(a[15]), "r"(a[16]), "r"(a[17]), "r"(a[18]), "r"(a[19]), "r"(a[20]), "r"(a[21]),
        "r"(a[22]), "r"(a[23]), "r"(a[24]), "r"(a[25]), "r"(a[26]), "r"(a[27]), "r"(b[0]),
        "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(b[8]),
        "r"(b[9]), "r"(b[10]), "r"(b[11]), "r"(b[12]), "r"(b[13]), "r"(b[14]), "r"(b[15]),
        "r"(b[16]), "r"(b[17]), "r"(b[18]), "r"(b[19]), "r"(b[20]), "r"(b[21]), "r"(b[22]),
        "r"(b[23]), "r"(b[24]), "r"(b[25]), "r"(b[26]), "r"(b[27]));
}
template <int N>
__device__ __forceinline__ void add_run(uint32_t *s, const uint32_t *a, const uint32_t *b) {
  static_assert(N >= 4 && N <= 28, "run length");
#define NGIA_RUN(K) \
  if constexpr (N == K) add_run##K(s, a, b);
  NGIA_RUN(4) NGIA_RUN(5) NGIA_RUN(6) NGIA_RUN(7) NGIA_RUN(8) NGIA_RUN(9) NGIA_RUN(10)
  NGIA_RUN(11) NGIA_RUN(12) NGIA_RUN(14) NGIA_RUN(16) NGIA_RUN(18) NGIA_RUN(20) NGIA_RUN(24) NGIA_RUN(28)
#undef NGIA_RUN
}

}  // namespace ngia
