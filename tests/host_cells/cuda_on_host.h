// cuda_on_host.h — the CUDA intrinsics that the per-cell headers use, as their
// IEEE operations on the CPU (compiled with -ffp-contract=off).
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <memory>
#include <vector>

#include <cuda_runtime.h>

#define __noinline__ __attribute__((noinline))  // after the standard headers, which use the word themselves

static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
static inline double __dadd_rn(double a, double b) { return a + b; }
static inline double __dsub_rn(double a, double b) { return a - b; }
static inline double __dmul_rn(double a, double b) { return a * b; }
static inline double __fma_rn(double a, double b, double c) { return fma(a, b, c); }
static inline float __double2float_rn(double d) { return (float)d; }
template <class A, class B>
static inline A bits_as(B b) {
  static_assert(sizeof(A) == sizeof(B), "sizes");
  A a;
  memcpy(&a, &b, sizeof a);
  return a;
}
static inline unsigned __float_as_uint(float f) { return bits_as<unsigned>(f); }
static inline int __float_as_int(float f) { return bits_as<int>(f); }
static inline float __uint_as_float(unsigned u) { return bits_as<float>(u); }
static inline int __double2hiint(double d) { return (int)(bits_as<uint64_t>(d) >> 32); }
static inline int __double2loint(double d) { return (int)bits_as<uint64_t>(d); }
static inline double __hiloint2double(int h, int l) {
  return bits_as<double>(((uint64_t)(unsigned)h << 32) | (unsigned)l);
}
static inline int __clz(int v) { return v == 0 ? 32 : __builtin_clz((unsigned)v); }
template <class T>
static inline T __ldg(const T* p) {
  return *p;
}
static inline unsigned atomicOr(unsigned* p, unsigned v) {
  const unsigned o = *p;
  *p |= v;
  return o;
}
using std::min;
