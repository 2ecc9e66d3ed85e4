// Stand-ins for the CUDA keywords and intrinsics that the FP64 device headers use, so that
// a host compiler (-ffp-contract=off) evaluates the same operations.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <cuda_runtime.h>

static inline double __dmul_rn(double a, double b) { return a * b; }
static inline double __dadd_rn(double a, double b) { return a + b; }
static inline double __dsub_rn(double a, double b) { return a - b; }
static inline double __fma_rn(double a, double b, double c) { return fma(a, b, c); }
static inline int64_t __double_as_longlong(double a) { int64_t v; memcpy(&v, &a, 8); return v; }
static inline double __longlong_as_double(int64_t v) { double a; memcpy(&a, &v, 8); return a; }
static inline int __double2hiint(double a) { return (int)((uint64_t)__double_as_longlong(a) >> 32); }
static inline int __double2loint(double a) { return (int)(uint32_t)__double_as_longlong(a); }
static inline double __hiloint2double(int hi, int lo) {
  return __longlong_as_double((int64_t)(((uint64_t)(uint32_t)hi << 32) | (uint32_t)lo));
}
static inline unsigned max(unsigned a, unsigned b) { return a > b ? a : b; }
#ifndef __noinline__
#define __noinline__
#endif
