// rbk_sample_scan.h -- what one thread of sample_scan_kernel does with its run
// of values [lo, hi), in a form that the host compiles too.
//
// The scanned values have to be exact in two ways whatever their rounding: they
// never decrease, and a value of zero leaves the one before it as it is (a chunk
// of zero weight would be drawn otherwise).  The lanes of a scan add in different
// orders, so the ends of the runs are made so afterwards: each is the largest of
// the ends up to it, those of runs of zeros left out.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define RBK_HD __host__ __device__ __forceinline__
#else
#define RBK_HD inline
#endif

namespace rbk {

// The run's sum; *last: one past its last value that is not zero (lo if all are).
RBK_HD double scan_run(const double* v, uint64_t lo, uint64_t hi, uint64_t* last)
{
  double run = 0.0;
  *last = lo;
#ifdef __CUDACC__
#pragma unroll 8
#endif
  for (uint64_t i = lo; i < hi; ++i) {
    const double x = v[i];
    run += x;
    if (x != 0.0) *last = i + 1;
  }
  return run;
}

// The later of two ends of runs, a first: the larger, NaN if either is.
RBK_HD double scan_later(double a, double b) { return b != b || a <= b ? b : a; }

// Writes the run's scanned values: from `before`, the end of the runs before it,
// to its own end.
RBK_HD void scan_write(double* v, uint64_t lo, uint64_t hi, uint64_t last, double before, double end)
{
  double acc = before;
#ifdef __CUDACC__
#pragma unroll 8
#endif
  for (uint64_t i = lo; i < hi; ++i) {
    acc += v[i];
    v[i] = i + 1 >= last ? end : (acc < end ? acc : end);
  }
}

}  // namespace rbk
