// Declarations of the FP64-accurate tensor-core list-1 path.
#pragma once

#include <cuda_fp16.h>

namespace vl1 {

// Operand geometry of one plan: source points padded to whole units of 16,
// output columns (interleaved real / imaginary parts for complex tables)
// padded to whole chunks of nch (16, 32 or 64 columns per CTA).
struct WideGeom {
  int kp, np, nch;
};

// source points of a work item of several keys: its digit sums of weights
// 2^-56 .. 2^-72 must fit an int32, (2^16 + 7 * 2^14) K < 2^31
constexpr int kItemPoints = 8192;

struct WidePlan {
  WideGeom geom;
  __half *adig;    // table digits (nullptr until first needed)
  int *key_exp;    // exponent per (table level, case) block
};

}  // namespace vl1
