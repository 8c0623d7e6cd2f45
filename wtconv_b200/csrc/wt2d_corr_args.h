// Kernel argument of the parameter-gradient launches (see wt2d_corr.cuh).
#pragma once

namespace wt {

struct CorrArgs {
  float* stats;            // (1 + 4 L, K*K + 1, C), zeroed before the first launch
  int C, set0;             // set of sub-band 0 of the (first) level
  float* llx;              // (B, C, h1, w1) low-pass planes for the next level, may be null
  float* llg;
  int nsplit;              // CTAs per channel group (corr) or per channel (deep)
  long long gs[4];         // strides of the gradient (n, c, row, col)
  int gvec;                // pixels of a gradient row per access
};

}  // namespace wt
