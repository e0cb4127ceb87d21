// Device memory of a GEMM that divides the tiles of its last waves between CTA pairs: partial sums and start counter / flags.
#pragma once
#include <stdint.h>

namespace sb200 {

// Asked for by the launcher only when the product is in a form that may divide tiles.
struct SplitSpace {
  // partial: gemm_split_floats() floats; sync: gemm_split_sync_ints() ints that are zero when the kernel starts and used by no
  // other launch.  False: none to be had (the product runs undivided).
  virtual bool get(float** partial, int** sync) = 0;
  virtual ~SplitSpace() = default;
};
int64_t gemm_split_floats();
int gemm_split_sync_ints();

}  // namespace sb200
