// The order of a block's columns by their norms. Plain C++: host code too.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define KG_HOST_DEVICE __host__ __device__
#else
#define KG_HOST_DEVICE
#endif

namespace kg {

// Whether column a of norm na comes before column b of norm nb: by descending norm, NaNs last,
// ties to the lower column. A strict total order whatever the norms hold, so that counting the
// columns before each one gives every place once (with "not smaller" for "equal", a NaN ties
// with every norm, two columns get one place, and another stays unwritten).
KG_HOST_DEVICE inline bool column_before(double na, uint32_t a, double nb, uint32_t b) {
  const bool nan_a = na != na, nan_b = nb != nb;
  if (nan_a || nan_b) return nan_a == nan_b ? a < b : nan_b;
  return na > nb || (na == nb && a < b);
}

}  // namespace kg
