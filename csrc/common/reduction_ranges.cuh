// Several products of one shape side by side, each over a range of the reduction index of its own: product g reduces over [offsets[g], offsets[g + 1]) (experts' weight
// gradients), or over `per` indices each where there are no offsets (the parts of a split reduction), and writes D + g * stride.
#pragma once

namespace dewb {

struct Ranges {
  const int* offsets;
  int per, count;
  long long stride;
};

struct Range {
  int k0, k_iters;        // the first index, and steps of `step`
  long long d_off;
};

__device__ __forceinline__ Range range_of(const Ranges& r, int g, int K, int step) {
  const int k0 = r.offsets != nullptr ? r.offsets[g] : g * r.per;
  const int end = r.offsets != nullptr ? r.offsets[g + 1] : min(K, k0 + r.per);
  return {k0, (end - k0 + step - 1) / step, g * r.stride};
}

}  // namespace dewb
