// split.cuh -- how a block of four warps splits its elements' work, for the adjoint
// split kernel (adjoint_split.cuh): 32 elements per block, one per lane; the warp
// index r is the part of the element's work that thread does, so every table
// operand is the same for a warp's 32 lanes.
#pragma once
#include <type_traits>

#include "element.cuh"

namespace nzb {

constexpr int SPLIT_T = 4;   // threads (warps) per element
constexpr int SPLIT_EB = 32; // elements per block, one per lane

struct SplitRanges {
  int first[SPLIT_T];
  int count[SPLIT_T];
};

template <int K, int P>
struct SplitPlan {
  using S = Shape<K, P>;
  // Costs in instruction units: a volume point (interpolation, Euler flux,
  // contravariant flux, stores; the vertex Jacobian for general geometry) and
  // a face (two traces, the flux and the lift at each face point).
  static constexpr int VCOST = 4 * S::NP + 40 + (K == 1 ? 16 : 0);
  static constexpr int FCOST = S::NQF * (12 * S::NE + 150);

  // Phase A1: a warp without a face (triangles: warp 3) evaluates the last
  // LATE volume points while the others evaluate their faces' fluxes; their
  // FV slots must lie beyond the NF * NE * 4 slots that stage the neighbours'
  // edge coefficients.  The rest go to phase A2, evenly.
  static constexpr int late() {
    if (S::NF >= SPLIT_T) return 0;
    const int first_free = (S::NF * S::NE * 4 + 7) / 8;  // first point whose FV slots are free
    int n = FCOST / VCOST;
    if (n > S::NQV - first_free) n = S::NQV - first_free;
    return n < 0 ? 0 : n;
  }
  static constexpr int LATE = late();

  // An even split of n items over the warps.
  static constexpr SplitRanges even(int n) {
    SplitRanges R{};
    int f = 0;
    for (int r = 0; r < SPLIT_T; ++r) {
      R.count[r] = n / SPLIT_T + (r < n % SPLIT_T ? 1 : 0);
      R.first[r] = f;
      f += R.count[r];
    }
    return R;
  }
};

// Calls fn(integral_constant<int, r>) for the runtime warp index r (uniform
// across a warp), so each warp runs code compiled for its own share.
template <class F>
__device__ __forceinline__ void for_part(int r, F&& fn) {
  switch (r) {
    case 0: fn(std::integral_constant<int, 0>{}); break;
    case 1: fn(std::integral_constant<int, 1>{}); break;
    case 2: fn(std::integral_constant<int, 2>{}); break;
    default: fn(std::integral_constant<int, 3>{}); break;
  }
}

}  // namespace nzb
