// Tensor-core form of the DFT for fluxes tabulated per coarse plane (dft_tc.cuh):
// the rows lie in one plane each and carry its flux.
#include "dft_tc.cuh"

namespace obit {

namespace {

template <int MA, int NJ, int T>
TcFn pick_shape(int kind, bool crossPt, int mixed) {
  constexpr int S = kExSpec | kExTab, B = kExBoth | kExTab;
  if (kind == kPointTSpec)
    return crossPt ? dft_tc_kernel<MA, NJ, T, S, true, 0> : dft_tc_kernel<MA, NJ, T, S, false, 0>;
  if (mixed) return crossPt ? dft_tc_kernel<MA, NJ, T, B, true, 2> : dft_tc_kernel<MA, NJ, T, B, true, 1>;
  return dft_tc_kernel<MA, NJ, T, B, true, 0>;
}

}  // namespace

TcFn tc_pick_tab(const TcPlan& pl) {
  if (pl.MA == 2 && pl.NJ == 2 && pl.T == 2) return pick_shape<2, 2, 2>(pl.kind, pl.crossPt, pl.mixed);
  if (pl.MA == 2 && pl.NJ == 2 && pl.T == 1) return pick_shape<2, 2, 1>(pl.kind, pl.crossPt, pl.mixed);
  if (pl.MA == 1 && pl.NJ == 2 && pl.T == 1) return pick_shape<1, 2, 1>(pl.kind, pl.crossPt, pl.mixed);
  if (pl.MA == 1 && pl.NJ == 1 && pl.T == 1) return pick_shape<1, 1, 1>(pl.kind, pl.crossPt, pl.mixed);
  return nullptr;
}

}  // namespace obit
