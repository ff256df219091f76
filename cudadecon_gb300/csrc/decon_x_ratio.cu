// Inverse x pass of the first convolution: C2R, RL ratio, and R2C of the
// ratio for the second convolution.
#include "decon_x_kernels.cuh"
#include "x_gen_dispatch.h"

namespace cdx {

int launch_x_inv_ratio_fwd(const Geom& g, const FftLen& fx, float2* S, const float* raw,
                           const float* mean, float eps, cudaStream_t st) {
  if (g.pair) {
    bool done = false;
    const PairGeom up = pair_geom(g);
    const int rc = past_l2(g) ? pxgen_ratio(pair_geom_down(g), fx.d_pair, last_slice(up, S),
                                            last_slice_real(up, raw), mean, eps, st, &done)
                              : pxgen_ratio(up, fx.d_pair, S, raw, mean, eps, st, &done);
    if (done || rc) return rc;
  }
  if (fx.has_tc && dft_form() == 1)
    return launch_xtc_ratio(g, fx.tc, S, raw, eps, fx.tc.d_err, st);
  const int P = x_pairs(g.nx);
  return x_ratio_go<GenericRunner>(g, fx.dev, S, raw, eps, P, threads_for((long long)P * g.nx), st);
}

}  // namespace cdx
