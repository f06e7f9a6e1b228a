// Host face of the product on pairs of CTAs (csrc/kernels/gemm_pair.cu).
#pragma once

#include "xpool/api.h"
#include "xpool/gemm_ws.cuh"

namespace xpool {
namespace gemm {

// Width of the activation tile (256 or 128) with which pairs take the call, 0 if the single-CTA kernel should.
int pair_width(const XpGemmArgs& a, int sms);
// `p` as for the single-CTA kernel, without its tile plan.
int pair_launch(const XpGemmArgs& a, Problem p, const CUtensorMap& tmap_w, int width, bool wide_epilogue, int sms);

}  // namespace gemm
}  // namespace xpool
