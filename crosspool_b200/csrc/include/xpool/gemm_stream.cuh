// Host face of the register-streaming product for few activation rows (csrc/kernels/gemm_stream.cu).
#pragma once

#include "xpool/api.h"

namespace xpool {
namespace gemm {

constexpr int kStreamMaxRows = 16;   // why there: see stream_applies

bool stream_applies(const XpGemmArgs& a);
int stream_launch(const XpGemmArgs& a);

}  // namespace gemm
}  // namespace xpool
