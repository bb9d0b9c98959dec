// gradient.cuh — the size of vi_gradient's workspace, for the gradient itself
// and for the server's admission.
#pragma once

#include <cstddef>

#include "common.cuh"

namespace vb {

// Bytes for nslots state slots (checkpoints, segment and adjoint), the adjoint
// sweep's scratch, `copied` medium planes and the traces.
size_t gradient_bytes(const vi_config &c, long long nslots, int nt, int nrec, int copied);

}  // namespace vb
