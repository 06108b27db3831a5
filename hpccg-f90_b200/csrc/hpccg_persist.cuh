// hpccg_persist.cuh -- the one-kernel CG of small stored systems (hpccg_persist.cu).
#pragma once
#include "hpccg_internal.cuh"

namespace hpccg {

// Rows up to which the one-kernel form runs (it wins at 1.0 million, loses at 2.1).
constexpr int kPersistRows = 1 << 20;
constexpr int kPersistBoxRows = 460000;  // where the graph's rows are box walks

// Whether the context's CG runs in one kernel (its row kernel settled as row patterns).
bool cg_persist_fits(const hpccg_ctx *c);
// Launches it on the context's stream: b, x, state and history as the graph's kernels take them.
int cg_persist(hpccg_ctx *c);

}  // namespace hpccg
