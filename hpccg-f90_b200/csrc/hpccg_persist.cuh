// hpccg_persist.cuh -- the one-kernel CG of small stored systems (hpccg_persist.cu).
#pragma once
#include "hpccg_internal.cuh"

namespace hpccg {

// Rows up to which the one-kernel form runs (it wins at 1.0 million, loses at 2.1).
constexpr int kPersistRows = 1 << 20;
constexpr int kPersistBoxRows = 460000;  // where the graph's rows are box walks

// What a thread reports when its part of the kernel ends: `ok` = every wait of its block
// came, `status` = how the solve ended.  HPCCG_OK is what the word starts as and is never
// stored, and a wait that ran out stands over any other status, so the word does not
// depend on the order of the blocks.  Word: set(v), and set_if_ok(v) where it is HPCCG_OK.
template <class Word>
__host__ __device__ inline void persist_report(Word &&word, bool lead, bool ok, int status) {
  if (!ok)
    word.set(HPCCG_ERR_TIMEOUT);
  else if (lead && status != HPCCG_OK)
    word.set_if_ok(status);
}

// Whether the context's CG runs in one kernel (its row kernel settled as row patterns).
bool cg_persist_fits(const hpccg_ctx *c);
// Launches it on the context's stream: b, x, state and history as the graph's kernels take
// them.  *launched = false where its second p finds no memory or its blocks cannot all
// be resident: nothing has run, and the graph takes the solve.
int cg_persist(hpccg_ctx *c, bool *launched);

}  // namespace hpccg
