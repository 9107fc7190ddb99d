// Launchers of the river CFR kernel (river_cfr.cu).
#pragma once
#include <cuda_runtime.h>

#include <atomic>

#include "layout.h"

namespace prb {

enum { kModeCFR = 0, kModeBR = 1 };

// Device memory of split passes (few roots: see launch_river), taken and given back in stream order, so
// that passes on several streams and threads do not share it. It comes from one pool per device, which
// keeps at most kMaxScratch bytes between passes, whatever the number of builders, and goes with the last
// of those that drew on it. No memory is handed out while the stream is capturing: those passes run
// unsplit.
struct RiverScratch {
    static constexpr size_t kMaxScratch = (size_t)256 << 20;
    int device = 0;
    std::atomic<int> splits{0};  // CTAs per root of the last pass, 0 before the first
    std::atomic<cudaMemPool_t> pool{nullptr};
    bool attach();
    void *take(size_t bytes, cudaStream_t stream);
    void give_back(void *p, cudaStream_t stream);
    ~RiverScratch();
};

// Shared memory per CTA for a pass; max_groups / max_card_groups are the largest tie-group
// counts over the flop's boards.
size_t river_smem_bytes(int mode, int fp64, int max_groups, int max_card_groups);

// One pass over n river subgames: CFR (regret update of `updater`'s edges, results are
// counterfactual values) or best response (results are best-response values, regrets
// read only). ranges / results: n rows of kRangeStride values; regrets: n * 26 * 256.
// In CFR mode with own_ranges (the updater's ranges, same rows) and avg_sums (n * 26 * 256)
// the pass also accumulates average-strategy sums. With `scratch`, passes over few roots spread each
// root's river cards over several CTAs (same values, bucket sums and regrets, bit for bit).
cudaError_t launch_river(int mode, const SubgameDesc *desc, int n, const float *ranges, float *results,
                         float *regrets, const BoardPack *packs, unsigned long long flop, int updater,
                         int max_groups, int max_card_groups, const float *own_ranges, float *avg_sums,
                         RiverScratch *scratch, cudaStream_t stream);

// Best response in double precision.
cudaError_t launch_river_br64(const SubgameDesc *desc, int n, const double *ranges, double *results,
                              float *regrets, const BoardPack *packs, unsigned long long flop, int updater,
                              int max_groups, int max_card_groups, RiverScratch *scratch, cudaStream_t stream);

}  // namespace prb
