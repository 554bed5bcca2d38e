// Forward pair column kernel, cf32 samples.
#include "acq_pairs_fwd.cuh"

namespace ugsdr_gpu {
	void launch_fwd_cols_pair_cf32(const BatchedParams& p, int items, int sm_count, cudaStream_t stream) {
		launch_fwd_cols_pair<UGSDR_SAMPLES_CF32>(p, items, sm_count, stream);
	}
}
