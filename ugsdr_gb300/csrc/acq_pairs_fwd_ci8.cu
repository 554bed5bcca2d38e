// Forward pair column kernel, ci8 samples.
#include "acq_pairs_fwd.cuh"

namespace ugsdr_gpu {
	void launch_fwd_cols_pair_ci8(const BatchedParams& p, int items, int sm_count, cudaStream_t stream) {
		launch_fwd_cols_pair<UGSDR_SAMPLES_CI8>(p, items, sm_count, stream);
	}
}
