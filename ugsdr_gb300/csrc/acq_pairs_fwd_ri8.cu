// Forward pair column kernel, ri8 samples.
#include "acq_pairs_fwd.cuh"

namespace ugsdr_gpu {
	void launch_fwd_cols_pair_ri8(const BatchedParams& p, int items, int sm_count, cudaStream_t stream) {
		launch_fwd_cols_pair<UGSDR_SAMPLES_RI8>(p, items, sm_count, stream);
	}
}
