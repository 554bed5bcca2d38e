// Pair column kernels, eight columns per CTA.
#include "acq_pairs_cols.cuh"

namespace ugsdr_gpu {
	void launch_inv_cols_pair8(const BatchedParams& p, cudaStream_t stream) { launch_inv_cols_pair_width<8>(p, stream); }
}
