// Pair column kernels, four columns per CTA, and the choice of the width.
#include "acq_pairs_cols.cuh"

namespace ugsdr_gpu {
	void launch_inv_cols_pair8(const BatchedParams& p, cudaStream_t stream);

	void launch_inv_cols_pair(const BatchedParams& p, cudaStream_t stream) {
		if (p.pair.cw_shift == 3)
			launch_inv_cols_pair8(p, stream);
		else
			launch_inv_cols_pair_width<4>(p, stream);
	}
}
