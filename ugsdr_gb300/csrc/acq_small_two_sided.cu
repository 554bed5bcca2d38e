// Single-CTA inverse kernel of lone CTAs, two-sided spectra.
#include "acq_small.cuh"

namespace ugsdr_gpu {
	void launch_inv_small_two_sided(const AcqParams& p, const SmallPlan& plan, int rows, cudaStream_t stream) {
		launch_inv_small(acq_inv_small_kernel<32, false, false>, p, plan, rows, stream);
	}
}
