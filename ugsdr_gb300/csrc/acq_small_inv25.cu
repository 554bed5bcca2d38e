// Single-CTA inverse kernel, one-sided spectra, radices up to 25.
#include "acq_small.cuh"

namespace ugsdr_gpu {
	void launch_inv_small25(const AcqParams& p, const SmallPlan& plan, int rows, cudaStream_t stream) {
		launch_inv_small(acq_inv_small_kernel<25, true>, p, plan, rows, small_inv_bytes(plan), stream);
	}

	void launch_inv_4000(const AcqParams& p, const SmallPlan& plan, bool half, int rows, cudaStream_t stream) {
		if (half)
			launch_inv_small(acq_inv_three_kernel<25, 10, 16, true>, p, plan, rows, small_inv_bytes(plan), stream);
		else
			launch_inv_small(acq_inv_three_kernel<25, 10, 16, false>, p, plan, rows, small_inv_bytes(plan), stream);
	}
}
