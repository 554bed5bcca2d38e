// Single-CTA inverse kernels of lone CTAs, one-sided spectra, radices up to
// 25; blocks of 4,000 points.
#include "acq_small.cuh"

namespace ugsdr_gpu {
	void launch_inv_small25_cluster(const AcqParams& p, const SmallPlan& plan, int rows, cudaStream_t stream);

	void launch_inv_small25(const AcqParams& p, const SmallPlan& plan, int rows, cudaStream_t stream) {
		if (plan.split > 1)
			launch_inv_small25_cluster(p, plan, rows, stream);
		else
			launch_inv_small(acq_inv_small_kernel<25, true, false>, p, plan, rows, stream);
	}

	template <bool HALF>
	static void launch_4000(const AcqParams& p, const SmallPlan& plan, int rows, cudaStream_t stream) {
		if (plan.split > 1)
			launch_inv_small(acq_inv_three_kernel<25, 10, 16, HALF, true>, p, plan, rows, stream);
		else
			launch_inv_small(acq_inv_three_kernel<25, 10, 16, HALF, false>, p, plan, rows, stream);
	}
	void launch_inv_4000(const AcqParams& p, const SmallPlan& plan, bool half, int rows, cudaStream_t stream) {
		(half ? launch_4000<true> : launch_4000<false>)(p, plan, rows, stream);
	}
}
