// Single-CTA inverse kernel of lone CTAs, one-sided spectra, radices up to 32,
// and the choice among those of that class and the two-sided ones.
#include "acq_small.cuh"

namespace ugsdr_gpu {
	void launch_inv_small32_cluster(const AcqParams& p, const SmallPlan& plan, int rows, cudaStream_t stream);
	void launch_inv_small_two_sided(const AcqParams& p, const SmallPlan& plan, int rows, cudaStream_t stream);
	void launch_inv_small_two_sided_cluster(const AcqParams& p, const SmallPlan& plan, int rows, cudaStream_t stream);

	void launch_inv_small32(const AcqParams& p, const SmallPlan& plan, int rows, cudaStream_t stream) {
		if (!p.one_sided)
			(plan.split > 1 ? launch_inv_small_two_sided_cluster : launch_inv_small_two_sided)(p, plan, rows, stream);
		else if (plan.split > 1)
			launch_inv_small32_cluster(p, plan, rows, stream);
		else
			launch_inv_small(acq_inv_small_kernel<32, true, false>, p, plan, rows, stream);
	}
}
