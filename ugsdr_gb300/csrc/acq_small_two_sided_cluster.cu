// Single-CTA inverse kernel of clusters, two-sided spectra.
#include "acq_small.cuh"

namespace ugsdr_gpu {
	void launch_inv_small_two_sided_cluster(const AcqParams& p, const SmallPlan& plan, int rows, cudaStream_t stream) {
		launch_inv_small(acq_inv_small_kernel<32, false, true>, p, plan, rows, stream);
	}
}
