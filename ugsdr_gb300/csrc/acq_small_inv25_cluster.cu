// Single-CTA inverse kernel of clusters, one-sided spectra, radices up to 25.
#include "acq_small.cuh"

namespace ugsdr_gpu {
	void launch_inv_small25_cluster(const AcqParams& p, const SmallPlan& plan, int rows, cudaStream_t stream) {
		launch_inv_small(acq_inv_small_kernel<25, true, true>, p, plan, rows, stream);
	}
}
