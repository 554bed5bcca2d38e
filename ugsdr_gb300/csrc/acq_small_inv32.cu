// Single-CTA inverse kernels, radices up to 32, and two-sided spectra.
#include "acq_small.cuh"

namespace ugsdr_gpu {
	void launch_inv_small32(const AcqParams& p, const SmallPlan& plan, int rows, cudaStream_t stream) {
		launch_inv_small(p.one_sided ? acq_inv_small_kernel<32, true> : acq_inv_small_kernel<32, false>, p, plan, rows,
			small_inv_bytes(plan), stream);
	}
}
