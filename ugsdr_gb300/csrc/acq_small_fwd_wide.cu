// Single-CTA forward kernels, 16-bit and float samples.
#include "acq_small.cuh"

namespace ugsdr_gpu {
	void launch_fwd_small_wide(const AcqParams& p, const SmallPlan& plan, int sample_type, int items, cudaStream_t stream) {
		launch_fwd_small(sample_type == UGSDR_SAMPLES_CI16 ? acq_fwd_small_kernel<UGSDR_SAMPLES_CI16> : acq_fwd_small_kernel<UGSDR_SAMPLES_CF32>,
			p, plan, items, stream);
	}
}
