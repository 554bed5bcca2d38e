// Single-CTA forward kernels, 8-bit samples.
#include "acq_small.cuh"

namespace ugsdr_gpu {
	void launch_fwd_small_8bit(const AcqParams& p, const SmallPlan& plan, int sample_type, int items, cudaStream_t stream) {
		launch_fwd_small(sample_type == UGSDR_SAMPLES_CI8 ? acq_fwd_small_kernel<UGSDR_SAMPLES_CI8> : acq_fwd_small_kernel<UGSDR_SAMPLES_RI8>,
			p, plan, items, stream);
	}
}
