// Forward pair row kernel.
#include "acq_pairs_fwd.cuh"

namespace ugsdr_gpu {
	void launch_fwd_rows_pair(const BatchedParams& p, int items, int sm_count, cudaStream_t stream) {
		const PairSplit& s = p.pair;
		const PairRows lay(s.b0, s.b1, s.rw, 0);
		const int smem = lay.cs_at + static_cast<int>(sizeof(float2)) * lay.tws * s.b0;
		const int parts = (p.n1 + s.rw - 1) / s.rw, per = pair_items(items, parts, sm_count);
		const int grid = (items + per - 1) / per * parts;
		auto kernel = max(p.pair.b0, p.pair.b1) <= 25 ? fwd_rows_pair_kernel<25> : fwd_rows_pair_kernel<32>;
		cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem);
		kernel<<<grid, pair_fwd_threads(s.rw * min(s.b0, s.b1)), smem, stream>>>(p, items, per);
	}
}
