// Row kernels of the pair splits, one per register class and spectrum mode.
#include "internal.hpp"
#include "acq_pairs.cuh"

#include <algorithm>

namespace ugsdr_gpu {
	void launch_inv_rows_pair(const BatchedParams& p, bool half, cudaStream_t stream) {
		const PairSplit& s = p.pair;
		const PairRows lay(s.b0, s.b1, s.rw, half ? 1 : 0);
		const int grid = p.rows * ((p.n1 + s.rw - 1) / s.rw);
		auto launch = [&](auto kernel) {
			UG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem));
			kernel<<<grid, s.row_threads, lay.bytes, stream>>>(p);
			UG_CUDA(cudaGetLastError());
		};
		if (std::max(s.b0, s.b1) <= 25)
			half ? launch(inv_rows_pair_kernel<25, true>) : launch(inv_rows_pair_kernel<25, false>);
		else
			half ? launch(inv_rows_pair_kernel<32, true>) : launch(inv_rows_pair_kernel<32, false>);
	}
}
