// Launch of the pair column kernels of one tile width (compiled per width).
#pragma once

#include "internal.hpp"
#include "acq_pairs.cuh"

#include <algorithm>

namespace ugsdr_gpu {
	template <int CW>
	void launch_inv_cols_pair_width(const BatchedParams& p, cudaStream_t stream) {
		const PairSplit& s = p.pair;
		const PairCols lay(s.a0, s.a1, CW);
		const int grid = p.rows * (p.n2p / CW);
		auto launch = [&](auto kernel) {
			UG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem));
			kernel<<<grid, s.col_threads, lay.bytes, stream>>>(p);
			UG_CUDA(cudaGetLastError());
		};
		if (std::max(s.a0, s.a1) <= 25)
			p.base.stat ? launch(inv_cols_pair_kernel<CW, 25, 1>) : launch(inv_cols_pair_kernel<CW, 25, 0>);
		else
			p.base.stat ? launch(inv_cols_pair_kernel<CW, 32, 1>) : launch(inv_cols_pair_kernel<CW, 32, 0>);
	}
}
