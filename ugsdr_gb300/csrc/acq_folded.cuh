// Folded searches (ReshapeAndSum of GetOneMsPeak, fse.hpp:201-220) on
// transforms of the folded length.
//
// With N = F M, the fold of the correlation y over its F segments is an
// M-point inverse transform of every F-th bin:
//   sum_f y[i + f M] = (1 / M) sum_{q < M} X[q F] C[q F] exp(2 pi i q i / M),
// and X[q F] is the M-point transform of the folded input
//   x'[i] = sum_f x[i + f M],
// so the search mixes the whole block, folds it, and runs M-point transforms:
// F times fewer points in both directions, no atomics, no finishing pass.
// One-sided spectra stay one-sided: q F > N / 2 exactly when q > M / 2.
// A replica that repeats every M samples has C[k] = 0 off the multiples of F,
// so y itself repeats and the folded magnitudes are F equal values.
#pragma once

#include "acq_kernels.cuh"

namespace ugsdr_gpu {

	constexpr int kFoldCodes = 32;  // codes per launch (their pointers travel as kernel parameters)
	constexpr int kFoldBins = 4;    // Doppler bins per thread of the mix

	struct FoldCodesParams {
		const float2* in[kFoldCodes];
		int m, folds;
		int n1_in, n1_out;  // layout: natural (0) or k1-major, X_T[k1][k2] = X[k1 + n1 k2]
		float scale;
		float2* out;        // [code][m]
	};

	// out[q] = scale C[q F]; grid: ceil(m / 256) x codes.  A gather of n_codes
	// x M values per job (2.4 MB for 32 codes of 9,548 points), 3 us.
	static __global__ void __launch_bounds__(256) fold_codes_kernel(const __grid_constant__ FoldCodesParams p) {
		const int e = blockIdx.x * blockDim.x + threadIdx.x;
		if (e >= p.m)
			return;
		int q = e;
		if (p.n1_out) {
			const int n2 = p.m / p.n1_out;
			q = e / n2 + p.n1_out * (e % n2);
		}
		int k = q * p.folds;
		if (p.n1_in) {
			const int n2 = p.m * p.folds / p.n1_in;
			k = (k % p.n1_in) * n2 + k / p.n1_in;
		}
		const float2 v = __ldg(p.in[blockIdx.y] + k);
		p.out[static_cast<size_t>(blockIdx.y) * p.m + e] = c2(v.x * p.scale, v.y * p.scale);
	}

	// out[d][blk][i] = sum_f mix(x[blk F m + f m + i]) for bins d_base + d, d <
	// nd, p.n = m.  Each thread takes one i for kFoldBins bins: the F samples
	// are loaded, converted and translated once for all of them, the NCO
	// holders step by constants.  Issue-bound (two table reads and six flops per
	// sample and bin).  grid: ceil(m / 256) * K * ceil(nd / kFoldBins).
	template <int ST>
	__global__ void __launch_bounds__(256) fold_mix_kernel(const __grid_constant__ AcqParams p, int folds, int nd, float2* out) {
		__shared__ float lut[80];
		for (int i = threadIdx.x; i < 80; i += blockDim.x)
			lut[i] = p.lut[i];
		__syncthreads();
		const int m = p.n;
		const int parts = (m + 255) / 256;
		const int item = blockIdx.x / parts;  // (bin group, block)
		const int i = (blockIdx.x - item * parts) * 256 + threadIdx.x;
		if (i >= m)
			return;
		const int group = item / p.k_blocks;
		const int blk = item - group * p.k_blocks, d0 = group * kFoldBins;
		uint64_t g = static_cast<uint64_t>(blk) * folds * m + i;
		const uint32_t gl = static_cast<uint32_t>(g), mu = static_cast<uint32_t>(m);
		uint32_t hf = gl * p.fe_adder;
		const uint32_t dhf = mu * p.fe_adder;
		uint32_t h[kFoldBins], dh[kFoldBins];
		float2 acc[kFoldBins];
#pragma unroll
		for (int u = 0; u < kFoldBins; ++u) {
			const uint32_t adder = d0 + u < nd ? p.adders[p.d_base + d0 + u] : 0u;
			h[u] = p.phase0 + gl * adder;
			dh[u] = mu * adder;
			acc[u] = c2(0.f, 0.f);
		}
#pragma unroll 4
		for (int f = 0; f < folds; ++f) {
			float2 v = load_sample<ST>(p.samples, g);
			if (p.fe_on)
				v = table_mix_holder(v, hf, lut);
#pragma unroll
			for (int u = 0; u < kFoldBins; ++u) {
				acc[u] = cadd(acc[u], table_mix_holder(v, h[u], lut));
				h[u] += dh[u];
			}
			hf += dhf;
			g += m;
		}
#pragma unroll
		for (int u = 0; u < kFoldBins; ++u)
			if (d0 + u < nd)
				out[(static_cast<size_t>(d0 + u) * p.k_blocks + blk) * m + i] = acc[u];
	}
}
