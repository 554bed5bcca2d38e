// Forward four-step kernels of the pair splits (acq_pairs.cuh): signal items
// and the per-op DFT's whole signal, one item (code spectra keep
// fwd_cols_kernel / fwd_rows_kernel).
//
// fwd_cols_pair_kernel: pass 0 loads, converts and mixes its samples straight
// into the butterfly's registers (the row index steps by a1, the NCO holders
// by constants), pass 1 applies the inter-step twiddle and stores; one tile,
// two barriers per item.  fwd_rows_pair_kernel: pass 0 reads its rows from
// global memory, pass 1 writes the spectrum over them (the part the inverse
// gather reads).  A CTA takes up to four (Doppler, block) items of its columns
// or rows, so that its tables and twiddle seeds are built once; fewer when the
// items are too few to fill the SMs (36 items of 50,000 points: 128 -> 121 us a
// search).  Splits of radices up to 25 run at 80 registers a thread (24 warps
// per SM, not 15): 656 items of 50,000 points and 16 x 41 x 40 more, columns
// 5.4 -> 4.8 ms, rows 4.6 -> 3.9.
// Bound: issue (72 % in the columns) and the latency of the loads.
#pragma once

#include "acq_pairs.cuh"

namespace ugsdr_gpu {

	// launches, one file per kernel (acq_pairs_fwd_*.cu)
	void launch_fwd_cols_pair_cf32(const BatchedParams& p, int items, int sm_count, cudaStream_t stream);
	void launch_fwd_cols_pair_ci8(const BatchedParams& p, int items, int sm_count, cudaStream_t stream);
	void launch_fwd_cols_pair_ci16(const BatchedParams& p, int items, int sm_count, cudaStream_t stream);
	void launch_fwd_cols_pair_ri8(const BatchedParams& p, int items, int sm_count, cudaStream_t stream);
	void launch_fwd_rows_pair(const BatchedParams& p, int items, int sm_count, cudaStream_t stream);

	// items per CTA: four, or as many as leave every SM eight CTAs
	inline int pair_items(int items, int parts, int sm_count) {
		const long long ctas = static_cast<long long>(items) * parts;
		return static_cast<int>(ctas >= 32LL * sm_count ? 4 : ctas >= 16LL * sm_count ? 2 : 1);
	}

	inline int pair_fwd_threads(int butterflies) {
		return butterflies >= kPairThreads ? kPairThreads : butterflies <= 32 ? 32 : (butterflies + 31) / 32 * 32;
	}

	// grid: ceil(items / per) * ceil(N2 / 8)
	template <int ST, int MAXR>
	__global__ void __launch_bounds__(kPairThreads, kPairMinBlocks<MAXR>) fwd_cols_pair_kernel(const __grid_constant__ BatchedParams p, int items,
		int per) {
		extern __shared__ __align__(16) unsigned char raw[];
		__shared__ float lut[80];
		constexpr int CW = 8;
		const AcqParams& q = p.base;
		const int a0 = p.pair.a0, a1 = p.pair.a1, n2 = p.n2;
		const PairCols lay(a0, a1, CW);
		float2* const work = reinterpret_cast<float2*>(raw);
		float2* const tw = reinterpret_cast<float2*>(raw + lay.tw_at);
		float2* const seeds = reinterpret_cast<float2*>(raw + lay.acc_at);  // [column][a0 + 1 + kTwiddleJumps]
		for (int i = threadIdx.x; i < 80; i += blockDim.x)
			lut[i] = q.lut[i];
		const int chunks = (n2 + CW - 1) / CW;
		const int group = blockIdx.x / chunks;
		const int c0 = (blockIdx.x - group * chunks) * CW;
		const uint32_t n = static_cast<uint32_t>(q.n);
		for (int e = threadIdx.x; e < a0 * (a1 - 1); e += blockDim.x) {
			const int k = e / (a1 - 1), r = e - k * (a1 - 1) + 1;
			tw[k * lay.tws + r - 1] = __ldg(p.p1.tw + r * k);
		}
		// W_N^{(c0 + c) j}, j < a0, the recurrence's step W_N^{(c0 + c) a0} and its
		// restarts
		const float inv_n2 = 2.0f / static_cast<float>(q.n);
		constexpr int J = kTwiddleJumps;
		for (int e = threadIdx.x; e < CW * (a0 + 1 + J); e += blockDim.x) {
			const int c = e / (a0 + 1 + J), j = e - c * (a0 + 1 + J);
			const uint32_t power = j <= a0 ? j : kTwiddleRun * a0 * (j - a0);
			seeds[e] = tw_n((power * static_cast<uint32_t>(c0 + c)) % n, n, inv_n2, false);
		}
		__syncthreads();
		const int it1 = min(items, (group + 1) * per);
		for (int item = group * per; item < it1; ++item) {
			const int d = item / q.k_blocks;
			const int blk = item - d * q.k_blocks;
			const uint32_t adder = q.adders[q.d_base + d], fe_adder = q.fe_adder;
			const int fe_on = q.fe_on;
			// pass 0: radix a0, sample n2 (j + r a1) + c0 + c (u = j CW + c)
			with_radix<MAXR>(a0, [&](auto rc) {
				constexpr int R = decltype(rc)::value;
				constexpr int PAD = (R & 1) ^ 1;
				const uint32_t dg = static_cast<uint32_t>(n2) * static_cast<uint32_t>(a1);
				for (int u = threadIdx.x; u < CW * a1; u += blockDim.x) {
					const int c = u % CW;
					if (c0 + c >= n2)
						continue;
					const uint64_t g = static_cast<uint64_t>(blk) * n + static_cast<uint64_t>(n2) * (u / CW) + c0 + c;
					float2 v[R];
#pragma unroll
					for (int r = 0; r < R; ++r)
						v[r] = load_sample<ST>(q.samples, g + static_cast<uint64_t>(r) * dg);
					uint32_t hd = q.phase0 + static_cast<uint32_t>(g) * adder;
					const uint32_t dhd = dg * adder;
					if (fe_on) {
						uint32_t hf = static_cast<uint32_t>(g) * fe_adder;
						const uint32_t dhf = dg * fe_adder;
#pragma unroll
						for (int r = 0; r < R; ++r) {
							v[r] = table_mix_holder(v[r], hf, lut);
							hf += dhf;
						}
					}
#pragma unroll
					for (int r = 0; r < R; ++r) {
						v[r] = table_mix_holder(v[r], hd, lut);
						hd += dhd;
					}
					Dft<R, false>::run(v);
					float2* o = work + (u / CW) * ((R + PAD) * CW) + c;
#pragma unroll
					for (int r = 0; r < R; ++r)
						o[r * CW] = v[r];
				}
			});
			__syncthreads();
			// pass 1: radix a1, output k1 = j + r a0, times W_N^{(c0 + c) k1}
			float2* out = p.out + static_cast<size_t>(item) * n + c0;
			with_radix<MAXR>(a1, [&](auto rc) {
				constexpr int R = decltype(rc)::value;
				const size_t inc = static_cast<size_t>(a0) * n2;
				for (int u = threadIdx.x; u < CW * a0; u += blockDim.x) {
					const int j = u / CW, c = u % CW;
					if (c0 + c >= n2)
						continue;
					const float2* wk = tw + j * lay.tws - 1;
					float2 v[R];
#pragma unroll
					for (int r = 0; r < R; ++r)
						v[r] = work[u + r * lay.stride];
#pragma unroll
					for (int r = 1; r < R; ++r)
						v[r] = cmul(v[r], wk[r]);
					Dft<R, false>::run(v);
					const float2* const sc = seeds + c * (a0 + 1 + J);
					float2 w = sc[j];
					const float2 step = sc[a0];
					float2* o = out + static_cast<size_t>(j) * n2 + c;
#pragma unroll
					for (int r = 0; r < R; ++r) {
						*o = cmul(v[r], w);
						w = (r + 1) % kTwiddleRun ? cmul(w, step) : cmul(sc[j], sc[a0 + (r + 1) / kTwiddleRun]);
						o += inc;
					}
				}
			});
			__syncthreads();  // the next item's pass 0 rewrites the tile
		}
	}

	template <int ST>
	void launch_fwd_cols_pair(const BatchedParams& p, int items, int sm_count, cudaStream_t stream) {
		const PairCols lay(p.pair.a0, p.pair.a1, 8);
		const int seeds = lay.acc_at + static_cast<int>(sizeof(float2)) * 8 * (p.pair.a0 + 1 + kTwiddleJumps);
		const int parts = (p.n2 + 7) / 8, per = pair_items(items, parts, sm_count);
		const int grid = (items + per - 1) / per * parts;
		auto kernel = max(p.pair.a0, p.pair.a1) <= 25 ? fwd_cols_pair_kernel<ST, 25> : fwd_cols_pair_kernel<ST, 32>;
		cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem);
		kernel<<<grid, pair_fwd_threads(8 * min(p.pair.a0, p.pair.a1)), seeds, stream>>>(p, items, per);
	}

	// grid: ceil(items / per) * ceil(N1 / rw); spectra elements k2 <
	// row_keep (0: all) of each row stored
	template <int MAXR>
	__global__ void __launch_bounds__(kPairThreads, kPairMinBlocks<MAXR>) fwd_rows_pair_kernel(const __grid_constant__ BatchedParams p, int items,
		int per) {
		extern __shared__ __align__(16) unsigned char raw[];
		const int b0 = p.pair.b0, b1 = p.pair.b1, n1 = p.n1, n2 = p.n2;
		const PairRows lay(b0, b1, p.pair.rw, 0);
		float2* const b = reinterpret_cast<float2*>(raw);
		float2* const tw = reinterpret_cast<float2*>(raw + lay.cs_at);  // no staged code rows
		const int chunks = (n1 + p.pair.rw - 1) / p.pair.rw;
		const int group = blockIdx.x / chunks;
		const int r0 = (blockIdx.x - group * chunks) * p.pair.rw;
		const int rw = min(p.pair.rw, n1 - r0);
		for (int e = threadIdx.x; e < b0 * (b1 - 1); e += blockDim.x) {
			const int k = e / (b1 - 1), r = e - k * (b1 - 1) + 1;
			tw[k * lay.tws + r - 1] = __ldg(p.p2.tw + r * k);
		}
		__syncthreads();
		const int keep = p.row_keep > 0 ? p.row_keep : n2;
		const float inv_b1 = 1.0f / static_cast<float>(b1), inv_b0 = 1.0f / static_cast<float>(b0);
		const int it1 = min(items, (group + 1) * per);
		for (int item = group * per; item < it1; ++item) {
			float2* rows = p.out + static_cast<size_t>(item) * p.base.n + static_cast<size_t>(r0) * n2;
			with_radix<MAXR>(b0, [&](auto rc) {
				constexpr int R = decltype(rc)::value;
				constexpr int PAD = (R & 1) ^ 1;
				for (int u = threadIdx.x; u < rw * b1; u += blockDim.x) {
					const int f = fdiv(u, inv_b1), j = u - f * b1;
					const float2* x = rows + f * n2 + j;
					float2 v[R];
#pragma unroll
					for (int r = 0; r < R; ++r)
						v[r] = x[r * b1];
					Dft<R, false>::run(v);
					float2* o = b + f * lay.ldb + j * (R + PAD);
#pragma unroll
					for (int r = 0; r < R; ++r)
						o[r] = v[r];
				}
			});
			__syncthreads();  // the CTA's rows are read: pass 1 may write over them
			with_radix<MAXR>(b1, [&](auto rc) {
				constexpr int R = decltype(rc)::value;
				const int stride = b0 + lay.pad;
				for (int u = threadIdx.x; u < rw * b0; u += blockDim.x) {
					const int f = fdiv(u, inv_b0), j = u - f * b0;
					const float2* src = b + f * lay.ldb + j;
					const float2* wk = tw + j * lay.tws - 1;
					float2 v[R];
#pragma unroll
					for (int r = 0; r < R; ++r)
						v[r] = src[r * stride];
#pragma unroll
					for (int r = 1; r < R; ++r)
						v[r] = cmul(v[r], wk[r]);
					Dft<R, false>::run(v);
					float2* o = rows + f * n2 + j;
					int k2 = j;
#pragma unroll
					for (int r = 0; r < R; ++r) {
						if (k2 < keep)
							o[r * b0] = v[r];
						k2 += b0;
					}
				}
			});
			__syncthreads();  // the next item's pass 0 rewrites the tile
		}
	}
}
