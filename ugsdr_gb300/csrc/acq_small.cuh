// Single-CTA acquisition kernels for any block size that fits: each pass of
// the plan switches on its radix once (radix_switch.cuh), the first pass
// gathers its inputs from global memory (samples through the mixers, or X C)
// and the last one stores the spectrum or accumulates the magnitude, so a
// transform of two or three passes takes as many barriers and no separate
// load, store or magnitude loop.  The pass twiddles W_N^{r k N / (NS R)} come
// from a per-size table in the order [r - 1][k] (coalesced over the lanes'
// consecutive k; L1).
// acq_inv_small_kernel splits the K blocks of a (code, Doppler) row over the
// CTAs of a cluster when the rows alone leave SMs idle; the first CTA adds the
// others' accumulators through distributed shared memory.
// Bound: issue and the barriers between the passes.
#pragma once

#include "acq_kernels.cuh"
#include "radix_switch.cuh"

#include <cuda_runtime.h>

namespace ugsdr_gpu {

	constexpr int kSmallThreads = 256;

	struct SmallPlan {
		int n, n_pass;
		int radix[12];
		const float2* tables;  // pass s >= 1 at offset sum of the earlier passes' NS (R - 1)
		int threads;
		int split;             // CTAs per row (inverse)
	};

	// elements of pass 0's tile
	UG_HD int small_tile(const SmallPlan& plan) { return plan.n + (plan.radix[0] % 2 == 0 ? plan.n / plan.radix[0] : 0); }
	// the tiles of a transform (a second one with a middle pass), bytes
	inline int small_tiles_bytes(const SmallPlan& plan) {
		return static_cast<int>(sizeof(float2)) * (small_tile(plan) + (plan.n_pass > 2 ? plan.n : 0));
	}
	inline int small_inv_bytes(const SmallPlan& plan) {
		return static_cast<int>(sizeof(float2)) * ((plan.n + 1) / 2) + small_tiles_bytes(plan);
	}
	// every kernel's limit, set to it always: a context with smaller blocks
	// never lowers it under another's launch
	constexpr int kSmallSmem = 224 * 1024;

	// launches, by sample type (forward) and largest radix (inverse; the
	// two-sided spectra share one kernel)
	void launch_fwd_small_8bit(const AcqParams& p, const SmallPlan& plan, int sample_type, int items, cudaStream_t stream);
	void launch_fwd_small_wide(const AcqParams& p, const SmallPlan& plan, int sample_type, int items, cudaStream_t stream);
	void launch_inv_small25(const AcqParams& p, const SmallPlan& plan, int rows, cudaStream_t stream);
	void launch_inv_small32(const AcqParams& p, const SmallPlan& plan, int rows, cudaStream_t stream);

	// Runs the passes after the first: `a` holds pass 0's output (padded by one
	// element per butterfly when its radix is even), middle passes ping-pong
	// between the tiles, the last one hands each butterfly to emit(u, NS, v):
	// output element u + r NS is v[r], u < NS.  Ends without a barrier.
	template <int MAXR, bool INV, class Emit>
	__device__ __forceinline__ void small_passes(float2* a, float2* b, const SmallPlan& plan, Emit&& emit) {
		const int n = plan.n;
		int ns = plan.radix[0];
		const int pad = (ns & 1) ^ 1;
		const float2* tab = plan.tables;
		for (int s = 1; s < plan.n_pass; ++s) {
			const int radix = plan.radix[s];
			const int nb = n / radix;
			const float inv_ns = 1.0f / static_cast<float>(ns);
			const bool last = s + 1 == plan.n_pass;
			// pass 1 reads the padded tile: element u + r nb at u + u / ns pad + r (nb + nb / ns pad)
			const int p1 = s == 1 ? pad : 0;
			const int stride = nb + p1 * (nb / ns);
			with_radix<MAXR>(radix, [&](auto rc) {
				constexpr int R = decltype(rc)::value;
				for (int u = threadIdx.x; u < nb; u += blockDim.x) {
					const int uq = fdiv(u, inv_ns);
					const int k = u - uq * ns;
					const float2* src = a + u + p1 * uq;
					float2 v[R];
#pragma unroll
					for (int r = 0; r < R; ++r)
						v[r] = src[r * stride];
#pragma unroll
					for (int r = 1; r < R; ++r) {
						const float2 w = __ldg(tab + (r - 1) * ns + k);
						v[r] = INV ? cmulc(v[r], w) : cmul(v[r], w);
					}
					Dft<R, INV>::run(v);
					if (last) {
						emit(u, ns, v, rc);
					}
					else {
						float2* dst = b + uq * (R * ns) + k;
#pragma unroll
						for (int r = 0; r < R; ++r)
							dst[r * ns] = v[r];
					}
				}
			});
			if (last)
				return;
			__syncthreads();
			tab += ns * (radix - 1);
			ns *= radix;
			float2* t = a;
			a = b;
			b = t;
		}
	}

	// grid: Doppler bins x K blocks, one transform each
	template <int ST>
	__global__ void __launch_bounds__(kSmallThreads, 2) acq_fwd_small_kernel(const __grid_constant__ AcqParams p,
		const __grid_constant__ SmallPlan plan) {
		extern __shared__ float2 smem[];
		__shared__ float lut[80];
		for (int i = threadIdx.x; i < 80; i += blockDim.x)
			lut[i] = p.lut[i];
		__syncthreads();
		const int n = plan.n;
		const int d = blockIdx.x / p.k_blocks;
		const int blk = blockIdx.x - d * p.k_blocks;
		const uint32_t adder = p.adders[p.d_base + d];
		const uint64_t base = static_cast<uint64_t>(blk) * n;
		float2* a = smem;
		with_radix<32>(plan.radix[0], [&](auto rc) {
			constexpr int R = decltype(rc)::value;
			constexpr int PAD = (R & 1) ^ 1;
			const int nb = n / R;
			for (int u = threadIdx.x; u < nb; u += blockDim.x) {
				const uint64_t g = base + u;
				float2 v[R];
#pragma unroll
				for (int r = 0; r < R; ++r)
					v[r] = load_sample<ST>(p.samples, g + static_cast<uint64_t>(r) * nb);
				if (p.fe_on) {
					uint32_t hf = static_cast<uint32_t>(g) * p.fe_adder;
#pragma unroll
					for (int r = 0; r < R; ++r) {
						v[r] = table_mix_holder(v[r], hf, lut);
						hf += static_cast<uint32_t>(nb) * p.fe_adder;
					}
				}
				uint32_t hd = p.phase0 + static_cast<uint32_t>(g) * adder;
#pragma unroll
				for (int r = 0; r < R; ++r) {
					v[r] = table_mix_holder(v[r], hd, lut);
					hd += static_cast<uint32_t>(nb) * adder;
				}
				Dft<R, false>::run(v);
				float2* o = a + u * (R + PAD);
#pragma unroll
				for (int r = 0; r < R; ++r)
					o[r] = v[r];
			}
		});
		__syncthreads();
		float2* dst = p.spectra + (static_cast<size_t>(d) * p.k_blocks + blk) * n;
		const int limit = p.one_sided ? n / 2 + 1 : n;
		small_passes<32, false>(a, a + small_tile(plan), plan, [&](int u, int ns, auto& v, auto rc) {
			constexpr int R = decltype(rc)::value;
#pragma unroll
			for (int r = 0; r < R; ++r)
				if (u + r * ns < limit)
					dst[u + r * ns] = v[r];
		});
	}

	// grid: (rows x split) CTAs in clusters of `split`; unfolded rows (m == N).
	// HALF: one-sided spectra (Z is zero above N / 2: pass 0 reads R / 2 + 1 of
	// its R inputs)
	template <int MAXR, bool HALF>
	__global__ void __launch_bounds__(kSmallThreads, !HALF ? 1 : MAXR <= 25 ? 3 : 2) acq_inv_small_kernel(const __grid_constant__ AcqParams p,
		const __grid_constant__ SmallPlan plan) {
		extern __shared__ float2 smem[];
		const int n = plan.n;
		float* const acc = reinterpret_cast<float*>(smem);
		float2* const a = smem + (n + 1) / 2;
		float2* const b = a + small_tile(plan);
		const int row = blockIdx.x / plan.split;
		const int part = blockIdx.x - row * plan.split;
		const int c = row % p.n_codes;
		const int d = row / p.n_codes;
		const float2* code = p.codes[c];
		for (int i = threadIdx.x; i < n; i += blockDim.x)
			acc[i] = 0.f;
		const float scale = (p.one_sided ? 2.0f : 1.0f) / static_cast<float>(n);
		const int stat = p.stat;
		// the last pass reads the tile that the next block's first pass rewrites
		// unless a middle pass (and its barrier) lies between
		const bool fence = (plan.n_pass & 1) == 0;
		for (int blk = part; blk < p.k_blocks; blk += plan.split) {
			const float2* x = p.spectra + (static_cast<size_t>(d) * p.k_blocks + blk) * n;
			with_radix<MAXR>(plan.radix[0], [&](auto rc) {
				constexpr int R = decltype(rc)::value;
				constexpr int RL = HALF ? R / 2 + 1 : R;
				constexpr int PAD = (R & 1) ^ 1;
				const int nb = n / R;
				for (int u = threadIdx.x; u < nb; u += blockDim.x) {
					float2 v[R];
#pragma unroll
					for (int r = 0; r < RL; ++r)
						v[r] = __ldg(x + u + r * nb);
					// one-sided spectra end at N / 2: beyond it (r = R / 2, u > 0) X is not
					// written, and an even radix's last live input counts for u = 0 only
#pragma unroll
					for (int r = 0; r < RL; ++r)
						v[r] = HALF && u + r * nb > n / 2 ? c2(0.f, 0.f) : cmul(v[r], __ldg(code + u + r * nb));
					if constexpr (RL < R)
						DftPruned<R, true, RL>::run(v);
					else
						Dft<R, true>::run(v);
					float2* o = a + u * (R + PAD);
#pragma unroll
					for (int r = 0; r < R; ++r)
						o[r] = v[r];
				}
			});
			__syncthreads();
			small_passes<MAXR, true>(a, b, plan, [&](int u, int ns, auto& v, auto rc) {
				constexpr int R = decltype(rc)::value;
#pragma unroll
				for (int r = 0; r < R; ++r)
					acc[u + r * ns] += stat_of(cscale(v[r], scale), stat);
			});
			if (fence)
				__syncthreads();
		}
		if (plan.split > 1) {
			// distributed shared memory: the first CTA of the cluster adds the others'
			// accumulators in order (every CTA arrives once before and once after)
			asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
			if (part == 0) {
				const uint32_t mine = static_cast<uint32_t>(__cvta_generic_to_shared(acc));
				for (int o = 1; o < plan.split; ++o) {
					uint32_t theirs;
					asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(theirs) : "r"(mine), "r"(o));
					for (int i = threadIdx.x; i < n; i += blockDim.x) {
						float v;
						asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(theirs + 4u * i) : "memory");
						acc[i] += v;
					}
				}
			}
			asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
			if (part != 0)
				return;
		}
		__syncthreads();
		reduce_cell(acc, n, p.cells + static_cast<size_t>(c) * p.n_doppler + p.d_base + d);
	}

	template <class K>
	void launch_fwd_small(K kernel, const AcqParams& p, const SmallPlan& plan, int items, cudaStream_t stream) {
		cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem);
		kernel<<<items, plan.threads, small_tiles_bytes(plan), stream>>>(p, plan);
	}

	// the launch error, if any, is the runtime's last error
	template <class K>
	void launch_inv_small(K kernel, const AcqParams& p, const SmallPlan& plan, int rows, cudaStream_t stream) {
		cudaLaunchConfig_t cfg{};
		cfg.gridDim = dim3(static_cast<unsigned>(rows) * plan.split);
		cfg.blockDim = dim3(plan.threads);
		cfg.dynamicSmemBytes = small_inv_bytes(plan);
		cfg.stream = stream;
		cudaLaunchAttribute cluster{};
		cluster.id = cudaLaunchAttributeClusterDimension;
		cluster.val.clusterDim.x = static_cast<unsigned>(plan.split);
		cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
		cfg.attrs = &cluster;
		cfg.numAttrs = plan.split > 1 ? 1 : 0;
		cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem);
		cudaLaunchKernelEx(&cfg, kernel, p, plan);
	}
}
