// Single-CTA acquisition kernels for any block size that fits: each pass of
// the plan switches on its radix once (radix_switch.cuh), the first pass
// gathers its inputs from global memory (samples through the mixers, or X C)
// and the last one stores the spectrum or accumulates the magnitude, so a
// transform of two or three passes takes as many barriers and no separate
// load, store or magnitude loop.  The pass twiddles W_N^{r k N / (NS R)} come
// from a per-size table in the order [r - 1][k] (coalesced over the lanes'
// consecutive k; L1).
// acq_inv_small_kernel splits the K blocks of a (code, Doppler) row over the
// CTAs of a cluster when the rows alone leave SMs idle; the CTAs add their
// magnitudes in block order through distributed shared memory.
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

	// Three passes in place (the inverse): pass 0's butterfly j leaves output
	// k0 at j s0 + (j / R2) pad + k0; the middle pass takes j = j1 + R2 r, r <
	// R1, of one (j1, k0) and leaves k1 at (j1 + R2 k1, k0), so no thread waits
	// between its reads and its writes; the last pass takes the R2 values j1 of
	// one (k0, k1), whose output k2 is element k0 + R0 k1 + R0 R1 k2.  s0 is
	// odd (pass 0's stores) and a group of R2 rows padded so that the last
	// pass's lanes run on through the banks from one k1 to the next.
	struct InPlace {
		int s0, pad, group, elems;
		UG_HD constexpr InPlace(int r0, int r1, int r2)
			: s0(r0 | 1), pad(((r0 - s0 * r2) % 16 + 16) % 16), group(s0 * r2 + pad), elems(group * r1) {}
	};

	// elements of pass 0's tile
	UG_HD int small_tile(const SmallPlan& plan) { return plan.n + (plan.radix[0] % 2 == 0 ? plan.n / plan.radix[0] : 0); }
	// the tiles of a transform (a second one with a middle pass), bytes
	inline int small_tiles_bytes(const SmallPlan& plan) {
		return static_cast<int>(sizeof(float2)) * (small_tile(plan) + (plan.n_pass > 2 ? plan.n : 0));
	}
	// accumulators, 16-byte pieces of them
	UG_HD constexpr int small_accs(int n) { return (n + 3) / 4 * 4; }
	inline int small_inv_bytes(const SmallPlan& plan) {
		const int tile = plan.n_pass == 3
			? static_cast<int>(sizeof(float2)) * InPlace(plan.radix[0], plan.radix[1], plan.radix[2]).elems : small_tiles_bytes(plan);
		return static_cast<int>(sizeof(float)) * small_accs(plan.n) + (tile + 15) / 16 * 16;
	}
	// beyond those, bytes: a cluster CTA's second buffer of magnitudes and its
	// share of the running sums
	UG_HD int small_cluster_bytes(const SmallPlan& plan) {
		const int step = 4 * plan.split * plan.threads;
		return plan.split > 1 ? static_cast<int>(sizeof(float)) * (small_accs(plan.n) + (plan.n + step - 1) / step * 4 * plan.threads) : 0;
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
	// blocks of 4,000 points as 25 x 10 x 16
	void launch_inv_4000(const AcqParams& p, const SmallPlan& plan, bool half, int rows, cudaStream_t stream);

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

	__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
	__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

	// Adds a round of a cluster's CTAs, the first `live` of which hold a block's n
	// magnitudes in mag, in block order to the running sums, of which every CTA
	// keeps its share in tot (a CTA alone reading the others' waits a round trip
	// per element and CTA: half the kernel's time at 168 rows of 2,500 points).
	// A cell's sum is so the one a lone CTA makes of its blocks, whatever the
	// split, and the split may follow the rows of a launch.  The last round
	// leaves the sums in the first CTA's mag.  Between a wait for the round's
	// magnitudes and an arrival.
	__device__ __forceinline__ void cluster_add(float* mag, float* tot, int n, int split, int part, int live, bool first, bool last) {
		const uint32_t mine = static_cast<uint32_t>(__cvta_generic_to_shared(mag));
		uint32_t at[8];
#pragma unroll
		for (int o = 0; o < 8; ++o)
			if (o < split)
				asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at[o]) : "r"(mine), "r"(o));
		// four sums a thread: a round trip per 4 x split x threads of them
		float4* const sums = reinterpret_cast<float4*>(tot);
		for (int i = part * blockDim.x + threadIdx.x, j = threadIdx.x; i < (n + 3) / 4; i += split * blockDim.x, j += blockDim.x) {
			float4 v[8];
#pragma unroll
			for (int o = 0; o < 8; ++o)
				if (o < live)
					asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
						: "=f"(v[o].x), "=f"(v[o].y), "=f"(v[o].z), "=f"(v[o].w) : "r"(at[o] + 16u * i) : "memory");
			float4 s = first ? make_float4(0.f, 0.f, 0.f, 0.f) : sums[j];
#pragma unroll
			for (int o = 0; o < 8; ++o)
				if (o < live)
					s = make_float4(s.x + v[o].x, s.y + v[o].y, s.z + v[o].z, s.w + v[o].w);
			if (last)
				asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};"
					:: "r"(at[0] + 16u * i), "f"(s.x), "f"(s.y), "f"(s.z), "f"(s.w) : "memory");
			else
				sums[j] = s;
		}
	}

	// grid: (rows x split) CTAs in clusters of `split`; unfolded rows (m == N).
	// Three passes run in place (InPlace) in one tile; the two tiles they took
	// before left two CTAs per SM from 4,000 points on: 672 rows x 10 blocks of
	// 4,092 points 307 -> 188 us, of 5,000 380 -> 178.  Two CTAs' worth of
	// registers (128 a thread): at 80 radices from 12 on spill, 672 x 10 of
	// 3,000 points 139 us against 110.
	// HALF: one-sided spectra (Z is zero above N / 2: pass 0 reads R / 2 + 1 of
	// its R inputs)
	// CLUSTER: split > 1 (apart, as its sums cost the lone CTAs' kernel registers:
	// 255 -> 267 us for 32 codes x 21 bins x 20 blocks of 2,046 points)
	template <int MAXR, bool HALF, bool CLUSTER>
	__global__ void __launch_bounds__(kSmallThreads, HALF ? 2 : 1) acq_inv_small_kernel(const __grid_constant__ AcqParams p,
		const __grid_constant__ SmallPlan plan, int mag_at) {
		extern __shared__ __align__(16) float2 smem[];
		const int n = plan.n;
		float* const acc = reinterpret_cast<float*>(smem);
		// (the same offset in a lone CTA spilled 500 bytes more at radix 31, 4 - 14 %)
		float2* const a = smem + (CLUSTER ? small_accs(n) / 2 : (n + 1) / 2);
		float2* const b = a + small_tile(plan);
		float* const mag = acc + mag_at;  // a cluster CTA's magnitudes: here and in acc by turns
		const int split = CLUSTER ? plan.split : 1;
		const int row = blockIdx.x / split;
		const int part = blockIdx.x - row * split;
		const int c = row % p.n_codes;
		const int d = row / p.n_codes;
		const float2* code = p.codes[c];
		for (int i = threadIdx.x; i < n; i += blockDim.x)
			acc[i] = 0.f;
		const float scale = (p.one_sided ? 2.0f : 1.0f) / static_cast<float>(n);
		const int stat = p.stat;
		constexpr bool alone = !CLUSTER;
		// the last pass reads the tile that the next block's first pass rewrites
		// unless a middle pass (and its barrier) lies between
		const bool fence = (plan.n_pass & 1) == 0;
		const bool three = plan.n_pass == 3;
		const int r0 = plan.radix[0], r1 = plan.radix[1], r2 = three ? plan.radix[2] : 1;
		const InPlace ip(r0, r1, r2);
		const float inv_r0 = 1.0f / static_cast<float>(r0), inv_r2 = 1.0f / static_cast<float>(r2);
		// A cluster's round of blocks is added while the next one's are on their
		// way, before their magnitudes are written: whoever waits for a round's
		// has added the one before it, so two buffers do
		bool odd = true;
		auto add_round = [&](int blk0, bool last) {
			cluster_wait();
			cluster_add(odd ? mag : acc, mag + small_accs(n), n, split, part, min(split, p.k_blocks - blk0), blk0 == 0, last);
		};
		for (int blk0 = 0; blk0 < p.k_blocks; blk0 += split) {
			const int blk = blk0 + part;
			if (CLUSTER && blk >= p.k_blocks) {  // a last round of fewer blocks than CTAs
				add_round(blk0 - split, false);
				odd = !odd;
				cluster_arrive();
				break;
			}
			const float2* x = p.spectra + (static_cast<size_t>(d) * p.k_blocks + blk) * n;
			with_radix<MAXR>(plan.radix[0], [&](auto rc) {
				constexpr int R = decltype(rc)::value;
				constexpr int RL = HALF ? R / 2 + 1 : R;
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
					float2* o = a + u * (R | 1) + (three ? fdiv(u, inv_r2) * ip.pad : 0);
#pragma unroll
					for (int r = 0; r < R; ++r)
						o[r] = v[r];
				}
			});
			__syncthreads();
			if (three) {
				with_radix<MAXR>(r1, [&](auto rc) {
					constexpr int R = decltype(rc)::value;
					for (int u = threadIdx.x; u < r0 * r2; u += blockDim.x) {  // u = k0 + R0 j1
						const int j1 = fdiv(u, inv_r0), k0 = u - j1 * r0;
						float2* e = a + j1 * ip.s0 + k0;
						const float2* w = plan.tables + k0;
						float2 v[R];
#pragma unroll
						for (int r = 0; r < R; ++r)
							v[r] = e[r * ip.group];
#pragma unroll
						for (int r = 1; r < R; ++r)
							v[r] = cmulc(v[r], __ldg(w + (r - 1) * r0));
						Dft<R, true>::run(v);
#pragma unroll
						for (int r = 0; r < R; ++r)
							e[r * ip.group] = v[r];
					}
				});
				__syncthreads();
				if (!alone && blk0)
					add_round(blk0 - split, false);
				odd = !odd;
				float* const to = odd ? mag : acc;
				with_radix<MAXR>(r2, [&](auto rc) {
					constexpr int R = decltype(rc)::value;
					const int ns = r0 * r1;
					for (int u = threadIdx.x; u < ns; u += blockDim.x) {  // u = k0 + R0 k1
						const int k1 = fdiv(u, inv_r0);
						const float2* e = a + k1 * ip.group + (u - k1 * r0);
						const float2* w = plan.tables + r0 * (r1 - 1) + u;
						float2 v[R];
#pragma unroll
						for (int r = 0; r < R; ++r)
							v[r] = e[r * ip.s0];
#pragma unroll
						for (int r = 1; r < R; ++r)
							v[r] = cmulc(v[r], __ldg(w + (r - 1) * ns));
						Dft<R, true>::run(v);
						float m[R];
						stats_of(v, scale, stat, m);
						if constexpr (alone) {
#pragma unroll
							for (int r = 0; r < R; ++r)
								acc[u + r * ns] += m[r];
						}
						else {
#pragma unroll
							for (int r = 0; r < R; ++r)
								to[u + r * ns] = m[r];
						}
					}
				});
				if (!alone)
					cluster_arrive();
				__syncthreads();  // the next block's pass 0 rewrites the tile
				continue;
			}
			if (!alone && blk0)
				add_round(blk0 - split, false);
			odd = !odd;
			float* const to = odd ? mag : acc;
			small_passes<MAXR, true>(a, b, plan, [&](int u, int ns, auto& v, auto rc) {
				constexpr int R = decltype(rc)::value;
				float m[R];
				stats_of(v, scale, stat, m);
				if constexpr (alone) {
#pragma unroll
					for (int r = 0; r < R; ++r)
						acc[u + r * ns] += m[r];
				}
				else {
#pragma unroll
					for (int r = 0; r < R; ++r)
						to[u + r * ns] = m[r];
				}
			});
			if (!alone)
				cluster_arrive();
			if (fence)
				__syncthreads();
		}
		if (!alone) {
			add_round((p.k_blocks - 1) / split * split, true);
			cluster_arrive();
			cluster_wait();
			if (part != 0)
				return;
		}
		__syncthreads();
		reduce_cell(alone || !odd ? acc : mag, n, p.cells + static_cast<size_t>(c) * p.n_doppler + p.d_base + d);
	}

	// The same for N = R0 R1 R2 with every pass compiled in.  At 4,000 points
	// 48 KB a CTA, so registers decide (three CTAs per SM); two tiles and a
	// staged twiddle table (112 KB) left two: 672 rows x 10 blocks 128 -> 90 us.
	// Bound: the L1 / shared-memory data pipe (60 %), issue (51 %) and the
	// barriers between the passes.
	template <int R0, int R1, int R2, bool HALF, bool CLUSTER>
	__global__ void __launch_bounds__(kSmallThreads, 3) acq_inv_three_kernel(const __grid_constant__ AcqParams p,
		const __grid_constant__ SmallPlan plan, int mag_at) {
		constexpr int N = R0 * R1 * R2, NB0 = N / R0, NB1 = N / R1, NB2 = N / R2;
		static_assert(R0 % 2 == 1, "rows of R0 elements: the middle pass's u runs along them");
		static_assert(NB0 <= kSmallThreads && NB1 <= 2 * kSmallThreads && NB2 <= kSmallThreads, "butterflies per thread");
		constexpr int RL = HALF ? R0 / 2 + 1 : R0;
		constexpr InPlace ip(R0, R1, R2);
		constexpr int GS = ip.group;
		extern __shared__ __align__(16) float2 smem[];
		float2* const t = smem;
		static_assert(ip.elems % 2 == 0, "16-byte aligned accumulators");
		float* const acc = reinterpret_cast<float*>(smem + ip.elems);
		float* const mag = reinterpret_cast<float*>(smem) + mag_at;  // a cluster CTA's magnitudes: here and in acc by turns
		const int tid = threadIdx.x;
		float2* const first = t + tid * R0 + tid / R2 * ip.pad;
		const float2* const last = t + tid / R0 * GS + tid % R0;
		const int split = CLUSTER ? plan.split : 1;
		const int row = blockIdx.x / split;
		const int part = blockIdx.x - row * split;
		const int c = row % p.n_codes;
		const int d = row / p.n_codes;
		const float2* code = p.codes[c] + tid;
		const float2* tw1 = plan.tables;
		const float2* tw2 = tw1 + R0 * (R1 - 1) + tid;
		if (tid < NB2)
#pragma unroll
			for (int r = 0; r < R2; ++r)
				acc[tid + r * NB2] = 0.f;
		const float scale = (p.one_sided ? 2.0f : 1.0f) / static_cast<float>(N);
		const int stat = p.stat;
		constexpr bool alone = !CLUSTER;
		bool odd = true;
		auto add_round = [&](int blk0, bool last) {  // as in acq_inv_small_kernel
			cluster_wait();
			cluster_add(odd ? mag : acc, mag + small_accs(N), N, split, part, min(split, p.k_blocks - blk0), blk0 == 0, last);
		};
		for (int blk0 = 0; blk0 < p.k_blocks; blk0 += split) {
			const int blk = blk0 + part;
			const bool live = alone || blk < p.k_blocks;  // else a last round of fewer blocks than CTAs
			// code and twiddle reads stay in the loop: held across it they spill
			asm volatile("" : "+l"(code), "+l"(tw1), "+l"(tw2));
			if (live && tid < NB0) {
				const float2* x = p.spectra + (static_cast<size_t>(d) * p.k_blocks + blk) * N + tid;
				float2 v[R0];
#pragma unroll
				for (int r = 0; r < RL; ++r)
					v[r] = __ldg(x + r * NB0);
#pragma unroll
				for (int r = 0; r < RL; ++r)
					v[r] = (HALF || p.one_sided) && tid + r * NB0 > N / 2 ? c2(0.f, 0.f) : cmul(v[r], __ldg(code + r * NB0));
				if constexpr (RL < R0)
					DftPruned<R0, true, RL>::run(v);
				else
					Dft<R0, true>::run(v);
#pragma unroll
				for (int r = 0; r < R0; ++r)
					first[r] = v[r];
			}
			__syncthreads();
			for (int u = live ? tid : NB1; u < NB1; u += kSmallThreads) {  // u = k0 + R0 j1
				const float2* w = tw1 + u % R0;
				float2 v[R1];
#pragma unroll
				for (int r = 0; r < R1; ++r)
					v[r] = t[u + r * GS];
#pragma unroll
				for (int r = 1; r < R1; ++r)
					v[r] = cmulc(v[r], __ldg(w + (r - 1) * R0));
				Dft<R1, true>::run(v);
#pragma unroll
				for (int r = 0; r < R1; ++r)
					t[u + r * GS] = v[r];
			}
			__syncthreads();
			if (!alone && blk0)
				add_round(blk0 - split, false);
			odd = !odd;
			if (live && tid < NB2) {
				float2 v[R2];
#pragma unroll
				for (int r = 0; r < R2; ++r)
					v[r] = last[r * R0];
#pragma unroll
				for (int r = 1; r < R2; ++r)
					v[r] = cmulc(v[r], __ldg(tw2 + (r - 1) * NB2));
				Dft<R2, true>::run(v);
				float m[R2];
				stats_of(v, scale, stat, m);
				if constexpr (alone) {
#pragma unroll
					for (int r = 0; r < R2; ++r)
						acc[tid + r * NB2] += m[r];
				}
				else {
					float* const to = (odd ? mag : acc) + tid;
#pragma unroll
					for (int r = 0; r < R2; ++r)
						to[r * NB2] = m[r];
				}
			}
			if (!alone)
				cluster_arrive();
			__syncthreads();  // the next block's pass 0 rewrites the tile
		}
		if (!alone) {
			add_round((p.k_blocks - 1) / split * split, true);
			cluster_arrive();
			cluster_wait();
			if (part != 0)
				return;
		}
		__syncthreads();
		reduce_cell(alone || !odd ? acc : mag, N, p.cells + static_cast<size_t>(c) * p.n_doppler + p.d_base + d);
	}

	template <class K>
	void launch_fwd_small(K kernel, const AcqParams& p, const SmallPlan& plan, int items, cudaStream_t stream) {
		cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem);
		kernel<<<items, plan.threads, small_tiles_bytes(plan), stream>>>(p, plan);
	}

	// the launch error, if any, is the runtime's last error
	template <class K>
	void launch_inv_small(K kernel, const AcqParams& p, const SmallPlan& plan, int rows, cudaStream_t stream) {
		const int smem = small_inv_bytes(plan);
		cudaLaunchConfig_t cfg{};
		cfg.gridDim = dim3(static_cast<unsigned>(rows) * plan.split);
		cfg.blockDim = dim3(plan.threads);
		cfg.dynamicSmemBytes = smem + small_cluster_bytes(plan);
		cfg.stream = stream;
		cudaLaunchAttribute cluster{};
		cluster.id = cudaLaunchAttributeClusterDimension;
		cluster.val.clusterDim.x = static_cast<unsigned>(plan.split);
		cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
		cfg.attrs = &cluster;
		cfg.numAttrs = plan.split > 1 ? 1 : 0;
		cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem);
		cudaLaunchKernelEx(&cfg, kernel, p, plan, smem / static_cast<int>(sizeof(float)));
	}
}
