// Inverse four-step kernels for any split N = N1 x N2 whose halves are
// products of two radices: N1 = a0 a1, N2 = b0 b1, each radix 2..32.
//
// The runtime plan (acq_batched.cuh RuntimeFft) switches on the radix inside
// every butterfly and derives each element's index from runtime sizes (154
// and 157 thread-instructions per point in the row and column kernels of
// 40,920-point blocks).  Here a pass switches once, uniformly for the CTA, to
// code with its radix compiled in; only the strides stay runtime values, one
// add per element.  One kernel per tile width and register class serves every
// length, so sizes need no plan of their own.
//
// Row stage (inv_rows_pair_kernel): a CTA takes rw rows k1 of one (code,
// Doppler) row through both passes for all K blocks.  Pass 0 gathers Z = X C:
// the X rows straight from global memory (every code's CTA reads the same
// rows: L2), the code rows staged in shared memory once.  With one-sided
// spectra (HALF) Z is zero from the middle of every row on, and pass 0 reads
// b0 / 2 + 1 of its b0 inputs into the pruned DFT.  Pass 1 applies the
// inter-step twiddle (seeds per row, a recurrence of eight products per butterfly) and stores B
// in the blocked layout B[n2 / CW][k1][n2 % CW].
// Column stage (inv_cols_pair_kernel): a CTA takes CW columns of a row over
// the K blocks; pass 0 reads its contiguous N1 x CW tile from global memory,
// pass 1 adds |y| or |y|^2 to accumulators in shared memory that only the
// owning thread touches.
// Both hold one work tile, so two barriers per block; the loads of pass 0 are
// a0 (or b0) independent requests per thread, and the CTAs sharing an SM cover
// their latency.  Elements of a tile are padded by one per pass-0 butterfly
// when the radix is even: its stride-R stores then fall in distinct banks.
// Bound: instruction issue.
#pragma once

#include "acq_batched.cuh"
#include "radix_switch.cuh"

namespace ugsdr_gpu {

	constexpr int kPairThreads = 256;
	// dynamic shared memory a pair kernel may ask for (227 KB less a kilobyte for
	// its static part): always set to this, so that contexts with other splits
	// never lower it under a launch
	constexpr int kPairSmem = 226 * 1024;

	// launches of the kernels below (acq_pairs_rows.cu, acq_pairs_cols.cu)
	void launch_inv_rows_pair(const BatchedParams& p, bool half, cudaStream_t stream);
	void launch_inv_cols_pair(const BatchedParams& p, cudaStream_t stream);

	// shared-memory layouts, in bytes (host and device walk the same code)
	struct PairCols {
		int pad, stride, tws, accs;  // pad per pass-0 butterfly, tile row stride, twiddle and accumulator strides
		int tw_at, acc_at, bytes;
		UG_HD PairCols(int a0, int a1, int cw) {
			pad = (a0 & 1) ^ 1;
			stride = (a0 + pad) * cw;
			tws = (a1 - 1) | 1;
			accs = a1 | 1;
			tw_at = static_cast<int>(sizeof(float2)) * stride * a1;
			acc_at = tw_at + static_cast<int>(sizeof(float2)) * tws * a0;
			bytes = acc_at + static_cast<int>(sizeof(float)) * accs * cw * a0;
		}
	};
	struct PairRows {
		int pad, ldb, live, lds, tws;  // tile row stride, live inputs of a pass-0 butterfly, staged code elements per row
		int cs_at, tw_at, seeds_at, bytes;
		// rw: a power of two >= 4.  Pass 1's half-warps read rw rows x 16 / rw
		// neighbours: a row stride of 16 / rw modulo 16 puts them in distinct banks.
		UG_HD PairRows(int b0, int b1, int rw, int half) {
			pad = (b0 & 1) ^ 1;
			ldb = (b0 + pad) * b1;
			const int want = rw < 16 ? 16 / rw : 1;
			ldb += (want - ldb % 16 + 16) % 16;
			live = half ? b0 / 2 + 1 : b0;
			lds = live * b1;
			tws = (b1 - 1) | 1;
			cs_at = static_cast<int>(sizeof(float2)) * ldb * rw;
			tw_at = cs_at + static_cast<int>(sizeof(float2)) * lds * rw;
			seeds_at = tw_at + static_cast<int>(sizeof(float2)) * tws * b0;
			bytes = seeds_at + static_cast<int>(sizeof(float2)) * rw * (b0 + 1 + kTwiddleJumps);
		}
	};

	// register classes: the DFTs up to radix 25 fit 80 registers (three CTAs of
	// 256 threads), the larger ones (31: 15 pairs of sums and differences) 128
	template <int MAXR>
	constexpr int kPairMinBlocks = MAXR <= 25 ? 3 : 2;

	// grid: rows * ceil(N1 / rw)
	template <int MAXR, bool HALF>
	__global__ void __launch_bounds__(kPairThreads, kPairMinBlocks<MAXR>) inv_rows_pair_kernel(const __grid_constant__ BatchedParams p) {
		extern __shared__ __align__(16) unsigned char raw[];
		const AcqParams& q = p.base;
		const int cw_shift = p.pair.cw_shift, cw = 1 << cw_shift, cw_mask = cw - 1;
		const int b0 = p.pair.b0, b1 = p.pair.b1, n1 = p.n1, n2 = p.n2, n = q.n;
		const PairRows lay(b0, b1, p.pair.rw, HALF);
		float2* const b = reinterpret_cast<float2*>(raw);
		float2* const cs = reinterpret_cast<float2*>(raw + lay.cs_at);
		float2* const tw = reinterpret_cast<float2*>(raw + lay.tw_at);
		float2* const seeds = reinterpret_cast<float2*>(raw + lay.seeds_at);
		const int chunks = (n1 + p.pair.rw - 1) / p.pair.rw;
		const int lrow = blockIdx.x / chunks;
		const int r0 = (blockIdx.x - lrow * chunks) * p.pair.rw;
		const int rw = min(p.pair.rw, n1 - r0);
		const int row = p.row0 + lrow;
		const int c = row % q.n_codes;
		const int d = row / q.n_codes;
		// pass-1 twiddles W_N2^{r k}, k < b0, laid out [k][r - 1]
		for (int e = threadIdx.x; e < b0 * (b1 - 1); e += blockDim.x) {
			const int k = e / (b1 - 1), r = e - k * (b1 - 1) + 1;
			tw[k * lay.tws + r - 1] = __ldg(p.p2.tw + r * k);
		}
		build_row_seeds(seeds, rw, b0, r0, static_cast<uint32_t>(n), row_gain(n), kTwiddleJumps);
		const float2* code = q.codes[c] + static_cast<size_t>(r0) * n2;
		for (int f = 0; f < rw; ++f)
			for (int e = threadIdx.x; e < lay.lds; e += blockDim.x)
				cs[f * lay.lds + e] = __ldg(code + f * n2 + e);
		__syncthreads();
		const float2* xg = q.spectra + static_cast<size_t>(d) * q.k_blocks * n + static_cast<size_t>(r0) * n2;
		const size_t out_block = static_cast<size_t>(n1) * p.n2p;
		float2* out = p.bbuf + static_cast<size_t>(lrow) * q.k_blocks * out_block + (r0 << cw_shift);
		const float inv_b1 = 1.0f / static_cast<float>(b1);
		const int rw_shift = 31 - __clz(p.pair.rw);
		const int chunk_elems = n1 << cw_shift;
		for (int blk = 0; blk < q.k_blocks; ++blk, xg += n, out += out_block) {
			// pass 0: radix b0, input k2 = j + r b1, j < b1
			with_radix<MAXR>(b0, [&](auto rc) {
				constexpr int R = decltype(rc)::value;
				constexpr int RL = HALF ? R / 2 + 1 : R;
				for (int u = threadIdx.x; u < rw * b1; u += blockDim.x) {
					const int f = fdiv(u, inv_b1), j = u - f * b1;
					const float2* x = xg + f * n2 + j;
					const float2* cc = cs + f * lay.lds + j;
					float2 v[R];
#pragma unroll
					for (int r = 0; r < RL; ++r)
						v[r] = __ldg(x + r * b1);
#pragma unroll
					for (int r = 0; r < RL; ++r)
						v[r] = cmul(v[r], cc[r * b1]);
					if constexpr (RL < R)
						DftPruned<R, true, RL>::run(v);
					else
						Dft<R, true>::run(v);
					constexpr int PAD = (R & 1) ^ 1;
					float2* o = b + f * lay.ldb + j * (R + PAD);
#pragma unroll
					for (int r = 0; r < R; ++r)
						o[r] = v[r];
				}
			});
			__syncthreads();
			// pass 1: radix b1, input j + r b0 at j + r (b0 + pad), output n2 = j + r b0
			with_radix<MAXR>(b1, [&](auto rc) {
				constexpr int R = decltype(rc)::value;
				const int stride = b0 + lay.pad;
				for (int u = threadIdx.x; u < b0 << rw_shift; u += blockDim.x) {
					// rows fastest: a warp's stores of one output are whole
					// 32-byte pieces of adjacent rows, 128-byte lines of B
					const int f = u & (p.pair.rw - 1), j = u >> rw_shift;
					if (f >= rw)
						continue;
					const float2* src = b + f * lay.ldb + j;
					const float2* wk = tw + j * lay.tws - 1;
					float2 v[R];
#pragma unroll
					for (int r = 0; r < R; ++r)
						v[r] = src[r * stride];
#pragma unroll
					for (int r = 1; r < R; ++r)
						v[r] = cmulc(v[r], wk[r]);
					Dft<R, true>::run(v);
					const float2* const sf = seeds + f * (b0 + 1 + kTwiddleJumps);
					float2 w = sf[j];
					const float2 step = sf[b0];
					auto next = [&](int r) {  // the twiddle of output r + 1
						w = (r + 1) % kTwiddleRun ? cmul(w, step) : cmul(sf[j], sf[b0 + (r + 1) / kTwiddleRun]);
					};
					float2* o = out + (f << cw_shift);
					if ((b0 & cw_mask) == 0) {
						// every output a fixed distance from the first
						o += (j >> cw_shift) * chunk_elems + (j & cw_mask);
						const int inc = (b0 >> cw_shift) * chunk_elems;
#pragma unroll
						for (int r = 0; r < R; ++r) {
							o[r * inc] = cmul(v[r], w);
							next(r);
						}
					}
					else {
						int i2 = j;
#pragma unroll
						for (int r = 0; r < R; ++r) {
							o[(i2 >> cw_shift) * chunk_elems + (i2 & cw_mask)] = cmul(v[r], w);
							next(r);
							i2 += b0;
						}
					}
				}
			});
			__syncthreads();  // the next block's pass 0 rewrites the tile
		}
	}

	// grid: rows * (n2p / CW).  STAT: the job's statistic
	template <int CW, int MAXR, int STAT>
	__global__ void __launch_bounds__(kPairThreads, kPairMinBlocks<MAXR>) inv_cols_pair_kernel(const __grid_constant__ BatchedParams p) {
		extern __shared__ __align__(16) unsigned char raw[];
		__shared__ MaxIdx s_max[kPairThreads / 32];
		__shared__ double s_sum[kPairThreads / 32], s_sq[kPairThreads / 32];
		__shared__ bool s_last;
		const AcqParams& q = p.base;
		const int a0 = p.pair.a0, a1 = p.pair.a1, n2 = p.n2;
		const PairCols lay(a0, a1, CW);
		float2* const work = reinterpret_cast<float2*>(raw);
		float2* const tw = reinterpret_cast<float2*>(raw + lay.tw_at);
		float* const acc = reinterpret_cast<float*>(raw + lay.acc_at);
		const int chunks = p.n2p / CW;
		const int lrow = blockIdx.x / chunks;
		const int chunk = blockIdx.x - lrow * chunks;
		// pass-1 twiddles W_N1^{r k}, k < a0, laid out [k][r - 1]
		for (int e = threadIdx.x; e < a0 * (a1 - 1); e += blockDim.x) {
			const int k = e / (a1 - 1), r = e - k * (a1 - 1) + 1;
			tw[k * lay.tws + r - 1] = __ldg(p.p1.tw + r * k);
		}
		for (int e = threadIdx.x; e < CW * a0 * lay.accs; e += blockDim.x)
			acc[e] = 0.f;
		const size_t block_elems = static_cast<size_t>(p.n1) * p.n2p;
		const float2* src = p.bbuf + static_cast<size_t>(lrow) * q.k_blocks * block_elems + static_cast<size_t>(chunk) * (p.n1 * CW);
		__syncthreads();
		for (int blk = 0; blk < q.k_blocks; ++blk, src += block_elems) {
			// pass 0: radix a0, input k1 = j + r a1, column c (u = j CW + c)
			with_radix<MAXR>(a0, [&](auto rc) {
				constexpr int R = decltype(rc)::value;
				const int stride = a1 * CW;
				for (int u = threadIdx.x; u < CW * a1; u += blockDim.x) {
					float2 v[R];
#pragma unroll
					for (int r = 0; r < R; ++r)
						v[r] = __ldg(src + u + r * stride);
					Dft<R, true>::run(v);
					constexpr int PAD = (R & 1) ^ 1;
					float2* o = work + (u / CW) * ((R + PAD) * CW) + u % CW;
#pragma unroll
					for (int r = 0; r < R; ++r)
						o[r * CW] = v[r];
				}
			});
			__syncthreads();
			// pass 1: radix a1, input j + r a0, output n1 = j + r a0
			with_radix<MAXR>(a1, [&](auto rc) {
				constexpr int R = decltype(rc)::value;
				for (int u = threadIdx.x; u < CW * a0; u += blockDim.x) {
					const float2* wk = tw + (u / CW) * lay.tws - 1;
					float2 v[R];
#pragma unroll
					for (int r = 0; r < R; ++r)
						v[r] = work[u + r * lay.stride];
#pragma unroll
					for (int r = 1; r < R; ++r)
						v[r] = cmulc(v[r], wk[r]);
					Dft<R, true>::run(v);
					float* ac = acc + u * lay.accs;
					float m[R];
#pragma unroll
					for (int r = 0; r < R; ++r)
						m[r] = v[r].x * v[r].x + v[r].y * v[r].y;
					if constexpr (!STAT)
						roots(m);
#pragma unroll
					for (int r = 0; r < R; ++r)
						ac[r] += m[r];
				}
			});
			__syncthreads();  // the next block's pass 0 rewrites the tile
		}
		// scale once: |s y| = s |y| with s = 2 / N one-sided (1 / N two-sided), less the row stage's gain
		const float s = column_scale(q.n, q.one_sided);
		const float sc = STAT ? s * s : s;
		MaxIdx best{-1.0f, 0xFFFFFFFFu};
		Moments own(threadIdx.x < CW * a0 && chunk * CW + threadIdx.x % CW < n2 ? acc[threadIdx.x * lay.accs] * sc : __int_as_float(0x7F800000));
		for (int u = threadIdx.x; u < CW * a0; u += blockDim.x) {
			const int j = u / CW, n2g = chunk * CW + u % CW;
			if (n2g >= n2)
				continue;
			for (int r = 0; r < a1; ++r) {
				const float v = acc[u * lay.accs + r] * sc;
				best = better(best, MaxIdx{v, static_cast<uint32_t>(n2) * static_cast<uint32_t>(j + r * a0) + static_cast<uint32_t>(n2g)});
				own.add(v);
			}
		}
		double dsum = 0.0, dsq = 0.0;
		own.reduce(&dsum, &dsq);
		auto reduce_max = [&] {
			for (int o = 16; o > 0; o >>= 1) {
				const MaxIdx other{__shfl_down_sync(0xffffffffu, best.v, o), __shfl_down_sync(0xffffffffu, best.i, o)};
				best = better(best, other);
			}
		};
		reduce_max();
		const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
		if (lane == 0) {
			s_max[warp] = best;
			s_sum[warp] = dsum;
			s_sq[warp] = dsq;
		}
		__syncthreads();
		if (threadIdx.x == 0) {
			for (int w = 1; w < warps; ++w) {
				s_max[0] = better(s_max[0], s_max[w]);
				s_sum[0] += s_sum[w];
				s_sq[0] += s_sq[w];
			}
			const size_t slot = static_cast<size_t>(lrow) * chunks + chunk;
			p.partials[slot] = make_float4(s_max[0].v, __uint_as_float(s_max[0].i), 0.f, 0.f);
			p.sums[slot] = make_double2(s_sum[0], s_sq[0]);
			__threadfence();
			s_last = atomicAdd(p.counters + lrow, 1u) == static_cast<unsigned>(chunks - 1);
		}
		__syncthreads();
		if (!s_last || threadIdx.x >= 32)
			return;
		// last chunk of this row: warp 0 combines every chunk's partial into the
		// cell (lanes over the chunks, then a fixed tree)
		__threadfence();
		best = MaxIdx{-1.0f, 0xFFFFFFFFu};
		dsum = dsq = 0.0;
		for (int k = lane; k < chunks; k += 32) {
			const size_t slot = static_cast<size_t>(lrow) * chunks + k;
			const float4 pt = __ldcg(p.partials + slot);
			const double2 sm = __ldcg(p.sums + slot);
			best = better(best, MaxIdx{pt.x, __float_as_uint(pt.y)});
			dsum += sm.x;
			dsq += sm.y;
		}
		reduce_max();
		for (int o = 16; o > 0; o >>= 1) {
			dsum += __shfl_down_sync(0xffffffffu, dsum, o);
			dsq += __shfl_down_sync(0xffffffffu, dsq, o);
		}
		if (lane != 0)
			return;
		const int row = p.row0 + lrow;
		const int c = row % q.n_codes;
		const int d = q.d_base + row / q.n_codes;
		const int m = q.m;
		const double mean = dsum / m;
		const double var = m > 1 ? (dsq - dsum * mean) / (m - 1) : 0.0;
		AcqCellDev cell;
		cell.level = best.v;
		cell.index = best.i;
		cell.mean = static_cast<float>(mean);
		cell.std = static_cast<float>(sqrt(var > 0 ? var : 0.0));
		q.cells[static_cast<size_t>(c) * q.n_doppler + d] = cell;
	}
}
