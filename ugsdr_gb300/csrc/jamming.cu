// Interference mitigation on the device: the STFT, the jamming detector and
// the suppression engine the digital front end runs after resampling
// (src/dfe/dfe.hpp:199-202).
//
//   detect_kernel       the detector's STFT, eight lanes per column with the
//                       128-point transform in registers and one exchange
//                       through shared memory (Octet128), then one thread per
//                       column for the eight strongest bins with their peak /
//                       sigma (JammingDetector::IntermediateDetection,
//                       src/antijamming/jamming_detection.hpp:113-128) and
//                       each CTA's occupation histograms
//   stft_kernel         the per-op STFT (spectra out): columns per CTA in
//                       shared memory (compile-time 128-point plan)
//   decide_kernel,      AnalyzeStftData (130-189): the occupation vote per
//   jn_sum_kernel       round, then the reported J/N sums; only the detection
//                       list goes back to the host
//   wideband_kernel     FilterWideband (src/antijamming/jse.hpp:70-87) fused,
//                       eight lanes per run of output slots: the covering columns
//                       re-transformed from the samples (Octet128), bins with
//                       |.| >= 20 zeroed, inverse transforms scaled 2/W,
//                       overlap-added in column order in registers
//   istft_cols_kernel,  the per-op OverlapAndAdd (src/math/stft.hpp:63-75):
//   overlap_add_kernel  inverse columns, then a gather in column order
//   null_bins_kernel    FilterInFreqencyDomain (jse.hpp:61-68): +-128 bins
//                       around each narrowband jammer of the whole-signal DFT
#include "internal.hpp"
#include "acq_batched.cuh"
#include "fft_static.cuh"

#include <algorithm>
#include <cmath>
#include <vector>

namespace ugsdr_gpu {
	namespace {
		constexpr int kJamThreads = 256;
		constexpr int kMaxCandidates = 8;      // max_inreference_cnt (jamming_detection.hpp:81)
		constexpr int kNullHalfWidth = 3;      // null_window_size (82)
		constexpr float kJnThreshold = 6.0f;   // j_s_threshold (78)
		constexpr double kProbability = 0.9;   // probability_threshold (79)
		constexpr int kNarrowNull = 128;       // null_window_size (jse.hpp:47)
		constexpr int kDetectWindow = 128;     // Transform's defaults (stft.hpp:19)
		constexpr int kDetectOverlap = 96;

		constexpr int kDetectBins = 128;        // the detector's window
		constexpr int kMaxDetections = 2 * kMaxCandidates;  // two per round at most
		constexpr int kSumCtas = 256;           // CTAs of the J/N sums
		constexpr uint8_t kNoBin = 0xFF;

		struct Detection {
			int type;
			int bin;
			double frequency;
			double jn;
		};

		struct DetectionList {
			int n;
			int pad;
			Detection d[kMaxDetections];
		};

		// Device scratch of the detector (one allocation, 256-byte regions):
		// per round r the occupation histogram over bins, the candidate count,
		// the decisions, the J/N partial sums and the detection list; then the
		// per-column candidates as rounds x columns arrays (bin, J/N).
		struct DetectScratch {
			int* hist;                  // [kMaxCandidates][kDetectBins]
			unsigned long long* total;  // candidates over all columns
			unsigned int* done;         // CTAs of jn_sum_kernel finished
			int* picks;                 // [kMaxCandidates][2]: narrowband, wideband bin or -1
			double* quantity;           // [kMaxCandidates]
			int* rounds;                // mean candidates per column
			DetectionList* list;
			double* partials;           // [kSumCtas][kMaxDetections]
			uint8_t* bins;              // [kMaxCandidates][cols], kNoBin past the column's count
			float* jn;                  // [kMaxCandidates][cols]
		};

		struct DetectLayout {
			size_t hist, total, done, picks, quantity, rounds, list, partials, bins, jn, bytes, zero_bytes;
			explicit DetectLayout(size_t cols) {
				size_t at = 0;
				auto take = [&](size_t b) {
					const size_t r = at;
					at = (at + b + 255) / 256 * 256;
					return r;
				};
				hist = take(sizeof(int) * kMaxCandidates * kDetectBins);
				total = take(sizeof(unsigned long long));
				done = take(sizeof(unsigned int));
				zero_bytes = at;  // hist, total and done start at zero
				picks = take(sizeof(int) * kMaxCandidates * 2);
				quantity = take(sizeof(double) * kMaxCandidates);
				rounds = take(sizeof(int));
				list = take(sizeof(DetectionList));
				partials = take(sizeof(double) * kSumCtas * kMaxDetections);
				bins = take(kMaxCandidates * cols);
				jn = take(sizeof(float) * kMaxCandidates * cols);
				bytes = at;
			}
			DetectScratch carve(void* base) const {
				char* b = static_cast<char*>(base);
				return DetectScratch{reinterpret_cast<int*>(b + hist), reinterpret_cast<unsigned long long*>(b + total),
					reinterpret_cast<unsigned int*>(b + done), reinterpret_cast<int*>(b + picks),
					reinterpret_cast<double*>(b + quantity), reinterpret_cast<int*>(b + rounds),
					reinterpret_cast<DetectionList*>(b + list), reinterpret_cast<double*>(b + partials),
					reinterpret_cast<uint8_t*>(b + bins), reinterpret_cast<float*>(b + jn)};
			}
		};

		struct StftParams {
			const float2* x;
			int w, hop;
			int cols;
			int per_cta;           // columns per CTA
			const float* window;   // w floats
			FftPlanDev plan;
			float2* s;             // cols x w spectra
		};

		template <class F>
		__global__ void __launch_bounds__(kJamThreads) stft_kernel(StftParams p) {
			extern __shared__ float2 sm[];
			const int w = fft_n<F>(p.plan.n);
			const int ld = w | 1;
			const int c0 = blockIdx.x * p.per_cta;
			const int nc = min(p.per_cta, p.cols - c0);
			float2* a = sm;
			float2* b = sm + p.per_cta * ld;
			float* win = reinterpret_cast<float*>(sm + 2 * p.per_cta * ld);
			const FftPlanDev plan = F::prepare(p.plan, win + w);
			for (int i = threadIdx.x; i < w; i += blockDim.x)
				win[i] = p.window[i];
			__syncthreads();
			// vec * complex(window, 0) (stft.hpp:55-56): both parts scaled
			for (int e = threadIdx.x; e < nc * w; e += blockDim.x) {
				const int f = e / w, i = e - f * w;
				const float2 v = p.x[static_cast<size_t>(c0 + f) * p.hop + i];
				a[f * ld + i] = c2(__fmul_rn(v.x, win[i]), __fmul_rn(v.y, win[i]));
			}
			__syncthreads();
			const float2* y = F::template run<false>(a, b, plan, nc, ld);
			for (int e = threadIdx.x; e < nc * w; e += blockDim.x) {
				const int f = e / w, i = e - f * w;
				p.s[static_cast<size_t>(c0 + f) * w + i] = y[f * ld + i];
			}
		}

		// 128-point DFT of one column by eight lanes, four columns per warp.  Lane
		// l holds v[j] = x[l + 8 j]: a 16-point DFT over j in registers, the twiddle
		// W_128^{l k1}, one exchange through shared memory, and for the lane's k1 =
		// l and l + 8 an 8-point DFT over the lanes' values; lane l then holds
		// X[l + 8 m] in v[m].  The inverse runs backwards with conjugate twiddles,
		// unnormalised (x 128).  16 stores and 16 loads per lane and four columns,
		// against the 40 two-word shuffles per column of one warp per column.
		// Exchange tiles: element (k1, l) at 9 k1 + l, columns 152 apart, so that
		// half-warps of stores and loads touch every bank once.
		constexpr int kOctetTile = 152;
		struct Octet128 {
			float2 tw[15];   // W_128^{l k1}, k1 = 1..15
			float2* tile;    // the column's exchange tile
			int l;
			__device__ __forceinline__ void init(const float2* __restrict__ table, float2* warp_tiles) {
				const int lane = threadIdx.x & 31;
				l = lane & 7;
				tile = warp_tiles + (lane >> 3) * kOctetTile;
#pragma unroll
				for (int k1 = 1; k1 < 16; ++k1)
					tw[k1 - 1] = __ldg(table + l * k1);
			}
			__device__ __forceinline__ void forward(float2 (&v)[16]) const {
				Dft<16, false>::run(v);
				tile[l] = v[0];
#pragma unroll
				for (int k1 = 1; k1 < 16; ++k1)
					tile[9 * k1 + l] = cmul(v[k1], tw[k1 - 1]);
				__syncwarp();
				float2 a[8], b[8];
#pragma unroll
				for (int i = 0; i < 8; ++i) {
					a[i] = tile[9 * l + i];
					b[i] = tile[9 * (l + 8) + i];
				}
				__syncwarp();  // the next exchange may write
				Dft<8, false>::run(a);
				Dft<8, false>::run(b);
#pragma unroll
				for (int i = 0; i < 8; ++i) {
					v[2 * i] = a[i];
					v[2 * i + 1] = b[i];
				}
			}
			__device__ __forceinline__ void inverse(float2 (&v)[16]) const {
				float2 a[8], b[8];
#pragma unroll
				for (int i = 0; i < 8; ++i) {
					a[i] = v[2 * i];
					b[i] = v[2 * i + 1];
				}
				Dft<8, true>::run(a);
				Dft<8, true>::run(b);
#pragma unroll
				for (int i = 0; i < 8; ++i) {
					tile[9 * l + i] = a[i];
					tile[9 * (l + 8) + i] = b[i];
				}
				__syncwarp();
				v[0] = tile[l];
#pragma unroll
				for (int k1 = 1; k1 < 16; ++k1)
					v[k1] = cmulc(tile[9 * k1 + l], tw[k1 - 1]);
				__syncwarp();
				Dft<16, true>::run(v);
			}
		};

		struct DetectParams {
			const float2* x;       // samples; column c starts at 32 c
			int cols;
			int per_octet;         // columns per octet of lanes and batch
			int batches;           // of 4 per_octet columns
			const float* window;   // 128 Hann coefficients
			const float2* tw;      // W_128^m, m < 128
			DetectScratch det;
		};

		constexpr int kDetectThreads = 64;
		constexpr int kMagStride = 137;   // odd: one thread per column reads without conflicts; 9 modulo 32 spreads the four columns of a store
		constexpr int kDetectWarpBytes = static_cast<int>(sizeof(float2)) * 4 * kOctetTile + static_cast<int>(sizeof(float)) * 32 * (kMagStride + 17);

		// One thread, one column: kMaxCandidates rounds of first-max over the
		// column's magnitudes (the largest, then the lowest bin holding it, as
		// std::max_element), each followed by nulling +-3 bins (NullRegion,
		// jamming_detection.hpp:101-110); then the float mean and unbiased sigma of
		// the nulled magnitudes with SequentialMeanStdDev's formula (src/math/
		// mean_stddev.hpp:29-42; the sums in four interleaved parts) and J/N = peak
		// / sigma.  Candidates with J/N < 6 are erased, the rest kept in order:
		// kept candidate r of column `col` goes to [r][col] and into the CTA's
		// round-r occupation histogram.  The maxima of the 16 groups of eight bins
		// are kept beside the magnitudes, so a round looks at 16 maxima, one group,
		// and the at most two groups that nulling touched.
		__device__ __forceinline__ void detect_column(float* mag, float* group, const DetectScratch& d, size_t col, size_t cols,
			int* s_hist, unsigned int* s_total) {
			// maxima of bit patterns, which order as non-negative floats do and put a
			// NaN above them all (a float maximum passes it over)
			auto bits = [](float m) { return __float_as_uint(m); };
			auto group_max = [&](int g) {
				unsigned int m = bits(mag[8 * g]);
#pragma unroll
				for (int i = 1; i < 8; ++i)
					m = max(m, bits(mag[8 * g + i]));
				group[g] = __uint_as_float(m);
			};
#pragma unroll 4
			for (int g = 0; g < 16; ++g)
				group_max(g);
			int bins[kMaxCandidates];
			float peaks[kMaxCandidates];
#pragma unroll
			for (int r = 0; r < kMaxCandidates; ++r) {
				unsigned int top = bits(group[0]);
				int g = 0;
#pragma unroll
				for (int i = 1; i < 16; ++i) {
					const unsigned int m = bits(group[i]);
					g = m > top ? i : g;
					top = max(top, m);
				}
				int bi = 8 * g + 7;
#pragma unroll
				for (int i = 6; i >= 0; --i)
					bi = bits(mag[8 * g + i]) == top ? 8 * g + i : bi;
				bins[r] = bi;
				peaks[r] = __uint_as_float(top);
#pragma unroll
				for (int i = -kNullHalfWidth; i <= kNullHalfWidth; ++i)
					mag[(bi + i) & (kDetectBins - 1)] = 0.0f;
				if (r + 1 < kMaxCandidates) {
					const int ga = ((bi - kNullHalfWidth) & (kDetectBins - 1)) >> 3, gb = ((bi + kNullHalfWidth) & (kDetectBins - 1)) >> 3;
					group_max(ga);
					if (gb != ga)
						group_max(gb);
				}
			}
			float q[4] = {0.f, 0.f, 0.f, 0.f}, s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
			for (int i = 0; i < kDetectBins; i += 4)
#pragma unroll
				for (int k = 0; k < 4; ++k) {
					const float m = mag[i + k];
					q[k] = __fadd_rn(q[k], __fmul_rn(m, m));
					s[k] = __fadd_rn(s[k], m);
				}
			const float qs = __fadd_rn(__fadd_rn(q[0], q[1]), __fadd_rn(q[2], q[3])), ss = __fadd_rn(__fadd_rn(s[0], s[1]), __fadd_rn(s[2], s[3]));
			const float fw = static_cast<float>(kDetectBins);
			const float var = __fdiv_rn(__fsub_rn(qs, __fdiv_rn(__fmul_rn(ss, ss), fw)), static_cast<float>(kDetectBins - 1));
			const float sigma = __fsqrt_rn(var);
			int c = 0;
#pragma unroll
			for (int r = 0; r < kMaxCandidates; ++r) {
				// double(peak) / double(sigma) < 6 exactly when peak - 6 sigma < 0
				// (two floats' double quotient cannot round onto 6 unless it is 6),
				// and fmaf rounds that difference once, keeping its sign: the
				// reference's double test without FP64 (a NaN stays, as in
				// remove_if(jn < threshold)).  The kept J/N is the float quotient.
				if (!(fmaf(-kJnThreshold, sigma, peaks[r]) < 0.0f)) {
					d.bins[static_cast<size_t>(c) * cols + col] = static_cast<uint8_t>(bins[r]);
					d.jn[static_cast<size_t>(c) * cols + col] = __fdiv_rn(peaks[r], sigma);
					atomicAdd(&s_hist[c * kDetectBins + bins[r]], 1);
					++c;
				}
			}
			for (int r = c; r < kMaxCandidates; ++r)
				d.bins[static_cast<size_t>(r) * cols + col] = kNoBin;
			atomicAdd(s_total, static_cast<unsigned int>(c));
		}

		// JammingDetector's STFT and per-column candidates: a warp takes batches of
		// 4 per_octet consecutive columns (grid-stride), each octet of lanes
		// per_octet (eight, fewer for short signals) of them in a row — a column's
		// samples are the previous one's moved by 32, so only 32 are loaded per
		// column — then each lane one column's candidates.  Bound:
		// issue, and shared memory for the warps in flight.
		__global__ void __launch_bounds__(kDetectThreads) detect_kernel(DetectParams p) {
			extern __shared__ __align__(16) unsigned char raw[];
			__shared__ int s_hist[kMaxCandidates * kDetectBins];
			__shared__ unsigned int s_total;
			for (int e = threadIdx.x; e < kMaxCandidates * kDetectBins; e += blockDim.x)
				s_hist[e] = 0;
			if (threadIdx.x == 0)
				s_total = 0;
			__syncthreads();
			const int lane = threadIdx.x & 31, octet = lane >> 3;
			unsigned char* mine = raw + (threadIdx.x >> 5) * kDetectWarpBytes;
			float* const mags = reinterpret_cast<float*>(mine + sizeof(float2) * 4 * kOctetTile);
			float* const groups = mags + 32 * kMagStride;
			Octet128 fft;
			fft.init(p.tw, reinterpret_cast<float2*>(mine));
			float win[16];
#pragma unroll
			for (int j = 0; j < 16; ++j)
				win[j] = p.window[fft.l + 8 * j];
			const int warps = gridDim.x * (blockDim.x >> 5);
			for (int batch = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); batch < p.batches; batch += warps) {
				const int c0 = (batch * 4 + octet) * p.per_octet;  // the octet's first column
				// samples of the last column on (clamped: columns past the end repeat it)
				const float2* x = p.x + static_cast<size_t>(min(c0, p.cols - 1)) * 32 + fft.l;
				float2 smp[16];
#pragma unroll
				for (int j = 0; j < 12; ++j)
					smp[j + 4] = x[8 * j];
#pragma unroll 1
				for (int i = 0; i < p.per_octet; ++i) {
#pragma unroll
					for (int j = 0; j < 12; ++j)
						smp[j] = smp[j + 4];
					if (c0 + i < p.cols) {
#pragma unroll
						for (int j = 12; j < 16; ++j)
							smp[j] = x[32 * i + 8 * j];
					}
					float2 v[16];
#pragma unroll
					for (int j = 0; j < 16; ++j)  // vec * complex(window, 0) (stft.hpp:55-56): both parts scaled
						v[j] = c2(__fmul_rn(smp[j].x, win[j]), __fmul_rn(smp[j].y, win[j]));
					fft.forward(v);
					float* m = mags + (octet * p.per_octet + i) * kMagStride + fft.l;
#pragma unroll
					for (int j = 0; j < 16; ++j)
						m[8 * j] = __fsqrt_rn(v[j].x * v[j].x + v[j].y * v[j].y);
				}
				__syncwarp();
				const int col = batch * 4 * p.per_octet + lane;
				if (lane < 4 * p.per_octet && col < p.cols)
					detect_column(mags + lane * kMagStride, groups + lane * 17, p.det, static_cast<size_t>(col), static_cast<size_t>(p.cols),
						s_hist, &s_total);
				__syncwarp();  // the next batch writes the magnitudes
			}
			__syncthreads();
			for (int e = threadIdx.x; e < kMaxCandidates * kDetectBins; e += blockDim.x)
				if (s_hist[e])
					atomicAdd(p.det.hist + e, s_hist[e]);
			if (threadIdx.x == 0 && s_total)
				atomicAdd(p.det.total, static_cast<unsigned long long>(s_total));
		}

		struct IstftParams {
			const float2* s;       // cols x w
			int w;
			int cols;
			int per_cta;
			FftPlanDev plan;
			float2* t;             // cols x w inverse columns
		};

		template <class F>
		__global__ void __launch_bounds__(kJamThreads) istft_cols_kernel(IstftParams p) {
			extern __shared__ float2 sm[];
			const int w = fft_n<F>(p.plan.n);
			const int ld = w | 1;
			const int c0 = blockIdx.x * p.per_cta;
			const int nc = min(p.per_cta, p.cols - c0);
			float2* a = sm;
			float2* b = sm + p.per_cta * ld;
			const FftPlanDev plan = F::prepare(p.plan, b + p.per_cta * ld);
			for (int e = threadIdx.x; e < nc * w; e += blockDim.x) {
				const int f = e / w, i = e - f * w;
				a[f * ld + i] = p.s[static_cast<size_t>(c0 + f) * w + i];
			}
			__syncthreads();
			const float2* y = F::template run<true>(a, b, plan, nc, ld);
			// SequentialDft inverse (src/math/dft.hpp:124-129): el /= size; el *= 2
			const float fw = static_cast<float>(w);
			for (int e = threadIdx.x; e < nc * w; e += blockDim.x) {
				const int f = e / w, i = e - f * w;
				const float2 v = y[f * ld + i];
				p.t[static_cast<size_t>(c0 + f) * w + i] =
					c2(__fmul_rn(__fdiv_rn(v.x, fw), 2.0f), __fmul_rn(__fdiv_rn(v.y, fw), 2.0f));
			}
		}

		// dst[i * hop + j] += column_i[j] for i = 0, 1, ... (stft.hpp:69-72)
		// gathered per output sample; samples past the synthesis length are the
		// zeros of the resize to n (jse.hpp:83-85).
		__global__ void overlap_add_kernel(const float2* __restrict__ t, int w, int hop, int cols, uint64_t n,
			float2* __restrict__ out) {
			const uint64_t len = static_cast<uint64_t>(w) + static_cast<uint64_t>(cols - 1) * hop;
			for (uint64_t k = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; k < n;
				 k += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
				float ax = 0.0f, ay = 0.0f;
				if (k < len) {
					const int lo = k >= static_cast<uint64_t>(w) ? static_cast<int>((k - w) / hop) + 1 : 0;
					const int hi = min(cols - 1, static_cast<int>(k / hop));
					for (int i = lo; i <= hi; ++i) {
						const float2 v = t[static_cast<size_t>(i) * w + (k - static_cast<uint64_t>(i) * hop)];
						ax = __fadd_rn(ax, v.x);
						ay = __fadd_rn(ay, v.y);
					}
				}
				out[k] = c2(ax, ay);
			}
		}

		struct WidebandParams {
			const float2* x;       // n input samples
			uint64_t n;
			int cols;
			int slots_per_octet;   // 32-sample output slots per run
			const float* window;
			const float2* tw;      // W_128^m, m < 128
			float2* out;           // n output samples (not x)
		};

		// float(|X|) >= 20 (jse.hpp:43) on the square: the root of the float below
		// 400 is the first to round to 20
		constexpr float kWidebandLevel2 = 0x1.8ffffep+8f;
		constexpr int kWidebandThreads = 128;

		// FilterWideband (jse.hpp:70-87) + OverlapAndAdd + resize to n, eight lanes
		// per run of 32-sample output slots: they walk the covering columns in
		// order (the first slot's three predecessors first), re-transforming each
		// from the samples as the detector did (Octet128; 32 new samples per
		// column), zeroing |.| >= 20, inverse-transforming and scaling (v / 128) *
		// 2; a column's samples 32 q .. belong to slot i + q, so four slot
		// accumulators take the columns in column order, and slot i is complete
		// after column i.  Bound: issue.
		__global__ void __launch_bounds__(kWidebandThreads) wideband_kernel(WidebandParams p) {
			__shared__ __align__(16) float2 tiles[kWidebandThreads / 8 * kOctetTile];
			const int octet = static_cast<int>(threadIdx.x >> 3);
			const long long total_slots = static_cast<long long>((p.n + 31) / 32);
			const long long s0 = (static_cast<long long>(blockIdx.x) * (kWidebandThreads / 8) + octet) * p.slots_per_octet;
			const long long s1 = min(s0 + p.slots_per_octet, total_slots);
			Octet128 fft;
			fft.init(p.tw, tiles + (threadIdx.x >> 5) * (4 * kOctetTile));
			float win[16];
#pragma unroll
			for (int j = 0; j < 16; ++j)
				win[j] = p.window[fft.l + 8 * j];
			// slot i + q's sums, samples fft.l + 8 k of the slot
			float2 acc[4][4];
#pragma unroll
			for (int q = 0; q < 4; ++q)
#pragma unroll
				for (int k = 0; k < 4; ++k)
					acc[q][k] = c2(0.0f, 0.0f);
			auto put = [&](long long s, const float2 (&v)[4]) {
#pragma unroll
				for (int k = 0; k < 4; ++k) {
					const uint64_t at = static_cast<uint64_t>(s) * 32 + fft.l + 8 * k;
					if (at < p.n)
						p.out[at] = v[k];
				}
			};
			const long long i_lo = s0 - 3;  // columns before the first and past the last add nothing
			float2 smp[16];
			{
				const long long first = max(0LL, min(i_lo, static_cast<long long>(p.cols) - 1));
#pragma unroll
				for (int j = 0; j < 12; ++j)
					smp[j + 4] = p.x[static_cast<size_t>(first) * 32 + fft.l + 8 * j];
			}
			// every octet of the warp walks the same number of columns (the
			// exchanges synchronise the warp)
			for (int step = 0; step < p.slots_per_octet + 3; ++step) {
				const long long i = i_lo + step;
				const bool live = i >= 0 && i < p.cols && i < s1;
				// the window moves on from the first column that exists
				if (i > 0) {
#pragma unroll
					for (int j = 0; j < 12; ++j)
						smp[j] = smp[j + 4];
				}
				else {
#pragma unroll
					for (int j = 0; j < 12; ++j)
						smp[j] = i == 0 ? smp[j + 4] : smp[j];
				}
				if (live) {
#pragma unroll
					for (int j = 12; j < 16; ++j)
						smp[j] = p.x[static_cast<size_t>(i) * 32 + fft.l + 8 * j];
				}
				float2 v[16];
#pragma unroll
				for (int j = 0; j < 16; ++j)
					v[j] = c2(__fmul_rn(smp[j].x, win[j]), __fmul_rn(smp[j].y, win[j]));
				fft.forward(v);
#pragma unroll
				for (int j = 0; j < 16; ++j)
					if (v[j].x * v[j].x + v[j].y * v[j].y >= kWidebandLevel2)
						v[j] = c2(0.0f, 0.0f);
				fft.inverse(v);
				if (live) {
					// (v / 128) * 2: exact powers of two
#pragma unroll
					for (int q = 0; q < 4; ++q)
#pragma unroll
						for (int k = 0; k < 4; ++k) {
							const float2 y = v[4 * q + k];
							acc[q][k] = c2(__fadd_rn(acc[q][k].x, __fmul_rn(y.x, 0.015625f)), __fadd_rn(acc[q][k].y, __fmul_rn(y.y, 0.015625f)));
						}
				}
				// slot i is complete; past the last column the synthesis tail (slots
				// cols .. cols + 2), then the zeros of the resize to n
				if (i >= s0 && i < s1)
					put(i, acc[0]);
#pragma unroll
				for (int k = 0; k < 4; ++k) {
					acc[0][k] = acc[1][k];
					acc[1][k] = acc[2][k];
					acc[2][k] = acc[3][k];
					acc[3][k] = c2(0.0f, 0.0f);
				}
			}
		}

		struct NullRange {
			uint64_t start;  // first bin (mod n)
			uint64_t len;
		};
		struct NullParams {
			NullRange r[2 * kMaxCandidates];
			int n_ranges;
		};

		__global__ void null_bins_kernel(float2* x, uint64_t n, NullParams p) {
			for (int d = 0; d < p.n_ranges; ++d)
				for (uint64_t j = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; j < p.r[d].len;
					 j += static_cast<uint64_t>(gridDim.x) * blockDim.x)
					x[(p.r[d].start + j) % n] = c2(0.0f, 0.0f);
		}

		int blocks_for(uint64_t n) {
			return static_cast<int>(std::min<uint64_t>((n + kJamThreads - 1) / kJamThreads, 152 * 16));
		}

		template <class Fn>
		void with_column_fft(int w, Fn&& fn) {
			if (w == 128)
				fn(StaticFft<128, 16, 8>{});
			else
				fn(RuntimeFft{});
		}

		FftPlanDev column_plan(ugsdr_ctx* ctx, int w) {
			const FftPlanDesc& d = get_plan(ctx, w);
			FftPlanDev p{};
			p.n = d.n;
			p.n_pass = d.n_pass;
			for (int i = 0; i < d.n_pass; ++i)
				p.radix[i] = d.radix[i];
			p.tw = d.tw;
			return p;
		}

		// columns per CTA and the shared memory they take: two tiles of
		// per_cta x (w | 1) + the plan's table (w entries) + the window
		int columns_per_cta(ugsdr_ctx* ctx, int w, size_t& smem) {
			const size_t ld = static_cast<size_t>(w | 1);
			int per = 16;
			auto bytes = [&](int c) { return 2 * sizeof(float2) * c * ld + sizeof(float2) * w + 16 + sizeof(float) * w; };
			while (per > 1 && bytes(per) > ctx->smem_optin - 2048)
				per /= 2;
			require(bytes(per) <= ctx->smem_optin - 2048, "STFT window too long for one CTA", UGSDR_E_UNSUPPORTED);
			smem = bytes(per);
			return per;
		}

		// SequentialStft::GetWindow (stft.hpp:34-40): computed in double, stored as float
		const float* hann_window(ugsdr_ctx* ctx, int w) {
			if (ctx->jam_window_len != w) {
				std::vector<float> h(w);
				const double pi = 3.14159265358979323846;
				for (int i = 0; i < w; ++i)
					h[i] = static_cast<float>(0.5 * (1 - std::cos(2.0 * pi * static_cast<double>(i) / w)));
				ctx->jam_window.reserve(sizeof(float) * w);
				UG_CUDA(cudaMemcpyAsync(ctx->jam_window.ptr, h.data(), sizeof(float) * w, cudaMemcpyHostToDevice, ctx->stream));
				UG_CUDA(cudaStreamSynchronize(ctx->stream));
				ctx->jam_window_len = w;
			}
			return ctx->jam_window.as<float>();
		}

		size_t stft_columns(size_t n, int w, int overlap) {
			require(w >= 2 * kNullHalfWidth + 2 && overlap >= 0 && overlap < w, "STFT window must be >= 8 and above the overlap");
			require(n >= static_cast<size_t>(w), "fewer samples than one STFT window");
			const size_t cols = (n - static_cast<size_t>(overlap)) / static_cast<size_t>(w - overlap);
			require(cols <= (1u << 30), "too many STFT columns");
			return cols;
		}

		// STFT of device samples x into ctx->jam_s (the per-op Transform)
		void stft_device(ugsdr_ctx* ctx, const float2* x, size_t cols, int w, int overlap) {
			size_t smem = 0;
			const int per = columns_per_cta(ctx, w, smem);
			ctx->jam_s.reserve(sizeof(float2) * cols * w);
			StftParams p{};
			p.x = x;
			p.w = w;
			p.hop = w - overlap;
			p.cols = static_cast<int>(cols);
			p.per_cta = per;
			p.window = hann_window(ctx, w);
			p.plan = column_plan(ctx, w);
			p.s = ctx->jam_s.as<float2>();
			KernelTimer timer(ctx, "jam_stft");
			with_column_fft(w, [&](auto f) {
				using F = decltype(f);
				UG_CUDA(cudaFuncSetAttribute(stft_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
				stft_kernel<F><<<static_cast<unsigned>((cols + per - 1) / per), kJamThreads, smem, ctx->stream>>>(p);
				note_launch(ctx);
			});
		}

		// inverse columns of ctx->jam_s into ctx->jam_t, overlap-added into n
		// samples at out
		void istft_device(ugsdr_ctx* ctx, size_t cols, int w, int overlap, float2* out, size_t n) {
			size_t smem = 0;
			const int per = columns_per_cta(ctx, w, smem);
			ctx->jam_t.reserve(sizeof(float2) * cols * w);
			IstftParams p{};
			p.s = ctx->jam_s.as<float2>();
			p.w = w;
			p.cols = static_cast<int>(cols);
			p.per_cta = per;
			p.plan = column_plan(ctx, w);
			p.t = ctx->jam_t.as<float2>();
			with_column_fft(w, [&](auto f) {
				using F = decltype(f);
				UG_CUDA(cudaFuncSetAttribute(istft_cols_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
				istft_cols_kernel<F><<<static_cast<unsigned>((cols + per - 1) / per), kJamThreads, smem, ctx->stream>>>(p);
			});
			overlap_add_kernel<<<blocks_for(n), kJamThreads, 0, ctx->stream>>>(ctx->jam_t.as<float2>(), w, w - overlap,
				static_cast<int>(cols), n, out);
			note_launch(ctx, 2);
		}

		// FilterWideband + OverlapAndAdd + resize to n, fused: x -> out
		void wideband_device(ugsdr_ctx* ctx, const float2* x, size_t n, float2* out) {
			WidebandParams p{};
			p.x = x;
			p.n = n;
			p.cols = static_cast<int>(stft_columns(n, kDetectWindow, kDetectOverlap));
			// runs of up to 64 slots (each walks three more columns), of the length
			// that makes whole waves of the CTAs three of which share an SM, two
			// slots at least
			const long long slots = static_cast<long long>((n + 31) / 32);
			const long long wave = static_cast<long long>(ctx->sm_count) * 3 * (kWidebandThreads / 8);  // octets
			const long long waves = (slots + 64 * wave - 1) / (64 * wave);
			p.slots_per_octet = static_cast<int>(std::max<long long>(2, (slots + waves * wave - 1) / (waves * wave)));
			p.window = hann_window(ctx, kDetectWindow);
			p.tw = get_plan(ctx, kDetectWindow).tw;
			p.out = out;
			const long long octets = (slots + p.slots_per_octet - 1) / p.slots_per_octet;
			const long long ctas = (octets + kWidebandThreads / 8 - 1) / (kWidebandThreads / 8);
			require(ctas < (1LL << 31), "signal too long");
			KernelTimer timer(ctx, "jam_wideband");
			wideband_kernel<<<static_cast<unsigned>(ctas), kWidebandThreads, 0, ctx->stream>>>(p);
			note_launch(ctx);
		}

		// deterministic block sum of per-thread doubles (fixed tree order)
		__device__ double block_sum(double v, double* scratch) {
			for (int o = 16; o > 0; o >>= 1)
				v += __shfl_down_sync(0xffffffffu, v, o);
			const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
			__syncthreads();
			if (lane == 0)
				scratch[warp] = v;
			__syncthreads();
			if (warp == 0) {
				v = lane < (blockDim.x >> 5) ? scratch[lane] : 0.0;
				for (int o = 16; o > 0; o >>= 1)
					v += __shfl_down_sync(0xffffffffu, v, o);
				if (lane == 0)
					scratch[0] = v;
			}
			__syncthreads();
			return scratch[0];
		}

		// AnalyzeStftData (jamming_detection.hpp:130-189), decisions.  Round i
		// looks at every column's i-th candidate: its occupation map is keyed
		// by frequency = bin * fs / w, which orders as the bins do, so the
		// reference's walk over the map is a walk over occupied bins in
		// increasing order of the round's histogram.
		// One warp per round, lane l on bins l, l + 32, ...; the walk's state at a
		// bin follows from the ballots of the bins below it.
		__global__ void __launch_bounds__(32 * kMaxCandidates) decide_kernel(DetectScratch d, unsigned long long cols) {
			const int rounds = static_cast<int>(*d.total / cols);
			if (threadIdx.x == 0)
				*d.rounds = rounds;
			const int i = threadIdx.x >> 5, lane = threadIdx.x & 31;
			if (i >= rounds)
				return;
			constexpr int J = kDetectBins / 32;
			int occ[J], sum = 0, occupied = 0;
			unsigned occupied_mask[J];
#pragma unroll
			for (int j = 0; j < J; ++j) {
				occ[j] = d.hist[i * kDetectBins + j * 32 + lane];
				sum += occ[j];
				occupied_mask[j] = __ballot_sync(0xffffffffu, occ[j] != 0);
				occupied += __popc(occupied_mask[j]);
			}
			const double quantity = static_cast<double>(__reduce_add_sync(0xffffffffu, sum));
			int narrow = -1, wide = -1, first = -1;
			unsigned long long cnt_wideband = 0;
#pragma unroll
			for (int j = 0; j < J; ++j) {
				const double probability = occ[j] / quantity;
				const unsigned sure = __ballot_sync(0xffffffffu, occ[j] != 0 && probability >= kProbability);
				unsigned many = __ballot_sync(0xffffffffu, occ[j] != 0 && probability >= kProbability / static_cast<double>(occupied));
				if (first < 0 && occupied_mask[j])
					first = j * 32 + __ffs(static_cast<int>(occupied_mask[j])) - 1;
				if (narrow >= 0)
					continue;  // the walk ended below these bins
				if (sure) {
					narrow = j * 32 + __ffs(static_cast<int>(sure)) - 1;
					many &= (1u << (narrow & 31)) - 1u;
				}
				if (many) {
					cnt_wideband += __popc(many);
					wide = j * 32 + 31 - __clz(static_cast<int>(many));
				}
			}
			if (wide < 0)
				wide = first;  // the reference's pointer starts at the map's first entry
			if (lane == 0) {
				d.picks[2 * i] = narrow;
				// one occupied bin makes the bound 0: reported as wideband too
				d.picks[2 * i + 1] = cnt_wideband >= static_cast<unsigned long long>(occupied * kProbability) ? wide : -1;
				d.quantity[i] = quantity;
			}
		}

		// The reported J/N of each pick: the mean of the round's candidate J/N
		// at that bin.  Per-CTA partial sums over a fixed column split, combined
		// in a fixed tree by the last CTA, which also writes the detection list —
		// deterministic, within rounding of the reference's column-order sum.
		__global__ void __launch_bounds__(kJamThreads) jn_sum_kernel(DetectScratch d, unsigned long long cols, double fs) {
			__shared__ double scratch[32];
			__shared__ bool s_last;
			const int rounds = *d.rounds;
			for (int i = 0; i < rounds; ++i)
				for (int k = 0; k < 2; ++k) {
					const int b = d.picks[2 * i + k];
					if (b < 0)
						continue;
					double part = 0;
					const uint8_t* bins = d.bins + static_cast<size_t>(i) * cols;
					const float* jn = d.jn + static_cast<size_t>(i) * cols;
					for (unsigned long long c = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; c < cols;
						 c += static_cast<unsigned long long>(gridDim.x) * blockDim.x)
						if (bins[c] == b)
							part += jn[c];
					const double sum = block_sum(part, scratch);
					if (threadIdx.x == 0)
						d.partials[blockIdx.x * kMaxDetections + 2 * i + k] = sum;
				}
			__syncthreads();
			if (threadIdx.x == 0) {
				__threadfence();
				s_last = atomicAdd(d.done, 1u) == gridDim.x - 1;
			}
			__syncthreads();
			if (!s_last)
				return;
			__threadfence();
			int n = 0;
			for (int i = 0; i < rounds; ++i)
				for (int k = 0; k < 2; ++k) {
					const int b = d.picks[2 * i + k];
					if (b < 0 || n >= kMaxDetections)
						continue;
					double part = 0;
					for (unsigned int g = threadIdx.x; g < gridDim.x; g += blockDim.x)
						part += __ldcg(d.partials + g * kMaxDetections + 2 * i + k);
					const double sum = block_sum(part, scratch);
					if (threadIdx.x != 0) {
						++n;
						continue;
					}
					Detection& out = d.list->d[n++];
					out.type = k == 0 ? UGSDR_INTERFERENCE_NARROWBAND : UGSDR_INTERFERENCE_WIDEBAND;
					out.bin = b;
					out.frequency = static_cast<double>(b) * fs / static_cast<double>(kDetectBins);
					out.jn = sum / d.quantity[i];
				}
			if (threadIdx.x == 0)
				d.list->n = n;
		}

		// detector over device samples x (n): STFT + candidates, decisions and
		// J/N sums on the device; only the detection list comes back
		std::vector<Detection> detect_device(ugsdr_ctx* ctx, const float2* x, size_t n, double fs) {
			require(fs > 0, "sampling rate must be positive");
			const size_t cols = stft_columns(n, kDetectWindow, kDetectOverlap);
			const DetectLayout lay(cols);
			ctx->jam_cand.reserve(lay.bytes);
			const DetectScratch d = lay.carve(ctx->jam_cand.ptr);
			UG_CUDA(cudaMemsetAsync(ctx->jam_cand.ptr, 0, lay.zero_bytes, ctx->stream));
			DetectParams dp{};
			dp.x = x;
			dp.cols = static_cast<int>(cols);
			// fewer columns in a row as long as one wave of warps (eight per SM) holds them:
			// 4,474 columns 17 us by eight in a row, 9 one at a time
			dp.per_octet = 8;
			while (dp.per_octet > 1 && cols <= static_cast<size_t>(2 * dp.per_octet) * 8 * ctx->sm_count)
				dp.per_octet /= 2;
			dp.batches = static_cast<int>((cols + 4 * dp.per_octet - 1) / (4 * dp.per_octet));
			dp.window = hann_window(ctx, kDetectWindow);
			dp.tw = get_plan(ctx, kDetectWindow).tw;
			dp.det = d;
			{
				KernelTimer timer(ctx, "jam_stft_detect");
				constexpr int kWarps = kDetectThreads / 32;
				const size_t smem = static_cast<size_t>(kWarps) * kDetectWarpBytes;
				UG_CUDA(cudaFuncSetAttribute(detect_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
				const int ctas = std::min((dp.batches + kWarps - 1) / kWarps, ctx->sm_count * 16);
				detect_kernel<<<ctas, kDetectThreads, smem, ctx->stream>>>(dp);
			}
			note_launch(ctx);
			decide_kernel<<<1, 32 * kMaxCandidates, 0, ctx->stream>>>(d, cols);
			jn_sum_kernel<<<kSumCtas, kJamThreads, 0, ctx->stream>>>(d, cols, fs);
			note_launch(ctx, 2);
			DetectionList host{};
			UG_CUDA(cudaMemcpyAsync(&host, d.list, sizeof(DetectionList), cudaMemcpyDeviceToHost, ctx->stream));
			UG_CUDA(cudaStreamSynchronize(ctx->stream));
			return std::vector<Detection>(host.d, host.d + std::min(host.n, kMaxDetections));
		}

		void report(const std::vector<Detection>& det, ugsdr_jamming_detection* out, int cap, int* n_detections) {
			if (n_detections)
				*n_detections = static_cast<int>(det.size());
			for (int i = 0; out && i < cap && i < static_cast<int>(det.size()); ++i) {
				out[i].type = det[i].type;
				out[i].frequency_bin = det[i].bin;
				out[i].frequency = det[i].frequency;
				out[i].jammer_to_noise = det[i].jn;
			}
		}

		// the samples on the device: the caller's pointer or a staged copy
		float2* stage(ugsdr_ctx* ctx, const float* iq, size_t n, int on_device) {
			require(iq != nullptr && n > 0, "null or empty signal");
			if (on_device)
				return reinterpret_cast<float2*>(const_cast<float*>(iq));
			ctx->jam_x.reserve(sizeof(float2) * n);
			UG_CUDA(cudaMemcpyAsync(ctx->jam_x.ptr, iq, sizeof(float2) * n, cudaMemcpyHostToDevice, ctx->stream));
			return ctx->jam_x.as<float2>();
		}
	}
}

using namespace ugsdr_gpu;

#define UG_JAM_ENTRY(ctx) \
	if (!(ctx))           \
		return UGSDR_E_INVALID; \
	std::lock_guard<std::mutex> lock_((ctx)->mutex); \
	return guarded((ctx), [&]

extern "C" {

int ugsdr_stft(ugsdr_ctx* ctx, const float* in_iq, size_t n, int window_length, int overlap_length, float* out_iq,
	size_t* n_columns) {
	UG_JAM_ENTRY(ctx) {
		require(in_iq != nullptr, "null signal");
		const size_t cols = stft_columns(n, window_length, overlap_length);
		if (n_columns)
			*n_columns = cols;
		if (!out_iq)
			return;
		const float2* x = stage(ctx, in_iq, n, 0);
		stft_device(ctx, x, cols, window_length, overlap_length);
		UG_CUDA(cudaMemcpyAsync(out_iq, ctx->jam_s.ptr, sizeof(float2) * cols * window_length, cudaMemcpyDeviceToHost, ctx->stream));
		UG_CUDA(cudaStreamSynchronize(ctx->stream));
	});
}

int ugsdr_istft(ugsdr_ctx* ctx, const float* in_iq, size_t n_columns, int window_length, int overlap_length,
	float* out_iq) {
	UG_JAM_ENTRY(ctx) {
		require(in_iq && out_iq && n_columns > 0, "null or empty columns");
		require(window_length >= 2 * kNullHalfWidth + 2 && overlap_length >= 0 && overlap_length < window_length,
			"STFT window must be >= 8 and above the overlap");
		const size_t w = static_cast<size_t>(window_length);
		const size_t len = w + (n_columns - 1) * (w - overlap_length);
		ctx->jam_s.reserve(sizeof(float2) * n_columns * w);
		UG_CUDA(cudaMemcpyAsync(ctx->jam_s.ptr, in_iq, sizeof(float2) * n_columns * w, cudaMemcpyHostToDevice, ctx->stream));
		ctx->jam_x.reserve(sizeof(float2) * len);
		istft_device(ctx, n_columns, window_length, overlap_length, ctx->jam_x.as<float2>(), len);
		UG_CUDA(cudaMemcpyAsync(out_iq, ctx->jam_x.ptr, sizeof(float2) * len, cudaMemcpyDeviceToHost, ctx->stream));
		UG_CUDA(cudaStreamSynchronize(ctx->stream));
	});
}

int ugsdr_jamming_detect(ugsdr_ctx* ctx, const float* iq, size_t n, double fs, int samples_on_device,
	ugsdr_jamming_detection* out, int cap, int* n_detections) {
	UG_JAM_ENTRY(ctx) {
		const float2* x = stage(ctx, iq, n, samples_on_device);
		report(detect_device(ctx, x, n, fs), out, cap, n_detections);
	});
}

int ugsdr_jamming_suppress(ugsdr_ctx* ctx, float* iq, size_t n, double fs, int samples_on_device,
	ugsdr_jamming_detection* out, int cap, int* n_detections) {
	UG_JAM_ENTRY(ctx) {
		float2* x = stage(ctx, iq, n, samples_on_device);
		const std::vector<Detection> det = detect_device(ctx, x, n, fs);
		report(det, out, cap, n_detections);
		if (det.empty())
			return;
		const bool wideband = std::any_of(det.begin(), det.end(), [](const Detection& d) { return d.type == UGSDR_INTERFERENCE_WIDEBAND; });
		if (wideband) {
			// out of place (a tile reads its neighbours' inputs), then back
			ctx->jam_t.reserve(sizeof(float2) * n);
			wideband_device(ctx, x, n, ctx->jam_t.as<float2>());
			if (samples_on_device)
				UG_CUDA(cudaMemcpyAsync(x, ctx->jam_t.ptr, sizeof(float2) * n, cudaMemcpyDeviceToDevice, ctx->stream));
			else
				x = ctx->jam_t.as<float2>();
		}
		else {
			// idx = size_t(frequency / fs * n); zero [idx - 128 + n, idx + 128]
			// (+ n when that wraps) modulo n (jse.hpp:50-59, 64-66)
			require(det.size() <= 2 * kMaxCandidates, "too many narrowband detections");
			NullParams np{};
			np.n_ranges = static_cast<int>(det.size());
			const long long nn = static_cast<long long>(n);
			for (size_t i = 0; i < det.size(); ++i) {
				const long long idx = static_cast<long long>(static_cast<size_t>(det[i].frequency / fs * static_cast<double>(n)));
				const long long start = idx - kNarrowNull + nn;
				long long finish = idx + kNarrowNull;
				if (finish < start)
					finish += nn;
				np.r[i].start = static_cast<uint64_t>(start);
				np.r[i].len = finish >= start ? static_cast<uint64_t>(finish - start + 1) : 0;
			}
			ctx->jam_t.reserve(sizeof(float2) * n);
			float2* spec = ctx->jam_t.as<float2>();
			dft_scaled(ctx, x, spec, n, false, ctx->jam_tmp);
			null_bins_kernel<<<blocks_for(2 * kNarrowNull + 1), kJamThreads, 0, ctx->stream>>>(spec, n, np);
			note_launch(ctx);
			dft_scaled(ctx, spec, x, n, true, ctx->jam_tmp);
		}
		if (!samples_on_device)
			UG_CUDA(cudaMemcpyAsync(iq, x, sizeof(float2) * n, cudaMemcpyDeviceToHost, ctx->stream));
		UG_CUDA(cudaStreamSynchronize(ctx->stream));
	});
}
}
