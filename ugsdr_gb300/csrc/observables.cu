// Tracking outputs -> measurements on the device (src/measurements/
// observable.hpp), for every channel of a tracking bank at once, reading the
// bank's n_epochs x n_channels output array where the bank left it.
//
//   sign_bits_kernel  the sign of the prompt I, one bit per epoch, channel by
//                     channel (adjacent threads on adjacent channels)
//   preamble_kernel   FindPreambleGps / FindPreambleGlonass's candidate
//                     search (observable.hpp:204-220, 260-277): the signs
//                     circularly correlated with the preamble upsampled to 1 ms,
//                     epochs above the threshold listed in order.  One CTA per
//                     channel over tiles of epochs; a correlation of +-1 values
//                     is the length less twice the bits that differ, exact.
//   obs_sums_kernel   one thread per (segment of epochs, channel), adjacent
//                     threads on adjacent channels: the carrier-phase increments
//                     summed per segment, and the prompt Q copied channel by channel
//   obs_sigma_kernel  CalculateSnr's sigma (observable.hpp:55-72): the
//                     reference's SequentialMeanStdDev over the prompt Q in
//                     float, in epoch order (mean_stddev.hpp:29-42), one warp
//                     per channel; and the segments' exclusive prefix sums
//   obs_emit_kernel   per epoch the unwrapped phase (prefix + running sum,
//                     snapped to the bank's wrapped 64-bit phase), pseudorange,
//                     pseudophase, Doppler and SNR (the Observable constructor,
//                     75-88), one thread per (segment, channel)
#include "internal.hpp"

#include <algorithm>
#include <cmath>
#include <vector>

namespace ugsdr_gpu {
	namespace {
		constexpr int kObsThreads = 256;
		constexpr int kObsWarps = kObsThreads / 32;
		constexpr int kPreambleTile = 8192;    // epochs per CTA pass: one 32-epoch word per thread
		constexpr int kMinSegment = 16;        // epochs per thread of the sums and the emit pass
		constexpr int kMaxSegment = 128;       // (a multiple of kObsUnroll)
		constexpr int kSegmentThreads = 64;    // per CTA of the sums and the emit pass: small, for an even last wave
		constexpr int kObsUnroll = 8;          // epochs whose loads are in flight per thread
		constexpr int kMaxPreambleLen = 400;   // symbols x upsampling, GLONASS
		constexpr double kTwoPi = 6.283185307179586476925286766559;
		constexpr double kInvTwoPi = 1.0 / kTwoPi;

		// Preambles as +-1 symbols per 20 ms (GPS) or 10 ms (GLONASS):
		// GetPreambleGps (observable.hpp:92-94), the LNAV preamble 10001011;
		// GetPreambleGlonass (143-146), the 30-chip time mark followed by ten
		// meander symbols.  Thresholds on |matched filter| from 219 and 276.
		__constant__ signed char kGpsPreamble[8] = {1, -1, -1, -1, 1, -1, 1, 1};
		__constant__ signed char kGloPreamble[40] = {
			-1, -1, -1, -1, -1, 1, 1, 1, -1, -1, 1, -1, -1, -1, 1, -1, 1, -1, 1, 1,
			1, 1, -1, 1, 1, -1, 1, -1, -1, 1, 1, -1, 1, -1, 1, -1, 1, -1, -1, 1};

		struct PreambleParams {
			const uint32_t* bits;           // [channel][words]: bit e % 32 of word e / 32 set when the prompt I of epoch e is > 0
			int words;                      // per channel
			int n_epochs, n_channels;
			const int* messages;            // per channel, ugsdr_nav_message
			int* counts;                    // per channel
			int* indexes;                   // [channel][cap]
			int cap;
		};

		// One thread per (32 epochs, channel), adjacent threads on adjacent
		// channels: a warp's loads of one epoch cover a contiguous 2.8 KB piece of
		// the record array, eight epochs in flight.  Bound: HBM, one 32-byte sector
		// per record.
		__global__ void __launch_bounds__(kObsThreads) sign_bits_kernel(const ugsdr_track_output* out, int n_epochs, int n_channels,
			int words, uint32_t* bits) {
			const long long t = static_cast<long long>(blockIdx.x) * kObsThreads + threadIdx.x;
			if (t >= static_cast<long long>(words) * n_channels)
				return;
			const int w = static_cast<int>(t / n_channels), c = static_cast<int>(t - static_cast<long long>(w) * n_channels);
			const int e0 = w * 32, cnt = min(32, n_epochs - e0);
			const ugsdr_track_output* r = out + static_cast<size_t>(e0) * n_channels + c;
			uint32_t b = 0;
#pragma unroll 8
			for (int k = 0; k < cnt; ++k)
				b |= (r[static_cast<size_t>(k) * n_channels].taps[2][0] > 0.f ? 1u : 0u) << k;
			bits[static_cast<size_t>(c) * words + w] = b;
		}

		// the 32 signs from epoch `pos` on (0 <= pos < 2 n), circular over n epochs
		__device__ __forceinline__ uint32_t circular_word(const uint32_t* row, int n, long long pos) {
			if (pos >= n)
				pos %= n;
			const int at = static_cast<int>(pos);
			if (at + 32 <= n) {
				const int i = at >> 5, sh = at & 31;
				return sh ? __funnelshift_r(row[i], row[i + 1], sh) : row[i];
			}
			uint32_t b = 0;
			for (int k = 0; k < 32; ++k) {
				const int e = (at + k) % n;
				b |= ((row[e >> 5] >> (e & 31)) & 1u) << k;
			}
			return b;
		}

		__global__ void __launch_bounds__(kObsThreads) preamble_kernel(PreambleParams p) {
			constexpr int kPatternWords = (kMaxPreambleLen + 31) / 32;
			__shared__ uint32_t win[kPreambleTile / 32 + kPatternWords + 1];
			__shared__ uint32_t hits[kPreambleTile / 32];
			__shared__ uint32_t pattern[kPatternWords], valid[kPatternWords];
			__shared__ int warp_hits[kObsWarps];
			const int c = blockIdx.x;
			const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
			const bool glonass = p.messages[c] == UGSDR_NAV_GLONASS;
			const int n_sym = glonass ? 40 : 8;
			const int up = glonass ? 10 : 20;
			const int threshold = glonass ? 370 : 153;
			const int n = p.n_epochs;
			// the preamble is cut to the prompt's length (preamble.resize(size))
			const int len = min(n_sym * up, n);
			const int pattern_words = (len + 31) / 32;
			const uint32_t* row = p.bits + static_cast<size_t>(c) * p.words;
			if (threadIdx.x < pattern_words) {
				uint32_t b = 0, v = 0;
				for (int k = 0; k < 32; ++k) {
					const int m = threadIdx.x * 32 + k;
					if (m < len) {
						const int q = m / up;
						b |= ((glonass ? kGloPreamble[q] : kGpsPreamble[q]) > 0 ? 1u : 0u) << k;
						v |= 1u << k;
					}
				}
				pattern[threadIdx.x] = b;
				valid[threadIdx.x] = v;
			}
			int found = 0;  // candidates so far, the same in every thread
			for (int k0 = 0; k0 < n; k0 += kPreambleTile) {
				__syncthreads();  // the previous tile's readers are done
				const int tile = min(kPreambleTile, n - k0);
				const int load = (tile + 31) / 32 + pattern_words + 1;
				for (int t = threadIdx.x; t < load; t += kObsThreads)
					win[t] = circular_word(row, n, static_cast<long long>(k0) + 32 * t);
				__syncthreads();
				for (int t = threadIdx.x; t < kPreambleTile; t += kObsThreads) {
					bool hit = false;
					if (t < tile) {
						// y[k] = 2 sum_m x[(k + m) mod n] p[m] (the 2/N inverse
						// of the reference's FFT matched filter)
						const int sh = t & 31;
						const uint32_t* x = win + (t >> 5);
						int differ = 0;
						uint32_t lo = x[0];
						for (int w = 0; w < pattern_words; ++w) {
							const uint32_t hi = x[w + 1];
							differ += __popc((__funnelshift_r(lo, hi, sh) ^ pattern[w]) & valid[w]);
							lo = hi;
						}
						hit = 2 * abs(len - 2 * differ) > threshold;
					}
					const unsigned mask = __ballot_sync(0xffffffffu, hit);
					if (lane == 0)
						hits[t >> 5] = mask;
				}
				__syncthreads();
				// one word per thread: its position from the counts before it
				const uint32_t mine = hits[threadIdx.x];
				const int count = __popc(mine);
				int scan = count;
				for (int o = 1; o < 32; o <<= 1) {
					const int up_count = __shfl_up_sync(0xffffffffu, scan, o);
					if (lane >= o)
						scan += up_count;
				}
				if (lane == 31)
					warp_hits[warp] = scan;
				__syncthreads();
				int pos = found + scan - count;
				for (int w = 0; w < kObsWarps; ++w) {
					pos += w < warp ? warp_hits[w] : 0;
					found += warp_hits[w];
				}
				for (uint32_t left = mine; left; left &= left - 1, ++pos)
					if (pos < p.cap)
						p.indexes[static_cast<size_t>(c) * p.cap + pos] = k0 + static_cast<int>(threadIdx.x) * 32 + __ffs(static_cast<int>(left)) - 1;
			}
			if (threadIdx.x == 0)
				p.counts[c] = found;
		}
		static_assert(kPreambleTile == 32 * kObsThreads, "one word of hits per thread");

		// per channel, precomputed on the host
		struct ObsChannel {
			double samples_to_ms;   // 1000 / sampling_rate
			double windup;          // intermediate_frequency / 1e3
			double intermediate_frequency;
			double phase0;          // carrier phase before epoch 0, cycles
			double frequency0;      // carrier frequency before epoch 0, Hz
			double correction;      // range_correction_ms
			long long position;     // preamble_position
		};

		struct ObsParams {
			const ugsdr_track_output* out;  // [epoch][channel]
			int n_epochs, n_channels, n_segments, segment;
			int q_stride;                   // epochs rounded up to a multiple of kObsUnroll
			const ObsChannel* ch;
			float* q;                       // prompt Q, [channel][q_stride]
			float* sigma;                   // per channel
			double* segsum;                 // [segment][channel]: sums, then exclusive prefixes
			ugsdr_observable* obs;          // [epoch][channel]
		};

		__device__ __forceinline__ const ugsdr_track_output& rec(const ObsParams& p, int e, int c) {
			return p.out[static_cast<size_t>(e) * p.n_channels + c];
		}

		// cycles the loop advanced the carrier phase at epoch e: UpdatePhase
		// with the frequency before the epoch's update (2 pi f / 1000 rad),
		// then Pll's phase_error * pi / 2 rad (tracking_parameters.hpp:163-165,
		// 495-511); f: the frequency after epoch e - 1
		__device__ __forceinline__ double phase_step(double phase, double f, double phase_error) {
			return fma(phase_error, 0.25, fma(f, 1e-3, phase));
		}

		// (double)x by integer operations: the conversion instruction runs on the
		// FP64 pipe, which bounds the emit pass
		__device__ __forceinline__ double widen(float x) {
			const uint32_t b = __float_as_uint(x), e = (b >> 23) & 0xFFu;
			if (e == 0u || e == 0xFFu)
				return static_cast<double>(x);  // zeros, subnormals, infinities, NaN
			return __hiloint2double(static_cast<int>((b & 0x80000000u) | (((b & 0x7FFFFFFFu) >> 3) + (896u << 20))), static_cast<int>(b << 29));
		}

		// The frequency before the first epoch of a thread's segment.
		__device__ __forceinline__ double start_frequency(const ObsParams& p, int e0, int c) {
			return e0 == 0 ? p.ch[c].frequency0 : rec(p, e0 - 1, c).carrier_frequency;
		}

		// Threads on adjacent channels read adjacent 88-byte records, so a
		// warp's loads of one field cover a contiguous 2.8 KB row piece (the
		// emit pass with lanes over epochs, 22.5 KB apart, took 677 us for 256
		// channels x 60,000 epochs, this way 438); kObsUnroll epochs' loads are in
		// flight per thread.  Bound: HBM (235 us, 86 % of its peak).
		__global__ void __launch_bounds__(kSegmentThreads) obs_sums_kernel(ObsParams p) {
			const long long t = static_cast<long long>(blockIdx.x) * kSegmentThreads + threadIdx.x;
			if (t >= static_cast<long long>(p.n_channels) * p.n_segments)
				return;
			const int g = static_cast<int>(t / p.n_channels), c = static_cast<int>(t - static_cast<long long>(g) * p.n_channels);
			const int e0 = g * p.segment, e1 = min(p.n_epochs, e0 + p.segment);
			double f = start_frequency(p, e0, c), s = 0.0;
			float* q = p.q + static_cast<size_t>(c) * p.q_stride;
			for (int e = e0; e < e1; e += kObsUnroll) {
				float qv[kObsUnroll];
				double fv[kObsUnroll], pv[kObsUnroll];
#pragma unroll
				for (int u = 0; u < kObsUnroll; ++u) {
					const bool in = e + u < e1;
					const ugsdr_track_output& r = rec(p, in ? e + u : e, c);
					qv[u] = in ? r.taps[2][1] : 0.f;
					fv[u] = r.carrier_frequency;
					pv[u] = r.phase_error;
				}
#pragma unroll
				for (int u = 0; u < kObsUnroll; ++u)
					if (e + u < e1) {
						s = phase_step(s, f, pv[u]);
						f = fv[u];
					}
				float4* q4 = reinterpret_cast<float4*>(q + e);
				q4[0] = make_float4(qv[0], qv[1], qv[2], qv[3]);
				q4[1] = make_float4(qv[4], qv[5], qv[6], qv[7]);
			}
			p.segsum[t] = s;
		}

		// One warp per channel, launched as 2-warp CTAs so the channels spread
		// over every SM.  Bound: the dependent adds in epoch order.  Before them
		// the warp turns its channel's segment sums into exclusive prefixes (each
		// lane a run of segments).
		constexpr int kSigmaWarps = 2;
		constexpr int kSigmaTile = 1024;
		__global__ void __launch_bounds__(32 * kSigmaWarps) obs_sigma_kernel(ObsParams p) {
			__shared__ __align__(16) float s_tiles[kSigmaWarps][2 * kSigmaTile];
			const int c = blockIdx.x * kSigmaWarps + (threadIdx.x >> 5);
			const int lane = threadIdx.x & 31;
			if (c >= p.n_channels)
				return;
			{
				const int run = (p.n_segments + 31) / 32;
				const int g0 = min(lane * run, p.n_segments), g1 = min(g0 + run, p.n_segments);
				double total = 0.0;
				for (int g = g0; g < g1; ++g)
					total += p.segsum[static_cast<size_t>(g) * p.n_channels + c];
				double scan = total;
				for (int o = 1; o < 32; o <<= 1) {
					const double up = __shfl_up_sync(0xffffffffu, scan, o);
					if (lane >= o)
						scan += up;
				}
				double before = __shfl_up_sync(0xffffffffu, scan, 1);
				if (lane == 0)
					before = 0.0;
				for (int g = g0; g < g1; ++g) {
					double* at = p.segsum + static_cast<size_t>(g) * p.n_channels + c;
					const double s = *at;
					*at = before;
					before += s;
				}
			}
			// tiles of kSigmaTile epochs, the next one's copy in flight behind the
			// current one's adds; every lane reads the same four epochs at a time
			// (broadcast) and replays the same serial adds.  60,000 epochs of 256
			// channels: 223 us, 308 with shuffles of strided record loads; squares
			// formed ahead by the lanes side by side (254) and one packed add for
			// both sums (296) were slower.
			const int n = p.n_epochs;
			const float* qc = p.q + static_cast<size_t>(c) * p.q_stride;
			float* const tiles = s_tiles[threadIdx.x >> 5];
			auto copy = [&](int t) {
				const int e0 = t * kSigmaTile, cnt = min(kSigmaTile, p.q_stride - e0);
				float* dst = tiles + (t & 1) * kSigmaTile;
				for (int e = 4 * lane; e < cnt; e += 128) {
					const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst + e));
					asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(qc + e0 + e));
				}
				asm volatile("cp.async.commit_group;\n" ::);
			};
			float q = 0.f, m = 0.f;
			copy(0);
			for (int t = 0; t * kSigmaTile < n; ++t) {
				if ((t + 1) * kSigmaTile < n) {
					copy(t + 1);
					asm volatile("cp.async.wait_group 1;\n" ::: "memory");
				}
				else {
					asm volatile("cp.async.wait_group 0;\n" ::: "memory");
				}
				__syncwarp();
				const float* x = tiles + (t & 1) * kSigmaTile;
				const int cnt = min(kSigmaTile, n - t * kSigmaTile);
				int e = 0;
				for (; e + 32 <= cnt; e += 32) {
					float4 v[8];
#pragma unroll
					for (int k = 0; k < 8; ++k)
						v[k] = *reinterpret_cast<const float4*>(x + e + 4 * k);
#pragma unroll
					for (int k = 0; k < 8; ++k) {
						const float y[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
						for (int i = 0; i < 4; ++i) {
							q = __fadd_rn(q, __fmul_rn(y[i], y[i]));
							m = __fadd_rn(m, y[i]);
						}
					}
				}
				for (; e < cnt; ++e) {
					q = __fadd_rn(q, __fmul_rn(x[e], x[e]));
					m = __fadd_rn(m, x[e]);
				}
				__syncwarp();  // the tile after next is copied over this one
			}
			if (lane == 0) {
				float s = 0.f;
				if (n >= 2) {
					const float nf = static_cast<float>(n);
					const float var = __fdiv_rn(__fsub_rn(q, __fdiv_rn(__fmul_rn(m, m), nf)), static_cast<float>(n - 1));
					s = __fsqrt_rn(var);
				}
				p.sigma[c] = s;
			}
		}

		// Bound: the FP64 pipe (two lanes per SM and cycle) beside HBM: eight FP64
		// operations per record at a zero IF.  Twelve, in 256-thread CTAs that left
		// a nearly empty last wave, took 603 us for 256 channels x 60,000 epochs
		// with the pipe 85 % active.
		__global__ void __launch_bounds__(kSegmentThreads) obs_emit_kernel(ObsParams p) {
			const long long t = static_cast<long long>(blockIdx.x) * kSegmentThreads + threadIdx.x;
			if (t >= static_cast<long long>(p.n_channels) * p.n_segments)
				return;
			const int g = static_cast<int>(t / p.n_channels), c = static_cast<int>(t - static_cast<long long>(g) * p.n_channels);
			const int e0 = g * p.segment, e1 = min(p.n_epochs, e0 + p.segment);
			const ObsChannel ch = p.ch[c];
			// Observable: pseudorange_offset = int32(code_phases[position] * samples_to_ms_rate)
			const double range_offset = static_cast<double>(__double2int_rz(__dmul_rn(rec(p, static_cast<int>(ch.position), c).code_phase,
				ch.samples_to_ms)));
			const float sigma = p.sigma[c];
			const bool no_if = ch.intermediate_frequency == 0.0;
			double f = start_frequency(p, e0, c);
			// phase before the segment: channel start + the earlier segments
			double approx = p.segsum[t] + ch.phase0;
			constexpr int U = kObsUnroll / 2;
			for (int e = e0; e < e1; e += U) {
				float iv[U];
				double fv[U], wv[U], cv[U], pv[U];
#pragma unroll
				for (int u = 0; u < U; ++u) {
					const ugsdr_track_output& r = rec(p, min(e + u, e1 - 1), c);
					iv[u] = r.taps[2][0];
					fv[u] = r.carrier_frequency;
					wv[u] = r.carrier_phase;
					cv[u] = r.code_phase;
					pv[u] = r.phase_error;
				}
#pragma unroll
				for (int u = 0; u < U; ++u) {
					if (e + u >= e1)
						break;
					approx = phase_step(approx, f, pv[u]);  // within far less than half a cycle
					f = fv[u];
					// the bank keeps the phase as a 64-bit fraction of a cycle: its
					// whole cycles come from the running sum (the fraction is the
					// carrier phase times 1 / 2 pi)
					const double whole = rint(fma(-wv[u], kInvTwoPi, approx));
					ugsdr_observable o;
					o.pseudorange = __dadd_rn(__dsub_rn(__dmul_rn(cv[u], ch.samples_to_ms), range_offset), ch.correction);
					// phases[i] = -carrier_phase / 2 pi, plus (i + 1) * IF / 1e3, which
					// at a zero IF adds nothing
					o.pseudophase = fma(-wv[u], kInvTwoPi, -whole);
					if (!no_if)
						o.pseudophase = __dadd_rn(o.pseudophase, __dmul_rn(static_cast<double>(e + u + 1), ch.windup));
					o.doppler = no_if ? f : __dsub_rn(f, ch.intermediate_frequency);
					// 27 + 20 * std::log10(|I| / sigma), all in float
					const float ratio = __fdiv_rn(fabsf(iv[u]), sigma);
					o.snr = widen(__fadd_rn(27.f, __fmul_rn(20.f, log10f(ratio))));
					p.obs[static_cast<size_t>(e + u) * p.n_channels + c] = o;
				}
			}
		}

		// device copy of the bank outputs (or the caller's device pointer)
		const ugsdr_track_output* stage_outputs(ugsdr_ctx* ctx, const ugsdr_track_output* outputs, int on_device,
			size_t records) {
			if (on_device)
				return outputs;
			ctx->obs_in.reserve(sizeof(ugsdr_track_output) * records);
			UG_CUDA(cudaMemcpyAsync(ctx->obs_in.ptr, outputs, sizeof(ugsdr_track_output) * records,
				cudaMemcpyHostToDevice, ctx->stream));
			return ctx->obs_in.as<ugsdr_track_output>();
		}
	}
}

using namespace ugsdr_gpu;

#define UG_OBS_ENTRY(ctx) \
	if (!(ctx))           \
		return UGSDR_E_INVALID; \
	std::lock_guard<std::mutex> lock_((ctx)->mutex); \
	return guarded((ctx), [&]

extern "C" {

int ugsdr_preamble_search(ugsdr_ctx* ctx, const ugsdr_track_output* outputs, int outputs_on_device, int n_epochs,
	int n_channels, const int* messages, int* counts, int* indexes, int cap) {
	UG_OBS_ENTRY(ctx) {
		require(outputs && messages && counts, "null outputs, messages or counts");
		require(n_epochs >= 1 && n_epochs <= (1 << 30) && n_channels >= 1, "bad output array shape");
		require(cap >= 0 && (cap == 0 || indexes), "null indexes");
		for (int c = 0; c < n_channels; ++c)
			require(messages[c] == UGSDR_NAV_GPS_LNAV || messages[c] == UGSDR_NAV_GLONASS, "unknown navigation message");
		const size_t records = static_cast<size_t>(n_epochs) * n_channels;
		const ugsdr_track_output* d_out = stage_outputs(ctx, outputs, outputs_on_device, records);
		const size_t list_bytes = sizeof(int) * static_cast<size_t>(n_channels) * cap;
		const int words = (n_epochs + 31) / 32;
		const size_t word_threads = static_cast<size_t>(words) * n_channels;
		ctx->obs_tmp.reserve(sizeof(int) * 2 * static_cast<size_t>(n_channels) + list_bytes + sizeof(uint32_t) * word_threads + 16);
		int* d_msg = ctx->obs_tmp.as<int>();
		int* d_counts = d_msg + n_channels;
		int* d_idx = d_counts + n_channels;
		uint32_t* d_bits = reinterpret_cast<uint32_t*>(d_idx + static_cast<size_t>(n_channels) * cap);
		UG_CUDA(cudaMemcpyAsync(d_msg, messages, sizeof(int) * n_channels, cudaMemcpyHostToDevice, ctx->stream));
		PreambleParams p{d_bits, words, n_epochs, n_channels, d_msg, d_counts, d_idx, cap};
		{
			KernelTimer timer(ctx, "obs_preamble");
			sign_bits_kernel<<<static_cast<unsigned>((word_threads + kObsThreads - 1) / kObsThreads), kObsThreads, 0, ctx->stream>>>(
				d_out, n_epochs, n_channels, words, d_bits);
			preamble_kernel<<<static_cast<unsigned>(n_channels), kObsThreads, 0, ctx->stream>>>(p);
			UG_CUDA(cudaGetLastError());
			note_launch(ctx, 2);
		}
		UG_CUDA(cudaMemcpyAsync(counts, d_counts, sizeof(int) * n_channels, cudaMemcpyDeviceToHost, ctx->stream));
		if (list_bytes)
			UG_CUDA(cudaMemcpyAsync(indexes, d_idx, list_bytes, cudaMemcpyDeviceToHost, ctx->stream));
		UG_CUDA(cudaStreamSynchronize(ctx->stream));
	});
}

int ugsdr_observables(ugsdr_ctx* ctx, const ugsdr_track_output* outputs, int outputs_on_device, int n_epochs,
	int n_channels, const ugsdr_observable_channel* channels, ugsdr_observable* out) {
	UG_OBS_ENTRY(ctx) {
		require(outputs && channels && out, "null outputs, channels or observables");
		require(n_epochs >= 1 && n_epochs <= (1 << 30) && n_channels >= 1, "bad output array shape");
		std::vector<ObsChannel> ch(n_channels);
		for (int c = 0; c < n_channels; ++c) {
			const ugsdr_observable_channel& in = channels[c];
			require(in.sampling_rate > 0, "sampling rate must be positive");
			require(in.preamble_position >= 0 && in.preamble_position < n_epochs, "preamble position outside the epochs");
			ch[c].samples_to_ms = 1000 / in.sampling_rate;
			ch[c].windup = in.intermediate_frequency / 1e3;
			ch[c].intermediate_frequency = in.intermediate_frequency;
			ch[c].phase0 = in.carrier_phase / kTwoPi;
			ch[c].frequency0 = in.carrier_frequency;
			ch[c].correction = in.range_correction_ms;
			ch[c].position = in.preamble_position;
		}
		const size_t records = static_cast<size_t>(n_epochs) * n_channels;
		const ugsdr_track_output* d_out = stage_outputs(ctx, outputs, outputs_on_device, records);
		// segments long enough for whole groups of loads, short enough that the
		// threads (one per segment and channel) fill the SMs
		const size_t wanted = records / (static_cast<size_t>(ctx->sm_count) * 768) + 1;
		const int segment = static_cast<int>(std::min<size_t>(kMaxSegment,
			std::max<size_t>(kMinSegment, (wanted + kObsUnroll - 1) / kObsUnroll * kObsUnroll)));
		const int n_segments = (n_epochs + segment - 1) / segment;
		const size_t threads = static_cast<size_t>(n_channels) * n_segments;
		const int q_stride = (n_epochs + kObsUnroll - 1) / kObsUnroll * kObsUnroll;
		// scratch: channels | sigma | segment sums | prompt Q (256-byte aligned regions)
		auto align = [](size_t b) { return (b + 255) & ~static_cast<size_t>(255); };
		const size_t ch_bytes = align(sizeof(ObsChannel) * n_channels), sig_bytes = align(sizeof(float) * n_channels);
		const size_t seg_bytes = align(sizeof(double) * threads);
		ctx->obs_tmp.reserve(ch_bytes + sig_bytes + seg_bytes + sizeof(float) * static_cast<size_t>(q_stride) * n_channels);
		char* base = ctx->obs_tmp.as<char>();
		ObsChannel* d_ch = reinterpret_cast<ObsChannel*>(base);
		float* d_sigma = reinterpret_cast<float*>(base + ch_bytes);
		double* d_seg = reinterpret_cast<double*>(base + ch_bytes + sig_bytes);
		float* d_q = reinterpret_cast<float*>(base + ch_bytes + sig_bytes + seg_bytes);
		UG_CUDA(cudaMemcpyAsync(d_ch, ch.data(), sizeof(ObsChannel) * n_channels, cudaMemcpyHostToDevice, ctx->stream));
		ugsdr_observable* d_obs = out;
		if (!outputs_on_device) {
			ctx->obs_out.reserve(sizeof(ugsdr_observable) * records);
			d_obs = ctx->obs_out.as<ugsdr_observable>();
		}
		ObsParams p{d_out, n_epochs, n_channels, n_segments, segment, q_stride, d_ch, d_q, d_sigma, d_seg, d_obs};
		{
			KernelTimer timer(ctx, "observables");
			const unsigned blocks = static_cast<unsigned>((threads + kSegmentThreads - 1) / kSegmentThreads);
			obs_sums_kernel<<<blocks, kSegmentThreads, 0, ctx->stream>>>(p);
			obs_sigma_kernel<<<(n_channels + kSigmaWarps - 1) / kSigmaWarps, 32 * kSigmaWarps, 0, ctx->stream>>>(p);
			obs_emit_kernel<<<blocks, kSegmentThreads, 0, ctx->stream>>>(p);
			UG_CUDA(cudaGetLastError());
			note_launch(ctx, 3);
		}
		if (!outputs_on_device)
			UG_CUDA(cudaMemcpyAsync(out, d_obs, sizeof(ugsdr_observable) * records, cudaMemcpyDeviceToHost, ctx->stream));
		UG_CUDA(cudaStreamSynchronize(ctx->stream));
	});
}

}
