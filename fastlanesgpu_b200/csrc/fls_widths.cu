// fls_widths.cu -- GPU decode of FastLanes columns of 8-, 16- and 64-bit
// lanes (FOR with one base and bit width per column), to HBM and/or fused
// with a sum.  The reference decodes only 32-bit lanes on the GPU
// (fls_gen/unpack/unpack.cuh); its host packer covers all four widths
// (fastlanes/src/pack.cpp:29521, 29552, 29607, 29710), whose layout this
// reads: 1024/T lanes, row r of lane i is value (1024/T)*r + i, word k of
// lane i at (1024/T)*k + i, 128-byte rows, 128*bw bytes per vector.
//
// 8/16-bit lanes: one warp per vector; thread t reads the 32-bit word t of
// each 128-byte row, which holds 32/T consecutive lanes, and extracts row r
// of all of them at once (SIMD within a register: every lane of a word has
// the same bit offset r*bw, so one shift and a per-lane mask serve all; the
// base is added lane-wise without carries between lanes), at constant widths.
// 64-bit lanes: a half-warp per vector, one lane per thread.  Both read and
// write 128-byte rows per instruction.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "fls_pipeline.cuh"

namespace fls {
namespace {

template <int B>
struct Narrow {
	static constexpr uint32_t kRep  = B == 8 ? 0x01010101u : 0x00010001u; // one per lane of a word
	static constexpr uint32_t kLow  = (1u << B) - 1u;
	static constexpr uint32_t kHigh = (1u << (B - 1)) * kRep; // lane top bits
};

// Lane-wise sum of the 32/B lanes of x.
template <int B>
__device__ __forceinline__ uint32_t lane_sum(uint32_t x) {
	if constexpr (B == 8) {
		const uint32_t t = (x & 0x00ff00ffu) + ((x >> 8) & 0x00ff00ffu);
		return (t & 0xffffu) + (t >> 16);
	} else {
		return (x & 0xffffu) + (x >> 16);
	}
}

// The block's sum into the result with one atomic: one per warp, 18,944 on one
// address, took 5 of the 17 us of 90 M 8-bit values at width 3.
__device__ __forceinline__ void add_block_sum(unsigned long long acc, unsigned long long* sum) {
	__shared__ unsigned long long part[8];
	const uint32_t lane = threadIdx.x & 31u;
	acc                 = warp_sum_u64(acc);
	if (lane == 0) { part[threadIdx.x >> 5] = acc; }
	__syncthreads();
	if (threadIdx.x < 32u) {
		acc = warp_sum_u64(lane < 8u ? part[lane] : 0ull);
		if (lane == 0 && acc) { atomicAdd(sum, acc); }
	}
}

// One vector of 8/16-bit lanes at width BW: rows of the 32/B lanes of thread
// word t.  OUT / SUM: write the values / add them to part; TAIL: the column's
// last, partial vector (rem values).  NOWRAP: the host proved base + 2^bw - 1 <
// 2^B, so no value wraps: a packed add gives the values, and whole vectors sum
// their fields packed (while 2^B holds a thread's rows of them) or in 2B-bit
// halves, with the base added once per thread (32 values).
//
// With the width a constant every shift and mask is one too and a thread
// reads its BW words once: about 6 instructions per row, 37 with the width at
// run time (two clamped reads per row among them).  90 M values, us before ->
// after: to memory 8-bit at width 3 33 -> 23, 16-bit at width 5 59 -> 41 and 13
// 66 -> 54 (write bound); sums 8-bit at width 3 35 -> 16, 16-bit at width 5 61
// -> 20 and 13 63 -> 30.
template <int B, int BW, bool OUT, bool SUM, bool TAIL, bool NOWRAP>
__device__ __forceinline__ void narrow_vector(const uint32_t* __restrict src, uint32_t* __restrict dst,
                                              uint32_t base_rep, uint32_t t, uint64_t rem, uint32_t& part) {
	using N              = Narrow<B>;
	constexpr uint32_t L = 32u / B;   // lanes per thread word
	constexpr uint32_t S = 1024u / B; // lanes per vector
	constexpr uint32_t V = (1u << BW) - 1u;
	constexpr bool     kFields = SUM && !TAIL && NOWRAP;         // fields are summed, not values
	constexpr bool     kPacked = BW + (B == 8 ? 3 : 4) <= B;     // B rows of them fit a lane
	uint32_t           w[BW > 0 ? BW : 1];
#pragma unroll
	for (int k = 0; k < BW; ++k) { w[k] = __ldg(src + 32 * k + t); }
	uint32_t ev = 0, od = 0;
#pragma unroll
	for (int r = 0; r < B; ++r) {
		const int o = r * BW, k = o / B, sh = o % B;
		uint32_t  x = 0;
		if constexpr (BW > 0) {
			x = (w[k] >> sh) & ((N::kLow >> sh & V) * N::kRep);
			if (sh + BW > B) { x |= (w[k + 1] << (B - sh)) & ((N::kLow << (B - sh) & V) * N::kRep); }
		}
		uint32_t y = x;
		if constexpr (NOWRAP) {
			y = x + base_rep;
		} else {
			y = ((x & ~N::kHigh) + (base_rep & ~N::kHigh)) ^ ((x ^ base_rep) & N::kHigh);
		}
		if constexpr (OUT) { __stcs(dst + 32 * r + t, y); }
		if constexpr (kFields && kPacked) {
			ev += x;
		} else if constexpr (kFields) {
			if constexpr (B == 8) {
				ev += x & 0x00ff00ffu;
				od += (x >> 8) & 0x00ff00ffu;
			} else {
				ev += x & 0xffffu;
				od += x >> 16;
			}
		} else if constexpr (SUM) {
			uint32_t keep = y;
			if constexpr (TAIL) {
				keep = 0;
#pragma unroll
				for (uint32_t j = 0; j < L; ++j) {
					keep |= (S * r + L * t + j < rem) ? (y & (N::kLow << (B * j))) : 0u;
				}
			}
			part += lane_sum<B>(keep);
		}
	}
	if constexpr (kFields) {
		if constexpr (kPacked) {
			part += lane_sum<B>(ev);
		} else if constexpr (B == 8) {
			part += (ev & 0xffffu) + (ev >> 16) + (od & 0xffffu) + (od >> 16);
		} else {
			part += ev + od;
		}
		part += 32u * (base_rep & N::kLow); // the thread's 32 values
	}
}

// Resident 256-thread blocks per SM asked of the compiler (it trades
// registers for warps): enough warps to cover the reads, and registers for
// two vectors' words.
constexpr int kNarrowMinBlocks = 4;

// A column of width BW: one warp per vector.
template <int B, int BW, bool OUT, bool SUM, bool NOWRAP>
__device__ __forceinline__ void narrow_column(const uint32_t* __restrict in, uint64_t n, uint64_t n_vec,
                                              uint32_t base_rep, uint32_t* __restrict out, unsigned long long& acc) {
	const uint32_t t  = threadIdx.x & 31u;
	const uint64_t wg = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
	const uint64_t nw = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
	const uint64_t full = SUM ? n / 1024u : n_vec; // vectors that need no test of their rows
	uint64_t       v    = wg;
	// Several vectors at a time while their words are few, so that enough
	// reads are in flight (sum of 90 M 8-bit values at width 3, whole call: 22.2
	// us one by one, 20.5 four at a time).
	constexpr uint32_t U = BW <= 4 ? 4u : BW <= 8 ? 2u : 1u;
	for (; U > 1u && v + (U - 1u) * nw < full; v += U * nw) {
#pragma unroll
		for (uint32_t u = 0; u < U; ++u) {
			uint32_t part = 0;
			narrow_vector<B, BW, OUT, SUM, false, NOWRAP>(in + (v + u * nw) * (32u * BW),
			                                              OUT ? out + (v + u * nw) * (32u * B) : nullptr, base_rep, t,
			                                              1024u, part);
			acc += part;
		}
	}
	for (; v < n_vec; v += nw) {
		const uint32_t* src  = in + v * (32u * BW);
		uint32_t*       dst  = OUT ? out + v * (32u * B) : nullptr;
		uint32_t        part = 0;
		if (v < full) {
			narrow_vector<B, BW, OUT, SUM, false, NOWRAP>(src, dst, base_rep, t, 1024u, part);
		} else {
			narrow_vector<B, BW, OUT, SUM, true, NOWRAP>(src, dst, base_rep, t, n - v * 1024u, part);
		}
		acc += part;
	}
}

// 8/16-bit lanes: one warp per vector (a 0-bit column reads no payload); the
// width is a switch ahead of the loop over the vectors.
template <int B, bool OUT, bool SUM, bool NOWRAP>
__global__ void __launch_bounds__(256, kNarrowMinBlocks) decode_narrow_kernel(const uint32_t* __restrict in, uint64_t n,
                                                                             uint64_t n_vec, uint32_t bw,
                                                                             uint32_t base_rep,
                                                                             uint32_t* __restrict out,
                                                                             unsigned long long* sum) {
	unsigned long long acc = 0;
	switch (bw) {
#define FLS_NARROW_CASE(W)                                                                                             \
	case W:                                                                                                            \
		if constexpr (W <= B) { narrow_column<B, W, OUT, SUM, NOWRAP>(in, n, n_vec, base_rep, out, acc); }             \
		break;
		FLS_NARROW_CASE(0)
		FLS_NARROW_CASE(1)
		FLS_NARROW_CASE(2)
		FLS_NARROW_CASE(3)
		FLS_NARROW_CASE(4)
		FLS_NARROW_CASE(5)
		FLS_NARROW_CASE(6)
		FLS_NARROW_CASE(7)
		FLS_NARROW_CASE(8)
		FLS_NARROW_CASE(9)
		FLS_NARROW_CASE(10)
		FLS_NARROW_CASE(11)
		FLS_NARROW_CASE(12)
		FLS_NARROW_CASE(13)
		FLS_NARROW_CASE(14)
		FLS_NARROW_CASE(15)
		FLS_NARROW_CASE(16)
#undef FLS_NARROW_CASE
	default: break;
	}
	if constexpr (SUM) { add_block_sum(acc, sum); }
}

// 64-bit lanes: a half-warp per vector, one lane per thread.
template <bool OUT, bool SUM>
__global__ void __launch_bounds__(256, 3) decode_u64_kernel(const uint64_t* __restrict in, uint64_t n, uint64_t n_vec,
                                                         uint32_t bw, uint64_t base, uint64_t* __restrict out,
                                                         unsigned long long* sum) {
	const uint32_t     i   = threadIdx.x & 15u; // lane of the vector
	const uint64_t     h0  = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 4;
	const uint64_t     nh  = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 4;
	const uint64_t     m    = bw >= 64 ? ~0ull : (1ull << bw) - 1ull;
	const uint32_t     m_lo = static_cast<uint32_t>(m), m_hi = static_cast<uint32_t>(m >> 32);
	const uint32_t     last = bw ? bw - 1u : 0u;
	unsigned long long acc = 0;
	// every half-warp runs the same number of iterations, so full-warp
	// shuffles at the end see every lane
	const uint64_t iters = (n_vec + nh - 1) / nh;
	for (uint64_t it = 0; it < iters; ++it) {
		const uint64_t v = h0 + it * nh;
		if (v >= n_vec) { continue; }
		const auto*    src = reinterpret_cast<const unsigned long long*>(in + v * 16u * bw);
		const uint64_t rem = n - v * 1024u;
		if (bw == 0) { // every value is the base; no payload to read
			for (uint32_t r = 0; r < 64; ++r) {
				if constexpr (OUT) { __stcs(reinterpret_cast<unsigned long long*>(out) + v * 1024u + 16u * r + i, base); }
				if constexpr (SUM) { acc += 16u * r + i < rem ? base : 0ull; }
			}
			continue;
		}
		// Row r's field starts at bit s of word row k.  Both word rows are
		// read unconditionally (the second clamped inside the vector) and
		// the field is cut from their four 32-bit halves by two 32-bit
		// funnel shifts; bits of the second row past a field that does not
		// straddle fall under the mask.
		auto row = [&](uint32_t r) -> uint64_t {
			const uint32_t o = r * bw, k = o >> 6, s = o & 63u;
			const uint2    a = __ldg(reinterpret_cast<const uint2*>(src + 16u * k + i));
			const uint2    b = __ldg(reinterpret_cast<const uint2*>(src + 16u * min(k + 1u, last) + i));
			const bool     up = s >= 32u;
			const uint32_t w0 = up ? a.y : a.x, w1 = up ? b.x : a.y, w2 = up ? b.y : b.x;
			const uint32_t xl = __funnelshift_r(w0, w1, s) & m_lo, xh = __funnelshift_r(w1, w2, s) & m_hi;
			return ((static_cast<uint64_t>(xh) << 32) | xl) + base;
		};
		if (rem >= 1024u) {
#pragma unroll 16
			for (uint32_t r = 0; r < 64; ++r) {
				const uint64_t y = row(r);
				if constexpr (OUT) { __stcs(reinterpret_cast<unsigned long long*>(out) + v * 1024u + 16u * r + i, y); }
				if constexpr (SUM) { acc += y; }
			}
		} else {
#pragma unroll 4
			for (uint32_t r = 0; r < 64; ++r) {
				const uint64_t y = row(r);
				if constexpr (OUT) { __stcs(reinterpret_cast<unsigned long long*>(out) + v * 1024u + 16u * r + i, y); }
				if constexpr (SUM) { acc += 16u * r + i < rem ? y : 0ull; }
			}
		}
	}
	if constexpr (SUM) {
		acc = warp_sum_u64(acc);
		if ((threadIdx.x & 31u) == 0 && acc) { atomicAdd(sum, acc); }
	}
}

template <class K>
void launch_mode(bool out, bool sum, K&& k) {
	if (out && sum) {
		k(std::integral_constant<int, 3> {});
	} else if (out) {
		k(std::integral_constant<int, 1> {});
	} else {
		k(std::integral_constant<int, 2> {});
	}
}

fls_status launch_decode(uint32_t bits, const void* d_in, uint64_t n, uint8_t bw, uint64_t base, void* d_out,
                         uint64_t* d_sum, fls_stream_t stream, const char* who) {
	if (!d_in || n == 0 || (!d_out && !d_sum)) {
		return set_error(FLS_ERR_INVALID_ARG, std::string(who) + ": null pointer, n == 0 or no output");
	}
	if (bw > bits) { return set_error(FLS_ERR_BAD_BW, std::string(who) + ": bit width larger than the values"); }
	if (fls_status s = check_n_values(n, who); s != FLS_OK) { return s; }
	if ((reinterpret_cast<uintptr_t>(d_in) | reinterpret_cast<uintptr_t>(d_out)) & 15u) {
		return set_error(FLS_ERR_ALIGNMENT, std::string(who) + ": buffers must be 16-byte aligned");
	}
	DeviceInfo di;
	fls_status s = device_info(di);
	if (s != FLS_OK) { return s; }
	cudaStream_t   st    = reinterpret_cast<cudaStream_t>(stream);
	const uint64_t n_vec = (n + 1023u) / 1024u;
	if (d_sum && (s = cuda_check(cudaMemsetAsync(d_sum, 0, sizeof(uint64_t), st), "cudaMemsetAsync")) != FLS_OK) {
		return s;
	}
	auto* sum = reinterpret_cast<unsigned long long*>(d_sum);
	if (bits == 64) {
		const uint32_t grid = static_cast<uint32_t>(std::min<uint64_t>((n_vec + 15u) / 16u, static_cast<uint64_t>(di.sms) * 16u));
		launch_mode(d_out != nullptr, d_sum != nullptr, [&](auto mode) {
			constexpr int M = decltype(mode)::value;
			decode_u64_kernel<(M & 1) != 0, (M & 2) != 0><<<grid, 256, 0, st>>>(
			    static_cast<const uint64_t*>(d_in), n, n_vec, bw, base, static_cast<uint64_t*>(d_out), sum);
		});
	} else {
		const uint32_t rep  = bits == 8 ? static_cast<uint32_t>(base & 0xffu) * 0x01010101u
		                                : static_cast<uint32_t>(base & 0xffffu) * 0x00010001u;
		// no decoded value wraps: base + 2^bw - 1 < 2^bits
		const bool nowrap = (base & ((1ull << bits) - 1u)) + ((1ull << bw) - 1u) < (1ull << bits);
		const uint32_t grid = static_cast<uint32_t>(std::min<uint64_t>((n_vec + 7u) / 8u, static_cast<uint64_t>(di.sms) * 16u));
		launch_mode(d_out != nullptr, d_sum != nullptr, [&](auto mode) {
			constexpr int  M   = decltype(mode)::value;
			constexpr bool O = (M & 1) != 0, S = (M & 2) != 0;
			const auto     run = [&](auto* kernel) {
                kernel<<<grid, 256, 0, st>>>(static_cast<const uint32_t*>(d_in), n, n_vec, bw, rep,
                                             static_cast<uint32_t*>(d_out), sum);
			};
			if (bits == 8) {
				nowrap ? run(decode_narrow_kernel<8, O, S, true>) : run(decode_narrow_kernel<8, O, S, false>);
			} else {
				nowrap ? run(decode_narrow_kernel<16, O, S, true>) : run(decode_narrow_kernel<16, O, S, false>);
			}
		});
	}
	count_launch();
	return cuda_check(cudaGetLastError(), "decode kernel launch");
}

} // namespace
} // namespace fls

using namespace fls;

extern "C" {

fls_status fls_decode_u8(const uint8_t* d_in, uint64_t n, uint8_t bw, uint8_t base, uint8_t* d_out, uint64_t* d_sum,
                         fls_stream_t stream) {
	return launch_decode(8, d_in, n, bw, base, d_out, d_sum, stream, "fls_decode_u8");
}

fls_status fls_decode_u16(const uint16_t* d_in, uint64_t n, uint8_t bw, uint16_t base, uint16_t* d_out,
                          uint64_t* d_sum, fls_stream_t stream) {
	return launch_decode(16, d_in, n, bw, base, d_out, d_sum, stream, "fls_decode_u16");
}

fls_status fls_decode_u64(const uint64_t* d_in, uint64_t n, uint8_t bw, uint64_t base, uint64_t* d_out,
                          uint64_t* d_sum, fls_stream_t stream) {
	return launch_decode(64, d_in, n, bw, base, d_out, d_sum, stream, "fls_decode_u64");
}

} // extern "C"
