// fls_selector.cuh -- device parts of the learned scheme selector that the
// statistics kernel, the network's kernels (fls_mlp.cu) and the encoder
// (fls_encode.cu) share: the 16 statistics of a staged vector and the
// network's parameter layout.
//
// Parameter layout (FLS_MLP_N_PARAMS floats): W1[64][16], b1[64], W2[64][64],
// b2[64], W3[5][64], b3[5]; ReLU after layers 1 and 2, softmax cross-entropy.
#pragma once

#include "fls_pipeline.cuh"

namespace fls {
namespace sel {

constexpr int kIn = FLS_MLP_IN, kH = FLS_MLP_HIDDEN, kOut = FLS_MLP_OUT;
constexpr int kW1 = 0, kB1 = kW1 + kH * kIn, kW2 = kB1 + kH, kB2 = kW2 + kH * kH, kW3 = kB2 + kH,
              kB3 = kW3 + kOut * kH, kNP = kB3 + kOut;
static_assert(kNP == FLS_MLP_N_PARAMS, "parameter layout");

// Words of a vector staged with one pad word per 32 values: lane L's chunk
// (values 32L..32L+31) is then read without bank conflicts.
constexpr uint32_t kPadded = 33u * 32u;
constexpr uint32_t kBuckets = 1024; // of the distinct-value estimate, one byte each

// The vector's counts that the statistics and the schemes' sizes derive from.
struct Counts {
	uint32_t max_d; // largest delta inside a 32-value chunk (unsigned)
	uint32_t runs;  // runs of rle.hpp: a change of value, or every 256 values
};

// Stages vector v (the last one padded with the column's last value, as the
// host encoder pads) 33-padded in shared memory; mn, mx: the vector's range.
__device__ __forceinline__ void stage_vector(const int32_t* __restrict__ values, uint64_t n, uint64_t v, int32_t* sv,
                                             uint32_t lane, int32_t& mn, int32_t& mx) {
	mn                = INT32_MAX;
	mx                = INT32_MIN;
	const uint64_t v0 = v * 1024u;
	if (v0 + 1024u <= n && (reinterpret_cast<uintptr_t>(values) & 15u) == 0) { // warp-uniform
		// a whole vector from a 16-byte aligned column: eight 16-byte loads
		// per lane (values 128 k + 4 lane .. + 3), all in flight at once
		int4 q[8];
#pragma unroll
		for (uint32_t k = 0; k < 8; ++k) { q[k] = __ldg(reinterpret_cast<const int4*>(values + v0) + 32u * k + lane); }
		asm volatile("" ::: "memory"); // every load issued before the first store below
#pragma unroll
		for (uint32_t k = 0; k < 8; ++k) {
			const uint32_t j = 128u * k + 4u * lane; // conflict-free: (j + j / 32) mod 32 differs across lanes
			const int32_t  e[4] = {q[k].x, q[k].y, q[k].z, q[k].w};
#pragma unroll
			for (uint32_t t = 0; t < 4; ++t) {
				sv[(j + t) + ((j + t) >> 5)] = e[t];
				mn                           = min(mn, e[t]);
				mx                           = max(mx, e[t]);
			}
		}
	} else {
		const int32_t last = __ldg(values + (n - 1));
#pragma unroll 4
		for (uint32_t r = 0; r < 32; ++r) {
			const uint64_t idx = v0 + 32u * r + lane;
			const int32_t  x   = idx < n ? __ldg(values + idx) : last;
			sv[33u * r + lane] = x;
			mn                 = min(mn, x);
			mx                 = max(mx, x);
		}
	}
	__syncwarp();
	mn = __reduce_min_sync(0xffffffffu, mn);
	mx = __reduce_max_sync(0xffffffffu, mx);
}

// One pass of lane L over its chunk.  WIDE: the sum of the chunk's absolute
// differences may pass 32 bits.
template <bool WIDE>
__device__ __forceinline__ void chunk_pass(const int32_t* c, int32_t mn, int32_t before, uint32_t tm_h, uint32_t tm_q,
                                           uint8_t* buckets, uint32_t& max_d, uint32_t& up, uint32_t& eqs, uint32_t& lh,
                                           uint32_t& lq, unsigned long long& sabs) {
	int32_t  p    = before;
	uint32_t s32  = 0;
	max_d = up = eqs = lh = lq = 0;
	sabs               = 0;
#pragma unroll 8
	for (uint32_t s = 0; s < 32; ++s) {
		const int32_t  x = c[s];
		const uint32_t u = static_cast<uint32_t>(x) - static_cast<uint32_t>(mn);
		const uint32_t d = static_cast<uint32_t>(x) - static_cast<uint32_t>(p);
		lh += u <= tm_h ? 1u : 0u;
		lq += u <= tm_q ? 1u : 0u;
		buckets[(static_cast<uint32_t>(x) * 0x9e3779b1u) >> 22] = 1;
		const uint32_t ad = x > p ? d : 0u - d;
		if constexpr (WIDE) {
			sabs += ad;
		} else {
			s32 += ad;
		}
		up += x > p ? 1u : 0u;
		eqs += d == 0u ? 1u : 0u;
		if (s != 0) { max_d = max(max_d, d); }
		p = x;
	}
	if constexpr (!WIDE) { sabs = s32; }
}

// The 16 statistics of a staged vector, exactly those of vector_stats()
// (fls_host.cpp): statistic `lane` on lanes 0..15, 0 on the others.
// buckets: kBuckets bytes of the warp's own, 16-byte aligned.
//
// Bounded by integer issue: about 20 instructions per value.  Distinct values
// are marked by plain byte stores, where bits of 32 shared words took an
// atomic each (43 instructions per value, many lanes on one word).
__device__ __forceinline__ float vector_features(const int32_t* sv, int32_t mn, int32_t mx, uint8_t* buckets,
                                                 uint32_t lane, Counts& n) {
	const auto bits32 = [](uint32_t v) { return 32u - static_cast<uint32_t>(__clz(v)); };
	auto*      b4     = reinterpret_cast<uint4*>(buckets);
	b4[lane] = b4[lane + 32u] = make_uint4(0u, 0u, 0u, 0u);
	__syncwarp();
	const uint32_t rbw = bits32(static_cast<uint32_t>(mx) - static_cast<uint32_t>(mn));
	const int32_t* c   = sv + 33u * lane; // this lane's chunk: values 32 lane .. 32 lane + 31
	// u <= tm_h (tm_q): the value lies in the lower half (sixteenth) of the
	// range's bit width; every value counts when the width is 0 (<= 4)
	const uint32_t tm_h = rbw == 0 ? 0xffffffffu : (1u << (rbw / 2)) - 1u;
	const uint32_t tm_q = rbw <= 4 ? 0xffffffffu : (1u << (rbw - 4)) - 1u;
	// the value before the chunk; the vector's first value is compared with
	// itself (an equal pair, corrected below)
	const int32_t      c0 = c[0], pb = lane ? c[-2] : c0;
	uint32_t           max_d, up, eqs, lh, lq;
	unsigned long long sabs;
	if (rbw <= 27) { // 32 differences below 2^27
		chunk_pass<false>(c, mn, pb, tm_h, tm_q, buckets, max_d, up, eqs, lh, lq, sabs);
	} else {
		chunk_pass<true>(c, mn, pb, tm_h, tm_q, buckets, max_d, up, eqs, lh, lq, sabs);
	}
	__syncwarp();
	// deltas of the lane: 32 (31 for lane 0, whose first value has no
	// predecessor); runs: the chunks of lanes 0, 8, 16, 24 open one whether or
	// not the value changes, lane 0's first value included
	const uint32_t at_start = c0 == pb ? 1u : 0u;
	uint32_t       eq       = eqs - (lane == 0 ? 1u : 0u);
	uint32_t       down     = 32u - up - eqs;
	uint32_t       runs     = 32u - eqs + ((lane & 7u) == 0 ? at_start : 0u);
	const uint4    o0 = b4[lane], o1 = b4[lane + 32u]; // bytes of 0 or 1
	const uint32_t occ = __reduce_add_sync(
	    0xffffffffu, static_cast<uint32_t>(__popc(o0.x) + __popc(o0.y) + __popc(o0.z) + __popc(o0.w) + __popc(o1.x) +
	                                       __popc(o1.y) + __popc(o1.z) + __popc(o1.w)));
	// counts of at most 1024 share words: up | down, eq | runs, lh | lq
	const uint32_t r0 = __reduce_add_sync(0xffffffffu, up | (down << 16));
	const uint32_t r1 = __reduce_add_sync(0xffffffffu, eq | (runs << 16));
	const uint32_t r2 = __reduce_add_sync(0xffffffffu, lh | (lq << 16));
	n.max_d           = __reduce_max_sync(0xffffffffu, max_d);
	n.runs            = r1 >> 16;
	const uint32_t cc = static_cast<uint32_t>(__popc(__ballot_sync(0xffffffffu, eqs - at_start == 31u)));
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) { sabs += __shfl_xor_sync(0xffffffffu, sabs, o); }
	const unsigned long long mean_d = sabs >> 10;
	const uint32_t amin = mn < 0 ? static_cast<uint32_t>(-static_cast<long long>(mn)) : static_cast<uint32_t>(mn);
	// statistic `lane` as an integer over a power of two
	uint32_t num = 0;
	float    scale = 0.0f;
	switch (lane) {
	case 0: num = rbw, scale = 1.0f / 32.0f; break;
	case 1: num = bits32(n.max_d), scale = 1.0f / 32.0f; break;
	case 2: num = n.runs, scale = 1.0f / 1024.0f; break;
	case 3: num = r0 & 0xffffu, scale = 1.0f / 1024.0f; break;
	case 4: num = r0 >> 16, scale = 1.0f / 1024.0f; break;
	case 5: num = r1 & 0xffffu, scale = 1.0f / 1024.0f; break;
	case 6: num = occ, scale = 1.0f / 1024.0f; break;
	case 7: num = bits32(occ), scale = 1.0f / 16.0f; break;
	case 8: num = bits32(static_cast<uint32_t>(min(mean_d, 0xffffffffull))), scale = 1.0f / 32.0f; break;
	case 9: num = r2 & 0xffffu, scale = 1.0f / 1024.0f; break;
	case 10: num = r2 >> 16, scale = 1.0f / 1024.0f; break;
	case 11: num = bits32(amin), scale = 1.0f / 32.0f; break;
	case 12: num = mn == mx ? 1u : 0u, scale = 1.0f; break;
	case 13: num = bits32(n.runs), scale = 1.0f / 16.0f; break;
	case 14: num = cc, scale = 1.0f / 32.0f; break;
	case 15: num = 1u, scale = 1.0f; break;
	default: break;
	}
	return static_cast<float>(num) * scale;
}

__device__ __forceinline__ void softmax5(float (&z)[kOut]) {
	float m = z[0];
#pragma unroll
	for (int k = 1; k < kOut; ++k) { m = fmaxf(m, z[k]); }
	float s = 0.0f;
#pragma unroll
	for (int k = 0; k < kOut; ++k) {
		z[k] = expf(z[k] - m);
		s += z[k];
	}
	const float inv = 1.0f / s;
#pragma unroll
	for (int k = 0; k < kOut; ++k) { z[k] *= inv; }
}

// The largest probability and its scheme (the first of equals).
__device__ __forceinline__ int top_of(const float (&z)[kOut], float& top) {
	int arg = 0;
	top     = z[0];
#pragma unroll
	for (int k = 1; k < kOut; ++k) {
		if (z[k] > top) {
			top = z[k];
			arg = k;
		}
	}
	return arg;
}

// The network on one sample by one warp, two units of each layer per lane,
// with the parameters in shared memory.  Weight rows are padded to a multiple
// of four floats plus four, so that the 16-byte reads of eight neighbouring
// units fall on different banks.  Every sum runs in the order of the
// one-sample form (forward_one in fls_mlp.cu): the same roundings.
struct WarpNet {
	static constexpr int kS1 = kIn + 4, kS2 = kH + 4;
	static constexpr int kOW1 = 0, kOB1 = kOW1 + kH * kS1, kOW2 = kOB1 + kH, kOB2 = kOW2 + kH * kS2,
	                     kOW3 = kOB2 + kH, kOB3 = kOW3 + kOut * kS2, kFloats = kOB3 + 8;
	static constexpr int kScratch = kIn + 2 * kH; // floats of the warp's own, 16-byte aligned
	static_assert(kOW2 % 4 == 0 && kOW3 % 4 == 0 && kIn % 4 == 0 && kH == 64, "16-byte rows");

	// All threads of the CTA; the caller synchronises before forward().
	static __device__ __forceinline__ void load(const float* __restrict__ g, float* s) {
		for (int i = threadIdx.x; i < kNP; i += blockDim.x) {
			int at;
			if (i < kB1) {
				at = kOW1 + i / kIn * kS1 + i % kIn;
			} else if (i < kW2) {
				at = kOB1 + (i - kB1);
			} else if (i < kB2) {
				at = kOW2 + (i - kW2) / kH * kS2 + (i - kW2) % kH;
			} else if (i < kW3) {
				at = kOB2 + (i - kB2);
			} else if (i < kB3) {
				at = kOW3 + (i - kW3) / kH * kS2 + (i - kW3) % kH;
			} else {
				at = kOB3 + (i - kB3);
			}
			s[at] = g[i];
		}
	}

	// x: input `lane` on lanes 0..15.  z: the logits, on every lane.
	static __device__ __forceinline__ void forward(const float* s, float* scratch, float x, uint32_t lane,
	                                               float (&z)[kOut]) {
		float *h1 = scratch + kIn, *h2 = h1 + kH;
		if (lane < kIn) { scratch[lane] = x; }
		__syncwarp();
#pragma unroll
		for (int t = 0; t < 2; ++t) {
			const uint32_t unit = lane + 32u * t;
			const float4*  w = reinterpret_cast<const float4*>(s + kOW1 + unit * kS1);
			float          a = s[kOB1 + unit];
#pragma unroll
			for (int i4 = 0; i4 < kIn / 4; ++i4) {
				const float4 q = w[i4], v = reinterpret_cast<const float4*>(scratch)[i4];
				a              = fmaf(q.x, v.x, a);
				a              = fmaf(q.y, v.y, a);
				a              = fmaf(q.z, v.z, a);
				a              = fmaf(q.w, v.w, a);
			}
			h1[unit] = fmaxf(a, 0.0f);
		}
		__syncwarp();
		{
			const float4 *w0 = reinterpret_cast<const float4*>(s + kOW2 + lane * kS2), *w1 = w0 + 32 * kS2 / 4;
			float         a[2][4] = {{s[kOB2 + lane], 0.0f, 0.0f, 0.0f}, {s[kOB2 + lane + 32], 0.0f, 0.0f, 0.0f}};
#pragma unroll 8
			for (int i4 = 0; i4 < kH / 4; ++i4) {
				const float4 h = reinterpret_cast<const float4*>(h1)[i4], p = w0[i4], q = w1[i4];
				a[0][0]        = fmaf(p.x, h.x, a[0][0]);
				a[0][1]        = fmaf(p.y, h.y, a[0][1]);
				a[0][2]        = fmaf(p.z, h.z, a[0][2]);
				a[0][3]        = fmaf(p.w, h.w, a[0][3]);
				a[1][0]        = fmaf(q.x, h.x, a[1][0]);
				a[1][1]        = fmaf(q.y, h.y, a[1][1]);
				a[1][2]        = fmaf(q.z, h.z, a[1][2]);
				a[1][3]        = fmaf(q.w, h.w, a[1][3]);
			}
#pragma unroll
			for (int t = 0; t < 2; ++t) {
				h2[lane + 32u * t] = fmaxf((a[t][0] + a[t][1]) + (a[t][2] + a[t][3]), 0.0f);
			}
		}
		__syncwarp();
		const uint32_t k = lane < kOut ? lane : 0u;
		const float4*  w = reinterpret_cast<const float4*>(s + kOW3 + k * kS2);
		float          a = s[kOB3 + k];
#pragma unroll 8
		for (int j4 = 0; j4 < kH / 4; ++j4) {
			const float4 q = w[j4], h = reinterpret_cast<const float4*>(h2)[j4];
			a = fmaf(q.x, h.x, a);
			a = fmaf(q.y, h.y, a);
			a = fmaf(q.z, h.z, a);
			a = fmaf(q.w, h.w, a);
		}
#pragma unroll
		for (int i = 0; i < kOut; ++i) { z[i] = __shfl_sync(0xffffffffu, a, i); }
	}
};

} // namespace sel
} // namespace fls
