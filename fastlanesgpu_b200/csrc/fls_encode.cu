// fls_encode.cu -- the FastLanes column encoder on the GPU.
//
// Produces exactly the words and metadata of the host encoder
// (fls_encode_column, fls_host.cpp encode_vector) for a column already in
// device memory, with a per-vector scheme that may itself come from the GPU
// (the learned selector's picks), so a column can be selected and encoded
// without leaving the device.  One kernel reads the values once: a CTA takes
// tiles of eight consecutive vectors in order; one warp per vector stages its
// 1024 values in shared memory and computes the chosen scheme's bit width, aux
// and payload words; the tile's word offset comes from a look-back over the
// tiles before it; the warp then writes the payload it still holds.
//
// Layout facts restated from the reference: the lane/word order of
// fastlanes/src/pack.cpp:1954-1990, the transposed order of
// fastlanes/src/transpose.cpp:4110 with the rsum visiting order of
// fls_gen/rsum/rsum.cuh:4-107, unrsum.cpp:120-256, and rle.hpp:8-44's run
// dictionary restarting every 256 values.
#include <cuda_runtime.h>

#include <algorithm>

#include "fls_pipeline.cuh"

namespace fls {
namespace {

constexpr uint32_t kEncWarps    = 8;                 // warps per CTA
constexpr uint32_t kValWords    = 33u * 32u;         // the vector, 33-padded rows
constexpr uint32_t kEncWarpWords = 2u * kValWords;   // the vector; sort buffer, then dictionary
constexpr uint32_t kKeyedBits    = 22;               // widest range whose sort keys carry the value's index
constexpr uint32_t kPollLimit   = 1u << 22;          // bounded look-back waits (each poll is an L2 round trip)

struct EncParams {
	const int32_t* values;
	uint64_t       n;
	uint64_t       n_vec;
	const uint8_t* schemes; // per vector, or null: `scheme` for all
	uint32_t       scheme;
	uint32_t       layout;
	uint32_t       round4;
	uint32_t       pad_;
	uint32_t*      out;
	fls_vec_meta*  meta;
	uint64_t       n_tiles;
	uint32_t*      counter; // next tile to take (zeroed before the launch)
	uint64_t*      tiles;   // per tile: look-back state (zeroed before the launch)
	uint64_t*      info;    // [0] total words, [1] max vector words, [2] scheme mask
	uint32_t*      err;
};

// Look-back state of a tile, one 64-bit word: payload words (42 bits: at most
// 2^30 vectors of kMaxVecWords), largest vector (11 bits), scheme mask (5
// bits), and a flag: not there yet, of the tile alone, of all tiles up to it,
// or given up.
constexpr uint64_t kTileSum = (1ull << 42) - 1ull, kTileBody = (1ull << 62) - 1ull;
constexpr uint64_t kTileOwn = 1ull << 62, kTileAll = 2ull << 62, kTileLost = 3ull << 62;
static_assert(kMaxVecWords < (1u << 11) && FLS_N_SCHEMES <= 5 && FLS_MAX_VALUES / 1024u * kMaxVecWords <= kTileSum,
              "look-back state fields");

__device__ __forceinline__ uint64_t tile_state(uint64_t words, uint32_t max_words, uint32_t mask) {
	return words | (static_cast<uint64_t>(max_words) << 42) | (static_cast<uint64_t>(mask) << 53);
}
__device__ __forceinline__ uint32_t tile_max(uint64_t s) { return static_cast<uint32_t>(s >> 42) & 0x7ffu; }
__device__ __forceinline__ uint32_t tile_mask(uint64_t s) { return static_cast<uint32_t>(s >> 53) & 0x1fu; }
__device__ __forceinline__ uint64_t tile_join(uint64_t a, uint64_t b) {
	return tile_state((a & kTileSum) + (b & kTileSum), max(tile_max(a), tile_max(b)), tile_mask(a) | tile_mask(b));
}

__device__ __forceinline__ uint64_t tile_load(const uint64_t* p) {
	uint64_t v;
	asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
	return v;
}
__device__ __forceinline__ void tile_store(uint64_t* p, uint64_t v) {
	asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// One warp: the joined state of all tiles before `tile` (no flag), after
// publishing this tile's own; kTileLost when a wait gave up (the bound is
// never met by a running grid: tiles are taken in order, so every tile before
// this one belongs to a resident CTA).  A round reads kLookGroups x 32 tiles,
// all loads in flight: tiles finish at one window per L2 round trip at most,
// so a window of 32 tiles held a large column to 1.5 TB/s of values (it
// measured 0.90-0.97x of separate plan, scan and write kernels).
constexpr uint32_t kLookGroups = 4;
__device__ __forceinline__ uint64_t tile_lookback(uint64_t* tiles, uint64_t tile, uint64_t own, uint32_t lane) {
	if (tile == 0) {
		if (lane == 0) { tile_store(tiles, own | kTileAll); }
		return 0;
	}
	if (lane == 0) { tile_store(tiles + tile, own | kTileOwn); }
	uint64_t before = 0;
	for (uint64_t end = tile;;) { // tiles [0, end) are still to be joined
		uint64_t s[kLookGroups];
		uint32_t take[kLookGroups]; // lanes joined from each group
		bool     got = false, done = false, lost = false;
		for (uint32_t poll = 0; poll < kPollLimit && !got; ++poll) {
#pragma unroll
			for (uint32_t g = 0; g < kLookGroups; ++g) {
				const uint32_t back = 32u * g + lane;
				s[g]                = back < end ? tile_load(tiles + (end - 1u - back)) : kTileAll;
			}
			got  = true;
			done = false;
#pragma unroll
			for (uint32_t g = 0; g < kLookGroups; ++g) {
				const uint64_t flag = s[g] & ~kTileBody;
				const uint32_t all  = __ballot_sync(0xffffffffu, flag >= kTileAll);
				const uint32_t none = __ballot_sync(0xffffffffu, flag == 0);
				take[g]             = done ? 0u : all ? all ^ (all - 1u) : 0xffffffffu; // up to the first that knows all
				got                 = got && (none & take[g]) == 0;
				done                = done || all != 0;
			}
		}
		uint64_t sum = 0;
		uint32_t mx = 0, mask = 0;
#pragma unroll
		for (uint32_t g = 0; g < kLookGroups; ++g) {
			const bool mine = (take[g] >> lane) & 1u;
			lost            = lost || (mine && (s[g] & ~kTileBody) == kTileLost);
			const uint64_t b = mine ? s[g] & kTileBody : 0ull;
			sum += b & kTileSum;
			mx = max(mx, tile_max(b));
			mask |= tile_mask(b);
		}
		if (!got || __any_sync(0xffffffffu, lost)) {
			if (lane == 0) { tile_store(tiles + tile, kTileLost); }
			return kTileLost;
		}
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) { sum += __shfl_xor_sync(0xffffffffu, sum, o); }
		before = tile_join(before, tile_state(sum, __reduce_max_sync(0xffffffffu, mx), __reduce_or_sync(0xffffffffu, mask)));
		if (done) { break; } // also at the column's start: tiles before it count as known
		end -= 32u * kLookGroups;
	}
	if (lane == 0) { tile_store(tiles + tile, tile_join(before, own) | kTileAll); }
	return before;
}

__device__ __forceinline__ uint32_t bits_of(uint32_t v) { return v ? 32u - __clz(v) : 0u; }
__device__ __forceinline__ uint32_t round_words4(uint32_t w) { return (w + 3u) & ~3u; }

// Value j of the staged vector (33-padded: row and chunk reads are
// bank-conflict-free).
__device__ __forceinline__ int32_t val_at(const int32_t* v, uint32_t j) { return v[j + (j >> 5)]; }

__device__ __forceinline__ uint32_t payload_words(uint32_t scheme, uint32_t bw, uint32_t aux) {
	switch (scheme) {
	case FLS_SCHEME_FOR: return 32u * bw;
	case FLS_SCHEME_DELTA: return 32u + 32u * bw;
	case FLS_SCHEME_RLE: return 48u + round_words4((aux * bw + 31u) / 32u);
	case FLS_SCHEME_CONST: return 0u;
	default: return 32u * bits_of(aux - 1u) + round_words4((aux * bw + 31u) / 32u); // DICT
	}
}

// Loads vector v (the last one padded with the column's last value, as the
// host encoder pads) into shared memory; returns this lane's min and max.
__device__ __forceinline__ void stage_vector(const EncParams& P, uint64_t v, int32_t* sv, uint32_t lane, int32_t& mn,
                                             int32_t& mx) {
	const int32_t last = __ldg(P.values + (P.n - 1));
	mn                 = INT32_MAX;
	mx                 = INT32_MIN;
	const uint64_t v0  = v * 1024u;
	if (v0 + 1024u <= P.n && (reinterpret_cast<uintptr_t>(P.values) & 15u) == 0) { // warp-uniform
		// a whole vector from a 16-byte aligned column: eight 16-byte loads
		// per lane (values 128 k + 4 lane .. + 3), all in flight at once
		int4 q[8];
#pragma unroll
		for (uint32_t k = 0; k < 8; ++k) { q[k] = __ldg(reinterpret_cast<const int4*>(P.values + v0) + 32u * k + lane); }
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
#pragma unroll 4
		for (uint32_t r = 0; r < 32; ++r) {
			const uint64_t idx = v0 + 32u * r + lane;
			const int32_t  x   = idx < P.n ? __ldg(P.values + idx) : last;
			sv[33u * r + lane] = x;
			mn                 = min(mn, x);
			mx                 = max(mx, x);
		}
	}
	__syncwarp();
	mn = __reduce_min_sync(0xffffffffu, mn);
	mx = __reduce_max_sync(0xffffffffu, mx);
}

__device__ __forceinline__ void order(uint32_t& a, uint32_t& b) {
	const uint32_t lo = min(a, b), hi = max(a, b);
	a = lo;
	b = hi;
}

// Compare-exchange of registers J apart.
template <int J>
__device__ __forceinline__ void order_step(uint32_t (&k)[32]) {
#pragma unroll
	for (int r = 0; r < 32; ++r) {
		if (!(r & J)) { order(k[r], k[r | J]); }
	}
}

// Ascending bitonic sort of a warp's 1024 keys, lane L holding elements
// 32 L .. 32 L + 31 in registers before and after.  Steps less than 32 apart
// are between a lane's own registers; for the others the keys are turned by
// way of buf (33-padded, conflict-free) so that lane L holds elements L, L +
// 32, ...  A block that sorts downwards holds its keys complemented, so every
// step is one min and one max.  About 2500 instructions per vector, against
// 12000 for the same network on shared memory (low-cardinality dictionary of
// 6 M values, whole encoder call: 308 -> 126 us).
__device__ __forceinline__ void sort1024(uint32_t (&k)[32], uint32_t* buf, uint32_t lane) {
	uint32_t flip = 0u - (lane & 1u);
#pragma unroll
	for (int r = 0; r < 32; ++r) { k[r] ^= flip; }
#pragma unroll
	for (int w = 2; w <= 32; w *= 2) {
#pragma unroll
		for (int j = w / 2; j > 0; j /= 2) {
#pragma unroll
			for (int r = 0; r < 32; ++r) {
				if (!(r & j)) { (r & w) ? order(k[r | j], k[r]) : order(k[r], k[r | j]); }
			}
		}
	}
#pragma unroll 1
	for (uint32_t p = 0; p < 5; ++p) { // blocks of 64 << p
		const uint32_t next = p < 4 ? 0u - ((lane >> (p + 1u)) & 1u) : 0u, turn = flip ^ next;
		flip                = next;
#pragma unroll
		for (int r = 0; r < 32; ++r) { buf[33u * lane + r] = k[r] ^ turn; }
		__syncwarp();
#pragma unroll
		for (int r = 0; r < 32; ++r) { k[r] = buf[33u * r + lane]; }
		if (p >= 4) { order_step<16>(k); }
		if (p >= 3) { order_step<8>(k); }
		if (p >= 2) { order_step<4>(k); }
		if (p >= 1) { order_step<2>(k); }
		order_step<1>(k);
#pragma unroll
		for (int r = 0; r < 32; ++r) { buf[33u * r + lane] = k[r]; }
		__syncwarp();
#pragma unroll
		for (int r = 0; r < 32; ++r) { k[r] = buf[33u * lane + r]; }
		order_step<16>(k);
		order_step<8>(k);
		order_step<4>(k);
		order_step<2>(k);
		order_step<1>(k);
		__syncwarp(); // buf is read before its next use
	}
}

// Sorts the staged vector's values minus mn (range bits rbw) into k, each
// with its index below it when both fit 32 bits, and returns the number of
// distinct values; first: the registers that hold the first of a value.
__device__ __forceinline__ uint32_t sort_distinct(const int32_t* sv, uint32_t* buf, uint32_t lane, int32_t mn,
                                                  uint32_t rbw, uint32_t (&k)[32], uint32_t& first, uint32_t& before) {
	const bool     keyed = rbw <= kKeyedBits;
	const uint32_t sh    = keyed ? 10u : 0u;
#pragma unroll
	for (uint32_t r = 0; r < 32; ++r) {
		const uint32_t d = static_cast<uint32_t>(sv[33u * lane + r]) - static_cast<uint32_t>(mn);
		k[r]             = keyed ? (d << 10) | (32u * lane + r) : d;
	}
	__syncwarp();
	sort1024(k, buf, lane);
	const uint32_t last = __shfl_up_sync(0xffffffffu, k[31], 1);
	first               = lane == 0 || ((k[0] ^ last) >> sh) != 0u ? 1u : 0u;
#pragma unroll
	for (uint32_t r = 1; r < 32; ++r) { first |= (((k[r] ^ k[r - 1]) >> sh) != 0u ? 1u : 0u) << r; }
	const uint32_t cnt  = static_cast<uint32_t>(__popc(first));
	uint32_t       incl = cnt;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
		if (lane >= static_cast<uint32_t>(o)) { incl += y; }
	}
	before = incl - cnt;
	return __shfl_sync(0xffffffffu, incl, 31);
}

// Dictionary of the sorted keys: the distinct values minus mn, ascending, in
// u; with keys that carry the index, also the code of every value over the
// staged vector (16-bit, 34-padded rows of 32).
__device__ __forceinline__ uint16_t* codes_of(int32_t* sv) { return reinterpret_cast<uint16_t*>(sv); }
__device__ __forceinline__ uint32_t  code_pos(uint32_t j) { return j + 2u * (j >> 5); }

__device__ __forceinline__ void write_dict(const uint32_t (&k)[32], uint32_t first, uint32_t before, bool keyed,
                                           int32_t* sv, uint32_t* u) {
	uint32_t n = before;
#pragma unroll
	for (uint32_t r = 0; r < 32; ++r) {
		const bool f = (first >> r) & 1u;
		if (f) { u[n] = keyed ? k[r] >> 10 : k[r]; }
		n += f ? 1u : 0u;
		if (keyed) { codes_of(sv)[code_pos(k[r] & 1023u)] = static_cast<uint16_t>(n - 1u); }
	}
	__syncwarp();
}

// Run starts of rle.hpp (every 256 values, or a change of value): lane L
// counts the starts of chunk L (values 32L..32L+31).
__device__ __forceinline__ uint32_t chunk_starts(const int32_t* sv, uint32_t lane) {
	uint32_t f = 0;
#pragma unroll 4
	for (uint32_t s = 0; s < 32; ++s) {
		const uint32_t j = 32u * lane + s;
		f |= ((j & 255u) == 0 || val_at(sv, j) != val_at(sv, j ? j - 1u : 0u) ? 1u : 0u) << s;
	}
	return f;
}

// Element of the lane's row r in the column's layout.
__device__ __forceinline__ uint32_t layout_index(uint32_t layout, uint32_t lane, uint32_t r) {
	return layout == FLS_LAYOUT_NORMAL ? 32u * r + lane : 32u * dev::chunk_of_lane(lane) + dev::step_of_row(r);
}

// FastLanes packing of the lane's 32 rows (x[r] < 2^BW) into words
// out[32k + lane]; a switch on the width (warp-uniform) makes every shift a
// constant: about 2 instructions per row, 12 with the width at run time.
template <int BW>
__device__ __forceinline__ void pack_rows(const uint32_t (&x)[32], uint32_t* out, uint32_t lane) {
	uint32_t w = 0;
#pragma unroll
	for (int r = 0; r < 32; ++r) {
		const int k = r * BW / 32, s = r * BW % 32;
		w = s ? w | (x[r] << s) : x[r];
		if (s + BW >= 32) {
			out[32 * k + lane] = w;
			w                  = s + BW > 32 ? x[r] >> (32 - s) : 0u;
		}
	}
}

__device__ __forceinline__ void pack_lane(const uint32_t (&x)[32], uint32_t bw, uint32_t* out, uint32_t lane) {
	switch (bw) {
#define FLS_PACK_CASE(B)                                                                                               \
	case B: if constexpr (B > 0) { pack_rows<B>(x, out, lane); } break;
		FLS_BW_CASES_0_32(FLS_PACK_CASE)
#undef FLS_PACK_CASE
	default: break;
	}
}

// Sequential LSB-first packing of u[0..n) at bw bits, zero-padded to a
// multiple of 4 words (the host's pack_sequential).  The word's first entry
// is found by a reciprocal: 32 w < 2^15 and bw <= 32, so the product with
// ceil(2^32 / bw) divides exactly.
__device__ __forceinline__ void pack_sequential(const uint32_t* u, uint32_t n, uint32_t bw, uint32_t* out,
                                                uint32_t lane) {
	if (bw == 0) { return; }
	const uint32_t words = round_words4((n * bw + 31u) / 32u);
	const uint32_t inv   = 0xffffffffu / bw + 1u; // bw == 1: 0
	for (uint32_t w = lane; w < words; w += 32) {
		const uint32_t bit0 = 32u * w;
		const uint32_t k0   = bw == 1u ? bit0 : __umulhi(bit0, inv);
		uint32_t       word = 0;
		if (k0 < n) {
			word = u[k0] >> (bit0 - k0 * bw);
			uint32_t k = k0 + 1u;
			for (uint32_t sh = (k0 + 1u) * bw - bit0; sh < 32u && k < n; sh += bw) { word |= u[k++] << sh; }
		}
		out[w] = word;
	}
}

struct Plan {
	uint32_t scheme, bw, aux;
	int32_t  base;
};

// Scheme parameters of the staged vector (CONST on a non-constant vector
// becomes FOR, as on the host).
__device__ __forceinline__ Plan plan_vector(const EncParams& P, uint64_t v, int32_t* sv, uint32_t* u, uint32_t lane,
                                            int32_t mn, int32_t mx) {
	uint32_t s = P.schemes ? P.schemes[v] : P.scheme;
	if (s >= FLS_N_SCHEMES) {
		if (lane == 0) { atomicOr(P.err, kErrBadMeta); }
		s = FLS_SCHEME_FOR;
	}
	if (s == FLS_SCHEME_CONST && mn != mx) { s = FLS_SCHEME_FOR; }
	const uint32_t range = static_cast<uint32_t>(mx) - static_cast<uint32_t>(mn);
	Plan           p {s, 0u, 0u, 0};
	switch (s) {
	case FLS_SCHEME_CONST: p.base = mn; break;
	case FLS_SCHEME_FOR:
		p.bw = bits_of(range);
		if (P.round4 && p.bw) { p.bw = (p.bw + 3u) & ~3u; }
		p.base = mn;
		break;
	case FLS_SCHEME_DELTA: {
		const uint32_t c = dev::chunk_of_lane(lane);
		uint32_t       mxd = 0;
		int32_t        prev = val_at(sv, 32u * c);
		for (uint32_t t = 1; t < 32; ++t) {
			const int32_t cur = val_at(sv, 32u * c + t);
			mxd               = max(mxd, static_cast<uint32_t>(cur) - static_cast<uint32_t>(prev));
			prev              = cur;
		}
		p.bw = bits_of(__reduce_max_sync(0xffffffffu, mxd));
		break;
	}
	case FLS_SCHEME_RLE:
		p.aux  = __reduce_add_sync(0xffffffffu, __popc(chunk_starts(sv, lane)));
		p.bw   = bits_of(range);
		p.base = mn;
		break;
	default: { // DICT: leaves the dictionary in u, and the codes in sv when the keys carry them
		uint32_t k[32], first, before;
		p.bw   = bits_of(range);
		p.base = mn;
		p.aux  = sort_distinct(sv, u, lane, mn, p.bw, k, first, before);
		write_dict(k, first, before, p.bw <= kKeyedBits, sv, u);
		break;
	}
	}
	return p;
}

// ------------------------------------------------ learned selection

struct SelParams {
	const int32_t*      values;
	uint64_t            n, n_vec;
	const uint8_t*      mlp_best; // the network's pick per vector
	const float*        conf;     // and its probability
	float               threshold;
	uint32_t            pad_;
	double              kappa;
	uint8_t*            schemes;  // the chosen scheme per vector
	unsigned long long* n_fallback;
};

// The exhaustive choice for vectors the network is unsure of (confidence
// below threshold), else the network's pick.  The exact encoded sizes of
// every scheme (payload + 16 B metadata) are the host exhaustive encoder's
// (fls_host.cpp scheme_sizes), the choice the label rule of the learned
// selector: argmin of size x (1 + kappa (decode cost - 1)) with the decode
// costs FOR 1, DELTA 1.5, RLE 2, CONST 1, DICT 4.5, ties to the cheaper
// decode (FOR, CONST, DELTA, RLE, DICT), in IEEE double with each product and
// sum rounded separately (no fused multiply-add), as numpy computes it.
__global__ void __launch_bounds__(kEncWarps * 32) enc_select_kernel(const __grid_constant__ SelParams S) {
	extern __shared__ __align__(16) int32_t esmem[];
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	int32_t*       sv   = esmem + warp * kEncWarpWords;
	uint32_t*      u    = reinterpret_cast<uint32_t*>(sv + kValWords);
	EncParams      P {};
	P.values = S.values;
	P.n      = S.n;
	for (uint64_t v = static_cast<uint64_t>(blockIdx.x) * kEncWarps + warp; v < S.n_vec;
	     v += static_cast<uint64_t>(gridDim.x) * kEncWarps) {
		if (!(S.conf[v] < S.threshold)) {
			if (lane == 0) { S.schemes[v] = S.mlp_best[v]; }
			continue;
		}
		int32_t mn, mx;
		stage_vector(P, v, sv, lane, mn, mx);
		const uint32_t rbw = bits_of(static_cast<uint32_t>(mx) - static_cast<uint32_t>(mn));
		uint32_t       mxd = 0;
		{
			const uint32_t c    = dev::chunk_of_lane(lane);
			int32_t        prev = val_at(sv, 32u * c);
			for (uint32_t t = 1; t < 32; ++t) {
				const int32_t cur = val_at(sv, 32u * c + t);
				mxd               = max(mxd, static_cast<uint32_t>(cur) - static_cast<uint32_t>(prev));
				prev              = cur;
			}
		}
		const uint32_t dbw    = bits_of(__reduce_max_sync(0xffffffffu, mxd));
		const uint32_t n_runs = __reduce_add_sync(0xffffffffu, __popc(chunk_starts(sv, lane)));
		uint32_t       k[32], first, before;
		const uint32_t n_dist = sort_distinct(sv, u, lane, mn, rbw, k, first, before);
		if (lane == 0) {
			uint32_t size[FLS_N_SCHEMES];
			size[FLS_SCHEME_FOR]   = 16u + 4u * payload_words(FLS_SCHEME_FOR, rbw, 0u);
			size[FLS_SCHEME_DELTA] = 16u + 4u * payload_words(FLS_SCHEME_DELTA, dbw, 0u);
			size[FLS_SCHEME_RLE]   = 16u + 4u * payload_words(FLS_SCHEME_RLE, rbw, n_runs);
			size[FLS_SCHEME_CONST] = mn == mx ? 16u : 0xffffffffu;
			size[FLS_SCHEME_DICT]  = 16u + 4u * payload_words(FLS_SCHEME_DICT, rbw, n_dist);
			const uint32_t order[FLS_N_SCHEMES] = {FLS_SCHEME_FOR, FLS_SCHEME_CONST, FLS_SCHEME_DELTA, FLS_SCHEME_RLE,
			                                       FLS_SCHEME_DICT};
			const double cost[FLS_N_SCHEMES] = {1.0, 1.5, 2.0, 1.0, 4.5}; // by scheme id
			uint32_t     best = order[0];
			double       best_score = 0.0;
			for (uint32_t i = 0; i < FLS_N_SCHEMES; ++i) {
				const uint32_t sc = order[i];
				if (size[sc] == 0xffffffffu) { continue; }
				const double f     = __dadd_rn(1.0, __dmul_rn(S.kappa, cost[sc] - 1.0));
				const double score = __dmul_rn(static_cast<double>(size[sc]), f);
				if (i == 0 || score < best_score) {
					best       = sc;
					best_score = score;
				}
			}
			S.schemes[v] = static_cast<uint8_t>(best);
			atomicAdd(S.n_fallback, 1ull);
		}
		__syncwarp();
	}
}

// Writes the planned vector's payload (staged in sv; DICT: planned) at `out`.
__device__ __forceinline__ void write_vector(const EncParams& P, const Plan& p, const int32_t* sv, uint32_t* u,
                                             uint32_t* out, uint32_t lane) {
	const uint32_t base  = static_cast<uint32_t>(p.base);
	uint32_t       x[32] = {}, bw = 0, skip = 0; // rows to pack, their width, words before them
	if (p.scheme == FLS_SCHEME_FOR) {
		bw = p.bw;
		if (P.layout == FLS_LAYOUT_NORMAL) {
#pragma unroll
			for (uint32_t r = 0; r < 32; ++r) { x[r] = static_cast<uint32_t>(sv[33u * r + lane]) - base; }
		} else {
			const uint32_t c = 33u * dev::chunk_of_lane(lane);
#pragma unroll
			for (uint32_t r = 0; r < 32; ++r) { x[r] = static_cast<uint32_t>(sv[c + dev::step_of_row(r)]) - base; }
		}
	} else if (p.scheme == FLS_SCHEME_DELTA) {
		const uint32_t c = 33u * dev::chunk_of_lane(lane);
		bw               = p.bw;
		skip             = 32u;
		out[lane]        = static_cast<uint32_t>(sv[c]);
		uint32_t prev    = static_cast<uint32_t>(sv[c]);
#pragma unroll
		for (uint32_t t = 0; t < 32; ++t) {
			const uint32_t cur    = static_cast<uint32_t>(sv[c + t]);
			x[dev::rsum_row(t)] = cur - prev;
			prev                  = cur;
		}
	} else if (p.scheme == FLS_SCHEME_RLE) {
		// Run index of every value: starts before its chunk + starts in it.
		const uint32_t f   = chunk_starts(sv, lane);
		const uint32_t cnt = __popc(f);
		uint32_t       pre = cnt;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const uint32_t y = __shfl_up_sync(0xffffffffu, pre, o);
			if (lane >= static_cast<uint32_t>(o)) { pre += y; }
		}
		pre -= cnt;
		// run dictionary: the value at each start, in order
		uint32_t ff = f, k = pre;
		while (ff) {
			const uint32_t t = __ffs(ff) - 1u;
			ff &= ff - 1u;
			u[k++] = static_cast<uint32_t>(sv[33u * lane + t]) - base;
		}
		// transposed lane L holds chunk c(L): base = run index of its first
		// value, then 1-bit deltas (a start) in rsum row order
		const uint32_t c  = dev::chunk_of_lane(lane);
		const uint32_t fc = __shfl_sync(0xffffffffu, f, c);
		const uint32_t pc = __shfl_sync(0xffffffffu, pre, c);
		reinterpret_cast<uint16_t*>(out)[lane] = static_cast<uint16_t>(pc + (fc & 1u) - 1u);
		uint32_t bits = 0;
#pragma unroll
		for (uint32_t r = 0; r < 32; ++r) {
			const uint32_t t = dev::step_of_row(r);
			bits |= (t != 0 ? (fc >> t) & 1u : 0u) << r;
		}
		out[16 + lane] = bits;
		__syncwarp();
		pack_sequential(u, p.aux, p.bw, out + 48, lane);
	} else if (p.scheme == FLS_SCHEME_DICT) {
		const uint32_t n = p.aux;
		bw               = bits_of(n - 1u);
		if (p.bw <= kKeyedBits) {
			const uint16_t* codes = reinterpret_cast<const uint16_t*>(sv);
#pragma unroll
			for (uint32_t r = 0; r < 32; ++r) { x[r] = codes[code_pos(layout_index(P.layout, lane, r))]; }
		} else {
#pragma unroll
			for (uint32_t r = 0; r < 32; ++r) {
				const uint32_t val = static_cast<uint32_t>(val_at(sv, layout_index(P.layout, lane, r))) - base;
				uint32_t       lo  = 0; // the value's position: it is there, so ten halvings find it
#pragma unroll 1
				for (uint32_t step = 512; step > 0; step >>= 1) {
					if (lo + step < n && u[lo + step] <= val) { lo += step; }
				}
				x[r] = lo;
			}
		}
		pack_sequential(u, n, p.bw, out + 32u * bw, lane);
	}
	pack_lane(x, bw, out + skip, lane);
}

// Bounded by the per-vector work of planning and packing (DICT: the sort) and,
// for large columns, by how many vectors an SM has in flight: two 33-padded
// buffers per warp let three CTAs (24 warps) share an SM.  Against separate
// plan, scan and write kernels, which read and sorted everything twice, whole
// encoder calls took (us, before -> after): 6 M values DICT 437 -> 126,
// 33.5 M values FOR 187 -> 168, DELTA 188 -> 165, RLE 186 -> 174, DICT 1918
// -> 325; of each about 60 are the call's host side and its read-back.
__global__ void __launch_bounds__(kEncWarps * 32, 3) enc_kernel(const __grid_constant__ EncParams P) {
	extern __shared__ __align__(16) int32_t esmem[];
	__shared__ uint32_t s_tile;
	__shared__ uint64_t s_own[kEncWarps], s_before;
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	int32_t*       sv   = esmem + warp * kEncWarpWords;
	uint32_t*      u    = reinterpret_cast<uint32_t*>(sv + kValWords);
	for (;;) {
		if (threadIdx.x == 0) { s_tile = atomicAdd(P.counter, 1u); }
		__syncthreads();
		const uint64_t tile = s_tile;
		if (tile >= P.n_tiles) { break; }
		const uint64_t v    = tile * kEncWarps + warp;
		const bool     live = v < P.n_vec;
		Plan           p {};
		uint32_t       words = 0;
		if (live) {
			int32_t mn, mx;
			stage_vector(P, v, sv, lane, mn, mx);
			p     = plan_vector(P, v, sv, u, lane, mn, mx);
			words = payload_words(p.scheme, p.bw, p.aux);
		}
		if (lane == 0) { s_own[warp] = live ? tile_state(words, words, 1u << p.scheme) : 0ull; }
		__syncthreads();
		if (warp == 0) {
			uint64_t own = 0;
#pragma unroll
			for (uint32_t w = 0; w < kEncWarps; ++w) { own = tile_join(own, s_own[w]); }
			const uint64_t before = tile_lookback(P.tiles, tile, own, lane);
			if (lane == 0) {
				s_before = before;
				if (before == kTileLost) {
					atomicOr(P.err, kErrTimeout);
				} else if (tile + 1u == P.n_tiles) {
					const uint64_t all = tile_join(before, own);
					P.info[0]          = all & kTileSum;
					P.info[1]          = tile_max(all);
					P.info[2]          = tile_mask(all);
				}
			}
		}
		__syncthreads();
		const uint64_t before = s_before;
		if (live && before != kTileLost) {
			uint64_t offset = before & kTileSum;
			for (uint32_t w = 0; w < warp; ++w) { offset += s_own[w] & kTileSum; }
			if (lane == 0) {
				fls_vec_meta m;
				m.offset  = offset;
				m.base    = p.base;
				m.scheme  = static_cast<uint8_t>(p.scheme);
				m.bw      = static_cast<uint8_t>(p.bw);
				m.aux     = static_cast<uint16_t>(p.aux);
				P.meta[v] = m;
			}
			write_vector(P, p, sv, u, P.out + offset, lane);
		}
		__syncthreads(); // s_own and the staged vector are read before the next tile's
	}
}

} // namespace
} // namespace fls

using namespace fls;

extern "C" {

uint64_t fls_encode_gpu_workspace_bytes(uint64_t n) {
	const uint64_t n_vec = (n + 1023u) / 1024u, n_tiles = (n_vec + kEncWarps - 1) / kEncWarps;
	return 8u * n_tiles + 256u; // the counter and the tiles' states, after alignment
}

fls_status fls_encode_column_gpu(const int32_t* d_values, uint64_t n, const uint8_t* d_schemes, uint32_t scheme,
                                 uint32_t layout, int round4, uint32_t* d_out, uint64_t out_capacity_words,
                                 fls_vec_meta* d_meta, uint64_t* d_info, void* d_workspace, uint64_t workspace_bytes,
                                 fls_stream_t stream) {
	if (!d_values || !d_out || !d_meta || !d_info || !d_workspace || n == 0) {
		return set_error(FLS_ERR_INVALID_ARG, "fls_encode_column_gpu: null pointer or n == 0");
	}
	if (fls_status s = check_n_values(n, "fls_encode_column_gpu"); s != FLS_OK) { return s; }
	if (!d_schemes && scheme >= FLS_N_SCHEMES) { return set_error(FLS_ERR_INVALID_ARG, "fls_encode_column_gpu: bad scheme"); }
	if (layout > FLS_LAYOUT_TRANSPOSED) { return set_error(FLS_ERR_INVALID_ARG, "fls_encode_column_gpu: bad layout"); }
	if ((reinterpret_cast<uintptr_t>(d_out) | reinterpret_cast<uintptr_t>(d_meta)) & 15u) {
		return set_error(FLS_ERR_ALIGNMENT, "fls_encode_column_gpu: output and metadata must be 16-byte aligned");
	}
	const uint64_t n_vec = (n + 1023u) / 1024u;
	if (out_capacity_words < n_vec * kMaxVecWords) {
		return set_error(FLS_ERR_CAPACITY, "fls_encode_column_gpu: output smaller than fls_encode_bound_words(n)");
	}
	if (workspace_bytes < fls_encode_gpu_workspace_bytes(n)) {
		return set_error(FLS_ERR_CAPACITY, "fls_encode_column_gpu: workspace smaller than fls_encode_gpu_workspace_bytes(n)");
	}
	DeviceInfo di;
	fls_status s = device_info(di);
	if (s != FLS_OK) { return s; }
	cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
	EncParams    P {};
	P.values  = d_values;
	P.n       = n;
	P.n_vec   = n_vec;
	P.schemes = d_schemes;
	P.scheme  = scheme;
	P.layout  = layout;
	P.round4  = round4 ? 1u : 0u;
	P.out     = d_out;
	P.meta    = d_meta;
	char* ws  = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(d_workspace) + 15u) & ~uintptr_t {15u});
	P.n_tiles = (n_vec + kEncWarps - 1) / kEncWarps;
	P.counter = reinterpret_cast<uint32_t*>(ws);
	P.tiles   = reinterpret_cast<uint64_t*>(ws + 16);
	P.info    = d_info;
	P.err     = device_error_word(st);
	const size_t smem = 4u * kEncWarps * kEncWarpWords;
	{
		static std::mutex mu;
		static uint64_t   configured = 0;
		int               dev        = 0;
		cudaGetDevice(&dev);
		std::lock_guard<std::mutex> lk(mu);
		if (dev >= 64 || !(configured & (1ull << dev))) {
			if ((s = cuda_check(cudaFuncSetAttribute(enc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
			                                         static_cast<int>(smem)),
			                    "cudaFuncSetAttribute")) != FLS_OK) {
				return s;
			}
			if (dev < 64) { configured |= 1ull << dev; }
		}
	}
	if ((s = cuda_check(cudaMemsetAsync(ws, 0, 16u + 8u * P.n_tiles, st), "cudaMemsetAsync")) != FLS_OK) { return s; }
	const uint32_t grid = static_cast<uint32_t>(std::min<uint64_t>(P.n_tiles, static_cast<uint64_t>(di.sms) * 8u));
	enc_kernel<<<grid, kEncWarps * 32, smem, st>>>(P);
	count_launch();
	return cuda_check(cudaGetLastError(), "enc_kernel launch");
}

uint64_t fls_encode_learned_workspace_bytes(uint64_t n) {
	const uint64_t n_vec = (n + 1023u) / 1024u;
	auto           a256  = [](uint64_t b) { return (b + 255u) & ~uint64_t {255u}; };
	return a256(64u * n_vec) + a256(4u * n_vec) + 2u * a256(n_vec) + fls_encode_gpu_workspace_bytes(n);
}

fls_status fls_encode_learned_gpu(const int32_t* d_values, uint64_t n, const float* d_params, float threshold,
                                  double kappa, uint32_t layout, uint32_t* d_out, uint64_t out_capacity_words,
                                  fls_vec_meta* d_meta, uint64_t* d_info, uint8_t* d_schemes, void* d_workspace,
                                  uint64_t workspace_bytes, fls_stream_t stream) {
	if (!d_values || !d_params || !d_info || !d_workspace || n == 0) {
		return set_error(FLS_ERR_INVALID_ARG, "fls_encode_learned_gpu: null pointer or n == 0");
	}
	if (fls_status s = check_n_values(n, "fls_encode_learned_gpu"); s != FLS_OK) { return s; }
	if (!(kappa >= 0.0)) { return set_error(FLS_ERR_INVALID_ARG, "fls_encode_learned_gpu: kappa must be >= 0"); }
	if (workspace_bytes < fls_encode_learned_workspace_bytes(n) || (reinterpret_cast<uintptr_t>(d_workspace) & 255u)) {
		return set_error(FLS_ERR_CAPACITY,
		                 "fls_encode_learned_gpu: workspace smaller than fls_encode_learned_workspace_bytes(n) "
		                 "or not 256-byte aligned");
	}
	const uint64_t n_vec = (n + 1023u) / 1024u;
	auto           a256  = [](uint64_t b) { return (b + 255u) & ~uint64_t {255u}; };
	char*          w     = static_cast<char*>(d_workspace);
	float*         stats = reinterpret_cast<float*>(w);
	float*         conf  = reinterpret_cast<float*>(w + a256(64u * n_vec));
	uint8_t*       best  = reinterpret_cast<uint8_t*>(w + a256(64u * n_vec) + a256(4u * n_vec));
	uint8_t*       own   = best + a256(n_vec);
	void*          enc   = own + a256(n_vec);
	uint8_t*       pick  = d_schemes ? d_schemes : own;
	cudaStream_t   st    = reinterpret_cast<cudaStream_t>(stream);
	DeviceInfo     di;
	fls_status     s = device_info(di);
	if (s != FLS_OK) { return s; }
	if ((s = fls_vector_stats_gpu(d_values, n, stats, stream)) != FLS_OK) { return s; }
	if ((s = fls_mlp_infer(d_params, stats, n_vec, nullptr, best, conf, stream)) != FLS_OK) { return s; }
	const size_t smem = 4u * kEncWarps * kEncWarpWords;
	{
		static std::mutex mu;
		static uint64_t   configured = 0;
		int               dev        = 0;
		cudaGetDevice(&dev);
		std::lock_guard<std::mutex> lk(mu);
		if (dev >= 64 || !(configured & (1ull << dev))) {
			if ((s = cuda_check(cudaFuncSetAttribute(enc_select_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
			                                         static_cast<int>(smem)),
			                    "cudaFuncSetAttribute")) != FLS_OK) {
				return s;
			}
			if (dev < 64) { configured |= 1ull << dev; }
		}
	}
	if ((s = cuda_check(cudaMemsetAsync(d_info + 3, 0, sizeof(uint64_t), st), "cudaMemsetAsync")) != FLS_OK) {
		return s;
	}
	SelParams S {};
	S.values     = d_values;
	S.n          = n;
	S.n_vec      = n_vec;
	S.mlp_best   = best;
	S.conf       = conf;
	S.threshold  = threshold;
	S.kappa      = kappa;
	S.schemes    = pick;
	S.n_fallback = reinterpret_cast<unsigned long long*>(d_info + 3);
	const uint32_t grid = static_cast<uint32_t>(
	    std::min<uint64_t>((n_vec + kEncWarps - 1) / kEncWarps, static_cast<uint64_t>(di.sms) * 8u));
	enc_select_kernel<<<grid, kEncWarps * 32, smem, st>>>(S);
	count_launch(1);
	if ((s = cuda_check(cudaGetLastError(), "enc_select_kernel launch")) != FLS_OK) { return s; }
	return fls_encode_column_gpu(d_values, n, pick, 0u, layout, 0, d_out, out_capacity_words, d_meta, d_info, enc,
	                             fls_encode_gpu_workspace_bytes(n), stream);
}

} // extern "C"
