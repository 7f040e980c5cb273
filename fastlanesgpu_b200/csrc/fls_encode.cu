// fls_encode.cu -- the FastLanes column encoder on the GPU.
//
// Produces exactly the words and metadata of the host encoder
// (fls_encode_column, fls_host.cpp encode_vector) for a column already in
// device memory, with a per-vector scheme that may itself come from the GPU
// (the learned selector's picks), so a column can be selected and encoded
// without leaving the device.  One kernel reads the values once: a CTA takes
// tiles of eight consecutive vectors in order; one warp per vector stages its
// 1024 values in shared memory and computes the chosen scheme's bit width, aux
// and payload words; a warp of one more CTA adds up the tiles' words in order
// and answers with each tile's offset; the warp then writes the payload it
// still holds.
//
// Layout facts restated from the reference: the lane/word order of
// fastlanes/src/pack.cpp:1954-1990, the transposed order of
// fastlanes/src/transpose.cpp:4110 with the rsum visiting order of
// fls_gen/rsum/rsum.cuh:4-107, unrsum.cpp:120-256, and rle.hpp:8-44's run
// dictionary restarting every 256 values.
#include <cuda_runtime.h>

#include <algorithm>

#include "fls_selector.cuh"

namespace fls {
namespace {

constexpr uint32_t kEncWarps    = 8;                 // warps per CTA
// A warp's shared memory, in words: the staged vector (33-padded), which is
// also the sort's buffer; in its place afterwards a DICT vector's 16-bit codes
// (34-padded) and its dictionary, or an RLE vector's run values; past the
// staged vector, before that, the statistics' buckets and the network's
// activations.
constexpr uint32_t kCodeWords    = 34u * 32u / 2u;
constexpr uint32_t kEncWarpWords = kCodeWords + 1024u;
constexpr uint32_t kNetWords     = sel::kPadded + sel::kBuckets / 4u; // offset of the activations
static_assert(kEncWarpWords % 4 == 0 && kEncWarpWords >= kNetWords + sel::WarpNet::kScratch, "the warp's words");
constexpr uint32_t kKeyedBits    = 22;               // widest range whose sort keys carry the value's index
constexpr uint32_t kPollLimit   = 1u << 22;          // bounded waits on other tiles (each poll is an L2 round trip)
// Idle rounds (some 5 ms) after which the scan looks whether any tile is taken:
// encodes that share the GPU with others wait for places for a while, and a tile
// by the scanning CTA holds up the answers to all others (64 columns on four
// streams, whole calls: 4.4 ms at 64 rounds, 4.2 so).
constexpr uint32_t kAloneRounds = 1u << 13;

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
	uint32_t*      counter; // next ticket, CTAs done (zeroed before the launch)
	uint32_t*      lost;    // set by a tile that gave up waiting (zeroed before the launch)
	uint64_t*      reports; // per tile (zeroed before the launch)
	uint64_t*      offsets; // per tile (zeroed before the launch)
	uint32_t       scan_polls, tile_polls; // limits of the scan's and of a tile's wait
	uint64_t*      info;    // [0] total words, [1] max vector words, [2] scheme mask; learned: [3] fallbacks
	uint32_t*      err;
	// learned selection
	const float*        params;
	float               threshold;
	double              kappa;
	uint8_t*            picks;      // the chosen scheme per vector, or null
	unsigned long long* n_fallback; // vectors below the threshold (zeroed before the launch)
};

// What a tile reports, one 64-bit word: its payload words (low half), its
// largest vector (16 bits), its scheme mask (8 bits) and a mark that it is
// there.  What it gets back: its word offset and the mark, or kTileLost.
constexpr uint64_t kTileMark = 1ull << 63, kTileLost = ~0ull;
static_assert(kMaxVecWords < (1u << 16) && FLS_N_SCHEMES <= 8 && FLS_MAX_VALUES / 1024u * kMaxVecWords < kTileMark,
              "tile report fields");

__device__ __forceinline__ uint64_t tile_report(uint32_t words, uint32_t max_words, uint32_t mask) {
	return kTileMark | (static_cast<uint64_t>(mask << 16 | max_words) << 32) | words;
}
__device__ __forceinline__ uint64_t tile_load(const uint64_t* p) {
	uint64_t v;
	asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
	return v;
}
__device__ __forceinline__ void tile_store(uint64_t* p, uint64_t v) {
	asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// The scan of the tiles' reports.
struct ScanState {
	uint64_t pos, run; // tiles answered, their words
	uint32_t mx, mask;
};

// An encode that is lost: no totals (a column that is there has at least one
// bit in its scheme mask).
__device__ __forceinline__ void void_info(const EncParams& P) {
	tile_store(P.info, 0ull);
	tile_store(P.info + 1, 0ull);
	tile_store(P.info + 2, 0ull);
}

// One warp: takes the tiles' reports in order, answers each with its offset
// and leaves the column's totals in info.  A round reads kScanGroups x 32
// reports, all loads in flight, and answers those that are there.  Returns 0
// when nothing is left to do.
//
// Only tiles that running CTAs have taken are waited for, so the next report
// always comes; should scan_polls rounds bring none all the same, the tiles
// still waiting are told so.  A tile that no CTA has taken may be long in
// coming: other work may hold every other place on the GPU for as long as it
// likes.  So where all tiles taken are answered, the scan takes the next one
// (by compare and swap: it is the next to be answered too) and returns its
// ticket, with its own state in S, for the CTA to encode it: one resident CTA
// finishes the column.
//
// Why one warp: a look-back by every tile over those before it (256 reports
// per round trip) cost the tiles 4-7 us each on a column of 733 tiles, since
// all of a GPU's tiles finish planning together and walk the same states.
constexpr uint32_t kScanGroups = 8;
__device__ __forceinline__ uint32_t scan_tiles(const EncParams& P, ScanState& S, uint32_t alone_rounds, uint32_t lane) {
	uint64_t pos = S.pos, run = S.run;
	uint32_t mx = S.mx, mask = S.mask, idle = 0;
	while (pos < P.n_tiles) {
		uint64_t s[kScanGroups];
#pragma unroll
		for (uint32_t g = 0; g < kScanGroups; ++g) {
			const uint64_t t = pos + 32u * g + lane;
			s[g]             = t < P.n_tiles ? tile_load(P.reports + t) : 0ull;
		}
		const uint64_t pos0 = pos;
		bool           more = true;
#pragma unroll
		for (uint32_t g = 0; g < kScanGroups; ++g) {
			if (!more) { continue; }
			const uint32_t none = __ballot_sync(0xffffffffu, s[g] == 0ull);
			const uint32_t n    = none ? static_cast<uint32_t>(__ffs(none)) - 1u : 32u;
			const bool     mine = lane < n;
			const uint32_t hi   = mine ? static_cast<uint32_t>(s[g] >> 32) & 0x7fffffffu : 0u;
			const uint32_t w    = mine ? static_cast<uint32_t>(s[g]) : 0u;
			uint32_t       incl = w; // at most 32 tiles x 8 vectors of kMaxVecWords
#pragma unroll
			for (int o = 1; o < 32; o <<= 1) {
				const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
				if (lane >= static_cast<uint32_t>(o)) { incl += y; }
			}
			if (mine) { tile_store(P.offsets + pos + lane, kTileMark | (run + incl - w)); }
			run += __shfl_sync(0xffffffffu, incl, 31);
			mx = max(mx, hi & 0xffffu);
			mask |= hi >> 16;
			pos += n;
			more = n == 32u;
		}
		idle = pos == pos0 ? idle + 1u : 0u;
		if (idle >= alone_rounds && idle % kAloneRounds == alone_rounds % kAloneRounds) {
			const uint32_t next = static_cast<uint32_t>(pos) + 1u; // the ticket after those of the tiles answered
			uint32_t       had  = 0;
			if (lane == 0) { had = atomicCAS(P.counter, next, next + 1u); }
			if (__shfl_sync(0xffffffffu, had, 0) == next) {
				S = ScanState {pos, run, __reduce_max_sync(0xffffffffu, mx), __reduce_or_sync(0xffffffffu, mask)};
				return next;
			}
		}
		if (idle >= P.scan_polls) {
			if (lane == 0) {
				atomicOr(P.err, kErrTimeout);
				void_info(P);
			}
			for (uint64_t t = pos + lane; t < P.n_tiles; t += 32u) { tile_store(P.offsets + t, kTileLost); }
			return 0;
		}
	}
	mx   = __reduce_max_sync(0xffffffffu, mx);
	mask = __reduce_or_sync(0xffffffffu, mask);
	if (lane == 0) {
		tile_store(P.info, run);
		tile_store(P.info + 1, mx);
		tile_store(P.info + 2, mask);
		__threadfence(); // see tile_lost
		if (*static_cast<const volatile uint32_t*>(P.lost)) { void_info(P); }
	}
	return 0;
}

// A tile whose wait has run out.  Either the scan, which looks for the mark
// after it has written its totals, sees it and takes them back, or the totals
// were there before the mark was, and are taken back here.
__device__ __forceinline__ void tile_lost(const EncParams& P) {
	atomicOr(P.err, kErrTimeout);
	atomicExch(P.lost, 1u);
	__threadfence();
	void_info(P);
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
// 12000 for the same network on shared memory (6 M values as a dictionary,
// whole encoder call: 308 -> 126 us).
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
// distinct values; first: the registers that hold the first of a value, of
// which `before` are on lower lanes.  The staged vector is lost.
__device__ __forceinline__ uint32_t sort_distinct(int32_t* sv, uint32_t lane, int32_t mn, uint32_t rbw,
                                                  uint32_t (&k)[32], uint32_t& first, uint32_t& before) {
	const bool     keyed = rbw <= kKeyedBits;
	const uint32_t sh    = keyed ? 10u : 0u;
#pragma unroll
	for (uint32_t r = 0; r < 32; ++r) {
		const uint32_t d = static_cast<uint32_t>(sv[33u * lane + r]) - static_cast<uint32_t>(mn);
		k[r]             = keyed ? (d << 10) | (32u * lane + r) : d;
	}
	__syncwarp();
	sort1024(k, reinterpret_cast<uint32_t*>(sv), lane);
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

// Dictionary of the sorted keys: the distinct values minus mn, ascending, and,
// with keys that carry the index, the code of every value.
__device__ __forceinline__ uint16_t* codes_of(int32_t* sv) { return reinterpret_cast<uint16_t*>(sv); }
__device__ __forceinline__ uint32_t* dict_of(int32_t* sv) { return reinterpret_cast<uint32_t*>(sv) + kCodeWords; }
__device__ __forceinline__ uint32_t  code_pos(uint32_t j) { return j + 2u * (j >> 5); }

__device__ __forceinline__ void write_dict(const uint32_t (&k)[32], uint32_t first, uint32_t before, bool keyed,
                                           int32_t* sv) {
	uint32_t *u = dict_of(sv), n = before;
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
	const uint32_t n_bits = n * bw;
	if (bw >= 11) {
		// a word meets at most four entries: read without a loop, so that the
		// reads of several words are in flight together (past the last entry
		// whatever lies there, masked off)
#pragma unroll 4
		for (uint32_t w = lane; w < words; w += 32) {
			const uint32_t bit0 = 32u * w, k0 = __umulhi(bit0, inv), s0 = bit0 - k0 * bw;
			uint32_t       word = u[min(k0, 1023u)] >> s0;
#pragma unroll
			for (uint32_t i = 1; i < 4; ++i) {
				const uint32_t s = i * bw - s0, e = u[min(k0 + i, 1023u)];
				word |= s < 32u ? e << s : 0u;
			}
			const uint32_t left = bit0 < n_bits ? n_bits - bit0 : 0u;
			out[w]              = left < 32u ? word & ((1u << left) - 1u) : word;
		}
		return;
	}
	for (uint32_t w = lane; w < words; w += 32) {
		const uint32_t bit0 = 32u * w;
		uint32_t       k    = bw == 1u ? bit0 : __umulhi(bit0, inv), word = 0;
		if (k < n) {
			uint32_t sh = (k + 1u) * bw - bit0;
			word        = u[k++] >> (bw - sh);
			for (; sh < 32u && k < n; sh += bw) { word |= u[k++] << sh; }
		}
		out[w] = word;
	}
}

struct Plan {
	uint32_t scheme, bw, aux;
	int32_t  base;
};

// The exhaustive choice among the exact encoded sizes (payload + 16 B
// metadata) of every scheme, as the host exhaustive encoder gives them
// (fls_host.cpp scheme_sizes), by the label rule of the learned selector:
// argmin of size x (1 + kappa (decode cost - 1)) with the decode costs FOR 1,
// DELTA 1.5, RLE 2, CONST 1, DICT 4.5, ties to the cheaper decode (FOR, CONST,
// DELTA, RLE, DICT), in IEEE double with each product and sum rounded
// separately (no fused multiply-add), as numpy computes it.
__device__ uint32_t exhaustive_choice(double kappa, uint32_t range_bits, uint32_t delta_bits, uint32_t runs,
                                      uint32_t distinct, bool constant) {
	uint32_t size[FLS_N_SCHEMES];
	size[FLS_SCHEME_FOR]   = 16u + 4u * payload_words(FLS_SCHEME_FOR, range_bits, 0u);
	size[FLS_SCHEME_DELTA] = 16u + 4u * payload_words(FLS_SCHEME_DELTA, delta_bits, 0u);
	size[FLS_SCHEME_RLE]   = 16u + 4u * payload_words(FLS_SCHEME_RLE, range_bits, runs);
	size[FLS_SCHEME_CONST] = constant ? 16u : 0xffffffffu;
	size[FLS_SCHEME_DICT]  = 16u + 4u * payload_words(FLS_SCHEME_DICT, range_bits, distinct);
	const uint32_t order[FLS_N_SCHEMES] = {FLS_SCHEME_FOR, FLS_SCHEME_CONST, FLS_SCHEME_DELTA, FLS_SCHEME_RLE,
	                                       FLS_SCHEME_DICT};
	const double cost[FLS_N_SCHEMES] = {1.0, 1.5, 2.0, 1.0, 4.5}; // by scheme id
	uint32_t     best = order[0];
	double       best_score = 0.0;
#pragma unroll
	for (uint32_t i = 0; i < FLS_N_SCHEMES; ++i) {
		const uint32_t sc = order[i];
		if (size[sc] == 0xffffffffu) { continue; }
		const double f     = __dadd_rn(1.0, __dmul_rn(kappa, cost[sc] - 1.0));
		const double score = __dmul_rn(static_cast<double>(size[sc]), f);
		if (i == 0 || score < best_score) {
			best       = sc;
			best_score = score;
		}
	}
	return best;
}

// Scheme parameters of the staged vector (CONST on a non-constant vector
// becomes FOR, as on the host).  LEARNED: `counts` are known, and a vector the
// network is `unsure` of takes the exhaustive choice instead of `s`, which
// receives it.
template <bool LEARNED>
__device__ __forceinline__ Plan plan_vector(const EncParams& P, uint64_t v, int32_t* sv, uint32_t lane, int32_t mn,
                                            int32_t mx, uint32_t& s, const sel::Counts& counts, bool unsure) {
	const uint32_t range_bits = bits_of(static_cast<uint32_t>(mx) - static_cast<uint32_t>(mn));
	uint32_t       k[32], first = 0, before = 0, distinct = 0;
	if (s == FLS_SCHEME_DICT || (LEARNED && unsure)) {
		distinct = sort_distinct(sv, lane, mn, range_bits, k, first, before);
	}
	if constexpr (LEARNED) {
		if (unsure) {
			s = exhaustive_choice(P.kappa, range_bits, bits_of(counts.max_d), counts.runs, distinct, mn == mx);
			if (s != FLS_SCHEME_DICT) { // the sort took the staged values' place
				int32_t mn2, mx2;
				__syncwarp();
				sel::stage_vector(P.values, P.n, v, sv, lane, mn2, mx2);
			}
		}
	}
	Plan p {s, 0u, 0u, 0};
	if (s == FLS_SCHEME_CONST && mn != mx) { p.scheme = FLS_SCHEME_FOR; }
	switch (p.scheme) {
	case FLS_SCHEME_CONST: p.base = mn; break;
	case FLS_SCHEME_FOR:
		p.bw = range_bits;
		if (P.round4 && p.bw) { p.bw = (p.bw + 3u) & ~3u; }
		p.base = mn;
		break;
	case FLS_SCHEME_DELTA: {
		uint32_t mxd = counts.max_d;
		if constexpr (!LEARNED) {
			int32_t prev = sv[33u * lane];
			mxd          = 0;
#pragma unroll 8
			for (uint32_t t = 1; t < 32; ++t) {
				const int32_t cur = sv[33u * lane + t];
				mxd               = max(mxd, static_cast<uint32_t>(cur) - static_cast<uint32_t>(prev));
				prev              = cur;
			}
			mxd = __reduce_max_sync(0xffffffffu, mxd);
		}
		p.bw = bits_of(mxd);
		break;
	}
	case FLS_SCHEME_RLE:
		p.aux  = LEARNED ? counts.runs : __reduce_add_sync(0xffffffffu, __popc(chunk_starts(sv, lane)));
		p.bw   = range_bits;
		p.base = mn;
		break;
	default: // DICT: the dictionary and the codes take the staged values' place
		p.aux  = distinct;
		p.bw   = range_bits;
		p.base = mn;
		write_dict(k, first, before, p.bw <= kKeyedBits, sv);
		break;
	}
	return p;
}

// Writes the planned vector's payload (staged in sv; DICT: planned) at `out`.
__device__ __forceinline__ void write_vector(const EncParams& P, uint64_t v, const Plan& p, int32_t* sv, uint32_t* out,
                                             uint32_t lane) {
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
		// run dictionary: the value at each start, in order, in the place of
		// the values
		auto*    u = reinterpret_cast<uint32_t*>(sv);
		uint32_t k = pre;
#pragma unroll
		for (uint32_t t = 0; t < 32; ++t) { x[t] = static_cast<uint32_t>(sv[33u * lane + t]) - base; }
		__syncwarp();
#pragma unroll
		for (uint32_t t = 0; t < 32; ++t) {
			if ((f >> t) & 1u) { u[k++] = x[t]; }
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
		const uint32_t  n = p.aux;
		const uint32_t* u = dict_of(sv);
		bw                = bits_of(n - 1u);
		if (p.bw <= kKeyedBits) {
#pragma unroll
			for (uint32_t r = 0; r < 32; ++r) { x[r] = codes_of(sv)[code_pos(layout_index(P.layout, lane, r))]; }
		} else { // the values once more, from the column
			const uint64_t v0 = v * 1024u;
#pragma unroll
			for (uint32_t r = 0; r < 32; ++r) {
				const uint64_t i   = min(v0 + layout_index(P.layout, lane, r), P.n - 1u);
				const uint32_t val = static_cast<uint32_t>(__ldg(P.values + i)) - base;
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

// What the warps of a CTA share on a tile.
struct TileShared {
	uint32_t words[kEncWarps], mask[kEncWarps];
	uint64_t offset;
};

// The scanning CTA's own tile is the next to be answered.
__device__ __forceinline__ void offset_alone(TileShared& T, ScanState* scan, uint64_t own, uint32_t lane) {
	const uint32_t hi = static_cast<uint32_t>(own >> 32) & 0x7fffffffu;
	if (lane == 0) { T.offset = kTileMark | scan->run; }
	__syncwarp();
	scan->pos += 1u;
	scan->run += static_cast<uint32_t>(own);
	scan->mx = max(scan->mx, hi & 0xffffu);
	scan->mask |= hi >> 16;
}

// One tile by the CTA; returns whether the warp's vector fell back to the
// exhaustive choice.  ALONE: by the scanning CTA (scan: warp 0's state).
template <bool LEARNED, bool ALONE>
__device__ __forceinline__ bool encode_tile(const EncParams& P, uint64_t tile, int32_t* sv, const float* net,
                                            TileShared& T, ScanState* scan, uint32_t warp, uint32_t lane) {
	const uint64_t v    = tile * kEncWarps + warp;
	const bool     live = v < P.n_vec;
	Plan           p {};
	uint32_t       words = 0;
	int32_t        mn = 0, mx = 0;
	sel::Counts    counts {};
	uint32_t       scheme = 0;
	bool           unsure = false;
	if (live) { sel::stage_vector(P.values, P.n, v, sv, lane, mn, mx); }
	// the vector this warp is likely to take next: from memory to L2
	const uint64_t ahead = v + static_cast<uint64_t>(gridDim.x) * kEncWarps;
	if ((ahead + 1u) * 1024u <= P.n) {
		asm volatile("prefetch.global.L2 [%0];" ::"l"(P.values + ahead * 1024u + 32u * lane));
	}
	if constexpr (LEARNED) {
		if (live) {
			const float f = sel::vector_features(sv, mn, mx, reinterpret_cast<uint8_t*>(sv + sel::kPadded), lane, counts);
			float       z[sel::kOut], top;
			sel::WarpNet::forward(net, reinterpret_cast<float*>(sv + kNetWords), f, lane, z);
			sel::softmax5(z);
			scheme = static_cast<uint32_t>(sel::top_of(z, top));
			unsure = top < P.threshold;
			__syncwarp(); // the activations are read before the warp's words serve something else
		}
	} else if (live) {
		scheme = P.schemes ? P.schemes[v] : P.scheme;
		if (scheme >= FLS_N_SCHEMES) {
			if (lane == 0) { atomicOr(P.err, kErrBadMeta); }
			scheme = FLS_SCHEME_FOR;
		}
	}
	if (live) {
		p     = plan_vector<LEARNED>(P, v, sv, lane, mn, mx, scheme, counts, unsure);
		words = payload_words(p.scheme, p.bw, p.aux);
		if (LEARNED && P.picks && lane == 0) { P.picks[v] = static_cast<uint8_t>(scheme); }
	}
	if (lane == 0) {
		T.words[warp] = words;
		T.mask[warp]  = live ? 1u << p.scheme : 0u;
	}
	__syncthreads();
	if (warp == 0) {
		const uint32_t w = lane < kEncWarps ? T.words[lane] : 0u, m = lane < kEncWarps ? T.mask[lane] : 0u;
		const uint64_t own = tile_report(__reduce_add_sync(0xffffffffu, w), __reduce_max_sync(0xffffffffu, w),
		                                 __reduce_or_sync(0xffffffffu, m));
		if (ALONE) {
			offset_alone(T, scan, own, lane);
		} else if (lane == 0) {
			tile_store(P.reports + tile, own);
			uint64_t got = 0;
			for (uint32_t poll = 0; poll < P.tile_polls && got == 0ull; ++poll) { got = tile_load(P.offsets + tile); }
			if (got == 0ull) {
				tile_lost(P);
				got = kTileLost;
			}
			T.offset = got;
		}
	}
	__syncthreads();
	const uint64_t before = T.offset;
	if (live && before != kTileLost) {
		uint64_t offset = before & ~kTileMark;
		for (uint32_t w = 0; w < warp; ++w) { offset += T.words[w]; }
		if (lane == 0) {
			fls_vec_meta m;
			m.offset  = offset;
			m.base    = p.base;
			m.scheme  = static_cast<uint8_t>(p.scheme);
			m.bw      = static_cast<uint8_t>(p.bw);
			m.aux     = static_cast<uint16_t>(p.aux);
			P.meta[v] = m;
		}
		write_vector(P, v, p, sv, P.out + offset, lane);
	} else if (live && lane == 0) { // metadata that every decoder refuses
		fls_vec_meta m {};
		m.scheme  = FLS_N_SCHEMES;
		P.meta[v] = m;
	}
	__syncthreads(); // T is read before the next tile's
	return unsure;
}

// The rest of the column by the scanning CTA, from the tile of `ticket` on, with
// whatever tiles other CTAs have taken in between.  Returns the warp's
// fallbacks.  Apart from the kernel's loop, so that the registers of the scan and
// of a tile stay apart there (33.5 M values as a dictionary, kernel: 264 us
// without it, 270 with it, 276 where the scan went back into the loop).
template <bool LEARNED>
__device__ __forceinline__ uint32_t encode_alone(const EncParams& P, uint32_t ticket, int32_t* sv, const float* net,
                                              TileShared& T, uint32_t& s_tile, ScanState scan, uint32_t warp,
                                              uint32_t lane) {
	uint32_t fallbacks = 0;
	while (ticket != 0u) {
		fallbacks += encode_tile<LEARNED, true>(P, ticket - 1u, sv, net, T, &scan, warp, lane) ? 1u : 0u;
		if (warp == 0) {
			ticket = scan_tiles(P, scan, 1u, lane); // still alone: the next tile at once
			if (lane == 0) { s_tile = ticket; }
		}
		__syncthreads();
		ticket = s_tile;
		__syncthreads();
	}
	return fallbacks;
}

// Bounded by the per-vector work of planning (DICT: the sort; LEARNED: the
// statistics and the network, about 6 us of a round of 24 vectors per SM) and,
// in columns of few rounds, by the round trip of a tile's offset, 2-4 us.
// 1568 words per warp let three CTAs (24 warps) share an SM.  Against separate
// plan, scan and write kernels, which read and sorted everything twice, whole
// encoder calls took (us, before -> after; about 40 of each are the call's
// host side and its read-back): 6 M values DICT 437 -> 104, 33.5 M values FOR
// 186 -> 120, DELTA 185 -> 118, RLE 185 -> 145, DICT 1920 -> 315.
//
// LEARNED: a warp first takes its vector's statistics and runs the network on
// them (fls_selector.cuh), so the values are still read once and the column
// takes one launch instead of eight (four columns of 8.4 M values: statistics
// 20, network 21, choice 6, plan 18, scans 10, write 18-41 us each -> 40-50;
// the whole call 576 -> 325 us).
template <bool LEARNED>
__global__ void __launch_bounds__(kEncWarps * 32, 3) enc_kernel(const __grid_constant__ EncParams P) {
	extern __shared__ __align__(16) int32_t esmem[];
	__shared__ uint32_t   s_tile;
	__shared__ TileShared s_shared;
	__shared__ ScanState  s_scan; // of the CTA with the first ticket
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	int32_t*       sv   = esmem + warp * kEncWarpWords;
	float*         net  = reinterpret_cast<float*>(esmem + kEncWarps * kEncWarpWords); // LEARNED
	uint32_t       fallbacks = 0; // of this warp's vectors
	if constexpr (LEARNED) { sel::WarpNet::load(P.params, net); }
	for (;;) {
		// taken only now: a tile taken ahead of its work would hold up every
		// tile after it
		if (threadIdx.x == 0) { s_tile = atomicAdd(P.counter, 1u); }
		__syncthreads();
		if (s_tile == 0u) { // the first ticket: this CTA adds up the tiles
			__syncthreads(); // s_tile is read
			if (warp == 0) {
				if (lane == 0) { s_scan = ScanState {}; }
				__syncwarp();
				const uint32_t ticket = scan_tiles(P, s_scan, kAloneRounds, lane);
				if (lane == 0) { s_tile = ticket; }
			}
			__syncthreads();
			break;
		}
		const uint64_t tile = s_tile - 1u;
		if (tile >= P.n_tiles) { break; }
		fallbacks += encode_tile<LEARNED, false>(P, tile, sv, net, s_shared, nullptr, warp, lane) ? 1u : 0u;
	}
	// s_tile: past the last tile, or, in the scanning CTA, 0 or a tile to go on with
	if (s_tile != 0u && s_tile <= P.n_tiles) {
		fallbacks += encode_alone<LEARNED>(P, s_tile, sv, net, s_shared, s_tile, s_scan, warp, lane);
	}
	if constexpr (LEARNED) {
		// The last CTA to get here reports the fallbacks of all.
		if (lane == 0 && fallbacks) { atomicAdd(P.n_fallback, static_cast<unsigned long long>(fallbacks)); }
		__threadfence();
		__syncthreads();
		if (threadIdx.x == 0 && atomicAdd(P.counter + 1, 1u) + 1u == gridDim.x) {
			__threadfence();
			P.info[3] = atomicAdd(P.n_fallback, 0ull);
		}
	}
}

uint64_t workspace_bytes_of(uint64_t n) {
	const uint64_t n_vec = (n + 1023u) / 1024u, n_tiles = (n_vec + kEncWarps - 1) / kEncWarps;
	return 16u * n_tiles + 256u; // the counters, the tiles' reports and offsets, after alignment
}

// Checks the arguments both encoders share, fills in the rest of P and
// launches the kernel: one memset of the tiles' states, one launch.  max_ctas:
// of the launch (0: as many as are resident).
template <bool LEARNED>
fls_status encode_launch(EncParams& P, uint64_t out_capacity_words, void* d_workspace, uint64_t workspace_bytes,
                         cudaStream_t st, const std::string& who, uint32_t max_ctas = 0) {
	if (!P.values || !P.out || !P.meta || !P.info || !d_workspace || P.n == 0) {
		return set_error(FLS_ERR_INVALID_ARG, who + ": null pointer or n == 0");
	}
	if (fls_status s = check_n_values(P.n, who.c_str()); s != FLS_OK) { return s; }
	if (P.layout > FLS_LAYOUT_TRANSPOSED) { return set_error(FLS_ERR_INVALID_ARG, who + ": bad layout"); }
	if ((reinterpret_cast<uintptr_t>(P.out) | reinterpret_cast<uintptr_t>(P.meta)) & 15u) {
		return set_error(FLS_ERR_ALIGNMENT, who + ": output and metadata must be 16-byte aligned");
	}
	P.n_vec = (P.n + 1023u) / 1024u;
	if (out_capacity_words < P.n_vec * kMaxVecWords) {
		return set_error(FLS_ERR_CAPACITY, who + ": output smaller than fls_encode_bound_words(n)");
	}
	if (workspace_bytes < workspace_bytes_of(P.n)) {
		return set_error(FLS_ERR_CAPACITY, who + ": workspace smaller than " +
		                                       (LEARNED ? "fls_encode_learned_workspace_bytes(n)" : "fls_encode_gpu_workspace_bytes(n)"));
	}
	DeviceInfo di;
	fls_status s = device_info(di);
	if (s != FLS_OK) { return s; }
	char* ws     = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(d_workspace) + 15u) & ~uintptr_t {15u});
	P.n_tiles    = (P.n_vec + kEncWarps - 1) / kEncWarps;
	P.counter    = reinterpret_cast<uint32_t*>(ws);
	P.n_fallback = reinterpret_cast<unsigned long long*>(ws + 8);
	P.lost       = reinterpret_cast<uint32_t*>(ws + 16);
	P.reports    = reinterpret_cast<uint64_t*>(ws + 32);
	P.offsets    = P.reports + P.n_tiles;
	P.err        = device_error_word(st);
	const size_t smem = 4u * (kEncWarps * kEncWarpWords + (LEARNED ? sel::WarpNet::kFloats : 0u));
	{
		static std::mutex mu;
		static uint64_t   configured = 0;
		int               dev        = 0;
		cudaGetDevice(&dev);
		std::lock_guard<std::mutex> lk(mu);
		if (dev >= 64 || !(configured & (1ull << dev))) {
			if ((s = cuda_check(cudaFuncSetAttribute(enc_kernel<LEARNED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
			                                         static_cast<int>(smem)),
			                    "cudaFuncSetAttribute")) != FLS_OK) {
				return s;
			}
			if (dev < 64) { configured |= 1ull << dev; }
		}
	}
	if ((s = cuda_check(cudaMemsetAsync(ws, 0, 32u + 16u * P.n_tiles, st), "cudaMemsetAsync")) != FLS_OK) { return s; }
	const uint32_t grid = static_cast<uint32_t>(
	    std::min<uint64_t>(P.n_tiles + 1u, max_ctas ? max_ctas : static_cast<uint64_t>(di.sms) * 3u));
	enc_kernel<LEARNED><<<grid, kEncWarps * 32, smem, st>>>(P);
	count_launch();
	return cuda_check(cudaGetLastError(), "enc_kernel launch");
}

} // namespace
} // namespace fls

using namespace fls;

extern "C" {

uint64_t fls_encode_gpu_workspace_bytes(uint64_t n) { return workspace_bytes_of(n); }

fls_status fls_encode_column_gpu(const int32_t* d_values, uint64_t n, const uint8_t* d_schemes, uint32_t scheme,
                                 uint32_t layout, int round4, uint32_t* d_out, uint64_t out_capacity_words,
                                 fls_vec_meta* d_meta, uint64_t* d_info, void* d_workspace, uint64_t workspace_bytes,
                                 fls_stream_t stream) {
	if (!d_schemes && scheme >= FLS_N_SCHEMES) { return set_error(FLS_ERR_INVALID_ARG, "fls_encode_column_gpu: bad scheme"); }
	EncParams P {};
	P.values  = d_values;
	P.n       = n;
	P.schemes = d_schemes;
	P.scheme  = scheme;
	P.layout  = layout;
	P.round4  = round4 ? 1u : 0u;
	P.out     = d_out;
	P.meta    = d_meta;
	P.info    = d_info;
	P.scan_polls = P.tile_polls = kPollLimit;
	return encode_launch<false>(P, out_capacity_words, d_workspace, workspace_bytes,
	                            reinterpret_cast<cudaStream_t>(stream), "fls_encode_column_gpu");
}

uint64_t fls_encode_learned_workspace_bytes(uint64_t n) { return workspace_bytes_of(n); }

fls_status fls_encode_learned_gpu(const int32_t* d_values, uint64_t n, const float* d_params, float threshold,
                                  double kappa, uint32_t layout, uint32_t* d_out, uint64_t out_capacity_words,
                                  fls_vec_meta* d_meta, uint64_t* d_info, uint8_t* d_schemes, void* d_workspace,
                                  uint64_t workspace_bytes, fls_stream_t stream) {
	if (!d_params) { return set_error(FLS_ERR_INVALID_ARG, "fls_encode_learned_gpu: null pointer or n == 0"); }
	if (!(kappa >= 0.0)) { return set_error(FLS_ERR_INVALID_ARG, "fls_encode_learned_gpu: kappa must be >= 0"); }
	if (reinterpret_cast<uintptr_t>(d_workspace) & 255u) {
		return set_error(FLS_ERR_CAPACITY, "fls_encode_learned_gpu: workspace not 256-byte aligned");
	}
	EncParams P {};
	P.values    = d_values;
	P.n         = n;
	P.layout    = layout;
	P.out       = d_out;
	P.meta      = d_meta;
	P.info      = d_info;
	P.params    = d_params;
	P.threshold = threshold;
	P.kappa     = kappa;
	P.picks     = d_schemes;
	P.scan_polls = P.tile_polls = kPollLimit;
	return encode_launch<true>(P, out_capacity_words, d_workspace, workspace_bytes,
	                           reinterpret_cast<cudaStream_t>(stream), "fls_encode_learned_gpu");
}

fls_status fls_selftest_encode_waits(const int32_t* d_values, uint64_t n, uint32_t scheme, const float* d_params,
                                     uint32_t* d_out, uint64_t out_capacity_words, fls_vec_meta* d_meta,
                                     uint64_t* d_info, void* d_workspace, uint64_t workspace_bytes, uint32_t ctas,
                                     uint32_t scan_polls, uint32_t tile_polls, fls_stream_t stream) {
	if (scheme >= FLS_N_SCHEMES || ctas == 0 || scan_polls > kPollLimit || tile_polls > kPollLimit) {
		return set_error(FLS_ERR_INVALID_ARG, "fls_selftest_encode_waits: bad scheme, CTAs or limits");
	}
	EncParams P {};
	P.values     = d_values;
	P.n          = n;
	P.scheme     = scheme;
	P.layout     = FLS_LAYOUT_TRANSPOSED;
	P.out        = d_out;
	P.meta       = d_meta;
	P.info       = d_info;
	P.scan_polls = scan_polls;
	P.tile_polls = tile_polls;
	P.params     = d_params;
	P.threshold  = 0.9f;
	const auto st = reinterpret_cast<cudaStream_t>(stream);
	return d_params ? encode_launch<true>(P, out_capacity_words, d_workspace, workspace_bytes, st, __func__, ctas)
	                : encode_launch<false>(P, out_capacity_words, d_workspace, workspace_bytes, st, __func__, ctas);
}

} // extern "C"
