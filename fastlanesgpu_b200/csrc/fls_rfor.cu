// fls_rfor.cu -- GPU decoder of the tile-based run-length format (RFOR) of
// the reference's tile_based codecs: decode to HBM and decode fused with a
// uint64 sum.
//
// The reference decodes a 512-value tile with a CTA of 128 threads
// (LoadRBinPack, tile_based/src/include/rlebinpack_kernel.cuh:20-145): the
// runs' values and lengths are unpacked, an exchange and a block scan turn
// the lengths into run ends, the ends are marked in shared memory, a second
// block scan turns the marks into each position's run index, and the values
// are gathered.  Here one warp decodes a tile with no block-wide barrier:
//   1. lane l takes runs l, l + 32, ...: 32 fields of a packed block fill
//      exactly bw words, so a lane's fields all start at the same bit and its
//      shift and mask are constants; a warp scan of the lengths per 32 runs
//      gives each run's first position (a tile of many runs: contiguous chunks
//      and one scan, see many_runs);
//   2. the sum needs no more: a run adds its value times its length, and a
//      whole tile's not even the positions;
//   3. to memory, each lane writes its runs' values to shared memory and sets
//      the bit of each run's first position in a 512-bit mask (16 words);
//   4. a lane writes four consecutive positions at a time: the first is in run
//      popc(mask bits up to it) - 1, each next one a run further where its bit
//      is set; the values are gathered from shared memory.
// Runs of length 0 cover no position: they add nothing to the sum and, to
// memory, set no bit and keep no value (the values kept are those of the runs
// that have a bit, in order).
// A tile whose block is inconsistent is skipped and flagged, never read past
// its stream.
//
// Bounded by integer issue (68 % of it active, 430 warp instructions per tile to
// memory) and, in the rest, by reads and chains of shuffles that too few warps
// cover.  16.8 M values of geometric runs (mean 16), whole call, against
// contiguous chunks of runs per lane, one position per lane and row and the sum
// over expanded positions: to memory 22.7 -> 20.7 us, sum 22.8 -> 14.5.
#include "fls_pipeline.cuh"

namespace fls {
namespace {

constexpr uint32_t kTile      = FLS_RFOR_TILE;
constexpr uint32_t kRforWarps = 8;

struct RforParams {
	const uint32_t *vals, *rls, *val_off, *rl_off;
	uint64_t        n_values, n_tiles, n_val_words, n_rl_words;
	uint32_t*       out;
	unsigned long long* sum;
	uint32_t*       err;
};

__device__ __forceinline__ uint32_t packed_words(uint32_t count, uint32_t bw) {
	const uint32_t bits = count * bw; // count <= 512, bw <= 32
	return bits == 0 ? 1u : (bits + 31u) >> 5;
}

// A lane's fields lane, lane + 32, ... of a sequentially packed block (bit
// k*bw, LSB first): word row i of bw words holds fields 32 i .. 32 i + 31.
// Never reads past the block's last packed word.
struct LaneFields {
	const uint32_t* p;
	uint32_t        bw, sh, mask, next;
	__device__ __forceinline__ LaneFields(const uint32_t* block, uint32_t width, uint32_t lane) {
		const uint32_t bit = lane * width;
		p    = block + (bit >> 5);
		bw   = width;
		sh   = bit & 31u;
		mask = width >= 32 ? 0xffffffffu : ((1u << width) - 1u);
		next = sh + width > 32u ? 1u : 0u; // without a second word the first is read twice and masked off
	}
	// Row i's field; the caller has checked that it is one of the block's.
	__device__ __forceinline__ uint32_t get(uint32_t i) const {
		if (bw == 0) { return 0u; } // warp-uniform
		const uint32_t* q = p + i * bw;
		return __funnelshift_r(__ldg(q), __ldg(q + next), sh) & mask;
	}
	__device__ __forceinline__ const uint32_t* block(uint32_t lane) const { return p - ((lane * bw) >> 5); }
	// Field k of the block, whichever lane's it is (a block of width 0 still has one word).
	__device__ __forceinline__ uint32_t any(const uint32_t* block, uint32_t k) const {
		const uint32_t  bit = k * bw, s = bit & 31u;
		const uint32_t* q = block + (bit >> 5);
		return __funnelshift_r(__ldg(q), s + bw > 32u ? __ldg(q + 1) : 0u, s) & mask;
	}
};

// The values of a tile's positions, four consecutive ones at a time per lane
// (positions 128 j + 4 lane .. + 3), handed to f(first position, values);
// words[w] = {mask bits of positions 32 w .. 32 w + 31, run starts before them
// minus one}.
template <class F>
__device__ __forceinline__ void expand_rows(const uint2* words, const uint32_t* vals, uint32_t lane, F&& f) {
	const uint32_t sh = 4u * (lane & 7u), upto = 0xffffffffu >> (31u - sh);
#pragma unroll
	for (uint32_t j = 0; j < kTile / 128; ++j) {
		const uint2 w = words[4u * j + (lane >> 3)];
		uint32_t    k = w.y + __popc(w.x & upto);
		uint4       v;
		v.x = vals[k];
		k += (w.x >> (sh + 1u)) & 1u;
		v.y = vals[k];
		k += (w.x >> (sh + 2u)) & 1u;
		v.z = vals[k];
		k += (w.x >> (sh + 3u)) & 1u;
		v.w = vals[k];
		f(128u * j + 4u * lane, v);
	}
}

// A tile's two blocks {minimum, bit width per byte, count, fields}, read and
// checked by one lane: 32 tiles of the warp at a time, so that a tile costs
// five shuffles where every lane read and checked the same words, two round
// trips to memory one after the other.
constexpr uint32_t kBadTile = 0xffffffffu;
struct TileHead {
	uint32_t vo, ro;     // 32-bit word offsets of the blocks
	uint32_t vmin, rmin;
	uint32_t widths;     // count | value width << 16 | length width << 24, or kBadTile
};

__device__ __forceinline__ TileHead load_head(const RforParams& P, uint64_t t) {
	TileHead h {0u, 0u, 0u, 0u, kBadTile};
	if (t >= P.n_tiles) { return h; }
	const uint32_t vo = __ldg(P.val_off + t), ve = __ldg(P.val_off + t + 1);
	const uint32_t ro = __ldg(P.rl_off + t), re = __ldg(P.rl_off + t + 1);
	bool           ok = static_cast<uint64_t>(vo) + 3u <= ve && ve <= P.n_val_words &&
	          static_cast<uint64_t>(ro) + 3u <= re && re <= P.n_rl_words;
	if (ok) {
		const uint32_t *v = P.vals + vo, *r = P.rls + ro;
		const uint32_t  vbw = __ldg(v + 1) & 0xffu, rbw = __ldg(r + 1) & 0xffu, cnt = __ldg(v + 2);
		h.vmin = __ldg(v);
		h.rmin = __ldg(r);
		ok     = vbw <= 32u && rbw <= 32u && cnt >= 1u && cnt <= kTile && __ldg(r + 2) == cnt &&
		     static_cast<uint64_t>(vo) + 3u + packed_words(cnt, vbw) <= ve &&
		     static_cast<uint64_t>(ro) + 3u + packed_words(cnt, rbw) <= re;
		h.vo     = vo;
		h.ro     = ro;
		h.widths = ok ? cnt | (vbw << 16) | (rbw << 24) : kBadTile;
	}
	if (!ok) { raise_err(P.err, kErrBadMeta); }
	return h;
}

// Tiles of more than kFewRuns runs: each lane takes a contiguous chunk of the
// runs, so that a tile takes one scan, its words are all asked for by the first
// run of the chunks, and neighbouring starts are marked by one lane after the
// other.  32 runs at a time take a chain of five shuffles and a round trip to
// memory per 32 runs, and their starts, close together, meet in a word or two,
// one atomic after the other (16.8 M values, whole call, 32 at a time -> this:
// to memory, runs of mean 2 57 -> 37 and 4 37 -> 27 us; 1 stays at 104, bound by
// the bank conflicts of chunks of 16; sums 64 -> 51, 48 -> 34 and 31 -> 23 with
// the whole tiles' sums below).  `total`: the positions covered; SUM (of the
// positions below `live`) into part.  False where a run has length 0 or passes
// the tile: nothing that counts is done then.
constexpr uint32_t kFewRuns = 64;
template <bool SUM>
__device__ __forceinline__ bool many_runs(const LaneFields& vf, const LaneFields& rf, uint32_t vmin, uint32_t rmin,
                                          uint32_t cnt, uint32_t live, uint32_t* vals, uint16_t* lens, uint2* words,
                                          uint32_t lane, uint32_t& total, unsigned long long& part) {
	const uint32_t *vb = vf.block(lane), *rb = rf.block(lane);
	const uint32_t chunk = (cnt + 31u) >> 5, k0 = min(cnt, lane * chunk), k1 = min(cnt, k0 + chunk);
	uint32_t       own = 0, most = 0; // most: the largest length minus one
	for (uint32_t k = k0; k < k1; ++k) {
		const uint32_t l = rmin + rf.any(rb, k);
		if constexpr (!SUM) {
			vals[k] = vmin + vf.any(vb, k);
			lens[k] = static_cast<uint16_t>(l);
		}
		most = max(most, l - 1u);
		own += l;
	}
	if (!__all_sync(0xffffffffu, most < kTile)) {
		__syncwarp(); // the values are written once more
		return false;
	}
	uint32_t incl = own;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
		if (lane >= static_cast<uint32_t>(o)) { incl += x; }
	}
	total = __shfl_sync(0xffffffffu, incl, 31);
	if (total == kTile) { // every run starts inside the tile
		uint32_t pos = incl - own;
		for (uint32_t k = k0; k < k1; ++k) {
			if constexpr (SUM) {
				const uint32_t l = rmin + rf.any(rb, k);
				part += static_cast<unsigned long long>(vmin + vf.any(vb, k)) * (min(pos + l, live) - min(pos, live));
				pos += l;
			} else { // each lane reads back its own lengths
				atomicOr(&words[pos >> 5].x, 1u << (pos & 31u));
				pos += lens[k];
			}
		}
	}
	return true;
}

// WIDE: the output is 16-byte aligned.  To memory five CTAs share an SM: at six
// the 40 registers a thread spill (runs of mean 16 20.6 -> 23.8 us).
template <bool SUM, bool WIDE>
__global__ void __launch_bounds__(kRforWarps * 32, SUM ? 6 : 5) rfor_kernel(const __grid_constant__ RforParams P) {
	__shared__ uint32_t s_vals[SUM ? 1 : kRforWarps][kTile];
	__shared__ uint2    s_words[SUM ? 1 : kRforWarps][kTile / 32];
	__shared__ uint16_t s_lens[SUM ? 1 : kRforWarps][kTile];
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	uint32_t*      vals  = s_vals[SUM ? 0 : warp];
	uint2*         words = s_words[SUM ? 0 : warp];
	uint16_t*      lens  = s_lens[SUM ? 0 : warp];
	unsigned long long acc = 0;
	const uint64_t total = static_cast<uint64_t>(gridDim.x) * kRforWarps;
	const uint64_t first = static_cast<uint64_t>(blockIdx.x) * kRforWarps + warp;
	TileHead       head {};
	uint32_t       j = 31u; // lane that holds the current tile
	for (uint64_t t = first; t < P.n_tiles; t += total) {
		j = (j + 1u) & 31u;
		if (j == 0) { head = load_head(P, t + lane * total); }
		const uint32_t widths = __shfl_sync(0xffffffffu, head.widths, j);
		if (widths == kBadTile) { continue; } // flagged by the lane that read it
		const uint32_t cnt  = widths & 0xffffu;
		const uint32_t vmin = __shfl_sync(0xffffffffu, head.vmin, j), rmin = __shfl_sync(0xffffffffu, head.rmin, j);
		const LaneFields vf(P.vals + __shfl_sync(0xffffffffu, head.vo, j) + 3u, (widths >> 16) & 0xffu, lane);
		const LaneFields rf(P.rls + __shfl_sync(0xffffffffu, head.ro, j) + 3u, widths >> 24, lane);
		const uint64_t   row0 = t * kTile;
		const uint32_t   live = static_cast<uint32_t>(min(static_cast<uint64_t>(kTile), P.n_values - row0));
		if constexpr (!SUM) {
			if (lane < kTile / 32) { words[lane] = make_uint2(0u, 0u); }
			__syncwarp();
		}
		uint32_t           start = 0; // of the next 32 runs
		unsigned long long part  = 0;
		bool               fits  = true, grouped = true;
		if (SUM && live == kTile) {
			// A whole tile's sum needs no positions: no scan, every read
			// independent of the one before.  (Unrolled it is slower, 34 -> 41
			// us at runs of mean 2.)
			grouped        = false;
			uint32_t cover = 0;
#pragma unroll 1
			for (uint32_t i = 0; 32u * i < cnt; ++i) {
				if (32u * i + lane < cnt) {
					const uint32_t l = rmin + rf.get(i), v = vmin + vf.get(i);
					fits             = fits && l <= kTile;
					cover += l;
					part += static_cast<unsigned long long>(v) * l;
				}
			}
			start = __reduce_add_sync(0xffffffffu, cover);
		}
		if (cnt > kFewRuns && grouped) {
			grouped = !many_runs<SUM>(vf, rf, vmin, rmin, cnt, live, vals, lens, words, lane, start, part);
		}
		if (grouped) {
			// Runs 32 i + lane, until the tile's runs are used up (a tile whose
			// runs do not cover it exactly is found out at the end: nothing of
			// it has been added or written by then).
			[[maybe_unused]] uint32_t empty = 0; // runs of length 0 so far
			for (uint32_t i = 0; 32u * i < cnt; ++i) {
				const uint32_t k    = 32u * i + lane;
				const bool     mine = k < cnt;
				uint32_t       l = 0, v = 0;
				if (mine) {
					l = rmin + rf.get(i);
					v = vmin + vf.get(i);
				}
				fits          = fits && l <= kTile; // sums of 32 lengths below stay far from 32 bits
				uint32_t incl = l;
#pragma unroll
				for (int o = 1; o < 32; o <<= 1) {
					const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
					if (lane >= static_cast<uint32_t>(o)) { incl += x; }
				}
				const uint32_t pos = start + incl - l;
				if constexpr (SUM) {
					// the run's positions below `live`
					part += static_cast<unsigned long long>(v) * (min(pos + l, live) - min(pos, live));
				} else {
					uint32_t       at   = k - empty;
					const uint32_t none = __ballot_sync(0xffffffffu, mine && l == 0u);
					if (none) { // not in this library's streams
						at -= __popc(none & ((1u << lane) - 1u));
						empty += __popc(none);
					}
					if (l != 0u && pos < kTile) { // past the tile: found out below
						vals[at] = v;
						atomicOr(&words[pos >> 5].x, 1u << (pos & 31u));
					}
				}
				start += __shfl_sync(0xffffffffu, incl, 31);
				if (!__all_sync(0xffffffffu, fits)) { break; }
			}
		}
		if (start != kTile || !__all_sync(0xffffffffu, fits)) { // the runs must cover the tile exactly
			if (lane == 0) { raise_err(P.err, kErrBadMeta); }
			__syncwarp();
			continue;
		}
		if constexpr (SUM) {
			acc += part;
		} else {
			__syncwarp();
			// run starts before each mask word, minus one
			const uint32_t own = lane < kTile / 32 ? __popc(words[lane].x) : 0u;
			uint32_t       c   = own;
#pragma unroll
			for (int o = 1; o < 16; o <<= 1) {
				const uint32_t x = __shfl_up_sync(0xffffffffu, c, o);
				if (lane >= static_cast<uint32_t>(o)) { c += x; }
			}
			if (lane < kTile / 32) { words[lane].y = c - own - 1u; }
			__syncwarp();
			uint32_t* out = P.out + row0;
			if (WIDE && live == kTile) {
				expand_rows(words, vals, lane,
				            [&](uint32_t p, const uint4& v) { __stcs(reinterpret_cast<uint4*>(out + p), v); });
			} else {
				expand_rows(words, vals, lane, [&](uint32_t p, const uint4& v) {
					const uint32_t e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
					for (uint32_t i = 0; i < 4; ++i) {
						if (p + i < live) { __stcs(out + p + i, e[i]); }
					}
				});
			}
			__syncwarp();
		}
	}
	if constexpr (SUM) {
		const unsigned long long s = warp_sum_u64(acc);
		if (lane == 0 && s) { atomicAdd(P.sum, s); }
	}
}

fls_status rfor_launch(const fls_rfor_column* col, uint32_t* d_out, uint64_t* d_sum, fls_stream_t stream,
                       const char* who) {
	if (!col || !col->values || !col->run_lengths || !col->val_offsets || !col->rl_offsets || (!d_out && !d_sum)) {
		return set_error(FLS_ERR_INVALID_ARG, std::string(who) + ": null pointer");
	}
	if (col->n_values == 0 || col->n_values > 0xffffffffull) {
		return set_error(FLS_ERR_INVALID_ARG, std::string(who) + ": 1..2^32-1 values");
	}
	DeviceInfo di;
	fls_status s = device_info(di);
	if (s != FLS_OK) { return s; }
	cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
	RforParams   P {};
	P.vals        = col->values;
	P.rls         = col->run_lengths;
	P.val_off     = col->val_offsets;
	P.rl_off      = col->rl_offsets;
	P.n_values    = col->n_values;
	P.n_tiles     = (col->n_values + kTile - 1) / kTile;
	P.n_val_words = col->n_val_words;
	P.n_rl_words  = col->n_rl_words;
	P.out         = d_out;
	P.sum         = reinterpret_cast<unsigned long long*>(d_sum);
	P.err         = device_error_word(st);
	if (d_sum && (s = cuda_check(cudaMemsetAsync(d_sum, 0, sizeof(uint64_t), st), "cudaMemsetAsync")) != FLS_OK) {
		return s;
	}
	const uint32_t grid = static_cast<uint32_t>(
	    std::min<uint64_t>((P.n_tiles + kRforWarps - 1) / kRforWarps, static_cast<uint64_t>(di.sms) * (d_sum ? 6u : 5u))); // resident
	if (d_sum) {
		rfor_kernel<true, false><<<grid, kRforWarps * 32, 0, st>>>(P);
	} else if ((reinterpret_cast<uintptr_t>(d_out) & 15u) == 0) {
		rfor_kernel<false, true><<<grid, kRforWarps * 32, 0, st>>>(P);
	} else {
		rfor_kernel<false, false><<<grid, kRforWarps * 32, 0, st>>>(P);
	}
	count_launch();
	return cuda_check(cudaGetLastError(), "rfor_kernel launch");
}

} // namespace
} // namespace fls

using namespace fls;

extern "C" {

fls_status fls_rfor_decode_u32(const fls_rfor_column* col, uint32_t* d_out, fls_stream_t stream) {
	if (!d_out) { return set_error(FLS_ERR_INVALID_ARG, "fls_rfor_decode_u32: null output"); }
	return rfor_launch(col, d_out, nullptr, stream, "fls_rfor_decode_u32");
}

fls_status fls_rfor_decode_sum_u32(const fls_rfor_column* col, uint64_t* d_sum, fls_stream_t stream) {
	if (!d_sum) { return set_error(FLS_ERR_INVALID_ARG, "fls_rfor_decode_sum_u32: null output"); }
	return rfor_launch(col, nullptr, d_sum, stream, "fls_rfor_decode_sum_u32");
}

} // extern "C"
