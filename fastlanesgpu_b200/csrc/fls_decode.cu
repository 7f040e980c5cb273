// fls_decode.cu -- decode-to-HBM and decode-fused-sum operators.
//
// Reference counterparts: unpack_global (fastlanes/src/include/fls_gen/unpack/
// unpack.cuh:3436), QueryKernel of bitpack_shared_memory.cu:21 /
// bitpack_register.cu:21 (decode + sum), delta_shared_memory.cu:24 (delta +
// sum) and delta_global_memory.cu:24 (delta to global memory).
#include <algorithm>

#include "fls_pipeline.cuh"

namespace fls {
namespace {

// ------------------------------------------------------- column pipeline
//
// One column, vector by vector: warp w of the grid takes vectors w, w + total,
// ... and keeps a ring of `slots` of them in flight, one bulk copy and one
// mbarrier each.  Lane l holds the metadata of the warp's l-th next vector
// (read and checked 32 vectors at a time, the following 32 a window ahead), so
// a vector costs a few shuffles where a tile of the general pipeline reads,
// checks and shares its metadata anew (about 200 instructions per tile, of one
// to three vectors).  50 M values, us before -> after: sum FOR 35 -> 27, DELTA
// 27 -> 23, RLE 37 -> 33, DICT 62 -> 46; to memory, bound by the writes, RLE 41
// -> 38, DICT 78 -> 57, FOR and DELTA unchanged at 5.5 TB/s; 4 M values, which
// now reach every SM, 10.2 -> 8.0 to 8.9.
//
// A uniform column's vectors lie one after the other at one size, so there a
// ring's slot holds a tile of several of them, by one copy, and their metadata is
// the column's.  Sums only: to memory the writes bind.  (134 M values, sum, in
// tiles of the general pipeline -> vector by vector -> now: DELTA of 2 bits 45.5
// -> 55.5 -> 35.4 us, of 9 bits 51.3 -> 56.3 -> 39.1; FOR of 4 bits by the general
// kernel 49.6 -> 60.0 -> 41.2.)
struct ColumnCfg {
	DevCol    col;
	uint64_t  n_vec, n_values;
	uint64_t  n_items;    // what the ring holds: vectors, or tiles of a uniform column
	uint32_t  tile;       // vectors per item
	uint32_t  slots;      // ring depth
	uint32_t  slot_words; // multiple of 4
	uint32_t  warps;
	uint32_t  warp_words; // per-warp region (multiple of 4)
	uint32_t  dict_off, extra_off, bar_off; // into it
	uint32_t  has_dict;
	uint32_t* err;
};

constexpr uint32_t kMaxSlots = 16; // a window ahead covers any ring

// Metadata of one vector, as a lane holds it.
struct LaneMeta {
	uint64_t offset;
	uint32_t base, packed; // scheme | bw << 8 | aux << 16
	uint32_t words;        // 0 when nothing is to be copied
};

// The warp's vectors 32 w .. 32 w + 31: lane l reads and checks the l-th.
__device__ __forceinline__ LaneMeta load_window(const ColumnCfg& cfg, uint64_t first, uint64_t total, uint64_t w,
                                                uint32_t lane) {
	LaneMeta       m {0, 0, kBadScheme, 0};
	const uint64_t v = first + (32u * w + lane) * total;
	if (v < cfg.n_vec) {
		VecInfo vi {};
		bool    ok = dev::vec_info(cfg.col, v, dev::load_meta(cfg.col, v), vi);
		// RLE / DICT vectors need the dictionary scratch
		ok = ok && (cfg.has_dict || (vi.scheme != FLS_SCHEME_RLE && vi.scheme != FLS_SCHEME_DICT));
		if (ok) {
			m = LaneMeta {vi.offset, static_cast<uint32_t>(vi.base), vi.scheme | (vi.bw << 8) | (vi.aux << 16), vi.words};
		} else {
			raise_err(cfg.err, kErrBadMeta);
		}
	}
	return m;
}

// Copies the vector held by lane `src` into a slot.  Words is a multiple of 4
// and the offset too (checked), so the copy's ends are 16-byte aligned.
__device__ __forceinline__ void issue_vector(const ColumnCfg& cfg, uint32_t* slot, uint64_t* bar, const LaneMeta& m,
                                             uint32_t src, uint32_t lane, uint64_t pol) {
	if (lane == src) {
		dev::mbar_arrive_expect_tx(bar, 4u * m.words);
		if (m.words) { dev::bulk_g2s(slot, cfg.col.data + m.offset, 4u * m.words, bar, pol); }
	}
}

// The operator's view of a staged vector.
struct ColumnVec {
	VecInfo         vi;
	const uint32_t* s;
	uint32_t*       dict;
	uint32_t*       extra;
	uint64_t        v;
	__device__ uint32_t rows(const ColumnCfg& cfg, uint32_t lane) const {
		const uint64_t start = v * 1024u;
		if (start + 1024u <= cfg.n_values) { return 0xffffffffu; }
		return dev::tail_rows(cfg.col.layout, lane, static_cast<uint32_t>(cfg.n_values - start));
	}
};

// Copies tile t of a uniform column; the host has checked that the data covers
// every vector.
__device__ __forceinline__ void issue_tile(const ColumnCfg& cfg, uint32_t* slot, uint64_t* bar, uint64_t t,
                                           uint32_t lane, uint64_t pol) {
	if (lane == 0) {
		const uint64_t v0    = t * cfg.tile;
		const uint32_t bytes = static_cast<uint32_t>(min(static_cast<uint64_t>(cfg.tile), cfg.n_vec - v0)) * cfg.col.vec_words * 4u;
		dev::mbar_arrive_expect_tx(bar, bytes);
		if (bytes) { dev::bulk_g2s(slot, cfg.col.data + v0 * cfg.col.vec_words, bytes, bar, pol); }
	}
}

template <class Op, bool UNIFORM>
__global__ void __launch_bounds__(Op::kWarps * 32, 1)
    column_kernel(const __grid_constant__ ColumnCfg cfg, const __grid_constant__ Op op) {
	extern __shared__ __align__(128) uint32_t smem[];
	const uint32_t     lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	uint32_t*          base = smem + warp * cfg.warp_words;
	uint64_t*          bars = reinterpret_cast<uint64_t*>(base + cfg.bar_off);
	typename Op::State state {};
	const uint64_t     total = static_cast<uint64_t>(gridDim.x) * cfg.warps;
	const uint64_t     first = static_cast<uint64_t>(blockIdx.x) * cfg.warps + warp;
	const uint64_t     n     = first < cfg.n_items ? (cfg.n_items - first + total - 1u) / total : 0u;
	LaneMeta           now {}, next {};
	if constexpr (!UNIFORM) {
		now  = load_window(cfg, first, total, 0, lane);
		next = load_window(cfg, first, total, 1, lane);
	}
	if (lane < cfg.slots) { dev::mbar_init(bars + lane, 1); }
	dev::fence_mbar_init();
	__syncwarp();
	const uint64_t pol = dev::l2_evict_first_policy();
	for (uint32_t q = 0; q < cfg.slots && q < n; ++q) {
		if constexpr (UNIFORM) {
			issue_tile(cfg, base + q * cfg.slot_words, bars + q, first + q * total, lane, pol);
		} else {
			issue_vector(cfg, base + q * cfg.slot_words, bars + q, now, q, lane, pol);
		}
	}
	uint32_t slot = 0, phase = 0;
	for (uint64_t q = 0; q < n; ++q) {
		const uint32_t j = static_cast<uint32_t>(q) & 31u;
		if (!UNIFORM && j == 0 && q != 0) {
			now  = next;
			next = load_window(cfg, first, total, (q >> 5) + 1u, lane);
		}
		if (!dev::mbar_wait_bounded(bars + slot, phase, kWaitPolls)) {
			raise_err(cfg.err, kErrTimeout);
			// Give the copies still in flight a bounded chance to land before exit.
			for (uint32_t s = 0; s < cfg.slots; ++s) {
				dev::mbar_wait_bounded(bars + s, phase, 1u << 10);
				dev::mbar_wait_bounded(bars + s, phase ^ 1u, 1u << 10);
			}
			return;
		}
		ColumnVec cv;
		cv.s     = base + slot * cfg.slot_words;
		cv.dict  = base + cfg.dict_off;
		cv.extra = base + cfg.extra_off;
		if constexpr (UNIFORM) {
			cv.vi.base   = cfg.col.base;
			cv.vi.scheme = cfg.col.scheme;
			cv.vi.bw     = cfg.col.bw;
			cv.vi.aux    = 0;
			cv.v         = (first + q * total) * cfg.tile;
			const uint64_t end = min(cv.v + cfg.tile, cfg.n_vec);
			for (; cv.v < end; ++cv.v, cv.s += cfg.col.vec_words) { op.process(state, cv, lane, cfg); }
		} else {
			const uint32_t packed = __shfl_sync(0xffffffffu, now.packed, j);
			cv.vi.base   = static_cast<int32_t>(__shfl_sync(0xffffffffu, now.base, j));
			cv.vi.scheme = packed & 0xffu;
			cv.vi.bw     = (packed >> 8) & 0xffu;
			cv.vi.aux    = packed >> 16;
			cv.v         = first + q * total;
			if (cv.vi.scheme != kBadScheme) { op.process(state, cv, lane, cfg); }
		}
		__syncwarp();
		if (q + cfg.slots < n) {
			dev::fence_proxy_async_smem();
			if constexpr (UNIFORM) {
				issue_tile(cfg, base + slot * cfg.slot_words, bars + slot, first + (q + cfg.slots) * total, lane, pol);
			} else {
				const uint32_t ahead = j + cfg.slots; // below 64
				issue_vector(cfg, base + slot * cfg.slot_words, bars + slot, ahead < 32u ? now : next, ahead & 31u, lane, pol);
			}
		}
		if (++slot == cfg.slots) {
			slot = 0;
			phase ^= 1u;
		}
	}
	op.finish(state, lane, cfg);
}

// Lays out and launches: as many warps as the operator takes and shared
// memory holds at two slots or more, then slots up to the launch
// configuration's bytes in flight per warp (stages x tile bytes), or a third
// of them where every vector is also written out (half in original order):
// past that the reads in flight only disturb the writes (67 M values to
// memory: DELTA 59.0 us at 4 KB a warp, 61.7 at 6 KB; in original order 59.4
// at 6 KB, 59.8 at 4 and 61.0 at 8; FOR of mixed widths 68.5, 69.3 at 12; at 1 to
// 8 M values a warp has few vectors and the share makes no difference).  A
// column of fewer items than warps spreads over the SMs.  A uniform column's
// tiles are as long as a tile of the launch configuration, or shorter so that
// every warp gets four.
template <class Op, bool UNIFORM>
fls_status launch_column_as(const fls_column& col, const Op& op, uint32_t extra_words, cudaStream_t stream) {
	ColumnCfg  cfg {};
	DeviceInfo di;
	fls_status s = device_info(di);
	if (s != FLS_OK) { return s; }
	if ((s = make_devcol(col, cfg.col)) != FLS_OK) { return s; }
	uint32_t warps = 0, stages = 0, ctas = 0, tile_bytes = 0;
	fls_get_launch_config(&warps, &stages, &ctas, &tile_bytes);
	warps        = std::min(launch_warps(Op::kWarps), Op::kWarps);
	cfg.has_dict = col.meta && (col.scheme_mask & ((1u << FLS_SCHEME_RLE) | (1u << FLS_SCHEME_DICT))) ? 1u : 0u;
	cfg.n_values = col.n_values;
	cfg.n_vec    = (col.n_values + 1023u) / 1024u;
	const auto round4 = [](uint32_t w) { return (w + 3u) & ~3u; };
	const uint32_t fixed = kSlotSlackWords + (cfg.has_dict ? kDictWords : 0u) + round4(extra_words) + 2u * kMaxSlots;
	const uint32_t avail = static_cast<uint32_t>(di.max_smem) / 4u;
	cfg.tile             = 1;
	if (UNIFORM) { // two tiles of all warps fit
		const uint64_t all   = static_cast<uint64_t>(di.sms) * ctas * warps;
		const uint32_t words = std::min<uint32_t>(tile_bytes / 4u, (avail / warps - fixed) / 2u);
		cfg.tile             = std::max<uint32_t>(1u, std::min<uint32_t>(kMaxTile, words / std::max<uint32_t>(cfg.col.vec_words, 32u)));
		while (cfg.tile > 1 && cfg.n_vec / cfg.tile < 4u * all) { cfg.tile /= 2u; }
	}
	cfg.n_items           = (cfg.n_vec + cfg.tile - 1u) / cfg.tile;
	cfg.slot_words        = round4(cfg.tile * cfg.col.slot_words);
	const uint32_t flight = stages * tile_bytes / op.flight_share();
	const uint32_t want   = std::max<uint32_t>(1u, flight / std::max<uint32_t>(4u * cfg.slot_words, 256u));
	const auto     fits  = [&](uint32_t w, uint32_t slots) { return w * (slots * cfg.slot_words + fixed) <= avail; };
	while (warps > 1 && !fits(warps, 2)) { --warps; }
	if (!fits(warps, 1)) { return set_error(FLS_ERR_CAPACITY, "vectors too large for shared-memory staging"); }
	cfg.slots = std::min<uint32_t>(std::max<uint32_t>(want, 2u), kMaxSlots);
	while (cfg.slots > 1 && !fits(warps, cfg.slots)) { --cfg.slots; }
	uint64_t grid = std::min<uint64_t>((cfg.n_items + warps - 1u) / warps, static_cast<uint64_t>(di.sms) * ctas);
	if (grid < static_cast<uint64_t>(di.sms)) {
		grid  = std::min<uint64_t>(cfg.n_items, static_cast<uint64_t>(di.sms));
		warps = static_cast<uint32_t>((cfg.n_items + grid - 1u) / grid);
	}
	cfg.warps      = warps;
	cfg.dict_off   = cfg.slots * cfg.slot_words + kSlotSlackWords;
	cfg.extra_off  = cfg.dict_off + (cfg.has_dict ? kDictWords : 0u);
	cfg.bar_off    = cfg.extra_off + round4(extra_words);
	cfg.warp_words = cfg.bar_off + 2u * kMaxSlots;
	cfg.err        = device_error_word(stream);
	{
		static std::mutex mu;
		static uint64_t   configured = 0; // bit d: device d's shared-memory attribute raised
		int               dev        = 0;
		cudaGetDevice(&dev);
		std::lock_guard<std::mutex> lk(mu);
		if (dev >= 64 || !(configured & (1ull << dev))) {
			s = cuda_check(cudaFuncSetAttribute(column_kernel<Op, UNIFORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, di.max_smem),
			               "cudaFuncSetAttribute");
			if (s != FLS_OK) { return s; }
			if (dev < 64) { configured |= 1ull << dev; }
		}
	}
	column_kernel<Op, UNIFORM><<<static_cast<uint32_t>(grid), 32u * warps, 4ull * cfg.warp_words * warps, stream>>>(cfg, op);
	count_launch();
	return cuda_check(cudaGetLastError(), "column_kernel launch");
}

template <class Op>
fls_status launch_column(const fls_column& col, const Op& op, uint32_t extra_words, cudaStream_t stream) {
	if constexpr (Op::kTiles) {
		if (!col.meta) { return launch_column_as<Op, true>(col, op, extra_words, stream); }
	}
	return launch_column_as<Op, false>(col, op, extra_words, stream);
}

// -------------------------------------------------------------- operators

struct NoState {};

// Decode to HBM.  Values of a vector are written as 32 coalesced 128-byte rows
// with streaming stores; transposed columns can instead be reordered through
// shared memory into original order.
//
// The reordering buffer holds chunk c (32 consecutive values) at words 32 c ..
// 32 c + 31, its groups of four exchanged by c mod 8 and turned inside by c /
// 8, so that a lane's column of chunk positions falls on 32 different banks
// and four consecutive values still leave by one 16-byte read and one 16-byte
// store: 48 memory instructions per vector instead of 96 with padded rows
// (67 M DELTA values in original order: 59.4 -> 58.4 us, 50 M RLE 47.6 ->
// 46.3).
struct DecodeOp {
	static constexpr uint32_t kWarps = 16;
	static constexpr bool     kTiles = false; // bound by the writes: no faster in tiles
	uint32_t flight_share() const { return original ? 2u : 3u; }
	using State = NoState;
	uint32_t* out;
	uint32_t  original;
	uint32_t  wide; // out is 16-byte aligned
	__device__ void process(State&, const ColumnVec& cv, uint32_t lane, const ColumnCfg&) const {
		uint32_t vals[32];
		dev::decode_vals(cv.s, cv.vi, cv.dict, lane, vals);
		uint32_t* dst = out + cv.v * 1024u;
		if (original) {
			uint32_t*      tb = cv.extra;
			const uint32_t c = dev::chunk_of_lane(lane), turn = c >> 3, swap = (c & 7u) << 2;
#pragma unroll
			for (uint32_t r = 0; r < 32; ++r) {
				const uint32_t t = dev::step_of_row(r);
				tb[32u * c + ((t & 28u) ^ swap) + (((t & 3u) + turn) & 3u)] = vals[r];
			}
			__syncwarp();
			if (wide) {
#pragma unroll
				for (uint32_t m = 0; m < 8; ++m) { // values 128 m + 4 lane .. + 3: chunk 4 m + lane / 8, group lane mod 8
					const uint32_t k = 4u * m + (lane >> 3);
					const uint4    q = *reinterpret_cast<const uint4*>(tb + 32u * k + (((lane & 7u) ^ (k & 7u)) << 2));
					const uint32_t e[4] = {q.x, q.y, q.z, q.w};
					// turned by k / 8 = m / 2
					__stcs(reinterpret_cast<uint4*>(dst + 128u * m + 4u * lane),
					       make_uint4(e[(m >> 1) & 3u], e[((m >> 1) + 1u) & 3u], e[((m >> 1) + 2u) & 3u],
					                  e[((m >> 1) + 3u) & 3u]));
				}
			} else {
#pragma unroll
				for (uint32_t r = 0; r < 32; ++r) {
					dev::st_stream(dst + 32u * r + lane,
					               tb[32u * r + ((lane & 28u) ^ ((r & 7u) << 2)) + (((lane & 3u) + (r >> 3)) & 3u)]);
				}
			}
			__syncwarp();
		} else {
#pragma unroll
			for (uint32_t r = 0; r < 32; ++r) { dev::st_stream(dst + 32u * r + lane, vals[r]); }
		}
	}
	__device__ void finish(State&, uint32_t, const ColumnCfg&) const {}
};

struct AccState {
	unsigned long long acc;
};

// Decode fused with a uint64 sum; four independent partial sums per lane, one
// atomic per warp at the end.
struct DecodeSumOp {
	static constexpr uint32_t kWarps = 16;
	static constexpr bool     kTiles = true;
	uint32_t flight_share() const { return 1u; }
	using State = AccState;
	unsigned long long* sum;
	__device__ void process(State& S, const ColumnVec& cv, uint32_t lane, const ColumnCfg& cfg) const {
		uint32_t vals[32];
		// Values are summed as uint32 (base added per value: it may wrap).
		dev::decode_vals(cv.s, cv.vi, cv.dict, lane, vals);
		const uint32_t     m = cv.rows(cfg, lane);
		unsigned long long p[4] = {0, 0, 0, 0};
		if (m == 0xffffffffu) { // every vector but the column's last
#pragma unroll
			for (uint32_t r = 0; r < 32; ++r) { p[r & 3] += vals[r]; }
		} else {
#pragma unroll
			for (uint32_t r = 0; r < 32; ++r) { p[r & 3] += ((m >> r) & 1u) ? vals[r] : 0u; }
		}
		S.acc += (p[0] + p[1]) + (p[2] + p[3]);
	}
	__device__ void finish(State& S, uint32_t lane, const ColumnCfg&) const {
		const unsigned long long s = warp_sum_u64(S.acc);
		if (lane == 0 && s) { atomicAdd(sum, s); }
	}
};

// ------------------------------------------------------------------------
// Decode fused with a sum for columns whose vectors all share one scheme
// (DELTA, RLE or DICT; scheme_mask has one bit), as the encoder produces for
// sorted keys, runs and dictionaries.  The scheme is a template parameter, so
// the per-vector scheme switch and the value array of the general operator
// disappear: each decoded value goes straight into the lane's sum.  The bit
// width stays a warp-uniform switch per vector (vectors of one column differ
// in width).  Values whose 32-row lane sum cannot exceed 32 bits (every value
// below 2^27, known from the vector's base and width) are summed in 32 bits.
//
// The reference times delta decode + sum as delta_shared_memory.cu:24-61
// (unpack to shared memory, d_rsum_32, BlockLoad, BlockSum per 1024 values).

template <int BW>
__device__ __forceinline__ unsigned long long delta_lane_sum(const uint32_t* __restrict__ s, uint32_t lane,
                                                             uint32_t rows) {
	dev::LaneWords<BW> lw;
	dev::load_words<BW>(s + 32, lane, lw);
	uint32_t           x   = s[lane];
	unsigned long long acc = 0;
	if constexpr (BW <= 22) {
		if (rows == 0xffffffffu) {
			// Value s is base + p_s with p_s the running sum of the deltas.
			// For BW <= 22, p_31 < 2^27 and the sum of the 32 p_s < 2^32, so
			// the p_s sum in 32 bits and the base is added once -- exact
			// unless base + p_31 wraps (then the full path below runs).
			uint32_t p = 0, ps = 0;
#pragma unroll
			for (int st = 0; st < 32; ++st) {
				p += dev::extract<BW>(lw, static_cast<int>(dev::rsum_row(st)));
				ps += p;
			}
			if (static_cast<uint64_t>(x) + p < (1ull << 32)) {
				return 32ull * x + ps;
			}
		}
	}
	if (rows == 0xffffffffu) {
#pragma unroll
		for (int st = 0; st < 32; ++st) {
			x += dev::extract<BW>(lw, static_cast<int>(dev::rsum_row(st)));
			acc += x;
		}
	} else {
#pragma unroll
		for (int st = 0; st < 32; ++st) {
			const int r = static_cast<int>(dev::rsum_row(st));
			x += dev::extract<BW>(lw, r);
			acc += ((rows >> r) & 1u) ? x : 0u;
		}
	}
	return acc;
}

// The rows `rows` of a column's last, partial vector, any code width (one
// vector per column: a plain loop).
__device__ __noinline__ unsigned long long dict_lane_sum_rows(const uint32_t* __restrict__ s,
                                                             const uint32_t* __restrict__ dict, uint32_t lane,
                                                             uint32_t cbw, uint32_t rows) {
	unsigned long long acc = 0;
	const uint32_t     m   = cbw >= 32 ? 0xffffffffu : ((1u << cbw) - 1u);
	for (uint32_t r = 0; r < 32; ++r) {
		if (cbw == 0 || !((rows >> r) & 1u)) {
			acc += ((rows >> r) & 1u) ? dict[0] : 0u;
			continue;
		}
		const uint32_t bit = r * cbw, w = bit >> 5, sh = bit & 31u;
		const uint32_t lo = s[32u * w + lane], hi = sh + cbw > 32u ? s[32u * (w + 1u) + lane] : 0u;
		acc += dict[(__funnelshift_r(lo, hi, sh) & m) & 1023u];
	}
	return acc;
}

// True when every value of the vector (base + a bw-bit field) is below 2^27.
__device__ __forceinline__ bool small_values(const VecInfo& m) {
	const uint64_t top = static_cast<uint64_t>(static_cast<uint32_t>(m.base)) +
	                     (m.bw >= 32 ? 0xffffffffull : ((1ull << m.bw) - 1ull));
	return top < (1ull << 27);
}

// FULL: every row of the lane holds a value (all vectors but a column's
// last), so no row is tested.
template <bool Small, bool FULL>
__device__ __forceinline__ unsigned long long rle_lane_sum(const uint32_t* __restrict__ s,
                                                           const uint32_t* __restrict__ dict, uint32_t lane,
                                                           uint32_t rows) {
	uint32_t           idx  = reinterpret_cast<const uint16_t*>(s)[lane];
	const uint32_t     bits = s[16 + lane];
	uint32_t           s32  = 0;
	unsigned long long s64  = 0;
#pragma unroll
	for (int st = 0; st < 32; ++st) {
		const int r = static_cast<int>(dev::rsum_row(st));
		idx += (bits >> r) & 1u;
		const uint32_t v = (FULL || ((rows >> r) & 1u)) ? dict[idx & 1023u] : 0u;
		if constexpr (Small) {
			s32 += v;
		} else {
			s64 += v;
		}
	}
	return Small ? static_cast<unsigned long long>(s32) : s64;
}

// A whole vector (every row holds a value) at code width CBW.
template <int CBW, bool Small>
__device__ __forceinline__ unsigned long long dict_lane_sum(const uint32_t* __restrict__ s,
                                                            const uint32_t* __restrict__ dict, uint32_t lane) {
	dev::LaneWords<CBW> lw;
	dev::load_words<CBW>(s, lane, lw);
	uint32_t           s32 = 0;
	unsigned long long s64 = 0;
#pragma unroll
	for (int r = 0; r < 32; ++r) {
		const uint32_t v = dict[dev::extract<CBW>(lw, r) & 1023u];
		if constexpr (Small) {
			s32 += v;
		} else {
			s64 += v;
		}
	}
	return Small ? static_cast<unsigned long long>(s32) : s64;
}

template <uint32_t SCHEME>
struct SchemeSumOp {
	// 50 M values, kernel at 16, 24 and 32 warps (us): DELTA 20.2, 18.1, 18.4; RLE
	// 29.7, 27.3, 26.5; DICT 43.5, 39.9, 39.9.  Short columns, whole call at 16 and
	// 24: DICT 1 M 8.3, 8.3, 4 M (two vectors for some warps of 24) 10.4, 12.3, 8 M
	// 14.5, 14.3; RLE 4 M 8.3, 9.9, 8 M 10.4, 10.6; DELTA 4 M 8.3, 8.3.
	static constexpr uint32_t kWarps = 24;
	static constexpr bool     kTiles = SCHEME == FLS_SCHEME_DELTA; // the one that a uniform column may have
	uint32_t flight_share() const { return 1u; }
	using State = AccState;
	unsigned long long* sum;
	__device__ void process(State& S, const ColumnVec& sv, uint32_t lane, const ColumnCfg& cfg) const {
		const uint32_t rows = sv.rows(cfg, lane);
		if (sv.vi.scheme != SCHEME) { // the host saw one scheme; any other vector is flagged, not read
			if (lane == 0) { raise_err(cfg.err, kErrBadMeta); }
			return;
		}
		if constexpr (SCHEME == FLS_SCHEME_DELTA) {
			switch (sv.vi.bw) {
#define FLS_DELTA_SUM(B)                                                                                               \
	case B: S.acc += delta_lane_sum<B>(sv.s, lane, rows); break;
				FLS_BW_CASES_0_32(FLS_DELTA_SUM)
#undef FLS_DELTA_SUM
			default: break;
			}
		} else if constexpr (SCHEME == FLS_SCHEME_RLE) {
			uint32_t* dict = sv.dict;
			dev::unpack_dict(sv.s + 48, sv.vi.aux, sv.vi.bw, sv.vi.base, dict, lane);
			if (__all_sync(0xffffffffu, rows == 0xffffffffu)) {
				S.acc += small_values(sv.vi) ? rle_lane_sum<true, true>(sv.s, dict, lane, rows)
				                             : rle_lane_sum<false, true>(sv.s, dict, lane, rows);
			} else {
				S.acc += small_values(sv.vi) ? rle_lane_sum<true, false>(sv.s, dict, lane, rows)
				                             : rle_lane_sum<false, false>(sv.s, dict, lane, rows);
			}
			__syncwarp();
		} else {
			uint32_t*      dict = sv.dict;
			const uint32_t cbw  = dev::bits_of(sv.vi.aux - 1u);
			dev::unpack_dict(sv.s + 32u * cbw, sv.vi.aux, sv.vi.bw, sv.vi.base, dict, lane);
			const bool small = small_values(sv.vi);
			if (!__all_sync(0xffffffffu, rows == 0xffffffffu)) {
				S.acc += dict_lane_sum_rows(sv.s, dict, lane, cbw, rows);
			} else {
				switch (cbw) {
#define FLS_DICT_SUM(B)                                                                                                \
	case B: S.acc += small ? dict_lane_sum<B, true>(sv.s, dict, lane) : dict_lane_sum<B, false>(sv.s, dict, lane); break;
					FLS_BW_CASES_0_10(FLS_DICT_SUM)
#undef FLS_DICT_SUM
				default: break;
				}
			}
			__syncwarp();
		}
	}
	__device__ void finish(State& S, uint32_t lane, const ColumnCfg&) const {
		const unsigned long long s = warp_sum_u64(S.acc);
		if (lane == 0 && s) { atomicAdd(sum, s); }
	}
};

// The single scheme of a column, if it has a specialised sum, or FLS_N_SCHEMES.
uint32_t single_scheme(const fls_column& c) {
	const uint32_t m = c.meta ? c.scheme_mask : 1u << c.scheme;
	if (m == (1u << FLS_SCHEME_DELTA)) { return FLS_SCHEME_DELTA; }
	if (m == (1u << FLS_SCHEME_RLE)) { return FLS_SCHEME_RLE; }
	if (m == (1u << FLS_SCHEME_DICT)) { return FLS_SCHEME_DICT; }
	return FLS_N_SCHEMES;
}

} // namespace
} // namespace fls

using namespace fls;

extern "C" {

fls_status fls_decode_u32(const fls_column* col, uint32_t* d_out, uint32_t order, fls_stream_t stream) {
	if (!col || !d_out) { return set_error(FLS_ERR_INVALID_ARG, "fls_decode_u32: null pointer"); }
	if (order > FLS_ORDER_ORIGINAL) { return set_error(FLS_ERR_INVALID_ARG, "fls_decode_u32: bad order"); }
	const bool   orig = order == FLS_ORDER_ORIGINAL && col->layout == FLS_LAYOUT_TRANSPOSED;
	cudaStream_t st   = reinterpret_cast<cudaStream_t>(stream);
	if (tuning_jit() && !orig) {
		bool       used = false;
		fls_status s    = jit_decode(col, 1, d_out, nullptr, st, used);
		if (s != FLS_OK || used) { return s; }
	}
	DecodeOp op {};
	op.out      = d_out;
	op.original = orig ? 1u : 0u;
	op.wide     = (reinterpret_cast<uintptr_t>(d_out) & 15u) == 0 ? 1u : 0u;
	return launch_column(*col, op, orig ? 1024u : 0u, st);
}

fls_status fls_decode_sum_u32(const fls_column* col, uint64_t* d_sum, fls_stream_t stream) {
	if (!col || !d_sum) { return set_error(FLS_ERR_INVALID_ARG, "fls_decode_sum_u32: null pointer"); }
	DeviceInfo di;
	DevCol     checked;
	fls_status s = device_info(di);
	if (s == FLS_OK) { s = make_devcol(*col, checked); }
	if (s != FLS_OK) { return s; }
	cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
	if ((s = cuda_check(cudaMemsetAsync(d_sum, 0, sizeof(uint64_t), st), "cudaMemsetAsync")) != FLS_OK) { return s; }
	auto* sum = reinterpret_cast<unsigned long long*>(d_sum);
	if (tuning_jit()) {
		bool used = false;
		s         = jit_decode(col, 0, nullptr, d_sum, st, used);
		if (s != FLS_OK || used) { return s; }
		switch (single_scheme(*col)) {
		case FLS_SCHEME_DELTA: return launch_column(*col, SchemeSumOp<FLS_SCHEME_DELTA> {sum}, 0u, st);
		case FLS_SCHEME_RLE: return launch_column(*col, SchemeSumOp<FLS_SCHEME_RLE> {sum}, 0u, st);
		case FLS_SCHEME_DICT: return launch_column(*col, SchemeSumOp<FLS_SCHEME_DICT> {sum}, 0u, st);
		default: break;
		}
	}
	return launch_column(*col, DecodeSumOp {sum}, 0u, st);
}

} // extern "C"
