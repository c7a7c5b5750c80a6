// The B200 decode engine: one persistent kernel that walks a queue of (column, vector) work items and decodes
// each FastLanes vector with one warp.
//
//   stage 1  packed words of the vector -> shared memory with a bulk TMA copy (cp.async.bulk + mbarrier),
//            STAGES vectors ahead of the one being decoded (per-warp ring)
//   stage 2  bit-unpack + FOR add (+ per-lane running sum for DELTA) in registers, values in run order
//   stage 3  optional gather: RLE expansion from the run values staged next to the packed words, or a
//            dictionary lookup
//   stage 4  store: transposed order straight from registers, original order through a swizzled staging
//            buffer and row-wise 16-byte stores (every decoded byte crosses HBM exactly once)
//
// Reference semantics (cwida/FastLanes): unpack/unffor = primitives/fls_generated/fallback/scalar_aav_uf1/
// *_unpack_src.cpp:17277 / *_unffor_src.cpp:22971 (u32 dispatch), rsum = *_rsum_src.cpp:100-410,
// untranspose_i = *_untranspose_src.cpp:4110, RLE expansion = src/cor/lyt/vec.cpp:318-332 (Vec::flatten_to),
// dictionary gather = include/fls/encoder/assert_eq.hpp:257-400.
#include "fls_device.cuh"
#include "fls_plan.h"

namespace flsgpu {

struct Plan {
	const uint8_t* src;        // packed words of the stream
	const uint8_t* lane_bases; // ENC_DELTA
	const uint8_t* gsrc;       // RLE run values
	const uint8_t* dict;
	uint8_t*       out;
	uint64_t       for_base;
	uint32_t       bytes;  // packed bytes = bw * 128
	uint32_t       gbytes; // run-value bytes
	uint32_t       bw;
	uint32_t       entry_c;
	uint32_t       n_runs;
	uint32_t       ghead; // offset of the run values inside the staged (16-byte aligned) copy
	uint8_t        ws, e, enc, post, order;
	uint8_t        cmp; // OUT_BITMAP_* of filter plans, else OUT_VALUES
	bool           ok;
	bool           lb_exact; // lane bases outside a page: copy exactly 128 bytes, never a window around them
};

__device__ __forceinline__ uint64_t ld_le(const uint8_t* p, uint32_t n) {
	const uintptr_t a = reinterpret_cast<uintptr_t>(p);
	if ((a & (n - 1)) == 0) {
		switch (n) {
		case 1: return *p;
		case 2: return *reinterpret_cast<const uint16_t*>(p);
		case 4: return *reinterpret_cast<const uint32_t*>(p);
		default: return *reinterpret_cast<const uint64_t*>(p);
		}
	}
	if (n == 8 && (a & 3u) == 0) {
		const uint32_t* w = reinterpret_cast<const uint32_t*>(p);
		return static_cast<uint64_t>(w[0]) | (static_cast<uint64_t>(w[1]) << 32);
	}
	uint64_t x = 0;
	for (uint32_t i = 0; i < n; ++i) { x |= static_cast<uint64_t>(p[i]) << (8 * i); }
	return x;
}

// Entry points sit at page offset 8 + 4*arr_c; a page may be placed at any byte address (it is placed so that
// its packed buffer is 16-byte aligned), so they are read alignment-agnostically.
// Little-endian load of 4 / 8 bytes at any byte address inside a shared-memory staging area that has at least 8
// readable bytes after it: aligned words joined by funnel shifts instead of byte loads.
__device__ __forceinline__ uint32_t sld4(const uint8_t* p) {
	const uintptr_t a = reinterpret_cast<uintptr_t>(p);
	const uint32_t* w = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3));
	return (a & 3u) ? __funnelshift_r(w[0], w[1], (a & 3u) * 8u) : w[0];
}
__device__ __forceinline__ uint64_t sld8(const uint8_t* p) {
	const uintptr_t a = reinterpret_cast<uintptr_t>(p);
	const uint32_t* w = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3));
	const uint32_t  s = (a & 3u) * 8u;
	const uint32_t  lo = s ? __funnelshift_r(w[0], w[1], s) : w[0];
	const uint32_t  hi = s ? __funnelshift_r(w[1], w[2], s) : w[1];
	return (static_cast<uint64_t>(hi) << 32) | lo;
}
template <int E>
__device__ __forceinline__ uint64_t sld(const uint8_t* p) {
	if constexpr (E == 8) {
		return sld8(p);
	} else if constexpr (E == 4) {
		return sld4(p);
	} else {
		return ld_le(p, E);
	}
}

__device__ __forceinline__ uint32_t ep_of(const ColDesc& c, uint32_t v, uint32_t i) {
	if (v == 0) { return 0u; }
	return static_cast<uint32_t>(ld_le(reinterpret_cast<const uint8_t*>(c.ep) + 4ull * ((v - 1) * c.arr_c + i), 4));
}

__device__ __forceinline__ Plan make_plan(const ColDesc& c, uint32_t v) {
	Plan p;
	p.ws      = c.ws;
	p.e       = c.e;
	p.enc     = c.enc;
	p.post    = c.post;
	p.order   = c.order;
	p.entry_c = c.entry_c;
	p.dict    = c.dict;
	p.cmp     = c.out_mode;
	p.out     = c.out + static_cast<uint64_t>(v) * (c.out_mode != OUT_VALUES ? 128u : kVec * c.e);
	p.ok      = v < c.n_vec;
	p.lb_exact   = c.layout == LAYOUT_ARRAYS;
	p.for_base   = 0;
	p.lane_bases = nullptr;
	p.gsrc       = nullptr;
	p.gbytes     = 0;
	p.n_runs     = 0;
	p.ghead      = 0;
	const uint32_t wb = c.ws / 8;
	if (c.layout == LAYOUT_ARRAYS) {
		p.bw               = c.bw_arr ? c.bw_arr[v] : c.bw_const;
		const uint64_t off = c.byte_off ? c.byte_off[v] : static_cast<uint64_t>(v) * c.bw_const * 128u;
		p.src              = c.packed + off;
		if (c.base_arr) { p.for_base = ld_le(c.base_arr + static_cast<uint64_t>(v) * wb, wb); }
		if (c.lane_base_arr) { p.lane_bases = c.lane_base_arr + static_cast<uint64_t>(v) * 128u; }
	} else {
		if (c.enc == ENC_RAW) {
			p.bw = c.ws;
		} else {
			const uint32_t obw = ep_of(c, v, c.ib_bw);
			const uint32_t obs = ep_of(c, v, c.ib_base);
			if (obw >= c.buf_size[c.ib_bw] || obs + wb > c.buf_size[c.ib_base]) { p.ok = false; }
			p.bw       = p.ok ? c.buf[c.ib_bw][obw] : 0;
			p.for_base = p.ok ? ld_le(c.buf[c.ib_base] + obs, wb) : 0;
		}
		const uint32_t opk = ep_of(c, v, c.ib_packed);
		p.src              = c.buf[c.ib_packed] + opk;
		if (static_cast<uint64_t>(opk) + p.bw * 128ull > c.buf_size[c.ib_packed]) { p.ok = false; }
		if (c.enc == ENC_DELTA) {
			const uint32_t olb = ep_of(c, v, c.ib_lane_bases);
			if (olb + 128ull > c.buf_size[c.ib_lane_bases]) { p.ok = false; }
			p.lane_bases = c.buf[c.ib_lane_bases] + olb;
		}
		if (post_is_patch(c.post)) {
			// exceptions (gsrc, gbytes) and their positions / bitmap / chain head (dict, entry_c bytes)
			const uint32_t oe = ep_of(c, v, c.ib_exc), os = ep_of(c, v, c.ib_side);
			const uint64_t ee = (v + 1 < c.n_vec) ? ep_of(c, v + 1, c.ib_exc) : c.buf_size[c.ib_exc];
			const uint64_t es = (v + 1 < c.n_vec) ? ep_of(c, v + 1, c.ib_side) : c.buf_size[c.ib_side];
			if (ee < oe || ee > c.buf_size[c.ib_exc] || es < os || es > c.buf_size[c.ib_side]) { p.ok = false; }
			p.gsrc    = c.buf[c.ib_exc] + oe;
			p.gbytes  = p.ok ? static_cast<uint32_t>(ee - oe) : 0u;
			p.dict    = c.buf[c.ib_side] + os;
			p.entry_c = p.ok ? static_cast<uint32_t>(es - os) : 0u;
		}
		if (c.post == POST_RLE || c.post == POST_RLE_DICT) {
			const uint32_t ov  = ep_of(c, v, c.ib_vals);
			const uint64_t end = (v + 1 < c.n_vec) ? ep_of(c, v + 1, c.ib_vals) : c.buf_size[c.ib_vals];
			if (end < ov || end > c.buf_size[c.ib_vals]) { p.ok = false; }
			p.gsrc   = c.buf[c.ib_vals] + ov;
			p.gbytes = p.ok ? static_cast<uint32_t>(end - ov) : 0;
		}
	}
	if (p.bw > p.ws) { p.ok = false; }
	p.bytes = p.ok ? p.bw * 128u : 0u;
	if (p.post == POST_RLE || p.post == POST_RLE_DICT) {
		const uint32_t ve = p.post == POST_RLE ? p.e : 4u;
		if (p.gbytes > kVec * ve) { p.ok = false; }
		p.n_runs = p.ok ? p.gbytes / ve : 0u;
		p.ghead  = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p.gsrc) & 15u);
	}
	return p;
}

#ifndef FLS_HOST_EMULATION
// Copy one vector's inputs into its stage and arm the stage's mbarrier.  Called by all 32 lanes with the same
// plan.  16-byte aligned packed words go through the TMA engine; anything else is copied by the warp.
// The run values of an RLE vector are fetched as the enclosing 16-byte aligned window (pages are placed
// with at least 16 bytes of slack on both sides), so they always take the TMA path.
// The 128 lane bases of a DELTA vector travel with its packed words: the 16-byte aligned window around them
// (at most 144 bytes, inside the page) lands in a per-slot area of kLaneWindow bytes.
constexpr uint32_t kLaneWindow = 256;

template <uint32_t GSTAGE>
__device__ __forceinline__ void issue(const Plan& p, uint8_t* stage, uint8_t* gstage, uint8_t* lbstage, uint64_t* bar,
                                      uint32_t lane, bool stall = false) {
	uint32_t       tx     = 0;
	const uint32_t lbhead = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p.lane_bases) & 15u);
	// 16-byte aligned lane bases: exactly their 128 bytes by TMA; inside a page: the aligned 144-byte window by
	// TMA; otherwise (a misaligned caller array) the warp copies the 128 bytes
	const bool lbtma  = p.ok && p.lane_bases != nullptr && (lbhead == 0 || !p.lb_exact);
	const bool lbwarp = p.ok && p.lane_bases != nullptr && !lbtma;
	const uint32_t lbbytes = lbhead ? 144u : 128u;
	if (lbwarp) {
		for (uint32_t i = lane; i < 128; i += 32) { lbstage[lbhead + i] = p.lane_bases[i]; }
	}
	const bool tma_pk  = p.ok && p.bytes > 0 && (reinterpret_cast<uintptr_t>(p.src) & 15u) == 0;
	uint32_t   gwindow = 0;
	if (GSTAGE > 0 && p.ok && p.gbytes > 0) { gwindow = (p.ghead + p.gbytes + 15u) & ~15u; }
	if (GSTAGE > 0 && gwindow > GSTAGE) { gwindow = 0; }
	if (p.ok && p.bytes > 0 && !tma_pk) {
		if ((reinterpret_cast<uintptr_t>(p.src) & 3u) == 0) {
			const uint32_t* s = reinterpret_cast<const uint32_t*>(p.src);
			uint32_t*       d = reinterpret_cast<uint32_t*>(stage);
			for (uint32_t i = lane; i < p.bytes / 4; i += 32) { d[i] = s[i]; }
		} else {
			for (uint32_t i = lane; i < p.bytes; i += 32) { stage[i] = p.src[i]; }
		}
	}
	__syncwarp();
	if (lane == 0) {
		if (tma_pk) { tx += p.bytes; }
		tx += gwindow;
		if (lbtma) { tx += lbbytes; }
		mbar_arrive_expect_tx(bar, tx);
		// stall (failure injection): the byte count is armed, no copy is issued, so the wait runs out
		if (tma_pk && !stall) { bulk_g2s(stage, p.src, p.bytes, bar); }
		if (gwindow && !stall) { bulk_g2s(gstage, p.gsrc - p.ghead, gwindow, bar); }
		if (lbtma && !stall) { bulk_g2s(lbstage, p.lane_bases - lbhead, lbbytes, bar); }
		// without a staging area the run values are gathered from global memory: start them towards L2 now
		if (GSTAGE == 0 && p.ok && p.gbytes > 0) { bulk_prefetch_l2(p.gsrc - p.ghead, (p.ghead + p.gbytes + 15u) & ~15u); }
	}
}

#endif // FLS_HOST_EMULATION

// ---------------------------------------------------------------------------------------------------------
// Per-width decode of the staged stream into registers (run order).
// ---------------------------------------------------------------------------------------------------------
template <int WS>
struct StreamT {
	using T = uint32_t;
};
template <>
struct StreamT<64> {
	using T = uint64_t;
};

// Patch one vector's unpacked values (after the FOR add, before rsum) through `scratch` (1024 values in
// transposed order; the stage the packed words came from, free once they are in registers).  Exceptions are
// at p.gsrc (p.gbytes bytes), their positions / bitmap / chain head at p.dict (p.entry_c bytes).
template <int WS>
__device__ __forceinline__ void apply_patch(const Plan& p, typename StreamT<WS>::T (&v)[32], uint8_t* scratch,
                                            uint32_t t, int* status) {
	using T = typename StreamT<WS>::T;
	if constexpr (WS == 32 || WS == 64) {
		T*             s   = reinterpret_cast<T*>(scratch);
		const uint32_t n_e = p.gbytes / sizeof(T);
		__syncwarp();
#pragma unroll
		for (int q = 0; q < 32; ++q) { s[run_tpos<WS>(t, 0, q)] = v[q]; }
		__syncwarp();
		bool bad = false;
		if (p.post == POST_PATCH_S) {
			const uint32_t c = p.entry_c >= 2 ? static_cast<uint32_t>(ld_le(p.dict, 2)) : 0u;
			bad              = p.entry_c < 2 || 2u + 2u * c > p.entry_c || c > n_e;
			for (uint32_t i = t; !bad && i < c; i += 32) {
				const uint32_t pos = static_cast<uint32_t>(ld_le(p.dict + 2 + 2 * i, 2));
				if (pos < kVec) { s[pos] = static_cast<T>(ld_le(p.gsrc + static_cast<uint64_t>(i) * sizeof(T), sizeof(T))); }
			}
		} else if (p.post == POST_PATCH_B) {
			// 16 bitmap words, one per lane 0..15; exceptions follow the set bits in ascending order
			bad              = p.entry_c < 128;
			const uint64_t w = (!bad && t < 16) ? ld_le(p.dict + 8 * t, 8) : 0ull;
			const uint32_t c   = static_cast<uint32_t>(__popcll(w));
			uint32_t       inc = c; // inclusive warp scan of the per-word counts
#pragma unroll
			for (uint32_t d = 1; d < 32; d <<= 1) {
				const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, d);
				if (t >= d) { inc += y; }
			}
			const uint32_t i0  = inc - c;
			const uint32_t tot = __shfl_sync(0xFFFFFFFFu, inc, 31);
			bad |= tot > n_e;
			uint64_t rest = bad ? 0ull : w;
			for (uint32_t k = 0; rest != 0; ++k) {
				const uint32_t r = __ffsll(static_cast<long long>(rest)) - 1;
				rest &= rest - 1;
				s[64 * t + r] = static_cast<T>(ld_le(p.gsrc + static_cast<uint64_t>(i0 + k) * sizeof(T), sizeof(T)));
			}
		} else if (t == 0) {
			// LL: the packed value at an exception is the distance to the next one minus one
			const uint32_t c     = p.entry_c >= 4 ? static_cast<uint32_t>(ld_le(p.dict, 2)) : 0u;
			uint64_t       cur   = p.entry_c >= 4 ? ld_le(p.dict + 2, 2) : 0u;
			const T        base  = static_cast<T>(p.for_base);
			bad                  = p.entry_c < 4 || c > n_e;
			for (uint32_t i = 0; !bad && i < c; ++i) {
				if (cur >= kVec) {
					bad = true;
					break;
				}
				const T off = static_cast<T>(s[cur] - base + T(1));
				s[cur]      = static_cast<T>(ld_le(p.gsrc + static_cast<uint64_t>(i) * sizeof(T), sizeof(T)));
				cur += static_cast<uint64_t>(off);
			}
		}
		if (__any_sync(0xFFFFFFFFu, bad) && t == 0) { atomicOr(status, STATUS_BAD_INDEX); }
		__syncwarp();
#pragma unroll
		for (int q = 0; q < 32; ++q) { v[q] = s[run_tpos<WS>(t, 0, q)]; }
		__syncwarp();
	}
}

// The 32 values of half-lane h of lane l (values 2m + h, m = 0..31, in run order) of a 64-bit stream of bit
// width BW <= 16, as 32-bit words.  The thread's values sit at bits h*BW + 2m*BW of the lane: the lane's
// 32-bit words are first shifted by h*BW (one funnel shift each, every word read once), after which every
// value's word and shift are compile-time constants.
template <uint32_t BW>
__device__ __forceinline__ void extract_w64_small_bw(const uint32_t* __restrict__ S, uint32_t l, uint32_t h,
                                                     uint32_t (&x)[32]) {
	constexpr uint32_t mask = BW == 0 ? 0u : (1u << BW) - 1u;
	if constexpr (BW == 0) {
#pragma unroll
		for (int i = 0; i < 32; ++i) { x[i] = 0; }
	} else {
		const uint32_t hb  = h * BW;
		// lane word k (k = 0, 1, ...: the low and high halves of the lane's 64-bit words in order)
		auto           raw = [&](uint32_t k) { return S[2 * (l + 16 * (k >> 1)) + (k & 1u)]; };
#pragma unroll
		for (uint32_t m = 0; m < 32; ++m) {
			const uint32_t b  = 2 * m * BW;
			const uint32_t k  = b >> 5;
			const uint32_t sh = b & 31u;
			const uint32_t s0 = __funnelshift_r(raw(k), raw(k + 1), hb);
			if (sh + BW <= 32) {
				x[run32_pos(m)] = (s0 >> sh) & mask;
			} else {
				const uint32_t s1 = __funnelshift_r(raw(k + 1), raw(k + 2), hb);
				x[run32_pos(m)]   = __funnelshift_r(s0, s1, sh) & mask;
			}
		}
	}
}

// Bit widths up to 26 (values below 2^26): compile-time layouts up to 16 bits, computed offsets above.
__device__ __forceinline__ void extract_w64_small(const uint32_t* __restrict__ S, uint32_t l, uint32_t h,
                                                  uint32_t bw, uint32_t (&x)[32]) {
	switch (bw) {
#define FLS_W64_SMALL(B)                                                                                               \
	case B: extract_w64_small_bw<B>(S, l, h, x); return;
		FLS_W64_SMALL(0) FLS_W64_SMALL(1) FLS_W64_SMALL(2) FLS_W64_SMALL(3) FLS_W64_SMALL(4) FLS_W64_SMALL(5)
		FLS_W64_SMALL(6) FLS_W64_SMALL(7) FLS_W64_SMALL(8) FLS_W64_SMALL(9) FLS_W64_SMALL(10) FLS_W64_SMALL(11)
		FLS_W64_SMALL(12) FLS_W64_SMALL(13) FLS_W64_SMALL(14) FLS_W64_SMALL(15) FLS_W64_SMALL(16)
#undef FLS_W64_SMALL
	default: break;
	}
	const uint32_t mlo = (1u << bw) - 1u;
#pragma unroll
	for (uint32_t m = 0; m < 32; ++m) {
		const uint32_t b  = (2 * m + h) * bw;
		const uint32_t h2 = b >> 5;
		const uint32_t lo = S[2 * (l + 16 * (h2 >> 1)) + (h2 & 1u)];
		const uint32_t h3 = h2 + 1;
		const uint32_t hi = S[2 * (l + 16 * (h3 >> 1)) + (h3 & 1u)];
		x[run32_pos(m)]   = __funnelshift_r(lo, hi, b & 31u) & mlo;
	}
}

// DELTA vectors of a 64-bit stream whose deltas and FOR base are below 2^26 (the common case of sorted 64-bit
// keys): every delta + FOR base is below 2^27, so a half-lane's running sum of 32 of them fits 32 bits.
__device__ __forceinline__ bool small_deltas(const Plan& p) {
	return p.enc == ENC_DELTA && p.bw <= 26 && p.for_base < (1ull << 26);
}

// Their running sums in run order (x, non-decreasing) and what to add to each of them (returned): value i of
// thread t is the returned 64-bit word + x[i].
__device__ __forceinline__ uint64_t small_delta_sums(const Plan& p, const uint32_t* S, uint32_t t, uint32_t (&x)[32]) {
	const uint32_t l   = t & 15u;
	const uint32_t h   = t >> 4;
	const uint32_t b32 = static_cast<uint32_t>(p.for_base);
	extract_w64_small(S, l, h, p.bw, x);
	uint32_t acc = 0;
#pragma unroll
	for (int i = 0; i < 32; ++i) {
		acc += x[i] + b32;
		x[i] = acc;
	}
	const uint32_t lower = __shfl_sync(0xFFFFFFFFu, acc, l); // total of the lane's first half
	return ld_le(p.lane_bases + 8 * l, 8) + (h ? lower : 0u);
}

// PATCH: the kernel may meet patched items (plain-stream kernels and the catch-all one; gather kernels never do)
template <int WS, bool PATCH = true>
__device__ __forceinline__ void decode_stream(const Plan& p, const uint32_t* S, uint32_t t,
                                              typename StreamT<WS>::T (&v)[32], uint8_t* scratch = nullptr,
                                              int* status = nullptr) {
	using T = typename StreamT<WS>::T;
	if constexpr (WS == 64) {
		if (small_deltas(p) && !(PATCH && scratch && post_is_patch(p.post))) {
			// the 64-bit add happens once per value
			uint32_t x[32];
			const T  add = small_delta_sums(p, S, t, x);
#pragma unroll
			for (int i = 0; i < 32; ++i) { v[i] = add + x[i]; }
			return;
		}
		extract_w64(S, t, p.bw, v);
	} else if constexpr (WS == 32) {
		extract_w32(S, t, p.bw, v);
	} else if constexpr (WS == 16) {
		extract_w16(S, t, p.bw, v);
	} else {
		extract_w8(S, t, p.bw, v);
	}
	constexpr T wmask = WS == 64 ? ~T(0) : static_cast<T>((1ull << WS) - 1ull);
	// 16- and 8-bit DELTA streams without patches add the FOR base inside the running sum: sums of at most 16
	// terms below 2^16 stay exact in 32 bits, so the wrap to the stream width comes once per value, off the
	// chain of dependent adds
	const bool fold = WS <= 16 && p.enc == ENC_DELTA && !(PATCH && scratch && post_is_patch(p.post));
	if (p.enc != ENC_RAW && !fold) {
		const T base = static_cast<T>(p.for_base);
#pragma unroll
		for (int i = 0; i < 32; ++i) { v[i] = (v[i] + base) & wmask; }
	}
	if constexpr (PATCH) {
		if (scratch && post_is_patch(p.post)) { apply_patch<WS>(p, v, scratch, t, status); }
	}
	if (p.enc == ENC_DELTA) {
		// rsum: running sum along each lane in original order, seeded by the lane's base.
		if constexpr (WS == 32) {
			T acc = static_cast<T>(ld_le(p.lane_bases + 4 * t, 4));
#pragma unroll
			for (int i = 0; i < 32; ++i) {
				acc += v[i];
				v[i] = acc;
			}
		} else if constexpr (WS == 64) {
			const uint32_t l   = t & 15u;
			const uint32_t h   = t >> 4;
			T              acc = 0;
#pragma unroll
			for (int i = 0; i < 32; ++i) {
				acc += v[i];
				v[i] = acc;
			}
			const T lower = __shfl_sync(0xFFFFFFFFu, acc, l); // total of the lane's first half
			T       add   = static_cast<T>(ld_le(p.lane_bases + 8 * l, 8));
			if (h) { add += lower; }
#pragma unroll
			for (int i = 0; i < 32; ++i) { v[i] += add; }
		} else if constexpr (WS == 16) {
			const T base = fold ? static_cast<T>(p.for_base) & wmask : T(0);
#pragma unroll
			for (int q = 0; q < 2; ++q) {
				T acc = static_cast<T>(ld_le(p.lane_bases + 2 * (2 * t + q), 2));
#pragma unroll
				for (int i = 0; i < 16; ++i) {
					acc += v[16 * q + i] + base;
					v[16 * q + i] = acc;
				}
			}
#pragma unroll
			for (int i = 0; i < 32; ++i) { v[i] &= wmask; }
		} else {
			const T base = fold ? static_cast<T>(p.for_base) & wmask : T(0);
#pragma unroll
			for (int q = 0; q < 4; ++q) {
				T acc = p.lane_bases[4 * t + q];
#pragma unroll
				for (int i = 0; i < 8; ++i) {
					acc += v[8 * q + i] + base;
					v[8 * q + i] = acc;
				}
			}
#pragma unroll
			for (int i = 0; i < 32; ++i) { v[i] &= wmask; }
		}
	}
}

// ---------------------------------------------------------------------------------------------------------
// Store of 32 values per thread (run order) for stream width WS and element size E.
// ---------------------------------------------------------------------------------------------------------
template <int E>
struct OutT {
	using T = uint32_t;
};
template <>
struct OutT<8> {
	using T = uint64_t;
};
// exact element type of an E-byte output
template <int E>
struct ElemT;
template <>
struct ElemT<1> {
	using T = uint8_t;
};
template <>
struct ElemT<2> {
	using T = uint16_t;
};
template <>
struct ElemT<4> {
	using T = uint32_t;
};
template <>
struct ElemT<8> {
	using T = uint64_t;
};

// 16 decoded bytes to global memory.  The output's address comes out of a plan in shared memory, so that to the compiler
// an ordinary store through it might change the staging buffer: every read of the buffer then waited for the store
// before it.  Nothing in a launch reads an output.
__device__ __forceinline__ void store_out16(uint8_t* out, const uint4& x) {
#ifdef FLS_HOST_EMULATION
	*reinterpret_cast<uint4*>(out) = x;
#else
	asm volatile("st.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(__cvta_generic_to_global(out)), "r"(x.x), "r"(x.y), "r"(x.z),
	             "r"(x.w));
#endif
}

// two neighbouring E-byte values, the first one on a multiple of 2 * E bytes
template <int E>
__device__ __forceinline__ void store_pair(typename ElemT<E>::T* out, typename OutT<E>::T a, typename OutT<E>::T b) {
	if constexpr (E == 8) {
		*reinterpret_cast<uint4*>(out) = make_uint4(static_cast<uint32_t>(a), static_cast<uint32_t>(a >> 32), static_cast<uint32_t>(b),
		                                            static_cast<uint32_t>(b >> 32));
	} else if constexpr (E == 4) {
		*reinterpret_cast<uint2*>(out) = make_uint2(a, b);
	} else {
		*reinterpret_cast<uint32_t*>(out) = (a & 0xFFFFu) | (b << 16);
	}
}

template <int WS, int E>
__device__ __forceinline__ void store_vector(const typename OutT<E>::T (&o)[32], uint8_t* out, uint8_t* ost,
                                             bool original, uint32_t t) {
	constexpr uint32_t RL = run_len<WS>();
	constexpr uint32_t RC = run_count<WS>();
	if (original) {
		__syncwarp(); // the staging buffer is the stage the packed words were just read from
#pragma unroll
		for (uint32_t r = 0; r < RC; ++r) {
			const uint32_t b0 = run_start<WS>(t, r) * E;
			if constexpr (RL * E >= 16) {
				constexpr uint32_t PER = 16 / E; // values per 16-byte chunk
#pragma unroll
				for (uint32_t c = 0; c < RL * E / 16; ++c) {
					uint32_t w[4];
#pragma unroll
					for (uint32_t k = 0; k < 4; ++k) {
						if constexpr (E == 8) {
							const uint64_t x = o[r * RL + c * PER + k / 2];
							w[k]             = (k & 1) ? static_cast<uint32_t>(x >> 32) : static_cast<uint32_t>(x);
						} else if constexpr (E == 4) {
							w[k] = static_cast<uint32_t>(o[r * RL + c * PER + k]);
						} else if constexpr (E == 2) {
							w[k] = (o[r * RL + c * PER + 2 * k] & 0xFFFFu) | (o[r * RL + c * PER + 2 * k + 1] << 16);
						} else {
							const uint32_t i0 = r * RL + c * PER + 4 * k;
							w[k] = (o[i0] & 0xFFu) | ((o[i0 + 1] & 0xFFu) << 8) | ((o[i0 + 2] & 0xFFu) << 16) |
							       (o[i0 + 3] << 24);
						}
					}
					*reinterpret_cast<uint4*>(ost + stage_off(b0 + 16 * c)) = make_uint4(w[0], w[1], w[2], w[3]);
				}
			} else {
				// WS = 8, E = 1: an 8-byte run
				const uint32_t i0 = r * RL;
				const uint32_t lo = (o[i0] & 0xFFu) | ((o[i0 + 1] & 0xFFu) << 8) | ((o[i0 + 2] & 0xFFu) << 16) |
				                    (o[i0 + 3] << 24);
				const uint32_t hi = (o[i0 + 4] & 0xFFu) | ((o[i0 + 5] & 0xFFu) << 8) |
				                    ((o[i0 + 6] & 0xFFu) << 16) | (o[i0 + 7] << 24);
				*reinterpret_cast<uint2*>(ost + stage_off(b0)) = make_uint2(lo, hi);
			}
		}
		__syncwarp();
		if ((reinterpret_cast<uintptr_t>(out) & 15u) == 0) {
#pragma unroll
			for (uint32_t j = 0; j < 2u * E; ++j) {
				const uint32_t c = 32 * j + t;
				store_out16(out + 16 * c, *reinterpret_cast<const uint4*>(ost + stage_off(16 * c)));
			}
		} else {
			for (uint32_t b = t; b < 1024u * E; b += 32) { out[b] = ost[stage_off(b)]; }
		}
		__syncwarp();
	} else {
		using ET = typename ElemT<E>::T;
#pragma unroll
		for (uint32_t p = 0; p < RL; ++p) {
			// the thread's RC lanes are adjacent in the transposed order
			const uint32_t k0 = run_tpos<WS>(t, 0, p);
#pragma unroll
			for (uint32_t r = 0; r < RC; ++r) { reinterpret_cast<ET*>(out)[k0 + r] = static_cast<ET>(o[r * RL + p]); }
		}
	}
}

// ---------------------------------------------------------------------------------------------------------
// Predicate of 32 values per thread (run order) into the vector's 1024-bit bitmap at out (predicate pushdown:
// the decoded values never leave the registers).  Bit i of the bitmap is value i of the vector in the plan's
// order (original or transposed).
// ---------------------------------------------------------------------------------------------------------
// The predicate for E-byte values as one range test: value OP constant holds exactly when x - lo <= span in
// unsigned arithmetic, or exactly when it does not (flip).  EQ is the range [constant, constant]; LT and LE start
// at the type's lowest value; NE, GE and GT are the complements of EQ, LT and LE.  One subtraction and one
// compare a value where testing below / equal / above took two compares and a class lookup, the complement
// applied once to the finished bitmap word.
template <int E>
struct PredE {
	using T = typename OutT<E>::T;
	static constexpr uint32_t kSh = E < 4 ? 32 - 8 * E : 0; // narrow values are compared in the top bytes of a word
	T        lo, span;
	uint32_t flip; // all ones: the complement

	__device__ __forceinline__ PredE(const Pred& pr, bool sgn) {
		const uint32_t op = pr.op < 6 ? pr.op : 0;
		const T  s = sgn ? T(1) << (8 * sizeof(T) - 1) : T(0); // the lowest value
		const T  c = static_cast<T>(static_cast<T>(pr.value) << kSh);
		flip       = (op == PRED_NE || op == PRED_GT || op == PRED_GE) ? ~0u : 0u;
		if constexpr (E < 8) {
			// a constant outside a narrow column's range: every value is below (or above) it
			const int64_t v     = static_cast<int64_t>(pr.value);
			const bool    above = sgn ? v < -(1ll << (8 * E - 1)) : false;
			const bool    below = sgn ? v > (1ll << (8 * E - 1)) - 1 : pr.value > (1ull << (8 * E)) - 1;
			if (above || below) {
				const bool all = op == PRED_NE || (below ? op == PRED_LT || op == PRED_LE : op == PRED_GT || op == PRED_GE);
				lo   = 0;
				span = ~T(0);
				flip = all ? 0u : ~0u;
				return;
			}
		}
		if (op == PRED_EQ || op == PRED_NE) {
			lo   = c;
			span = 0;
		} else if (op == PRED_LE || op == PRED_GT) {
			lo   = s;
			span = c - s;
		} else {
			// value < constant: nothing is below the lowest value
			lo   = s;
			span = c - s - 1;
			if (c == s) { flip = ~flip; } // span is all ones: the complement of everything
		}
	}
	// x is in the range (the predicate up to flip)
	__device__ __forceinline__ bool in(T x) const { return static_cast<T>(static_cast<T>(x << kSh) - lo) <= span; }
	__device__ __forceinline__ bool operator()(T x) const { return in(x) != (flip != 0); }
};

// 16 bits to the even bits of a word
__device__ __forceinline__ uint32_t spread16(uint32_t x) {
	x = (x | (x << 8)) & 0x00FF00FFu;
	x = (x | (x << 4)) & 0x0F0F0F0Fu;
	x = (x | (x << 2)) & 0x33333333u;
	return (x | (x << 1)) & 0x55555555u;
}

template <int WS, int E>
__device__ __forceinline__ void filter_vector(const typename OutT<E>::T (&o)[32], const Plan& p, uint8_t* ost,
                                              uint32_t t, const Pred& pr) {
	constexpr uint32_t RL = run_len<WS>();
	constexpr uint32_t RC = run_count<WS>();
	const PredE<E>     holds(pr, p.cmp == OUT_BITMAP_S);
	uint32_t*          out  = reinterpret_cast<uint32_t*>(p.out);
	uint32_t           mine = 0; // bitmap word t
	if (p.order) {
		if constexpr (RL == 32) {
			// the thread's run is one aligned bitmap word
#pragma unroll
			for (uint32_t j = 0; j < 32; ++j) { mine |= static_cast<uint32_t>(holds.in(o[j])) << j; }
			out[run_start<WS>(t, 0) / 32] = mine ^ holds.flip;
			return;
		} else {
			// runs of RL (16 or 8) values start at multiples of 8: every bitmap byte belongs to one run
			__syncwarp(); // the stage was just read into registers
#pragma unroll
			for (uint32_t r = 0; r < RC; ++r) {
				uint32_t m = 0;
#pragma unroll
				for (uint32_t j = 0; j < RL; ++j) { m |= static_cast<uint32_t>(holds.in(o[r * RL + j])) << j; }
				m ^= holds.flip;
				const uint32_t s = run_start<WS>(t, r) / 8;
#pragma unroll
				for (uint32_t b = 0; b < RL / 8; ++b) { ost[s + b] = static_cast<uint8_t>(m >> (8 * b)); }
			}
			__syncwarp();
			mine = reinterpret_cast<const uint32_t*>(ost)[t];
		}
	} else if constexpr (WS == 32 || WS == 64) {
		// run position j of every thread lands on bit t of bitmap word run32_val(j)
#pragma unroll
		for (uint32_t j = 0; j < 32; ++j) {
			const uint32_t b = __ballot_sync(0xFFFFFFFFu, holds.in(o[j]));
			if (run32_val(j) == t) { mine = b; }
		}
		mine ^= holds.flip;
	} else if constexpr (WS == 16) {
		// run position j of the thread's two lanes: bits 2t and 2t + 1 of the 64 at 64 * run16_val(j)
#pragma unroll
		for (uint32_t j = 0; j < 16; ++j) {
			const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, holds(o[j]));
			const uint32_t b1 = __ballot_sync(0xFFFFFFFFu, holds(o[16 + j]));
			const uint32_t g  = 2 * run16_val(j);
			if (t == g) { mine = spread16(b0 & 0xFFFFu) | (spread16(b1 & 0xFFFFu) << 1); }
			if (t == g + 1) { mine = spread16(b0 >> 16) | (spread16(b1 >> 16) << 1); }
		}
	} else {
		uint32_t* bm = reinterpret_cast<uint32_t*>(ost);
		__syncwarp();
		bm[t] = 0;
		__syncwarp();
#pragma unroll
		for (uint32_t r = 0; r < RC; ++r) {
#pragma unroll
			for (uint32_t j = 0; j < RL; ++j) {
				if (holds(o[r * RL + j])) {
					const uint32_t k = run_tpos<WS>(t, r, j);
					atomicOr(bm + k / 32, 1u << (k & 31u));
				}
			}
		}
		__syncwarp();
		mine = bm[t];
	}
	out[t] = mine;
	__syncwarp();
}

// The predicate over a DELTA vector of small deltas, original order: the values are add + x[i] (small_delta_sums),
// so the range test moves to the 32-bit sums: with D = add - lo, the sums x with D + x <= span (mod 2^64) are one
// interval [a, a + s] of 32-bit numbers, found once a thread; a value then costs a 32-bit subtraction and compare.
// Two intervals (the sums wrap past lo inside a range that also holds D) take the 64-bit test value by value.
// The filter of 16,001 vectors of 64-bit timestamps (7-bit deltas): 38.2 us with two 64-bit compares a value, 26.4 us
// so (cold caches); what is left is the extraction and too few warps for its latency.
__device__ __forceinline__ void filter_small_deltas(const Plan& p, const uint32_t* S, uint32_t t, const Pred& pr) {
	const PredE<8> holds(pr, p.cmp == OUT_BITMAP_S);
	uint32_t       x[32];
	const uint64_t add = small_delta_sums(p, S, t, x);
	const uint64_t D    = add - holds.lo;
	const uint64_t top  = x[31]; // the largest sum
	const bool     wrap = D + top < D;
	uint32_t       mine = 0;
	if (!wrap || holds.span < D) {
		const uint64_t first = wrap ? 0ull - D : 0ull; // at most top
		const uint64_t room  = top - first;
		const uint64_t len   = wrap ? holds.span : holds.span - D;
		const uint32_t a = static_cast<uint32_t>(first), n = static_cast<uint32_t>(len < room ? len : room);
		// a sum below `first` is at least 2^32 - first past it, above room >= n
#pragma unroll
		for (uint32_t j = 0; j < 32; ++j) { mine |= (x[j] - a <= n ? 1u : 0u) << j; }
		if (!wrap && D > holds.span) { mine = 0; }
	} else {
#pragma unroll
		for (uint32_t j = 0; j < 32; ++j) { mine |= (holds.in(add + x[j]) ? 1u : 0u) << j; }
	}
	reinterpret_cast<uint32_t*>(p.out)[run_start<64>(t, 0) / 32] = mine ^ holds.flip;
}

// ---------------------------------------------------------------------------------------------------------
// Full decode of one staged vector.
// ---------------------------------------------------------------------------------------------------------
// GSMEM: RLE run values / run codes staged in shared memory at gstage + ghead (else read from p.gsrc).
// KIND: bit 0 = the kernel handles RLE / DICT gathers, bit 1 = patched FFOR / DELTA items; a kernel that meets
// an item outside its kind flags a layout error (plans never route one there).  Bit 2 (KIND_FILTER): the
// vector's predicate bitmap is written instead of its values.
enum : int { KIND_PLAIN = 0, KIND_GATHER = 1, KIND_PATCH = 2, KIND_ALL = 3, KIND_FILTER = 4 };

// The value behind an index of a gathered stream: run value (RLE), dictionary entry (DICT), or the entry of a run's
// code (RLE_DICT).  FAST (the usual case): the arrays lie at multiples of their element sizes and every index of the
// vector is known to be in range, so that a run value or dictionary entry costs its address and its load; a run's code
// is still checked.  The arrays are read-only for the launch, so the loads need not wait for the stores before them.
// Otherwise every index is checked.  GSMEM: the run values / run codes are staged in shared memory with at least 8
// readable bytes behind them.
template <int E, int POST, bool FAST, bool GSMEM>
struct Gathered {
	using OT = typename OutT<E>::T;
	using ET = typename ElemT<E>::T;
	const uint8_t *runs, *dict;
	uint32_t       n_runs, entry_c;
	bool           bad = false;

	__device__ __forceinline__ Gathered(const Plan& p, const uint8_t* gstage)
	    : runs(GSMEM ? gstage + p.ghead : p.gsrc), dict(p.dict), n_runs(p.n_runs), entry_c(p.entry_c) {}
	__device__ __forceinline__ OT operator()(uint32_t i) {
		const uint8_t* table = POST == POST_RLE ? runs : dict;
		if constexpr (FAST && POST != POST_RLE_DICT) {
			return static_cast<OT>(__ldg(reinterpret_cast<const ET*>(table) + i));
		} else if constexpr (FAST) {
			i             = __ldg(reinterpret_cast<const uint32_t*>(runs) + i);
			const bool in = i < entry_c;
			bad |= !in;
			return in ? static_cast<OT>(__ldg(reinterpret_cast<const ET*>(table) + i)) : OT(0);
		} else {
			if constexpr (POST == POST_RLE_DICT) {
				const bool in = i < n_runs;
				bad |= !in;
				i = !in ? 0u : GSMEM ? sld4(runs + 4ull * i) : static_cast<uint32_t>(ld_le(runs + 4ull * i, 4));
			}
			const bool     in = i < (POST == POST_RLE ? n_runs : entry_c);
			const uint8_t* a  = table + static_cast<uint64_t>(i) * E;
			bad |= !in;
			return !in ? OT(0) : GSMEM && POST == POST_RLE ? static_cast<OT>(sld<E>(a)) : static_cast<OT>(ld_le(a, E));
		}
	}
};

// Indices of a vector (32 a thread, run order) to values or bitmap.  Original order: the indices go through the
// staging buffer, 2 or 4 bytes each, and are looked up where the values leave: 32 lanes then read 32 to 256
// neighbouring positions, whose run indices are neighbours too (one or two sectors a load where lanes 64 positions
// apart touched 32), the buffer holds indices instead of values, and no thread keeps 32 values, so that more warps
// fit.  32,768 vectors of RLE int32: 51.2 us with the lookups in run order, 41.0 us so; 16,000 of DICT int32 47.9, 28.7 us.
template <int WS, int E, int POST, bool FAST, bool GSMEM, int KIND>
__device__ __forceinline__ bool gather_post(const Plan& p, const typename StreamT<WS>::T (&v)[32], const uint8_t* gstage,
                                            uint8_t* ost, uint32_t t, const Pred& pr) {
	using OT = typename OutT<E>::T;
	using ET = typename ElemT<E>::T;
	constexpr uint32_t              IW = WS / 8; // bytes of a staged index
	Gathered<E, POST, FAST, GSMEM> get(p, gstage);
	const bool filter = (KIND & KIND_FILTER) != 0 && p.cmp != OUT_VALUES;
	if constexpr ((KIND & KIND_FILTER) != 0) {
		// a bitmap of transposed order takes the values as they come; so does one of run values in original order, where a
		// thread's neighbouring values come from the same runs (24,000 vectors of 4 bytes: 37 us, 59 through the staging
		// buffer; of 8 bytes 46 and 63).  For dictionary entries the buffer is the faster way: 55 against 96.
		if (filter && (!p.order || POST == POST_RLE)) {
			OT o[32];
#pragma unroll
			for (int i = 0; i < 32; ++i) { o[i] = get(static_cast<uint32_t>(v[i])); }
			filter_vector<WS, E>(o, p, ost, t, pr);
			return get.bad;
		}
	}
	if (!p.order) {
		// a thread's lanes are neighbours: their values go out together, looked up some steps ahead (24,000 vectors of RLE
		// int64: 53 us, 72 with one lane's stores after the other's)
		constexpr uint32_t RC = run_count<WS>(), RL = run_len<WS>(), STEP = 16 / RC;
		const bool         paired = (reinterpret_cast<uintptr_t>(p.out) & (2 * E - 1)) == 0;
#pragma unroll
		for (uint32_t q0 = 0; q0 < RL; q0 += STEP) {
			OT o[STEP][RC];
#pragma unroll
			for (uint32_t q = 0; q < STEP; ++q) {
#pragma unroll
				for (uint32_t r = 0; r < RC; ++r) { o[q][r] = get(static_cast<uint32_t>(v[r * RL + q0 + q])); }
			}
#pragma unroll
			for (uint32_t q = 0; q < STEP; ++q) {
				ET* at = reinterpret_cast<ET*>(p.out) + run_tpos<WS>(t, 0, q0 + q);
				if (RC == 2 && paired) {
					store_pair<E>(at, o[q][0], o[q][RC - 1]);
				} else {
#pragma unroll
					for (uint32_t r = 0; r < RC; ++r) { at[r] = static_cast<ET>(o[q][r]); }
				}
			}
		}
		return get.bad;
	}
	__syncwarp(); // the staging buffer is the stage the packed words were just read from
#pragma unroll
	for (uint32_t r = 0; r < run_count<WS>(); ++r) {
#pragma unroll
		for (uint32_t c = 0; c < run_len<WS>() * IW / 16; ++c) {
			uint32_t w[4];
#pragma unroll
			for (uint32_t k = 0; k < 4; ++k) {
				if constexpr (WS == 16) {
					const uint32_t i = r * 16 + c * 8 + 2 * k;
					w[k]             = v[i] | (v[i + 1] << 16);
				} else {
					w[k] = static_cast<uint32_t>(v[c * 4 + k]);
				}
			}
			*reinterpret_cast<uint4*>(ost + stage_off(run_start<WS>(t, r) * IW + 16 * c)) = make_uint4(w[0], w[1], w[2], w[3]);
		}
	}
	__syncwarp();
	auto index = [&](uint32_t pos) {
		const uint8_t* a = ost + stage_off(pos * IW);
		return WS == 16 ? static_cast<uint32_t>(*reinterpret_cast<const uint16_t*>(a)) : *reinterpret_cast<const uint32_t*>(a);
	};
	if constexpr ((KIND & KIND_FILTER) != 0) {
		if (filter) {
			const PredE<E> holds(pr, p.cmp == OUT_BITMAP_S);
			uint32_t       mine = 0;
#pragma unroll 8
			for (uint32_t w = 0; w < 32; ++w) {
				const uint32_t b = __ballot_sync(0xFFFFFFFFu, holds.in(get(index(32 * w + t))));
				if (w == t) { mine = b; }
			}
			reinterpret_cast<uint32_t*>(p.out)[t] = mine ^ holds.flip;
			__syncwarp();
			return get.bad;
		}
	}
	if ((reinterpret_cast<uintptr_t>(p.out) & 15u) == 0) {
		constexpr uint32_t PER = 16 / E; // values a 16-byte store
		constexpr uint32_t kUnroll = !FAST ? 1 : E == 8 ? 4 : 2 * E; // (8-byte values: more code in line costs small batches)
#pragma unroll kUnroll
		for (uint32_t j = 0; j < 2u * E; ++j) { // (a trip count known without t)
			const uint32_t c = 32 * j + t;
			// the PER indices lie in one 16-byte piece (two for 2-byte values of 4-byte indices)
			uint32_t       idx[PER];
			const uint8_t* a = ost + stage_off(c * PER * IW);
			if constexpr (PER * IW == 4) {
				const uint32_t x = *reinterpret_cast<const uint32_t*>(a);
				idx[0] = x & 0xFFFFu, idx[1] = x >> 16;
			} else if constexpr (PER * IW == 8 && IW == 2) {
				const uint2 x = *reinterpret_cast<const uint2*>(a);
				idx[0] = x.x & 0xFFFFu, idx[1] = x.x >> 16, idx[2] = x.y & 0xFFFFu, idx[3] = x.y >> 16;
			} else if constexpr (PER * IW == 8) {
				const uint2 x = *reinterpret_cast<const uint2*>(a);
				idx[0] = x.x, idx[1] = x.y;
			} else if constexpr (PER * IW == 16 && IW == 4) {
				const uint4 x = *reinterpret_cast<const uint4*>(a);
				idx[0] = x.x, idx[1] = x.y, idx[2] = x.z, idx[3] = x.w;
			} else {
#pragma unroll
				for (uint32_t i = 0; i < PER; ++i) { idx[i] = index(c * PER + i); }
			}
			OT o[PER];
#pragma unroll
			for (uint32_t i = 0; i < PER; ++i) { o[i] = get(idx[i]); }
			uint32_t w[4];
#pragma unroll
			for (uint32_t k = 0; k < 4; ++k) {
				if constexpr (E == 8) {
					w[k] = static_cast<uint32_t>(o[k / 2] >> (32 * (k & 1)));
				} else if constexpr (E == 4) {
					w[k] = static_cast<uint32_t>(o[k]);
				} else {
					w[k] = (static_cast<uint32_t>(o[2 * k]) & 0xFFFFu) | (static_cast<uint32_t>(o[2 * k + 1]) << 16);
				}
			}
			store_out16(p.out + 16 * c, make_uint4(w[0], w[1], w[2], w[3]));
		}
	} else {
		for (uint32_t i = t; i < kVec; i += 32) { reinterpret_cast<ET*>(p.out)[i] = static_cast<ET>(get(index(i))); }
	}
	__syncwarp();
	return get.bad;
}

template <int WS, int E, bool GSMEM, int KIND>
__device__ __forceinline__ void gather_vector(const Plan& p, const typename StreamT<WS>::T (&v)[32], const uint8_t* gstage,
                                              uint8_t* ost, uint32_t t, int* status, const Pred& pr) {
	// the largest index decides once for the vector whether its indices need checking
	uint32_t top = 0;
#pragma unroll
	for (int i = 0; i < 32; ++i) { top = top < static_cast<uint32_t>(v[i]) ? static_cast<uint32_t>(v[i]) : top; }
	const bool rle    = WS == 16;
	bool       direct = top < (rle ? p.n_runs : p.entry_c);
	direct            = !__any_sync(0xFFFFFFFFu, !direct);
	const uintptr_t dict = reinterpret_cast<uintptr_t>(p.dict), runs = reinterpret_cast<uintptr_t>(p.gsrc);
	bool            bad;
	if constexpr (WS == 16) {
		if (p.post == POST_RLE) {
			bad = !GSMEM && direct && (runs & (E - 1)) == 0
			          ? gather_post<WS, E, POST_RLE, true, false, KIND>(p, v, gstage, ost, t, pr)
			          : gather_post<WS, E, POST_RLE, false, GSMEM, KIND>(p, v, gstage, ost, t, pr);
		} else {
			bad = !GSMEM && direct && (runs & 3u) == 0 && (dict & (E - 1)) == 0
			          ? gather_post<WS, E, POST_RLE_DICT, true, false, KIND>(p, v, gstage, ost, t, pr)
			          : gather_post<WS, E, POST_RLE_DICT, false, GSMEM, KIND>(p, v, gstage, ost, t, pr);
		}
	} else {
		bad = direct && (dict & (E - 1)) == 0 ? gather_post<WS, E, POST_DICT, true, false, KIND>(p, v, gstage, ost, t, pr)
		                                      : gather_post<WS, E, POST_DICT, false, false, KIND>(p, v, gstage, ost, t, pr);
	}
	if (__any_sync(0xFFFFFFFFu, bad) && t == 0) { atomicOr(status, STATUS_BAD_INDEX); }
}

template <int WS, int E, bool GSMEM = true, int KIND = KIND_ALL>
__device__ __forceinline__ void decode_vector(const Plan& p, const uint8_t* stage, const uint8_t* gstage, uint8_t* ost,
                                              uint32_t t, int* status, const Pred& pr = Pred {}) {
	using ST = typename StreamT<WS>::T;
	using OT = typename OutT<E>::T;
	constexpr bool GATHER = (KIND & KIND_GATHER) != 0;
	constexpr bool PATCH  = (KIND & KIND_PATCH) != 0;
	if constexpr ((KIND & KIND_FILTER) != 0 && WS == 64) {
		if (p.order && p.post == POST_NONE && p.cmp != OUT_VALUES && small_deltas(p)) {
			filter_small_deltas(p, reinterpret_cast<const uint32_t*>(stage), t, pr);
			return;
		}
	}
	ST v[32];
	decode_stream<WS, PATCH>(p, reinterpret_cast<const uint32_t*>(stage), t, v, ost, status);
	if (!PATCH && post_is_patch(p.post) && t == 0) { atomicOr(status, STATUS_BAD_LAYOUT); }
	if constexpr (GATHER && (WS == 16 || WS == 32)) {
		if (post_is_gather(p.post)) {
			gather_vector<WS, E, GSMEM, KIND>(p, v, gstage, ost, t, status, pr);
			return;
		}
	}
	// streams of other widths are never gathered from, and a kernel for gathers alone has no room to stage values
	if (post_is_gather(p.post) || (KIND & KIND_ALL) == KIND_GATHER) {
		if (t == 0) { atomicOr(status, STATUS_BAD_LAYOUT); }
		return;
	}
	OT o[32];
#pragma unroll
	for (int i = 0; i < 32; ++i) { o[i] = static_cast<OT>(v[i]); }
	if constexpr ((KIND & KIND_FILTER) != 0) {
		bool values = false;
		if constexpr ((KIND & KIND_PATCH) != 0) {
			// an intermediate stream of a filter plan (a DICT page's patched codes, a patched item)
			values = p.cmp == OUT_VALUES;
			if (values) { store_vector<WS, E>(o, p.out, ost, p.order != 0, t); }
		}
		if (!values) { filter_vector<WS, E>(o, p, ost, t, pr); }
	} else {
		store_vector<WS, E>(o, p.out, ost, p.order != 0, t);
	}
}

// Compact plan kept in shared memory between the lane-parallel metadata fetch and the use of the plan.
struct __align__(16) PlanS {
	const uint8_t* src;
	uint8_t*       out;
	uint64_t       for_base;
	const uint8_t* lane_bases;
	const uint8_t* gsrc;
	const uint8_t* dict;
	uint32_t       gbytes;
	uint32_t       entry_c;
	uint16_t       bytes;
	uint8_t        bw, ws, e, enc, post, flags; // flags: bit0 original order, bit1 ok, bit2 valid, bit3 lb_exact,
	                                            // bits 4-5 cmp
};
static_assert(sizeof(PlanS) == 64, "PlanS layout");

__device__ __forceinline__ PlanS pack_plan(const Plan& p, bool valid) {
	PlanS s;
	s.src        = p.src;
	s.out        = p.out;
	s.for_base   = p.for_base;
	s.lane_bases = p.lane_bases;
	s.gsrc       = p.gsrc;
	s.dict       = p.dict;
	s.gbytes     = p.gbytes;
	s.entry_c    = p.entry_c;
	s.bytes      = static_cast<uint16_t>(p.bytes);
	s.bw         = static_cast<uint8_t>(p.bw > 255 ? 255 : p.bw);
	s.ws         = p.ws;
	s.e          = p.e;
	s.enc        = p.enc;
	s.post       = p.post;
	s.flags      = static_cast<uint8_t>((p.order ? 1 : 0) | (p.ok ? 2 : 0) | (valid ? 4 : 0) | (p.lb_exact ? 8 : 0) |
	                                    ((p.cmp & 3u) << 4));
	return s;
}

__device__ __forceinline__ Plan unpack_plan(const PlanS& s) {
	Plan p;
	p.src        = s.src;
	p.out        = s.out;
	p.for_base   = s.for_base;
	p.lane_bases = s.lane_bases;
	p.gsrc       = s.gsrc;
	p.dict       = s.dict;
	p.gbytes     = s.gbytes;
	p.entry_c    = s.entry_c;
	p.bytes      = s.bytes;
	p.bw         = s.bw;
	p.ws         = s.ws;
	p.e          = s.e;
	p.enc        = s.enc;
	p.post       = s.post;
	p.order      = s.flags & 1u;
	p.ok         = (s.flags & 2u) != 0;
	p.lb_exact   = (s.flags & 8u) != 0;
	p.cmp        = (s.flags >> 4) & 3u;
	const uint32_t ve = p.post == POST_RLE ? p.e : 4u;
	p.n_runs     = (p.post == POST_RLE || p.post == POST_RLE_DICT) ? p.gbytes / ve : 0u;
	p.ghead      = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p.gsrc) & 15u);
	return p;
}

#ifndef FLS_HOST_EMULATION
__device__ __forceinline__ uint32_t item_col(uint32_t it, uint32_t shift) { return it >> shift; }
__device__ __forceinline__ uint32_t item_vec(uint32_t it, uint32_t shift) { return it & ((1u << shift) - 1u); }

__device__ __forceinline__ Plan plan_of(const DecodeArgs& a, uint64_t item) {
	if (a.queue == nullptr) { return make_plan(a.col0, static_cast<uint32_t>(item)); }
	const uint32_t it = a.queue[item];
	const ColDesc& c  = a.cols ? a.cols[item_col(it, a.col_shift)] : a.col0;
	return make_plan(c, item_vec(it, a.col_shift));
}

// Kernel family: MAXWS bounds the staged stream (MAXWS * 128 bytes), GSTAGE the run-value window, EMAX the
// output element size.  The original-order staging reuses the stage once its packed words are in registers,
// so a slot is max(stream, output) bytes plus the run-value window.  Plans of the warp's next 2*PB items
// live in shared memory (64 bytes each).
template <int MAXWS, uint32_t GSTAGE, int EMAX, int WARPS, int STAGES, int KIND = KIND_ALL>
struct Geometry {
	static constexpr uint32_t kPB      = 16;
	static constexpr uint32_t kStage   = MAXWS * 128u;
	// what a vector is staged in on its way out: its values, or (gathers) its indices, at most 4 bytes each; a filter of
	// plain streams keeps its values in registers
	static constexpr uint32_t kOut     = (KIND & KIND_ALL) == KIND_GATHER ? 4096u : KIND == (KIND_PLAIN | KIND_FILTER) ? 1024u : EMAX * 1024u;
	static constexpr uint32_t kMain    = kStage > kOut ? kStage : kOut;
	static constexpr uint32_t kSlot    = kMain + kLaneWindow + GSTAGE;
	static constexpr uint32_t kPlans   = 2 * kPB * sizeof(PlanS);
	static constexpr uint32_t kPerWarp = 64u + kPlans + STAGES * kSlot;
	static constexpr uint32_t kSlack   = 256u; // extraction reads one row past the last stage
	static constexpr uint32_t kSmem    = WARPS * kPerWarp + kSlack;
	static constexpr int      kThreads = WARPS * 32;
	static_assert(STAGES < kPB, "plans must run ahead of the copies");
	static_assert(kSmem <= 232448u, "at most 227 KB of shared memory per CTA");
};

template <int MAXWS, uint32_t GSTAGE, int EMAX, int KIND>
__device__ __forceinline__ void decode_dispatch(const Plan& p, uint8_t* st, const uint8_t* gs, uint32_t lane,
                                                int* status, const Pred& pr) {
	if (p.ws == 64) {
		if constexpr (MAXWS >= 64) { decode_vector<64, 8, (GSTAGE > 0), KIND>(p, st, gs, st, lane, status, pr); }
	} else if (p.ws == 32) {
		if constexpr (MAXWS >= 32) {
			if (p.e == 8) {
				if constexpr (EMAX >= 8) { decode_vector<32, 8, (GSTAGE > 0), KIND>(p, st, gs, st, lane, status, pr); }
			} else {
				decode_vector<32, 4, (GSTAGE > 0), KIND>(p, st, gs, st, lane, status, pr);
			}
		}
	} else if (p.ws == 16) {
		if (p.e == 8) {
			if constexpr (EMAX >= 8) { decode_vector<16, 8, (GSTAGE > 0), KIND>(p, st, gs, st, lane, status, pr); }
		} else if (p.e == 4) {
			if constexpr (EMAX >= 4) { decode_vector<16, 4, (GSTAGE > 0), KIND>(p, st, gs, st, lane, status, pr); }
		} else {
			decode_vector<16, 2, (GSTAGE > 0), KIND>(p, st, gs, st, lane, status, pr);
		}
	} else {
		decode_vector<8, 1, (GSTAGE > 0), KIND>(p, st, gs, st, lane, status, pr);
	}
}

template <int MAXWS, uint32_t GSTAGE, int EMAX, int WARPS, int STAGES, int KIND>
__global__ void __launch_bounds__(WARPS * 32, 1) k_decode(const DecodeArgs a) {
	using G = Geometry<MAXWS, GSTAGE, EMAX, WARPS, STAGES, KIND>;
	constexpr uint32_t PB = G::kPB;
	extern __shared__ __align__(128) uint8_t smem[];
	const uint32_t lane   = threadIdx.x & 31u;
	const uint32_t warp   = threadIdx.x >> 5;
	uint8_t*       wbase  = smem + warp * G::kPerWarp;
	uint64_t*      bars   = reinterpret_cast<uint64_t*>(wbase);
	PlanS*         plans  = reinterpret_cast<PlanS*>(wbase + 64);
	uint8_t*       stages = wbase + 64 + G::kPlans;

	// fewer items than warps: they go to the CTAs in turn, so that a small batch spreads over the SMs (100 vectors on
	// 100 SMs instead of 7)
	const uint64_t n  = a.n_items;
	const uint64_t nw = static_cast<uint64_t>(gridDim.x) * WARPS;
	const uint64_t gw = n < nw ? static_cast<uint64_t>(warp) * gridDim.x + blockIdx.x : static_cast<uint64_t>(blockIdx.x) * WARPS + warp;
	if (gw >= n) { return; } // (warps never wait for one another)

	if (lane == 0) {
		for (int s = 0; s < STAGES; ++s) { mbar_init(&bars[s], 1); }
		fence_mbar_init();
	}

	auto stage_ptr  = [&](uint32_t s) { return stages + s * G::kSlot; };
	auto lb_ptr     = [&](uint32_t s) { return stages + s * G::kSlot + G::kMain; };
	auto gstage_ptr = [&](uint32_t s) { return stages + s * G::kSlot + G::kMain + kLaneWindow; };
	// Lane-parallel metadata fetch: lane j resolves the plan of the warp's item blk*PB + j (count of them).
	static_assert(PB == 16, "the first fill takes both halves of the ring");
	auto fill = [&](uint32_t blk, uint32_t count) {
		if (lane < count) {
			const uint64_t k    = static_cast<uint64_t>(blk) * PB + lane;
			const uint64_t item = gw + k * nw;
			Plan           p {};
			const bool     valid = item < n;
			if (valid) { p = plan_of(a, item); }
			plans[k % (2 * PB)] = pack_plan(p, valid);
		}
	};
	auto issue_k = [&](uint64_t k, uint32_t s) {
		const PlanS& ps = plans[k % (2 * PB)];
		if (ps.flags & 4u) {
			const bool stall = a.test_stall != 0 && gw + k * nw == a.test_stall - 1;
			issue<GSTAGE>(unpack_plan(ps), stage_ptr(s), gstage_ptr(s), lb_ptr(s), &bars[s], lane, stall);
		}
	};
	const uint32_t limit = a.spin_limit ? a.spin_limit : kMbarSpinLimit;

	fill(0, 32); // both halves of the ring at once
	__syncwarp();
	for (uint32_t s = 0; s < STAGES; ++s) { issue_k(s, s); }

	uint32_t k       = 0;
	bool     aborted = false;
	for (uint64_t item = gw; item < n; item += nw, ++k) {
		if (k % PB == 0 && k > 0) {
			fill(k / PB + 1, PB);
			__syncwarp();
		}
		const uint32_t s      = k % STAGES;
		const uint32_t parity = (k / STAGES) & 1u;
		Plan           p      = unpack_plan(plans[k % (2 * PB)]);
		if (!mbar_wait(&bars[s], parity, limit)) {
			if (lane == 0) { atomicOr(a.status, STATUS_TIMEOUT); }
			aborted = true;
			break;
		}
		if (!p.ok) {
			if (lane == 0) { atomicOr(a.status, p.bw > p.ws ? STATUS_BAD_BW : STATUS_BAD_LAYOUT); }
		} else {
			// the lane bases were staged with the packed words
			if (p.lane_bases) { p.lane_bases = lb_ptr(s) + (reinterpret_cast<uintptr_t>(p.lane_bases) & 15u); }
			decode_dispatch<MAXWS, GSTAGE, EMAX, KIND>(p, stage_ptr(s), gstage_ptr(s), lane, a.status, a.pred);
		}
		__syncwarp();
		issue_k(k + STAGES, s);
	}
	if (aborted) {
		// Drain: every later stage this warp armed must land before the block's shared memory goes away (full
		// bound: these copies were issued)
		for (uint32_t j = k + 1; j < k + STAGES; ++j) {
			const uint64_t item = gw + static_cast<uint64_t>(j) * nw;
			if (item >= n) { break; }
			(void)mbar_wait(&bars[j % STAGES], (j / STAGES) & 1u);
		}
	}
}
#endif // FLS_HOST_EMULATION

} // namespace flsgpu
