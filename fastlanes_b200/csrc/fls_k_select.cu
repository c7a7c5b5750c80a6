// Expression selection on the B200 (include/fls_select.h): the exact-size wizard, the per-vector statistics of
// the learned selector, and the MLP kernels (forward, gradient, Adam, graph-replayed training).
//
// Per-vector work runs warp per vector with every thread holding 32 contiguous values in registers: thread t
// holds original positions R(t) = (t % 16) * 64 + 32 * (t / 16) .. + 31.  In the unified transposed layout
// that run is exactly
//   * W = 32: the whole lane t;
//   * W = 64: half of lane t % 16, the other half in thread t ^ 16;
//   * W = 16 (the RLE run index): two whole lanes, [0,16) and [16,32) of the run.
// and the rsum / unrsum chains visit a lane in ascending original order, so FFOR, DELTA and RLE sizes come out
// of one read of the values.
#include "fls_device.cuh"
#include "fls_runtime.h"
#include "fls_b200.h"
#include "fls_cd_queue.cuh"
#include "fls_select.h"
#include "fls_smem_limit.h"
#include "fls_strings.cuh"
#include "fls_strplan.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <memory>
#include <random>
#include <vector>

namespace flsgpu {
namespace sel {

constexpr int      K        = FLS_SEL_K;
constexpr int      NF       = FLS_SEL_FEATURES;
constexpr int      H        = FLS_SEL_HIDDEN;
constexpr uint32_t kMaxVecPerChunk = 64;
constexpr int      kWarps   = 8;

struct Col {
	const uint8_t* values;
	uint64_t       n_vec;
	uint32_t       width;
	uint32_t       sgn;
};

// A work item: vector `vec` of column `col`; `chunk` its chunk, `cpos` its index inside the chunk.
struct Item {
	uint32_t col;
	uint32_t chunk;
	uint32_t vec;
	uint32_t cpos;
};

template <int W>
struct UT;
template <>
struct UT<32> {
	using T = uint32_t;
};
template <>
struct UT<64> {
	using T = uint64_t;
};

__device__ __forceinline__ uint32_t bits_of(uint64_t d) { return d ? 64u - static_cast<uint32_t>(__clzll(d)) : 0u; }

template <class T>
__device__ __forceinline__ T warp_min(T x) {
#pragma unroll
	for (int d = 16; d > 0; d >>= 1) {
		const T y = __shfl_xor_sync(0xFFFFFFFFu, x, d);
		x         = y < x ? y : x;
	}
	return x;
}
template <class T>
__device__ __forceinline__ T warp_max(T x) {
#pragma unroll
	for (int d = 16; d > 0; d >>= 1) {
		const T y = __shfl_xor_sync(0xFFFFFFFFu, x, d);
		x         = y > x ? y : x;
	}
	return x;
}

__device__ __forceinline__ uint32_t thread_run(uint32_t t) { return (t % 16) * 64 + 32 * (t / 16); }
// Lane whose run holds original position R(t) - 1 (t > 0).
__device__ __forceinline__ uint32_t prev_run_lane(uint32_t t) { return t >= 16 ? t - 16 : t + 15; }
// Thread runs in original order: virtual position u = 2 (t % 16) + t / 16.
__device__ __forceinline__ uint32_t lane_of_virtual(uint32_t u) { return (u >> 1) + 16 * (u & 1); }
__device__ __forceinline__ uint32_t virtual_of_lane(uint32_t t) { return 2 * (t % 16) + t / 16; }

// Exclusive sum of c over the thread runs in original order.
__device__ __forceinline__ uint32_t run_exclusive(uint32_t c, uint32_t lane) {
	const uint32_t cv  = __shfl_sync(0xFFFFFFFFu, c, lane_of_virtual(lane));
	const uint32_t inc = warp_inclusive_scan(cv, lane);
	return __shfl_sync(0xFFFFFFFFu, inc - cv, virtual_of_lane(lane));
}

template <int W>
__device__ __forceinline__ void load_run(const Col& c, uint64_t v, uint32_t lane, typename UT<W>::T (&x)[32]) {
	using T          = typename UT<W>::T;
	const uint4* src = reinterpret_cast<const uint4*>(c.values + (v * 1024 + thread_run(lane)) * sizeof(T));
	constexpr int n  = 32 * sizeof(T) / 16;
	uint4         b[n];
#pragma unroll
	for (int i = 0; i < n; ++i) { b[i] = __ldg(src + i); }
#pragma unroll
	for (int i = 0; i < n; ++i) {
		if constexpr (W == 32) {
			x[4 * i] = b[i].x, x[4 * i + 1] = b[i].y, x[4 * i + 2] = b[i].z, x[4 * i + 3] = b[i].w;
		} else {
			x[2 * i]     = (static_cast<uint64_t>(b[i].y) << 32) | b[i].x;
			x[2 * i + 1] = (static_cast<uint64_t>(b[i].w) << 32) | b[i].z;
		}
	}
}

// The size-model quantities of one vector (warp-uniform results).
struct Parts {
	uint32_t bw_f, bw_d, bw_i, runs;
	uint32_t start_mask; // this thread's run starts (bit i: original position R(t) + i starts a run)
	uint64_t lo, hi;     // lowest and highest value, in the column's order (signed: the top bit flipped)
};

template <int W>
__device__ __forceinline__ Parts vector_parts(const typename UT<W>::T (&x)[32], uint32_t lane, bool sgn) {
	using T      = typename UT<W>::T;
	const T flip = sgn ? (T(1) << (W - 1)) : T(0);
	Parts   P;
	// FFOR: range of the values (signed order through the flipped top bit)
	T mn = x[0] ^ flip, mx = mn;
#pragma unroll
	for (int i = 1; i < 32; ++i) {
		const T k = x[i] ^ flip;
		mn        = k < mn ? k : mn;
		mx        = k > mx ? k : mx;
	}
	mn     = warp_min(mn);
	mx     = warp_max(mx);
	P.bw_f = bits_of(static_cast<uint64_t>(static_cast<T>(mx - mn)));
	P.lo   = mn;
	P.hi   = mx;
	// DELTA: the unrsum chains of the transposed layout visit a lane's values in ascending original order, so
	// a chain is a run of contiguous original positions (W = 32: this thread's 32; W = 64: 64, this thread's
	// and its partner's); every chain's first difference is 0
	T dmn = flip, dmx = flip;
#pragma unroll
	for (int c = 1; c < 32; ++c) {
		const T k = static_cast<T>(x[c] - x[c - 1]) ^ flip;
		dmn       = k < dmn ? k : dmn;
		dmx       = k > dmx ? k : dmx;
	}
	if constexpr (W == 64) {
		const T lower = __shfl_xor_sync(0xFFFFFFFFu, x[31], 16);
		if (lane >> 4) {
			const T k = static_cast<T>(x[0] - lower) ^ flip;
			dmn       = k < dmn ? k : dmn;
			dmx       = k > dmx ? k : dmx;
		}
	}
	dmn    = warp_min(dmn);
	dmx    = warp_max(dmx);
	P.bw_d = bits_of(static_cast<uint64_t>(static_cast<T>(dmx - dmn)));
	// RLE: run starts in original order
	const T  prev = __shfl_sync(0xFFFFFFFFu, x[31], prev_run_lane(lane));
	uint32_t sm   = (lane == 0 || x[0] != prev) ? 1u : 0u;
#pragma unroll
	for (int i = 1; i < 32; ++i) { sm |= (x[i] != x[i - 1] ? 1u : 0u) << i; }
	P.start_mask = sm;
	P.runs       = warp_sum(static_cast<uint32_t>(__popc(sm)));
	// the u16 run index: each of its chains is 16 contiguous positions (this thread's [0,16) and [16,32)), so
	// its deltas are the run starts inside a chain (0 or 1) and the range is 1 as soon as one run starts there
	P.bw_i = __any_sync(0xFFFFFFFFu, (sm & 0xFFFEFFFEu) != 0) ? 1u : 0u;
	return P;
}

__device__ __forceinline__ uint32_t pack_parts(const Parts& p) {
	return p.bw_f | (p.bw_d << 7) | (p.bw_i << 14) | (p.runs << 19);
}

// ---------------------------------------------------------------------------------------------------------
// Statistics of the learned selector (one warp, one vector).  slots: this warp's table, 2048 entries of 11 hash bits,
// the 10-bit position of the key's first value put in (the key itself: vals holds the vector) and an 11-bit count.
// 4 bytes an entry instead of 12 let 16 warps run on an SM instead of 8, and the loop over the vector's rows, instead
// of 32 inserts in line, fits the instruction cache: the kernel waited on latency and on instruction fetch.
// 3,660 vectors: 105 us, 79 us so.
// ---------------------------------------------------------------------------------------------------------
constexpr uint32_t kHSlots = 2048;

// the odd multipliers are xxHash's 32-bit primes 1, 2 and 3 (Collet)
template <class T>
__device__ __forceinline__ uint32_t feat_hash(T x) {
	uint32_t a = static_cast<uint32_t>(x) * 0x9E3779B1u;
	if constexpr (sizeof(T) == 8) { a += static_cast<uint32_t>(x >> 32) * 0x85EBCA77u; }
	a ^= a >> 15;
	a *= 0xC2B2AE3Du;
	return a ^ (a >> 13);
}

// Counts of the vector's values into the (empty) table: a row of 32 neighbouring values a step, one insert a run.
template <class T>
__device__ __forceinline__ void count_values(const T* vals, uint32_t lane, uint32_t* slots) {
#pragma unroll 2
	for (uint32_t r = 0; r < 32; ++r) {
		const T        x     = __ldg(vals + 32 * r + lane);
		const T        prev  = __shfl_up_sync(0xFFFFFFFFu, x, 1);
		const bool     start = lane == 0 || x != prev;
		const uint32_t after = (__ballot_sync(0xFFFFFFFFu, start) >> lane) >> 1; // the starts past this lane
		if (start) {
			const uint32_t weight = after ? __ffs(after) : 32 - lane;
			const uint32_t h      = feat_hash(x);
			const uint32_t tag = h << 21, mine = tag | ((32 * r + lane) << 11) | weight;
			uint32_t       s   = h >> 21;
			for (uint32_t probe = 0; probe < kHSlots; ++probe) {
				uint32_t e = *reinterpret_cast<volatile uint32_t*>(slots + s);
				if (e == 0) {
					e = atomicCAS(slots + s, 0u, mine);
					if (e == 0) { break; }
				}
				if ((e ^ tag) < (1u << 21) && __ldg(vals + ((e >> 11) & 1023u)) == x) {
					atomicAdd(slots + s, weight);
					break;
				}
				s = (s + 1) & (kHSlots - 1);
			}
		}
	}
	__syncwarp();
}

template <int W>
__device__ void vector_features(const typename UT<W>::T (&x)[32], uint32_t lane, bool sgn, const Parts& P,
                                const typename UT<W>::T* vals, uint32_t* slots, float* out) {
	using T             = typename UT<W>::T;
	const T        flip = sgn ? (T(1) << (W - 1)) : T(0);
	const uint32_t sm   = P.start_mask;
	// distinct values and the top multiplicity (exact: 1024 values in 2048 slots)
	count_values(vals, lane, slots);
	uint32_t dv = 0, top = 0;
	for (uint32_t s = lane; s < kHSlots / 4; s += 32) {
		const uint4    e    = reinterpret_cast<const uint4*>(slots)[s];
		const uint32_t w[4] = {e.x, e.y, e.z, e.w};
#pragma unroll
		for (int i = 0; i < 4; ++i) {
			const uint32_t c = w[i] & 0x7FFu;
			dv += c ? 1u : 0u;
			top = c > top ? c : top;
		}
		reinterpret_cast<uint4*>(slots)[s] = make_uint4(0, 0, 0, 0);
	}
	dv  = warp_sum(dv);
	top = warp_max(top);
	__syncwarp();
	// adjacency in original order: increases, decreases, largest |difference|
	const T  prev = __shfl_sync(0xFFFFFFFFu, x[31], prev_run_lane(lane));
	uint32_t inc = 0, dec = 0, bw_a = 0;
#pragma unroll
	for (int i = 0; i < 32; ++i) {
		if (i == 0 && lane == 0) { continue; }
		const T a = (i == 0 ? prev : x[i - 1]);
		const T b = x[i];
		inc += ((b ^ flip) > (a ^ flip)) ? 1u : 0u;
		dec += ((b ^ flip) < (a ^ flip)) ? 1u : 0u;
		T d = static_cast<T>(b - a);
		if (d >> (W - 1)) { d = static_cast<T>(T(0) - d); }
		bw_a = max(bw_a, bits_of(static_cast<uint64_t>(d)));
	}
	inc  = warp_sum(inc);
	dec  = warp_sum(dec);
	bw_a = warp_max(bw_a);
	// longest run: the run in progress entering each thread comes from a scan (original order) of
	// f(L) = (no start in the thread) ? L + 32 : length of the thread's last run
	const uint32_t u    = virtual_of_lane(lane);
	uint32_t       cont = sm == 0 ? 1u : 0u;
	uint32_t       cval = sm == 0 ? 32u : static_cast<uint32_t>(__clz(sm)) + 1u;
	{
		uint32_t a = __shfl_sync(0xFFFFFFFFu, cont, lane_of_virtual(lane));
		uint32_t c = __shfl_sync(0xFFFFFFFFu, cval, lane_of_virtual(lane));
#pragma unroll
		for (int d = 1; d < 32; d <<= 1) {
			const uint32_t pa = __shfl_up_sync(0xFFFFFFFFu, a, d);
			const uint32_t pc = __shfl_up_sync(0xFFFFFFFFu, c, d);
			if (lane >= static_cast<uint32_t>(d)) {
				c = a ? pc + c : c;
				a = pa & a;
			}
		}
		// virtual lane `lane` now holds the composition up to it; the run entering virtual u is that of u - 1
		const uint32_t entering_v = __shfl_up_sync(0xFFFFFFFFu, c, 1);
		const uint32_t ent        = __shfl_sync(0xFFFFFFFFu, lane == 0 ? 0u : entering_v, u);
		uint32_t       best       = 0;
		if (sm != 0) {
			const uint32_t head = static_cast<uint32_t>(__ffs(sm)) - 1u;
			best                = ent + head; // the run in progress ends at the first start (0 when nothing entered)
			int last            = -1;
#pragma unroll
			for (int i = 0; i < 32; ++i) {
				if ((sm >> i) & 1u) {
					if (last >= 0) { best = max(best, static_cast<uint32_t>(i - last)); }
					last = i;
				}
			}
		}
		if (u == 31) { best = max(best, sm == 0 ? ent + 32u : static_cast<uint32_t>(__clz(sm)) + 1u); }
		cval = warp_max(best);
	}
	const uint32_t maxrun = cval;
	// values with the top bit of (x - min) set, block ranges, zeros, min / max counts, magnitude
	T mnk = x[0] ^ flip, mxk = mnk;
#pragma unroll
	for (int i = 1; i < 32; ++i) {
		const T k = x[i] ^ flip;
		mnk       = k < mnk ? k : mnk;
		mxk       = k > mxk ? k : mxk;
	}
	const uint32_t blk = bits_of(static_cast<uint64_t>(static_cast<T>(mxk - mnk)));
	mnk                = warp_min(mnk);
	mxk                = warp_max(mxk);
	const T  mn = mnk ^ flip, mx = mxk ^ flip;
	uint32_t cnt_top = 0, nzero = 0, nmin = 0, nmax = 0, mag = 0;
#pragma unroll
	for (int i = 0; i < 32; ++i) {
		if (P.bw_f > 0) { cnt_top += static_cast<uint32_t>((static_cast<T>(x[i] - mn) >> (P.bw_f - 1)) & 1u); }
		nzero += x[i] == 0 ? 1u : 0u;
		nmin += x[i] == mn ? 1u : 0u;
		nmax += x[i] == mx ? 1u : 0u;
		T a = x[i];
		if (sgn && (a >> (W - 1))) { a = static_cast<T>(T(0) - a); }
		mag = max(mag, bits_of(static_cast<uint64_t>(a)));
	}
	cnt_top              = warp_sum(cnt_top);
	nzero                = warp_sum(nzero);
	nmin                 = warp_sum(nmin);
	nmax                 = warp_sum(nmax);
	mag                  = warp_max(mag);
	const uint32_t blk_s = warp_sum(blk);
	// lane f writes feature f
	const float    w = static_cast<float>(W), raw = 1024.0f * (W / 8), sz = static_cast<float>(W / 8);
	const float    r = static_cast<float>(P.runs), fdv = static_cast<float>(dv);
	const uint32_t cb = bits_of(dv - 1);
	float          f  = 0.0f;
	switch (lane) {
	case 0: f = P.bw_f / w; break;
	case 1: f = P.bw_d / w; break;
	case 2: f = r / 1024.0f; break;
	case 3: f = P.bw_i / 16.0f; break;
	case 4: f = fdv / 1024.0f; break;
	case 5: f = log2f(fdv) / 10.0f; break;
	case 6: f = cb / 16.0f; break;
	case 7: f = inc / 1023.0f; break;
	case 8: f = dec / 1023.0f; break;
	case 9: f = bw_a / w; break;
	case 10: f = maxrun / 1024.0f; break;
	case 11: f = log2f(1024.0f / r) / 10.0f; break;
	case 12: f = top / 1024.0f; break;
	case 13: f = cnt_top / 1024.0f; break;
	case 14: f = blk_s / (32.0f * w); break;
	case 15: f = w / 64.0f; break;
	case 16: f = sgn ? 1.0f : 0.0f; break;
	case 17: f = (1.0f + sz + 128.0f * P.bw_f) / raw; break;
	case 18: f = (129.0f + sz + 128.0f * P.bw_d) / raw; break;
	case 19: f = (r * sz + 131.0f + 128.0f * P.bw_i) / raw; break;
	case 20: f = (fdv * sz + 5.0f + 128.0f * cb) / raw; break;
	case 21: f = (fdv * sz + 4.0f * r + 131.0f + 128.0f * P.bw_i) / raw; break;
	case 22: f = mag / w; break;
	case 23: f = nzero / 1024.0f; break;
	case 24: f = fdv / r; break;
	case 25: f = log2f(static_cast<float>(maxrun)) / 10.0f; break;
	case 26: f = bits_of(top) / 11.0f; break;
	case 27: f = nmin / 1024.0f; break;
	case 28: f = nmax / 1024.0f; break;
	case 29: f = (static_cast<float>(P.bw_f) - blk_s / 32.0f) / w; break;
	case 30: f = P.bw_f == 0 ? 1.0f : 0.0f; break;
	default: f = dec == 0 ? 1.0f : 0.0f; break;
	}
	out[lane] = f;
}

// ---------------------------------------------------------------------------------------------------------
// Kernels over work items (warp per vector)
// ---------------------------------------------------------------------------------------------------------
// What k_parts notes of every vector for the chunk dictionary: in the column's order (signed columns with the top bit
// flipped) its lowest, highest, first and last value, its runs and whether its values never fall.
struct VecInfo {
	uint64_t lo, hi, first, last;
	uint32_t runs, sorted;
};

template <int W>
__device__ __forceinline__ void note_vector(const typename UT<W>::T (&x)[32], uint32_t lane, bool sgn, const Parts& P,
                                            VecInfo* out) {
	using T         = typename UT<W>::T;
	const T  flip   = sgn ? (T(1) << (W - 1)) : T(0);
	const T  prev   = __shfl_sync(0xFFFFFFFFu, x[31], prev_run_lane(lane));
	bool     falls  = lane > 0 && (x[0] ^ flip) < (prev ^ flip);
#pragma unroll
	for (int i = 1; i < 32; ++i) { falls |= (x[i] ^ flip) < (x[i - 1] ^ flip); }
	falls        = __any_sync(0xFFFFFFFFu, falls);
	const T last = __shfl_sync(0xFFFFFFFFu, x[31], lane_of_virtual(31));
	if (lane == 0) { *out = VecInfo {P.lo, P.hi, static_cast<uint64_t>(x[0] ^ flip), static_cast<uint64_t>(last ^ flip), P.runs, falls ? 0u : 1u}; }
}

struct ItemArgs {
	const Col*  cols;
	const Item* items;
	uint64_t    n_items;
};

__global__ void __launch_bounds__(kWarps * 32) k_parts(ItemArgs a, uint32_t* parts, VecInfo* info) {
	const uint32_t lane = threadIdx.x & 31u;
	for (uint64_t it = blockIdx.x * static_cast<uint64_t>(kWarps) + (threadIdx.x >> 5); it < a.n_items;
	     it += static_cast<uint64_t>(gridDim.x) * kWarps) {
		const Item m = a.items[it];
		const Col  c = a.cols[m.col];
		if (c.width == 64) {
			uint64_t x[32];
			load_run<64>(c, m.vec, lane, x);
			const Parts P = vector_parts<64>(x, lane, c.sgn != 0);
			if (lane == 0) { parts[it] = pack_parts(P); }
			if (info) { note_vector<64>(x, lane, c.sgn != 0, P, info + it); }
		} else {
			uint32_t x[32];
			load_run<32>(c, m.vec, lane, x);
			const Parts P = vector_parts<32>(x, lane, c.sgn != 0);
			if (lane == 0) { parts[it] = pack_parts(P); }
			if (info) { note_vector<32>(x, lane, c.sgn != 0, P, info + it); }
		}
	}
}

constexpr uint32_t kFeatSmem = kWarps * kHSlots * 4;

__global__ void __launch_bounds__(kWarps * 32, 2) k_features(ItemArgs a, float* feat) {
	extern __shared__ __align__(16) uint8_t fsm[];
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	uint32_t*      hs   = reinterpret_cast<uint32_t*>(fsm) + warp * kHSlots;
	for (uint32_t s = lane; s < kHSlots; s += 32) { hs[s] = 0; }
	__syncwarp();
	for (uint64_t it = blockIdx.x * static_cast<uint64_t>(kWarps) + warp; it < a.n_items;
	     it += static_cast<uint64_t>(gridDim.x) * kWarps) {
		const Item m = a.items[it];
		const Col  c = a.cols[m.col];
		if (c.width == 64) {
			uint64_t x[32];
			load_run<64>(c, m.vec, lane, x);
			const Parts P = vector_parts<64>(x, lane, c.sgn != 0);
			vector_features<64>(x, lane, c.sgn != 0, P, reinterpret_cast<const uint64_t*>(c.values) + m.vec * 1024ull, hs, feat + it * NF);
		} else {
			uint32_t x[32];
			load_run<32>(c, m.vec, lane, x);
			const Parts P = vector_parts<32>(x, lane, c.sgn != 0);
			vector_features<32>(x, lane, c.sgn != 0, P, reinterpret_cast<const uint32_t*>(c.values) + m.vec * 1024ull, hs, feat + it * NF);
		}
		__syncwarp();
	}
}

// ---------------------------------------------------------------------------------------------------------
// Dictionary of a chunk (wizard), one CTA per chunk: the chunk's distinct values, numbered in first-occurrence
// order (src/cor/lyt/dic/dic_fac.cpp:19-40), give the dictionary size and every vector's code bit width.  Codes
// rise with the first position, so a vector's code range is the rank of the largest first position among its values
// minus that of the smallest: two ranks a vector (popcounts of the bitmap of first positions), none a value.
//   sorted    a chunk whose values never fall (k_parts says) needs no table: every run is a new code;
//   direct    a chunk whose values span fewer than 47 Ki keeps first positions by value - lowest, no hash;
//   unique    a chunk of nearly all different values: every run start sets a bit of a 1 Mbit filter by its hash; the
//             few that find theirs set mark a coarser filter, and only the values whose mark is set (a few percent)
//             need the table: the others are the only ones of their kind, their first position is their own;
//   table     47 Ki slots of 32 bits in shared memory, open addressing: 16 bits of the key's hash and the 16-bit
//             position of its first occurrence seen so far (the chunk's values stay in L2, so the key itself is read
//             back from that position when the hash bits agree).  A slot of 4 bytes instead of a 64-bit key and a
//             position (12) is what lets one table hold most of a chunk of distinct values;
//   queue     a warp takes whole vectors (in chunks of few, some rows of one), and every step looks at one slot for each
//             of 32 keys from the warp's queue in shared memory; keys that have to look further go back on it.  So
//             runs, other parts' keys and long probes cost no idle lanes (a loop of its own for every warp of keys
//             went round for its unluckiest lane, 200 to 300 instructions a step);
//   parts     a chunk of more distinct values goes through the table in parts of the hash space (2, then 4); the count
//             beside the rows done says early whether it will;
//   sort      keys that crowd, whatever the reason (every hash has such keys), spend a warp's looks or overflow four
//             parts: their chunk's positions are sorted by value instead.
// Exact for every chunk: the hash only decides how long it takes.  Instruction-bound.  28 integer columns (30 M values, 462
// chunks): 1,855 us with 16 Ki slots of keys and positions and a bucket pass through global memory, 275 us so; 5.7 M
// string hashes (90 chunks): 710 us, 139 us.
// ---------------------------------------------------------------------------------------------------------
constexpr uint32_t kCdThreads = 1024;
constexpr uint32_t kCdWarps   = kCdThreads / 32;
constexpr uint32_t kCdSlots   = 47 * 1024;
constexpr uint32_t kCdCap     = 43 * 1024; // keys the table takes (eleven twelfths), and those in flight
constexpr uint32_t kCdMaxParts = 4; // two hold every chunk whose keys spread
// looks a warp may spend on the keys of one filling of the table.  Keys that spread leave it far away (a table filled to
// kCdCap takes some 300 a warp, a warp whose 2,048 keys all come last some 5,000); keys that crowd are sorted instead.
constexpr uint32_t kCdLooks    = 1u << 14;
constexpr uint32_t kCdWords   = kMaxVecPerChunk * 1024 / 32;
constexpr uint64_t kCdGBytes  = kMaxVecPerChunk * 1024 * 2; // per CTA: the slots of every vector's keys
// unique: the filter (2^20 bits) lies where the table of the marked values then goes; behind it the marks (2^18 bits)
constexpr uint32_t kCdUniqueSlots = 32 * 1024;
constexpr uint32_t kCdMarkWords   = 8 * 1024;
constexpr uint32_t kCdUniqueMax   = 8 * 1024;  // values that may find their bit set; marked are about twice as many
constexpr uint32_t kCdUniqueCap   = 28 * 1024; // keys its table takes (keys chosen to share marks could be more)
static_assert(kCdUniqueSlots + kCdMarkWords <= kCdSlots, "filter and marks lie in the table's space");
static_assert(kCdCap + 2 * kCdThreads < kCdSlots && kCdSlots < 0xFFFFu, "free slots always; slots in 16 bits");

struct ChunkDictSmem {
	uint32_t table[kCdSlots]; // at the end: the exclusive prefix of the bitmap words' popcounts
	uint32_t bits[kCdWords];  // first positions
	uint64_t qkey[kCdWarps][kCdQueue];
	uint16_t qpos[kCdWarps][kCdQueue], qslot[kCdWarps][kCdQueue], qtag[kCdWarps][kCdQueue];
	uint32_t vrange[kMaxVecPerChunk][2]; // smallest and largest first position of a vector's values
	uint32_t wsum[33];
	uint32_t chunk, over, spent, count, mode, distinct;
	uint64_t lo;    // direct: the lowest value
	uint64_t dw[2]; // weights of the first positions
};
static_assert(sizeof(ChunkDictSmem) <= 227 * 1024, "chunk dictionary tables fit one CTA");
enum : uint32_t { CD_SORTED, CD_DIRECT, CD_UNIQUE /* to be tried */, CD_TABLE };

struct ChunkDictArgs {
	const Col*      cols;
	const Item*     items;       // the chunks' vectors, chunk by chunk
	const VecInfo*  info;        // per item
	const uint32_t* chunk_items; // item range of every chunk (n_chunks + 1)
	uint32_t        n_chunks;
	uint32_t*       dict_n;  // per chunk: distinct values
	uint32_t*       bw_code; // per item: FFOR bit width of its codes
	int*            status;
	// string columns (optional): per-row weights of every column (row = vector * 1024 + position), summed over
	// the first occurrences of a chunk's distinct values into dict_w[chunk][0..1] (the dictionary's raw and
	// FSST-compressed bytes)
	const uint32_t* const* w0;
	const uint32_t* const* w1;
	uint64_t*       dict_w;
	uint16_t*       gslots; // gridDim.x regions of kCdGBytes
	uint32_t*       ticket; // zero: the next chunk to take
};

// How the chunk of items [i0, i0 + nv) is done (warp 0; CD_*), from its vectors' notes.
__device__ __forceinline__ void cd_choose(const ChunkDictArgs& a, uint32_t i0, uint32_t nv, uint32_t lane,
                                          ChunkDictSmem& S) {
	uint64_t lo = ~0ull, hi = 0;
	uint32_t runs = 0, borders = 0, unsorted = 0;
	for (uint32_t v = lane; v < nv; v += 32) {
		const VecInfo m = a.info[i0 + v];
		lo              = m.lo < lo ? m.lo : lo;
		hi              = m.hi > hi ? m.hi : hi;
		runs += m.runs;
		unsorted |= m.sorted ? 0u : 1u;
		if (v + 1 < nv) { // a run across the border of two vectors is one code
			const uint64_t next = a.info[i0 + v + 1].first;
			unsorted |= next < m.last ? 1u : 0u;
			borders += next == m.last ? 1u : 0u;
		}
	}
	lo       = warp_min(lo);
	hi       = warp_max(hi);
	runs     = warp_sum(runs);
	borders  = warp_sum(borders);
	unsorted = __any_sync(0xFFFFFFFFu, unsorted != 0);
	if (lane == 0) {
		S.lo       = lo;
		S.spent    = 0;
		S.distinct = runs - borders; // of a sorted chunk
		// fewer runs than the table takes in one part with room to spare go straight to it
		S.mode = !unsorted && !a.w0 ? CD_SORTED : hi - lo < kCdSlots ? CD_DIRECT : runs > kCdCap / 2 ? CD_UNIQUE : CD_TABLE;
	}
}

// First positions and vector ranges of a chunk without a hash: its positions (order: space for them in global memory)
// sorted by value and then position with Batcher's merge exchange (Knuth, The Art of Computer Programming 3, algorithm
// 5.2.2M), so that the positions of a value stand side by side, the first one in front.  136 passes over 65,536
// positions: 15 ms for a chunk with the looks spent before, however its keys are made (0.13 ms for keys that spread).
template <class T>
__device__ __noinline__ void cd_sort(const T* vals, uint32_t nv, uint16_t* order, const uint32_t* w0, const uint32_t* w1,
                                     ChunkDictSmem& S) {
	const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, n = nv * 1024;
	for (uint32_t i = tid; i < n; i += kCdThreads) { order[i] = static_cast<uint16_t>(i); }
	__syncthreads();
	const uint32_t top = 1u << (31 - __clz(n - 1)); // the largest power of two below n
	for (uint32_t p = top; p > 0; p >>= 1) {
		uint32_t r = 0, d = p;
		for (uint32_t q = top;; q >>= 1) {
			for (uint32_t i = tid; i + d < n; i += kCdThreads) {
				if ((i & p) != r) { continue; }
				const uint32_t a = order[i], b = order[i + d];
				const T        x = __ldg(vals + a), y = __ldg(vals + b);
				if (x > y || (x == y && a > b)) {
					order[i]     = static_cast<uint16_t>(b);
					order[i + d] = static_cast<uint16_t>(a);
				}
			}
			__syncthreads();
			if (q == p) { break; }
			d = q - p;
			r = p;
		}
	}
	// nv neighbouring positions a thread; each takes its value's first position from the last head (the first position
	// of a value) up to it, which may lie in an earlier thread's stretch: a scan hands it on
	const uint32_t i0 = tid * nv;
	auto           is_head = [&](uint32_t i) { return i == 0 || __ldg(vals + order[i]) != __ldg(vals + order[i - 1]); };
	uint32_t       head = 0; // the stretch's last one, plus one
	uint64_t       s0 = 0, s1 = 0;
	for (uint32_t i = i0; i < i0 + nv; ++i) {
		if (!is_head(i)) { continue; }
		const uint32_t f = order[i];
		head             = i + 1;
		atomicOr(S.bits + (f >> 5), 1u << (f & 31u));
		if (w0) {
			s0 += __ldg(w0 + f);
			s1 += __ldg(w1 + f);
		}
	}
	if (w0) {
		atomicAdd(reinterpret_cast<unsigned long long*>(S.dw), static_cast<unsigned long long>(s0));
		atomicAdd(reinterpret_cast<unsigned long long*>(S.dw + 1), static_cast<unsigned long long>(s1));
	}
	uint32_t upto = head; // the last head of the warp's lanes up to this one
	for (uint32_t d = 1; d < 32; d <<= 1) {
		const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, upto, d);
		if (lane >= d) { upto = max(upto, y); }
	}
	uint32_t before = __shfl_up_sync(0xFFFFFFFFu, upto, 1);
	if (lane == 0) { before = 0; }
	if (lane == 31) { S.wsum[warp] = upto; }
	__syncthreads();
	for (uint32_t w = 0; w < warp; ++w) { before = max(before, S.wsum[w]); }
	uint32_t f = before ? order[before - 1] : 0u;
	for (uint32_t i = i0; i < i0 + nv; ++i) {
		const uint32_t pos = order[i];
		if (is_head(i)) { f = pos; }
		atomicMin(&S.vrange[pos >> 10][0], f);
		atomicMax(&S.vrange[pos >> 10][1], f);
	}
	__syncthreads();
}

template <int W>
__device__ __forceinline__ void chunk_dict(const ChunkDictArgs& a, const Col& col, uint32_t c, ChunkDictSmem& S) {
	using T             = typename UT<W>::T;
	const uint32_t tid  = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
	const uint32_t i0   = a.chunk_items[c], nv = a.chunk_items[c + 1] - i0;
	const Item     m0   = a.items[i0];
	const uint64_t row0 = static_cast<uint64_t>(m0.vec - m0.cpos) * 1024; // the chunk's first value
	const T*       vals = reinterpret_cast<const T*>(col.values) + row0;
	uint16_t*      slots = a.gslots + blockIdx.x * (kCdGBytes / 2);
	if (warp == 0) { cd_choose(a, i0, nv, lane, S); }
	__syncthreads();
	const uint32_t mode = S.mode;
	if (mode == CD_SORTED) {
		if (tid < nv) { a.bw_code[i0 + tid] = bits_of(a.info[i0 + tid].runs - 1); }
		if (tid == 0) { a.dict_n[c] = S.distinct; }
		__syncthreads(); // S is read to the end before the next chunk's choice
		return;
	}
	const T            flip = col.sgn ? (T(1) << (W - 1)) : T(0);
	const T            low  = static_cast<T>(S.lo);
	const uint32_t*    w0   = a.w0 ? a.w0[m0.col] + row0 : nullptr;
	const uint32_t*    w1   = a.w0 ? a.w1[m0.col] + row0 : nullptr;
	volatile uint32_t* over = &S.over;
	uint64_t           sw0 = 0, sw1 = 0; // weights of the first positions this thread finds
	CdQueue<T>         Q {reinterpret_cast<T*>(S.qkey[warp]), S.qpos[warp], S.qslot[warp], S.qtag[warp], nullptr, 0, 0, 0};
	// a warp's units: warp, warp + kCdWarps.  A unit is a vector, or some of its rows where there are fewer vectors than
	// half the warps (4,096 chunks of one vector: 973 us with a warp each, 293 so)
	constexpr uint32_t kPer  = kMaxVecPerChunk / kCdWarps;
	const uint32_t     split = nv < kCdWarps ? 31 - __clz(kCdWarps / nv) : 0; // log2 of a vector's units
	const uint32_t     units = nv << split, unit_rows = 32u >> split;
	auto               first_row = [&](uint32_t u) { return (u << (5 - split)) & 31u; };
	uint32_t           listed[kPer];
	auto clear = [&](uint32_t words) { // of the table
		for (uint32_t k = tid; k < words / 4; k += kCdThreads) {
			reinterpret_cast<uint4*>(S.table)[k] = make_uint4(kCdFree, kCdFree, kCdFree, kCdFree);
		}
	};
	auto reset = [&]() { // before anything is found
		for (uint32_t k = tid; k < kCdWords; k += kCdThreads) { S.bits[k] = 0; }
		if (tid < kMaxVecPerChunk) {
			S.vrange[tid][0] = ~0u;
			S.vrange[tid][1] = 0u;
		}
		sw0 = sw1 = 0;
	};
	// row r of vector v: this lane's value, and whether it starts a run (the first value of row r0, a unit's first, counts
	// as one)
	T    last = 0;
	auto row  = [&](uint32_t v, uint32_t r, uint32_t r0, T* x) {
		*x     = __ldg(vals + v * 1024 + r * 32 + lane);
		T prev = __shfl_up_sync(0xFFFFFFFFu, *x, 1);
		if (lane == 0) { prev = last; }
		last = __shfl_sync(0xFFFFFFFFu, *x, 31);
		return *x != prev || (r == r0 && lane == 0);
	};
	// the ranges of the warp's vectors from their slots (the table holds the first positions), and the first positions
	// themselves; the table is read to the end at the closing barrier
	auto collect = [&](uint32_t n_slots) {
#pragma unroll
		for (uint32_t j = 0; j < kPer; ++j) {
			const uint32_t  u    = warp + j * kCdWarps;
			const uint16_t* list = slots + u * unit_rows * 32;
			uint32_t        lo = ~0u, hi = 0u;
#pragma unroll 4
			for (uint32_t i = lane; i < listed[j]; i += 32) {
				const uint32_t f = S.table[list[i]] & 0xFFFFu;
				lo               = min(lo, f);
				hi               = max(hi, f);
			}
			lo = __reduce_min_sync(0xFFFFFFFFu, lo);
			hi = __reduce_max_sync(0xFFFFFFFFu, hi);
			if (lane == 0 && lo != ~0u) {
				atomicMin(&S.vrange[u >> split][0], lo);
				atomicMax(&S.vrange[u >> split][1], hi);
			}
		}
#pragma unroll 4
		for (uint32_t k = tid; k < n_slots; k += kCdThreads) {
			const uint32_t e = S.table[k];
			if (e != kCdFree) {
				const uint32_t f = e & 0xFFFFu;
				atomicOr(S.bits + (f >> 5), 1u << (f & 31u));
				if (w0) {
					sw0 += __ldg(w0 + f);
					sw1 += __ldg(w1 + f);
				}
			}
		}
		__syncthreads();
	};
	if (tid < 2) { S.dw[tid] = 0; }
	bool found = false;
	if (mode == CD_DIRECT) {
		reset();
		clear(kCdSlots);
		__syncthreads();
		auto entry = [&](T x) { return S.table + static_cast<uint32_t>(static_cast<T>((x ^ flip) - low)); };
		for (uint32_t u = warp; u < units; u += kCdWarps) {
#pragma unroll 8
			for (uint32_t r = 0; r < unit_rows; ++r) {
				const uint32_t pos = (u * unit_rows + r) * 32 + lane;
				uint32_t*      e   = entry(__ldg(vals + pos));
				if (pos < *reinterpret_cast<volatile uint32_t*>(e)) { atomicMin(e, pos); }
			}
		}
		__syncthreads();
		for (uint32_t u = warp; u < units; u += kCdWarps) {
			uint32_t lo = ~0u, hi = 0u;
#pragma unroll 8
			for (uint32_t r = 0; r < unit_rows; ++r) {
				const uint32_t f = *entry(__ldg(vals + (u * unit_rows + r) * 32 + lane));
				lo               = min(lo, f);
				hi               = max(hi, f);
			}
			lo = __reduce_min_sync(0xFFFFFFFFu, lo);
			hi = __reduce_max_sync(0xFFFFFFFFu, hi);
			if (lane == 0) {
				atomicMin(&S.vrange[u >> split][0], lo);
				atomicMax(&S.vrange[u >> split][1], hi);
			}
		}
#pragma unroll
		for (uint32_t j = 0; j < kPer; ++j) { listed[j] = 0; }
		collect(kCdSlots);
		found = true;
	}
	if (mode == CD_UNIQUE) {
		uint32_t* filter = S.table;
		uint32_t* marks  = S.table + kCdUniqueSlots;
		reset();
		for (uint32_t k = tid; k < kCdUniqueSlots + kCdMarkWords; k += kCdThreads) { S.table[k] = 0; }
		if (tid == 0) { S.count = S.over = 0; }
		__syncthreads();
		bool stop = false;
		for (uint32_t v = warp; v < nv && !stop; v += kCdWarps) {
			for (uint32_t r0 = 0; r0 < 32 && !stop; r0 += 4) {
				uint32_t set = 0;
#pragma unroll
				for (uint32_t i = 0; i < 4; ++i) {
					T          x;
					const bool start = row(v, r0 + i, 0, &x);
					uint32_t   place, other;
					cd_hash(x, &place, &other);
					const uint32_t b = place >> 12;
					if (start && ((atomicOr(filter + (b >> 5), 1u << (b & 31u)) >> (b & 31u)) & 1u)) {
						atomicOr(marks + (b >> 7), 1u << ((b >> 2) & 31u));
						++set;
					}
				}
				set = __reduce_add_sync(0xFFFFFFFFu, set);
				if (lane == 0) {
					// too many already, or on the way there
					const uint32_t now = atomicAdd(&S.count, (4u << 16) + set) + (4u << 16) + set;
					const uint32_t n = now & 0xFFFFu, done = now >> 16;
					if (n > kCdUniqueMax || (done >= 4 * nv && n * nv > done * (kCdUniqueMax / 32) * 2)) { *over = 1; }
				}
				stop = __any_sync(0xFFFFFFFFu, *over != 0);
			}
		}
		__syncthreads();
		found = S.over == 0;
		__syncthreads(); // S.over is read before it is cleared
		if (found) {
			clear(kCdUniqueSlots);
			if (tid == 0) { S.count = 0; }
			Q.left = kCdLooks;
			__syncthreads();
#pragma unroll
			for (uint32_t j = 0; j < kPer; ++j) {
				const uint32_t v = warp + j * kCdWarps;
				uint32_t       lo = ~0u, hi = 0u;
				Q.list = slots + v * 1024;
				Q.q = Q.n = 0;
				for (uint32_t r = 0; r < 32 && v < nv; ++r) {
					if (__any_sync(0xFFFFFFFFu, *over != 0)) { break; } // one answer for the whole warp
					T          x;
					const bool start = row(v, r, 0, &x);
					uint32_t   place, other;
					cd_hash(x, &place, &other);
					const uint32_t pos  = v * 1024 + r * 32 + lane;
					const bool     mark = start && ((marks[place >> 19] >> ((place >> 14) & 31u)) & 1u);
					const uint32_t only = __ballot_sync(0xFFFFFFFFu, start && !mark);
					if (lane == 0) { S.bits[pos >> 5] = only; }
					if (only) {
						lo = min(lo, pos - lane + __ffs(only) - 1);
						hi = pos - lane + 31 - __clz(only);
					}
					if (w0 && start && !mark) {
						sw0 += __ldg(w0 + pos);
						sw1 += __ldg(w1 + pos);
					}
					Q.push(mark, x, pos, __umulhi(place, kCdUniqueSlots), cd_tag(other), lane);
					uint32_t fresh = 0;
					if (!Q.drain(S.table, kCdUniqueSlots, vals, r == 31, lane, &fresh)) {
						if (lane == 0) { S.spent = *over = 1; }
						break;
					}
					if (lane == 0 && fresh && atomicAdd(&S.count, fresh) + fresh > kCdUniqueCap) { *over = 1; }
				}
				listed[j] = Q.n;
				if (lane == 0 && lo != ~0u) {
					S.vrange[v][0] = lo;
					S.vrange[v][1] = hi;
				}
			}
			__syncthreads();
			found = S.over == 0;
			__syncthreads(); // S.over is read before it is cleared
			if (found) { collect(kCdUniqueSlots); }
		}
	}
	for (uint32_t parts_log = 0; !found && (1u << parts_log) <= kCdMaxParts && S.spent == 0; ++parts_log) {
		reset();
		for (uint32_t part = 0; part < (1u << parts_log); ++part) {
			clear(kCdSlots);
			if (tid == 0) { S.count = S.over = 0; }
			Q.left = kCdLooks;
			__syncthreads();
#pragma unroll
			for (uint32_t j = 0; j < kPer; ++j) {
				const uint32_t u = warp + j * kCdWarps, v = u >> split, r0 = first_row(u), r1 = r0 + unit_rows;
				uint32_t       rows = 0;
				Q.list = slots + u * unit_rows * 32;
				Q.q = Q.n = 0;
				for (uint32_t r = r0; r < r1 && v < nv; ++r) {
					if (__any_sync(0xFFFFFFFFu, *over != 0)) { break; } // one answer for the whole warp
					T        x;
					bool     need = row(v, r, r0, &x);
					uint32_t place, other;
					cd_hash(x, &place, &other);
					need = need && cd_part(other, parts_log) == part;
					const uint32_t pos = v * 1024 + r * 32 + lane, s = __umulhi(place, kCdSlots), tag = cd_tag(other);
					uint32_t       fresh = 0;
					bool           looked = true;
					if (Q.q == 0 && __all_sync(0xFFFFFFFFu, need)) { // a full warp as it is
						fresh = Q.look(S.table, kCdSlots, vals, true, x, pos, s, tag, lane);
					} else {
						Q.push(need, x, pos, s, tag, lane);
						looked = Q.q >= 32;
					}
					if (!Q.drain(S.table, kCdSlots, vals, r + 1 == r1, lane, &fresh)) {
						if (lane == 0) { S.spent = *over = 1; }
						break;
					}
					++rows;
					if (lane == 0 && (looked || r + 1 == r1)) {
						// room left, and room for the chunk if the keys go on coming at this rate?
						const uint32_t now = atomicAdd(&S.count, (rows << 16) + fresh) + (rows << 16) + fresh;
						const uint32_t n = now & 0xFFFFu, done = now >> 16;
						if (n > kCdCap || (done >= 4 * nv && n * nv > done * (kCdCap / 32))) { *over = 1; }
					}
					if (looked) { rows = 0; }
				}
				listed[j] = Q.n;
			}
			__syncthreads();
			const bool full = S.over != 0;
			__syncthreads(); // S.over is read before it is cleared
			if (full) { break; }
			collect(kCdSlots);
			found = part + 1 == (1u << parts_log);
		}
	}
	if (!found) {
		reset();
		__syncthreads();
		cd_sort<T>(vals, nv, slots, w0, w1, S);
	}
	if (w0) {
		sw0 = warp_sum(sw0);
		sw1 = warp_sum(sw1);
		if (lane == 0) {
			atomicAdd(reinterpret_cast<unsigned long long*>(S.dw), static_cast<unsigned long long>(sw0));
			atomicAdd(reinterpret_cast<unsigned long long*>(S.dw + 1), static_cast<unsigned long long>(sw1));
		}
	}
	// exclusive prefix of the bitmap words' popcounts: words 2 * tid, 2 * tid + 1
	static_assert(kCdWords == 2 * kCdThreads, "two bitmap words a thread");
	uint32_t*      pref = S.table;
	const uint32_t p0 = __popc(S.bits[2 * tid]), p1 = __popc(S.bits[2 * tid + 1]);
	const uint32_t inc = warp_inclusive_scan(p0 + p1, lane);
	if (lane == 31) { S.wsum[warp] = inc; }
	__syncthreads();
	if (warp == 0) {
		const uint32_t w  = S.wsum[lane];
		const uint32_t wi = warp_inclusive_scan(w, lane);
		S.wsum[lane]      = wi - w;
		if (lane == 31) { S.wsum[32] = wi; }
	}
	__syncthreads();
	pref[2 * tid]     = S.wsum[warp] + inc - p0 - p1;
	pref[2 * tid + 1] = S.wsum[warp] + inc - p1;
	__syncthreads();
	if (tid < nv) {
		auto rank = [&](uint32_t f) { return pref[f >> 5] + __popc(S.bits[f >> 5] & ((1u << (f & 31u)) - 1u)); };
		const uint32_t lo = S.vrange[tid][0], hi = S.vrange[tid][1];
		a.bw_code[i0 + tid] = lo <= hi ? bits_of(rank(hi) - rank(lo)) : 0u;
	}
	if (tid == 0) {
		a.dict_n[c] = S.wsum[32];
		if (a.dict_w) {
			a.dict_w[2ull * c]     = S.dw[0];
			a.dict_w[2ull * c + 1] = S.dw[1];
		}
	}
	__syncthreads();
}

__global__ void __launch_bounds__(kCdThreads) k_chunk_dict(ChunkDictArgs a) {
	extern __shared__ __align__(16) uint8_t smem[];
	ChunkDictSmem&                          S = *reinterpret_cast<ChunkDictSmem*>(smem);
	for (;;) {
		// chunks differ in cost by their distinct values: the next free CTA takes the next one
		if (threadIdx.x == 0) { S.chunk = atomicAdd(a.ticket, 1u); }
		__syncthreads();
		const uint32_t c = S.chunk;
		if (c >= a.n_chunks) { return; }
		const Col col = a.cols[a.items[a.chunk_items[c]].col];
		if (col.width == 64) {
			chunk_dict<64>(a, col, c, S);
		} else {
			chunk_dict<32>(a, col, c, S);
		}
	}
}

// ---------------------------------------------------------------------------------------------------------
// String columns.  The selection works on a 64-bit hash of every row (distinct rows, runs and first-occurrence
// codes come from the integer machinery run on the hashes), the row's length and its FSST-compressed length
// under the column's symbol table (the encoder's greedy longest match; a byte no symbol starts with costs an
// escape and itself, 2 bytes).  Candidates (string pool, no patches; src/cor/exp_pool.cpp:66-101):
//   0 BYTE_ARR (pool id 0)   1 DICT FFOR over an FSST dictionary (id 3)   2 FSST (id 13)
//   3 DICT_RLE with raw run codes and a raw u16 run index (id 15)
// ---------------------------------------------------------------------------------------------------------
constexpr int kStrK = FLS_SEL_STR_K;

// An FSST symbol table arranged for greedy matching by the next two bytes of a string:
//   one    bitmap of the bytes that are symbols by themselves; two: the two-byte symbols;
//   groups the longer symbols, grouped by their first two bytes (pair), longest first.  Group ids start at kStrGroup;
//          g_short is what a string takes when none of the group's symbols matches: 2, 1 or 0 (an escape).  A table
//          with more pairs than ids shares the id of another group with the same g_short: every symbol of a group
//          is compared in full, so that only costs comparisons.
constexpr uint32_t kStrGroup  = 3;
constexpr uint32_t kStrGroups = 256 - kStrGroup;
struct StrTab {
	ulonglong2 sym[256]; // the groups' symbols: value, mask of its bytes
	uint32_t one[8];
	uint16_t two[256];
	uint16_t pair[256];  // first two bytes (the first in the low byte)
	uint16_t start[258]; // symbols of group g: [start[g], start[g + 1]), g counted from 0
	uint16_t n_two, n_pair;
	uint8_t  pair_group[256];
	uint8_t  len[256];
	uint8_t  g_short[256];
};

struct StrCol {
	const uint8_t*  bytes;
	const uint64_t* offsets; // n_rows + 1
	uint64_t        n_bytes; // offsets[n_rows]
	const StrTab*   tab;
	uint32_t        tab_bytes; // the exported table's size (the FSST page's dictionary slot)
	uint64_t*       hash;      // per row
	uint32_t*       len;
	uint32_t*       clen;
};

__device__ __forceinline__ uint64_t str_mix(uint64_t h) {
	h ^= h >> 33;
	h *= 0xff51afd7ed558ccdull;
	h ^= h >> 33;
	h *= 0xc4ceb9fe1a85ec53ull;
	h ^= h >> 33;
	return h;
}

// 8 bytes of a string from byte position p (bytes past the column's last byte read as the last word's)
__device__ __forceinline__ uint64_t str_load8(const StrCol& c, uint64_t p) {
	const uint32_t* w    = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(c.bytes) & ~uintptr_t(3));
	const uint64_t  a    = (reinterpret_cast<uintptr_t>(c.bytes) & 3u) + p; // byte index from w
	const uint64_t  last = ((reinterpret_cast<uintptr_t>(c.bytes) & 3u) + (c.n_bytes ? c.n_bytes - 1 : 0)) >> 2;
	const uint64_t  q    = a >> 2;
	const uint32_t  x0 = __ldg(w + (q < last ? q : last)), x1 = __ldg(w + (q + 1 < last ? q + 1 : last)),
	               x2  = __ldg(w + (q + 2 < last ? q + 2 : last));
	const uint32_t  sh = 8u * static_cast<uint32_t>(a & 3u);
	const uint32_t  lo = sh ? __funnelshift_r(x0, x1, sh) : x0, hi = sh ? __funnelshift_r(x1, x2, sh) : x1;
	return (static_cast<uint64_t>(hi) << 32) | lo;
}

// str_load8 for a row that ends at least 12 bytes before the column's last byte
__device__ __forceinline__ uint64_t str_load8_inside(const StrCol& c, uint64_t p) {
	const uintptr_t a  = reinterpret_cast<uintptr_t>(c.bytes) + p;
	const uint32_t* w  = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3));
	const uint32_t  x0 = __ldg(w), x1 = __ldg(w + 1), x2 = __ldg(w + 2);
	const uint32_t  sh = 8u * static_cast<uint32_t>(a & 3u);
	return (static_cast<uint64_t>(__funnelshift_r(x1, x2, sh)) << 32) | __funnelshift_r(x0, x1, sh);
}

// Hash and length of each of a vector's 1024 rows, and the compressed length of every rs-th row (rs = 1: every
// row, the exact figure the wizard's sizes need; rs > 1, the learned selector's features: the other rows'
// compressed lengths are written as 0 and the vector's sum is scaled by rs).  The CTAs go through the columns one
// after the other, a warp taking units of kStrUnit rows.
//   memo     rows that another row of the column equals take its compressed length from the column's part of a table in
//            global memory, cleared for every call: an entry says where a row's bytes are, and both rows' bytes are
//            compared (nothing follows from a hash).  A first launch over every `stride`-th vector fills it -- all
//            units start at once, so that it finds nothing -- and counts the rows that it would have found; columns
//            whose rows repeat (a quarter of those) look theirs up in the second launch.  With one table for all
//            columns, those whose rows all differ would push the others' entries out;
//   match    greedy matching looks at the next two bytes in a 64 KB table in shared memory (what they start: nothing,
//            a one- or two-byte symbol, or a group of longer ones), so that only the few symbols of one group are
//            compared, where the symbols sharing a first byte were walked one after the other;
//   lanes    draw rows from the warp's list as they finish (8 at a time), four codes between two looks: rows of 1 to 20
//            codes would otherwise leave most lanes idle.
// 5.7 M rows of 6 columns (a third of the rows all different, 17 codes each): 1,677 us by rows and first-byte lists,
// 45 + 312 us so.  Bound by instructions and the latency of the rows' loads (issue slots half used, registers full).  Whole
// calls: the memo is worth 1,156 against 930 us for those (and 28 integer columns); of 4.6 M rows all different it
// would cost 709 us where 488 are needed, so the columns are told apart.
constexpr int      kStrWarps = 16;
// log2 of a vector's units: of 128 rows, and of 32, one a lane, where those would leave warps without one
constexpr uint32_t kStrPer = 3, kStrUnit = 1024 >> kStrPer, kStrSmallPer = 5;
// log2 of a column's memo entries: as many as the largest column has rows, at most 1 MB, and (down to the least) all
// columns' at most 8 MB, which is cleared in a few microseconds and stays in L2
constexpr uint32_t kStrMemoMin = 13, kStrMemoMax = 17, kStrMemoAll = 20;
// a column's vectors, on average: at least for a memo, and in the launch that fills it
constexpr uint32_t kStrMemoVecs = 32, kStrMemoFill = 8;
struct StrRowsSmem {
	// by the next two bytes: 0 escape, 1 / 2 a symbol of that length, kStrGroup + g; behind them, by a row's last byte
	uint8_t  pair[65536 + 256];
	StrTab   t;
	uint32_t off[kStrWarps][kStrUnit + 1]; // a unit's row offsets from its first row's
	uint16_t list[kStrWarps][kStrUnit];    // rows to match
};

// What the string bytes in x, `left` of them still in the row, start (an entry of pair; its first two bytes are read).
__device__ __forceinline__ uint32_t str_look(const StrRowsSmem& S, uint32_t x, uint32_t left) {
	return S.pair[left == 1 ? 65536u + (x & 0xFFu) : x & 0xFFFFu];
}

// The next code's bytes and (*cost grows by) its compressed size: 1, or 2 for an escaped byte.  x: the next 8 bytes.
__device__ __forceinline__ uint32_t str_next_code(const StrRowsSmem& S, uint64_t x, uint32_t left, uint32_t* cost) {
	uint32_t what = str_look(S, static_cast<uint32_t>(x), left);
	if (what >= kStrGroup) {
		const uint32_t g = what - kStrGroup;
		for (uint32_t k = S.t.start[g]; k < S.t.start[g + 1]; ++k) {
			const ulonglong2 m = S.t.sym[k];
			if ((x & m.y) == m.x && S.t.len[k] <= left) {
				*cost += 1;
				return S.t.len[k];
			}
		}
		what = S.t.g_short[g];
	}
	*cost += what ? 1u : 2u;
	return what == 2 ? 2u : 1u;
}

// the string bytes in x, `left` of them (at least one) still in the row, zero past them
__device__ __forceinline__ uint64_t str_row_bytes(uint64_t x, uint64_t left) {
	return left >= 8 ? x : (x & ((1ull << (8 * left)) - 1));
}
__device__ __forceinline__ uint64_t str_hash_step(uint64_t h, uint64_t x) { return str_mix(h ^ x) + 0x9E3779B97F4A7C15ull; }
constexpr uint64_t kStrHashSeed = 0x243F6A8885A308D3ull;
// The hash of a row of m bytes whose words gave h, the last one x.  A row that ends in a zero byte has its length mixed in
// once more: the length that h starts from can cancel against a first byte, and a shorter row's words are the same then
// ("a" and "b\0" shared a hash).  (Another hash for all rows would change their columns' statistics.)
__device__ __forceinline__ uint64_t str_hash_end(uint64_t h, uint64_t x, uint64_t m) {
	return m && (x >> (8 * ((m - 1) & 7u)) & 0xFFu) == 0 ? str_mix(h + m * 0x9E3779B97F4A7C15ull) : h;
}

// A unit whose offsets do not fit 31 bits from its first one (rows of gigabytes, or corrupt offsets), row by row.
__device__ __noinline__ void str_unit_wide(const StrRowsSmem& S, const StrCol& c, uint64_t r0, uint32_t unit, uint32_t rs,
                                           uint32_t lane, uint64_t* sl, uint64_t* sc) {
	for (uint32_t j = lane; j < unit; j += 32) {
		const uint64_t r = r0 + j, b = __ldg(c.offsets + r), e = __ldg(c.offsets + r + 1), m = e >= b ? e - b : 0;
		uint64_t       h = kStrHashSeed ^ m, x = 0;
		for (uint64_t p = 0; p < m; p += 8) {
			x = str_row_bytes(str_load8(c, b + p), m - p);
			h = str_hash_step(h, x);
		}
		h = str_hash_end(h, x, m);
		uint32_t cl = 0;
		if ((r & 1023u) % rs == 0) {
			for (uint64_t p = 0; p < m;) {
				const uint64_t left = m - p;
				p += str_next_code(S, str_load8(c, b + p), left < 8 ? static_cast<uint32_t>(left) : 8u, &cl);
			}
		}
		c.hash[r] = h;
		c.len[r]  = static_cast<uint32_t>(m);
		c.clen[r] = cl;
		*sl += m;
		*sc += cl;
	}
}

// A memo entry: a row's compressed length + 1 (0: no entry), its length, where it starts in the column's bytes, and 8 bits
// of its hash, so that few other rows' bytes are looked at.  Rows of more bytes, or further in, have none.  The place is
// a pair of entries, told by the low bits - 1 bits of the hash: strings that share a place push each other out for good,
// and a warp waits for its few rows that miss: 4,096 strings in 64 Ki single entries, of which 6 % share one, 83 + 667 us
// for 7.4 M rows of 12 columns, 81 + 541 us so.
constexpr uint32_t kStrMemoClenBits = 11, kStrMemoLenBits = 11, kStrMemoAtBits = 34;
constexpr uint32_t kStrMemoClen = (1u << kStrMemoClenBits) - 2, kStrMemoLen = (1u << kStrMemoLenBits) - 1; // at most
constexpr uint32_t kStrMemoAtPos = kStrMemoClenBits + kStrMemoLenBits, kStrMemoTagPos = kStrMemoAtPos + kStrMemoAtBits;
constexpr uint64_t kStrMemoAtEnd = 1ull << kStrMemoAtBits;
static_assert(kStrMemoTagPos == 56, "8 bits of the hash");

// what an entry of a row of hash h and length m has beside the row's place and compressed length
__device__ __forceinline__ uint64_t str_memo_key(uint64_t h, uint32_t m) {
	return (h & ~((1ull << kStrMemoTagPos) - 1)) | (static_cast<uint64_t>(m) << kStrMemoClenBits);
}
constexpr uint64_t kStrMemoKey = ~((1ull << kStrMemoTagPos) - 1) | (((1ull << kStrMemoLenBits) - 1) << kStrMemoClenBits);

struct StrRowsArgs {
	const StrCol* cols;
	const Item*   items; // by column
	uint64_t      n_items;
	uint64_t *    vlen, *vclen; // optional: sums of every item, zero before the first launch
	uint64_t*     memo;   // 1 << memo_bits entries for every column; null: no memo
	uint32_t*     repeats; // with it, for every column: rows of the launch that fills the memo, and how many another equals
	uint32_t      memo_bits;
	uint32_t      rs;
	uint32_t      stride; // every stride-th item in the first launch, the others in the next one
	uint32_t      first;
	uint32_t      per; // log2 of a vector's units
};

__global__ void __launch_bounds__(kStrWarps * 32, 2) k_str_rows(const StrRowsArgs a) {
	extern __shared__ __align__(16) uint8_t smem[];
	StrRowsSmem&       S  = *reinterpret_cast<StrRowsSmem*>(smem);
	constexpr uint32_t nt = kStrWarps * 32;
	const uint32_t     per = a.per, unit = 1024u >> per; // rows of a unit
	const uint32_t     tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, rs = a.rs;
	// this launch's items: i * stride (first), or the others in order; number i of them
	const uint64_t n_first = (a.n_items + a.stride - 1) / a.stride;
	const uint64_t n       = a.first ? n_first : a.n_items - n_first;
	auto           item    = [&](uint64_t i) { return a.first ? i * a.stride : a.stride == 1 ? i : i + i / (a.stride - 1) + 1; };
	const uint64_t gw = static_cast<uint64_t>(blockIdx.x) * kStrWarps, nw = static_cast<uint64_t>(gridDim.x) * kStrWarps;
	// units are dealt to the warps round robin, over the columns' borders; a CTA goes from the column of its first unit to
	// that of its first unit past it
	for (uint64_t u0 = 0;;) {
		const uint64_t turn = u0 % nw; // whose unit u0 is
		u0 += turn < gw ? gw - turn : turn < gw + kStrWarps ? 0 : nw - turn + gw;
		if (u0 >= n << per) { break; }
		const uint32_t col = a.items[item(u0 >> per)].col;
		// the column's end among the items, the first of another column: by doubling steps, then halving
		uint64_t lo = (u0 >> per) + 1, hi = lo;
		for (uint64_t d = 1; hi < n && a.items[item(hi)].col == col; d *= 2) {
			lo = hi + 1;
			hi = lo + d < n ? lo + d : n;
		}
		while (lo < hi) {
			const uint64_t mid = (lo + hi) / 2;
			if (a.items[item(mid)].col == col) {
				lo = mid + 1;
			} else {
				hi = mid;
			}
		}
		const uint64_t    u1   = lo << per;
		const StrCol      c    = a.cols[col];
		ulonglong2* const memo = reinterpret_cast<ulonglong2*>(a.memo + (static_cast<uint64_t>(col) << a.memo_bits));
		const uint32_t    pairs = (1u << (a.memo_bits - 1)) - 1;
		// rows are looked up only where the first launch found that they repeat
		const bool look = a.memo && !a.first && a.repeats[2 * col + 1] >= a.repeats[2 * col] / 4;
		uint32_t   rows = 0, repeats = 0;
		__syncthreads(); // the previous column's table is read to the end
		for (uint32_t k = tid; k < sizeof(StrTab) / 4; k += nt) {
			reinterpret_cast<uint32_t*>(&S.t)[k] = __ldg(reinterpret_cast<const uint32_t*>(c.tab) + k);
		}
		__syncthreads();
		for (uint32_t k = tid; k < 65536 / 4; k += nt) { // bytes 4k .. 4k + 3: the low byte of the pair
			const uint32_t m                       = S.t.one[(k & 63u) >> 3] >> (4 * (k & 7u));
			reinterpret_cast<uint32_t*>(S.pair)[k] = (m & 1u) | ((m & 2u) << 7) | ((m & 4u) << 14) | ((m & 8u) << 21);
			if (k < 64) { reinterpret_cast<uint32_t*>(S.pair)[65536 / 4 + k] = reinterpret_cast<uint32_t*>(S.pair)[k]; }
		}
		__syncthreads();
		for (uint32_t k = tid; k < S.t.n_two; k += nt) { S.pair[S.t.two[k]] = 2; }
		__syncthreads();
		for (uint32_t k = tid; k < S.t.n_pair; k += nt) { S.pair[S.t.pair[k]] = static_cast<uint8_t>(kStrGroup + S.t.pair_group[k]); }
		__syncthreads();
		for (uint64_t u = u0 + (gw + warp + nw - u0 % nw) % nw; u < u1; u += nw) {
			const uint64_t it = item(u >> per);
			uint64_t       sl = 0, sc = 0;
			{
				const uint64_t r0   = static_cast<uint64_t>(a.items[it].vec) * 1024 + (u & ((1u << per) - 1u)) * unit;
				const uint64_t o0   = __ldg(c.offsets + r0);
				uint32_t*      off  = S.off[warp];
				uint16_t*      list = S.list[warp];
				bool           wide = false;
				__syncwarp(); // the warp's previous unit is read to the end
				for (uint32_t j = lane; j <= unit; j += 32) {
					const uint64_t o = __ldg(c.offsets + r0 + j) - o0;
					wide |= o >= (1ull << 31);
					off[j] = static_cast<uint32_t>(o);
				}
				__syncwarp();
				if (__any_sync(0xFFFFFFFFu, wide)) {
					str_unit_wide(S, c, r0, unit, rs, lane, &sl, &sc);
				} else {
					// offsets from o0 below this lie at least 12 bytes before the column's end
					const uint64_t room  = c.n_bytes > o0 ? c.n_bytes - o0 : 0;
					const uint32_t limit = room < 12 ? 0u : room < (1u << 31) ? static_cast<uint32_t>(room) - 11 : 1u << 31;
					auto load8 = [&](uint32_t p, bool inside) { return inside ? str_load8_inside(c, o0 + p) : str_load8(c, o0 + p); };
					uint32_t todo = 0;
					uint32_t row = 0, ask = 0; // the look into the memo of the row before
					uint64_t key = 0;
					ulonglong2 seen = make_ulonglong2(0, 0);
					for (uint32_t j = lane; j < unit + 32; j += 32) {
						uint32_t row_next = j, ask_next = 0;
						uint64_t key_next = 0;
						ulonglong2 seen_next = make_ulonglong2(0, 0);
						if (j < unit) {
							const uint32_t b = off[j], e = off[j + 1], m = e >= b ? e - b : 0;
							const bool     inside = e < limit;
							uint64_t       h = kStrHashSeed ^ m;
							uint64_t       x = 0;
							for (uint32_t p = 0; p < m; p += 8) {
								x = str_row_bytes(load8(b + p, inside), m - p);
								h = str_hash_step(h, x);
							}
							h = str_hash_end(h, x, m);
							const uint64_t r = r0 + j;
							c.hash[r]        = h;
							c.len[r]         = m;
							sl += m;
							if ((r & 1023u) % rs == 0) {
								ask_next = look && m <= kStrMemoLen && e <= room ? 1u : 2u; // 2: not looked up, to be matched
								if (ask_next == 1) {
									key_next  = str_memo_key(h, m);
									seen_next = __ldcg(memo + (static_cast<uint32_t>(h) & pairs));
								}
							} else {
								c.clen[r] = 0;
							}
						}
						const uint64_t found = (seen.x & kStrMemoKey) == key ? seen.x : seen.y;
						bool           hit   = ask == 1 && found != 0 && (found & kStrMemoKey) == key;
						if (hit) { // the same bytes?
							const uint64_t q = (found >> kStrMemoAtPos) & (kStrMemoAtEnd - 1);
							const uint32_t b = off[row], m = static_cast<uint32_t>(key >> kStrMemoClenBits) & kStrMemoLen;
							const bool     inside = b + m < limit && q + m + 12 <= c.n_bytes;
							if (inside) { // two words a step: their loads are in flight together
								for (uint32_t p = 0; p < m && hit; p += 16) {
									const uint32_t p1 = p + 8 < m ? p + 8 : p;
									const uint64_t x0 = str_load8_inside(c, o0 + b + p), y0 = str_load8_inside(c, q + p);
									const uint64_t x1 = str_load8_inside(c, o0 + b + p1), y1 = str_load8_inside(c, q + p1);
									hit = (str_row_bytes(x0 ^ y0, m - p) | str_row_bytes(x1 ^ y1, m - p1)) == 0;
								}
							} else {
								for (uint32_t p = 0; p < m && hit; p += 8) {
									hit = str_row_bytes(str_load8(c, o0 + b + p) ^ str_load8(c, q + p), m - p) == 0;
								}
							}
						}
						if (hit) {
							const uint32_t cl = static_cast<uint32_t>(found & ((1u << kStrMemoClenBits) - 1)) - 1;
							c.clen[r0 + row]  = cl;
							sc += cl;
						}
						const bool     miss = ask && !hit;
						const uint32_t m    = __ballot_sync(0xFFFFFFFFu, miss);
						if (miss) { list[todo + __popc(m & ((1u << lane) - 1u))] = static_cast<uint16_t>(row); }
						todo += __popc(m);
						row = row_next, ask = ask_next, key = key_next, seen = seen_next;
					}
					__syncwarp();
					uint32_t next = 0, j = 0, p = 0, left = 0, cl = 0;
					bool     have = false, inside = false;
					for (;;) {
						const uint32_t idle = __ballot_sync(0xFFFFFFFFu, !have);
						if (next < todo && (__popc(idle) >= 8 || idle == 0xFFFFFFFFu)) {
							if (!have) {
								const uint32_t k = next + __popc(idle & ((1u << lane) - 1u));
								have             = k < todo;
								if (have) {
									j                = list[k];
									p                = off[j];
									const uint32_t e = off[j + 1];
									left             = e >= p ? e - p : 0;
									inside           = e < limit;
									cl               = 0;
								}
							}
							next += __popc(idle);
						} else if (idle == 0xFFFFFFFFu) {
							break;
						}
						// four codes between two looks at who is idle, from one load of eight bytes while they are of one
						// and two bytes: straight through, as no more is asked of them than the table's entry
						uint64_t x   = left ? load8(p, inside) : 0;
						uint32_t got = 8;
#pragma unroll
						for (uint32_t k = 0; k < 4; ++k) {
							const uint32_t what = str_look(S, static_cast<uint32_t>(x), left);
							const bool     on   = left != 0;
							uint32_t       step = on ? 1u + (what >> 1) : 0u;
							if (on && what >= kStrGroup) {
								if (got < 8) {
									x   = load8(p, inside);
									got = 8;
								}
								step = str_next_code(S, x, left, &cl);
								if (got < step + 2 * (3 - k)) { // the codes to come may need two bytes each
									x   = left > step ? load8(p + step, inside) : 0;
									got = 8 + step;
								} else {
									x = step < 8 ? x >> (8 * step) : 0;
								}
							} else {
								cl += on ? 1u + (what == 0) : 0u;
								x >>= 8 * step;
							}
							p += step;
							left -= step;
							got -= step;
						}
						if (have && left == 0) {
							c.clen[r0 + j] = cl;
							sc += cl;
							have = false;
						}
					}
					__syncwarp();
					for (uint32_t k = a.memo && (a.first || look) ? lane : todo; k < todo; k += 32) { // what was matched, for the rows to come
						const uint32_t i = list[k];
						const uint64_t r = r0 + i;
						const uint32_t l = c.clen[r];
						const uint32_t b = off[i], e = off[i + 1], n = e >= b ? e - b : 0;
						++rows;
						if (n <= kStrMemoLen && l <= kStrMemoClen && e <= room && o0 + b < kStrMemoAtEnd) {
							const uint64_t   h = c.hash[r], key = str_memo_key(h, n);
							ulonglong2*      at = memo + (static_cast<uint32_t>(h) & pairs);
							const ulonglong2 had = __ldcg(at);
							if ((had.x != 0 && (had.x & kStrMemoKey) == key) || (had.y != 0 && (had.y & kStrMemoKey) == key)) {
								++repeats;
							} else { // into the entry of the pair that is free, or over one of the two
								const uint32_t slot = had.x == 0 ? 0u : had.y == 0 ? 1u : static_cast<uint32_t>(h >> 57) & 1u;
								__stcg(reinterpret_cast<uint64_t*>(at) + slot, key | ((o0 + b) << kStrMemoAtPos) | (l + 1));
							}
						}
					}
				}
			}
			sl = warp_sum(sl);
			sc = warp_sum(sc);
			if (lane == 0) {
				if (a.vlen) { atomicAdd(reinterpret_cast<unsigned long long*>(a.vlen + it), static_cast<unsigned long long>(sl)); }
				if (a.vclen) { atomicAdd(reinterpret_cast<unsigned long long*>(a.vclen + it), static_cast<unsigned long long>(sc * rs)); }
			}
		}
		if (a.memo && a.first) {
			rows    = warp_sum(rows);
			repeats = warp_sum(repeats);
			if (lane == 0 && rows) {
				atomicAdd(a.repeats + 2 * col, rows);
				atomicAdd(a.repeats + 2 * col + 1, repeats);
			}
		}
		u0 = u1;
	}
}

// k_str_rows over n_items vectors, two CTAs a SM; with the memo in two launches, the first over as many vectors as give
// every warp a unit of 32 rows, or more.
cudaError_t launch_str_rows(const StrCol* cols, const Item* items, uint64_t n_items, uint64_t* vlen, uint64_t* vclen,
                            uint32_t rs, uint64_t* memo, uint32_t memo_bits, uint64_t n_cols, cudaStream_t s) {
	Device* d = current_device();
	if (!d) { return cudaErrorInvalidDevice; }
	static SmemLimit limit;
	cudaError_t      e = limit.need(reinterpret_cast<const void*>(k_str_rows), sizeof(StrRowsSmem));
	if (e != cudaSuccess) { return e; }
	if (vlen) { e = cudaMemsetAsync(vlen, 0, n_items * 8, s); }
	if (e == cudaSuccess && vclen) { e = cudaMemsetAsync(vclen, 0, n_items * 8, s); }
	const uint64_t most = static_cast<uint64_t>(d->sm_count) * 2, warps = most * kStrWarps; // CTAs, warps
	uint64_t       step = std::max<uint64_t>(1, ((n_items << kStrSmallPer) + warps - 1) / warps);
	// the memo pays for columns of some vectors, when every row is matched; the first launch takes at least some of each
	const uint64_t vecs = n_items / n_cols;
	const bool     keep = memo && rs == 1 && step > 1 && vecs >= kStrMemoVecs;
	step                = keep ? std::min<uint64_t>(step, vecs / kStrMemoFill) : 1;
	if (e == cudaSuccess && keep) { e = cudaMemsetAsync(memo, 0, (n_cols << memo_bits) * 8 + n_cols * 8, s); }
	if (e != cudaSuccess) { return e; }
	StrRowsArgs a {cols, items, n_items, vlen, vclen, keep ? memo : nullptr, reinterpret_cast<uint32_t*>(memo + (n_cols << memo_bits)),
	               memo_bits, rs, static_cast<uint32_t>(step), 1, 0};
	for (const uint32_t first : {1u, 0u}) {
		const uint64_t n_first = (n_items + step - 1) / step, n = first ? n_first : n_items - n_first;
		a.first = first;
		a.per   = (n << kStrPer) < warps ? kStrSmallPer : kStrPer;
		const uint64_t ctas = std::min(((n << a.per) + kStrWarps - 1) / kStrWarps, most);
		if (ctas) {
			k_str_rows<<<static_cast<unsigned>(ctas), kStrWarps * 32, sizeof(StrRowsSmem), s>>>(a);
			++launch_counter();
		}
	}
	return cudaGetLastError();
}

// The features of a string vector: those of its row hashes (distinct rows, runs, multiplicities), with the
// slots that mean nothing for hashes replaced by the rows' lengths and compressibility.
__global__ void __launch_bounds__(kWarps * 32) k_str_features(const StrCol* cols, const Item* items, uint64_t n_items,
                                                              float* feat, uint32_t rs) {
	const uint32_t lane = threadIdx.x & 31u;
	for (uint64_t it = blockIdx.x * static_cast<uint64_t>(kWarps) + (threadIdx.x >> 5); it < n_items;
	     it += static_cast<uint64_t>(gridDim.x) * kWarps) {
		const Item   m  = items[it];
		const StrCol c  = cols[m.col];
		float        sl = 0, sc = 0, sq = 0, mx = 0, mn = 1e30f;
		for (uint32_t i = 0; i < 32; ++i) {
			const uint64_t r = static_cast<uint64_t>(m.vec) * 1024 + lane + 32 * i;
			const float    l = static_cast<float>(c.len[r]);
			sl += l;
			sq += l * l;
			sc += static_cast<float>(c.clen[r]);
			mx = fmaxf(mx, l);
			mn = fminf(mn, l);
		}
		sl = warp_sum(sl);
		sq = warp_sum(sq);
		sc = warp_sum(sc) * static_cast<float>(rs); // every rs-th row's compressed length, scaled
		mx = warp_max(mx);
		mn = warp_min(mn);
		const float mean = sl / 1024.0f;
		const float var  = fmaxf(sq / 1024.0f - mean * mean, 0.0f);
		float*      f    = feat + it * NF;
		if (lane == 0) {
			f[0]  = mean / 64.0f;
			f[1]  = sl > 0 ? sc / sl : 1.0f;
			f[9]  = sqrtf(var) / 64.0f;
			f[14] = mx / 256.0f;
			f[15] = mn / 64.0f;
			f[16] = 1.0f; // a string column
			f[22] = log2f(mean + 1.0f) / 8.0f;
			f[29] = sc / (1024.0f * 64.0f);
		}
	}
}

struct StrSizeArgs {
	const uint32_t* chunk_col;
	const uint32_t* chunk_items; // item range of every chunk (n_chunks + 1)
	const uint32_t* parts;       // per item: runs of the row hashes in bits 19..
	const uint32_t* bw_code;     // per item
	const uint64_t* vlen;        // per item
	const uint64_t* vclen;       // per item
	const uint32_t* dict_n;      // per chunk
	const uint64_t* dict_w;      // per chunk: the dictionary's raw and compressed bytes
	const StrCol*   cols;
	uint32_t        n_chunks;
	uint64_t*       sizes; // n_chunks x FLS_SEL_K (the string candidates in 0..3, the rest ~0)
	uint8_t*        best;
};

// Exact page bytes of the string candidates (page = header, buffer offsets, per-vector entry points, buffers;
// the dictionary page of DICT and DICT_RLE = dict_hdr_t, the FSST_MAXHEADER table slot, u32 compressed lengths
// and the compressed entries, src/cor/lyt/dic/dic.cpp:88-111; the FSST column's = dict_hdr_t and the table).
__global__ void k_str_sizes(StrSizeArgs a) {
	const uint32_t lane = threadIdx.x & 31u;
	for (uint32_t c = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); c < a.n_chunks; c += gridDim.x * (blockDim.x / 32)) {
		const uint32_t i0 = a.chunk_items[c], i1 = a.chunk_items[c + 1];
		uint64_t       L = 0, C = 0, R = 0, B = 0;
		for (uint32_t i = i0 + lane; i < i1; i += 32) {
			L += a.vlen[i];
			C += a.vclen[i];
			R += a.parts[i] >> 19;
			B += a.bw_code[i];
		}
		L = warp_sum(L), C = warp_sum(C), R = warp_sum(R), B = warp_sum(B);
		if (lane == 0) {
			const uint64_t nv    = i1 - i0;
			auto           frame = [&](uint64_t arr) { return 8 + 4 * arr + 4 * arr * (nv ? nv - 1 : 0); };
			const uint64_t dpage = 8 + 2066 + 4ull * a.dict_n[c] + a.dict_w[2ull * c + 1];
			uint64_t       z[FLS_SEL_K];
			z[0] = frame(2) + L + 4096 * nv;
			z[1] = frame(3) + nv + 4 * nv + 128 * B + dpage;
			z[2] = frame(2) + C + 4096 * nv + 8 + a.cols[a.chunk_col[c]].tab_bytes;
			z[3] = frame(2) + 4 * R + 2048 * nv + dpage;
			for (int k = kStrK; k < FLS_SEL_K; ++k) { z[k] = ~0ull; }
			uint32_t b = 0;
			for (int k = 0; k < FLS_SEL_K; ++k) {
				a.sizes[static_cast<uint64_t>(c) * FLS_SEL_K + k] = z[k];
				if (z[k] < z[b]) { b = k; }
			}
			a.best[c] = static_cast<uint8_t>(b);
		}
	}
}

// Exact sizes of every candidate of every chunk, and the smallest (lowest index on ties).
struct SizeArgs {
	const Col*      cols;
	const uint32_t* chunk_col;
	const uint32_t* chunk_items; // item range of every chunk (n_chunks + 1)
	const uint32_t* parts;       // per item
	const uint32_t* bw_code;     // per item
	const uint32_t* dict_n;      // per chunk
	uint32_t        n_chunks;
	uint64_t*       sizes;
	uint8_t*        best;
};

__global__ void k_chunk_sizes(SizeArgs a) {
	const uint32_t lane = threadIdx.x & 31u;
	for (uint32_t c = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); c < a.n_chunks; c += gridDim.x * (blockDim.x / 32)) {
		const uint32_t i0 = a.chunk_items[c], i1 = a.chunk_items[c + 1];
		uint64_t       sf = 0, sd = 0, si = 0, sr = 0, sc = 0;
		for (uint32_t i = i0 + lane; i < i1; i += 32) {
			const uint32_t p = a.parts[i];
			sf += p & 127u;
			sd += (p >> 7) & 127u;
			si += (p >> 14) & 31u;
			sr += p >> 19;
			sc += a.bw_code[i];
		}
		sf = warp_sum(sf), sd = warp_sum(sd), si = warp_sum(si), sr = warp_sum(sr), sc = warp_sum(sc);
		if (lane == 0) {
			const uint64_t nv = i1 - i0, sz = a.cols[a.chunk_col[c]].width / 8;
			const uint64_t dp = 8 + 12 + static_cast<uint64_t>(a.dict_n[c]) * sz;
			uint64_t       s[K];
			s[0] = 8 + 4 * nv + 1024 * sz * nv;
			s[1] = 8 + 12 * nv + nv + sz * nv + 128 * sf;
			s[2] = 8 + 20 * nv + sz * sr + 128 * nv + nv + 2 * nv + 128 * si;
			s[3] = 8 + 16 * nv + 128 * nv + nv + sz * nv + 128 * sd;
			s[4] = dp + 8 + 12 * nv + nv + 4 * nv + 128 * sc;
			s[5] = dp + 8 + 20 * nv + 4 * sr + 128 * nv + nv + 2 * nv + 128 * si;
			uint32_t b = 0;
			for (int k = 0; k < K; ++k) {
				a.sizes[static_cast<uint64_t>(c) * K + k] = s[k];
				if (s[k] < s[b]) { b = k; }
			}
			a.best[c] = static_cast<uint8_t>(b);
		}
	}
}

// Per-chunk vote of the learned selector over its sampled rows: mean log-probability, argmax, mean top
// probability as the confidence.
__global__ void k_vote(const float* prob, const uint32_t* chunk_rows, uint32_t n_chunks, uint8_t* choice, float* conf,
                       int k_use) {
	const uint32_t lane = threadIdx.x & 31u;
	for (uint32_t c = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); c < n_chunks; c += gridDim.x * (blockDim.x / 32)) {
		const uint32_t r0 = chunk_rows[c], r1 = chunk_rows[c + 1];
		float          lp[K] = {}, pp[K] = {};
		for (uint32_t r = r0 + lane; r < r1; r += 32) {
#pragma unroll
			for (int k = 0; k < K; ++k) {
				const float p = prob[static_cast<uint64_t>(r) * K + k];
				lp[k] += logf(fmaxf(p, 1e-30f));
				pp[k] += p;
			}
		}
		uint32_t b = 0;
#pragma unroll
		for (int k = 0; k < K; ++k) {
			lp[k] = warp_sum(lp[k]);
			pp[k] = warp_sum(pp[k]);
			if (k < k_use && lp[k] > lp[b]) { b = k; }
		}
		if (lane == 0) {
			choice[c] = static_cast<uint8_t>(b);
			if (conf) { conf[c] = r1 > r0 ? pp[b] / static_cast<float>(r1 - r0) : 0.0f; }
		}
	}
}

// ---------------------------------------------------------------------------------------------------------
// MLP kernels (float32)
// ---------------------------------------------------------------------------------------------------------
enum : int { EPI_NONE = 0, EPI_BIAS = 1, EPI_RELU = 2, EPI_MASK = 4 };

// C[M x N] = op(A)[M x Kd] * op(B)[Kd x N] with op = transpose when ta / tb; epilogue: + bias[n], ReLU, or
// zero where mask[m, n] <= 0 (the ReLU derivative).  64 x 64 tiles, 16-deep, 4 x 4 outputs per thread.
__global__ void __launch_bounds__(256) k_gemm(int M, int N, int Kd, const float* __restrict__ A, int lda, int ta,
                                              const float* __restrict__ B, int ldb, int tb, float* __restrict__ C,
                                              int ldc, const float* __restrict__ bias, const float* __restrict__ mask,
                                              int epi) {
	__shared__ float As[16][64 + 4];
	__shared__ float Bs[16][64 + 4];
	const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
	const int m0 = blockIdx.y * 64, n0 = blockIdx.x * 64;
	float     acc[4][4] = {};
	for (int k0 = 0; k0 < Kd; k0 += 16) {
		// consecutive threads walk the operand's contiguous dimension
		for (int e = threadIdx.x; e < 16 * 64; e += 256) {
			const int kk = ta ? e / 64 : e % 16, mm = ta ? e % 64 : e / 16;
			const int m = m0 + mm, k = k0 + kk;
			As[kk][mm]  = (m < M && k < Kd) ? (ta ? A[static_cast<int64_t>(k) * lda + m] : A[static_cast<int64_t>(m) * lda + k]) : 0.0f;
		}
		for (int e = threadIdx.x; e < 16 * 64; e += 256) {
			const int kk = tb ? e % 16 : e / 64, nn = tb ? e / 16 : e % 64;
			const int n = n0 + nn, k = k0 + kk;
			Bs[kk][nn]  = (n < N && k < Kd) ? (tb ? B[static_cast<int64_t>(n) * ldb + k] : B[static_cast<int64_t>(k) * ldb + n]) : 0.0f;
		}
		__syncthreads();
#pragma unroll
		for (int kk = 0; kk < 16; ++kk) {
			float a[4], b[4];
#pragma unroll
			for (int i = 0; i < 4; ++i) {
				a[i] = As[kk][ty + 16 * i];
				b[i] = Bs[kk][tx + 16 * i];
			}
#pragma unroll
			for (int i = 0; i < 4; ++i) {
#pragma unroll
				for (int j = 0; j < 4; ++j) { acc[i][j] = fmaf(a[i], b[j], acc[i][j]); }
			}
		}
		__syncthreads();
	}
#pragma unroll
	for (int i = 0; i < 4; ++i) {
		const int m = m0 + ty + 16 * i;
		if (m >= M) { continue; }
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			const int n = n0 + tx + 16 * j;
			if (n >= N) { continue; }
			float v = acc[i][j];
			if (epi & EPI_BIAS) { v += bias[n]; }
			if (epi & EPI_RELU) { v = fmaxf(v, 0.0f); }
			if ((epi & EPI_MASK) && !(mask[static_cast<int64_t>(m) * ldc + n] > 0.0f)) { v = 0.0f; }
			C[static_cast<int64_t>(m) * ldc + n] = v;
		}
	}
}

// Class probabilities of n feature rows: the whole forward pass of the MLP, 32 rows a CTA, every layer's activations
// and all weights in shared memory.  Each sum runs over k in order, as k_gemm's do, and the softmax is k_softmax's, so
// the results are theirs bit for bit.  The three products, the softmax and their round trips through global memory
// were four launches of 3 to 30 us (each of 116 CTAs of 64-row tiles, a quarter of the SMs idle); this one takes 23 us from cold
// caches for 3,660 rows.
constexpr uint32_t kMlpRows = 32;
struct MlpSmem {
	float w2[H][H], w1[NF][H], w3[H][K + 2];
	float b1[H], b2[H], b3[K + 2];
	float x[kMlpRows][NF + 1], h1[kMlpRows][H + 4], h2[kMlpRows][H + 4];
};

// out[rows][H] = relu(in[rows][KD] * w + b): thread (tx, ty) takes columns 4 tx .. + 3 of rows ty, ty + 8, + 16, + 24
template <int KD, int LDA>
__device__ __forceinline__ void mlp_layer(const float (*in)[LDA], const float (*w)[H], const float* b, float (*out)[H + 4],
                                          uint32_t tx, uint32_t ty) {
	float acc[4][4] = {};
#pragma unroll 8
	for (int k = 0; k < KD; ++k) {
		const float4 wv = *reinterpret_cast<const float4*>(&w[k][4 * tx]);
#pragma unroll
		for (int i = 0; i < 4; ++i) {
			const float a = in[ty + 8 * i][k];
			acc[i][0] = fmaf(a, wv.x, acc[i][0]), acc[i][1] = fmaf(a, wv.y, acc[i][1]);
			acc[i][2] = fmaf(a, wv.z, acc[i][2]), acc[i][3] = fmaf(a, wv.w, acc[i][3]);
		}
	}
#pragma unroll
	for (int i = 0; i < 4; ++i) {
#pragma unroll
		for (int j = 0; j < 4; ++j) { out[ty + 8 * i][4 * tx + j] = fmaxf(acc[i][j] + b[4 * tx + j], 0.0f); }
	}
}

__global__ void __launch_bounds__(256) k_mlp(const float* __restrict__ params, const float* __restrict__ X, uint64_t n,
                                             float* __restrict__ P) {
	extern __shared__ __align__(16) uint8_t smem[];
	MlpSmem&       S   = *reinterpret_cast<MlpSmem*>(smem);
	const uint32_t tid = threadIdx.x, tx = tid % 32, ty = tid / 32;
	const float*   w1 = params;
	const float *  b1 = w1 + NF * H, *w2 = b1 + H, *b2 = w2 + H * H, *w3 = b2 + H, *b3 = w3 + H * K;
	// unrolled so that the weights' loads are in flight together: every CTA waits for them once, before its first row
#pragma unroll 8
	for (uint32_t e = tid; e < NF * H; e += 256) { S.w1[e / H][e % H] = __ldg(w1 + e); }
#pragma unroll 16
	for (uint32_t e = tid; e < H * H; e += 256) { S.w2[e / H][e % H] = __ldg(w2 + e); }
	for (uint32_t e = tid; e < H * K; e += 256) { S.w3[e / K][e % K] = __ldg(w3 + e); }
	if (tid < H) {
		S.b1[tid] = b1[tid];
		S.b2[tid] = b2[tid];
	}
	if (tid < K) { S.b3[tid] = b3[tid]; }
	for (uint64_t r0 = static_cast<uint64_t>(blockIdx.x) * kMlpRows; r0 < n; r0 += static_cast<uint64_t>(gridDim.x) * kMlpRows) {
		for (uint32_t e = tid; e < kMlpRows * NF; e += 256) {
			S.x[e / NF][e % NF] = r0 + e / NF < n ? __ldg(X + r0 * NF + e) : 0.0f;
		}
		__syncthreads();
		mlp_layer<NF, NF + 1>(S.x, S.w1, S.b1, S.h1, tx, ty);
		__syncthreads();
		mlp_layer<H, H + 4>(S.h1, S.w2, S.b2, S.h2, tx, ty);
		__syncthreads();
		if (tid < kMlpRows * K) { // a logit a thread, into x
			const uint32_t r = tid / K, c = tid % K;
			float          acc = 0.0f;
#pragma unroll 8
			for (int k = 0; k < H; ++k) { acc = fmaf(S.h2[r][k], S.w3[k][c], acc); }
			S.x[r][c] = acc + S.b3[c];
		}
		__syncthreads();
		if (tid < kMlpRows && r0 + tid < n) {
			float z[K], mx = -INFINITY, s = 0.0f;
#pragma unroll
			for (int k = 0; k < K; ++k) {
				z[k] = S.x[tid][k];
				mx   = fmaxf(mx, z[k]);
			}
#pragma unroll
			for (int k = 0; k < K; ++k) {
				z[k] = expf(z[k] - mx);
				s += z[k];
			}
#pragma unroll
			for (int k = 0; k < K; ++k) { P[(r0 + tid) * K + k] = z[k] / s; }
		}
		__syncthreads(); // x is read to the end before the next rows
	}
}

// Softmax of every labelled row of Z (n x K): dZ = (P - onehot) / n and the mean loss added to *loss (and to
// loss_hist[*step] when given).
__global__ void k_softmax(const float* Z, uint64_t n, const int32_t* y, float* dZ, float* loss,
                          float* loss_hist, const uint32_t* step) {
	float l = 0.0f;
	for (uint64_t r = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; r < n;
	     r += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
		float z[K], mx = -INFINITY, s = 0.0f;
#pragma unroll
		for (int k = 0; k < K; ++k) {
			z[k] = Z[r * K + k];
			mx   = fmaxf(mx, z[k]);
		}
#pragma unroll
		for (int k = 0; k < K; ++k) {
			z[k] = expf(z[k] - mx);
			s += z[k];
		}
#pragma unroll
		for (int k = 0; k < K; ++k) {
			z[k] /= s;
		}
		const int32_t t = y[r];
		l -= logf(fmaxf(z[t], 1e-30f));
#pragma unroll
		for (int k = 0; k < K; ++k) { dZ[r * K + k] = (z[k] - (k == t ? 1.0f : 0.0f)) / static_cast<float>(n); }
	}
	l = warp_sum(l);
	if ((threadIdx.x & 31u) == 0) {
		if (loss) { atomicAdd(loss, l / static_cast<float>(n)); }
		if (loss_hist) { atomicAdd(loss_hist + *step, l / static_cast<float>(n)); }
	}
}

// out[j] = sum over the n rows of X[r * ld + j] (bias gradients), one block per column.
__global__ void k_colsum(const float* X, uint64_t n, int cols, int ld, float* out) {
	__shared__ float ws[8];
	for (int j = blockIdx.x; j < cols; j += gridDim.x) {
		float s = 0.0f;
		for (uint64_t r = threadIdx.x; r < n; r += blockDim.x) { s += X[r * ld + j]; }
		s = warp_sum(s);
		if ((threadIdx.x & 31u) == 0) { ws[threadIdx.x >> 5] = s; }
		__syncthreads();
		if (threadIdx.x == 0) {
			float t = 0.0f;
			for (int w = 0; w < static_cast<int>(blockDim.x / 32); ++w) { t += ws[w]; }
			out[j] = t;
		}
		__syncthreads();
	}
}

// Adam (Kingma & Ba 2015, Algorithm 1); the step count comes from step_host, or from *step_dev + 1.
__global__ void k_adam(float* p, const float* g, float* m, float* v, uint64_t n, float lr, float b1, float b2,
                       float eps, uint32_t step_host, const uint32_t* step_dev) {
	const float t   = static_cast<float>(step_dev ? *step_dev + 1u : step_host);
	const float c1  = 1.0f - powf(b1, t);
	const float c2  = 1.0f - powf(b2, t);
	for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
	     i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
		const float gi = g[i];
		const float mi = b1 * m[i] + (1.0f - b1) * gi;
		const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
		m[i]           = mi;
		v[i]           = vi;
		p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
	}
}

// Rows perm[step * B ..) of X / y into the contiguous batch.
__global__ void k_gather(const float* X, const int32_t* y, const uint32_t* perm, const uint32_t* step, uint32_t B,
                         float* Xb, int32_t* yb) {
	const uint64_t base = static_cast<uint64_t>(*step) * B;
	for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < B * NF; i += gridDim.x * blockDim.x) {
		const uint32_t r = i / NF, f = i % NF;
		const uint32_t src = perm[base + r];
		Xb[i]              = X[static_cast<uint64_t>(src) * NF + f];
		if (f == 0) { yb[r] = y[src]; }
	}
}

__global__ void k_step_inc(uint32_t* step) { ++*step; }

} // namespace sel
} // namespace flsgpu

// =========================================================================================================
// Host side
// =========================================================================================================
using namespace flsgpu;
using namespace flsgpu::sel;

namespace {

struct DevMem {
	void* p = nullptr;
	~DevMem() {
		if (p) { cudaFree(p); }
	}
	bool alloc(size_t n) {
		if (p) {
			cudaFree(p);
			p = nullptr;
		}
		return cudaMalloc(&p, n ? n : 1) == cudaSuccess;
	}
	template <class T>
	T* as() const {
		return static_cast<T*>(p);
	}
};

// Device scratch that only grows: a plan's calls reuse it instead of allocating (cudaFree synchronises the device).
struct Scratch {
	DevMem m;
	size_t cap = 0;
	bool   need(size_t n) {
		if (n <= cap && m.p) { return true; }
		if (!m.alloc(n)) {
			cap = 0;
			return false;
		}
		cap = n;
		return true;
	}
	template <class T>
	T* as() const {
		return m.as<T>();
	}
};

struct ItemSet {
	DevMem   items, chunk_items, row_chunk;
	uint64_t n = 0;
};

uint64_t param_count() { return NF * H + H + H * H + H + H * K + K; }

struct ParamView {
	const float *w1, *b1, *w2, *b2, *w3, *b3;
};
ParamView view(const float* p) {
	ParamView v;
	v.w1 = p;
	v.b1 = v.w1 + NF * H;
	v.w2 = v.b1 + H;
	v.b2 = v.w2 + H * H;
	v.w3 = v.b2 + H;
	v.b3 = v.w3 + H * K;
	return v;
}

cudaError_t gemm(cudaStream_t s, int M, int N, int Kd, const float* A, int lda, int ta, const float* B, int ldb, int tb,
                 float* C, int ldc, const float* bias, const float* mask, int epi) {
	if (M <= 0 || N <= 0) { return cudaSuccess; }
	// the grid's y extent is limited: tall row-major products go in slices of rows
	constexpr int kRows = 65535 * 64;
	if (M > kRows && ta) { return cudaErrorInvalidValue; }
	for (int m0 = 0; m0 < M; m0 += kRows) {
		const int  mm = std::min(kRows, M - m0);
		const dim3 grid((N + 63) / 64, (mm + 63) / 64);
		k_gemm<<<grid, 256, 0, s>>>(mm, N, Kd, A + static_cast<int64_t>(m0) * lda, lda, ta, B, ldb, tb,
		                            C + static_cast<int64_t>(m0) * ldc, ldc, bias,
		                            mask ? mask + static_cast<int64_t>(m0) * ldc : nullptr, epi);
		++launch_counter();
	}
	return cudaGetLastError();
}

// forward: H1, H2, Z of n rows
cudaError_t forward(cudaStream_t s, const float* params, const float* X, uint64_t n, float* H1, float* H2, float* Z) {
	const ParamView p = view(params);
	cudaError_t     e;
	if ((e = gemm(s, (int)n, H, NF, X, NF, 0, p.w1, H, 0, H1, H, p.b1, nullptr, EPI_BIAS | EPI_RELU)) != cudaSuccess) { return e; }
	if ((e = gemm(s, (int)n, H, H, H1, H, 0, p.w2, H, 0, H2, H, p.b2, nullptr, EPI_BIAS | EPI_RELU)) != cudaSuccess) { return e; }
	return gemm(s, (int)n, K, H, H2, H, 0, p.w3, K, 0, Z, K, p.b3, nullptr, EPI_BIAS);
}

// class probabilities of n rows
cudaError_t probabilities(cudaStream_t s, const float* params, const float* X, uint64_t n, float* P) {
	Device* d = current_device();
	if (!d) { return cudaErrorInvalidDevice; }
	static SmemLimit  limit;
	const cudaError_t e = limit.need(reinterpret_cast<const void*>(k_mlp), sizeof(MlpSmem));
	if (e != cudaSuccess) { return e; }
	const uint64_t tiles = (n + kMlpRows - 1) / kMlpRows;
	k_mlp<<<static_cast<unsigned>(std::min<uint64_t>(tiles, d->sm_count)), 256, sizeof(MlpSmem), s>>>(params, X, n, P);
	++launch_counter();
	return cudaGetLastError();
}

// backward from dZ (n x K): gradients into G (parameter layout); dH2 / dH1: n x H scratch
cudaError_t backward(cudaStream_t s, const float* params, const float* X, uint64_t n, const float* H1, const float* H2,
                     const float* dZ, float* dH2, float* dH1, float* G) {
	const ParamView p = view(params);
	float*          gw1 = G;
	float*          gb1 = gw1 + NF * H;
	float*          gw2 = gb1 + H;
	float*          gb2 = gw2 + H * H;
	float*          gw3 = gb2 + H;
	float*          gb3 = gw3 + H * K;
	const int       nn  = static_cast<int>(n);
	cudaError_t     e;
	if ((e = gemm(s, H, K, nn, H2, H, 1, dZ, K, 0, gw3, K, nullptr, nullptr, EPI_NONE)) != cudaSuccess) { return e; }
	k_colsum<<<K, 256, 0, s>>>(dZ, n, K, K, gb3);
	++launch_counter();
	if ((e = gemm(s, nn, H, K, dZ, K, 0, p.w3, K, 1, dH2, H, nullptr, H2, EPI_MASK)) != cudaSuccess) { return e; }
	if ((e = gemm(s, H, H, nn, H1, H, 1, dH2, H, 0, gw2, H, nullptr, nullptr, EPI_NONE)) != cudaSuccess) { return e; }
	k_colsum<<<H, 256, 0, s>>>(dH2, n, H, H, gb2);
	++launch_counter();
	if ((e = gemm(s, nn, H, H, dH2, H, 0, p.w2, H, 1, dH1, H, nullptr, H1, EPI_MASK)) != cudaSuccess) { return e; }
	if ((e = gemm(s, NF, H, nn, X, NF, 1, dH1, H, 0, gw1, H, nullptr, nullptr, EPI_NONE)) != cudaSuccess) { return e; }
	k_colsum<<<H, 256, 0, s>>>(dH1, n, H, H, gb1);
	++launch_counter();
	return cudaGetLastError();
}

cudaError_t launch_features(const ItemArgs& a, float* feat, cudaStream_t s);

int grid_for(uint64_t warps_needed) {
	Device* d = current_device();
	if (!d) { return 0; }
	const uint64_t blocks = (warps_needed + kWarps - 1) / kWarps;
	const uint64_t cap    = static_cast<uint64_t>(d->sm_count) * 8;
	return static_cast<int>(std::max<uint64_t>(1, std::min(blocks, cap)));
}

cudaError_t launch_features(const ItemArgs& a, float* feat, cudaStream_t s) {
	static SmemLimit  limit;
	const cudaError_t e = limit.need(reinterpret_cast<const void*>(k_features), kFeatSmem);
	if (e != cudaSuccess) { return e; }
	k_features<<<grid_for(a.n_items), kWarps * 32, kFeatSmem, s>>>(a, feat);
	++launch_counter();
	return cudaGetLastError();
}

__global__ void k_scatter_best(const uint8_t* best, const uint32_t* chunks, uint32_t n, uint8_t* out) {
	for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) { out[chunks[i]] = best[i]; }
}

} // namespace

struct fls_sel_plan {
	DevMem                cols_d, items_d, chunk_col_d, chunk_items_d;
	std::vector<Col>      cols;
	std::vector<Item>     items; // every vector, plan order
	std::vector<uint32_t> chunk_col, chunk_items;
	std::vector<uint64_t> chunk_first;
	uint64_t              n_chunks = 0;
	uint32_t              chunk_vectors = 64;
	// wizard scratch (gtab: the chunk dictionary's slot scratch, one region per CTA; the subset lists of a
	// wizard run over some chunks) and the learned selector's; all grow-only
	Scratch bw_code, parts, info, dict_n, gtab, sub_lists, sub_sizes, sub_best, vlen, vclen,
	    dict_w, l_work, l_conf;
	// string columns (fls_sel_plan_create_strings): the plan's columns are the row hashes; these are the strings
	bool                str = false;
	std::vector<StrCol> scols;
	DevMem              scols_d, tabs_d, hash_d, len_d, clen_d, wptr_d, str_memo;
	uint32_t            memo_bits = 0;
	std::map<uint32_t, ItemSet> samples; // stride -> sampled items
};

namespace {

int upload(DevMem& m, const void* h, size_t n) {
	if (!m.alloc(n)) { return FLS_ERR_CUDA; }
	if (n && cudaMemcpy(m.p, h, n, cudaMemcpyHostToDevice) != cudaSuccess) { return FLS_ERR_CUDA; }
	return FLS_OK;
}

// Sampled items (vectors 0, stride, ... of every chunk) with their chunk row ranges.
int sample_set(fls_sel_plan* p, uint32_t stride, ItemSet** out) {
	auto f = p->samples.find(stride);
	if (f == p->samples.end()) {
		std::vector<Item>     it;
		std::vector<uint32_t> rows(p->n_chunks + 1, 0), row_chunk;
		for (uint64_t c = 0; c < p->n_chunks; ++c) {
			rows[c] = static_cast<uint32_t>(it.size());
			for (uint32_t i = p->chunk_items[c]; i < p->chunk_items[c + 1]; i += stride) {
				it.push_back(p->items[i]);
				row_chunk.push_back(static_cast<uint32_t>(c));
			}
		}
		rows[p->n_chunks] = static_cast<uint32_t>(it.size());
		ItemSet& s        = p->samples[stride];
		s.n               = it.size();
		int rc;
		if ((rc = upload(s.items, it.data(), it.size() * sizeof(Item))) != FLS_OK) { return rc; }
		if ((rc = upload(s.chunk_items, rows.data(), rows.size() * 4)) != FLS_OK) { return rc; }
		if ((rc = upload(s.row_chunk, row_chunk.data(), row_chunk.size() * 4)) != FLS_OK) { return rc; }
		f = p->samples.find(stride);
	}
	*out = &f->second;
	return FLS_OK;
}

// Exact sizes of the chunks listed (all when chunks is empty).
int wizard_run(fls_sel_plan* p, const std::vector<uint32_t>& subset, uint64_t* d_sizes, uint8_t* d_best,
               uint32_t* d_dict_n, cudaStream_t s) {
	Device* dev = current_device();
	if (!dev) { return FLS_ERR_CUDA; }
	const bool            all = subset.empty();
	std::vector<uint32_t> chunks;
	if (all) {
		chunks.resize(p->n_chunks);
		for (uint64_t c = 0; c < p->n_chunks; ++c) { chunks[c] = static_cast<uint32_t>(c); }
	} else {
		chunks = subset;
	}
	// item list of the selected chunks (in chunk order) and their ranges: the plan's own device lists for all
	// chunks; for a subset, lists built here and copied in stream order into the plan's scratch
	const Item*     items_d  = p->items_d.as<Item>();
	const uint32_t* ranges_d = p->chunk_items_d.as<uint32_t>();
	const uint32_t* ccol_d   = p->chunk_col_d.as<uint32_t>();
	const uint32_t* ids_d    = nullptr;
	uint64_t        n_items  = p->items.size();
	if (!all) {
		std::vector<Item>     it;
		std::vector<uint32_t> ranges(chunks.size() + 1), ccol(chunks.size());
		for (size_t i = 0; i < chunks.size(); ++i) {
			const uint32_t c = chunks[i];
			ranges[i]        = static_cast<uint32_t>(it.size());
			ccol[i]          = p->chunk_col[c];
			for (uint32_t j = p->chunk_items[c]; j < p->chunk_items[c + 1]; ++j) {
				Item m  = p->items[j];
				m.chunk = static_cast<uint32_t>(i); // local chunk numbering for this run
				it.push_back(m);
			}
		}
		ranges[chunks.size()] = static_cast<uint32_t>(it.size());
		n_items               = it.size();
		if (it.empty()) { return FLS_OK; }
		// one copy for the four lists, and no wait (a copy from pageable memory is staged before the call returns)
		const size_t         o1 = it.size() * sizeof(Item), o2 = o1 + ranges.size() * 4, o3 = o2 + ccol.size() * 4;
		std::vector<uint8_t> lists(o3 + chunks.size() * 4);
		std::memcpy(lists.data(), it.data(), o1);
		std::memcpy(lists.data() + o1, ranges.data(), ranges.size() * 4);
		std::memcpy(lists.data() + o2, ccol.data(), ccol.size() * 4);
		std::memcpy(lists.data() + o3, chunks.data(), chunks.size() * 4);
		if (!p->sub_lists.need(lists.size()) ||
		    cudaMemcpyAsync(p->sub_lists.m.p, lists.data(), lists.size(), cudaMemcpyHostToDevice, s) != cudaSuccess) {
			return FLS_ERR_CUDA;
		}
		items_d  = p->sub_lists.as<Item>();
		ranges_d = reinterpret_cast<const uint32_t*>(p->sub_lists.as<uint8_t>() + o1);
		ccol_d   = reinterpret_cast<const uint32_t*>(p->sub_lists.as<uint8_t>() + o2);
		ids_d    = reinterpret_cast<const uint32_t*>(p->sub_lists.as<uint8_t>() + o3);
	}
	if (n_items == 0) { return FLS_OK; }
	if (!p->parts.need(n_items * 4) || !p->bw_code.need(n_items * 4) || !p->info.need(n_items * sizeof(VecInfo)) || !p->dict_n.need(chunks.size() * 4)) {
		return FLS_ERR_CUDA;
	}
	if (p->str) {
		// the rows of every vector: hashes (the columns the integer passes read), lengths, compressed lengths
		if (!p->vlen.need(n_items * 8) || !p->vclen.need(n_items * 8) || !p->dict_w.need(chunks.size() * 16)) {
			return FLS_ERR_CUDA;
		}
		if (launch_str_rows(p->scols_d.as<StrCol>(), items_d, n_items, p->vlen.as<uint64_t>(), p->vclen.as<uint64_t>(), 1u,
		                    p->str_memo.as<uint64_t>(), p->memo_bits, p->scols.size(), s) != cudaSuccess) {
			return FLS_ERR_CUDA;
		}
	}
	ItemArgs ia {p->cols_d.as<Col>(), items_d, n_items};
	k_parts<<<grid_for(n_items), kWarps * 32, 0, s>>>(ia, p->parts.as<uint32_t>(), p->info.as<VecInfo>());
	++launch_counter();
	// dictionary of every chunk: one CTA per chunk, tables in shared memory
	{
		static SmemLimit limit;
		if (limit.need(reinterpret_cast<const void*>(k_chunk_dict), sizeof(ChunkDictSmem)) != cudaSuccess) { return FLS_ERR_CUDA; }
		// one CTA per SM, each with its own slot scratch
		const uint32_t grid = static_cast<uint32_t>(std::min<size_t>(chunks.size(), static_cast<size_t>(dev->sm_count)));
		if (!p->gtab.need(kCdGBytes * grid + 4)) { return FLS_ERR_CUDA; }
		uint32_t* ticket = reinterpret_cast<uint32_t*>(p->gtab.as<uint8_t>() + kCdGBytes * grid);
		if (cudaMemsetAsync(ticket, 0, 4, s) != cudaSuccess) { return FLS_ERR_CUDA; }
		ChunkDictArgs a {p->cols_d.as<Col>(), items_d, p->info.as<VecInfo>(), ranges_d,
		                 static_cast<uint32_t>(chunks.size()), p->dict_n.as<uint32_t>(), p->bw_code.as<uint32_t>(),
		                 dev->status, nullptr, nullptr, nullptr, p->gtab.as<uint16_t>(), ticket};
		if (p->str) {
			const uint32_t* const* wp = p->wptr_d.as<const uint32_t*>();
			a.w0                      = wp;
			a.w1                      = wp + p->scols.size();
			a.dict_w                  = p->dict_w.as<uint64_t>();
		}
		k_chunk_dict<<<grid, kCdThreads, sizeof(ChunkDictSmem), s>>>(a);
		++launch_counter();
		if (cudaGetLastError() != cudaSuccess) { return FLS_ERR_CUDA; }
	}
	uint64_t* sizes = d_sizes;
	uint8_t*  best  = d_best;
	if (!all) {
		if (!p->sub_sizes.need(chunks.size() * K * 8) || !p->sub_best.need(chunks.size())) { return FLS_ERR_CUDA; }
		sizes = p->sub_sizes.as<uint64_t>();
		best  = p->sub_best.as<uint8_t>();
	}
	if (p->str) {
		StrSizeArgs sa {ccol_d, ranges_d, p->parts.as<uint32_t>(), p->bw_code.as<uint32_t>(),
		                p->vlen.as<uint64_t>(), p->vclen.as<uint64_t>(), p->dict_n.as<uint32_t>(), p->dict_w.as<uint64_t>(),
		                p->scols_d.as<StrCol>(), static_cast<uint32_t>(chunks.size()), sizes, best};
		k_str_sizes<<<static_cast<unsigned>((chunks.size() + 7) / 8), 256, 0, s>>>(sa);
	} else {
		SizeArgs sa {p->cols_d.as<Col>(), ccol_d, ranges_d, p->parts.as<uint32_t>(),
		             p->bw_code.as<uint32_t>(), p->dict_n.as<uint32_t>(), static_cast<uint32_t>(chunks.size()), sizes, best};
		k_chunk_sizes<<<static_cast<unsigned>((chunks.size() + 7) / 8), 256, 0, s>>>(sa);
	}
	++launch_counter();
	if (cudaGetLastError() != cudaSuccess) { return FLS_ERR_CUDA; }
	if (!all) {
		// the subset's choices go to their chunks (sizes of a subset are not reported)
		if (d_best) {
			k_scatter_best<<<64, 256, 0, s>>>(best, ids_d, static_cast<uint32_t>(chunks.size()), d_best);
			++launch_counter();
		}
	} else if (d_dict_n) {
		if (cudaMemcpyAsync(d_dict_n, p->dict_n.m.p, chunks.size() * 4, cudaMemcpyDeviceToDevice, s) != cudaSuccess) {
			return FLS_ERR_CUDA;
		}
	}
	return cudaStreamSynchronize(s) == cudaSuccess ? FLS_OK : FLS_ERR_CUDA;
}

} // namespace

extern "C" {

int fls_sel_plan_create(const fls_sel_column* cols, uint32_t n_cols, uint32_t chunk_vectors, fls_sel_plan** out) {
	if (!out || (!cols && n_cols) || chunk_vectors == 0 || chunk_vectors > kMaxVecPerChunk) { return FLS_ERR_ARG; }
	*out = nullptr;
	if (!current_device()) { return FLS_ERR_CUDA; }
	auto p           = std::make_unique<fls_sel_plan>();
	p->chunk_vectors = chunk_vectors;
	for (uint32_t c = 0; c < n_cols; ++c) {
		const fls_sel_column& s = cols[c];
		if ((s.width != 32 && s.width != 64) || (s.n_vec && !s.d_values) ||
		    (reinterpret_cast<uintptr_t>(s.d_values) & 15u) != 0 || s.n_vec >= (1ull << 32)) {
			return FLS_ERR_ARG;
		}
		p->cols.push_back(Col {static_cast<const uint8_t*>(s.d_values), s.n_vec, s.width, s.is_signed ? 1u : 0u});
		for (uint64_t v0 = 0; v0 < s.n_vec; v0 += chunk_vectors) {
			const uint32_t chunk = static_cast<uint32_t>(p->chunk_col.size());
			p->chunk_col.push_back(c);
			p->chunk_first.push_back(v0);
			p->chunk_items.push_back(static_cast<uint32_t>(p->items.size()));
			const uint64_t v1 = std::min<uint64_t>(s.n_vec, v0 + chunk_vectors);
			for (uint64_t v = v0; v < v1; ++v) {
				p->items.push_back(Item {c, chunk, static_cast<uint32_t>(v), static_cast<uint32_t>(v - v0)});
			}
		}
	}
	if (p->items.size() >= (1ull << 32)) { return FLS_ERR_TOO_LARGE; }
	p->n_chunks = p->chunk_col.size();
	p->chunk_items.push_back(static_cast<uint32_t>(p->items.size()));
	int rc;
	if ((rc = upload(p->cols_d, p->cols.data(), p->cols.size() * sizeof(Col))) != FLS_OK) { return rc; }
	if ((rc = upload(p->items_d, p->items.data(), p->items.size() * sizeof(Item))) != FLS_OK) { return rc; }
	if ((rc = upload(p->chunk_items_d, p->chunk_items.data(), p->chunk_items.size() * 4)) != FLS_OK) { return rc; }
	if ((rc = upload(p->chunk_col_d, p->chunk_col.data(), p->chunk_col.size() * 4)) != FLS_OK) { return rc; }
	*out = p.release();
	return FLS_OK;
}

} // extern "C"

namespace flsgpu {
int fsst_import_table(const uint8_t* buf, uint64_t avail, FsstTable* t, uint64_t* used);
}

namespace {
// An exported FSST table (fsst_export format) arranged for greedy matching (StrTab); the codes past the table's
// symbol count, which decode as "corrupt", are not symbols.
int arrange_table(const uint8_t* tab, uint64_t n, StrTab* out) {
	FsstTable t {};
	const int rc = fsst_import_table(tab, n, &t, nullptr);
	if (rc != FLS_OK) { return rc; }
	const uint32_t zt = tab[8] & 1u;
	uint32_t       count = 0;
	for (uint32_t l = 0; l < 8; ++l) { count += tab[9 + l]; }
	if (zt && count) { --count; }
	std::vector<uint32_t> codes;
	for (uint32_t c = zt; c < zt + count && c < 255; ++c) { codes.push_back(c); }
	std::memset(out, 0, sizeof(*out));
	std::vector<uint32_t> longer;
	std::vector<bool>     is_two(65536, false);
	for (const uint32_t c : codes) {
		const uint32_t b = static_cast<uint32_t>(t.sym[c]);
		if (t.len[c] == 1) {
			out->one[(b & 0xFFu) >> 5] |= 1u << (b & 31u);
		} else if (t.len[c] == 2) {
			out->two[out->n_two++] = static_cast<uint16_t>(b);
			is_two[b & 0xFFFFu]    = true;
		} else if (t.len[c] > 2) {
			longer.push_back(c);
		}
	}
	auto pair_of  = [&](uint32_t c) { return static_cast<uint32_t>(t.sym[c]) & 0xFFFFu; };
	auto short_of = [&](uint32_t pair) { return is_two[pair] ? 2u : (out->one[(pair & 0xFFu) >> 5] >> (pair & 31u)) & 1u; };
	// group id of every pair: its own while ids last, then one of the same g_short
	std::map<uint32_t, uint32_t> id;
	uint32_t                     groups = 0;
	for (const uint32_t c : longer) {
		const uint32_t pair = pair_of(c);
		if (id.count(pair)) { continue; }
		const uint32_t sh = short_of(pair);
		uint32_t       g  = groups;
		if (groups + 3 >= kStrGroups) { // the last three ids: one for each g_short
			for (g = 0; g < groups && out->g_short[g] != sh; ++g) {}
		}
		if (g == groups) { ++groups; }
		out->g_short[g]                 = static_cast<uint8_t>(sh);
		out->pair[out->n_pair]          = static_cast<uint16_t>(pair);
		out->pair_group[out->n_pair++]  = static_cast<uint8_t>(g);
		id[pair]                        = g;
	}
	std::stable_sort(longer.begin(), longer.end(), [&](uint32_t x, uint32_t y) {
		const uint32_t gx = id[pair_of(x)], gy = id[pair_of(y)];
		return gx != gy ? gx < gy : t.len[x] > t.len[y];
	});
	for (size_t k = 0; k < longer.size(); ++k) {
		out->len[k] = t.len[longer[k]];
		out->sym[k] = make_ulonglong2(t.sym[longer[k]], ~0ull >> (64 - 8 * out->len[k]));
		out->start[id[pair_of(longer[k])] + 1] = static_cast<uint16_t>(k + 1);
	}
	for (uint32_t g = 0; g < 257; ++g) { out->start[g + 1] = std::max(out->start[g], out->start[g + 1]); }
	return FLS_OK;
}
} // namespace

extern "C" {

int fls_sel_plan_create_strings(const fls_sel_str_column* cols, uint32_t n_cols, uint32_t chunk_vectors,
                                fls_sel_plan** out) {
	if (!out || (!cols && n_cols)) { return FLS_ERR_ARG; }
	*out = nullptr;
	uint64_t rows = 0;
	for (uint32_t c = 0; c < n_cols; ++c) {
		if (cols[c].n_rows % 1024 || (cols[c].n_rows && (!cols[c].d_offsets || !cols[c].table)) ||
		    cols[c].n_rows >= (1ull << 41)) {
			return FLS_ERR_ARG;
		}
		rows += cols[c].n_rows;
	}
	DevMem hash, len, clen, tabs;
	if (!hash.alloc(rows * 8 + 16) || !len.alloc(rows * 4 + 16) || !clen.alloc(rows * 4 + 16) ||
	    !tabs.alloc(sizeof(StrTab) * (n_cols ? n_cols : 1))) {
		return FLS_ERR_CUDA;
	}
	// the plan's integer columns are the row hashes
	std::vector<fls_sel_column> hc(n_cols);
	std::vector<StrCol>         sc(n_cols);
	std::vector<StrTab>         st(n_cols);
	uint64_t                    r0 = 0;
	for (uint32_t c = 0; c < n_cols; ++c) {
		const fls_sel_str_column& x = cols[c];
		if (x.n_rows) {
			const int rc = arrange_table(x.table, x.table_size, &st[c]);
			if (rc != FLS_OK) { return rc; }
		}
		uint64_t nb = 0;
		if (x.n_rows && cudaMemcpy(&nb, x.d_offsets + x.n_rows, 8, cudaMemcpyDeviceToHost) != cudaSuccess) {
			return FLS_ERR_CUDA;
		}
		hc[c]          = fls_sel_column {};
		hc[c].d_values = hash.as<uint64_t>() + r0;
		hc[c].n_vec    = x.n_rows / 1024;
		hc[c].width    = 64;
		sc[c] = StrCol {x.d_bytes, x.d_offsets, nb, tabs.as<StrTab>() + c, static_cast<uint32_t>(x.table_size),
		                hash.as<uint64_t>() + r0, len.as<uint32_t>() + r0, clen.as<uint32_t>() + r0};
		r0 += x.n_rows;
	}
	fls_sel_plan* p  = nullptr;
	int           rc = fls_sel_plan_create(hc.data(), n_cols, chunk_vectors, &p);
	if (rc != FLS_OK) { return rc; }
	std::unique_ptr<fls_sel_plan> own(p);
	std::vector<const uint32_t*>  wp(2 * n_cols);
	for (uint32_t c = 0; c < n_cols; ++c) {
		wp[c]          = sc[c].len;
		wp[n_cols + c] = sc[c].clen;
	}
	if (n_cols && (cudaMemcpy(tabs.p, st.data(), sizeof(StrTab) * n_cols, cudaMemcpyHostToDevice) != cudaSuccess ||
	               (rc = upload(own->scols_d, sc.data(), sizeof(StrCol) * n_cols)) != FLS_OK ||
	               (rc = upload(own->wptr_d, wp.data(), sizeof(void*) * wp.size())) != FLS_OK)) {
		return rc != FLS_OK ? rc : FLS_ERR_CUDA;
	}
	uint64_t most = 1; // rows of a column
	for (uint32_t c = 0; c < n_cols; ++c) { most = std::max<uint64_t>(most, cols[c].n_rows); }
	own->memo_bits = kStrMemoMax;
	while (own->memo_bits > kStrMemoMin && ((1ull << (own->memo_bits - 1)) >= most ||
	                                        (static_cast<uint64_t>(n_cols) << own->memo_bits) > (1ull << kStrMemoAll))) {
		--own->memo_bits;
	}
	if (n_cols && rows / 1024 / n_cols >= kStrMemoVecs &&
	    !own->str_memo.alloc(((static_cast<uint64_t>(n_cols) << own->memo_bits) + n_cols) * 8)) {
		return FLS_ERR_CUDA;
	}
	own->str   = true;
	own->scols = sc;
	own->hash_d.p = hash.p, hash.p = nullptr;
	own->len_d.p  = len.p, len.p = nullptr;
	own->clen_d.p = clen.p, clen.p = nullptr;
	own->tabs_d.p = tabs.p, tabs.p = nullptr;
	*out          = own.release();
	return FLS_OK;
}

int fls_sel_plan_info(const fls_sel_plan* p, uint64_t* n_chunks, uint64_t* n_vectors) {
	if (!p) { return FLS_ERR_ARG; }
	if (n_chunks) { *n_chunks = p->n_chunks; }
	if (n_vectors) { *n_vectors = p->items.size(); }
	return FLS_OK;
}

int fls_sel_plan_chunks(const fls_sel_plan* p, uint32_t* h_col, uint64_t* h_first, uint32_t* h_count) {
	if (!p) { return FLS_ERR_ARG; }
	for (uint64_t c = 0; c < p->n_chunks; ++c) {
		if (h_col) { h_col[c] = p->chunk_col[c]; }
		if (h_first) { h_first[c] = p->chunk_first[c]; }
		if (h_count) { h_count[c] = p->chunk_items[c + 1] - p->chunk_items[c]; }
	}
	return FLS_OK;
}

int fls_sel_plan_destroy(fls_sel_plan* p) {
	delete p;
	return FLS_OK;
}

int fls_sel_vector_parts(const fls_sel_plan* p, uint32_t* d_parts, void* stream) {
	if (!p || (!d_parts && !p->items.empty())) { return FLS_ERR_ARG; }
	if (p->items.empty()) { return FLS_OK; }
	cudaStream_t s = static_cast<cudaStream_t>(stream);
	ItemArgs     a {p->cols_d.as<Col>(), p->items_d.as<Item>(), p->items.size()};
	k_parts<<<grid_for(p->items.size()), kWarps * 32, 0, s>>>(a, d_parts, nullptr);
	++launch_counter();
	return cudaGetLastError() == cudaSuccess ? FLS_OK : FLS_ERR_CUDA;
}

int fls_sel_wizard(fls_sel_plan* p, uint64_t* d_sizes, uint8_t* d_best, uint32_t* d_dict_n, void* stream) {
	if (!p || ((!d_sizes || !d_best) && p->n_chunks)) { return FLS_ERR_ARG; }
	return wizard_run(p, {}, d_sizes, d_best, d_dict_n, static_cast<cudaStream_t>(stream));
}

} // extern "C"

namespace {
// Statistics of the items of a: for a string plan, the sampled vectors' rows first (hashes and lengths of every
// row, compressed lengths of every kStrFeatRowStride-th row), then the hash features with the string slots
// filled in.
constexpr uint32_t kStrFeatRowStride = 4;
cudaError_t        sample_features(fls_sel_plan* p, const ItemArgs& a, float* feat, cudaStream_t s) {
	if (p->str) {
		const cudaError_t e =
		    launch_str_rows(p->scols_d.as<StrCol>(), a.items, a.n_items, nullptr, nullptr, kStrFeatRowStride,
		                    p->str_memo.as<uint64_t>(), p->memo_bits, p->scols.size(), s);
		if (e != cudaSuccess) { return e; }
	}
	cudaError_t e = launch_features(a, feat, s);
	if (e != cudaSuccess || !p->str) { return e; }
	k_str_features<<<grid_for(a.n_items), kWarps * 32, 0, s>>>(p->scols_d.as<StrCol>(), a.items, a.n_items, feat,
	                                                           kStrFeatRowStride);
	++launch_counter();
	return cudaGetLastError();
}
} // namespace

extern "C" {

int fls_sel_features(fls_sel_plan* p, uint32_t stride, float* d_feat, uint32_t* d_row_chunk, uint64_t* n_rows,
                     void* stream) {
	if (!p || stride == 0 || !n_rows) { return FLS_ERR_ARG; }
	ItemSet* set = nullptr;
	int      rc  = sample_set(p, stride, &set);
	if (rc != FLS_OK) { return rc; }
	*n_rows = set->n;
	if (!d_feat || set->n == 0) { return FLS_OK; }
	cudaStream_t s = static_cast<cudaStream_t>(stream);
	ItemArgs     a {p->cols_d.as<Col>(), set->items.as<Item>(), set->n};
	if (sample_features(p, a, d_feat, s) != cudaSuccess) { return FLS_ERR_CUDA; }
	if (d_row_chunk && cudaMemcpyAsync(d_row_chunk, set->row_chunk.p, set->n * 4, cudaMemcpyDeviceToDevice, s) != cudaSuccess) {
		return FLS_ERR_CUDA;
	}
	return cudaGetLastError() == cudaSuccess ? FLS_OK : FLS_ERR_CUDA;
}

int fls_sel_learned(fls_sel_plan* p, const float* d_params, uint32_t stride, float threshold, uint8_t* d_choice,
                    float* d_conf, uint64_t* n_fallback, void* stream) {
	if (!p || !d_params || stride == 0 || (!d_choice && p->n_chunks)) { return FLS_ERR_ARG; }
	if (n_fallback) { *n_fallback = 0; }
	if (p->n_chunks == 0) { return FLS_OK; }
	cudaStream_t s   = static_cast<cudaStream_t>(stream);
	ItemSet*     set = nullptr;
	int          rc  = sample_set(p, stride, &set);
	if (rc != FLS_OK) { return rc; }
	const uint64_t n = set->n;
	if (!p->l_work.need(n * (NF + K) * 4) || !p->l_conf.need(p->n_chunks * 4)) { return FLS_ERR_CUDA; }
	float*   conf = d_conf ? d_conf : p->l_conf.as<float>();
	float*   feat = p->l_work.as<float>();
	float*   prob = feat + n * NF;
	ItemArgs a {p->cols_d.as<Col>(), set->items.as<Item>(), n};
	if (sample_features(p, a, feat, s) != cudaSuccess) { return FLS_ERR_CUDA; }
	if (probabilities(s, d_params, feat, n, prob) != cudaSuccess) { return FLS_ERR_CUDA; }
	k_vote<<<static_cast<unsigned>((p->n_chunks + 7) / 8), 256, 0, s>>>(prob, set->chunk_items.as<uint32_t>(),
	                                                                     static_cast<uint32_t>(p->n_chunks), d_choice,
	                                                                     conf, p->str ? kStrK : K);
	++launch_counter();
	if (cudaGetLastError() != cudaSuccess) { return FLS_ERR_CUDA; }
	if (threshold > 0.0f) {
		std::vector<float> hc(p->n_chunks);
		if (cudaMemcpyAsync(hc.data(), conf, hc.size() * 4, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
		    cudaStreamSynchronize(s) != cudaSuccess) {
			return FLS_ERR_CUDA;
		}
		std::vector<uint32_t> low;
		for (uint64_t c = 0; c < p->n_chunks; ++c) {
			if (hc[c] < threshold) { low.push_back(static_cast<uint32_t>(c)); }
		}
		if (n_fallback) { *n_fallback = low.size(); }
		if (!low.empty() && (rc = wizard_run(p, low, nullptr, d_choice, nullptr, s)) != FLS_OK) { return rc; }
	}
	return cudaStreamSynchronize(s) == cudaSuccess ? FLS_OK : FLS_ERR_CUDA;
}

uint64_t fls_sel_param_count(void) { return param_count(); }

int fls_sel_mlp_init(float* d_params, uint64_t seed) {
	if (!d_params) { return FLS_ERR_ARG; }
	std::vector<float>              h(param_count(), 0.0f);
	std::mt19937_64                 rng(seed);
	std::normal_distribution<float> nd(0.0f, 1.0f);
	float*                          w1 = h.data();
	float*                          w2 = w1 + NF * H + H;
	float*                          w3 = w2 + H * H + H;
	for (int i = 0; i < NF * H; ++i) { w1[i] = nd(rng) * std::sqrt(2.0f / NF); }
	for (int i = 0; i < H * H; ++i) { w2[i] = nd(rng) * std::sqrt(2.0f / H); }
	for (int i = 0; i < H * K; ++i) { w3[i] = nd(rng) * std::sqrt(2.0f / H); }
	return cudaMemcpy(d_params, h.data(), h.size() * 4, cudaMemcpyHostToDevice) == cudaSuccess ? FLS_OK : FLS_ERR_CUDA;
}

int fls_sel_mlp_forward(const float* d_params, const float* d_x, uint64_t n, float* d_prob, void* stream) {
	if (!d_params || ((!d_x || !d_prob) && n) || n >= (1ull << 31)) { return FLS_ERR_ARG; }
	if (n == 0) { return FLS_OK; }
	cudaStream_t s = static_cast<cudaStream_t>(stream);
	if (probabilities(s, d_params, d_x, n, d_prob) != cudaSuccess) { return FLS_ERR_CUDA; }
	return cudaStreamSynchronize(s) == cudaSuccess ? FLS_OK : FLS_ERR_CUDA;
}

int fls_sel_mlp_grad(const float* d_params, const float* d_x, const int32_t* d_y, uint64_t n, float* d_grad,
                     float* d_loss, void* stream) {
	if (!d_params || !d_x || !d_y || !d_grad || !d_loss || n == 0 || n >= (1ull << 31)) { return FLS_ERR_ARG; }
	cudaStream_t s = static_cast<cudaStream_t>(stream);
	DevMem       w;
	if (!w.alloc(n * (4 * H + 2 * K) * 4)) { return FLS_ERR_CUDA; }
	float* h1  = w.as<float>();
	float* h2  = h1 + n * H;
	float* z   = h2 + n * H;
	float* dz  = z + n * K;
	float* dh2 = dz + n * K;
	float* dh1 = dh2 + n * H;
	if (cudaMemsetAsync(d_loss, 0, 4, s) != cudaSuccess) { return FLS_ERR_CUDA; }
	if (forward(s, d_params, d_x, n, h1, h2, z) != cudaSuccess) { return FLS_ERR_CUDA; }
	k_softmax<<<static_cast<unsigned>(std::min<uint64_t>((n + 255) / 256, 4096)), 256, 0, s>>>(z, n, d_y, dz, d_loss,
	                                                                                            nullptr, nullptr);
	++launch_counter();
	if (backward(s, d_params, d_x, n, h1, h2, dz, dh2, dh1, d_grad) != cudaSuccess) { return FLS_ERR_CUDA; }
	return cudaStreamSynchronize(s) == cudaSuccess ? FLS_OK : FLS_ERR_CUDA;
}

int fls_sel_adam_step(float* d_params, const float* d_grad, float* d_m, float* d_v, float lr, float beta1, float beta2,
                      float eps, uint32_t step, void* stream) {
	if (!d_params || !d_grad || !d_m || !d_v || step == 0) { return FLS_ERR_ARG; }
	cudaStream_t s = static_cast<cudaStream_t>(stream);
	k_adam<<<64, 256, 0, s>>>(d_params, d_grad, d_m, d_v, param_count(), lr, beta1, beta2, eps, step, nullptr);
	++launch_counter();
	return cudaGetLastError() == cudaSuccess ? FLS_OK : FLS_ERR_CUDA;
}

int fls_sel_train(float* d_params, const float* d_x, const int32_t* d_y, const uint32_t* d_perm, uint32_t batch,
                  uint32_t steps, float lr, float* d_loss_hist, void* stream) {
	if (!d_params || !d_x || !d_y || !d_perm || batch == 0 || batch > (1u << 20)) { return FLS_ERR_ARG; }
	if (steps == 0) { return FLS_OK; }
	// capture needs a stream other than the legacy default one: a private stream ordered after the caller's
	cudaStream_t caller = static_cast<cudaStream_t>(stream);
	cudaStream_t s      = nullptr;
	cudaEvent_t  ev     = nullptr;
	if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) { return FLS_ERR_CUDA; }
	struct Guard {
		cudaStream_t s;
		cudaEvent_t* ev;
		~Guard() {
			if (*ev) { cudaEventDestroy(*ev); }
			cudaStreamSynchronize(s);
			cudaStreamDestroy(s);
		}
	} guard {s, &ev};
	if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess || cudaEventRecord(ev, caller) != cudaSuccess ||
	    cudaStreamWaitEvent(s, ev, 0) != cudaSuccess) {
		return FLS_ERR_CUDA;
	}
	const uint64_t P = param_count(), B = batch;
	DevMem         w;
	if (!w.alloc((B * (NF + 4 * H + 2 * K) + 3 * P) * 4 + B * 4 + 64)) { return FLS_ERR_CUDA; }
	float*    xb  = w.as<float>();
	float*    h1  = xb + B * NF;
	float*    h2  = h1 + B * H;
	float*    z   = h2 + B * H;
	float*    dz  = z + B * K;
	float*    dh2 = dz + B * K;
	float*    dh1 = dh2 + B * H;
	float*    g   = dh1 + B * H;
	float*    m   = g + P;
	float*    v   = m + P;
	int32_t*  yb  = reinterpret_cast<int32_t*>(v + P);
	uint32_t* st  = reinterpret_cast<uint32_t*>(yb + B);
	if (cudaMemsetAsync(m, 0, 2 * P * 4, s) != cudaSuccess || cudaMemsetAsync(st, 0, 4, s) != cudaSuccess) {
		return FLS_ERR_CUDA;
	}
	if (d_loss_hist && cudaMemsetAsync(d_loss_hist, 0, steps * 4ull, s) != cudaSuccess) { return FLS_ERR_CUDA; }
	// one training step, captured once and replayed `steps` times
	cudaGraph_t     graph = nullptr;
	cudaGraphExec_t exec  = nullptr;
	const uint64_t launches0 = launch_counter();
	if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) { return FLS_ERR_CUDA; }
	k_gather<<<64, 256, 0, s>>>(d_x, d_y, d_perm, st, batch, xb, yb);
	forward(s, d_params, xb, B, h1, h2, z);
	k_softmax<<<static_cast<unsigned>((B + 255) / 256), 256, 0, s>>>(z, B, yb, dz, nullptr, d_loss_hist, st);
	backward(s, d_params, xb, B, h1, h2, dz, dh2, dh1, g);
	k_adam<<<64, 256, 0, s>>>(d_params, g, m, v, P, lr, 0.9f, 0.999f, 1e-8f, 0, st);
	k_step_inc<<<1, 1, 0, s>>>(st);
	const cudaError_t ce = cudaStreamEndCapture(s, &graph);
	launch_counter()     = launches0;
	if (ce != cudaSuccess || !graph) { return FLS_ERR_CUDA; }
	const cudaError_t ie = cudaGraphInstantiate(&exec, graph, 0);
	cudaGraphDestroy(graph);
	if (ie != cudaSuccess) { return FLS_ERR_CUDA; }
	int rc = FLS_OK;
	for (uint32_t i = 0; i < steps && rc == FLS_OK; ++i) {
		if (cudaGraphLaunch(exec, s) != cudaSuccess) { rc = FLS_ERR_CUDA; }
	}
	launch_counter() += static_cast<uint64_t>(steps) * 15; // kernels per replayed step
	if (cudaStreamSynchronize(s) != cudaSuccess) { rc = FLS_ERR_CUDA; }
	cudaGraphExecDestroy(exec);
	return rc;
}

} // extern "C"
