// The warp-level parts of the wizard's chunk dictionary (k_chunk_dict): how its keys are placed, one look at a slot of
// its table, and a warp's queue of keys on their way into it.
#pragma once

#include "fls_device.cuh"

namespace flsgpu {
namespace sel {

constexpr uint32_t kCdFree = 0xFFFFFFFFu; // a slot without a key

// A key's hash: *place places it (by its top bits), *other's upper half is what its slot keeps of it (*tag: never all
// ones, so that no slot reads as free) and that half's low bits choose its part.
// 32-bit keys: the 32-bit finaliser of MurmurHash3 (Appleby), a bijection.
__device__ __forceinline__ void cd_hash(uint32_t x, uint32_t* place, uint32_t* other) {
	x ^= x >> 16;
	x *= 0x85ebca6bu;
	x ^= x >> 13;
	x *= 0xc2b2ae35u;
	x ^= x >> 16;
	*place = x;
	*other = x << 16;
}
// 64-bit keys: a bijection of all 64 bits, three Feistel rounds on the halves (the odd multipliers are xxHash's 32-bit
// primes, Collet).  A linear combination of the halves, a multiplication more, put the 65,536 keys (a << 56) | (b << 24)
// on 256 places, 331 looks a key where spread keys take 2.
__device__ __forceinline__ void cd_hash(uint64_t x, uint32_t* place, uint32_t* other) {
	uint32_t lo = static_cast<uint32_t>(x), hi = static_cast<uint32_t>(x >> 32), f;
	f = lo * 0x9E3779B1u;
	hi += f ^ (f >> 15);
	f = hi * 0x85EBCA77u;
	lo += f ^ (f >> 13);
	f = lo * 0xC2B2AE3Du;
	hi += f ^ (f >> 16);
	*place = hi;
	*other = lo;
}
__device__ __forceinline__ uint32_t cd_tag(uint32_t other) {
	const uint32_t t = other & 0xFFFF0000u;
	return t == 0xFFFF0000u ? 0u : t;
}
// the part, of 1 << parts_log (at most 256), that a key belongs to
__device__ __forceinline__ uint32_t cd_part(uint32_t other, uint32_t parts_log) {
	return (other >> 16) & ((1u << parts_log) - 1u);
}

// One look at slot *s for value x at position pos: done (it is the key's slot now) or not (*s is the next one).
template <class T>
__device__ __forceinline__ bool cd_step(uint32_t* table, uint32_t n_slots, const T* vals, T x, uint32_t pos, uint32_t tag,
                                        uint32_t* s, bool* fresh) {
	uint32_t e = *reinterpret_cast<volatile uint32_t*>(table + *s);
	if (e == kCdFree) {
		e = atomicCAS(table + *s, kCdFree, tag | pos);
		if (e == kCdFree) {
			*fresh = true;
			return true;
		}
	}
	if ((e ^ tag) < 0x10000u && __ldg(vals + (e & 0xFFFFu)) == x) {
		if (pos < (e & 0xFFFFu)) { atomicMin(table + *s, tag | pos); }
		return true;
	}
	*s = *s + 1 == n_slots ? 0 : *s + 1;
	return false;
}

// A warp's queue of keys on their way into the table, and the list of the slots they ended in (the current vector's).
// It holds at most kCdQueue keys: fewer than 32 between two rows (drain sees to that), 32 more from a row.
constexpr uint32_t kCdQueue = 64;

template <class T>
struct CdQueue {
	T*         key;
	uint16_t * pos, *slot, *tag;
	uint16_t*  list;
	uint32_t   q, n; // keys queued, slots listed
	uint32_t   left; // looks the warp may still spend

	__device__ __forceinline__ void push(bool take, T x, uint32_t at_pos, uint32_t s, uint32_t t, uint32_t lane) {
		const uint32_t m = __ballot_sync(0xFFFFFFFFu, take);
		if (take) {
			const uint32_t at = q + __popc(m & ((1u << lane) - 1u));
			key[at]           = x;
			pos[at]           = static_cast<uint16_t>(at_pos);
			slot[at]          = static_cast<uint16_t>(s);
			tag[at]           = static_cast<uint16_t>(t >> 16);
		}
		q += __popc(m);
		__syncwarp();
	}
	// One look for every lane's key (those of `have`); the unfinished ones go on the queue.  Returns the new keys.
	__device__ __forceinline__ uint32_t look(uint32_t* table, uint32_t n_slots, const T* vals, bool have, T x,
	                                         uint32_t at_pos, uint32_t s, uint32_t t, uint32_t lane) {
		bool fresh = false, done = false;
		if (have) { done = cd_step<T>(table, n_slots, vals, x, at_pos, t, &s, &fresh); }
		const uint32_t m = __ballot_sync(0xFFFFFFFFu, done);
		if (done) { list[n + __popc(m & ((1u << lane) - 1u))] = static_cast<uint16_t>(s); }
		n += __popc(m);
		push(have && !done, x, at_pos, s, t, lane);
		return __popc(__ballot_sync(0xFFFFFFFFu, fresh));
	}
	// The last up to 32 queued keys take a look each.
	__device__ __forceinline__ uint32_t pop(uint32_t* table, uint32_t n_slots, const T* vals, uint32_t lane) {
		const uint32_t take = q < 32 ? q : 32;
		q -= take;
		const bool     have = lane < take;
		const uint32_t at   = q + (have ? lane : 0u);
		const T        x    = key[at];
		const uint32_t p = pos[at], s = slot[at], t = static_cast<uint32_t>(tag[at]) << 16;
		__syncwarp(); // read before the unfinished ones are written back
		return look(table, n_slots, vals, have, x, p, s, t, lane);
	}
	// Looks while a whole warp of keys waits (last: while any key does); *fresh grows by the new keys.  False when the
	// looks are spent: the keys that wait are then dropped (the next row's would not fit behind them), and the caller
	// gives the chunk up to the sort.
	__device__ __forceinline__ bool drain(uint32_t* table, uint32_t n_slots, const T* vals, bool last, uint32_t lane,
	                                      uint32_t* fresh) {
		while (q >= 32 || (last && q > 0)) {
			if (left == 0) {
				q = 0;
				return false;
			}
			--left;
			*fresh += pop(table, n_slots, vals, lane);
		}
		return true;
	}
};

} // namespace sel
} // namespace flsgpu
