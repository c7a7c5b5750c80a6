// Selections of filter plans (predicate pushdown): bitmaps -> index lists, bitmap combination, and the
// intersection of index lists (src/primitive/predicate/equal.cpp:12-28 and :100-119 of the reference).  One
// warp per vector; a vector's bitmap is 32 u32 words, one per lane.
#include "fls_b200.h"
#include "fls_plan.h"
#include "fls_runtime.h"
#include "fls_strings.cuh"

namespace flsgpu {

namespace {

// Positions of the set bits of the vector's bitmap (lane l holds word l, bits 32l .. 32l + 31) in ascending
// order into idx (global, 1024 entries); returns the count (every lane).  s: the warp's 1024 entries of shared
// memory, 16-byte aligned.
// A lane walks its own word's bits, as many steps as the fullest word has bits: straight to global memory when those are
// few, else into shared memory, from where the list leaves in 16-byte stores.  Where fewer words hold a bit than the
// fullest has bits (nearly all bits set, or clusters), one word a step, a bit a lane: its positions land side by side,
// without bank conflicts, and words without a bit cost nothing.  40,000 vectors (us, lanes walking to global memory / a
// word a step / now): 3 % of the bits set 12.3 / 34.8 / 12.3, 15 % 22.5 / 49.2 / 18.4, half 121 / 49 / 27, all 266 / 49 / 21.
__device__ __forceinline__ uint32_t compact_bits(uint32_t word, uint32_t lane, uint16_t* s, uint16_t* idx) {
	if (__all_sync(0xFFFFFFFFu, word == ~0u)) { // the whole vector, as a filter of sorted values has it
		if ((reinterpret_cast<uintptr_t>(idx) & 15u) == 0) {
#pragma unroll
			for (uint32_t j = 0; j < 4; ++j) {
				const uint32_t i = j * 32 + lane, x = i * 0x00080008u + 0x00010000u; // positions 8 i, 8 i + 1
				reinterpret_cast<uint4*>(idx)[i] = make_uint4(x, x + 0x00020002u, x + 0x00040004u, x + 0x00060006u);
			}
		} else {
			for (uint32_t i = lane; i < 1024; i += 32) { idx[i] = static_cast<uint16_t>(i); }
		}
		return 1024;
	}
	uint32_t       n    = 0;
	const uint32_t some = __ballot_sync(0xFFFFFFFFu, word != 0); // words that hold a bit
	const uint32_t mine = __popc(word), most = __reduce_max_sync(0xFFFFFFFFu, mine);
	const bool     direct = most <= 8;
	if (direct || most < static_cast<uint32_t>(__popc(some))) {
		const uint32_t inc = warp_inclusive_scan(mine, lane);
		uint16_t*      to  = direct ? idx : s;
		for (uint32_t at = inc - mine; word; word &= word - 1) { to[at++] = static_cast<uint16_t>(32 * lane + __ffs(word) - 1); }
		n = __shfl_sync(0xFFFFFFFFu, inc, 31);
		if (direct) { return n; }
	} else {
		for (uint32_t rest = some; rest; rest &= rest - 1) {
			const uint32_t k = __ffs(rest) - 1;
			const uint32_t w = __shfl_sync(0xFFFFFFFFu, word, k);
			if ((w >> lane) & 1u) { s[n + __popc(w & ((1u << lane) - 1u))] = static_cast<uint16_t>(32 * k + lane); }
			n += __popc(w);
		}
	}
	__syncwarp();
	if ((reinterpret_cast<uintptr_t>(idx) & 15u) == 0) {
		const uint32_t full = n / 8; // whole 16-byte pieces; entries past the count stay as they are
		for (uint32_t i = lane; i < full; i += 32) { reinterpret_cast<uint4*>(idx)[i] = reinterpret_cast<const uint4*>(s)[i]; }
		const uint32_t i = 8 * full + lane;
		if (i < n) { idx[i] = s[i]; }
	} else {
		for (uint32_t i = lane; i < n; i += 32) { idx[i] = s[i]; }
	}
	__syncwarp(); // the next vector's positions reuse s
	return n;
}

// (8 CTAs an SM, 32 registers a thread, here and in the next kernel: with 6 of them the intersection of full lists took 399
// us, 313 so)
__global__ void __launch_bounds__(256, 8) k_bitmap_to_selection(const uint32_t* __restrict__ bm, uint64_t n_vec,
                                                                uint16_t* __restrict__ idx, uint16_t* __restrict__ count) {
	__shared__ __align__(16) uint16_t list[8][1024];
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x / 32;
	const uint64_t nw   = static_cast<uint64_t>(gridDim.x) * (blockDim.x / 32);
	for (uint64_t v = static_cast<uint64_t>(blockIdx.x) * (blockDim.x / 32) + warp; v < n_vec; v += nw) {
		const uint32_t n = compact_bits(bm[32 * v + lane], lane, list[warp], idx + 1024 * v);
		if (lane == 0) { count[v] = static_cast<uint16_t>(n); }
	}
}

__global__ void k_bitmap_combine(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, uint32_t* out,
                                 uint64_t n_words, int op) {
	for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n_words;
	     i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
		const uint32_t x = a[i], y = b[i];
		out[i]           = op == FLS_BITMAP_AND ? (x & y) : op == FLS_BITMAP_OR ? (x | y) : (x & ~y);
	}
}

// Bits of an index list in shared memory (32 words per warp); false when a position or the count is out of
// range.
__device__ __forceinline__ bool list_bits(const uint16_t* idx, uint32_t n, uint32_t* bits, uint32_t lane) {
	bits[lane] = 0;
	__syncwarp();
	bool bad = n > 1024;
	n        = n > 1024 ? 1024 : n;
	for (uint32_t i = lane; i < n; i += 32) {
		const uint32_t p = idx[i];
		if (p < 1024) {
			atomicOr(bits + p / 32, 1u << (p % 32));
		} else {
			bad = true;
		}
	}
	__syncwarp();
	return !__any_sync(0xFFFFFFFFu, bad);
}

__global__ void __launch_bounds__(256, 8) k_selection_and(const uint16_t* __restrict__ i0, const uint16_t* __restrict__ c0,
                                                          const uint16_t* __restrict__ i1, const uint16_t* __restrict__ c1,
                                                          uint16_t* io, uint16_t* co, uint64_t n_vec, int* status) {
	__shared__ uint32_t               bits[8][2][32];
	__shared__ __align__(16) uint16_t list[8][1024];
	const uint32_t      lane = threadIdx.x & 31u, warp = threadIdx.x / 32;
	const uint64_t      nw   = static_cast<uint64_t>(gridDim.x) * (blockDim.x / 32);
	for (uint64_t v = static_cast<uint64_t>(blockIdx.x) * (blockDim.x / 32) + warp; v < n_vec; v += nw) {
		const bool ok0 = list_bits(i0 + 1024 * v, c0[v], bits[warp][0], lane);
		const bool ok1 = list_bits(i1 + 1024 * v, c1[v], bits[warp][1], lane);
		if (!(ok0 && ok1) && lane == 0) { atomicOr(status, STATUS_BAD_INDEX); }
		const uint32_t n = compact_bits(bits[warp][0][lane] & bits[warp][1][lane], lane, list[warp], io + 1024 * v);
		if (lane == 0) { co[v] = static_cast<uint16_t>(n); }
		__syncwarp();
	}
}

unsigned grid_for(uint64_t warps_needed) {
	const Device* d    = current_device();
	const uint64_t cap = static_cast<uint64_t>(d ? d->sm_count : 148) * 8; // 8 CTAs of 8 warps per SM
	const uint64_t g   = (warps_needed + 7) / 8;
	return static_cast<unsigned>(g < cap ? (g ? g : 1) : cap);
}

} // namespace

} // namespace flsgpu

extern "C" {

int fls_gpu_bitmap_to_selection(const uint64_t* d_bitmaps, uint64_t n_vec, uint16_t* d_idx, uint16_t* d_count,
                                fls_stream_t stream) {
	using namespace flsgpu;
	if (n_vec == 0) { return FLS_OK; }
	if (!d_bitmaps || !d_idx || !d_count) { return FLS_ERR_ARG; }
	k_bitmap_to_selection<<<grid_for(n_vec), 256, 0, static_cast<cudaStream_t>(stream)>>>(
	    reinterpret_cast<const uint32_t*>(d_bitmaps), n_vec, d_idx, d_count);
	++launch_counter();
	return cudaGetLastError() == cudaSuccess ? FLS_OK : FLS_ERR_CUDA;
}

int fls_gpu_bitmap_combine(const uint64_t* d_a, const uint64_t* d_b, uint64_t* d_out, uint64_t n_vec, int op,
                           fls_stream_t stream) {
	using namespace flsgpu;
	if (op < FLS_BITMAP_AND || op > FLS_BITMAP_ANDNOT) { return FLS_ERR_ARG; }
	if (n_vec == 0) { return FLS_OK; }
	if (!d_a || !d_b || !d_out) { return FLS_ERR_ARG; }
	const uint64_t words = 32 * n_vec;
	k_bitmap_combine<<<grid_for(words / 32), 256, 0, static_cast<cudaStream_t>(stream)>>>(
	    reinterpret_cast<const uint32_t*>(d_a), reinterpret_cast<const uint32_t*>(d_b),
	    reinterpret_cast<uint32_t*>(d_out), words, op);
	++launch_counter();
	return cudaGetLastError() == cudaSuccess ? FLS_OK : FLS_ERR_CUDA;
}

int fls_gpu_selection_and(const uint16_t* d_idx0, const uint16_t* d_count0, const uint16_t* d_idx1,
                          const uint16_t* d_count1, uint16_t* d_idx_out, uint16_t* d_count_out, uint64_t n_vec,
                          fls_stream_t stream) {
	using namespace flsgpu;
	if (n_vec == 0) { return FLS_OK; }
	if (!d_idx0 || !d_count0 || !d_idx1 || !d_count1 || !d_idx_out || !d_count_out) { return FLS_ERR_ARG; }
	Device* d = current_device();
	if (!d) { return FLS_ERR_CUDA; }
	k_selection_and<<<grid_for(n_vec), 256, 0, static_cast<cudaStream_t>(stream)>>>(
	    d_idx0, d_count0, d_idx1, d_count1, d_idx_out, d_count_out, n_vec, d->status);
	++launch_counter();
	return cudaGetLastError() == cudaSuccess ? FLS_OK : FLS_ERR_CUDA;
}

} // extern "C"
