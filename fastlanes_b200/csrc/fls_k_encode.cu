// Encoder-side kernels: transposing a column's vectors, deltas, FOR bases and bit widths, bit packing, and the packed
// vectors' offsets (generated::transpose / unrsum / ffor of the reference and ffor_analyze,
// src/cor/prm/ffor/ffor_analyze.cpp:77-102).
#include "fls_b200.h"
#include "fls_device.cuh"
#include "fls_runtime.h"
#include "fls_strings.cuh"

#include <type_traits>

namespace flsgpu {

namespace {

__host__ __device__ __forceinline__ uint32_t transposed_index(uint32_t o) {
	// inverse of original_index: o = 64a + 8b + c  ->  k = a + 16*O[b] + 128*c   (O is an involution)
	return (o / 64) + 16 * fls_order((o / 8) % 8) + 128 * (o % 8);
}

// Original to transposed order, a warp a vector.  A vector is a matrix of 16 blocks of 64 values in original order;
// transposed row m holds value O[m % 8] * 8 + m / 8 of every block.  The blocks go into shared memory as they come
// (16-byte loads) and leave as 16-byte pieces of transposed rows; column c of block i lies at c ^ tr_swz(i), which
// keeps 16-byte pieces whole and puts the values that a warp gathers at a time (rows m, m + 8, ... are neighbouring
// columns) on different banks.  HBM-bound: 16,385 vectors of u64 (268 MB moved) took 75 us with a thread a value
// reading 8 bytes 512 bytes apart, 43 us so.
template <typename T>
__device__ __forceinline__ uint32_t tr_swz(uint32_t i) {
	return sizeof(T) == 8 ? (i & 14u) : sizeof(T) == 4 ? (i & 12u) * 2 : sizeof(T) == 2 ? (i & 8u) * 2 : 0u;
}

constexpr uint32_t kTrWarps = 4;

template <typename T, bool ALIGNED>
__global__ void __launch_bounds__(kTrWarps * 32) k_transpose(const T* __restrict__ in, T* __restrict__ out, uint64_t n_vec) {
	constexpr uint32_t PER = 16 / sizeof(T), LPR = 16 / PER, ROWS = 32 / LPR; // values a piece, pieces a row, rows a step
	__shared__ __align__(16) T tile[kTrWarps][kVec];
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	const uint64_t v    = static_cast<uint64_t>(blockIdx.x) * kTrWarps + warp;
	if (v >= n_vec) { return; }
	T*       s   = tile[warp];
	const T* src = in + v * kVec;
	T*       dst = out + v * kVec;
	if constexpr (ALIGNED) {
		uint4 x[kVec / PER / 32];
#pragma unroll
		for (uint32_t j = 0; j < kVec / PER / 32; ++j) { x[j] = __ldg(reinterpret_cast<const uint4*>(src) + j * 32 + lane); }
#pragma unroll
		for (uint32_t j = 0; j < kVec / PER / 32; ++j) {
			const uint32_t e = (j * 32 + lane) * PER, i = e / 64;
			*reinterpret_cast<uint4*>(s + i * 64 + ((e % 64) ^ tr_swz<T>(i))) = x[j];
		}
	} else {
		for (uint32_t e = lane; e < kVec; e += 32) { s[(e / 64) * 64 + ((e % 64) ^ tr_swz<T>(e / 64))] = src[e]; }
	}
	__syncwarp();
#pragma unroll
	for (uint32_t j = 0; j < 64 / ROWS; ++j) {
		const uint32_t g = j * ROWS + lane / LPR, m = g / 8 + 8 * (g % 8), q = lane % LPR;
		const uint32_t c = fls_order(m % 8) * 8 + m / 8;
		union {
			T     t[PER];
			uint4 u;
		} p;
#pragma unroll
		for (uint32_t k = 0; k < PER; ++k) {
			const uint32_t i = q * PER + k;
			p.t[k]           = s[i * 64 + (c ^ tr_swz<T>(i))];
		}
		if constexpr (ALIGNED) {
			*reinterpret_cast<uint4*>(dst + m * 16 + q * PER) = p.u;
		} else {
#pragma unroll
			for (uint32_t k = 0; k < PER; ++k) { dst[m * 16 + q * PER + k] = p.t[k]; }
		}
	}
}

// Bit packing, a thread a lane of a vector: the lane's values in order through an accumulator, each word stored as it
// fills (lane l's word w at out[l + L * w], so loads and stores are 128-byte rows).  Reading every value once, 8 loads
// in flight, instead of walking the words and re-reading the values across their borders: 38.2 to 25.8 us for
// 16,385 vectors of u64 at 7 bits (134 MB read).
template <typename T, int W>
__global__ void k_ffor(const T* __restrict__ in, T* __restrict__ out, const uint8_t* __restrict__ bw,
                       const T* __restrict__ base, const uint64_t* __restrict__ byte_off, uint64_t n_vec) {
	constexpr uint32_t L = 1024 / W;
	using A              = typename std::conditional<W == 64, uint64_t, uint32_t>::type;
	const uint64_t i     = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
	if (i >= n_vec * L) { return; }
	const uint64_t v = i / L;
	const uint32_t l = static_cast<uint32_t>(i % L);
	const uint32_t b = bw[v];
	if (b == 0 || b > W) { return; }
	T*       o    = reinterpret_cast<T*>(reinterpret_cast<uint8_t*>(out) + (byte_off ? byte_off[v] : v * b * 128ull)) + l;
	const T  bs   = base ? base[v] : T(0);
	const T* src  = in + v * kVec + l;
	const A  mask = ~A(0) >> (8 * sizeof(A) - b);
	A        acc  = 0; // the word being filled (its low nb bits)
	uint32_t nb   = 0;
#pragma unroll 8
	for (uint32_t j = 0; j < static_cast<uint32_t>(W); ++j) {
		const A x = static_cast<A>(static_cast<T>(src[L * j] - bs)) & mask;
		acc |= x << nb;
		nb += b;
		if (nb >= W) {
			*o = static_cast<T>(acc);
			o += L;
			nb -= W;
			acc = nb ? x >> (b - nb) : A(0); // the value's bits past the word
		}
	}
}

template <typename T, int W>
__global__ void k_unrsum(const T* __restrict__ in, T* __restrict__ out, uint64_t n_vec) {
	constexpr uint32_t L = 1024 / W;
	const uint64_t     i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
	if (i >= n_vec * L) { return; }
	const uint64_t v = i / L;
	const uint32_t l = static_cast<uint32_t>(i % L);
	// lane l covers a contiguous run of original positions; walk it in order
	uint32_t start;
	if constexpr (W == 64) {
		start = l * 64;
	} else if constexpr (W == 32) {
		start = (l % 16) * 64 + 32 * (l / 16);
	} else {
		start = (l % 16) * 64 + fls_order(l / 16) * 8;
	}
	const T* src  = in + v * kVec;
	T*       dst  = out + v * kVec;
	T        prev = 0;
	for (uint32_t p = 0; p < static_cast<uint32_t>(W); ++p) {
		const uint32_t k = transposed_index(start + p);
		const T        x = src[k];
		dst[k]           = p == 0 ? T(0) : static_cast<T>(x - prev);
		prev             = x;
	}
}

template <typename T, int W>
__global__ void k_analyze(const T* __restrict__ in, uint8_t* __restrict__ bw, T* __restrict__ base, uint64_t n_vec,
                          bool is_signed) {
	// one warp per vector
	const uint64_t v    = static_cast<uint64_t>(blockIdx.x) * (blockDim.x / 32) + threadIdx.x / 32;
	const uint32_t lane = threadIdx.x & 31u;
	if (v >= n_vec) { return; }
	const T* src  = in + v * kVec;
	const T  flip = is_signed ? static_cast<T>(T(1) << (W - 1)) : T(0);
	T        mn = static_cast<T>(~T(0)), mx = 0;
	for (uint32_t k = lane; k < kVec; k += 32) {
		const T x = static_cast<T>(src[k] ^ flip);
		mn        = x < mn ? x : mn;
		mx        = x > mx ? x : mx;
	}
	for (int o = 16; o > 0; o >>= 1) {
		const T a = __shfl_xor_sync(0xFFFFFFFFu, mn, o);
		const T b = __shfl_xor_sync(0xFFFFFFFFu, mx, o);
		mn        = a < mn ? a : mn;
		mx        = b > mx ? b : mx;
	}
	if (lane == 0) {
		const uint64_t d = static_cast<uint64_t>(static_cast<T>(mx - mn));
		bw[v]            = static_cast<uint8_t>(d == 0 ? 0 : 64 - __clzll(static_cast<long long>(d)));
		base[v]          = static_cast<T>(mn ^ flip);
	}
}

// Byte offsets of densely packed vectors (bw[v] * 128 bytes each) and their total.  Every CTA takes a stretch of
// `per` vectors (a multiple of kPoTurn), 4 a thread and turn, and sums the widths before it itself: a byte a vector,
// 16 a load, is less to read than waiting for another CTA costs.  total[1]: whether a width is above max_bw (the last
// CTA reads them all).  One CTA scanning 16,385 widths took 13.8 us from cold caches; half a dozen small torch kernels
// before that, 35 us.
constexpr uint32_t kPoTurn = 4096;

__device__ __forceinline__ uint32_t block_sum_1024(uint32_t x, uint32_t* wsum) {
	const uint32_t lane = threadIdx.x & 31u;
	x                   = warp_sum(x);
	if (lane == 0) { wsum[threadIdx.x >> 5] = x; }
	__syncthreads();
	x = warp_sum(wsum[lane]);
	__syncthreads();
	return x;
}

__global__ void __launch_bounds__(1024) k_pack_offsets(const uint8_t* __restrict__ bw, uint64_t n, uint32_t max_bw,
                                                       uint64_t* __restrict__ off, uint64_t* __restrict__ total,
                                                       uint64_t per) {
	__shared__ uint32_t wsum[33];
	const uint32_t      tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
	const uint64_t      v0 = blockIdx.x * per, v1 = v0 + per < n ? v0 + per : n;
	const bool          wide = (reinterpret_cast<uintptr_t>(bw) & 15u) == 0, wide_out = (reinterpret_cast<uintptr_t>(off) & 15u) == 0;
	uint64_t            before = 0; // widths of the vectors before v0 (a multiple of kPoTurn)
	uint32_t            bad    = 0;
	for (uint64_t u0 = 0; u0 < v0; u0 += 1024 * 1024) { // sums of a turn fit 32 bits
		const uint64_t u1  = u0 + 1024 * 1024 < v0 ? u0 + 1024 * 1024 : v0;
		uint32_t       sum = 0;
		for (uint64_t u = u0 + tid * 16; u < u1; u += 1024 * 16) {
			__align__(16) uint8_t b[16];
			if (wide) {
				*reinterpret_cast<uint4*>(b) = __ldg(reinterpret_cast<const uint4*>(bw + u));
			} else {
#pragma unroll
				for (uint32_t i = 0; i < 16; ++i) { b[i] = bw[u + i]; }
			}
#pragma unroll
			for (uint32_t i = 0; i < 16; ++i) {
				sum += b[i];
				bad |= b[i] > max_bw ? 1u : 0u;
			}
		}
		before += block_sum_1024(sum, wsum);
	}
	for (uint64_t t0 = v0; t0 < v1; t0 += kPoTurn) {
		const uint64_t v = t0 + tid * 4;
		uint32_t       b[4], sum = 0;
#pragma unroll
		for (uint32_t i = 0; i < 4; ++i) {
			b[i] = v + i < v1 ? bw[v + i] : 0u;
			sum += b[i];
			bad |= b[i] > max_bw ? 1u : 0u;
		}
		const uint32_t inc = warp_inclusive_scan(sum, lane);
		if (lane == 31) { wsum[warp] = inc; }
		__syncthreads();
		if (warp == 0) {
			const uint32_t w  = wsum[lane];
			const uint32_t wi = warp_inclusive_scan(w, lane);
			wsum[lane]        = wi - w;
			if (lane == 31) { wsum[32] = wi; }
		}
		__syncthreads();
		const uint64_t o0 = (before + wsum[warp] + inc - sum) * 128, o1 = o0 + b[0] * 128ull, o2 = o1 + b[1] * 128ull,
		               o3 = o2 + b[2] * 128ull;
		before += wsum[32];
		if (wide_out && v + 4 <= v1) {
			*reinterpret_cast<ulonglong2*>(off + v)     = make_ulonglong2(o0, o1);
			*reinterpret_cast<ulonglong2*>(off + v + 2) = make_ulonglong2(o2, o3);
		} else {
			const uint64_t o[4] = {o0, o1, o2, o3};
#pragma unroll
			for (uint32_t i = 0; i < 4; ++i) {
				if (v + i < v1) { off[v + i] = o[i]; }
			}
		}
		__syncthreads(); // wsum is read to the end before the next turn
	}
	if (blockIdx.x + 1 == gridDim.x) {
		bad = __syncthreads_or(bad != 0) ? 1u : 0u;
		if (tid == 0) {
			total[0] = before * 128;
			total[1] = bad;
		}
	}
}

int to_status(cudaError_t e) { return e == cudaSuccess ? FLS_OK : FLS_ERR_CUDA; }

template <typename T>
int run_transpose(const T* in, T* out, uint64_t n_vec, fls_stream_t stream) {
	if (n_vec == 0) { return FLS_OK; }
	if (!in || !out) { return FLS_ERR_ARG; }
	const bool al = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0;
	const auto grid = static_cast<unsigned>((n_vec + kTrWarps - 1) / kTrWarps);
	if (al) {
		k_transpose<T, true><<<grid, kTrWarps * 32, 0, static_cast<cudaStream_t>(stream)>>>(in, out, n_vec);
	} else {
		k_transpose<T, false><<<grid, kTrWarps * 32, 0, static_cast<cudaStream_t>(stream)>>>(in, out, n_vec);
	}
	++launch_counter();
	return to_status(cudaGetLastError());
}

template <typename T, int W>
int run_ffor(const T* in, T* out, const uint8_t* bw, const T* base, const uint64_t* off, uint64_t n_vec,
             fls_stream_t stream) {
	if (n_vec == 0) { return FLS_OK; }
	if (!in || !out || !bw) { return FLS_ERR_ARG; }
	const uint64_t n = n_vec * (1024 / W);
	k_ffor<T, W><<<static_cast<unsigned>((n + 127) / 128), 128, 0, static_cast<cudaStream_t>(stream)>>>(in, out, bw,
	                                                                                                   base, off, n_vec);
	++launch_counter();
	return to_status(cudaGetLastError());
}

template <typename T, int W>
int run_unrsum(const T* in, T* out, uint64_t n_vec, fls_stream_t stream) {
	if (n_vec == 0) { return FLS_OK; }
	if (!in || !out || in == out) { return FLS_ERR_ARG; }
	const uint64_t n = n_vec * (1024 / W);
	k_unrsum<T, W><<<static_cast<unsigned>((n + 127) / 128), 128, 0, static_cast<cudaStream_t>(stream)>>>(in, out,
	                                                                                                     n_vec);
	++launch_counter();
	return to_status(cudaGetLastError());
}

template <typename T, int W>
int run_analyze(const T* in, uint8_t* bw, T* base, uint64_t n_vec, int is_signed, fls_stream_t stream) {
	if (n_vec == 0) { return FLS_OK; }
	if (!in || !bw || !base) { return FLS_ERR_ARG; }
	k_analyze<T, W><<<static_cast<unsigned>((n_vec + 7) / 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
	    in, bw, base, n_vec, is_signed != 0);
	++launch_counter();
	return to_status(cudaGetLastError());
}

} // namespace

} // namespace flsgpu

using namespace flsgpu;

extern "C" {

#define FLS_ENC(T, W)                                                                                                 \
	int fls_gpu_transpose_i_u##W(const T* in, T* out, uint64_t n, fls_stream_t s) {                                 \
		return run_transpose<T>(in, out, n, s);                                                                     \
	}                                                                                                               \
	int fls_gpu_ffor_u##W(const T* in, T* out, const uint8_t* bw, const T* base, const uint64_t* off, uint64_t n,   \
	                      fls_stream_t s) {                                                                         \
		return run_ffor<T, W>(in, out, bw, base, off, n, s);                                                        \
	}

FLS_ENC(uint8_t, 8)
FLS_ENC(uint16_t, 16)
FLS_ENC(uint32_t, 32)
FLS_ENC(uint64_t, 64)

#define FLS_ENC2(T, W)                                                                                                \
	int fls_gpu_unrsum_u##W(const T* in, T* out, uint64_t n, fls_stream_t s) { return run_unrsum<T, W>(in, out, n, s); } \
	int fls_gpu_analyze_u##W(const T* in, uint8_t* bw, T* base, uint64_t n, int sg, fls_stream_t s) {               \
		return run_analyze<T, W>(in, bw, base, n, sg, s);                                                           \
	}

FLS_ENC2(uint16_t, 16)
FLS_ENC2(uint32_t, 32)
FLS_ENC2(uint64_t, 64)

int fls_gpu_pack_offsets(const uint8_t* d_bw, uint64_t n_vec, uint32_t width, uint64_t* d_byte_off, uint64_t* d_total,
                         fls_stream_t stream) {
	if (!d_total || ((!d_bw || !d_byte_off) && n_vec)) { return FLS_ERR_ARG; }
	const Device* d = current_device();
	if (!d) { return FLS_ERR_CUDA; }
	// stretches of whole turns, as many as there are turns up to one a SM
	const uint64_t sms = static_cast<uint64_t>(d->sm_count), turns = (n_vec + kPoTurn - 1) / kPoTurn;
	const uint64_t per = kPoTurn * ((turns + sms - 1) / sms);
	const unsigned grid  = static_cast<unsigned>(per ? (n_vec + per - 1) / per : 1);
	k_pack_offsets<<<grid, 1024, 0, static_cast<cudaStream_t>(stream)>>>(d_bw, n_vec, width, d_byte_off, d_total, per);
	++launch_counter();
	return to_status(cudaGetLastError());
}

} // extern "C"
