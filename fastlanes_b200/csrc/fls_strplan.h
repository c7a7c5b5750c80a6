// Arguments of the string kernels (shared by the host string plan and fls_k_strings.cu).
#pragma once

#include "fls_plan.h"
#include <cstdint>
#include <cuda_runtime.h>

namespace flsgpu {

// FSST symbol table as the decoder uses it: symbol c (little-endian) and its length.
struct FsstTable {
	uint64_t sym[256];
	uint8_t  len[256];
};

// FSST12 symbol table (include/fls/cor/prm/fsst12/fsst12.h:74-79): 4096 codes of 12 bits, symbol c
// (little-endian) and its length.
struct Fsst12Table {
	uint64_t sym[4096];
	uint8_t  len[4096];
};

enum : uint8_t {
	STR_DICT  = 0, // rows are dictionary codes (DICT / DICT_RLE pages), dictionary FSST-decoded once per plan
	STR_FSST  = 1, // rows are FSST-compressed in the page (FSST pages)
	STR_BYTES = 2, // rows are plain bytes in the page (BYTE_ARR pages)
	STR_FSST12 = 3, // rows are FSST12-compressed in the page (FSST12 pages)
};

constexpr int      kStrMaxWarps   = 32;        // warps per CTA of the string kernels (at most)
constexpr int      kStrLenWarps   = 16;        // warps per CTA of the lengths pass
constexpr uint32_t kStrEndsSmemMax = 64 * 1024; // largest dictionary end-offset array copied to shared memory
// static shared memory of the FSST12 string kernels (the symbol table), taken from the dynamic budget
constexpr uint32_t kStrFsst12Smem = sizeof(Fsst12Table);

struct StrArgs {
	ColDesc          col; // the row stream: codes or cumulative end offsets, page layout
	uint8_t          kind;
	bool             dict_in_smem; // materialising pass: decoded dictionary bytes in shared memory
	bool             ends_in_smem; // lengths pass: dictionary end offsets in shared memory
	bool             rows16;       // DICT with fewer than 65535 entries: codes kept as 16-bit rows
	uint32_t         entry_c;
	const uint32_t*  dict_ends;
	// materialising pass: entry c as start | length << 24 (dictionaries of < 16 MiB decoded bytes whose
	// entries are all < 256 bytes), one load per row instead of two end offsets; null otherwise
	const uint32_t*  dict_rows;
	// FSST12 pages: every row's decoded length, written by the lengths pass and read by the materialising pass
	// instead of walking the row's codes a second time (null: both walk them)
	uint32_t*        row_len;
	const uint8_t*   dict_bytes;
	uint64_t         dict_bytes_n;
	const FsstTable* table;
	const Fsst12Table* table12; // FSST12 pages
	uint64_t*        vec_total;
	const uint64_t*  vec_base;
	uint32_t*        offsets;
	uint8_t*         bytes;
	uint64_t         bytes_cap;
	int*             status;
	uint64_t         item_base; // single-pass DICT decode: index of the column's vector 0 among the look-back words
	// single-pass DICT decode: the dictionary with every entry on an 8-byte boundary, zero between them, and entry c as
	// (start / 8) | length << 24
	const uint8_t*   dict8;
	const uint32_t*  rows8;
	uint64_t         dict8_n;
};

// One launch of the single-pass DICT decode (k_dict_pass) over the vectors of one or more DICT string columns.
// Every column has a ticket; a CTA stays with a column, its dictionary in shared memory, while the column's ticket has
// vectors left, and each of its warps takes them one by one; then it goes on to another column.  Every vector publishes
// its decoded byte total and, once its predecessors' totals are known, its inclusive prefix (a decoupled look-back within
// its column), so each vector learns its first output byte without a separate lengths pass.
struct StrSetArgs {
	const StrArgs*  cols;      // per-column arguments in device memory (each with dict8 and rows8)
	uint32_t        n_cols;
	uint32_t        active;    // warps of a CTA that take vectors (fewer for sets of fewer vectors than warps)
	uint64_t        n_items;   // vectors of all columns
	const uint64_t* first;     // the first vector of every column among all, and n_items behind them (one column: null)
	uint64_t*       flags;     // [0] the cursor over the columns, [1 + c] the ticket of column c, [1 + n_cols + item_base
	                           // + v] the look-back word of vector v; zeroed before every launch
	int*            status;
	uint32_t*       out_offsets; // one-column launches: the outputs (null: each column's own)
	uint8_t*        out_bytes;
	uint64_t        out_cap;
	uint32_t        dict_cap; // shared memory held for a dictionary's bytes (a multiple of 16)
};

// dynamic shared memory of a k_dict_pass CTA (227 KB less its static words)
constexpr uint32_t kDictPassSmem = 226 * 1024;
// of a warp of it beside its window: the vector's rows
constexpr uint32_t kDictRows16 = 2048 + 128, kDictRows32 = 4096 + 128;

constexpr uint32_t kDictWindow = 1536, kDictWideWindow = 2048; // a warp's output window

// Where k_dict_pass has its dictionaries: entries on 8-byte boundaries (dict8, rows8) in global or shared memory, or
// byte after byte (dict_bytes, dict_rows) in shared memory.
enum : uint32_t { DICT_GLOBAL, DICT_SMEM8, DICT_SMEM_PACKED };

struct DictLayout {
	uint32_t mode, warps, window;
	uint32_t dict_cap, smem; // shared memory held for the dictionary's bytes, and in all
};

// How a k_dict_pass CTA is laid out for dictionaries of at most `d8` bytes (entries padded to 8) or `packed` bytes
// (unpadded), `entries` entries and `mean` bytes an entry.  Measured on columns of 12,000 vectors (us):
//   window   2 KB costs warps, 1.5 KB splits the batches of long rows.  Entries of 40 to 60 bytes (2,000 of them): 267 with
//            27 warps of 2 KB, 355 with 31 of 1.5 KB; of 5 to 40 bytes (4,096): 191 with 25, 181 with 29.  So 2 KB for
//            means of 40 bytes on, and wherever 32 warps fit all the same (20 to 40 bytes, 300 entries: 198 against 204).
//   mode     whole 8-byte loads pay for entries of some length: 173 against 189 packed (5 to 40 bytes, 300 entries), 400
//            against 445 (5 to 20 bytes, 200 columns of 500 entries and 200 vectors), but 146 against 138 (9 bytes),
//            120 against 109 (1 byte).  The padding costs warps: 204 with 17 against 165
//            with 28 packed (6,000 of 17 bytes), 251 with 14 against 243 with 19 (6,000 of 5 to 40 bytes).  So padded
//            from 10 bytes on, if four fifths of the packed form's warps fit.
//   global   below about 13 warps the dictionary does better in the L1 and L2 caches: 302 against 409 with 8 (7,500
//            of 5 to 40 bytes), 224 against 323 with 8 (10,000 of 9 bytes, padded); with 18 warps 214 against 173
//            (18,000 of 5 bytes), with 14 304 against 251.
inline DictLayout dict_layout(uint64_t d8, uint64_t packed, uint64_t entries, uint64_t mean, bool rows16) {
	constexpr uint64_t kMinWarps = 13;
	const uint64_t     tab = (4 * entries + 15) & ~15ull;
	d8     = (d8 + 15) & ~15ull;
	packed = (packed + 15) & ~15ull;
	DictLayout l {};
	auto       warps = [&](uint64_t held) { // that fit beside `held` bytes
		const uint64_t w = held < kDictPassSmem ? (kDictPassSmem - held) / ((rows16 ? kDictRows16 : kDictRows32) + l.window) : 0;
		return w < static_cast<uint64_t>(kStrMaxWarps) ? w : static_cast<uint64_t>(kStrMaxWarps);
	};
	for (const uint32_t window : {kDictWideWindow, kDictWindow}) {
		l.window          = window;
		const uint64_t w8 = warps(d8 + tab), wp = warps(packed + tab);
		l.mode            = mean >= 10 && w8 >= kMinWarps && 5 * w8 >= 4 * wp ? DICT_SMEM8 : wp >= kMinWarps ? DICT_SMEM_PACKED : DICT_GLOBAL;
		l.dict_cap        = static_cast<uint32_t>(l.mode == DICT_SMEM8 ? d8 : l.mode == DICT_SMEM_PACKED ? packed : 0);
		const uint64_t held = l.mode == DICT_GLOBAL ? 0 : l.dict_cap + tab;
		l.warps           = static_cast<uint32_t>(warps(held));
		l.smem            = static_cast<uint32_t>(held) + l.warps * ((rows16 ? kDictRows16 : kDictRows32) + window);
		if (mean >= 40 || (l.mode != DICT_GLOBAL && l.warps == static_cast<uint32_t>(kStrMaxWarps))) { break; }
	}
	return l;
}
cudaError_t launch_dict_pass(const StrSetArgs& a, bool rows16, const DictLayout& l, cudaStream_t s, int sm_count = 0);

// The dictionary's entries (rows: start | length << 24) from bytes to their places in bytes8 (rows8), zero behind them.
cudaError_t launch_dict_align(const uint8_t* bytes, const uint32_t* rows, const uint32_t* rows8, uint32_t entry_c,
                              uint8_t* bytes8, cudaStream_t s);

cudaError_t launch_fsst_dict(const uint8_t* lens, const uint8_t* comp, uint64_t comp_size, uint32_t entry_c,
                             const FsstTable* tab, uint32_t* ends, uint8_t* bytes, uint64_t cap, int* status,
                             cudaStream_t s);
// sm_count: the device's SM count, or 0 to take it from the library's per-device state (current_device())
cudaError_t launch_str_lengths(const StrArgs& a, int sm_count, cudaStream_t s);
// Single-pass FSST / BYTE_ARR decode (k_stream_single): lb = a ticket word then one zeroed look-back word per
// vector; writes a.offsets / a.bytes (capacity a.bytes_cap).
cudaError_t launch_stream_single(const StrArgs& a, uint64_t* lb, cudaStream_t s, int sm_count = 0);
cudaError_t launch_scan_totals(const uint64_t* total, uint64_t* base, uint64_t n, cudaStream_t s);
// warps: warps per CTA (at most kStrMaxWarps); dyn_smem: warps * str_smem_per_warp(a.rows16) plus the
// 16-byte rounded dictionary bytes when a.dict_in_smem
cudaError_t launch_str_materialize(const StrArgs& a, int warps, uint32_t dyn_smem, cudaStream_t s, int sm_count = 0);
uint32_t    str_smem_per_warp(bool rows16);
// shared-memory bytes of the dictionary end offsets (16-byte rounded)
__host__ __device__ inline uint32_t str_ends_smem(const StrArgs& a) { return (a.entry_c * 4u + 15u) & ~15u; }

} // namespace flsgpu
