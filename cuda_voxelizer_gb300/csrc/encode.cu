// encode.cu -- output encoders on the GPU: the binvox run-length payload and the .vox voxel list.
//
// Reference: write_binvox (src/util_io.cpp:202-246) walks the voxels with x outermost, then z, then
// y, and writes (value, count) byte pairs, a run ending where the value changes or after 255
// voxels; write_vox (src/util_io.cpp:249-285) walks x, then y over [0, gz), then z over [0, gy) and
// hands every set voxel to VoxWriter::AddVoxel as (x, gz - z, y).  Both read the table in linear
// order through checkVoxel (src/util.h:25-38).
//
// Both start from the same step: the table re-read in the writer's traversal order into a stream of
// bits (order_rows).  The stream is cut into tiles of kTileWords words, one CTA each; a first pass
// summarises every tile, one CTA turns the summaries into each tile's place in the output, and a
// second pass writes it.  The whole sequence is launched without waiting for the host; the caller's
// capacity is checked on the device, and the host reads the total once.
#include <cuda_runtime.h>

#include <string>

#include "cvx.h"
#include "engine.h"

namespace cvx {
namespace {

constexpr unsigned FULL = 0xFFFFFFFFu;
constexpr uint32_t kThreads = 256;
constexpr uint32_t kChunkWords = 8;                       // consecutive stream words of a thread
constexpr uint32_t kTileWords = kThreads * kChunkWords;
constexpr uint32_t kScanThreads = 1024;

// ---- the table in a writer's traversal order -------------------------------------------------
// Stream bit o = ((x * A) + a) * B + b for voxel (x, y, z), where (a, b) = (z, y) for binvox and
// (y, z) for the voxel list (A = gz, B = gy in both: y < gz, z < gy on the list's cubic grids).
// A row of the stream is the B bits of one (x, a); it begins on a word, `nib` words per row, and the
// bits after B in its last word are zero and do not count.  Grids with gy <= 16 that would waste
// more than half of every word are kept dense instead: one row of all the bits.
struct Order {
	uint32_t gx, A, B;    // extents of x, a, b
	uint64_t sa, sb;      // table bits from one a (b) to the next
	uint64_t n_bits;
	uint64_t row_bits;    // bits per row of the stream: B, or n_bits when dense
	uint64_t nib;         // words per row
	uint64_t words;       // words of the stream
	bool dense;
};

Order order_of(const cvx_voxinfo& v, bool inner_is_y) {
	Order o;
	const uint64_t gx = v.gridsize[0], gy = v.gridsize[1];
	o.gx = v.gridsize[0];
	o.A = v.gridsize[2];
	o.B = v.gridsize[1];
	o.sa = inner_is_y ? gx * gy : gx;
	o.sb = inner_is_y ? gx : gx * gy;
	o.n_bits = gx * gy * v.gridsize[2];
	o.dense = o.B <= 16;
	o.row_bits = o.dense ? o.n_bits : o.B;
	o.nib = (o.row_bits + 31) / 32;
	o.words = o.dense ? o.nib : gx * o.A * o.nib;
	return o;
}

__device__ __forceinline__ uint32_t voxel_bit(const uint32_t* table, uint64_t idx) {
	return (table[idx >> 5] >> (31u - (uint32_t)(idx & 31u))) & 1u;
}

// Dense streams: one thread per stream word, 32 gathered bits.
__global__ void __launch_bounds__(kThreads) order_gather(const uint32_t* __restrict__ table, uint32_t* __restrict__ out,
                                                         const __grid_constant__ Order O) {
	const uint64_t w = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
	if (w >= O.words) return;
	uint32_t word = 0;
	for (uint32_t i = 0; i < 32; i++) {
		const uint64_t o = (w << 5) + i;
		if (o >= O.n_bits) break;
		const uint64_t b = o % O.B, rest = o / O.B, a = rest % O.A, x = rest / O.A;
		word |= voxel_bit(table, x + a * O.sa + b * O.sb) << (31u - i);
	}
	out[w] = word;
}

// 32 x 32 bit transpose in registers (MSB first): bit 31 - j of v[i] becomes bit 31 - i of v[j].  Five
// exchanges of register-index bits with bit-position bits, as in morton_block.cuh.
__device__ __forceinline__ void transpose32(uint32_t v[32]) {
#pragma unroll
	for (int i = 0; i < 16; i++) {
		const uint32_t x = v[i], y = v[i + 16];
		v[i] = __byte_perm(y, x, 0x7632);
		v[i + 16] = __byte_perm(y, x, 0x5410);
	}
#pragma unroll
	for (int i = 0; i < 32; i++)
		if (!(i & 8)) {
			const uint32_t x = v[i], y = v[i + 8];
			v[i] = __byte_perm(y, x, 0x7351);
			v[i + 8] = __byte_perm(y, x, 0x6240);
		}
#pragma unroll
	for (int s = 4; s >= 1; s >>= 1) {
		const uint32_t m = s == 4 ? 0x0F0F0F0Fu : (s == 2 ? 0x33333333u : 0x55555555u);
#pragma unroll
		for (int i = 0; i < 32; i++)
			if (!(i & s)) {
				const uint32_t x = v[i], y = v[i + s];
				v[i] = (x & ~m) | ((y >> s) & m);
				v[i + s] = (y & m) | ((x << s) & ~m);
			}
	}
}

// One thread per block of 32 x by 32 inner coordinates of one outer coordinate: 32 row pieces in, 32
// stream words out.  The lowest thread bits take up to 8 inner blocks and 4 x blocks, so that a warp
// writes whole 32-byte sectors of the stream and reads neighbouring words of table rows.  kAligned: gx
// is a multiple of 32; otherwise a piece is cut from two words.  512^3: 10 us; 63 us with a warp
// ballot per bit, each warp reading one word of 32 rows and writing one word of 32 stream rows.
template <bool kAligned>
__global__ void __launch_bounds__(128) order_rows(const uint32_t* __restrict__ table, uint32_t* __restrict__ out,
                                                  const __grid_constant__ Order O) {
	const uint32_t nxb = (O.gx + 31u) >> 5, nib = (uint32_t)O.nib;
	const uint32_t nI = min(8u, nib), nX = min(4u, nxb), cI = (nib + nI - 1u) / nI, cX = (nxb + nX - 1u) / nX;
	uint32_t t = blockIdx.x * 128u + threadIdx.x;
	uint32_t ib = t % nI;
	t /= nI;
	uint32_t xb = t % nX;
	t /= nX;
	ib += (t % cI) * nI;
	t /= cI;
	xb += (t % cX) * nX;
	const uint32_t a = t / cX;
	if (a >= O.A || ib >= nib || xb >= nxb) return;
	const uint32_t rows = min(32u, O.B - (ib << 5));
	const uint64_t bit0 = ((uint64_t)xb << 5) + a * O.sa + ((uint64_t)ib << 5) * O.sb;
	uint32_t v[32];
#pragma unroll
	for (uint32_t i = 0; i < 32; i++) {
		v[i] = 0u;
		if (i < rows) {
			const uint64_t bit = bit0 + i * O.sb;
			if constexpr (kAligned) {
				v[i] = table[bit >> 5];
			} else {
				const uint64_t w = bit >> 5;
				const uint32_t s = (uint32_t)(bit & 31u);
				v[i] = __funnelshift_l(s && (w + 1) << 5 < O.n_bits ? table[w + 1] : 0u, table[w], s);
			}
		}
	}
	transpose32(v);
	uint32_t* dst = out + (((uint64_t)xb << 5) * O.A + a) * nib + ib;
	const uint32_t cols = min(32u, O.gx - (xb << 5));
	const uint64_t step = (uint64_t)O.A * nib;
#pragma unroll
	for (uint32_t j = 0; j < 32; j++)
		if (j < cols) dst[j * step] = v[j];
}

cudaError_t traversal_stream(const Order& O, const uint32_t* table, uint32_t* stream_words, cudaStream_t s) {
	if (O.dense) {
		order_gather<<<(unsigned)((O.words + kThreads - 1) / kThreads), kThreads, 0, s>>>(table, stream_words, O);
	} else {
		const uint64_t nxb = (O.gx + 31) / 32, nI = O.nib < 8 ? O.nib : 8, nX = nxb < 4 ? nxb : 4;
		const uint64_t threads = (O.nib + nI - 1) / nI * nI * ((nxb + nX - 1) / nX * nX) * O.A;
		const unsigned blocks = (unsigned)((threads + 127) / 128);
		if (O.gx % 32 == 0) order_rows<true><<<blocks, 128, 0, s>>>(table, stream_words, O);
		else order_rows<false><<<blocks, 128, 0, s>>>(table, stream_words, O);
	}
	return cudaGetLastError();
}

// Row of word w and the word's place in it (32-bit division, a fifth of the instructions, where it fits).
__device__ __forceinline__ void word_row(const Order& O, uint64_t w, uint64_t& row, uint64_t& ib) {
	if (O.words >> 32) {
		row = w / O.nib;
		ib = w % O.nib;
	} else {
		row = (uint32_t)w / (uint32_t)O.nib;
		ib = (uint32_t)w % (uint32_t)O.nib;
	}
}

// Stream position (bits) of word w, or the end of the stream.
__device__ __forceinline__ uint64_t word_pos(const Order& O, uint64_t w) {
	uint64_t row, ib;
	word_row(O, w, row, ib);
	return w < O.words ? row * O.row_bits + (ib << 5) : O.n_bits;
}

// ---- block scans ---------------------------------------------------------------------------------

struct Sum {
	__device__ uint64_t operator()(uint64_t a, uint64_t b) const { return a + b; }
};
struct Max {
	__device__ uint64_t operator()(uint64_t a, uint64_t b) const { return a > b ? a : b; }
};

// Exclusive scan over the CTA (identity 0) and the total over it.
template <uint32_t N, class Op>
__device__ __forceinline__ uint64_t block_exclusive(uint64_t v, uint64_t* s_warp, uint64_t* total, Op op) {
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	uint64_t incl = v;
#pragma unroll
	for (int d = 1; d < 32; d <<= 1) {
		const uint64_t u = __shfl_up_sync(FULL, incl, d);
		if (lane >= (uint32_t)d) incl = op(incl, u);
	}
	if (lane == 31) s_warp[warp] = incl;
	__syncthreads();
	if (warp == 0) {
		uint64_t w = lane < N / 32 ? s_warp[lane] : 0ull;
#pragma unroll
		for (int d = 1; d < 32; d <<= 1) {
			const uint64_t u = __shfl_up_sync(FULL, w, d);
			if (lane >= (uint32_t)d) w = op(w, u);
		}
		if (lane < N / 32) s_warp[lane] = w;
	}
	__syncthreads();
	*total = s_warp[N / 32 - 1];
	uint64_t excl = __shfl_up_sync(FULL, incl, 1);
	if (lane == 0) excl = 0;
	if (warp) excl = op(s_warp[warp - 1], excl);
	__syncthreads();  // s_warp is reused by the caller's next scan
	return excl;
}

// ---- binvox runs ---------------------------------------------------------------------------------
// A run starts where a bit differs from its predecessor (and at bit 0); a pair starts at every run
// start r and at r + 255, r + 510, ... within the run.  So the pairs that start in a tile depend on
// what precedes it only through the last run start before it.  Positions are kept as position + 1, 0
// for none.

// Pairs of the run started at r that start in [begin, end), r <= begin.
__device__ __forceinline__ uint64_t pairs_in(uint64_t r, uint64_t begin, uint64_t end) {
	return (end - r + 254) / 255 - (begin - r + 254) / 255;
}

// A thread's chunk of the stream: its words, and the value of the bit before it.
struct Chunk {
	uint64_t w0, n;        // words [w0, w0 + n)
	uint64_t ib;           // place of word w0 in its row
	uint64_t begin;        // position
	uint32_t cur[kChunkWords];
	uint32_t before;       // value of the bit before `begin` (the complement of the first bit at begin = 0)
};

// Bits of a word's row beyond the row's end, in the last word of a row.
__device__ __forceinline__ uint32_t pad_of(const Order& O) { return (uint32_t)(O.nib * 32u - O.row_bits); }

__device__ __forceinline__ void load_chunk(const Order& O, const uint32_t* __restrict__ st, uint64_t w0, Chunk& c) {
	c.w0 = w0;
	c.n = w0 < O.words ? umin64(kChunkWords, O.words - w0) : 0;
	uint64_t row;
	word_row(O, w0, row, c.ib);
	c.begin = c.n ? row * O.row_bits + (c.ib << 5) : O.n_bits;
	if (c.n == kChunkWords) {  // the stream buffer is 16-byte aligned, w0 a multiple of kChunkWords
		const uint4 p = reinterpret_cast<const uint4*>(st + w0)[0], q = reinterpret_cast<const uint4*>(st + w0)[1];
		c.cur[0] = p.x; c.cur[1] = p.y; c.cur[2] = p.z; c.cur[3] = p.w;
		c.cur[4] = q.x; c.cur[5] = q.y; c.cur[6] = q.z; c.cur[7] = q.w;
	} else {
#pragma unroll
		for (uint32_t i = 0; i < kChunkWords; i++) c.cur[i] = i < c.n ? st[w0 + i] : 0u;
	}
	if (w0 == 0) c.before = ~c.cur[0] >> 31;
	else if (c.n) c.before = (st[w0 - 1] >> (c.ib ? 0u : pad_of(O))) & 1u;
	else c.before = 0u;
}

// The run starts of the chunk's word i: bits that differ from their predecessor, and the bits of the
// row the word belongs to.  `prev`, `ib` walk along.
__device__ __forceinline__ uint32_t start_bits(const Order& O, uint32_t pad, const Chunk& c, uint32_t i, uint32_t& prev,
                                               uint64_t& ib, uint32_t& bits) {
	const bool row_end = ib + 1 == O.nib;
	const uint32_t cur = c.cur[i];
	uint32_t d = cur ^ ((cur >> 1) | (prev << 31));
	if (row_end) d &= ~0u << pad;
	prev = (cur >> (row_end ? pad : 0u)) & 1u;
	bits = row_end ? 32u - pad : 32u;
	ib = row_end ? 0 : ib + 1;
	return d;
}

struct ChunkRuns {
	uint64_t first = 0, last = 0;  // run starts in the chunk (position + 1)
	uint32_t pairs = 0;            // pairs that start from `first` on
	uint32_t bits = 0;             // bits of the chunk
};
__device__ __forceinline__ ChunkRuns chunk_runs(const Order& O, const Chunk& c) {
	ChunkRuns r;
	const uint32_t pad = pad_of(O);
	uint64_t ib = c.ib;
	uint32_t prev = c.before, first = ~0u, last = 0;
	uint32_t& at = r.bits;
#pragma unroll
	for (uint32_t i = 0; i < kChunkWords; i++) {
		if (i < c.n) {
			uint32_t bits;
			const uint32_t d = start_bits(O, pad, c, i, prev, ib, bits);
			if (d) {
				first = min(first, at + __clz(d));
				last = at + 32u - __ffs(d);
			}
			r.pairs += __popc(d);
			at += bits;
		}
	}
	// two starts of one chunk of at most 256 bits are at most 255 apart: one pair each; the last run may
	// have a second one, 255 bits on
	if (r.pairs) {
		r.first = c.begin + first + 1;
		r.last = c.begin + last + 1;
		r.pairs += at - last > 255u ? 1u : 0u;
	}
	return r;
}
// Pairs of a chunk, given the last run start before it (position + 1; 0: not known, only from its
// first run start on).
__device__ __forceinline__ uint64_t chunk_pairs(const ChunkRuns& r, const Chunk& c, uint64_t before) {
	return r.pairs + (before ? pairs_in(before - 1, c.begin, r.first ? r.first - 1 : c.begin + r.bits) : 0);
}

struct RunTile {
	uint64_t first, last;  // run starts of the tile (position + 1); then: last start before it, pairs before it
	uint64_t pairs;        // pairs that start from `first` on
};

__global__ void __launch_bounds__(kThreads) run_tiles(const uint32_t* __restrict__ st, const __grid_constant__ Order O,
                                                      RunTile* tiles) {
	__shared__ uint64_t s_warp[kThreads / 32];
	Chunk c;
	load_chunk(O, st, (uint64_t)blockIdx.x * kTileWords + threadIdx.x * kChunkWords, c);
	const ChunkRuns r = chunk_runs(O, c);
	uint64_t last, pairs, inv_first;
	const uint64_t before = block_exclusive<kThreads>(r.last, s_warp, &last, Max());
	block_exclusive<kThreads>(chunk_pairs(r, c, before), s_warp, &pairs, Sum());
	block_exclusive<kThreads>(r.first ? ~r.first : 0, s_warp, &inv_first, Max());
	if (threadIdx.x == 0) tiles[blockIdx.x] = RunTile{inv_first ? ~inv_first : 0, last, pairs};
}

// One CTA: every tile's last run start before it and pairs before it, in place; the total.
__global__ void __launch_bounds__(kScanThreads) run_scan(RunTile* tiles, uint64_t n, const __grid_constant__ Order O,
                                                         uint64_t* total_pairs) {
	__shared__ uint64_t s_warp[kScanThreads / 32];
	uint64_t last = 0, pairs = 0;  // before the tiles of this step
	for (uint64_t t0 = 0; t0 < n; t0 += kScanThreads) {
		const uint64_t t = t0 + threadIdx.x;
		RunTile m = {0, 0, 0};
		if (t < n) m = tiles[t];
		uint64_t step_last, step_pairs;
		uint64_t before = block_exclusive<kScanThreads>(m.last, s_warp, &step_last, Max());
		before = before ? before : last;
		uint64_t p = m.pairs;
		if (t < n && before)
			p += pairs_in(before - 1, word_pos(O, t * kTileWords), m.first ? m.first - 1 : word_pos(O, (t + 1) * kTileWords));
		const uint64_t off = pairs + block_exclusive<kScanThreads>(p, s_warp, &step_pairs, Sum());
		if (t < n) tiles[t] = RunTile{before, off, 0};
		if (step_last) last = step_last;
		pairs += step_pairs;
	}
	if (threadIdx.x == 0) *total_pairs = pairs;
}

// Writes the pairs that start in each tile.  A pair's length is the distance to the next pair, in the
// next chunk if need be, at most 255 voxels on.
__global__ void __launch_bounds__(kThreads) run_emit(const uint32_t* __restrict__ st, const __grid_constant__ Order O,
                                                     const RunTile* __restrict__ tiles,
                                                     const uint64_t* __restrict__ total_pairs, uint64_t capacity,
                                                     uint8_t* __restrict__ out) {
	__shared__ uint64_t s_warp[kThreads / 32];
	if (2 * *total_pairs > capacity) return;  // nothing is written into a buffer that is too small
	const RunTile tile = tiles[blockIdx.x];
	Chunk c;
	load_chunk(O, st, (uint64_t)blockIdx.x * kTileWords + threadIdx.x * kChunkWords, c);
	const ChunkRuns r = chunk_runs(O, c);
	uint64_t dummy;
	uint64_t before = block_exclusive<kThreads>(r.last, s_warp, &dummy, Max());
	before = before ? before : tile.first;
	uint64_t k = tile.last + block_exclusive<kThreads>(chunk_pairs(r, c, before), s_warp, &dummy, Sum());
	if (c.n == 0) return;
	// From here on positions are relative to the chunk, so 32 bits hold them.
	uint8_t* dst = out + 2 * k;
	const bool aligned = (reinterpret_cast<uintptr_t>(out) & 1u) == 0;
	uint32_t pending = ~0u;  // a pair whose length is not known yet: its position
	uint32_t pending_value = 0;
	auto pair_at = [&](uint32_t p, uint32_t value) {
		if (pending != ~0u) {
			const uint32_t len = p - pending;
			if (aligned) {
				*reinterpret_cast<uint16_t*>(dst) = (uint16_t)(pending_value | len << 8);
			} else {
				dst[0] = (uint8_t)pending_value;
				dst[1] = (uint8_t)len;
			}
			dst += 2;
		}
		pending = p;
		pending_value = value;
	};
	const uint32_t pad = pad_of(O);
	uint32_t value = c.before, prev = c.before, at = 0;
	uint32_t next = before ? (uint32_t)((before - 1) + (c.begin - (before - 1) + 254) / 255 * 255 - c.begin) : ~0u;  // the run's next pair
	uint64_t ib = c.ib;
#pragma unroll
	for (uint32_t i = 0; i < kChunkWords; i++) {
		if (i < c.n) {
			uint32_t bits;
			uint32_t d = start_bits(O, pad, c, i, prev, ib, bits);
			while (d) {
				const uint32_t j = __clz(d);  // MSB-first offset
				d &= ~(0x80000000u >> j);
				const uint32_t p = at + j;
				if (next < p) pair_at(next, value);  // at most one: the chunk has 256 bits
				value = (c.cur[i] >> (31u - j)) & 1u;
				pair_at(p, value);
				next = p + 255u;
			}
			at += bits;
		}
	}
	for (; next < at; next += 255) pair_at(next, value);
	if (pending == ~0u) return;
	// the pending pair ends at `next`, at the first bit after the chunk that differs, or at the stream's end
	uint32_t e = (uint32_t)umin64(next, O.n_bits - c.begin);
	for (uint64_t w = c.w0 + c.n; w < O.words && at < e; w++) {
		const bool row_end = ib + 1 == O.nib;
		uint32_t d = st[w] ^ (0u - value);
		if (row_end) d &= ~0u << pad;
		if (d) {
			e = min(e, at + __clz(d));
			break;
		}
		at += row_end ? 32u - pad : 32u;
		ib = row_end ? 0 : ib + 1;
	}
	pair_at(e, 0u);
}

// ---- voxel list ----------------------------------------------------------------------------------

__global__ void __launch_bounds__(kThreads) count_bits(const uint32_t* __restrict__ table, uint64_t n_bits,
                                                       unsigned long long* total) {
	__shared__ uint64_t s_warp[kThreads / 32];
	const uint64_t words = (n_bits + 31) >> 5;
	uint64_t n = 0, sum;
	for (uint64_t w = (uint64_t)blockIdx.x * kThreads + threadIdx.x; w < words; w += (uint64_t)gridDim.x * kThreads) {
		uint32_t v = table[w];
		if (w + 1 == words && (n_bits & 31u)) v &= ~0u << (32u - (uint32_t)(n_bits & 31u));
		n += __popc(v);
	}
	block_exclusive<kThreads>(n, s_warp, &sum, Sum());
	if (threadIdx.x == 0 && sum) atomicAdd(total, (unsigned long long)sum);
}

__global__ void __launch_bounds__(kThreads) voxel_tiles(const uint32_t* __restrict__ st, const __grid_constant__ Order O,
                                                        uint64_t* counts) {
	__shared__ uint64_t s_warp[kThreads / 32];
	uint32_t n = 0;
	for (uint32_t i = 0; i < kChunkWords; i++) {
		const uint64_t w = (uint64_t)blockIdx.x * kTileWords + i * kThreads + threadIdx.x;
		if (w < O.words) n += __popc(st[w]);
	}
	uint64_t sum;
	block_exclusive<kThreads>(n, s_warp, &sum, Sum());
	if (threadIdx.x == 0) counts[blockIdx.x] = sum;
}

// One CTA: exclusive sums of the tiles' counts, in place; the total.
__global__ void __launch_bounds__(kScanThreads) voxel_scan(uint64_t* counts, uint64_t n, uint64_t* total) {
	__shared__ uint64_t s_warp[kScanThreads / 32];
	uint64_t sum = 0;
	for (uint64_t t0 = 0; t0 < n; t0 += kScanThreads) {
		const uint64_t t = t0 + threadIdx.x;
		uint64_t step;
		const uint64_t off = sum + block_exclusive<kScanThreads>(t < n ? counts[t] : 0, s_warp, &step, Sum());
		if (t < n) counts[t] = off;
		sum += step;
	}
	if (threadIdx.x == 0) *total = sum;
}

// A warp takes 256 consecutive words, 32 at a time, and turns them into triples one word after another:
// a full word (most of a filled mesh) is 96 ints whose component and bit are the same for a lane each
// time; of any other word the lanes of the set bits put their triples into shared memory, from where they
// are written as consecutive ints.  Bound by instructions: 80 us for the filled icosphere at 512^3
// (20.7 M voxels, 248 MB written); 94 us with a list of every word's bits made by its lane, 327 us with a
// thread per word that wrote its triples one after another.
template <bool kDense>
__global__ void __launch_bounds__(kThreads) voxel_emit(const uint32_t* __restrict__ st, const __grid_constant__ Order O,
                                                       const uint64_t* __restrict__ offsets,
                                                       const uint64_t* __restrict__ total, uint64_t capacity,
                                                       int32_t* __restrict__ xyz) {
	__shared__ uint64_t s_warp[kThreads / 32];
	__shared__ int4 s_word[kThreads / 32][32];        // x, gz - first inner coordinate, a, first int
	__shared__ int32_t s_out[kThreads / 32][2 * 96];  // the triples of a word, twice
	if (*total > capacity) return;
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	const uint64_t w0 = (uint64_t)blockIdx.x * kTileWords + warp * (32u * kChunkWords);
	uint32_t n = 0;
#pragma unroll
	for (uint32_t i = 0; i < kChunkWords; i++) {
		const uint64_t w = w0 + i * 32u + lane;
		n += w < O.words ? __popc(st[w]) : 0u;
	}
	uint64_t sum;
	const uint64_t thread_off = block_exclusive<kThreads>(n, s_warp, &sum, Sum());
	int32_t* dst = xyz + 3 * (offsets[blockIdx.x] + __shfl_sync(FULL, thread_off, 0));  // of the warp's first word
	int4* info = s_word[warp];
	uint32_t half = 0;
#pragma unroll 1
	for (uint32_t i = 0; i < kChunkWords; i++) {
		const uint64_t w = w0 + i * 32u + lane;
		const uint32_t word = w < O.words ? st[w] : 0u;
		const uint32_t any = __ballot_sync(FULL, word != 0u);
		if (!any) continue;
		uint32_t full = kDense ? 0u : __ballot_sync(FULL, word == 0xFFFFFFFFu);
		const uint32_t cnt = 3u * __popc(word);
		uint32_t incl = cnt;
#pragma unroll
		for (int d = 1; d < 32; d <<= 1) {
			const uint32_t u = __shfl_up_sync(FULL, incl, d);
			if (lane >= (uint32_t)d) incl += u;
		}
		if constexpr (!kDense) {
			uint64_t row, ib;
			word_row(O, w, row, ib);
			const uint32_t x = (uint32_t)(O.words >> 32 ? row / O.A : (uint32_t)row / O.A);
			info[lane] = make_int4((int)x, (int)O.A - (int)((uint32_t)ib << 5), (int)((uint32_t)row - x * O.A), (int)(incl - cnt));
		} else {
			info[lane].w = (int)(incl - cnt);
		}
		__syncwarp();
		uint32_t part = any & ~full;
		while (full) {
			const uint32_t src = __ffs(full) - 1u;
			full &= full - 1u;
			const int4 c = info[src];
			int32_t* p = dst + c.w;
#pragma unroll
			for (uint32_t h = 0; h < 3; h++) {
				const uint32_t k = lane + 32u * h, comp = k % 3u;
				p[k] = comp == 0u ? c.x : (comp == 1u ? c.y - (int)(k / 3u) : c.z);  // AddVoxel(x, -z + gz, y)
			}
		}
		while (part) {
			const uint32_t src = __ffs(part) - 1u;
			part &= part - 1u;
			const uint32_t v = __shfl_sync(FULL, word, src);
			int4 c = info[src];
			if ((v >> (31u - lane)) & 1u) {
				int32_t* o = s_out[warp] + half + 3u * (lane ? __popc(v >> (32u - lane)) : 0u);
				if constexpr (kDense) {
					const uint64_t bit = ((w0 + i * 32u + src) << 5) + lane, rest = bit / O.B;
					c.x = (int)(rest / O.A);
					c.y = (int)O.A - (int)(bit % O.B) + (int)lane;
					c.z = (int)(rest % O.A);
				}
				o[0] = c.x;
				o[1] = c.y - (int)lane;
				o[2] = c.z;
			}
			__syncwarp();  // (the next word uses the other half: this one's readers are past the next barrier)
			const uint32_t m = 3u * __popc(v);
			int32_t* p = dst + c.w;
#pragma unroll
			for (uint32_t k = lane; k < 96u; k += 32)
				if (k < m) p[k] = s_out[warp][half + k];
			half ^= 96u;
		}
		dst += __shfl_sync(FULL, incl, 31);
		__syncwarp();
	}
}

// ---- scratch -------------------------------------------------------------------------------------

// The total, the tiles' summaries and the stream.  Both encoders' orders have the same size.
struct Layout {
	uint64_t tiles, off_tiles, off_stream, end;
};
Layout layout_of(const Order& O) {
	Layout l;
	l.tiles = (O.words + kTileWords - 1) / kTileWords;
	l.off_tiles = 256;
	l.off_stream = (l.off_tiles + l.tiles * sizeof(RunTile) + 255) / 256 * 256;
	l.end = (l.off_stream + O.words * 4 + 255) / 256 * 256;
	return l;
}

struct DevBuf {
	void* p = nullptr;
	cudaStream_t s;
	explicit DevBuf(cudaStream_t st) : s(st) {}
	cudaError_t alloc(size_t bytes) { return cudaMallocAsync(&p, bytes ? bytes : 16, s); }
	~DevBuf() {
		if (p) cudaFreeAsync(p, s);
	}
};

cvx_status invalid(const std::string& m) {
	set_message(m);
	return CVX_ERR_INVALID_VALUE;
}

cvx_status cuda_status(cudaError_t e, const char* what) {
	if (e == cudaSuccess) return CVX_OK;
	set_message(std::string(what) + ": " + cudaGetErrorString(e));
	return CVX_ERR_CUDA;
}

cvx_status check_info(const cvx_voxinfo* info, const void* table, const void* out_n, const char* fn) {
	if (!info || !table || !out_n) return invalid(std::string(fn) + ": null argument");
	for (int i = 0; i < 3; i++)
		if (info->gridsize[i] == 0) return invalid(std::string(fn) + ": gridsize has a zero dimension");
	return CVX_OK;
}

cvx_status check_list(const cvx_voxinfo* info) {
	if (info->gridsize[1] == info->gridsize[2]) return CVX_OK;
	// the reference's loops run y to gz and z to gy through checkVoxel's (x, y, z): only grids with
	// gy == gz stay inside the table
	set_message("cvx_encode_voxel_list: needs gridsize y == z");
	return CVX_ERR_UNSUPPORTED;
}

cvx_status check_ws(const cvx_voxinfo* info, const void* ws, uint64_t bytes, const char* fn) {
	if (!ws) return invalid(std::string(fn) + ": workspace is null");
	if (reinterpret_cast<uintptr_t>(ws) % 256) return invalid(std::string(fn) + ": workspace not 256-byte aligned");
	if (bytes < layout_of(order_of(*info, true)).end) return invalid(std::string(fn) + ": workspace too small");
	return CVX_OK;
}

#define CVX_TRY(expr, what)                                           \
	do {                                                              \
		const cvx_status st_ = cuda_status((expr), (what));           \
		if (st_ != CVX_OK) return st_;                                \
	} while (0)

cvx_status read_total(const uint64_t* d_total, uint64_t* n, cudaStream_t s) {
	CVX_TRY(cudaMemcpyAsync(n, d_total, 8, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
	CVX_TRY(cudaStreamSynchronize(s), "cudaStreamSynchronize");
	return CVX_OK;
}

cvx_status encode_binvox(const cvx_voxinfo& info, const uint32_t* d_table, char* ws, uint8_t* d_out, uint64_t capacity,
                         uint64_t* out_bytes, cudaStream_t s) {
	const Order O = order_of(info, true);
	const Layout l = layout_of(O);
	uint64_t* total = reinterpret_cast<uint64_t*>(ws);
	RunTile* tiles = reinterpret_cast<RunTile*>(ws + l.off_tiles);
	uint32_t* st = reinterpret_cast<uint32_t*>(ws + l.off_stream);
	CVX_TRY(traversal_stream(O, d_table, st, s), "binvox order");
	run_tiles<<<(unsigned)l.tiles, kThreads, 0, s>>>(st, O, tiles);
	run_scan<<<1, kScanThreads, 0, s>>>(tiles, l.tiles, O, total);
	if (d_out) run_emit<<<(unsigned)l.tiles, kThreads, 0, s>>>(st, O, tiles, total, capacity, d_out);
	CVX_TRY(cudaGetLastError(), "binvox runs");
	uint64_t pairs = 0;
	const cvx_status r = read_total(total, &pairs, s);
	if (r != CVX_OK) return r;
	*out_bytes = 2 * pairs;
	if (d_out && capacity < 2 * pairs) return invalid("cvx_encode_binvox: output buffer too small (see out_bytes)");
	return CVX_OK;
}

cvx_status encode_list(const cvx_voxinfo& info, const uint32_t* d_table, char* ws, int32_t* d_xyz, uint64_t capacity,
                       uint64_t* out_count, cudaStream_t s) {
	const Order O = order_of(info, false);
	const Layout l = layout_of(O);
	uint64_t* total = reinterpret_cast<uint64_t*>(ws);
	if (!d_xyz) {  // the count does not depend on the order
		CVX_TRY(cudaMemsetAsync(total, 0, 8, s), "cudaMemsetAsync");
		const uint64_t blocks = (O.n_bits / 32 + kTileWords) / kTileWords;
		count_bits<<<(unsigned)(blocks < 2048 ? blocks : 2048), kThreads, 0, s>>>(
		    d_table, O.n_bits, reinterpret_cast<unsigned long long*>(total));
		CVX_TRY(cudaGetLastError(), "count_bits");
		return read_total(total, out_count, s);
	}
	uint64_t* counts = reinterpret_cast<uint64_t*>(ws + l.off_tiles);
	uint32_t* st = reinterpret_cast<uint32_t*>(ws + l.off_stream);
	CVX_TRY(traversal_stream(O, d_table, st, s), "vox order");
	voxel_tiles<<<(unsigned)l.tiles, kThreads, 0, s>>>(st, O, counts);
	voxel_scan<<<1, kScanThreads, 0, s>>>(counts, l.tiles, total);
	if (O.dense) voxel_emit<true><<<(unsigned)l.tiles, kThreads, 0, s>>>(st, O, counts, total, capacity, d_xyz);
	else voxel_emit<false><<<(unsigned)l.tiles, kThreads, 0, s>>>(st, O, counts, total, capacity, d_xyz);
	CVX_TRY(cudaGetLastError(), "voxel list");
	const cvx_status r = read_total(total, out_count, s);
	if (r != CVX_OK) return r;
	if (capacity < *out_count) return invalid("cvx_encode_voxel_list: output buffer too small (see out_count)");
	return CVX_OK;
}

}  // namespace
}  // namespace cvx

using namespace cvx;

extern "C" {

uint64_t cvx_encode_workspace_size(const cvx_voxinfo* info) {
	if (!info || !info->gridsize[0] || !info->gridsize[1] || !info->gridsize[2]) return 0;
	return layout_of(order_of(*info, true)).end;
}

cvx_status cvx_encode_binvox_ws(const cvx_voxinfo* info, const uint32_t* d_table, void* d_ws, uint64_t ws_bytes,
                                uint8_t* d_out, uint64_t out_capacity, uint64_t* out_bytes, cvx_stream_t stream) {
	cvx_status st = check_info(info, d_table, out_bytes, "cvx_encode_binvox_ws");
	if (st == CVX_OK) st = check_ws(info, d_ws, ws_bytes, "cvx_encode_binvox_ws");
	if (st != CVX_OK) return st;
	return encode_binvox(*info, d_table, static_cast<char*>(d_ws), d_out, out_capacity, out_bytes, (cudaStream_t)stream);
}

cvx_status cvx_encode_binvox(const cvx_voxinfo* info, const uint32_t* d_table, uint8_t* d_out, uint64_t out_capacity,
                             uint64_t* out_bytes, cvx_stream_t stream) {
	const cvx_status st = check_info(info, d_table, out_bytes, "cvx_encode_binvox");
	if (st != CVX_OK) return st;
	DevBuf ws((cudaStream_t)stream);
	CVX_TRY(ws.alloc(cvx_encode_workspace_size(info)), "cudaMallocAsync");
	return encode_binvox(*info, d_table, static_cast<char*>(ws.p), d_out, out_capacity, out_bytes, (cudaStream_t)stream);
}

cvx_status cvx_encode_voxel_list_ws(const cvx_voxinfo* info, const uint32_t* d_table, void* d_ws, uint64_t ws_bytes,
                                    int32_t* d_xyz, uint64_t capacity, uint64_t* out_count, cvx_stream_t stream) {
	cvx_status st = check_info(info, d_table, out_count, "cvx_encode_voxel_list_ws");
	if (st == CVX_OK) st = check_list(info);
	if (st == CVX_OK) st = check_ws(info, d_ws, ws_bytes, "cvx_encode_voxel_list_ws");
	if (st != CVX_OK) return st;
	return encode_list(*info, d_table, static_cast<char*>(d_ws), d_xyz, capacity, out_count, (cudaStream_t)stream);
}

cvx_status cvx_encode_voxel_list(const cvx_voxinfo* info, const uint32_t* d_table, int32_t* d_xyz, uint64_t capacity,
                                 uint64_t* out_count, cvx_stream_t stream) {
	cvx_status st = check_info(info, d_table, out_count, "cvx_encode_voxel_list");
	if (st == CVX_OK) st = check_list(info);
	if (st != CVX_OK) return st;
	DevBuf ws((cudaStream_t)stream);
	CVX_TRY(ws.alloc(d_xyz ? cvx_encode_workspace_size(info) : 256), "cudaMallocAsync");
	return encode_list(*info, d_table, static_cast<char*>(ws.p), d_xyz, capacity, out_count, (cudaStream_t)stream);
}

}  // extern "C"
