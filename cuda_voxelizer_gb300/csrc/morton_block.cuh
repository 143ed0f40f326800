// morton_block.cuh -- register-level conversion between linear rows and Morton words.
//
// A Morton word holds a 4 x 4 x 2 block of voxels (x and y in their two low bits, z in its low bit);
// a linear word holds 32 voxels of one row.  Eight rows (4 y x 2 z) of one linear word are the same
// 256 bits as the eight Morton words of its eight x groups, so the conversion is a permutation of
// the bits of eight registers.  Number those bits by (register r2 r1 r0, bit p4 p3 p2 p1 p0): the rows
// have (r, p) = (y1 y0 z0, x4 x3 x2 x1 x0), the Morton words (x4 x3 x2, y1 x1 z0 y0 x0) -- both up to
// a complement of every index bit, because bits are stored MSB first, which is why the callers number
// their registers downwards.  Four exchanges of one register-index bit with one bit-position bit do
// it:  y1 <-> x4 (p4), y0 <-> x1 (p1), x1 <-> x3 (p3), z0 <-> x2 (p2).  An exchange of halves or
// bytes is one byte permute per register, the others a shift and a three-input logic operation: 6
// instructions per word, where assembling a word from eight 4-bit row pieces took about 80.
// Each exchange is its own inverse, so Morton to linear runs them backwards.
#pragma once
#include "cvx_device.cuh"

namespace cvx {

// Exchange register-index bit (a: 0, b: 1) with bit-position bit K (positions with bit K set: M).
template <int K>
__device__ __forceinline__ void bit_exchange(uint32_t& a, uint32_t& b) {
	const uint32_t x = a, y = b;
	if constexpr (K == 4) {
		a = __byte_perm(x, y, 0x5410);  // low halves of both
		b = __byte_perm(x, y, 0x7632);  // high halves of both
	} else if constexpr (K == 3) {
		a = __byte_perm(x, y, 0x6240);
		b = __byte_perm(x, y, 0x7351);
	} else {
		constexpr uint32_t M = K == 2 ? 0xF0F0F0F0u : 0xCCCCCCCCu;
		a = (x & ~M) | ((y << (1 << K)) & M);
		b = (y & M) | ((x >> (1 << K)) & ~M);
	}
}

// Rows -> Morton words, in place.  In: v[7 - (2 * dy + dz)] is the row (dy, dz) of the linear word
// (dy < 4, dz < 2).  Out: v[7 - j] is the Morton word of x group j (x = 4j .. 4j + 3 of the word).
__device__ __forceinline__ void rows_to_morton(uint32_t v[8]) {
#pragma unroll
	for (int i = 0; i < 4; i++) bit_exchange<4>(v[i], v[i + 4]);
#pragma unroll
	for (int i = 0; i < 4; i++) bit_exchange<1>(v[(i & 1) + (i & 2) * 2], v[(i & 1) + (i & 2) * 2 + 2]);
#pragma unroll
	for (int i = 0; i < 4; i++) bit_exchange<3>(v[(i & 1) + (i & 2) * 2], v[(i & 1) + (i & 2) * 2 + 2]);
#pragma unroll
	for (int i = 0; i < 8; i += 2) bit_exchange<2>(v[i], v[i + 1]);
}

// Morton words -> rows: the inverse of rows_to_morton.
__device__ __forceinline__ void morton_to_rows(uint32_t v[8]) {
#pragma unroll
	for (int i = 0; i < 8; i += 2) bit_exchange<2>(v[i], v[i + 1]);
#pragma unroll
	for (int i = 0; i < 4; i++) bit_exchange<3>(v[(i & 1) + (i & 2) * 2], v[(i & 1) + (i & 2) * 2 + 2]);
#pragma unroll
	for (int i = 0; i < 4; i++) bit_exchange<1>(v[(i & 1) + (i & 2) * 2], v[(i & 1) + (i & 2) * 2 + 2]);
#pragma unroll
	for (int i = 0; i < 4; i++) bit_exchange<4>(v[i], v[i + 4]);
}

// How threads cover a table of g^3 voxels (g a power of two, at least 32): one thread holds a column
// of one linear word in 16 rows (4 y x 4 z), i.e. 16 Morton words, which lie in four runs of four
// (z1 and x2 are the two low bits of a Morton word's index).  The lowest thread bits take up to 8
// neighbouring words of a row, the next two neighbouring 4 x 4 row groups (y2, z2), so that a warp
// reads whole 32-byte sectors of rows and writes whole sectors of Morton words; then the rest of the
// row, so that a CTA reads whole rows; then the rest of y and of z.
struct MortonCols {
	uint32_t lg;    // log2(g)
	uint32_t lgw;   // log2(words per row)
	uint32_t lgc;   // log2(neighbouring words of a row in the lowest thread bits)
};
__host__ __device__ __forceinline__ MortonCols morton_cols(uint32_t lg) {
	MortonCols m;
	m.lg = lg;
	m.lgw = lg - 5;
	m.lgc = m.lgw < 3 ? m.lgw : 3;
	return m;
}

// Row group number q (of (g / 4)^2) -> (Y, Z) = (y / 4, z / 4), in the order y2, z2, the rest of y, the rest of z.
__device__ __forceinline__ void morton_row_group(const MortonCols& m, uint64_t q, uint32_t& Y, uint32_t& Z) {
	const uint64_t rest = q >> 2;
	Y = ((uint32_t)q & 1u) | ((uint32_t)rest & ((1u << (m.lg - 3)) - 1u)) << 1;
	Z = ((uint32_t)(q >> 1) & 1u) | (uint32_t)(rest >> (m.lg - 3)) << 1;
}

// Column t (of (g / 4)^2 * (g / 32)): its linear word w and row group (Y, Z) = (y / 4, z / 4).
__device__ __forceinline__ void morton_column(const MortonCols& m, uint64_t t, uint32_t& w, uint32_t& Y, uint32_t& Z) {
	const uint32_t whi = (uint32_t)(t >> (m.lgc + 2)) & ((1u << (m.lgw - m.lgc)) - 1u);
	w = ((uint32_t)t & ((1u << m.lgc) - 1u)) | whi << m.lgc;
	morton_row_group(m, ((t >> m.lgc) & 3u) | (t >> (m.lgw + 2)) << 2, Y, Z);
}

// First Morton word of the column at linear word w of row group (Y, Z); its 16 words are base + c +
// 16 * x3 + 128 * x4, c < 4 (c = z1 + 2 * x2).
__device__ __forceinline__ uint64_t morton_col_base(uint32_t w, uint32_t Y, uint32_t Z) {
	return morton3(w << 5, Y << 2, Z << 2) >> 5;
}

}  // namespace cvx
