// transcode.cu -- Morton <-> linear conversion of a bit table (cubic power-of-two grids).
//
// The reference's writers read tables in linear order only (checkVoxel, src/util.h:25-38), and a
// Morton table (src/voxelize.cuh:20-34, bits MSB-first like the linear one) is written out raw
// (src/util_io.cpp:192-200).  These kernels let any caller move between the two layouts on the
// GPU.  A Morton word holds the codes 32m..32m+31: a 4 x 4 x 2 block of voxels (x and y in their two
// low bits, z in its low bit), i.e. eight 4-bit x-runs of eight linear rows.
#include <cuda_runtime.h>

#include "cvx.h"
#include "engine.h"
#include "morton_block.cuh"

namespace cvx {
namespace {

// g < 32 (several rows per linear word).  One thread per Morton word: gather the block's eight row nibbles from the linear table.
__global__ void __launch_bounds__(256) linear_to_morton(const uint32_t* __restrict__ lin, uint32_t* __restrict__ mor,
                                                        uint64_t words, uint32_t lg) {
	const uint64_t m = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (m >= words) return;
	const uint64_t code = m << 5;
	const uint64_t x0 = compact3(code), y0 = compact3(code >> 1), z0 = compact3(code >> 2);
	uint32_t out = 0;
#pragma unroll
	for (uint32_t dz = 0; dz < 2; dz++)
#pragma unroll
		for (uint32_t dy = 0; dy < 4; dy++) {
			const uint64_t bit = x0 + ((y0 + dy) << lg) + ((z0 + dz) << (2 * lg));
			const uint32_t nib = (lin[bit >> 5] >> (28u - (uint32_t)(bit & 31u))) & 0xFu;
			out |= nibble_mask(nib) >> (2u * (dy & 1u) + 4u * dz + 16u * (dy >> 1));
		}
	mor[m] = out;
}

// One thread per linear word (several rows): eight 4-voxel groups from eight Morton words.
__global__ void __launch_bounds__(256) morton_to_linear(const uint32_t* __restrict__ mor, uint32_t* __restrict__ lin,
                                                        uint64_t words, uint32_t lg) {
	const uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (w >= words) return;
	const uint32_t g = 1u << lg;
	uint32_t out = 0;
	for (uint32_t q = 0; q < 8; q++) {
		// voxel run q of this word: bits 4q..4q+3 (MSB first) are x .. x + 3 of row (y, z)
		const uint32_t b = (uint32_t)(w << 5) + 4 * q;
		const uint64_t code = morton3(b & (g - 1), (b >> lg) & (g - 1), b >> (2 * lg));
		const uint32_t word = mor[code >> 5], off = (uint32_t)(code & 31u);
		const uint32_t nib = (((word >> (31u - off)) & 1u) << 3) | (((word >> (30u - off)) & 1u) << 2) |
		                     (((word >> (23u - off)) & 1u) << 1) | ((word >> (22u - off)) & 1u);
		out |= nib << (28u - 4u * q);
	}
	lin[w] = out;
}

// g >= 32: one thread per column of one linear word in 16 rows, i.e. 16 Morton words in four runs of
// four, converted in registers (morton_block.cuh).  Bound by the L1's request rate (a warp's load
// touches four rows), close to memory: 1024^3 in 51 us, 268 MB at 5.2 TB/s (0.77 of a copy's rate);
// 16 x 16-row slabs in shared memory, each word assembled from its eight row pieces, took 125 us.
// Walking whole rows per CTA matters: with the words of a row far apart in the grid it took 96 us.
// kVec: both tables are 16-byte aligned, so a run of four Morton words is one access.
constexpr uint32_t kColThreads = 128;

template <bool kVec>
__global__ void __launch_bounds__(kColThreads) linear_to_morton_cols(const uint32_t* __restrict__ lin,
                                                                     uint32_t* __restrict__ mor, uint64_t columns,
                                                                     uint32_t lg) {
	const uint64_t t = (uint64_t)blockIdx.x * kColThreads + threadIdx.x;
	if (t >= columns) return;
	const MortonCols m = morton_cols(lg);
	uint32_t w, Y, Z;
	morton_column(m, t, w, Y, Z);
	const uint32_t* src = lin + ((((uint64_t)Z << (lg + 2)) + (Y << 2)) << m.lgw) + w;
	uint32_t v[2][8];
#pragma unroll
	for (uint32_t dz = 0; dz < 4; dz++)
#pragma unroll
		for (uint32_t dy = 0; dy < 4; dy++)
			v[dz >> 1][7 - (2 * dy + (dz & 1))] = src[(((uint64_t)dz << lg) + dy) << m.lgw];
	rows_to_morton(v[0]);
	rows_to_morton(v[1]);
	uint32_t* dst = mor + morton_col_base(w, Y, Z);
#pragma unroll
	for (uint32_t j = 0; j < 8; j += 2) {  // x3 = j bit 1, x4 = j bit 2
		const uint4 o = make_uint4(v[0][7 - j], v[1][7 - j], v[0][6 - j], v[1][6 - j]);
		uint32_t* d = dst + 8 * (j & 2) + 32 * (j & 4);
		if constexpr (kVec) {
			*reinterpret_cast<uint4*>(d) = o;
		} else {
			d[0] = o.x; d[1] = o.y; d[2] = o.z; d[3] = o.w;
		}
	}
}

template <bool kVec>
__global__ void __launch_bounds__(kColThreads) morton_to_linear_cols(const uint32_t* __restrict__ mor,
                                                                     uint32_t* __restrict__ lin, uint64_t columns,
                                                                     uint32_t lg) {
	const uint64_t t = (uint64_t)blockIdx.x * kColThreads + threadIdx.x;
	if (t >= columns) return;
	const MortonCols m = morton_cols(lg);
	uint32_t w, Y, Z;
	morton_column(m, t, w, Y, Z);
	const uint32_t* src = mor + morton_col_base(w, Y, Z);
	uint32_t v[2][8];
#pragma unroll
	for (uint32_t j = 0; j < 8; j += 2) {
		const uint32_t* d = src + 8 * (j & 2) + 32 * (j & 4);
		uint4 o;
		if constexpr (kVec) o = *reinterpret_cast<const uint4*>(d);
		else o = make_uint4(d[0], d[1], d[2], d[3]);
		v[0][7 - j] = o.x; v[1][7 - j] = o.y; v[0][6 - j] = o.z; v[1][6 - j] = o.w;
	}
	morton_to_rows(v[0]);
	morton_to_rows(v[1]);
	uint32_t* dst = lin + ((((uint64_t)Z << (lg + 2)) + (Y << 2)) << m.lgw) + w;
#pragma unroll
	for (uint32_t dz = 0; dz < 4; dz++)
#pragma unroll
		for (uint32_t dy = 0; dy < 4; dy++)
			dst[(((uint64_t)dz << lg) + dy) << m.lgw] = v[dz >> 1][7 - (2 * dy + (dz & 1))];
}

}  // namespace
}  // namespace cvx

using namespace cvx;

extern "C" cvx_status cvx_transcode(const uint32_t* d_src, uint32_t* d_dst, uint32_t gridsize, int to_morton,
                                    cvx_stream_t stream) {
	if (!d_src || !d_dst) {
		set_message("cvx_transcode: null argument");
		return CVX_ERR_INVALID_VALUE;
	}
	if (d_src == d_dst) {
		set_message("cvx_transcode: source and destination must not overlap");
		return CVX_ERR_INVALID_VALUE;
	}
	if (gridsize < 4 || (gridsize & (gridsize - 1)) || gridsize > (1u << 16)) {
		set_message("cvx_transcode: needs a cubic power-of-two grid between 4 and 65536");
		return CVX_ERR_UNSUPPORTED;
	}
	const uint32_t lg = 31u - (uint32_t)__builtin_clz(gridsize);
	const uint64_t words = ((uint64_t)gridsize * gridsize * gridsize) >> 5;
	const unsigned blocks = (unsigned)((words + 255) / 256);
	cudaStream_t s = (cudaStream_t)stream;
	const bool aligned = ((reinterpret_cast<uintptr_t>(d_src) | reinterpret_cast<uintptr_t>(d_dst)) & 15u) == 0;
	if (gridsize >= 32) {
		const uint64_t columns = words >> 4;
		const unsigned cb = (unsigned)((columns + kColThreads - 1) / kColThreads);
		if (to_morton) {
			if (aligned) linear_to_morton_cols<true><<<cb, kColThreads, 0, s>>>(d_src, d_dst, columns, lg);
			else linear_to_morton_cols<false><<<cb, kColThreads, 0, s>>>(d_src, d_dst, columns, lg);
		} else {
			if (aligned) morton_to_linear_cols<true><<<cb, kColThreads, 0, s>>>(d_src, d_dst, columns, lg);
			else morton_to_linear_cols<false><<<cb, kColThreads, 0, s>>>(d_src, d_dst, columns, lg);
		}
	} else if (to_morton) {
		linear_to_morton<<<blocks, 256, 0, s>>>(d_src, d_dst, words, lg);
	} else {
		morton_to_linear<<<blocks, 256, 0, s>>>(d_src, d_dst, words, lg);
	}
	const cudaError_t e = cudaGetLastError();
	if (e != cudaSuccess) {
		set_message(std::string("cvx_transcode: ") + cudaGetErrorString(e));
		return CVX_ERR_CUDA;
	}
	return CVX_OK;
}
