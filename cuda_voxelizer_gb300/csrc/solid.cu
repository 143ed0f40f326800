// solid.cu -- solid voxelization kernels (reference: voxelize_triangle_solid,
// src/voxelize_solid.cu:16-145).
//
// The reference casts, for every voxel-centre column (y, z) inside a triangle's YZ projection, the
// column onto the triangle's plane and XORs every voxel x in [0, xmax] (:115-135): O(g) single-bit
// atomics per column hit, and parity along +x yields the solid.  The engine computes the same
// column hits with the same arithmetic, but records each hit as two toggles in a linear-order flip
// table (the start of the row and xmax + 1), then resolves all rows with one prefix-XOR pass and
// XORs the resolved bits into the caller's table (or scatters them into Morton order).  The XOR of
// any set of [0, xmax] ranges is exactly what this produces.
//
// Kernels, in launch order:
//   solid_classify      a warp per 32 triangles (staged by a bulk copy); the columns of the triangles
//                       with few columns are dealt over the warp, the other triangles queued.
//   solid_cols          persistent; each warp takes items of up to kColsPerItem columns in turn.
//   solid_resolve       linear jobs: a warp per run of whole rows, 128 words at a time: prefix XOR
//                       along x, XORed into the linear table (every word stored, for
//                       JOB_TABLE_OVERWRITE jobs), flip table cleared.
//   solid_morton_cols   Morton jobs with g >= 32: a warp resolves row groups of 4 x 4 rows along x and
//                       converts them to Morton words in registers.
//   solid_morton_small  Morton jobs with g < 32 (one word at a time), then solid_zero clears the
//                       flip table.
#include <algorithm>

#include "engine.h"
#include "morton_block.cuh"
#include "stage.cuh"

namespace cvx {

namespace {

constexpr double kFloatError = 0.000001;  // src/voxelize_solid.cu:13 (a double literal)
// For a float f, (double)f < 0.000001 exactly when f <= 0x1.0c6f7ap-20f, the largest float below the
// double 1e-6 (floats are exact in double, and 0x1.0c6f7ap-20 < 1e-6 < its successor).
constexpr float kFloatErrorBelow = 0x1.0c6f7ap-20f;
static_assert((double)kFloatErrorBelow < kFloatError && (double)0x1.0c6f7cp-20f >= kFloatError,
              "kFloatErrorBelow is the largest float below the reference's float_error");

// floor((double)q - 0.5) and ceil(...) for a float q: q - 0.5f is exact in float when |q| < 2^22
// (its ulp is at most 0.5 there), so float floor/ceil give the double result; else use double.
__device__ __forceinline__ float floor_half(float q) {
	return fabsf(q) < 4194304.0f ? floorf(__fsub_rn(q, 0.5f)) : (float)floor((double)q - 0.5);
}
__device__ __forceinline__ float ceil_half(float q) {
	return fabsf(q) < 4194304.0f ? ceilf(__fsub_rn(q, 0.5f)) : (float)ceil((double)q - 0.5);
}
// floor_half / ceil_half of fl(a / u), using the reciprocal shortcut when the approximate
// quotient is clearly away from the decision boundary (the half-integers).
__device__ __forceinline__ float div_floor_half(float a, float u, float inv) {
	const float q = __fmul_rn(a, inv);
	const float h = __fsub_rn(q, 0.5f);
	const float f = floorf(h);
	const float room = 4.0f * __fmul_rn(fabsf(q), 1.1920929e-07f) + 1.0e-30f;
	if (fabsf(q) < 4194304.0f && h - f > room && (f + 1.0f) - h > room) return f;
	return floor_half(__fdiv_rn(a, u));
}
__device__ __forceinline__ float div_ceil_half(float a, float u, float inv) {
	const float q = __fmul_rn(a, inv);
	const float h = __fsub_rn(q, 0.5f);
	const float f = floorf(h);
	const float room = 4.0f * __fmul_rn(fabsf(q), 1.1920929e-07f) + 1.0e-30f;
	if (fabsf(q) < 4194304.0f && h - f > room && (f + 1.0f) - h > room) return f + 1.0f;
	return ceil_half(__fdiv_rn(a, u));
}

// int((double)q - 0.5) (truncation, saturating as cvt.rzi.s32.f64 does)
__device__ __forceinline__ int trunc_half(float q) {
	return fabsf(q) < 4194304.0f ? __float2int_rz(__fsub_rn(q, 0.5f)) : __double2int_rz((double)q - 0.5);
}

struct SolidTri {
	float nx, ny, nz;
	float v0x, v0y, v0z;
	float ax, ay, bx, by, cx, cy;  // v0_yz, v1_yz, v2_yz after the counter-clockwise swap
	int y0, y1, z0, z1;            // column range, clipped to the grid
	bool skip;
};

// Triangle setup, src/voxelize_solid.cu:83-119.
template <class P>
__device__ __forceinline__ void solid_setup(const float* t, const float* bmin, const float* unit, const float* inv,
                                            const uint32_t* grid, SolidTri& S) {
	const float v0x = __fsub_rn(t[0], bmin[0]), v0y = __fsub_rn(t[1], bmin[1]), v0z = __fsub_rn(t[2], bmin[2]);
	const float v1x = __fsub_rn(t[3], bmin[0]), v1y = __fsub_rn(t[4], bmin[1]), v1z = __fsub_rn(t[5], bmin[2]);
	const float v2x = __fsub_rn(t[6], bmin[0]), v2y = __fsub_rn(t[7], bmin[1]), v2z = __fsub_rn(t[8], bmin[2]);
	const float e0x = __fsub_rn(v1x, v0x), e0y = __fsub_rn(v1y, v0y), e0z = __fsub_rn(v1z, v0z);
	const float e1x = __fsub_rn(v2x, v1x), e1y = __fsub_rn(v2y, v1y), e1z = __fsub_rn(v2z, v1z);
	const float cx = mul_sub<P::cross>(e0y, e1z, e0z, e1y);
	const float cy = mul_sub<P::cross>(e0z, e1x, e0x, e1z);
	const float cz = mul_sub<P::cross>(e0x, e1y, e0y, e1x);
	const float rlen = rsqrtf(dot3<P::dot3>(cx, cy, cz, cx, cy, cz));
	S.nx = __fmul_rn(cx, rlen);
	S.ny = __fmul_rn(cy, rlen);
	S.nz = __fmul_rn(cz, rlen);
	S.v0x = v0x; S.v0y = v0y; S.v0z = v0z;
	S.skip = fabsf(S.nx) <= kFloatErrorBelow;  // :92, (double)|n.x| < 1e-6 (the thread returns)
	// YZ projection, made counter-clockwise (:95-105; checkCCW :55-64)
	float ax = v0y, ay = v0z, bx = v1y, by = v1z, qx = v2y, qy = v2z;
	const float ccw = mul_sub<P::ccw>(__fsub_rn(bx, ax), __fsub_rn(qy, ay), __fsub_rn(qx, ax), __fsub_rn(by, ay));
	if (!(ccw > 0.0f)) {
		float tx = bx, ty = by;
		bx = qx; by = qy; qx = tx; qy = ty;
	}
	S.ax = ax; S.ay = ay; S.bx = bx; S.by = by; S.cx = qx; S.cy = qy;
	// column range (:109-119): floor/ceil(q - 0.5) evaluated in double, loop y from (int)min while
	// (float)y <= max.  Columns outside the grid are dropped (the reference writes them outside the
	// table or into neighbouring rows).
	const float mxy = fmaxf(ax, fmaxf(bx, qx)), mxz = fmaxf(ay, fmaxf(by, qy));
	const float mny = fminf(ax, fminf(bx, qx)), mnz = fminf(ay, fminf(by, qy));
	const float gmaxy = div_floor_half(mxy, unit[1], inv[1]);
	const float gmaxz = div_floor_half(mxz, unit[2], inv[2]);
	const float gminy = div_ceil_half(mny, unit[1], inv[1]);
	const float gminz = div_ceil_half(mnz, unit[2], inv[2]);
	int y0 = __float2int_rz(gminy), z0 = __float2int_rz(gminz);
	// last integer y with (float)y <= gmax (gmax holds an integer value, or is not finite)
	int y1 = gmaxy >= 2147483520.0f ? 2147483647 : (gmaxy >= -2147483648.0f ? (int)gmaxy : (-2147483647 - 1));
	int z1 = gmaxz >= 2147483520.0f ? 2147483647 : (gmaxz >= -2147483648.0f ? (int)gmaxz : (-2147483647 - 1));
	if (!(gmaxy == gmaxy)) y1 = y0 - 1;  // NaN bound: the loop never runs
	if (!(gmaxz == gmaxz)) z1 = z0 - 1;
	S.y0 = max(y0, 0); S.z0 = max(z0, 0);
	S.y1 = min(y1, (int)grid[1] - 1); S.z1 = min(z1, (int)grid[2] - 1);
}

__device__ __forceinline__ bool top_left(float v0x, float v0y, float v1x, float v1y) {
	return (v1y < v0y) || (v1y == v0y && v0x > v1x);  // :67-70
}

// Column test for voxel-centre column (y, z): returns true and xmax on a hit (:119-123).  `morton`
// selects the contraction of get_x_coordinate the reference uses for that table order.
template <class P>
__device__ __forceinline__ bool column_hit(const SolidTri& S, const float* unit, int y, int z, bool morton, int& xmax) {
	// ((y + 0.5) * unit.y) in double then rounded to float == the float product of the exact y+0.5f
	// for |y| < 2^22 (the double product is exact, so both round the same real number once).
	const float px = __fmul_rn(__int2float_rn(y) + 0.5f, unit[1]);
	const float py = __fmul_rn(__int2float_rn(z) + 0.5f, unit[2]);
	// check_point_triangle (:24-46)
	const float PAx = __fsub_rn(px, S.ax), PAy = __fsub_rn(py, S.ay);
	const float PBx = __fsub_rn(px, S.bx), PBy = __fsub_rn(py, S.by);
	const float PCx = __fsub_rn(px, S.cx), PCy = __fsub_rn(py, S.cy);
	int check;
	const float t1 = mul_sub<P::pt>(PAx, PBy, PAy, PBx);
	const float t2 = mul_sub<P::pt>(PBx, PCy, PBy, PCx);
	const float t3 = mul_sub<P::pt>(PCx, PAy, PCy, PAx);
	if (fabsf(t1) <= kFloatErrorBelow && __fmul_rn(PAx, PBx) <= 0.0f && __fmul_rn(PAy, PBy) <= 0.0f) check = 1;
	else if (fabsf(t2) <= kFloatErrorBelow && __fmul_rn(PBx, PCx) <= 0.0f && __fmul_rn(PBy, PCy) <= 0.0f) check = 2;
	else if (fabsf(t3) <= kFloatErrorBelow && __fmul_rn(PCx, PAx) <= 0.0f && __fmul_rn(PCy, PAy) <= 0.0f) check = 3;
	else if (__fmul_rn(t1, t2) > 0.0f && __fmul_rn(t1, t3) > 0.0f) check = 0;
	else check = -1;
	const bool in = (check == 1 && top_left(S.ax, S.ay, S.bx, S.by)) || (check == 2 && top_left(S.bx, S.by, S.cx, S.cy)) ||
	                (check == 3 && top_left(S.cx, S.cy, S.ax, S.ay)) || (check == 0);
	if (!in) return false;
	// get_x_coordinate (:49-52): -(n.y*(p.x - v0.y) + n.z*(p.y - v0.z)) / n.x + v0.x
	const float A = __fsub_rn(px, S.v0y), B = __fsub_rn(py, S.v0z);
	const float m = morton ? mul_add<P::getx_morton>(S.ny, A, S.nz, B) : mul_add<P::getx>(S.ny, A, S.nz, B);
	const float xh = __fadd_rn(__fdiv_rn(-m, S.nx), S.v0x);
	xmax = trunc_half(__fdiv_rn(xh, unit[0]));  // int(... / unit.x - 0.5), the 0.5 a double
	return true;
}

__device__ __forceinline__ void toggle(uint32_t* flips, uint64_t bit) { atomicXor(flips + (bit >> 5), bit_of(bit)); }

// Record column hit (y, z, xmax): the reference flips bits [0, xmax] of the column's row, i.e. the
// linear bit range [r*gx, r*gx + xmax]; a range longer than the row continues into the following
// rows (:124-135).  Morton order has no such continuation (x is encoded on its own), the range is
// clipped at the row end there (beyond it the reference writes outside the table).
__device__ __forceinline__ void record_hit(uint32_t* flips, const uint32_t* grid, bool morton, int y, int z, int xmax) {
	if (xmax < 0) return;
	const uint64_t gx = grid[0];
	const uint64_t rows = (uint64_t)grid[1] * grid[2];
	const uint64_t row = (uint64_t)y + (uint64_t)z * grid[1];
	const uint64_t len = (uint64_t)xmax + 1;
	if (morton || len <= gx) {
		toggle(flips, row * gx);
		const uint64_t e = len < gx ? len : gx;
		if (e < gx) toggle(flips, row * gx + e);
		return;
	}
	const uint64_t q = len / gx, rem = len % gx;
	for (uint64_t k = 0; k < q && row + k < rows; k++) toggle(flips, (row + k) * gx);
	if (rem && row + q < rows) {
		toggle(flips, (row + q) * gx);
		toggle(flips, (row + q) * gx + rem);
	}
}

// A small triangle's solid setup parked in shared memory between the classify phases.  16 words
// padded to 20: records stay 16-byte aligned for vector access, and the 8 lanes of a quarter warp
// touching 8 records start on banks 0, 20, 8, 28, 16, 4, 24, 12 -- no conflicts (at 16 words, 4-way).
struct __align__(16) SmallSolid {
	float nx, ny, nz, v0x, v0y, v0z, ax, ay, bx, by, cx, cy;
	int y0, z0;
	uint32_t nyc;    // columns along y
	uint32_t start;  // columns of the warp's triangles before this one
	uint32_t pad[4];
};
static_assert(sizeof(SmallSolid) == 80, "SmallSolid stride");

// Four independent warps per CTA, 32 triangles each; nothing waits on a CTA barrier.  Phase 1: one
// lane per triangle: setup, then the triangles of up to kColsPerSmall * small_cols columns park it in
// the warp's shared memory, packed, and the larger ones are queued for solid_cols.  Phase 2: the
// parked triangles' columns, 32 at a time, one per lane: a lane finds its triangle by counting the
// triangles that start at or before its column (one warp-wide OR of start bits and a population
// count), so no list of columns is written.
// Bound by instructions on large meshes, by latency on small ones.  A triangle that stays costs its
// columns; one that is queued costs solid_cols a chain of dependent loads and a second setup.  Times
// of solid_classify + solid_cols, triangles of up to 128 / up to 16 columns staying, in us:
//   icosphere 8 at 1024^3 77 + 12 / 150 + 81, 6 at 500^3 28 + 13 / 17 + 36 (10,240 and 640 CTAs).
// In a launch of few CTAs the split (classify_split) spreads the columns; a limit of 448 columns to a
// warp, with the rest left to solid_cols, gained nothing beside it.
// With item lists dealt over the CTA and 16 columns the same meshes took 150 + 76, 18 + 36, 12 + 21.
template <class P>
__global__ void __launch_bounds__(kTile, 12) solid_classify(const __grid_constant__ LaunchDesc L, const uint32_t small_cols,
                                                              const uint32_t split) {
	__shared__ __align__(16) union {
		float tri[32 * 9];
		SmallSolid small[32];
	} s_warp[kTile / 32];
	__shared__ __align__(8) uint64_t s_bar[kTile / 32];
	const uint32_t tile = blockIdx.x >> split;
	const uint32_t j = job_of_tile(L, tile);
	const JobDesc& J = job_at(L, j);
	const uint64_t n = J.n_tri;
	const bool morton = (J.flags & JOB_MORTON) != 0;
	const float bmin[3] = {J.bmin[0], J.bmin[1], J.bmin[2]};
	const float unit[3] = {J.unit[0], J.unit[1], J.unit[2]};
	const float inv[3] = {J.inv_unit[0], J.inv_unit[1], J.inv_unit[2]};
	const uint32_t grid[3] = {J.grid[0], J.grid[1], J.grid[2]};
	uint32_t* flips = J.flips;
	const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
	const uint32_t part = (blockIdx.x - (tile << split)) * (kTile / 32) + wid;
	const uint64_t t0 = (uint64_t)(tile - J.tile_begin) * kTile + part * (32u >> split);
	if (t0 >= n) return;
	auto& sm = s_warp[wid];
	const uint32_t cnt = (uint32_t)umin64(32u >> split, n - t0);
	if (!stage_warp(L, J.tris + t0 * 9, cnt, sm.tri, &s_bar[wid], (J.flags & JOB_PLAIN_LOADS) != 0)) return;  // error word set

	const bool valid = lane < cnt;
	float t[9];
#pragma unroll
	for (int k = 0; k < 9; k++) t[k] = valid ? sm.tri[lane * 9 + k] : 0.0f;
	__syncwarp();  // the triangles are consumed; the shared memory now holds records

	SolidTri S;
	bool is_mid = false, is_big = false;
	uint32_t n_items = 0, n_cols = 0;
	uint64_t ncols = 0;
	if (valid) {
		solid_setup<P>(t, bmin, unit, inv, grid, S);
		if (!S.skip && S.y0 <= S.y1 && S.z0 <= S.z1)
			ncols = (uint64_t)(S.y1 - S.y0 + 1) * (uint64_t)(S.z1 - S.z0 + 1);
	}
	if (ncols <= kColsPerSmall * small_cols) n_cols = (uint32_t)ncols;
	if (ncols > n_cols) {
		const uint64_t it = (ncols + kColsPerItem - 1) / kColsPerItem;
		n_items = (uint32_t)umin64(it, 0xFFFFFFu);
		is_mid = n_items == 1;
		is_big = n_items > 1;
	}
	const uint32_t lt = (1u << lane) - 1u;
	const uint32_t mid_ballot = __ballot_sync(FULL, is_mid);
	if (mid_ballot) {
		uint32_t base = 0;
		const uint32_t leader = __ffs(mid_ballot) - 1;
		if (lane == leader) base = atomicAdd(&L.scr.ctr->mid, (unsigned)__popc(mid_ballot));
		base = __shfl_sync(FULL, base, leader);
		const uint32_t slot = base + __popc(mid_ballot & lt);
		if (is_mid) {
			if (slot < L.scr.cap) L.scr.mid[slot] = MidRec{j, (uint32_t)(t0 + lane)};
			else set_error(L, kErrQueueOverflow);
		}
	}
	const uint32_t big_ballot = __ballot_sync(FULL, is_big);
	if (big_ballot) {
		uint32_t incl = is_big ? n_items : 0u;
#pragma unroll
		for (int d = 1; d < 32; d <<= 1) {
			const uint32_t v = __shfl_up_sync(FULL, incl, d);
			if (lane >= (uint32_t)d) incl += v;
		}
		const uint32_t total = __shfl_sync(FULL, incl, 31);
		unsigned long long old = 0;
		if (lane == 0)
			old = atomicAdd(&L.scr.ctr->big, ((unsigned long long)__popc(big_ballot) << kBigShift) | (unsigned long long)total);
		old = __shfl_sync(FULL, old, 0);
		if (is_big) {
			const uint32_t rec = (uint32_t)(old >> kBigShift) + __popc(big_ballot & lt);
			const uint64_t first = (old & kBigItemMask) + incl - n_items;
			if (rec < L.scr.cap && first + n_items <= kBigItemMask)
				L.scr.big[rec] = BigRec{first, j, (uint32_t)(t0 + lane), n_items, 0u};
			else
				set_error(L, kErrQueueOverflow);
		}
	}

	// Phase 2: columns of the small triangles (src/voxelize_solid.cu:115-139).
	uint32_t incl = n_cols;
#pragma unroll
	for (int d = 1; d < 32; d <<= 1) {
		const uint32_t v = __shfl_up_sync(FULL, incl, d);
		if (lane >= (uint32_t)d) incl += v;
	}
	const uint32_t total = __shfl_sync(FULL, incl, 31);
	const uint32_t start = incl - n_cols;
	const uint32_t parked = __ballot_sync(FULL, n_cols != 0u);
	if (n_cols) {
		SmallSolid& o = sm.small[__popc(parked & lt)];
		o.nx = S.nx; o.ny = S.ny; o.nz = S.nz; o.v0x = S.v0x; o.v0y = S.v0y; o.v0z = S.v0z;
		o.ax = S.ax; o.ay = S.ay; o.bx = S.bx; o.by = S.by; o.cx = S.cx; o.cy = S.cy;
		o.y0 = S.y0; o.z0 = S.z0;
		o.nyc = (uint32_t)(S.y1 - S.y0 + 1);
		o.start = start;
	}
	__syncwarp();
	uint32_t begun = 0;  // triangles that start before this step's columns
	for (uint32_t base = 0; base < total; base += 32) {
		const uint32_t at = start - base;
		const uint32_t starts = __reduce_or_sync(FULL, n_cols && at < 32u ? 1u << at : 0u);
		const uint32_t rec = begun + __popc(starts & (0xFFFFFFFFu >> (31u - lane))) - 1u;
		begun += __popc(starts);
		const uint32_t k = base + lane;
		if (k >= total) break;
		const SmallSolid& o = sm.small[rec];
		SolidTri T;
		T.nx = o.nx; T.ny = o.ny; T.nz = o.nz; T.v0x = o.v0x; T.v0y = o.v0y; T.v0z = o.v0z;
		T.ax = o.ax; T.ay = o.ay; T.bx = o.bx; T.by = o.by; T.cx = o.cx; T.cy = o.cy;
		// column c = dy + dz * nyc, c and nyc at most kColsPerSmall * kSmallCols = 128: the approximate
		// quotient is more than 1e-3 away from the next integer and truncates exactly
		const uint32_t c = k - o.start, nyc = o.nyc;
		const uint32_t dz = (uint32_t)__fdividef((float)c + 0.5f, (float)nyc);
		const int y = o.y0 + (int)(c - dz * nyc), z = o.z0 + (int)dz;
		int xmax;
		if (column_hit<P>(T, unit, y, z, morton, xmax)) record_hit(flips, grid, morton, y, z, xmax);
	}
}

template <class P>
__global__ void __launch_bounds__(kRowsThreads) solid_cols(const __grid_constant__ LaunchDesc L) {
	const uint32_t lane = threadIdx.x & 31u;
	Counters* C = L.scr.ctr;
	clear_next_counters(L);
	__shared__ unsigned long long s_bigc;  // read once per CTA (see surf_rows)
	__shared__ unsigned s_mid;
	if (threadIdx.x == 0) {
		s_bigc = *reinterpret_cast<volatile unsigned long long*>(&C->big);
		s_mid = *reinterpret_cast<volatile unsigned*>(&C->mid);
	}
	__syncthreads();
	const unsigned long long bigc = s_bigc;
	const uint32_t n_big = min((uint32_t)(bigc >> kBigShift), L.scr.cap);
	const uint64_t n_big_items = bigc & kBigItemMask;
	const uint32_t n_mid = min(s_mid, L.scr.cap);
	const uint64_t total = n_big_items + n_mid;
	// Items are of about the same size (at most kColsPerItem columns), so every warp takes its share in
	// turn, without a counter (the icosphere 5 at 1000^3, 60,000 items: 154 us -> 63 us).
	const uint32_t n_warps = gridDim.x * (blockDim.x >> 5);
	for (uint64_t tk = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); tk < total; tk += n_warps) {
		uint32_t job, tri, chunk, slices;
		if (!queue_item(L, tk, n_big, n_big_items, lane, job, tri, chunk, slices)) continue;
		const JobDesc& J = job_at(L, job);
		const float unit[3] = {J.unit[0], J.unit[1], J.unit[2]};
		const uint32_t grid[3] = {J.grid[0], J.grid[1], J.grid[2]};
		const bool morton = (J.flags & JOB_MORTON) != 0;
		uint32_t* flips = J.flips;
		float tv = lane < 9 ? J.tris[(uint64_t)tri * 9 + lane] : 0.0f;
		float t[9];
#pragma unroll
		for (int k = 0; k < 9; k++) t[k] = __shfl_sync(FULL, tv, k);
		SolidTri S;
		solid_setup<P>(t, J.bmin, unit, J.inv_unit, grid, S);
		const uint64_t nyc = (uint64_t)(S.y1 - S.y0 + 1);
		const uint64_t ncols = nyc * (uint64_t)(S.z1 - S.z0 + 1);
		const uint64_t c0 = (uint64_t)chunk * kColsPerItem;
		const uint64_t c1 = umin64(ncols, c0 + kColsPerItem);
		// column c is (y0 + c % nyc, z0 + c / nyc): one division for the lane's first column, then
		// steps of 32 columns (dz slices and dy rows, carrying y into z)
		const uint64_t cf = c0 + lane;
		if (cf < c1) {  // (no lane enters when the range is empty: nyc may be 0 then)
			const bool small = (ncols >> 32) == 0;
			int z = (int)(small ? (uint32_t)cf / (uint32_t)nyc : cf / nyc), y = (int)(cf - (uint64_t)z * nyc);
			const int dz = (int)(32u / (uint32_t)nyc), dy = 32 - dz * (int)nyc;
			y += S.y0;
			z += S.z0;
			for (uint64_t c = cf; c < c1; c += 32) {
				int xmax;
				if (column_hit<P>(S, unit, y, z, morton, xmax)) record_hit(flips, grid, morton, y, z, xmax);
				z += dz;
				y += dy;
				if (y > S.y1) {
					y -= (int)nyc;
					z++;
				}
			}
		}
	}
}

__device__ __forceinline__ uint32_t prefix_xor_msb(uint32_t t) {
	t ^= t >> 1;
	t ^= t >> 2;
	t ^= t >> 4;
	t ^= t >> 8;
	t ^= t >> 16;
	return t;
}

// XOR a resolved word into the table (the reference's semantics: the caller's table is XORed), or
// store it, zero or not, when the engine owns the table's content (JOB_TABLE_OVERWRITE).
__device__ __forceinline__ void xor_out(uint32_t* dest, uint64_t w, uint32_t v, bool overwrite) {
	if (overwrite) dest[w] = v;
	else if (v) dest[w] ^= v;
}

// Linear grids whose rows solid_resolve gives to one lane each.
constexpr uint32_t kLaneRow = 640;
__host__ __device__ __forceinline__ bool lane_rows(uint32_t gx) { return gx % 128u == 0 && gx <= kLaneRow; }

// Linear jobs: table ^= resolved bits, toggles cleared.  Morton jobs (g < 32): toggles replaced by
// the resolved bits for solid_morton_small to gather.
//
// One warp per unit of unit_words words, which begins with a row; the warp takes 128 consecutive
// words at a time, four per lane in one access.  A word's bits are the prefix XOR of its toggles,
// started again at every row start inside it; the bits before its first row start also take the
// parity carried in.  So a lane needs two bits of every lane before it -- its last bit, and whether a
// row starts in it -- and two ballots give both.  The same code serves rows that begin on words and
// rows that begin inside them.  Bound by memory: the flip table is read, the table read and written.
// Times here and of one thread per run of rows, which walked rows that begin inside words bit by bit:
// 100^3 6 / 37 us, 500^3 16 / 188 us, 1024^3 57 / 73 us.
//
// Short rows of whole 16-byte groups need less: a lane walks a row of its own, 32 rows to a unit, with a
// third of the instructions and no exchange.  The lanes then read 16 bytes of a row at a time and rely on
// the L1 for the rest of its sector, which long rows, or loads made ahead, push out.  Ten jobs of 512^3 at
// once 69 us (88 with the warp on consecutive words, 111 with the next load made ahead), forty of 256^3
// 49 / 70, one of 384^3 8 / 10, of 640^3 16 / 20; of 768^3 39 / 26, of 1024^3 92 / 57, hence kLaneRow.
// Six CTAs per SM at 40 registers with 12 B of spills; seven and eight spill more and are no faster.
__global__ void __launch_bounds__(256, 6) solid_resolve(const __grid_constant__ LaunchDesc L) {
	const uint32_t unit_id = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
	if (unit_id >= L.n_units) return;
	const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
	const uint32_t j = warp_job(L, unit_id, [](const JobDesc& d) { return (uint64_t)d.unit_begin; });
	const JobDesc& J = job_at(L, j);
	const uint32_t gx = J.grid[0];
	const uint64_t bits = (uint64_t)gx * J.grid[1] * J.grid[2];
	const bool morton = (J.flags & JOB_MORTON) != 0;
	const bool overwrite = (J.flags & JOB_TABLE_OVERWRITE) != 0 || morton;
	uint32_t* flips = J.flips;
	uint32_t* dest = morton ? flips : J.table;
	const bool vec = ((reinterpret_cast<uintptr_t>(flips) | reinterpret_cast<uintptr_t>(dest)) & 15u) == 0;
	const uint64_t w0 = (uint64_t)(unit_id - J.unit_begin) * J.unit_words;
	const uint64_t w1 = umin64((bits + 31) >> 5, w0 + J.unit_words);
	if (lane_rows(gx) && vec) {  // rows of the unit, one per lane
		uint64_t w = w0 + (uint64_t)lane * (gx >> 5);
		if (w >= w1) return;
		uint32_t in = 0u;  // all ones where the row's parity is odd
		for (const uint64_t end = w + (gx >> 5); w < end; w += 4) {
			const uint4 t = *reinterpret_cast<const uint4*>(flips + w);
			const bool toggles = (t.x | t.y | t.z | t.w) != 0u;
			uint4 r = make_uint4(in, in, in, in);
			if (toggles) {
				r.x ^= prefix_xor_msb(t.x), in = 0u - (r.x & 1u);
				r.y = prefix_xor_msb(t.y) ^ in, in = 0u - (r.y & 1u);
				r.z = prefix_xor_msb(t.z) ^ in, in = 0u - (r.z & 1u);
				r.w = prefix_xor_msb(t.w) ^ in, in = 0u - (r.w & 1u);
				*reinterpret_cast<uint4*>(flips + w) = make_uint4(0u, 0u, 0u, 0u);
			} else if (!overwrite && !in) {
				continue;
			}
			if (!overwrite) {
				const uint4 d = *reinterpret_cast<const uint4*>(dest + w);
				r.x ^= d.x, r.y ^= d.y, r.z ^= d.z, r.w ^= d.w;
			}
			*reinterpret_cast<uint4*>(dest + w) = r;
		}
		return;
	}
	const bool quad = gx % 128u == 0;
	const uint32_t step = 4096u % gx;         // bits of a warp's words, past whole rows
	uint32_t pos = (lane * 128u) % gx;        // position in its row of the lane's first bit
	uint32_t carry = 0;                       // parity of the row before the warp's words
	auto load = [&](uint64_t w) {
		if (vec && w + 4 <= w1) return *reinterpret_cast<const uint4*>(flips + w);
		return make_uint4(w < w1 ? flips[w] : 0u, w + 1 < w1 ? flips[w + 1] : 0u, w + 2 < w1 ? flips[w + 2] : 0u,
		                  w + 3 < w1 ? flips[w + 3] : 0u);
	};
	uint4 next = load(w0 + lane * 4u);
	for (uint64_t wc = w0; wc < w1; wc += 128) {
		const uint64_t w = wc + lane * 4u;
		const uint4 t4 = next;
		if (wc + 128 < w1) next = load(w + 128);
		const uint32_t t[4] = {t4.x, t4.y, t4.z, t4.w};
		uint32_t r[4] = {0u, 0u, 0u, 0u};
		const bool toggles = (t[0] | t[1] | t[2] | t[3]) != 0u;
		uint32_t p = pos;
		pos += step;
		if (pos >= gx) pos -= gx;
		if (carry || __any_sync(FULL, toggles)) {
			uint32_t in[4];       // the bits that the parity carried into the lane reaches
			uint32_t last = 0;    // the lane's last bit, for an even parity carried in
			bool starts = false;  // a row starts in the lane's words
			if (quad) {           // rows of whole 16-byte groups: a row starts with the lane's words or not at all
				starts = p == 0u;
#pragma unroll
				for (int k = 0; k < 4; k++) {
					r[k] = prefix_xor_msb(t[k]) ^ (0u - last);
					last = r[k] & 1u;
					in[k] = starts ? 0u : 0xFFFFFFFFu;
				}
			} else {
#pragma unroll
				for (int k = 0; k < 4; k++) {
					r[k] = prefix_xor_msb(t[k]);
					uint32_t m = 0xFFFFFFFFu;  // the bits before the word's first row start
					const uint32_t o0 = p ? gx - p : 0u;
					if (o0 < 32u) {
						m = ~(0xFFFFFFFFu >> o0);
						for (uint32_t o = o0; o < 32u; o += gx)
							if (o && ((r[k] >> (32u - o)) & 1u)) r[k] ^= 0xFFFFFFFFu >> o;
					}
					r[k] ^= last ? m : 0u;
					last = r[k] & 1u;
					in[k] = starts ? 0u : m;
					starts = starts || o0 < 32u;
					p += 32u;
					while (p >= gx) p -= gx;
				}
			}
			const uint32_t lasts = __ballot_sync(FULL, last != 0u), rows = __ballot_sync(FULL, starts);
			// parity at the end of the lanes in `from`: their last bits, back to the last row start
			auto parity = [&](uint32_t from) {
				const uint32_t s = rows & from;
				return s ? __popc(lasts & from & (0xFFFFFFFFu << (31 - __clz(s)))) & 1u : (__popc(lasts & from) & 1u) ^ carry;
			};
			const uint32_t c = parity(below);
			carry = parity(FULL);
			if (c) {
#pragma unroll
				for (int k = 0; k < 4; k++) r[k] ^= in[k];
			}
		}
		const uint32_t any = r[0] | r[1] | r[2] | r[3];
		if (vec && w + 4 <= w1) {
			if (overwrite || any) {
				if (!overwrite) {
					const uint4 d = *reinterpret_cast<const uint4*>(dest + w);
					r[0] ^= d.x; r[1] ^= d.y; r[2] ^= d.z; r[3] ^= d.w;
				}
				*reinterpret_cast<uint4*>(dest + w) = make_uint4(r[0], r[1], r[2], r[3]);
			}
			if (toggles && !morton) *reinterpret_cast<uint4*>(flips + w) = make_uint4(0u, 0u, 0u, 0u);
		} else {
#pragma unroll
			for (int k = 0; k < 4; k++)
				if (w + k < w1) {
					xor_out(dest, w + k, r[k], overwrite);
					if (t[k] && !morton) flips[w + k] = 0u;
				}
		}
	}
}

// Morton jobs with g >= 32: resolve, convert and clear in one pass, in registers.  A thread holds one
// linear word of 16 rows (4 y x 4 z: 16 Morton words, morton_block.cuh); the C = min(8, g / 32) lowest
// lane bits take neighbouring words of the rows, the others neighbouring 4 x 4 row groups, and the
// warp walks along x, C words at a time.  A word's incoming parity is the XOR of its row's earlier
// words' parities: the 16 rows' parities of a lane are one 16-bit mask, scanned over the C lanes with
// log2(C) shuffles.  Where no lane's words hold a toggle -- most of the inside and the outside of a
// solid -- every word is all zeros or all ones and nothing is scanned.  Bound by memory latency (the
// flip table read, the table read and written); the filled icosphere at 512^3 takes 12.6 us, 4.2 M
// warp instructions, where resolving 16 x 16-row slabs in shared memory and assembling words from
// their eight row pieces took 27.8 us and 19.2 M.  72 registers keep 512^3's 1,024 CTAs in one wave
// (7 per SM); at 64 (8 per SM) the kernel spills and takes 16 us.
constexpr uint32_t kMortonThreads = 128;

__global__ void __launch_bounds__(kMortonThreads, 7) solid_morton_cols(const __grid_constant__ LaunchDesc L) {
	const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	if (warp >= L.n_mwarps) return;
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t j = warp_job(L, warp, [](const JobDesc& d) { return d.mwarp_begin; });
	const JobDesc& J = job_at(L, j);
	const uint32_t lg = 31u - __clz(J.grid[0]);
	const MortonCols m = morton_cols(lg);
	const uint32_t C = 1u << m.lgc, col = lane & (C - 1u);
	uint32_t w, Y, Z;  // this lane's first word (w = col) and its row group
	morton_row_group(m, ((warp - J.mwarp_begin) << (5 - m.lgc)) + (lane >> m.lgc), Y, Z);
	uint32_t* flips = J.flips + ((((uint64_t)Z << (lg + 2)) + (Y << 2)) << m.lgw);
	uint32_t* table = J.table;
	const bool overwrite = (J.flags & JOB_TABLE_OVERWRITE) != 0;
	const bool vec = (reinterpret_cast<uintptr_t>(table) & 15u) == 0;
	uint32_t carry = 0;  // bit i: parity of row i = 4 * dz + dy before this chunk of words
	for (w = col; w < (1u << m.lgw); w += C) {
		uint32_t* src = flips + w;
		uint32_t t[16], any = 0;
#pragma unroll
		for (uint32_t i = 0; i < 16; i++) {
			t[i] = src[(((uint64_t)(i >> 2) << lg) + (i & 3u)) << m.lgw];
			any |= t[i];
		}
		uint32_t v[2][8];  // the resolved rows as rows_to_morton takes them
		if (__any_sync(FULL, any != 0u)) {
			uint32_t par = 0;  // bit i: parity of row i's word
#pragma unroll
			for (uint32_t i = 0; i < 16; i++) {
				if (t[i]) src[(((uint64_t)(i >> 2) << lg) + (i & 3u)) << m.lgw] = 0u;
				t[i] = prefix_xor_msb(t[i]);
				par = __funnelshift_r(par, t[i], 1);  // its last bit in at the top
			}
			par >>= 16;
			uint32_t incl = par;
			for (uint32_t d = 1; d < C; d <<= 1) {
				const uint32_t u = __shfl_up_sync(FULL, incl, d, C);
				if (col >= d) incl ^= u;
			}
			const uint32_t in = carry ^ incl ^ par;
			carry ^= __shfl_sync(FULL, incl, C - 1u, C);
#pragma unroll
			for (uint32_t i = 0; i < 16; i++)
				v[i >> 3][7 - (2 * (i & 3u) + ((i >> 2) & 1u))] = t[i] ^ (uint32_t)((int)(in << (31 - i)) >> 31);
		} else if (__any_sync(FULL, carry != 0u)) {
#pragma unroll
			for (uint32_t i = 0; i < 16; i++)
				v[i >> 3][7 - (2 * (i & 3u) + ((i >> 2) & 1u))] = (uint32_t)((int)(carry << (31 - i)) >> 31);
		} else {
			if (!overwrite) continue;
#pragma unroll
			for (uint32_t i = 0; i < 16; i++) v[i >> 3][i & 7u] = 0u;
		}
		rows_to_morton(v[0]);
		rows_to_morton(v[1]);
		uint32_t* dst = table + morton_col_base(w, Y, Z);
#pragma unroll
		for (uint32_t k = 0; k < 8; k += 2) {  // x groups k and k + 1: x3 = k bit 1, x4 = k bit 2
			uint4 o = make_uint4(v[0][7 - k], v[1][7 - k], v[0][6 - k], v[1][6 - k]);
			uint32_t* d = dst + 8 * (k & 2) + 32 * (k & 4);
			if (!overwrite && (o.x | o.y | o.z | o.w) == 0u) continue;
			if (vec) {
				if (!overwrite) {
					const uint4 q = *reinterpret_cast<const uint4*>(d);
					o = make_uint4(o.x ^ q.x, o.y ^ q.y, o.z ^ q.z, o.w ^ q.w);
				}
				*reinterpret_cast<uint4*>(d) = o;
			} else {
				xor_out(d, 0, o.x, overwrite);
				xor_out(d, 1, o.y, overwrite);
				xor_out(d, 2, o.z, overwrite);
				xor_out(d, 3, o.w, overwrite);
			}
		}
	}
}

// Morton jobs with g < 32: one Morton word per thread, 32 codes decoded one by one.
__global__ void __launch_bounds__(256) solid_morton_small(const __grid_constant__ LaunchDesc L) {
	const uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (idx >= L.n_mwords) return;
	const uint32_t j = job_search(L, idx, [](const JobDesc& d) { return d.mword_begin; });
	const JobDesc& J = job_at(L, j);
	const uint64_t m = idx - J.mword_begin;
	const uint64_t g = J.grid[0];
	const uint32_t* flips = J.flips;
	uint32_t out = 0;
	const uint64_t total = g * g * g;
	for (uint32_t i = 0; i < 32; i++) {
		const uint64_t c = m * 32 + i;
		if (c >= total) break;
		const uint64_t x = compact3(c), y = compact3(c >> 1), z = compact3(c >> 2);
		const uint64_t lin = x + g * (y + g * z);
		out |= ((flips[lin >> 5] >> (31u - (uint32_t)(lin & 31u))) & 1u) << (31u - i);
	}
	xor_out(J.table, m, out, (J.flags & JOB_TABLE_OVERWRITE) != 0);
}

// Morton jobs with g < 32: clear the resolved flip table, one warp per resolve unit
// (solid_morton_cols clears its own words).
__global__ void __launch_bounds__(256) solid_zero(const __grid_constant__ LaunchDesc L) {
	const uint32_t unit_id = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
	if (unit_id >= L.n_units) return;
	const uint32_t j = warp_job(L, unit_id, [](const JobDesc& d) { return (uint64_t)d.unit_begin; });
	const JobDesc& J = job_at(L, j);
	if (!(J.flags & JOB_MORTON)) return;
	const uint64_t words = ((uint64_t)J.grid[0] * J.grid[1] * J.grid[2] + 31) >> 5;
	const uint64_t w0 = (uint64_t)(unit_id - J.unit_begin) * J.unit_words, w1 = umin64(words, w0 + J.unit_words);
	for (uint64_t w = w0 + (threadIdx.x & 31u); w < w1; w += 32) J.flips[w] = 0u;
}

}  // namespace

SolidUnits solid_units(const uint32_t grid[3]) {
	const uint64_t words = ((uint64_t)grid[0] * grid[1] * grid[2] + 31) / 32;
	uint32_t a = grid[0], b = 32;
	while (b) { const uint32_t r = a % b; a = b; b = r; }
	uint32_t run = grid[0] / a;  // words of the shortest run of rows that begins and ends on words
	run *= run % 4 == 0 ? 1 : (run % 2 == 0 ? 2 : 4);
	const uint32_t target = words >= (1u << 23) ? 512 : (words >= (1u << 20) ? 256 : 128);
	SolidUnits s;
	s.unit_words = lane_rows(grid[0]) ? grid[0] : run * std::max(1u, target / run);
	s.units = (words + s.unit_words - 1) / s.unit_words;
	return s;
}

template <class P>
static cudaError_t launch_solid_t(const LaunchDesc& L, const Tune& tune, int cols_grid, cudaStream_t s, unsigned phases,
                                  const Prof* prof) {
	cudaError_t e = cudaSuccess;
	if (prof) (*prof)(nullptr, s);
	if ((phases & kSolidToggles) && L.n_tiles) {
		// split while there are fewer classify CTAs than solid_cols has (4 per SM; the classify kernel itself
		// holds 12: a line at its own residency has not been measured)
		const uint32_t split = classify_split(L.n_tiles, (uint32_t)cols_grid);
		solid_classify<P><<<L.n_tiles << split, kTile, 0, s>>>(L, std::min(tune.small_cols, kSmallCols), split);
		if ((e = cudaGetLastError()) != cudaSuccess) return e;
		if (prof) (*prof)("solid_classify", s);
		if ((e = launch_k(solid_cols<P>, (unsigned)cols_grid, kRowsThreads, 0, s, L)) != cudaSuccess) return e;
		if (prof) (*prof)("solid_cols", s);
	}
	if (phases & kSolidResolve) {
		if (L.n_units) {
			if ((e = launch_k(solid_resolve, (L.n_units + 7) / 8, 256, 0, s, L)) != cudaSuccess) return e;
			if (prof) (*prof)("solid_resolve", s);
		}
		if (L.n_mwarps) {
			if ((e = launch_k(solid_morton_cols, (unsigned)((L.n_mwarps * 32 + kMortonThreads - 1) / kMortonThreads), kMortonThreads, 0, s, L)) != cudaSuccess) return e;
			if (prof) (*prof)("solid_morton_cols", s);
		}
		if (L.n_mwords) {
			if ((e = launch_k(solid_morton_small, (unsigned)((L.n_mwords + 255) / 256), 256, 0, s, L)) != cudaSuccess)
				return e;
			if ((e = launch_k(solid_zero, (L.n_units + 7) / 8, 256, 0, s, L)) != cudaSuccess) return e;
			if (prof) (*prof)("solid_morton_small", s);
		}
	}
	return cudaSuccess;
}

cudaError_t launch_solid(const LaunchDesc& L, const Tune& tune, int cols_grid, cudaStream_t s, unsigned phases,
                         const Prof* prof) {
	return launch_solid_t<RefFma>(L, tune, cols_grid, s, phases, prof);
}

int solid_cols_blocks_per_sm() {
	int n = 0;
	cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, solid_cols<RefFma>, kRowsThreads, 0);
	return n > 0 ? n : 1;
}

}  // namespace cvx
