// surface.cu -- surface voxelization kernels (reference: voxelize_triangle, src/voxelize.cu:58-190).
//
// Two kernels per launch sequence, both over a job table so that one mesh and a batch of meshes
// run through the same code:
//   surf_classify  a warp per 32 triangles of one job, staged into shared memory with one
//                  cp.async.bulk (TMA bulk copy) when aligned.  Each lane sets up its triangle;
//                  triangles of at most kLocalRows rows of at most kMaskRowVoxels voxels are finished
//                  by the warp, their rows dealt over its lanes, every voxel tested like in the
//                  reference; the others are queued, one record per triangle, as one item ("mid"),
//                  as one item per 4 to 32 z-slices ("big"), or, of few but long rows, in a queue of
//                  their own ("long").
//   surf_rows      persistent CTAs; each warp takes its share of the long triangles, up to 32 at a
//                  time, their rows dealt over its lanes; then work tickets (big items first, then
//                  mid triangles): it finds the bounds that the tests of the three projections put on the
//                  item's slices and rows, one test per slice or row instead of one per voxel row,
//                  narrows every row to its exact x-interval with the plane test and ORs it into the
//                  table one word at a time (the whole warp for long rows).  Jobs whose indices fit
//                  32 bits (JOB_NARROW) write with 32-bit index arithmetic.
#include "engine.h"
#include "stage.cuh"
#include "surface.cuh"

namespace cvx {

namespace {

// Triangles of few rows, each longer than kMaskRowVoxels but of at most kLongVoxels voxels, are queued for
// long_triangles: those of at most kLongRows rows, or of fewer rows than voxels in a row.  One by one as items of
// surf_rows 200,000 triangles in boxes of 17 x 3 x 3 voxels took 220 us (50 this way), of 60 x 6 x 6 223 / 140, the
// icosphere 7 on 4096 x 64 x 64 230 / 40; up to 64 rows whatever their length, icosphere 6 at 1000^3 86 us, 83
// with this rule.
constexpr uint32_t kLongRows = 32, kLongVoxels = 512;
constexpr uint32_t kCollectRows = 384;  // rows of a classify warp from which those that pass the YZ tests are collected
constexpr uint32_t kQueueRows = 64;     // fewer than 32 rows wait when 32 more are tested

// The place of row r = dy + dz * ny of a parked triangle, r and ny at most kLocalRows: the approximate quotient is
// more than 1e-3 away from the next integer and truncates exactly.
__device__ __forceinline__ void row_place(const float4& box, uint32_t r, int& y, int& z) {
	const uint32_t by = __float_as_uint(box.y), bz = __float_as_uint(box.z), ny = (by >> 24) + 1u;
	const uint32_t dz = (uint32_t)__fdividef((float)r + 0.5f, (float)ny);
	y = (int)((by & 0xFFFFFFu) + r - dz * ny);
	z = (int)((bz & 0xFFFFFFu) + dz);
}

// Four independent warps per CTA, 32 triangles each (fewer in a launch with few tiles); nothing waits
// on a CTA barrier.  Phase 1: one lane per triangle: setup, then the triangles of up to local_rows
// rows of up to kMaskRowVoxels voxels park it in the warp's shared memory, packed, and the larger ones
// are queued for surf_rows (or the brick kernels).  Phase 2: the parked triangles' rows, 32 at a time,
// one per lane: a lane finds its triangle by counting the triangles that start at or before its row
// (one warp-wide OR of start bits and a population count), and tests every voxel of its row.
// Where the triangles have many rows, about half fail the YZ tests, and a warp tests the voxels of 32
// rows that passed at a time: the 512^3 meshes of a 256-mesh mix 546 -> 507 us, its 256^3 meshes 356 ->
// 343.  With few rows most pass: the icosphere at 512^3 (125 rows a warp) takes 77 us that way, and 74 with
// one loop for both.
// Bound by instructions (82% of issue slots busy on the icosphere at 512^3, 45 per triangle).  There
// 71 us; 90 us with the rows listed in shared memory and dealt over the CTA behind three barriers, the
// tests combined with short-circuit branches (15% of all instructions) and the edge sums added up
// before they are compared.  Nine CTAs per SM at 56 registers; ten at 48 are 1% slower.
// Triangles with more rows cost less in surf_rows, which shares one setup over a warp, and so do those with
// longer ones, whose voxels need not all be tested (few such rows: long_triangles): with
// up to 256 rows of any length kept here, the soup of 300,000 at 300^3 took 148 + 642 us in the two
// kernels, 44 + 701 with this rule.  A warp keeps all such triangles, also in a launch of few CTAs:
// leaving those of a warp with more than 384 rows to surf_rows took 31 + 75 us instead of 43 + 37 on
// icosphere 6 at 700^3 (640 CTAs), 31 + 44 / 35 + 19 at 500^3, and the same on meshes of up to 160 CTAs.
template <class P, bool kDense>
__global__ void __launch_bounds__(kTile, 9) surf_classify(const __grid_constant__ LaunchDesc L, const uint32_t local_rows,
                                                             const uint32_t item_rows, const uint32_t split) {
	__shared__ __align__(16) union {
		float tri[32 * 9];
		SmallTri small[32];
	} s_warp[kTile / 32];
	__shared__ __align__(8) uint64_t s_bar[kTile / 32];
	__shared__ uint16_t s_queue[kTile / 32][kQueueRows];
	const uint32_t tile = blockIdx.x >> split;
	const uint32_t j = job_of_tile(L, tile);
	const JobDesc& J = job_at(L, j);
	const uint64_t n = J.n_tri;
	const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
	const uint32_t part = (blockIdx.x - (tile << split)) * (kTile / 32) + wid;
	const uint64_t t0 = (uint64_t)(tile - J.tile_begin) * kTile + part * (32u >> split);
	if (t0 >= n) return;
	uint32_t* table = J.table;
	const uint32_t jflags = J.flags;
	const float unit[3] = {J.unit[0], J.unit[1], J.unit[2]};
	const uint32_t grid[3] = {J.grid[0], J.grid[1], J.grid[2]};
	auto& sm = s_warp[wid];
	const uint32_t cnt = (uint32_t)umin64(32u >> split, n - t0);
	if (!stage_warp(L, J.tris + t0 * 9, cnt, sm.tri, &s_bar[wid], (jflags & JOB_PLAIN_LOADS) != 0)) return;  // error word set

	const bool valid = lane < cnt;
	float t[9];
#pragma unroll
	for (int k = 0; k < 9; k++) t[k] = valid ? sm.tri[lane * 9 + k] : 0.0f;
	__syncwarp();  // the triangles are consumed; the shared memory now holds records

	SurfTri S;
	uint32_t n_items = 0, n_rows = 0, slices = kZch;
	bool tiny = false;
	if (valid) {
		const float bmin[3] = {J.bmin[0], J.bmin[1], J.bmin[2]};
		const float inv[3] = {J.inv_unit[0], J.inv_unit[1], J.inv_unit[2]};
		surf_setup<P>(t, bmin, unit, inv, J.box_near, grid, S);
		const uint32_t ex = (uint32_t)(S.bx1 - S.bx0), ey = (uint32_t)(S.by1 - S.by0), ez = (uint32_t)(S.bz1 - S.bz0);
		const uint64_t rows = (uint64_t)(ey + 1) * (uint64_t)(ez + 1);
		while (slices > kMinSlices && (uint64_t)(ey + 1) * slices > item_rows) slices >>= 1;
		n_items = ez / slices + 1u;
		if (rows <= local_rows) {
			if (ex < kMaskRowVoxels) n_rows = (uint32_t)rows;
			else if (ex < kLongVoxels && rows <= max(kLongRows, ex)) slices = 0u;  // for long_triangles
		}
		tiny = plane_underflows(S.d1, S.d2);
	}
	uint32_t incl = n_rows;
#pragma unroll
	for (int d = 1; d < 32; d <<= 1) {
		const uint32_t v = __shfl_up_sync(FULL, incl, d);
		if (lane >= (uint32_t)d) incl += v;
	}
	const uint32_t total_rows = __shfl_sync(FULL, incl, 31);
	const uint32_t start = incl - n_rows;
	const uint32_t lt = (1u << lane) - 1u;
	const uint32_t parked = __ballot_sync(FULL, n_rows != 0u);
	if (n_rows) pack_small(S, start, sm.small[__popc(parked & lt)]);
	if (n_rows && tiny) {  // bounds of the plane test where its product may underflow
		SmallTri& o = sm.small[__popc(parked & lt)];
		plane_widen(S.nx, S.ny, S.nz, unit, o.q[4].z, o.q[4].w);
	}
	const bool queued = n_items && !n_rows;
	// Queue the other triangles: warp-aggregated appends.
	if (__any_sync(FULL, queued)) {
		const bool is_brick = queued && (jflags & JOB_BRICKS);  // rasterized in shared-memory bricks (bricks.cu)
		const bool is_long = queued && !is_brick && slices == 0u;
		const bool is_item = queued && !is_brick && slices != 0u;
		const bool is_mid = is_item && n_items == 1, is_big = is_item && n_items > 1;
		const uint32_t brick_ballot = __ballot_sync(FULL, is_brick);
		if (brick_ballot) {
			uint32_t base = 0;
			const uint32_t leader = __ffs(brick_ballot) - 1;
			if (lane == leader) base = atomicAdd(&L.scr.ctr->bq, (unsigned)__popc(brick_ballot));
			base = __shfl_sync(FULL, base, leader);
			const uint32_t slot = base + __popc(brick_ballot & lt);
			if (is_brick) {
				if (slot < L.scr.cap) L.scr.bq[slot] = MidRec{j, (uint32_t)(t0 + lane)};
				else set_error(L, kErrQueueOverflow);
			}
		}
		const uint32_t mid_ballot = __ballot_sync(FULL, is_mid), long_ballot = __ballot_sync(FULL, is_long);
		if (mid_ballot | long_ballot) {  // both counters with one atomic: 68 triangles of all sizes at 128^3 14.4 / 13.1 us
			unsigned long long base = 0;
			if (lane == 0)
				base = atomicAdd(reinterpret_cast<unsigned long long*>(&L.scr.ctr->mid),
				                 ((unsigned long long)__popc(long_ballot) << 32) | (unsigned long long)__popc(mid_ballot));
			base = __shfl_sync(FULL, base, 0);
			if (is_mid || is_long) {
				const uint32_t slot = is_mid ? (uint32_t)base + __popc(mid_ballot & lt) : (uint32_t)(base >> 32) + __popc(long_ballot & lt);
				if (slot < L.scr.cap) L.scr.mid[is_mid ? slot : L.scr.cap - 1u - slot] = MidRec{j, (uint32_t)(t0 + lane)};
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
					L.scr.big[rec] = BigRec{first, j, (uint32_t)(t0 + lane), n_items, slices};
				else
					set_error(L, kErrQueueOverflow);
			}
		}
	}

	// Phase 2: the rows of the parked triangles.
	__syncwarp();
	auto test_row = [&](const SmallTri& o, const float4& box, int y, int z) {
		const uint32_t bx = __float_as_uint(box.x);
		const int x0 = (int)(bx & 0xFFFFFFu);
		const uint32_t pm = row_mask<P>(o, unit[0], __fmul_rn(__int2float_rn(y), unit[1]), __fmul_rn(__int2float_rn(z), unit[2]),
		                                x0, (bx >> 24) + 1u);
		if (!pm) return;
		if (kDense && (jflags & JOB_DENSE))
			write_row_mask<true>(table, (jflags & JOB_MORTON) != 0, (jflags & JOB_NARROW) != 0, grid, y, z, x0, pm);
		else
			write_row_mask<false>(table, (jflags & JOB_MORTON) != 0, (jflags & JOB_NARROW) != 0, grid, y, z, x0, pm);
	};
	uint32_t begun = 0;  // triangles that start before this step's rows
	// Row k's triangle and its row of it, y and z; whether the row passes the YZ tests.  Every lane calls it.
	auto find_row = [&](uint32_t base, uint32_t& rec, uint32_t& r, float4& box, int& y, int& z) {
		const uint32_t at = start - base;
		const uint32_t starts = __reduce_or_sync(FULL, n_rows && at < 32u ? 1u << at : 0u);
		rec = begun + __popc(starts & (0xFFFFFFFFu >> (31u - lane))) - 1u;
		begun += __popc(starts);
		const uint32_t k = base + lane;
		if (k >= total_rows) return false;
		const SmallTri& o = sm.small[rec];
		box = o.q[0];
		r = k - __float_as_uint(box.w);
		row_place(box, r, y, z);
		return row_in_yz<P>(o, __fmul_rn(__int2float_rn(y), unit[1]), __fmul_rn(__int2float_rn(z), unit[2]));
	};
	uint32_t rec, r;
	float4 box;
	int y, z;
	if (total_rows < kCollectRows) {
		for (uint32_t base = 0; base < total_rows; base += 32)
			if (find_row(base, rec, r, box, y, z)) test_row(sm.small[rec], box, y, z);
		return;
	}
	uint16_t* queue = s_queue[wid];      // a ring of rows that passed
	uint32_t filled = 0, done = 0;       // rows put into it and taken out
	for (uint32_t base = 0; base < total_rows || done < filled;) {
		while (base < total_rows && filled - done < 32u) {
			const bool pass = find_row(base, rec, r, box, y, z);
			const uint32_t passed = __ballot_sync(FULL, pass);
			if (pass) queue[(filled + __popc(passed & lt)) % kQueueRows] = (uint16_t)(rec | r << 5);
			filled += __popc(passed);
			base += 32;
		}
		__syncwarp();
		if (done + lane < filled) {
			const uint32_t e = queue[(done + lane) % kQueueRows];
			const SmallTri& o = sm.small[e & 31u];
			box = o.q[0];
			row_place(box, e >> 5, y, z);
			test_row(o, box, y, z);
		}
		done = min(done + 32u, filled);
		__syncwarp();  // read before the places are filled again
	}
}

// Persistent CTAs of four warps; a warp takes one item (a triangle, or 4 to 32 z-slices of a larger one) at
// a time.  Lane = slice: the YZ tests' interval of y and the ZX tests' bounds on x.  Lane = y: the XY
// tests' bounds on x, into a table of the warp in shared memory (kRowsWindow values of y at a time).
// Then the item's rows, 32 at a time, one per lane: the row's slice is found by counting the slices that
// start at or before it, its bounds on x are read from both tables, the plane test narrows them to
// the row's exact interval, and the interval is ORed into the table.
// kGrouped: a warp claims up to kRowsGroup items and sets their triangles up at once, one per lane, in shared
// memory: the setup, a third of the instructions of an item of 100 rows, is paid once per group, and the
// loads it waits for come together.  An item alone costs 1 - 2 us more that way, so launches whose warps
// would claim one at a time do without.  Grouped / not: the 512^3 surface meshes of a 256-mesh mix 252 /
// 300 us, its 256^3 ones 83 / 95, icosphere 6 at 1000^3 68 / 80, 7 at 1000^3 39 / 45; icosphere 5 at 600^3
// (20,480 triangles) 35 / 33, 4 at 512^3 25 / 24.
// Bound by the L2's scattered atomics on large tables (issue slots 53% busy), by instructions and, with
// few items, by the latency of one item elsewhere.  The soup of 2 M triangles at 1024^3: 26.9 ms for
// 3.36 G word updates (125 G/s); 39.8 ms with all eight x-dependent tests evaluated per row (41 G warp
// instructions).  The soup of 300,000 at 300^3 384 us / 697 us.  Six CTAs per SM at 80 registers; five
// are 2% faster on the first soup and 3% slower on the second, seven spill (at six only the part for long
// triangles does, 76 B and 108 B).  Reading a word before the
// atomic, to skip it where its bits are set, cost as many L2 requests as it saved (27.4 - 28.2 ms, and
// 30% to 90% more where the table fits the L2), and walking the items twice or four times, each time for
// a half or quarter of the table that stays in the L2, was 2% to 7% slower.
constexpr uint32_t kRowsCtaThreads = 128;
constexpr int kRowsWindow = 128;

constexpr uint32_t kRowsGroup = 8;  // items that a warp of the grouped kernel sets up at once

struct __align__(16) RowsTri {
	SurfTri S;             // bz0: the item's first slice
	uint32_t job, slices;
};
static_assert(sizeof(RowsTri) == 160, "RowsTri is ten 16-byte vectors");

struct RowsWarp {
	float4 xy[kRowsWindow];  // per y of the window: bounds of x from the XY tests, ny * py, its part of the row's place
	float4 slice[32];        // per slice with rows in the window: start - first y, its part, bounds of x from the ZX tests
	float kz[32];            // and its nz * pz
};

// A row's place in a narrow job's table is the sum of a part of its y and a part of its slice: linear
// index y * gx + z * gx * gy, or the Morton code's y and z bits.  (Other jobs keep y and z.)
__device__ __forceinline__ uint32_t y_part(const uint32_t* grid, bool morton, bool narrow, int y) {
	return !narrow ? (uint32_t)y : (morton ? spread3_narrow((uint32_t)y) << 1 : (uint32_t)y * grid[0]);
}
__device__ __forceinline__ uint32_t z_part(const uint32_t* grid, bool morton, bool narrow, int z) {
	return !narrow ? (uint32_t)z : (morton ? spread3_narrow((uint32_t)z) << 2 : (uint32_t)z * grid[1] * grid[0]);
}

// Writes of one row's interval [xl, xh] in a narrow job: its own lane's, of a few words, and the whole
// warp's, one row at a time with the lanes on consecutive words (linear) or x groups (Morton) -- a
// scattered atomic costs an L2 transaction of its own, a warp's atomics on one row share a few lines.
__device__ __forceinline__ void write_linear(uint32_t* table, uint32_t place, uint32_t xl, uint32_t xh) {
	const uint32_t lo = place + xl, hi = place + xh, w0 = lo >> 5, w1 = hi >> 5;  // at most three words
	const uint32_t m0 = 0xFFFFFFFFu >> (lo & 31u), m1 = 0xFFFFFFFFu << (~hi & 31u);
	atomicOr(table + w0, w0 == w1 ? m0 & m1 : m0);
	if (w0 != w1) {
		atomicOr(table + w1, m1);
		if (w1 - w0 > 1u) atomicOr(table + w0 + 1, 0xFFFFFFFFu);
	}
}
__device__ __forceinline__ void write_linear_warp(uint32_t* table, uint32_t place, uint32_t xl, uint32_t xh, uint32_t lane) {
	const uint32_t lo = place + xl, hi = place + xh, w0 = lo >> 5, w1 = hi >> 5;
	for (uint32_t w = w0 + lane; w <= w1; w += 32)
		atomicOr(table + w, (w == w0 ? 0xFFFFFFFFu >> (lo & 31u) : 0xFFFFFFFFu) & (w == w1 ? 0xFFFFFFFFu << (~hi & 31u) : 0xFFFFFFFFu));
}
// Bits of x offsets j0 .. j1 of the 4-voxel group k of a Morton row, at their place in its word.
__device__ __forceinline__ void write_morton_group(uint32_t* table, uint32_t code, int k, int xl, int xh) {
	const int j0 = max(xl - (k << 2), 0), j1 = min(xh - (k << 2), 3);
	const uint32_t n = (0xFu << j0) & (0xFu >> (3 - j1));
	const uint32_t m = ((n & 1u) << 31) | ((n & 2u) << 29) | ((n & 4u) << 21) | ((n & 8u) << 19);
	atomicOr(table + (code >> 5), m >> (code & 31u));
}
__device__ __forceinline__ void write_morton(uint32_t* table, uint32_t place, int xl, int xh) {
	uint32_t xd = spread3_narrow((uint32_t)(xl & ~3));
	for (int k = xl >> 2; k <= (xh >> 2); k++) {
		write_morton_group(table, xd | place, k, xl, xh);
		xd = morton_x_add_t<uint32_t>(xd, (uint32_t)kMortonX4);
	}
}
__device__ __forceinline__ void write_morton_warp(uint32_t* table, uint32_t place, int xl, int xh, uint32_t lane) {
	for (int k = (xl >> 2) + (int)lane; k <= (xh >> 2); k += 32)
		write_morton_group(table, spread3_narrow((uint32_t)(k << 2)) | place, k, xl, xh);
}

// Queued triangles of few rows that are too long to test every voxel.
struct LongWarp {
	SmallTri tri[32];  // q[0].w: rows of the warp's triangles before this one | voxels of a row - 1 << 16
	uint32_t job[32];
};

// A warp sets up up to 32 of them at a time, one per lane (in a launch with few of them fewer, so that all warps
// have some), parks them and deals their rows over its lanes: the bounds that the six tests of x and the plane
// test put on a row are found as in surf_rows, and the row is its lane's to write.  (As a call it took registers
// from surf_rows' own loop: the soup of 2 M at 1024^3 27.55 ms, 27.10 inline.)
template <class P>
__device__ __forceinline__ void long_triangles(const LaunchDesc& L, LongWarp& W, uint32_t n_long, uint32_t warp,
                                                   uint32_t n_warps) {
	const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
	const uint32_t turns = (n_long + 32u * n_warps - 1u) / (32u * n_warps), each = (n_long + turns * n_warps - 1u) / (turns * n_warps);
	for (uint64_t first = (uint64_t)warp * each; first < n_long; first += (uint64_t)n_warps * each) {
		SurfTri S;
		uint32_t n_rows = 0, job = 0;
		if (lane < each && first + lane < n_long) {
			const MidRec m = L.scr.mid[L.scr.cap - 1u - (uint32_t)(first + lane)];
			if (m.job < L.n_jobs && m.tri < job_at(L, m.job).n_tri) {  // (not so only after a queue overflow)
				const JobDesc& J = job_at(L, m.job);
				const float unit[3] = {J.unit[0], J.unit[1], J.unit[2]};
				const uint32_t grid[3] = {J.grid[0], J.grid[1], J.grid[2]};
				float t[9];
#pragma unroll
				for (int k = 0; k < 9; k++) t[k] = J.tris[(uint64_t)m.tri * 9 + k];
				surf_setup<P>(t, J.bmin, unit, J.inv_unit, J.box_near, grid, S);
				n_rows = (uint32_t)((S.by1 - S.by0 + 1) * (S.bz1 - S.bz0 + 1));
				job = m.job;
			}
		}
		uint32_t start = n_rows;
#pragma unroll
		for (int d = 1; d < 32; d <<= 1) {
			const uint32_t v = __shfl_up_sync(FULL, start, d);
			if (lane >= (uint32_t)d) start += v;
		}
		const uint32_t total = __shfl_sync(FULL, start, 31);
		start -= n_rows;
		const uint32_t slot = __popc(__ballot_sync(FULL, n_rows != 0u) & lt);
		if (n_rows) {
			SmallTri& o = W.tri[slot];
			pack_small(S, start | (uint32_t)(S.bx1 - S.bx0) << 16, o);
			if (plane_underflows(S.d1, S.d2)) plane_widen(S.nx, S.ny, S.nz, job_at(L, job).unit, o.q[4].z, o.q[4].w);
			W.job[slot] = job;
		}
		__syncwarp();
		uint32_t begun = 0;  // triangles that start before this step's rows
		for (uint32_t base = 0; base < total; base += 32) {
			const uint32_t at = start - base;
			const uint32_t starts = __reduce_or_sync(FULL, n_rows && at < 32u ? 1u << at : 0u);
			const uint32_t rec = begun + __popc(starts & (0xFFFFFFFFu >> (31u - lane))) - 1u;
			begun += __popc(starts);
			if (base + lane >= total) continue;
			const SmallTri& o = W.tri[rec];
			const JobDesc& J = job_at(L, W.job[rec]);
			const float4 box = o.q[0];
			const uint32_t w = __float_as_uint(box.w);
			int y, z;
			row_place(box, base + lane - (w & 0xFFFFu), y, z);
			const float ux = J.unit[0], py = __fmul_rn(__int2float_rn(y), J.unit[1]), pz = __fmul_rn(__int2float_rn(z), J.unit[2]);
			if (!row_in_yz<P>(o, py, pz)) continue;
			const float4 a = o.q[3], b = o.q[4], c = o.q[5], d = o.q[6], e = o.q[7], f = o.q[8];
			const float b0 = (float)(__float_as_uint(box.x) & 0xFFFFFFu), b1 = b0 + (float)(w >> 16);
			float x0 = b0, x1 = b1;
			clip_test_lane(c.x, __fmul_rn(c.z, py), -e.z, ux, b0, b1, x0, x1);
			clip_test_lane(c.y, __fmul_rn(c.w, py), -e.w, ux, b0, b1, x0, x1);
			clip_test_lane(d.x, __fmul_rn(b.x, py), -f.x, ux, b0, b1, x0, x1);
			clip_test_lane(d.y, __fmul_rn(b.y, pz), -f.y, ux, b0, b1, x0, x1);
			clip_test_lane(d.z, __fmul_rn(e.x, pz), -f.z, ux, b0, b1, x0, x1);
			clip_test_lane(d.w, __fmul_rn(e.y, pz), -f.w, ux, b0, b1, x0, x1);
			clip_plane(a.y, __fmul_rn(a.z, py), __fmul_rn(a.w, pz), b.z, b.w, fmaxf(fabsf(b.z), fabsf(b.w)),
			           __fdividef(-1.0f, a.y * ux), ux, b0, b1, x0, x1);
			if (!(x0 <= x1)) continue;
			const uint32_t grid[3] = {J.grid[0], J.grid[1], J.grid[2]};
			const bool morton = (J.flags & JOB_MORTON) != 0;
			if (J.flags & JOB_NARROW) write_row_t<uint32_t>(J.table, morton, grid, y, z, (int)x0, (int)x1);
			else write_row_t<uint64_t>(J.table, morton, grid, y, z, (int)x0, (int)x1);
		}
		__syncwarp();  // the records are written again
	}
}

template <class P, bool kGrouped>
__global__ void __launch_bounds__(kRowsCtaThreads, 6) surf_rows(const __grid_constant__ LaunchDesc L) {
	static_assert(P::plane == 2 && P::edge_xy == 1 && P::edge_yz == 1 && P::edge_zx == 2,
	              "the one-test bounds follow the pinned fused-multiply-add pattern");
	__shared__ __align__(16) union {
		RowsWarp rows;
		LongWarp longs;
	} s_warp[kRowsCtaThreads / 32];
	const uint32_t lane = threadIdx.x & 31u;
	RowsWarp& W = s_warp[threadIdx.x >> 5].rows;
	__shared__ RowsTri s_group[kGrouped ? kRowsCtaThreads / 32 : 1][kGrouped ? kRowsGroup : 1];
	RowsTri* group = s_group[kGrouped ? threadIdx.x >> 5 : 0];
	Counters* C = L.scr.ctr;
	clear_next_counters(L);
	// One thread per CTA reads the queue counters (thousands of warps reading one line would
	// serialise on its L2 slice), the CTA shares them through shared memory.
	__shared__ unsigned long long s_bigc;
	__shared__ uint2 s_mids;
	if (threadIdx.x == 0) {
		s_bigc = *reinterpret_cast<volatile unsigned long long*>(&C->big);
		const unsigned long long mids = *reinterpret_cast<volatile unsigned long long*>(&C->mid);  // and C->longs
		s_mids = make_uint2((uint32_t)mids, (uint32_t)(mids >> 32));
	}
	__syncthreads();
	// (Warps of different CTAs first, from the last one on: the first ones have the first items.  In launches of
	// few triangles, 3,223 of all sizes at 128^3: 18.5 us / 16.4.)
	if (s_mids.y)
		long_triangles<P>(L, s_warp[threadIdx.x >> 5].longs, min(s_mids.y, L.scr.cap),
		                  (threadIdx.x >> 5) * gridDim.x + gridDim.x - 1u - blockIdx.x, gridDim.x * (blockDim.x >> 5));
	const unsigned long long bigc = s_bigc;
	const uint32_t n_big = min((uint32_t)(bigc >> kBigShift), L.scr.cap);
	const uint64_t n_big_items = bigc & kBigItemMask;
	const uint32_t n_mid = min(s_mids.x, L.scr.cap);
	const uint64_t total = n_big_items + n_mid;
	// Warps beyond the number of queued items have nothing to claim (all of them when only small
	// triangles were queued).
	if ((uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5) >= total) return;
	// Where few items are parts of big triangles the items are of like size, and longer claims set up more
	// triangles together (icosphere 6 at 1000^3 68 us, 86 with eight turns); the others differ more (the
	// soup of 30,000 at 600^3 152 us, 191 with two turns).
	const uint32_t turns = kGrouped && 4 * n_big_items < total ? 2u : 8u;
	SpreadTickets wt(total, blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), gridDim.x * (blockDim.x >> 5), turns);
	for (;;) {
		SurfTri S;
		uint32_t job = 0, tri = 0, chunk = 0, slices = kZch;  // (grouped: of lane i, item i's at first)
		uint32_t items = 1u;
		unsigned long long first;
		float t[9];
		if constexpr (kGrouped) {
			uint32_t count;
			if (!wt.claim(L.scr.tickets, total, lane, kRowsGroup, first, count)) break;
			bool found = false;
			for (uint32_t i = 0; i < count && first + i * kTicketQueues < n_big_items; i++) {
				uint32_t a, b, c, e;
				const bool ok = queue_item(L, first + i * kTicketQueues, n_big, n_big_items, lane, a, b, c, e);
				if (lane == i) {
					found = ok;
					job = a;
					tri = b;
					chunk = c;
					slices = e;
				}
			}
			const unsigned long long mine = first + lane * kTicketQueues;
			if (lane < count && mine >= n_big_items) {
				const MidRec m = L.scr.mid[mine - n_big_items];
				job = m.job;
				tri = m.tri;
				found = job < L.n_jobs && tri < job_at(L, job).n_tri;
			}
			if (found) {
				const float* v = job_at(L, job).tris + (uint64_t)tri * 9;
#pragma unroll
				for (int k = 0; k < 9; k++) t[k] = v[k];
				const JobDesc& J = job_at(L, job);
				const float unit[3] = {J.unit[0], J.unit[1], J.unit[2]};
				const uint32_t grid[3] = {J.grid[0], J.grid[1], J.grid[2]};
				RowsTri g;
				surf_setup<P>(t, J.bmin, unit, J.inv_unit, J.box_near, grid, g.S);
				g.S.bz0 += (int)(chunk * slices);
				g.job = job;
				g.slices = slices;
				group[lane] = g;
			}
			items = __ballot_sync(FULL, found);
			__syncwarp();
		} else {
			if (!wt.take(L.scr.tickets, total, lane, first)) break;
			if (!queue_item(L, first, n_big, n_big_items, lane, job, tri, chunk, slices)) continue;
		}
		for (; items; items &= items - 1u) {
			if constexpr (kGrouped) {
				const RowsTri g = group[__ffs(items) - 1];
				S = g.S;
				job = g.job;
				slices = g.slices;
			}
			const JobDesc& J = job_at(L, job);
			const float unit[3] = {J.unit[0], J.unit[1], J.unit[2]};
			const uint32_t grid[3] = {J.grid[0], J.grid[1], J.grid[2]};
			const bool morton = (J.flags & JOB_MORTON) != 0;
			const bool narrow = (J.flags & JOB_NARROW) != 0;
			uint32_t* table = J.table;
			if constexpr (!kGrouped) {
				float tv = lane < 9 ? J.tris[(uint64_t)tri * 9 + lane] : 0.0f;
#pragma unroll
				for (int k = 0; k < 9; k++) t[k] = __shfl_sync(FULL, tv, k);
				surf_setup<P>(t, J.bmin, unit, J.inv_unit, J.box_near, grid, S);
			}
			float lo, hi;
			plane_bounds(S, lo, hi);
			if (plane_underflows(lo, hi)) plane_widen(S.nx, S.ny, S.nz, unit, lo, hi);
			const float plane_m = fmaxf(fabsf(lo), fabsf(hi)), plane_inv = __fdividef(-1.0f, S.nx * unit[0]);
			const float bx0 = (float)S.bx0, bx1 = (float)S.bx1;

			// this lane's z-slice
			const int z0 = kGrouped ? S.bz0 : S.bz0 + (int)(chunk * slices), z = z0 + (int)lane;
			float fy0 = (float)S.by0, fy1 = (float)S.by1, zx0 = bx0, zx1 = bx1, kz;
			{
				const float pz = __fmul_rn(__int2float_rn(z), unit[2]);
				kz = __fmul_rn(S.nz, pz);
				const float b0 = fy0, b1 = fy1;
	#pragma unroll
				for (int i = 0; i < 3; i++) {
					clip_test(S.eyz[i][0], __fmul_rn(S.eyz[i][1], pz), S.dyz[i], unit[1], b0, b1, fy0, fy1);
					clip_test(S.ezx[i][1], __fmul_rn(S.ezx[i][0], pz), S.dzx[i], unit[0], bx0, bx1, zx0, zx1);
				}
			}
			const bool rows = lane < slices && z <= S.bz1 && fy0 <= fy1 && zx0 <= zx1;
			const int ya = rows ? (int)fy0 : 0x7FFFFFFF, yb = rows ? (int)fy1 : -1;
			const int y_begin = __reduce_min_sync(FULL, ya), y_last = __reduce_max_sync(FULL, yb);
			for (int yw = y_begin; yw <= y_last; yw += kRowsWindow) {
				const int yw1 = min(yw + kRowsWindow - 1, y_last);
				for (int y = yw + (int)lane; y <= yw1; y += 32) {
					const float py = __fmul_rn(__int2float_rn(y), unit[1]);
					float x0 = bx0, x1 = bx1;
	#pragma unroll
					for (int i = 0; i < 3; i++)
						clip_test(S.exy[i][0], __fmul_rn(S.exy[i][1], py), S.dxy[i], unit[0], bx0, bx1, x0, x1);
					W.xy[y - yw] = make_float4(x0, x1, __fmul_rn(S.ny, py), __uint_as_float(y_part(grid, morton, narrow, y)));
				}
				const int first = max(ya, yw);
				const uint32_t cnt = rows ? (uint32_t)max(min(yb, yw1) - first + 1, 0) : 0u;
				uint32_t incl = cnt;
	#pragma unroll
				for (int d = 1; d < 32; d <<= 1) {
					const uint32_t v = __shfl_up_sync(FULL, incl, d);
					if (lane >= (uint32_t)d) incl += v;
				}
				const uint32_t R = __shfl_sync(FULL, incl, 31), start = incl - cnt;
				const uint32_t slot = __popc(__ballot_sync(FULL, cnt != 0u) & ((1u << lane) - 1u));
				if (cnt) {
					W.slice[slot] = make_float4(__int_as_float((int)start - first), __uint_as_float(z_part(grid, morton, narrow, z)),
					                            zx0, zx1);
					W.kz[slot] = kz;
				}
				__syncwarp();
				uint32_t begun = 0;  // slices that start before this step's rows
				for (uint32_t base = 0; base < R; base += 32) {
					const uint32_t at = start - base;
					const uint32_t starts = __reduce_or_sync(FULL, cnt && at < 32u ? 1u << at : 0u);
					const uint32_t rec = begun + __popc(starts & (0xFFFFFFFFu >> (31u - lane))) - 1u;
					begun += __popc(starts);
					const uint32_t k = base + lane;
					uint32_t yp = 0, zp = 0;  // the row's place
					int xl = 0, xh = -1;
					if (k < R) {
						const float4 q = W.slice[rec];
						const int y = (int)k - __float_as_int(q.x);
						const float4 e = W.xy[y - yw];
						yp = __float_as_uint(e.w);
						zp = __float_as_uint(q.y);
						float x0 = fmaxf(q.z, e.x), x1 = fminf(q.w, e.y);
						clip_plane(S.nx, e.z, W.kz[rec], lo, hi, plane_m, plane_inv, unit[0], bx0, bx1, x0, x1);
						if (x0 <= x1) {  // integers of [0, 2^22]: their bits after adding 2^23
							xl = __float_as_int(__fadd_rn(x0, 8388608.0f)) & 0x7FFFFF;
							xh = __float_as_int(__fadd_rn(x1, 8388608.0f)) & 0x7FFFFF;
						}
					}
					// Short rows are written by their own lane, long ones by the whole warp.
					const bool has = xh >= xl;
					const bool wide = has && (morton ? (xh >> 2) - (xl >> 2) >= 4 : (xh >> 5) - (xl >> 5) >= 2);
					uint32_t todo = __ballot_sync(FULL, wide);
					if (narrow && !morton) {
						if (has && !wide) write_linear(table, yp + zp, (uint32_t)xl, (uint32_t)xh);
					} else if (narrow) {
						if (has && !wide) write_morton(table, yp | zp, xl, xh);
					} else {
						if (has && !wide) write_row_t<uint64_t>(table, morton, grid, (int)yp, (int)zp, xl, xh);
					}
					while (todo) {
						const int src = __ffs(todo) - 1;
						todo &= todo - 1u;
						const uint32_t wy = __shfl_sync(FULL, yp, src), wz = __shfl_sync(FULL, zp, src);
						const int wl = __shfl_sync(FULL, xl, src), wh = __shfl_sync(FULL, xh, src);
						if (narrow && !morton) write_linear_warp(table, wy + wz, (uint32_t)wl, (uint32_t)wh, lane);
						else if (narrow) write_morton_warp(table, wy | wz, wl, wh, lane);
						else write_row_warp_t<uint64_t>(table, morton, grid, (int)wy, (int)wz, wl, wh, lane);
					}
				}
				__syncwarp();  // the tables are rewritten for the next window or item
			}
		}
		if constexpr (kGrouped) __syncwarp();  // and the triangles for the next group
	}
}

}  // namespace

// ---- host-side launchers ------------------------------------------------------------------------

template <class P>
static cudaError_t launch_surface_t(const LaunchDesc& L, const Tune& tune, int rows_grid, int raster_grid,
                                    cudaStream_t s, const Prof* prof) {
	if (L.n_tiles == 0) return cudaSuccess;
	if (prof) (*prof)(nullptr, s);
	// Rows (of the bounding box) that a queued triangle's items may have: with few triangles there are
	// fewer items than surf_rows has warps, and one item of a large triangle is its time.  In surf_rows,
	// with items of up to 1024 rows / 4096 / 32 slices whatever their rows: icosphere 3 at 1000^3 (1,280
	// triangles) 45 / 55 / 59 us, soups of 5,000 at 400^3 32 / 56 / 61 us, of 30,000 at 600^3 197 / 161 / 179,
	// of 300,000 at 300^3 488 / 410 / 411 us.
	const uint64_t triangles = (uint64_t)L.n_tiles * kTile, warps = (uint64_t)rows_grid * (kRowsCtaThreads / 32);
	const uint32_t item_rows = triangles < 4 * warps ? 1024u : (triangles < 16 * warps ? 4096u : 0xFFFFFFFFu);
	const uint32_t split = classify_split(L.n_tiles, (uint32_t)rows_grid);
	// (a kernel of its own for launches with dense jobs: their code costs the others 1% to 2%)
	const auto classify = L.any_dense ? surf_classify<P, true> : surf_classify<P, false>;
	classify<<<L.n_tiles << split, kTile, 0, s>>>(L, std::min(tune.small_vox, kLocalRows), item_rows, split);
	cudaError_t e = cudaGetLastError();
	if (e != cudaSuccess) return e;
	if (prof) (*prof)("surf_classify", s);
	if (L.n_bricks) {  // with no pair area (pair_cap 0) brick_bin queues every triangle for surf_rows
		e = launch_bricks(L, rows_grid, raster_grid, s, prof);
		if (e != cudaSuccess) return e;
	}
	// Grouped where the warps can expect to claim several items at a time: many triangles in meshes whose
	// triangles are larger than a few voxels (both sides at surf_rows; icosphere 6 at 500^3, 205 faces a warp,
	// 20 us grouped and 19 not, at 700^3, 403 a warp, 35 and 37).
	const bool grouped = L.coarse_tri >= 16 * warps && L.coarse_faces >= 256 * warps;
	e = launch_k(grouped ? surf_rows<P, true> : surf_rows<P, false>, (unsigned)rows_grid, kRowsCtaThreads, 0, s, L);
	if (e != cudaSuccess) return e;
	if (prof) (*prof)("surf_rows", s);
	return cudaGetLastError();
}

cudaError_t launch_surface(const LaunchDesc& L, const Tune& tune, int rows_grid, int raster_grid, cudaStream_t s,
                           const Prof* prof) {
	return launch_surface_t<RefFma>(L, tune, rows_grid, raster_grid, s, prof);
}

int surf_rows_blocks_per_sm() {
	int n = 0;
	cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, surf_rows<RefFma, true>, kRowsCtaThreads, 0);
	return n > 0 ? n : 1;
}

}  // namespace cvx
