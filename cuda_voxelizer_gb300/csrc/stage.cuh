// stage.cuh -- staging of a warp's triangles in shared memory, shared by the classify kernels.
#pragma once
#include "engine.h"

namespace cvx {

constexpr unsigned FULL = 0xFFFFFFFFu;

// Bounded wait on an mbarrier phase.  Returns false if the phase did not complete in time.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
	for (uint32_t it = 0; it < (1u << 24); it++) {
		uint32_t ok;
		asm volatile(
		    "{\n\t.reg .pred p;\n\t"
		    "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
		    "selp.u32 %0, 1, 0, p;\n\t}"
		    : "=r"(ok)
		    : "r"(bar), "r"(parity)
		    : "memory");
		if (ok) return true;
	}
	return false;
}

// Stage a warp's `cnt` <= 32 triangles (9 floats each) from global memory into shared memory.  A
// multiple of four aligned triangles of plain device memory goes through one bulk copy completing on
// the warp's own mbarrier; anything else (a ragged or unaligned group, managed or host memory:
// `plain`) is loaded by the lanes.  Returns false (in every lane) if the bulk copy did not complete within the bounded wait: the
// error word is set, the warp waits once more (again bounded) for the copy still in flight, and the
// caller skips the triangles without touching the shared memory the copy may still write.
__device__ __forceinline__ bool stage_warp(const LaunchDesc& L, const float* src, uint32_t cnt, float* s_tri,
                                           uint64_t* s_bar, bool plain) {
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t bytes = cnt * 36u;
	const bool bulk = (cnt & 3u) == 0u && ((reinterpret_cast<uintptr_t>(src) & 15u) == 0) && !plain;
	if (bulk) {
		const uint32_t bar = (uint32_t)__cvta_generic_to_shared(s_bar);
		const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_tri);
		if (lane == 0) {
			asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
			asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
			asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
			asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
			             "l"(src), "r"(bytes), "r"(bar)
			             : "memory");
		}
		__syncwarp();  // barrier initialised before anyone waits on it
		const bool late = !mbar_wait(bar, 0);
		if (__any_sync(FULL, late)) {
			if (lane == 0) set_error(L, kErrBulkTimeout);
			mbar_wait(bar, 0);
			return false;
		}
		return true;
	}
	for (uint32_t i = lane; i < cnt * 9u; i += 32) s_tri[i] = src[i];
	__syncwarp();
	return true;
}

// The persistent kernels clear the counters of the next launch sequence (whose kernels follow in the
// stream), so that it needs no memset: 2 us of a small call.  With them go the error words of other
// calls: of the one before, and the word that the next one will use.
__device__ __forceinline__ void clear_next_counters(const LaunchDesc& L) {
	if (L.scr.next && blockIdx.x + 1 == gridDim.x) {
		for (uint32_t i = threadIdx.x; i < L.scr.next_words; i += blockDim.x) L.scr.next[i] = 0u;
		if (threadIdx.x < kErrorWords && L.scr.errors + threadIdx.x != L.scr.error) L.scr.errors[threadIdx.x] = 0u;
	}
}

// The queued item of ticket `tk` of a persistent kernel: big items (n_big records, n_big_items items)
// first, then the mid triangles.  Every lane calls it with the same ticket and gets the same answer;
// false for a malformed record (only possible after a queue overflow).  The big record is found by a
// search with 32 probes per round: three dependent loads for 32,768 records instead of fifteen.
__device__ __forceinline__ bool queue_item(const LaunchDesc& L, unsigned long long tk, uint32_t n_big,
                                           uint64_t n_big_items, uint32_t lane, uint32_t& job, uint32_t& tri,
                                           uint32_t& chunk, uint32_t& slices) {
	chunk = 0;
	slices = kZch;
	if (tk < n_big_items) {
		if (n_big == 0) return false;
		uint32_t first = 0, n = n_big;  // the last record with item_begin <= tk is among n from `first`
		while (n > 1) {
			const uint32_t step = (n + 31u) >> 5, at = lane * step;
			const bool le = at < n && (at == 0u || L.scr.big[first + at].item_begin <= tk);
			const uint32_t last = 31u - __clz(__ballot_sync(FULL, le));
			first += last * step;
			n = min(step, n - last * step);
		}
		const BigRec r = L.scr.big[first];
		job = r.job;
		tri = r.tri;
		slices = r.slices;
		chunk = (uint32_t)(tk - r.item_begin);
		if (tk < r.item_begin || chunk >= r.n_items) return false;
	} else {
		const MidRec r = L.scr.mid[tk - n_big_items];
		job = r.job;
		tri = r.tri;
	}
	return job < L.n_jobs && tri < job_at(L, job).n_tri;
}

// Triangles of a classify warp: 32, or in a launch with few tiles 32 >> split, so that its warps are
// spread over the chip and none has many rows or columns to walk.  Split while the launch has fewer CTAs
// than `enough`, those of the persistent kernel that follows (6 per SM for surface jobs, 4 for solid
// ones; the classify kernels themselves hold 9 and 12), up to kMaxSplit; a split of s launches 2^s CTAs
// per tile.  (9,216-triangle torus: surf_classify 64^3 11.7 -> 9.5 us, 128^3 16 ->
// 11.3 us, 256^3 with surf_rows 39 -> 27 us; solid_classify + solid_cols 256^3 28 -> 18 us.)
constexpr uint32_t kMaxSplit = 3;
inline uint32_t classify_split(uint32_t n_tiles, uint32_t enough) {
	uint32_t s = 0;
	while (s < kMaxSplit && (n_tiles << s) < enough) s++;
	return s;
}

}  // namespace cvx
