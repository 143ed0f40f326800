// mesh.cu -- mesh ingest on the GPU: the vertex bounding box of a triangle soup and the expansion
// of an indexed mesh into the soup the voxelizer reads.
//
// Reference: src/main.cpp:61-80 (meshToGPU_managed: a host loop copying each face's three vertices
// into managed memory, 9 floats per triangle) and src/main.cpp:179 (Trimesh need_bbox: min/max over
// the vertices), followed by createMeshBBCube and the voxinfo constructor (src/main.cpp:180-186).
// Min and max are exact, so the device box equals the host one for finite coordinates.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>

#include "cvx.h"
#include "engine.h"

namespace cvx {
namespace {

constexpr uint32_t kReduceThreads = 256;

// Order-preserving map of a float to an unsigned key (finite values and infinities); never 0.
__device__ __forceinline__ uint32_t order_key(float f) {
	const uint32_t b = __float_as_uint(f);
	return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// out[0..2] = maxima of the complemented keys (the minima), out[3..5] = maxima of the keys; zeroed by
// the host.  kVec: the soup is 16-byte aligned, and a thread reads four vertices in three accesses
// (1.05 M triangles, 38 MB, in 9.3 us; 11.5 us reading one vertex float by float).
template <bool kVec>
__global__ void __launch_bounds__(kReduceThreads) bbox_reduce(const float* __restrict__ tris, uint64_t n_vertices,
                                                              uint32_t* out) {
	float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
	auto add = [&](int k, float c) {
		lo[k] = fminf(lo[k], c);
		hi[k] = fmaxf(hi[k], c);
	};
	const uint64_t id = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
	uint64_t done = 0;
	if constexpr (kVec) {
		const float4* q = reinterpret_cast<const float4*>(tris);
#pragma unroll 2
		for (uint64_t i = id; i < n_vertices / 4; i += stride) {
			const float4 a = q[3 * i], b = q[3 * i + 1], c = q[3 * i + 2];
			add(0, a.x); add(1, a.y); add(2, a.z); add(0, a.w);
			add(1, b.x); add(2, b.y); add(0, b.z); add(1, b.w);
			add(2, c.x); add(0, c.y); add(1, c.z); add(2, c.w);
		}
		done = n_vertices / 4 * 4;
	}
	for (uint64_t v = done + id; v < n_vertices; v += stride)
#pragma unroll
		for (int k = 0; k < 3; k++) add(k, tris[3 * v + k]);
	// (the keys in integers: one reduction instruction per value instead of five shuffles)
	__shared__ uint32_t s_key[6][kReduceThreads / 32];
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
	for (int k = 0; k < 3; k++) {
		const uint32_t l = __reduce_max_sync(0xFFFFFFFFu, ~order_key(lo[k]));
		const uint32_t h = __reduce_max_sync(0xFFFFFFFFu, order_key(hi[k]));
		if (lane == 0) {
			s_key[k][warp] = l;
			s_key[3 + k][warp] = h;
		}
	}
	__syncthreads();
	if (threadIdx.x < 6) {
		uint32_t m = 0;
		for (uint32_t w = 0; w < kReduceThreads / 32; w++) m = max(m, s_key[threadIdx.x][w]);
		atomicMax(out + threadIdx.x, m);
	}
}

constexpr uint32_t kGatherFaces = 256;

// A CTA per 256 faces, one thread each: three vertex indices -> 9 floats, staged in shared memory (9 words
// per face: no bank conflicts) so that the soup is written in consecutive 16-byte pieces.  A face with
// an index out of range becomes a NaN triangle and is counted in *bad (the caller must not voxelize
// such a soup).  kVec: the soup is 16-byte aligned.  Bound by memory: 12.8 us for 1.05 M faces (69 MB,
// 5.4 TB/s); 36 us with each thread writing its nine floats 36 bytes from the next one's.
template <bool kVec>
__global__ void __launch_bounds__(kGatherFaces) gather_faces(const float* __restrict__ verts, uint64_t n_verts,
                                                             const uint32_t* __restrict__ faces, uint64_t n_faces,
                                                             float* __restrict__ soup, unsigned long long* bad) {
	__shared__ __align__(16) float s_soup[kGatherFaces * 9];
	__shared__ uint32_t s_faces[kGatherFaces * 3];
	const uint64_t f0 = (uint64_t)blockIdx.x * kGatherFaces;
	const uint32_t n = (uint32_t)umin64(kGatherFaces, n_faces - f0);
	for (uint32_t i = threadIdx.x; i < 3 * n; i += kGatherFaces) s_faces[i] = faces[3 * f0 + i];
	__syncthreads();
	if (threadIdx.x < n) {
		const uint32_t idx[3] = {s_faces[3 * threadIdx.x], s_faces[3 * threadIdx.x + 1], s_faces[3 * threadIdx.x + 2]};
		const bool ok = idx[0] < n_verts && idx[1] < n_verts && idx[2] < n_verts;
		float* o = s_soup + 9 * threadIdx.x;
#pragma unroll
		for (int c = 0; c < 3; c++)
#pragma unroll
			for (int k = 0; k < 3; k++) o[3 * c + k] = ok ? verts[3 * (uint64_t)idx[c] + k] : __int_as_float(0x7FC00000);
		if (!ok && bad) atomicAdd(bad, 1ull);
	}
	__syncthreads();
	float* dst = soup + 9 * f0;
	uint32_t done = 0;
	if constexpr (kVec) {
		done = 9 * n / 4 * 4;
		for (uint32_t i = threadIdx.x; i < done / 4; i += kGatherFaces)
			reinterpret_cast<float4*>(dst)[i] = reinterpret_cast<const float4*>(s_soup)[i];
	}
	for (uint32_t i = done + threadIdx.x; i < 9 * n; i += kGatherFaces) dst[i] = s_soup[i];
}

float key_to_float(uint32_t k) {
	const uint32_t b = (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k;
	float f;
	std::memcpy(&f, &b, 4);
	return f;
}

cvx_status cuda_status(cudaError_t e, const char* what) {
	if (e == cudaSuccess) return CVX_OK;
	set_message(std::string(what) + ": " + cudaGetErrorString(e));
	return CVX_ERR_CUDA;
}

}  // namespace
}  // namespace cvx

using namespace cvx;

extern "C" {

static cvx_status check_box(const float* d_triangles, uint64_t n_triangles, const float* out_min, const float* out_max) {
	if (!d_triangles || !out_min || !out_max) {
		set_message("cvx_mesh_bbox_device: null argument");
		return CVX_ERR_INVALID_VALUE;
	}
	if (n_triangles == 0) {
		set_message("cvx_mesh_bbox_device: empty mesh has no bounding box");
		return CVX_ERR_INVALID_VALUE;
	}
	return CVX_OK;
}

cvx_status cvx_mesh_bbox_device_ws(const float* d_triangles, uint64_t n_triangles, void* d_ws, uint64_t ws_bytes,
                                   float out_min[3], float out_max[3], cvx_stream_t stream) {
	cvx_status st = check_box(d_triangles, n_triangles, out_min, out_max);
	if (st != CVX_OK) return st;
	if (!d_ws || ws_bytes < CVX_BBOX_WORKSPACE || reinterpret_cast<uintptr_t>(d_ws) % 16) {
		set_message("cvx_mesh_bbox_device_ws: workspace null, too small or not 16-byte aligned");
		return CVX_ERR_INVALID_VALUE;
	}
	cudaStream_t s = (cudaStream_t)stream;
	uint32_t* d_out = static_cast<uint32_t*>(d_ws);
	uint32_t keys[6];
	int dev = 0, sms = 0;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	const uint64_t nv = 3 * n_triangles;
	const uint64_t want = (nv + kReduceThreads * 8 - 1) / (kReduceThreads * 8);
	const uint32_t blocks = (uint32_t)(want < (uint64_t)sms * 8 ? (want ? want : 1) : (uint64_t)sms * 8);
	st = cuda_status(cudaMemsetAsync(d_out, 0, sizeof(keys), s), "cudaMemsetAsync");
	if (st == CVX_OK) {
		if (reinterpret_cast<uintptr_t>(d_triangles) % 16 == 0) bbox_reduce<true><<<blocks, kReduceThreads, 0, s>>>(d_triangles, nv, d_out);
		else bbox_reduce<false><<<blocks, kReduceThreads, 0, s>>>(d_triangles, nv, d_out);
		st = cuda_status(cudaGetLastError(), "bbox_reduce");
	}
	if (st == CVX_OK)
		st = cuda_status(cudaMemcpyAsync(keys, d_out, sizeof(keys), cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
	if (st == CVX_OK) st = cuda_status(cudaStreamSynchronize(s), "cudaStreamSynchronize");
	if (st != CVX_OK) return st;
	for (int k = 0; k < 3; k++) {
		out_min[k] = key_to_float(~keys[k]);
		out_max[k] = key_to_float(keys[3 + k]);
	}
	return CVX_OK;
}

cvx_status cvx_mesh_bbox_device(const float* d_triangles, uint64_t n_triangles, float out_min[3], float out_max[3],
                                cvx_stream_t stream) {
	cvx_status st = check_box(d_triangles, n_triangles, out_min, out_max);
	if (st != CVX_OK) return st;
	cudaStream_t s = (cudaStream_t)stream;
	void* ws = nullptr;
	st = cuda_status(cudaMallocAsync(&ws, CVX_BBOX_WORKSPACE, s), "cudaMallocAsync");
	if (st != CVX_OK) return st;
	st = cvx_mesh_bbox_device_ws(d_triangles, n_triangles, ws, CVX_BBOX_WORKSPACE, out_min, out_max, stream);
	cudaFreeAsync(ws, s);
	return st;
}

static cvx_status voxinfo_of_box(cvx_status st, const float lo[3], const float hi[3], const uint32_t gridsize[3],
                                 uint64_t n_triangles, cvx_voxinfo* out) {
	float clo[3], chi[3];
	if (st != CVX_OK) return st;
	if ((st = cvx_bbox_cube(lo, hi, clo, chi)) != CVX_OK) return st;
	return cvx_voxinfo_init(out, clo, chi, gridsize, n_triangles);
}

cvx_status cvx_voxinfo_from_device_ws(const float* d_triangles, uint64_t n_triangles, const uint32_t gridsize[3],
                                      void* d_ws, uint64_t ws_bytes, cvx_voxinfo* out, cvx_stream_t stream) {
	if (!gridsize || !out) {
		set_message("cvx_voxinfo_from_device: null argument");
		return CVX_ERR_INVALID_VALUE;
	}
	float lo[3], hi[3];
	const cvx_status st = cvx_mesh_bbox_device_ws(d_triangles, n_triangles, d_ws, ws_bytes, lo, hi, stream);
	return voxinfo_of_box(st, lo, hi, gridsize, n_triangles, out);
}

cvx_status cvx_voxinfo_from_device(const float* d_triangles, uint64_t n_triangles, const uint32_t gridsize[3],
                                   cvx_voxinfo* out, cvx_stream_t stream) {
	if (!gridsize || !out) {
		set_message("cvx_voxinfo_from_device: null argument");
		return CVX_ERR_INVALID_VALUE;
	}
	float lo[3], hi[3];
	const cvx_status st = cvx_mesh_bbox_device(d_triangles, n_triangles, lo, hi, stream);
	return voxinfo_of_box(st, lo, hi, gridsize, n_triangles, out);
}

cvx_status cvx_gather_soup(const float* d_vertices, uint64_t n_vertices, const uint32_t* d_faces, uint64_t n_faces,
                           float* d_soup, unsigned long long* d_bad_faces, cvx_stream_t stream) {
	if ((n_faces && (!d_faces || !d_soup)) || (n_vertices && !d_vertices)) {
		set_message("cvx_gather_soup: null argument");
		return CVX_ERR_INVALID_VALUE;
	}
	if (n_faces == 0) return CVX_OK;
	cudaStream_t s = (cudaStream_t)stream;
	const unsigned blocks = (unsigned)((n_faces + kGatherFaces - 1) / kGatherFaces);
	if (reinterpret_cast<uintptr_t>(d_soup) % 16 == 0)
		gather_faces<true><<<blocks, kGatherFaces, 0, s>>>(d_vertices, n_vertices, d_faces, n_faces, d_soup, d_bad_faces);
	else
		gather_faces<false><<<blocks, kGatherFaces, 0, s>>>(d_vertices, n_vertices, d_faces, n_faces, d_soup, d_bad_faces);
	return cuda_status(cudaGetLastError(), "gather_faces");
}

}  // extern "C"
