// Host-level test of cvx_device_status: error words planted where a failed device-side check leaves
// them, then calls that go through.  Compiled with api.cu itself, whose per-stream scratch it reads.
#include "../cuda_voxelizer_gb300/csrc/api.cu"

static int g_bad = 0;
static void expect(bool ok, const char* what) {
	if (!ok) g_bad++;
	std::printf("%s %s\n", ok ? "ok  " : "FAIL", what);
}
static void need(cvx_status st) {
	if (st != CVX_OK) {
		std::printf("FAIL call: %s\n", cvx_last_error_message());
		std::exit(2);
	}
}

struct Mesh {
	cvx_voxinfo info;
	float* tris = nullptr;
	uint32_t* table = nullptr;
	Mesh(uint32_t gx, uint32_t gy, uint32_t gz, uint32_t n) {
		const float lo[3] = {0, 0, 0}, hi[3] = {(float)gx, (float)gy, (float)gz};
		const uint32_t g[3] = {gx, gy, gz};
		need(cvx_voxinfo_init(&info, lo, hi, g, n));
		std::vector<float> t(9 * n);
		uint32_t r = 1;
		for (uint32_t i = 0; i < 9 * n; i++) {
			r = r * 1664525u + 1013904223u;
			t[i] = hi[i % 3] * ((float)(r >> 8) / 16777216.0f);
		}
		cudaMalloc((void**)&tris, t.size() * 4);
		cudaMemcpy(tris, t.data(), t.size() * 4, cudaMemcpyHostToDevice);
		cudaMalloc((void**)&table, cvx_table_words(&info) * 4);
	}
	cvx_job job(int solid) const { return cvx_job{info, tris, table, 0, solid}; }
};

static void plant(cudaStream_t s, uint32_t word) {
	const unsigned code = kErrQueueOverflow;
	cudaStreamSynchronize(s);
	char* rec = static_cast<char*>(g_ws[{0, s}].rec);
	cudaMemcpy(reinterpret_cast<unsigned*>(rec + rec_layout(0, 0).errors) + word, &code, 4, cudaMemcpyHostToDevice);
}
static uint32_t last_direct(cudaStream_t s) { return g_ws[{0, s}].error ^ 1u; }  // the word of the last direct call

int main() {
	Mesh small(64, 64, 64, 300), large(1024, 1024, 512, 50);
	cudaStream_t s, fresh;
	cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
	cudaStreamCreateWithFlags(&fresh, cudaStreamNonBlocking);
	auto direct = [&](int solid) {
		need(solid ? cvx_voxelize_solid(&small.info, small.tris, small.table, 0, s) : cvx_voxelize(&small.info, small.tris, small.table, 0, s));
	};
	auto batch = [&]() {  // two launch sequences in one call
		const cvx_job jobs[2] = {small.job(0), large.job(1)};
		need(cvx_voxelize_batch(jobs, 2, s));
	};
	auto bricks = [&](cudaStream_t on) {
		cvx_tuning t, b;
		need(cvx_get_tuning(0, &t));
		b = t;
		b.brick_pairs = 16;
		need(cvx_set_tuning(0, &b));
		need(cvx_voxelize(&large.info, large.tris, large.table, 0, on));
		need(cvx_set_tuning(0, &t));
	};

	// a new area, in memory that was used before, whose first call has brick jobs
	std::vector<void*> used(64);
	for (void*& p : used) {
		cudaMalloc(&p, 4 << 20);
		cudaMemset(p, 0x5A, 4 << 20);
	}
	for (void* p : used) cudaFree(p);
	bricks(fresh);
	expect(cvx_device_status(fresh) == CVX_OK, "first call of a stream with brick jobs");

	bricks(s);  // the scratch has its final size before the capture
	batch();
	direct(0);
	direct(1);
	cudaStreamSynchronize(s);
	cudaGraph_t graph;
	cudaGraphExec_t exec;
	cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
	direct(0);
	cudaStreamEndCapture(s, &graph);
	cudaGraphInstantiate(&exec, graph, 0);

	const char* names[] = {"direct surface", "direct solid", "batch", "replay", "bricks"};
	auto call = [&](int k) {
		if (k == 0) direct(0);
		if (k == 1) direct(1);
		if (k == 2) batch();
		if (k == 3) cudaGraphLaunch(exec, s);
		if (k == 4) bricks(s);
	};
	for (int failed = 0; failed < 5; failed++)
		for (int next = 0; next < 5; next++) {
			call(failed);
			expect(cvx_device_status(s) == CVX_OK, names[failed]);
			plant(s, failed < 3 ? last_direct(s) : kCaptureError);
			expect(cvx_device_status(s) == CVX_ERR_DEVICE_CHECK, "a failed check is reported");
			expect(cvx_device_status(s) == CVX_ERR_DEVICE_CHECK, "and reported again");
			call(next);
			char what[128];
			std::snprintf(what, sizeof(what), "%s that fails, then %s", names[failed], names[next]);
			expect(cvx_device_status(s) == CVX_OK, what);
		}
	std::printf("%d failures\n", g_bad);
	return g_bad ? 1 : 0;
}
