"""A thread that submits to the server does not wait for the launch of a batch: server.cu
compiled for the host against stand-ins for the index and the CUDA calls, one launch held
until another request has been submitted."""
import os
import subprocess

from conftest import PKG, ROOT

SRC = r"""
#include "server.cu"
#include <atomic>
#include <cstdio>
#include <cstdlib>

static std::atomic<int> launches{0}, submitted{0}, held{0};
static std::string      err;

namespace vann { void set_last_error(const char* m) { err = m; } }
extern "C" {
const char* vann_last_error(void) { return err.c_str(); }
vann_status vann_get_info(const vann_index*, vann_info* i) { *i = vann_info{}; i->dim = 4; return VANN_OK; }
vann_status vann_search_uneven(vann_index*, const float*, uint64_t, const vann_search_params*, const uint32_t*,
                               const uint32_t*, uint32_t* ids, float*, void*) {
    if (++launches == 1) {  // two seconds at most
        held = 1;
        for (int i = 0; i < 2000 && !submitted; ++i) std::this_thread::sleep_for(std::chrono::milliseconds(1));
        held = submitted ? 2 : 3;
    }
    ids[0] = 7;
    return VANN_OK;
}
vann_status vann_insert(vann_index*, const float*, uint64_t, uint32_t*, void*) { return VANN_OK; }
vann_status vann_delete(vann_index*, const uint32_t*, uint64_t, void*) { return VANN_OK; }
vann_status vann_consolidate(vann_index*, void*) { return VANN_OK; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = calloc(n, 1); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = calloc(n, 1); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = calloc(n, 1); return cudaSuccess; }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free((void*)s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free((void*)e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
}

int main() {
    vann_server_params p{};
    p.max_batch = 8; p.slots = 2; p.max_k = 4;
    vann_server* s = nullptr;
    float        q[4] = {1, 2, 3, 4};
    uint64_t     a = 0, b = 0;
    if (vann_server_create((vann_index*)&p, &p, &s) != VANN_OK) return 2;
    if (vann_server_submit_search(s, q, 1, 1, 4, &a) != VANN_OK) return 3;
    while (!held) std::this_thread::sleep_for(std::chrono::milliseconds(1));
    if (vann_server_submit_search(s, q, 1, 1, 4, &b) != VANN_OK) return 4;
    submitted = 1;
    uint32_t ids[2] = {0, 0};
    float    d[2];
    if (vann_server_wait(s, a, ids, d, nullptr, nullptr, 5000) != VANN_OK) return 5;
    if (vann_server_wait(s, b, ids + 1, d, nullptr, nullptr, 5000) != VANN_OK) return 6;
    vann_server_stats st{};
    vann_server_get_stats(s, &st);
    printf("%s %u %u %llu %llu\n", held == 2 ? "free" : "held", ids[0], ids[1], (unsigned long long)st.batches,
           (unsigned long long)st.queries);
    vann_server_destroy(s);
}
"""


def test_submit_during_a_launch(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-w", "-pthread", "-I", os.path.join(PKG, "csrc"), "-I", os.path.join(ROOT, "include"),
                    "-I", "/usr/local/cuda/include", str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True, timeout=60).stdout
    assert out == "free 7 7 2 2\n"
