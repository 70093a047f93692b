"""Host copies against the kernels that read them. A cudaMemcpy from pageable memory
returns when the data has been staged; only its stream (the legacy one) knows when it
has arrived, and a kernel on a non-blocking stream does not wait for that stream. The
library's host code runs here against a CUDA runtime that does nothing but follow
copies, synchronisations and launches: no launch may come before the arrival of a copy
made on another stream. No GPU is needed."""
import glob
import os
import subprocess

from conftest import ROOT

RUNTIME = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
static std::set<cudaStream_t> pending;   // streams with a copy that may still be on its way
static std::map<void*, size_t> live;
static bool capturing = false;
int bad = 0, launches = 0;
const char* phase = "";
static void launch(cudaStream_t s)
{
    if (capturing) return;
    ++launches;
    for (cudaStream_t p : pending)
        if (p != s) ++bad, std::printf("%s: a launch does not wait for a copy on %s\n", phase, p ? "another stream" : "the legacy stream");
}
static void copy(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st, bool sync)
{
    if (capturing) return;
    std::memcpy(d, s, n);
    if (k == cudaMemcpyHostToDevice) pending.insert(st);
    else if (sync) pending.erase(st);
}
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { live[*p = std::calloc(n, 1)] = n; return cudaSuccess; }
cudaError_t cudaFree(void* p) { live.erase(p); std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { copy(d, s, n, k, nullptr, true); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) { copy(d, s, n, k, st, false); return cudaSuccess; }
cudaError_t cudaMemset(void*, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { if (v == 0) std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { pending.erase(s); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { pending.clear(); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { pending.erase(s); return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { capturing = true; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { capturing = false; *g = nullptr; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { *e = (cudaGraphExec_t)1; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) { launch(s); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t*) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) { *t = 0; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) { std::memset(p, 0, sizeof *p); return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = (size_t)1 << 33; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 2; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPeekAtLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void*, void**) { launch(c->stream); return cudaSuccess; }
cudaError_t cudaLaunchCooperativeKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t s) { launch(s); return cudaSuccess; }
static cudaStream_t next_stream;
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void* s) { next_stream = (cudaStream_t)s; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void* s) { *(cudaStream_t*)s = next_stream; return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t*, const void*) { return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t s) { launch(s); return cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
}
"""

PROG = r"""
#include <vector>
#include "runtime.h"
#include "troute_gb300.h"
static void ok(int rc) { if (rc) std::printf("%s: %d %s\n", phase, rc, troute_last_error()), std::exit(1); }
int main()
{
    // a main stem of 60 reaches with a short tributary at every second
    std::vector<int> ptr{0}, idx, start, len;
    int stem = -1, n = 0;
    auto reach = [&](std::vector<int> ups) {
        for (int u : ups) idx.push_back(u);
        ptr.push_back((int)idx.size());
        start.push_back(n);
        len.push_back(1);
        return n++;
    };
    for (int k = 0; k < 60; ++k) {
        std::vector<int> ups;
        if (stem >= 0) ups.push_back(stem);
        if (stem >= 0 && k % 2) ups.push_back(reach({}));
        stem = reach(ups);
    }
    const troute_topo topo{n, n, start.data(), len.data(), ptr.data(), idx.data()};
    const int T = 70;
    std::vector<float> c(n, 0.25f), ql((size_t)T * n, 0.1f), q(n, 1.0f), out(n);
    cudaStream_t st;
    cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);

    phase = "linear route";
    ok(troute_linear_route(&topo, c.data(), c.data(), c.data(), c.data(), ql.data(), q.data(), T, out.data()));
    phase = "linear handle";
    troute_linear* L;
    ok(troute_linear_create(&L, &topo, c.data(), c.data(), c.data(), c.data()));
    for (int t : {1, 9, 17, 70, 9})
        for (cudaStream_t s : {(cudaStream_t) nullptr, st}) ok(troute_linear_run_device(L, ql.data(), t, out.data(), 0, s));
    troute_linear_destroy(L);

    phase = "matrix route";
    ok(troute_matrix_route(n, ptr.data(), idx.data(), c.data(), c.data(), c.data(), c.data(), 0.0f, ql.data(), q.data(), T, out.data()));
    phase = "matrix handle";
    troute_matrix* M;
    ok(troute_matrix_create(&M, n, ptr.data(), idx.data(), c.data(), c.data(), c.data(), c.data(), 0.0f));
    for (cudaStream_t s : {(cudaStream_t) nullptr, st}) ok(troute_matrix_run_device(M, ql.data(), 3, out.data(), s));
    troute_matrix_destroy(M);

    phase = "diffusive";
    std::vector<troute_diff_reach> rp(4, troute_diff_reach{5, 0.5f, 300.0f});
    std::vector<float> a(40, 1.0f), b(40);
    ok(troute_diffusive_tridiag(rp.data(), a.data(), a.data(), nullptr, a.data(), b.data(), 4, 10));

    phase = "reach-parallel";
    std::vector<troute_chparams> p(n, troute_chparams{1000, 5, 15, 25, 0.05, 0.1, 1, 0.001});
    std::vector<double> x(n, 1.0), y(n), z(n), w(n);
    ok(troute_mc_reach_parallel(p.data(), x.data(), start.data(), len.data(), x.data(), x.data(), x.data(), y.data(), z.data(), w.data(),
                                1.0, 300.0, n));

    phase = "routing handle";
    troute_cfg cfg;
    troute_cfg_default(&cfg);
    cfg.warm_start = 1;
    troute_handle* H;
    ok(troute_create(&H, &topo, p.data(), 300.0, &cfg));
    ok(troute_set_state(H, x.data(), x.data(), nullptr));
    troute_warm* W;
    ok(troute_warm_create(&W, 1));
    std::vector<float> state(4801 + 18, 0.5f);
    ok(troute_warm_set(W, state.data(), (int)state.size()));
    ok(troute_set_warm_start(H, W, 0.05));
    std::vector<double> in((size_t)T * n, 0.1);
    ok(troute_run(H, in.data(), T, nullptr));
    ok(troute_run_device(H, in.data(), T, st));
    ok(troute_sync(H, nullptr));
    ok(troute_destroy(H));
    ok(troute_warm_destroy(W));
    std::printf("%d launches, %d of them early\n", launches, bad);
    return launches > 20 && bad == 0 ? 0 : 1;
}
"""


def test_no_launch_comes_before_its_uploads(tmp_path):
    from troute_gb300 import build as B

    B.build()
    (tmp_path / "runtime.h").write_text(RUNTIME)
    (tmp_path / "t.cpp").write_text(PROG)
    objects = [o for o in glob.glob(os.path.join(B.BUILD, "*.o")) if os.path.basename(o)[:-2] in B.CU_SOURCES + B.CPP_SOURCES]
    assert len(objects) == len(B.CU_SOURCES + B.CPP_SOURCES)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-w", "-I", os.path.join(B.CUDA_HOME, "include"), "-I", os.path.join(ROOT, "include"),
                    str(tmp_path / "t.cpp"), *objects, "-o", exe, "-lpthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
