// The host code of the library on a stand-in for the CUDA runtime: device memory is host memory, kernels are only noted.  It follows
// which clears of device memory are still on their way (a cudaMemset returns before the default stream has run it, and nothing orders the
// default stream and a non-blocking one) and reports a kernel that is launched beside one.  Built and driven by test_host_runtime.py.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "../llm170_b200/csrc/dec.h"

namespace {

struct Clear {
    void* p;
    cudaStream_t st;
};
std::vector<Clear> pending;
std::map<const void*, std::string>& kernels() {       // (filled before this file's own statics are there)
    static std::map<const void*, std::string> m;
    return m;
}
int launches = 0, fail_at = -1;       // which kernel launch fails (0 = the first), -1 = none
cudaError_t last = cudaSuccess;
w4a16_dec* dec = nullptr;
const char matmul[] = "matmul";

std::string label(void* p) {
    const auto& d = dec->d;
    return p == d.mb.cnt ? "counts" : p == d.counters ? "tickets" : p == d.gemm_status ? "status" : p == d.err_flag ? "flags" : p == d.tp_block ? "exchange" : "block";
}
std::string name(cudaStream_t st) {
    char b[32];
    snprintf(b, sizeof b, st ? "stream%d" : "default", (int)(size_t)st);
    return b;
}
void note(const std::string& s) { printf("%s\n", s.c_str()); }
void finish(bool all, cudaStream_t st) {
    std::vector<Clear> left;
    for (const Clear& c : pending) {
        if (!all && c.st != st) {
            left.push_back(c);
        }
    }
    pending = left;
}
cudaError_t clear(void* p, int v, size_t n, cudaStream_t st) {
    memset(p, v, n);
    pending.push_back({p, st});
    note("clear " + label(p) + " " + name(st));
    return cudaSuccess;
}
cudaError_t start(const void* f, cudaStream_t st) {
    std::string k = kernels().count(f) ? kernels()[f] : "?";
    if (launches++ == fail_at) {
        note("refused " + k);
        return last = cudaErrorLaunchOutOfResources;
    }
    for (const Clear& c : pending) {
        if (c.st != st) {
            note("UNORDERED " + label(c.p) + " " + name(c.st) + " beside " + k + " " + name(st));
        }
    }
    note("kernel " + k + " " + name(st));
    return cudaSuccess;
}

}  // namespace

extern "C" {
void** __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* device, int, uint3*, uint3*, dim3*, dim3*, int*) { kernels()[host] = device; }
static dim3 cfg_g, cfg_b;
static size_t cfg_m;
static cudaStream_t cfg_s;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, cudaStream_t s) {
    cfg_g = g, cfg_b = b, cfg_m = m, cfg_s = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
    *g = cfg_g, *b = cfg_b, *m = cfg_m, *(cudaStream_t*)s = cfg_s;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t st) { return start(f, st); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) { return start(f, c->stream); }
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = malloc(n);
    memset(*p, 0xA5, n);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { return clear(p, v, n, nullptr); }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) { return clear(p, v, n, st); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    memcpy(d, s, n);
    finish(false, nullptr);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    memcpy(d, s, n);
    note("copy " + name(st));
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
    finish(true, nullptr);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    finish(false, st);
    note("wait " + name(st));
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "stand-in error"; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t* h, void*) {
    memset(h, 0, sizeof *h);
    return cudaSuccess;
}
}

namespace w4 {
// the grouped matmuls: only that they are asked for
bool moe_gemv_plan(int, int, int, int, int, int, MoeGemvPlan&) { return true; }
cudaError_t launch_gemv_moe(const GemvArgs&, const MoeGemvPlan&, cudaStream_t st) { return start(matmul, st); }
int Dec::gemm_ts_grouped(const Lin*, const void*, int, void*, int, const MoeBufs&, int, int, const float*, cudaStream_t st, bool) { return start(matmul, st); }
int Dec::gemm_grouped(const Lin*, const void*, int, void*, int, const MoeBufs&, int, const float*, cudaStream_t st) { return start(matmul, st); }
}  // namespace w4

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (argc > 2) {
        fail_at = atoi(argv[2]);
    }
    kernels()[matmul] = matmul;
    dec = new w4a16_dec();
    auto& d = dec->d;
    const cudaStream_t own = (cudaStream_t)1, other = (cudaStream_t)2;
    d.stream = own;
    cudaMalloc((void**)&d.gemm_status, 4);
    cudaMalloc((void**)&d.err_flag, 16);
    *d.gemm_status = 0;
    int rc = 0;
    if (what == "moe") {
        d.moe = {true, 16, 8, 64, 64, 32, 0, 16};
        d.lins["\x01moe.0.w13"] = w4::Lin{};
        d.lins["\x01moe.0.w2"] = w4::Lin{};
        void* x = aligned_alloc(16, 4096);
        const int t = argc > 3 ? atoi(argv[3]) : 256;
        rc = d.moe_ffn(0, (const float*)x, x, x, t, W4A16_OUT_F32, other);
        note("returned " + std::to_string(rc));
        fail_at = -1;
        rc = d.moe_ffn(0, (const float*)x, x, x, t, W4A16_OUT_F32, other);       // with the scratch of the first call
    } else if (what == "scratch") {
        rc = d.ensure_scratch(1000, 100, other);
        start(matmul, other);
    } else if (what == "status") {
        cudaMalloc((void**)&d.counters, 4);
        d.counters_cap = 1;
        *d.gemm_status = 7 << 16;
        rc = w4a16_kernel_status(dec);
        start(matmul, own);
    } else if (what == "exchange") {
        char h[64];
        rc = w4a16_tp_create(dec, 0, 2, 64, h);
        start(matmul, own);
    } else if (what == "timeline") {
        rc = w4a16_set_tuning(dec, "debug_timeline", 1);
        start(matmul, own);
    } else if (what == "upload") {
        const int n = 32, k = 256, group = argc > 3 ? atoi(argv[3]) : 128, bf16 = argc > 4 ? atoi(argv[4]) : 0;
        std::vector<uint32_t> q(n * k / 8);
        std::vector<uint16_t> s(n * k / group, bf16 ? 0x3c00 : 0x2000);
        rc = d.upload_common("u", q.data(), s.data(), n, k, group, bf16, 0);
    }
    note("returned " + std::to_string(rc));
    return 0;
}
