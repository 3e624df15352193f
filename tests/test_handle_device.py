"""A handle belongs to the device it was made on: with another device current every entry point that would launch,
copy or queue something refuses on the host and leaves the handle as it was, and the readers of status words
synchronise the handle's own device. Two devices are played by a fake CUDA runtime, on the CPU."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "f2k_cuda_b200" / "csrc"
CUDA = Path("/usr/local/cuda/include")

# The runtime calls and launchers that the host sources use. `work` counts what would reach a GPU; the
# fake allocations are host memory, so that status words can be read and cleared.
PROGRAM = r"""
#include "f2k_attn.h"
#include "attn_launch.h"
#include <cstdio>
#include <cstdlib>
#include <cstring>
static int current = 0, work = 0, synchronised = -1;
static CUresult fake_encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                            const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                            CUtensorMapL2promotion, CUtensorMapFloatOOBfill) { return CUDA_SUCCESS; }
static CUresult fake_stream_op(CUstream, CUdeviceptr, cuuint32_t, unsigned int) { ++work; return CUDA_SUCCESS; }
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { current = d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) { *v = a == cudaDevAttrComputeCapabilityMajor ? 10 : 148; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { synchronised = current; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { ++work; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { ++work; return cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void*, size_t, const void*, size_t, size_t, size_t, cudaMemcpyKind, cudaStream_t) { ++work; return cudaSuccess; }
cudaError_t cudaMemcpy3DAsync(const cudaMemcpy3DParms*, cudaStream_t) { ++work; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { ++work; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { ++work; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t*, void*) { return cudaSuccess; }
cudaError_t cudaIpcOpenMemHandle(void**, cudaIpcMemHandle_t, unsigned) { return cudaSuccess; }
cudaError_t cudaIpcCloseMemHandle(void*) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char* name, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *fn = std::strcmp(name, "cuTensorMapEncodeTiled") == 0 ? reinterpret_cast<void*>(fake_encode) : reinterpret_cast<void*>(fake_stream_op);
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
}
namespace f2k {
cudaError_t attn_fwd_prepare() { return cudaSuccess; }
cudaError_t attn_fwd_launch(const AttnParams&, cudaStream_t) { ++work; return cudaSuccess; }
cudaError_t qk_prologue_prepare() { return cudaSuccess; }
cudaError_t qk_prologue_launch(const QkPrologueParams&, cudaStream_t) { ++work; return cudaSuccess; }
cudaError_t qkv_scatter_launch(const QkvScatterParams&, cudaStream_t) { ++work; return cudaSuccess; }
cudaError_t rmsnorm_rows_launch(const void*, const void*, void*, int, int, float, cudaStream_t) { return cudaSuccess; }
cudaError_t rope4_rows_launch(void*, const float*, const float*, const int32_t*, int, int, int, cudaStream_t) { return cudaSuccess; }
}
template <class Call, class Error>
static void refused_elsewhere(const char* name, Call call, Error last_error) {
    current = 0; work = 0;
    if (call() != F2K_ERR_INVALID || work != 0 || !std::strstr(last_error(), "made on device 1, device 0 is current")) {
        std::printf("%s with device 0 current: %d calls reached the GPU, message '%s'\n", name, work, last_error());
        std::exit(1);
    }
    current = 1;
    if (call() != F2K_OK || work == 0) { std::printf("%s with its own device current: '%s'\n", name, last_error()); std::exit(1); }
}
static void status_of(const char* name, int rc) {
    if (rc != F2K_OK || synchronised != 1 || current != 0) {
        std::printf("%s: rc %d, synchronised device %d, device %d current afterwards\n", name, rc, synchronised, current);
        std::exit(1);
    }
    synchronised = -1;
}
int main() {
    alignas(16) static float x[4];                 // never read: only its address is looked at
    alignas(16) static unsigned char host[1 << 16];
    current = 1;
    const f2k_attn_config one_pass{2, 8, 8, 1, 128, 0.f}, row_chunks{1, 0, 1100, 8, 128, 0.f};
    const f2k_seqpar_config rank{1, 64, 2, 128, 1, 0, 0.f}, rank0{1, 64, 2, 128, 2, 0, 0.f};
    f2k_attn *h = nullptr, *rows = nullptr;
    f2k_seqpar* sp = nullptr;
    f2k_hx* hx = nullptr;
    if (f2k_attn_create(&one_pass, &h) || f2k_attn_create(&row_chunks, &rows) || f2k_seqpar_create(&rank0, &sp) || f2k_hx_create(&rank, &hx))
        { std::printf("create\n"); return 1; }
    void* peers[2] = {nullptr, host};
    if (f2k_seqpar_attach(sp, peers)) { std::printf("attach\n"); return 1; }
    auto err = [&] { return f2k_attn_last_error(h); };
    refused_elsewhere("forward", [&] { return f2k_attn_forward(h, x, x, x, x, x, x, x, x, nullptr, 0, nullptr); }, err);
    refused_elsewhere("forward_fused", [&] {
        return f2k_attn_forward_fused(h, x, x, x, x, x, x, x, x, x, x, x, x, x, x, 1e-6f, x, x, host, sizeof host, nullptr); }, err);
    f2k_attn_strides st{};
    refused_elsewhere("forward_fused_strided", [&] {
        return f2k_attn_forward_fused_strided(h, x, x, x, x, x, x, x, x, x, x, x, x, x, x, 1e-6f, x, x, &st, host, sizeof host, nullptr); }, err);
    refused_elsewhere("forward_fused_host", [&] {
        return f2k_attn_forward_fused_host(h, x, x, x, x, x, x, x, x, x, x, x, x, x, x, 1e-6f, x, x, nullptr); }, err);
    refused_elsewhere("forward_fused_host, row chunks", [&] {
        return f2k_attn_forward_fused_host(rows, nullptr, nullptr, nullptr, x, x, x, nullptr, nullptr, x, x, nullptr, nullptr, x, x, 1e-6f,
                                           nullptr, x, nullptr); }, [&] { return f2k_attn_last_error(rows); });
    // own copy stream and compute stream are both the null handle here, which only the form without overlap takes
    refused_elsewhere("seqpar_forward", [&] { return f2k_seqpar_forward(sp, x, x, 0, nullptr, nullptr); }, [&] { return f2k_seqpar_last_error(sp); });
    auto hx_err = [&] { return f2k_hx_last_error(hx); };
    void* o = nullptr;
    for (int form = 0; form < 3; ++form) {
        refused_elsewhere("hx exchange", [&] {
            return (form == 0 ? f2k_hx_exchange_in : form == 1 ? f2k_hx_exchange_in_copy : f2k_hx_forward)(hx, x, x, x, x, x, x, x, 1e-6f, nullptr); }, hx_err);
        if (form < 2) refused_elsewhere("hx_attend", [&] { return f2k_hx_attend(hx, nullptr); }, hx_err);
        refused_elsewhere("hx_output", [&] { return f2k_hx_output(hx, &o, nullptr); }, hx_err);
    }
    current = 0;
    int word = 0;
    status_of("attn status", f2k_attn_device_status(h, &word));
    status_of("seqpar status", f2k_seqpar_device_status(sp, &word));
    status_of("hx status", f2k_hx_device_status(hx, &word));
    f2k_attn_destroy(h); f2k_attn_destroy(rows); f2k_seqpar_destroy(sp); f2k_hx_destroy(hx);
    return 0;
}
"""


def test_calls_with_another_device_current_are_refused(tmp_path):
    if not (CUDA / "cuda.h").exists():
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "devices.cpp", tmp_path / "devices"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "include"), "-I", str(CSRC), "-I", str(CUDA),
                    "-x", "c++", *(str(p) for p in (src, CSRC / "capi.cu", CSRC / "seqpar.cu", CSRC / "headswap.cu")),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
