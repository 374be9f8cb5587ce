"""The ring copies (csrc/hostcopy.cu) when host memory runs out: built for the
host against stand-ins of the CUDA calls, with every allocation in turn
refused.  A copy then goes the plain way with the same bytes; nothing throws
out of an entry, and a refused start is reported."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CUDA = r"""
#pragma once
#include <cstddef>
#include <cstdlib>
#include <cstring>
enum cudaError_t { cudaSuccess, cudaErrorMemoryAllocation, cudaErrorNotReady };
typedef struct S* cudaStream_t;
typedef char* cudaEvent_t;
enum { cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost, cudaEventDisableTiming, cudaHostAllocDefault };
enum cudaStreamCaptureStatus { cudaStreamCaptureStatusNone, cudaStreamCaptureStatusActive };
enum cudaMemoryType { cudaMemoryTypeUnregistered, cudaMemoryTypeHost };
struct cudaPointerAttributes { cudaMemoryType type; };
inline cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaHostAlloc(void** p, size_t n, int) { *p = std::malloc(n); return cudaSuccess; }
inline cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, int) { static char c; *e = &c; return cudaSuccess; }
inline cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, int, cudaStream_t) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
inline cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
"""

MAIN = r"""
#include <atomic>
#include <cstdio>
#include <new>
#include <type_traits>
#include <vector>
#include "hostcopy.cuh"
static std::atomic<long> left{1L << 60};
static std::atomic<long> refused{0};
void* operator new(size_t n) {
    if (left.fetch_sub(1) == 0) {
        ++refused;
        throw std::bad_alloc();
    }
    if (void* p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void* operator new(size_t n, const std::nothrow_t&) noexcept {
    if (left.fetch_sub(1) == 0) {
        ++refused;
        return nullptr;
    }
    return std::malloc(n ? n : 1);
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
// attach's answer; one without an answer cannot refuse
template <class F>
bool attach(F f) {
    if constexpr (std::is_void_v<decltype(f())>) {
        f();
        return true;
    } else {
        return f();
    }
}
int main(int argc, char** argv) {
    const long k = std::atol(argv[1]);  // the allocation to refuse
    const size_t n = (25u << 20) + 77;  // several laps of the ring, both ways, helped
    std::vector<unsigned char> host(n), dev(n), back(n);
    for (size_t i = 0; i < n; ++i) host[i] = (unsigned char)(i * 2654435761u >> 13);
    left = k;
    if (!attach([] { return rcmvs::host_copy_attach(); })) {
        left = 1L << 60;
        std::puts("refused");
        return 0;
    }
    const bool ok = rcmvs::host_upload(dev.data(), host.data(), n, nullptr) == cudaSuccess &&
                    rcmvs::host_download(back.data(), dev.data(), n, nullptr) == cudaSuccess;
    left = 1L << 60;
    rcmvs::host_copy_detach();
    std::puts(ok && back == host ? (refused ? "copied" : "untouched") : "wrong");
    return 0;
}
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="needs g++")
def test_copies_survive_refused_allocations(tmp_path):
    csrc = os.path.join(ROOT, "rustcolmap_b200", "csrc")
    (tmp_path / "cuda_runtime.h").write_text(CUDA)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "copies"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{tmp_path}", f"-I{csrc}", str(tmp_path / "main.cpp"),
                    "-x", "c++", os.path.join(csrc, "hostcopy.cu"), "-o", str(exe)], check=True)
    seen = set()
    for k in range(200):
        p = subprocess.run([str(exe), str(k)], capture_output=True, text=True, timeout=60)
        assert p.returncode == 0, f"allocation {k}: {p.returncode} {p.stderr[-200:]}"
        out = p.stdout.strip()
        assert out in ("refused", "copied", "untouched"), f"allocation {k}: {out}"
        seen.add(out)
        if out == "untouched":  # fewer allocations than k
            break
    assert seen == {"refused", "copied", "untouched"}
