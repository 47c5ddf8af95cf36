"""Launchers in a process with several devices: function attributes belong to a device, so whatever a launcher sets once, it
sets once per device.  The launchers' own objects are linked against a stand-in for the runtime that has two devices, notes the
attributes and refuses what the real one refuses: more dynamic shared memory than the device's kernel was allowed."""

import ctypes
import os
import subprocess

import pytest

from paged_llm_b200.csrc import build

FAKE = r"""
#include <cstdint>
#include <map>
#include <mutex>
#include <utility>
#include <cuda_runtime_api.h>
static thread_local int device = 0;
static std::mutex mu;
static std::map<std::pair<int, const void*>, int> allowed;
static int launches = 0;
extern "C" {
void fake_use(int d) { device = d; }
int fake_launches() { return launches; }
void** __cudaRegisterFatBinary(void*) { static void* p; return &p; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
char __cudaInitModule(void**) { return 1; }
cudaError_t __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st*) { return cudaSuccess; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "refused"; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) {
    std::lock_guard<std::mutex> lock(mu);
    allowed[{device, f}] = v;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    std::lock_guard<std::mutex> lock(mu);
    auto it = allowed.find({device, f});
    if ((int)c->dynamicSmemBytes > (it == allowed.end() ? 48 * 1024 : it->second)) return cudaErrorInvalidValue;
    ++launches;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyFromSymbol(void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* c) {
    *n = (device == 0 ? 148 : 74) / c->attrs[0].val.clusterDim.x;
    return cudaSuccess;
}
static int encode(...) { return 0; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *f = (void*)encode;
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char* s, void** f, unsigned, unsigned long long x, cudaDriverEntryPointQueryResult* q) {
    return cudaGetDriverEntryPoint(s, f, x, q);
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    work = tmp_path_factory.mktemp("per_device")
    (work / "fake.cpp").write_text(FAKE)
    nvcc = build.find_nvcc()
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    jobs, objs = [], []
    for src in ("common.cu", "gemm_f32.cu", "attention_f32.cu", "gemm_mid.cu"):
        objs.append(str(work / (src + ".o")))
        jobs.append(subprocess.Popen([nvcc, *build.NVCC_FLAGS, "-Xptxas", "-O0", "-I", build.HERE, "-c", os.path.join(build.HERE, src), "-o", objs[-1]]))
    objs.append(str(work / "fake.o"))
    jobs.append(subprocess.Popen(["g++", "-O1", "-fPIC", "-I", cuda, "-c", str(work / "fake.cpp"), "-o", objs[-1]]))
    assert [j.wait() for j in jobs] == [0] * len(jobs)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs", "-o", str(work / "lib.so"), *objs, "-lpthread"], check=True)
    lib = ctypes.CDLL(str(work / "lib.so"))
    lib.pl_last_error.restype = ctypes.c_char_p
    return lib


def on_both_devices(lib, call):
    for device in (0, 1, 0):
        lib.fake_use(device)
        before = lib.fake_launches()
        assert call() == 0, f"device {device}: {lib.pl_last_error().decode()}"
        assert lib.fake_launches() == before + 1
    lib.fake_use(0)


P, I = ctypes.c_void_p, ctypes.c_int


@pytest.mark.parametrize("M", [1, 8, 32, 2048])
def test_float32_product(lib, M):
    on_both_devices(lib, lambda: lib.pl_gemm_f32(P(4096), P(4096), P(4096), I(M), I(4096), I(2048), I(2048), I(2048), I(4096), P(0)))


@pytest.mark.parametrize("kv", [4096, 4100])
@pytest.mark.parametrize("d", [64, 128, 256])
def test_float32_attention(lib, d, kv):
    from paged_llm_b200.kernels.ops import AttnParams
    p = AttnParams()
    p.q = p.out = p.block_table = p.cu_q = p.k_lens = p.work = 4096
    p.kv = kv
    p.nh, p.nkv, p.d, p.ps, p.n_work, p.max_splits, p.num_pages = 4, 2, d, 16, 3, 1, 8
    on_both_devices(lib, lambda: lib.pl_attention_f32(ctypes.byref(p), P(0)))


@pytest.mark.parametrize("out_float32", [0, 1])
def test_product_of_few_tokens(lib, out_float32):
    on_both_devices(lib, lambda: lib.pl_gemm_mid(P(4096), I(2048), P(4096), P(4096), I(2560), I(24), I(2560), I(2048), I(out_float32),
                                                 P(0), ctypes.c_float(0), P(0)))


def test_threads_meet_at_the_first_call(lib):
    """The first calls of eight threads at once, on two devices: every one is let through."""
    import threading
    codes, gate = [], threading.Barrier(8)

    def work(i):
        lib.fake_use(i % 2)
        gate.wait()
        for _ in range(20):
            codes.append(lib.pl_gemm_mid_silu(P(4096), I(2048), P(4096), P(4096), I(5632), I(24), I(5632), I(2048), I(0), P(0),
                                              ctypes.c_float(0), P(0)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(8)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert codes == [0] * 160
