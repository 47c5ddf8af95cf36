"""More launchers in a process with several devices (see tests/test_per_device.py): the products of few and of many tokens, the
attention of prompt tiles, the scans of the recurrent mixers, the draw.  The stand-in here also notes what an ordinary launch
asks for, and the size of the last grid."""

import ctypes
import os
import subprocess

import pytest

from paged_llm_b200.csrc import build
from tests.test_per_device import FAKE

PLAIN = "cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }"
COUNTED = r"""
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t) {
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    return last = cudaLaunchKernelExC(&c, f, args);
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int d) { *v = d == 0 ? 148 : 74; return cudaSuccess; }
"""
CONFIG = r"""
static thread_local dim3 pushed_grid, pushed_block;
static thread_local size_t pushed_smem = 0;
static thread_local cudaError_t last = cudaSuccess;
static int grid_x = 0;
extern "C" int fake_grid() { return grid_x; }
"""


def stand_in() -> str:
    text = FAKE.replace('extern "C" {', CONFIG + 'extern "C" {', 1)
    for old, new in (
            (PLAIN, COUNTED),
            ("cudaError_t __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st*) { return cudaSuccess; }",
             "unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, struct CUstream_st*)"
             " { pushed_grid = g; pushed_block = b; pushed_smem = s; return 0; }"),
            ("cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }",
             "cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void*)"
             " { *g = pushed_grid; *b = pushed_block; *s = pushed_smem; return cudaSuccess; }"),
            ("cudaError_t cudaGetLastError() { return cudaSuccess; }",
             "cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }"),
            ("cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) {", "cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {"),
            ("    allowed[{device, f}] = v;\n", "    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) allowed[{device, f}] = v;\n"),
            ("    ++launches;\n", "    ++launches;\n    grid_x = (int)c->gridDim.x;\n")):
        assert text.count(old) == 1, old
        text = text.replace(old, new)
    return text


# a library per source: two of them may name the same entry point
SOURCES = ("gemm_tc", "gemm_skinny", "attention_bf16_d64", "attention_bf16_d128", "ssm", "general_delta", "recurrent", "sampling")


@pytest.fixture(scope="module")
def libs(tmp_path_factory):
    work = tmp_path_factory.mktemp("per_device_launchers")
    (work / "fake.cpp").write_text(stand_in())
    nvcc = build.find_nvcc()
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    # (no device code is run, so none is assembled: PTX alone)
    flags = [f.replace("code=sm_100a", "code=compute_100a") for f in build.NVCC_FLAGS]
    jobs = [subprocess.Popen([nvcc, *flags, "-I", build.HERE, "-c", os.path.join(build.HERE, src + ".cu"), "-o", str(work / (src + ".o"))])
            for src in ("common", *SOURCES)]
    jobs.append(subprocess.Popen(["g++", "-O1", "-fPIC", "-I", cuda, "-c", str(work / "fake.cpp"), "-o", str(work / "fake.o")]))
    assert [j.wait() for j in jobs] == [0] * len(jobs)
    out = {}
    for src in SOURCES:
        path = str(work / (src + ".so"))
        subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs", "-o", path,
                        *[str(work / (o + ".o")) for o in ("common", src, "fake")], "-lpthread"], check=True)
        out[src] = ctypes.CDLL(path)
        out[src].pl_last_error.restype = ctypes.c_char_p
    return out


def on_both_devices(lib, call, launches=1):
    """The call on device 0, 1 and 0 again; the sizes of the last grids."""
    grids = []
    for device in (0, 1, 0):
        lib.fake_use(device)
        before = lib.fake_launches()
        assert call() == 0, f"device {device}: {lib.pl_last_error().decode()}"
        assert lib.fake_launches() == before + launches
        grids.append(lib.fake_grid())
    lib.fake_use(0)
    return grids


P, I, L, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float


def test_product_of_many_tokens(libs):
    lib = libs["gemm_tc"]
    # as many pairs of blocks as the device has pairs of SMs
    assert on_both_devices(lib, lambda: lib.pl_gemm_tc(P(4096), I(2048), P(4096), P(4096), I(8192), P(0), I(2048), I(8192), I(2048), I(2),
                                                       P(0))) == [148, 74, 148]


def test_threads_meet_at_the_first_product(libs):
    """The first calls of eight threads at once, on two devices: every one is let through."""
    import threading
    lib, codes, gate = libs["gemm_skinny"], [], threading.Barrier(8)

    def work(i):
        lib.fake_use(i % 2)
        gate.wait()
        for _ in range(20):
            codes.append(lib.pl_gemm_skinny_silu(P(4096), I(2048), P(4096), P(4096), I(5632), I(8), I(5632), I(2048), P(0), P(0), I(0),
                                                 F(0), I(0), P(0)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(8)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert codes == [0] * 160


@pytest.mark.parametrize("M", [1, 8, 16])
def test_product_of_few_tokens(libs, M):
    lib = libs["gemm_skinny"]
    assert on_both_devices(lib, lambda: lib.pl_gemm_skinny(P(4096), I(2048), P(4096), P(4096), I(32000), I(M), I(32000), I(2048), I(0), P(0),
                                                           P(0), I(0), F(0), I(0), P(0))) == [148, 74, 148]


# pages of 16 tokens, and of 12 (not a power of two: head size 64 alone has a tcgen05 kernel for them); queries that are rotated
# already or not yet
@pytest.mark.parametrize("d,ps,rotated_later", [(64, 16, False), (64, 12, False), (64, 16, True), (128, 16, False), (128, 16, True)])
def test_prompt_tiles(libs, d, ps, rotated_later):
    from paged_llm_b200.kernels.ops import AttnParams
    lib = libs[f"attention_bf16_d{d}"]
    p = AttnParams()
    p.q = p.out = p.kv = p.block_table = p.cu_q = p.k_lens = p.work = 4096
    p.nh, p.nkv, p.d, p.ps, p.n_work, p.max_splits, p.num_pages = 8, 2, d, ps, 3, 1, 8
    p.ps_shift = ps.bit_length() - 1 if ps & (ps - 1) == 0 else -1
    p.q_stride, p.out_stride, p.scale = 12 * d, 8 * d, d ** -0.5
    if rotated_later:
        p.rope_table, p.rope_len = 4096, 1024
    on_both_devices(lib, lambda: getattr(lib, f"pl_attention_bf16_d{d}")(ctypes.byref(p), P(0)))


@pytest.mark.parametrize("N,tokens", [(256, 64), (128, 64), (256, 1)])
def test_state_space_scan(libs, N, tokens):
    lib, H, D, G = libs["ssm"], 4, 64, 1
    inner = H * D
    C = inner + 2 * G * N
    on_both_devices(lib, lambda: lib.pl_ssm_scan(P(4096), I(C), I(inner), I(G), I(N), I(H), I(D), P(4096), P(4096), P(4096), P(4096),
                                                 L(1 << 16), L(0), P(4096), P(4096), I(1), I(tokens), P(4096), P(0)))


@pytest.mark.parametrize("d", [64, 128])
def test_general_delta_step(libs, d):
    lib, H, rank = libs["general_delta"], 4, 64
    on_both_devices(lib, lambda: lib.pl_general_delta_step(P(4096), I(1), I(5 * H * d + rank), P(4096), I(rank), P(4096), P(4096), I(H), I(d),
                                                           F(-0.5), F(1e-6), P(4096), F(1e-6), P(4096), L(1 << 18), P(4096), P(4096), I(2),
                                                           P(4096), P(0)))


@pytest.mark.parametrize("d", [64, 128, 256])
def test_general_delta_chunks(libs, d):
    lib, H = libs["general_delta"], 4
    on_both_devices(lib, lambda: lib.pl_general_delta_chunks(P(4096), I(1), I(5 * H * d), P(4096), P(4096), P(4096), I(H), I(d), F(-0.5),
                                                             F(1e-6), P(4096), I(3), P(4096), L(1 << 18), P(4096), P(4096), I(2), P(4096),
                                                             P(0)), launches=2)


@pytest.mark.parametrize("lanes", [8, 16, 32])
def test_delta_rule_scan(libs, lanes):
    lib, H, G, d, dv = libs["recurrent"], 4, 4, 256, 128
    C = 2 * G * d + H * dv
    on_both_devices(lib, lambda: lib.pl_delta_rule(P(4096), I(C), P(4096), I(1), I(C + 2 * H), I(C), P(4096), P(4096), I(H), I(G), I(d), I(dv),
                                                   F(1e-6), F(1.0), P(4096), P(4096), L(1 << 20), L(0), P(4096), P(4096), I(2), L(64),
                                                   P(4096), I(lanes), P(0)), launches=2)


def test_draw(libs):
    """64 rows of a large vocabulary: two blocks each where the device has an SM for both, else one."""
    lib = libs["sampling"]
    assert on_both_devices(lib, lambda: lib.pl_sample(P(4096), P(4096), I(64), I(128256), L(128256), P(4096), P(4096), P(4096), P(4096),
                                                      P(4096), P(0))) == [128, 64, 128]
