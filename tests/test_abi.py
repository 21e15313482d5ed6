"""The shared library loads and exports every symbol the header declares (no GPU needed)."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def built():
    from cinnamon_b200 import build
    return build.build()


def _declared():
    text = open(os.path.join(ROOT, "include", "cinnamon_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(cinn_[a-z0-9_]+)\s*\(", text)))


def test_every_declared_symbol_is_exported(built):
    lib = ctypes.CDLL(built)
    names = _declared()
    assert len(names) >= 10
    for n in names:
        assert hasattr(lib, n), f"{n} declared in include/cinnamon_b200.h but not exported"


def test_binding_table_matches_header(built):
    from cinnamon_b200 import _lib
    assert sorted(_lib.SIGNATURES) == _declared()
    assert _lib.lib.cinn_version() >= 100


def test_bad_arguments_are_reported_not_crashed(built):
    from cinnamon_b200 import _lib
    L = _lib.lib
    # null pointers / bad modes are rejected on the host before any CUDA call
    st = L.cinn_quant_rowwise(None, 0, 4, 128, 128, 1, None, None, 128, 0, 0, None)
    assert st == _lib.ERR_INVALID and "null" in _lib.last_error()
    st = L.cinn_quant_rowwise(ctypes.c_void_p(16), 0, 4, 128, 128, 1, ctypes.c_void_p(16), ctypes.c_void_p(16), 128, 0, 7, None)
    assert st == _lib.ERR_INVALID and "div_mode" in _lib.last_error()
    st = L.cinn_fp8_gemm(ctypes.c_void_p(16), ctypes.c_void_p(16), 1, ctypes.c_void_p(16), ctypes.c_void_p(16), 1, 1,
                         ctypes.c_void_p(16), 128, 128, 100, 0, 0, None)
    assert st == _lib.ERR_INVALID and "multiple of 16" in _lib.last_error()
    with pytest.raises(AssertionError):
        _lib.check(st, "cinn_fp8_gemm")
    # a combine without gates is refused, with and without an addend
    p = ctypes.c_void_p(256)
    assert L.cinn_moe_combine(p, 0, p, None, p, 4, 8, 2, 64, None) == _lib.ERR_INVALID
    assert L.cinn_moe_combine_add(p, 0, p, None, p, 0, p, 4, 8, 2, 64, None) == _lib.ERR_INVALID and "null" in _lib.last_error()
    # empty problems are a successful no-op
    assert L.cinn_quant_rowwise(None, 0, 0, 128, 128, 1, None, None, 128, 0, 0, None) == 0
    assert L.cinn_fp8_gemm(None, None, 1, None, None, 1, 1, None, 0, 128, 128, 0, 0, None) == 0


def test_gemm_plans_under_a_cap_of_one_sm(built):
    """Planning divides tiles by SM pairs: with a cap below two SMs there are none (in a process of its own: this once ended it)."""
    import subprocess
    import sys
    code = ("from cinnamon_b200 import kernels as K\n"
            "for cap in (1, 2, 3):\n"
            "    K.set_gemm_sm_limit(cap)\n"
            "    for M, N, Kd in ((512, 512, 512), (64, 512, 7168), (4096, 4096, 4096)):\n"
            "        for layout in (0, 1):\n"
            "            assert K._L.cinn_fp8_gemm_workspace_bytes(M, N, Kd, layout) >= 0\n")
    p = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, (p.returncode, p.stderr)


def test_routing_workspace_keeps_what_the_built_in_scratch_serves(built):
    """Tokens per CTA grow with the tokens, and the workspace fits the built-in scratch wherever it does at
    the most tokens per CTA."""
    from cinnamon_b200 import _lib
    ints, limit = _lib.lib.cinn_moe_route_workspace_ints, _lib.lib.cinn_moe_route_static_max_ints()
    for E in (1, 8, 33, 256, 511, 1024):
        last = 0
        for T in sorted({int(1.07 ** i) for i in range(1, 200)} | {8192, 8193, 32768, 32769, 65536, 65537}):
            ctas = ints(T, E) // E - 1
            per = -(-T // ctas)
            assert ctas >= -(-T // 128) and per >= 0.9 * last, (T, E, ctas)
            last = per if per > 8 else 0
            if -(-T // 128) * E + E <= limit:
                assert ints(T, E) <= limit, (T, E)


def test_cpu_tensors_assert_like_the_reference(built):
    import torch
    from cinnamon_b200 import kernels as K
    x = torch.randn(4, 128)
    for fn in (K.quantize_fp8_rowwise, K.quantize_fp8_blockwise):
        with pytest.raises(AssertionError, match="CUDA"):
            fn(x)
    with pytest.raises(AssertionError):
        K.dequantize_fp8(x.to(torch.float8_e4m3fn), torch.ones(1, 1))
    # FP8Linear on CPU is an unquantised linear, as in the reference (src/kernels.py:823-824)
    lin = K.FP8Linear(128, 256)
    assert torch.equal(lin(x), torch.nn.functional.linear(x, lin.weight))


def test_convert_to_fp8_selection_rules(built):
    import torch
    from cinnamon_b200 import kernels as K

    class Blk(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.w1 = torch.nn.Linear(256, 512, bias=False)
            self.w3 = torch.nn.Linear(512, 256, bias=True)
            self.attn_proj = torch.nn.Linear(256, 256)
            self.router = torch.nn.Linear(256, 8)
            self.tiny = torch.nn.Linear(64, 256)

    m = torch.nn.Sequential(Blk())
    K.convert_to_fp8(m)
    b = m[0]
    assert isinstance(b.w1, K.FP8Linear) and b.w1.round_scale
    assert isinstance(b.w3, K.FP8Linear) and not b.w3.round_scale and b.w3.bias is not None
    assert type(b.attn_proj) is torch.nn.Linear and type(b.router) is torch.nn.Linear and type(b.tiny) is torch.nn.Linear
    assert sorted(n for n, _ in b.w1.named_parameters()) == ["weight"]


# a CUDA runtime whose launches end as they are told and whose last error is cleared when it is read
RUNTIME = """
int last = 0, next = 0, capturing = 0;                        // errors: what is pending, what the next launch ends with
static int launched() { if (next != 0) last = next; return next; }
extern "C" {
int cudaGetLastError() { const int e = last; last = 0; return e; }
int cudaPeekAtLastError() { return last; }
const char* cudaGetErrorString(int) { return "refused"; }
int cudaLaunchKernel() { return launched(); }
int cudaLaunchKernelExC() { return launched(); }
int cudaStreamIsCapturing(void*, int* status) { *status = capturing; return 0; }
unsigned __cudaPushCallConfiguration() { return 0; }
int __cudaPopCallConfiguration() { return 0; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction() {}
char __cudaInitModule(void**) { return 0; }
}
"""


def _run_over_runtime(tmp_path, program):
    import subprocess
    from cinnamon_b200 import build as B
    exe, runtime, calls = tmp_path / "launch", tmp_path / "runtime.cpp", tmp_path / "calls.cu"
    runtime.write_text(RUNTIME)
    calls.write_text("""
#include "common.cuh"
extern int last, next, capturing;
namespace cinn {
std::atomic<int64_t> g_launches{0};
void set_error(const char*, ...) {}
}
""" + program)
    p = subprocess.run([B._nvcc(), *B.NVCC_FLAGS, "-cudart", "none", "-I" + B.CSRC, str(calls), str(runtime), "-o", str(exe)],
                       capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    return subprocess.run([str(exe)], timeout=60).returncode


def test_a_launch_that_fails_is_reported(built, tmp_path):
    """Early or plain, a launch that the CUDA runtime refuses is an error of the call and counts as none."""
    assert _run_over_runtime(tmp_path, """
__global__ void kernel(int) {}
static int call(bool early) {
    cinn::launch_early_if(early, kernel, dim3(1), dim3(32), 0, nullptr, 1);
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}
int main() {
    for (int early = 0; early < 2; ++early) {
        next = 0;
        if (call(early) != CINN_OK || cinn::g_launches != early + 1) return 10 + early;
        next = cudaErrorInvalidConfiguration;
        if (call(early) != CINN_ERR_CUDA || cinn::g_launches != early + 1 || last != 0) return 20 + early;
    }
    return 0;
}
""") == 0


def test_quantisers_start_early_for_short_rows_and_outside_a_capture(built, tmp_path):
    assert _run_over_runtime(tmp_path, """
int main() {
    using cinn::quantise_early;
    const cudaStream_t s = reinterpret_cast<cudaStream_t>(0x1000);
    if (!quantise_early(4096, 512, s) || quantise_early(4096, 4096, s) || quantise_early(1 << 20, 1024, s)) return 1;
    capturing = cudaStreamCaptureStatusActive;
    if (quantise_early(4096, 512, s) || !cinn::captured(s) || cinn::captured(nullptr)) return 2;
    return 0;
}
""") == 0
