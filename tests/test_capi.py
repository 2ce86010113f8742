"""CPU checks of the C-ABI boundary: the library builds/loads and exports what the header declares."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _header_functions():
    text = open(os.path.join(ROOT, "include", "ghost_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(ghost_[a-z0-9_]+)\s*\(", text)))


def test_header_declares_expected_entry_points():
    names = _header_functions()
    for required in ("ghost_gram_dot_bf16", "ghost_wgrad_bf16", "ghost_persample_dot_bf16",
                     "ghost_colsum", "ghost_layernorm_persample", "ghost_embedding_dot",
                     "ghost_embedding_wgrad", "ghost_gradproj_dense_bf16", "ghost_last_error"):
        assert required in names


def test_library_builds_and_exports_every_declared_symbol():
    from ghostsuite_b200 import build, _lib
    path = build.build()
    assert os.path.exists(path)
    lib = ctypes.CDLL(path)
    for name in _header_functions():
        assert hasattr(lib, name), f"{name} declared in ghost_b200.h but not exported"
    # the ctypes prototypes cover exactly the header
    assert sorted(_lib.PROTOTYPES) == _header_functions()
    lib.ghost_version.restype = ctypes.c_char_p
    assert b"ghost_b200" in lib.ghost_version()


def test_ops_fail_loudly_without_cuda():
    import torch
    from ghostsuite_b200 import ops
    if torch.cuda.is_available():
        pytest.skip("CUDA present")
    A = torch.randn(4, 3, 8)
    with pytest.raises(RuntimeError):
        ops.gram_dot(A, A, 1)
    with pytest.raises(RuntimeError):
        ops.colsum(A)


def test_kernel_switches_validate_their_argument():
    """The process-wide kernel switches need no device: modes 0..2 are accepted, others rejected."""
    from ghostsuite_b200 import build
    lib = ctypes.CDLL(build.build())
    for name, default in (("ghost_set_persample_pair_mode", 1), ("ghost_set_wgrad_pair_mode", 1),
                          ("ghost_set_gram_pair_mode", 1)):
        fn = getattr(lib, name)
        fn.argtypes = [ctypes.c_int]
        fn.restype = ctypes.c_int
        assert fn(-1) < 0 and fn(3) < 0
        for mode in (0, 2, default):
            assert fn(mode) == 0


def test_small_dense_layers_are_bounded_by_the_rows_of_a_tile():
    """A gradient tile of the one-launch kernel walks all train rows in turn: long chains are the GEMM's."""
    from ghostsuite_b200 import _lib
    fits = _lib.load().ghost_dense_small_fits
    # (is_f32, n_train, n_val, T, d, p)
    for args in ((1, 64, 16, 1, 512, 1024), (1, 64, 16, 1, 1024, 10), (1, 768, 8, 1, 64, 64), (1, 1024, 8, 1, 1024, 128),
                 (1, 32, 8, 16, 64, 64), (0, 512, 8, 1, 64, 64)):
        assert fits(*args) == 1, args
    for args in ((1, 16384, 8, 1, 64, 64), (1, 8192, 8, 1, 128, 10), (0, 256, 1, 16, 64, 64), (0, 2048, 1, 8, 128, 10),
                 (1, 2048, 1, 1, 1024, 128), (0, 1024, 1, 1, 64, 64), (1, 64, 1, 16, 64, 64)):
        assert fits(*args) == 0, args


def test_binding_of_another_torch_is_stale(tmp_path, monkeypatch):
    """The binding is compiled against torch's C++ headers: after an upgrade it is built again, not loaded."""
    import shutil
    import torch
    from ghostsuite_b200 import _lib, build
    build.build()
    assert build._torch()[1] == torch.__version__
    assert _lib.binding_built_for(torch.__version__) and not build._binding_stale()
    other = tmp_path / "_ghost_torch.so"
    shutil.copyfile(build.BINDING, other)
    os.utime(other)
    other.write_bytes(other.read_bytes().replace(b"built for torch " + torch.__version__.encode(), b"built for torch 0"))
    monkeypatch.setattr(build, "BINDING", str(other))
    assert build._binding_stale() and not _lib.binding_built_for(torch.__version__, str(other))


_FAKE_RUNTIME = r"""
#include "common.cuh"
namespace gb { int fail(int code, const char*, ...) { return code; } }
static cudaError_t last = cudaSuccess, query = cudaSuccess;      // the runtime's last error; what the query answers
extern "C" {
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = cudaStreamCaptureStatusNone; return last = query; }
cudaError_t cudaGetLastError(void) { cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return ""; }
}
static int refused_launch() { GB_CUDA_OK(last = cudaErrorInvalidConfiguration); return GHOST_OK; }
int main() {
  cudaLaunchAttribute a;
  if (gb::early_start(&a, nullptr) != 1 || last != cudaSuccess) return 1;
  query = cudaErrorStreamCaptureImplicit;
  if (gb::early_start(&a, nullptr) != 0 || last != cudaSuccess) return 2;
  if (refused_launch() != GHOST_ERR_CUDA || last != cudaSuccess) return 3;
  return 0;
}
"""


def test_failed_runtime_calls_leave_no_error_for_the_next_caller(tmp_path):
    """A status that is returned, or dropped, is taken out of the runtime's last error too: the next launch check
    of any library would report it again.  The runtime is a fake here."""
    import subprocess
    from ghostsuite_b200 import build
    cuda = os.path.dirname(os.path.dirname(build._nvcc()))
    src, exe = tmp_path / "fake.cpp", tmp_path / "fake"
    src.write_text(_FAKE_RUNTIME)
    subprocess.run(["g++", "-std=c++17", f"-I{cuda}/include", f"-I{build.CSRC}", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
