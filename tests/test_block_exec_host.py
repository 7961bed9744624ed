"""Host side of a decoder block queued by one call (``csrc/block_exec.cu``), on the CPU: its launches are stand-ins that note their arguments."""
import ctypes
import os
import shutil
import subprocess
from pathlib import Path

import pytest

from mini_trainer_b200.ops import block_exec as B

CSRC = Path(__file__).resolve().parent.parent / "mini_trainer_b200" / "csrc"
CUDA_INC = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"

STUBS = r"""
#include "block_exec.cu"
extern "C" {
long long noted[64][2];   // splits and epoch of every product and of the attention backward, in the order of their launches
const char* entered[64];   // by the products among them
int n_noted;
float* last_rstd;
#define GEMM(name) int name(const void*, long long, int, const void*, long long, int, void*, long long, int, const void*, long long, const void*, int, int, int, \
  float, int splits, u64*, u64 epoch, float*, long long, float2*, int*, cudaStream_t) { entered[n_noted] = #name; noted[n_noted][0] = splits; noted[n_noted++][1] = epoch; return 0; }
GEMM(mtb200_gemm_bf16)
GEMM(mtb200_gemm2_bf16)
GEMM(mtb200_gemm2_wide_bf16)
GEMM(mtb200_gemm_n64_bf16)
GEMM(mtb200_gemm_n128_bf16)
int mtb200_gemm_act(const void*, long long, const void*, void*, void*, const void*, int, int, int, int, int, int, int*, cudaStream_t) { return 0; }
int mtb200_swiglu_fwd(const void*, void*, long long, int, cudaStream_t) { return 0; }
int mtb200_geglu_fwd(const void*, void*, long long, int, cudaStream_t) { return 0; }
int mtb200_gelu_fwd(const void*, void*, long long, cudaStream_t) { return 0; }
int mtb200_swiglu_bwd(const void*, const void*, void*, long long, int, cudaStream_t) { return 0; }
int mtb200_swiglu_bwd_act(void*, const void*, void*, long long, int, cudaStream_t) { return 0; }
int mtb200_geglu_bwd(const void*, const void*, void*, long long, int, cudaStream_t) { return 0; }
int mtb200_geglu_bwd_act(void*, const void*, void*, long long, int, cudaStream_t) { return 0; }
int mtb200_gelu_bwd(const void*, const void*, void*, long long, cudaStream_t) { return 0; }
int mtb200_gelu_bwd_act(void*, const void*, void*, long long, cudaStream_t) { return 0; }
int mtb200_rmsnorm_fwd(const void*, const void*, void*, float* rstd, float, int, int, int*, cudaStream_t) { last_rstd = rstd; return 0; }
int mtb200_layernorm_fwd(const void*, const void*, const void*, void*, float*, float* rstd, float, int, int, int*, cudaStream_t) { last_rstd = rstd; return 0; }
int mtb200_norm_bwd_blocks(int, int) { return 148; }
int mtb200_rmsnorm_bwd(const void*, const void*, const float*, const void*, const void*, void*, float*, void*, int, int, int*, cudaStream_t) { return 0; }
int mtb200_layernorm_bwd(const void*, const void*, const float*, const float*, const void*, const void*, void*, float*, void*, void*, int, int, int*,
                         cudaStream_t) { return 0; }
int mtb200_rope(void*, const int*, const float*, int, long long, int, int, int, cudaStream_t) { return 0; }
int mtb200_head_rmsnorm_fwd(void*, const void*, const void*, void*, float*, const int*, const float*, float, int, long long, int, int, int, cudaStream_t) { return 0; }
int mtb200_head_rmsnorm_bwd_blocks(int, int) { return 148; }
int mtb200_head_rmsnorm_bwd(void*, const void*, const float*, const void*, const void*, float*, void*, void*, const int*, const float*, int, long long,
                            long long, int, int, int, cudaStream_t) { return 0; }
int mtb200_attn_fwd(const void*, long long, void*, long long, float*, const int*, int, int, int, int, int, int, float, int*, cudaStream_t) { return 0; }
int mtb200_attn_fwd_one(const void*, long long, void*, long long, float*, const int*, int, int, int, int, int, float, int*, cudaStream_t) { return 0; }
int mtb200_attn_bwd(const void*, long long, const void*, long long, const void*, long long, void*, long long, const float*, float*, float*, const int*, int,
                    int, int, int, int, int splits, u64*, u64 epoch, float*, long long, float, int, int*, cudaStream_t) {
  noted[n_noted][0] = splits; noted[n_noted++][1] = epoch; return 0;
}
int mtb200_colsum(const void*, long long, void*, float*, int, int, cudaStream_t) { return 0; }
}
"""
WS = 1 << 40   # addresses that nothing reads


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None or not CUDA_INC.exists():
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("block_exec")
    (d / "stubs.cpp").write_text(STUBS)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", f"-I{CUDA_INC}", "-o", str(d / "lib.so"), str(d / "stubs.cpp")], check=True)
    lib = ctypes.CDLL(str(d / "lib.so"))
    lib.mtb200_block_workspace.restype = ctypes.c_longlong
    return lib


def make(gated=1, layernorm=0, T=300):
    s = B.Spec(T, 256, 384, 4, 2, 64, gated, 0, layernorm, 0, 1e-5, 0.125, 1.0)
    s.form[:], s.splits[:] = [k % 5 for k in range(B.GEMMS)], [2] * B.GEMMS
    s.need_out, s.bwd_splits = 1, 2
    io = B.IO()
    for name, kind in B.IO._fields_:
        if kind is ctypes.c_void_p and name not in ("n1", "n2", "act", "mean1", "mean2", "qk_pre", "rstd_qk"):
            setattr(io, name, 1 << 20)
    io.ws = WS
    return s, io


def queue(lib, s, io, bwd):
    """(splits, epoch) of the launches that may split."""
    count = ctypes.c_int.in_dll(lib, "n_noted")
    count.value = 0
    epochs = (ctypes.c_ulonglong * (B.GEMMS + 1))(*range(100, 101 + B.GEMMS))
    io.epochs = ctypes.addressof(epochs)
    n, p = ctypes.c_int(0), B.Params()
    args = [ctypes.byref(s), ctypes.byref(p)] + ([ctypes.byref(p)] if bwd else []) + [ctypes.byref(io), ctypes.byref(n), None]
    assert (lib.mtb200_block_backward if bwd else lib.mtb200_block_forward)(*args) == 0
    return [tuple(e) for e in ((ctypes.c_longlong * 2) * count.value).in_dll(lib, "noted")]


@pytest.mark.parametrize("gated", [0, 1])
@pytest.mark.parametrize("bwd", [0, 1])
def test_split_launches_are_numbered_in_the_order_they_are_queued(lib, bwd, gated):
    """Arrivals that a launch which gave up leaves behind do not count in those after it only if these have larger numbers."""
    s, io = make(gated)
    got = queue(lib, s, io, bwd)
    assert len(got) == (9 if bwd else 4) and all(k == 2 for k, _ in got)
    assert all(a < b for (_, a), (_, b) in zip(got, got[1:])), got


@pytest.mark.parametrize("layernorm", [0, 1])
@pytest.mark.parametrize("keep", [(), ("n1",), ("n2",)])
def test_workspace_is_what_the_call_lays_out(lib, keep, layernorm):
    """Statistics of a norm that is formed again come last."""
    s, io = make(layernorm=layernorm, T=321)
    for name in keep:
        setattr(io, name, 1 << 20)
    size = lib.mtb200_block_workspace(ctypes.byref(s), ctypes.byref(io), 1)
    queue(lib, s, io, 1)
    end = ctypes.c_void_p.in_dll(lib, "last_rstd").value - WS + 321 * 4   # the second of two rows
    assert size == -(-end // 256) * 256


def test_structures_have_the_layout_of_the_library(lib, monkeypatch):
    B.check_layout(lib)
    s, io = make(T=321)   # and the sizes it reads give the workspace they should
    per_token = 2 * (768 + 384 + 4 * 256) + 4 * 4 + 4 * 256 + 8   # dgu, dact, dn, n2, dh1, dattn; delta; dq; statistics
    rows, cols = 148 * 256 * 4, 32 * 768 * 4
    size = lib.mtb200_block_workspace(ctypes.byref(s), ctypes.byref(io), 1)
    assert 0 <= size - (321 * per_token + rows + cols) < 16 * 256

    class Short(ctypes.Structure):
        _fields_ = B.Spec._fields_[:-1]
    monkeypatch.setattr(B, "Spec", Short)
    with pytest.raises(RuntimeError, match="another version"):
        B.check_layout(lib)


def test_kernels_of_a_product_are_those_the_plan_names(lib, monkeypatch):
    names = list(B.gemm_plan.FORMS)
    entered = (ctypes.c_char_p * 64).in_dll(lib, "entered")
    for first in range(len(names)):
        s, io = make()
        s.form[:] = [(first + k) % len(names) for k in range(B.GEMMS)]
        queue(lib, s, io, 0)
        assert [entered[k].decode() for k in range(4)] == [names[s.form[k]] for k in range(4)]
    s.form[0] = len(names)   # not a kernel
    n, p = ctypes.c_int(0), B.Params()
    assert lib.mtb200_block_forward(ctypes.byref(s), ctypes.byref(p), ctypes.byref(io), ctypes.byref(n), None) == -10
    monkeypatch.setattr(B.gemm_plan, "FORMS", dict(zip(reversed(names), range(len(names)))))
    with pytest.raises(RuntimeError, match="another version"):
        B.check_layout(lib)
