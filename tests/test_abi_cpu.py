"""The C-ABI library loads without a GPU and exports every symbol the header declares."""
import ctypes
import os
import re

import numpy as np
import pytest

from conftest import ROOT, problem_by_name


def header_functions():
    text = open(os.path.join(ROOT, "include", "oeq_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(oeq_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    from openequivariance_b200 import _native
    lib = _native.lib()
    names = header_functions()
    assert len(names) >= 20
    for name in names:
        assert hasattr(lib, name), f"{name} is declared in include/oeq_b200.h but not exported"
        assert name in _native.SYMBOLS, f"{name} has no ctypes signature"
    assert b"sm_100a" in lib.oeq_version()


def test_torch_library_shares_the_cxx_runtime(monkeypatch, tmp_path):
    """A private copy of libstdc++ (what a compiler named by $CXX may link) crashes on the first formatted message."""
    import subprocess
    from openequivariance_b200 import build
    fake = tmp_path / "cxx"
    fake.write_text("#!/bin/sh\nexec g++ -static-libstdc++ \"$@\"\n")
    fake.chmod(0o755)
    monkeypatch.setenv("CXX", str(fake))
    monkeypatch.setattr(build, "torch_library_path", lambda: str(tmp_path / "lib.so"))
    out = subprocess.run(["readelf", "-d", build.build_torch_library()], capture_output=True, text=True, check=True).stdout
    assert "libstdc++.so" in out


def test_descriptor_errors_are_reported_not_fatal():
    from openequivariance_b200 import _native
    lib = _native.lib()
    out = ctypes.c_void_p()
    assert lib.oeq_tp_create(None, ctypes.byref(out)) == 1
    assert b"null" in lib.oeq_last_error()
    p = problem_by_name("uvw_small")
    d = _native.Descriptor(p)
    d.struct.dtype = 7
    assert lib.oeq_tp_create(d.ref(), ctypes.byref(out)) == 1
    # a fused convolution over a 'uvw' problem is outside the supported set
    d2 = _native.Descriptor(p)
    assert lib.oeq_conv_create(d2.ref(), 1, ctypes.byref(out)) == 2
    assert b"uvu" in lib.oeq_last_error()


def test_front_end_rejects_what_the_reference_rejects():
    import openequivariance_b200 as oeq
    with pytest.raises(AssertionError):      # mixed connection modes
        oeq.TensorProduct(oeq.TPProblem("2x0e", "2x0e", "2x0e", [(0, 0, 0, "uvu", True), (0, 0, 0, "uvw", True)],
                                        shared_weights=False, internal_weights=False), torch_op=True)
    with pytest.raises(AssertionError):      # conv needs multiplicity 1 in the second input
        oeq.TensorProductConv(problem_by_name("uvu_v2"), torch_op=True)
    with pytest.raises(AssertionError):      # dtypes must agree
        oeq.TensorProduct(problem_by_name("readme", irrep_dtype=np.float64), torch_op=True)


def test_kernels_specialise_without_a_gpu(tmp_path):
    """Run-time specialisation (NVRTC for sm_100a) needs no device; the cache is keyed by content."""
    from openequivariance_b200 import _native
    lib = _native.lib()
    lib.oeq_set_cache_dir(str(tmp_path).encode())
    try:
        _native.precompile(problem_by_name("readme"), _native.KIND_BATCH | _native.KIND_CONV_DET)
        files = sorted(os.listdir(tmp_path))
        # batch forward / backward / one-pass second derivatives, convolution forward, sender-order and
        # receiver-order backward
        assert len(files) == 6 and all(f.endswith(".cubin") for f in files)
        _native.precompile(problem_by_name("readme"), _native.KIND_BATCH)
        assert sorted(os.listdir(tmp_path)) == files
    finally:
        lib.oeq_set_cache_dir(os.path.join(os.path.dirname(_native.library_path()), "_kcache").encode())


@pytest.mark.parametrize("mul,in1,in2,dtype,atomic,kernels", [
    (128, "0e+1o+2e", "0e+1o+2e", "float32", True, 3),      # forward and backward in slices, the sender-order kernel behind
    (128, "0e+1o+2e", "0e+1o+2e", "float32", False, 3),
    (64, "0e+1o+2e+3o", "0e+1o+2e", "float32", False, 3),
    (128, "0e+1o+2e", "0e+1o+2e", "float64", False, 3),
    (128, "0e+1o+2e", "0e+1o", "float64", False, 3),
    (128, "0e+1o+2e", "0e+1o", "float64", True, 4),         # the additions of wide FP64 rows: receiver-order kernel for large lists
    (64, "0e+1o+2e", "0e+1o", "float64", True, 3),
    (128, "0e+1o", "0e+1o+2e", "float64", True, 3),
])
def test_edge_sums_leave_large_lists_to_the_slice_kernels(tmp_path, mul, in1, in2, dtype, atomic, kernels):
    """Group kernels for large lists are specialised where they are the faster ones, which sums of products hardly ever are."""
    import openequivariance_b200 as oeq
    from openequivariance_b200 import _native
    from openequivariance_b200.conv import UVWConvPlan
    wide, dt = "+".join(f"{mul}x{ir}" for ir in in1.split("+")), getattr(np, dtype)
    p = oeq.FullyConnectedTPProblem(wide, in2, wide, irrep_dtype=dt, weight_dtype=dt)
    lib = _native.lib()
    lib.oeq_set_cache_dir(str(tmp_path).encode())
    try:
        _native.precompile(UVWConvPlan(p).edge_sum, _native.KIND_CONV_ATOMIC if atomic else _native.KIND_CONV_DET, unit_weights=True)
        assert len(os.listdir(tmp_path)) == kernels
    finally:
        lib.oeq_set_cache_dir(os.path.join(os.path.dirname(_native.library_path()), "_kcache").encode())
