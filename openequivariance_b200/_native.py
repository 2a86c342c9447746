"""ctypes binding of ``liboeq_b200.so`` (C ABI declared in ``include/oeq_b200.h``).

This is the counterpart of the reference's pybind11 module import
(reference: openequivariance/extlib/__init__.py:22-65): the library is built
in-tree with nvcc on first use if it is missing, and every failure surfaces as
a Python exception carrying ``oeq_last_error()``.  There is no fallback path:
if the library cannot be built or loaded the operators do not work.
"""

from __future__ import annotations

import ctypes as C
import os
import threading

import numpy as np

from .wigner import cg_nonzeros

OEQ_OK = 0
OEQ_ERR_INVALID = 1
OEQ_ERR_UNSUPPORTED = 2
ERR_NAMES = {1: "invalid argument", 2: "unsupported problem", 3: "kernel specialisation failed",
             4: "CUDA error", 5: "device-side wait abandoned"}

KIND_BATCH, KIND_CONV_DET, KIND_CONV_ATOMIC = 1, 2, 4
KIND_CONV_SECOND = 8    # with a convolution kind: also the second-derivative kernels of that convolution


class OeqError(RuntimeError):
    def __init__(self, code, message):
        super().__init__(f"oeq_b200: {ERR_NAMES.get(code, code)}: {message}")
        self.code = code


class _Irrep(C.Structure):
    _fields_ = [("mul", C.c_int32), ("l", C.c_int32), ("parity", C.c_int32)]


class _Instruction(C.Structure):
    _fields_ = [("i_in1", C.c_int32), ("i_in2", C.c_int32), ("i_out", C.c_int32), ("mode", C.c_int32),
                ("path_weight", C.c_double), ("cg_nnz", C.c_int32),
                ("cg_i", C.POINTER(C.c_int32)), ("cg_j", C.POINTER(C.c_int32)), ("cg_k", C.POINTER(C.c_int32)),
                ("cg_value", C.POINTER(C.c_double))]


class _ProblemDesc(C.Structure):
    _fields_ = [("n_in1", C.c_int32), ("n_in2", C.c_int32), ("n_out", C.c_int32), ("n_instr", C.c_int32),
                ("in1", C.POINTER(_Irrep)), ("in2", C.POINTER(_Irrep)), ("out", C.POINTER(_Irrep)),
                ("instr", C.POINTER(_Instruction)), ("dtype", C.c_int32), ("shared_weights", C.c_int32)]


# every symbol include/oeq_b200.h declares: name -> (restype, argtypes)
_P, _I64, _SZ, _INT = C.c_void_p, C.c_int64, C.c_size_t, C.c_int
_PI = C.POINTER(C.c_int)
SYMBOLS = {
    "oeq_version": (C.c_char_p, []),
    "oeq_last_error": (C.c_char_p, []),
    "oeq_set_kernel_dir": (_INT, [C.c_char_p]),
    "oeq_set_cache_dir": (_INT, [C.c_char_p]),
    "oeq_precompile": (_INT, [C.POINTER(_ProblemDesc), _INT]),
    "oeq_tp_create": (_INT, [C.POINTER(_ProblemDesc), C.POINTER(_P)]),
    "oeq_tp_destroy": (_INT, [_P]),
    "oeq_tp_weight_numel": (_I64, [_P]),
    "oeq_tp_forward": (_INT, [_P, _I64, _P, _P, _P, _P, _P]),
    "oeq_tp_forward_workspace_bytes": (_SZ, [_P]),
    "oeq_tp_forward_ws": (_INT, [_P, _I64, _P, _P, _P, _P, _P, _SZ, _P]),
    "oeq_tp_workspace_bytes": (_SZ, [_P, _I64]),
    "oeq_tp_backward": (_INT, [_P, _I64, _P, _P, _P, _P, _P, _P, _P, _P, _SZ, _P]),
    "oeq_tp_backward_noalloc": (_INT, [_P, _I64, _P, _P, _P, _P, _P, _P, _P, _P]),
    "oeq_tp_has_double_backward": (_INT, [_P]),
    "oeq_tp_double_backward": (_INT, [_P, _I64, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P]),
    "oeq_tp_check": (_INT, [_P]),
    "oeq_conv_create": (_INT, [C.POINTER(_ProblemDesc), _INT, C.POINTER(_P)]),
    "oeq_conv_destroy": (_INT, [_P]),
    "oeq_conv_workspace_bytes": (_SZ, [_P, _I64, _I64]),
    "oeq_conv_forward": (_INT, [_P, _I64, _I64, _P, _P, _P, _P, _P, _P, _P, _SZ, _P]),
    "oeq_conv_backward": (_INT, [_P, _I64, _I64, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _SZ, _P]),
    "oeq_conv_check": (_INT, [_P]),
    "oeq_conv_last_backward_launches": (_INT, [_P]),
    "oeq_conv_has_double_backward": (_INT, [_P]),
    "oeq_conv_double_backward": (_INT, [_P, _I64, _I64] + [_P] * 14 + [_P, _SZ, _P]),
    "oeq_selftest_bounded_wait": (_INT, [_INT, _P]),
    "oeq_tp_launch_info": (_INT, [_P, _INT, _PI, _PI, _PI, _PI, _PI, _PI]),
    "oeq_conv_launch_info": (_INT, [_P, _INT, _PI, _PI, _PI, _PI, _PI, _PI]),
}

_lib = None
_lock = threading.Lock()


def library_path() -> str:
    return os.path.join(os.path.dirname(os.path.abspath(__file__)), "liboeq_b200.so")


def lib():
    """Load (building first if needed) the shared library; raises if impossible."""
    global _lib
    with _lock:
        if _lib is None:
            from .build import build_library
            path = build_library()
            handle = C.CDLL(path)
            for name, (restype, argtypes) in SYMBOLS.items():
                fn = getattr(handle, name)
                fn.restype, fn.argtypes = restype, argtypes
            _lib = handle
    return _lib


_torch_lib = None
_registered = []    # handles of the registered ops: an op can be called as long as the process lives


def register_ops(forward, gradient, handle, *, deterministic=False, shared=False, has_weights=True, f64=False, dims=(),
                 second=None):
    """Register the torch ops ``openequivariance_b200::<forward>`` and ``::<gradient>`` of one operator (native kernels
    and autograd, ``csrc/oeq_torch.cpp``) and return their overloads.  ``dims``: x, y, z row lengths and the number of
    weights; ``second``: an op already registered that may replace the second derivatives (``call_second``)."""
    global _torch_lib
    import torch
    lib()
    with _lock:
        if _torch_lib is None:
            from .build import build_torch_library
            t = C.CDLL(build_torch_library())
            t.oeq_torch_error.restype = C.c_char_p
            t.oeq_torch_register.argtypes = [C.c_char_p] * 3 + [_P, _P] + [_INT] * 4 + [_I64] * 4
            t.oeq_torch_call_second.argtypes = [C.c_char_p, _INT]
            t.oeq_torch_conv_gradients.argtypes = [C.c_char_p] + [_I64] * 2 + [_P] * 14 + [C.POINTER(_I64), C.POINTER(_P)]
            _torch_lib = t
    is_conv = isinstance(handle, ConvHandle)
    code = _torch_lib.oeq_torch_register(forward.encode(), gradient.encode(), second.encode() if second else None,
                                         None if is_conv else handle.ptr, handle.ptr if is_conv else None,
                                         int(deterministic), int(shared), int(has_weights), int(f64), *dims)
    if code:
        raise RuntimeError("registering torch ops failed: " + _torch_lib.oeq_torch_error().decode(errors="replace"))
    _registered.append(handle)
    ns = torch.ops.openequivariance_b200
    ops = getattr(ns, forward).default, getattr(ns, gradient).default
    z_dim = dims[2]

    @torch.library.register_fake(f"openequivariance_b200::{forward}")
    def _(L1_in, *args):
        return L1_in.new_empty(L1_in.shape[0], z_dim)

    @torch.library.register_fake(f"openequivariance_b200::{gradient}")
    def _(*args):
        return [t.new_empty(*t.shape) for t in args[:3 if has_weights else 2]]

    return ops


def call_second(forward, call: bool):
    """Let the second backward pass of the operator with this forward op call its registered ``second`` op."""
    _torch_lib.oeq_torch_call_second(forward.encode(), int(call))


def conv_gradients(forward, nodes, edges, *pointers):
    """First (``EX``, ``EY``, ``EW``, ``GdZ`` 0) or second derivatives on the current device and stream, with the scratch
    memory that the ops of the operator with this forward op keep.  Returns that memory's size and address."""
    size, address = _I64(0), _P(None)
    code = _torch_lib.oeq_torch_conv_gradients(forward.encode(), nodes, edges, *pointers, C.byref(size), C.byref(address))
    if code < 0:
        raise RuntimeError(_torch_lib.oeq_torch_error().decode(errors="replace"))
    check(code)
    return size.value, address.value or 0


def check(code: int):
    if code != OEQ_OK:
        raise OeqError(code, lib().oeq_last_error().decode(errors="replace"))


class Descriptor:
    """Owns the ctypes arrays behind one ``oeq_problem_desc``."""

    def __init__(self, problem, unit_weights=False):
        modes = {ins.connection_mode for ins in problem.instructions}
        if len(problem.instructions) == 0:
            raise ValueError("Tensor product problem has no valid intructions!")
        assert len(modes) == 1, "all instructions must use the same connection mode"
        mode = modes.pop()
        assert mode in ("uvu", "uvw"), f"connection mode {mode!r} is not supported (uvu and uvw are)"
        assert problem.irrep_dtype == problem.weight_dtype, "irrep_dtype and weight_dtype must match"
        assert problem.irrep_dtype in (np.float32, np.float64)
        for ins in problem.instructions:
            assert ins.has_weight, "every instruction must carry weights"
        self._keep = []

        def irreps(src):
            arr = (_Irrep * max(1, len(src)))()
            for n, (mul, ir) in enumerate(src):
                arr[n] = _Irrep(mul, ir.l, ir.p)
            self._keep.append(arr)
            return arr

        in1, in2, out = irreps(problem.irreps_in1), irreps(problem.irreps_in2), irreps(problem.irreps_out)
        instr = (_Instruction * len(problem.instructions))()
        for n, ins in enumerate(problem.instructions):
            l1 = problem.irreps_in1[ins.i_in1].ir.l
            l2 = problem.irreps_in2[ins.i_in2].ir.l
            l3 = problem.irreps_out[ins.i_out].ir.l
            nz = cg_nonzeros(l1, l2, l3)
            ci = (C.c_int32 * len(nz))(*[t[0] for t in nz])
            cj = (C.c_int32 * len(nz))(*[t[1] for t in nz])
            ck = (C.c_int32 * len(nz))(*[t[2] for t in nz])
            cv = (C.c_double * len(nz))(*[t[3] for t in nz])
            self._keep += [ci, cj, ck, cv]
            instr[n] = _Instruction(ins.i_in1, ins.i_in2, ins.i_out, 0 if mode == "uvu" else 1,
                                    float(ins.path_weight), len(nz), ci, cj, ck, cv)
        self._keep.append(instr)
        self.struct = _ProblemDesc(len(problem.irreps_in1), len(problem.irreps_in2), len(problem.irreps_out),
                                   len(problem.instructions), in1, in2, out, instr,
                                   1 if problem.irrep_dtype == np.float64 else 0,
                                   2 if unit_weights else (1 if problem.shared_weights else 0))

    def ref(self):
        return C.byref(self.struct)


def precompile(problem, kinds: int, unit_weights: bool = False):
    """Specialise the kernels of ``problem`` into the on-disk cache (no GPU needed)."""
    d = Descriptor(problem, unit_weights=unit_weights)
    check(lib().oeq_precompile(d.ref(), kinds))


class _Handle:
    _destroy = None

    def __init__(self):
        self.ptr = _P()

    def __del__(self):
        try:
            if self.ptr and _lib is not None:
                getattr(_lib, self._destroy)(self.ptr)
        except Exception:
            pass

    def _info(self, fn, which):
        vals = [C.c_int() for _ in range(6)]
        check(fn(self.ptr, which, *[C.byref(v) for v in vals]))
        keys = ("threads", "groups_per_cta", "partitions", "stages", "smem_bytes", "registers")
        return dict(zip(keys, (v.value for v in vals)))


class TPHandle(_Handle):
    _destroy = "oeq_tp_destroy"

    def __init__(self, problem):
        super().__init__()
        self.desc = Descriptor(problem)
        check(lib().oeq_tp_create(self.desc.ref(), C.byref(self.ptr)))

    def forward_workspace_bytes(self):
        return lib().oeq_tp_forward_workspace_bytes(self.ptr)

    def forward(self, batch, x, y, w, z, stream, ws=0, ws_bytes=0):
        check(lib().oeq_tp_forward_ws(self.ptr, batch, x, y, w, z, ws, ws_bytes, stream))

    def workspace_bytes(self, batch):
        return lib().oeq_tp_workspace_bytes(self.ptr, batch)

    def backward(self, batch, x, y, w, dz, dx, dy, dw, ws, ws_bytes, stream):
        check(lib().oeq_tp_backward(self.ptr, batch, x, y, w, dz, dx, dy, dw, ws, ws_bytes, stream))

    def has_double_backward(self):
        return bool(lib().oeq_tp_has_double_backward(self.ptr))

    def double_backward(self, batch, x, y, w, dz, ex, ey, ew, gx, gy, gw, gdz, stream):
        check(lib().oeq_tp_double_backward(self.ptr, batch, x, y, w, dz, ex, ey, ew, gx, gy, gw, gdz, stream))

    def check(self):
        check(lib().oeq_tp_check(self.ptr))

    def launch_info(self, which):
        return self._info(lib().oeq_tp_launch_info, which)


class ConvHandle(_Handle):
    _destroy = "oeq_conv_destroy"

    def __init__(self, problem, deterministic, unit_weights=False):
        super().__init__()
        self.desc = Descriptor(problem, unit_weights=unit_weights)
        check(lib().oeq_conv_create(self.desc.ref(), 1 if deterministic else 0, C.byref(self.ptr)))

    def workspace_bytes(self, nodes, edges):
        return lib().oeq_conv_workspace_bytes(self.ptr, nodes, edges)

    def forward(self, nodes, edges, x, y, w, rows, cols, z, ws, ws_bytes, stream):
        check(lib().oeq_conv_forward(self.ptr, nodes, edges, x, y, w, rows, cols, z, ws, ws_bytes, stream))

    def backward(self, nodes, edges, x, y, w, dz, rows, cols, perm, dx, dy, dw, ws, ws_bytes, stream):
        check(lib().oeq_conv_backward(self.ptr, nodes, edges, x, y, w, dz, rows, cols, perm, dx, dy, dw,
                                      ws, ws_bytes, stream))

    def check(self):
        check(lib().oeq_conv_check(self.ptr))

    def last_backward_launches(self):
        return int(lib().oeq_conv_last_backward_launches(self.ptr))

    def has_double_backward(self):
        return bool(lib().oeq_conv_has_double_backward(self.ptr))

    def double_backward(self, nodes, edges, x, y, w, dz, ex, ey, ew, rows, cols, perm, gx, gy, gw, gdz,
                        ws, ws_bytes, stream):
        check(lib().oeq_conv_double_backward(self.ptr, nodes, edges, x, y, w, dz, ex, ey, ew, rows, cols, perm,
                                             gx, gy, gw, gdz, ws, ws_bytes, stream))

    def launch_info(self, which):
        return self._info(lib().oeq_conv_launch_info, which)
