"""The extension that packs torch tensors for the packed calls: what a callee sees of every kind of
argument, including more arguments than fit its stack arrays."""
import ctypes
import os
import subprocess
import sys

import pytest
import torch

from sparsetir_b200 import _lib as L
from sparsetir_b200 import build
from sparsetir_b200 import ops


def record(args):
    """Calls a ctypes function through the extension; (return code, what the callee saw)."""
    seen = []

    def callee(values, codes, n, ret, ret_code, handle):
        for i in range(n):
            if codes[i] == L.kTVMDLTensorHandle:
                d = ctypes.cast(values[i].v_handle, ctypes.POINTER(L.DLTensor)).contents
                shape = tuple(d.shape[k] for k in range(d.ndim))
                strides = tuple(d.strides[k] for k in range(d.ndim)) if d.strides else None
                seen.append((d.data, d.device.device_type, shape, strides, d.dtype.code, d.dtype.bits, d.dtype.lanes, d.byte_offset))
            elif codes[i] == L.kTVMArgFloat:
                seen.append(values[i].v_float64)
            elif codes[i] == L.kTVMNullptr:
                seen.append(values[i].v_handle)
            else:
                seen.append((codes[i], values[i].v_int64))
        return 7

    fn = ctypes.CFUNCTYPE(ctypes.c_int, *L.PACKED_ARGTYPES)(callee)
    stream = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_int, ctypes.c_void_p)(lambda device, st: 0)
    rc = L.pycall().invoke(L.entry_address(fn), L.entry_address(stream), args)
    return rc, seen


@pytest.mark.parametrize("dtype,code,bits", [(torch.float32, L.kDLFloat, 32), (torch.float16, L.kDLFloat, 16),
                                             (torch.float64, L.kDLFloat, 64), (torch.int32, L.kDLInt, 32),
                                             (torch.int64, L.kDLInt, 64), (torch.uint8, L.kDLUInt, 8)])
@pytest.mark.parametrize("copies", [1, 60])
def test_callee_sees_the_tensors(dtype, code, bits, copies):
    t = torch.zeros(4, 6, dtype=dtype)
    rc, seen = record((t, t[:, ::2], t.reshape(-1)[5:], t[:0]) * copies + (3, True, 2.5, None, -1))
    assert rc == 7
    row = [(t.data_ptr(), L.kDLCPU, (4, 6), None, code, bits, 1, 0),
           (t.data_ptr(), L.kDLCPU, (4, 3), (6, 2), code, bits, 1, 0),
           (t.data_ptr() + 5 * t.element_size(), L.kDLCPU, (19,), None, code, bits, 1, 0),
           (None, L.kDLCPU, (0, 6), None, code, bits, 1, 0)]
    assert seen == row * copies + [(L.kTVMArgInt, 3), (L.kTVMArgInt, 1), 2.5, None, (L.kTVMArgInt, -1)]


def test_other_arguments_are_left_to_the_general_path():
    assert record((torch.zeros(2, dtype=torch.bfloat16),)) == (None, [])
    assert record((torch.zeros(2), "text")) == (None, [])
    with pytest.raises(TypeError, match="bfloat16"):
        ops.csrmm(torch.zeros(2, dtype=torch.bfloat16))
    with pytest.raises(ops.SparseTIRError, match="no CPU path"):
        ops.csrmm(*[torch.zeros(2)] * 5)


def test_argument_lists_hold_flat_tensors():
    x, y, w, rows, cols = torch.zeros(4, 8), torch.zeros(32), torch.zeros(2, 2), torch.zeros(2), torch.zeros(2, 2)
    args = ops.hyb_args(x, y, [(w, rows, cols)], 8, 4)
    assert [a.dim() for a in args[:5]] == [1] * 5 and args[5:] == [8, 4]
    assert args[0].data_ptr() == x.data_ptr() and args[1] is y


WITHOUT_STORAGE = {
    "vmap": "torch.vmap(call)(torch.zeros(3, 4))",
    "jvp": "torch.func.jvp(call, (torch.zeros(4),), (torch.ones(4),))",
    "fake": """
from torch._subclasses.fake_tensor import FakeTensorMode
with FakeTensorMode():
    call(torch.zeros(4))
""",
}


@pytest.mark.parametrize("where", sorted(WITHOUT_STORAGE))
def test_a_tensor_without_storage_is_a_python_error(where):
    # in a process of its own: the fault to be seen here ends the process
    calls = ["ops.csrmm(t, t, t, t, t)", "ops.csrmm(*[t] * 60)", "ops.hyb_spmm(*ops.hyb_args(t.view(1, -1), t, [(t, t, t)], 4))"]
    code = "import torch\nfrom sparsetir_b200 import ops\n"
    for op in calls:
        body = "".join(f"    {line}\n" for line in WITHOUT_STORAGE[where].strip().splitlines())
        code += f"def call(t):\n    {op}\n    return t\ntry:\n{body}except RuntimeError:\n    print('RuntimeError')\n"
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert (r.returncode, r.stdout.split()) == (0, ["RuntimeError"] * 3), r.stderr[-2000:]


def test_another_torch_builds_the_extension_anew(monkeypatch):
    build.build_pycall()
    ran = []
    monkeypatch.setattr(build.subprocess, "run", lambda cmd, **_: ran.append(cmd) or subprocess.CompletedProcess(cmd, 1, "", ""))
    assert build.build_pycall() == build.PYCALL_PATH and not ran
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    with pytest.raises(RuntimeError, match="g\\+\\+ failed"):
        build.build_pycall()
    assert len(ran) == 1 and '-DSPTIR_TORCH_VERSION="0.0.1"' in ran[0]
    monkeypatch.setattr(L, "_pycall", None)
    with pytest.raises(L.LibraryError, match="this is torch 0.0.1"):
        L.pycall()


def test_the_library_builds_without_torch(monkeypatch):
    monkeypatch.setitem(sys.modules, "torch", None)  # import torch raises ImportError
    assert build.build_pycall(force=True) is None


def test_the_extension_builds_without_cuda(tmp_path):
    out = build.build_pycall(cuda=False, out=str(tmp_path / "_pycall.so"))
    code = ("import importlib.util, torch\n"
            f"spec = importlib.util.spec_from_file_location('_pycall', {out!r})\n"
            "module = importlib.util.module_from_spec(spec)\nspec.loader.exec_module(module)\n"
            "t = torch.zeros(3, 4)\nprint(module.flatten([t])[0].shape == (12,), module.invoke(8, 8, ('text',)))\n")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.stdout.split() == ["True", "None"], r.stderr[-2000:]
    needed = subprocess.run(["readelf", "-d", out], capture_output=True, text=True).stdout
    assert "libc10.so" in needed and "cuda" not in needed.replace("torch_cuda", "")
