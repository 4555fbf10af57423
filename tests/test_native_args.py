"""Argument handling of the native half of ``kaio_b200.ops``, as far as it shows without a GPU: what a call
took and refused when every argument went through ctypes."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from kaio_b200 import ops

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def refused(exc, fn, *args, match=None):
    with pytest.raises(exc, match=match):
        fn(ops.KaioDevice(0), *args)


def test_integers_of_other_types_are_integers():
    """Sizes come from numpy shapes and integer tensors too.  A budget of 0 is refused by the library and
    anything else needs a device, so no call gets as far as a kernel."""
    for zero in (0, np.int64(0), np.uint32(0), torch.tensor(0), False):
        with pytest.raises(Exception) as e:
            ops.selftest_bounded_wait(ops.KaioDevice(0), zero)
        assert not isinstance(e.value, TypeError), e.value
    for bad in (0.0, "0", None):
        refused(TypeError, ops.selftest_bounded_wait, bad, match="budget_us: expected an int")


def test_more_addresses_than_ranks_are_refused():
    t = torch.zeros(1)
    for fn, args in [
            (ops.matmul_int4_allgather, (t, t, t, [1, 2, 3], 8, 2, 0, 1, 16, 128, 128)),
            (ops.matmul_int4_allgather_multicast, (t, t, t, range(1, 11), 8, 4096, 8, 0, 1, 64, 128, 128)),
            (ops.matmul_int4_peer_partials, (t, t, t, [1, 2], 8, 1, 0, False, 1, 16, 128, 128))]:
        refused(IndexError, fn, *args, match="device addresses for")


def test_a_scale_that_is_no_tensor_is_named():
    t, s = torch.zeros(1), torch.ones(1)
    refused(TypeError, ops.qkv_project_w8a8, t, t, t, t, 0.5, s, s, t, t, t, 1, 16, 32, match="scale_q: expected a torch.Tensor")
    refused(TypeError, ops.qkv_project_w8a8, t, t, t, t, s, s, None, t, t, t, 1, 16, 32, match="scale_v: expected a torch.Tensor")
    refused(TypeError, ops.qkv_project_int8, t, t, t, t, s, 0.5, s, t, t, t, 1, 16, 32, match="scale_k: expected a torch.Tensor")


def test_a_device_of_another_type_is_asked_for_its_stream():
    class Pool(ops.KaioDevice):
        def stream_handle(self):
            raise KeyError("no stream left")

    class Plain:
        ordinal = 0

        def stream_handle(self):
            raise KeyError("no stream left")

    for d in (Pool(0), Plain()):
        with pytest.raises(KeyError):
            ops.selftest_bounded_wait(d, 5)


def test_a_wrong_dtype_is_named_as_torch_names_it():
    a = torch.zeros(4, dtype=torch.int8)
    for dtype in (torch.float64, torch.bfloat16, torch.uint8, torch.int16, torch.int64, torch.bool, torch.float32):
        refused(TypeError, ops.matmul_int8, a.to(dtype), a, a, 1.0, 1, 1, 32, match=f"a: expected dtype torch.int8, got {dtype}")


def test_the_extension_is_rebuilt_for_another_torch(monkeypatch, tmp_path):
    from kaio_b200 import build
    for name in ("NATIVE", "NATIVE_STAMP"):
        monkeypatch.setattr(build, name, str(tmp_path / name))
    (tmp_path / "NATIVE").write_text("")
    assert not build.native_is_current()  # no stamp
    (tmp_path / "NATIVE_STAMP").write_text(build._native_key())
    assert build.native_is_current()
    monkeypatch.setattr(torch, "__version__", "0.0")
    assert not build.native_is_current()


def test_the_extension_of_another_torch_does_not_load():
    code = ("import torch; torch.__version__ = '0.0'\n"
            "from kaio_b200 import ops\n"
            "try: ops.selftest_bounded_wait(ops.KaioDevice(0), 0)\n"
            "except RuntimeError as e: print(e)")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert "built for torch" in r.stdout and "kaio_b200.build" in r.stdout, r.stdout + r.stderr
