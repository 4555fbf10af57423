"""Argument handling of the native half of ``kaio_b200.ops``, as far as it shows without a GPU: what a call
took and refused when every argument went through ctypes."""
import numpy as np
import pytest
import torch

from kaio_b200 import ops


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
