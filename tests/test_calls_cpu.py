"""The extension module's calls take and refuse what ctypes does, and reach the same library."""
import ctypes

import numpy as np
import pytest

from cunn_b200._lib import calls, lib

GEO = (64, 32, 112, 112, 1, 3, 3, 1, 1, 1, 1)


def outcome(f, *args):
    try:
        return f(*args)
    except (ctypes.ArgumentError, TypeError) as e:
        return type(e)


@pytest.mark.parametrize("arg", [64, True, np.int32(7), np.int64(3), -1, 2 ** 31, 2 ** 32 + 5, -2 ** 70, 1.0, "1", None, [1]])
def test_integers(arg):
    for name in ("cunn_b200_dwconv_acc_grad_workspace", "cunn_b200_convmm_acc_grad_workspace"):
        assert outcome(getattr(calls, name), arg, *GEO[1:]) == outcome(getattr(lib, name), arg, *GEO[1:])
    assert outcome(calls.cunn_b200_maxpool_out_size, arg, 3, 2, 1, 1, 1) == outcome(lib.cunn_b200_maxpool_out_size, arg, 3, 2, 1, 1, 1)


@pytest.mark.parametrize("arg", [None, 0, 1.0, np.float32(1), True])
def test_pointers_and_numbers(arg):
    """n = 0 returns before anything is read."""
    for L in (calls, lib):
        assert outcome(L.cunn_b200_sgd_update, None, None, 0, 0.5, None) == 0
    for at in (0, 3):
        args = [None, None, 0, 0.5, None]
        args[at] = arg
        assert outcome(calls.cunn_b200_sgd_update, *args) == outcome(lib.cunn_b200_sgd_update, *args)


def test_too_few_arguments():
    assert outcome(calls.cunn_b200_dwconv_acc_grad_workspace, *GEO[1:]) is TypeError


def test_errors_reach_the_caller():
    """A call that is refused leaves its message for the thread that made it."""
    assert calls.cunn_b200_dwconv_forward(None, None, None, None, *GEO, None) != 0
    assert b"null" in lib.cunn_b200_last_error()


def test_small_pointwise_layers_have_no_use_for_scratch():
    """What functional.py does not ask for is 0: both sides of the limit, by the tensor that the pass reads."""
    limit = calls.CONV_POINT_VALUES
    N, H, W = 8, 7, 9
    for which in range(3):
        sizes = []
        for C in range(limit // (N * H * W) - 300, limit // (N * H * W) + 300, 50):
            cin, cout = (64, C) if which == 1 else (C, 512)
            need = calls.cunn_b200_conv_scratch(which, N, cin, H, W, cout, 1, 1, 1, 1, 0, 0, 1, 1)
            assert need == 0 or N * C * H * W >= limit
            sizes.append(need)
        assert which == 2 or any(sizes)


def test_module_of_this_python():
    """A module built for another version of Python is another file: it is neither loaded nor taken for one that is up to date."""
    import os
    import sysconfig
    from cunn_b200 import build
    assert os.path.basename(calls.__spec__.origin) == os.path.basename(build.CALLS) == "_calls" + sysconfig.get_config_var("EXT_SUFFIX")
