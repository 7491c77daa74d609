"""The update's split of a volume into runs of slices, at shapes that are
checked to be split on the device at hand: a last run of one slice, of two and
of seven, runs of more than eight slices, several tiles, odd widths and even
ones, with and without rejected attempts.  Reference and tolerance are those
of test_gpu_update_runs.py (the FP64 oracle's run2, 1e-4)."""
import ctypes

import pytest

from tomocam_b200 import _lib

from . import test_gpu_update_runs as base

TILE_X, TILE_Y, CTAS = 64, 32, 2  # the update's tile and its CTAs per SM


def _run(n, S, sms):
    f = _lib.lib()["_ZN2tc10update_runEiii"]
    f.argtypes, f.restype = [ctypes.c_int] * 3, ctypes.c_int
    return f(-(-n // TILE_X) * -(-n // TILE_Y), S, CTAS * sms)


@pytest.mark.parametrize("n,S,run", [(24, 8, 8), (24, 9, 9), (24, 10, 8), (300, 24, 8), (512, 64, 32),
                                     (767, 40, 40), (1024, 16, 16), (1024, 256, 64), (1400, 96, 32),
                                     (2048, 256, 256), (2908, 256, 64)])
def test_rule(n, S, run):
    """The runs whose times stand beside the rule, on 148 SMs."""
    assert _run(n, S, 148) == run


@pytest.mark.gpu
@pytest.mark.parametrize("n,S,last", [(24, 10, 2), (25, 17, 1), (32, 31, 7), (100, 25, 1), (129, 18, 2),
                                      (40, 1500, None)])
@pytest.mark.parametrize("reject", [False, True])
def test_split(n, S, last, reject):
    import torch
    run = _run(n, S, torch.cuda.get_device_properties(0).multi_processor_count)
    assert run % 8 == 0 and run < S
    if last is not None:
        assert run == 8 and S % run == last
    else:
        assert run > 8
    base.test_runs(n, S, reject)
