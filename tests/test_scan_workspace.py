"""Workspace of programs with many short steps (host arithmetic, no GPU)."""
import ctypes as C

import pytest


def _bytes(B, D, H, L, steps):
    from lact_b200 import _lib, build
    build.build()
    cfg = _lib.ScanConfig()
    cfg.B, cfg.L, cfg.D, cfg.H, cfg.out_len, cfg.act_dtype, cfg.renorm = B, L, D, H, L, _lib.LACT_BF16, 1
    n = len(steps)
    kind, start, end = ((t * n)(*[s[j] for s in steps]) for j, t in enumerate((C.c_int32, C.c_int64, C.c_int64)))
    need = C.c_size_t(0)
    assert _lib.lib().lact_scan_workspace_bytes(C.byref(cfg), n, kind, start, end, C.byref(need)) == 0
    return need.value - (4 * B * n + 255) // 256 * 256   # (a momentum factor per step and entry)


# APPLY steps of a run keep their weights: 128 MB of them at most beside the ones in force, and 12 tiles of 128 x 128 hidden activations
# per SM (148 where there is no GPU, here or on the device) beside one step's
@pytest.mark.parametrize("B,D,H,chunk", [(1, 384, 384, 64), (4, 512, 512, 64), (1, 1024, 1024, 128), (12, 128, 256, 1), (64, 1024, 1024, 64),
                                         (1, 16, 16, 8)])
@pytest.mark.parametrize("n", [2, 20, 2000])
def test_short_steps_take_a_bounded_workspace(B, D, H, chunk, n):
    from lact_b200 import program as P
    steps = [x for i in range(n) for x in ((P.UPDATE, i * chunk, (i + 1) * chunk), (P.APPLY, i * chunk, (i + 1) * chunk))]
    extra = _bytes(B, D, H, n * chunk, steps) - _bytes(B, D, H, n * chunk, steps[:2])
    assert 0 <= extra <= (128 << 20) + 12 * 148 * 128 * 128 * 2 + 4096


def test_steps_that_form_no_run_take_no_more_than_one():
    from lact_b200 import program as P
    one = _bytes(2, 64, 64, 1000, [(P.UPDATE, 0, 100), (P.APPLY, 0, 100)])
    apart = [(P.UPDATE, 0, 100), (P.APPLY, 0, 100), (P.APPLY, 100, 200), (P.UPDATE, 0, 90), (P.UPDATE, 0, 90), (P.APPLY, 200, 300),
             (P.UPDATE, 0, 90), (P.APPLY, 100, 200), (P.UPDATE, 0, 90), (P.APPLY, 300, 399)]
    assert _bytes(2, 64, 64, 1000, apart) == one
    two = apart + [(P.UPDATE, 0, 90), (P.APPLY, 400, 499), (P.UPDATE, 0, 90), (P.APPLY, 505, 604)]   # uneven: two steps at most
    assert _bytes(2, 64, 64, 1000, two) == _bytes(2, 64, 64, 1000, [(P.UPDATE, 0, 100), (P.APPLY, 0, 99), (P.UPDATE, 0, 90), (P.APPLY, 100, 199)])
