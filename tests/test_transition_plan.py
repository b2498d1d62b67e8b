"""The row ranges of the Transition backward, through the scratch they ask for (no GPU: the plan is host arithmetic)."""
import ctypes as C

import pytest
import torch

from megafold_b200 import _lib

DIM, INNER = 128, 32


def align(n):
    return -(-n // 256) * 256


def scratch(M):
    a = _lib.TransitionBwdArgs()
    a.M, a.dim, a.inner, a.dtype = M, DIM, INNER, _lib.MF_BF16
    for f in ("x", "ln_w", "w1", "w2", "dy", "dx", "dw1", "dw2", "d_ln_w"):
        setattr(a, f, 256)
    return _lib.lib().mf_transition_bwd_workspace_bytes(C.byref(a))


@pytest.mark.skipif(torch.cuda.is_available(), reason="without a device the plan is that of 148 SMs")
@pytest.mark.parametrize("M", [1, 129, 262144, 262145, 500001, 524288, 524289, *(L * L for L in (800, 1024, 1922, 1924, 1990, 2049, 2500, 4096)), 3694081, 10 ** 7])
def test_ranges_cover_the_rows_once(M):
    """Every range holds rows, none more than the limit in whole waves, and the partial sums are those of the ranges."""
    limit, wave = 262144, 128 * 148
    n = -(-M // limit)
    rows = min(M, M if n == 1 else -(-(-(-M // n)) // wave) * wave)
    n = -(-M // rows)
    assert (n - 1) * rows < M <= n * rows and rows <= -(-limit // wave) * wave
    blocks = min(-(-rows // 128), 148)
    want = align(rows * 64 * 2) + align(rows * 2 * INNER * 2) + align(4 * DIM * 2 * INNER) + align(4 * n * blocks * 2 * DIM)
    assert scratch(M) == want
