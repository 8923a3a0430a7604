"""The batched in-place inverses of the mode solver's line blocks
(FDTD_mode_invert) against numpy: sizes around the panel (16 columns, 8 or
4 for blocks of more than 640 or 1280 rows) and the 64 x 64 tile,
a permutation (every pivot off the diagonal), lines in any order with untouched
ones between, and singular blocks.

Tolerance: Gauss-Jordan with partial pivoting leaves a residual of about
n eps |A| |X|; |I - A X| / (n eps |A| |X|) stays below 1 by far on random blocks
(16 allows for the growth of the elimination)."""
import ctypes

import numpy as np
import pytest
import torch

from emopt_b200 import fdtd_ctypes as ct
from emopt_b200 import modes  # noqa: F401  (declares the two routines)

pytestmark = pytest.mark.gpu
lib = ct.libFDTD


def _invert(W, lines):
    dev = torch.device("cuda", 0)
    nb = W.shape[1]
    d = torch.as_tensor(W, device=dev).contiguous()
    l32 = torch.as_tensor(lines, dtype=torch.int32, device=dev)
    need = lib.FDTD_mode_invert_work(nb, len(lines))
    assert need > 0
    work = torch.empty(need, dtype=torch.uint8, device=dev)
    info = torch.full((len(lines),), 7, dtype=torch.int32, device=dev)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    assert lib.FDTD_mode_invert(nb, 0, torch.cuda.current_stream(dev).cuda_stream, p(d), p(l32), len(lines), p(work),
                                need, p(info)) == ct.FDTD_OK
    return d.cpu().numpy(), info.cpu().numpy()


@pytest.mark.parametrize("nb", [1, 2, 6, 15, 16, 17, 33, 64, 65, 130, 606, 641, 900, 1290])
def test_inverse_of_random_blocks(nb):
    rng = np.random.default_rng(nb)
    n = 5 if nb < 600 else 2
    W = rng.standard_normal((n, nb, nb)) + 1j * rng.standard_normal((n, nb, nb))
    W[0] = np.roll(np.eye(nb), 1, axis=0) * (1 + 2j)
    lines = [n - 1, 0] if n == 2 else [3, 0, 4]
    X, info = _invert(W, lines)
    assert not info.any()
    for q in range(n):
        if q not in lines:
            assert np.array_equal(X[q], W[q])
            continue
        res = np.linalg.norm(np.eye(nb) - W[q] @ X[q])
        assert res <= 16 * nb * np.finfo(float).eps * np.linalg.norm(W[q]) * np.linalg.norm(X[q])


def test_singular_blocks_are_reported():
    W = np.stack([np.eye(20, dtype=complex) * 3, np.zeros((20, 20), dtype=complex), np.eye(20, dtype=complex)])
    W[2, 4, 4] = np.nan
    X, info = _invert(W, [0, 1, 2])
    assert list(info) == [0, 1, 1]
    assert np.allclose(X[0], np.eye(20) / 3)
    assert lib.FDTD_mode_invert_work(100000, 1) == 0
