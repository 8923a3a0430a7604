"""The automatic choice of the stepping kernel, read from the solve's result:
only the fused step cuts z chunks (zchunk), the split pair has two launches per
half step but counts as the pair."""
import numpy as np
import pytest

from emopt_b200 import problems as P

pytestmark = pytest.mark.gpu

# precision, shape (Nz, Ny, Nx), CPML cells, is the fused step taken?
CASES = [
    # rows of at most 16 vectors
    ("fp32", (44, 48, 64), 10, False), ("fp32", (44, 48, 65), 10, True),
    ("fp64", (44, 48, 32), 10, False), ("fp64", (44, 48, 33), 10, True),
    # launch- and latency-bound grids, one row of cells among them
    ("fp64", (90, 90, 62), 15, True), ("fp64", (100, 1, 128), 10, True), ("fp32", (100, 1, 256), 10, True),
    ("fp32", (59, 87, 149), 12, True), ("fp64", (65, 76, 101), 15, True), ("fp64", (51, 81, 161), 10, True),
    # few rows on a long grid: 16.8 us a step against 39.4 by the fused step
    ("fp64", (1082, 1, 324), 0, False), ("fp64", (171, 33, 126), 15, False),
    ("fp32", (500, 1, 512), (0, 0, 0, 0, 120, 120), False),
    ("fp64", (486, 1, 88), 10, False), ("fp64", (791, 2, 179), 0, False),
    # where the pair would be the split one (20.8 us against 13.9; 28.0 against 33.8)
    ("fp32", (300, 1, 512), 10, True), ("fp32", (947, 1, 580), 12, False),
    # x-slab state of a tile wider than a box copy: 35.1 us against 40.0
    ("fp64", (90, 90, 72), 15, False), ("fp64", (136, 79, 62), 12, False),
    # x slabs that share a vector (the fused step is not possible)
    ("fp32", (12, 13, 70), (33, 36, 2, 2, 2, 2), False),
]


def _solve(p, precision, kernel):
    sim = P.make_solver(p, precision=precision, kernel=kernel)
    names = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
    t0 = [getattr(sim, "_%s_fwd_t0" % c) for c in names]
    info = sim._solve(t0, t0, sim._sources)
    return np.stack([sim._raw(c, False) for c in names]), info


@pytest.mark.parametrize("precision,shape,w,fused", CASES)
def test_auto_choice(precision, shape, w, fused):
    if isinstance(w, int):
        w = tuple(min(w, n // 3) if n >= 12 else 0 for n in shape[::-1] for _ in range(2))
    p = P.random_box(seed=91, shape=shape, w_pml=w, fixed_steps=4)
    _, info = _solve(p, precision, "auto")
    assert (info["zchunk"] > 0) == fused


def test_auto_gives_the_bits_of_either_kernel():
    p = P.random_box(seed=92, shape=(136, 79, 62), w_pml=(12,) * 6, fixed_steps=20, n_sources=2)
    A, info = _solve(p, "fp64", "auto")
    B, forced = _solve(p, "fp64", "fused")
    assert info["zchunk"] == 0 and forced["zchunk"] > 0
    assert np.array_equal(A, B)
