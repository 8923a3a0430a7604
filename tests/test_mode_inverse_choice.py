"""Which line blocks FDTD_mode_invert takes (host rule), and that the mode solver
gives the same modes whichever routine inverts them (GPU)."""
import numpy as np
import pytest

from emopt_b200 import modes


@pytest.mark.parametrize("nb,n,own", [
    (1, 1, True), (606, 1, True), (640, 80, True), (640, 5000, True),       # always up to 640 rows
    (641, 1, False), (641, 2, True), (641, 70, True), (641, 71, False),     # one block: the library
    (900, 50, True), (900, 51, False), (900, 80, False), (1280, 24, True), (1280, 50, False),
    (1281, 7, True), (1281, 8, False), (1400, 16, False), (2400, 3, True), (2400, 16, False),
    (2560, 3, True), (2560, 4, False),
])
def test_rule(nb, n, own):
    assert modes._own_inverse(nb, n) is own


@pytest.mark.gpu
@pytest.mark.parametrize("pick", [lambda nb, n: False, lambda nb, n: n != 1, lambda nb, n: n == 1])
def test_modes_do_not_depend_on_the_choice(pick, monkeypatch):
    from test_gpu_modes import D, WL, strip
    from emopt_b200.grid import FunctionMaterial3D
    from emopt_b200.misc import DomainCoordinates

    def solve():
        dom = DomainCoordinates.from_indices(5, 6, 0, 36, 0, 24, D, D, D)
        m = modes.ModeFullVector(WL, FunctionMaterial3D(strip(0.7, 0.46), D, D, D),
                                 FunctionMaterial3D(lambda x, y, z: np.ones(np.shape(x)) + 0j, D, D, D), dom, n0=3.0,
                                 neigs=3, device=0)
        m.bc = ["0", "0"]
        m.build()
        m.solve()
        return np.array(m.neff)

    ref = solve()
    monkeypatch.setattr(modes, "_own_inverse", pick)
    # both residuals are at rounding level; the tolerance of the oracle comparison
    assert np.max(np.abs(solve() - ref) / np.abs(ref)) < 1e-10
