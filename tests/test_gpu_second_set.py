"""The second field set of the fused step (kernel 3): coefficients survive a
change of kernel, automatic choice goes on with the pair when the set does not
fit, and a set that an earlier solve left behind makes room for arrays that
every kernel needs.  All results bit for bit those of the pair."""
import numpy as np
import pytest

from emopt_b200 import problems as P
from emopt_b200.fdtd_ctypes import libFDTD

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

NAMES = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
MATS = ("_eps_x", "_eps_y", "_eps_z", "_mu_x", "_mu_y", "_mu_z")
KERNEL = {"fused": 3, "vector": 5}


def _solve(sim):
    t0 = [getattr(sim, "_%s_fwd_t0" % c) for c in NAMES]
    info = sim._solve(t0, t0, sim._sources)
    return np.stack([sim._raw(c, False) for c in NAMES]), info


def _overwrite(sim):
    """What a program does that prepares its next design in the arrays it gave
    to the solver, before it says so."""
    for a in MATS:
        getattr(sim, a)[:] = 5.0


@pytest.mark.parametrize("order", [("vector", "fused"), ("fused", "vector"), ("vector", "auto", "vector")])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_coefficients_survive_a_change_of_kernel(precision, order):
    # x slabs of 3 and 5 cells: the fused step keeps their state in longer rows
    p = P.random_box(seed=81, shape=(9, 10, 70), w_pml=(3, 5, 2, 3, 2, 2), bc="0EH", complex_eps=True, mu_random=True,
                     n_sources=2, fixed_steps=50)
    sim = P.make_solver(p, precision=precision, kernel=order[0])
    ref, _ = _solve(sim)
    _overwrite(sim)
    for k in order[1:]:
        libFDTD.FDTD_set_kernel(sim._libfdtd, KERNEL.get(k, 0))
        F, info = _solve(sim)                       # materials_unchanged = 1
        assert (info["zchunk"] > 0) == (k != "vector")
        assert np.array_equal(F, ref)


# ---- with most of the GPU's memory taken by another allocation
SHAPE = (150, 150, 256)                             # 46 MB an array in float64
ARRAY = 8 * SHAPE[0] * SHAPE[1] * SHAPE[2]


def _problem(lossy):
    return P.random_box(seed=82, shape=SHAPE, w_pml=(8,) * 6, complex_eps=lossy, n_sources=1, fixed_steps=6)


def _free():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _fill_but(leave):
    return torch.empty(_free() - int(leave), dtype=torch.uint8, device="cuda")


def _load_kernels():
    for lossy in (False, True):
        for k in ("vector", "fused"):
            _solve(P.make_solver(P.random_box(seed=83, shape=(6, 7, 70), w_pml=(2,) * 6, complex_eps=lossy,
                                              fixed_steps=6), kernel=k))


@pytest.mark.parametrize("lossy", [False, True])
def test_auto_keeps_the_pair_when_the_second_set_does_not_fit(lossy):
    _load_kernels()
    p = _problem(lossy)
    before = _free()
    sim = P.make_solver(p, kernel="vector")
    ref, _ = _solve(sim)
    pair_bytes = before - _free()
    del sim
    assert _free() >= before - ARRAY
    # the pair's arrays and half a second set (six fields and state): lossy, the
    # pair's arrays without the three factors and a whole second set fit as well
    fill = _fill_but(pair_bytes + 3 * ARRAY)
    sim = P.make_solver(p, kernel="auto")
    F, info = _solve(sim)
    assert info["zchunk"] == 0 and np.array_equal(F, ref)
    _overwrite(sim)
    F, info = _solve(sim)                           # the coefficients stay, also without room
    assert info["zchunk"] == 0 and np.array_equal(F, ref)
    del fill
    _free()
    F, info = _solve(sim)                           # ... and when there is room again
    assert info["zchunk"] > 0 and np.array_equal(F, ref)


def test_a_second_set_left_behind_makes_room():
    _load_kernels()
    p = _problem(False)
    sim = P.make_solver(p, kernel="auto")
    _, info = _solve(sim)
    assert info["zchunk"] > 0
    fill = _fill_but(2 * ARRAY)
    libFDTD.FDTD_set_complex_eps(sim._libfdtd, True)   # three more arrays
    F, info = _solve(sim)
    assert info["zchunk"] == 0
    del fill
    _free()
    q = _problem(False)
    q.complex_eps = True
    ref, _ = _solve(P.make_solver(q, kernel="vector"))
    assert np.array_equal(F, ref)
