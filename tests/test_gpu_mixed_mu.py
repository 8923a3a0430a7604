"""Permeability that varies in one or two components only: every stepping
kernel against the CPU oracle, and the vector forms bit for bit against each
other.  Tolerances as for the other small blocks (test_gpu_parity): float64 to
rounding, float32 storage to 1e-4."""
import numpy as np
import pytest

from emopt_b200 import problems as P
from helpers import oracle_for, oracle_lib, rel_l2

pytestmark = pytest.mark.gpu

VARYING = ((0,), (1,), (2,), (0, 1), (0, 2), (1, 2))


def _problem(varying):
    p = P.random_box(seed=71, shape=(7, 9, 70), w_pml=(3, 4, 2, 3, 2, 2), bc="0EH", mu_random=True, n_sources=2,
                     fixed_steps=60)
    mats = list(p.mats)
    for c in range(3):
        if c not in varying:
            mats[3 + c] = np.full(p.shape, 1.0 + 0.25 * c, dtype=np.complex128)
    p.mats = tuple(mats)
    return p


def _fields(p, precision, kernel):
    sim = P.make_solver(p, precision=precision, kernel=kernel)
    names = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
    t0 = [getattr(sim, "_%s_fwd_t0" % c) for c in names]
    sim._solve(t0, t0, sim._sources)
    return np.stack([sim._raw(c, False) for c in names])


@pytest.mark.parametrize("varying", VARYING, ids=lambda v: "mu_" + "".join("xyz"[c] for c in v))
def test_mixed_mu_matches_the_oracle(varying):
    p = _problem(varying)
    ref = np.stack(oracle_for(p, oracle_lib()).solve(fixed_steps=p.fixed_steps)["fields"])
    for precision, tol in (("fp64", 1e-11), ("fp32", 1e-4)):
        F = {k: _fields(p, precision, k) for k in ("scalar", "vector", "split", "fused", "auto")}
        for k, f in F.items():
            assert rel_l2(f, ref) < tol, (precision, k)
        assert np.array_equal(F["fused"], F["vector"])
