"""A request whose handle was solved by itself before admission holds no more of
the engine's budget than a fresh one (the fused step's second field set is given
up), and is served with the same result."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
from emopt_b200 import fdtd_ctypes as ct  # noqa: E402
from emopt_b200 import serving  # noqa: E402

pytestmark = pytest.mark.gpu


def _request(ones):
    spec = serving.RequestSpec(0, (72, 76, 80), 0.04, 1.55, [(-9.0, 9.0, 1.2, 1.7, 1.2, 1.6, 12.25)], w_pml=10, src_k=15,
                               src_yz=(1.5, 1.4), src_w0=0.4, src_phase_y=0.1, fixed_steps=40, precision=32)
    return serving.Request(spec, 0, ones)


def test_budget_after_a_solve_of_its_own():
    ones = torch.ones(72 * 76 * 80, dtype=torch.complex128, device="cuda")
    eng = serving.ServeEngine(0, 10e9, 4, 16)
    used = []
    for solve_first in (False, True):
        req = _request(ones)
        if solve_first:
            req.set_outputs()
            res = ct.SolveResult()
            assert ct.libFDTD.FDTD_solve_cw(req.h, ctypes.byref(req.opt), ctypes.byref(res)) == ct.FDTD_OK
            assert res.zchunk > 0                    # the fused step and its second set
            alone = [a.clone() for a in req.out]
        before = eng.info()[0]
        assert eng.admit(req)
        used.append(eng.info()[0] - before)
        while not (ready := eng.advance()):
            pass
        (done, r), = eng.collect(ready)
        assert done is req and r["steps"] > 40
        torch.cuda.synchronize()
    assert used[1] <= 1.01 * used[0]
    assert all(torch.equal(a, b) for a, b in zip(alone, req.out))
    eng.close()
