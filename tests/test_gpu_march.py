"""The fused time step (kernel 3, auto's choice for most grids) against the
kernels it replaces, bit for bit: grids around the edges of its tiles (120
float32 / 60 float64 cells, 7 rows, z chunks), CPML slabs that are absent, a
few cells wide or wider than what one box copy of their state holds, every
boundary letter, lossy media, mu arrays, and current boxes on faces, across
tiles and as a whole x-normal sheet."""
import numpy as np
import pytest

from emopt_b200 import problems as P

pytestmark = pytest.mark.gpu

# shape (Nz, Ny, Nx), six CPML widths, further arguments of random_box
GRIDS = {
    "tile_edge": ((9, 7, 128), (3, 4, 2, 3, 2, 3), dict(bc="000", n_sources=2)),
    "tile_edge_plus_1": ((9, 8, 129), (3, 4, 2, 3, 2, 3), dict(bc="E0H", n_sources=2, edge_source=True)),
    "two_tiles": ((14, 15, 248), (2, 0, 0, 4, 3, 0), dict(bc="0EH", complex_eps=True, n_sources=3)),
    "f64_tile_edge": ((5, 14, 64), (0, 3, 3, 0, 0, 2), dict(bc="HE0", mu_random=True, n_sources=2)),
    "one_plane": ((1, 9, 70), (3, 3, 2, 2, 0, 0), dict(bc="000")),
    "one_row": ((12, 1, 70), (0, 0, 0, 0, 3, 4), dict(bc="000")),
    "narrow": ((6, 5, 6), (2, 1, 1, 2, 1, 2), dict(bc="EEE", n_sources=2)),
    "wide_slabs": ((21, 23, 200), (47, 61, 9, 10, 7, 8), dict(bc="000", complex_eps=True, mu_random=True)),
    "no_slabs": ((33, 16, 181), (0,) * 6, dict(bc="H0E", n_sources=16)),
    "mostly_interior": ((40, 40, 640), (2,) * 6, dict(bc="000", n_sources=2)),
}
SPLIT = ("no_slabs", "mostly_interior")


def _fields(p, precision, kernel):
    sim = P.make_solver(p, precision=precision, kernel=kernel)
    names = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
    t0 = [getattr(sim, "_%s_fwd_t0" % c) for c in names]
    info = sim._solve(t0, t0, sim._sources)
    return np.stack([sim._raw(c, False) for c in names]), info


def _with_sheet(p):
    Nz, Ny, Nx = p.shape
    rng = np.random.default_rng(5)
    k = min(5, Nx - 1)
    p.sources = p.sources[:15] + [([rng.standard_normal((Nz, Ny, 1)) + 1j * rng.standard_normal((Nz, Ny, 1))
                                    for _ in range(6)], 0, 0, k)]
    return p


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("name", list(GRIDS))
def test_fused_step_equals_the_pair(name, precision):
    shape, w, kw = GRIDS[name]
    p = _with_sheet(P.random_box(seed=60, shape=shape, w_pml=w, fixed_steps=41, **kw))
    Ff, fi = _fields(p, precision, "fused")
    # the pair that auto would take without it: split where at least 60% of the
    # float32 warp tasks lie in no slab (its interior body rounds the tasks a
    # source touches differently)
    Fp, pi = _fields(p, precision, "split" if name in SPLIT and precision == "fp32" else "vector")
    assert fi["steps"] == pi["steps"]
    assert np.all(np.isfinite(Fp)) and np.abs(Fp).max() > 0
    assert np.array_equal(Ff, Fp)


def test_chunk_length_changes_no_bit():
    from emopt_b200.fdtd_ctypes import libFDTD
    p = _with_sheet(P.random_box(seed=61, shape=(23, 9, 90), w_pml=(3, 4, 2, 3, 4, 5), fixed_steps=33, n_sources=2))
    ref, _ = _fields(p, "fp32", "fused")
    for planes in (1, 5, 23):
        sim = P.make_solver(p, precision="fp32", kernel="fused")
        libFDTD.FDTD_set_zchunk(sim._libfdtd, planes)
        t0 = [getattr(sim, "_%s_fwd_t0" % c) for c in ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")]
        info = sim._solve(t0, t0, sim._sources)
        assert info["zchunk"] == planes
        assert np.array_equal(np.stack([sim._raw(c, False) for c in ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")]), ref)
