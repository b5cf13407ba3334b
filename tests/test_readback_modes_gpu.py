"""Fields are rebuilt either all together or without the twelve that are
rarely read (rho, u, phi, |grad phi| only). Whatever is read in which order,
with TMA-fed or plain-load kernels, on aligned and padded rows: the same
values bit for bit, ghost shell included."""
import numpy as np
import pytest

from test_parity_gpu import ALL18, droplet_cfg, jet_cfg

pytestmark = pytest.mark.gpu

ORDERS = (ALL18, tuple(reversed(ALL18)), ("phi", "pxy", "uz", "ind", "rho"), ("ind", "ux"), ("vort_z", "fsx", "uy"))


@pytest.mark.parametrize("case,vs,storage,nx", [("jet", 19, 0, 32), ("jet", 27, 1, 32), ("jet", 19, 2, 29),
                                                ("droplet", 27, 0, 24), ("droplet", 19, 3, 25), ("jet", 27, 0, 33)])
def test_fields_do_not_depend_on_what_else_is_read(pflbm, monkeypatch, case, vs, storage, nx):
    c = jet_cfg(pflbm, vs, nx=nx, ny=27, nz=34, diam=6, noise=1) if case == "jet" else droplet_cfg(pflbm, vs, n=24, radius=6)
    c.nx, c.storage, c.flags = nx, storage, pflbm.FLAG_VORTICITY
    monkeypatch.setenv("PFLBM_NO_PAIR", "1")
    want, mass = {}, None
    for plain in (True, False):
        for name in ("PFLBM_NO_TMA", "PFLBM_NO_VEC"):
            monkeypatch.setenv(name, "1") if plain else monkeypatch.delenv(name, raising=False)
        for order in ORDERS:
            with pflbm.Simulation(c) as s:
                for _ in range(2):  # the second time some field beyond the base ones may have been read
                    s.step(9)
                    got = {f: s.get_field(f, dtype=np.float64) for f in order}
                    d = s.reduce()
                for f, a in got.items():
                    assert np.array_equal(want.setdefault(f, a), a), (plain, order, f)
                mass = mass or d.phi_mass
                assert d.phi_mass == mass


def test_ensemble_boxes_read_in_any_order(pflbm):
    cfgs = pflbm.ensemble_configs(3, seed=5)
    for k, c in enumerate(cfgs):
        c.nx = c.ny = c.nz = 32 + 16 * (k % 2)
        c.radius, c.diam = 6, 12
    with pflbm.Ensemble(cfgs) as a, pflbm.Ensemble(cfgs) as b:
        a.step(5), b.step(5)
        want = {(k, f): a.get_field(k, f) for f in ALL18 for k in range(3)}
        order = [(k, f) for k in range(3) for f in ("phi", "uz", "normx", "rho", "fsz", "ind")]
        assert all(np.array_equal(b.get_field(*o), want[o]) for o in order)
        a.step(1), b.step(1)
        assert b.reduce(1).phi_mass == a.reduce(1).phi_mass
        assert np.array_equal(a.get_field(1, "uz"), b.get_field(1, "uz"))
        assert not np.array_equal(a.get_field(1, "uz"), want[(1, "uz")])
        b.init()
        assert np.array_equal(b.get_field(1, "pxy"), np.zeros_like(want[(1, "pxy")]))
