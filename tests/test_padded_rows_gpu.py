"""Grids whose rows do not start on 16-byte boundaries: their device arrays
have padded rows and run the TMA-fed collide and the float4 phase step. Bit
for bit the plain-load kernels on unpadded rows (PFLBM_NO_TMA=1,
PFLBM_NO_VEC=1), and files move freely between the two layouts."""
import numpy as np
import pytest

from test_parity_gpu import ALL18, AVG_FIELDS, BASIC, droplet_cfg, jet_cfg

pytestmark = pytest.mark.gpu


def _cfg(pf, case, vs, storage, nx, flags=0):
    c = jet_cfg(pf, vs, nx=nx, ny=27, nz=33, diam=6, noise=1) if case == "jet" else droplet_cfg(pf, vs, n=26, radius=6)
    if case == "droplet":
        c.nx = nx
    c.storage, c.flags = storage, flags
    return c


def _plain(monkeypatch, on):
    for name in ("PFLBM_NO_TMA", "PFLBM_NO_VEC"):
        monkeypatch.setenv(name, "1") if on else monkeypatch.delenv(name, raising=False)


@pytest.mark.parametrize("case,vs,storage,nx", [
    ("jet", 19, 0, 29), ("jet", 27, 0, 33), ("jet", 27, 0, 65), ("jet", 19, 0, 31), ("droplet", 27, 0, 23),
    ("droplet", 19, 0, 67), ("jet", 19, 1, 36), ("jet", 27, 2, 33), ("droplet", 19, 2, 35), ("jet", 19, 3, 29),
    ("droplet", 27, 3, 25),
])
def test_padded_rows_bit_identical(pflbm, monkeypatch, case, vs, storage, nx):
    flags = pflbm.FLAG_TIME_AVERAGE | pflbm.FLAG_REYNOLDS_MOMENTS | pflbm.FLAG_VORTICITY if nx % 2 else 0
    names = ALL18 + ((*AVG_FIELDS, "vort_x", "vort_mag") if flags else ())
    out = {}
    for plain in (False, True):
        _plain(monkeypatch, plain)
        with pflbm.Simulation(_cfg(pflbm, case, vs, storage, nx, flags)) as s:
            assert s.collide_variant == ("plain" if plain else "tma")
            s.step(21)
            out[plain] = {f: s.get_field(f, dtype=np.float64) for f in names}
            d = s.reduce()
            out[plain]["mass"] = np.array([d.phi_mass, d.rho_mass, d.max_speed])
    for f, a in out[True].items():
        assert np.array_equal(out[False][f], a), f


@pytest.mark.parametrize("storage,first", [(0, False), (0, True), (1, False)])
def test_checkpoints_move_between_layouts(pflbm, monkeypatch, tmp_path, storage, first):
    c = _cfg(pflbm, "jet", 27, storage, 29, pflbm.FLAG_TIME_AVERAGE)
    ck = tmp_path / "c.ckpt"
    _plain(monkeypatch, first)
    with pflbm.Simulation(c) as a:
        a.step(13)
        a.save_checkpoint(ck)
        a.step(10)
        want = {f: a.get_field(f) for f in BASIC + ("avg_uz",)}
    _plain(monkeypatch, not first)
    with pflbm.Simulation(c, init=False) as b:
        b.load_checkpoint(ck)
        b.save_checkpoint(tmp_path / "d.ckpt")
        b.step(10)
        for f, v in want.items():
            assert np.array_equal(b.get_field(f), v), f
    assert ck.read_bytes() == (tmp_path / "d.ckpt").read_bytes()


def test_no_room_for_padding_keeps_the_grid(pflbm, monkeypatch):
    c = _cfg(pflbm, "jet", 19, 1, 33)
    _plain(monkeypatch, True)
    with pflbm.Simulation(c) as s:
        dense = s.device_bytes
        s.step(9)
        want = s.get_field("uz")
    _plain(monkeypatch, False)
    with pflbm.Simulation(c) as s:
        assert s.device_bytes > dense and s.uses_tma
    monkeypatch.setenv("PFLBM_ALLOC_LIMIT_BYTES", str(dense))
    with pflbm.Simulation(c) as s:
        assert s.device_bytes == dense and not s.uses_tma
        s.step(9)
        assert np.array_equal(s.get_field("uz"), want)
