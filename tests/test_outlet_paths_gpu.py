"""The kernels' variants on jets that have reached the outlet (phi above 0.5
on the last fluid plane), where the outflow rebuild works on a developed flow:
TMA-fed collide and float4 phase step against the plain-load collide and the
scalar phase step, on aligned and padded rows, bit for bit."""
import numpy as np
import pytest

from test_parity_gpu import ALL18, AVG_FIELDS, BASIC, jet_cfg

pytestmark = pytest.mark.gpu


def _cfg(pf, vs, storage, nx, flags=0):
    c = jet_cfg(pf, vs, nx=nx, ny=27, nz=24, diam=6, noise=1)
    c.storage, c.flags = storage, flags
    return c


def _plain(monkeypatch, on):
    monkeypatch.setenv("PFLBM_NO_PAIR", "1")
    for name in ("PFLBM_NO_TMA", "PFLBM_NO_VEC"):
        monkeypatch.setenv(name, "1") if on else monkeypatch.delenv(name, raising=False)


@pytest.mark.parametrize("vs,storage,nx", [
    (27, 0, 33), (19, 0, 29), (27, 0, 32), (19, 0, 32), (27, 1, 33), (19, 1, 32), (19, 2, 35), (27, 2, 40),
    (19, 3, 29), (27, 3, 32),
])
def test_developed_jets_bit_identical(pflbm, monkeypatch, vs, storage, nx):
    flags = pflbm.FLAG_TIME_AVERAGE | pflbm.FLAG_REYNOLDS_MOMENTS if storage in (0, 3) else 0
    out = {}
    for plain in (False, True):
        _plain(monkeypatch, plain)
        with pflbm.Simulation(_cfg(pflbm, vs, storage, nx, flags)) as s:
            assert s.collide_variant == ("plain" if plain else "tma")
            s.step(860)
            out[plain] = {f: s.get_field(f, dtype=np.float64) for f in ALL18 + (AVG_FIELDS if flags else ())}
    assert out[True]["phi"][-2].max() > 0.5
    for f, a in out[True].items():
        assert np.array_equal(out[False][f], a), f


@pytest.mark.parametrize("storage,nx", [(0, 33), (1, 33)])
def test_developed_checkpoints_move_between_layouts(pflbm, monkeypatch, tmp_path, storage, nx):
    c = _cfg(pflbm, 27, storage, nx)
    _plain(monkeypatch, False)
    with pflbm.Simulation(c) as a:
        a.step(860)
        a.save_checkpoint(tmp_path / "c.ckpt")
        a.step(25)
        want = {f: a.get_field(f) for f in BASIC}
    assert want["phi"][-2].max() > 0.5
    _plain(monkeypatch, True)
    with pflbm.Simulation(c, init=False) as b:
        b.load_checkpoint(tmp_path / "c.ckpt")
        b.save_checkpoint(tmp_path / "d.ckpt")
        b.step(25)
        for f, v in want.items():
            assert np.array_equal(b.get_field(f), v), f
    assert (tmp_path / "c.ckpt").read_bytes() == (tmp_path / "d.ckpt").read_bytes()
