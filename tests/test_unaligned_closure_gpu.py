"""The learned closure on grids whose rows do not start on 16-byte boundaries
(padded on the device): the TMA-fed collide bit for bit the plain-load one on
unpadded rows, time averages included, and training snapshots of such a run the
same samples from either layout."""
import numpy as np
import pytest

from test_closure_gpu import _features
from test_parity_gpu import AVG_FIELDS, BASIC, jet_cfg

pytestmark = pytest.mark.gpu


def _plain(monkeypatch, on):
    for name in ("PFLBM_NO_TMA", "PFLBM_NO_VEC"):
        monkeypatch.setenv(name, "1") if on else monkeypatch.delenv(name, raising=False)


@pytest.mark.parametrize("vs,storage,nx", [(19, 0, 41), (27, 0, 34), (19, 3, 35), (27, 3, 33)])
@pytest.mark.parametrize("avg", [False, True])
def test_closure_on_padded_rows_bit_identical(pflbm, monkeypatch, vs, storage, nx, avg):
    c = jet_cfg(pflbm, vs, nx=nx, ny=27, nz=33, diam=8, noise=1)
    c.storage = storage
    if avg:
        c.flags = pflbm.FLAG_TIME_AVERAGE | pflbm.FLAG_REYNOLDS_MOMENTS
    with pflbm.Closure(2048) as k:
        k.set_samples(_features(2048, 7), np.full(2048, 2e-3))
        k.init_params(seed=9)
        blob = k.blob.copy()
    blob[:1377] += np.random.default_rng(8).normal(0.0, 0.1, 1377).astype(np.float32)
    out = {}
    for plain in (False, True):
        _plain(monkeypatch, plain)
        with pflbm.Simulation(c) as s:
            assert s.uses_tma != plain
            s.step(3)
            s.set_closure(blob, strength=1.0)
            s.step(30)
            out[plain] = {f: s.get_field(f, dtype=np.float64) for f in BASIC + (AVG_FIELDS if avg else ())}
    for f, a in out[True].items():
        assert np.array_equal(out[False][f], a), f


@pytest.mark.parametrize("vs,storage,nx", [(19, 0, 34), (27, 1, 36), (19, 2, 38)])
def test_snapshots_of_padded_rows(pflbm, monkeypatch, vs, storage, nx):
    c = jet_cfg(pflbm, vs, nx=nx, ny=28, nz=40, diam=8, noise=1)
    c.storage = storage
    got = {}
    for plain in (False, True):
        _plain(monkeypatch, plain)
        with pflbm.Simulation(c) as s, pflbm.Closure(20000) as k:
            assert s.uses_tma != plain
            s.step(40)
            assert k.add_snapshot(s, stride=1) > 0
            got[plain] = (*k.samples(), k.interface_scale())
    assert np.array_equal(got[False][0], got[True][0]) and np.array_equal(got[False][1], got[True][1])
    assert got[False][2] == got[True][2]
