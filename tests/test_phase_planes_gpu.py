"""The boundary planes of a jet in the float4 phase step: on small planes a
thread per rebuilt direction, on larger ones a thread per node, and blocks of
32, 16 or 8 segments along x. Bit for bit the scalar step (PFLBM_NO_VEC=1)."""
import numpy as np
import pytest

from test_parity_gpu import ALL18, jet_cfg

pytestmark = pytest.mark.gpu


# the last plane with a thread per direction and the first without (152 SMs:
# 30 and 16 blocks of 256 nodes), the smallest, ragged ones, each block width
@pytest.mark.parametrize("vs,storage,nx,ny", [
    (19, 0, 96, 80), (19, 0, 96, 84), (27, 0, 64, 64), (27, 0, 68, 64), (19, 0, 32, 32), (27, 2, 37, 41),
    (19, 1, 129, 33), (27, 0, 33, 127),
])
def test_shared_rebuild_bit_identical(pflbm, monkeypatch, vs, storage, nx, ny):
    c = jet_cfg(pflbm, vs, nx=nx, ny=ny, nz=24, diam=8, noise=1)
    c.storage = storage
    out = []
    for scalar in (False, True):
        monkeypatch.setenv("PFLBM_NO_VEC", "1") if scalar else monkeypatch.delenv("PFLBM_NO_VEC", raising=False)
        with pflbm.Simulation(c) as s:
            s.step(37)
            out.append({f: s.get_field(f, dtype=np.float64) for f in ALL18})
    for f in ALL18:
        assert np.array_equal(out[0][f], out[1][f]), f
    assert np.ptp(out[0]["phi"]) > 0.5
