"""The last boundary plane that is rebuilt with a thread per direction and the
first with a thread per node, for the number of SMs of the device that runs the
test: bit for bit the scalar phase step."""
import numpy as np
import pytest

from test_parity_gpu import ALL18, jet_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vs,nx", [(19, 96), (27, 64), (27, 61)])
@pytest.mark.parametrize("past", [False, True])
def test_planes_at_the_line_between_the_rebuilds(pflbm, monkeypatch, vs, nx, past):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    directions = 5 if vs == 19 else 9
    ny = sms // directions * 256 // nx
    if past:
        while -(-nx * ny // 256) * directions <= sms:
            ny += 1
    assert (-(-nx * ny // 256) * directions <= sms) != past
    c = jet_cfg(pflbm, vs, nx=nx, ny=ny, nz=24, diam=8, noise=1)
    out = []
    for scalar in (False, True):
        monkeypatch.setenv("PFLBM_NO_VEC", "1") if scalar else monkeypatch.delenv("PFLBM_NO_VEC", raising=False)
        with pflbm.Simulation(c) as s:
            s.step(37)
            out.append({f: s.get_field(f, dtype=np.float64) for f in ALL18})
    for f in ALL18:
        assert np.array_equal(out[0][f], out[1][f]), f
