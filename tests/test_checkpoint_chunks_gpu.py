"""Checkpoints whose arrays are written and read in several chunks (64 MB each,
the last one partial), from padded and unpadded device rows: the same file, and
a load brings the state back bit for bit."""
import numpy as np
import pytest

from test_parity_gpu import jet_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,nx", [(0, 101), (0, 100), (1, 203), (3, 51)])
def test_checkpoints_in_several_chunks(pflbm, monkeypatch, tmp_path, storage, nx):
    c = jet_cfg(pflbm, 27, nx=nx, ny=93, nz=151, diam=14, noise=1)
    c.storage = storage
    files = []
    for plain in (False, True):
        for name in ("PFLBM_NO_TMA", "PFLBM_NO_VEC"):
            monkeypatch.setenv(name, "1") if plain else monkeypatch.delenv(name, raising=False)
        files.append(tmp_path / f"{plain}.ckpt")
        with pflbm.Simulation(c) as a:
            a.step(5)
            a.save_checkpoint(files[-1])
            a.step(5)
            want = a.get_field("uz")
        assert files[-1].stat().st_size > 2 * 2 ** 27
        with pflbm.Simulation(c, init=False) as b:
            b.load_checkpoint(files[-1])
            b.step(5)
            assert np.array_equal(b.get_field("uz"), want)
            b.load_checkpoint(files[0])
            b.save_checkpoint(tmp_path / "again.ckpt")
        assert files[0].read_bytes() == (tmp_path / "again.ckpt").read_bytes()
    assert files[0].read_bytes() == files[1].read_bytes()
