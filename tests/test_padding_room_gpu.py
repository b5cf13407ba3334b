"""What padded rows cost: the fewest elements that the row's alignment needs
(16 bytes; whole 32-byte sectors for FP32 where they make the row at most an
eighth longer), and only where the device keeps 256 MB free beside them."""
import pytest

from test_parity_gpu import jet_cfg

pytestmark = pytest.mark.gpu

BYTES = {0: (4, 4), 1: (2, 4), 2: (2, 4), 3: (8, 8)}  # populations, fields


def _cfg(pf, storage, nx):
    c = jet_cfg(pf, 19, nx=nx, ny=27, nz=33, diam=6, noise=1)
    c.storage = storage
    return c


def _bytes(pf, monkeypatch, c, plain):
    monkeypatch.setenv("PFLBM_NO_TMA", "1") if plain else monkeypatch.delenv("PFLBM_NO_TMA", raising=False)
    with pf.Simulation(c) as s:
        assert s.uses_tma != plain
        return s.device_bytes


@pytest.mark.parametrize("storage,nx,pad", [(1, 17, 7), (1, 33, 7), (2, 97, 7), (1, 98, 6), (1, 20, 4), (0, 17, 3),
                                            (0, 33, 3), (0, 34, 2), (0, 65, 7), (0, 97, 7), (0, 102, 2), (3, 33, 1)])
def test_padding_takes_what_the_alignment_needs(pflbm, monkeypatch, storage, nx, pad):
    c = _cfg(pflbm, storage, nx)
    s, t = BYTES[storage]
    extra = _bytes(pflbm, monkeypatch, c, False) - _bytes(pflbm, monkeypatch, c, True)
    per_element = c.ny * (c.nz * (2 * 19 * s + 2 * t + 3 * t) + 22 * t)  # f and phi twice, J, boundary planes
    assert extra == pad * per_element


def test_padding_leaves_room_on_the_device(pflbm, monkeypatch):
    c = _cfg(pflbm, 0, 33)
    padded = _bytes(pflbm, monkeypatch, c, False)
    for spare, pads in ((0, False), (2**20, False), (2**28 - 1, False), (2**28, True)):
        monkeypatch.setenv("PFLBM_ALLOC_LIMIT_BYTES", str(padded + spare))
        with pflbm.Simulation(c) as s:
            assert s.uses_tma == pads, spare
            s.step(3)
