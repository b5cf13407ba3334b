"""Index safety of the plain-load collide and the scalar phase step, which grids
run whose padded rows find no room: the bounds-checked test build with
PFLBM_NO_TMA=1 and PFLBM_NO_VEC=1, and on padded rows with time averages. No
guard may fire (pflbm_step would return PFLBM_ERR_DEVICE); the fields equal the
normal build's to rounding (the guards change which multiply-adds the compiler
contracts)."""
import numpy as np
import pytest

from conftest import rel_l2
from test_closure_gpu import _features
from test_parity_gpu import BASIC, droplet_cfg, jet_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("plain", [True, False])
def test_checked_build_on_unaligned_rows(pflbm, monkeypatch, plain):
    from phasefieldlbm_gb300 import build

    for name in ("PFLBM_NO_TMA", "PFLBM_NO_VEC"):
        monkeypatch.setenv(name, "1") if plain else monkeypatch.delenv(name, raising=False)
    checked = pflbm.load_library(str(build.build_checked()))
    normal = pflbm.load_library()
    with pflbm.Closure(2048) as k:
        k.set_samples(_features(2048, 7), np.full(2048, 2e-3))
        k.init_params(seed=9)
        blob = k.blob.copy()
    avg = pflbm.FLAG_TIME_AVERAGE | pflbm.FLAG_REYNOLDS_MOMENTS
    try:
        for vs, storage, nx, flags, closure in ((19, 0, 30, 0, False), (27, 0, 29, avg, False), (19, 1, 33, 0, False),
                                                (27, 2, 35, avg, False), (19, 3, 31, avg, False),
                                                (19, 0, 41, avg, True), (27, 3, 27, 0, True)):
            c = jet_cfg(pflbm, vs, nx=nx, ny=27, nz=33, diam=6, noise=1)
            c.storage, c.flags = storage, flags
            d = droplet_cfg(pflbm, vs, n=nx, radius=6)
            d.storage, d.flags = storage, flags
            for cfg in (c, d):
                out = []
                for lib in (checked, normal):
                    pflbm._LIB = lib
                    with pflbm.Simulation(cfg) as s:
                        assert s.uses_tma != plain
                        if closure:
                            s.set_closure(blob, strength=1.0)
                        s.step(23)
                        out.append({f: s.get_field(f, dtype=np.float64) for f in BASIC + (("avg_uz",) if flags else ())})
                for f in out[0]:
                    if storage in (0, 3) and (cfg is c or f in ("rho", "phi")):
                        assert rel_l2(out[0][f], out[1][f]) <= (1e-12 if storage == 3 else 1e-5), (vs, nx, f)
                    else:  # 16-bit stores round the contraction's last bit up; a droplet's u is near its floor
                        assert np.isfinite(out[0][f]).all()
    finally:
        pflbm._LIB = normal
