"""A launch that the runtime refuses: the test build _build/faillaunch
(-DPFLBM_TEST_FAIL_LAUNCH) asks for an empty grid while PFLBM_FAIL_LAUNCH=1, so
that the call fails on the host and nothing reaches the device. The call must
report it (PFLBM_ERR_CUDA, 2), count only what has run, and the same call must
give the right results once launches succeed again."""
import numpy as np
import pytest

from test_closure_gpu import _features
from test_closure_sums_gpu import _targets
from test_parity_gpu import AVG_FIELDS, BASIC, droplet_cfg, jet_cfg

pytestmark = pytest.mark.gpu


@pytest.fixture
def failing(pflbm, monkeypatch):
    """The test build in the library's place; failing(True) makes launches fail."""
    from phasefieldlbm_gb300 import build

    normal = pflbm.load_library()
    pflbm._LIB = pflbm.load_library(str(build.build_fail_launch()))
    yield lambda on: monkeypatch.setenv("PFLBM_FAIL_LAUNCH", "1") if on else monkeypatch.delenv("PFLBM_FAIL_LAUNCH")
    pflbm._LIB = normal


def _refused(pflbm, call):
    with pytest.raises(pflbm.PflbmError) as e:
        call()
    assert e.value.code == 2, e.value


@pytest.mark.parametrize("vs,storage,nx", [(19, 0, 32), (27, 0, 30), (19, 1, 32), (19, 3, 32)])
@pytest.mark.parametrize("profiled", [False, True])
def test_steps_that_were_not_launched_do_not_count(pflbm, failing, vs, storage, nx, profiled):
    c = jet_cfg(pflbm, vs, nx=nx, ny=24, nz=30, diam=6, noise=1)
    c.storage = storage
    c.flags = pflbm.FLAG_TIME_AVERAGE | pflbm.FLAG_REYNOLDS_MOMENTS if storage == 0 else 0
    fields = BASIC + (AVG_FIELDS if c.flags else ())
    with pflbm.Simulation(c) as s:
        s.step(21)
        s.get_field("phi")
        s.step(12)
        want = {f: s.get_field(f, dtype=np.float64) for f in fields}
    with pflbm.Simulation(c) as s:
        s.step(21)
        failing(True)
        _refused(pflbm, lambda: s.get_field("phi"))
        _refused(pflbm, (lambda: s.step_profiled(5)) if profiled else (lambda: s.step(13)))
        failing(False)
        done = 21 if profiled else 29  # a graph of 8 steps had been launched
        assert s.current_step == done
        s.step(33 - done)
        for f in fields:
            assert np.array_equal(s.get_field(f, dtype=np.float64), want[f]), f


def test_ensemble_readback_that_was_not_launched_is_not_served(pflbm, failing):
    cfgs = [droplet_cfg(pflbm, 19, n=n, radius=6) for n in (32, 36)]
    with pflbm.Ensemble(cfgs) as e:
        e.step(7)
        want = {(k, f): e.get_field(k, f) for k in (0, 1) for f in ("phi", "pxy")}
    with pflbm.Ensemble(cfgs) as e:
        e.get_field(1, "phi")
        e.step(7)
        failing(True)
        for k, f in want:
            _refused(pflbm, lambda: e.get_field(k, f))
        _refused(pflbm, lambda: e.reduce(1))
        failing(False)
        for (k, f), a in want.items():
            assert np.array_equal(e.get_field(k, f), a), (k, f)


def test_training_that_was_not_launched_does_not_count(pflbm, failing):
    x = _features(3000, 51)
    y = _targets(x, 52)
    blobs = []
    for interrupted in (False, True):
        with pflbm.Closure(3000) as c:
            c.set_samples(x, y)
            c.init_params(seed=3)
            c.train(40, batch=700, lr=2e-3, seed=5)
            if interrupted:
                failing(True)
                _refused(pflbm, lambda: c.train(300, batch=700, lr=2e-3, seed=5))
                failing(False)
            c.train(40, batch=700, lr=2e-3, seed=5)
            blobs.append(c.blob.copy())
    assert np.array_equal(*blobs)
