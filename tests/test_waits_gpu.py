"""Bounded device-side waits made to run out, each where it stands: the test
builds make one wait of a kernel poll something that nothing sets, with a
short limit. The kernel reports through the device error word and returns, the
call returns PFLBM_ERR_DEVICE (8), and the device stays usable."""
import numpy as np
import pytest

from test_closure_gpu import _features
from test_closure_sums_gpu import _targets
from test_faults_gpu import _small_jet

pytestmark = pytest.mark.gpu


# error word: 1 = a plane's wait in the collide loop, 8 = the wait for a
# tile's first phi planes
@pytest.mark.parametrize("where,word", [("wait", 1), ("warmup", 8)])
def test_collide_reports_which_wait_ran_out(pflbm, where, word):
    from phasefieldlbm_gb300 import build

    dead = pflbm.load_library(str(getattr(build, f"build_dead_{where}")()))
    normal = pflbm.load_library()
    boxes = pflbm.ensemble_configs(3, seed=5)
    for c in boxes:
        c.nx = c.ny = c.nz = 32
        c.radius, c.diam = 6, 12
    closure_blob = np.zeros(1395, np.float32)
    try:
        pflbm._LIB = dead
        # one node per thread with a 4-plane and a 3-plane normal ring, node pairs
        for vs, storage, variant, closure in ((19, 0, "tma", False), (27, 0, "tma", False), (19, 1, "tma_pairs", False),
                                              (19, 3, "tma", False), (19, 0, "tma", True)):
            c = _small_jet(pflbm)
            c.velocity_set, c.storage = vs, storage
            with pflbm.Simulation(c) as s:
                assert s.collide_variant == variant
                if closure:
                    s.set_closure(closure_blob, 1.0)
                with pytest.raises(pflbm.PflbmError) as e:
                    s.step(3)
                assert e.value.code == 8 and f"error word {word})" in str(e.value), e.value
        with pflbm.Ensemble(boxes) as ens:
            with pytest.raises(pflbm.PflbmError) as e:
                ens.step(2)
            # the CTAs that did not see the wait run out give up at the grid barrier (2)
            got = int(str(e.value).split("error word ")[1].split(")")[0])
            assert e.value.code == 8 and got | 2 == word | 2, e.value
    finally:
        pflbm._LIB = normal
    with pflbm.Simulation(_small_jet(pflbm)) as s:
        s.step(5)
        assert int(s.reduce().nonfinite) == 0


def test_training_barrier_runs_out_and_reports(pflbm):
    """The grid barrier of the training kernel: after it has run out the
    parameters are those of no known iteration, and every call that would use
    them refuses until new ones are set."""
    from phasefieldlbm_gb300 import build

    dead = pflbm.load_library(str(build.build_dead_grid()))
    normal = pflbm.load_library()
    x = _features(3000, 61)
    y = _targets(x, 62)
    try:
        pflbm._LIB = dead
        with pflbm.Closure(3000) as c:
            c.set_samples(x, y)
            c.init_params(seed=3)
            before = c.blob.copy()
            with pytest.raises(pflbm.PflbmError) as e:
                c.train(300, batch=700, lr=2e-3, seed=5)  # several launches
            assert e.value.code == 8, e.value
            for call in (lambda: c.train(1, batch=700), lambda: c.gradient(700), c.loss):
                with pytest.raises(pflbm.PflbmError) as e:
                    call()
                assert e.value.code == 4, e.value
            c.blob = before
            g, loss = c.gradient(700)
    finally:
        pflbm._LIB = normal
    with pflbm.Closure(3000) as c:
        c.set_samples(x, y)
        c.blob = before
        g2, loss2 = c.gradient(700)
        assert np.array_equal(g, g2) and loss == loss2
        hist = c.train(300, batch=700, lr=2e-3, seed=5)
        assert np.isfinite(hist).all() and hist[-1] < hist[0]
