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
