"""Reading any field at step 0 leaves the initial fields that the caller has
set as they are, whether the simulation was initialised, restored from a
checkpoint of step 0, or had stepped before."""
import numpy as np
import pytest

from test_parity_gpu import ALL18, BASIC, jet_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["init", "load", "load_after_steps"])
@pytest.mark.parametrize("read_first", [False, True])
def test_reading_at_step_0_keeps_the_initial_fields(pflbm, tmp_path, how, read_first):
    c = jet_cfg(pflbm, 19, nx=32, ny=24, nz=30, diam=6, noise=1)
    ck = tmp_path / "zero.ckpt"
    rng = np.random.default_rng(4)
    with pflbm.Simulation(c) as a:
        a.save_checkpoint(ck)
        want = {f: a.get_field(f) for f in BASIC}
        for f, amp in zip(BASIC, (1e-3, 1e-3, 1e-3, 1e-3, 0.1)):
            want[f] = (want[f] + amp * rng.random(want[f].shape)).astype(np.float32)
            a.set_initial_field(f, want[f])
        a.step(21)
        after = {f: a.get_field(f) for f in BASIC}
    with pflbm.Simulation(c, init=how != "load") as b:
        if how != "init":
            if how == "load_after_steps":
                b.step(9)
                b.get_field("phi")
            b.load_checkpoint(ck)
        if read_first:
            b.get_field("uz")
        for f in BASIC:
            b.set_initial_field(f, want[f])
        for f in ALL18:
            b.get_field(f)
        for f in BASIC:
            assert np.array_equal(b.get_field(f), want[f]), f
        b.set_initial_field("phi", want["phi"])  # the state is rebuilt from the fields once more
        b.step(21)
        for f in BASIC:
            assert np.array_equal(b.get_field(f), after[f]), f
