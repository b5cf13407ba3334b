"""The FP64 diagnostics over fields with every kind of float: normal numbers
of all magnitudes, zeros of both signs, denormals (widened by the conversion
instruction, the others on the integer units), infinities and NaN (counted).
Sums against numpy in FP64: the same values in another order, 1e-12 of the sum
of magnitudes; maxima and counts exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 5, 5), (7, 34, 19), (40, 9, 67)])
@pytest.mark.parametrize("special", [False, True])
def test_reduce_over_all_kinds_of_floats(pflbm, shape, special):
    rng = np.random.default_rng(shape[0] + special)
    c = pflbm.config_reference(pflbm.CASE_DROPLET, pflbm.VS_D3Q19)
    c.nz, c.ny, c.nx = shape
    c.radius, c.diam = 1, 2
    fields = {}
    for k, name in enumerate(("rho", "ux", "uy", "uz", "phi")):
        a = (rng.standard_normal(shape) * 10.0 ** rng.integers(-30, 3, shape)).astype(np.float32)
        a[rng.random(shape) < 0.2] = 0.0
        a[rng.random(shape) < 0.1] = -0.0
        if special:
            a[rng.random(shape) < 0.2] = np.float32(1e-42) * (1 if k % 2 else -1)
            a[rng.random(shape) < 0.02] = (np.inf, -np.inf, np.nan, np.inf, np.nan)[k]
        if name == "phi":
            a[rng.random(shape) < 0.3] = np.float32(0.9)
            a[rng.random(shape) < 0.3] = np.nextafter(np.float32(0.9), np.float32(1))
            a[rng.random(shape) < 0.3] = np.float32(0.1)
        fields[name] = a
    with pflbm.Simulation(c) as s:
        for name, a in fields.items():
            s.set_initial_field(name, a)
        d = s.reduce()
    f = {k: a[1:-1, 1:-1, 1:-1].astype(np.float64) for k, a in fields.items()}
    ok = np.logical_and.reduce([np.isfinite(a) for a in f.values()])
    assert int(d.nonfinite) == int((~ok).sum())
    rho, ux, uy, uz, phi = (f[k][ok] for k in ("rho", "ux", "uy", "uz", "phi"))

    def near(got, terms):
        assert abs(got - terms.sum()) <= 1e-12 * np.abs(terms).sum()

    near(d.phi_mass, phi)
    near(d.rho_mass, rho)
    for got, u in zip(d.momentum, (ux, uy, uz)):
        near(got, rho * u)
    assert d.max_speed == pytest.approx(np.sqrt((ux ** 2 + uy ** 2 + uz ** 2).max()), rel=1e-15)
    inside, outside = phi > 0.9, phi < 0.1
    assert (int(d.n_in), int(d.n_out)) == (int(inside.sum()), int(outside.sum()))
    if inside.any():
        assert abs(d.rho_in - rho[inside].mean()) <= 1e-12 * np.abs(rho[inside]).mean()
