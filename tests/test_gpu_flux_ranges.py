"""The plain FP64 form's branch-free division and square root: bit for bit
the oracle's IEEE arithmetic on both sides of every range they are limited
to (states marked and unmarked, normals along the axes and tilted by
rounding), in every launch shape."""
import numpy as np
import pytest

import meshes

pytestmark = pytest.mark.gpu


def values(rng, kind, shape):
    if kind == "plain":
        return rng.uniform(-1.0, 1.0, shape)
    # zeros of both signs and magnitudes on both sides of 2^-120 and 2^60
    pool = np.array([0.0, -0.0, 1e-300, -1e-40, 2.0 ** -120, -np.nextafter(2.0 ** -120, 0.0), 1e-17, 0.3, -0.7])
    return rng.choice(pool, shape)


def state(rng, kind, cells):
    rho = rng.uniform(0.5, 1.5, cells)
    p = rng.uniform(0.5, 1.5, cells)
    mu, mv = values(rng, kind, cells), values(rng, kind, cells)
    if kind == "scaled":
        # units that put rho, rho E and the momenta below, at and above the
        # edges 2^-40 and 2^40, each pair of cells with a ratio of O(1)
        k = rng.choice([2.0 ** -41, 2.0 ** -40, 2.0 ** -39, 1.0, 2.0 ** 38, 2.0 ** 39, 2.0 ** 40])
        rho, p, mu, mv = rho * k, p * k, mu * k, mv * k
    return np.stack([rho, mu, mv, p / 0.4 + 0.5 * (mu * mu + mv * mv) / rho], axis=1).reshape(-1)


@pytest.mark.parametrize("scale", [4.0, 0.7], ids=["axis", "tilted"])
@pytest.mark.parametrize("kind", ["plain", "tiny", "scaled"])
@pytest.mark.parametrize("n", [4, 8, 16])
def test_residual_bits(ag, oracle, n, kind, scale):
    f = meshes.hanging(n, 2, lo=(0.1, -0.3, 0.0) if scale != 4.0 else (-2.0, -2.0, 0.0), scale=scale)
    m = f.mesh(n)
    cfg = meshes.make_config(n, h=scale, bc=(1, 0, 2, 1))
    cfg.apply()
    for seed in range(3):
        s0 = state(np.random.default_rng(seed), kind, m.ncells)
        want = oracle.rhs(m, s0, oracle.make_config(n, cfg))
        assert np.isfinite(want).all()
        s = ag.Session(m, cfg, form=ag.FORM_FP64_EXACT)
        s.upload(s0)
        dt = oracle.time_step(m, s0, oracle.make_config(n, cfg))
        assert s.cfl_dt() == dt
        for k in range(len(s.launch_variants())):
            s.set_launch_variant(k)
            got = s.rhs()
            assert np.array_equal(got, want), (k, np.abs(got - want).max())
        s.close()
