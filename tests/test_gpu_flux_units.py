"""The plain FP64 form in other units than O(1): residuals bit for bit the
oracle's on both sides of the ranges that the branch-free division and square
root are limited to, in density, energy and speed, in every launch shape."""
import numpy as np
import pytest

import meshes

pytestmark = pytest.mark.gpu


def state(rng, kind, cells):
    rho = rng.uniform(0.5, 1.5, cells)
    u, v = rng.uniform(-1.0, 1.0, cells), rng.uniform(-1.0, 1.0, cells)
    p = rng.uniform(0.5, 1.5, cells)
    # rho by a factor, speeds by another, p with them; per cell where several are given
    k, c = {"cgs": ([2.0 ** -80], [2.0 ** 20]), "si": ([1.2], [340.0]),
            "density": (2.0 ** np.array([-111.0, -110, -109, -30]), [1.0]),
            "dense": (2.0 ** np.array([30.0, 108, 109, 110, 111]), [1.0]),
            "slow": ([1.0], 2.0 ** np.array([-42.0, -41, -40, -39])),
            "fast": ([1.0], 2.0 ** np.array([38.0, 39, 40, 41]))}[kind]
    k, c = rng.choice(k, cells), rng.choice(c, cells)
    # a velocity of its own scale, zeros among them
    u = u * rng.choice([1.0, 1.0, 0.0, 2.0 ** -100, 2.0 ** -159, 2.0 ** -170], cells)
    rho, u, v, p = rho * k, u * c, v * c, p * k * c * c
    return np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)], axis=1).reshape(-1)


@pytest.mark.parametrize("scale", [4.0, 0.7], ids=["axis", "tilted"])
@pytest.mark.parametrize("kind", ["cgs", "si", "density", "dense", "slow", "fast"])
@pytest.mark.parametrize("n", [4, 8, 16])
def test_residual_bits(ag, oracle, n, kind, scale):
    f = meshes.hanging(n, 2, lo=(0.1, -0.3, 0.0) if scale != 4.0 else (-2.0, -2.0, 0.0), scale=scale)
    m = f.mesh(n)
    cfg = meshes.make_config(n, h=scale, bc=(1, 0, 2, 1))
    cfg.apply()
    s0 = state(np.random.default_rng(n), kind, m.ncells)
    want = oracle.rhs(m, s0, oracle.make_config(n, cfg))
    assert np.isfinite(want).all()
    s = ag.Session(m, cfg, form=ag.FORM_FP64_EXACT)
    s.upload(s0)
    for k in range(len(s.launch_variants())):
        s.set_launch_variant(k)
        got = s.rhs()
        assert np.array_equal(got, want), (k, np.abs(got - want).max())
    s.close()
