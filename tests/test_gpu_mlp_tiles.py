"""The learned indicator's tile and weight-gradient kernels at the edges of
their tiles (128 rows a tile, 256 rows a partial sum, 16 rows a K step), and
the judge on the device against the same rule on the host."""
import numpy as np
import pytest

import meshes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L(ag):
    from amrgpu import learned
    return learned


@pytest.fixture(scope="module")
def M():
    from oracle import mlp_oracle
    return mlp_oracle


@pytest.mark.parametrize("B", [8, 24, 120, 136, 248, 264, 512, 4104])
def test_gradient_at_tile_edges(L, M, B):
    """Rounding as in the whole-batch gradient test: BF16 at the same points
    as the oracle, FP32 sums in another order (logits within 2e-2, every
    tensor within 1e-2 relative)."""
    rng = np.random.default_rng(B)
    m = L.Mlp(seed=3)
    p = (M.init_params(3) * 3.0).astype(np.float32)
    m.set_params(p)
    xb = M.f32_to_bf16_bits(rng.normal(scale=1.5, size=(B, M.NIN)).astype(np.float32))
    y = rng.integers(0, 3, B).astype(np.int32)
    logits, g, loss = m.grad(xb, y)
    want, loss_ref, g_ref = M.forward_backward(p.astype(np.float64), M.bf16_bits_to_f64(xb), y)
    assert np.abs(logits - want).max() <= 2e-2
    assert np.array_equal(m.predict(xb), logits)
    assert abs(loss - loss_ref) <= 1e-3 * abs(loss_ref)
    o = 0
    for name, k in (("W1", 128 * 400), ("b1", 128), ("W2", 64 * 128), ("b2", 64), ("W3", 3 * 64), ("b3", 3)):
        a, b = g[o:o + k].astype(np.float64), g_ref[o:o + k]
        o += k
        assert np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(b), name
    m.close()


def sample(seed, quads, fraction):
    z = (np.uint64(seed) * np.uint64(0x9E3779B97F4A7C15)
         + np.arange(quads, dtype=np.uint64) * np.uint64(0xD1B54A32D192ED03) + np.uint64(0x8CB92BA72F3D8DD7))
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    z ^= z >> np.uint64(31)
    return (z >> np.uint64(11)).astype(np.float64) * (1.0 / 9007199254740992.0) < fraction


@pytest.mark.parametrize("n,level,fraction", [(8, 2, 0.3), (16, 2, 1.0), (8, 4, 0.05), (8, 2, 0.0)])
def test_judge_counts(ag, L, n, level, fraction):
    f = meshes.hanging(n, level=level, refine=(3, 6), periodic=(1, 0))
    cfg = meshes.make_config(n, ic=1, h=4.0)
    cfg.apply()
    s = ag.Session(f.mesh(n), cfg, form=1)
    s.upload(meshes.perturbed(f.initialize(n), 3, amp=3e-2))
    m = L.Mlp(seed=1)
    m.set_params((m.get_params() * 3.0).astype(np.float32))
    tol = 0.03
    for seed in (0, 12345678901):
        with np.errstate(over="ignore"):
            which = sample(seed, f.num_quads, fraction)
        plain = L.plain_classes(L.session_jumps(s), tol)
        tags, j = m.tags(s, tol, judge_fraction=fraction, seed=seed)
        logits = m.predict(L.session_features(s))
        assert np.array_equal(tags, np.argmax(logits, axis=1))
        p, t = plain[which], tags[which]
        assert j["judged"] == which.sum()
        assert j["disagree"] == (p != t).sum()
        assert j["coarser"] == (((p == L.REFINE) & (t != L.REFINE)) | ((t == L.COARSEN) & (p != L.COARSEN))).sum()
    m.close()
    s.close()


@pytest.mark.parametrize("at", [0, 100, 299])
@pytest.mark.parametrize("entry", [-1, -2 ** 31, "rows", 2 ** 31 - 1])
def test_permutation_entries_out_of_range_are_refused(ag, L, at, entry):
    """Before anything is trained: the parameters stay as they were. Entry
    299 is in no whole batch and is refused as well."""
    f = meshes.uniform(8, 3, periodic=(1, 1))
    s = ag.Session(f.mesh(8), meshes.make_config(8).apply(), form=1)
    s.upload(f.initialize(8))
    m = L.Mlp(seed=2)
    while m.size() < 300:
        m.append(s, 0.02)
    before = m.get_params()
    perm = np.arange(300, dtype=np.int32)
    m.train_epoch(perm[:0], batch=128)
    perm[at] = m.size() if entry == "rows" else entry
    with pytest.raises(ag.AmrGpuError):
        m.train_epoch(perm, batch=128)
    assert np.array_equal(m.get_params(), before)
    perm[at] = m.size() - 1
    m.train_epoch(perm, batch=128)
    assert not np.array_equal(m.get_params(), before)
    m.close()
    s.close()
