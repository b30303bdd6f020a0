"""What a program that uses amrgpu has it do, as cases that can be timed.

Kinds of pass (the field "kind" of a case):

  march     steps of a device-resident session (Session.step): the inner loop
            of every run, on uniform and on refined meshes, in both forms
  evolve    one hpc_amr_evolve_solver call on ordinary host arrays: what the
            reference's driver calls once per regrid interval
  amr       one turn of the adaptive loop: steps, report, indicator tags,
            regrid; the region of interest moves out and back again, so a
            pass ends on the mesh it began with
  classify  the learned indicator's classes of a session's quads
  train     one epoch of the learned indicator's training

Meshes are bricks of trees_x x trees_y quadtrees in n x n patches, uniform
(finest == level) or refined around a circle up to the level `finest`.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "amr-demo_b200"))
os.environ.setdefault("AMRGPU_QUIET", "1")
# launch shapes are tuned in each process, not read from an earlier program's file
os.environ.setdefault("AMRGPU_TUNE_CACHE", "")

FP64, FP32 = 0, 1  # amrgpu.FORM_FP64_EXACT, amrgpu.FORM_FP32_FLUX
STAGES = {1: 1, 3: 3, 4: 4, 5: 5}  # time_scheme: RK1, SSP-RK3, RK4, LSERK45
NPARAMS = 59779
REACH = 2.5  # a quad is refined when the circle passes within this many of its widths


def _mesh(kind, trees, level, finest, n, form, scheme, steps, **more):
    return dict(kind=kind, trees_x=trees[0], trees_y=trees[1], level=level, finest=finest, n=n, form=form,
                scheme=scheme, steps=steps, periodic=finest == level, **more)


def listed():
    return [
        # the smallest run: 64 x 64 cells in 64 patches of 8 x 8, one call of the reference's entry point per
        # regrid interval of 10 steps; latency of one call
        dict(name="evolve 64^2 fp64", **_mesh("evolve", (1, 1), 3, 3, 8, FP64, 3, 10)),
        # the same entry point at the benchmark's 1024 x 1024 cells: the state goes in and out by every call
        dict(name="evolve 1024^2 fp32", **_mesh("evolve", (1, 1), 6, 6, 16, FP32, 3, 10)),
        # a small study run: 256 quads, far fewer than the GPU could hold; a graph of steps per launch
        dict(name="march 256^2 fp32", **_mesh("march", (1, 1), 4, 4, 16, FP32, 3, 24, graph=True)),
        # the benchmark's mesh in both forms
        dict(name="march 1024^2 fp32", **_mesh("march", (1, 1), 6, 6, 16, FP32, 3, 10)),
        dict(name="march 1024^2 fp64", **_mesh("march", (1, 1), 6, 6, 16, FP64, 3, 5)),
        # the largest uniform mesh, four times the benchmark's
        dict(name="march 2048^2 fp32", **_mesh("march", (1, 1), 7, 7, 16, FP32, 3, 5)),
        # 8 x 8 patches on a refined mesh, as the learned indicator's workload has them
        dict(name="march refined 8x8 fp32", **_mesh("march", (1, 1), 3, 7, 8, FP32, 3, 5)),
        # hanging faces and walls in the bit-exact form, an odd brick, classical RK4
        dict(name="march refined 16x16 fp64 rk4", **_mesh("march", (3, 1), 3, 6, 16, FP64, 4, 3)),
        # the adaptive loop at a four-quadrant run's levels and at a shock-bubble run's
        dict(name="amr levels 4-8", **_mesh("amr", (1, 1), 4, 8, 16, FP32, 3, 5)),
        dict(name="amr levels 5-10", **_mesh("amr", (2, 1), 5, 10, 16, FP32, 3, 5)),
        # the learned indicator on a refined mesh of 8 x 8 patches, and its training
        dict(name="classify refined 8x8", **_mesh("classify", (1, 1), 3, 8, 8, FP32, 3, 0)),
        dict(name="train 65536 rows", kind="train", rows=65536, batch=8192),
    ]


def draw(rng):
    kind = rng.choice(["march"] * 6 + ["amr"] * 2 + ["evolve", "classify", "train"])
    if kind == "train":
        batch = 128 * int(round(2 ** rng.uniform(2, 6)))
        return dict(kind="train", rows=min(65536, batch * rng.randint(2, 24)), batch=batch)
    n = rng.choice([8, 16, 16])
    form = rng.choice([FP64, FP32])
    if kind == "amr":
        level = rng.randint(3, 4)
        return _mesh("amr", (rng.randint(1, 2), rng.randint(1, 2)), level, level + rng.randint(2, 4), n, FP32, 3,
                     rng.randint(2, 6))
    trees = (rng.randint(1, 7), rng.randint(1, 7))
    refined = kind == "classify" or (kind == "march" and rng.random() < 0.5)
    most = 4096 if n == 16 else 16384  # quads of 1024^2 cells
    quads = int(math.exp(rng.uniform(math.log(64), math.log(most // (4 if refined else 1)))))
    level = max(0, min(6, round(math.log(max(1.0, quads / (trees[0] * trees[1])), 4))))
    while trees[0] * trees[1] * 4 ** level > most // (4 if refined else 1):
        level -= 1
    if kind == "classify":
        return _mesh("classify", trees, max(level, 1), max(level, 1) + 2, n, FP32, 3, 0)
    if kind == "evolve":
        return _mesh("evolve", trees, level, level, n, form, 3, rng.randint(5, 12))
    scheme = rng.choice([3, 3, 3, 1, 4, 5])
    c = _mesh("march", trees, level, level + (rng.randint(1, 2) if refined else 0), n, form, scheme,
              rng.randint(1, 5))
    return dict(c, graph=True, steps=12) if rng.random() < 0.2 else c


# ------------------------------------------------------------------ meshes and initial states
def _circle(case, moved=0.0):
    """Centre and radius of the circle that meshes are refined around, in tree widths."""
    w, h = case["trees_x"], case["trees_y"]
    return 0.47 * w, 0.53 * h, 0.29 * min(w, h) + moved


def _hit(case, level, x, y, moved=0.0, parents=0):
    """Quads (their ancestors, with `parents`) that the circle passes within REACH widths of."""
    cx, cy, r = _circle(case, moved)
    d = 0.5 ** (level - parents)
    x, y = x >> parents, y >> parents
    return np.abs(np.hypot((x + 0.5) * d - cx, (y + 0.5) * d - cy) - r) < REACH * d


def _interleave(v):
    v = v.astype(np.uint64)
    for s, m in ((16, 0x0000FFFF0000FFFF), (8, 0x00FF00FF00FF00FF), (4, 0x0F0F0F0F0F0F0F0F), (2, 0x3333333333333333),
                 (1, 0x5555555555555555)):
        v = (v | (v << np.uint64(s))) & np.uint64(m)
    return v


def _leaves(case):
    """(level, x, y) of the mesh's quads in Morton order, x and y in widths of the quad from the brick's corner. A
    refined mesh is 2:1 balanced as it is: REACH is over 2.13, so neighbours differ by one level at most."""
    w, h, lv = case["trees_x"], case["trees_y"], case["level"]
    y, x = np.divmod(np.arange((w << lv) * (h << lv), dtype=np.int64), w << lv)
    level = np.full(len(x), lv, np.int64)
    for _ in range(lv, case["finest"]):
        hit = _hit(case, level, x, y) & (level == level.max())
        if not hit.any():
            break
        k = np.where(hit, 4, 1)
        at = np.repeat(np.arange(len(x)), k)
        sub = np.arange(len(at)) - np.repeat(np.cumsum(k) - k, k)
        f = hit[at].astype(np.int64)
        level, x, y = level[at] + f, (x[at] << f) + f * (sub & 1), (y[at] << f) + f * (sub >> 1)
    up = case["finest"] - level
    order = np.argsort(_interleave(x << up) | (_interleave(y << up) << np.uint64(1)), kind="stable")
    return level[order], x[order], y[order]


def _state(case, leaves, seed):
    """Conserved variables at the cell centres, (quads, n, n, 4): smooth waves on a stream and a density step at the
    circle, all from the seed."""
    g = np.random.default_rng(seed)
    n, w, h = case["n"], case["trees_x"], case["trees_y"]
    lv, qx, qy = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in leaves)
    d = torch.exp2(-lv.double())[:, None]
    c = ((torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) / n)[None, :]
    x = ((qx[:, None] + c) * d)[:, None, :].expand(-1, n, n)
    y = ((qy[:, None] + c) * d)[:, :, None].expand(-1, n, n)

    def waves(mean, size):
        v = torch.full_like(x, mean)
        for _ in range(3):
            kx, ky = g.integers(1, 4), g.integers(1, 4)
            v += size * g.uniform(0.3, 1.0) * torch.sin(2 * math.pi * (kx * x / w + g.uniform())) \
                * torch.sin(2 * math.pi * (ky * y / h + g.uniform()))
        return v

    u, v, p = waves(g.uniform(0.2, 0.5), 0.1), waves(g.uniform(0.2, 0.5), 0.1), waves(1.0, 0.05)
    cx, cy, r = _circle(case)
    step = torch.tanh((torch.hypot(x - cx, y - cy) - r) * 2.0 ** (case["finest"] - 1))
    rho = waves(1.0, 0.05) + g.uniform(0.1, 0.3) * step
    return torch.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)], dim=-1)


def _forest(case):
    import amrgpu as ag
    f = ag.Forest(case["trees_x"], case["trees_y"], periodic=(int(case["periodic"]),) * 2, scale=1.0,
                  level=case["level"])
    level, x, y = _leaves(dict(case, finest=case["level"]))
    for finest in range(case["level"], case["finest"]):
        f.refine((_hit(case, level, x, y) & (level == finest)).astype(np.int32), max_level=case["finest"])
        level, x, y = _leaves(dict(case, finest=finest + 1))
    f.balance()
    if f.num_quads != len(level):
        raise RuntimeError("the forest's quads are not the case's")
    return f


def _config(case):
    import amrgpu as ag
    cfg = ag.Config.from_input(cfl=0.5, time_scheme=case["scheme"], nelem_subgrid=case["n"], coarse_grid_h=1.0,
                               time_steps=10 ** 9, dt=1.0, bc=[1] * 6, gamma=1.4, form=case["form"],
                               regrid_interval=max(case["steps"], 1), amr_ntag_methods=1,
                               amr_tag_methods=[5, 0, 0, 0, 0], amr_tag_tolerances=[0.9, 0, 0, 0, 0])
    return cfg.apply()


class _Device:
    """A session's state, (4, cells) in device memory, as torch sees it; the session lives as long as that."""

    def __init__(self, session, ptr, pitch, cells):
        self.session = session
        self.__cuda_array_interface__ = dict(shape=(4, cells), strides=(8 * pitch, 8), typestr="<f8",
                                             data=(ptr, False), version=3)


def _view(st):
    s = st["session"]
    ptr, cells = s.state_ptr(0), s.mesh.ncells
    v = st["views"].get((ptr, cells))
    if v is None:
        v = st["views"][ptr, cells] = torch.as_tensor(_Device(s, ptr, (s.state_ptr(1) - ptr) // 8, cells),
                                                          device="cuda")
    return v


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    return dict(march=_prepare_march, evolve=_prepare_evolve, amr=_prepare_amr, classify=_prepare_classify,
                train=_prepare_train)[case["kind"]](case, seed)


def _session(case, seed):
    import amrgpu as ag
    torch.cuda.current_device()
    f, cfg = _forest(case), _config(case)
    s = ag.Session(f.mesh(case["n"]), cfg, form=case["form"])
    s.upload(_state(case, _leaves(case), seed).cpu().numpy().reshape(-1))
    return f, cfg, s


def _prepare_march(case, seed):
    f, cfg, s = _session(case, seed)
    if s.mesh.ncell >= 256:
        s.autotune()
    return dict(case=case, forest=f, config=cfg, session=s, views={})


def _prepare_evolve(case, seed):
    f, cfg = _forest(case), _config(case)
    return dict(case=case, config=cfg, mesh=f.mesh(case["n"]),
                soln=_state(case, _leaves(case), seed).cpu().numpy().reshape(-1))


def _roi(case, forest, moved):
    """The program's own wish for every quad: 1 refine, 2 keep, 0 coarsen, from the circle's place."""
    tree, level, x, y = forest.quads()
    lv = level.astype(np.int64)
    w, h = case["trees_x"], case["trees_y"]
    ty, tx = np.divmod(np.arange(w * h), w)
    order = np.argsort(_interleave(tx) | (_interleave(ty) << np.uint64(1)), kind="stable")
    gx = (tx[order][tree] << lv) + (x >> (30 - lv))
    gy = (ty[order][tree] << lv) + (y >> (30 - lv))
    near = _hit(case, lv, gx, gy, moved)
    keep = (lv > case["level"]) & _hit(case, lv, gx, gy, moved, parents=1)
    return np.where(near, 1, np.where(keep, 2, 0)).astype(np.int32)


def _prepare_amr(case, seed):
    f, cfg, s = _session(case, seed)
    s.reserve(3 * s.mesh.ncells, 3 * s.mesh.ncell)
    # the circle grows by half of the second-finest width and shrinks again; the mesh is led through that
    # until it comes back to what it was, and the wishes of that round are kept
    places = (0.5 ** case["finest"], 0.0)
    before = None
    for _ in range(12):
        rois = []
        for moved in places:
            rois.append(_roi(case, f, moved))
            s.adapt_regrid(f, case["level"], case["finest"], tags=rois[-1])
        after = np.stack(f.quads()[:2])
        if before is not None and before.shape == after.shape and (before == after).all():
            break
        before = after
    else:
        raise RuntimeError("the mesh does not come back")
    leaves = f.quads()
    lv = leaves[1].astype(np.int64)
    w, h = case["trees_x"], case["trees_y"]
    ty, tx = np.divmod(np.arange(w * h), w)
    order = np.argsort(_interleave(tx) | (_interleave(ty) << np.uint64(1)), kind="stable")
    gx = (tx[order][leaves[0]] << lv) + (leaves[2] >> (30 - lv))
    gy = (ty[order][leaves[0]] << lv) + (leaves[3] >> (30 - lv))
    s.upload(_state(case, (lv, gx, gy), seed).cpu().numpy().reshape(-1))
    if s.mesh.ncell >= 256:
        s.autotune()
    return dict(case=case, forest=f, config=cfg, session=s, rois=rois, views={})


def _prepare_classify(case, seed):
    from amrgpu import learned
    f, cfg, s = _session(case, seed)
    g = np.random.default_rng(seed)
    m = learned.Mlp(seed=0)
    params = []
    for rows, cols in ((128, 400), (64, 128), (3, 64)):
        params += [g.normal(size=rows * cols) * 1.5 / math.sqrt(cols), g.normal(size=rows) * 0.1]
    m.set_params(np.concatenate(params).astype(np.float32))
    return dict(case=case, forest=f, config=cfg, session=s, mlp=m)


def _prepare_train(case, seed):
    from amrgpu import learned
    mesh = _mesh("march", (1, 1), 6, 6, 8, FP32, 3, 10)
    f, cfg, s = _session(mesh, seed)
    m = learned.Mlp(seed=seed % 1000)
    while m.size() < case["rows"]:
        m.append(s, 0.02)
        s.step(10)
    s.sync()
    s.close()
    perm = np.random.default_rng(seed).permutation(m.size())[: case["rows"]].astype(np.int32)
    return dict(case=case, mlp=m, perm=perm)


# ------------------------------------------------------------------ run
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "march":
        st["session"].step(case["steps"], graph_steps=12 if case.get("graph") else 0)
        return _view(st)
    if kind == "evolve":
        import amrgpu as ag
        ag.evolve_solver(st["mesh"], st["soln"], 0)
        return st["soln"]
    if kind == "amr":
        s = st["session"]
        for roi in st["rois"]:
            s.step(case["steps"])
            rep = s.sync()
            tags = s.tag()
            s.adapt_regrid(st["forest"], case["level"], case["finest"], tags=np.maximum(tags, roi))
        return dict(state=_view(st), tags=tags, quads=s.mesh.ncell, time=rep["time"], dt=rep["dt_last"])
    if kind == "classify":
        cls, judge = st["mlp"].tags(st["session"], 0.02, judge_fraction=0.05, seed=7)
        return dict(classes=cls, judged=judge["judged"], disagree=judge["disagree"], coarser=judge["coarser"])
    loss, accuracy = st["mlp"].train_epoch(st["perm"], batch=case["batch"], lr=1e-3)
    return dict(loss=loss, accuracy=accuracy, params=st["mlp"].get_params())


# ------------------------------------------------------------------ work
def work(case):
    if case["kind"] == "train":
        rows = case["rows"] // case["batch"] * case["batch"]
        mults = 400 * 128 + 128 * 64 + 64 * 3
        # a row's 400 BF16 features once; forward, input gradients and weight gradients
        return dict(bytes=rows * 804 + 8 * NPARAMS, flops=rows * (4 * mults + 2 * (128 * 64 + 64 * 3)))
    quads = len(_leaves(case)[0])
    cells = quads * case["n"] ** 2
    if case["kind"] == "classify":
        return dict(bytes=32 * cells + 4 * quads, flops=2 * quads * NPARAMS + 4 * cells)
    # a step reads a state and writes a state; a stage takes about 330 operations a cell (two faces, the record, the
    # update). An adaptive turn has two runs of steps and moves the state to another mesh twice.
    turns = 2 if case["kind"] == "amr" else 1
    steps = turns * case["steps"]
    moves = steps + (2 if case["kind"] == "amr" else 0)
    return dict(bytes=64 * cells * moves, flops=330 * cells * steps * STAGES[case["scheme"]])


# ------------------------------------------------------------------ the same in 64 bits
def _sides(case, leaves):
    """Per side (x-, x+, y-, y+) of every quad: its neighbours (two where it is the coarse one of a hanging face; -1:
    none, a wall) and how much of the quad's width its face has."""
    level, x, y = leaves
    w, h = case["trees_x"], case["trees_y"]
    lo, hi = int(level.min()), int(level.max())
    grid = {}
    for lv in range(lo - 1, hi + 2):
        grid[lv] = np.full((max(1, int(h * 2.0 ** lv)), max(1, int(w * 2.0 ** lv))), -1, np.int64)
    for lv in range(lo, hi + 1):
        at = np.nonzero(level == lv)[0]
        grid[lv][y[at], x[at]] = at
    first = np.full((4, len(x)), -1, np.int64)
    second = np.full((4, len(x)), -1, np.int64)
    share = np.ones((4, len(x)))
    for lv in range(lo, hi + 1):
        at = np.nonzero(level == lv)[0]
        for s, (dx, dy) in enumerate(((-1, 0), (1, 0), (0, -1), (0, 1))):
            ax, ay = x[at] + dx, y[at] + dy
            if case["periodic"]:
                ax, ay = ax % (w << lv), ay % (h << lv)
            inside = (ax >= 0) & (ay >= 0) & (ax < w << lv) & (ay < h << lv)
            q, ax, ay = at[inside], ax[inside], ay[inside]
            same = grid[lv][ay, ax]
            first[s, q] = same
            if lv > lo:
                m = same < 0
                first[s, q[m]] = grid[lv - 1][ay[m] >> 1, ax[m] >> 1]
            m = first[s, q] < 0
            if m.any():
                a, b = 2 * ax[m] + (dx < 0), 2 * ay[m] + (dy < 0)
                first[s, q[m]] = grid[lv + 1][b, a]
                second[s, q[m]] = grid[lv + 1][b + (dx != 0), a + (dy != 0)]
                share[s, q[m]] = 0.5
    return first, second, share


def _flux(ql, qr, d):
    """The solver's face flux along axis d, per unit length: HLLE with the contact and shear waves restored at the
    Roe average. States are (..., 4)."""
    def prims(q):
        r, mu, mv, e = q.unbind(-1)
        u, v = mu / r, mv / r
        p = 0.4 * (e - 0.5 * r * (u * u + v * v))
        return r, u, v, p, (e + p) / r
    rl, ul, vl, pl, hl = prims(ql)
    rr, ur, vr, pr, hr = prims(qr)
    nl, nr = (ul, ur) if d == 0 else (vl, vr)
    sl, sr = rl.sqrt(), rr.sqrt()
    t = 1.0 / (sl + sr)
    rb = (rl * rr).sqrt()
    ub, vb, hb = (ul * sl + ur * sr) * t, (vl * sl + vr * sr) * t, (hl * sl + hr * sr) * t
    ab = (0.4 * (hb - 0.5 * (ub * ub + vb * vb))).sqrt()
    nb = ub if d == 0 else vb
    bp = torch.maximum(nb + ab, nr + ab).clamp(min=0.0)
    bm = torch.minimum(nb - ab, nl - ab).clamp(max=0.0)
    bc = bp * bm / (bp - bm)
    bk = bc / (1.0 + (nb / ab).abs())
    d1 = (rr - rl) - (pr - pl) / (ab * ab)
    dn = nr - nl
    wave = torch.stack([d1, d1 * ub + rb * (ur - ul - (dn if d == 0 else 0.0)),
                        d1 * vb + rb * (vr - vl - (dn if d == 1 else 0.0)), d1 * hb + rb * (hr - hl)], dim=-1)

    def phys(q, un, p):
        f = q * un[..., None]
        f[..., 1 + d] += p
        f[..., 3] += p * un
        return f
    jump = qr - ql
    jump = torch.cat([jump[..., :3], (rr * hr - rl * hl)[..., None]], dim=-1)
    return ((bp[..., None] * phys(ql, nl, pl) - bm[..., None] * phys(qr, nr, pr)) / (bp - bm)[..., None]
            + bc[..., None] * jump - bk[..., None] * wave)


def _wall(q, d):
    """Flux of a slip wall: the pressure of the state without its velocity into the wall."""
    t = q[..., 2 - d]
    f = torch.zeros_like(q)
    f[..., 1 + d] = 0.4 * (q[..., 3] - 0.5 * t * t / q[..., 0])
    return f


class _Exact:
    def __init__(self, case, leaves):
        self.n = case["n"]
        first, second, share = _sides(case, leaves)
        self.first, self.second, self.share = (torch.from_numpy(v).cuda() for v in (first, second, share))
        self.width = torch.exp2(-torch.from_numpy(leaves[0]).double()).cuda()[:, None, None, None] / self.n
        self.cfl = 0.25 * 0.5 * case["scheme"]
        self.scheme = case["scheme"]

    @staticmethod
    def _edge(q, s):
        return (q[:, :, 0], q[:, :, -1], q[:, 0], q[:, -1])[s]

    def rate(self, q):
        """dQ/dt."""
        out = torch.zeros_like(q)
        f = _flux(q[:, :, :-1], q[:, :, 1:], 0)
        out[:, :, :-1] -= f
        out[:, :, 1:] += f
        f = _flux(q[:, :-1], q[:, 1:], 1)
        out[:, :-1] -= f
        out[:, 1:] += f
        for s in range(4):
            d, sign = s // 2, -1.0 if s % 2 else 1.0
            own, facing = self._edge(q, s), self._edge(q, s ^ 1)
            total = torch.zeros_like(own)
            for nbr in (self.first[s], self.second[s]):
                at = torch.nonzero(nbr >= 0)[:, 0]
                other = facing[nbr[at]]
                f = _flux(own[at], other, d) if s % 2 else _flux(other, own[at], d)
                total[at] += f * self.share[s][at][:, None, None]
            at = torch.nonzero(self.first[s] < 0)[:, 0]
            total[at] = _wall(own[at], d)
            self._edge(out, s).add_(total, alpha=sign)
        return out / self.width

    def dt(self, q):
        r = q[..., 0]
        v2 = (q[..., 1] ** 2 + q[..., 2] ** 2) / r ** 2
        c = (1.4 * 0.4 * (q[..., 3] / r - 0.5 * v2)).sqrt()
        return min(1.0, float((self.cfl * self.width[..., 0] / (v2.sqrt() + c)).min()))

    def step(self, q):
        h, k = self.dt(q), self.rate(q)
        if self.scheme == 1:
            return q + h * k
        if self.scheme == 3:
            q1 = q + h * k
            q2 = 0.75 * q + 0.25 * (q1 + h * self.rate(q1))
            return q / 3.0 + 2.0 / 3.0 * (q2 + h * self.rate(q2))
        if self.scheme == 4:
            k2 = self.rate(q + 0.5 * h * k)
            k3 = self.rate(q + 0.5 * h * k2)
            return q + h / 6.0 * (k + 2.0 * k2 + 2.0 * k3 + self.rate(q + h * k3))
        a = (0.0, -567301805773 / 1357537059087, -2404267990393 / 2016746695238, -3550918686646 / 2091501179385,
             -1275806237668 / 842570457699)
        b = (1432997174477 / 9575080441755, 5161836677717 / 13612068292357, 1720146321549 / 2090206949498,
             3134564353537 / 4481467310338, 2277821191437 / 14882151754819)
        w = torch.zeros_like(q)
        for i in range(5):
            w = a[i] * w + h * (k if i == 0 else self.rate(q))
            q = q + b[i] * w
        return q


def exact(case, seed):
    # the adaptive loop's outputs are copies and averages on a mesh that follows from the library's own regrid
    # rules; classes are whole numbers; training rounds to BF16 at every layer, which has no 64-bit counterpart
    if case["kind"] not in ("march", "evolve"):
        return None
    leaves = _leaves(case)
    e = _Exact(case, leaves)
    q = _state(case, leaves, seed)
    for _ in range(case["steps"]):
        q = e.step(q)
    if case["kind"] == "evolve":
        return q.reshape(-1)
    return q.reshape(-1, 4).T.contiguous()
