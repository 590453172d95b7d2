"""Learned absorbing boundary on the GPU, through the C ABI (part 4), against
the CPU oracle (oracle/abc_mlp.py).

* the training kernel's loss and gradient vs the oracle's analytic FP64
  gradient with the same FP16 roundings: relative L2 <= 1e-3 (FP32
  accumulation);
* the tensor-core inference path vs the oracle's forward: within 3e-2 of
  the outputs' RMS (tanh.approx and FP16 rounding of the activations);
* collected training samples (features and targets of ghost cells) vs the
  oracle's restatement at the same cells;
* one step of the resident one-way layer: the fixed-coefficient form equals
  the oracle's box-scheme update of the plain step (1e-6), the learned form
  equals it with the oracle network's coefficients (1e-2 of the update's
  size), and nothing outside the ghost zone changes;
* end to end at 96^3: training lowers the loss, and the learned layer
  reflects clearly less than the one-way layer without the network and the
  32-cell random shell.
"""
import numpy as np
import pytest

from conftest import gpu_available
from fletcher_petrobras_gb300 import Propagator
from fletcher_petrobras_gb300 import learned
from fletcher_petrobras_gb300._lib import iptr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not gpu_available():
        pytest.fail("these tests need a CUDA GPU")


def rel(a, b):
    a = np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def random_features(n, seed):
    g = np.random.default_rng(seed)
    f = np.empty((n, 40), np.float32)
    f[:, :36] = g.uniform(-1, 1, (n, 36))
    f[:, 36] = g.uniform(0.37, 1.0, n)
    f[:, 37] = g.uniform(0, 0.3, n)
    f[:, 38] = f[:, 37] * g.uniform(0, 1, n)
    f[:, 39] = g.integers(5, 9, n) / 8.0
    return f


def test_gradient_vs_cpu_oracle():
    from oracle import abc_mlp

    learned.init(3)
    P = learned.get_weights()
    X = random_features(300, 1)
    T = np.random.default_rng(2).normal(0, 1, (300, 4)).astype(np.float32)
    loss, g = learned.gradient(X, T)
    oloss, og = abc_mlp.loss_and_grad(P, X, T)
    assert abs(loss - oloss) <= 1e-4 * oloss
    assert rel(g, og) < 1e-3
    for name, (o, s) in abc_mlp.OFF.items():
        assert rel(g[o:o + s], og[o:o + s]) < 3e-3, name


def test_inference_path_vs_cpu_oracle():
    from oracle import abc_mlp

    learned.init(4)
    P = learned.get_weights()
    X = random_features(1000, 5)  # not a multiple of 16: the last tile is partial
    y = learned.forward(X)
    oy, _ = abc_mlp.forward(P, X)
    rms = np.sqrt(np.mean(oy ** 2))
    assert np.max(np.abs(y - oy)) < 3e-2 * rms
    assert rel(y, oy) < 1e-2


@pytest.mark.parametrize("n", [1, 15, 16, 17, 63, 64, 65, 129, 13312, 13313, 19521])
def test_network_batch_edges_vs_cpu_oracle(n):
    """Loss, gradient and outputs where a training block of 64 samples and an
    inference tile of 16 rows begin and end, and where a block begins to take
    several chunks of 64 (from 13 313 samples).  In few samples an FP16
    rounding that falls the other way is not averaged out: it changes one of
    a sample's 32 activations by 2^-11 of itself, so loss and gradient are
    held to 2^-10."""
    from oracle import abc_mlp

    learned.init(6)
    P = learned.get_weights()
    X = random_features(n, 11 + n)
    T = np.random.default_rng(12 + n).normal(0, 1, (n, 4)).astype(np.float32)
    loss, g = learned.gradient(X, T)
    oloss, og = abc_mlp.loss_and_grad(P, X, T)
    assert abs(loss - oloss) <= 2.0 ** -10 * oloss
    assert rel(g, og) < 2.0 ** -10
    y = learned.forward(X)
    oy, _ = abc_mlp.forward(P, X)
    assert np.max(np.abs(y - oy)) < 3e-2 * np.sqrt(np.mean(oy ** 2))


def test_collected_samples_vs_cpu_restatement():
    from oracle import abc_mlp

    prob, lo, hi = learned.training_problem(0, n_virtual=16, steps=60)
    prop = Propagator()
    prop.initialize(prob.sx, prob.sy, prob.sz, prob.bord, prob.dx, prob.dy, prob.dz, prob.dt, prob.raw_model())
    prop.run(60, prob.i_source, prob.sources(60))
    prop.synchronize()
    lib = prop.lib
    assert lib.FLETCHER_AbcReserve(200000) == 0
    lo_a, hi_a = np.array(lo, np.int32), np.array(hi, np.int32)
    assert lib.FLETCHER_AbcCollect(iptr(lo_a), iptr(hi_a), learned.LAYER, 1.0, 5, 0.0) == 0
    f, t, cells = learned.samples()
    shape = (prob.sz, prob.sy, prob.sx)
    cur = np.stack([prop.field(0).reshape(shape), prop.field(1).reshape(shape)])
    prev = np.stack([prop.field(2).reshape(shape), prop.field(3).reshape(shape)])
    coef = prop.coefficients().reshape((10,) + shape)
    prop.finalize()
    # every ghost cell with a wave on it, once
    ghost = {c[:3] + (c[3] + 8 * c[4],) for c in abc_mlp.ghost_cells(lo, hi, learned.LAYER)}
    got = {tuple(int(v) for v in c) for c in cells}
    assert len(f) > 1000 and len(got) == len(f) and got <= ghost
    pick = np.random.default_rng(0).choice(len(f), 200, replace=False)
    sel = [(int(c[0]), int(c[1]), int(c[2]), int(c[3]) % 8, int(c[3]) // 8) for c in cells[pick]]
    of, ot = abc_mlp.features_targets(cur, prev, coef, lo, hi, learned.LAYER, sel, (prob.dx, prob.dy, prob.dz),
                                      prob.dt)
    assert np.max(np.abs(f[pick] - of)) < 1e-5
    # a and b are differences of O(1) values (over s): FP32 rounding of the update
    assert np.max(np.abs(t[pick] - ot)) < 1e-5 * np.max(np.abs(ot)) + 1e-5


def _one_step(prob, model, fields, mode):
    prop = Propagator()
    prop.initialize(prob.sx, prob.sy, prob.sz, prob.bord, prob.dx, prob.dy, prob.dz, prob.dt, model, *fields)
    assert prop.lib.FLETCHER_SetBoundary(mode, learned.LAYER, 0.0) == 0
    ncells = prop.lib.FLETCHER_AbcLayerCells()
    prop.run(1)
    prop.synchronize()
    out = np.stack([prop.field(0), prop.field(1)])
    prop.lib.FLETCHER_SetBoundary(learned.BOUNDARY_PLAIN, 0, 0.0)
    prop.finalize()
    return out, ncells


def test_resident_oneway_steps_vs_cpu_oracle():
    """One step with the fixed-coefficient and the learned ghost zone: the
    plain step followed by the oracle's box-scheme update (with the
    medium's coefficients, and with sigmoid of the oracle network on the
    oracle's inputs), and no change outside the ghost zone."""
    from oracle import abc_mlp

    learned.init(6)
    P = learned.get_weights()
    prob = learned.boundary_problem("learned", 16, 150)
    model = prob.raw_model()
    prop = Propagator()
    prop.initialize(prob.sx, prob.sy, prob.sz, prob.bord, prob.dx, prob.dy, prob.dz, prob.dt, model)
    prop.run(150, prob.i_source, prob.sources(150))
    prop.synchronize()
    f = [prop.field(k) for k in (2, 0, 3, 1)]  # pp pc qp qc
    coef = prop.coefficients()
    prop.finalize()
    shape = (prob.sz, prob.sy, prob.sx)
    plain, _ = _one_step(prob, model, f, learned.BOUNDARY_PLAIN)
    fixed, n_fixed = _one_step(prob, model, f, learned.BOUNDARY_ONEWAY)
    lrn, n_lrn = _one_step(prob, model, f, learned.BOUNDARY_LEARNED)
    b, L = prob.bord, learned.LAYER
    lo, hi = (b + L,) * 3, (prob.sx - b - L, prob.sy - b - L, prob.sz - b - L)
    cells = abc_mlp.ghost_cells(lo, hi, L)
    assert n_fixed == n_lrn == len(cells)
    cur = np.stack([f[1].reshape(shape), f[3].reshape(shape)]).astype(np.float64)
    prev = np.stack([f[0].reshape(shape), f[2].reshape(shape)]).astype(np.float64)
    base = plain.reshape((2,) + shape).astype(np.float64)
    mask = np.zeros(shape, bool)
    for (x, y, z, _, _) in cells:
        mask[z, y, x] = True
    scale = np.abs(cur).max()
    assert scale > 0
    # fixed coefficients, from the medium in FP32 as the library computes them
    c4 = coef.reshape((10,) + shape)
    k = np.empty((len(cells), 2))
    dt, h = np.float32(prob.dt), (prob.dx, prob.dy, prob.dz)
    for i, (x, y, z, fc, d) in enumerate(cells):
        v2pz, v2px = np.float32(c4[7, z, y, x]), np.float32(c4[6, z, y, x])
        vpz = np.sqrt(v2pz)
        eps = np.float32(0.5) * (v2px / v2pz - np.float32(1))
        a = abc_mlp.face_axis(fc)
        c = vpz if a == 2 else vpz * np.sqrt(np.float32(1) + np.float32(2) * eps)
        r = c * dt / np.float32(h[a])
        k[i] = (1 - r) / (1 + r)
    want = abc_mlp.oneway_update(cur, base.copy(), lo, hi, L, k)
    got = fixed.reshape((2,) + shape)
    assert np.max(np.abs(got - want)) < 1e-6 * scale
    assert np.array_equal(got[:, ~mask], plain.reshape((2,) + shape)[:, ~mask])
    # learned coefficients
    X, _ = abc_mlp.features_targets(cur, prev, c4, lo, hi, L, cells, h, prob.dt, targets=False)
    y, _ = abc_mlp.forward(P, X)
    want = abc_mlp.oneway_update(cur, base.copy(), lo, hi, L, abc_mlp.sigmoid(y))
    got = lrn.reshape((2,) + shape)
    size = np.max(np.abs(want - base)[:, mask])
    assert size > 0
    assert np.max(np.abs(got - want)) < 1e-2 * size + 1e-6 * scale
    assert np.array_equal(got[:, ~mask], plain.reshape((2,) + shape)[:, ~mask])


def _ghost_update(cur, prev, base, c4, prob, weights):
    """The oracle's features, network and box-scheme update (the medium's
    coefficients where weights is None), a slab of one distance at a time."""
    from oracle import abc_mlp

    b, L = prob.bord, learned.LAYER
    dims = (prob.sx, prob.sy, prob.sz)
    h = (prob.dx, prob.dy, prob.dz)
    nxt = base.astype(np.float64)
    vpz = np.sqrt(c4[7])
    eps, delta = (np.float32(0.5) * (c4[k] / c4[7] - np.float32(1)) for k in (6, 9))
    for f in range(6):
        a, sgn = abc_mlp.face_axis(f), abc_mlp.face_sign(f)

        def slab(F, d):  # the kept box's cells at distance d outward
            n = b + L - d if sgn < 0 else dims[a] - b - L - 1 + d
            ix = [slice(b, dims[t] - b) for t in (2, 1, 0)]
            ix[2 - a] = n
            return F[(Ellipsis, *ix)]

        for d in range(L - 3, L + 1):
            g = slab(cur, d)
            if weights is None:
                c = slab(vpz, d) if a == 2 else slab(vpz, d) * np.sqrt(np.float32(1) + np.float32(2) * slab(eps, d))
                r = c * np.float32(prob.dt) / np.float32(h[a])
                k = np.broadcast_to((1 - r) / (1 + r), g.shape)
            else:
                st = [slab(F, d + o)[c] if d + o <= L else np.zeros(g.shape[1:])
                      for F in (cur, prev) for c in (0, 1) for o in range(-4, 5)]
                st = np.stack(st, -1).reshape(-1, 36)
                s = np.abs(st).max(1, keepdims=True)
                X = np.concatenate([st / s] + [np.reshape(np.broadcast_to(m, g.shape[1:]), (-1, 1)) for m in (
                    slab(vpz, d) / 4000.0, slab(eps, d), slab(delta, d), d / L)], 1)
                y, _ = abc_mlp.forward(weights, X)
                k = abc_mlp.sigmoid(y).T.reshape(g.shape)
            slab(nxt, d)[...] = slab(cur, d - 1) + k * (g - slab(nxt, d - 1))
    return nxt


@pytest.mark.parametrize("n", [(1, 1, 1), (3, 30, 7), (95, 91, 2), (2, 290, 281)])
def test_ghost_update_on_ragged_boxes(n):
    """The boundary kernels where a face's rays are no multiple of a warp's
    group and where a pass takes one round of the grid or several (16 200
    rays for the network kernel, 150 000 for the other), against the oracle's
    update of the plain step; the network's bound as in the test above."""
    b, L = 4, learned.LAYER
    prob = learned.Problem("ghost", *n, absorb=L, bord=b, dt=0.0006, steps=1, kind="layered", layers=3, seed=5)
    shape = (prob.sz, prob.sy, prob.sx)
    g = np.random.default_rng(sum(n))
    f = []
    for _ in range(4):  # pp pc qp qc
        v = np.zeros(shape, np.float32)
        v[b:-b, b:-b, b:-b] = g.uniform(-1, 1, tuple(s - 2 * b for s in shape))
        f.append(v.ravel())
    model = prob.raw_model()
    learned.init(6)
    plain, _ = _one_step(prob, model, f, learned.BOUNDARY_PLAIN)
    prop = Propagator()
    prop.initialize(prob.sx, prob.sy, prob.sz, b, prob.dx, prob.dy, prob.dz, prob.dt, model)
    c4 = prop.coefficients().reshape((10,) + shape)
    prop.finalize()
    cur = np.stack([f[1], f[3]]).reshape((2,) + shape).astype(np.float64)
    prev = np.stack([f[0], f[2]]).reshape((2,) + shape).astype(np.float64)
    base = plain.reshape((2,) + shape)
    for mode, weights in ((learned.BOUNDARY_ONEWAY, None), (learned.BOUNDARY_LEARNED, learned.get_weights())):
        got, _ = _one_step(prob, model, f, mode)
        want = _ghost_update(cur, prev, base, c4, prob, weights)
        size = np.max(np.abs(want - base))
        # Fixed: four cells' FP32 rounding and that of k, 3 ulp of up to 5 / 4 of size each.
        tol = (2e-6 if weights is None else 1e-2) * size
        assert np.max(np.abs(got.reshape(want.shape) - want)) < tol


def test_training_and_reflected_energy_small():
    """What the trained network gains over the method without it.  Training on
    32 padded models (the library's kernels, reproducible), then the
    reflected energy of each form against the wide-domain run at 96^3 x 900
    steps.  The one-way layer with the medium's coefficients (the method
    without the network) and the learned one both beat the bare 8-cell
    layer, and the learned layer reflects clearly less than both the one-way
    layer and the 32-cell random shell (measured 0.0071 vs 0.0112 and
    0.0102)."""
    n_s = learned.collect(models=32, n_virtual=48, keep=0.1, capacity=3_000_000)
    assert n_s > 500_000
    learned.init(0)
    loss = learned.train(iters=3000, batch=8192, lr=3e-3)
    print(f"samples {n_s}, loss {loss[:20].mean():.4g} -> {loss[-50:].mean():.4g}")
    assert loss[-50:].mean() < 0.3 * loss[:20].mean()
    res = learned.compare(n=96, steps=900, nsnap=3, kinds=("random", "learned", "oneway", "plain8"))
    for k, v in res.items():
        print(k, v)
    e = {k: v["reflected_energy"] for k, v in res.items() if k != "snapshots"}
    assert e["wide"] == 0.0
    assert 0.0 < e["random"] < e["plain8"]
    assert 0.0 < e["oneway"] < e["plain8"]
    assert 0.0 < e["learned"] < 0.8 * e["oneway"]
    assert e["learned"] < e["random"]
    assert res["learned"]["launches_per_step"] == 2 and res["oneway"]["launches_per_step"] == 2


def test_interval_reuses_the_coefficients():
    """With the network every 2 steps the first step equals the every-step
    run bit for bit (both evaluate it), the second differs (it reuses the
    first step's coefficients)."""
    learned.init(7)
    prob = learned.boundary_problem("learned", 16, 150)
    model = prob.raw_model()
    prop = Propagator()
    prop.initialize(prob.sx, prob.sy, prob.sz, prob.bord, prob.dx, prob.dy, prob.dz, prob.dt, model)
    prop.run(150, prob.i_source, prob.sources(150))
    prop.synchronize()
    f = [prop.field(k) for k in (2, 0, 3, 1)]
    prop.finalize()
    out = {}
    for interval in (1, 2):
        prop = Propagator()
        prop.initialize(prob.sx, prob.sy, prob.sz, prob.bord, prob.dx, prob.dy, prob.dz, prob.dt, model, *f)
        assert prop.lib.FLETCHER_AbcSetInterval(interval) == 0
        assert prop.lib.FLETCHER_SetBoundary(learned.BOUNDARY_LEARNED, learned.LAYER, 0.0) == 0
        prop.run(1)
        a = prop.field(0)
        prop.run(1)
        out[interval] = (a, prop.field(0))
        prop.lib.FLETCHER_SetBoundary(learned.BOUNDARY_PLAIN, 0, 0.0)
        prop.lib.FLETCHER_AbcSetInterval(1)
        prop.finalize()
    assert np.array_equal(out[1][0], out[2][0])
    assert not np.array_equal(out[1][1], out[2][1])
    assert np.max(np.abs(out[1][1] - out[2][1])) < 0.1 * np.max(np.abs(out[1][1]))


def test_collection_and_training_are_reproducible():
    """The training set lands in cell order and the gradient sums are added
    in block order, so collecting and training twice gives the same samples,
    losses and weights bit for bit."""
    runs = []
    for _ in range(2):
        learned.collect(models=2, n_virtual=16, times=(40, 60), keep=0.5, capacity=200_000)
        f, t, c = learned.samples()
        learned.init(5)
        loss = learned.train(iters=40, batch=1024, lr=3e-3)
        runs.append((f, t, c, loss, learned.get_weights()))
    assert len(runs[0][0]) > 100
    for a, b in zip(runs[0], runs[1]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("interval", [1, 2])
def test_fused_boundary_rollout_vs_cpu_oracle(interval, orc):
    """Four steps of the learned layer (one boundary launch per step: the
    network kernel on evaluation steps, the ray kernel in between) against
    a CPU rollout: the oracle's plain step, its features of (t, t-1) --
    after the first step the GPU takes t-1 from the line buffer it carried
    over, not from the field -- its network and its box-scheme update.  The
    network's k is held for `interval` steps."""
    from oracle import abc_mlp

    learned.init(6)
    P = learned.get_weights()
    prob = learned.boundary_problem("learned", 16, 150)
    model = prob.raw_model()
    prop = Propagator()
    prop.initialize(prob.sx, prob.sy, prob.sz, prob.bord, prob.dx, prob.dy, prob.dz, prob.dt, model)
    prop.run(150, prob.i_source, prob.sources(150))
    prop.synchronize()
    f = [prop.field(k) for k in (2, 0, 3, 1)]  # pp pc qp qc
    coef = prop.coefficients()
    prop.finalize()
    steps = 4
    prop = Propagator()
    prop.initialize(prob.sx, prob.sy, prob.sz, prob.bord, prob.dx, prob.dy, prob.dz, prob.dt, model, *f)
    assert prop.lib.FLETCHER_AbcSetInterval(interval) == 0
    assert prop.lib.FLETCHER_SetBoundary(learned.BOUNDARY_LEARNED, learned.LAYER, 0.0) == 0
    prop.run(steps)
    prop.synchronize()
    got = np.stack([prop.field(0), prop.field(1)])
    prop.lib.FLETCHER_SetBoundary(learned.BOUNDARY_PLAIN, 0, 0.0)
    prop.lib.FLETCHER_AbcSetInterval(1)
    prop.finalize()
    # CPU rollout.  The oracle's time loop always adds a source; it is put at
    # grid cell 0, which no update reads, and that cell is left out below.
    shape = (prob.sz, prob.sy, prob.sx)
    quiet = prob.with_(source=(0, 0, 0))
    b, L = prob.bord, learned.LAYER
    lo, hi = (b + L,) * 3, (prob.sx - b - L, prob.sy - b - L, prob.sz - b - L)
    cells = abc_mlp.ghost_cells(lo, hi, L)
    c4 = coef.reshape((10,) + shape)
    h = (prob.dx, prob.dy, prob.dz)
    prev = np.stack([f[0], f[2]]).astype(np.float32)
    cur = np.stack([f[1], f[3]]).astype(np.float32)
    k = None
    size = 0.0
    for s in range(steps):
        p1, q1, _, _ = orc.run_f32(quiet, model, steps=1, coef=coef, fields=(prev[0], cur[0], prev[1], cur[1]))
        base = np.stack([p1, q1]).reshape((2,) + shape).astype(np.float64)
        c64 = cur.reshape((2,) + shape).astype(np.float64)
        if s % interval == 0:
            X, _ = abc_mlp.features_targets(c64, prev.reshape((2,) + shape).astype(np.float64), c4, lo, hi, L, cells,
                                            h, prob.dt, targets=False)
            y, _ = abc_mlp.forward(P, X)
            k = abc_mlp.sigmoid(y)
        new = abc_mlp.oneway_update(c64, base.copy(), lo, hi, L, k)
        size = max(size, float(np.max(np.abs(new - base))))
        prev, cur = cur, new.reshape(2, -1).astype(np.float32)
    want = cur.reshape(2, -1).astype(np.float64)
    g = got.astype(np.float64)
    g[:, 0] = want[:, 0] = 0.0
    assert size > 0
    err = float(np.max(np.abs(g - want)))
    print(f"interval {interval}: max |GPU - oracle| {err:.3g} against an update size {size:.3g}")
    assert err < 3e-2 * size + 1e-6 * np.abs(want).max()
