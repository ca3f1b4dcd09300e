"""CUDA kernels at the sizes where their tilings end: tile edges, remainders, the smallest and the
largest of a range, odd strides and alignments -- each against the repository's oracle or against
the general path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def rel_rms(a, b):
    return float(np.sqrt(np.sum((a - b) ** 2) / np.sum(b ** 2)))


def network_rows(n, seed, width=8):
    rng = np.random.default_rng(seed)
    f = np.zeros((n, width), dtype=np.float32)
    u, v = rng.uniform(-3, 3, size=(2, n))
    f[:, 0], f[:, 1], f[:, 2:5], f[:, 5] = u, v, rng.uniform(0, 0.2, (n, 3)), 1.0 / np.sqrt(u * u + v * v + 0.1)
    t = np.stack([np.sin(u) * 0.3, np.cos(v) * 0.2], axis=1).astype(np.float32)
    return f, t


# Forward: BF16 operands at the oracle's rounding points, so 2e-2 as in the network's own tests.
# 152 SMs x 8 tiles of 128 rows in flight: 155,649 rows leave a second round of one row.
@pytest.mark.parametrize("n,width", [(1, 6), (127, 7), (128, 8), (129, 9), (257, 12), (155649, 6)])
def test_network_forward_rows_and_strides(n, width):
    from barneshut.gb300.learned import LearnedCorrection
    from oracle import mlp_oracle

    mlp = LearnedCorrection(seed=21)
    f, _ = network_rows(n, n, width)
    out = mlp.forward(torch.from_numpy(f)).cpu().numpy()
    ref, _ = mlp_oracle.forward(mlp.params.cpu().numpy(), f[:, :8].astype(np.float64))
    assert out.shape == (n, 2) and rel_rms(out, ref) < 2e-2
    mlp.check_errors()


# Gradients: cosine and loss as in the network's own tests; 19,457 rows give one SM a second tile
# of a single row; the shifted gradient buffer takes the scalar additions.
@pytest.mark.parametrize("n,width,shift", [(1, 6, 0), (128, 8, 0), (129, 7, 1), (19457, 8, 0), (19457, 6, 3)])
def test_network_gradient_rows_and_alignment(n, width, shift):
    import ctypes

    from barneshut.gb300.learned import LearnedCorrection
    from oracle import mlp_oracle

    mlp = LearnedCorrection(seed=22)
    f, t = network_rows(n, n, width)
    F, T = torch.from_numpy(f).cuda(), torch.from_numpy(t).cuda()
    store = torch.zeros(10448 + 4, dtype=torch.float32, device="cuda")
    grad = store[shift:shift + 10448]
    loss = torch.zeros(1, device="cuda")
    rc = mlp.L.bh_mlp_train_batch(*[ctypes.c_void_p(F.data_ptr()), width, ctypes.c_void_p(T.data_ptr()), n,
                                    mlp._img(), ctypes.c_void_p(mlp.params.data_ptr()),
                                    ctypes.c_void_p(grad.data_ptr()), ctypes.c_void_p(loss.data_ptr()),
                                    ctypes.c_void_p(mlp.err.data_ptr()), mlp._st()])
    assert rc == 0
    g = grad.cpu().numpy().astype(np.float64)
    ref_loss, rg = mlp_oracle.loss_and_grad(mlp.params.cpu().numpy(), f[:, :8].astype(np.float64), t)
    assert abs(float(loss.item()) / (2 * n) - ref_loss) < 2e-2 * ref_loss
    assert float(np.dot(g, rg) / np.linalg.norm(g) / np.linalg.norm(rg)) > 0.998
    assert not store[:shift].any() and not store[shift + 10448:].any()
    mlp.check_errors()


# The correction over work items of at most 128 targets (streamed lists) and of at most 512 (the
# walk): the same groups, so the same band cells and the same network outputs in another tiling.
# Its sums are FP32 (2^-24 relative a term, some hundred terms) and are read off as the difference
# of two accelerations some ten times larger: 1e-4 relative RMS.
@pytest.mark.parametrize("n,grid,group", [(700, 8, 2), (5003, 16, 4), (20011, 24, 8), (20011, 64, 2), (60011, 64, 2)])
def test_learned_correction_item_sizes(n, grid, group):
    from barneshut.gb300 import learned, native, workloads

    s = workloads.cluster_mixture(n, seed=n)
    p = learned.init_params(23)
    mlp = learned.LearnedCorrection(params=p)
    corr = []
    for walk in (0, native.BH_FLAG_WALK):
        acc = []
        for flag in (0, native.BH_FLAG_LEARNED):
            prm = native.make_params(1.0, 1e-5, 1e-4, 0.0, 0.8, group, native.BH_PREC_FP32_KAHAN, walk | flag,
                                     correction_theta=0.5)
            plan = native.Plan([n], [grid], prm)
            if flag:
                plan.set_correction(mlp)
            plan.load(*s)
            plan.create_tree()
            plan.summarize()
            plan.evaluate()
            out = plan.store()
            assert plan.error_flags() == 0
            acc.append(torch.stack([out["ax"], out["ay"]]).cpu().numpy())
        corr.append(acc[1] - acc[0])
    assert np.abs(corr[0]).max() > 0
    assert rel_rms(corr[0], corr[1]) < 1e-4


# FP64 sums of at most 1e5 terms: 1e-16 a rounding, far below 1e-12.  Tiles of 4 to 64 targets, one
# chunk and many, a target count over the scratch, softened and not.
@pytest.mark.parametrize("n,nt,eps", [(1, 1, 0.1), (5, 5, 0.0), (1000, 3, 1e-4), (1000, 1000, 0.0), (4099, 65, 1e-2),
                                      (100003, 1, 1e-4), (30011, 700, 0.0)])
def test_direct_sample_tiles_and_chunks(n, nt, eps):
    from barneshut.gb300 import native

    rng = np.random.default_rng(n + nt)
    x, y, vx, vy = rng.random((4, n))
    m = 1.0 + rng.random(n)
    plan = native.Plan([n], [4], native.make_params(0.7, 1e-5, eps, 0.0, 0.5))
    plan.load(x, y, m, vx, vy)
    plan.step(1)
    state = {k: v.cpu().numpy() for k, v in plan.store().items()}
    x, y = state["x"], state["y"]
    t = rng.choice(n, nt, replace=False)
    ax, ay = plan.direct_sample(t)
    rx, ry = np.empty(nt), np.empty(nt)
    for k, i in enumerate(t):
        dx, dy = np.delete(x, i) - x[i], np.delete(y, i) - y[i]
        w = np.delete(m, i) / (dx * dx + dy * dy + eps * eps)
        rx[k], ry[k] = 0.7 * np.sum(w * dx), 0.7 * np.sum(w * dy)
    got, ref = np.concatenate([ax.cpu().numpy(), ay.cpu().numpy()]), np.concatenate([rx, ry])
    assert np.linalg.norm(got - ref) <= 1e-12 * np.linalg.norm(ref)
    after = plan.store()  # the sampler leaves the state alone
    assert all(np.array_equal(after[k].cpu().numpy(), state[k]) for k in state)


def test_direct_sample_of_a_system_in_a_batch():
    from barneshut.gb300 import native

    rng = np.random.default_rng(5)
    n = [300, 2000]
    x, y, v = rng.random((3, 2300))
    m = 1.0 + rng.random(2300)
    plan = native.Plan(n, [2, 4], native.make_params(1.0, 1e-5, 1e-3, 0.0, 0.5))
    plan.load(x, y, m, v, v)
    alone = native.Plan([2000], [4], native.make_params(1.0, 1e-5, 1e-3, 0.0, 0.5))
    alone.load(x[300:], y[300:], m[300:], v[300:], v[300:])
    t = np.array([300, 1234, 2299, 299, 0])
    ax, _ = plan.direct_sample(t, sys=1)
    bx, _ = alone.direct_sample(t[:3] - 300)
    assert torch.allclose(ax[:3], bx, rtol=1e-12, atol=0)
    assert torch.isnan(ax[3:]).all()  # not particles of the system


# The walking force kernel with one CTA per item (a batch whose items fill the chip) and with two (a
# system alone): the same sums.  Leaf sums differ by their chunk offsets (1e-7 of a box edge), so
# accelerations agree within 1e-5 relative RMS, the oracle tests' own bound.
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("cutoff,eps", [(0.0, 0.0), (1e-5, 0.0), (1e-5, 1e-3), (0.0, 1e-3)])
def test_walk_items_one_or_two_ctas(prec, cutoff, eps):
    from barneshut.gb300 import native, workloads

    sizes, grids = [1, 3, 700, 2049, 5000, 9000, 1500, 4000, 6001], [1, 2, 2, 3, 4, 8, 16, 16, 12]
    systems = [workloads.uniform(n, seed=n) for n in sizes]
    prm = native.make_params(1.0, 1e-5, eps, cutoff, 0.0, 1, prec)

    def accel(n, g, cols):
        plan = native.Plan(n, g, prm)
        plan.load(*cols)
        plan.create_tree()
        plan.summarize()
        plan.evaluate()
        out = plan.store()
        assert plan.error_flags() == 0
        return torch.stack([out["ax"], out["ay"]]).cpu().numpy(), plan.pair_counts()

    big, pairs = accel(sizes, grids, [np.concatenate([s[k] for s in systems]) for k in range(5)])
    o, near, far = 0, 0, 0
    for s, n, g in zip(systems, sizes, grids):
        one, (a, b) = accel([n], [g], s)
        near, far = near + a, far + b
        if n > 1:
            assert rel_rms(big[:, o:o + n], one) < 1e-5
        o += n
    assert pairs == (near, far)


# A small plan splits its heaviest work items over several warps: half or a quarter of each quad of
# targets with the same slices and the same order of sources.  The same system in a batch whose other
# systems raise the item bound past the rule runs whole items; without boxes that straddle leaf chunks
# (every system's particle count a multiple of 32) its leaf sums are the same, and so is every bit.
@pytest.mark.parametrize("n,grid,group,dense,quad,layout", [(32, 1, 1, 16, -1, "uniform"), (4096, 8, 1, 16, 128, "cluster"),
                                                            (20000, 16, 2, 0, 0, "cluster"), (65536, 8, 4, 16, -1, "uniform")])
@pytest.mark.parametrize("prec,tune", [(0, 0), (1, 0), (1, 1)])
def test_split_items_are_the_same_bits(n, grid, group, dense, quad, layout, prec, tune):
    from barneshut.gb300 import native, workloads

    s = (workloads.uniform if layout == "uniform" else workloads.cluster_mixture)(n, seed=n)
    rest = workloads.uniform(1 << 21, seed=7)
    prm = native.make_params(1.0, 1e-5, 1e-4, 0.0, 0.5, group, prec, 0, tune, dense_min=dense, quad_min=quad)

    def accel(sizes, grids, cols):
        plan = native.Plan(sizes, grids, prm)
        plan.load(*cols)
        plan.step(1)
        out = plan.store()
        assert plan.error_flags() == 0
        return [out[k][:n].cpu().numpy() for k in ("ax", "ay", "x", "y", "vx", "vy")]

    alone = accel([n], [grid], s)
    both = accel([n, 1 << 21], [grid, 181], [np.concatenate([s[k], rest[k]]) for k in range(5)])
    assert all(np.array_equal(a, b) for a, b in zip(alone, both))


# Download of a state whose box order is far from the pid order (gathered from 262,144 particles on) or
# close to it (scattered): create_tree reorders the state and changes nothing else.
@pytest.mark.parametrize("n", [1, 262143, 262144, 300007])
@pytest.mark.parametrize("order", ["file", "box"])
def test_store_returns_the_state(n, order):
    from barneshut.gb300 import native, workloads

    s = workloads.cluster_mixture(n, seed=3)
    if order == "box":
        o = workloads.box_order(s[0], s[1], 64)
        s = tuple(a[o] for a in s)
    plan = native.Plan([n], [64], native.make_params(1.0, 1e-5, 1e-4, 0.0, 0.5))
    vx, vy = np.random.default_rng(n).random((2, n))
    plan.load(s[0], s[1], s[2], vx, vy)
    for _ in range(2):
        out = plan.store()
        rec = plan.store_records().cpu().numpy()
        for k, a in (("x", s[0]), ("y", s[1]), ("vx", vx), ("vy", vy)):
            assert np.array_equal(out[k].cpu().numpy(), a)
        assert np.array_equal(rec[:, :5], np.stack([s[0], s[1], s[2], vx, vy], axis=1))
        assert np.array_equal(rec[:, 9], np.arange(n)) and not rec[:, 5:7].any()
        plan.create_tree()
    assert plan.error_flags() == 0


# The order within a quadrant is the input order whatever slots the placement handed out: quadrants at
# the edges of the sorting forms (registers of a thread, of a warp, merged runs, radix passes), in random
# input order against the same particles loaded in box order; one system (the small-system kernel) and two.
@pytest.mark.parametrize("systems", [1, 2])
@pytest.mark.parametrize("count", [2, 16, 17, 32, 33, 64, 65, 128, 129, 256, 257, 512, 513, 1024, 1025, 3000, 4096, 4097])
def test_quadrant_sort_sizes(count, systems):
    from barneshut.gb300 import native, workloads

    rng = np.random.default_rng(count)
    counts = np.array([count, count, max(1, count - 1), 3])
    q = np.repeat(np.arange(4), counts)
    n = len(q) + 2
    x = np.concatenate([[0.0, 1.0], 0.25 * (q >> 1) + 0.01 + 0.22 * rng.random(len(q))])
    y = np.concatenate([[0.0, 1.0], 0.25 * (q & 1) + 0.01 + 0.22 * rng.random(len(q))])
    o = rng.permutation(n)
    x, y = x[o], y[o]
    m = 1.0 + rng.random(n)
    z = np.zeros(n)
    prm = native.make_params(1.0, 1e-5, 1e-3, 0.0, 0.5, 1, quad_min=128)

    def accel(cols):
        plan = native.Plan([n] * systems, [2] * systems, prm)
        plan.load(*(np.tile(c, systems) for c in (*cols, z, z)))
        plan.step(1)
        out = plan.store()
        assert plan.error_flags() == 0
        return torch.stack([out["ax"], out["ay"]]).cpu().numpy().reshape(2, systems, n)[:, -1]

    b = workloads.box_order(x, y, 2)
    assert np.array_equal(accel((x, y, m))[:, b], accel((x[b], y[b], m[b])))


# A batch of more systems than a block has threads, empty ones among them: each with its own box.
def test_bounding_boxes_of_many_systems():
    from barneshut.gb300 import native

    rng = np.random.default_rng(9)
    sizes = [int(v) for v in rng.integers(0, 40, 300)] + [5000, 0, 8192, 1]
    shift = rng.uniform(-5, 5, (len(sizes), 2))
    pts = [shift[k] + rng.random((v, 2)) for k, v in enumerate(sizes)]
    x, y = np.concatenate(pts).T.copy()
    n = len(x)
    plan = native.Plan(sizes, [3] * len(sizes), native.make_params(1.0, 1e-5, 1e-3, 0.0, 0.5))
    plan.load(x, y, np.ones(n), np.zeros(n), np.zeros(n))
    plan.create_tree()
    for k, p in enumerate(pts):
        if len(p):
            g = plan.grid_info(k)
            assert (g["min_x"], g["min_y"]) == (p[:, 0].min(), p[:, 1].min())
    assert plan.error_flags() == 0


# One small system's tree, work items and moments by one cluster against the general kernels (the same
# system first in a batch; its particle count a multiple of 32 keeps the leaf chunks' offsets): the same
# bits, phase by phase and fused.  Quadrants of 0 to 8,192 particles and more, one box to 64 x 64.
@pytest.mark.parametrize("n,grid,layout", [(32, 1, "uniform"), (32, 64, "uniform"), (1056, 3, "cluster"), (8192, 17, "uniform"), (16384, 64, "cluster"), (16384, 2, "coincident"),
                                           (16416, 64, "cluster"), (2048, 16, "coincident")])
@pytest.mark.parametrize("mode", ["stream", "walk", "flat", "fp64"])
def test_cluster_tree_is_the_general_tree(n, grid, layout, mode):
    from barneshut.gb300 import native, workloads

    if layout == "coincident":  # half of them in one point
        s = list(workloads.uniform(n, seed=1))
        s[0][: n // 2], s[1][: n // 2] = 0.37, 0.61
        o = np.random.default_rng(2).permutation(n)
        s = tuple(a[o] for a in s)
    else:
        s = (workloads.uniform if layout == "uniform" else workloads.cluster_mixture)(n, seed=n + grid)
    rest = workloads.uniform(64, seed=8)
    kw = dict(stream=dict(theta=0.5, softening=1e-3, cutoff_r2=0.0), flat=dict(theta=0.0, cutoff_r2=1e-5),
              walk=dict(theta=0.6, softening=1e-3, cutoff_r2=0.0, flags=native.BH_FLAG_WALK),
              fp64=dict(theta=0.5, softening=1e-3, cutoff_r2=0.0, precision=native.BH_PREC_FP64))[mode]
    prm = native.make_params(1.0, 1e-6, group_dim=0 if mode == "flat" else 2, **kw)

    def result(sizes, grids, cols):
        plan = native.Plan(sizes, grids, prm)
        out = []
        for fused in (False, True):
            plan.load(*cols)
            if fused:
                plan.step(2)
            else:
                plan.create_tree()
                plan.summarize()
                plan.evaluate()
                out.append(plan.box_moments(0))
            st = plan.store()
            out += [st[k][:n] for k in ("x", "y", "vx", "vy", "ax", "ay")]
            out.append(plan.store_records()[:n])
        assert plan.error_flags() == 0
        return [a.cpu().numpy() for a in out]

    alone = result([n], [grid], s)
    batch = result([n, 64], [grid, 2], [np.concatenate([s[k], rest[k]]) for k in range(5)])
    for a, b in zip(alone, batch):
        assert np.array_equal(a, b)


def test_adam_with_images_is_adam_then_pack():
    from barneshut.gb300.learned import LearnedCorrection

    rng = np.random.default_rng(31)
    f, t = network_rows(500, 31)
    F, T = torch.from_numpy(f).cuda(), torch.from_numpy(t).cuda()
    a = LearnedCorrection(seed=31)
    a.grad_batch(F, T)
    b = LearnedCorrection(seed=31)
    b.grad.copy_(a.grad)
    a.adam_step(1e-3)
    b.step_count += 1
    assert b.L.bh_mlp_adam(b.params.data_ptr(), b.m.data_ptr(), b.v.data_ptr(), b.grad.data_ptr(), 1, 1e-3, b._st()) == 0
    b.pack()
    assert torch.equal(a.params, b.params) and torch.equal(a.m, b.m) and torch.equal(a.v, b.v)
    x = torch.from_numpy(rng.standard_normal((300, 6)).astype(np.float32)).cuda()
    assert torch.equal(a.forward(x), b.forward(x))
    a.grad_batch(F, T)
    b.grad_batch(F, T)
    assert torch.allclose(a.grad, b.grad, rtol=1e-4, atol=1e-6)  # (FP32 additions in another order)


# Long direct sums: coincident and very close pairs, one mass far above the others, a system far from the
# origin; and a target of another system.
@pytest.mark.parametrize("kind", ["plain", "close", "heavy", "offset"])
@pytest.mark.parametrize("eps", [0.0, 1e-3])
def test_direct_sample_long_sums(kind, eps):
    from barneshut.gb300 import native

    n, nt = 524287 + 1024, 37
    rng = np.random.default_rng(len(kind))
    x, y = rng.random((2, n))
    m = 1.0 + rng.random(n)
    t = rng.choice(n - 200, nt, replace=False)
    if kind == "close":
        x[n - 100:n - 63], y[n - 100:n - 63] = x[t] + 1e-9 * rng.random(nt), y[t] - 1e-12
        if eps > 0.0:
            x[n - 50:n - 13], y[n - 50:n - 13] = x[t], y[t]
    elif kind == "heavy":
        m[5] = 1e25
    elif kind == "offset":
        x, y = x + 12345.0, y - 77.0
    z = np.zeros(n)
    plan = native.Plan([100, n], [2, 4], native.make_params(1.0, 1e-5, eps, 0.0, 0.5))
    pad = rng.random((2, 100))
    plan.load(np.r_[pad[0], x], np.r_[pad[1], y], np.r_[np.ones(100), m], np.r_[z[:100], z], np.r_[z[:100], z])
    ax, ay = plan.direct_sample(np.r_[t + 100, 3], sys=1)
    got = np.stack([ax.cpu().numpy(), ay.cpu().numpy()])
    assert np.isnan(got[:, nt]).all()
    for k, i in enumerate(t):
        dx, dy = np.delete(x, i) - x[i], np.delete(y, i) - y[i]
        w = np.delete(m, i) / (dx * dx + dy * dy + eps * eps)
        ref = np.array([np.sum(w * dx), np.sum(w * dy)])
        assert np.linalg.norm(got[:, k] - ref) <= 1e-12 * np.linalg.norm(ref)


# FP64 forces with every pair near (8,200 particles): close and coincident pairs, pairs at the cutoff, a mass
# far above the others, a system far off, another in the batch.  FP64 sums of 8,000 terms: 1e-12.
@pytest.mark.parametrize("kind", ["plain", "close", "cutoff", "heavy", "offset"])
@pytest.mark.parametrize("theta,eps,cutoff", [(0.0, 0.0, 1e-5), (0.0, 0.0, 0.0), (0.5, 1e-3, 0.0), (0.0, 1e-2, 1e-4)])
def test_fp64_forces_in_split_floats(kind, theta, eps, cutoff):
    from barneshut.gb300 import native

    n, extra = 8200, 300
    rng = np.random.default_rng(len(kind) + 7)
    x, y = rng.random((2, n))
    m = 1.0 + rng.random(n)
    t = rng.choice(n - 200, 40, replace=False)
    if kind == "close":
        x[n - 100:n - 60], y[n - 100:n - 60] = x[t] + 1e-7, y[t]
        x[n - 60:n - 20], y[n - 60:n - 20] = x[t], y[t]
    elif kind == "cutoff" and cutoff > 0.0:
        f = np.sqrt(cutoff) * (1.0 + np.array([1e-4, -1e-4, 1e-7, -1e-7] * 10))
        x[n - 100:n - 60], y[n - 100:n - 60] = x[t] + f * np.cos(t), y[t] + f * np.sin(t)
    elif kind == "heavy":
        m[3] = 1e22
    elif kind == "offset":
        x, y = x + 4321.0, y - 99.0
    o = rng.random((2, extra))
    z = np.zeros(n + extra)
    prm = native.make_params(1.0, 1e-5, eps, cutoff, theta, 1, native.BH_PREC_FP64)
    plan = native.Plan([extra, n], [1, 2], prm)
    plan.load(np.r_[o[0], x], np.r_[o[1], y], np.r_[np.ones(extra), m], z, z)
    for _ in range(2):  # (the sampler and a second evaluation use the same scratch)
        plan.create_tree()
        plan.summarize()
        plan.evaluate()
    out = plan.store()
    assert plan.error_flags() == 0
    got = np.stack([out["ax"].cpu().numpy(), out["ay"].cpu().numpy()])[:, extra:]
    for i in t:
        dx, dy = x - x[i], y - y[i]
        r2 = dx * dx + dy * dy
        with np.errstate(divide="ignore", invalid="ignore"):
            w = np.where(r2 > cutoff, m / (r2 + eps * eps), 0.0)
        w[i] = 0.0
        ref = np.array([np.sum(w * dx), np.sum(w * dy)])
        assert np.linalg.norm(got[:, i] - ref) <= 1e-12 * np.linalg.norm(ref)


# Kernels set up while their predecessor runs still wait for everything before them: tensors written on
# another stream that the plan's stream was made to wait for (after kernels of its own), and a step captured
# in a caller's graph, whole call sequence and all, give the results of a plain sequence.
@pytest.mark.parametrize("n,grid", [(10000, 16), (40000, 32)])
def test_launches_wait_for_other_streams_and_capture(n, grid):
    from barneshut.gb300 import native

    rng = np.random.default_rng(n)
    prm = native.make_params(1.0, 1e-5, 1e-3, 0.0, 0.5, 1)
    sets = [[torch.from_numpy(rng.random(n)).cuda() for _ in range(3)] for _ in range(2)]
    z = torch.zeros(n, dtype=torch.float64, device="cuda")

    def run(plan, s):
        plan.load(*s, z, z)
        plan.step(2)
        out = plan.store()
        return torch.stack([out[k] for k in ("x", "y", "vx", "vy", "ax", "ay")])

    plan = native.Plan([n], [grid], prm)
    want = [run(plan, s).clone() for s in sets]
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    cols = [torch.empty_like(c) for c in sets[0]]
    big = torch.ones(64 << 20, device="cuda")
    torch.cuda.synchronize()
    got = []
    for k in range(6):
        with torch.cuda.stream(b):
            for _ in range(4):
                big.mul_(1.0)  # keeps the copies below late
            for c, src in zip(cols, sets[k & 1]):
                c.copy_(src)
        with torch.cuda.stream(a):
            a.wait_stream(b)
            got.append(run(plan, cols))
        b.wait_stream(a)
    torch.cuda.synchronize()
    assert all(torch.equal(g, want[k & 1]) for k, g in enumerate(got))

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = run(plan, cols)
    for k in range(4):
        for c, src in zip(cols, sets[k & 1]):
            c.copy_(src)
        g.replay()
        assert torch.equal(out, want[k & 1])
    assert plan.error_flags() == 0


# Queues of fewer entries than CTAs or warps, of as many, and of more: every item is taken once and the
# accelerations match FP64 sums (all pairs are near with 2 x 2 boxes).  Tolerance: FP32 pairs of 3e-7 and FP32
# sums of at most n terms (a random walk of 2^-24 steps).
@pytest.mark.parametrize("n", [1, 5, 129, 1025, 6007])
@pytest.mark.parametrize("theta", [0.0, 0.5])
def test_queue_entries_taken_once(n, theta):
    from barneshut.gb300 import native

    rng = np.random.default_rng(n)
    x, y, m = rng.random(n), rng.random(n), rng.uniform(1, 2, n)
    z = np.zeros(n)
    plan = native.Plan([n], [2], native.make_params(1.0, 1e-5, 1e-3, 0.0, theta))
    for _ in range(2):  # the queue starts again for the next launch
        plan.load(x, y, m, z, z)
        plan.create_tree()
        plan.summarize()
        plan.evaluate()
        out = plan.store()
        dx, dy = x[None, :] - x[:, None], y[None, :] - y[:, None]
        w = m[None, :] / (dx * dx + dy * dy + 1e-6)
        got = np.stack([out["ax"].cpu().numpy(), out["ay"].cpu().numpy()])
        ref = np.stack([(w * dx).sum(1), (w * dy).sum(1)])
        assert np.sqrt(((got - ref) ** 2).sum()) <= 1e-5 * max(np.sqrt((ref ** 2).sum()), 1e-30)
    assert plan.error_flags() == 0


# Pairs at the cutoff: a jittered lattice whose neighbours' r^2 straddles it by parts in 1e7, where the FP64
# positions decide, in half items (few groups) and whole ones (20 x 20 groups), with groups of sources and the
# remainders of a slice.  A wrong decision changes a force by m / r, a thousand times the tolerance (that of
# FP32 pairs and sums against FP64 ones).
@pytest.mark.parametrize("side,grid", [(3, 1), (9, 1), (23, 2), (60, 3), (80, 20), (101, 21)])
def test_cutoff_decided_in_groups(side, grid):
    from barneshut.gb300 import native
    from oracle import oracle

    rng = np.random.default_rng(side)
    h = np.sqrt(1e-5)
    i, j = np.meshgrid(np.arange(side), np.arange(side))
    x = (i.ravel() + rng.uniform(-1, 1, side * side) * 1e-7) * h + 0.25
    y = (j.ravel() + rng.uniform(-1, 1, side * side) * 1e-7) * h + 0.5
    m = rng.uniform(1, 2, side * side)
    z = np.zeros(side * side)
    plan = native.Plan([side * side], [grid], native.make_params(1.0, 1e-5, 0.0, 1e-5, 0.0))
    plan.load(x, y, m, z, z)
    plan.create_tree()
    plan.summarize()
    plan.evaluate()
    out = plan.store()
    ref = oracle.reference_evaluate(x, y, m, G=grid, gconst=1.0)
    assert oracle.rel_rms(out["ax"].cpu().numpy(), out["ay"].cpu().numpy(), ref["ax"], ref["ay"]) <= 1e-5
    assert plan.error_flags() == 0
