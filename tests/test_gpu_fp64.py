"""FP64 results against extended precision, at the rounding errors of FP64 arithmetic: what the header
calls FP64 pairs and an FP64 direct sum is computed in 53 bits, whatever the number of terms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

EPS = 2.0 ** -53


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def direct_sums(x, y, m, eps, at):
    """Accelerations of the particles `at` and the sums of their terms' magnitudes, in long double."""
    x, y, m = (np.asarray(a, dtype=np.longdouble) for a in (x, y, m))
    e2 = np.longdouble(eps * eps)
    a, size = np.zeros((2, len(at)), np.longdouble), np.zeros(len(at), np.longdouble)
    for k, i in enumerate(at):
        dx, dy = x - x[i], y - y[i]
        s = dx * dx + dy * dy + e2
        s[i] = 1.0
        w = m / s
        w[i] = 0.0
        a[:, k] = np.sum(w * dx), np.sum(w * dy)
        size[k] = np.sum(w * np.sqrt(dx * dx + dy * dy))
    return a, size


# Systems of few particles, 8,400 and more in the batch: short sums, where no errors average out.  All
# coordinates are multiples of 2^-20 with corners at 0 and 1, so differences and box-relative offsets
# are exact in FP64 and a pair's error is that of its arithmetic: r^2 + eps^2 two roundings, the
# reciprocal 1.02, the weight one, the product and its addition one, each 2^-53 of the term at most.  A
# target's sum adds ceil(n / 32) terms a slice and at most min(n, 128) slices.
@pytest.mark.parametrize("n,systems", [(2, 4200), (9, 1000), (65, 150), (501, 17)])
@pytest.mark.parametrize("theta,eps", [(0.0, 0.0), (0.5, 2.0 ** -10), (0.5, 0.3)])
@pytest.mark.parametrize("heavy", [False, True])
def test_fp64_forces_of_small_systems(n, systems, theta, eps, heavy):
    from barneshut.gb300 import native

    rng = np.random.default_rng(n + 2 * systems + heavy)
    xy = np.zeros((systems, 2, n))
    for s in range(systems):  # distinct points, so no pair is coincident
        c = rng.choice((1 << 20) - 1, (2, n), replace=False) + 1.0
        xy[s] = c / (1 << 20)
        xy[s, :, 0], xy[s, :, -1] = 0.0, 1.0
    m = rng.uniform(0.5, 1.0, (systems, n))
    if heavy:
        m[:, n // 2] *= 1e9
    z = np.zeros(n * systems)
    prm = native.make_params(1.0, 1e-5, eps, 0.0, theta, 1, native.BH_PREC_FP64)
    plan = native.Plan([n] * systems, [2] * systems, prm)
    plan.load(xy[:, 0].ravel(), xy[:, 1].ravel(), m.ravel(), z, z)
    plan.create_tree()
    plan.summarize()
    plan.evaluate()
    out = plan.store()
    assert plan.error_flags() == 0
    got = torch.stack([out["ax"], out["ay"]]).cpu().numpy().reshape(2, systems, n)
    bound = (5.1 + np.ceil(n / 32) + min(n, 128)) * EPS
    for s in range(0, systems, max(1, systems // 150)):
        ref, size = direct_sums(xy[s, 0], xy[s, 1], m[s], eps, range(n))
        err = np.sqrt((((got[:, s] - ref) / size) ** 2).sum(0))
        assert float(err.max()) <= bound, float(err.max()) / EPS


# The sampler over half a million sources and more of which eight have mass, or one has 1e9 times the
# others': its result is an FP64 sum also where no errors average out.  A pair has 8.1 roundings of at most
# 2^-53 (two differences, two of r^2's own and their two in it, reciprocal, weight and product).  Eight
# terms: seven additions more, at most.  A heavy one: every addition after it rounds the whole sum; at most
# 96 of them in a row (runs of 16, a thread's runs, slices, chunks), whose errors, 2^-53 at most and
# independent, add up as a random walk.
@pytest.mark.parametrize("nt", [16, 37])
@pytest.mark.parametrize("eps", [0.0, 1e-3])
@pytest.mark.parametrize("heavy", [False, True])
def test_direct_sample_of_few_masses(nt, eps, heavy):
    from barneshut.gb300 import native

    n = (1 << 19) + 77
    rng = np.random.default_rng(nt)
    x, y = rng.random((2, n))
    if heavy:
        m = rng.uniform(0.5, 1.0, n)
        m[n // 3] = 1e9
    else:
        m = np.zeros(n)
        m[rng.choice(n, 8, replace=False)] = rng.uniform(0.5, 1.0, 8)
    z = np.zeros(n)
    plan = native.Plan([n], [64], native.make_params(1.0, 1e-5, eps, 0.0, 0.5))
    plan.load(x, y, m, z, z)
    t = rng.choice(n, nt, replace=False)
    ax, ay = plan.direct_sample(t)
    got = np.stack([ax.cpu().numpy(), ay.cpu().numpy()])
    if heavy:  # (half a million terms a target in extended precision)
        t, got = t[:8], got[:, :8]
    used = np.unique(np.r_[np.flatnonzero(m), t])
    ref, size = direct_sums(x[used], y[used], m[used], eps, np.searchsorted(used, t))
    err = np.sqrt((((got - ref) / size) ** 2).sum(0))
    if heavy:
        assert float(np.sqrt(np.mean(err ** 2))) <= np.sqrt(8.1 + 96) * EPS
    else:
        assert float(err.max()) <= (8.1 + 7) * EPS


# Samplers on several streams of one plan, of the same system and of two, beside each other and beside an
# FP64 evaluation: each gives what it gives alone, bit for bit, and so does the evaluation.
def test_overlapping_samplers_and_evaluation():
    from barneshut.gb300 import native

    rng = np.random.default_rng(3)
    sizes = [60000, 90000]
    n = sum(sizes)
    x, y, m = rng.random(n), rng.random(n), rng.uniform(0.5, 1.0, n)
    z = np.zeros(n)
    plan = native.Plan(sizes, [64, 64], native.make_params(1.0, 1e-5, 1e-3, 0.0, 0.6, 2, native.BH_PREC_FP64))
    plan.load(x, y, m, z, z)
    plan.create_tree()
    plan.summarize()
    calls = [(rng.choice(sizes[s], k, replace=False) + s * sizes[0], s) for s, k in ((0, 9), (1, 300), (1, 50), (0, 1200))]
    alone = [torch.stack(plan.direct_sample(t, sys=s)) for t, s in calls]
    plan.evaluate()
    want = [plan.store()[k] for k in ("ax", "ay")]
    streams = [torch.cuda.Stream() for _ in calls]
    torch.cuda.synchronize()
    for _ in range(3):
        plan.create_tree()
        plan.summarize()
        got = []
        for st in streams:
            st.wait_stream(torch.cuda.current_stream())
        plan.evaluate()
        for st, (t, s) in zip(streams, calls):
            with torch.cuda.stream(st):
                got.append(torch.stack(plan.direct_sample(t, sys=s)))
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(alone, got))
        out = plan.store()
        assert torch.equal(out["ax"], want[0]) and torch.equal(out["ay"], want[1])
    assert plan.error_flags() == 0


# Target and source counts at the edges of the sampler's tiles, chunks and thread layouts: one target a
# thread and four, tiles of 4 to 64 with idle targets, one chunk to eight, against extended precision.
# 32 + 16 + 8 + 8 additions of a sum's roundings beside a pair's 8.1, of the terms' magnitudes.
@pytest.mark.parametrize("n,nt", [(2, 1), (255, 7), (257, 75), (511, 76), (2049, 303), (2048, 304), (4097, 305), (3001, 2433),
                                  (1500, 1216), (70001, 5), (300, 1000)])
def test_direct_sample_layouts(n, nt):
    from barneshut.gb300 import native

    rng = np.random.default_rng(n + nt)
    x, y, m = rng.random(n), rng.random(n), rng.uniform(0.5, 1.0, n)
    z = np.zeros(n)
    plan = native.Plan([n], [2], native.make_params(1.0, 1e-5, 1e-3, 0.0, 0.5))
    plan.load(x, y, m, z, z)
    t = np.resize(rng.permutation(n), nt)  # (targets may repeat)
    ax, ay = plan.direct_sample(t)
    got = np.stack([ax.cpu().numpy(), ay.cpu().numpy()])
    some = np.unique(np.r_[np.arange(min(nt, 12)), rng.choice(nt, min(nt, 12), replace=False), nt - 1])
    ref, size = direct_sums(x, y, m, 1e-3, t[some])
    err = np.sqrt((((got[:, some] - ref) / size) ** 2).sum(0))
    assert float(err.max()) <= (8.1 + 64) * EPS
    for i in set(t.tolist()) if nt > n else ():
        assert len(np.unique(got[0, t == i])) == 1


# The FP64 pairs' reciprocal against the division, element by element, through the sampler: a source of mass
# m at the origin and a target at (-2^k, -y) give m / s * 2^k with s = 2^2k + y^2 (y^2 rounded, then the sum),
# an exact multiple of the weight.  Within one unit in the last place of the rounded quotient, and equal to
# it where the division is taken.
def reciprocal_case(e, rng, mantissa=None):
    """(k, y, s) of an r^2 near 2^e."""
    y = np.ldexp(np.sqrt(rng.uniform(1.0, 4.0) if mantissa is None else mantissa), e // 2)
    k = e // 2 - 1
    s = np.float64(np.longdouble(np.ldexp(1.0, 2 * k)) + np.longdouble(y * y))
    return k, y, s


def test_reciprocal_random_mantissas():
    from barneshut.gb300 import native

    n = 40000
    rng = np.random.default_rng(77)
    e = rng.integers(-300, 300, n)
    k, y, s = (np.array(v) for v in zip(*(reciprocal_case(int(v), rng) for v in e)))
    x = -np.ldexp(1.0, k)
    m = np.zeros(n)
    x[0], y[0], m[0] = 0.0, 0.0, 1.0
    plan = native.Plan([n], [4], native.make_params(1.0, 1e-5, 0.0, 0.0, 0.5))
    plan.load(x, -y, m, np.zeros(n), np.zeros(n))
    ax, _ = plan.direct_sample(np.arange(1, n))
    got, want = np.ldexp(ax.cpu().numpy(), -k[1:]), 1.0 / s[1:]
    assert np.abs((got - want) / np.spacing(want)).max() <= 1.0
    assert (got == want).mean() > 0.9  # (half a unit and 2^-7 of one: nearly always the rounded quotient)


def test_reciprocal_every_exponent():
    from barneshut.gb300 import native

    rng = np.random.default_rng(78)
    cases = []
    for e in list(range(-1074, 1024)) + 4 * [-1000, -999, -998, 1001, 1002, 1003]:
        cases.append(reciprocal_case(e, rng) + (1.0,))
        if not -990 < e < 990:  # a mass whose quotient is in range where the reciprocal is not
            cases.append(reciprocal_case(e, rng) + (float(np.ldexp(rng.uniform(1.0, 2.0), np.clip(e, -1000, 1000))),))
    cases += [(-10, 1e200, np.inf, 1.0), (0, np.inf, np.inf, 1.0), (0, np.nan, np.nan, 1.0), (0, 0.0, 1.0, np.inf)]
    S = len(cases)
    xy, m = np.zeros((2, 2 * S)), np.zeros(2 * S)
    for c, (k, y, s, mass) in enumerate(cases):
        xy[:, 2 * c + 1] = -np.ldexp(1.0, k), -y
        m[2 * c] = mass
    plan = native.Plan([2] * S, [1] * S, native.make_params(1.0, 1e-5, 0.0, 0.0, 0.5))
    plan.load(xy[0], xy[1], m, np.zeros(2 * S), np.zeros(2 * S))
    got = torch.cat([plan.direct_sample([2 * c + 1], sys=c)[0] for c in range(S)]).cpu().numpy()
    for (k, y, s, mass), a in zip(cases, got):
        with np.errstate(all="ignore"):
            want = np.float64(mass) / s * np.ldexp(1.0, k)
        usual = np.isfinite(s) and s > 0 and 24 <= np.frexp(s)[1] + 1022 <= 2024
        if not usual or np.isinf(want):
            assert a == want or (np.isnan(a) and np.isnan(want)), (k, y, s, mass, a, want)
        else:
            assert abs(a - want) <= np.spacing(abs(want)), (k, y, s, mass, a, want)
