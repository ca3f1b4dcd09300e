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
