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
# 152 SMs x 4 CTAs x 2 tiles of 128 rows in flight: 155,649 rows leave a second round of one row.
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
@pytest.mark.parametrize("n,grid,group", [(700, 8, 2), (5003, 16, 4), (20011, 24, 8)])
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
