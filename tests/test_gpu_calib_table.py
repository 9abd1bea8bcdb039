"""The table gather and fold of the calibration against the torch operations they stand for: gathered values bit for bit,
the gradient within FP64 rounding of the sums (n positions of one row: n * 2^-53 relative to the sum of magnitudes)."""
import numpy as np
import pytest

from gatk_gb300 import calibration as C
from gatk_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    pytest.importorskip("torch")
    from gatk_gb300.pairhmm import Engine

    e = Engine()
    yield e
    e.close()


@pytest.mark.parametrize("n,rows,spread", [(1, 1, 1), (31, 160, 160), (32, 160, 1), (33, 160, 3), (5000, 160, 160),
                                           (100003, 160, 2), (70001, 2048, 2048), (64, 7, 7)])
def test_gather_and_fold(engine, n, rows, spread):
    import torch

    rng = np.random.default_rng(n)
    index = torch.from_numpy(rng.integers(-1, spread, n)).cuda()
    table = torch.from_numpy(rng.normal(size=(rows, 2))).cuda()
    g, c = torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    L, h = engine.L, engine.handle
    native.check(L.ghmm_calib_gather(h, table.data_ptr(), rows, index.data_ptr(), n, -4.5, -1.0, g.data_ptr(), c.data_ptr(),
                                     s), h)
    fixed = index < 0
    at = index.clamp(min=0)
    assert torch.equal(g, torch.where(fixed, torch.tensor(-4.5, dtype=torch.float64, device="cuda"), table[at, 0]).float())
    assert torch.equal(c, torch.where(fixed, torch.tensor(-1.0, dtype=torch.float64, device="cuda"), table[at, 1]).float())
    gg, gc = (torch.from_numpy(rng.normal(size=n).astype(np.float32)).cuda() for _ in range(2))
    out = torch.full((rows, 2), 7.0, dtype=torch.float64, device="cuda")
    native.check(L.ghmm_calib_fold(h, index.data_ptr(), n, gg.data_ptr(), gc.data_ptr(), rows, out.data_ptr(), s), h)
    keep = ~fixed
    for k, v in enumerate((gg, gc)):
        want = torch.zeros(rows, dtype=torch.float64, device="cuda").index_add_(0, at[keep], v[keep].double())
        size = torch.zeros(rows, dtype=torch.float64, device="cuda").index_add_(0, at[keep], v[keep].double().abs())
        assert bool(((out[:, k] - want).abs() <= 2 * n * 2.0 ** -53 * size).all())


def test_table_gradient_through_either_path(engine):
    """log10_likelihoods against position_params (torch operations) followed by the likelihood function: same values, and
    the same gradient but for the order of the FP32 atomics per position (one pair a read here, so none) and FP64 sums."""
    import torch

    from gatk_gb300 import workload

    cs = C.CalibrationSet(workload.generate(3, regions=20))
    for table in (C.default_theta(), C.default_theta().cuda(), C.default_theta().double().cuda()):
        a, b = (table.clone().requires_grad_(True) for _ in range(2))
        la = C.log10_likelihoods(a, cs, engine)
        lb = C._FN.apply(*cs.position_params(b), cs, engine, 0)
        assert torch.equal(la, lb)
        w = torch.linspace(0.5, 2.0, cs.n_pairs, dtype=torch.float64, device="cuda")
        (la * w).sum().backward()
        (lb * w).sum().backward()
        assert a.grad.dtype == table.dtype and a.grad.device == table.device
        assert torch.allclose(a.grad, b.grad, rtol=2e-7, atol=0)
    with pytest.raises(IndexError):
        C.log10_likelihoods(torch.zeros(1, 2), cs, engine)
