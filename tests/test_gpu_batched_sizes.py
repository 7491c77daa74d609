"""The batched Toeplitz passes at every transform length (64 .. 4096), odd and
even widths (a last row block that is not full), one to three slices: each
scan against its own mbir_solve, to the 1e-5 that the batched solver's other
tests use (the two take the same sums in another order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_every_length():
    import torch
    from tomocam_b200.plan import BatchScan, Plan, mbir_batched
    sizes = [(5, 2), (17, 1), (32, 3), (33, 2), (64, 1), (100, 3), (129, 1), (255, 2), (301, 1),
             (512, 1), (513, 1), (700, 3), (1023, 1), (1027, 2), (1500, 1)]
    scans, plans, starts = [], [], []
    for i, (n, S) in enumerate(sizes):
        ang = (np.arange(9 + i) * (np.pi / (9 + i))).astype(np.float32)
        pl = Plan(n, ang, pow2_toeplitz=True)
        g = torch.Generator("cuda").manual_seed(i)
        x = torch.rand((S, n, n), device="cuda", generator=g)
        aty = pl.toeplitz_grad(x)
        sq = 1.05 * float((x.double() * aty).sum())
        x0 = 0.8 * x
        plans.append(pl)
        starts.append((aty, sq, x0))
        scans.append(BatchScan(pl, aty, sq, x0.clone(), 50.0, 1.2, 0.5 + 0.1 * i))
    hist = mbir_batched(scans, 3)
    for pl, (aty, sq, x0), s, h in zip(plans, starts, scans, hist):
        ref, hr = pl.mbir_solve(aty, sq, x0, 3, s.sigma, s.p, s.prior_weight)
        assert np.array_equal(h[:, 2], hr[:, 2])
        assert float((s.x - ref).norm()) <= 1e-5 * float(ref.norm())
        pl.close()
