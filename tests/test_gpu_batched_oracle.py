"""The batched solver at every transform length (64 .. 4096) against the FP64
oracle's run2: odd and even widths, one to three slices, a last row block and
a last slice pair that are not full, scans with rejected attempts beside scans
without.  1e-4, the solver's tolerance; the point-spread functions are the
plans' own (FP64, held to the oracle elsewhere)."""
import math

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [(5, 2), (31, 3), (32, 1), (33, 2), (64, 1), (100, 3), (129, 1), (255, 2), (301, 1), (512, 1),
         (700, 2), (1027, 1)]


def test_against_run2():
    import torch
    from tomocam_b200.plan import BatchScan, Plan, mbir_batched
    iters, scans, plans, refs = 3, [], [], []
    for i, (n, S) in enumerate(SIZES):
        P, reject = 9 + i, i % 3 == 2
        pl = Plan(n, (np.arange(P) * (np.pi / P)).astype(np.float32), pow2_toeplitz=True)
        H = O.ToeplitzCache(pl.psf())
        x = np.random.default_rng(i).uniform(0.0, 1.0, (S, n, n))
        scale, weight, sigma = (1e-4, 1e-3, 1.0) if reject else (1.0, 1.0, 50.0)
        aty = (O.toeplitz_apply(x, H.spec) * scale).astype(np.float32)
        x0 = (0.8 * x * scale).astype(np.float32)
        sq = 1.01 * float(np.sum(x * scale * aty))
        step = O.lipschitz_step(H.spec, n)[0] * (2.5 if reject else 1.0)

        def grad(v):
            return H.gradient2(v, aty) + weight * O.qggmrf_grad(v, sigma, 1.2)

        def err(v):
            return math.sqrt(H.function_value2(v, aty, sq))

        rec = O.Run2Record()
        refs.append((O.run2(x0, iters, step, grad, err, rec), rec.attempts))
        plans.append(pl)
        scans.append(BatchScan(pl, torch.from_numpy(aty).cuda(), sq, torch.from_numpy(x0).cuda(), sigma, 1.2,
                               weight, step=step))
    hist = mbir_batched(scans, iters)
    for (n, S), pl, s, h, (ref, attempts) in zip(SIZES, plans, scans, hist, refs):
        assert int(h[:, 2].sum()) == attempts, (n, S)
        assert np.linalg.norm(s.x.cpu().numpy() - ref) <= 1e-4 * np.linalg.norm(ref), (n, S)
        pl.close()
    assert max(a for _, a in refs) > iters and min(a for _, a in refs) == iters
