"""The update's split of a volume into runs of slices: small images with many
slices (runs of 8, a short last run, one slice more than a run) against the
FP64 oracle's run2, with and without rejected attempts, odd widths (no
tensor copies) and even ones.  1e-4, the solver's tolerance."""
import math

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,S", [(24, 8), (24, 9), (25, 16), (32, 17), (33, 31), (70, 25)])
@pytest.mark.parametrize("reject", [False, True])
def test_runs(n, S, reject):
    import torch
    from tomocam_b200.plan import Plan
    P, iters = 12, 4
    ang = (np.arange(P) * (np.pi / P)).astype(np.float32)
    psf = O.psf_kernel(n, ang.astype(np.float64))
    rng = np.random.default_rng(n * S)
    x = rng.uniform(0.0, 1.0, (S, n, n))
    scale, weight, sigma = (1e-4, 1e-3, 1.0) if reject else (1.0, 1.0, 50.0)
    aty = (O.toeplitz_apply(x, psf) * scale).astype(np.float32)
    x0 = (0.8 * x * scale).astype(np.float32)
    sq = 1.01 * float(np.sum(x * scale * aty))
    step, _ = O.lipschitz_step(psf, n)
    step *= 2.5 if reject else 1.0

    def grad(v):
        return O.gradient2(v, aty, psf) + weight * O.qggmrf_grad(v, sigma, 1.2)

    def err(v):
        return math.sqrt(O.function_value2(v, aty, psf, sq))

    rec = O.Run2Record()
    ref = O.run2(x0, iters, step, grad, err, rec)
    with Plan(n, ang) as pl:
        out, hist = pl.mbir_solve(torch.from_numpy(aty).cuda(), sq, torch.from_numpy(x0).cuda(), iters,
                                  sigma, 1.2, weight, step=step)
        out = out.cpu().numpy()
    assert int(hist[:, 2].sum()) == rec.attempts
    assert np.linalg.norm(out - ref) <= 1e-4 * np.linalg.norm(ref)
