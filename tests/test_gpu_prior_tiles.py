"""The standalone prior kernels (gradient, Hessian-vector product) where their
32 x 8 tiles, their runs of slices and the clamp can go wrong, against the
FP64 oracle: single voxels, rows and columns, one voxel past a tile, one
slice, and more slices than one run takes.

Tolerance 1e-5 relative L2: each edge is good to a few 1e-7, and a sum of 26
random edges loses at most about an order to cancellation; the two dot
products are held to 1e-5 of the sum of their terms' magnitudes (bounded by
|v| |grad| in the 2-norm)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 40), (3, 19, 1), (1, 8, 32), (1, 9, 33), (2, 7, 31),
                                   (4, 16, 64), (5, 17, 65), (37, 10, 34), (700, 3, 5)])
@pytest.mark.parametrize("sigma,p", [(0.7, 1.2), (5.0, 1.6)])
def test_gradient_and_hvp(shape, sigma, p):
    import torch
    from tomocam_b200.plan import qggmrf_grad, qggmrf_hvp
    rng = np.random.default_rng(sum(shape))
    x, v, g0 = (rng.standard_normal(shape).astype(np.float32) for _ in range(3))
    xt, vt = torch.from_numpy(x).cuda(), torch.from_numpy(v).cuda()
    ref = O.qggmrf_grad(x, sigma, p)
    g = qggmrf_grad(xt, torch.from_numpy(g0).cuda(), sigma, p, 0.5).cpu().numpy()
    assert np.linalg.norm(g - (g0 + 0.5 * ref)) <= 1e-5 * np.linalg.norm(np.abs(g0) + np.abs(0.5 * ref))
    hr, ar, br = O.qggmrf_hvp(x, v, sigma, p, 0.5)
    hv, a, b = qggmrf_hvp(xt, vt, sigma, p, 0.5)
    assert np.linalg.norm(hv.cpu().numpy() - hr) <= 1e-5 * np.linalg.norm(hr)
    bound = 1e-5 * np.linalg.norm(v) * np.linalg.norm(ref)
    assert abs(a - ar) <= bound
    # |d grad / d sigma| <= (2 - p + 1) |grad| / sigma per edge, of either sign
    assert abs(b - br) <= 10 * bound / sigma + 1e-5 * abs(br)
