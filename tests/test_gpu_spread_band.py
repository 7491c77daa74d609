"""Band spreading (type-1 pass 1): every lane shape (1 to 8 complex lines),
every kernel width, bands split over several chunks, against the oracle's
exact non-uniform DFT.

Tolerances: 1e-5 relative L2 at the default kernel (the operators' own);
10 tol + 1e-5 for a kernel of accuracy tol (the ES kernel of width
ceil(log10(1/tol)) + 1 is accurate to a small multiple of tol)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(n, P, S, tol=0.0, bound=1e-5, **kw):
    import torch
    from tomocam_b200.plan import Plan
    ang = (np.arange(P) * (np.pi / P)).astype(np.float32)
    y = np.random.default_rng(n + S).standard_normal((S, P, n)).astype(np.float32)
    ref = O.backproject(y, ang.astype(np.float64))
    with Plan(n, ang, nufft_tol=tol, psf=False, **kw) as pl:
        out = pl.iradon(torch.from_numpy(y).cuda()).cpu().numpy()
    for s in range(S):
        assert np.linalg.norm(out[s] - ref[s]) <= bound * np.linalg.norm(ref[s])


@pytest.mark.parametrize("n", [32, 45])
@pytest.mark.parametrize("S", [1, 2, 3, 4, 5, 6, 7, 9, 11, 14, 16])
def test_lines(n, S):
    _check(n, 24, S)


@pytest.mark.parametrize("S", [1, 2, 3, 5, 8])
def test_one_slice_per_line(S):
    _check(40, 24, S, paired=False)


@pytest.mark.parametrize("w", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("S", [1, 4, 8, 16])
def test_widths(w, S):
    tol = 10.0 ** (1 - w)
    _check(33, 20, S, tol=tol, bound=10 * tol + 1e-5)


@pytest.mark.parametrize("S", [1, 3, 6, 16])
def test_split_bands(S):
    # 700 rays cross the central bands: more points than one chunk takes
    _check(36, 700, S)
