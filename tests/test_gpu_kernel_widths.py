"""The NUFFT kernels of every width, the narrow ones above all, against an
FP64 evaluation of the same approximation: the same ES kernel, fine grid and
correction factors on the host, so that the approximation's own error (0.1 and
0.01 at the widths 2 and 3) cancels and only the arithmetic is compared.

1e-5 relative L2, the operators' own bound: an FP32 kernel weight is good to
about 1e-6, the transforms to a few 1e-7.  The angles are random, so that no
point lies where a weight is a jump (a tap at exactly the kernel's edge); the
closest one is checked to be 1e-5 of a half width away, where the FP32 offset
(1e-7) moves the weight, exp(-beta) there, by less than 1e-3 of itself."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

P = 20


def _angles(n, w):
    return np.random.default_rng(100 * n + w).uniform(0.05, np.pi / 2 - 0.05, P).astype(np.float32) + \
        np.float32(np.pi / 2) * (np.arange(P, dtype=np.float32) % 2)


def _edge_distance(n, ang, nf, w):
    """Smallest distance of a tap to the kernel's edge, in half widths (the
    centre of the polar grid, exactly on a grid cell, apart)."""
    pts = np.stack(O.polar_grid(P, n, ang.astype(np.float64)))
    pts = np.delete(pts, n // 2, axis=2) * nf / (2 * np.pi)
    r = np.mod(pts - 0.5 * w, 1.0)
    return np.minimum(r, 1 - r).min() * 2 / w


def _plan(n, w, **kw):
    from tomocam_b200.plan import Plan
    ang = _angles(n, w)
    pl = Plan(n, ang, nufft_tol=10.0 ** (1 - w), psf=False, **kw)
    info = pl.info
    assert info["kernel_width"] == w and info["band_chunk"] > 0 and info["interp_tile"] > 0
    assert O.ESParams(10.0 ** (1 - w)).w == w
    assert _edge_distance(n, ang, info["nf"], w) > 1e-5
    return pl, ang, info["nf"]


def _close(out, ref):
    for s in range(len(ref)):
        assert np.linalg.norm(out[s] - ref[s]) <= 1e-5 * np.linalg.norm(ref[s])


# slices: one, two and four lines of two slices, eight lines, and a last odd slice
@pytest.mark.parametrize("w", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("n", [32, 33])
@pytest.mark.parametrize("S", [1, 4, 7, 16])
def test_paired(monkeypatch, n, w, S):
    _both(monkeypatch, n, w, S)


@pytest.mark.parametrize("w", [2, 3, 8])
@pytest.mark.parametrize("S", [1, 2, 5])
def test_unpaired(monkeypatch, w, S):
    _both(monkeypatch, 45, w, S, paired=False)


def _both(monkeypatch, n, w, S, **kw):
    import torch
    rng = np.random.default_rng(n + S)
    y = rng.standard_normal((S, P, n)).astype(np.float32)
    x = rng.standard_normal((S, n, n)).astype(np.float32)
    pl, ang, nf = _plan(n, w, **kw)
    with pl:
        back = pl.iradon(torch.from_numpy(y).cuda()).cpu().numpy()
        proj = pl.radon(torch.from_numpy(x).cuda()).cpu().numpy()
    monkeypatch.setattr(O, "es_fine_size", lambda _: nf)
    tol, ang = 10.0 ** (1 - w), ang.astype(np.float64)
    _close(back, O.backproject(y, ang, method="es", tol=tol))
    _close(proj, O.project(x, ang, method="es", tol=tol))
