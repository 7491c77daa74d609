"""An autotuned plan holds only lists that its operators read: where the bands
spread every type-1 transform no tile lists are built or timed, and where they
cannot (kernel widths above 8) the tile choice is still measured."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plans(n, P, **kw):
    from tomocam_b200.plan import Plan
    ang = (np.arange(P) * (np.pi / P)).astype(np.float32)
    return Plan(n, ang, psf=False, **kw), Plan(n, ang, psf=False, autotune=True, **kw)


@pytest.mark.parametrize("n,P", [(64, 90), (200, 150)])
@pytest.mark.parametrize("paired", [True, False])
def test_bands_without_tile_lists(n, P, paired):
    """Tile lists are at least one 4-byte index per point.  The autotuned
    plan's other choices (a band list in chunks of 128 points: 16 bytes for
    every 128 of at most 4 entries per point; interpolation tiles) stay below."""
    a, b = _plans(n, P, paired=paired)
    with a, b:
        assert a.info["band_chunk"] > 0 and b.info["band_chunk"] > 0
        assert b.info["table_bytes"] - a.info["table_bytes"] < 4 * P * n


def test_wide_kernel_keeps_the_tile_choice():
    import torch
    n, P = 64, 90
    a, b = _plans(n, P, nufft_tol=1e-9)
    with a, b:
        assert a.info["band_chunk"] == 0 and b.info["band_chunk"] == 0
        assert b.info["table_bytes"] >= 4 * P * n
        assert b.info["spread_tile"] in (16, 32, 64)
        y = torch.randn((3, P, n), device="cuda", generator=torch.Generator("cuda").manual_seed(1))
        ra, rb = a.iradon(y), b.iradon(y)
        # same points and weights, another order of the atomic adds
        assert float((ra - rb).norm()) <= 1e-5 * float(ra.norm())
