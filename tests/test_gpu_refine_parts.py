"""refine_support with the parts found on the device, against the host's
label_parts and FP64 numpy: shapes around the kernels' tiles (32 x 32 pixels,
64 taps, warps of 32 columns, fewer than 3 rows or columns) and masks whose
parts wrap round, nest, fill whole rows or consist of single pixels.  The blur
is the same FP64 sum in another order (1e-12 relative); a pixel could only
change sides of a threshold if it lay within that of it."""
import numpy as np
import pytest

from als_speckle_b200 import masking

pytestmark = pytest.mark.gpu


def _mask(kind, R, C, rng):
    r, c = np.indices((R, C))
    if kind == "empty":
        return np.zeros((R, C), bool)
    if kind == "full":
        return np.ones((R, C), bool)
    if kind == "rows":  # full rows, joined round the edge
        return r % 3 != 1
    if kind == "cols":
        return c % 4 < 2
    if kind == "singles":
        return (r % 2 == 0) & (c % 2 == 0)
    if kind == "spiral":
        d = np.maximum(abs(r - R // 2), abs(c - C // 2))
        m = d % 2 == 0
        m[R // 2, :C // 2] = True
        return m
    return rng.random((R, C)) < {"sparse": 0.15, "percolating": 0.41, "dense": 0.75}[kind]


def _want(sup, avg, blur, lt, gt, kill):
    mag = np.abs(avg).astype(np.float64)
    ks = []
    for n in mag.shape:
        g = np.fft.fftshift(np.exp(-(np.arange(n) - n // 2) ** 2 / (2 * blur ** 2)))
        ks.append(g / g.sum())
    b = np.zeros_like(mag)
    for i, k in enumerate(ks[1]):
        b += k * np.roll(mag, i, 1)
    b2 = np.zeros_like(mag)
    for i, k in enumerate(ks[0]):
        b2 += k * np.roll(b, i, 0)
    lab, n = masking.label_parts(sup)
    out = np.zeros(mag.shape)
    sums = [mag[lab == k].sum() for k in range(1, n + 1)]
    drop = int(np.argmin(sums)) + 1 if kill and n else -1
    for k in range(1, n + 1):
        if k != drop:
            part = b2 * (lab == k)
            out += (part > max(part.max(), 0.0) * lt)
    return out * (b2 > b2.max() * gt), b2


@pytest.mark.parametrize("kind", ["empty", "full", "rows", "cols", "singles", "spiral", "sparse",
                                  "percolating", "dense"])
@pytest.mark.parametrize("R,C", [(1, 40), (40, 1), (2, 33), (33, 2), (3, 3), (8, 32), (31, 65), (64, 64),
                                 (97, 130), (340, 341)])
def test_refine_support_parts(kind, R, C):
    import torch
    from als_speckle_b200.phasing import refine_support
    rng = np.random.default_rng(R * 1000 + C)
    sup = _mask(kind, R, C, rng).astype(np.float32)
    avg = (rng.random((R, C)) * np.exp(1j * rng.random((R, C)))).astype(np.complex64)
    for kill in (False, True):
        got, blurred = refine_support(sup, torch.from_numpy(avg).cuda(), blur=0.8, local_threshold=0.7,
                                      global_threshold=0.3, kill_weakest=kill)
        want, b = _want(sup, avg, 0.8, 0.7, 0.3, kill)
        assert np.allclose(blurred, b, rtol=1e-6, atol=0)  # |avg| is FP32 there
        # parts, thresholds and the dropped part; values of the two blurs differ
        # by FP32 rounding of |avg|, so pixels within 1e-6 of a threshold may differ
        diff = np.argwhere(got != want)
        lab = masking.label_parts(sup)[0]
        for r, c in diff:
            p = b[lab == lab[r, c]].max() * 0.7 if lab[r, c] else np.inf
            assert min(abs(b[r, c] - p) / p, abs(b[r, c] - b.max() * 0.3) / b.max()) < 1e-6
        assert len(diff) <= 2


@pytest.mark.parametrize("shape", [(530000, 2), (2, 530000)])  # more tiles than a grid has in y
def test_refine_support_of_long_thin_maps(shape):
    """A constant map stays constant under the blur, so every pixel of the support is
    above its thresholds and the support comes back, hole and all."""
    import torch
    from als_speckle_b200.phasing import refine_support
    sup = np.ones(shape, np.float32)
    sup.ravel()[1000:2000] = 0
    avg = torch.full(shape, 2j, dtype=torch.complex64, device="cuda")
    got, blurred = refine_support(sup, avg, blur=1.0, local_threshold=0.5)
    assert np.allclose(blurred, 2.0, rtol=1e-12)
    np.testing.assert_array_equal(got, sup)


@pytest.mark.parametrize("kind", ["empty", "full", "rows", "singles", "spiral", "sparse", "percolating"])
@pytest.mark.parametrize("R,C", [(33, 2), (97, 130), (340, 341)])
def test_parts_from_the_host_match(kind, R, C, monkeypatch):
    """The route of supports too large for the device's 32-bit pixel numbers (parts
    labelled by the caller, sp_shrinkwrap) on small ones: the same blur bit for bit,
    the same support."""
    import torch
    from als_speckle_b200 import phasing
    rng = np.random.default_rng(R + C)
    sup = _mask(kind, R, C, rng).astype(np.float64)
    avg = torch.from_numpy((rng.random((R, C)) * 1j).astype(np.complex64)).cuda()
    for kill in (False, True):
        args = dict(blur=0.8, local_threshold=0.7, global_threshold=0.3, kill_weakest=kill)
        got, blurred = phasing.refine_support(sup, avg, **args)
        with monkeypatch.context() as m:
            m.setattr(phasing, "_HOST_PARTS", 1)
            host, b = phasing.refine_support(sup, avg, **args)
        np.testing.assert_array_equal(b, blurred)
        np.testing.assert_array_equal(host, got)


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int64])
def test_results_hold_no_more_than_themselves(dtype):
    """The refined support and the blurred map do not share memory: a program that
    keeps a support for every round keeps 4 bytes a pixel of it."""
    import torch
    from als_speckle_b200.phasing import refine_support
    n = 64
    got = refine_support(np.ones((n, n), dtype), torch.ones((n, n), dtype=torch.complex64, device="cuda"))
    for a in got:
        root = a
        while isinstance(root.base, np.ndarray):
            root = root.base
        held = root.base.untyped_storage().nbytes() if isinstance(root.base, torch.Tensor) else root.nbytes
        assert held == a.nbytes
    assert not np.shares_memory(*got)
