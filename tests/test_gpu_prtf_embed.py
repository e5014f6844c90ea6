"""PRTF phasor sums of embedded frames (rows and columns fewer than N, chunks
of frames) at every transform size, against FP64 numpy.

Bound: a phasor's error is the transform's error over |F|.  The transform of
white noise is good to ~3e-7 of its rms (the FFT's own bound here is 2e-6
relative norm); |F|^2 is exponentially distributed, so the least of P pixels
times F frames is ~rms/sqrt(P F) >= rms/1500 at these sizes, and one frame's
phasor weighs 1/F: 2e-6 * 1500 / F per pixel at worst."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,frames,rows,cols", [
    (8, 3, 8, 8), (8, 5, 3, 7), (16, 4, 9, 16), (32, 7, 32, 5), (64, 33, 17, 40), (128, 20, 101, 67),
    (256, 9, 180, 181), (512, 5, 512, 1), (512, 13, 173, 400), (1024, 2, 33, 1000), (2048, 2, 70, 51),
    (4096, 1, 33, 65)])
def test_prtf_of_embedded_frames(N, frames, rows, cols):
    import torch
    from als_speckle_b200.phasing import prtf
    from als_speckle_b200._lib import call, ptr, stream_ptr
    rng = np.random.default_rng(N + frames)
    x = (rng.standard_normal((frames, rows, cols)) + 1j * rng.standard_normal((frames, rows, cols)))
    x = x.astype(np.complex64)
    acc = np.zeros((N, N), np.complex128)
    for f in x:
        F = np.fft.fft2(f.astype(np.complex128), s=(N, N))
        acc += F / np.abs(F)
    t = torch.from_numpy(x).cuda()
    tol = 2e-6 * 1500 / frames
    got = prtf(t, N=N).cpu().numpy()
    assert np.max(np.abs(got - np.fft.fftshift(np.abs(acc) / frames))) < tol
    # the two halves: phasor sums added to what acc holds, in its own layout
    out = torch.full((N, N), 1.5 - 0.5j, dtype=torch.complex64, device="cuda")
    work = torch.empty((frames, N, N), dtype=torch.complex64, device="cuda")
    call("sp_prtf_phasors", ptr(t), frames, rows, cols, N, ptr(work), ptr(out), stream_ptr())
    assert np.max(np.abs(out.cpu().numpy() - (acc + 1.5 - 0.5j))) < tol * frames


@pytest.mark.parametrize("N,frames,rows,cols", [
    (8, 3, 8, 8), (16, 4, 9, 16), (64, 33, 17, 40), (256, 9, 180, 181), (512, 13, 173, 400),
    (1024, 2, 33, 1000), (4096, 1, 33, 65)])
def test_rftf_of_embedded_frames(N, frames, rows, cols):
    """gpu_rftf without an ipsf against FP64 numpy.  A summand's slope in |F|
    is at most 0.385/g; with g >= 0.2 rms and a pixel's transform good to 1e-5
    of the rms (2e-6 in norm) it is good to 2e-5.  Where g = 0 it is 0."""
    import torch
    from als_speckle_b200.phasing import gpu_rftf
    rng = np.random.default_rng(N + frames)
    x = (rng.standard_normal((frames, rows, cols)) + 1j * rng.standard_normal((frames, rows, cols)))
    x = x.astype(np.complex64)
    rms = np.sqrt(2.0 * rows * cols)
    g = ((0.2 + 2 * rng.random((N, N))) * rms).astype(np.float32)
    g[N // 3, N // 5] = 0
    want = np.zeros((N, N))
    with np.errstate(divide="ignore"):
        for f in x:
            F = np.abs(np.fft.fft2(f.astype(np.complex128), s=(N, N)))
            want += 1 / np.sqrt(1 + (g.astype(np.float64) - F) ** 2 / g.astype(np.float64) ** 2)
    got = gpu_rftf(None, torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda()).cpu().numpy()
    assert np.max(np.abs(got - np.fft.fftshift(want / frames))) < 2e-5


def test_rftf_of_extreme_magnitudes():
    """Transforms whose squares leave the float range count as the summand's
    limits: 0 where |F|^2 overflows, g-only where |F| = 0."""
    import torch
    from als_speckle_b200.phasing import gpu_rftf
    x = np.zeros((2, 4, 4), np.complex64)
    x[0, 0, 0] = 3e19  # |F|^2 = inf everywhere
    g = np.ones((16, 16), np.float32)
    got = gpu_rftf(None, torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda()).cpu().numpy()
    # frame 1: F = 0, summand 1/sqrt(2)
    assert np.allclose(got, 0.5 / np.sqrt(2.0), rtol=1e-6)


@pytest.mark.parametrize("N", [32, 1024])
@pytest.mark.parametrize("goal", [9e18, 9.3e18, 1e19, 1.8e19])
def test_rftf_of_large_goals(goal, N):
    """Goals whose square's reciprocal lies below the float range (from 9.2e18 on)
    beside ordinary ones, F the same everywhere (a frame that is one point).  A
    summand is a few roundings: 1e-6."""
    import torch
    from als_speckle_b200.phasing import gpu_rftf
    x = np.zeros((3, 4, 4), np.complex64)
    x[:, 0, 0] = [4e18, 1e18, 1.2e19]
    g = np.full((N, N), goal, np.float32)
    g[::3, ::2] = 3e18
    g[5, 7] = 0
    got = gpu_rftf(None, torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda()).cpu().numpy()
    with np.errstate(divide="ignore"):
        want = np.mean([1 / np.sqrt(1 + (g.astype(np.float64) - f) ** 2 / g.astype(np.float64) ** 2)
                        for f in np.abs(x[:, 0, 0]).astype(np.float64)], axis=0)
    np.testing.assert_allclose(np.fft.ifftshift(got), want, rtol=1e-6, atol=1e-7)


@pytest.mark.parametrize("N,frames", [(32, 600), (64, 900), (256, 300)])
def test_mean_of_many_frames(N, frames):
    """Frames that are one point, whose transforms are the same everywhere: the
    RFTF's summand is 1/sqrt(2), the PRTF's phasor a quarter turn's.  A summand is
    good to 1.5 units of its last place and the means of equal ones, added up in
    FP64 but for runs of a few, to little more: 4e-7 relative."""
    import torch
    from als_speckle_b200.phasing import gpu_rftf, prtf
    x = torch.zeros((frames, 3, 2), dtype=torch.complex64, device="cuda")
    x[:, 0, 0] = 1.2 + 1.6j
    g = torch.ones((N, N), device="cuda")
    got = gpu_rftf(None, x, g).cpu().numpy()
    np.testing.assert_allclose(got, np.full((N, N), 1 / np.sqrt(2.0)), rtol=4e-7)
    np.testing.assert_allclose(prtf(x, N=N).cpu().numpy(), np.ones((N, N)), rtol=4e-7)


@pytest.mark.parametrize("N,rows,cols", [(8, 5, 8), (64, 40, 33), (512, 180, 181), (2048, 300, 77), (4096, 300, 321)])
def test_phasors_of_the_standalone_transform(N, rows, cols):
    """One frame's phasors are those of sp_fft2's transform of the embedded frame,
    to the phasor's own few roundings (3e-7): the transforms are the same bits, where
    another order of operations would show wherever F is small."""
    import torch
    from als_speckle_b200._lib import call, ptr, stream_ptr
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    x = torch.view_as_complex(torch.randn((rows, cols, 2), generator=g, device="cuda"))
    F = torch.zeros((N, N), dtype=torch.complex64, device="cuda")
    F[:rows, :cols] = x
    call("sp_fft2", ptr(F), ptr(F), N, 1, 0, stream_ptr())
    got = torch.zeros((N, N), dtype=torch.complex64, device="cuda")
    work = torch.empty((1, N, N), dtype=torch.complex64, device="cuda")
    call("sp_prtf_phasors", ptr(x), 1, rows, cols, N, ptr(work), ptr(got), stream_ptr())
    F = F.to(torch.complex128)
    assert (got.to(torch.complex128) - F / F.abs()).abs().max().item() < 3e-7
