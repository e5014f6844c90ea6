"""Partially coherent batches of every grid shape (one CTA per SM to several
rounds) equal their trials run alone, bit for bit: the launches overlap
programmatically, and a kernel that read a plane too early would differ."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["ipsf", "spectrum", "both"])
@pytest.mark.parametrize("N,counts", [(32, (3,)), (64, (2, 40)), (256, (3, 10, 37)), (512, (2, 5, 11)),
                                      (1024, (2,))])
@pytest.mark.parametrize("alg", ["hio", "dm"])
def test_batches_match_alone(N, counts, mode, alg):
    import torch
    from als_speckle_b200.engine import Engine, TrialSpec
    from als_speckle_b200.workloads import gaussian_ipsf
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    S = torch.zeros((N, N), device="cuda")
    S[N // 8:N // 2, N // 4:N // 2 + 3] = 1
    ipsf = torch.from_numpy(gaussian_ipsf(N, 1.5)).cuda() if mode != "spectrum" else None
    e = np.linspace(0.9, 1.12, 19)  # rows skipped and repeated, more than one table fill
    spec = None
    if mode != "ipsf":
        spec = (torch.from_numpy(e.astype(np.float32)).cuda(),
                torch.from_numpy(np.exp(-(e - 1) ** 2 * 50).astype(np.float32)).cuda())
    Ms = [20 * torch.rand((N, N), generator=g, device="cuda") for _ in range(2)]
    eng = Engine(use_graph=False)

    def run(trials):
        psi = torch.zeros((len(trials), N, N), dtype=torch.complex64, device="cuda")
        eng.solve([TrialSpec(psi=psi[i], modulus=Ms[k % 2], support=S, iterations=4, order=((alg, 9),),
                             beta=0.9, random_phase=True, seed=5, trial=k, ipsf=ipsf, spectrum=spec)
                   for i, k in enumerate(trials)])
        return psi.cpu().numpy()

    alone = {k: run([k])[0] for k in (0, 1, counts[-1] - 1)}
    for c in counts:
        batch = run(list(range(c)))
        for k in alone:
            if k < c:
                np.testing.assert_array_equal(batch[k], alone[k])
    eng.close()


@pytest.mark.parametrize("mode", ["ipsf", "both"])
@pytest.mark.parametrize("N,counts", [(64, (75, 149)), (128, (19, 38)), (256, (6, 19))])
def test_batches_match_alone_at_small_n(N, counts, mode):
    """Counts of one to a few CTAs per SM at the sizes whose row kernel is compiled
    for two CTAs on an SM."""
    test_batches_match_alone(N, counts, mode, "hio")
