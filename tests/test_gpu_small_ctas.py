"""Small-CTA passes of lone trials and small batches: the same bits as the
large CTAs of a batch, at every size that has both, on both sides of the rule
that picks them."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alg", ["hio", "raar", "dm"])
@pytest.mark.parametrize("N,E,counts", [
    # counts: alone, the last count in small CTAs, the first in large ones
    # (148 SMs; items per trial x 4 small CTAs, at most 2 per SM, 1 at 512)
    (64, 32, (1, 148, 149)), (128, 32, (1, 37, 38)), (128, 16, (1, 18, 19)), (256, 16, (1, 4, 5)),
    (256, 8, (1, 2, 3)), (512, 32, (1, 2)), (512, 16, (1, 2))])
def test_small_ctas_match_large(N, E, counts, alg):
    from als_speckle_b200.engine import Engine, TrialSpec
    g = torch.Generator(device="cuda")
    g.manual_seed(N + E)
    M = 100 * torch.rand((N, N), generator=g, device="cuda")
    S = torch.zeros((N, N), device="cuda")
    S[N // 8:N // 2, N // 4:N // 2 + 3] = 1
    eng = Engine(use_graph=False, e_per_n={N: E})
    box = (N // 8, N // 4 + 1, 7, N // 4)

    def run(count):
        psi = torch.zeros((count, N, N), dtype=torch.complex64, device="cuda")
        save = torch.zeros((count,) + box[2:], dtype=torch.complex64, device="cuda")
        err = torch.zeros((count, 5, 2), dtype=torch.float64, device="cuda")
        eng.solve([TrialSpec(psi=psi[k], modulus=M, support=S, iterations=5, order=((alg, 4), ("er", 1)),
                             beta=0.9, random_phase=True, seed=3, trial=k, box=box, save=save[k],
                             errors=err[k]) for k in range(count)])
        torch.cuda.synchronize()
        return psi.cpu().numpy(), save.cpu().numpy(), err.cpu().numpy()

    runs = [run(c) for c in counts]
    large = runs[-1]
    for psi, save, err in runs[:-1]:
        for k in {0, len(psi) - 1}:
            if k >= len(large[0]):
                continue
            np.testing.assert_array_equal(psi[k], large[0][k])
            np.testing.assert_array_equal(save[k], large[1][k])
            # FP64 sums of the same FP32 partials, added in any order
            np.testing.assert_allclose(err[k], large[2][k], rtol=1e-12)
    eng.close()


@pytest.mark.parametrize("alg", ["hio", "dm"])
@pytest.mark.parametrize("N,E,counts", [
    # the other pairs that have both; small CTAs of a trial: (64, 8) and (64, 16)
    # 8 and 4, the other two 32; at (64, 32) above an item is two, not four
    (64, 8, (1, 37, 38)), (64, 16, (1, 74, 75)), (128, 8, (1, 9, 10)), (256, 32, (1, 9, 10))])
def test_small_ctas_match_large_for_every_e(N, E, counts, alg):
    test_small_ctas_match_large(N, E, counts, alg)
