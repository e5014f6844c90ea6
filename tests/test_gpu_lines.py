"""Batches whose sizes fill the chip run in one line of overlapping launches,
the others beside it: every trial equals itself alone, bit for bit, whatever it
shares the call with, for different iteration counts and algorithms, eager, as
a graph, and with a partially coherent size in the line."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mix", [
    # (N, trials, iterations, algorithm), sizes in more than one round of SMs among them
    ((512, 10, 5, "hio"), (1024, 3, 7, "raar")),
    ((256, 40, 4, "dm"), (512, 9, 6, "hio"), (1024, 2, 3, "dm"), (2048, 1, 5, "er")),
    ((128, 2, 9, "hio"), (512, 1, 4, "raar"), (2048, 1, 3, "hio")),
    ((256, 38, 6, "er"), (512, 9, 4, "ipsf"), (1024, 2, 5, "hio")),
    # so many rounds that every size gets a line of its own
    ((256, 20, 4, "dm"), (1024, 40, 2, "hio"), (2048, 18, 3, "raar"))])
def test_mixed_lines_match_alone(mix):
    import torch
    from als_speckle_b200.engine import Engine, TrialSpec
    from als_speckle_b200.workloads import gaussian_ipsf
    g = torch.Generator(device="cuda")
    g.manual_seed(11)
    pat = {}
    for N, _, _, _ in mix:
        S = torch.zeros((N, N), device="cuda")
        S[N // 8:N // 2, N // 4:N // 2 + 3] = 1
        pat[N] = (30 * torch.rand((N, N), generator=g, device="cuda"), S)

    def specs(sel):
        out, k = [], 0
        for N, count, its, alg in mix:
            for _ in range(count):
                if sel is None or k in sel:
                    ip = torch.from_numpy(gaussian_ipsf(N, 1.5)).cuda() if alg == "ipsf" else None
                    out.append(TrialSpec(
                        psi=torch.zeros((N, N), dtype=torch.complex64, device="cuda"), modulus=pat[N][0],
                        support=pat[N][1], iterations=its, order=((alg if ip is None else "hio", its),),
                        beta=0.9, random_phase=True, seed=2, trial=k, ipsf=ip))
                k += 1
        return out, k

    _, total = specs(set())
    stream = torch.cuda.Stream()
    batches = []
    for use_graph in (False, True):
        eng = Engine(use_graph=use_graph)
        sp, _ = specs(None)
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            for _ in range(3):  # back to back: a round of launches right behind the last one's
                eng.solve(sp, stream=stream)
        stream.synchronize()
        batches.append([s.psi.cpu().numpy() for s in sp])
        eng.close()
    ends = np.cumsum([m[1] for m in mix])
    picks = sorted({0, total - 1} | {int(e) - 1 for e in ends} | {int(e) for e in ends[:-1]})
    eng = Engine(use_graph=False)
    for k in picks:
        sp, _ = specs({k})
        eng.solve(sp)
        torch.cuda.synchronize()
        alone = sp[0].psi.cpu().numpy()
        for b in batches:
            np.testing.assert_array_equal(b[k], alone)
    for a, b in zip(*batches):
        np.testing.assert_array_equal(a, b)
    eng.close()


@pytest.mark.parametrize("mix", [
    # several rounds of the SMs each, so that a size's pass starts early, on SMs
    # that read its planes a tick ago: 8-byte copies through L1 at every size but 512
    ((256, 40, 30, "hio"), (1024, 4, 30, "raar")),
    ((1024, 3, 24, "hio"), (2048, 1, 24, "hio")),
    ((256, 24, 24, "dm"), (512, 12, 24, "hio"), (1024, 3, 24, "er"))])
def test_early_passes_read_what_the_last_tick_wrote(mix):
    """Every trial of a long mixed batch, bit for bit, against its size alone
    (one size in a call never starts early)."""
    import torch
    from als_speckle_b200.engine import Engine, TrialSpec
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    specs = []
    for N, count, its, alg in mix:
        S = torch.zeros((N, N), device="cuda")
        S[N // 8:N // 2, N // 4:N // 2 + 3] = 1
        M = 30 * torch.rand((N, N), generator=g, device="cuda")
        for _ in range(count):
            specs.append(dict(modulus=M, support=S, iterations=its, order=((alg, its),), beta=0.9,
                              random_phase=True, seed=6, trial=len(specs)))

    def solve(eng, sel):
        sp = [TrialSpec(psi=torch.zeros(tuple(s["modulus"].shape), dtype=torch.complex64, device="cuda"), **s)
              for s in sel]
        for _ in range(2):
            eng.solve(sp)
        torch.cuda.synchronize()
        return [s.psi for s in sp]

    eng = Engine(use_graph=False)
    mixed = solve(eng, specs)
    alone, k = [], 0
    for _, count, _, _ in mix:
        alone += solve(eng, specs[k:k + count])
        k += count
    for k, (a, b) in enumerate(zip(mixed, alone)):
        assert torch.equal(torch.view_as_real(a), torch.view_as_real(b)), k
    eng.close()


def test_graphs_of_different_lines_are_kept_apart():
    """16 x 256^2 share the other sizes' line while they are less than a fifth of the
    work, and get their own once they run DM (twice the work): a batch of the same
    shape in the same workspace must not replay the other's graph."""
    import torch
    from als_speckle_b200 import _lib
    from als_speckle_b200.engine import Engine, TrialSpec
    mix = ((256, 16), (512, 9), (1024, 2))

    def specs(alg):
        out = []
        for N, count in mix:
            M = torch.ones((N, N), device="cuda")
            a = alg if N == 256 else "hio"
            out += [TrialSpec(psi=torch.zeros((N, N), dtype=torch.complex64, device="cuda"), modulus=M,
                              support=M, iterations=3, order=((a, 3),), beta=0.9, random_phase=True,
                              seed=2, trial=k) for k in range(count)]
        return out

    eng = Engine(use_graph=True)
    stream = torch.cuda.Stream()
    counts = [_lib.lib.sp_engine_graph_count()]
    for alg in ("dm", "hio", "dm", "raar"):  # DM first: its workspace is the larger one
        sp = specs(alg)
        stream.wait_stream(torch.cuda.current_stream())
        eng.solve(sp, stream=stream)
        stream.synchronize()
        counts.append(_lib.lib.sp_engine_graph_count())
    assert [c - counts[0] for c in counts] == [0, 1, 2, 2, 2]
    eng.close()
