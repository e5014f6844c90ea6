"""Which sizes of a mixed batch share a line of launches, read off the streams their
passes run on, and that every trial equals its size alone, bit for bit."""
import json

import pytest

pytestmark = pytest.mark.gpu


def _kernels(run, tmp_path):
    import torch
    run()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    path = str(tmp_path / "trace.json")
    prof.export_chrome_trace(path)
    with open(path) as f:
        return [e for e in json.load(f)["traceEvents"] if e.get("cat") == "kernel"]


def _specs(mix, ipsf=()):
    import torch
    from als_speckle_b200.engine import TrialSpec
    from als_speckle_b200.workloads import gaussian_ipsf
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    specs = []
    for N, count in mix:
        M = 30 * torch.rand((N, N), generator=g, device="cuda")
        S = torch.zeros((N, N), device="cuda")
        S[N // 8:N // 2, N // 4:N // 2 + 3] = 1
        ip = torch.from_numpy(gaussian_ipsf(N, 1.5)).cuda() if N in ipsf else None
        specs += [TrialSpec(psi=torch.zeros((N, N), dtype=torch.complex64, device="cuda"), modulus=M,
                            support=S, iterations=4, order=(("hio", 4),), beta=0.9, random_phase=True,
                            seed=6, trial=k, ipsf=ip) for k in range(count)]
    return specs


def _check(mix, lines, tmp_path, ipsf=(), **options):
    import torch
    from als_speckle_b200.engine import Engine
    eng = Engine(use_graph=False, e_per_n={128: 32, 256: 16, 512: 32, 1024: 32, 2048: 32}, **options)
    specs = _specs(mix, ipsf)
    kernels = _kernels(lambda: eng.solve(specs), tmp_path)
    mixed = [s.psi.clone() for s in specs]
    k = 0
    for _, count in mix:
        eng.solve(specs[k:k + count])
        k += count
    torch.cuda.synchronize()
    for a, s in zip(mixed, specs):
        assert torch.equal(torch.view_as_real(a), torch.view_as_real(s.psi))
    eng.close()
    if not kernels:
        pytest.skip("the profiler records no kernels here")
    streams = {}
    for e in kernels:
        for N, _ in mix:
            if "_pass" in e["name"] and "<%d," % N in e["name"]:
                streams.setdefault(e["args"]["stream"], set()).add(N)
    assert sorted(map(sorted, streams.values())) == sorted(map(sorted, lines))
    return kernels


@pytest.mark.parametrize("mix,ipsf,lines", [
    # 10 x 512^2 fill the SMs twice, 3 x 1024^2 and 38 x 256^2 as well
    (((512, 10), (1024, 3)), (1024,), [{512}, {1024}]),
    (((256, 38), (512, 10), (1024, 3), (2048, 1)), (512,), [{512}, {256, 1024, 2048}]),
    (((512, 10), (1024, 3), (2048, 1)), (512,), [{512}, {1024, 2048}])])
def test_partially_coherent_sizes_run_beside_the_line(mix, ipsf, lines, tmp_path):
    """In a line of their own, and without the shared memory that keeps other CTAs off
    their SMs when they are alone."""
    kernels = _check(mix, lines, tmp_path, ipsf)
    alone = _check([m for m in mix if m[0] in ipsf], [set(ipsf)], tmp_path, ipsf)
    for name in ("pc_cols_a", "pc_rows_w", "pc_cols_b"):
        shared = [{e["args"]["shared memory"] for e in ks if name in e["name"]} for ks in (kernels, alone)]
        assert len(shared[0]) == 1 and max(shared[0]) < 64 * 1024
        assert max(shared[0]) <= min(shared[1])


@pytest.mark.parametrize("mix", [((512, 10), (1024, 3)), ((256, 20), (512, 10), (1024, 3))])
def test_capped_sizes_run_side_by_side(mix, tmp_path):
    _check(mix, [{N} for N, _ in mix], tmp_path, ctas_per_sm=1)


@pytest.mark.parametrize("mix,lines", [
    (((256, 19), (512, 5)), [{256}, {512}]), (((256, 37), (1024, 3)), [{256}, {1024}]),
    (((512, 5), (1024, 2)), [{512, 1024}]), (((1024, 2), (2048, 1)), [{1024, 2048}]),
    (((256, 19), (512, 5), (1024, 2)), [{256, 512, 1024}]),
    (((128, 100), (256, 20), (512, 6)), [{128}, {256}, {512}]),
    (((128, 4), (512, 5), (1024, 2)), [{128}, {512, 1024}])])
def test_sizes_of_a_pair_share_a_line_when_they_fill_their_sms(mix, lines, tmp_path):
    _check(mix, lines, tmp_path)


@pytest.mark.parametrize("mix", [((128, 30), (512, 1)), ((256, 4), (1024, 2)), ((128, 8), (256, 2), (512, 1))])
def test_small_ctas_are_for_a_size_alone(mix, tmp_path):
    """Sizes side by side run in the large CTAs (of 128 or 256 threads); alone the small
    counts here run in 64-thread ones, with the same results."""
    for e in _check(mix, [{N} for N, _ in mix], tmp_path):
        if "_pass" in e["name"]:
            assert e["args"]["block"][0] > 64
    alone = _check(mix[:1], [{mix[0][0]}], tmp_path)
    assert {e["args"]["block"][0] for e in alone if "_pass" in e["name"]} == {64}
