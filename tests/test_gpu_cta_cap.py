"""sp_run_opts.ctas_per_sm, read off the launched grids: it caps CTAs of the large
kind, and calls that run in 64-thread CTAs keep as many threads as before them."""
import json

import pytest

pytestmark = pytest.mark.gpu


def _passes(eng, specs, tmp_path):
    """(grid, block) of every pass kernel of one solve."""
    import torch
    eng.solve(specs)
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        eng.solve(specs)
        torch.cuda.synchronize()
    path = str(tmp_path / "trace.json")
    prof.export_chrome_trace(path)
    with open(path) as f:
        events = json.load(f)["traceEvents"]
    return [(e["args"]["grid"][0], e["args"]["block"][0]) for e in events
            if e.get("cat") == "kernel" and "_pass" in e["name"]]


@pytest.mark.parametrize("N,count,cap", [(256, 1, 1), (256, 4, 1), (256, 4, 2), (128, 30, 1), (256, 40, 1),
                                         (1024, 2, 1)])
def test_cap_counts_large_ctas(N, count, cap, tmp_path):
    import torch
    from als_speckle_b200.engine import Engine, TrialSpec
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    M = torch.ones((N, N), device="cuda")
    specs = [TrialSpec(psi=torch.zeros((N, N), dtype=torch.complex64, device="cuda"), modulus=M, support=M,
                       iterations=2, order=(("hio", 2),), beta=0.9, random_phase=True, seed=1, trial=k)
             for k in range(count)]
    free, capped = Engine(use_graph=False), Engine(use_graph=False, ctas_per_sm=cap)
    a, b = _passes(free, specs, tmp_path), _passes(capped, specs, tmp_path)
    if not a:
        pytest.skip("the profiler records no kernels here")
    assert len(a) == len(b)
    for (grid, block), (grid_c, block_c) in zip(a, b):
        assert block == block_c
        assert grid_c == min(grid, cap * sms * (256 // block if block == 64 else 1))
    free.close()
    capped.close()
