"""sp_engine_run_static on several sizes: sizes of more than one round of the SMs
share a line of overlapping launches, the others follow one another on the
caller's stream (interleaved they were up to 17% slower than one after another).
Every trial equals its size alone, bit for bit, and the kernels launched are those
of the rule."""
import ctypes as C
import json

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mix,line", [
    # (N, trials, iterations); the sizes in the shared line on 148 SMs at the tuned E
    (((256, 16, 6), (512, 4, 6)), ()),
    (((512, 4, 5), (1024, 1, 8)), ()),
    (((256, 30, 4), (512, 5, 7)), (256, 512)),
    (((64, 40, 4), (256, 20, 6), (512, 6, 3), (1024, 1, 5)), (256, 512))])
def test_static_batches_of_several_sizes(mix, line, tmp_path):
    import torch
    from als_speckle_b200 import _lib
    from als_speckle_b200.engine import Engine, TrialSpec, _to_struct
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    specs = []
    for N, count, its in mix:
        M = 30 * torch.rand((N, N), generator=g, device="cuda")
        S = torch.zeros((N, N), device="cuda")
        S[N // 8:N // 2, N // 4:N // 2 + 3] = 1
        specs += [dict(modulus=M, support=S, iterations=its, order=(("hio", its),), beta=0.9,
                       random_phase=True, seed=6, trial=len(specs) + k) for k in range(count)]
    eng = Engine(use_graph=False, e_per_n={64: 32, 256: 16, 512: 32, 1024: 32})
    opts = eng.opts()

    def run(sel):
        sp = [TrialSpec(psi=torch.zeros(tuple(s["modulus"].shape), dtype=torch.complex64, device="cuda"), **s)
              for s in sel]
        arr = (_lib.sp_trial * len(sp))(*[_to_struct(t) for t in sp])
        _lib.call("sp_engine_run_static", arr, len(sp), C.byref(opts), _lib.stream_ptr())
        torch.cuda.synchronize()
        return [t.psi for t in sp]

    mixed, alone, k = run(specs), [], 0
    for _, count, _ in mix:
        alone += run(specs[k:k + count])
        k += count
    for a, b in zip(mixed, alone):
        assert torch.equal(torch.view_as_real(a), torch.view_as_real(b))
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        run(specs)
    path = str(tmp_path / "trace.json")
    prof.export_chrome_trace(path)
    with open(path) as f:
        names = {e["name"] for e in json.load(f)["traceEvents"] if e.get("cat") == "kernel"}
    if not names:
        pytest.skip("the profiler records no kernels here")
    shared = {N for N, _, _ in mix if any("_pass" in n and "<%d," % N in n and "true>" in n for n in names)}
    assert shared == set(line)
    eng.close()
