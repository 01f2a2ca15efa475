"""What a launch may do besides launching, and which kernel the autotuner times."""
import pytest

from conftest import small_problem

pytestmark = pytest.mark.gpu


def _big(torch, seed):
    few = 80 * torch.cuda.get_device_properties(0).multi_processor_count
    return small_problem("dop853", n=12, npart=few + 1, periods=0.03, seed=seed, nsteps=3)


def _buffers(torch, prob):
    npart = prob["state"].shape[0]
    return dict(time=torch.tensor(prob["time"], device="cuda"), state=torch.tensor(prob["state"], device="cuda"),
                cnt=torch.zeros((npart, 3), dtype=torch.int64, device="cuda"))


def _run(f, prob, b, stream=0):
    f.run_device("dop853", prob["params"], b["time"], b["state"], b["cnt"], stream=stream)


@pytest.mark.parametrize("captured", ["another_stream", "its_own_stream"])
def test_first_large_run_of_a_handle_during_a_capture(cuda, captured):
    """A capture in the default (global) mode survives the first run of a handle
    that is large enough to hand particles over, whichever stream that run is on."""
    torch = cuda
    from particles_gb300 import Fields
    prob = _big(torch, 61)
    uu, bb = prob["fields"]
    ref = _buffers(torch, prob)
    _run(Fields(uu, bb), prob, ref)                       # loads the kernels; the results to compare with
    f, b = Fields(uu, bb), _buffers(torch, prob)
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    x = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        g.capture_begin(capture_error_mode="global")
        x.add_(1.0)
        _run(f, prob, b, side.cuda_stream if captured == "its_own_stream" else other.cuda_stream)
        g.capture_end()
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    assert f.run_check() == 0
    assert x.tolist() == [1.0] * 8
    assert torch.equal(b["cnt"], ref["cnt"])
    assert torch.equal(b["state"].view(torch.int64), ref["state"].view(torch.int64))


def test_autotune_times_the_variants_on_a_small_sample(cuda):
    """Variants are of the kernel with one lane per particle.  A sample that a run
    would give to the eight-lane kernel, at about a third of the time per attempt
    (170 and 52 us of a DOP853 attempt), is timed on the former all the same."""
    torch = cuda
    from particles_gb300 import Fields
    prob = small_problem("dop853", n=16, npart=1000, periods=0.5, seed=62)
    f, b = Fields(*prob["fields"]), _buffers(torch, prob)
    start = b["state"].clone()
    ms = []
    for _ in range(4):
        b["state"].copy_(start)
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        ev[0].record()
        f.run_device("dop853", prob["params"], b["time"], b["state"], b["cnt"], max_steps=32)
        ev[1].record()
        torch.cuda.synchronize()
        ms.append(ev[0].elapsed_time(ev[1]))
    _, tried = f.autotune("dop853", prob["params"], b["time"], start, max_steps=32)
    print(min(ms), tried)
    assert min(tried.values()) > 1.6 * min(ms[1:])


def test_a_small_ensemble_holds_no_hand_over_list(cuda):
    """An ensemble that fits the eight-lane machine from its first window on never
    hands particles over, so it does not pay for the list (5.8 MB, mapped and
    unmapped with every ensemble)."""
    torch = cuda
    from particles_gb300 import Ensemble, Fields
    prob = small_problem("rk5", n=12, npart=30, periods=0.05, seed=64, nsteps=2)
    f = Fields(*prob["fields"])
    z = lambda *shape, dtype: torch.zeros(shape, dtype=dtype, device="cuda")
    member = dict(_buffers(torch, prob), fields=f, params=prob["params"], status=z(30, dtype=torch.int32),
                  carry=z(128 * 30, dtype=torch.uint8))
    Ensemble("rk5", [member]).close()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    held = Ensemble("rk5", [member])
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] < 2 << 20
    held.run(0.0)
    assert held.check() == 0 and held.counts()[0].sum() == 0
    held.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_the_last_particles_of_a_queue_start_with_the_others(cuda, native, precision):
    """13,000 particles leave the last warp eight.  With the same number of attempts
    each, a run in which warps may hand over takes as long as one in which they
    may not (it took a third longer while that warp handed over at once)."""
    torch = cuda
    from particles_gb300 import Fields
    prob = small_problem("rk5", n=16, npart=13000, periods=1.0, seed=65)
    f, b = Fields(*prob["fields"], precision=precision), _buffers(torch, prob)
    ms = {}
    for cap in (0, -1):
        native.pt_debug_machines(0, cap)
        times = []
        for _ in range(6):
            b["state"].copy_(torch.tensor(prob["state"]))
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            ev[0].record()
            f.run_device("rk5", prob["params"], b["time"], b["state"], b["cnt"], max_steps=16)
            ev[1].record()
            torch.cuda.synchronize()
            times.append(ev[0].elapsed_time(ev[1]))
        ms[cap] = min(times[1:])
    native.pt_debug_machines(-1, -1)
    print(ms)
    assert (b["cnt"][:, 0] == 16).all()
    assert ms[-1] < 1.12 * ms[0]
