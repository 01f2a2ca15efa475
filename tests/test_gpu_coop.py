"""Eight lanes per particle (csrc/pt_coop.cuh): small runs from the start, larger
ones from where their queue runs dry.  Every particle goes through the same
operations in the same order in both machines, so the exact build is the
oracle's bits at every size."""
import numpy as np
import pytest

from conftest import small_problem

pytestmark = pytest.mark.gpu

PER_SM = 80                       # particles per SM up to which a run starts on eight lanes


def _sizes(torch):
    few = PER_SM * torch.cuda.get_device_properties(0).multi_processor_count
    return {"one": 1, "odd": 33, "last_small": few, "first_handed": few + 1}


@pytest.mark.parametrize("size", ["one", "odd", "last_small", "first_handed"])
@pytest.mark.parametrize("method,with_j,near", [("rk5", False, False), ("dop853", True, False),
                                                ("dop853", False, False), ("rk5", True, True)])
def test_exact_bitwise_at_every_size(cuda, oracle_lib, method, with_j, near, size):
    torch = cuda
    import oracle
    from particles_gb300 import Fields
    npart = _sizes(torch)[size]
    prob = small_problem(method, n=12, npart=npart, periods=0.06, seed=71, with_j=with_j,
                         nsteps=3, gamma_range=(1.001, 50.0))
    uu, bb, jj = (*prob["fields"], None)[:3]
    eta = 1e-3 if with_j else 0.0
    so, co, sto = oracle.integrate(method, prob["params"], prob["time"], uu, bb, prob["state"].copy(),
                                   eta=eta, jj=jj, near=near)
    f = Fields(uu, bb, jj)
    t = lambda a: torch.tensor(a, device="cuda")
    s, c = t(prob["state"]), torch.zeros((npart, 3), dtype=torch.int64, device="cuda")
    st = torch.zeros(npart, dtype=torch.int32, device="cuda")
    carry = torch.zeros(128 * npart, dtype=torch.uint8, device="cuda")
    for stop in (0.4 * prob["time"][-1], 0.0):       # two windows: resumed particles too
        f.run_device(method, prob["params"], t(prob["time"]), s, c, st, carry, eta=eta, t_stop=stop,
                     interpolation="near" if near else "linear")
    assert f.run_check() == 0
    assert np.array_equal(st.cpu().numpy(), sto)
    assert np.array_equal(c.cpu().numpy(), co)
    assert np.array_equal(s.cpu().numpy().view(np.int64), so.view(np.int64))
