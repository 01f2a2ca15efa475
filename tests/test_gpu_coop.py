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


@pytest.mark.parametrize("method,tol", [("rk5", 1e-8), ("dop853", 1e-8)])
@pytest.mark.parametrize("prec,kw", [("fp64_fma", {}), ("fp64_fma", dict(face_steps=True)), ("fp32", {}),
                                     ("fp32", dict(face_steps=True, noise_floor=True)),
                                     ("bf16", dict(noise_floor=True)),
                                     ("fp64", dict(learned=True)), ("fp64_fma", dict(learned=True)),
                                     ("fp32", dict(learned=True, face_steps=True))])
@pytest.mark.parametrize("with_j", [False, True])
def test_both_machines_give_the_same_bits(cuda, method, tol, prec, kw, with_j):
    """A particle's result does not depend on how many others run with it: a
    few of them alone (eight lanes throughout) against the same ones in a run
    that starts on one lane each and hands over."""
    torch = cuda
    from particles_gb300 import Fields, learned
    few = 333
    kw = dict(kw)
    if kw.pop("learned", False):
        norm = np.concatenate([np.zeros(9), np.full(9, 3.0), [-8.0, 1.0]]).astype(np.float32)
        kw["model"] = learned.Model(learned.init_params(5), norm, safety=0.9)
    npart = 3 * PER_SM * torch.cuda.get_device_properties(0).multi_processor_count + 17
    prob = small_problem(method, n=20, npart=npart, periods=0.1, seed=72, with_j=with_j, nsteps=7,
                         gamma_range=(1.001, 50.0), tol=tol)
    t = lambda a: torch.tensor(a, device="cuda")
    f = Fields(*prob["fields"], precision=prec)
    out = []
    for n in (npart, few):
        s, c = t(prob["state"][:n]), torch.zeros((n, 3), dtype=torch.int64, device="cuda")
        st = torch.zeros(n, dtype=torch.int32, device="cuda")
        f.run_device(method, prob["params"], t(prob["time"]), s, c, st, eta=1e-3 if with_j else 0.0, **kw)
        assert f.run_check() == 0
        out.append((s[:few].cpu(), c[:few].cpu(), st[:few].cpu()))
    for a, b in zip(*out):
        assert torch.equal(a.view(torch.int64) if a.is_floating_point() else a,
                           b.view(torch.int64) if b.is_floating_point() else b)
    # finished, with output rows (the last one's time may round past tmax)
    assert (out[0][2] == 0).all() and (out[0][0][:, -2, 6] > 1.0).all()


def test_ensemble_of_few_and_many(cuda, oracle_lib):
    """An ensemble's windows go to one machine or the other by the particles
    that are left; the members' bits stay the oracle's."""
    torch = cuda
    import oracle
    from particles_gb300 import Ensemble, Fields
    few = PER_SM * torch.cuda.get_device_properties(0).multi_processor_count
    z = lambda shape, dt: torch.zeros(shape, dtype=dt, device="cuda")
    for counts in ((40, 7), (few, 50)):
        probs = [small_problem("dop853", n=12, npart=n, periods=0.05, seed=80 + k, nsteps=3,
                               gamma_range=(1.001, 50.0)) for k, n in enumerate(counts)]
        mem = [dict(fields=Fields(*p["fields"]), params=p["params"], time=torch.tensor(p["time"], device="cuda"),
                    state=torch.tensor(p["state"], device="cuda"), cnt=z((n, 3), torch.int64),
                    status=z(n, torch.int32), carry=z(128 * n, torch.uint8)) for p, n in zip(probs, counts)]
        es = Ensemble("dop853", mem)
        for stop in (0.3 * probs[0]["time"][-1], 0.6 * probs[0]["time"][-1], 0.0):
            es.run(stop)
        live, _ = es.counts()
        assert es.check() == 0 and (live == 0).all()
        for p, m in zip(probs, mem):
            so, co, _ = oracle.integrate("dop853", p["params"], p["time"], *p["fields"], p["state"].copy())
            assert np.array_equal(m["cnt"].cpu().numpy(), co)
            assert np.array_equal(m["state"].cpu().numpy().view(np.int64), so.view(np.int64))


def test_noalloc_grid_longer_than_16_bits(cuda, oracle_lib):
    """The no-allocation entry point takes axes of up to 64^3 nodes: node
    indices beyond 2^16 in the eight-lane gather."""
    torch = cuda
    import ctypes as C
    import oracle
    from particles_gb300 import _native as N
    from particles_gb300 import initial, params
    dm = (100003, 1, 2)
    rng = np.random.default_rng(7)
    uu = 0.01 * rng.normal(size=(3, 2, 1, dm[0]))
    bb = 0.1 * rng.normal(size=uu.shape)
    bb[0] += 1.0
    tmax = 1e-3 * 2 * np.pi / 200.0
    prm = params.pack_params(qom=200.0, vunit=0.05, tmax=tmax, dtmax=tmax, atol=1e-6, rtol=1e-6)
    tg = params.time_grid(2, tmax)
    st = np.zeros((40, tg.size, 8))
    st[:, 0, :6] = initial.isotropic_state(40, 9, speed=0.5)
    so, co, _ = oracle.integrate("rk5", prm, tg, uu, bb, st.copy())
    t = lambda a: torch.tensor(a, device="cuda")
    p = lambda a: C.c_void_p(a.data_ptr())
    d = dict(t=t(tg), u=t(uu), b=t(bb), s=t(st), c=torch.zeros((40, 3), dtype=torch.int64, device="cuda"))
    L = N.load()
    N.check(L.pt_integrate_device_noalloc(1, 40, tg.size, np.array(dm, np.int32).ctypes.data_as(C.c_void_p),
                                          prm.ctypes.data_as(C.c_void_p), p(d["t"]), p(d["u"]), p(d["b"]),
                                          p(d["s"]), p(d["c"]), None, None), "noalloc")
    assert L.pt_integrate_device_noalloc_check(None) == 0
    assert np.array_equal(d["c"].cpu().numpy(), co)
    assert np.array_equal(d["s"].cpu().numpy().view(np.int64), so.view(np.int64))
