"""The machine with one lane per particle (csrc/pt_integrator.cuh) on runs that
would go to the one with eight: the tests of launch variants, failures,
windows, ensembles, gathers and controllers once more with every run started on
one lane, alone to its end, with its last particles handed over, and with a
hand-over list that fills up."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import small_problem
from test_gpu_checked import ROOT, SCRIPT
from test_gpu_ensemble import (test_ensemble_exact_matches_oracle_per_member,        # noqa: F401
                               test_ensemble_graph_replay_equals_stepwise,
                               test_ensemble_graph_replay_matches_oracle_per_member)
from test_gpu_face import (test_face_steps_in_an_ensemble,                           # noqa: F401
                           test_face_steps_turbulent_fewer_rejections_same_accuracy)
from test_gpu_failures import (test_attempt_cap_matches_oracle,                      # noqa: F401
                               test_bad_queue_order_entries_are_skipped_and_reported,
                               test_checkpoint_file_resume_is_bit_identical,
                               test_nonfinite_field_stops_particles_like_the_oracle,
                               test_time_budget_interrupts_and_the_carry_resumes)
from test_gpu_grids import test_exact_bitwise_noncubic_offset_domain_eta_open        # noqa: F401
from test_gpu_learned import test_learned_controller_in_the_integrator               # noqa: F401
from test_gpu_mixed import (test_mixed_turbulent_statistics,                         # noqa: F401
                            test_mixed_windowed_resume_matches_single_run,
                            test_near_gather_mixed_statistics, test_noise_floor_norm)
from test_gpu_parity import (test_dop853_pi_controller_bitwise,                      # noqa: F401
                             test_fused_exact_bitwise, test_near_gather_exact_bitwise,
                             test_tiny_and_ragged_batches_bitwise)
from test_gpu_variants import (test_autotune_choice_keeps_results,                   # noqa: F401
                               test_exact_variants_bitwise, test_mixed_learned_variants_agree)

pytestmark = pytest.mark.gpu

HAND_CAP = {"alone": 0, "handed": -1, "list_full": 37}


@pytest.fixture(autouse=True, params=list(HAND_CAP))
def machine(request, native):
    assert native.pt_debug_machines(0, HAND_CAP[request.param]) == 0
    yield request.param
    native.pt_debug_machines(-1, -1)


def test_bounds_checked_gathers(cuda, machine):
    first = "from particles_gb300 import _native; _native.load().pt_debug_machines(0, %d)\n" % HAND_CAP[machine]
    r = subprocess.run([sys.executable, "-c", first + SCRIPT], cwd=ROOT, env=dict(os.environ, PT_CHECKED="1"),
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    assert "checked ok" in r.stdout


def _run(torch, f, prob, **kw):
    npart = prob["state"].shape[0]
    s = torch.tensor(prob["state"], device="cuda")
    c = torch.zeros((npart, 3), dtype=torch.int64, device="cuda")
    st = torch.zeros(npart, dtype=torch.int32, device="cuda")
    f.run_device(prob["method"], prob["params"], torch.tensor(prob["time"], device="cuda"), s, c, st, **kw)
    assert f.run_check() == 0
    return s.cpu().view(torch.int64), c.cpu(), st.cpu()


@pytest.mark.parametrize("precision", ["fp64", "fp64_fma", "fp32", "bf16"])
@pytest.mark.parametrize("method", ["rk5", "dop853"])
@pytest.mark.parametrize("with_j", [False, True])
def test_every_variant_gives_the_bits_of_eight_lanes(cuda, native, machine, precision, method, with_j):
    """Register caps and block sizes, open x faces and a queue order."""
    torch = cuda
    from particles_gb300 import Fields
    prob = small_problem(method, n=20, npart=777, periods=0.1, seed=63, with_j=with_j, nsteps=5,
                         gamma_range=(1.001, 50.0), tol=1e-8)
    prob["state"][:200, 0, 0] = 0.001                       # next to an open face
    f = Fields(*prob["fields"], precision=precision)
    order = torch.tensor(np.random.default_rng(1).permutation(777).astype(np.int32), device="cuda")
    kw = dict(eta=1e-3 if with_j else 0.0, open_x=True, open_x_margin=0.002)
    native.pt_debug_machines(-1, -1)
    want = _run(torch, f, prob, **kw)
    native.pt_debug_machines(0, HAND_CAP[machine])
    assert (want[2] == 2).any() and (want[2] == 0).any()    # some escaped, some finished
    for v in (2, 3, 4):
        for tpb in (64, 128, 256):
            got = _run(torch, f, prob, order=order, blocks_per_sm=v, threads_per_block=tpb, **kw)
            for a, b in zip(got, want):
                assert torch.equal(a, b), (v, tpb)
