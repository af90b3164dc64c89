"""Lanes of the batched sparse-LU time advance (csrc/kernels_lanes_impl.cuh) that held a sample with non-finite
values and take another from the queue: the later samples come out as the oracle's. The batches are larger than
the shapes' lanes, so that a lane is refilled, and the last FP32 cases have a tail block with more rows than the
matrix (32 rows at one and two samples per CTA and 8 rows at sixteen, on 152 SMs).
Bounds are the forms' own: 1e-6 per species for the full-Newton FP32 form, 1e-8 for the plain form."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from helpers import rel_error  # noqa: E402
from oracle import Oracle  # noqa: E402
from tchem_gb import AtmosphericChemistry, KineticModel, tadv_to_device, time_advance_array  # noqa: E402
from tchem_gb.generator import MechanismSpec, mechanism_yaml, sample_states  # noqa: E402

pytestmark = pytest.mark.gpu

TN = [1e-18, 1e-8]
BOUND = {"plain": 1e-8, "mixed": 1e-6}


def dev(a):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64)).cuda()


@pytest.mark.parametrize("form", ["mixed", "plain"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("m,R,B,horizon", [(8, 20, 290, 1e-3), (4, 9, 2000, 1e-2), (20, 60, 580, 1e-3), (3, 5, 4500, 1.0),
                                           (51, 156, 290, 1e-6), (12, 36, 180, 1e-3), (20, 60, 500, 1e-3),
                                           (4, 9, 19600, 1e-4)])
def test_samples_after_a_non_finite_one(m, R, B, horizon, bad, form):
    km = KineticModel.from_string(mechanism_yaml(MechanismSpec(n_species=m, n_reactions=R, seed=1000 + m)))
    state = sample_states(B, m, seed=7)
    lost = np.arange(0, B, 9)
    state[lost, 3 + m // 2] = bad
    tadv = time_advance_array(B, tend=horizon, dt=1e-10, dtmin=1e-10, dtmax=horizon, max_num_newton_iterations=20,
                              num_time_iterations_per_interval=2000)
    tol = np.tile([1e-12, 1e-6], (m, 1))
    d_state = dev(state)
    out = torch.full_like(d_state, float("nan"))
    t, dt = torch.zeros(B, dtype=torch.float64, device="cuda"), torch.zeros(B, dtype=torch.float64, device="cuda")
    st = AtmosphericChemistry.runDeviceBatch(dev(TN), dev(tol), None, tadv_to_device(tadv), d_state, t, dt, out, km,
                                             form=form).cpu().numpy()
    keep = np.setdiff1d(np.arange(B), lost)
    ref = Oracle([km]).time_advance(tadv[keep], state[keep], TN, tol)
    assert np.array_equal(st[keep], ref[3]) and np.all(st[lost] != 0)
    assert rel_error(out.cpu().numpy()[keep, 3:3 + m], ref[0][:, 3:3 + m], 1e-12).max() <= BOUND[form]
    assert np.array_equal(t.cpu().numpy()[keep], ref[1])
