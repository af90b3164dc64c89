"""The one-warp dense FP64 factorisation and solves of the general plain kernel and the adjoint
(csrc/fp64_core.cuh, csrc/kernels_adjoint.cu) at the edges of their 32-row chunks and on both sides of the
128 species up to which the unknowns stand in the sparse LU's order. The general kernel is reached by
a Jacobian interval of 2. Bounds: the plain form's 1e-8 per species against the FP64 oracle, and for the
gradients 1e-6 of a sample's largest against the oracle's on the same recorded steps (two Newton solves to
1e-8)."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from helpers import rel_error  # noqa: E402
from oracle import Oracle  # noqa: E402
from oracle import binding as ob  # noqa: E402
from tchem_gb import AtmosphericChemistry, KineticModel, tadv_to_device, time_advance_array  # noqa: E402
from tchem_gb import adjoint as adj  # noqa: E402
from tchem_gb.generator import MechanismSpec, mechanism_yaml, sample_states  # noqa: E402

pytestmark = pytest.mark.gpu

TN = [1e-18, 1e-8]
SIZES = [(3, 5, 1.0), (32, 90, 1e-4), (33, 90, 1e-4), (64, 192, 1e-5), (65, 193, 1e-5), (128, 384, 1e-6), (129, 400, 1e-6)]


def dev(a):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64)).cuda()


def problem(m, R, horizon, interval):
    km = KineticModel.from_string(mechanism_yaml(MechanismSpec(n_species=m, n_reactions=R, seed=1000 + m)))
    B = 5
    state = sample_states(B, km.n_active, seed=7)
    tadv = time_advance_array(B, tend=horizon, dt=1e-10, dtmin=1e-10, dtmax=horizon, max_num_newton_iterations=20,
                              num_time_iterations_per_interval=1_000_000)
    tadv["jacobian_interval"] = interval
    return km, B, state, tadv, np.tile([1e-12, 1e-6], (km.n_active, 1))


@pytest.mark.parametrize("m,R,horizon", SIZES)
def test_general_plain_kernel(m, R, horizon):
    km, B, state, tadv, tol = problem(m, R, horizon, 2)
    d_state = dev(state)
    out = torch.full_like(d_state, float("nan"))
    t, dt = torch.zeros(B, dtype=torch.float64, device="cuda"), torch.zeros(B, dtype=torch.float64, device="cuda")
    st = AtmosphericChemistry.runDeviceBatch(dev(TN), dev(tol), None, tadv_to_device(tadv), d_state, t, dt, out, km,
                                             form="plain")
    ref = Oracle([km]).time_advance(tadv, state, TN, tol)
    assert np.array_equal(st.cpu().numpy(), ref[3])
    n = km.n_active
    assert rel_error(out.cpu().numpy()[:, 3:3 + n], ref[0][:, 3:3 + n], 1e-12).max() <= 1e-8


@pytest.mark.parametrize("m,R,horizon", SIZES)
def test_adjoint_sizes(m, R, horizon):
    km, B, state, tadv, tol = problem(m, R, horizon, 1)
    d_state = dev(state)
    t, dt = torch.zeros(B, dtype=torch.float64, device="cuda"), torch.zeros(B, dtype=torch.float64, device="cuda")
    tape = adj.new_tape(B, km.n_active, 1024)
    st = adj.record(km, dev(TN), dev(tol), tadv_to_device(tadv), d_state, t, dt, torch.empty_like(d_state), tape)
    assert int((st != 0).sum()) == 0
    lam = np.random.default_rng(m).normal(size=(B, km.n_active))
    gx, gk, ast = adj.adjoint(km, dev(TN), tadv_to_device(tadv), d_state, tape, dev(lam))
    assert int((ast != 0).sum()) == 0
    rx, rk = ob.adjoint(Oracle([km]), tadv, state, TN, ob.Tape(tape.dt.cpu().numpy(), tape.nsteps.cpu().numpy()), lam)
    for got, ref in ((gx, rx), (gk, rk)):
        scale = np.abs(ref).max(axis=1, keepdims=True) + 1e-300
        assert (np.abs(got.cpu().numpy() - ref) / scale).max() <= 1e-6
