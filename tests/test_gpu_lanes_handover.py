"""Samples that the batched sparse-LU time advance leaves to the general kernel of the same call, in every path that
runs the two one behind the other: box model, E3SM, trajectory record and batches of mixed mechanisms (the gas-aerosol
path is in test_gpu_lanes_aero.py). The workspace header's counts say how many were left, per structure group; results
are the oracle's to the forms' bounds."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from helpers import GOLDEN, mech_path, rel_error  # noqa: E402
from oracle import E3smOracle, Oracle  # noqa: E402
from oracle import binding as ob  # noqa: E402
from tchem_gb import (AtmosphericChemistry, KineticModel, set_scenario_conditions,  # noqa: E402
                      set_scenario_external_forcing, set_scenario_photolysis_rates, tadv_to_device, time_advance_array)
from tchem_gb import adjoint as adj  # noqa: E402
from tchem_gb.e3sm import AtmosphericChemistryE3SM  # noqa: E402
from tchem_gb.generator import MechanismSpec, mechanism_yaml, sample_states  # noqa: E402

pytestmark = pytest.mark.gpu

TN = [1e-18, 1e-8]
BOUND = {"plain": 1e-8, "mixed": 1e-6}
REDO_WORD = 192 // 4


def dev(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a)).to(device="cuda", dtype=dtype)


def tadv_of(B, horizon, dt0=1e-10):
    return time_advance_array(B, tend=horizon, dt=dt0, dtmin=dt0, dtmax=horizon, max_num_newton_iterations=20,
                              num_time_iterations_per_interval=1_000_000)


def left(ws, groups=1):
    return ws.view(torch.int32)[REDO_WORD:REDO_WORD + groups].cpu().tolist()


# A -> 200 B, B -> C, C -> 0.001 A and a ring of nine more: the multiplier of A's column is near 200 for long steps.
# Without the last of the three nothing but A itself is in A's row, which is then subtracted from no other.
def growth(feedback=True):
    lines = ["NCAR-version: v1.0", "constant_species:", "- name: M", "species:"]
    names = ["A", "B", "C"] + [f"X{i}" for i in range(9)]
    lines += [f"- name: {n}" for n in names] + ["reactions:"]
    steps = [("A", "B", 200, 1.0e3), ("B", "C", 1, 0.5), ("C", "A" if feedback else "X0", 0.001, 0.1)]
    steps += [(f"X{i}", f"X{(i + 1) % 9}", 1, 0.1 * (i + 1)) for i in range(9)]
    for a, b, n, k in steps:
        lines += ["- reactants:", f"    {a}: 1", "  products:", f"    {b}: {n}", "  type: ARRHENIUS", "  coefficients:",
                  f"    A: {k}", "    B: 0.0", "    C: 0.0", "    D: 300.0", "    E: 0.0"]
    return KineticModel.from_string("\n".join(lines) + "\n")


@pytest.mark.parametrize("form", ["mixed", "plain"])
@pytest.mark.parametrize("feedback", [True, False])
def test_multipliers_beyond_the_bound_are_handed_over(feedback, form):
    km, B = growth(feedback), 19
    m = km.n_active
    state, tadv, tol = sample_states(B, m, seed=11), tadv_of(B, 50.0), np.tile([1e-12, 1e-6], (12, 1))
    ws = torch.zeros(AtmosphericChemistry.getWorkSpaceSize(km, B, form), dtype=torch.uint8, device="cuda")
    d_state, t = dev(state), torch.zeros(B, dtype=torch.float64, device="cuda")
    out = torch.empty_like(d_state)
    st = AtmosphericChemistry.runDeviceBatch(dev(TN), dev(tol), None, tadv_to_device(tadv), d_state, t,
                                             torch.zeros_like(t), out, km, form=form, workspace=ws)
    ref = Oracle([km]).time_advance(tadv, state, TN, tol)
    assert left(ws) == [B if feedback else 0]
    assert np.array_equal(st.cpu().numpy(), ref[3]) and np.array_equal(t.cpu().numpy(), ref[1])
    assert rel_error(out.cpu().numpy()[:, 3:3 + m], ref[0][:, 3:3 + m], 1e-12).max() <= BOUND[form]


@pytest.mark.parametrize("form", ["mixed", "plain"])
def test_e3sm_columns(form):
    km = KineticModel.from_file(mech_path("uci_v2_test3.yaml"))
    scenario = GOLDEN / "e3sm" / "uci_col_input_conditions.yaml"
    state = set_scenario_conditions(scenario, km)
    B, m = state.shape[0], km.n_active
    photo, ext = set_scenario_photolysis_rates(scenario, B), set_scenario_external_forcing(scenario, km, B)
    tadv, tol = tadv_of(B, 300.0, 1e-20), np.tile([1e-12, 1e-6], (m, 1))
    tadv["jacobian_interval"][3::7] = 2
    ws = torch.zeros(AtmosphericChemistryE3SM.getWorkSpaceSize(km, B, form), dtype=torch.uint8, device="cuda")
    d_state, t = dev(state), torch.zeros(B, dtype=torch.float64, device="cuda")
    out = torch.empty_like(d_state)
    st = AtmosphericChemistryE3SM.runDeviceBatch(dev(TN), dev(tol), None, tadv_to_device(tadv), d_state, dev(photo),
                                                 dev(ext), t, torch.zeros_like(t), out, km, form=form, workspace=ws)
    ref = E3smOracle(km).time_advance(tadv, state, photo, ext, TN, tol)
    assert left(ws) == [len(range(3, B, 7))]
    assert np.array_equal(st.cpu().numpy(), ref[3]) and np.array_equal(t.cpu().numpy(), ref[1])
    assert rel_error(out.cpu().numpy()[:, 3:3 + m], ref[0][:, 3:3 + m], 1e-12).max() <= BOUND[form]


def test_trajectory_record():
    km, B = KineticModel.from_string(mechanism_yaml(MechanismSpec())), 23
    m = km.n_active
    state, tadv, tol = sample_states(B, m, seed=5), tadv_of(B, 1e-4), np.tile([1e-12, 1e-6], (m, 1))
    tadv["jacobian_interval"][2::5] = 3
    d_state, t = dev(state), torch.zeros(B, dtype=torch.float64, device="cuda")
    out, tape = torch.empty_like(d_state), adj.new_tape(B, m, 512)
    st = adj.record(km, dev(TN), dev(tol), tadv_to_device(tadv), d_state, t, torch.zeros_like(t), out, tape)
    ref = Oracle([km]).time_advance(tadv, state, TN, tol)
    assert np.array_equal(st.cpu().numpy(), ref[3]) and np.array_equal(tape.nsteps.cpu().numpy(), ref[4]["n_steps"])
    assert rel_error(out.cpu().numpy()[:, 3:3 + m], ref[0][:, 3:3 + m], 1e-12).max() <= BOUND["plain"]
    # the recorded steps, run again from the start, lead to the recorded end state
    y = ob.replay(Oracle([km]), tadv, state, TN, ob.Tape(tape.dt.cpu().numpy(), tape.nsteps.cpu().numpy()))
    assert rel_error(y, out.cpu().numpy()[:, 3:3 + m], 1e-12).max() <= BOUND["plain"]
    lam = np.random.default_rng(1).uniform(0.5, 1.5, (B, m))
    gx, gk, ast = adj.adjoint(km, dev(TN), tadv_to_device(tadv), d_state, tape, dev(lam))
    assert not bool(ast.any())
    rx, rk = ob.adjoint(Oracle([km]), tadv, state, TN, ob.Tape(tape.dt.cpu().numpy(), tape.nsteps.cpu().numpy()), lam)
    for got, want in ((gx, rx), (gk, rk)):  # each Newton solve to 1e-8, two a step
        assert (np.abs(got.cpu().numpy() - want) / (np.abs(want).max(axis=1, keepdims=True) + 1e-300)).max() <= 1e-6


@pytest.mark.parametrize("form", ["mixed", "plain"])
def test_mixed_mechanisms(form):
    big = KineticModel.from_string(mechanism_yaml(MechanismSpec()))
    small = KineticModel.from_string(mechanism_yaml(MechanismSpec(n_species=40, n_reactions=120, seed=1040)))
    B, rng = 61, np.random.default_rng(2)
    mos = rng.integers(0, 2, B).astype(np.int32)
    state = np.zeros((B, big.state_dim))
    for k, km in enumerate((big, small)):
        rows = sample_states(B, km.n_active, seed=20 + k)
        state[mos == k, :rows.shape[1]] = rows[mos == k]
    tadv, tol = tadv_of(B, 1e-4), np.tile([1e-12, 1e-6], (big.n_active, 1))
    tadv["jacobian_interval"][1::4] = 2
    mechs = [big, small]
    ws = torch.zeros(AtmosphericChemistry.getWorkSpaceSize(mechs, B, form), dtype=torch.uint8, device="cuda")
    d_state, t = dev(state), torch.zeros(B, dtype=torch.float64, device="cuda")
    out = torch.zeros_like(d_state)
    st = AtmosphericChemistry.runDeviceBatch(dev(TN), dev(tol), None, tadv_to_device(tadv), d_state, t,
                                             torch.zeros_like(t), out, mechs, mech_of_sample=dev(mos, torch.int32),
                                             form=form, workspace=ws)
    ref = Oracle(mechs).time_advance(tadv, state, TN, tol, mech_of_sample=mos)
    assert left(ws, 2) == [int((mos[1::4] == k).sum()) for k in (0, 1)]
    assert np.array_equal(st.cpu().numpy(), ref[3]) and np.array_equal(t.cpu().numpy(), ref[1])
    y = out.cpu().numpy()
    for k, km in enumerate(mechs):
        sel, m = mos == k, km.n_active
        assert rel_error(y[sel, 3:3 + m], ref[0][sel, 3:3 + m], 1e-12).max() <= BOUND[form]
