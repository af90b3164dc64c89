"""The gas-aerosol problem in the batched sparse-LU kernel (csrc/kernels_lanes_impl.cuh) against the oracle: ragged
batches over every shape, with cells left to the general kernel; steps that follow a rejected one; and advances captured in a graph after the number of particles changed."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from helpers import compare_tchem  # noqa: E402
from oracle import AerosolOracle  # noqa: E402
from tchem_gb import _capi, tadv_to_device, time_advance_array  # noqa: E402
from tchem_gb.aerosol import AerosolChemistry  # noqa: E402
from test_zzz_gpu_aerosol import dev, models, perturbed  # noqa: E402

pytestmark = pytest.mark.gpu

TN = [1e-30, 1e-8]
REDO_WORD = 192 // 4  # of the workspace: samples that the batched kernel left to the general one


def advance(km, am, tadv, state, nc, tol):
    """Results, work counters and the number of samples left to the general kernel."""
    B = state.shape[0]
    d_state = dev(state)
    out, t = d_state.clone(), torch.zeros(B, dtype=torch.float64, device="cuda")
    dt = torch.zeros_like(t)
    ws = torch.zeros(AerosolChemistry.getWorkSpaceSize(km, am, B), dtype=torch.uint8, device="cuda")
    stats = torch.zeros(B * _capi.SAMPLE_STATS_DTYPE.itemsize // 4, dtype=torch.int32, device="cuda")
    status = AerosolChemistry.runDeviceBatch(dev(TN), dev(tol), None, tadv_to_device(tadv, torch.device("cuda")),
                                             d_state, dev(nc), t, dt, out, km, am, stats=stats, workspace=ws)
    torch.cuda.synchronize()
    st = np.frombuffer(stats.cpu().numpy().tobytes(), dtype=_capi.SAMPLE_STATS_DTYPE)
    return out.cpu().numpy(), t.cpu().numpy(), status.cpu().numpy(), st, int(ws.view(torch.int32)[REDO_WORD])


def ragged(case, particles, B):
    km, am, gas, parts = models(case)
    am.set_number_of_particles(particles)
    state, nc = perturbed(km, am, gas, parts, B, B)
    tadv = time_advance_array(B, tend=1e-5, dt=1e-8, dtmin=1e-20, dtmax=1e-5, max_num_newton_iterations=20,
                              num_time_iterations_per_interval=100000)
    tadv["jacobian_interval"][4::7] = 2
    return km, am, state, nc, tadv, np.tile([1e-12, 1e-6], (am.n_ode, 1))


# two cells to a CTA, four, eight, and more than eight to a CTA hold (152 SMs); every seventh cell has a Jacobian
# interval of 2, which the batched kernel leaves
@pytest.mark.parametrize("particles,B", [(3, 153), (1, 305), (3, 609), (1, 1301)])
def test_every_shape_on_ragged_batches(particles, B):
    km, am, state, nc, tadv, tol = ragged("simpol", particles, B)
    out, t, status, st, left = advance(km, am, tadv, state, nc, tol)
    ref, t_ref, _, status_ref, st_ref = AerosolOracle(km, am).time_advance(tadv, state, nc, TN, tol)
    assert left == len(range(4, B, 7))
    assert np.array_equal(status, status_ref) and np.array_equal(t, t_ref)
    assert np.array_equal(st["n_steps"], st_ref["n_steps"])
    assert compare_tchem(out[:, 3:], ref[:, 3:]) <= 1e-8


# The same for CB05 with its gases at zero concentration, where the oracle is no reference for the first microseconds: at
# zero its difference step is 1e-28 and its columns of the Jacobian are lost to rounding. The cells in batches of 100, one
# to a CTA, are the reference: the shapes differ in the order of sums, 1e-16 with multipliers up to 64 over some ten steps.
@pytest.mark.parametrize("particles,B", [(1, 153), (3, 305), (1, 609)])
def test_every_shape_equals_one_cell_per_cta(particles, B):
    km, am, state, nc, tadv, tol = ragged("cb05", particles, B)
    out, t, status, st, left = advance(km, am, tadv, state, nc, tol)
    assert left == len(range(4, B, 7)) and not status.any()
    for a in range(0, B, 100):
        s = slice(a, a + 100)
        one = advance(km, am, tadv[s], state[s], nc[s], tol)
        assert np.array_equal(t[s], one[1]) and np.array_equal(st["n_steps"][s], one[3]["n_steps"])
        assert compare_tchem(out[s, 3:], one[0][:, 3:]) <= 1e-9


# Steps of seconds, where the entries between rows in kg m-3 and in ppm are 1e5 and more: no cell needs pivoting, so none is
# left to the general kernel. Bound as for the perturbed batches over 100 s: 1e-8 in the reference's norms.
@pytest.mark.parametrize("case,particles", [("simpol", 1), ("simpol", 30), ("cb05", 1), ("cb05", 3)])
def test_no_cell_is_left_for_its_units(case, particles):
    km, am, gas, parts = models(case)
    am.set_number_of_particles(particles)
    state, nc = perturbed(km, am, gas, parts, 5, 2)
    tadv = time_advance_array(5, tend=30.0, dt=1e-6, dtmin=1e-20, dtmax=10.0, max_num_newton_iterations=20,
                              num_time_iterations_per_interval=100000)
    tol = np.tile([1e-12, 1e-6], (am.n_ode, 1))
    out, t, status, st, left = advance(km, am, tadv, state, nc, tol)
    ref, t_ref, _, status_ref, st_ref = AerosolOracle(km, am).time_advance(tadv, state, nc, TN, tol)
    assert left == 0 and np.array_equal(status, status_ref) and np.array_equal(t, t_ref)
    assert compare_tchem(out[:, 3:], ref[:, 3:]) <= 1e-8


# Few particles of 1e-18 to 1e-16 kg grow by orders of magnitude within a step, so the first attempts are rejected, and
# the Newton test, on the norm of the gas, ends each stage after one iteration: what the matrix holds for the particles
# goes straight into the result. Bound: the oracle's difference Jacobian is within 1e-8 of the exact one, over the twelve
# attempts, with a factor 8 for what a step carries on.
@pytest.mark.parametrize("rtol", [1e-4, 1e-6])
def test_matrix_after_a_rejected_step(rtol):
    km, am, gas, particles = models("simpol")
    B, first = 16, 3 + km.nSpec
    state, nc = perturbed(km, am, gas, particles, B, 2)
    state[:, first:] = 10.0 ** np.random.default_rng(8).uniform(-18.0, -16.0, (B, state.shape[1] - first))
    nc *= 1e-12
    tadv = time_advance_array(B, tend=1000.0, dt=100.0, dtmin=1e-20, dtmax=1000.0, max_num_newton_iterations=20,
                              num_time_iterations_per_interval=12)
    tol = np.tile([1e-14, rtol], (am.n_ode, 1))
    tol[km.n_active:, 0] = 1e-30
    out, t, status, st, left = advance(km, am, tadv, state, nc, tol)
    ref, t_ref, _, status_ref, st_ref = AerosolOracle(km, am).time_advance(tadv, state, nc, TN, tol)
    assert left == 0 and np.array_equal(status, status_ref)
    assert st_ref["n_rejected"].sum() > B and np.array_equal(st["n_rejected"], st_ref["n_rejected"])
    assert (np.abs(t - t_ref) / t_ref).max() <= 1e-6
    assert (np.abs(out[:, first:] - ref[:, first:]) / ref[:, first:]).max() <= 1e-6


@pytest.mark.parametrize("query", [True, False])
def test_capture_after_a_change_of_particles(query):
    km, am, gas, particles = models("simpol")
    B = 5
    state, nc = perturbed(km, am, gas, particles, B, 3)
    tadv = time_advance_array(B, tend=1.0, dt=1e-6, dtmin=1e-20, dtmax=1.0, max_num_newton_iterations=20,
                              num_time_iterations_per_interval=100000)
    advance(km, am, tadv, state, nc, np.tile([1e-12, 1e-6], (am.n_ode, 1)))  # warm-up with one particle
    ws_bytes = AerosolChemistry.getWorkSpaceSize(km, am, B)
    am.set_number_of_particles(3)
    if query:  # the query builds the new tables; without them the general kernel takes the call
        ws_bytes = AerosolChemistry.getWorkSpaceSize(km, am, B)
    state, nc = perturbed(km, am, gas, particles, B, 3)
    tol = np.tile([1e-12, 1e-6], (am.n_ode, 1))
    d = [dev(TN), dev(tol), None, tadv_to_device(tadv, torch.device("cuda")), dev(state), dev(nc)]
    t, out = torch.zeros(B, dtype=torch.float64, device="cuda"), dev(state).clone()
    dt, status = torch.zeros_like(t), torch.full((B,), -1, dtype=torch.int32, device="cuda")
    ws = torch.zeros(ws_bytes, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        t.zero_()
        AerosolChemistry.runDeviceBatch(*d, t, dt, out, km, am, status=status, workspace=ws)
    ref = AerosolOracle(km, am).time_advance(tadv, state, nc, TN, tol)
    for _ in range(2):
        out.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(status.cpu().numpy(), ref[3]) and np.array_equal(t.cpu().numpy(), ref[1])
        assert compare_tchem(out.cpu().numpy()[:, 3:], ref[0][:, 3:]) <= 1e-8
