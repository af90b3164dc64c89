"""The batched sparse-LU time advance (csrc/kernels_lanes_impl.cuh) against the FP64 oracle at the edges of
its shapes: batches that fill, overfill and underfill the lanes of every shape, mechanisms from three
species to the tail block's largest, and the samples it leaves to the general kernel (a Jacobian
interval above 1, a negative step size, multipliers beyond the bound of the factorization without
pivot search). Bounds are the forms' own: 1e-8 per species for the plain form, 1e-6 for the full-Newton
FP32 form, with the same step counts within 3 %."""
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


def advance(km, state, tadv, form, in_place=False):
    B, m = state.shape[0], km.n_active
    tol = np.tile([1e-12, 1e-6], (m, 1))
    d_state = dev(state)
    out = d_state if in_place else torch.full_like(d_state, float("nan"))
    t = torch.zeros(B, dtype=torch.float64, device="cuda")
    dt = torch.full_like(t, -7.0)
    stats = torch.full((B, 8), -7, dtype=torch.int32, device="cuda")
    st = AtmosphericChemistry.runDeviceBatch(dev(TN), dev(tol), None, tadv_to_device(tadv), d_state, t, dt, out, km,
                                             stats=stats, form=form)
    torch.cuda.synchronize()
    assert AtmosphericChemistry.device_error() == 0
    return (out.cpu().numpy(), t.cpu().numpy(), dt.cpu().numpy(), st.cpu().numpy(), stats.cpu().numpy(),
            Oracle([km]).time_advance(tadv, state, TN, tol))


def check(km, got, form):
    out, t, dt, st, stats, ref = got
    m = km.n_active
    assert np.array_equal(st, ref[3])
    assert rel_error(out[:, 3:3 + m], ref[0][:, 3:3 + m], 1e-12).max() <= BOUND[form]
    assert np.array_equal(out[:, :3], ref[0][:, :3]) and np.array_equal(out[:, 3 + m:], ref[0][:, 3 + m:])
    assert np.array_equal(t, ref[1])
    steps, ref_steps = stats[:, 0].sum(), ref[4]["n_steps"].sum()
    assert abs(int(steps) - int(ref_steps)) <= 0.03 * ref_steps


def tadv_of(B, horizon, **kw):
    return time_advance_array(B, tend=horizon, dt=1e-10, dtmin=1e-10, dtmax=horizon, max_num_newton_iterations=20,
                              num_time_iterations_per_interval=kw.pop("budget", 1_000_000), **kw)


# one sample per CTA, two, four, eight, sixteen with one and with two CTAs per SM (152 SMs): a full
# shape, one sample more, and odd remainders
@pytest.mark.parametrize("form", ["mixed", "plain"])
@pytest.mark.parametrize("B", [1, 152, 153, 305, 609, 1217, 2433, 19459])
def test_every_shape_on_ragged_batches(B, form):
    km = KineticModel.from_string(mechanism_yaml(MechanismSpec()))
    state = sample_states(B, km.n_active, seed=B)
    tadv = tadv_of(B, 1e-6)
    check(km, advance(km, state, tadv, form), form)


# fewer species than the smallest tail, a tail that is the whole matrix, more species than slots of the
# wide shapes, the tail's largest block
@pytest.mark.parametrize("form", ["mixed", "plain"])
@pytest.mark.parametrize("m,R,B,horizon", [(3, 5, 5, 1.0), (8, 20, 700, 1e-3), (33, 90, 17, 1e-2), (64, 192, 40, 1e-3),
                                           (65, 193, 2500, 1e-7), (128, 384, 9, 1e-4), (129, 400, 3, 1e-5),
                                           (200, 640, 3, 1e-6), (320, 1024, 2, 1e-7)])
def test_mechanism_sizes(m, R, B, horizon, form):
    if form == "plain" and m > 200:
        horizon = 1e-8
    km = KineticModel.from_string(mechanism_yaml(MechanismSpec(n_species=m, n_reactions=R, seed=1000 + m)))
    state = sample_states(B, km.n_active, seed=7)
    check(km, advance(km, state, tadv_of(B, horizon), form), form)


@pytest.mark.parametrize("form", ["mixed", "plain"])
def test_samples_left_to_the_general_kernel(form):
    km = KineticModel.from_string(mechanism_yaml(MechanismSpec()))
    B = 37
    state = sample_states(B, km.n_active, seed=3)
    tadv = tadv_of(B, 1e-3)
    tadv["jacobian_interval"][5::7] = 3
    tadv["dt"][6] = -1.0
    tadv["num_time_iterations_per_interval"][8] = 0
    tadv["num_time_iterations_per_interval"][9] = 4
    out, t, dt, st, stats, ref = advance(km, state, tadv, form, in_place=True)
    m = km.n_active
    assert np.array_equal(st, ref[3]) and st[6] == 3
    keep = np.arange(B) != 6
    assert rel_error(out[keep, 3:3 + m], ref[0][keep, 3:3 + m], 1e-12).max() <= BOUND[form]
    assert np.array_equal(out[6], state[6]) and dt[6] == -7.0 and t[6] == 0.0
    assert np.array_equal(stats[[8, 9], 0], [0, 4]) and t[8] == 0.0 and np.array_equal(out[8], state[8])


# A -> 200 B with B -> A: the multiplier of A's column is near 200 for long steps
GROWTH = """
NCAR-version: v1.0
constant_species:
- name: M
species:
- name: A
- name: B
- name: C
reactions:
- reactants: {}
""".replace("- reactants: {}\n", "") + "".join(
    f"- reactants:\n    {a}: 1\n  products:\n    {b}: {n}\n  type: ARRHENIUS\n  coefficients:\n    A: {k}\n    B: 0.0\n"
    "    C: 0.0\n    D: 300.0\n    E: 0.0\n"
    for a, b, n, k in (("A", "B", 200, 1.0e3), ("B", "C", 1, 0.5), ("C", "A", 0.001, 0.1)))


@pytest.mark.parametrize("form", ["mixed", "plain"])
def test_multipliers_beyond_the_bound(form):
    km = KineticModel.from_string(GROWTH)
    B = 19
    state = sample_states(B, km.n_active, seed=11)
    check(km, advance(km, state, tadv_of(B, 50.0), form), form)
