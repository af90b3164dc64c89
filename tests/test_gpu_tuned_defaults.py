"""The tuned preference (tchem_gb_autotune) and the default kernels: where the full-Newton form's default is the fastest,
tuning keeps it, and an E3SM advance takes its default whatever the box model's preference is. Seen by the launches of
a call: the batched kernel and the general one behind it, or one kernel alone."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from helpers import GOLDEN, mech_path  # noqa: E402
from tchem_gb import (AtmosphericChemistry, KineticModel, set_scenario_conditions,  # noqa: E402
                      set_scenario_external_forcing, set_scenario_photolysis_rates, tadv_to_device, time_advance_array)
from tchem_gb.atmospheric_chemistry import kernel_launches  # noqa: E402
from tchem_gb.e3sm import AtmosphericChemistryE3SM  # noqa: E402
from tchem_gb.generator import MechanismSpec, mechanism_yaml, sample_states  # noqa: E402

pytestmark = pytest.mark.gpu

TN = [1e-18, 1e-8]


def dev(a):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64)).cuda()


def arrays(state, m, horizon, dt0):
    B = state.shape[0]
    tadv = time_advance_array(B, tend=horizon, dt=dt0, dtmin=dt0, dtmax=horizon, max_num_newton_iterations=20,
                              num_time_iterations_per_interval=100_000)
    d_state, t = dev(state), torch.zeros(B, dtype=torch.float64, device="cuda")
    return dev(TN), dev(np.tile([1e-12, 1e-6], (m, 1))), tadv_to_device(tadv), d_state, t, torch.zeros_like(t), \
        torch.empty_like(d_state)


@pytest.mark.parametrize("m,R", [(20, 60), (32, 90), (51, 156)])
def test_tuning_keeps_the_default_where_it_is_fastest(m, R):
    # 76 samples: one to an SM of the batched kernel, 1.4 to 2 times the register kernels' speed
    km = KineticModel.from_string(mechanism_yaml(MechanismSpec(n_species=m, n_reactions=R, seed=1000 + m)))
    tn, tt, tadv, state, t, dt, out = arrays(sample_states(76, m, seed=3), m, 1e-4, 1e-10)
    chosen, times = AtmosphericChemistry.autotune(km, tn, tt, tadv, state, form="mixed")
    assert chosen in (0, 32) and 32 in times
    before = kernel_launches()
    st = AtmosphericChemistry.runDeviceBatch(tn, tt, None, tadv, state, t, dt, out, km, form="mixed")
    assert kernel_launches() - before == 2 and not bool(st.any())


@pytest.mark.parametrize("pref", [0, 32, 64])
def test_e3sm_default_whatever_the_preference(pref):
    km = KineticModel.from_file(mech_path("uci_v2_test3.yaml"))
    scenario = GOLDEN / "e3sm" / "uci_col_input_conditions.yaml"
    state = set_scenario_conditions(scenario, km)
    B = state.shape[0]
    photo, ext = set_scenario_photolysis_rates(scenario, B), set_scenario_external_forcing(scenario, km, B)
    tn, tt, tadv, d_state, t, dt, out = arrays(state, km.n_active, 60.0, 1e-20)
    AtmosphericChemistry.set_threads_per_sample(km, pref, form="mixed")
    before = kernel_launches()
    st = AtmosphericChemistryE3SM.runDeviceBatch(tn, tt, None, tadv, d_state, dev(photo), dev(ext), t, dt, out, km,
                                                 form="mixed")
    assert kernel_launches() - before == 3 and not bool(st.any())  # rate constants, batched and general kernel
