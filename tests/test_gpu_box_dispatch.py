"""Which kernel a box-model batch takes by default (lanes_pay_for_box in csrc/lane_tables.cu) at the lines of the
rule, seen by the launches of a call: the batched kernel and the general one behind it, or one kernel alone. On both
sides of a line the results are the oracle's to the form's bound."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from helpers import rel_error  # noqa: E402
from oracle import Oracle  # noqa: E402
from tchem_gb import AtmosphericChemistry, KineticModel, tadv_to_device, time_advance_array  # noqa: E402
from tchem_gb.atmospheric_chemistry import kernel_launches  # noqa: E402
from tchem_gb.generator import MechanismSpec, mechanism_yaml, sample_states  # noqa: E402

pytestmark = pytest.mark.gpu

TN = [1e-18, 1e-8]
BOUND = {"plain": 1e-8, "mixed": 1e-6}


def dev(a):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64)).cuda()


# (species, form, first batch size of the other side, in samples per SM as a fraction, batched kernel below the line)
@pytest.mark.parametrize("m,R,form,num,den,below", [(8, 20, "mixed", 128, 1, False), (20, 60, "mixed", 400, 120, True),
                                                    (32, 90, "mixed", 1024, 120, True), (33, 90, "mixed", 11, 2, True),
                                                    (64, 192, "mixed", 14, 1, False), (3, 5, "plain", 1, 1, True),
                                                    (3, 5, "plain", 13, 1, False)])
def test_sides_of_the_line(m, R, form, num, den, below):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    # the rule's lines are "up to" but for the two-CTA shape's, which is "from"
    last = sms * num // den - (1 if num == 128 else 0)
    km = KineticModel.from_string(mechanism_yaml(MechanismSpec(n_species=m, n_reactions=R, seed=1000 + m)))
    for B in (last, last + 1):
        state = sample_states(B, m, seed=7)
        tadv = time_advance_array(B, tend=1e-6, dt=1e-10, dtmin=1e-10, dtmax=1e-6, max_num_newton_iterations=20,
                                  num_time_iterations_per_interval=100_000)
        tol = np.tile([1e-12, 1e-6], (m, 1))
        d_state = dev(state)
        out, t = torch.empty_like(d_state), torch.zeros(B, dtype=torch.float64, device="cuda")
        before = kernel_launches()
        st = AtmosphericChemistry.runDeviceBatch(dev(TN), dev(tol), None, tadv_to_device(tadv), d_state, t,
                                                 torch.zeros_like(t), out, km, form=form)
        assert kernel_launches() - before == (2 if below == (B == last) else 1)
        ref = Oracle([km]).time_advance(tadv, state, TN, tol)
        assert np.array_equal(st.cpu().numpy(), ref[3])
        assert rel_error(out.cpu().numpy()[:, 3:3 + m], ref[0][:, 3:3 + m], 1e-12).max() <= BOUND[form]
