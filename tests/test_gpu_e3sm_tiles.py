"""The E3SM rate kernels at the edges of their two layouts (lanes over reactions up to four samples per SM,
32-sample tiles above): ragged batches give, row by row, what the rows give in small batches, bit for bit
(both layouts evaluate the same expressions in the same order), with and without photolysis input and
external sources, and small batches match the oracle's rate constants."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from helpers import GOLDEN, mech_path  # noqa: E402
from oracle import E3smOracle  # noqa: E402
from tchem_gb import (KineticModel, set_scenario_conditions, set_scenario_external_forcing,  # noqa: E402
                      set_scenario_photolysis_rates)
from tchem_gb.e3sm import NetProductionRates, RateofProgress, ReactionRates  # noqa: E402

pytestmark = pytest.mark.gpu

SCENARIO = GOLDEN / "e3sm" / "uci_col_input_conditions.yaml"


def dev(a):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64)).cuda()


def evaluate(km, state, photo, ext):
    B, R, m = state.shape[0], km.nReac, km.n_active
    k = torch.full((B, R), float("nan"), dtype=torch.float64, device="cuda")
    q, w = k.clone(), torch.full((B, m), float("nan"), dtype=torch.float64, device="cuda")
    ReactionRates.runDeviceBatch(state, k, km, photo_rates=photo)
    RateofProgress.runDeviceBatch(state, photo, q, km)
    NetProductionRates.runDeviceBatch(state, photo, ext, w, km)
    torch.cuda.synchronize()
    return [v.cpu().numpy() for v in (k, q, w)]


@pytest.mark.parametrize("inputs", [True, False])
@pytest.mark.parametrize("B", [609, 640, 641, 2433])
def test_tiles_equal_small_batches(B, inputs):
    km = KineticModel.from_file(mech_path("uci_v2_test3.yaml"))
    base = set_scenario_conditions(SCENARIO, km)
    n = base.shape[0]
    rng = np.random.default_rng(B)
    idx = np.arange(B) % n
    state = base[idx] * rng.uniform(0.9, 1.1, (B, 1))
    photo = set_scenario_photolysis_rates(SCENARIO, n)[idx] * rng.uniform(0.5, 1.5, (B, 1))
    ext = set_scenario_external_forcing(SCENARIO, km, n)[idx] * rng.uniform(0.5, 1.5, (B, 1))
    d = [dev(state), dev(photo) if inputs else None, dev(ext) if inputs else None]
    whole = evaluate(km, *d)
    for a in range(0, B, 300):
        part = evaluate(km, *[None if v is None else v[a:a + 300].contiguous() for v in d])
        for x, y in zip(whole, part):
            assert np.array_equal(x[a:a + 300], y)
    oracle = E3smOracle(km)
    for b in (0, B - 1):
        ref = oracle.kforward(state[b, 2], state[b, 1], state[b, 3:], photo[b] if inputs else np.zeros(0))
        assert (np.abs(whole[0][b] - ref) / np.maximum(np.abs(ref), 1e-300)).max() <= 1e-12
