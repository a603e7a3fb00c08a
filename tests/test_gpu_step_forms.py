"""The FP32 and FP16-deviation step at sizes where its flat cell index can go wrong (rows
shorter and longer than a warp and a block, a last block of one cell, lattices one cell
deep) against the FP64 restatement, for one, two and three population sets and LES."""
import numpy as np
import pytest

from lbcases import make_case, pop_items, run_restatement

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import ch4b200  # noqa: E402

STEPS = 4


@pytest.mark.parametrize("storage", [1, 2], ids=["f32", "f16"])
@pytest.mark.parametrize("name", ["kolmogorov", "rb", "scalar", "les", "les_vd", "les_ts"])
@pytest.mark.parametrize("dims", [(33, 5, 4), (129, 4, 3), (31, 7, 6), (3, 43, 1), (128, 3, 3), (34, 9, 33)])
def test_step_forms(name, dims, storage):
    _, cfg, state = make_case(name, seed=3, storage=storage, dims=dims)
    ref = run_restatement(cfg, state, STEPS)
    with ch4b200.Simulation(cfg) as sim:
        for k, v in pop_items(state):
            sim.set_pop(k, v)
        sim.initialize()
        sim.step(STEPS)
        got = {k: sim.get_pop(k) for k, _ in pop_items(state)}
    for k, v in pop_items(state):
        shift = {"p": 1.0, "g": 0.5 * (cfg.T_bot + cfg.T_top), "h": 0.5 * (cfg.S_bot + cfg.S_top)}[k]
        w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
        # a step rounds some twenty operations on values up to the largest population (FP32),
        # and every stored deviation once to 11 bits (FP16); errors add over the steps
        bound = (STEPS + 1) * 20 * 2.0 ** -24 * np.abs(v).max()
        if storage == 2:
            bound += (STEPS + 1) * 2 * 2.0 ** -11 * max(np.abs(a - w * shift).max() for a in (v, ref[k]))
        assert np.abs(got[k] - ref[k]).max() <= bound, (k, np.abs(got[k] - ref[k]).max(), bound)
