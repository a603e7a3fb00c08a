"""Particle state over several re-sorts of its slots, bit for bit.

The slots are re-sorted every 16 steps and only the planes that a kernel writes, or that differ
between particles, move: a plane left out would keep the values of the slot's last owner.  36 steps
cross three re-sorts (steps 1, 17, 33; with a deposit 2, 18, 34) of a state in which every plane
that is ever written has been.  Every field of every particle against the restatement."""
import numpy as np
import pytest

import oracle as O
from lbcases import make_case, pop_items, run_restatement

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import ch4b200  # noqa: E402

STEPS = 36
EXACT = ["particles", "particles_t", "particles_g", "particles_1w", "particles_or", "particles_tc", "particles_tt",
         "particles_ttc", "particles_rb", "particles_duct", "particles_slip", "particles_reinj", "particles_bc",
         "particles_or2", "particles_swimt", "particles_swimb", "particles_swims", "particles_swimn",
         "particles_rdiff", "particles_rand", "particles_rjr", "particles_orbc", "particles_sed", "particles_rad"]


def both(name):
    _, cfg, state = make_case(name, seed=61)
    ref = run_restatement(cfg, state, STEPS)
    with ch4b200.Simulation(cfg) as sim:
        for k, v in pop_items(state):
            sim.set_pop(k, v)
        sim.set_particles(state["part"])
        sim.initialize()
        sim.step(STEPS)
        pops = {k: sim.get_pop(k) for k, _ in pop_items(state)}
        parts = O.particles_as_dict(sim.get_particles(len(state["part"])))
    return ref, pops, parts


@pytest.mark.parametrize("name", EXACT)
def test_every_field_after_three_resorts(name):
    ref, pops, parts = both(name)
    for f, v in ref["part"].items():
        assert np.array_equal(parts[f], v), "%s: max |d| %g" % (f, np.abs(parts[f] - v).max())
    for k, v in pops.items():
        assert np.array_equal(v, ref[k]), k


@pytest.mark.parametrize("name", ["particles_jump", "particles_jumpt"])
def test_every_field_of_the_jumping_swimmers(name):
    """The device's exp is within an ulp of the host's (one call a step): 1e-12 of a field's
    largest value, where a value of another particle would be off by the field's own size."""
    ref, pops, parts = both(name)
    for f, v in ref["part"].items():
        assert np.abs(parts[f] - v).max() <= 1e-12 * max(np.abs(v).max(), 1e-300), f
