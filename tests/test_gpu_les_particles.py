"""LES with particles: from the second step on u^n of the eddy viscosity is taken from the vectors
that the last step formed for the particles, instead of a pass of its own.  FP64.

One-way particles do not act on the fluid: the populations are bit for bit those of the same run
without particles (whose u^n has its own pass), also after new populations in the middle of a
run.  Two-way particles against the restatement, with the deposit in both."""
import numpy as np
import pytest

import oracle as O
from ch4b200 import abi
from lbcases import make_case, make_particles, pop_items

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import ch4b200  # noqa: E402

ONE_WAY = ["LAGRANGE", "LAGRANGE_WRAP", "LAGRANGE_GRADIENT", "LAGRANGE_ADDEDMASS"]
TWO_WAY = ONE_WAY + ["LAGRANGE_TWOWAY", "LAGRANGE_TWOWAY_MOMENTUM"]


def les_case(name, more, storage=0):
    """The case with further flags, and 200 particles (inertial ones at rest, tracers)."""
    _, cfg, state = make_case(name, seed=5, storage=storage)
    abi.set_flags(cfg, O.FLAGSETS[make_case(name)[0]] + more)
    parts = make_particles(np.random.default_rng(5), 200, cfg.NX, cfg.NY, cfg.NZ)
    for i, p in enumerate(parts):
        if p.tau_drag:
            p.tau_drag, p.beta_coeff = [0.8, 1.5][i % 2], [1.0, 0.5][i // 4 % 2]
    return cfg, state, parts


def upload(sim, state, parts=None):
    for k, v in pop_items(state):
        sim.set_pop(k, v)
    if parts is not None:
        sim.set_particles(parts)
    sim.initialize()


@pytest.mark.parametrize("name", ["les", "les_lilly", "les_sism", "les_kalman", "les_vd", "les_ls", "les_wale",
                                  "trt_les"])
@pytest.mark.parametrize("storage", [0, 1])
def test_one_way_particles_leave_the_fluid_alone(name, storage):
    cfg, state, parts = les_case(name, ONE_WAY, storage)
    _, plain, other = make_case(name, seed=6, storage=storage)
    with ch4b200.Simulation(cfg) as a, ch4b200.Simulation(plain) as b:
        upload(a, state, parts)
        upload(b, state)
        for s in (a, b):
            s.step(20)
        moved = O.particles_as_dict(a.get_particles(len(parts)))
        assert np.isfinite(moved["x"]).all() and np.abs(moved["ux"]).max() > 0
        for k, _ in pop_items(state):
            assert np.array_equal(a.get_pop(k), b.get_pop(k)), k
        for s in (a, b):  # other populations: the vectors at hand are not theirs
            upload(s, other)
            s.step(5)
        for k, _ in pop_items(state):
            assert np.array_equal(a.get_pop(k), b.get_pop(k)), k


@pytest.mark.parametrize("name", ["les", "les_sism", "les_kalman", "les_vd"])
def test_two_way_particles_bit_identical(name):
    cfg, state, parts = les_case(name, TWO_WAY)
    ref = O.Restatement(cfg)
    with ch4b200.Simulation(cfg) as sim:
        for s in (ref, sim):
            upload(s, state, parts)
            s.step(20)
        want = O.particles_as_dict(ref.get_particles(len(parts)))
        assert np.isfinite(want["x"]).all()
        got = O.particles_as_dict(sim.get_particles(len(parts)))
        for f, v in want.items():
            assert np.array_equal(got[f], v), f
        assert np.array_equal(sim.get_pop("p"), ref.get_pop("p"))
    ref.close()
