"""Read-back formed on the device (csrc/part_records.cuh, ch4_ensemble_get_fields) where its
tiles and chunks end: particle counts about the tile of 32 slots and about the chunk of the
staging buffer's halves, slots re-sorted meanwhile, fewer records asked for than there are;
ensemble lattices of one and of several chunks.  Copies: every value is exact."""
import ctypes as C

import numpy as np
import pytest

from ch4b200 import abi
from lbcases import make_case, make_particles
from test_gpu_ensemble import rb_case

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import ch4b200  # noqa: E402

CHUNK = (1 << 20) // 2 // C.sizeof(abi.Particle)  # records of a half of the smallest staging buffer


def records(parts):
    return np.frombuffer(parts, dtype=np.float64).reshape(len(parts), -1)


@pytest.mark.parametrize("n", [1, 31, 32, 33, CHUNK - 1, CHUNK, CHUNK + 1, 3 * CHUNK + 5])
def test_particle_records(n):
    _, cfg, state = make_case("particles", seed=3, dims=(9, 8, 7))
    parts = make_particles(np.random.default_rng(n), n, 9, 8, 7)
    for i, p in enumerate(parts):
        p.tau_drag, p.beta_coeff, p.name = 0.0, 0.0, i  # tracers: nothing is deposited
    before = records((abi.Particle * n)(*parts))
    with ch4b200.Simulation(cfg) as sim:
        sim.set_pop("p", state["p"])
        sim.set_particles((abi.Particle * n)(*parts))
        assert np.array_equal(records(sim.get_particles(n)), before)
        sim.initialize()
        sim.step(17)  # the slots are in home-cell order now
        got = records(sim.get_particles(n))
        name = abi.PARTICLE_FIELDS.index("name")
        assert np.array_equal(got[:, name], before[:, name])
        moved = np.abs(got - before).max(axis=0) > 0
        assert moved[abi.PARTICLE_FIELDS.index("x")] and np.isfinite(got).all()
        some = n // 2 + 1
        assert np.array_equal(records(sim.get_particles(some)), got[:some])
        sim.set_particles((abi.Particle * n).from_buffer(got.copy()))
        assert np.array_equal(records(sim.get_particles(n)), got)


# 11 x 7 x 5: one chunk; 300 x 200 x 20: 24 MB of values, two chunks of planes
@pytest.mark.parametrize("dims", [[(11, 7, 5), (40, 3, 1)], [(33, 5, 2), (300, 200, 20)]])
def test_ensemble_fields(dims):
    cases = [rb_case(*d, 1e5, 5 + i) for i, d in enumerate(dims)]
    with ch4b200.Ensemble(abi.STORE_F32) as ens:
        slots = []
        for cfg, st in cases:
            s = ens.add(cfg)
            for k, v in st.items():
                ens.set_pop(s, k, v)
            ens.initialize(s)
            slots.append(s)
        ens.step(3)
        got = [ens.fields(s) for s in slots]
    for (cfg, st), g in zip(cases, got):
        with ch4b200.Simulation(cfg) as sim:
            for k, v in st.items():
                sim.set_pop(k, v)
            sim.initialize()
            sim.step(3)
            ref = sim.fields()
        for k in ref:
            assert np.abs(g[k] - ref[k]).max() <= 1e-6, k  # as the populations agree; a misplaced cell would not
