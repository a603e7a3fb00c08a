"""The two-way deposit by lattice rows (csrc/deposit_rows.cuh) where its lists are unusual:
rows of two and three segments (particles at the segment ends included), lists longer than
the chunk that a warp merges at a time, runs that re-sort the slots, a particle count that
leaves most lists empty, and uploads in the middle of a run.  FP64, bit-identical to the
restatement; FP32 the same from call to call."""
import numpy as np
import pytest

import oracle as O
from ch4b200 import abi
from lbcases import make_case, make_particles, run_restatement

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import ch4b200  # noqa: E402


def small_particles(rng, n, size, box, at=None):
    """Inertial particles (radius small against a cell) and tracers in the corner `box`."""
    parts = make_particles(rng, n, *size)
    for i, p in enumerate(parts):
        p.tau_drag = [0.8, 0.0, 1.5, 1.0][i % 4]
        p.beta_coeff = [1.0, 0.5, 0.0][i % 3]
        p.x, p.y, p.z = (rng.random() * b for b in box)
        if at and i % 3 == 0:  # about the homes at a segment's end
            p.x = at[i % len(at)] + 0.9 * (rng.random() - 0.5)
    return parts


CASES = {
    "segments": dict(dims=(530, 3, 3), n=700, box=(530, 3, 3), at=(255.5, 256.5, 511.5, 512.5, 0.3, 529.7), steps=6),
    "dense": dict(dims=(10, 8, 7), n=600, box=(2, 2, 2), at=None, steps=3),
    "dense_segments": dict(dims=(300, 4, 3), n=500, box=(300, 2, 2), at=(255.6, 256.2), steps=3),
    "sparse": dict(dims=(40, 9, 8), n=5, box=(40, 9, 8), at=None, steps=10),
}


def run(cfg, state, parts, steps):
    with ch4b200.Simulation(cfg) as sim:
        sim.set_pop("p", state["p"])
        sim.set_particles(parts)
        sim.initialize()
        sim.step(1)
        sim.set_particles(sim.get_particles(len(parts)))  # the state as it is, re-uploaded
        sim.step(steps - 1)
        return sim.get_pop("p"), O.particles_as_dict(sim.get_particles(len(parts)))


@pytest.mark.parametrize("name", sorted(CASES))
def test_rows_bit_identical(name):
    c = CASES[name]
    _, cfg, state = make_case("particles", seed=2, dims=c["dims"])
    parts = small_particles(np.random.default_rng(7), c["n"], c["dims"], c["box"], c["at"])
    ref = run_restatement(cfg, dict(state, part=parts), c["steps"])
    assert np.isfinite(ref["p"]).all()
    p, got = run(cfg, state, parts, c["steps"])
    assert np.array_equal(p, ref["p"])
    for k, v in ref["part"].items():
        assert np.array_equal(got[k], v), k


@pytest.mark.parametrize("nx,ends", [(257, (128, 256)), (300, (128, 256)), (512, (128, 256, 384)), (515, (128, 384, 512))])
@pytest.mark.parametrize("n,steps", [(150, 6), (900, 3)])
def test_cut_rows(nx, ends, n, steps):
    """Rows of three to five segments, a third of the particles about the segments' ends: in the
    lists of the segment and in the edge lists of the one before; up to and beyond the 32 and the
    64 entries that a warp takes at once."""
    dims = (nx, 4, 3)
    _, cfg, state = make_case("particles", seed=2, dims=dims)
    at = tuple(e + d for e in ends for d in (0.0, 0.5, 1.0))
    parts = small_particles(np.random.default_rng(nx), n, dims, (nx, 2, 2), at)
    ref = run_restatement(cfg, dict(state, part=parts), steps)
    assert np.isfinite(ref["p"]).all()
    p, got = run(cfg, state, parts, steps)
    assert np.array_equal(p, ref["p"])
    for k, v in ref["part"].items():
        assert np.array_equal(got[k], v), k


def flyers(n, size, gather):
    """Heavy particles that keep their velocity: towards the middle, where they meet after 100
    steps, or out of two home rows."""
    rng = np.random.default_rng(n)
    parts = make_particles(rng, n, *size)
    for i, p in enumerate(parts):
        p.tau_drag, p.beta_coeff = 1e4, 1e-9 * (1 + i % 3)
        for a, s in zip("xyz", size):
            v = 0.1 * (rng.random() - 0.5)
            if gather:
                v = (0.5 * s + 0.25 - getattr(p, a)) / 100
            elif a != "x":
                setattr(p, a, 2.0 + rng.random())
            setattr(p, "v" + a, v)
    return parts


@pytest.mark.parametrize("gather", [False, True])
@pytest.mark.parametrize("size", [(10, 8, 7), (260, 5, 4)])
def test_both_routes_and_their_change(size, gather):
    """Lists beyond the limit deposit by home cells: from the upload on where the particles are
    gathered then, and from the second look after they have met.  530 steps hold looks at 2, 258
    and 514.  Bit-identical to the restatement all the way."""
    _, cfg, state = make_case("particles", seed=2, dims=size, time_dt_lagr_factor=1.0, Amp_x=1e-5, Amp_y=1e-5,
                              Amp_z=1e-5)
    parts = flyers(600, size, gather)
    with ch4b200.Simulation(cfg) as sim:
        ref = O.Restatement(cfg)
        for s in (ref, sim):
            s.set_pop("p", state["p"])
            s.set_particles(parts)
            s.initialize()
        for steps in (5, 525):
            ref.step(steps)
            sim.step(steps)
            want = ref.get_pop("p")
            assert np.isfinite(want).all()
            assert np.array_equal(sim.get_pop("p"), want)
            assert np.abs(sim.force() - ref.force()).max() == 0
            got, want = (O.particles_as_dict(s.get_particles(len(parts))) for s in (sim, ref))
            for k, v in want.items():
                assert np.array_equal(got[k], v), k
        ref.close()


@pytest.mark.parametrize("name", ["segments", "dense"])
def test_rows_f32_reproducible(name):
    c = CASES[name]
    _, cfg, state = make_case("particles", seed=2, dims=c["dims"], storage=1)
    parts = small_particles(np.random.default_rng(7), c["n"], c["dims"], c["box"], c["at"])
    a, b = run(cfg, state, parts, c["steps"]), run(cfg, state, parts, c["steps"])
    assert np.array_equal(a[0], b[0])
    assert all(np.array_equal(a[1][k], b[1][k]) for k in a[1])


@pytest.mark.parametrize("name", ["particles", "particles_tc", "particles_tt"])
def test_nothing_deposits_once_the_particles_are_removed(name):
    """By rows, by home cells (tricubic) and with the heat deposit; bit-identical to the
    restatement, whose particles are removed at the same step."""
    _, cfg, state = make_case(name, seed=8)
    sets = [k for k in ("p", "g") if k in state]
    none = (abi.Particle * 0)()
    ref = O.Restatement(cfg)
    with ch4b200.Simulation(cfg) as sim:
        for s in (ref, sim):
            for k in sets:
                s.set_pop(k, state[k])
            s.set_particles(state["part"])
            s.initialize()
            s.step(6)
            s.set_particles(none)
            s.step(5)
        for k in sets:
            assert np.array_equal(sim.get_pop(k), ref.get_pop(k)), k
    ref.close()
