"""Read-backs from several threads: they take turns at the buffers of a handle (populations, fields
and particle records pass through the same one) and of an ensemble, so each gets what a single
thread gets.  Copies: every value is exact."""
import threading

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

ROUNDS = 25


def in_threads(reads):
    """Every read ROUNDS times in a thread of its own, all begun together; [results] per read."""
    out, errors, gate = [[] for _ in reads], [], threading.Barrier(len(reads))

    def work(k):
        try:
            gate.wait()
            for _ in range(ROUNDS):
                out[k].append(reads[k]())
        except Exception as e:  # reported by the caller's thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(reads))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    return out


@pytest.mark.parametrize("storage", [0, 1])
def test_one_handle(storage):
    _, cfg, state = make_case("particles", seed=4, storage=storage, dims=(40, 30, 20))
    n = 5000
    parts = make_particles(np.random.default_rng(1), n, 40, 30, 20)
    for p in parts:
        p.beta_coeff = 0.0  # nothing is deposited
    with ch4b200.Simulation(cfg) as sim:
        sim.set_pop("p", state["p"])
        sim.set_particles((abi.Particle * n)(*parts))
        sim.initialize()
        sim.step(3)
        reads = [lambda: sim.get_pop("p"), lambda: sim.fields()["u"], lambda: sim.fields()["dens"],
                 lambda: np.frombuffer(sim.get_particles(n), dtype=np.float64).copy()]
        alone = [r() for r in reads]
        for want, got in zip(alone, in_threads(reads)):
            assert all(np.array_equal(g, want) for g in got)


def test_slots_of_an_ensemble():
    dims = [(33, 20, 9), (70, 41, 5), (18, 64, 30)]
    with ch4b200.Ensemble(abi.STORE_F32) as ens:
        slots = []
        for i, d in enumerate(dims):
            cfg, st = rb_case(*d, 1e5, 9 + i)
            s = ens.add(cfg)
            for k, v in st.items():
                ens.set_pop(s, k, v)
            ens.initialize(s)
            slots.append(s)
        ens.step(3)
        reads = [lambda s=s, k=k: ens.fields(s)[k] for s in slots for k in ("u", "t")]
        alone = [r() for r in reads]
        for want, got in zip(alone, in_threads(reads)):
            assert all(np.array_equal(g, want) for g in got)
