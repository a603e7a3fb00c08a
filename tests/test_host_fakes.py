"""The host code of the library (csrc/ch4_host.cpp) over a faked CUDA runtime and faked kernel
launchers (host_fakes.cpp): what it launches, in which order, and what it leaves behind when a
call fails.  No GPU; the failures are error codes that a fake returns."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from ch4b200 import abi
from lbcases import make_case

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
CUDA_INC = "/usr/local/cuda/include"

if not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime.h")):
    pytest.skip("no CUDA headers", allow_module_level=True)


@pytest.fixture(scope="module")
def fakes(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fakes") / "libfakes.so")
    csrc = os.path.join(REPO, "ch4-project_b200", "csrc")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", CUDA_INC, "-I", csrc,
                    os.path.join(csrc, "ch4_host.cpp"), os.path.join(csrc, "h5file.cpp"),
                    os.path.join(HERE, "host_fakes.cpp"), "-o", so], check=True)
    L = C.CDLL(so)
    L.fake_log.restype = L.fake_faults.restype = C.c_char_p
    L.fake_refuse.argtypes = [C.c_size_t]
    return L


class Handle:
    """A handle of the faked library holding a case's populations and particles."""

    def __init__(self, L, cfg, state):
        self.L, self.h, self.cfg = L, C.c_void_p(), cfg
        L.fake_reset()
        assert L.ch4_create(C.byref(cfg), C.byref(self.h)) == 0
        for k in ("p", "g", "h"):
            if k in state:
                a = np.ascontiguousarray(state[k])
                assert L.ch4_set_pop(self.h, C.c_char(k.encode()), a.ctypes.data_as(C.c_void_p), 0) == 0

    def set_particles(self, parts):
        assert self.L.ch4_set_particles(self.h, parts, len(parts)) == 0

    def initialize(self):
        assert self.L.ch4_initialize(self.h) == 0

    def step(self, n=1):
        return self.L.ch4_step(self.h, n)

    def log(self):
        out = self.L.fake_log().decode().split("\n")[:-1]
        faults = self.L.fake_faults().decode()
        self.L.fake_reset()
        assert faults == ""
        return out

    def close(self):
        self.L.ch4_destroy(self.h)


@pytest.fixture
def handle(fakes):
    made = []

    def make(name, **over):
        _, cfg, state = make_case(name, seed=1, **over)
        made.append(Handle(fakes, cfg, state))
        return made[-1], state

    yield make
    for h in made:
        h.close()


@pytest.mark.parametrize("name", ["kolmogorov", "les_vd", "cpower", "particles", "particles_tc"])
def test_uploads_are_ordered_with_the_steps(handle, name):
    """Every table, clear and upload is ordered with the first launch that may read it."""
    h, state = handle(name)
    if "part" in state:
        h.set_particles(state["part"])
    h.initialize()
    assert h.step(3) == 0
    if "part" in state:
        h.set_particles(state["part"])
        assert h.step(2) == 0
        h.set_particles((abi.Particle * 0)())
        assert h.step(2) == 0
    h.log()


def test_ensemble_tables_are_ordered_with_the_steps(fakes):
    _, cfg, state = make_case("kolmogorov", seed=1)
    fakes.fake_reset()
    ens, slot = C.c_void_p(), C.c_int()
    assert fakes.ch4_ensemble_create(abi.STORE_F32, C.c_size_t(1 << 30), C.byref(ens)) == 0
    assert fakes.ch4_ensemble_add(ens, C.byref(cfg), C.byref(slot)) == 0
    assert fakes.ch4_ensemble_initialize(ens, slot) == 0
    assert fakes.ch4_ensemble_step(ens, 3) == 0
    assert fakes.fake_faults().decode() == ""
    fakes.ch4_ensemble_destroy(ens)


EXCHANGE = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_size_t, C.c_void_p, C.c_void_p)


@pytest.mark.parametrize("name", ["particles_1w", "particles"])
@pytest.mark.parametrize("removed", [False, True])
def test_slab_without_particles(fakes, name, removed):
    """A slab whose lattice never had particles, or has lost them, has no exchange buffers: it
    steps without them (and clears its deposit)."""
    _, cfg, state = make_case(name, seed=1, dims=(6, 5, 8))
    cfg.nz_global, cfg.z_offset, cfg.NZ = 8, 0, 4
    state["p"] = state["p"][:4]
    h = Handle(fakes, cfg, state)
    moved = EXCHANGE(lambda *a: 0)
    assert fakes.ch4_set_exchange(h.h, moved, None) == 0 and fakes.ch4_set_face_exchange(h.h, moved, None) == 0
    if removed:
        h.set_particles(state["part"])
    h.initialize()
    if removed:
        assert h.step(2) == 0
        h.set_particles((abi.Particle * 0)())
    h.log()
    assert h.step(3) == 0
    log = h.log()
    assert log.count("launch_step") == 6  # the face planes, then the interior
    assert not any("ghosts" in x or "leave" in x or "arrive" in x for x in log)
    if name == "particles":
        assert log.count("launch_deposit stage 0") == (3 if removed else 2)
    h.close()


@pytest.mark.parametrize("storage,at,word", [(0, (0, 0), 8), (0, (4, 0), 4), (0, (0, 12), 4), (0, (8, 2), 2), (1, (4, 8), 4),
                                             (1, (0, 6), 2), (2, (2, 0), 2), (0, (1, 0), None), (2, (0, 3), None)])
def test_face_buffers_of_any_alignment(fakes, storage, at, word):
    """Face buffers aligned to less than a stored value go through narrower words; an odd
    address is refused."""
    _, cfg, state = make_case("rb", seed=1, storage=storage)
    h = Handle(fakes, cfg, state)
    h.log()
    down, up = (C.c_void_p((1 << 20) + a) for a in at)
    for call in (fakes.ch4_halo_pack, fakes.ch4_halo_unpack):
        assert call(h.h, down, up) == (abi.ERR_ARG if word is None else abi.OK)
        assert h.log() == ([] if word is None else ["launch_halo_faces word %d" % word])
    h.close()


@pytest.mark.parametrize("failing", ["launch_step", "launch_hydro", "launch_deposit", "launch_particle_substep"])
def test_deposit_after_a_failed_step_takes_the_state(handle, fakes, failing):
    """The lists that the last sub-step began serve one deposit.  A step that fails after it, or
    in it, is followed by a deposit that lists the particles itself, from cleared counters."""
    h, state = handle("particles")
    h.set_particles(state["part"])
    h.initialize()
    assert h.step(3) == 0
    assert h.log().count("launch_deposit stage 0 ready") == 2
    fakes.fake_fail(failing.encode())
    assert h.step() != 0
    bins = (h.cfg.NY + 1) * (h.cfg.NZ + 1)
    failed = h.log()
    assert ("clear %d" % (4 * (bins + 1)) in failed) == (failing == "launch_deposit")
    assert h.step() == 0
    assert [x for x in h.log() if "deposit" in x] == ["launch_deposit stage 0"]
    assert h.step() == 0
    assert "launch_deposit stage 0 ready" in h.log()


def test_u_of_the_les_after_a_failed_step(handle, fakes):
    """With particles the LES takes u^n from the vectors the last step formed for them; where
    that step failed before it formed them, u^n is computed."""
    h, state = handle("particles_1w")
    h.cfg.flags |= abi.FLAGS["LB_FLUID_LES"]
    les = Handle(fakes, h.cfg, {"p": state["p"]})
    les.initialize()
    les.log()
    counts = []
    for fail in (False, False, True, False, False):
        if fail:
            fakes.fake_fail(b"launch_hydro")
        assert (les.step() != 0) == fail
        counts.append(les.log().count("launch_hydro"))
    assert counts == [2, 1, 1, 2, 1]
    les.close()


LOOK = 256  # steps between two looks at the lists: every 16th re-sort


def routes(h):
    """Steps that deposited by home cells, among the deposits since the last call."""
    return ["cells" in x for x in h.log() if "deposit" in x]


def crowd(parts, cfg, rows):
    """The particles, all depositing, in one home row or spread."""
    parts = type(parts)(*parts)
    for i, p in enumerate(parts):
        p.tau_drag, p.beta_coeff = 1.0, 1.0
        p.y, p.z = (2.0, 2.0) if rows else (i % cfg.NY + 0.5, i // cfg.NY % cfg.NZ + 0.5)
    return parts


def test_deposit_route_follows_the_longest_list(handle, fakes):
    """At ch4_set_particles by the positions, then at every look by the figure of the one before."""
    fakes.fake_longest(0)
    h, state = handle("particles")
    h.set_particles(crowd(state["part"], h.cfg, True))  # 300 particles in one row
    h.initialize()
    assert h.step(2 + LOOK - 1) == 0
    assert routes(h) == [True] * LOOK  # the first step deposits nothing
    assert h.step(1) == 0  # the first look found no long list
    assert routes(h) == [False]
    fakes.fake_longest(91)
    assert h.step(LOOK) == 0  # longer than to return to rows, not than to leave them
    assert routes(h) == [False] * LOOK
    fakes.fake_longest(121)
    assert h.step(LOOK) == 0
    assert routes(h) == [False] * LOOK
    fakes.fake_longest(91)
    assert h.step(LOOK) == 0
    assert routes(h) == [False] * (LOOK - 1) + [True]
    assert h.step(LOOK) == 0
    assert routes(h) == [True] * LOOK
    h.set_particles(crowd(state["part"], h.cfg, False))
    assert h.step(1) == 0
    assert routes(h) == [False]
    h.set_particles((abi.Particle * 0)())
    assert h.step(2) == 0
    h.set_particles(crowd(state["part"], h.cfg, True))
    assert h.step(1) == 0
    assert routes(h) == [False, False, True]
    fakes.fake_longest(0)


def test_deposit_stays_by_rows_without_memory(handle, fakes):
    """Where the buffers of the home cells are refused the deposit goes by rows as before, and
    takes them when there is room."""
    h, state = handle("particles")
    parts = crowd(state["part"], h.cfg, True)
    h.set_particles(crowd(state["part"], h.cfg, False))
    h.initialize()
    h.log()
    for refused in (1, 8 * 9 * len(parts)):  # the first buffer, and the last
        fakes.fake_refuse(refused)
        h.set_particles(parts)
        assert h.step(2) == 0
        fakes.fake_refuse(0)
        assert not any(routes(h))
    h.set_particles(parts)
    assert h.step(1) == 0
    assert routes(h) == [True]
