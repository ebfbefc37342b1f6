"""GPU tests of the cell form of the persistent evaluation (sweep_cells: units of up to 32 i
particles of a cell against the j particles of all its tasks; MDB_SWEEP_FORM=cells selects it
as the autotuner otherwise does): pairs, exclusions and the sorted sweep's candidate count
exact, energy, virial and forces within the parity bounds of the oracle, at the sizes where
its strips, lists and masks end (cells of 0 to 90 particles, a cell of 1,000, a vapour, list
and mask exclusions, many tables), and the same results alone, in a batch,
resident and through engine_step.  Every test asserts the form that ran; the rules by which it is
chosen, its limits and its graphs have tests of their own."""
import ctypes as C

import numpy as np
import pytest

import mdcore_b200 as M
import oracle as O
import workloads as W
from helpers import force_errors, load_golden, tables_of
from test_gpu_edges import lj_system
from test_gpu_parity import cells_of_every_size, cells_of_every_size_2nm

pytestmark = pytest.mark.gpu


def one_large_cell():
    rng = np.random.default_rng(3)
    dense = rng.uniform(0.0, 1.0, size=(1000, 3))
    sparse = rng.uniform(0.0, 3.0, size=(200, 3))
    return lj_system(np.concatenate([dense, sparse[(sparse >= 1.0).any(axis=1)]]), L=3.0, scale=1e-4)


def far_exclusions():
    base, _ = load_golden("argon_1372.npz")
    rng = np.random.default_rng(5)
    pairs = set()
    while len(pairs) < 200:
        i, j = (int(v) for v in rng.integers(0, base.n, size=2))
        d = base.x[i] - base.x[j]
        d -= np.round(d / base.dim) * base.dim
        if i != j and (d ** 2).sum() < 0.8:
            pairs.add((i, j))
    return W.System(**{**base.__dict__, "excl": np.array(sorted(pairs), np.int32), "name": "argon-far-excl"})


def on_cell_faces():
    """Particles on the faces of their cells."""
    rng = np.random.default_rng(8)
    x = rng.uniform(0.0, 4.0, size=(1500, 3))
    x[:300, rng.integers(0, 3)] = np.round(x[:300, 0])
    return lj_system(np.mod(x, 4.0), L=4.0, scale=1e-4)


SYSTEMS = {
    "cells-0-40": cells_of_every_size,
    "cells-0-90": cells_of_every_size_2nm,
    "cell-1000": one_large_cell,
    "faces": on_cell_faces,
    "far-exclusions": far_exclusions,
    "water": lambda: W.water_spce(11, seed=2),
    "vapour": lambda: W.lj_slab(nx=22, nz=11, n_total=22 * 22 * 11 + 1000, box=(8.0, 8.0, 24.0), slab=4.0, seed=4),
    "dilute-water": lambda: W.water_spce(nside=8, density=1.0, seed=3),
    "chains": lambda: W.chains_water(nchains=4, length=20, nwater=150, box=(6.0, 6.0, 6.0), seed=2,
                                     angles_dihedrals=False),
    "single": lambda: lj_system(np.full((1, 3), 0.5)),
}


_ORACLE = {}


@pytest.mark.parametrize("cells", ["cells", "cells24"])
@pytest.mark.parametrize("name", SYSTEMS)
def test_cell_form_vs_oracle_and_queue_form(name, cells, monkeypatch):
    sysm = SYSTEMS[name]()
    if name not in _ORACLE:
        _ORACLE[name] = O.nonbond(sysm, tables_of(sysm))
    o = _ORACLE[name]
    out = {}
    for form in (cells, "queue"):
        monkeypatch.setenv("MDB_SWEEP_FORM", form)
        e = M.Engine.from_system(sysm)
        e.nonbond()
        assert e.form() == (("queue", 0) if form == "queue" else ("cells", 24 if form == "cells24" else 32)) + (False,)
        out[form] = e.forces(), e.stats(), [e.sortkeys(c, int((e.cells() == c).sum())) for c in (0, 1, 5)]
        e.close()
    f, st, keys = out[cells]
    q = out["queue"][1]
    assert st.status == 0
    assert (st.pairs, st.excluded, st.candidates) == (o["pairs"], o["excluded"], q.candidates)
    assert abs(st.epot - o["epot"]) <= 1e-6 * o["epot_abs"] and abs(st.virial - o["virial"]) <= 1e-6 * o["virial_abs"]
    if st.pairs:
        err = force_errors(f, o["f"])
        assert err["global_rel"] <= 2e-6 and err["max_over_frms"] <= 2e-5, err
    assert all(np.array_equal(a, b) for a, b in zip(keys, out["queue"][2]))     # sorted on demand


@pytest.mark.parametrize("name", ["water", "replicas"])
def test_cell_form_is_the_same_alone_in_a_batch_and_resident(name, monkeypatch):
    monkeypatch.setenv("MDB_SWEEP_FORM", "cells")
    systems = [W.with_rigid_water(W.water_spce(10), 300.0)] if name == "water" else W.argon_replicas(5, seed=9)
    for s in systems:
        if s.v is None:
            s.v = W.maxwell_velocities(s, 100.0, seed=1)
    engines = [M.Engine.from_system(s, start=False) for s in systems]
    b = M.Batch(engines)
    b.graph(True)
    b.resident_begin().resident_steps(7)
    assert b.form()[:2] == ("cells", 32)
    b.resident_sync()
    for s, r in zip(systems, engines):
        e = M.Engine.from_system(s)
        for _ in range(7):
            e.step()
        assert e.form().name == "cells"
        assert all(np.array_equal(x, y) for x, y in zip(e.parts(), r.parts()))
        assert e.energies() == r.energies()
        st = e.stats()
        if len(systems) == 1:
            assert st.candidates == b.stats().candidates
        e.close()
    b.close()


def test_candidates_of_the_last_step_of_every_call(monkeypatch):
    """The count is taken in the last step of a call only; it is the queue form's."""
    sysm = W.argon_fcc(7, jitter=0.05)
    sysm.v = W.maxwell_velocities(sysm, 150.0, seed=3)
    got = {}
    for form in ("cells", "queue"):
        monkeypatch.setenv("MDB_SWEEP_FORM", form)
        e = M.Engine.from_system(sysm)
        e.graph(True)
        e.resident_begin()
        got[form] = []
        for k in (1, 3, 1, 2):
            e.resident_steps(k)
            e.resident_sync()
            got[form].append((e.stats().pairs, e.stats().candidates))
            assert e.form().name == form
        e.close()
    assert got["cells"] == got["queue"]


def test_steps_of_several_tables_keep_the_queue_form(monkeypatch):
    """Default engines of many tables: force evaluations run the cell form, time steps (device
    and host-threaded) give the queue form's trajectory bit for bit."""
    sysm = chain_mix()
    out = []
    for form, host in ((None, False), (None, True), ("queue", False)):
        if form:
            monkeypatch.setenv("MDB_SWEEP_FORM", form)
        e = M.Engine.from_system(sysm)
        for _ in range(3):
            e.step_host() if host else e.step()
            assert e.form().name == "queue"
        out.append(e.parts())
        e.nonbond()
        assert e.form().name == (form or "cells")
        e.close()
    for other in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(out[0][:2], other[:2]))


def chain_mix():
    """Many tables, few large cells, no bonds: force evaluations run the cell form by default, steps
    the queue form."""
    s = W.chains_water(nchains=6, length=20, nwater=900, box=(4.0, 4.0, 4.0), seed=2, gap=0.3,
                       angles_dihedrals=False)
    s.bonds = None
    return s


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("calls", ["step, nonbond", "nonbond, resident steps", "nonbond, resident steps, end",
                                   "resident steps, nonbond, end"])
def test_keys_of_mixed_calls_are_the_queue_forms(calls, graph, monkeypatch):
    """Host evaluations and resident steps have sort keys of their own; an engine whose evaluations
    run the cell form and whose steps run the queue form answers as one of the queue form only."""
    out = []
    for form in (None, "queue"):
        if form:
            monkeypatch.setenv("MDB_SWEEP_FORM", form)
        e = M.Engine.from_system(chain_mix())
        e.graph(graph)
        for call in calls.split(", "):
            if call == "resident steps":
                e.resident_begin()
                e.resident_steps(5)
            else:
                for _ in range(1 if call == "end" else 4):
                    {"step": e.step, "nonbond": e.nonbond, "end": e.resident_end}[call]()
        counts = np.bincount(e.cells(), minlength=8)
        keys = [] if "end" in calls else [e.sortkeys(c, int(counts[c])) for c in range(8)]
        out.append(keys + [e.sched_features()])
        e.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))


def positions(e):
    """The engine's own cell-relative position (3 floats) of every particle by id."""
    partlist = C.c_void_p.from_address(e.ptr.value + 8 + 168).value     # struct space, after its flags
    out = []
    for i, p in enumerate((C.c_void_p * e.n).from_address(partlist)):
        assert C.c_int.from_address(p + 52).value == i                  # struct part: id
        out.append(np.frombuffer((C.c_float * 3).from_address(p), np.float32))
    return out


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 1e12])
@pytest.mark.parametrize("name", ["far-exclusions", "water", "chains"])
def test_non_finite_positions_have_no_pairs(name, bad, monkeypatch):
    """Particles at every place of a cell's list lost to infinity, or far away and from each other:
    no pairs and no force of their own, the others' forces those of the queue form."""
    sysm = SYSTEMS[name]()
    out = {}
    for form in ("queue", "cells", "cells24"):
        monkeypatch.setenv("MDB_SWEEP_FORM", form)
        e = M.Engine.from_system(sysm)
        x = positions(e)
        c = e.cells()
        lost = [np.flatnonzero(c == k)[k % 24] for k in range(c.max() + 1) if (c == k).sum() > k % 24]
        lost += [i for k in range(0, c.max() + 1, 3) for i in np.flatnonzero(c == k)[:1]]
        for k, i in enumerate(lost):
            x[i][k % 3] = bad * (k + 1)
        e.nonbond()
        assert e.form().name == form[:5]
        st = e.stats()
        out[form] = e.forces(), (st.status, st.pairs, st.excluded, st.candidates), st.epot
        e.close()
    f0, counts, epot = out["queue"]
    assert counts[0] == 0 and counts[1] > 1000 and not f0[lost].any()
    for form in ("cells", "cells24"):
        f, n, ep = out[form]
        assert n == counts and abs(ep - epot) <= 2e-6 * abs(epot)
        err = force_errors(f, f0)          # each form within the parity bounds (2e-6, 2e-5) of the exact forces
        assert err["global_rel"] <= 4e-6 and err["max_over_frms"] <= 4e-5, err


def test_autotuner_choice_and_what_undoes_it():
    """A large system of one table is tuned to the cell form (some 20 % ahead there); the returned
    shape stands for it, any other shape and a queue order given afterwards select the queue form."""
    e = M.Engine.from_system(W.argon_fcc(30, seed=1, jitter=0.02))
    e.nonbond()
    assert e.form() == ("queue", 0, False)
    warps, layout, stages, occupancy, _ = e.autotune(5)

    def form():
        e.nonbond()
        return e.form().name

    assert form() == "cells" and e.form().rows in (24, 32)
    e.set_layout(layout, stages, occupancy)
    assert form() == "cells"
    e.set_layout(1 - layout, 1, 640)
    assert form() == "queue"
    e.set_layout(layout, stages, occupancy)
    assert form() == "cells"
    e.set_order(e.get_order())
    assert form() == "queue"
    for other, same in (((e.tune, 4 if warps != 4 else 8), (e.tune, warps)), ((e.set_window, 8), (e.set_window, 4))):
        other[0](other[1])
        assert form() == "queue"
        e.set_layout(layout, stages, occupancy)
        assert form() == "queue"              # not the whole shape
        same[0](same[1])
        assert form() == "cells"
    e.tune(0, plain=True)
    assert form() == "plain"
    e.tune(0)
    assert form() == "cells"
    e.close()


def test_launch_shapes_select_the_queue_form_untuned():
    """An engine whose evaluations run the cell form by default."""
    for give in (lambda e: e.tune(8), lambda e: e.tune(4), lambda e: e.set_window(8), lambda e: e.set_layout(1),
                 lambda e: e.set_layout(0)):
        e = M.Engine.from_system(chain_mix())
        e.nonbond()
        assert e.form().name == "cells"
        e.tune(0)
        e.nonbond()
        assert e.form().name == "cells"
        give(e)
        e.nonbond()
        assert e.form().name == "queue"
        e.close()


def test_task_clocks_run_the_queue_form(monkeypatch):
    monkeypatch.setenv("MDB_SWEEP_FORM", "cells")
    e = M.Engine.from_system(W.argon_fcc(7))
    e.task_clocks(True)
    e.nonbond()
    assert e.form().name == "queue" and (e.task_clocks(True, read=True)[0] > 0).any()
    e.close()


@pytest.mark.parametrize("graph", [False, True])
def test_on_a_stream_of_the_caller(graph, monkeypatch):
    """The candidate count's own stream forks from and joins whatever stream is set."""
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("MDB_SWEEP_FORM", "cells")
    sysm = W.argon_fcc(10, seed=2, jitter=0.05)
    sysm.v = W.maxwell_velocities(sysm, 150.0, seed=3)
    out = []
    for stream in (None, torch.cuda.Stream()):
        e = M.Engine.from_system(sysm)
        e.graph(graph)
        if stream:
            e.set_stream(stream.cuda_stream)
        for _ in range(4):
            e.nonbond()
        counts = e.stats().candidates
        for _ in range(5):
            e.step()
        assert e.form() == ("cells", 32, graph)
        out.append([counts, e.stats().candidates, *e.parts()])
        e.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))


def test_grouped_batch_steps(monkeypatch):
    monkeypatch.setenv("MDB_SWEEP_FORM", "cells")
    out = []
    for groups in (1, 3):
        systems = W.argon_replicas(7, seed=5)
        for k, s in enumerate(systems):
            s.v = W.maxwell_velocities(s, 100.0, seed=k)
        engines = [M.Engine.from_system(s, start=False) for s in systems]
        b = M.Batch(engines)
        b.set_groups(groups)
        for _ in range(4):
            b.step()
        assert b.form().name == "cells"
        out.append([b.stats().pairs, b.stats().candidates] + [a for e in engines for a in e.parts()])
        b.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))


def test_shares_of_a_large_cell_in_resident_steps(monkeypatch):
    """A cell of 1,000 particles: its strips' j particles are split between units, in resident
    steps as in host-buffer evaluations."""
    monkeypatch.setenv("MDB_SWEEP_FORM", "cells")
    sysm = one_large_cell()
    sysm.v = W.maxwell_velocities(sysm, 50.0, seed=1)
    out = []
    for host in (False, True):
        e = M.Engine.from_system(sysm)
        if host:
            for _ in range(5):
                e.step_host()
        else:
            e.resident_begin().resident_steps(5).resident_end()
        assert e.form().name == "cells"
        out.append(e.parts())
        e.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("graph", [False, True])
def test_an_overflowing_unit_list_is_an_error(graph, monkeypatch):
    """Units past the list's room are dropped and reported, and none past it is read."""
    monkeypatch.setenv("MDB_SWEEP_FORM", "cells")
    sysm = W.argon_fcc(10, seed=2, jitter=0.05)
    e = M.Engine.from_system(sysm)
    e.graph(graph)
    for _ in range(3):
        e.nonbond()
    f, pairs = e.forces(), e.stats().pairs
    for units in (1, 50):
        e.celllimits_test(units=units)
        for _ in range(3):
            with pytest.raises(M.MdcoreError, match="Max. number of parts per cell"):
                e.nonbond()
            assert e.stats().status == 2 and 0 < e.stats().pairs < pairs
    e.celllimits_test()
    for _ in range(3):
        e.nonbond()
        assert np.array_equal(e.forces(), f) and e.stats().pairs == pairs
    e.celllimits_test(units=1)
    with pytest.raises(M.MdcoreError, match="Max. number of parts per cell"):
        e.step()
    e.close()


@pytest.mark.parametrize("graph", [False, True])
def test_more_slots_than_the_cell_form_numbers(graph, monkeypatch):
    """The slot limit (lowered here) is looked at for every evaluation on its own, on host buffers
    and in resident blocks, and blocks past it do not switch the form off for later ones."""
    monkeypatch.setenv("MDB_SWEEP_FORM", "cells")
    e = M.Engine.from_system(W.argon_fcc(10, seed=2, jitter=0.05))
    e.graph(graph)
    slots = int(((np.bincount(e.cells()) + 3) // 4 * 4).sum())

    def forms():
        out = []
        for _ in range(3):
            e.nonbond()
            out.append(e.form().name)
        for margin in (0, 400):
            e.resident_begin(margin)
            e.resident_steps(5)
            out.append(e.form().name)
            e.resident_end()
        return out

    assert forms() == ["cells"] * 5
    e.celllimits_test(slots=slots // 2)
    assert forms() == ["queue"] * 5
    e.celllimits_test(slots=3 * slots)
    assert forms() == ["cells"] * 4 + ["queue"]
    assert forms() == ["cells"] * 4 + ["queue"]
    e.celllimits_test()
    assert forms() == ["cells"] * 5
    e.close()


@pytest.mark.parametrize("form", ["queue", "cells", "cells24"])
@pytest.mark.parametrize("ncell", [7, 30])
def test_the_autotuner_keeps_the_form_asked_for(form, ncell, monkeypatch):
    """MDB_SWEEP_FORM overrides the autotuner's choice (by itself the queue form for the small
    system, the cell form for the large one)."""
    monkeypatch.setenv("MDB_SWEEP_FORM", form)
    e = M.Engine.from_system(W.argon_fcc(ncell, seed=1, jitter=0.02))
    _, layout, stages, occupancy, _ = e.autotune(3)
    want = {"queue": ("queue", 0), "cells": ("cells", 32), "cells24": ("cells", 24)}[form]
    assert e.form()[:2] == want
    e.nonbond()
    assert e.form()[:2] == want
    e.step()
    assert e.form()[:2] == want
    e.set_layout(layout, stages, occupancy)
    e.nonbond()
    assert e.form()[:2] == want
    e.close()


def test_the_autotuners_time_is_an_evaluations():
    """The cell form is timed with its candidate count, which every evaluation takes (without it
    these replicas' evaluations come out 22 % shorter than they are)."""
    engines = [M.Engine.from_system(s, start=False) for s in W.argon_replicas(64, seed=64)]
    b = M.Batch(engines)
    b.load_parts()
    ms = b.autotune(15)[4]
    assert b.form().name == "cells"
    t = []
    for _ in range(15):
        b.resident()
        t.append(b.kernel_times()[0])
    assert 0.9 * np.median(t) < ms < 1.1 * np.median(t), (ms, t)
    b.close()


def test_alternating_forms_replay_a_graph_each():
    """Force evaluations (cell form) and host-threaded steps (queue form) of one engine in turn: each
    is captured at its second launch and replayed from then on (the steps are too short for a
    particle to change cells)."""
    sysm = chain_mix()
    sysm.dt = 1e-9
    out = []
    for graph in (True, False):
        e = M.Engine.from_system(sysm)
        e.graph(graph)
        for k in range(4):
            e.nonbond()
            assert e.form() == ("cells", 24, graph and k > 0)
            e.step_host()
            assert e.form() == ("queue", 0, graph and k > 0)
        out.append(e.parts())
        e.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("cells, per_cell, form", [(3, 60, "queue"), (3, 100, "cells"), (6, 100, "cells"),
                                                   (7, 100, "queue")])
def test_default_form_by_number_and_size_of_cells(cells, per_cell, form):
    """Tables in global memory: the cell form where the queue form's tasks are few and large."""
    n = 22 * (cells ** 3 * per_cell // 22)
    s = W.chains_water(nchains=1, length=22, nwater=0, box=(1.2 * cells + 0.01,) * 3, seed=2, angles_dihedrals=False)
    rng = np.random.default_rng(1)
    s.x = rng.uniform(0.0, 1.2 * cells, size=(n, 3))
    s.type = np.tile(np.arange(22, dtype=np.int32), n // 22)
    s.q = np.zeros(n)
    s.excl, s.bonds, s.rigid = np.zeros((0, 2), np.int32), None, None
    e = M.Engine.from_system(s)
    e.load_parts()
    e.resident()
    assert e.form().name == form
    e.close()


@pytest.mark.parametrize("form", ["queue", "cells"])
def test_evaluation_inside_a_capture_of_the_caller(form, monkeypatch):
    """Uploaded particles are evaluated without an allocation, whatever has changed since the device
    state was built, so that a caller can capture the evaluation on its own stream."""
    torch = pytest.importorskip("torch")
    if form == "queue":
        monkeypatch.setenv("MDB_SWEEP_FORM", form)
    sysm = chain_mix()                                   # steps run the queue form
    sysm.rigid = None
    sysm.v = W.maxwell_velocities(sysm, 600.0, seed=3)
    e = M.Engine.from_system(sysm)
    most = np.bincount(e.cells()).max()
    while np.bincount(e.cells()).max() < most + 4:       # larger cells than at first
        e.resident_begin().resident_steps(5).resident_end()
    stream = torch.cuda.Stream()
    e.set_stream(stream.cuda_stream)
    e.load_parts()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        e.resident()
    assert e.form() == (form, 24 if form == "cells" else 0, False)
    g.replay()
    torch.cuda.synchronize()
    e.unload_parts()
    f, pairs = e.forces(), e.stats().pairs
    e.set_stream(0)
    e.nonbond()
    assert np.array_equal(e.forces(), f) and e.stats().pairs == pairs
    del g
    e.close()
