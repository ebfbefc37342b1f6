"""GPU test of the 8-lanes-per-cell re-binning and update kernels, which systems of at least
16,384 cells with at most 32 particles per cell on average run (others run a warp per cell):
a hot dilute gas beside a dense layer, so that cells hold 0 to about 60 particles and many
particles change cells every step, against engine_step_host (re-binning and update on the host
by the same rule) bit for bit, also through a block overflow and with rigid groups (the slots by
id), and with the Verlet skin's copies against the oracle."""
import numpy as np
import pytest

import mdcore_b200 as M
import oracle as O
import workloads as W
from helpers import tables_of

pytestmark = pytest.mark.gpu


def layered_gas(seed=4):
    s = W.lj_slab(nx=60, nz=10, n_total=60 * 60 * 10 + 9000, box=(26.0, 26.0, 26.0), slab=2.6, seed=seed)
    s.v = W.maxwell_velocities(s, 3000.0, seed=seed)
    return s


@pytest.mark.parametrize("graph", [False, True])
def test_resident_steps_equal_host_steps(graph):
    sysm = layered_gas()
    assert np.prod(np.floor(sysm.dim / sysm.L)) >= 16384
    a = M.Engine.from_system(sysm)
    a.graph(graph)
    a.resident_begin()
    a.resident_steps(6)
    a.resident_end()
    b = M.Engine.from_system(sysm)
    for _ in range(6):
        b.step_host()
    for x, y in zip(a.parts(), b.parts()):
        assert np.array_equal(x, y)
    a.close()
    b.close()


def test_block_overflow_regrows():
    """Everything drifts towards the middle of the box: blocks outgrow their margin."""
    sysm = layered_gas(seed=6)
    sysm.v = (np.array([13.0, 13.0, 13.0]) - sysm.x) * 2.0
    e = M.Engine.from_system(sysm)
    e.resident_begin(4)
    for _ in range(6):
        e.resident_steps(5)
    info = e.resident_info()
    e.resident_end()
    assert info.steps == 30 and info.regrows > 0, info
    h = M.Engine.from_system(sysm)
    for _ in range(30):
        h.step_host()
    for x, y in zip(e.parts(), h.parts()):
        assert np.array_equal(x, y)
    e.close()
    h.close()


def test_verlet_skin_copies():
    """Cells of 1.1 nm (a skin of 0.1 nm): between rebuilds the blocks are copied in order.  Every
    step's pairs are the oracle's on the same particles."""
    sysm = W.lj_slab(nx=60, nz=10, n_total=60 * 60 * 10 + 9000, box=(28.7, 28.7, 28.7), slab=3.0, seed=8)
    sysm.L = np.full(3, 1.1)
    sysm.v = W.maxwell_velocities(sysm, 500.0, seed=8)
    sysm.dt *= 0.2                  # some of the vapour starts in contact
    tables = tables_of(sysm)
    cdim = np.floor(sysm.dim / sysm.L).astype(np.int32)
    assert np.prod(cdim) >= 16384
    e = M.Engine.from_system(sysm, flags=M.engine_flag_cuda | M.engine_flag_verlet_pseudo)
    e.resident_begin()
    for _ in range(16):
        e.resident_sync()
        x, _, _, c = e.parts()
        o = O.nonbond(sysm, tables, binned=dict(cdim=cdim, h=sysm.dim / cdim, cell=c, xrel=x))
        before = e.resident_info().pairs
        e.resident_steps(1)
        assert e.resident_info().pairs - before == o["pairs"]
    assert 2 <= e.verlet_rebuilds() < 16, e.verlet_rebuilds()
    e.close()


def dilute(kind):
    if kind == "rigid water":       # every particle in a group: the constraint kernel updates them
        return W.with_rigid_water(W.water_spce(24, density=0.78, seed=2), 300.0)
    s = W.chains_water(nchains=60, length=20, nwater=2000, box=(32.0, 32.0, 32.0), seed=2, gap=0.25,
                       angles_dihedrals=False)
    s.bonds = None                  # engine_step_host has none
    s.v = W.maxwell_velocities(s, 50.0, seed=2)
    return s


@pytest.mark.parametrize("kind", ["rigid water", "water and free beads"])
def test_slots_by_id_of_rigid_systems(kind):
    sysm = dilute(kind)
    assert np.prod(np.floor(sysm.dim / sysm.L)) >= 16384
    a, b = M.Engine.from_system(sysm), M.Engine.from_system(sysm)
    a.resident_begin()
    a.resident_steps(6)
    a.resident_end()
    for _ in range(6):
        b.step_host()
    for x, y in zip(a.parts()[:2] + a.parts()[3:], b.parts()[:2] + b.parts()[3:]):
        assert np.array_equal(x, y)
    a.close()
    b.close()
