"""GPU test of the 8-lanes-per-cell re-binning and update kernels, which systems of at least
16,384 cells with at most 32 particles per cell on average run (others run a warp per cell):
a hot dilute gas beside a dense layer, so that cells hold 0 to about 60 particles and many
particles change cells every step, against engine_step_host (re-binning and update on the host
by the same rule) bit for bit, also through a block overflow and the Verlet skin's copies."""
import numpy as np
import pytest

import mdcore_b200 as M
import workloads as W

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
    """Everything drifts towards one corner cell layer: blocks outgrow their margin."""
    sysm = layered_gas(seed=6)
    sysm.v = (np.array([13.0, 13.0, 13.0]) - sysm.x) * 2.0
    e = M.Engine.from_system(sysm)
    e.resident_begin(4)
    for _ in range(6):
        e.resident_steps(5)
    info = e.resident_info()
    e.resident_end()
    x, v, f, c = e.parts()
    assert info.steps == 30 and info.regrows > 0, info
    assert (c >= 0).all() and np.isfinite(x).all()
    e.close()
