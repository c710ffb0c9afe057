"""The matrix of a Newton iteration on the device: the closed forms of the fully wet elements, their
gather and their Dirichlet rows, which sw2gpu_load (the differenced Jacobian) does not launch; the
launch variants of the differenced kernel where steps do use it; and what the autotuner leaves alone."""
import dataclasses

import numpy as np
import pytest

from adhv8_kraken_b200 import capi, meshgen
from adhv8_kraken_b200.model import BCT_VEL_DIR, BCT_VEL_PRS_DIR, Series, StringSpec
from adhv8_kraken_b200.sw2 import SW2GPU, run

pytestmark = pytest.mark.gpu


def _channel(nx, ny, held, flag):
    """A channel whose nodes `held` have their velocity (and depth) given."""
    m = meshgen.channel(nx=nx, ny=ny, length=10.0 * nx, width=10.0 * ny)
    ns = len(m.series)
    t = np.array([0.0, 100.0 * m.dt])
    m.series = list(m.series) + [Series(t, np.full(2, v)) for v in (0.1, -0.05, 1.02)]
    m.strings = list(m.strings) + [StringSpec("node", bc_flag=flag, ivx=ns, ivy=ns + 1, iu0=ns + 2)]
    m.node_string = m.node_string.copy()
    m.node_string[list(held)] = len(m.strings) - 1
    return m


# 126 triangles (not a multiple of the kernel's 64), 64, and fewer than one CTA's; nodes 0 to 2, whose
# flags the reference reads as those of the element's own vertices (fe_sw2_load.c:103), held and not
@pytest.mark.parametrize("nx,ny", [(9, 7), (8, 4), (3, 2)])
@pytest.mark.parametrize("held,flag", [((), BCT_VEL_DIR), ((0, 2), BCT_VEL_DIR), ((1,), BCT_VEL_PRS_DIR), ((5,), BCT_VEL_PRS_DIR)])
def test_first_increment_solves_the_differenced_system(nx, ny, held, flag):
    m = _channel(nx, ny, held, flag)
    V, dt = m.nnodes, m.dt
    rng = np.random.default_rng(nx)
    wave = lambda a: a * np.sin(3.0 * m.x / np.ptp(m.x) + rng.uniform(0, 6)) * np.cos(2.0 * m.y / np.ptp(m.y) + rng.uniform(0, 6))  # noqa: E731
    levels = [(1.0 + wave(0.03), 0.2 + wave(0.05), wave(0.05)) for _ in range(2)]   # current, old
    g = SW2GPU(m, precond=capi.SW2GPU_PREC_BAND, overrides=dict(max_nonlin_it=1, tol_nonlin=1e30))
    g.set_state(0, *levels[0])
    g.set_state(1, *levels[1])
    st = g.step(dt, 0.0)
    assert st["status"] == 0 and st["newton_its"] == 1 and st["wd_elems"] == 0
    got = np.stack(g.get_state(0), 1)
    g.close()
    # the same iteration from the pieces: the step starts from the old level with the held values in
    start = np.stack(levels[0], 1)
    for n in held:
        start[n, 1:] = 0.1, -0.05
        if flag == BCT_VEL_PRS_DIR:
            start[n, 0] = 1.02
    s = SW2GPU(m)
    s.set_state(0, *start.T)
    s.set_state(1, *levels[0])
    s.set_state(2, *levels[1])
    s.set_dt(dt, m.series_values(0.0, dt))
    s.resid()
    rp, col, val, R = s.load()
    s.close()
    A = np.zeros((V, 3, V, 3))
    A[np.repeat(np.arange(V), np.diff(rp)), :, col, :] = val
    x = np.linalg.solve(A.reshape(3 * V, 3 * V), R).reshape(V, 3)   # u, v, h
    want = start + x[:, [2, 0, 1]]
    # the quotients are good to 1e-8 (rounding of the residual over the step), times the condition of
    # the system, up to 1e4
    assert np.abs(got - want).max() <= 1e-4 * np.abs(x).max()


def test_variants_of_the_differenced_kernel_give_identical_steps():
    """Estimated viscosity: the steps launch k_jac_elem_wet in the variant that is set."""
    m = meshgen.bumpy_basin(1500, seed=7, size=3000.0, nsteps=3, dt=7.0, nbins=3)
    m = dataclasses.replace(m, materials=[dataclasses.replace(x, eev_mode=3, eev_coef=0.2) for x in m.materials])
    ref = None
    for jac in (1, 2):
        g = SW2GPU(m)
        g.set_variant(jac, 3)
        g.resid()
        val = g.load()[2]
        its = [(s["newton_its"], s["linear_its"]) for s in run(g, 3)]
        got = [np.concatenate(g.get_state(lvl)) for lvl in range(3)] + [val]
        g.close()
        if ref is None:
            ref = got, its
            continue
        assert its == ref[1]
        for a, b in zip(got, ref[0]):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("jac", [1, 2])
def test_autotune_leaves_a_kernel_alone_that_no_step_launches(jac):
    m = meshgen.bumpy_basin(1500, seed=7, size=3000.0, nsteps=3, dt=7.0, nbins=3)
    g = SW2GPU(m)
    g.set_variant(jac, 3)
    assert g.autotune()[0] == jac == g.variant()[0]
    g.close()
