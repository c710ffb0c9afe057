"""Meshes whose node numbering has no locality: the shares of the Krylov solve are cut into several
sub-ranges there (sw2_halo.h), and every launch variant still steps to the same bits."""
import dataclasses

import numpy as np
import pytest

from adhv8_kraken_b200 import capi, meshgen
from adhv8_kraken_b200.sw2 import SW2GPU


def renumbered(m, seed):
    """The mesh with its nodes in random order."""
    perm = np.random.default_rng(seed).permutation(m.nnodes)   # perm[new] = old
    inv = np.empty(m.nnodes, np.int32)
    inv[perm] = np.arange(m.nnodes, dtype=np.int32)
    return dataclasses.replace(m, x=m.x[perm].copy(), y=m.y[perm].copy(), z=m.z[perm].copy(), tri=inv[m.tri], edges=inv[m.edges],
                               node_string=m.node_string[perm].copy(), h0=m.h0[perm].copy(), u0=m.u0[perm].copy(),
                               v0=m.v0[perm].copy())


def _steps(g, n=2):
    sts = [g.step() for _ in range(n)]
    assert all(s["status"] == 0 for s in sts)
    out = [np.concatenate(g.get_state(lvl)) for lvl in range(2)], [(s["newton_its"], s["linear_its"]) for s in sts]
    g.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [capi.SW2GPU_FP64, capi.SW2GPU_MIXED])
def test_variants_give_identical_steps_on_a_scattered_numbering(precision):
    # 48,000 nodes: more rows and neighbours per CTA of the device than one operand buffer holds
    m = renumbered(meshgen.bumpy_basin(48000, seed=11, size=6200.0, nsteps=3), 3)
    ref = None
    for stages in (3, 2, 0):
        g = SW2GPU(m, precision=precision)
        g.set_variant(2, stages)
        assert g.variant() == (2, stages)
        got = _steps(g)
        if ref is None:
            ref = got
            continue
        assert got[1] == ref[1], stages
        for a, b in zip(got[0], ref[0]):
            assert np.array_equal(a, b), stages


@pytest.mark.gpu
@pytest.mark.parametrize("points", [97, 3001, 20000])
def test_solve_and_step_do_not_depend_on_the_numbering(points):
    """The Krylov solve takes the rows of a scattered mesh in its own order: a linear system with a
    known solution, and whole time steps against those of the mesh as it was numbered."""
    m = meshgen.bumpy_basin(points, seed=5, size=28.3 * points**0.5, nsteps=3, nbins=3)
    perm = np.random.default_rng(2).permutation(m.nnodes)
    r = renumbered(m, 2)
    assert np.array_equal(r.x, m.x[perm])
    g = SW2GPU(m)
    for _ in range(2):
        assert g.step()["status"] == 0
    want = g.get_state(0)
    g.close()
    if points < 10000:   # above, 1e-10 is at the limit of what BiCGSTAB reaches in any order of the rows
        g = SW2GPU(r, lin_rtol=1e-10, lin_atol=0.0)
        assert g.step()["status"] == 0
        rp, col, val, _ = g.load()
        x_ref = np.random.default_rng(3).standard_normal((r.nnodes, 3))
        b = np.zeros((r.nnodes, 3))
        np.add.at(b, np.repeat(np.arange(r.nnodes), np.diff(rp)), np.einsum("kij,kj->ki", val, x_ref[col]))
        x, its, rc = g.linear_solve(val, b.reshape(-1))
        # the bound of the solve against a direct one at this tolerance
        assert rc == 0 and its > 0 and np.abs(x - x_ref.reshape(-1)).max() <= 1e-7 * np.abs(x_ref).max()
        g.close()
    g = SW2GPU(r)
    for _ in range(2):
        assert g.step()["status"] == 0
    # each run is within 1e-10 of the exact steps (the bound against the reference), relative to the
    # largest value of the field
    for a, b in zip(g.get_state(0), want):
        assert np.abs(a - b[perm]).max() <= 1e-9 * max(np.abs(b).max(), 1e-3)
    g.close()
