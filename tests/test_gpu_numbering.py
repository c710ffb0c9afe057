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
