"""The two-CTAs-per-SM form of the Krylov solve: launches with more virtual CTAs than the device has
SMs.  It computes the bits of the one-CTA form, so a batch ends where its members end alone, and a
batch of any size the library takes is one launch per solve."""
import numpy as np
import pytest

from adhv8_kraken_b200 import capi, meshgen
from adhv8_kraken_b200.sw2 import SW2Batch, SW2Engine, SW2GPU


def _basin(points, seed):
    return meshgen.bumpy_basin(points, seed=seed, size=28.3 * points**0.5, nsteps=3, nbins=3)


def _state(g):
    return [np.concatenate(g.get_state(lvl)) for lvl in range(2)]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [capi.SW2GPU_FP64, capi.SW2GPU_MIXED])
def test_batch_with_more_virtual_ctas_than_sms_equals_alone(precision):
    # 5 to 96 virtual CTAs each (tiles at the edges of their rules), 290 together
    models = [_basin(n, 40 + k) for k, n in enumerate((320, 4095, 4097, 6001, 9000, 12000, 15359))]
    alone = []
    for m in models:
        g = SW2GPU(m, precision=precision)
        its = [g.step()["linear_its"] for _ in range(2)]
        alone.append((_state(g), its))
        g.close()
    solvers = [SW2GPU(m, precision=precision) for m in models]
    batch = SW2Batch(solvers)
    steps = [batch.step() for _ in range(2)]
    for k, g in enumerate(solvers):
        assert [s[k]["status"] for s in steps] == [0, 0]
        assert [s[k]["linear_its"] for s in steps] == alone[k][1]
        for a, b in zip(_state(g), alone[k][0]):
            assert np.array_equal(a, b), k
    batch.close()
    for g in solvers:
        g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision,points", [(capi.SW2GPU_MIXED, 119999), (capi.SW2GPU_MIXED, 121001), (capi.SW2GPU_FP64, 301000)])
def test_large_mesh_equals_the_direct_sweeps(precision, points):
    """Alone: either side of the size from which a mesh has two virtual CTAs per SM."""
    m = _basin(points, 9)
    got = []
    for stages in (3, 0):
        g = SW2GPU(m, precision=precision)
        g.set_variant(2, stages)
        st = g.step()
        assert st["status"] == 0
        got.append((_state(g), st["newton_its"], st["linear_its"]))
        g.close()
    assert got[0][1:] == got[1][1:]
    for a, b in zip(got[0][0], got[1][0]):
        assert np.array_equal(a, b)


@pytest.mark.gpu
def test_one_launch_per_solve_above_one_member_per_sm():
    """A member more than the device has SMs needs no launch more (the other kernels take members in
    groups of 30, so both sizes need the same number of those)."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert (sms + 29) // 30 == (sms + 30) // 30
    m = meshgen.channel(nx=6, ny=3, nsteps=2)
    launches = []
    for n in (sms, sms + 1):
        gs = [SW2GPU(m) for _ in range(n)]
        eng = SW2Engine(capi.SW2GPU_FP64)
        eng.set_rebalance(1)
        for g in gs:
            eng.add(g, 1)
        per_tick = []
        while eng.active:
            eng.tick()
            per_tick.append(eng.last_tick()["launches"])
        launches.append(per_tick)
        eng.close()
        for g in gs:
            g.close()
    assert launches[0] == launches[1]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [capi.SW2GPU_FP64, capi.SW2GPU_MIXED])
@pytest.mark.parametrize("rebalance", [(4, 0.5), (8, 0.0)], ids=["default", "every-iteration"])
def test_paused_solves_go_on_in_either_form(precision, rebalance):
    """An engine whose solves pause: a launch of two CTAs per SM resumes in another, and the last few
    members in launches of one per SM; each ends where it ends alone."""
    models = [_basin(n, 60 + k) for k, n in enumerate((900, 5000, 7001, 9000, 13000, 15001))]
    alone = []
    for m in models:
        g = SW2GPU(m, precision=precision)
        g.step()
        alone.append(_state(g))
        g.close()
    solvers = [SW2GPU(m, precision=precision) for m in models]
    eng = SW2Engine(precision)
    eng.set_rebalance(*rebalance)
    for g in solvers:
        eng.add(g, 1)
    done = eng.run()
    assert len(done) == len(models) and all(d["status"] == 0 for d in done)
    for g, want in zip(solvers, alone):
        for a, b in zip(_state(g), want):
            assert np.array_equal(a, b)
    eng.close()
    for g in solvers:
        g.close()
