"""The edges of the batched kernels: what a run leaves for the next one."""
import numpy as np
import pytest

from cudaprob3_gb300 import earth
from cudaprob3_gb300.batch import Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kinds", ["atmos", "beam", "both"])
@pytest.mark.parametrize("split", [0, 1])
def test_runs_leave_their_counters_cleared(kinds, split):
    """Every form of a run -- plain, in pieces, with other tile shapes, after a run that
    reported a time-out -- is followed by runs with the same results, and new parameters are
    taken over whichever problem they are set for."""
    import torch
    from cudaprob3_gb300._abi import CP3Error
    sets = earth.gaussian_sets(3, seed=21)
    cz, en = earth.cosine_grid(37), earth.log_energy_grid(45)
    b = Batch(0)
    b.set_earth(*earth.PREM_4LAYER, 22.0)
    for m in sets:
        if kinds != "beam":
            b.set_params(b.add_atmos(cz, en), m, False)
        if kinds != "atmos":
            b.set_params(b.add_beam(earth.lin_energy_grid(333), 2.6, [295.0, 1300.0]), m, False)
    b.set_split_tables(split)
    b.commit()
    n = b.info()["problems"]

    def results():
        b.run()
        b.synchronize()
        return [b.result(i).copy() for i in range(n)]

    def same(x, y):
        return all(np.array_equal(p, q) for p, q in zip(x, y))

    want = results()
    assert same(results(), want)
    host = torch.empty(b.info()["result_bytes"] // 4).pin_memory()
    for pieces in (1, 2, 3):
        b.run_to_host(host.data_ptr(), pieces)
        b.synchronize()
        assert same(results(), want)
    for rows, blocks, chunk in ((1, 1, 1), (16, 0, 64)):
        b.set_shape(rows, blocks, chunk)
        assert same(results(), want)
    b.set_shape(2, 0, 4)
    if kinds == "atmos" and split == 0:
        b.debug_withhold_tables(True)
        b.run()
        with pytest.raises(CP3Error, match="did not complete"):
            b.synchronize()
        b.debug_withhold_tables(False)
        assert same(results(), want)
    for i in range(n):
        b.set_params(i, sets[0], True)
    other = results()
    assert not any(np.array_equal(p, q) for p, q in zip(other, want))
    assert same(results(), other)


@pytest.mark.parametrize("last_fails", [False, True])
def test_a_status_belongs_to_its_run(last_fails):
    """Two runs queued without a wait between them, one of which times out (2 s): what the wait
    after them reports is the last one's end, whichever of the two failed."""
    import time
    import torch
    from cudaprob3_gb300._abi import CP3Error
    b = Batch(0)
    b.set_earth(*earth.PREM_4LAYER, 22.0)
    b.set_params(b.add_atmos(earth.cosine_grid(24), earth.log_energy_grid(40)), earth.NOMINAL, False)
    b.commit()
    b.run()
    b.synchronize()
    want = b.result(0).copy()
    s = torch.cuda.Stream()
    b.debug_withhold_tables(not last_fails)
    b.run(s.cuda_stream)
    time.sleep(0.3)  # the first run has read its descriptors
    b.debug_withhold_tables(last_fails)
    b.run()
    if last_fails:
        with pytest.raises(CP3Error, match="did not complete"):
            b.synchronize()
        b.debug_withhold_tables(False)
        b.run()
    b.synchronize()
    assert np.array_equal(b.result(0), want)


def test_a_run_cannot_be_captured():
    """Refused with its reason, and the batch runs on afterwards."""
    import torch
    from cudaprob3_gb300._abi import CP3Error
    b = Batch(0)
    b.set_params(b.add_beam(earth.lin_energy_grid(50), 2.6, [295.0]), earth.NOMINAL, False)
    b.commit()
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with pytest.raises(CP3Error, match="cannot be captured"):
        with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=s):
            b.run(s.cuda_stream)
    torch.cuda.synchronize()
    b.run()
    b.synchronize()
    assert np.abs(b.result(0).sum(axis=1) - 3.0).max() < 1e-4  # three initial flavours


MIXED_TOL = 1e-5  # the mixed path's bound against the oracle


@pytest.mark.parametrize("chunk", [1, 2, 3, 4, 64])
def test_beam_tile_edges(oracle, chunk):
    """A beam tile loads a group's energies one group ahead: problems that end inside, at and
    just after a group and a tile, every energy against the oracle."""
    from oracle.oracle import Mixing as OMix
    sizes = (1, 31, 32, 33, 32 * chunk - 1, 32 * chunk, 32 * chunk + 1)
    b = Batch(0)
    m = earth.gaussian_sets(1, seed=4)[0]
    om = OMix(m.theta12, m.theta13, m.theta23, m.dcp, m.dm12sq, m.dm23sq, 1)
    grids = [np.linspace(0.2, 9.0, n) if n > 1 else np.array([0.7]) for n in sizes]
    for en in grids:
        b.set_params(b.add_beam(en, 2.6, [295.0, 1300.0]), m, False)
    b.set_shape(beam_chunk=chunk)
    b.commit()
    b.run()
    b.synchronize()
    for i, en in enumerate(grids):
        got = b.result(i)
        for j, L in enumerate((295.0, 1300.0)):
            assert np.abs(got[j].T - oracle.beam(om, False, en, 2.6, L)).max() <= MIXED_TOL
