"""The SU(2) vertex flow of 49 to 64 sites around the node counts where an item's three transfer frequencies together have at most 64
nodes (their descriptors are built at once) or more: meshes and cutoffs whose items have 60 to 70, some with fewer and some with more
in one launch, alone and in a batch.  On a uniform mesh and a cutoff on its raster, so that the oracle's coordinates are exact.

Tolerance: normwise 1e-5, the bound of the other right-hand-side tests."""
import numpy as np
import pytest

import spinparser_gb300 as spn
from oracle import Oracle
from spinparser_gb300.batch import Su2Batch
from spinparser_gb300.driver import run_flow

pytestmark = pytest.mark.gpu


def tables(rng):
    return spn.Lattice("square", rng, "square-j1j2heisenberg", {"j1": "1", "j2": "0.3"}).tables()


@pytest.mark.parametrize("rng,n,cutoff", [(12, 9, 0.25), (14, 12, 1.0), (13, 11, 1.0), (12, 10, 0.25)])
def test_flow_at_node_counts(rng, n, cutoff):
    tab = tables(rng)
    assert 49 <= tab.n_sites <= 64
    freq = (np.arange(1, n + 1) * np.float32(0.5)).astype(np.float32)
    g = np.random.RandomState(rng * n)
    fn = n * n * (n + 1) // 2
    v2 = (0.2 * freq).astype(np.float32)
    ss, dd = g.uniform(-1, 1, (2, fn * tab.n_sites)).astype(np.float32)
    flow = spn.Su2Flow(tab, freq)
    flow.set_state(cutoff, v2, ss, dd)
    flow.compute_step()
    cnt = flow.node_counts()
    sums = [cnt[p] + cnt[q] + cnt[r] for p in range(n) for q in range(p + 1) for r in range(q + 1)]
    assert (min(sums), max(sums)) == {9: (60, 69), 10: (66, 75), 11: (51, 63), 12: (57, 69)}[n]
    dv2, *got = flow.get_flow()
    flow.close()
    want = Oracle(tab, freq).vertex_range(cutoff, v2, dv2, ss, dd, 0, fn)
    for a, b in zip(got, want):
        assert np.linalg.norm(a.astype(np.float64) - b) < 1e-5 * np.linalg.norm(b)


def test_batched_flows_equal_flows_alone():
    cut = spn.cutoff_exponential(20.0, 0.5, 0.5)
    specs = [(12, 9), (13, 12), (14, 13), (10, 12)]
    b = Su2Batch()
    ids = []
    for rng, n in specs:
        tab = tables(rng)
        ids.append(b.add(tab, spn.frequency_exponential(0.05, 50.0, n), cut, tab.initial_state(n)))
    b.run()
    for (rng, n), fid in zip(specs, ids):
        tab = tables(rng)
        flow = spn.Su2Flow(tab, spn.frequency_exponential(0.05, 50.0, n))
        measured, zz, dd, *_ = run_flow(flow, cut, tab.initial_state(n))
        r = b.result(fid)
        assert np.array_equal(r.zz, zz.reshape(r.zz.shape)) and np.array_equal(r.dd, dd.reshape(r.dd.shape))
        assert all(np.array_equal(x, y) for x, y in zip(b.state(fid), flow.get_state()))
        flow.close()
    b.close()
