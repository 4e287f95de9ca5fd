"""Grouped batches with more loop-frequency nodes than the grouped kernel builds at once (64 where a warp has several flows, 128 where
it has one), so that a flow's sums wait between chunks: every flow's measurements and final state are bit-identical to
the same flow run alone.  Subgroups of 1 to 16 flows of 6, 12 and 20 sites, so warps with none, some and all of their flows."""
import numpy as np
import pytest

import spinparser_gb300 as spn
from spinparser_gb300.batch import Su2Batch
from spinparser_gb300.driver import run_flow

pytestmark = pytest.mark.gpu

CUT = np.array([0.05, 0.045, 0.04], np.float32)  # at the lower end of the mesh, where every node counts


@pytest.mark.parametrize("cap_divisor", [1, 4])
@pytest.mark.parametrize("rng,n,flows", [(3, 34, 6), (3, 33, 16), (5, 34, 3), (5, 32, 7), (7, 65, 2)])
def test_flows_with_many_nodes(rng, n, flows, cap_divisor):
    freq = spn.frequency_exponential(0.05, 50.0, n)
    tabs = [spn.Lattice("square", rng, "square-j1j2heisenberg", {"j1": "1", "j2": f"{0.1 + 0.05 * i:.3f}"}).tables() for i in range(flows)]
    b = Su2Batch()
    b.set_grouping(2, cap_divisor)
    ids = [b.add(t, freq, CUT) for t in tabs]
    assert b.grouped_flows() == flows
    b.run()
    for i, (t, fid) in enumerate(zip(tabs, ids)):
        flow = spn.Su2Flow(t, freq)
        measured, zz, dd, cz, cd, diverged = run_flow(flow, CUT, t.initial_state(n))
        assert flow.node_counts().max() > (128 if rng == 7 else 64)
        r = b.result(fid)
        assert not r.diverged and not diverged
        for got, want in ((r.cutoffs, measured), (r.zz, zz), (r.dd, dd), (r.chi_zz, cz), (r.chi_dd, cd)):
            assert np.array_equal(got, want.reshape(got.shape)), i
        assert all(np.array_equal(x, y) for x, y in zip(b.state(fid), flow.get_state())), i
        flow.close()
    b.close()
