"""Grouped batches (spn_batch_set_grouping) of lattices on which a pair's exchange is another pair: full subgroups (16 flows up to 8
sites, 8 up to 16, 4 up to 24) share node supports, the other flows of a group do not, and every flow's measurements and final state
are bit-identical to the same flow run alone.  Tables no lattice has (6 and 12 sites) and pyrochlore lattices (9, 18 and 31
sites); the first member of a group diverges at its first step."""
from dataclasses import replace

import numpy as np
import pytest

import spinparser_gb300 as spn
from spinparser_gb300.batch import Su2Batch
from spinparser_gb300.driver import run_flow

pytestmark = pytest.mark.gpu

CUT = spn.cutoff_exponential(20.0, 1.0, 0.7)


def tables(lattice, rng, j2):
    tab = spn.Lattice(lattice, rng, f"{lattice}-j1j2heisenberg", {"j1": "1", "j2": f"{j2:.3f}"}).tables()
    if lattice == "square":  # an exchange that no lattice has
        tab = replace(tab, inv_sites_rid=np.random.RandomState(rng).randint(0, tab.n_sites, tab.n_sites).astype(np.int32))
    return tab


def start(tab, n, poison):
    v2, ss, dd = tab.initial_state(n)
    if poison:
        ss = ss.copy()
        ss[::tab.n_sites] = np.nan
    return v2, ss, dd


@pytest.mark.parametrize("cap_divisor", [1, 2])
@pytest.mark.parametrize("lattice,rng,n,flows,shared", [
    ("square", 3, 8, 18, 16), ("square", 5, 6, 8, 8), ("square", 5, 6, 7, 0), ("pyrochlore", 3, 7, 17, 16), ("pyrochlore", 4, 5, 9, 8),
    ("pyrochlore", 5, 5, 4, 0)])
def test_grouped_flows_equal_flows_alone(lattice, rng, n, flows, shared, cap_divisor):
    freq = spn.frequency_exponential(0.05, 50.0, n)
    tabs = [tables(lattice, rng, 0.05 + 0.9 * i / flows) for i in range(flows)]
    b = Su2Batch()
    b.set_grouping(2, cap_divisor)
    ids = [b.add(t, freq, CUT, start(t, n, i == 0)) for i, t in enumerate(tabs)]
    assert b.grouped_flows() == (shared if cap_divisor == 1 else 0)
    b.run()
    for i, (t, fid) in enumerate(zip(tabs, ids)):
        flow = spn.Su2Flow(t, freq)
        measured, zz, dd, cz, cd, diverged = run_flow(flow, CUT, start(t, n, i == 0))
        state = flow.get_state()
        flow.close()
        r = b.result(fid)
        assert r.diverged == diverged == (i == 0), i
        assert np.array_equal(r.cutoffs, measured), i
        for got, want in ((r.zz, zz), (r.dd, dd), (r.chi_zz, cz), (r.chi_dd, cd)):
            assert np.array_equal(got, want.reshape(got.shape), equal_nan=True), i
        if not diverged:
            assert all(np.array_equal(a, w) for a, w in zip(b.state(fid), state)), i
    b.close()
