"""Kernels that the other tests reach alone or not at all: batches of the classes of 33 to 64 sites whose pairs exchange with
others (a CTA per triple), and small SU(2) flows of both warp kernels stepped by several threads at once.  Every flow gives the
bits it gives alone."""
import threading
from dataclasses import replace

import numpy as np
import pytest

import spinparser_gb300 as spn
from spinparser_gb300.batch import Su2Batch
from spinparser_gb300.driver import run_flow

pytestmark = pytest.mark.gpu


def tables(lattice, rng, exchange=None):
    tab = spn.Lattice(lattice, rng, f"{lattice}-j1j2heisenberg", {"j1": "1", "j2": "0.3"}).tables()
    if exchange is not None:  # an exchange that no lattice has
        tab = replace(tab, inv_sites_rid=np.random.RandomState(exchange).randint(0, tab.n_sites, tab.n_sites).astype(np.int32))
    return tab


def test_batch_of_exchanged_pairs():
    tabs = [tables("pyrochlore", 6), tables("square", 13, 1), tables("square", 10, 2), tables("square", 14)]
    assert [t.n_sites for t in tabs] == [48, 56, 36, 64]
    cut = spn.cutoff_exponential(20.0, 1.0, 0.5)
    b = Su2Batch()
    ids = [b.add(t, spn.frequency_exponential(0.05, 50.0, n), cut) for t, n in zip(tabs, (6, 5, 7, 6))]
    b.run()
    for t, n, fid in zip(tabs, (6, 5, 7, 6), ids):
        flow = spn.Su2Flow(t, spn.frequency_exponential(0.05, 50.0, n))
        measured, zz, dd, *_ = run_flow(flow, cut, t.initial_state(n))
        r = b.result(fid)
        assert np.array_equal(r.zz, zz.reshape(r.zz.shape)) and np.array_equal(r.dd, dd.reshape(r.dd.shape)), t.n_sites
        assert all(np.array_equal(x, y) for x, y in zip(b.state(fid), flow.get_state())), t.n_sites
        flow.close()
    b.close()


def test_small_flows_side_by_side():
    flows, alone, bad = [], [], []
    for t, n in ((tables("square", 3), 12), (tables("pyrochlore", 4), 6), (tables("square", 6), 8), (tables("pyrochlore", 5), 5), (tables("square", 9), 6)):
        freq = spn.frequency_exponential(0.02, 20.0, n)
        flow = spn.Su2Flow(t, freq)
        g = np.random.RandomState(n)
        flow.set_state(0.37, (0.2 * freq).astype(np.float32), *g.uniform(-0.1, 0.1, (2, n * n * (n + 1) // 2 * t.n_sites)).astype(np.float32))
        flow.compute_step()
        flows.append(flow)
        alone.append([np.array(x) for x in (*flow.get_flow(), *flow.measure_correlation())])

    def work(flow, want):
        try:
            for _ in range(50):
                flow.compute_step()
                got = (*flow.get_flow(), *flow.measure_correlation())
                if flow.is_diverged() or not all(np.array_equal(x, y) for x, y in zip(got, want)):
                    bad.append("values")
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            bad.append(repr(e))

    threads = [threading.Thread(target=work, args=a) for a in zip(flows, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:3]
    for flow in flows:
        flow.close()
