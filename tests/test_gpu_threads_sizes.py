"""Flows of different sizes stepped by several threads at once: their kernels need different amounts of shared memory,
and none may lose it to another's launch.  Every flow gives the bits it gives alone."""
import os
import threading

import numpy as np
import pytest

import spinparser_gb300 as spn

pytestmark = pytest.mark.gpu

RES = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "res_honeycomb")


def make(core, rng, n):
    freq = spn.frequency_exponential(0.02, 20.0, n)
    g = np.random.RandomState(rng)
    v2 = (0.2 * freq).astype(np.float32)
    fn = n * n * (n + 1) // 2
    if core in ("su2", "fp64"):
        tab = spn.Lattice("square", rng, "square-j1j2heisenberg", {"j1": "1", "j2": "0.3"}).tables()
        flow = spn.Su2Flow(tab, freq, flags=spn.FP64 if core == "fp64" else 0)
        flow.set_state(0.37, v2, *g.uniform(-0.1, 0.1, (2, fn * tab.n_sites)).astype(np.float32))
        return flow
    lat = spn.Lattice("honeycomb", rng, "honeycomb-kitaev-gamma", {"j": "0.3", "k": "1", "g": "0" if core == "xyz" else "0.4"},
                      resource_dir=RES)
    tab, spin = lat.tables(), lat.spin_tables()
    flow = (spn.XyzFlow if core == "xyz" else spn.TriFlow)(tab, spin, freq)
    shape = (4, fn * tab.n_sites) if core == "xyz" else fn * 16 * tab.n_sites
    flow.set_state(0.37, v2, g.uniform(-0.1, 0.1, shape).astype(np.float32))
    return flow


@pytest.mark.parametrize("core,sizes", [("su2", (10, 13, 20, 17)), ("fp64", (3, 9, 5, 8)), ("xyz", (4, 9, 6, 8)), ("tri", (5, 9, 6, 8))])
def test_sizes_side_by_side(core, sizes):
    flows = [make(core, r, 6) for r in sizes]
    alone = []
    for f in flows:
        f.compute_step()
        alone.append(np.array(f.get_flow()[1]))
    bad = []

    def work(f, want):
        try:
            for _ in range(50):
                f.compute_step()
                if not np.array_equal(np.array(f.get_flow()[1]), want):
                    bad.append("values")
                f.measure_correlation()
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            bad.append(repr(e))

    threads = [threading.Thread(target=work, args=a) for a in zip(flows, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:3]
    for f in flows:
        f.close()
