"""The FP64 vertex flow's shared-node items (lattices of at most 32 sites) against the FP64 oracle: every width of
the outer products and its edges, meshes of 2 to 9 points, exchanged pairs that are other sites, and tables that no
lattice has.

Tolerance: normwise 1e-11, the bound of the other FP64 right-hand-side tests."""
from dataclasses import replace

import numpy as np
import pytest

import spinparser_gb300 as spn
from oracle import Oracle

pytestmark = pytest.mark.gpu

LATTICES = {
    "square": ("square-j1j2heisenberg", {"j1": "1", "j2": "0.3"}),
    "cubic": ("cubic-j1j2heisenberg", {"j1": "1", "j2": "0.3"}),
    "pyrochlore": ("pyrochlore-j1j2heisenberg", {"j1": "1", "j2": "0.3"}),
}


@pytest.mark.parametrize("tables", ["lattice", "arbitrary"])
@pytest.mark.parametrize("mesh", ["exponential", "uniform"])
@pytest.mark.parametrize("lattice,rng,n", [
    ("square", 2, 2), ("pyrochlore", 3, 5), ("square", 5, 9), ("square", 6, 3), ("cubic", 6, 4), ("pyrochlore", 5, 4),
])
def test_fp64_items_match_oracle(lattice, rng, n, mesh, tables):
    model, params = LATTICES[lattice]
    tab = spn.Lattice(lattice, rng, model, params).tables()
    g = np.random.RandomState(5 * rng + n)
    nl = tab.n_sites
    assert nl <= 32
    if tables == "arbitrary":
        tab = replace(tab, sites_rid=g.permutation(nl).astype(np.int32), inv_sites_rid=g.randint(0, nl, nl).astype(np.int32))
    freq = (np.arange(1, n + 1) * np.float32(0.5)).astype(np.float32) if mesh == "uniform" else spn.frequency_exponential(0.02, 20.0, n)
    fn = n * n * (n + 1) // 2
    v2 = 0.2 * freq.astype(np.float64)
    ss, dd = g.uniform(-1, 1, fn * nl), g.uniform(-1, 1, fn * nl)
    oracle = Oracle(tab, freq)
    flow = spn.Su2Flow(tab, freq, flags=spn.FP64)
    for cutoff in (0.4 * float(freq[0]), 0.37, float(freq[n // 2]), 1.5 * float(freq[-1])):
        cutoff = float(np.float32(cutoff))
        flow.set_state_f64(cutoff, v2, ss, dd)
        flow.compute_step()
        dv2, *got = flow.get_flow_f64()
        want = oracle.vertex_range(cutoff, v2, dv2, ss, dd, 0, fn, fp64=True)
        for what, a, b in zip(("spin", "density"), got, want):
            assert np.linalg.norm(a - b) <= 1e-11 * np.linalg.norm(b), (what, cutoff)
    flow.close()
