"""The XYZ vertex flow's shared-node items (lattices of at most 32 sites) against the oracle at the sizes where they
can go wrong: meshes of 2 to 7 points (degenerate index triples), both widths of the product matrices (at most
16 and at most 32 sites) with their edges, lattices with permuted spin components, and tables that no lattice has;
meshes on which loop frequencies cancel to exactly zero and hit mesh points.

Tolerance: 1e-5 of the largest value, the bound of the other right-hand-side tests (about 100 uncompensated FP32
terms of the oracle, 6e-8 each, with cancellation)."""
import os
from dataclasses import replace

import numpy as np
import pytest

import spinparser_gb300 as spn
from oracle import XyzOracle

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
LATTICES = {
    "square": ("square-heisenberg", {"j": "1.0"}, None),
    "honeycomb": ("honeycomb-kitaev-gamma", {"j": "0.3", "k": "1", "g": "0"}, "res_honeycomb"),
    "hyperhoneycomb": ("hyperhoneycomb-kitaev", {"j": "0.3", "k": "1"}, "res_hyperhoneycomb"),
}


def arbitrary_tables(tab, spin, seed):
    """Site tables that no lattice has: neither the identity nor an involution, permuted spin components."""
    g = np.random.RandomState(seed)
    nl = tab.n_sites
    perm = lambda: g.randint(0, 6, nl).astype(np.int32)
    return (replace(tab, sites_rid=g.permutation(nl).astype(np.int32), inv_sites_rid=g.randint(0, nl, nl).astype(np.int32)),
            replace(spin, sites_perm=perm(), inv_sites_perm=perm()))


@pytest.mark.parametrize("tables", ["lattice", "arbitrary"])
@pytest.mark.parametrize("mesh", ["exponential", "uniform"])
@pytest.mark.parametrize("lattice,rng,n", [
    ("square", 2, 2), ("honeycomb", 4, 7), ("square", 6, 3), ("honeycomb", 6, 4), ("hyperhoneycomb", 3, 5),
    ("honeycomb", 7, 5), ("honeycomb", 9, 3), ("square", 9, 4),
])
def test_xyz_items_match_oracle(lattice, rng, n, mesh, tables):
    model, params, res = LATTICES[lattice]
    lat = spn.Lattice(lattice, rng, model, params, **({"resource_dir": os.path.join(GOLDEN, res)} if res else {}))
    tab, spin = lat.tables(), lat.spin_tables()
    assert tab.n_sites <= 32
    if tables == "arbitrary":
        tab, spin = arbitrary_tables(tab, spin, rng)
    freq = (np.arange(1, n + 1) * np.float32(0.5)).astype(np.float32) if mesh == "uniform" else spn.frequency_exponential(0.02, 20.0, n)
    g = np.random.RandomState(11 * rng + n)
    fn = n * n * (n + 1) // 2
    v2 = (0.2 * freq).astype(np.float32)
    v4 = g.uniform(-0.05, 0.05, (4, fn * tab.n_sites)).astype(np.float32)
    oracle = XyzOracle(tab, spin, freq)
    flow = spn.XyzFlow(tab, spin, freq)
    for cutoff in (0.4 * float(freq[0]), 0.37, float(freq[n // 2]), 1.5 * float(freq[-1])):
        flow.set_state(cutoff, v2, v4)
        flow.compute_step()
        dv2, got = flow.get_flow()
        # the oracle's vertex flow from the same self-energy flow: that sum cancels on such states
        want = oracle.vertex(cutoff, v2, dv2, v4)
        for c in range(4):
            assert np.abs(np.asarray(got[c], np.float64) - want[c]).max() <= 1e-5 * np.abs(want[c]).max(), (c, cutoff)
    flow.close()
