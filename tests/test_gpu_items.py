"""The vertex flow's shared-node items (csrc/su2_item.cuh) against the oracle at the sizes where they can
go wrong: meshes of 2 to 9 points (degenerate index triples p = q, q = r), every outer-product width and
lane-group size, lattices whose exchanged pairs are the pairs themselves, another lattice site's, or (tables
no lattice has) arbitrary; meshes on which loop frequencies cancel to exactly zero and hit mesh points; and
states without the symmetries of a flow, whose density does not vanish at s = u.

Tolerance: normwise 1e-5, the bound of the other right-hand-side tests (about 100 uncompensated FP32
terms of the oracle, 6e-8 each, with cancellation)."""
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


def normwise(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def arbitrary_tables(tab, seed):
    """Site tables that no lattice has: neither the identity nor an involution."""
    g = np.random.RandomState(seed)
    nl = tab.n_sites
    return replace(tab, sites_rid=g.permutation(nl).astype(np.int32), inv_sites_rid=g.randint(0, nl, nl).astype(np.int32))


@pytest.mark.parametrize("tables", ["lattice", "arbitrary"])
@pytest.mark.parametrize("mesh", ["exponential", "uniform"])
@pytest.mark.parametrize("lattice,rng,n", [
    ("square", 2, 2), ("square", 3, 9), ("pyrochlore", 3, 5), ("square", 5, 3), ("square", 6, 7), ("cubic", 6, 5),
    ("square", 8, 4), ("pyrochlore", 5, 6), ("cubic", 7, 3), ("square", 10, 4), ("pyrochlore", 6, 4), ("square", 13, 5),
    ("pyrochlore", 7, 3), ("square", 17, 4), ("cubic", 12, 2), ("square", 20, 3),
])
def test_items_match_oracle(lattice, rng, n, mesh, tables):
    model, params = LATTICES[lattice]
    tab = spn.Lattice(lattice, rng, model, params).tables()
    if tables == "arbitrary":
        tab = arbitrary_tables(tab, rng)
    freq = (np.arange(1, n + 1) * np.float32(0.5)).astype(np.float32) if mesh == "uniform" else spn.frequency_exponential(0.02, 20.0, n)
    g = np.random.RandomState(7 * rng + n)
    fn = n * n * (n + 1) // 2
    v2 = (0.2 * freq).astype(np.float32)
    ss = g.uniform(-1, 1, fn * tab.n_sites).astype(np.float32)
    dd = g.uniform(-1, 1, fn * tab.n_sites).astype(np.float32)
    oracle = Oracle(tab, freq)
    flow = spn.Su2Flow(tab, freq)
    # below the mesh, between mesh points, on a mesh point, above the mesh
    for cutoff in (0.4 * float(freq[0]), 0.37, float(freq[n // 2]), 1.5 * float(freq[-1])):
        flow.set_state(cutoff, v2, ss, dd)
        flow.compute_step()
        dv2, *got = flow.get_flow()
        # the oracle's vertex flow from the same self-energy flow: that sum cancels on such states
        want = oracle.vertex_range(cutoff, v2, dv2, ss, dd, 0, fn)
        for what, a, b in zip(("spin", "density"), got, want):
            assert normwise(a, b) < 1e-5, (what, cutoff)
    flow.close()


@pytest.mark.parametrize("lattice,rng,n", [("square", 10, 40), ("square", 13, 40)])
def test_many_nodes_match_oracle(lattice, rng, n):
    """More loop frequencies than a CTA builds descriptors at once (64), on the first, middle and last triples.  In 64
    bits: at the highest frequencies of a random state the oracle's FP32 frequency sums cost it 6e-5."""
    model, params = LATTICES[lattice]
    tab = spn.Lattice(lattice, rng, model, params).tables()
    freq = spn.frequency_exponential(0.02, 20.0, n)
    g = np.random.RandomState(rng)
    fn = n * n * (n + 1) // 2
    v2 = (0.2 * freq).astype(np.float32)
    ss = g.uniform(-1, 1, fn * tab.n_sites).astype(np.float32)
    dd = g.uniform(-1, 1, fn * tab.n_sites).astype(np.float32)
    oracle = Oracle(tab, freq)
    flow = spn.Su2Flow(tab, freq)
    flow.set_state(0.01, v2, ss, dd)
    flow.compute_step()
    dv2, *got = flow.get_flow()
    for at in (0, fn // 2, fn - 150):
        want = oracle.vertex_range(float(np.float32(0.01)), v2, dv2, ss, dd, at, at + 150, fp64=True)
        for a, b in zip(got, want):
            assert normwise(a[at * tab.n_sites:(at + 150) * tab.n_sites], b) < 1e-5, at
    flow.close()
