"""The TRI vertex flow of lattices of at most 32 sites (a CTA per triple, the t channel's lattice sum on the tensor
cores from 10 sites on) against the oracle at the sizes where it can go wrong: meshes of 2 to 7 points, 8, 16
and 32 lanes a node with their edges, permuted spin components, tables that no lattice has, and loop sums of one
to six operand chunks (16 nodes each) with and without the second factor kept.

Tolerance: 1e-5 of the largest value, the bound of the other right-hand-side tests (about 100 uncompensated FP32
terms of the oracle, 6e-8 each, with cancellation).  The tensor-core products keep 24 bits of every operand."""
import os
from dataclasses import replace

import numpy as np
import pytest

import spinparser_gb300 as spn
from oracle import TriOracle

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
LATTICES = {
    "square": ("square-heisenberg", {"j": "1.0"}, None),
    "cubic": ("cubic-heisenberg", {"j": "1.0"}, None),
    "honeycomb": ("honeycomb-kitaev-gamma", {"j": "0.3", "k": "1", "g": "0.4"}, "res_honeycomb"),
}


def tables_of(lattice, rng):
    model, params, res = LATTICES[lattice]
    lat = spn.Lattice(lattice, rng, model, params, **({"resource_dir": os.path.join(GOLDEN, res)} if res else {}))
    return lat.tables(), lat.spin_tables()


def arbitrary_tables(tab, spin, seed):
    """Tables that no lattice has: exchanges that are no involution, any spin permutations in sites and pairs."""
    g = np.random.RandomState(seed)
    nl, no = tab.n_sites, len(tab.overlap_rid1)
    perm = lambda k: g.randint(0, 6, k).astype(np.int32)
    return (replace(tab, sites_rid=g.permutation(nl).astype(np.int32), inv_sites_rid=g.randint(0, nl, nl).astype(np.int32)),
            replace(spin, sites_perm=perm(nl), inv_sites_perm=perm(nl), overlap_perm1=perm(no), overlap_perm2=perm(no)))


def check(tab, spin, freq, cutoffs, seed):
    g = np.random.RandomState(seed)
    n = len(freq)
    v2 = (0.2 * freq).astype(np.float32)
    v4 = g.uniform(-0.5, 0.5, n * n * (n + 1) // 2 * 16 * tab.n_sites).astype(np.float32)
    oracle = TriOracle(tab, spin, freq)
    flow = spn.TriFlow(tab, spin, freq)
    for cutoff in cutoffs:
        flow.set_state(cutoff, v2, v4)
        flow.compute_step()
        dv2, got = flow.get_flow()
        # the oracle's vertex flow from the same self-energy flow: that sum cancels on such states
        want = oracle.vertex(cutoff, v2, dv2, v4).reshape(-1, 16, tab.n_sites)
        err = np.abs(np.asarray(got, np.float64).reshape(want.shape) - want).max(axis=(0, 2))
        assert err.max() <= 1e-5 * np.abs(want).max(), (cutoff, err)
        assert not flow.is_diverged()
    flow.close()


@pytest.mark.parametrize("tables", ["lattice", "arbitrary"])
@pytest.mark.parametrize("mesh", ["exponential", "uniform"])
@pytest.mark.parametrize("lattice,rng,n", [
    ("square", 2, 2), ("honeycomb", 3, 7), ("honeycomb", 4, 5), ("honeycomb", 5, 3), ("square", 6, 4), ("honeycomb", 7, 3),
    ("honeycomb", 8, 5), ("honeycomb", 9, 4), ("square", 9, 3),
])
def test_tri_flow_matches_oracle(lattice, rng, n, mesh, tables):
    tab, spin = tables_of(lattice, rng)
    assert tab.n_sites <= 32
    if tables == "arbitrary":
        tab, spin = arbitrary_tables(tab, spin, rng)
    freq = (np.arange(1, n + 1) * np.float32(0.5)).astype(np.float32) if mesh == "uniform" else spn.frequency_exponential(0.02, 20.0, n)
    check(tab, spin, freq, (0.4 * float(freq[0]), 0.37, float(freq[n // 2]), 1.5 * float(freq[-1])), 3 * rng + n)


@pytest.mark.parametrize("n", [12, 20, 24, 40])
def test_tri_operand_chunks_match_oracle(n):
    tab, spin = tables_of("honeycomb", 8)
    tab, spin = arbitrary_tables(tab, spin, n)
    keep = np.concatenate([np.arange(a, min(a + 2, b)) for a, b in zip(tab.overlap_ptr[:-1], tab.overlap_ptr[1:])])  # two pairs a site
    ptr = np.concatenate([[0], np.cumsum([min(2, b - a) for a, b in zip(tab.overlap_ptr[:-1], tab.overlap_ptr[1:])])])
    tab = replace(tab, overlap_ptr=ptr.astype(np.int32), overlap_rid1=tab.overlap_rid1[keep], overlap_rid2=tab.overlap_rid2[keep])
    spin = replace(spin, overlap_perm1=spin.overlap_perm1[keep], overlap_perm2=spin.overlap_perm2[keep])
    check(tab, spin, spn.frequency_exponential(0.02, 20.0, n), (0.01,), n)
