"""The XYZ vertex flow of lattices of at most 32 sites around the node counts where its kernel changes: up to 16 sites the descriptors of
an item's three transfer frequencies are built at once where any three have at most 64 nodes, and otherwise in batches of 64 a transfer
frequency.  On a uniform mesh and a cutoff on its raster, so that the oracle's coordinates are exact.

Tolerance: 1e-5 of the largest value, the bound of the other right-hand-side tests."""
import os
from dataclasses import replace

import numpy as np
import pytest

import spinparser_gb300 as spn
from oracle import XyzOracle

pytestmark = pytest.mark.gpu

RES = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "res_honeycomb")


def flow_tables(rng):
    """A lattice's tables with at most two pairs a site (the oracle's time)."""
    lat = spn.Lattice("honeycomb", rng, "honeycomb-kitaev-gamma", {"j": "0.3", "k": "1", "g": "0"}, resource_dir=RES)
    tab, spin = lat.tables(), lat.spin_tables()
    ptr = tab.overlap_ptr
    keep = np.concatenate([np.arange(a, min(a + 2, b)) for a, b in zip(ptr[:-1], ptr[1:])])
    return (replace(tab, overlap_ptr=np.concatenate([[0], np.cumsum(np.minimum(2, np.diff(ptr)))]).astype(np.int32),
                    overlap_rid1=tab.overlap_rid1[keep], overlap_rid2=tab.overlap_rid2[keep]),
            replace(spin, overlap_perm1=spin.overlap_perm1[keep], overlap_perm2=spin.overlap_perm2[keep]))


# (range, N, cutoff, nodes of the transfer frequency with the most)
@pytest.mark.parametrize("rng,n,cutoff,most", [
    (4, 11, 1.25, 20), (4, 11, 1.0, 21), (4, 11, 0.75, 23), (6, 11, 1.0, 21), (6, 12, 1.0, 23), (4, 29, 0.25, 63), (4, 30, 0.25, 65),
    (6, 33, 0.25, 71), (9, 30, 0.25, 65)])
def test_xyz_flow_at_node_counts(rng, n, cutoff, most):
    tab, spin = flow_tables(rng)
    freq = (np.arange(1, n + 1) * np.float32(0.5)).astype(np.float32)
    g = np.random.RandomState(rng * n)
    fn = n * n * (n + 1) // 2
    v2 = (0.2 * freq).astype(np.float32)
    su2 = spn.Su2Flow(tab, freq)  # the node counts depend on the mesh and the cutoff alone
    su2.set_state(cutoff, v2, np.zeros(fn * tab.n_sites, np.float32), np.zeros(fn * tab.n_sites, np.float32))
    su2.compute_step()
    assert su2.node_counts().max() == most
    su2.close()
    v4 = g.uniform(-0.05, 0.05, (4, fn * tab.n_sites)).astype(np.float32)
    flow = spn.XyzFlow(tab, spin, freq)
    flow.set_state(cutoff, v2, v4)
    flow.compute_step()
    dv2, got = flow.get_flow()
    flow.close()
    want = XyzOracle(tab, spin, freq).vertex(cutoff, v2, dv2, v4)
    for c in range(4):
        assert np.abs(np.asarray(got[c], np.float64) - want[c]).max() <= 1e-5 * np.abs(want[c]).max(), c
