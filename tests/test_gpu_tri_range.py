"""The lattice sum of TRI flows on the tensor cores at the ends of the FP32 range: its operands are split into bf16 terms,
which must not lose a finite value whose rounding to bf16 overflows, nor make NaN of an infinite one.  One stored vertex element is
large, of a transfer frequency and a site that neither the self-energy flow nor the site-local vertices read.

Tolerance: 1e-5 of the largest finite value, the bound of the other right-hand-side tests."""
import os
from dataclasses import replace

import numpy as np
import pytest

import spinparser_gb300 as spn
from oracle import TriOracle

pytestmark = pytest.mark.gpu

RES = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "res_honeycomb")


def flow_tables(rng):
    """A lattice's tables with at most two pairs a site, so that sums of infinite terms of both signs are few."""
    lat = spn.Lattice("honeycomb", rng, "honeycomb-kitaev-gamma", {"j": "0.3", "k": "1", "g": "0.4"}, resource_dir=RES)
    tab, spin = lat.tables(), lat.spin_tables()
    ptr = tab.overlap_ptr
    keep = np.concatenate([np.arange(a, min(a + 2, b)) for a, b in zip(ptr[:-1], ptr[1:])])
    return (replace(tab, overlap_ptr=np.concatenate([[0], np.cumsum(np.minimum(2, np.diff(ptr)))]).astype(np.int32),
                    overlap_rid1=tab.overlap_rid1[keep], overlap_rid2=tab.overlap_rid2[keep]),
            replace(spin, overlap_perm1=spin.overlap_perm1[keep], overlap_perm2=spin.overlap_perm2[keep]))


@pytest.mark.parametrize("value", [3.2e38, 3.35e38, -3.395e38, 3.4e38, np.inf, -np.inf])
@pytest.mark.parametrize("rng", [6, 9])
def test_large_elements(rng, value):
    tab, spin = flow_tables(rng)
    n, nl = 6, tab.n_sites
    # a uniform mesh, whose points the slabs hit (5, 4 at transfer 3 too), so that operands are as large as the element; off the points for the
    # infinite one, whose product with a zero weight is NaN
    freq = spn.frequency_exponential(0.1, 20.0, n) if np.isinf(value) else np.arange(1, n + 1, dtype=np.float32)
    cutoff = 1.0  # node coefficients below one, which operands are multiplied by
    g = np.random.RandomState(rng)
    v4 = g.uniform(-1e-3, 1e-3, (n * (n + 1) // 2, n, 16, nl)).astype(np.float32)
    v4[n * (n - 1) // 2 - 2, 2, g.randint(16), tab.overlap_rid1[tab.overlap_ptr[nl - 1]] or 1] = value
    v2 = (0.2 * freq).astype(np.float32)
    oracle = TriOracle(tab, spin, freq)
    flow = spn.TriFlow(tab, spin, freq)
    flow.set_state(cutoff, v2, v4.reshape(-1))
    flow.compute_step()
    dv2, got = flow.get_flow()
    flow.close()
    assert np.isfinite(dv2).all()
    want = oracle.vertex(cutoff, v2, dv2, v4.reshape(-1))
    got = np.asarray(got).reshape(want.shape)
    fin, inf = np.isfinite(want), np.isinf(want)
    assert fin.mean() > 0.5 and (inf.any() if np.isinf(value) else np.abs(want[fin]).max() > 1e30)
    assert np.isfinite(got[fin]).all()
    err = np.abs(got[fin].astype(np.float64) - want[fin]).max() / np.abs(want[fin]).max()
    assert err <= 1e-5, err
    if np.isinf(value):
        assert np.array_equal(got[inf], want[inf])
