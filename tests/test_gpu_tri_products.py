"""The TRI vertex flow's lattice sum on the tensor cores against the oracle in 64 bits: every bf16 term of an operand counts.  All pairs
of the lattices and operands of random signs, so that the lattice sum is most of the flow; on a uniform mesh and a cutoff on its
raster, so that coordinates are exact in 32 bits.  With more loop-frequency nodes than descriptors are built at once (112) for the
larger mesh.

Tolerance: 1e-6 of the largest value.  The sums over K slab products round by about sqrt(K) 6e-8 of their terms, 1e-7 of the largest
value; without an operand's third term the products are 2^-17 = 8e-6 off.

With operands of one sign the cuts of the tensor cores' sums add up: at most 4 of them, 0.5 units in the last place each, 2e-7, beside
the rounding of the ladders' sums of some 300 terms, 6e-8 sqrt(300) / 4 = 2.6e-7: in norm 5e-7."""
import os

import numpy as np
import pytest

import spinparser_gb300 as spn
from oracle import TriOracle

pytestmark = pytest.mark.gpu

RES = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "res_honeycomb")


def errors(rng, n, shift):
    lat = spn.Lattice("honeycomb", rng, "honeycomb-kitaev-gamma", {"j": "0.3", "k": "1", "g": "0.4"}, resource_dir=RES)
    tab, spin = lat.tables(), lat.spin_tables()
    freq = (np.arange(1, n + 1) * np.float32(0.5)).astype(np.float32)
    g = np.random.RandomState(rng)
    fn = n * n * (n + 1) // 2
    v2 = (0.2 * freq).astype(np.float32)
    v4 = (g.random_sample(fn * 16 * tab.n_sites) - shift).astype(np.float32)
    flow = spn.TriFlow(tab, spin, freq)
    flow.set_state(0.25, v2, v4)
    flow.compute_step()
    dv2, got = flow.get_flow()
    flow.close()
    triples = np.concatenate([[0, fn // 2, fn - 1], g.randint(0, fn, 13)])
    want = TriOracle(tab, spin, freq).vertex_sample64(0.25, v2, dv2, v4, triples)
    return np.asarray(got, np.float64).reshape(fn, -1)[triples] - want, want


@pytest.mark.parametrize("rng,n", [(9, 9), (6, 14), (5, 56)])
def test_tri_flow_in_64_bits(rng, n):
    err, want = errors(rng, n, 0.5)
    assert np.abs(err).max() <= 1e-6 * np.abs(want).max(), np.abs(err).max() / np.abs(want).max()


@pytest.mark.parametrize("rng,n", [(9, 16), (6, 48), (5, 56)])
def test_long_sums_of_one_sign(rng, n):
    err, want = errors(rng, n, 0.0)
    assert np.linalg.norm(err) <= 5e-7 * np.linalg.norm(want), np.linalg.norm(err) / np.linalg.norm(want)
