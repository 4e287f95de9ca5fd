"""The operand scratch of a TRI flow's lattice sum under a limit of device memory (no GPU: the allocator is a limit): a flow that
does not get all of it takes the same kernel with fewer CTAs, by halves, and fails only where not one CTA's fits; it never takes
another algorithm, whose sums would round differently."""
import ctypes as C

import pytest

import spinparser_gb300 as spn
from spinparser_gb300._capi import check, load_library

SMS = 152


def scratch(n, nl, free):
    ctas, size = C.c_int(), C.c_longlong()
    check(load_library().spn_tri_scratch(n, nl, SMS, free, C.byref(ctas), C.byref(size)))
    return ctas.value, size.value


@pytest.mark.parametrize("n", [2, 32, 256])
def test_fewer_ctas_where_memory_is_short(n):
    full = 1 << 50
    ctas, size = scratch(n, 28, full)
    assert ctas == SMS and size % SMS == 0
    one = size // SMS
    # 2 N + 8 nodes at most, two slabs each, in 24 operand terms of 128 bf16 rows; padded to 16 slab pairs
    assert 24 * 2 * 128 * 2 * (2 * n + 8) <= one <= 24 * 2 * 128 * (2 * (2 * n + 8) + 15)
    assert scratch(n, 28, size) == (SMS, size)
    assert scratch(n, 28, size - 1) == (76, 76 * one)
    assert scratch(n, 28, 5 * one) == (4, 4 * one)
    assert scratch(n, 28, one) == (1, one)
    with pytest.raises(spn.SpnError) as e:
        scratch(n, 28, one - 1)
    assert "out of memory" in str(e.value)


@pytest.mark.parametrize("nl", [1, 9, 33, 128])
def test_flows_without_products_take_none(nl):
    assert scratch(32, nl, 0) == (0, 0)
