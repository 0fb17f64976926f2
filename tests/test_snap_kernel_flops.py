"""The operation count of the SNAP kernels' formulation, by enumeration (CPU)."""
import itertools

import pytest

from examinimd_gb300.snap_flops import _entries, kernel_flops, product_counts


def _products(J):
    """Every product of one (T, q) and sign of T with its number of j: the pairs of
    elements (m1, n1) of U_j1 and (m - m1, m' - n1) of U_j2, unordered for j1 = j2."""
    products = weighted = zs = 0
    for T, q, _ in _entries(J):
        for s in ((1, -1) if T and q else (1,)):
            for j1 in range(J + 1):
                for j2 in range(j1 + 1):
                    js = [j for j in range(j1 - j2, min(J, j1 + j2) + 1, 2) if j >= q + T and (j - q - T) % 2 == 0]
                    if not js:
                        continue
                    M, N = (j1 + j2 - q - s * T) // 2, (j1 + j2 - q + s * T) // 2
                    seen = set()
                    for m1, n1 in itertools.product(range(j1 + 1), repeat=2):
                        m2, n2 = M - m1, N - n1
                        if 0 <= m2 <= j2 and 0 <= n2 <= j2:
                            seen.add(frozenset([(m1, n1), (m2, n2)]) if j1 == j2 else (m1, n1))
                    products += len(seen)
                    weighted += len(seen) * len(js)
                    zs += len(js)
    return products, weighted, zs


@pytest.mark.parametrize("J", [0, 1, 2, 3, 4, 6, 7, 8])
def test_products_by_enumeration(J):
    assert product_counts(J) == _products(J)


def test_phases_add_up_and_split_by_form():
    d = kernel_flops(8, 26)
    assert abs(sum(d["phases"].values()) - d["total"]) <= 1e-9 * d["total"]
    assert d["fp64"]["fp64"] == d["total"] and d["fp32"]["fp64"] == 0.0
    assert abs(d["fp64"]["mixed"] + d["fp32"]["mixed"] - d["total"]) <= 1e-9 * d["total"]
    # Y does not depend on the neighbours, the rest is linear in them
    e = kernel_flops(8, 52)
    assert e["phases"]["Y"] == d["phases"]["Y"] and e["phases"]["force"] == 2 * d["phases"]["force"]
