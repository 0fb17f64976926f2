"""Floating-point operation count of one SNAP force evaluation, per atom.

One operation per add, subtract or multiply (a fused multiply-add counts two)
and one per square root, division or transcendental call, for a given twojmax
and number of inside neighbours.

`kernel_flops` counts the formulation the GB300 kernels run
(`csrc/snap_kernel.cuh`): separated Wigner elements, shared products.

`snap_flops` counts the layered formulation (U by the layer recursion, one Z at
a time, reverse-mode pair forces through the layers), which already needs fewer
operations than the reference's (compute_ui / compute_zi / compute_duidrj /
compute_dbidrj, sna_impl.hpp).  It returns a dict of per-atom counts by phase
and by arithmetic type for each precision form:

- B, the U_tot recursion and its sums, is FP64 in both forms;
- the per-neighbour scalars are FP64 in both forms;
- C (Z and Y) and D (the pair forces) are FP32 in the mixed form and FP64 in
  the FP64 form; the FP64 tail of D (repulsion, scatter, sum for i) is FP64.
"""
from __future__ import annotations


def _triples(J: int):
    """Full (j1 >= j2, j) triples of the Z contraction (SNA::build_indexlist)."""
    for j1 in range(J + 1):
        for j2 in range(j1 + 1):
            for j in range(abs(j1 - j2), min(J, j1 + j2) + 1, 2):
                yield j1, j2, j


def _nh(j: int) -> int:
    """Elements of the half layer of j (mb <= j / 2)."""
    return (j + 1) * (j // 2 + 1)


def z_loop_counts(J: int) -> tuple[int, int, int]:
    """(jobs, outer iterations, inner iterations) of the Z contraction."""
    jobs = outer = inner = 0
    for j1, j2, j in _triples(J):
        for mb in range(j // 2 + 1):
            for ma in range(j + 1):
                jobs += 1
                ma1lo = max(0, (2 * ma - j - j2 + j1) // 2)
                ma1hi = min(j1, (2 * ma - j + j2 + j1) // 2)
                mb1lo = max(0, (2 * mb - j - j2 + j1) // 2)
                mb1hi = min(j1, (2 * mb - j + j2 + j1) // 2)
                na, nb = max(0, ma1hi - ma1lo + 1), max(0, mb1hi - mb1lo + 1)
                outer += na
                inner += na * nb
    return jobs, outer, inner


def snap_flops(twojmax: int, ninside: float) -> dict:
    """Per-atom operation counts of one force evaluation (see the module doc)."""
    J, n = twojmax, float(ninside)
    half = sum(_nh(j) for j in range(1, J + 1))  # half-layer elements, layers 1..J
    nyh = sum(_nh(j) for j in range(J + 1))
    # per-neighbour scalars (mixed form's closed forms; the FP64 form's
    # reference formulas are within a few operations of it): r, two sincos,
    # two divisions, a, b and their twelve derivatives, the switching function
    # and the r^-12 repulsion
    scalars = n * 80.0
    # B: 14 per element per neighbour (two complex multiply-adds), the layer
    # sums (2 per neighbour per element incl. layer 0) and the 1/f scaling
    b_stage = n * 14.0 * half + n * 2.0 * nyh + 4.0 * nyh
    # C: Z (complex product 6, CG scale 2, accumulate 2 per inner; 4 per
    # outer), Y (4 per job, 2 for the w / f scale per element)
    jobs, outer, inner = z_loop_counts(J)
    c_stage = 10.0 * inner + 4.0 * outer + 4.0 * jobs + 2.0 * nyh
    # D (reverse mode), per neighbour: forward 14 + 4 (Phi) per half element,
    # adjoint 18 per half element and 16 per gathered layer-(j-1) element,
    # then the pair force (3 components of about ten) and the lane sums
    gathered = sum(j * (j // 2 + 1) for j in range(2, J + 1))
    d_sweeps = n * (18.0 * half + 18.0 * half + 16.0 * gathered + 31.0 + 3 * 31.0)
    d_tail = n * (3.0 + 3.0 + 12.0)  # repulsion add, scatter, sum for i (FP64)
    total = scalars + b_stage + c_stage + d_sweeps + d_tail
    return {
        "twojmax": J,
        "ninside": n,
        "phases": {"scalars": scalars, "B": b_stage, "C": c_stage, "D": d_sweeps + d_tail},
        "total": total,
        "fp64": {"mixed": scalars + b_stage + d_tail, "fp64": total},
        "fp32": {"mixed": c_stage + d_sweeps, "fp64": 0.0},
    }


def _entries(J: int):
    """(T, q, highest k) of the separated elements conj(a)^q b^T P_k(x)."""
    for T in range(J + 1):
        for q in range(J - T + 1):
            yield T, q, (J - T - q) // 2


def product_counts(J: int) -> tuple[int, int, int]:
    """(products, weighted products, Z values) of the shared-product contraction:
    each U_j1 U_j2 product of one (m, m') once, weighted for every j; for j1 = j2
    the two orders of a pair are one product."""
    products = weighted = zs = 0
    for T, q, _ in _entries(J):
        for sign in ((1, -1) if T and q else (1,)):
            for j1 in range(J + 1):
                for j2 in range(j1 + 1):
                    hi = min(J - ((J + j1 + j2) & 1), j1 + j2)
                    if (j1 + j2 - q - T) & 1 or hi < max(j1 - j2, q + T):
                        continue
                    nj = (hi - max(j1 - j2, q + T)) // 2 + 1
                    M, Mp = (j1 + j2 - q - sign * T) // 2, (j1 + j2 - q + sign * T) // 2
                    na, nb = min(j1, M) - max(0, M - j2) + 1, min(j1, Mp) - max(0, Mp - j2) + 1
                    n = na * nb
                    if j1 == j2:  # pairs and the self-paired one, where there is one
                        n = (n + (1 if M % 2 == 0 and Mp % 2 == 0 else 0)) // 2
                    products += n
                    weighted += n * nj
                    zs += nj
    return products, weighted, zs


def kernel_flops(twojmax: int, ninside: float) -> dict:
    """Per-atom operation counts of the kernels' own formulation."""
    J, n = twojmax, float(ninside)
    sums = sum((j + 1) ** 2 for j in range(J + 1))
    # U, per neighbour: powers of a and b (6 each), x, their products with the
    # powers of x, one multiply-add per real sum; the sums are combined into the
    # polynomials' once per atom
    powers = sum((2 if T else 1) * ((J - T) // 2) for T in range(J + 1))
    combine = sum((2 if T else 1) * (2 if q else 1) * (k + 1) * (k + 2) for T, q, k in _entries(J))
    u_stage = n * (12.0 * J + 7 + 2.0 * sums + powers) + 3.0 * sums + combine
    products, weighted, zs = product_counts(J)
    y_stage = 6.0 * products + 4.0 * weighted + 4.0 * zs
    # pair forces, per neighbour: powers, P and P' (9 from k = 2 on), their sums
    # with E and O (values and derivatives), the sums over q and over T
    force = 12.0 * J + 7 + 60.0
    for T, q, k in _entries(J):
        w = 2 if T else 1
        force += (1 if k else 0) + 9 * max(0, k - 1) + w * (4 * min(k, 1) + 8 * max(0, k - 1)) + w * (24 if q else 4)
    force += 22.0 * J
    # the mixed form's FP64: r^2, the r^-14 term and the force sums; its scalars and
    # U sums run in FP32 pairs, each operation counted once although a product
    # takes six
    scalars, tail = n * 80.0, n * 26.0
    return {
        "twojmax": J,
        "ninside": n,
        "phases": {"scalars": scalars, "U": u_stage, "Y": y_stage, "force": n * force + tail},
        "total": scalars + u_stage + y_stage + n * force + tail,
        "fp64": {"mixed": tail, "fp64": scalars + u_stage + y_stage + n * force + tail},
        "fp32": {"mixed": scalars + u_stage + y_stage + n * force, "fp64": 0.0},
    }


__all__ = ["snap_flops", "z_loop_counts", "kernel_flops", "product_counts"]
