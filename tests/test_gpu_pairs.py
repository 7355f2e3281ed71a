"""The FP64 pair sweep (csrc/fock_pairs.cuh) at the edges of its tiers and of its rule: cofactors against the
long-double oracle.  A step runs it from 9 to 32 columns when at least two chosen rows have multiplicity 1 beside the
halved one; otherwise the term-by-term sweep does.  Tolerance: the FP64 bound of the parity tests (1e-10 to 24
columns, 1.8 times more per column beyond: the oracle's own FP64 sums deviate that much at 2^(K - 2) terms)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from photonic_engines_b200.clifford import laplace_cofactors_rows

pytestmark = pytest.mark.gpu


def _rows(K1: int, ones: int, mult: int) -> np.ndarray:
    """K1 chosen rows: `ones` modes once, the others `mult` times each (the last one takes what is left)."""
    rows = list(range(ones))
    mode = ones
    while len(rows) < K1:
        rows += [mode] * min(mult, K1 - len(rows))
        mode += 1
    return np.array(rows)


def _check(K: int, rows: np.ndarray, block: int = 128, tpl: int | None = None):
    S, m, K1 = 3, int(rows.max()) + 1, K - 1
    rng = np.random.default_rng(100 * K + len(set(rows.tolist())))
    A = rng.normal(size=(S, m, K)) + 1j * rng.normal(size=(S, m, K))
    R = np.stack([rng.permutation(rows) for _ in range(S)])
    P = laplace_cofactors_rows(torch.tensor(A, device="cuda"), torch.tensor(R, device="cuda"), block_threads=block,
                               tpl=tpl or (1 if K <= 20 else 2)).cpu().numpy()
    tol = 1e-10 * 1.8 ** max(0, K - 24)
    for s in range(S):
        ref, _ = O.cofactors(A[s][R[s]], R[s], precision="ld")
        assert np.abs(P[s] - ref).max() <= tol * np.abs(ref).max(), (K, rows.tolist(), s)


@pytest.mark.parametrize("K", [9, 10, 11, 12, 13, 16, 17, 18, 19, 20])
def test_tier_edges_with_distinct_rows(K):
    _check(K, _rows(K - 1, K - 1, 2))


@pytest.mark.parametrize("K", [21, 24, 25, 28, 29, 32])
def test_wide_tiers_with_repeated_rows(K):
    _check(K, _rows(K - 1, 5, 4))


@pytest.mark.parametrize("ones", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("K", [9, 18, 23])
def test_the_rule_around_two_single_rows(K, ones):
    _check(K, _rows(K - 1, ones, 3))


def test_zero_columns_stay_exact_and_lanes_of_a_small_cta():
    """Two zero columns in different pairs, and in one pair: every cofactor exactly zero; one warp per CTA."""
    rng = np.random.default_rng(5)
    K = 14
    for zero in ((0, 1), (2, 7)):
        A = rng.normal(size=(2, K, K)) + 1j * rng.normal(size=(2, K, K))
        A[:, :, list(zero)] = 0
        rows = torch.arange(K - 1, device="cuda").expand(2, -1)
        P = laplace_cofactors_rows(torch.tensor(A, device="cuda"), rows, block_threads=128, tpl=1).cpu().numpy()
        assert np.abs(P).max() == 0.0
    _check(K, _rows(K - 1, K - 1, 2), block=32)
