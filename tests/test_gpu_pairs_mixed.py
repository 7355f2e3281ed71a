"""The mixed form's pair sweep (csrc/fock_pairs.cuh, sweep_pairs_mixed) at the edges of its tiers and of its rule, and the
FP64 redo of a pair step inside the guard band.

Cofactors against the long-double oracle.  A term of K columns is some 3 K complex FP32 products, each off by at most
2^-24 or so of itself, with no common sign over the terms: the sum is off by about sqrt(3 K) 2^-24 times the root of
the sum of the squared terms (column sums counted as no smaller than their rms, since their own rounding is relative to
that).  Twice that is allowed; random blocks of these shapes reached half of it at most, in the term-by-term sweep four fifths."""
from math import comb

import numpy as np
import pytest
import torch

from oracle import oracle as O
from photonic_engines_b200.clifford import laplace_cofactors_rows, sample_chains

pytestmark = pytest.mark.gpu


def _rows(K1: int, ones: int, mult: int) -> np.ndarray:
    rows = list(range(ones))
    mode = ones
    while len(rows) < K1:
        rows += [mode] * min(mult, K1 - len(rows))
        mode += 1
    return np.array(rows)


def _spread(B: np.ndarray, rows: np.ndarray) -> np.ndarray:
    """Per column: root of the sum of squares of the collapsed sum's terms, scaled as the cofactors are."""
    d, first, mult = np.unique(rows, return_index=True, return_counts=True)
    s, w = np.zeros((1, B.shape[1]), complex), np.ones(1)
    for f, M in zip(first, mult):
        v = np.arange(M + 1)
        s = (s[:, None, :] + ((M - 2 * v)[:, None] * B[f])[None]).reshape(-1, B.shape[1])
        w = (w[:, None] * np.array([comb(int(M), int(x)) for x in v])).ravel()
    a = np.abs(s)
    a = np.log(np.maximum(a, np.sqrt((w[:, None] * a * a).sum(0) / w.sum())))
    return np.sqrt(((w[:, None] * np.exp(a.sum(1, keepdims=True) - a)) ** 2).sum(0)) * 2.0 ** -len(rows)


@pytest.mark.parametrize("K,ones,mult", [(K, K - 1, 2) for K in (9, 10, 11, 12, 13, 16, 17)]
                         + [(K, ones, 2) for K in (12, 16, 20) for ones in (5, 6, 7, 8)]
                         + [(K, ones, 3) for K in (13, 21) for ones in (5, 6, 7, 8)]
                         + [(K, ones, 4) for K in (24, 25) for ones in (5, 6, 7, 8)]
                         + [(28, 6, 6), (28, 7, 6), (29, 6, 6), (32, 7, 6)])
def test_tier_edges_and_the_rule_around_six_single_rows(K, ones, mult):
    rows = _rows(K - 1, ones, mult)
    S, m = 4, int(rows.max()) + 1
    rng = np.random.default_rng(1000 * K + 10 * ones + mult)
    A = rng.normal(size=(S, m, K)) + 1j * rng.normal(size=(S, m, K))
    R = np.stack([rng.permutation(rows) for _ in range(S)])
    for block in (32, 128):
        P = laplace_cofactors_rows(torch.tensor(A, device="cuda"), torch.tensor(R, device="cuda"), precision="mixed",
                                   block_threads=block, tpl=1 if K <= 20 else 2).cpu().numpy()
        for s in range(S):
            ref, _ = O.cofactors(A[s][R[s]], R[s], precision="ld")
            tol = 2 * np.sqrt(3 * K) * 2.0 ** -24 * _spread(A[s][R[s]], R[s])
            assert (np.abs(P[s] - ref) <= tol).all(), (K, ones, block, s, np.max(np.abs(P[s] - ref) / tol))


@pytest.mark.parametrize("split", [False, (11, 4)])
@pytest.mark.parametrize("n,m,tpl", [(14, 150, 1), (18, 300, 1)])
def test_a_pair_step_inside_the_guard_band_is_redone_in_fp64(n, m, tpl, split):
    """Every uniform from the ninth step on lies 1e-9 above or below a step of the cumulative weights, inside the guard
    band and far below the FP32 blocks' error (1e-7 and more) but above FP64's: the picks are the oracle's."""
    rng = np.random.default_rng(n)
    S = 12
    U = O.haar_unitary(m, n)
    sig = np.argsort(rng.random((S, n)), axis=1)
    u = rng.random((S, n))
    dp = np.zeros(S, np.int64)
    for k in range(8, n):
        ref = O.chain(U[:, :n], dp, sig, u, marg=True)
        cw = np.cumsum(ref["marg"][:, k], axis=1)
        side = np.where(rng.random(S) < 0.5, -1e-9, 1e-9)
        u[:, k] = np.clip(cw[np.arange(S), ref["rows"][:, k]], 1e-6, 1 - 1e-6) + side
    ref = O.chain(U[:, :n], dp, sig, u, marg=False)
    out = sample_chains(torch.tensor(U, device="cuda"), list(range(n)), sig, uniforms=u, precision="mixed", tpl=tpl,
                        mode="cta", split=split)
    assert np.array_equal(out["rows"].cpu().numpy(), ref["rows"])
