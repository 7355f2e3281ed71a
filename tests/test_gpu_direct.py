"""Steps of at most 8 columns, which sum over the chosen rows directly (no plan): cofactors and whole short chains in
the warp and CTA forms against the long-double oracle.  Tolerance 1e-12 for the cofactors (at most 64 terms of FP64
products, relative to the largest cofactor; the permanents of Gaussian blocks this small lose about two digits to
cancellation), 1e-11 for normalised marginals."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from photonic_engines_b200.clifford import laplace_cofactors_rows, sample_chains

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("K", [2, 3, 4, 5, 6, 7, 8, 9])
def test_cofactors_of_small_blocks(K, precision):
    rng = np.random.default_rng(K)
    S, m = 37, max(2, K - 1)
    A = rng.normal(size=(S, m, K)) + 1j * rng.normal(size=(S, m, K))
    R = rng.integers(0, m, size=(S, K - 1))
    P = laplace_cofactors_rows(torch.tensor(A, device="cuda"), torch.tensor(R, device="cuda"),
                               precision=precision).cpu().numpy()
    tol = 1e-12 if (precision == "f64" or K <= 8) else 2e-7 * 1.35 ** K
    for s in range(S):
        ref, _ = O.cofactors(A[s][R[s]], R[s], precision="ld")
        assert np.abs(P[s] - ref).max() <= tol * np.abs(ref).max(), (K, s)


@pytest.mark.parametrize("mode", ["warp", "cta"])
@pytest.mark.parametrize("n,m", [(1, 3), (2, 2), (5, 31), (6, 32), (7, 33), (8, 64), (9, 65), (12, 130)])
def test_chains_across_the_last_direct_step(n, m, mode):
    rng = np.random.default_rng(n)
    S = 70
    U = O.haar_unitary(m, n)
    sig = np.argsort(rng.random((S, n)), axis=1)
    u = rng.random((S, n))
    ref = O.chain(U[:, :n], np.zeros(S, np.int64), sig, u, marg=True)
    out = sample_chains(torch.tensor(U, device="cuda"), list(range(n)), sig, uniforms=u, want_marg=True, mode=mode)
    assert np.array_equal(out["rows"].cpu().numpy(), ref["rows"])
    assert np.abs(out["marg"].cpu().numpy() - ref["marg"]).max() <= 1e-11
