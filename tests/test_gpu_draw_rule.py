"""The CTA form's draw, bit by bit: modes in contiguous runs per thread, their sums scanned within a warp, the warps in
order, tot = cw[m - 1] as the last mode's thread forms it, marginal = weight / tot, and the pick
min(#{rho : cw[rho] < u tot}, m - 1).  One photon in a real circuit: the weights are squares rounded once, so the whole
draw can be followed in NumPy and compared exactly; uniforms at and next to 1 and trailing modes without weight."""
import numpy as np
import pytest
import torch

from photonic_engines_b200.clifford import sample_chains

pytestmark = pytest.mark.gpu


def _cumulative(w: np.ndarray, T: int) -> np.ndarray:
    m = len(w)
    C = (m + T - 1) // T
    lo = np.minimum(np.arange(T) * C, m)
    hi = np.minimum(lo + C, m)
    x = np.zeros(T)
    for i in range(C):
        use = lo + i < hi
        x[use] = x[use] + w[(lo + i)[use]]
    x = x.reshape(-1, 32)
    for o in (1, 2, 4, 8, 16):
        y = x.copy()
        x[:, o:] = y[:, o:] + y[:, :-o]
    E, before = np.zeros(T), 0.0
    for v in range(T // 32):
        for lane in range(32):
            E[32 * v + lane] = before + (x[v, lane - 1] if lane else 0.0)
        before = before + x[v, 31]
    cw = np.zeros(m)
    for t in range(T):
        c = E[t]
        for i in range(lo[t], hi[t]):
            c = c + w[i]
            cw[i] = c
    return cw


@pytest.mark.parametrize("block", [32, 128, 256])
@pytest.mark.parametrize("m", [1, 2, 31, 33, 127, 128, 129, 300, 1000, 2311])
def test_marginal_and_pick(m, block):
    rng = np.random.default_rng(m + block)
    for used in sorted({m, max(1, m - m // 3)}):
        U = np.zeros((m, m))
        U[:used, 0] = rng.normal(size=used) * 10.0 ** rng.uniform(-4, 0, size=used)
        w = U[:, 0] * U[:, 0]
        cw = _cumulative(w, block)
        u = np.concatenate([[0.0, 1.0, 1 - 2.0 ** -53, 1 - 2.0 ** -24], rng.random(60)])
        out = sample_chains(torch.tensor(U, dtype=torch.complex128, device="cuda"), [0],
                            np.zeros((len(u), 1), dtype=np.int64), uniforms=u[:, None], want_marg=True, mode="cta",
                            block_threads=block)
        assert np.array_equal(out["marg"].cpu().numpy()[:, 0], np.tile(w / cw[-1], (len(u), 1)))
        want = np.minimum((cw[None, :] < (u * cw[-1])[:, None]).sum(axis=1), m - 1)
        assert np.array_equal(out["rows"].cpu().numpy()[:, 0], want)
