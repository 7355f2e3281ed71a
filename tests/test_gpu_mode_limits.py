"""The most modes a CTA-form call may have: the layout of shared memory leaves 227 KB less its own size for one draw
weight per mode, and a layout that grows refuses calls that ran.  Chains of two photons in launches compiled for up to
n columns; their rows equal those of the FP64 form in the one-warp layout, which has no such limit."""
import numpy as np
import pytest
import torch

from photonic_engines_b200 import _native as N
from photonic_engines_b200.clifford.kernels import chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n,m", [("f64", 8, 23206), ("f64", 20, 23206), ("f64", 32, 23206), ("mixed", 20, 23206),
                                           ("mixed", 32, 23206), ("compensated", 20, 22182), ("compensated", 32, 22182),
                                           ("f64", 33, 17328), ("f64", 64, 17328)])
def test_largest_mode_counts(precision, n, m):
    assert N.load().pe_max_modes(0) >= 23206
    dev, S = torch.device("cuda"), 16
    g = torch.Generator(device=dev).manual_seed(n)
    acol = torch.view_as_complex(torch.randn(1, n, m, 2, generator=g, dtype=torch.float64, device=dev))
    off, mm, nn = (torch.tensor([x], dtype=t, device=dev) for x, t in ((0, torch.int64), (m, torch.int32), (n, torch.int32)))
    dp = torch.zeros(S, dtype=torch.int64, device=dev)
    cols = torch.argsort(torch.rand(S, n, generator=g, device=dev), dim=1)
    u = torch.rand(S, n, generator=g, dtype=torch.float64, device=dev)
    nk = torch.full((S,), 2, dtype=torch.int32, device=dev)
    rows = chain(acol, off, mm, nn, dp, cols, m_max=m, nk=nk, uniforms=u, precision=precision, mode="cta")[0]
    ref = chain(acol, off, mm, nn, dp, cols[:, :2].contiguous(), m_max=m, uniforms=u[:, :2].contiguous(), mode="warp")[0]
    assert np.array_equal(rows.cpu().numpy()[:, :2], ref.cpu().numpy())
