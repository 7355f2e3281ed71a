"""The packed instance is a copy of its own with resolved values, whatever view of memory the circuit is: the adjoint
and the conjugate are lazy views, a transpose shares memory, and the columns of a run of modes are a slice."""
import pytest
import torch

from photonic_engines_b200.clifford.kernels import pack_instances

VIEWS = {
    "plain": lambda V: V,
    "adjoint": lambda V: V.mH,
    "transpose": lambda V: V.mT,
    "conjugate": lambda V: V.conj(),
    "conjugate_of_column_major": lambda V: V.mT.contiguous().mT.conj(),
    "negative_view": lambda V: torch._neg_view(V),
    "strided": lambda V: torch.cat([V, V], dim=-1).contiguous()[..., ::2],
}


@pytest.mark.parametrize("modes", [[0, 1, 2], [1, 2], [0, 2, 5], [2, 1], [0, 0], list(range(6)), []])
@pytest.mark.parametrize("batch", [0, 1, 3])
@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("view", sorted(VIEWS))
def test_packed_columns_are_a_resolved_copy(view, dtype, batch, modes):
    shape = (6, 6) if batch == 0 else (batch, 6, 6)
    U = VIEWS[view](torch.randn(*shape, dtype=dtype, generator=torch.Generator().manual_seed(len(view))))
    acol, off, mm, nn = pack_instances(U, modes)
    want = U.resolve_conj().resolve_neg().clone().reshape(-1, 6, 6)[:, :, modes].to(torch.complex128).mT
    assert acol.dtype == torch.complex128 and acol.is_contiguous() and not acol.is_conj() and not acol.is_neg()
    assert torch.equal(acol, want)
    torch.view_as_real(acol)                                     # what the launches pass on
    assert acol.numel() == 0 or acol.untyped_storage().data_ptr() != U.untyped_storage().data_ptr()
    shared = pack_instances(U, modes, copy=False)[0]
    assert shared.dtype == torch.complex128 and shared.is_contiguous() and not shared.is_conj() and not shared.is_neg()
    assert torch.equal(shared, want)
    assert off.tolist() == [b * len(modes) * 6 for b in range(max(batch, 1))]
    assert mm.tolist() == [6] * max(batch, 1) and nn.tolist() == [len(modes)] * max(batch, 1)


def test_shared_columns_are_the_circuits_memory_only_where_the_kernels_can_read_it():
    """The kernels load 16 bytes at a time: a column-major circuit at an odd multiple of 8 bytes is copied."""
    n, m = 3, 6
    buf = torch.randn(2 * m * m + 4, dtype=torch.float64)
    first = (buf.data_ptr() // 8) % 2                            # 16-byte aligned start, in doubles
    for shift in (0, 1):
        raw = buf.numpy()[first + shift:][:2 * m * m]
        U = torch.from_numpy(raw.view("complex128").reshape(m, m)).mT
        assert U.data_ptr() % 16 == 8 * shift
        acol = pack_instances(U, range(n), copy=False)[0]
        assert (acol.data_ptr() == U.data_ptr()) == (shift == 0) and acol.data_ptr() % 16 == 0
        assert torch.equal(acol[0], U[:, :n].mT)
