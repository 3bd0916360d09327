"""Which tensors the autograd functions may hand over as pointers (no GPU)."""
import torch

from lynx_b200.autograd import _has_memory


def test_plain_tensors_have_memory():
    assert _has_memory(torch.ones(3)) and _has_memory(torch.ones(4, 3)[:, 1])


def test_batched_and_negated_tensors_have_not():
    seen = []
    torch.func.vmap(lambda t: seen.append(_has_memory(t)) or t)(torch.ones(2, 3))
    assert seen == [False]
    assert not _has_memory(torch.ones(3, dtype=torch.complex128).conj().imag)
