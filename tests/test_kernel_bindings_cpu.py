"""Python bindings of the kernels against a library that only notes its calls."""
import pytest
import torch

from hcache_deepspeed_b200.ops import kernels


class Library:

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *a: self.calls.append(name) or 0


def test_refused_norm_leaves_nothing_armed(monkeypatch):
    """The place for 8-bit codes is told to the library ahead of the norm that writes them: a call that is refused before that norm may not
    leave it there for the next one."""
    lib = Library()
    monkeypatch.setattr(kernels.native, "cuda_lib", lambda: lib)
    x = torch.zeros(2, 16)      # fp32: not a type of this kernel
    with pytest.raises(TypeError):
        kernels.norm(x, torch.ones(16), torch.empty(2, 16), fp8=(torch.zeros(2, 16, dtype=torch.uint8), torch.zeros(2)))
    assert lib.calls == []
