"""Helpers shared by the tensor classes (python/src/gelib/gelib_common.py:15-20 of GElib)."""
import torch

# Within ``with plain():`` attributes of the operands are read without the tensor classes' __torch_function__, whose Python
# handler costs several microseconds per access: a small product is bound by the host.
plain = torch._C.DisableTorchFunctionSubclass


def of_class(r, t):
    """``r``, made within ``plain()``, as the class that a torch function would have given it: t's, unless that class takes no
    part in __torch_function__ (torch.nn.Parameter: a gradient that were one would register itself as a weight)."""
    cls = type(t)
    if cls is torch.Tensor or cls.__torch_function__ is torch._C._disabled_torch_function_impl:
        return r
    return r.as_subclass(cls)


def zeros_like_all(tensors):
    """zeros_like of every tensor, filled by one launch; within ``plain()``."""
    r = [torch.empty_like(t) for t in tensors]
    if r:
        torch._foreach_zero_(r)
    return [of_class(z, t) for z, t in zip(r, tensors)]


def common_batch(x, y):
    """Batch size of a binary operation: equal batches, or one of them 1 (broadcast)."""
    assert x.dim() >= 1
    assert y.dim() >= 1
    if x.size(0) > 1 and y.size(0) > 1:
        assert x.size(0) == y.size(0)
    return max(x.size(0), y.size(0))


def output_memory(*operands):
    """torch.empty for the output of a product that writes all of it; torch.zeros when an operand is empty: the product then has
    no cells and writes nothing, and the reference's output is its zero-initialised tensor."""
    return torch.zeros if any(t.numel() == 0 for t in operands) else torch.empty
