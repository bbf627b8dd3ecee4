"""A diffusion block's norms run inside other kernels only where nobody would notice."""
import torch
import torch.nn.modules.module as every

from dew_b200.nn.dit import _bare
from dew_b200.nn.layers import LayerNorm


def test_a_norm_that_is_watched_or_replaced_is_called():
    norm = LayerNorm(8, affine=False)
    assert _bare(norm) and not _bare(LayerNorm(8)) and not _bare(torch.nn.Identity())
    look = lambda *args: None
    for register in (norm.register_forward_hook, norm.register_forward_pre_hook, norm.register_full_backward_hook, norm.register_full_backward_pre_hook,
                     every.register_module_forward_hook, every.register_module_forward_pre_hook, every.register_module_full_backward_hook,
                     every.register_module_full_backward_pre_hook):
        handle = register(look)
        assert not _bare(norm), register
        handle.remove()
    assert _bare(norm)
    norm.forward = lambda x: x
    assert not _bare(norm)
