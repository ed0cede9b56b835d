"""When a forward pass may be one library call: decided on the host, tested without a GPU (the passes
themselves: tests/test_network_gpu.py)."""
import types

import pytest
import torch

from strata_b200.pixel import StrataPixel3DBlock
from strata_b200.strata import FinalLayer, PatchEmbed3D, StrataTransformer3D, StrataTransformer3DBlock
from strata_b200.wrappers import StrataBackboneModel, StrataModel


def small_model(two_stage=False, **over):
    kw = dict(depth=4, height=16, width=16, n_layers=2, patch_size_horiz=4, in_chans=5, base_out_chans=4,
              embed_dim=128, num_heads=2, attn_kernel=3, do_rope_2d_stereographic=True, index_is_latlon=True)
    if two_stage:
        kw.update(embed_dim_pixel=64, n_layers_pixel=2, attn_kernel_pixel=3,
                  use_bilinear_dw_gelu_project_adaln_pixel=True)
    kw.update(over)
    return (StrataModel if two_stage else StrataBackboneModel)(**kw)


def parts(m):
    """(backbone, pixel stage or None) of a wrapper."""
    return (m.strata.backbone, m.strata) if isinstance(m, StrataModel) else (m.strata, None)


def is_stock(m):
    h = m.strata._network
    h._take_parts(*parts(m))
    return h._all_stock()


def _blocks(m):
    bb, px = parts(m)
    return (bb if px is None else px).__getattr__("blocks" if px is None else "pixel_blocks")


def _subclassed(cls, **methods):
    return type("Own" + cls.__name__, (cls,), methods)


def _swap_class(m, module, cls, **methods):
    module.__class__ = _subclassed(cls, **methods)


OWN = {
    "forward hook": lambda m: _blocks(m)[1].register_forward_hook(lambda *a: None),
    "forward pre-hook": lambda m: _blocks(m)[0].register_forward_pre_hook(lambda *a: None),
    "backward hook": lambda m: _blocks(m)[0].register_full_backward_hook(lambda *a: None),
    "block subclass": lambda m: _swap_class(m, _blocks(m)[1], type(_blocks(m)[1])),
    "block of another type": lambda m: _blocks(m).append(torch.nn.Identity()),
    "forward on the object": lambda m: setattr(_blocks(m)[0], "forward",
                                               types.MethodType(lambda s, *a, **k: a[0], _blocks(m)[0])),
    "weights on the object": lambda m: setattr(_blocks(m)[0], "device_weights", lambda: {}),
    "compiled block": lambda m: _blocks(m)[0].compile(backend="eager"),
    "backbone subclass": lambda m: _swap_class(m, parts(m)[0], StrataTransformer3D),
    "patch embedding subclass": lambda m: _swap_class(m, parts(m)[0].patch_embed, PatchEmbed3D),
}


@pytest.mark.parametrize("two_stage", [False, True])
@pytest.mark.parametrize("what", OWN)
def test_foreign_code_on_the_way_takes_the_step_by_step_path(what, two_stage):
    m = small_model(two_stage)
    assert is_stock(m)
    handle = OWN[what](m)
    assert not is_stock(m)
    if hasattr(handle, "remove"):
        handle.remove()
        assert is_stock(m)


def test_head_and_pixel_stage_subclasses_are_seen():
    m = small_model()
    _swap_class(m, m.strata.final_layer, FinalLayer)
    assert not is_stock(m)
    m = small_model(True)
    _swap_class(m, m.strata, type(m.strata))
    assert not is_stock(m)


@pytest.mark.parametrize("cls", [StrataTransformer3DBlock, StrataPixel3DBlock])
def test_a_method_replaced_on_the_class_is_seen(cls, monkeypatch):
    m = small_model(True)
    assert is_stock(m)
    monkeypatch.setattr(cls, "forward", lambda self, x, *a, **k: x)
    assert not is_stock(m)


def test_hooks_on_all_modules_are_seen():
    m = small_model()
    handle = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    try:
        assert not is_stock(m)
    finally:
        handle.remove()
    assert is_stock(m)
