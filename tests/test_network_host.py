"""When a forward pass may be one library call: decided on the host, tested without a GPU (the passes
themselves: tests/test_network_gpu.py)."""
import sys
import types

import pytest
import torch

from strata_b200 import _lib, network
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


def described(m, device="cpu"):
    return network.Described(*parts(m), torch.device(device))


@pytest.fixture(autouse=True)
def no_tables(monkeypatch):
    # (laying out the conditioning table is the one step of a description that needs the GPU)
    monkeypatch.setattr(_lib, "load", lambda: types.SimpleNamespace(
        strata_adaln_cond_table_floats=lambda *a: 0))


def is_stock(m):
    s = described(m)
    assert (s.desc is not None) == s.stock
    return s.stock


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


# ------------------------------------------------------------------ what the library call is handed
@pytest.mark.parametrize("two_stage", [False, True])
def test_host_fields_never_reach_the_library(two_stage):
    net = small_model(two_stage).strata
    x, lat = torch.zeros(1, 5, 4, 16, 16), torch.zeros(1, 16, 16)
    with pytest.raises(TypeError, match="CUDA float32"):
        net.forward_fused(x, None, lat=lat, lon=lat, concat_lat=True)


@pytest.mark.parametrize("two_stage", [False, True])
def test_weights_on_another_device_are_refused(two_stage):
    with pytest.raises(_lib.StrataLibraryError, match="is on cpu, the input on meta"):
        described(small_model(two_stage), "meta")


def _linear(n, k):
    return torch.nn.Linear(k, n)


WRONG = {
    "block 1: proj weight": lambda bb, px: setattr(bb.blocks[1].attn, "proj", _linear(64, 128)),
    "block 0: fc2 weight": lambda bb, px: bb.blocks[0].mlp.layers.__setitem__(2, _linear(128, 256)),
    "block 0: qkv weight": lambda bb, px: setattr(bb.blocks[0].attn, "qkv", _linear(256, 128)),
    "patch embedding weight": lambda bb, px: setattr(bb.patch_embed, "proj",
                                                     torch.nn.Conv3d(7, 64, (1, 4, 4), (1, 4, 4))),
    "final layer weight": lambda bb, px: setattr(px.pixel_final_layer if px else bb.final_layer, "linear",
                                                 _linear(64, 96)),
    "pixel block 1: fc1 weight": lambda bb, px: px.pixel_blocks[1].mlp.layers.__setitem__(0, _linear(256, 128)),
    "pixel block 0: modulation weight": lambda bb, px: setattr(px.pixel_blocks[0], "adaln_bilinear_dw_proj",
                                                               _linear(320, 128)),
}


@pytest.mark.parametrize("two_stage,what", [(t, w) for w in WRONG for t in (False, True)
                                            if t or not w.startswith("pixel")])
def test_weights_of_another_shape_are_refused(two_stage, what):
    m = small_model(two_stage)
    assert described(m).desc is not None
    WRONG[what](*parts(m))
    with pytest.raises(ValueError, match=what + " must have shape"):
        described(m)


# ------------------------------------------------------------------ what a description was read from
CHANGES = {
    "weight in place": lambda bb: bb.blocks[1].attn.proj.weight.mul_(2),
    "parameter": lambda bb: setattr(bb.blocks[0].attn.qkv, "weight", torch.nn.Parameter(torch.zeros(384, 128))),
    "module": lambda bb: bb.blocks[0].mlp.layers.__setitem__(2, _linear(128, 512)),
    "block gone": lambda bb: bb.blocks.__delitem__(1),
    "window": lambda bb: setattr(bb.blocks[0], "kernel", (3, 5, 5)),
    "q/k norm": lambda bb: setattr(bb.blocks[0], "qk_norm", True),
    "exact GELU": lambda bb: setattr(bb.blocks[0].mlp.layers[1], "approximate", "none"),
    "output channels": lambda bb: setattr(bb, "out_channels", 3),
    "dtype": lambda bb: bb.double(),
}


@pytest.mark.parametrize("two_stage", [False, True])
@pytest.mark.parametrize("what", CHANGES)
def test_a_changed_model_is_described_again(what, two_stage):
    m = small_model(two_stage)
    s = described(m)
    assert s.current(*parts(m), torch.device("cpu")) and not s.current(*parts(m), torch.device("meta"))
    with torch.no_grad():
        CHANGES[what](parts(m)[0])
    assert not s.current(*parts(m), torch.device("cpu"))


@pytest.mark.parametrize("two_stage", [False, True])
def test_a_described_model_is_freed_at_once(two_stage):
    """Its weights and their copies do not wait for the garbage collector."""
    import gc
    import weakref
    m = small_model(two_stage)
    m.strata._network._state = described(m)
    refs = [weakref.ref(t) for t in (m.strata, m.strata._network._state, parts(m)[0].blocks[0].attn.qkv.weight,
                                     parts(m)[0].blocks[0]._bf16_cache["w_qkv"])]
    gc.collect()
    gc.disable()
    try:
        del m
        assert [r() for r in refs] == [None] * 4
    finally:
        gc.enable()


@pytest.mark.parametrize("two_stage", [False, True])
def test_threads_share_a_model(two_stage, monkeypatch):
    """First calls and calls after a change, from several threads at once: none sees half a description,
    and none the sizes of another thread's call."""
    import threading
    m = small_model(two_stage)
    sizes, seen, errors = {}, [], []

    def forward_f32(dref, pref, x, lat, lon, B, D, H, W, *rest):
        d = dref._obj
        seen.append((threading.get_ident(), d.in_channels, d.concat_lat, d.u_idx, B))
        return 0
    monkeypatch.setattr(_lib, "load", lambda: types.SimpleNamespace(
        strata_adaln_cond_table_floats=lambda *a: 0, strata_network_workspace_bytes=lambda *a: 256,
        strata_network_forward_f32=forward_f32))
    monkeypatch.setattr(_lib, "on_device", lambda t: _lib._NOTHING)
    monkeypatch.setattr(_lib, "stream_of", lambda t: 0)
    monkeypatch.setattr(network.ops, "network_inputs", lambda x, lat, lon, c, bb: (x, lat, lon))
    bb, px = parts(m)
    start = threading.Barrier(6)

    def work(i):
        try:
            x, lat = torch.zeros(1 + i, 5 + 2 * (i % 2), 4, 16, 16), torch.zeros(1 + i, 16, 16)
            sizes[threading.get_ident()] = (x.shape[1], (i + 1) % 2, i - 1, 1 + i)
            for step in range(40):
                start.wait(60)
                if i == 0 and step % 4 == 0:
                    m.strata._network = network.NetworkHandle()
                y = m.strata._network.forward(bb, px, x, lat, lat, None if i == 0 else (i - 1, i), i % 2 == 0)
                assert y.shape == (1 + i, 4, 4, 16, 16)
        except BaseException as e:
            errors.append(e)
            start.abort()
    switch = sys.getswitchinterval()
    sys.setswitchinterval(1e-5)
    try:
        threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
        [t.start() for t in threads]
        [t.join() for t in threads]
    finally:
        sys.setswitchinterval(switch)
    assert not errors, errors
    assert len(seen) == 6 * 40 and all((s[1:]) == sizes[s[0]] for s in seen)


@pytest.mark.parametrize("settled", [True, False])
def test_casts_are_kept_only_once_settled(settled, monkeypatch):
    """What a module keeps for later calls was waited for; under capture (not settled) nothing is kept."""
    calls = []
    monkeypatch.setattr(_lib, "settle", lambda device: calls.append(device) or settled)
    bb, px = parts(small_model(True))
    makers = [bb.patch_embed._gemm_weights, px.pixel_final_layer._gemm_weights, bb.blocks[0].device_weights,
              px.pixel_blocks[1].device_weights]
    for make in makers:
        n = len(calls)
        first = make()
        assert len(calls) == n + 1
        assert (make() is first) == settled and len(calls) == n + (1 if settled else 2)


@pytest.mark.parametrize("settled", [True, False])
@pytest.mark.parametrize("two_stage", [False, True])
def test_a_description_waits_once(two_stage, settled, monkeypatch):
    calls = []
    monkeypatch.setattr(_lib, "settle", lambda device: calls.append(device) or settled)
    m = small_model(two_stage)
    with _lib.settled_together(torch.device("cpu")) as new:
        assert described(m).desc is not None
        kept = [b._bf16_cache for b in parts(m)[0].blocks]
        assert not calls and kept == [None, None]
    assert len(calls) == 1 and new.kept == settled
    assert all((b._bf16_cache is not None) == settled for b in parts(m)[0].blocks)
    with _lib.settled_together(torch.device("cpu")) as new:
        described(m)
    assert len(calls) == (1 if settled else 2)          # nothing new: nothing to wait for
    with pytest.raises(KeyError):
        with _lib.settled_together(torch.device("cpu")) as new:
            small_model().strata.blocks[0].device_weights()
            raise KeyError
    assert not new.kept and len(calls) == (1 if settled else 2) and _lib._filling.stores is None


def test_streams_are_found_without_the_private_lookup(monkeypatch):
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream",
                        lambda index: types.SimpleNamespace(cuda_stream=1000 + index))
    monkeypatch.setattr(_lib, "_current_stream", None)
    t = types.SimpleNamespace(device=torch.device("cuda", 3))
    assert _lib.stream_of(t) == 1003
