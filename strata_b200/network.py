"""Host side of `strata_network_forward_f32`: the descriptors of a live model, kept until one of
its parameters or modules changes, so that a forward pass is one call into the library.

A pass over a small tile is paced by the host: with a Python call per kernel the 25 launches of a
two-block model cost four times what the kernels take.
"""
from __future__ import annotations

import ctypes

import torch
from torch.nn.modules import module as _nn_module

from . import _lib, ops

_ROPE_MODES = {"none": 0, "axial": 1, "stereographic": 2}
_BLOCK_KEYS = ("qkv", "proj", "gate", "fc1", "fc2")


def _ptr(t):
    return None if t is None else t.data_ptr()


def _block_struct(weights: dict, out) -> None:
    for name in _BLOCK_KEYS:
        setattr(out, f"w_{name}", _ptr(weights.get(f"w_{name}")))
        setattr(out, f"b_{name}", _ptr(weights.get(f"b_{name}")))


class Stock:
    """A module class whose step the library call stands in for, with the methods that step goes
    through. The call may do so only where nothing else would have run: no subclass, no method replaced
    on the object or on the class and, for a module that the step calls (`called`), no hook."""

    HOOKS = ("_forward_hooks", "_forward_pre_hooks", "_backward_hooks", "_backward_pre_hooks")

    def __init__(self, cls, *methods, called=False):
        self.cls = cls
        self._lookup = vars(cls).get
        self._functions = {n: vars(cls)[n] for n in methods}
        self._stock = list(self._functions.values())
        # (_call_impl and _compiled_call_impl: what Module.__call__ and Module.compile() go through)
        self._names = (*methods, "_call_impl", "_compiled_call_impl") if called else methods
        self._hooks = self.HOOKS if called else ()

    def class_intact(self) -> bool:
        return list(map(self._lookup, self._functions)) == self._stock

    def holds(self, m) -> bool:
        if type(m) is not self.cls:
            return False
        v = vars(m)
        for n in self._names:
            if n in v:
                return False
        for h in self._hooks:
            if v[h]:
                return False
        return True

    def replaced(self, m, *methods) -> bool:
        """Whether m has one of these methods from somewhere else than the class."""
        return any(n in vars(m) or getattr(type(m), n) is not self._functions[n] for n in methods)


def _stock_parts(backbone, pixel):
    """(module, Stock) of every module whose own code a step-by-step pass would run."""
    out = [(backbone, STOCK["backbone"]), (backbone.patch_embed, STOCK["patch_embed"])]
    out += [(b, STOCK["block"]) for b in backbone.blocks]
    head = backbone.final_layer
    if pixel is not None:
        out += [(pixel, STOCK["pixel"]), (pixel.pixel_patch_embed, STOCK["patch_embed"])]
        out += [(b, STOCK["pixel_block"]) for b in pixel.pixel_blocks]
        head = pixel.pixel_final_layer
    return out + [(head, STOCK["final_layer"])]


_GLOBAL_HOOKS = tuple("_global" + h for h in Stock.HOOKS)


def _global_hooks() -> bool:
    """Hooks registered for every module (they run when a block is called)."""
    for name in _GLOBAL_HOOKS:
        if getattr(_nn_module, name, None):
            return True
    return False


# filled in by the modules that define the classes
STOCK: dict[str, Stock] = {}


class NetworkHandle:
    """Descriptors for one `StrataTransformer3D` (and, for the two-stage model, the `Strata` module
    around it). Belongs to the module that owns it; a copy of the module starts with an empty one."""

    def __init__(self):
        self._clear()

    def _clear(self):
        self._modules = self._params = self._attrs = None
        self._desc = self._pixel = None
        self._keep = None
        self._parts = self._classes = ()

    def __deepcopy__(self, memo):
        return NetworkHandle()

    def __reduce__(self):
        return (NetworkHandle, ())

    # ---------------------------------------------------------------- what may change
    def _watch(self, root, attrs) -> None:
        self._modules = [(m._modules, tuple(m._modules.items())) for m in root.modules() if m._modules]
        self._params = [(m._parameters, k, p, p.data_ptr(), p._version)
                        for m in root.modules() for k, p in m._parameters.items() if p is not None]
        self._attrs = attrs

    def _unchanged(self) -> bool:
        if self._modules is None:
            return False
        for d, items in self._modules:
            if len(d) != len(items):
                return False
            for k, m in items:
                if d.get(k) is not m:
                    return False
        for d, k, p, ptr, version in self._params:
            if d.get(k) is not p or p._version != version or p.data_ptr() != ptr:
                return False
        for obj, name, value in self._attrs:
            if getattr(obj, name, None) != value:
                return False
        return True

    def _take_parts(self, backbone, pixel) -> None:
        self._parts = _stock_parts(backbone, pixel)
        self._classes = {s for _, s in self._parts}

    def _all_stock(self) -> bool:
        for s in self._classes:
            if not s.class_intact():
                return False
        for m, s in self._parts:
            if not s.holds(m):
                return False
        return not _global_hooks()

    # ---------------------------------------------------------------- descriptors
    def _build(self, backbone, pixel) -> None:
        self._clear()
        self._take_parts(backbone, pixel)
        if not self._all_stock():
            return          # looked at again on the next call
        attrs = []
        keep = []

        def kernels_of(blocks):
            attrs.extend((b, "kernel", b.kernel) for b in blocks)
            flat = [v for b in blocks for v in b.kernel]
            return (ctypes.c_int32 * max(len(flat), 1))(*flat)

        def same(blocks, name, default):
            attrs.extend((b, name, getattr(b, name)) for b in blocks)
            values = {getattr(b, name) for b in blocks} or {default}
            return values.pop() if len(values) == 1 else None

        def usable(blocks):
            for b in blocks:
                attrs.append((b.mlp.layers[1], "approximate", "tanh"))
            return all(b._gelu_is_tanh() for b in blocks)

        bb = backbone
        blocks = list(bb.blocks)
        ok = usable(blocks) and same(blocks, "num_heads", bb.num_heads) == bb.num_heads
        qk_norm = same(blocks, "qk_norm", False)
        ok = ok and qk_norm is not None
        d = _lib.BackboneDesc()
        d.out_channels = bb.out_channels
        d.patch_v, d.patch_h, d.patch_w = bb.patch_size
        d.dim, d.heads, d.n_blocks = bb.embed_dim, bb.num_heads, len(blocks)
        d.hidden = blocks[0].mlp.layers[0].out_features if blocks else bb.embed_dim
        ok = ok and all(b.mlp.layers[0].out_features == d.hidden for b in blocks)
        d.qk_norm = 1 if qk_norm else 0
        wm, bias, _, kp = bb.patch_embed._gemm_weights()
        keep += [wm, bias]
        d.w_embed, d.b_embed, d.k_embed = _ptr(wm), _ptr(bias), kp
        structs = (_lib.BlockWeights * max(len(blocks), 1))()
        for s, b in zip(structs, blocks):
            w = b.device_weights()
            keep.append(w)
            _block_struct(w, s)
        kern = kernels_of(blocks)
        d.h_blocks = ctypes.cast(structs, ctypes.POINTER(_lib.BlockWeights))
        d.h_kernels = ctypes.cast(kern, ctypes.POINTER(ctypes.c_int32))
        keep += [structs, kern]
        if bb.final_layer is not None:
            d.w_head, d.b_head, d.n_head = self._head(bb.final_layer, keep)
        px = None
        if pixel is not None:
            pblocks = list(pixel.pixel_blocks)
            ok = ok and usable(pblocks) and same(pblocks, "num_heads", pixel.num_heads_pixel) == pixel.num_heads_pixel
            pqk = same(pblocks, "qk_norm", False)
            ok = ok and pqk is not None and not any(hasattr(b, "adaln_pixel_proj") for b in pblocks)
            px = _lib.PixelDesc()
            px.dim, px.heads, px.n_blocks = pixel.embed_dim_pixel, pixel.num_heads_pixel, len(pblocks)
            px.hidden = pblocks[0].mlp.layers[0].out_features if pblocks else pixel.embed_dim_pixel
            ok = ok and all(b.mlp.layers[0].out_features == px.hidden for b in pblocks)
            px.qk_norm = 1 if pqk else 0
            wm, bias, _, kp = pixel.pixel_patch_embed._gemm_weights()
            keep += [wm, bias]
            px.w_embed, px.b_embed, px.k_embed = _ptr(wm), _ptr(bias), kp
            if ok:
                px.cond_ks = self._pixel_blocks(pblocks, bb, px, keep)
                ok = px.cond_ks is not None
            kern = kernels_of(pblocks)
            px.h_kernels = ctypes.cast(kern, ctypes.POINTER(ctypes.c_int32))
            keep.append(kern)
            px.w_head, px.b_head, px.n_head = self._head(pixel.pixel_final_layer, keep)
        self._keep = keep
        if ok:
            self._desc, self._pixel = d, px
        self._watch(backbone if pixel is None else pixel, attrs)

    @staticmethod
    def _head(layer, keep):
        layer._refresh()
        wm, b, _ = layer._gemm_cache
        keep += [wm, b]
        return _ptr(wm), _ptr(b), wm.shape[0]

    @staticmethod
    def _pixel_blocks(pblocks, bb, px, keep):
        """Fills px.h_blocks; returns the depthwise kernel size (0: no block is modulated, None:
        the blocks disagree)."""
        lib = _lib.load()
        structs = (_lib.PixelBlockWeights * max(len(pblocks), 1))()
        sizes = set()
        for s, b in zip(structs, pblocks):
            w = b.device_weights()
            keep.append(w)
            _block_struct(w, s.block)
            if "w_mod" not in w:
                continue
            ks = w["w_dw"].shape[-1]
            sizes.add(ks)
            s.w_dw, s.b_dw = _ptr(w["w_dw"]), _ptr(w["b_dw"])
            s.w_mod, s.b_mod = _ptr(w["w_mod"]), _ptr(w["b_mod"])
            n = int(lib.strata_adaln_cond_table_floats(bb.embed_dim, bb.patch_size[1], ks))
            if n:
                table = torch.empty(n, dtype=torch.float32, device=w["w_dw"].device)
                with torch.cuda.device(table.device):
                    _lib.check(lib.strata_adaln_cond_table_f32(
                        w["w_dw"].data_ptr(), bb.embed_dim, bb.patch_size[1], ks, table.data_ptr(),
                        torch.cuda.current_stream().cuda_stream), "strata_adaln_cond_table_f32")
                keep.append(table)
                s.cond_table = table.data_ptr()
        px.h_blocks = ctypes.cast(structs, ctypes.POINTER(_lib.PixelBlockWeights))
        keep.append(structs)
        return None if len(sizes) > 1 else (sizes.pop() if sizes else 0)

    # ---------------------------------------------------------------- one pass
    def forward(self, backbone, pixel, x, lat, lon, wind, concat_lat):
        """x [B, C, D, H, W] fp32, lat / lon [B, H, W] fp32 on x's device -> fields, or None when
        the model has a part that only the step-by-step path runs."""
        if not (self._unchanged() and self._all_stock()):
            self._build(backbone, pixel)
        d, px = self._desc, self._pixel
        if d is None:
            return None
        x = x if x.is_contiguous() else x.contiguous()
        B, C, D, H, W = x.shape
        ops._check_fields(x, lat, lon, C + (2 if concat_lat else 0), backbone)
        d.in_channels = C
        d.concat_lat = 1 if concat_lat else 0
        d.u_idx, d.v_idx = (-1, -1) if wind is None else (int(wind[0]), int(wind[1]))
        d.rope_mode = _ROPE_MODES[backbone.rope_mode]
        d.rope_length_scale, d.rope_base = float(backbone.rope_length_scale), float(backbone.rope_base)
        pref = None
        if px is not None:
            px.rope_mode = _ROPE_MODES[pixel.rope_mode_pixel]
            px.rope_length_scale = float(pixel.rope_length_scale_pixel)
            px.rope_base = float(pixel.rope_base_pixel)
            pref = ctypes.byref(px)
        lib = _lib.load()
        dref = ctypes.byref(d)
        need = lib.strata_network_workspace_bytes(dref, pref, B, D, H, W)
        if need < 0:
            raise ValueError(f"input {tuple(x.shape)} does not fit the model (patch "
                             f"{backbone.patch_size})")
        out = torch.empty((B, backbone.out_channels, D, H, W), dtype=torch.float32, device=x.device)
        ws = torch.empty(max(need, 256), dtype=torch.uint8, device=x.device)
        with _lib.on_device(x):
            _lib.check(lib.strata_network_forward_f32(
                dref, pref, x.data_ptr(), lat.data_ptr(), lon.data_ptr(), B, D, H, W, out.data_ptr(),
                ws.data_ptr(), need, _lib.stream_of(x)),
                "strata_network_forward_f32")
        return out
