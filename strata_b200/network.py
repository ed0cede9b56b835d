"""Host side of `strata_network_forward_f32`: the descriptors of a live model, kept until one of
its parameters or modules changes, so that a forward pass is one call into the library.

A pass over a small tile is paced by the host: with a Python call per kernel the 20 launches of a
two-block model on 32 x 32 pixels take 260 us and more, as one call 90.
"""
from __future__ import annotations

import ctypes

import torch
from torch.nn.modules import module as _nn_module

from . import _lib, ops

_ROPE_MODES = {"none": 0, "axial": 1, "stereographic": 2}


class _Weights:
    """The tensors a descriptor points to, kept with it; each has the shape the kernels will read and
    is on the device they run on."""

    def __init__(self, device):
        self.device = device
        self.keep = []

    def ptr(self, t, shape, name):
        if t is None:
            return None
        if tuple(t.shape) != shape:
            raise ValueError(f"{name} must have shape {shape}, got {tuple(t.shape)}")
        if t.device != self.device:
            raise _lib.StrataLibraryError(f"{name} is on {t.device}, the input on {self.device}")
        self.keep.append(t)
        return t.data_ptr()

    def block(self, w: dict, dim: int, hidden: int, name: str, out) -> None:
        shapes = {"qkv": (3 * dim, dim), "proj": (dim, dim), "gate": (dim, dim), "fc1": (hidden, dim),
                  "fc2": (dim, hidden)}
        for key, shape in shapes.items():
            setattr(out, f"w_{key}", self.ptr(w.get(f"w_{key}"), shape, f"{name} {key} weight"))
            setattr(out, f"b_{key}", self.ptr(w.get(f"b_{key}"), shape[:1], f"{name} {key} bias"))

    def embed(self, layer, dim: int, name: str):
        """(weight, bias, columns of the patch rows) of a patch embedding."""
        wm, bias, _, kp = layer._gemm_weights()
        return (self.ptr(wm, (dim, kp), f"{name} weight"), self.ptr(bias, (dim,), f"{name} bias"), kp)

    def head(self, layer, dim: int, name: str):
        """(weight, bias, output columns) of a final layer."""
        wm, b, _ = layer._gemm_weights()
        n = wm.shape[0]
        return self.ptr(wm, (n, dim), f"{name} weight"), self.ptr(b, (n,), f"{name} bias"), n


class Stock:
    """A module class whose step the library call stands in for, with the methods that step goes
    through. The call may do so only where nothing else would have run: no subclass, no method replaced
    on the object or on the class and, for a module that the step calls (`called`), no hook."""

    HOOKS = ("_forward_hooks", "_forward_pre_hooks", "_backward_hooks", "_backward_pre_hooks")

    def __init__(self, cls, *methods, called=False):
        self.cls = cls
        self._functions = {n: vars(cls)[n] for n in methods}
        # what the class has to hold for them, to be looked up again: (lookup, name), function
        self.lookups = [((vars(cls).get, n), f) for n, f in self._functions.items()]
        # (_call_impl and _compiled_call_impl: what Module.__call__ and Module.compile() go through)
        self._names = (*methods, "_call_impl", "_compiled_call_impl") if called else methods
        self._hooks = self.HOOKS if called else ()

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
    """(module, Stock) of every module below the two whose own code a step-by-step pass would run."""
    out = [(backbone.patch_embed, STOCK["patch_embed"])]
    out += [(b, STOCK["block"]) for b in backbone.blocks]
    head = backbone.final_layer
    if pixel is not None:
        out.append((pixel.pixel_patch_embed, STOCK["patch_embed"]))
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


class Described:
    """The descriptors of a model as it is, and what they were read from. Complete when the constructor
    returns and never written afterwards, so threads that share the model may share it; a change of the
    model makes a new one (`current`). desc is None where only the step-by-step path will do. The module
    that owns it is not referred to: with such a cycle a model's memory would wait for the collector."""

    OWN = ("out_channels", "patch_size", "embed_dim", "num_heads")
    OWN_PIXEL = ("embed_dim_pixel", "num_heads_pixel")

    def __init__(self, backbone, pixel, device):
        self.device = device
        self.desc = self.pixel = None
        self.keep = None            # owns what the descriptors point to
        self._modules = self._owners = self._params = self._ptrs = self._versions = self._attrs = ()
        self._parts = _stock_parts(backbone, pixel)
        classes = {s for _, s in self._parts} | {STOCK["backbone"]} | ({STOCK["pixel"]} if pixel is not None else set())
        lookups = [e for s in classes for e in s.lookups]
        self._lookups, self._functions = [k for k, _ in lookups], [f for _, f in lookups]
        self._own = self._owned(backbone, pixel)
        self.stock = self._all_stock(backbone, pixel)
        if self.stock:
            self._describe(backbone, pixel)

    # ---------------------------------------------------------------- what may change
    def _owned(self, backbone, pixel):
        own = [getattr(backbone, n) for n in self.OWN]
        return own if pixel is None else own + [getattr(pixel, n) for n in self.OWN_PIXEL]

    def _all_stock(self, backbone, pixel) -> bool:
        if not STOCK["backbone"].holds(backbone) or not (pixel is None or STOCK["pixel"].holds(pixel)):
            return False
        if [get(n) for get, n in self._lookups] != self._functions:
            return False
        for m, s in self._parts:
            if not s.holds(m):
                return False
        return not _global_hooks()

    def _watch(self, root, attrs) -> None:
        self._modules = [(m._modules, dict(m._modules)) for m in root.modules() if m._modules]
        self._owners = [(m._parameters, k, p) for m in root.modules() for k, p in m._parameters.items()]
        self._params = [p for _, _, p in self._owners if p is not None]
        self._ptrs = [p.data_ptr() for p in self._params]
        self._versions = [p._version for p in self._params]
        self._attrs = attrs

    def current(self, backbone, pixel, device) -> bool:
        """Whether the model is still the one described, for inputs on `device`."""
        if not self.stock or self.device != device or not self._all_stock(backbone, pixel):
            return False
        if self._owned(backbone, pixel) != self._own:
            return False
        for d, was in self._modules:
            if d != was:
                return False
        for d, k, p in self._owners:
            if d.get(k) is not p:
                return False
        if [p._version for p in self._params] != self._versions or [p.data_ptr() for p in self._params] != self._ptrs:
            return False
        for own, name, value in self._attrs:
            if own.get(name) != value:
                return False
        return True

    # ---------------------------------------------------------------- descriptors
    def _describe(self, backbone, pixel) -> None:
        attrs = []
        weights = _Weights(self.device)
        keep = weights.keep

        def kernels_of(blocks):
            attrs.extend((vars(b), "kernel", b.kernel) for b in blocks)
            flat = [v for b in blocks for v in b.kernel]
            return (ctypes.c_int32 * max(len(flat), 1))(*flat)

        def same(blocks, name, default):
            attrs.extend((vars(b), name, getattr(b, name)) for b in blocks)
            values = {getattr(b, name) for b in blocks} or {default}
            return values.pop() if len(values) == 1 else None

        def usable(blocks):
            for b in blocks:
                attrs.append((vars(b.mlp.layers[1]), "approximate", "tanh"))
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
        d.w_embed, d.b_embed, d.k_embed = weights.embed(bb.patch_embed, bb.embed_dim, "patch embedding")
        structs = (_lib.BlockWeights * max(len(blocks), 1))()
        if ok:
            for i, (s, b) in enumerate(zip(structs, blocks)):
                weights.block(b.device_weights(), d.dim, d.hidden, f"block {i}:", s)
        kern = kernels_of(blocks)
        d.h_blocks = ctypes.cast(structs, ctypes.POINTER(_lib.BlockWeights))
        d.h_kernels = ctypes.cast(kern, ctypes.POINTER(ctypes.c_int32))
        keep += [structs, kern]
        if bb.final_layer is not None:
            d.w_head, d.b_head, d.n_head = weights.head(bb.final_layer, bb.embed_dim, "final layer")
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
            px.w_embed, px.b_embed, px.k_embed = weights.embed(pixel.pixel_patch_embed, px.dim,
                                                               "pixel patch embedding")
            if ok:
                px.cond_ks = self._pixel_blocks(pblocks, bb, px, weights)
                ok = px.cond_ks is not None
            kern = kernels_of(pblocks)
            px.h_kernels = ctypes.cast(kern, ctypes.POINTER(ctypes.c_int32))
            keep.append(kern)
            px.w_head, px.b_head, px.n_head = weights.head(pixel.pixel_final_layer, px.dim,
                                                           "pixel final layer")
        if ok:
            self.desc, self.pixel, self.keep = d, px, keep
        self._watch(backbone if pixel is None else pixel, attrs)

    @staticmethod
    def _pixel_blocks(pblocks, bb, px, weights):
        """Fills px.h_blocks; returns the depthwise kernel size (0: no block is modulated, None:
        the blocks disagree)."""
        lib = _lib.load()
        structs = (_lib.PixelBlockWeights * max(len(pblocks), 1))()
        sizes = set()
        keep, Cb = weights.keep, bb.embed_dim
        for i, (s, b) in enumerate(zip(structs, pblocks)):
            w, name = b.device_weights(), f"pixel block {i}:"
            weights.block(w, px.dim, px.hidden, name, s.block)
            if "w_mod" not in w:
                continue
            ks = w["w_dw"].shape[-1]
            sizes.add(ks)
            s.w_dw = weights.ptr(w["w_dw"], (Cb, ks, ks), f"{name} depthwise weight")
            s.b_dw = weights.ptr(w["b_dw"], (Cb,), f"{name} depthwise bias")
            s.w_mod = weights.ptr(w["w_mod"], (6 * px.dim, Cb), f"{name} modulation weight")
            s.b_mod = weights.ptr(w["b_mod"], (6 * px.dim,), f"{name} modulation bias")
            n = int(lib.strata_adaln_cond_table_floats(Cb, bb.patch_size[1], ks))
            if n:
                table = torch.empty(n, dtype=torch.float32, device=w["w_dw"].device)
                with torch.cuda.device(table.device):
                    _lib.check(lib.strata_adaln_cond_table_f32(
                        w["w_dw"].data_ptr(), Cb, bb.patch_size[1], ks, table.data_ptr(),
                        torch.cuda.current_stream().cuda_stream), "strata_adaln_cond_table_f32")
                keep.append(table)
                _lib.keep(table.device, lambda: None)     # (kept by this description, which waits for it)
                s.cond_table = table.data_ptr()
        px.h_blocks = ctypes.cast(structs, ctypes.POINTER(_lib.PixelBlockWeights))
        keep.append(structs)
        return None if len(sizes) > 1 else (sizes.pop() if sizes else 0)


class NetworkHandle:
    """The description of one `StrataTransformer3D` (and, for the two-stage model, the `Strata` module
    around it) that the last pass found. Belongs to the module that owns it; a copy of the module
    starts with an empty one."""

    def __init__(self):
        self._state = None      # read and replaced whole

    def __deepcopy__(self, memo):
        return NetworkHandle()

    def __reduce__(self):
        return (NetworkHandle, ())

    # ---------------------------------------------------------------- one pass
    def forward(self, backbone, pixel, x, lat, lon, wind, concat_lat):
        """x [B, C, D, H, W], lat / lon [B, H, W], CUDA fp32 on one device -> fields, or None when
        the model has a part that only the step-by-step path runs."""
        x, lat, lon = ops.network_inputs(x, lat, lon, x.shape[1] + (2 if concat_lat else 0), backbone)
        s = self._state
        if s is None or not s.current(backbone, pixel, x.device):
            with _lib.settled_together(x.device) as new:
                s = Described(backbone, pixel, x.device)
            if new.kept:
                self._state = s
        if s.desc is None or (backbone.rope_mode == "stereographic" and s.desc.patch_h != s.desc.patch_w):
            return None
        # the call's own copy takes the values that differ from call to call
        d = _lib.BackboneDesc.from_buffer_copy(s.desc)
        px = None if s.pixel is None else _lib.PixelDesc.from_buffer_copy(s.pixel)
        B, C, D, H, W = x.shape
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
