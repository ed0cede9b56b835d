"""ctypes binding of libstrata_b200.so (the C ABI declared in include/strata_b200.h).

There is no CPU or eager fallback: if the library is missing or an entry point reports an
error, the call raises.
"""
from __future__ import annotations

import ctypes
import threading
from ctypes import c_char_p, c_double, c_float, c_int, c_int32, c_int64, c_void_p, POINTER, Structure
from pathlib import Path

_LIB_PATH = Path(__file__).resolve().parent / "libstrata_b200.so"
_lib = None


class StrataLibraryError(RuntimeError):
    pass


class BlockWeights(Structure):
    """struct strata_block_weights (device pointers)."""
    _fields_ = [(n, c_void_p) for n in ("w_qkv", "b_qkv", "w_proj", "b_proj", "w_gate", "b_gate",
                                        "w_fc1", "b_fc1", "w_fc2", "b_fc2")]


class BackboneDesc(Structure):
    """struct strata_backbone_desc."""
    _fields_ = ([(n, c_int32) for n in ("in_channels", "out_channels", "patch_v", "patch_h", "patch_w",
                                        "dim", "heads", "hidden", "n_blocks", "qk_norm", "concat_lat",
                                        "u_idx", "v_idx", "rope_mode")]
                + [("rope_length_scale", c_double), ("rope_base", c_double), ("w_embed", c_void_p),
                   ("b_embed", c_void_p), ("k_embed", c_int64), ("h_blocks", POINTER(BlockWeights)),
                   ("h_kernels", POINTER(c_int32)), ("w_head", c_void_p), ("b_head", c_void_p),
                   ("n_head", c_int32)])


class PixelBlockWeights(Structure):
    """struct strata_pixel_block_weights."""
    _fields_ = [("block", BlockWeights)] + [(n, c_void_p) for n in ("cond_table", "w_dw", "b_dw", "w_mod",
                                                                   "b_mod")]


class PixelDesc(Structure):
    """struct strata_pixel_desc."""
    _fields_ = ([(n, c_int32) for n in ("dim", "heads", "hidden", "n_blocks", "qk_norm", "rope_mode",
                                        "cond_ks")]
                + [("rope_length_scale", c_double), ("rope_base", c_double), ("w_embed", c_void_p),
                   ("b_embed", c_void_p), ("k_embed", c_int64), ("h_blocks", POINTER(PixelBlockWeights)),
                   ("h_kernels", POINTER(c_int32)), ("w_head", c_void_p), ("b_head", c_void_p),
                   ("n_head", c_int32)])


_SIGNATURES = {
    "strata_abi_version": (c_int, []),
    "strata_error_string": (c_char_p, [c_int]),
    "strata_device_status": (c_int, [POINTER(c_int), c_int]),
    "strata_layernorm_bf16": (c_int, [c_void_p, c_int64, c_void_p, c_int64, c_int, c_int, c_float,
                                      c_void_p]),
    "strata_linear_bf16": (c_int, [c_void_p, c_int64, c_void_p, c_int64, c_void_p, c_void_p,
                                   c_int64, c_int, c_int, c_int, c_int, c_void_p, c_int64,
                                   c_void_p]),
    "strata_mlp_fused": (c_int, [c_int, c_int, c_int]),
    "strata_mlp_bf16": (c_int, [c_void_p, c_int64, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int64,
                                c_void_p, c_int64, c_void_p, c_int64, c_int, c_int, c_int, c_void_p]),
    "strata_qkv_rope_bf16": (c_int, [c_void_p, c_int64, c_void_p, c_int64, c_void_p, c_void_p,
                                     c_int64, c_int, c_int, c_int, c_void_p, c_int, c_int,
                                     c_int, c_float, c_void_p]),
    "strata_na3d_fwd_bf16": (c_int, [c_void_p, c_int64, c_void_p, c_int64, c_void_p, c_int64,
                                     c_void_p, c_int64, c_int, c_int, c_int, c_int, c_int, c_int,
                                     c_int, c_int, c_int, c_float, c_void_p]),
    "strata_block_workspace_bytes": (c_int64, [c_int64, c_int, c_int]),
    "strata_block_forward_bf16": (c_int, [c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int,
                                          c_int, c_int, c_int, c_int, c_int, POINTER(BlockWeights),
                                          c_void_p, c_int, c_float, c_float, c_void_p,
                                          c_int64, c_void_p]),
    "strata_halo_gather_tokens_bf16": (c_int, [c_void_p, POINTER(c_void_p), c_int, c_void_p,
                                               c_void_p, c_int, c_int, c_int, c_int, c_int, c_int,
                                               c_void_p]),
    "strata_halo_gather_fields_f32": (c_int, [c_void_p, POINTER(c_void_p), c_int, c_void_p, c_void_p,
                                              c_int, c_int, c_int, c_int64, c_void_p]),
    "strata_halo_gather_kv_bf16": (c_int, [c_void_p, POINTER(c_void_p), c_int, c_void_p, c_void_p,
                                           c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int,
                                           c_int, c_int64, c_void_p]),
    "strata_qkv_rope_padded_bf16": (c_int, [c_void_p, c_int64, c_void_p, c_int64, c_void_p, c_void_p,
                                            c_int64, c_int, c_int, c_int, c_void_p, c_int, c_int,
                                            c_int, c_float, c_int, c_int, c_int, c_void_p]),
    "strata_na3d_fwd_region_bf16": (c_int, [c_void_p, c_int64, c_void_p, c_int64, c_void_p, c_int64,
                                            c_void_p, c_int64, c_int, c_int, c_int, c_int, c_int,
                                            c_int, c_int, c_int, c_int, c_float, c_int, c_int,
                                            c_int, c_int, c_int, c_int, c_int, c_int, c_void_p]),
    "strata_halo_gather_knn_fields_f32": (c_int, [c_void_p, POINTER(c_void_p), c_int, c_void_p, c_void_p,
                                                  c_int, c_int, c_int, c_int, c_int64, c_void_p]),
    "strata_halo_adjoint_fields_f32": (c_int, [c_void_p, POINTER(c_void_p), c_int, c_void_p, c_void_p,
                                               c_void_p, c_void_p, c_void_p, c_int, c_int, c_int,
                                               c_int64, c_void_p]),
    "strata_preprocess_patches_bf16": (c_int, [c_void_p, c_int, c_int, c_int, c_int, c_int, c_void_p,
                                               c_void_p, c_void_p, c_void_p, c_int, c_int, c_int,
                                               c_int, c_int, c_int, c_void_p, c_int64, c_void_p]),
    "strata_postprocess_fields_f32": (c_int, [c_void_p, c_int64, c_int, c_int, c_int, c_int, c_int,
                                              c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int,
                                              c_int, c_int, c_int, c_void_p, c_void_p]),
    "strata_adaln_rows_bf16": (c_int, [c_void_p, c_int64, c_void_p, c_int64, c_void_p, c_int64,
                                       c_void_p, c_int64, c_void_p, c_void_p, c_int64, c_void_p,
                                       c_int64, c_int, c_int, c_float, c_void_p]),
    "strata_qk_norm_rows_bf16": (c_int, [c_void_p, c_int64, c_int64, c_int, c_float, c_void_p]),
    "strata_adaln_cond_bf16": (c_int, [c_void_p, c_int, c_int, c_int, c_int, c_int, c_int,
                                       c_void_p, c_void_p, c_int, c_int64, c_int64, c_void_p,
                                       c_void_p, c_void_p]),
    "strata_adaln_cond_table_floats": (c_int64, [c_int, c_int, c_int]),
    "strata_adaln_cond_table_f32": (c_int, [c_void_p, c_int, c_int, c_int, c_void_p, c_void_p]),
    "strata_tile_tables_workspace_bytes": (c_int64, [c_int, c_int, c_int]),
    "strata_tile_tables": (c_int, [c_void_p, c_void_p, c_int, c_int, c_int, c_void_p, c_void_p, c_int,
                                   c_int, c_double, c_double, c_int, c_void_p, c_void_p, c_int64,
                                   c_void_p]),
    "strata_network_workspace_bytes": (c_int64, [POINTER(BackboneDesc), POINTER(PixelDesc), c_int, c_int,
                                                 c_int, c_int]),
    "strata_network_forward_f32": (c_int, [POINTER(BackboneDesc), POINTER(PixelDesc), c_void_p, c_void_p,
                                           c_void_p, c_int, c_int, c_int, c_int, c_void_p, c_void_p,
                                           c_int64, c_void_p]),
    "strata_dealias_patches_bf16": (c_int, [c_void_p, c_int64, c_int, c_int, c_int, c_int, c_int,
                                            c_int, c_int, c_int, c_void_p, c_int, c_void_p, c_int64,
                                            c_void_p]),
    "strata_halo_barrier": (c_int, [POINTER(c_void_p), c_int, c_int, c_int, c_int, c_void_p]),
    "strata_ipc_alloc": (c_int, [c_int64, POINTER(c_void_p), c_void_p]),
    "strata_ipc_open": (c_int, [c_void_p, POINTER(c_void_p)]),
    "strata_ipc_close": (c_int, [c_void_p]),
    "strata_ipc_free": (c_int, [c_void_p]),
    "strata_block_forward_static_scratch_bf16": (c_int, [
        c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_int,
        POINTER(BlockWeights), c_void_p, c_int, c_float, c_float, c_void_p]),
}


def lib_path() -> Path:
    return _LIB_PATH


def load() -> ctypes.CDLL:
    """Load the shared library (once) and attach argument types."""
    global _lib
    if _lib is not None:
        return _lib
    if not _LIB_PATH.exists():
        raise StrataLibraryError(
            f"{_LIB_PATH} is missing: build it with `python -m strata_b200.build` "
            "(there is no fallback path)")
    lib = ctypes.CDLL(str(_LIB_PATH))
    for name, (res, args) in _SIGNATURES.items():
        fn = getattr(lib, name)
        fn.restype = res
        fn.argtypes = args
    _lib = lib
    return lib


class _Nothing:
    def __enter__(self):
        return None

    def __exit__(self, *exc):
        return False


_NOTHING = _Nothing()


def on_device(t):
    """Context in which t's device is current; free when it already is (torch's own guard costs
    3 us of a call that takes 10)."""
    import torch
    return _NOTHING if t.device.index == torch.cuda.current_device() else torch.cuda.device(t.device)


def _stream_lookup():
    """Device index -> raw handle of its current stream. torch's raw lookup is private; without it the
    stream object is asked (4 us more a call)."""
    import torch
    raw = getattr(torch._C, "_cuda_getCurrentRawStream", None)
    return raw if raw is not None else lambda index: torch.cuda.current_stream(index).cuda_stream


_current_stream = None


def stream_of(t) -> int:
    """Raw handle of the current stream of t's device."""
    global _current_stream
    if _current_stream is None:
        _current_stream = _stream_lookup()
    return _current_stream(t.device.index)


def settle(device) -> bool:
    """Waits for the device: what was filled on it before may then be read by any stream and thread, and
    nothing in flight reads what it replaces. False while a graph is being captured: nothing has run
    then."""
    import torch
    if device.type != "cuda":
        return True
    with torch.cuda.device(device):
        if torch.cuda.is_current_stream_capturing():
            return False
        torch.cuda.synchronize()
    return True


_filling = threading.local()


def keep(device, store) -> None:
    """Called with tensors that were just filled on the current stream and that a module will keep for
    later passes (weights cast for the kernels, tables): store() puts them where these look, once they are
    settled; under capture it is not called, and the tensors serve this pass only."""
    together = getattr(_filling, "stores", None)
    if together is not None:
        together.append(store)
    elif settle(device):
        store()


class settled_together:
    """Context in which this thread's keep() calls wait for the device once, at its end. `kept` then
    says whether what was filled inside may be kept."""

    def __init__(self, device):
        self.device = device
        self.kept = False

    def __enter__(self):
        self._outer = getattr(_filling, "stores", None)
        _filling.stores = self._stores = []
        return self

    def __exit__(self, kind, *exc):
        _filling.stores = self._outer
        if kind is None:
            self.kept = not self._stores or settle(self.device)
            if self.kept:
                for store in self._stores:
                    store()
        return False


def exported_names() -> list[str]:
    return sorted(_SIGNATURES)


def check(code: int, what: str) -> None:
    """Raise for a non-zero return code of an entry point."""
    if code == 0:
        return
    msg = load().strata_error_string(code).decode()
    if code in (-1,):
        raise ValueError(f"{what}: {msg} (code {code})")
    raise StrataLibraryError(f"{what}: {msg} (code {code})")


def device_status(reset: bool = True) -> int:
    """Synchronise and return the device status word (0 = ok)."""
    st = c_int(0)
    check(load().strata_device_status(ctypes.byref(st), 1 if reset else 0), "strata_device_status")
    return st.value
