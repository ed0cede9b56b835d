"""The work that is measured: whole calls through the public entry points, from the smallest
ones (where launches and host time count) to the largest.

A case is a dict of plain values with a "kind":

  model      StrataBackboneModel(x, index): fields in, fields out - what the inference and rollout
             tooling calls once per model step for a batch of tiles
  two_stage  StrataModel(x, index): backbone plus the AdaLN pixel stage at full resolution
  sphere     TiledSphereStepper(x): one step over a whole tiled cubed sphere (field halo, the
             backbone on the padded tiles, crop)
  block      ops.block_forward: one transformer block on tokens the caller holds
  tiled      TiledBlockRunner.block_forward: one block over all tiles of a sphere with the K/V
             halo exchanged inside the block
  attention  ops.na3d: neighbourhood attention alone
  halo       the field-space halo exchange: pad the tiles of a sphere (copied or interpolated
             halo), and un-pad by windowed overlap-add

Everything is inference (the library has no backward pass); tokens are bf16, fields fp32.
Weights and inputs are drawn from the seed on the GPU; what depends on the geometry alone (halo
plans, RoPE delta tables, peer buffers) is built once per geometry and kept, as a program
that steps one grid keeps it.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from strata_b200 import ops, rope
from strata_b200.halo import (DistributedTileCopyHaloPadding, DistributedTileKNNHaloPadding,
                              NormalizedHaloAdjoint, kbd_window)
from strata_b200.halo_block import TiledBlockRunner
from strata_b200.rollout import (TiledSphereStepper, equiangular_cubed_sphere_latlon,
                                 padded_face_latlon)
from strata_b200.topology import TileTopology
from strata_b200.wrappers import StrataBackboneModel, StrataModel


# ------------------------------------------------------------------------------- the cases
def _model(name, tiles, depth, height, width, patch, chans, dim, layers, kernel, *, gated=False,
           qk_norm=False, wind=False, rope_mode="stereographic"):
    return dict(name=name, kind="model", tiles=tiles, depth=depth, height=height, width=width,
                patch=patch, chans=chans, dim=dim, layers=layers, kd=kernel[0], kh=kernel[1],
                kw=kernel[2], gated=gated, qk_norm=qk_norm, wind=wind, rope=rope_mode)


def _two_stage(name, tiles, depth, height, width, chans, dim, layers, pixel_layers, pixel_kernel, *,
               wind=False, pixel_rope="none"):
    return dict(name=name, kind="two_stage", tiles=tiles, depth=depth, height=height, width=width,
                patch=4, chans=chans, dim=dim, layers=layers, pixel_layers=pixel_layers,
                pkd=pixel_kernel[0], pkh=pixel_kernel[1], pkw=pixel_kernel[2], wind=wind,
                pixel_rope=pixel_rope)


def _block(name, tiles, depth, height, width, dim, kernel, *, gated=False, qk_norm=False, with_rope=True):
    return dict(name=name, kind="block", tiles=tiles, depth=depth, height=height, width=width, dim=dim,
                kd=kernel[0], kh=kernel[1], kw=kernel[2], gated=gated, qk_norm=qk_norm, rope=with_rope)


def _attention(name, batch, depth, height, width, heads, kernel, packed):
    return dict(name=name, kind="attention", batch=batch, depth=depth, height=height, width=width,
                heads=heads, kd=kernel[0], kh=kernel[1], kw=kernel[2], packed=packed)


def _tiled(name, tile, per_dim, halo, depth, dim, kernel, *, gated=False, qk_norm=False):
    return dict(name=name, kind="tiled", tile=tile, per_dim=per_dim, halo=halo, depth=depth, dim=dim,
                kd=kernel[0], kh=kernel[1], kw=kernel[2], gated=gated, qk_norm=qk_norm)


def _halo(name, tile, per_dim, halo, chans, levels, source, unpad):
    return dict(name=name, kind="halo", tile=tile, per_dim=per_dim, halo=halo, chans=chans,
                levels=levels, source=source, unpad=unpad)


def _sphere(name, tile, per_dim, halo, depth, chans, dim, layers, kernel):
    return dict(name=name, kind="sphere", tile=tile, per_dim=per_dim, halo=halo, depth=depth,
                chans=chans, dim=dim, layers=layers, kd=kernel[0], kh=kernel[1], kw=kernel[2])


def listed():
    return [
        # one small tile through the single-stage model: the size the test-suite and a first
        # try-out use; latency of a step
        _model("model_small", 1, 4, 32, 32, 4, 5, 128, 2, (3, 3, 3)),
        # a batch of three tiles whose token planes fill no query or GEMM tile evenly, with
        # wind rotation, gate and q/k norm on
        _model("model_ragged", 3, 13, 88, 120, 4, 13, 384, 4, (3, 7, 7), gated=True, qk_norm=True,
               wind=True),
        # one production tile (24 levels of 256 x 256 columns, patch 4) through the default
        # backbone: 768 wide, 12 blocks
        _model("model_tile", 1, 24, 256, 256, 4, 13, 768, 12, (3, 3, 3)),
        # a small two-stage model on one tile: many short launches
        _two_stage("two_stage_small", 1, 4, 64, 64, 5, 128, 2, 2, (3, 5, 5)),
        # the production two-stage model on one production tile: the largest single call
        _two_stage("two_stage_tile", 1, 24, 256, 256, 13, 1024, 24, 4, (9, 9, 9), wind=True),
        # one block on one small tile (the reference's single-block CPU configuration in bf16)
        _block("block_small", 1, 8, 32, 32, 128, (3, 7, 7)),
        # the headline benchmark: four tiles of 16 x 64 x 64 tokens, 512 wide
        _block("block_tiles", 4, 16, 64, 64, 512, (3, 9, 9)),
        # wide window, gate and q/k norm on a grid that divides by nothing
        _block("block_ragged", 2, 11, 50, 71, 768, (5, 13, 13), gated=True, qk_norm=True),
        # a quarter of the attention sweep's batch at its middle window
        _attention("attention_sweep", 2, 32, 96, 96, 16, (3, 13, 13), False),
        # one block of the tiled encoder over a whole sphere with the K/V halo inside
        _tiled("tiled_block", 64, 2, 8, 16, 768, (5, 13, 13)),
        # field halo of one model step and the overlap-add back
        _halo("halo_fields", 64, 2, 8, 64, 8, "copy", True),
        # a whole sphere step on small tiles: halo, model on the padded tiles, crop
        _sphere("sphere_step", 32, 2, 8, 8, 8, 256, 2, (3, 5, 5)),
    ]


_KERNELS = ((3, 3, 3), (3, 5, 5), (3, 7, 7), (3, 9, 9), (5, 13, 13), (7, 7, 7), (5, 15, 15))


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _fitting(rng, depth, h, w):
    return rng.choice([k for k in _KERNELS if k[0] <= depth and k[1] <= h and k[2] <= w])


def _draw_once(rng):
    kind = rng.choice(["model", "model", "two_stage", "block", "block", "attention", "tiled", "halo",
                       "sphere"])
    flag = lambda: rng.random() < 0.5
    if kind == "model":
        depth, h, w = _log_int(rng, 3, 26), _log_int(rng, 8, 72), _log_int(rng, 8, 72)
        patch = rng.choice([1, 2, 4, 4])
        c = _model("", rng.randint(1, 4), depth, h * patch, w * patch, patch, rng.randint(3, 16),
                   64 * _log_int(rng, 2, 16), _log_int(rng, 2, 12), _fitting(rng, depth, h, w),
                   gated=flag(), qk_norm=flag(), wind=flag(),
                   rope_mode=rng.choice(["stereographic", "stereographic", "axial"]))
    elif kind == "two_stage":
        depth, h, w = _log_int(rng, 3, 24), _log_int(rng, 8, 64), _log_int(rng, 8, 64)
        c = _two_stage("", rng.randint(1, 2), depth, 4 * h, 4 * w, rng.randint(3, 16),
                       64 * _log_int(rng, 2, 16), _log_int(rng, 2, 24), rng.randint(1, 4),
                       rng.choice([k for k in ((3, 3, 3), (3, 5, 5), (7, 7, 7), (9, 9, 9)) if k[0] <= depth]),
                       wind=flag(), pixel_rope=rng.choice(["none", "none", "stereographic"]))
    elif kind == "block":
        depth, h, w = _log_int(rng, 3, 32), _log_int(rng, 16, 128), _log_int(rng, 16, 128)
        c = _block("", _log_int(rng, 1, 12), depth, h, w, 64 * _log_int(rng, 2, 16),
                   _fitting(rng, depth, h, w), gated=flag(), qk_norm=flag(), with_rope=rng.random() < 0.8)
    elif kind == "attention":
        depth, h, w = _log_int(rng, 3, 32), _log_int(rng, 16, 100), _log_int(rng, 16, 100)
        c = _attention("", _log_int(rng, 1, 8), depth, h, w, _log_int(rng, 1, 16),
                       _fitting(rng, depth, h, w), flag())
    elif kind == "tiled":
        k = rng.choice(_KERNELS[:5])
        depth = max(k[0], _log_int(rng, 4, 20))
        c = _tiled("", rng.choice([32, 64]), rng.choice([1, 2]), rng.randint(k[1] // 2, 14), depth,
                   64 * _log_int(rng, 2, 16), k, gated=flag(), qk_norm=flag())
    elif kind == "halo":
        tile = _log_int(rng, 12, 96)
        c = _halo("", tile, rng.choice([1, 2, 3]), rng.randint(1, min(16, tile // 2)), _log_int(rng, 1, 96),
                  _log_int(rng, 1, 24), rng.choice(["copy", "copy", "knn"]), flag())
    else:
        depth = _log_int(rng, 3, 16)
        tile, halo = rng.randint(8, 64), rng.randint(2, 8)
        c = _sphere("", tile, rng.choice([1, 2]), halo, depth, rng.randint(3, 16), 64 * _log_int(rng, 2, 12),
                    rng.randint(1, 4), rng.choice(_KERNELS[:3]))
    del c["name"]
    return c


def _cost(case):
    w = work(case)
    return w["flops"] / 5e14 + w["bytes"] / 2e12


def draw(rng):
    """One more case of the same ranges, no dearer than the largest listed one."""
    most = _cost(next(c for c in listed() if c["name"] == "two_stage_tile"))
    while True:
        c = _draw_once(rng)
        if _cost(c) <= most and _device_bytes(c) <= 24e9:
            return c


# ------------------------------------------------------------------------------- what a case needs
def _tokens(c):
    """(tiles, token grid) of the transformer tokens of a case."""
    if c["kind"] in ("model", "two_stage"):
        return c["tiles"], (c["depth"], c["height"] // c["patch"], c["width"] // c["patch"])
    if c["kind"] == "sphere":
        p = c["tile"] + 2 * c["halo"]
        return 6 * c["per_dim"] ** 2, (c["depth"], p, p)
    if c["kind"] == "tiled":
        return 6 * c["per_dim"] ** 2, (c["depth"], c["tile"], c["tile"])
    return c["tiles"], (c["depth"], c["height"], c["width"])


def _block_flops(n_tokens, dim, kernel, gated):
    keys = kernel[0] * kernel[1] * kernel[2]
    return n_tokens * ((26 if gated else 24) * dim * dim + 4 * keys * dim)


def _block_params(dim, gated):
    return (13 if gated else 12) * dim * dim


def work(case):
    """Bytes: every input, weight (bf16) and output once. Operations: the multiply-adds of the
    projections, of the keys inside each window, and of the embeddings."""
    c = case
    kind = c["kind"]
    if kind == "halo":
        tiles = 6 * c["per_dim"] ** 2
        t2, p2 = c["tile"] ** 2, (c["tile"] + 2 * c["halo"]) ** 2
        k = 4 if c["source"] == "knn" else 1
        cells = tiles * c["chans"] * c["levels"]
        # un-padding reads the padded tiles (an output of the same pass) and writes interiors
        return {"bytes": 4 * cells * (t2 + p2) * (2 if c["unpad"] else 1) + 8 * tiles * p2 * k,
                "flops": cells * p2 * (2 * k + (2 * k if c["unpad"] else 0))}
    if kind == "attention":
        n = c["batch"] * c["depth"] * c["height"] * c["width"] * c["heads"] * 64
        return {"bytes": 8 * n, "flops": 4 * c["kd"] * c["kh"] * c["kw"] * n}
    tiles, grid = _tokens(c)
    n = tiles * grid[0] * grid[1] * grid[2]
    dim = c["dim"]
    if kind in ("block", "tiled"):
        return {"bytes": 4 * n * dim + 2 * _block_params(dim, c["gated"]) + 4 * tiles * grid[1] * grid[2] * 32,
                "flops": _block_flops(n, dim, (c["kd"], c["kh"], c["kw"]), c["gated"])}
    # fields in, fields out
    if kind == "sphere":
        n_in = n_out = tiles * c["depth"] * c["tile"] ** 2
        cells_px, patch, gated, kernel = n, 1, False, (c["kd"], c["kh"], c["kw"])
    else:
        n_in = n_out = cells_px = tiles * c["depth"] * c["height"] * c["width"]
        patch = c["patch"]
        gated = True if kind == "two_stage" else c["gated"]
        kernel = (3, 3, 3) if kind == "two_stage" else (c["kd"], c["kh"], c["kw"])
    layers = c["layers"]
    embed = 2 * cells_px * (c["chans"] + 2) * dim            # patch embedding
    head = 2 * cells_px * c["chans"] * dim                   # final layer
    flops = embed + layers * _block_flops(n, dim, kernel, gated)
    params = layers * _block_params(dim, gated) + (2 * c["chans"] + 2) * patch * patch * dim
    if kind == "two_stage":
        pixels, pd = cells_px, 128
        keys = c["pkd"] * c["pkh"] * c["pkw"]
        # modulation: 5 x 5 depthwise taps on the upsampled tokens and the 6-fold projection
        flops += c["pixel_layers"] * pixels * (24 * pd * pd + 4 * keys * pd + 12 * pd * dim + 50 * dim)
        flops += 2 * pixels * pd * (2 * c["chans"] + 2)
        params += c["pixel_layers"] * (12 * pd * pd + 6 * pd * dim)
    else:
        flops += head
    return {"bytes": 4 * c["chans"] * (n_in + n_out) + 2 * params, "flops": flops}


def _device_bytes(c):
    """Rough device memory of one state and its pass."""
    if c["kind"] in ("halo", "attention"):
        return 3 * work(c)["bytes"]
    tiles, grid = _tokens(c)
    n = tiles * grid[0] * grid[1] * grid[2]
    b = n * c["dim"] * 26
    if c["kind"] == "tiled":
        b += n * ((c["tile"] + 2 * c["halo"]) / c["tile"]) ** 2 * c["dim"] * 12
    if c["kind"] == "two_stage":
        b += n * c["patch"] ** 2 * 128 * 32
    return b + 6 * c.get("layers", 1) * _block_params(c["dim"], True)


def tolerance(case):
    kind = case["kind"]
    if kind == "halo":
        # copies and the two-cell mean have one answer; weighted sums are fp32 sums of a few terms
        return "exact" if case["source"] == "copy" and not case["unpad"] else {"rel": 1e-6, "max": 1e-5}
    if kind in ("attention", "block", "tiled"):
        return {"rel": 6e-3, "max": 0.1}      # bf16 results, bf16 intermediates
    # the residual stream is rounded to bf16 twice per block
    return {"rel": 2e-2 if case["layers"] > 8 else 1e-2, "max": 0.15}


# ------------------------------------------------------------------------------- preparation
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, dtype=torch.float32, std=1.0):
    return torch.randn(*shape, generator=g, device="cuda").mul_(std).to(dtype)


def _latlon(g, tiles, height, width):
    """Smooth tiles somewhere on the sphere, columns about as dense as on the 2048-cell faces."""
    c = torch.rand(2, tiles, 1, 1, generator=g, device="cuda")
    step = math.pi / 2 / 2048
    i = torch.arange(height, device="cuda").view(1, -1, 1) * step
    j = torch.arange(width, device="cuda").view(1, 1, -1) * step
    lat = (-1.0 + 2.0 * c[0]) * 1.1 + i + 0.1 * j
    lon = 2 * math.pi * c[1] + j - 0.1 * i
    return (lat.expand(tiles, height, width).contiguous(), lon.expand(tiles, height, width).contiguous())


def _fill(module, g):
    """Weights of a trained model's size: fan-in scaled matrices, small biases (the AdaLN
    projections too, which start from zero in training)."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            std = 0.05 if p.dim() == 1 else p[0].numel() ** -0.5
            if "adaln" in name and p.dim() == 2:
                std *= 0.5
            p.copy_(torch.randn(p.shape, generator=g, device="cuda").mul_(std))
    return module


def _block_weights(g, dim, gated):
    shapes = {"qkv": (3 * dim, dim), "proj": (dim, dim), "fc1": (4 * dim, dim), "fc2": (dim, 4 * dim)}
    if gated:
        shapes["gate"] = (dim, dim)
    w = {}
    for name, (n, k) in shapes.items():
        w[f"w_{name}"] = _randn(g, n, k, dtype=torch.bfloat16, std=k ** -0.5)
        w[f"b_{name}"] = _randn(g, n, std=0.05)
    return w


@functools.lru_cache(maxsize=4)
def _topology(tile, per_dim, halo):
    return TileTopology(1, 0, tile * per_dim, tile, halo)


@functools.lru_cache(maxsize=2)
def _halo_modules(tile, per_dim, halo, source, unpad):
    topo = _topology(tile, per_dim, halo)
    if source == "knn":
        lat, lon = padded_face_latlon(topo.face_size, halo)
        pad = DistributedTileKNNHaloPadding.from_padded_face_grid(
            topology=topo, lon=torch.from_numpy(lon), lat=torch.from_numpy(lat), pad_width_data=halo,
            device="cuda")
    else:
        pad = DistributedTileCopyHaloPadding(topology=topo, device="cuda")
    back = None
    if unpad:
        p = topo.padded_tile_size
        back = NormalizedHaloAdjoint(pad, window=kbd_window(p) if p % 2 == 0 else None)
    return pad, back


@functools.lru_cache(maxsize=1)
def _runner(tile, per_dim, halo, depth, dim, kernel):
    topo = _topology(tile, per_dim, halo)
    face = topo.face_size
    lat, lon = equiangular_cubed_sphere_latlon(face)
    cut = lambda a: np.stack([a[f, i * tile:(i + 1) * tile, j * tile:(j + 1) * tile]
                              for f, i, j in topo.global_tiles])
    return TiledBlockRunner(topo, depth=depth, dim=dim, num_heads=dim // 64, kernel=kernel,
                            lat_deg=cut(lat), lon_deg=cut(lon),
                            rope_length_scale=float(np.radians(90.0 / face)))


def _model_kwargs(c):
    return dict(depth=c["depth"], height=c["height"], width=c["width"], n_layers=c["layers"],
                patch_size_vert=1, patch_size_horiz=c["patch"], in_chans=c["chans"],
                base_out_chans=c["chans"], embed_dim=c["dim"], num_heads=c["dim"] // 64,
                index_is_latlon=True, do_bf16_mixed=True, do_rotate_wind=c["wind"],
                wind_channel_indices=(0, 1) if c["wind"] else None)


def prepare(case, seed):
    c = case
    kind = c["kind"]
    g = _gen(seed)
    if kind == "halo":
        topo = _topology(c["tile"], c["per_dim"], c["halo"])
        pad, back = _halo_modules(c["tile"], c["per_dim"], c["halo"], c["source"], c["unpad"])
        x = _randn(g, c["chans"], c["levels"], topo.tiles_per_rank, c["tile"], c["tile"])
        return dict(kind=kind, x=x, pad=pad, back=back)
    if kind == "attention":
        shape = (c["batch"], c["depth"], c["height"], c["width"])
        if c["packed"]:       # slices of one packed projection, as the block holds them
            qkv = _randn(g, *shape, 3, c["heads"], 64, dtype=torch.bfloat16)
            q, k, v = (qkv[..., i, :, :] for i in range(3))
        else:
            q, k, v = (_randn(g, *shape, c["heads"], 64, dtype=torch.bfloat16) for _ in range(3))
        return dict(kind=kind, q=q, k=k, v=v, kernel=(c["kd"], c["kh"], c["kw"]))
    if kind == "block":
        tiles, grid = _tokens(c)
        n, dim = grid[0] * grid[1] * grid[2], c["dim"]
        w = _block_weights(g, dim, c["gated"])
        cs = None
        if c["rope"]:
            lat, lon = _latlon(g, tiles, grid[1], grid[2])
            cs = rope.pack_rope_tables(*rope.stereographic_rope_tables(
                torch.stack([lat, lon], 1), 64, 1, rope.default_rope_length_scale(1)))
        ws = torch.empty(ops.block_workspace_bytes(tiles * n, dim, 4 * dim), dtype=torch.uint8,
                         device="cuda")
        return dict(kind=kind, x=_randn(g, tiles, n, dim, dtype=torch.bfloat16), weights=w, cs=cs,
                    workspace=ws, grid=grid, heads=dim // 64, kernel=(c["kd"], c["kh"], c["kw"]),
                    qk_norm=c["qk_norm"])
    if kind == "tiled":
        tiles, grid = _tokens(c)
        run_ = _runner(c["tile"], c["per_dim"], c["halo"], c["depth"], c["dim"], (c["kd"], c["kh"], c["kw"]))
        return dict(kind=kind, runner=run_, weights=_block_weights(g, c["dim"], c["gated"]),
                    x=_randn(g, tiles, grid[0] * grid[1] * grid[2], c["dim"], dtype=torch.bfloat16),
                    qk_norm=c["qk_norm"])
    with torch.device("cuda"):
        if kind == "model":
            net = StrataBackboneModel(
                **_model_kwargs(c), attn_kernel=(c["kd"], c["kh"], c["kw"]), gated_attention=c["gated"],
                qk_norm=c["qk_norm"], do_rope_2d_stereographic=c["rope"] == "stereographic",
                do_rope_2d=c["rope"] == "axial")
        elif kind == "two_stage":
            # the production options: alternating (3,3,3) / (3,1,1) windows, gate, q/k norm
            net = StrataModel(
                **_model_kwargs(c), attn_kernel=3, do_alt_depthwise_attn=True, gated_attention=True,
                qk_norm=True, do_rope_2d_stereographic=True, embed_dim_pixel=128,
                n_layers_pixel=c["pixel_layers"], attn_kernel_pixel=(c["pkd"], c["pkh"], c["pkw"]),
                qk_norm_pixel=True, do_bf16_mixed_pixel=True,
                do_rope_2d_stereographic_pixel=c["pixel_rope"] == "stereographic",
                use_bilinear_dw_gelu_project_adaln_pixel=True)
        else:
            p = c["tile"] + 2 * c["halo"]
            net = StrataBackboneModel(
                depth=c["depth"], height=p, width=p, n_layers=c["layers"], patch_size=1,
                in_chans=c["chans"], base_out_chans=c["chans"], embed_dim=c["dim"],
                num_heads=c["dim"] // 64, attn_kernel=(c["kd"], c["kh"], c["kw"]),
                do_rope_2d_stereographic=True, index_is_latlon=True, do_bf16_mixed=True)
    net = _fill(net, g).eval()
    if kind == "sphere":
        topo = _topology(c["tile"], c["per_dim"], c["halo"])
        x = _randn(g, c["chans"], c["depth"], topo.tiles_per_rank, c["tile"], c["tile"])
        return dict(kind=kind, step=TiledSphereStepper(net, topo), x=x)
    lat, lon = _latlon(g, c["tiles"], c["height"], c["width"])
    x = _randn(g, c["tiles"], c["chans"], c["depth"], c["height"], c["width"])
    return dict(kind="network", net=net, x=x, index={"lat": lat, "lon": lon})


# ------------------------------------------------------------------------------- one pass
def run(state):
    s = state
    kind = s["kind"]
    with torch.inference_mode():
        if kind == "network":
            return s["net"](s["x"], s["index"])
        if kind == "sphere":
            return s["step"](s["x"])
        if kind == "block":
            return ops.block_forward(s["x"], s["weights"], grid=s["grid"], num_heads=s["heads"],
                                     kernel=s["kernel"], rope_cos=None, rope_sin=None, rope_cs=s["cs"],
                                     qk_norm=s["qk_norm"], workspace=s["workspace"])
        if kind == "tiled":
            return s["runner"].block_forward(s["x"], s["weights"], qk_norm=s["qk_norm"])
        if kind == "attention":
            return ops.na3d(s["q"], s["k"], s["v"], s["kernel"])
        padded = s["pad"](s["x"])
        return padded if s["back"] is None else {"padded": padded, "unpadded": s["back"](padded)}
