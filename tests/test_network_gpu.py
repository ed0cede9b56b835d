"""The one-call network forward and the tile-table kernels against the step-by-step path and the
tensor formulas they replace."""
import math

import pytest
import torch

from oracle import block_oracle as bo
from tests.util import tile_latlon

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W,patch", [(1, 8, 8, 4), (2, 33, 31, 1), (1, 32, 32, 1), (3, 36, 100, 4),
                                         (1, 64, 264, 8), (2, 18, 6, 2)])
def test_tile_tables_match_formulas(B, H, W, patch):
    # 1024 pixels is where the tile's sums move to a kernel of their own
    from strata_b200 import ops
    from strata_b200.wrappers import TileGeometry
    lat, lon = tile_latlon(B, H, W)
    lon = lon + 5.9                                            # tiles across the 2 pi seam
    scale = bo.default_rope_length_scale(patch) * 3
    lat0, lon0, cs = ops.tile_tables(lat.cuda(), lon.cuda(), centre=True, rope_mode="stereographic",
                                     patch=patch, length_scale=scale)
    cos, sin = bo.stereographic_rope_tables(lat, lon, 64, patch, scale)
    want = torch.stack([cos, sin], -1)
    assert cs.shape == want.shape
    assert (cs.float().cpu() - want).abs().max() < 6e-4        # half rounding of values up to 1
    w0, w1 = TileGeometry.tile_center(lat.double(), lon.double())
    assert torch.allclose(lat0.cpu().double(), w0.flatten(), atol=1e-6)
    d = (lon0.cpu().double() - w1.flatten() + math.pi) % (2 * math.pi) - math.pi
    assert d.abs().max() < 2e-6
    _, _, ax = ops.tile_tables(lat.cuda(), lon.cuda(), rope_mode="axial", patch=patch)
    cos, sin = bo.axial_rope_tables(H // patch, W // patch, 64)
    assert (ax.float().cpu() - torch.stack([cos, sin], -1)).abs().max() < 6e-4


def _randomised(m):
    g = torch.Generator(device="cuda").manual_seed(3)
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(torch.randn(p.shape, generator=g, device="cuda") * (0.05 if p.dim() == 1 else p[0].numel() ** -0.5))
    return m.eval()


@pytest.mark.parametrize("two_stage,over", [
    (False, dict()), (False, dict(do_rotate_wind=True, wind_channel_indices=(1, 0), gated_attention=True)),
    (False, dict(do_rope_2d_stereographic=False, do_rope_2d=True, qk_norm=True, patch_size_vert=2,
                 attn_kernel=(1, 3, 5))),
    (True, dict(do_rotate_wind=True, wind_channel_indices=(0, 2), qk_norm_pixel=True)),
    (True, dict(do_rope_2d_pixel=True, first_block_only_adaln_pixel=True)),
    (True, dict(do_rope_2d_stereographic_pixel=True, gated_attention_pixel=True)),
    # what the pixel block's two forms (C and Python) could differ in: gate, norm and rotation together, no
    # block modulated but the first, other widths, other factors and kernels (table and tap by tap), runs
    # of rows that do not end with the image, more pixels than one piece of the conditioning
    (True, dict(gated_attention_pixel=True, qk_norm_pixel=True, do_rope_2d_stereographic_pixel=True,
                do_rotate_wind=True, wind_channel_indices=(3, 1))),
    (True, dict(first_block_only_adaln_pixel=True, qk_norm_pixel=True, n_layers_pixel=3,
                attn_kernel_pixel=(1, 5, 7))),
    (True, dict(embed_dim_pixel=192, mlp_ratio_pixel=2.0, patch_size_horiz=8, attn_kernel=3)),
    (True, dict(patch_size_horiz=2, gated_attention=True)),
    (True, dict(depth=5, height=256, width=240, n_layers=1, n_layers_pixel=1))])
def test_one_call_equals_step_by_step(two_stage, over):
    from strata_b200.wrappers import StrataBackboneModel, StrataModel
    kw = dict(depth=4, height=40, width=24, n_layers=2, patch_size_horiz=4, in_chans=5, base_out_chans=4,
              embed_dim=128, num_heads=2, attn_kernel=(3, 3, 5), do_rope_2d_stereographic=True,
              index_is_latlon=True)
    if two_stage:
        kw.update(embed_dim_pixel=64, n_layers_pixel=2, attn_kernel_pixel=(3, 3, 3),
                  use_bilinear_dw_gelu_project_adaln_pixel=True)
    kw.update(over)
    m = _randomised((StrataModel if two_stage else StrataBackboneModel)(**kw).cuda())
    D, H, W = kw["depth"], kw["height"], kw["width"]
    x = torch.randn(2, 5, D, H, W, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    lat, lon = tile_latlon(2, H, W)
    idx = {"lat": lat.cuda(), "lon": lon.cuda()}

    class StepByStep:
        def forward(self, *a):
            return None
    with torch.no_grad():
        y = m(x, idx)
        one_call, m.strata._network = m.strata._network, StepByStep()
        assert torch.equal(m(x, idx), y)
        # a changed weight, module or option reaches the next call
        m.strata._network = one_call
        bb = m.strata.backbone if two_stage else m.strata
        bb.blocks[-1].attn.proj.weight.mul_(1.5)
        bb.blocks[0].mlp.layers[2] = torch.nn.Linear(512, 128).cuda()
        bb.rope_length_scale *= 2.0
        z = m(x, idx)
        m.strata._network = StepByStep()
        assert torch.equal(m(x, idx), z) and not torch.equal(y, z)


@pytest.mark.parametrize("dim,layers,size,gated", [(64, 3, (9, 72, 80), False), (128, 4, (5, 100, 92), True),
                                                   (192, 3, (9, 60, 72), False), (256, 3, (5, 100, 92), False),
                                                   (128, 1, (2, 12, 16), False), (320, 2, (3, 24, 40), False)])
def test_norms_written_by_the_kernels_before_them(dim, layers, size, gated):
    # up to 256 channels a block's second norm comes from its projection, up to 128 the next block's first and the
    # head's from its MLP; step by step they are kernels of their own: the same bits
    from strata_b200.wrappers import StrataBackboneModel
    D, H, W = size
    m = _randomised(StrataBackboneModel(depth=D, height=H, width=W, n_layers=layers, patch_size_vert=1, patch_size_horiz=4,
                                        in_chans=5, base_out_chans=5, embed_dim=dim, num_heads=dim // 64, attn_kernel=(1, 3, 3),
                                        do_rope_2d_stereographic=True, index_is_latlon=True, gated_attention=gated,
                                        do_bf16_mixed=True).cuda())
    x = torch.randn(2, 5, D, H, W, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    lat, lon = tile_latlon(2, H, W)
    idx = {"lat": lat.cuda(), "lon": lon.cuda()}

    class StepByStep:
        def forward(self, *a):
            return None
    with torch.no_grad():
        y = m(x, idx)
        m.strata._network = StepByStep()
        assert torch.equal(m(x, idx), y)


@pytest.mark.parametrize("two_stage,dim,ratio,size", [(False, 64, 2.0, (16, 172, 180)), (True, 64, 2.0, (5, 96, 72)),
                                                      (False, 128, 8.0, (4, 100, 92)), (True, 128, 8.0, (2, 40, 24))])
def test_short_and_long_hidden_layers(two_stage, dim, ratio, size):
    # 64 channels and 128 hidden ones on more rows than three 128-row tiles for each SM: the next norm written by the
    # MLP (one stage), the gated residual (pixel stage, whose single steps are the GEMMs). 128 channels and 1024 hidden
    # ones on so few rows that the two GEMMs are taken, though the projection writes the norm before them
    from strata_b200.wrappers import StrataBackboneModel, StrataModel
    D, H, W = size
    kw = dict(depth=D, height=H, width=W, n_layers=1 if two_stage else 3, patch_size_horiz=4, in_chans=5,
              base_out_chans=4, embed_dim=128 if two_stage else dim, num_heads=2 if two_stage else dim // 64,
              attn_kernel=(1, 3, 3),
              do_rope_2d_stereographic=True, index_is_latlon=True)
    if two_stage:
        kw.update(embed_dim_pixel=dim, n_layers_pixel=2, mlp_ratio_pixel=ratio, attn_kernel_pixel=(1, 3, 3),
                  use_bilinear_dw_gelu_project_adaln_pixel=True)
    else:
        kw.update(mlp_ratio=ratio)
    m = _randomised((StrataModel if two_stage else StrataBackboneModel)(**kw).cuda())
    x = torch.randn(2, 5, D, H, W, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    lat, lon = tile_latlon(2, H, W)
    idx = {"lat": lat.cuda(), "lon": lon.cuda()}

    class StepByStep:
        def forward(self, *a):
            return None
    with torch.no_grad():
        y = m(x, idx)
        m.strata._network = StepByStep()
        assert torch.equal(m(x, idx), y)


def _own_block_code(m, seen):
    """Replaces parts of a model's blocks; every replaced part reports itself in `seen`."""
    import types
    bb = getattr(m.strata, "backbone", m.strata)
    blocks = list(bb.blocks) + list(getattr(m.strata, "pixel_blocks", []))
    for i, b in enumerate(blocks):
        b.register_forward_pre_hook(lambda mod, a, i=i: seen.append(("pre", i)))
        b.register_forward_hook(lambda mod, a, out, i=i: seen.append(("post", i)))

    class Scaled(type(bb.blocks[1])):
        def forward(self, x, *a, **k):
            seen.append("subclass")
            return super().forward(x, *a, **k) * 0.5
    bb.blocks[1].__class__ = Scaled
    stock = bb.blocks[0].forward

    def patched(self, *a, **k):
        seen.append("object")
        return stock(*a, **k)
    bb.blocks[0].forward = types.MethodType(patched, bb.blocks[0])
    return len(blocks)


@pytest.mark.parametrize("two_stage", [False, True])
def test_hooks_and_own_blocks_run(two_stage):
    from tests.test_network_host import small_model
    m = _randomised(small_model(two_stage).cuda())
    x = torch.randn(2, 5, 4, 16, 16, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    lat, lon = tile_latlon(2, 16, 16)
    idx = {"lat": lat.cuda(), "lon": lon.cuda()}
    seen = []
    with torch.no_grad():
        plain = m(x, idx)
        n = _own_block_code(m, seen)
        y = m(x, idx)
    assert seen.count("subclass") == 1 and seen.count("object") == 1
    assert [s for s in seen if isinstance(s, tuple)] == [(w, i) for i in range(n) for w in ("pre", "post")]
    assert torch.isfinite(y).all() and not torch.equal(y, plain)


def test_a_hook_that_only_looks_changes_nothing():
    from tests.test_network_host import small_model
    m = _randomised(small_model().cuda())
    x = torch.randn(1, 5, 4, 16, 16, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    lat, lon = tile_latlon(1, 16, 16)
    idx = {"lat": lat.cuda(), "lon": lon.cuda()}
    got = []
    with torch.no_grad():
        y = m(x, idx)
        handle = m.strata.blocks[0].register_forward_hook(lambda mod, a, out: got.append(out.clone()))
        assert torch.equal(m(x, idx), y) and len(got) == 1 and got[0].shape == (1, 64, 128)
        handle.remove()
        assert torch.equal(m(x, idx), y) and len(got) == 1


@pytest.mark.parametrize("two_stage", [False, True])
@pytest.mark.parametrize("rope", ["none", "axial", "stereographic"])
def test_forward_fused_without_latitudes(two_stage, rope):
    """lat / lon are needed for the wind rotation, the latitude channels and the stereographic table only,
    and pos may bring the table's."""
    from tests.test_network_host import small_model
    over = dict(do_rope_2d_stereographic=rope == "stereographic", do_rope_2d=rope == "axial",
                do_concat_latitude=False)
    if two_stage and rope != "none":
        over["do_rope_2d_stereographic_pixel" if rope == "stereographic" else "do_rope_2d_pixel"] = True
    net = _randomised(small_model(two_stage, **over).cuda()).strata
    x = torch.randn(2, 5, 4, 16, 16, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    lat, lon = (t.cuda() for t in tile_latlon(2, 16, 16))
    pos = torch.stack([lat, lon], 1)
    with torch.no_grad():
        want = net.forward_fused(x, None, lat=lat, lon=lon)
        assert torch.equal(net.forward_fused(x, pos), want)
        # pos, not lat / lon, is the table's
        assert torch.equal(net.forward_fused(x, pos, lat=lat + 0.1, lon=lon), want)
        if rope == "stereographic":
            with pytest.raises(ValueError, match="lat"):
                net.forward_fused(x, None)
        else:
            assert torch.equal(net.forward_fused(x, None), want)
        with pytest.raises(ValueError):
            net.forward_fused(x, None if rope != "stereographic" else pos, wind=(0, 1))
        moved = net.forward_fused(x, None, lat=lat + 0.3 * torch.rand_like(lat), lon=lon)
        assert torch.equal(moved, want) == (rope != "stereographic")


def test_own_tables_and_block_loop_run():
    """A subclass's rope_tables and forward_tokens are what its pass goes through."""
    from strata_b200.strata import StrataTransformer3D
    from tests.test_network_host import small_model
    seen = []

    class Own(StrataTransformer3D):
        def rope_tables(self, pos, n_tiles, grid):
            seen.append(("tables", tuple(pos.shape)))
            return super().rope_tables(pos, n_tiles, grid)

        def forward_tokens(self, tokens, grid, rope_cos, rope_sin):
            seen.append(("tokens", rope_cos.dtype))
            return super().forward_tokens(tokens, grid, rope_cos, rope_sin)
    m = _randomised(small_model().cuda())
    x = torch.randn(1, 5, 4, 16, 16, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    lat, lon = tile_latlon(1, 16, 16)
    idx = {"lat": lat.cuda(), "lon": lon.cuda()}
    with torch.no_grad():
        want = m(x, idx)
        m.strata.__class__ = Own
        y = m(x, idx)
    assert seen == [("tables", (1, 2, 16, 16)), ("tokens", torch.float32)]
    # the table of tensor operations in fp32 against the kernel's in fp64: a few half values differ by one
    assert (y - want).norm() < 5e-3 * want.norm()


@pytest.mark.parametrize("two_stage", [False, True])
def test_inputs_are_checked_and_packed(two_stage):
    from strata_b200 import _lib
    from tests.test_network_host import small_model
    m = _randomised(small_model(two_stage).cuda())
    net = m.strata
    x = torch.randn(2, 5, 4, 16, 16, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    lat, lon = (t.cuda() for t in tile_latlon(2, 16, 16))
    call = lambda x, lat, lon: net.forward_fused(x, None, lat=lat, lon=lon, concat_lat=True)
    with torch.no_grad():
        want = call(x, lat, lon)
        # strided inputs are packed first
        wide = torch.stack([x, x], -1)[..., 0]
        rows = lat[:1, :, :1].expand(2, 16, 16)
        assert not wide.is_contiguous() and not rows.is_contiguous()
        assert torch.equal(call(wide, lat, lon), want)
        assert torch.equal(call(x, rows, lon), call(x, rows.contiguous(), lon))
        for bad in (x.bfloat16(), x.double(), x[0], x.cpu()):
            with pytest.raises((TypeError, ValueError)):
                call(bad, lat, lon)
        for bad in (lat.double(), lat.bfloat16(), lat.cpu()):
            with pytest.raises(TypeError):
                call(x, bad, lon)
        for bad in (lat[:1], lat[:, :8], lat.flatten()):
            with pytest.raises(ValueError):
                call(x, lat, bad)
        with pytest.raises(ValueError, match="input channels"):
            call(x[:, :4], lat, lon)
        with pytest.raises(ValueError, match="divisible"):
            call(x[..., :15], lat[..., :15], lon[..., :15])
        m.cpu()
        with pytest.raises(_lib.StrataLibraryError):
            m(x, {"lat": lat, "lon": lon})
        m.cuda()
        assert torch.equal(call(x, lat, lon), want)


@pytest.mark.parametrize("rope,wind", [("axial", None), ("axial", (0, 1)), ("none", (1, 2))])
@pytest.mark.parametrize("patch", [(1, 4, 2), (2, 2, 8)])
def test_rectangular_patches(rope, wind, patch):
    """The axial table is one of the token grid: patches need not be square (one call, steps, and the
    oracle)."""
    from strata_b200.strata import StrataTransformer3D
    from strata_b200.wrappers import _use_tanh_gelu
    net = StrataTransformer3D(in_channels=7, out_channels=5, input_shape=(4, 16, 24), patch_size=patch,
                              embed_dim=128, num_heads=2, num_layers=2, attn_kernel=(1, 3, 3),
                              rope_mode=rope).cuda()
    _use_tanh_gelu(net)
    _randomised(net)
    x = torch.randn(2, 5, 4, 16, 24, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    lat, lon = (t.cuda() for t in tile_latlon(2, 16, 24))
    with torch.no_grad():
        y = net.forward_fused(x, None, lat=lat, lon=lon, wind=wind, concat_lat=True)
        assert y.shape == x.shape and net._network._state.desc is not None
        handle = net.blocks[0].register_forward_hook(lambda *a: None)
        assert torch.equal(net.forward_fused(x, None, lat=lat, lon=lon, wind=wind, concat_lat=True), y)
        handle.remove()
        if wind is None:     # the same table by tensor operations, through the plain forward
            e = lat.view(2, 1, 1, 16, 24).expand(-1, 1, 4, -1, -1)
            z = net(torch.cat([x, e.cos(), e.sin()], 1), torch.stack([lat, lon], 1))
            assert (y - z).norm() < 5e-3 * z.norm()


def test_rectangular_patches_have_no_stereographic_table():
    from strata_b200.strata import StrataTransformer3D
    from strata_b200.wrappers import _use_tanh_gelu
    net = StrataTransformer3D(in_channels=5, out_channels=5, input_shape=(4, 16, 24), patch_size=(1, 4, 2),
                              embed_dim=128, num_heads=2, num_layers=1, rope_mode="stereographic").cuda()
    _use_tanh_gelu(net)
    x = torch.zeros(1, 5, 4, 16, 24, device="cuda")
    lat, lon = (t.cuda() for t in tile_latlon(1, 16, 24))
    with torch.no_grad(), pytest.raises(ValueError, match="square patches"):
        net.forward_fused(x, None, lat=lat, lon=lon)


@pytest.mark.parametrize("two_stage", [False, True])
def test_first_passes_on_two_streams(two_stage):
    """Weights are cast and tables laid out by the first pass, on its stream; a pass on another stream
    that is issued right behind it reads them whole."""
    from tests.test_network_host import small_model
    x = torch.randn(2, 5, 4, 16, 16, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    lat, lon = tile_latlon(2, 16, 16)
    idx = {"lat": lat.cuda(), "lon": lon.cuda()}
    m = _randomised(small_model(two_stage).cuda())
    with torch.no_grad():
        want = m(x, idx)
        m.strata._network = type(m.strata._network)()
        for mod in m.modules():
            for name in ("_gemm_cache", "_bf16_cache", "_cache"):
                if getattr(mod, name, None) is not None:
                    setattr(mod, name, None)
        torch.cuda.synchronize()
        out = []
        for _ in range(2):
            with torch.cuda.stream(torch.cuda.Stream()):
                torch.cuda._sleep(20_000_000)
                out.append(m(x, idx))
        torch.cuda.synchronize()
        assert all(torch.equal(y, want) for y in out)


@pytest.mark.parametrize("two_stage", [False, True])
def test_first_pass_under_capture(two_stage):
    """Casts that a capture records exist in its replays only; later calls make their own."""
    from tests.test_network_host import small_model
    x = torch.randn(2, 5, 4, 16, 16, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    lat, lon = tile_latlon(2, 16, 16)
    idx = {"lat": lat.cuda(), "lon": lon.cuda()}
    m = _randomised(small_model(two_stage).cuda())
    with torch.no_grad():
        want = m(x, idx)                              # (the library's kernels are loaded)
        fresh = _randomised(small_model(two_stage).cuda())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y = fresh(x, idx)
        assert fresh.strata._network._state is None
        assert torch.equal(fresh(x, idx), want)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)
        del graph


def test_step_by_step_passes_on_two_streams():
    """Passes that are in flight at the same time have scratch of their own."""
    from tests.test_network_host import small_model
    m = _randomised(small_model().cuda())
    m.strata.blocks[0].register_forward_hook(lambda *a: None)
    g = torch.Generator("cuda").manual_seed(1)
    xs = [torch.randn(2, 5, 4, 16, 16, device="cuda", generator=g) for _ in range(4)]
    lat, lon = tile_latlon(2, 16, 16)
    idx = {"lat": lat.cuda(), "lon": lon.cuda()}
    with torch.no_grad():
        want = [m(x, idx) for x in xs]
        torch.cuda.synchronize()
        spaces = []
        for _ in xs:
            with torch.cuda.stream(torch.cuda.Stream()):
                spaces.append(m.strata._get_workspace(512, xs[0].device))
        assert len({t.data_ptr() for t in spaces}) == len(xs)
        out = []
        for x in xs:
            with torch.cuda.stream(torch.cuda.Stream()):
                torch.cuda._sleep(10_000_000)
                out.append(m(x, idx))
        torch.cuda.synchronize()
    assert all(torch.equal(y, w) for y, w in zip(out, want))


def test_raw_stream_lookup_agrees(monkeypatch):
    from strata_b200 import _lib
    x = torch.zeros(1, device="cuda")
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        assert _lib.stream_of(x) == side.cuda_stream
        monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
        assert _lib._stream_lookup()(x.device.index) == side.cuda_stream


def test_blocks_that_differ_take_the_steps():
    """A model whose blocks have no common width of their hidden rows has no descriptors."""
    from strata_b200.strata import Mlp
    from tests.test_network_host import small_model
    from tests.util import rel_max_err
    m = small_model().cuda()
    mlp = Mlp(128, 256).cuda()
    mlp.layers[1] = torch.nn.GELU(approximate="tanh")
    m.strata.blocks[1].mlp = mlp
    x = torch.randn(2, 5, 4, 16, 16, generator=torch.Generator().manual_seed(1))
    lat, lon = tile_latlon(2, 16, 16)
    with torch.no_grad():
        y = m(x.cuda(), {"lat": lat.cuda(), "lon": lon.cuda()})
        assert m.strata._network._state.desc is None
        ref = bo.backbone_forward(x, {k: v.cpu() for k, v in m.state_dict().items()}, patch=(1, 4, 4),
                                  num_heads=2, kernel=3, num_layers=2, lat=lat, lon=lon)
        assert rel_max_err(y, ref) < 2e-2
        mlp.layers[1] = torch.nn.GELU()
        with pytest.raises(RuntimeError, match="tanh GELU"):
            m(x.cuda(), {"lat": lat.cuda(), "lon": lon.cuda()})


@pytest.mark.parametrize("two_stage", [False, True])
def test_threads_with_streams_of_their_own(two_stage):
    """One model, four threads, each with its stream, its batch size and its fields."""
    import threading
    from tests.test_network_host import small_model
    m = _randomised(small_model(two_stage).cuda())
    g = torch.Generator("cuda").manual_seed(1)
    calls = []
    for i in range(4):
        lat, lon = (t.cuda() for t in tile_latlon(1 + i, 16, 16))
        calls.append((torch.randn(1 + i, 5, 4, 16, 16, device="cuda", generator=g), {"lat": lat, "lon": lon}))
    with torch.no_grad():
        want = [m(*c) for c in calls]
    torch.cuda.synchronize()
    m.strata._network = type(m.strata._network)()
    bad, start = [], threading.Barrier(4)

    def work(i):
        try:
            stream = torch.cuda.Stream()
            start.wait(60)
            with torch.no_grad(), torch.cuda.stream(stream):
                out = [m(*calls[i]) for _ in range(30)]
            stream.synchronize()
            bad.extend(i for y in out if not torch.equal(y, want[i]))
        except BaseException as e:
            bad.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not bad, bad


@pytest.mark.parametrize("two_stage", [False, True])
def test_whole_forward_with_wind_beside_64_bits(two_stage, monkeypatch):
    """Against the oracle in 64 bits the model is as far off as the oracle that rounds to bf16 where the
    kernels do (a quarter more is allowed: other sums, other roundings on the way)."""
    from oracle import pixel_oracle as po
    from tests.util import in_double
    from tests.test_network_host import small_model
    over = dict(height=32, width=32, in_chans=5, base_out_chans=5, gated_attention=True, qk_norm=True,
                do_rotate_wind=True, wind_channel_indices=(0, 1))
    if two_stage:
        over.update(qk_norm_pixel=True, attn_kernel_pixel=(3, 5, 5))
    m = _randomised(small_model(two_stage, **over).cuda())
    if two_stage:
        with torch.no_grad():
            for n, p in m.named_parameters():
                if n.endswith("adaln_bilinear_dw_proj.weight"):
                    p.mul_(0.5)
    x = torch.randn(2, 5, 4, 32, 32, generator=torch.Generator().manual_seed(0))
    lat, lon = tile_latlon(2, 32, 32)
    with torch.no_grad():
        y = m(x.cuda(), {"lat": lat.cuda(), "lon": lon.cuda()}).cpu()
    state = {k: v.detach().cpu() for k, v in m.state_dict().items()}
    kw = dict(patch=(1, 4, 4), num_heads=2, kernel=3, num_layers=2, qk_norm=True, gated=True, wind_channels=(0, 1))
    fn = bo.backbone_forward
    if two_stage:
        fn = po.two_stage_forward
        kw.update(num_heads_pixel=1, kernel_pixel=(3, 5, 5), num_layers_pixel=2, qk_norm_pixel=True)
    exact = in_double(monkeypatch, fn, x, state, lat=lat, lon=lon, **kw)
    rounded = fn(x, state, lat=lat, lon=lon, emulate_bf16=True, **kw)
    err = lambda t: float((t.double() - exact).norm() / exact.norm())
    print(f"whole forward with wind vs 64 bits: model {err(y):.3e}, oracle with bf16 {err(rounded):.3e}")
    assert err(y) < 1.25 * err(rounded)
