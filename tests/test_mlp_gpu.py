"""The one-kernel MLP of narrow blocks against the two GEMMs it stands for (same bits) and the fp32 result."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from strata_b200 import ops
    return ops


def _data(M, C, H, seed, pad=0):
    g = torch.Generator("cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    rows = lambda: rnd(M, C + pad).bfloat16()[:, :C]       # pad: rows with a stride of their own
    return dict(x=rows(), aux=rows(), gate=rows(), w1=(rnd(H, C) * C ** -0.5).bfloat16(),
                w2=(rnd(C, H) * H ** -0.5).bfloat16(), b1=rnd(H) * 0.1, b2=rnd(C) * 0.1)


def _fused(ops, d, aux, gate, bias, out):
    from strata_b200 import _lib
    ptr = lambda t: None if t is None else t.data_ptr()
    ld = lambda t: 0 if t is None else t.stride(0)
    M, C = d["x"].shape
    H = d["w1"].shape[0]
    b1, b2 = (d["b1"], d["b2"]) if bias else (None, None)
    lib = _lib.load()
    assert lib.strata_mlp_bf16(ptr(d["x"]), ld(d["x"]), ptr(d["w1"]), ptr(b1), ptr(d["w2"]), ptr(b2), ptr(aux), ld(aux),
                               ptr(gate), ld(gate), ptr(out), ld(out), M, C, H,
                               torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert _lib.device_status() == 0


# rows: one, the edges of a 128-row tile and of a 32-row box, one tile more than the SMs, several tiles a CTA;
# hidden: one chunk, an odd number of them, several
@pytest.mark.parametrize("M,C,H,mode,pad", [
    (1, 64, 128, "residual", 0), (127, 64, 256, "bias", 0), (129, 128, 128, "residual", 8), (31, 128, 512, "gate", 0),
    (97, 192, 768, "gate", 8), (256, 192, 384, "residual", 0), (300, 256, 1024, "residual", 0), (160, 256, 128, "bias", 8),
    (149 * 128 + 5, 128, 512, "gate", 0), (149 * 128 + 5, 256, 384, "residual", 0), (45001, 64, 128, "residual", 0),
    (60007, 128, 384, "residual", 0), (60007, 192, 768, "gate", 0), (60007, 256, 1024, "bias", 0)])
@pytest.mark.parametrize("bias", [True, False])
def test_mlp_is_the_two_gemms(ops, M, C, H, mode, pad, bias):
    from strata_b200 import _lib
    d = _data(M, C, H, M + C + H, pad)
    b1, b2 = (d["b1"], d["b2"]) if bias else (None, None)
    aux = d["aux"] if mode != "bias" else None
    gate = d["gate"] if mode == "gate" else None
    out = torch.full((M, C + pad), float("nan"), device="cuda", dtype=torch.bfloat16)[:, :C]
    _fused(ops, d, aux, gate, bias, out)
    h = ops.linear(d["x"], d["w1"], b1, ops.EPI_GELU)
    if mode == "residual":
        want = ops.linear(h, d["w2"], b2, ops.EPI_RESIDUAL, aux)
    else:
        want = ops.linear(h, d["w2"], b2)
        if mode == "gate":
            y, want = want, torch.empty_like(want)
            assert _lib.load().strata_adaln_rows_bf16(
                aux.data_ptr(), aux.stride(0), y.data_ptr(), C, gate.data_ptr(), gate.stride(0), want.data_ptr(), C,
                None, None, 0, None, 0, M, C, 1e-6, torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(out, want)
    t = torch.nn.functional.gelu(d["x"].double() @ d["w1"].double().T + (b1.double() if bias else 0.0), approximate="tanh")
    t = t @ d["w2"].double().T + (b2.double() if bias else 0.0)
    if mode != "bias":
        t = aux.double() + (gate.double() if gate is not None else 1.0) * t
    # bf16 hidden channels and result: two roundings of 2^-9 relative rms at most, and bf16's own
    assert float((out.double() - t).norm() / t.norm()) < 4e-3


# 64 channels leave half of the epilogue warps without output columns, and with one chunk a tile those take only every
# other tile's: four tiles a CTA and more (148 x 128 rows are one), where such warps run ahead of the readers
@pytest.mark.parametrize("M,C,H,mode", [
    (60007, 64, 128, "residual"), (60007, 64, 256, "gate"), (200003, 64, 128, "gate"), (200003, 64, 128, "bias"),
    (200003, 64, 256, "residual"), (200003, 64, 384, "residual"), (100003, 128, 128, "residual")])
def test_mlp_of_many_tiles_a_cta(ops, M, C, H, mode):
    test_mlp_is_the_two_gemms(ops, M, C, H, mode, 0, True)


def test_mlp_in_place_and_through_ops(ops):
    d = _data(5000, 128, 512, 3)
    want = ops.linear(ops.linear(d["x"], d["w1"], d["b1"], ops.EPI_GELU), d["w2"], d["b2"], ops.EPI_RESIDUAL, d["aux"])
    assert torch.equal(ops.mlp(d["x"], d["w1"], d["b1"], d["w2"], d["b2"], d["aux"]), want)
    x = d["aux"].clone()
    _fused(ops, d, x, None, True, x)            # the result goes over the residual
    assert torch.equal(x, want)


def test_mlp_refuses_what_it_has_no_kernel_for(ops):
    from strata_b200 import _lib
    x = torch.zeros(128, 320, device="cuda", dtype=torch.bfloat16)
    f = _lib.load().strata_mlp_bf16
    p = x.data_ptr()
    assert f(p, 320, p, None, p, None, None, 0, None, 0, p, 320, 128, 320, 1280, 0) == -2     # too wide
    assert f(p, 320, p, None, p, None, None, 0, None, 0, p, 320, 128, 128, 320, 0) == -2      # part of a chunk
    assert f(p, 320, p, None, p, None, None, 0, p, 320, p, 320, 128, 128, 128, 0) == -1       # a gate without aux
    assert f(p + 2, 320, p, None, p, None, None, 0, None, 0, p, 320, 128, 128, 128, 0) == -1  # alignment


def test_mlp_of_wrong_weights_raises(ops):
    z = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.bfloat16)
    x, w1, w2 = z(256, 128), z(512, 128), z(128, 512)
    b1, b2 = torch.zeros(512, device="cuda"), torch.zeros(128, device="cuda")
    assert ops.mlp(x, w1, b1, w2, b2, x).shape == x.shape
    for bad in (z(512, 64), z(512, 192), z(512), z(512, 128, 1)):
        with pytest.raises(ValueError):
            ops.mlp(x, bad, b1, w2, b2, x)
    for bad in (z(128, 384), z(64, 512), z(128, 640)):
        with pytest.raises(ValueError):
            ops.mlp(x, w1, b1, bad, b2, x)
    for bad in (z(256, 64), z(128, 128)):
        with pytest.raises(ValueError):
            ops.mlp(x, w1, b1, w2, b2, bad)


def test_mlp_of_one_row_with_any_row_stride(ops):
    # the row stride of a single row says nothing: linear takes such a view, and so does this
    d = _data(1, 128, 512, 5)
    x, aux = (t.contiguous().view(128, 1).t() for t in (d["x"], d["aux"]))
    assert x.stride() == (1, 1)
    h = ops.linear(x, d["w1"], d["b1"], ops.EPI_GELU)
    want = ops.linear(h, d["w2"], d["b2"], ops.EPI_RESIDUAL, aux)
    assert torch.equal(ops.mlp(x, d["w1"], d["b1"], d["w2"], d["b2"], aux), want)


# the two ways as measured: turns of 148 row blocks (18944 rows), the last one's share, chunks of 128 hidden channels
@pytest.mark.parametrize("M,C,H,fused", [
    (37889, 192, 768, 0), (40000, 192, 768, 0), (45000, 192, 768, 0), (57000, 192, 768, 0), (75776, 192, 768, 1),
    (37889, 256, 1024, 0), (45000, 256, 1024, 1), (57000, 256, 1024, 1), (37889, 192, 1536, 1), (37889, 256, 2048, 1),
    (57000, 256, 512, 0), (45000, 192, 384, 0), (151552, 192, 384, 1), (9472, 256, 1024, 0), (9473, 256, 1024, 1),
    (18945, 192, 768, 0), (37888, 192, 768, 1), (128, 128, 512, 1), (128, 128, 1024, 0), (8192, 128, 1024, 1),
    (128, 64, 128, 1), (128, 128, 320, 0), (1 << 20, 320, 1280, 0)])
def test_mlp_rule(ops, M, C, H, fused):
    from strata_b200 import _lib
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the line lies by turns of 148 SMs")
    assert _lib.load().strata_mlp_fused(M, C, H) == fused
