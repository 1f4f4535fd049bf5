"""The extension module in front of the C ABI: what it takes gives bit for bit what the Python methods give by themselves, and
what it does not take (wrong types, shapes, pitches, devices; tensor subclasses) raises or runs there as before."""
import types

import pytest
import torch

import siglip_b200
from siglip_b200 import lib as L, synth

DEV = "cuda"


def _engines():
    fast, slow = siglip_b200.Engine(0), siglip_b200.Engine(0)
    slow._native = L.NoBinding()
    assert not isinstance(fast._native, L.NoBinding)
    return fast, slow


def _operands(M=300, d=256, ff=512):
    g = torch.Generator(device=DEV).manual_seed(7)
    codes = lambda r, c: synth.quantize_e4m3(torch.randn((r, c), generator=g, device=DEV) * 0.1)[0]
    bf = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)
    o = types.SimpleNamespace(A=codes(M, d), W1=codes(ff, d), W2=codes(d, ff), H=codes(M, ff), b1=bf(ff), b2=bf(d), res=bf(M, d), x=bf(M, d),
                              table=bf(100 + 128, d), sq=codes(d, d), one=torch.ones(1, device=DEV), s=torch.full((1,), 0.02, device=DEV),
                              px=torch.rand((2, 3, 64, 64), generator=g, device=DEV), M=M, d=d, ff=ff)
    o.pitched = lambda c: torch.zeros((M, synth.pitch128(c) + 128), dtype=torch.uint8, device=DEV)[:, :c]
    return o


CALLS = {
    "fc1": lambda e, o: e.fc1_gelu(o.A, o.W1, o.b1, scale_a=o.s, scale_b=o.s),
    "fc1_f32_bias": lambda e, o: e.fc1_gelu(o.A, o.W1, o.b1.float(), scale_a=o.s, flags=L.SL8_FLAG_GELU_HW_TANH),
    "fc1_new_e4m3": lambda e, o: e.fc1_gelu(o.A, o.W1, None, scale_a=o.s, out_dtype=torch.float8_e4m3fn, out_scale=o.s),
    "fc1_new_u8": lambda e, o: e.fc1_gelu(o.A.view(torch.uint8), o.W1, None, out_dtype=torch.uint8, out_scale=o.s),
    "fc1_out": lambda e, o: e.fc1_gelu(o.A, o.W1, o.b1, scale_a=o.s, out=o.pitched(o.ff), out_scale=o.s),
    "linear": lambda e, o: e.linear_bias(o.A, o.W1, o.b1, scale_a=o.s),
    "linear_out_and_type": lambda e, o: e.linear_bias(o.A, o.W1, o.b1, out=o.pitched(o.ff), out_dtype=torch.uint8, out_scale=o.s),
    "fc2": lambda e, o: e.fc2_residual(o.H, o.W2, o.b2, o.res, scale_a=o.s, scale_b=o.s),
    "fc2_rows": lambda e, o: e.fc2_residual(o.H[32:], o.W2, None, o.res[32:], scale_a=o.s, out=torch.empty_like(o.res)[32:]),
    "mlp": lambda e, o: e.mlp_chain(o.A, o.W1, o.b1, o.W2, o.b2, o.res, scale_a=o.s, scale_w1=o.s, scale_w2=o.s, hidden_scale=o.s, hidden=o.pitched(o.ff)),
    "embed": lambda e, o: e.patch_embed(o.A, o.sq, o.table, period=100, row_phase=7, scale_a=o.s),
    "embed_whole_table": lambda e, o: e.patch_embed(o.A, o.sq, o.table, out=torch.empty_like(o.res)),
    "patchify": lambda e, o: e.patchify_quantize(o.px, 16, o.s, out=torch.zeros((32, 768), dtype=torch.uint8, device=DEV)),
    "patchify_new": lambda e, o: e.patchify_quantize(o.px[..., :60].contiguous(), 14, o.s),
    "patchify_new_pitch": lambda e, o: e.patchify_quantize(o.px, 16, o.s, pitch=1024),
    "quantize_new": lambda e, o: e.quantize_e4m3(o.x[:, :200].float(), o.s),
    "layernorm_new": lambda e, o: e.layernorm_quantize(o.x[:, :200], None, None, 1e-6, o.s),
    "mlp_new": lambda e, o: e.mlp_chain(o.A, o.W1, o.b1, o.W2, o.b2, o.res, scale_a=o.s, scale_w1=o.s, scale_w2=o.s, hidden_scale=o.s),
    "amax": lambda e, o: torch.cat(e.amax_scale(o.x)),
    "quantize": lambda e, o: e.quantize_e4m3(o.x, o.s, out=o.pitched(o.d)),
    "layernorm": lambda e, o: e.layernorm_quantize(o.x, None, None, 1e-6, o.s, out=o.pitched(o.d)),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", CALLS)
def test_extension_and_python_agree(name):
    fast, slow = _engines()
    o = _operands()
    taken = []
    real = fast._native
    fast._native = types.SimpleNamespace(**{f: (lambda *a, f=f: taken.append(getattr(real, f)(*a)) or taken[-1])
                                            for f in dir(real) if not f.startswith("_")})
    got, want = CALLS[name](fast, o), CALLS[name](slow, o)
    assert got.dtype == want.dtype and got.shape == want.shape and torch.equal(got.contiguous().view(torch.uint8), want.contiguous().view(torch.uint8))
    assert got.stride() == want.stride() and got.untyped_storage().nbytes() == want.untyped_storage().nbytes()
    if name not in ("linear_out_and_type", "patchify_new_pitch"):
        assert len(taken) == 1 and taken[0] is not None      # the extension took the call
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        again = CALLS[name](fast, o)
    side.synchronize()
    assert torch.equal(again.contiguous().view(torch.uint8), want.contiguous().view(torch.uint8))


BAD = {
    "types": lambda e, o: e.fc1_gelu(o.x, o.W1, o.b1),
    "K": lambda e, o: e.fc1_gelu(o.A, o.W2, o.b1),
    "k_strided": lambda e, o: e.fc1_gelu(o.A.view(torch.uint8)[:, ::2], o.W1.view(torch.uint8)[:, ::2], None),
    "host": lambda e, o: e.fc1_gelu(o.A.cpu(), o.W1, None),
    "bias_type": lambda e, o: e.fc1_gelu(o.A, o.W1, o.b1.half()),
    "host_scale": lambda e, o: e.fc1_gelu(o.A, o.W1, None, scale_a=torch.ones(1)),
    "out_shape": lambda e, o: e.fc1_gelu(o.A, o.W1, None, out=o.res),
    "out_type": lambda e, o: e.fc2_residual(o.H, o.W2, None, o.res, out=o.pitched(o.d)),
    "residual": lambda e, o: e.fc2_residual(o.H, o.W2, None, o.res[1:]),
    "flags": lambda e, o: e.fc1_gelu(o.A, o.W1, None, flags=64),
    "table": lambda e, o: e.patch_embed(o.A, o.sq, o.table[:, ::2]),
    "period": lambda e, o: e.patch_embed(o.A, o.sq, o.table, period=10 ** 6),
    "hidden_scale": lambda e, o: e.mlp_chain(o.A, o.W1, o.b1, o.W2, o.b2, o.res, scale_a=o.s, scale_w1=o.s, scale_w2=o.s, hidden_scale=None, hidden=o.pitched(o.ff)),
    "hidden_shape": lambda e, o: e.mlp_chain(o.A, o.W1, o.b1, o.W2, o.b2, o.res, scale_a=o.s, scale_w1=o.s, scale_w2=o.s, hidden_scale=o.s, hidden=o.pitched(o.d)),
    "pixels": lambda e, o: e.patchify_quantize(o.px.transpose(2, 3)[..., ::2], 16, o.s, out=o.pitched(o.d)),
    "patch": lambda e, o: e.patchify_quantize(o.px, 0, o.s, out=o.pitched(o.d)),
    "quantize_type": lambda e, o: e.quantize_e4m3(o.x.half(), o.s, out=o.pitched(o.d)),
    "layernorm_width": lambda e, o: e.layernorm_quantize(o.x[:, :100], None, None, 1e-6, o.s, out=o.pitched(100)),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", BAD)
def test_refusals_are_the_same(name):
    errors = []
    for e in _engines():
        with pytest.raises(Exception) as info:
            BAD[name](e, _operands())
        errors.append((type(info.value), str(info.value)))
    assert errors[0] == errors[1]


@pytest.mark.gpu
def test_subclasses_go_through_python_and_outputs_are_the_tensor_given():
    fast, _ = _engines()
    o = _operands()

    class Tagged(torch.Tensor):
        pass

    want = fast.fc1_gelu(o.A, o.W1, o.b1)
    assert torch.equal(fast.fc1_gelu(o.A.as_subclass(Tagged), o.W1, o.b1), want)
    out = torch.empty_like(want)
    assert fast.fc1_gelu(o.A, torch.nn.Parameter(o.W1, requires_grad=False), o.b1, out=out) is out
    with pytest.raises(Exception):
        torch.func.vmap(lambda a: fast.fc1_gelu(a, o.W1, o.b1))(o.A.view(torch.uint8)[None])


@pytest.mark.gpu
@pytest.mark.parametrize("route", [0, 1])
def test_hidden_activations_stay_until_the_stream_is_done(route):
    """The scratch that mlp_chain allocates must not be handed out again while the stream it was given still has to use it."""
    e, M, d, ff = _engines()[route], 2048, 256, 4096
    g = torch.Generator(device=DEV).manual_seed(1)
    codes = lambda r, c: torch.randint(0, 256, (r, c), generator=g, device=DEV, dtype=torch.uint8) & 0xBF
    A, W1, W2, res, s = codes(M, d), codes(ff, d), codes(d, ff), torch.zeros((M, d), dtype=torch.bfloat16, device=DEV), torch.ones(1, device=DEV)
    out, side = torch.empty_like(res), torch.cuda.Stream()
    kw = dict(scale_a=s, scale_w1=s, scale_w2=s, hidden_scale=s, out=out)
    e.mlp_chain(A, W1, None, W2, None, res, **kw)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.empty((M, ff), dtype=torch.uint8, device=DEV)
    where = free.data_ptr()
    del free                                       # the one free block of that size: the call's scratch
    with torch.cuda.stream(side):
        torch.cuda._sleep(200_000_000)
    e.mlp_chain(A, W1, None, W2, None, res, stream=side, **kw)
    again = torch.empty((M, ff), dtype=torch.uint8, device=DEV)
    assert not side.query() and again.data_ptr() != where
    side.synchronize()
    e.device_status()
