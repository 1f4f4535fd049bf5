"""What the calls on device tensors refuse before any launch, and what they let through, with and without the extension module
in front of the C ABI.  No GPU: the calls meet a library that writes their arguments down (tests/fake_abi.py)."""
import json
import os
import shutil
import subprocess
import sys

import pytest
import torch

from tests import fake_abi
from tests.fake_abi import STREAM, cuda

U8, F8, BF16, F32, F16 = torch.uint8, torch.float8_e4m3fn, torch.bfloat16, torch.float32, torch.float16
S = dict(stream=STREAM)


def x(rows=8, cols=32, dtype=BF16, **kw):
    return cuda(rows, cols, dtype=dtype, **kw)


def one():
    return cuda(1, dtype=F32)


def pixels(dtype=F32):
    return cuda(2, 3, 32, 48, dtype=dtype)         # 2 x 2 x 3 patches of 16 x 16: rows of 768 codes


# Output buffers of the producer-side steps.
OUT_REFUSED = {
    "quantize_few_rows": lambda e: e.quantize_e4m3(x(), one(), out=cuda(7, 32), **S),
    "quantize_few_columns": lambda e: e.quantize_e4m3(x(), one(), out=cuda(8, 24, stride=(32, 1)), **S),
    "quantize_wide_type": lambda e: e.quantize_e4m3(x(), one(), out=cuda(8, 32, dtype=BF16), **S),
    "quantize_strided": lambda e: e.quantize_e4m3(x(), one(), out=cuda(8, 32, stride=(64, 2)), **S),
    "quantize_three_dimensions": lambda e: e.quantize_e4m3(x(), one(), out=cuda(2, 4, 32), **S),
    "layernorm_few_rows": lambda e: e.layernorm_quantize(x(), None, None, 1e-6, one(), out=cuda(7, 32), **S),
    "layernorm_wide_type": lambda e: e.layernorm_quantize(x(), None, None, 1e-6, one(), out=cuda(8, 32, dtype=F32), **S),
    "patchify_few_rows": lambda e: e.patchify_quantize(pixels(), 16, one(), out=cuda(11, 768), **S),
    "patchify_few_columns": lambda e: e.patchify_quantize(pixels(), 16, one(), out=cuda(12, 760, stride=(768, 1)), **S),
    "patchify_wide_type": lambda e: e.patchify_quantize(pixels(), 16, one(), out=cuda(12, 768, dtype=BF16), **S),
    # the rows are written whole up to a pitch that is a little wider: 16 bytes past the end of this buffer
    "patchify_pad_past_the_end": lambda e: e.patchify_quantize(pixels(), 16, one(), out=cuda(12, 768, stride=(800, 1), offset=32), **S),
}
OUT_TAKEN = {
    "quantize": lambda e: e.quantize_e4m3(x(), one(), out=cuda(8, 32), **S),
    "quantize_f32_codes": lambda e: e.quantize_e4m3(x(dtype=F32), None, out=cuda(8, 32, dtype=F8), **S),
    "quantize_more_rows": lambda e: e.quantize_e4m3(x(), one(), out=cuda(20, 32), **S),
    "quantize_more_columns": lambda e: e.quantize_e4m3(x(), one(), out=cuda(8, 128), **S),
    "quantize_pitched": lambda e: e.quantize_e4m3(x(), one(), out=cuda(8, 32, stride=(128, 1)), **S),
    "quantize_one_column": lambda e: e.quantize_e4m3(x(8, 1), one(), out=cuda(8, 1, stride=(16, 16)), **S),
    "layernorm": lambda e: e.layernorm_quantize(x(), None, None, 1e-6, one(), out=cuda(8, 32, stride=(48, 1)), **S),
    "layernorm_more_rows": lambda e: e.layernorm_quantize(x(), None, None, 1e-6, one(), out=cuda(9, 40), **S),
    "patchify": lambda e: e.patchify_quantize(pixels(), 16, one(), out=cuda(12, 768), **S),
    "patchify_whole_pitch": lambda e: e.patchify_quantize(pixels(BF16), 16, one(), out=cuda(12, 768, stride=(800, 1), elements=12 * 800), **S),
    "patchify_wide_pitch": lambda e: e.patchify_quantize(pixels(), 16, one(), out=cuda(12, 768, stride=(1024, 1)), **S),
    "patchify_more_rows": lambda e: e.patchify_quantize(pixels(), 16, one(), out=cuda(16, 896), **S),
}

# Operands that are not on the engine's GPU (pageable host memory, another GPU).
host = torch.zeros
PLACE_REFUSED = {
    "quantize_x": lambda e: e.quantize_e4m3(host(8, 32), one(), out=cuda(8, 32), **S),
    "quantize_x_new_out": lambda e: e.quantize_e4m3(host(8, 32), one(), **S),
    "quantize_x_other_gpu": lambda e: e.quantize_e4m3(x(device=1), one(), out=cuda(8, 32), **S),
    "quantize_scale": lambda e: e.quantize_e4m3(x(), host(1), out=cuda(8, 32), **S),
    "quantize_out": lambda e: e.quantize_e4m3(x(), one(), out=host(8, 32, dtype=U8), **S),
    "quantize_out_other_gpu": lambda e: e.quantize_e4m3(x(), one(), out=cuda(8, 32, device=1), **S),
    "amax_x": lambda e: e.amax_scale(host(8, 32), **S),
    "amax_x_other_gpu": lambda e: e.amax_scale(x(device=1), **S),
    "layernorm_x": lambda e: e.layernorm_quantize(host(8, 32), None, None, 1e-6, one(), out=cuda(8, 32), **S),
    "layernorm_gamma": lambda e: e.layernorm_quantize(x(), host(32), None, 1e-6, one(), out=cuda(8, 32), **S),
    "layernorm_beta": lambda e: e.layernorm_quantize(x(), None, host(32), 1e-6, one(), out=cuda(8, 32), **S),
    "layernorm_scale": lambda e: e.layernorm_quantize(x(), None, None, 1e-6, host(1), out=cuda(8, 32), **S),
    "layernorm_out": lambda e: e.layernorm_quantize(x(), None, None, 1e-6, one(), out=host(8, 32, dtype=U8), **S),
    "patchify_pixels": lambda e: e.patchify_quantize(host(2, 3, 32, 48), 16, one(), out=cuda(12, 768), **S),
    "patchify_pixels_new_out": lambda e: e.patchify_quantize(host(2, 3, 32, 48), 16, one(), **S),
    "patchify_scale": lambda e: e.patchify_quantize(pixels(), 16, host(1), out=cuda(12, 768), **S),
    "patchify_out": lambda e: e.patchify_quantize(pixels(), 16, one(), out=host(12, 768, dtype=U8), **S),
    "padded_table": lambda e: e.padded_table(host(100, 32, dtype=BF16), **S),
    "table_pos": lambda e: e.make_table(None, host(100, 32), **S),
    "table_bias": lambda e: e.make_table(host(32), cuda(100, 32, dtype=F32), **S),
}

# Activations whose rows are not what a base address and a row pitch describe.
ROWS_REFUSED = {
    "quantize_every_other_column": lambda e: e.quantize_e4m3(x(stride=(64, 2)), one(), out=cuda(8, 32), **S),
    "quantize_transposed": lambda e: e.quantize_e4m3(x(8, 8, stride=(1, 8)), one(), out=cuda(8, 8), **S),
    "quantize_one_row": lambda e: e.quantize_e4m3(x(1, 32, stride=(64, 2)), one(), out=cuda(1, 32), **S),
    "quantize_three_dimensions": lambda e: e.quantize_e4m3(cuda(2, 4, 32, dtype=BF16), one(), out=cuda(8, 32), **S),
    "amax_every_other_column": lambda e: e.amax_scale(x(stride=(64, 2)), **S),
    "amax_three_dimensions": lambda e: e.amax_scale(cuda(2, 4, 32, dtype=BF16), **S),
    "layernorm_every_other_column": lambda e: e.layernorm_quantize(x(stride=(64, 2)), None, None, 1e-6, one(), out=cuda(8, 32), **S),
    "padded_table_transposed": lambda e: e.padded_table(cuda(32, 32, dtype=BF16, stride=(1, 32)), **S),
    "padded_table_type": lambda e: e.padded_table(cuda(32, 32, dtype=F32), **S),
}
ROWS_TAKEN = {
    "quantize_one_column_of_many": lambda e: e.quantize_e4m3(x(8, 1, stride=(64, 64)), one(), out=cuda(8, 16), **S),
    "quantize_pitched": lambda e: e.quantize_e4m3(x(stride=(100, 1)), one(), out=cuda(8, 32), **S),
    "layernorm_one_row": lambda e: e.layernorm_quantize(x(1, 32), None, None, 1e-6, one(), out=cuda(1, 32), **S),
}

# Scales and affine vectors that are not fp32 values in a row, as many as are read.
def gemm(e, f, **kw):
    A, W, res, out = cuda(8, 32), cuda(64, 32), cuda(8, 64, dtype=BF16), cuda(8, 64, dtype=BF16)
    if f == "fc2":
        return e.fc2_residual(A, W, kw.pop("bias", None), res, out=out, **kw, **S)
    if f == "embed":
        return e.patch_embed(A, W, cuda(100, 64, dtype=BF16), out=out, **kw, **S)
    if f == "mlp":
        kw = dict(bias1=None, bias2=None, scale_a=None, scale_w1=None, scale_w2=None, hidden_scale=one()) | kw
        return e.mlp_chain(A, W, kw.pop("bias1"), cuda(32, 64), kw.pop("bias2"), cuda(8, 32, dtype=BF16), hidden=cuda(8, 64),
                           out=cuda(8, 32, dtype=BF16), **kw, **S)
    return (e.fc1_gelu if f == "fc1" else e.linear_bias)(A, W, kw.pop("bias", None), out=out, **kw, **S)


GEMM_SCALES = [(f, s) for f, names in (("fc1", "scale_a scale_b out_scale"), ("linear", "scale_a scale_b out_scale"), ("fc2", "scale_a scale_b"),
                                       ("embed", "scale_a scale_b"), ("mlp", "scale_a scale_w1 scale_w2 hidden_scale")) for s in names.split()]
FLOATS_REFUSED = {f"{f}_{s}_{t}": (lambda e, f=f, s=s, t=t: gemm(e, f, **{s: cuda(1, dtype=t) if t else cuda(0, dtype=F32, stride=(1,))}))
                  for f, s in GEMM_SCALES for t in (BF16, torch.float64, None)} | {
    "quantize_scale_bf16": lambda e: e.quantize_e4m3(x(), cuda(1, dtype=BF16), out=cuda(8, 32), **S),
    "patchify_scale_f64": lambda e: e.patchify_quantize(pixels(), 16, cuda(1, dtype=torch.float64), out=cuda(12, 768), **S),
    "layernorm_scale_int": lambda e: e.layernorm_quantize(x(), None, None, 1e-6, cuda(1, dtype=torch.int32), out=cuda(8, 32), **S),
    "layernorm_gamma_bf16": lambda e: e.layernorm_quantize(x(), cuda(32, dtype=BF16), None, 1e-6, one(), out=cuda(8, 32), **S),
    "layernorm_beta_short": lambda e: e.layernorm_quantize(x(), None, cuda(31, dtype=F32), 1e-6, one(), out=cuda(8, 32), **S),
    "layernorm_gamma_strided": lambda e: e.layernorm_quantize(x(), cuda(32, dtype=F32, stride=(2,)), None, 1e-6, one(), out=cuda(8, 32), **S),
}
FLOATS_TAKEN = {f"{f}_{s}": (lambda e, f=f, s=s: gemm(e, f, **{s: one()})) for f, s in GEMM_SCALES} | {
    "fc1_scale_of_more": lambda e: gemm(e, "fc1", scale_a=cuda(4, dtype=F32), scale_b=cuda(1, 1, dtype=F32)),
    "fc1_scale_expanded": lambda e: gemm(e, "fc1", scale_a=cuda(4, dtype=F32, stride=(0,))),
    "layernorm_affine": lambda e: e.layernorm_quantize(x(), cuda(32, dtype=F32), cuda(2, 32, dtype=F32), 1e-6, one(), out=cuda(8, 32), **S),
}

# Biases: bf16, or fp32 with the flag that says so, as many as the layer is wide.
BIAS_REFUSED = {f"{f}_{what}": (lambda e, f=f, b=b, kw=kw: gemm(e, f, bias=b(), **kw)) for f in ("fc1", "linear", "fc2") for what, b, kw in (
    ("fp16", lambda: cuda(64, dtype=F16), {}), ("fp64", lambda: cuda(64, dtype=torch.float64), {}),
    ("flag_contradicts", lambda: cuda(64, dtype=BF16), dict(flags=1)), ("short", lambda: cuda(63, dtype=BF16), {}),
    ("short_f32", lambda: cuda(48, dtype=F32), {}), ("strided", lambda: cuda(64, dtype=BF16, stride=(2,)), {}))} | {
    "mlp_bias2_fp16": lambda e: gemm(e, "mlp", bias2=cuda(32, dtype=F16)),
    "mlp_bias1_fp16": lambda e: gemm(e, "mlp", bias1=cuda(64, dtype=F16)),
    "mlp_types_differ": lambda e: gemm(e, "mlp", bias1=cuda(64, dtype=F32), bias2=cuda(32, dtype=BF16)),
    "mlp_types_differ_too": lambda e: gemm(e, "mlp", bias1=cuda(64, dtype=BF16), bias2=cuda(32, dtype=F32)),
    "table_short": lambda e: e.make_table(cuda(31, dtype=F32), cuda(100, 32, dtype=F32), **S),
    "mlp_bias1_short": lambda e: gemm(e, "mlp", bias1=cuda(32, dtype=BF16)),
    "mlp_bias2_short": lambda e: gemm(e, "mlp", bias2=cuda(31, dtype=BF16)),
}
BIAS_TAKEN = {f"{f}_{what}": (lambda e, f=f, b=b, kw=kw: gemm(e, f, bias=b(), **kw)) for f in ("fc1", "linear", "fc2") for what, b, kw in (
    ("bf16", lambda: cuda(64, dtype=BF16), {}), ("f32", lambda: cuda(64, dtype=F32), {}), ("f32_flag", lambda: cuda(64, dtype=F32), dict(flags=1)),
    ("none_flag", lambda: None, dict(flags=1)), ("row", lambda: cuda(1, 64, dtype=BF16), {}), ("longer", lambda: cuda(80, dtype=BF16), {}))} | {
    "mlp_bf16": lambda e: gemm(e, "mlp", bias1=cuda(64, dtype=BF16), bias2=cuda(32, dtype=BF16)),
    "mlp_f32": lambda e: gemm(e, "mlp", bias1=cuda(64, dtype=F32), bias2=cuda(32, dtype=F32)),
    "mlp_second_f32": lambda e: gemm(e, "mlp", bias2=cuda(32, dtype=F32)),
}

REFUSED = {f"bias_{k}": v for k, v in BIAS_REFUSED.items()} | {f"floats_{k}": v for k, v in FLOATS_REFUSED.items()} | {f"rows_{k}": v for k, v in ROWS_REFUSED.items()} | {f"place_{k}": v for k, v in PLACE_REFUSED.items()} | {f"out_{k}": v for k, v in OUT_REFUSED.items()}
TAKEN = {f"bias_{k}": v for k, v in BIAS_TAKEN.items()} | {f"floats_{k}": v for k, v in FLOATS_TAKEN.items()} | {f"rows_{k}": v for k, v in ROWS_TAKEN.items()} | {f"out_{k}": v for k, v in OUT_TAKEN.items()}


@pytest.mark.gpu
def test_pinned_operands_are_read_in_place(engine):
    """Host memory that the GPU reaches stays an operand of the producer-side steps."""
    g = torch.Generator().manual_seed(0)
    rows, px, scale = torch.randn((40, 64), generator=g).to(BF16), torch.rand((1, 3, 32, 32), generator=g), torch.tensor([0.05])
    gpu = lambda t: t.to("cuda")
    for size, call in (((40, 64), lambda f, out: engine.quantize_e4m3(f(rows), f(scale), out=out)),
                       ((40, 64), lambda f, out: engine.layernorm_quantize(f(rows), None, None, 1e-6, f(scale), out=out)),
                       ((4, 768), lambda f, out: engine.patchify_quantize(f(px), 16, f(scale), out=out))):
        want = call(gpu, torch.zeros(size, dtype=U8, device="cuda"))
        assert torch.equal(call(torch.Tensor.pin_memory, torch.zeros(size, dtype=U8, device="cuda")), want)
        onto = call(gpu, torch.zeros(size, dtype=U8).pin_memory())
        engine.device_status()
        assert torch.equal(onto, want.cpu())

# Calls whose stream is torch's current one: without a driver asking for it throws, in the middle of the extension's work.
THROWS = {"quantize": lambda e: e.quantize_e4m3(x(), one(), out=cuda(8, 32)), "fc1": lambda e: e.fc1_gelu(cuda(8, 32), cuda(64, 32), None, out=cuda(8, 64, dtype=BF16))}


@pytest.fixture(scope="module")
def folder(tmp_path_factory):
    path = tmp_path_factory.mktemp("fake_abi")
    fake_abi.install(path)
    return path


@pytest.fixture(scope="module")
def results(folder):
    out = {}
    for table in ("REFUSED", "TAKEN"):
        r = fake_abi.run_child(folder, __name__, table)
        assert r.returncode == 0, r.stdout + r.stderr
        out[table] = json.loads(r.stdout.splitlines()[-1])
    return out


@pytest.mark.parametrize("name", REFUSED)
def test_refused_before_any_launch(results, name):
    for route, (error, message, calls) in results["REFUSED"][name].items():
        assert error in ("ValueError", "TypeError") and not calls, f"{route}: {error} {message} {calls}"
    assert results["REFUSED"][name]["extension"] == results["REFUSED"][name]["python"]


@pytest.mark.skipif(torch.cuda.is_available(), reason="with a driver nothing throws here")
def test_a_throw_inside_the_extension_is_an_exception(folder):
    r = fake_abi.run_child(folder, __name__, "THROWS")
    assert r.returncode == 0, f"the process died ({r.returncode}): {r.stderr[-2000:]}"
    for name, routes in json.loads(r.stdout.splitlines()[-1]).items():
        assert routes["extension"][0] and not routes["extension"][2], (name, routes)


def test_the_extension_calls_the_library_beside_it(folder, tmp_path):
    """Another copy of the library on LD_LIBRARY_PATH must not get the handles of the one the engine loaded."""
    other = tmp_path / "libsiglip_fp8.so"
    (tmp_path / "other.c").write_text("int nothing;")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(other), str(tmp_path / "other.c")], check=True)      # holds none of the entry points
    r = fake_abi.run_child(folder, __name__, "OUT_TAKEN", LD_LIBRARY_PATH=f"{tmp_path}:{os.environ.get('LD_LIBRARY_PATH', '')}")
    assert r.returncode == 0 and "RuntimeWarning" not in r.stderr, r.stderr


@pytest.mark.parametrize("state", ["missing", "not a module", "another torch"])
def test_without_the_extension_the_calls_go_through_python(folder, tmp_path, state):
    """An engine needs libsiglip_fp8.so; a missing or stale extension module is said, and costs time only."""
    shutil.copy(folder / "libsiglip_fp8.so", tmp_path)
    if state == "not a module":
        (tmp_path / "sl8_torch.so").write_text("no ELF file")
    if state == "another torch":
        shutil.copy(folder / "sl8_torch.so", tmp_path)
    pretend = "import torch; torch.__version__ = '0.0.1'; " if state == "another torch" else ""
    code = (f"{pretend}import pathlib, warnings; from tests import fake_abi, test_operand_checks as t\n"
            "with warnings.catch_warnings(record=True) as said:\n    warnings.simplefilter('always')\n"
            f"    fast, _, calls = fake_abi.engines(pathlib.Path({str(tmp_path)!r}))\n"
            "assert any('python -m siglip_b200.build' in str(w.message) for w in said), said\n"
            "t.TAKEN['bias_fc1_bf16'](fast); t.TAKEN['out_quantize'](fast); assert len(calls()) == 2")
    r = subprocess.run([sys.executable, "-c", code], cwd=fake_abi.ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr


def test_the_build_asks_which_torch_the_extension_was_built_for(tmp_path, monkeypatch):
    from siglip_b200 import build
    monkeypatch.setattr(build, "BINDING", tmp_path / "sl8_torch.so")
    assert not build.binding_current()
    build.BINDING.touch()
    (tmp_path / "sl8_torch.tag").write_text(build.torch_tag())
    assert build.binding_current()
    (tmp_path / "sl8_torch.tag").write_text("0.0.1 cpython-38")
    assert not build.binding_current()


@pytest.mark.gpu
def test_a_new_output_without_memory_is_an_exception(engine):
    """Under a fake-tensor mode the output that the call allocates has no address: an error, as without the extension."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    A, W = torch.zeros((128, 64), dtype=U8, device="cuda"), torch.zeros((64, 64), dtype=U8, device="cuda")
    with FakeTensorMode(allow_non_fake_inputs=True), pytest.raises(Exception):
        engine.fc1_gelu(A, W, None)
    engine.device_status()


def test_the_flag_says_what_the_biases_are(results):
    """The last argument but the stream of mlp_chain: one bit for both biases, whichever is given."""
    flag = {k: int(results["TAKEN"][f"bias_mlp_{k}"]["python"][2][0].split()[-2]) for k in ("bf16", "f32", "second_f32")}
    assert flag == {"bf16": 0, "f32": 1, "second_f32": 1}


@pytest.mark.parametrize("name", TAKEN)
def test_taken_with_the_same_arguments(results, name):
    for route, (error, message, calls) in results["TAKEN"][name].items():
        assert error is None and len(calls) == 1, f"{route}: {error} {message} {calls}"
    assert results["TAKEN"][name]["extension"] == results["TAKEN"][name]["python"]
