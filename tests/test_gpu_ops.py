"""Parity of the CUDA kernels with the CPU oracle, through the C ABI (graph flavour via the
Python surface, eager flavour via raw ctypes in test_gpu_eager_abi.py).

Bars: bit-exact for quantize, argmax, gather, index_select, embedding;
<= 1e-5 relative for fp32 element-wise and reduction ops; bf16/f16 compared with the oracle run
in the same storage type. Shapes mirror the reference's tests (python/tests/test_transformer_ops.py,
test_batched_ops.py, crates/core/src/ops.rs tests) plus ragged / empty / non-multiple-of-vector sizes.
"""
import json
import os

import numpy as np
import pytest

from oracle import msl_ref as R

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
with open(os.path.join(HERE, "golden", "known_answers.json")) as f:
    CASES = json.load(f)["cases"]

REL = 1e-5  # fp32 bar from the north star


def close(got, ref, rel=REL, abs_=1e-6):
    got = np.asarray(got, np.float64); ref = np.asarray(ref, np.float64)
    assert got.shape == ref.shape, (got.shape, ref.shape)
    err = np.abs(got - ref)
    bound = abs_ + rel * np.abs(ref)
    assert np.all(err <= bound), f"max err {err.max()} at {np.unravel_index(err.argmax(), err.shape)}; ref there {ref.reshape(-1)[err.argmax()]}"


def bf16_bits(x):
    return R.to_bf16(np.asarray(x, np.float32))


def up_bf16(gpu, x):
    return gpu.from_bytes(bf16_bits(x).tobytes(), list(np.shape(x)), "bfloat16")


def run_gpu_case(gpu, c):
    f32 = lambda v: gpu.from_numpy(np.asarray(v, dtype=np.float32))
    i32 = lambda v: gpu.from_numpy(np.asarray(v, dtype=np.int32))
    op = c["op"]
    if op == "matmul": return (f32(c["a"]) @ f32(c["b"])).to_numpy()
    if op == "softmax": return gpu.softmax(f32(c["x"])).to_numpy()
    if op == "softmax_causal": return gpu.softmax_causal(f32(c["x"])).to_numpy()
    if op == "layer_norm": return gpu.layer_norm(f32(c["x"]), f32(c["gamma"]), f32(c["beta"]), c["eps"]).to_numpy()
    if op == "gelu": return gpu.gelu(f32(c["x"])).to_numpy()
    if op == "embedding": return gpu.embedding(f32(c["w"]), i32(c["idx"])).to_numpy()
    if op == "add_bias": return gpu.add_bias(f32(c["x"]), f32(c["bias"])).to_numpy()
    if op == "argmax": return gpu.argmax(f32(c["x"])).to_numpy()
    if op == "gather": return gpu.gather(f32(c["x"]), c["dim"], i32(c["idx"])).to_numpy()
    if op == "index_select": return gpu.index_select(f32(c["x"]), c["dim"], i32(c["idx"])).to_numpy()
    raise AssertionError(op)


@pytest.mark.parametrize("case", CASES, ids=[f'{c["op"]}@{c["src"].split(" ")[0]}' for c in CASES])
def test_reference_known_answers_on_gpu(gpu_dev, case):
    got = run_gpu_case(gpu_dev, case)
    exp = np.asarray(case["expect"])
    assert got.shape == exp.shape
    if case["tol"] == 0:
        assert np.array_equal(got.astype(np.float64), exp.astype(np.float64))
    else:
        assert np.max(np.abs(got.astype(np.float64) - exp)) <= case["tol"]


# ── element-wise ────────────────────────────────────────────────────────────
@pytest.mark.parametrize("n", [1, 3, 4, 1023, 4096, 100003])
@pytest.mark.parametrize("op", ["add", "sub", "mul", "div"])
def test_binary_f32(gpu_dev, op, n):
    rng = np.random.default_rng(n)
    a = rng.standard_normal(n).astype(np.float32); b = (rng.standard_normal(n).astype(np.float32) + 3.0)
    got = getattr(gpu_dev, op)(gpu_dev.from_numpy(a), gpu_dev.from_numpy(b)).to_numpy()
    assert np.array_equal(got, R.binary(a, b, op))   # one IEEE op per element: exact


def test_binary_broadcast_and_int(gpu_dev):
    rng = np.random.default_rng(0)
    a = rng.standard_normal((4, 1, 6)).astype(np.float32); b = rng.standard_normal((5, 6)).astype(np.float32)
    assert np.array_equal((gpu_dev.from_numpy(a) + gpu_dev.from_numpy(b)).to_numpy(), a + b)
    s = np.float32(2.5).reshape(1)
    assert np.array_equal((gpu_dev.from_numpy(a) * gpu_dev.from_numpy(s)).to_numpy(), a * s)
    ia = rng.integers(-50, 50, (7, 9)).astype(np.int32); ib = rng.integers(1, 9, (9,)).astype(np.int32)
    assert np.array_equal((gpu_dev.from_numpy(ia) + gpu_dev.from_numpy(ib)).to_numpy(), ia + ib)
    assert np.array_equal((gpu_dev.from_numpy(ia) * gpu_dev.from_numpy(ib)).to_numpy(), ia * ib)
    l = rng.integers(-2**40, 2**40, (5,)).astype(np.int64)
    assert np.array_equal((gpu_dev.from_numpy(l) - gpu_dev.from_numpy(l[::-1].copy())).to_numpy(), l - l[::-1])


@pytest.mark.parametrize("shape", [(5,), (3, 7), (8192, 32), (2, 3, 5, 7)])
def test_gelu_and_gelu_exact_f32(gpu_dev, shape):
    rng = np.random.default_rng(1)
    x = (rng.standard_normal(shape) * 3).astype(np.float32)
    close(gpu_dev.gelu(gpu_dev.from_numpy(x)).to_numpy(), R.gelu(x), rel=1e-5, abs_=1e-6)
    # the library evaluates erf with erff, the oracle with the reference's 7.1.26 polynomial
    # (max error 1.5e-7): the reference's own bar for this op is atol 1e-5 (test_gelu_exact.py:7-15)
    assert np.max(np.abs(gpu_dev.gelu_exact(gpu_dev.from_numpy(x)).to_numpy() - R.gelu_exact(x))) <= 1e-5


def test_gelu_has_no_nan_at_large_inputs(gpu_dev):
    x = np.array([20, -20, 50, -50, 1e4, -1e4], np.float32)       # ops.rs:3452-3469
    y = gpu_dev.gelu(gpu_dev.from_numpy(x)).to_numpy()
    # the library keeps the tiny negative tail (x * e^{2u} / (e^{2u} + 1)) that float32 tanh rounds to -0
    assert np.all(np.isfinite(y)) and np.allclose(y, R.gelu(x), rtol=1e-6, atol=1e-4)


def test_unary_ops_f32(gpu_dev):
    rng = np.random.default_rng(2)
    x = rng.standard_normal(1000).astype(np.float32)
    g = gpu_dev.from_numpy(x)
    assert np.array_equal(gpu_dev.neg(g).to_numpy(), -x)
    assert np.array_equal(gpu_dev.relu(g).to_numpy(), np.maximum(x, 0))
    assert np.array_equal(gpu_dev.abs(g).to_numpy(), np.abs(x))
    assert np.array_equal(gpu_dev.sign(g).to_numpy(), np.sign(x))
    close(gpu_dev.exp(g).to_numpy(), np.exp(x), rel=2e-6)
    close(gpu_dev.tanh(g).to_numpy(), np.tanh(x), rel=2e-6, abs_=1e-7)
    close(gpu_dev.sigmoid(g).to_numpy(), 1 / (1 + np.exp(-x.astype(np.float64))), rel=2e-6)
    close(gpu_dev.sqrt(gpu_dev.abs(g)).to_numpy(), np.sqrt(np.abs(x)), rel=1e-6)
    close(gpu_dev.scalar_mul(g, 0.125).to_numpy(), R.scalar_mul(x, 0.125), rel=0, abs_=0)


def test_fused_chains_execute_like_the_unfused_ops(gpu_dev):
    # fusion_integration.rs:6-104: add->relu, sqrt->neg->relu, add->gelu
    a = np.array([1.0, -2.0, 3.0, -4.0], np.float32); b = np.array([0.5, 0.5, 0.5, 0.5], np.float32)
    ga, gb = gpu_dev.from_numpy(a), gpu_dev.from_numpy(b)
    y = (ga + gb).relu()
    assert y.plan().startswith("fused_")
    assert y.to_list() == [1.5, 0.0, 3.5, 0.0]
    s = gpu_dev.from_numpy(np.array([1.0, 4.0, 9.0], np.float32))
    assert (-(s.sqrt())).relu().to_list() == [0.0, 0.0, 0.0]
    close(gpu_dev.gelu(ga + gb).to_numpy(), R.gelu(a + b), rel=1e-5)
    rng = np.random.default_rng(3)
    x = rng.standard_normal((33, 65)).astype(np.float32); r = rng.standard_normal((65,)).astype(np.float32)
    z = ((gpu_dev.from_numpy(x) * gpu_dev.from_numpy(r)) - gpu_dev.from_numpy(x)).tanh().exp()
    assert z.plan().count("\n") == 1
    close(z.to_numpy(), np.exp(np.tanh(x * r - x)), rel=3e-6)


@pytest.mark.parametrize("shape,bias_n", [((8192, 3072), 3072), ((7, 5), 5), ((2, 3, 2), 3), ((1, 2, 2, 2), 2), ((64, 772), 772)])
def test_add_bias_f32_exact(gpu_dev, shape, bias_n):
    rng = np.random.default_rng(4)
    x = rng.standard_normal(shape).astype(np.float32); b = rng.standard_normal(bias_n).astype(np.float32)
    assert np.array_equal(gpu_dev.add_bias(gpu_dev.from_numpy(x), gpu_dev.from_numpy(b)).to_numpy(), R.add_bias(x, b))


def test_add_bias_then_gelu_is_one_kernel(gpu_dev):
    rng = np.random.default_rng(21)
    x = rng.standard_normal((64, 3072)).astype(np.float32); b = rng.standard_normal(3072).astype(np.float32)
    y = gpu_dev.gelu(gpu_dev.add_bias(gpu_dev.from_numpy(x), gpu_dev.from_numpy(b)))
    assert y.plan().strip() == "add_bias[gelu]_f32 [64, 3072]"
    close(y.to_numpy(), R.gelu(R.add_bias(x, b)), rel=1e-5, abs_=1e-6)


# ── reductions ──────────────────────────────────────────────────────────────
@pytest.mark.parametrize("rows,cols", [(8192, 768), (3, 4), (5, 1), (17, 1280), (9, 1001), (2, 5120), (4, 20000), (1, 50257)])
def test_layer_norm_f32(gpu_dev, rows, cols):
    rng = np.random.default_rng(rows + cols)
    x = (rng.standard_normal((rows, cols)) * 2 + 0.5).astype(np.float32)
    g = rng.standard_normal(cols).astype(np.float32); b = rng.standard_normal(cols).astype(np.float32)
    got = gpu_dev.layer_norm(gpu_dev.from_numpy(x), gpu_dev.from_numpy(g), gpu_dev.from_numpy(b), 1e-5).to_numpy()
    # summation order differs from the serial reference loop; the bar is 1e-5 relative to each ROW's own scale
    # (max |ref| of that row, floored at 1), not to the largest value of the whole tensor
    ref = R.layer_norm(x, g, b, 1e-5)
    row_scale = np.maximum(1.0, np.max(np.abs(ref), axis=-1, keepdims=True))
    assert np.all(np.abs(got - ref) <= 1e-5 * row_scale)


def test_layer_norm_3d_and_eps(gpu_dev):
    rng = np.random.default_rng(5)
    x = rng.standard_normal((4, 6, 64)).astype(np.float32)
    g = np.ones(64, np.float32); b = np.zeros(64, np.float32)
    got = gpu_dev.layer_norm(gpu_dev.from_numpy(x), gpu_dev.from_numpy(g), gpu_dev.from_numpy(b), 1e-12).to_numpy()
    assert got.shape == (4, 6, 64)
    close(got, R.layer_norm(x, g, b, 1e-12), rel=1e-5, abs_=1e-5)


@pytest.mark.parametrize("shape", [(96, 128, 128), (3, 3), (2, 5, 7), (4, 1024), (2, 3, 1000), (2, 7, 3000), (1, 50257), (5, 2, 9, 16)])
def test_softmax_f32(gpu_dev, shape):
    rng = np.random.default_rng(6)
    x = (rng.standard_normal(shape) * 3).astype(np.float32)
    got = gpu_dev.softmax(gpu_dev.from_numpy(x)).to_numpy()
    x64 = x.astype(np.float64)
    e = np.exp(x64 - x64.max(-1, keepdims=True))
    exact = e / e.sum(-1, keepdims=True)
    assert np.max(np.abs(got - exact) / exact.max(-1, keepdims=True)) <= 1e-5         # the 1e-5 relative bar, against float64
    # the oracle sums each row serially in float32 like the reference kernel, so it carries up to
    # ~cols * 6e-8 of rounding itself; allow for that when comparing with it
    ref = R.softmax(x)
    assert np.max(np.abs(got - ref) / ref.max(-1, keepdims=True)) <= 1e-5 + shape[-1] * 6e-8
    np.testing.assert_allclose(got.sum(-1), 1.0, rtol=1e-5)


@pytest.mark.parametrize("shape", [(96, 128, 128), (3, 3), (2, 5, 7), (2, 7, 5), (3, 40, 1000), (2, 2100, 2100), (1, 1, 4)])
def test_softmax_causal_f32(gpu_dev, shape):
    rng = np.random.default_rng(7)
    x = (rng.standard_normal(shape) * 2).astype(np.float32)
    got = gpu_dev.softmax_causal(gpu_dev.from_numpy(x)).to_numpy()
    ref = R.softmax_causal(x)
    assert np.all(np.triu(got, 1) == 0)                      # explicit zeros right of the diagonal
    assert np.max(np.abs(got - ref)) <= 1e-5


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("rows,cols", [(4735, 768), (4736, 768), (4801, 256), (5000, 1000), (4737, 1024), (6001, 1280), (4800, 1288), (4736, 248),
                                       (16575, 768), (16576, 768), (16600, 256), (16577, 640), (9471, 512), (9473, 264), (23679, 1024), (23681, 904)])
def test_layer_norm_rows_by_bulk_copies(gpu_dev, dtype, rows, cols):
    """Both sides of the rule (32, 64, 112 or 160 rows an SM of 512 to 2560 bytes), every number of pieces a lane, a last piece that not every lane has."""
    import torch
    t = {"bfloat16": torch.bfloat16, "float16": torch.float16}[dtype]
    g = torch.Generator("cuda").manual_seed(rows + cols)
    x = (torch.randn((rows, cols), generator=g, device="cuda") * 3 + 5).to(t)
    gain, shift = torch.randn(cols, generator=g, device="cuda").to(t), torch.randn(cols, generator=g, device="cuda").to(t)
    got = torch.from_numpy(gpu_dev.layer_norm(gpu_dev.from_torch(x), gpu_dev.from_torch(gain), gpu_dev.from_torch(shift), 1e-5).to_numpy().astype(np.float32)).cuda().double()
    ref = torch.nn.functional.layer_norm(x.double(), (cols,), gain.double(), shift.double(), 1e-5)
    # one rounding to the type, half a step (2^-9 of the value in bfloat16, 2^-12 in float16), and float32 sums; where terms cancel, of their size
    assert torch.all((got - ref).abs() <= (2.0 ** -8 if dtype == "bfloat16" else 2.0 ** -11) * (ref.abs() + 2.0 ** -8 * (ref - shift.double()).abs()) + 1e-5)


@pytest.mark.parametrize("dtype", ["bfloat16", "float16", "float32"])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("shape", [(40, 128, 128), (19, 256, 256), (5, 1000, 1016), (6, 800, 1024), (3, 64, 2048), (2, 16, 4096), (3, 33, 8), (47, 256, 256), (93, 128, 128), (54, 764, 1020)])
def test_softmax_rows_in_registers_and_by_bulk_copies(gpu_dev, dtype, causal, shape):
    """Row lengths and counts on both sides of the rules, ragged diagonals, scores far from zero, -inf and the type's lowest value."""
    import torch
    t = {"bfloat16": torch.bfloat16, "float16": torch.float16, "float32": torch.float32}[dtype]
    g = torch.Generator("cuda").manual_seed(sum(shape))
    x = torch.randn(shape, generator=g, device="cuda") * 4
    x[0] += 300.0
    x[1, :, 3] = float("-inf")
    x = x.to(t)
    x[1, :, 5] = torch.finfo(t).min
    got = torch.from_numpy((gpu_dev.softmax_causal if causal else gpu_dev.softmax)(gpu_dev.from_torch(x)).to_numpy().astype(np.float32)).cuda().double()
    ref = x.double()
    if causal:
        ref = ref.masked_fill(torch.ones(shape[1:], dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    ref = torch.softmax(ref, -1)
    # 16 bits: the exponential and the result are rounded to the type (half a step each: 2^-8 of the value in bfloat16), float16 also at its
    # fixed step of 2^-24 for each; float32: exp2 within 2 ulp of an argument of up to 60 that is rounded once, 60 * 2^-24 * ln 2
    rel, tiny = {"bfloat16": (2.0 ** -7, 1e-37), "float16": (2.0 ** -10, 2.0 ** -23), "float32": (1e-5, 1e-37)}[dtype]
    assert torch.all((got - ref).abs() <= rel * ref + tiny)
    if causal:
        assert torch.all(got[ref == 0] == 0)


def test_rows_by_bulk_copies_are_whole_behind_a_failed_wait(gpu_dev):
    """A code that another kernel's wait left in the pipeline status word does not end the waits for rows: every row is written, and the
    code is still there to be read."""
    import torch
    from applegpu_runtime_b200 import _lib
    g = torch.Generator("cuda").manual_seed(11)
    x = torch.randn((40000, 768), generator=g, device="cuda").to(torch.bfloat16)
    s = torch.randn((24, 1024, 1024), generator=g, device="cuda").to(torch.bfloat16)
    gain, shift = torch.ones(768, device="cuda").to(torch.bfloat16), torch.zeros(768, device="cuda").to(torch.bfloat16)
    x, s, gain, shift = (gpu_dev.from_torch(t) for t in (x, s, gain, shift))
    want = [gpu_dev.layer_norm(x, gain, shift, 1e-5).to_numpy(), gpu_dev.softmax_causal(s).to_numpy()]
    assert gpu_dev.pipeline_status() == 0
    assert _lib.load().applegpu_test_wait_runs_out(77, 1000) == 0
    got = [gpu_dev.layer_norm(x, gain, shift, 1e-5).eval(), gpu_dev.softmax_causal(s).eval()]
    assert gpu_dev.pipeline_status() == 77
    for a, b in zip(got, want):
        assert np.array_equal(a.to_numpy().view(np.uint8), b.view(np.uint8))


def test_softmax_causal_all_masked_floor(gpu_dev):
    # the running max starts at -1e9 (kernel_templates.rs:478): values below it underflow to 0/0
    x = np.full((1, 2, 2), -2e9, np.float32); x[0, 1, 1] = 0.0
    got = gpu_dev.softmax_causal(gpu_dev.from_numpy(x)).to_numpy()
    ref = R.softmax_causal(x)
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    assert got[0, 1, 1] == 1.0 and got[0, 0, 1] == 0.0


@pytest.mark.parametrize("rows,cols", [(8, 50257), (3, 5), (1, 1), (300, 17), (2, 100000)])
def test_argmax_exact(gpu_dev, rows, cols):
    rng = np.random.default_rng(8)
    x = rng.standard_normal((rows, cols)).astype(np.float32)
    x[0, : min(cols, 3)] = x[0].max() + 1.0                   # a tie at the front: lowest index wins
    got = gpu_dev.argmax(gpu_dev.from_numpy(x)).to_numpy()
    assert got.dtype == np.int32 and np.array_equal(got, R.argmax(x))


def test_argmax_nan_rules(gpu_dev):
    x = np.array([[1.0, np.nan, 3.0, 2.0], [np.nan, 5.0, 1.0, 0.0], [-np.inf, -np.inf, -np.inf, -np.inf]], np.float32)
    got = gpu_dev.argmax(gpu_dev.from_numpy(x)).to_numpy()
    assert np.array_equal(got, R.argmax(x)) and got.tolist() == [2, 0, 0]


def test_sum_and_mean_last_dim(gpu_dev):
    rng = np.random.default_rng(9)
    x = rng.standard_normal((13, 257)).astype(np.float32)
    close(gpu_dev.sum(gpu_dev.from_numpy(x)).to_numpy(), x.astype(np.float64).sum(-1), rel=1e-5, abs_=1e-4)
    close(gpu_dev.mean(gpu_dev.from_numpy(x)).to_numpy(), x.astype(np.float64).mean(-1), rel=1e-5, abs_=1e-6)


# ── gather family (bit-exact) ───────────────────────────────────────────────
@pytest.mark.parametrize("dtype", ["float32", "float16"])
@pytest.mark.parametrize("vocab,dim,idx_shape", [(50257, 768, (1024,)), (5, 3, (3,)), (30522, 768, (4, 16)), (11, 7, (2, 3, 2)), (100, 1280, (0,))])
def test_embedding_exact(gpu_dev, dtype, vocab, dim, idx_shape):
    rng = np.random.default_rng(10)
    w = rng.standard_normal((vocab, dim)).astype(dtype)
    idx = rng.integers(0, vocab, idx_shape).astype(np.int32)
    got = gpu_dev.embedding(gpu_dev.from_numpy(w), gpu_dev.from_numpy(idx)).to_numpy()
    assert got.shape == idx_shape + (dim,)
    assert np.array_equal(got, R.embedding(w, idx))


def test_gather_and_index_select_exact(gpu_dev):
    rng = np.random.default_rng(11)
    x = rng.standard_normal((37, 53)).astype(np.float32)
    i0 = rng.integers(0, 37, (20, 53)).astype(np.int32); i1 = rng.integers(0, 53, (37, 9)).astype(np.int32)
    gx = gpu_dev.from_numpy(x)
    assert np.array_equal(gpu_dev.gather(gx, 0, gpu_dev.from_numpy(i0)).to_numpy(), R.gather(x, 0, i0))
    assert np.array_equal(gpu_dev.gather(gx, 1, gpu_dev.from_numpy(i1)).to_numpy(), R.gather(x, 1, i1))
    s0 = rng.integers(0, 37, (11,)).astype(np.int32); s1 = rng.integers(0, 53, (70,)).astype(np.int32)
    assert np.array_equal(gpu_dev.index_select(gx, 0, gpu_dev.from_numpy(s0)).to_numpy(), R.index_select(x, 0, s0))
    assert np.array_equal(gpu_dev.index_select(gx, 1, gpu_dev.from_numpy(s1)).to_numpy(), R.index_select(x, 1, s1))
    ii = rng.integers(-1000, 1000, (8, 6)).astype(np.int32)   # integer payloads go through the same kernel
    assert np.array_equal(gpu_dev.index_select(gpu_dev.from_numpy(ii), 0, gpu_dev.from_numpy(np.array([7, 0, 7], np.int32))).to_numpy(), ii[[7, 0, 7]])


# ── quantize / dequantize / cast (bit-exact) ────────────────────────────────
@pytest.mark.parametrize("n", [1, 15, 16, 17, 4099, 1 << 20])
@pytest.mark.parametrize("target,scale,zp", [("int8", 0.1, 0), ("int8", 0.037, -5), ("uint8", 0.05, 128), ("uint8", 1.0, 0)])
def test_quantize_bit_exact(gpu_dev, n, target, scale, zp):
    rng = np.random.default_rng(n)
    x = (rng.standard_normal(n) * 4).astype(np.float32)
    x[: min(n, 4)] = np.array([0.05, -0.05, 0.15, 1e6], np.float32)[: min(n, 4)] * np.float32(scale / 0.1)  # exact .5 ties and saturation
    got = gpu_dev.quantize(gpu_dev.from_numpy(x), target, scale=scale, zero_point=zp).to_numpy()
    assert np.array_equal(got, R.quantize(x, target, scale, zp))


def test_quantize_from_half_types_and_dequantize(gpu_dev):
    rng = np.random.default_rng(12)
    x = (rng.standard_normal(5000) * 3).astype(np.float16)
    assert np.array_equal(gpu_dev.quantize(gpu_dev.from_numpy(x), "int8", scale=0.05).to_numpy(), R.quantize(x, "int8", 0.05))
    xb = bf16_bits(rng.standard_normal(5000) * 3)
    gb = gpu_dev.from_bytes(xb.tobytes(), [5000], "bfloat16")
    assert np.array_equal(gpu_dev.quantize(gb, "uint8", scale=0.07, zero_point=100).to_numpy(), R.quantize(xb, "uint8", 0.07, 100, st=2))
    q = rng.integers(-128, 128, 4099).astype(np.int8)
    for dt in ("float32", "float16"):
        assert np.array_equal(gpu_dev.dequantize(gpu_dev.from_numpy(q), dt, scale=0.03, zero_point=7).to_numpy(), R.dequantize(q, dt, 0.03, 7))
    qu = rng.integers(0, 256, 333).astype(np.uint8)
    got = gpu_dev.dequantize(gpu_dev.from_numpy(qu), "bfloat16", scale=0.5, zero_point=128)
    assert np.array_equal(np.frombuffer(got.to_bytes(), np.uint16), R.dequantize(qu, "bfloat16", 0.5, 128))


def test_quantize_dequantize_round_trip_property(gpu_dev):
    # size-independent property at a large size: |dequant(quant(x)) - x| <= scale/2 inside the clamp range
    rng = np.random.default_rng(13)
    x = rng.uniform(-12, 12, 1 << 22).astype(np.float32)
    g = gpu_dev.from_numpy(x)
    y = gpu_dev.dequantize(gpu_dev.quantize(g, "int8", scale=0.1), "float32", scale=0.1).to_numpy()
    assert np.max(np.abs(y - x)) <= 0.05 + 1e-5


def test_per_channel_weight_quantisation_exact(gpu_dev):
    rng = np.random.default_rng(14)
    w = (rng.standard_normal((37, 129)) * 0.02).astype(np.float32); w[5] = 0
    q, s = gpu_dev.quantize_weight(gpu_dev.from_numpy(w))
    rq, rs = R.quantize_rows(w)
    assert np.array_equal(q.to_numpy(), rq) and np.array_equal(s.to_numpy(), rs)


def test_cast_matrix(gpu_dev):
    rng = np.random.default_rng(15)
    x = (rng.standard_normal(1000) * 50).astype(np.float32)
    g = gpu_dev.from_numpy(x)
    assert np.array_equal(gpu_dev.cast(g, "float16").to_numpy(), x.astype(np.float16))
    assert np.array_equal(gpu_dev.cast(g, "int32").to_numpy(), x.astype(np.int32))
    assert np.array_equal(np.frombuffer(gpu_dev.cast(g, "bfloat16").to_bytes(), np.uint16), R.to_bf16(x))
    i64 = rng.integers(0, 50257, 777).astype(np.int64)
    assert np.array_equal(gpu_dev.cast(gpu_dev.from_numpy(i64), "int32").to_numpy(), i64.astype(np.int32))   # the int64->int32 index cast of applegpu_backend.cpp:901-903
    assert np.array_equal(gpu_dev.cast(g, "bool").to_numpy(), x != 0)
    # int8 -> 16-bit floats (the widening of int8 weights before a tensor-core GEMM): every value, vector and scalar tails
    for n in (256 * 40, 16 * 3, 1000):
        q = np.resize(np.arange(-128, 128, dtype=np.int8), n)
        gq = gpu_dev.from_numpy(q)
        assert np.array_equal(gpu_dev.cast(gq, "float16").to_numpy(), q.astype(np.float16))
        assert np.array_equal(np.frombuffer(gpu_dev.cast(gq, "bfloat16").to_bytes(), np.uint16), R.to_bf16(q.astype(np.float32)))


# ── layout ops ──────────────────────────────────────────────────────────────
@pytest.mark.parametrize("dtype", ["float32", "bfloat16", "int32", "int8"])
def test_concat_is_bit_exact_on_every_axis_and_layout(gpu_dev, dtype):
    """Both halves of a concat are copied by one launch; the halves may allow different vector widths
    (odd extents, strided views), and either may be a view."""
    rng = np.random.default_rng(23)
    def make(shape):
        if dtype == "bfloat16":
            bits = R.to_bf16(rng.standard_normal(shape).astype(np.float32))
            return bits, gpu_dev.from_bytes(bits.tobytes(), list(shape), "bfloat16")
        x = (rng.standard_normal(shape) * 50).astype({"float32": np.float32, "int32": np.int32, "int8": np.int8}[dtype])
        return x, gpu_dev.from_numpy(x)
    def host(t):
        return np.frombuffer(t.to_bytes(), np.uint16).reshape(t.shape) if dtype == "bfloat16" else t.to_numpy()
    for shape_a, shape_b, dim in [((4, 6, 8), (4, 6, 8), 0), ((4, 6, 8), (4, 3, 8), 1), ((4, 6, 8), (4, 6, 5), 2), ((3, 5, 7), (3, 5, 1), 2),
                                  ((2, 3, 4, 16), (2, 3, 1, 16), 2), ((1, 64), (7, 64), 0), ((5, 1), (5, 9), 1)]:
        a, ga = make(shape_a); b, gb = make(shape_b)
        assert np.array_equal(host(gpu_dev.concat(ga, gb, dim=dim)), np.concatenate([a, b], dim)), (shape_a, shape_b, dim)
    # the decode KV append: cache [B, h, T, d] and a new entry that is a transposed view of [B, 1, h, d]
    cache, gc = make((2, 3, 5, 16)); new, gn = make((2, 1, 3, 16))
    got = gpu_dev.concat(gc, gpu_dev.transpose_dims(gn, 1, 2), dim=2)
    assert np.array_equal(host(got), np.concatenate([cache, new.transpose(0, 2, 1, 3)], 2))
    # both operands strided
    x, gx = make((6, 10)); y, gy = make((4, 10))
    got = gpu_dev.concat(gpu_dev.transpose(gx), gpu_dev.transpose(gy), dim=1)
    assert np.array_equal(host(got), np.concatenate([x.T, y.T], 1))


def test_views_and_copies_match_numpy(gpu_dev):
    rng = np.random.default_rng(16)
    x = rng.standard_normal((6, 10, 8)).astype(np.float32)
    g = gpu_dev.from_numpy(x)
    assert np.array_equal(gpu_dev.transpose(g).to_numpy(), x.transpose(0, 2, 1))
    assert np.array_equal(gpu_dev.transpose_dims(g, 0, 2).to_numpy(), x.transpose(2, 1, 0))
    assert np.array_equal(gpu_dev.slice(g, 1, 3, 7).to_numpy(), x[:, 3:7])
    assert np.array_equal(gpu_dev.slice(g, 2, 1, 2).to_numpy(), x[:, :, 1:2])
    assert np.array_equal(gpu_dev.reshape(gpu_dev.transpose_dims(g, 0, 1), [10, 48]).to_numpy(), x.transpose(1, 0, 2).reshape(10, 48))
    assert np.array_equal(gpu_dev.concat(g, g, dim=1).to_numpy(), np.concatenate([x, x], 1))
    assert np.array_equal(gpu_dev.concat(gpu_dev.slice(g, 0, 0, 2), gpu_dev.transpose_dims(gpu_dev.transpose_dims(g, 0, 1), 0, 1), dim=0).to_numpy(), np.concatenate([x[:2], x], 0))
    # a strided view feeding an element-wise op and a reduction
    v = gpu_dev.transpose_dims(g, 0, 1)
    assert np.array_equal((v + v).to_numpy(), 2 * x.transpose(1, 0, 2))
    assert np.max(np.abs(gpu_dev.softmax(v).to_numpy() - R.softmax(np.ascontiguousarray(x.transpose(1, 0, 2))))) < 1e-6
    h = gpu_dev.from_numpy(x.astype(np.float16))
    assert np.array_equal(gpu_dev.transpose(h).to_numpy(), x.astype(np.float16).transpose(0, 2, 1))


def test_empty_tensors(gpu_dev):
    e = gpu_dev.from_numpy(np.zeros((0, 4), np.float32))
    assert (e + e).to_numpy().shape == (0, 4)
    assert gpu_dev.gelu(e).to_numpy().shape == (0, 4)
    w = gpu_dev.from_numpy(np.zeros((4, 3), np.float32))
    assert (e @ w).to_numpy().shape == (0, 3)
    g = gpu_dev.from_numpy(np.ones(4, np.float32))
    assert gpu_dev.layer_norm(e, g, g).to_numpy().shape == (0, 4)


# ── half types against the oracle in the same storage type ──────────────────
def test_bf16_and_f16_bandwidth_ops(gpu_dev):
    rng = np.random.default_rng(17)
    x = (rng.standard_normal((64, 768)) * 2).astype(np.float32)
    g = rng.standard_normal(768).astype(np.float32); b = rng.standard_normal(768).astype(np.float32)
    xb, gb, bb = bf16_bits(x), bf16_bits(g), bf16_bits(b)
    got = gpu_dev.layer_norm(up_bf16(gpu_dev, x), up_bf16(gpu_dev, g), up_bf16(gpu_dev, b), 1e-5).to_numpy()
    ref = R.from_bf16(R.layer_norm(xb, gb, bb, 1e-5, st=2))
    assert np.max(np.abs(got - ref)) <= 2e-2 * np.max(np.abs(ref))          # bf16 bar of the north star
    assert np.mean(got == ref) > 0.98                                          # and nearly always the same bf16 value
    got = gpu_dev.softmax_causal(up_bf16(gpu_dev, x[:, :64].reshape(1, 64, 64))).to_numpy()
    ref = R.from_bf16(R.softmax_causal(bf16_bits(x[:, :64].reshape(1, 64, 64)), st=2))
    assert np.max(np.abs(got - ref)) <= 2e-2 and np.all(np.triu(got[0], 1) == 0)
    # gelu: the oracle evaluates x * 0.5 * (1 + tanh(u)) like the reference kernel, which loses
    # digits by cancellation for x < -3 (1 + tanh(u) ~ 1e-4); the library evaluates the same function
    # as x * e^{2u} / (e^{2u} + 1). The two agree to the storage precision except in that tail, where
    # values are ~1e-4 and differ by at most one unit in the last place.
    got = gpu_dev.gelu(up_bf16(gpu_dev, x)).to_numpy()
    ref = R.from_bf16(R.gelu(xb, st=2))
    assert np.mean(got == ref) > 0.97 and np.max(np.abs(got - ref)) <= 2e-2 * np.max(np.abs(ref))
    assert np.max(np.abs(got - ref) / np.maximum(np.abs(ref), 1e-3)) <= 2 ** -7   # <= 1 bf16 ulp where |y| > 1e-3
    xh = x.astype(np.float16)
    goth = gpu_dev.gelu(gpu_dev.from_numpy(xh)).to_numpy().astype(np.float32)
    refh = R.gelu(xh).astype(np.float32)
    assert np.mean(goth == refh) > 0.97 and np.max(np.abs(goth - refh) / np.maximum(np.abs(refh), 1e-3)) <= 2 ** -9
    got = gpu_dev.add_bias(up_bf16(gpu_dev, x), up_bf16(gpu_dev, g)).to_numpy()
    assert np.array_equal(got, R.from_bf16(R.add_bias(xb, gb, st=2)))


@pytest.mark.parametrize("rows,cols", [(3, 8191), (3, 8192), (1, 50257), (8, 32768), (148, 8200), (149, 8200)])
def test_argmax_of_long_rows(gpu_dev, rows, cols):
    """Both sides of the sizes at which a row takes a larger block: the lowest index among equals, NaNs never, a NaN in front always."""
    rng = np.random.default_rng(rows + cols)
    x = rng.integers(-50, 50, (rows, cols)).astype(np.float32)
    x[0, cols - 1] = 60
    want = x.argmax(-1)
    if rows > 2:
        x[1, 7] = x[1, want[1] + 1 if want[1] + 1 < cols else 3] = np.nan
        want[1] = np.nanargmax(x[1])
        x[2, 0] = np.nan
        want[2] = 0
    assert np.array_equal(gpu_dev.argmax(gpu_dev.from_numpy(x)).to_numpy().reshape(-1), want)
