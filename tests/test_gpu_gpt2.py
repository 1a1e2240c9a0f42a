"""GPT-2 forward and greedy decode against the golden fixture produced by the reference's CPU
path (tests/golden/gpt2_tiny.npz) and against the torch oracle at a larger random-init config.
Bars: fp32 logits atol 1e-3 and identical argmax (python/tests/test_cpp_backend.py:311-371),
greedy tokens identical; bf16 logits within 2e-2 relative of fp32."""
import os

import numpy as np
import pytest
import torch

from oracle import torch_ref

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def _fixture():
    z = np.load(os.path.join(HERE, "golden", "gpt2_tiny.npz"))
    c = z["config"].tolist()
    cfg = dict(n_layer=c[0], n_head=c[1], n_embd=c[2], vocab_size=c[3], n_positions=c[4])
    weights = {k[2:]: z[k] for k in z.files if k.startswith("w:")}
    return cfg, weights, z


def test_tiny_gpt2_logits_match_reference_cpu_path(gpu_dev):
    cfg, weights, z = _fixture()
    model = gpu_dev.load_gpt2_state_dict(weights, cfg)
    logits, kv = gpu_dev.gpt2_forward(model, z["ids"])
    got = logits.to_numpy()
    assert got.shape == z["logits"].shape
    np.testing.assert_allclose(got, z["logits"], atol=1e-3)
    assert np.array_equal(got.argmax(-1), z["logits"].argmax(-1))
    assert np.max(np.abs(got - z["logits"])) < 5e-5
    # list input = the reference's unbatched form
    l1, _ = gpu_dev.gpt2_forward(model, z["ids"][0].tolist())
    np.testing.assert_allclose(l1.to_numpy(), z["logits"][0], atol=1e-3)


def test_tiny_gpt2_greedy_tokens_identical_with_and_without_cache(gpu_dev):
    cfg, weights, z = _fixture()
    model = gpu_dev.load_gpt2_state_dict(weights, cfg)
    with_cache = gpu_dev.greedy_generate(model, z["ids"], max_tokens=6, use_cache=True)
    without = gpu_dev.greedy_generate(model, z["ids"], max_tokens=6, use_cache=False)
    assert with_cache.tolist() == z["greedy"].tolist()
    assert without.tolist() == z["greedy"].tolist()
    one = gpu_dev.generate(model, z["ids"][1].tolist(), max_tokens=6, temperature=0)
    assert one == z["greedy"][1].tolist()


def test_unfused_and_fused_forward_agree(gpu_dev):
    cfg, weights, z = _fixture()
    model = gpu_dev.load_gpt2_state_dict(weights, cfg)
    fused = gpu_dev.gpt2_forward(model, z["ids"])[0].to_numpy()
    gpu_dev.set_fusion(True, False)
    try:
        plain = gpu_dev.gpt2_forward(model, z["ids"])[0].to_numpy()
    finally:
        gpu_dev.set_fusion(True, True)
    np.testing.assert_allclose(fused, plain, atol=2e-5)


CFG_MID = dict(n_layer=3, n_head=4, n_embd=256, vocab_size=1003, n_positions=160)


def test_mid_gpt2_fp32_and_bf16_against_torch_oracle(gpu_dev):
    w = torch_ref.init_gpt2_weights(CFG_MID, seed=3)
    rng = np.random.default_rng(3)
    ids = rng.integers(0, CFG_MID["vocab_size"], (3, 160))
    with torch.no_grad():
        ref = torch_ref.gpt2_forward(w, CFG_MID, torch.from_numpy(ids))[0].numpy()
    m32 = gpu_dev.init_gpt2_weights(CFG_MID, seed=3, dtype="float32")       # same generator, same order
    got32 = gpu_dev.gpt2_forward(m32, ids)[0].to_numpy()
    np.testing.assert_allclose(got32, ref, atol=1e-3)
    assert np.mean(got32.argmax(-1) == ref.argmax(-1)) == 1.0
    m16 = gpu_dev.init_gpt2_weights(CFG_MID, seed=3, dtype="bfloat16")
    logits16 = gpu_dev.gpt2_forward(m16, ids)[0]
    plan16 = logits16.plan()
    assert plan16.count("fused_attention[causal,merge_heads]_bf16") == CFG_MID["n_layer"]   # the single-kernel tcgen05 attention
    assert plan16.count("fused_linear[") == 4 * CFG_MID["n_layer"] and "_f32" not in plan16
    x16 = gpu_dev.from_bytes(bytes(2 * 128 * 256), [128, 256], "bfloat16")
    assert gpu_dev.matmul_path(x16, m16["weights"]["transformer.h.0.attn.c_attn.weight"]) == "tcgen05"
    got16 = logits16.to_numpy()
    scale = float(np.max(np.abs(ref)))
    assert np.max(np.abs(got16 - ref)) <= 2e-2 * scale                      # bf16 bar: 2e-2 relative of fp32
    assert gpu_dev.pipeline_status() == 0


def test_mid_gpt2_greedy_decode_identical_to_torch_fp32(gpu_dev):
    w = torch_ref.init_gpt2_weights(CFG_MID, seed=4)
    rng = np.random.default_rng(4)
    ids = rng.integers(0, CFG_MID["vocab_size"], (4, 12))
    with torch.no_grad():
        ref = torch_ref.gpt2_greedy(w, CFG_MID, torch.from_numpy(ids), max_tokens=20).numpy()
    m32 = gpu_dev.init_gpt2_weights(CFG_MID, seed=4, dtype="float32")
    got = gpu_dev.greedy_generate(m32, ids, max_tokens=20, use_cache=True)
    assert got.tolist() == ref.tolist()


def test_gpt2_int8_weights_bf16_activations_against_dequantised_oracle(gpu_dev):
    """The int8 configuration: every linear weight quantised per output channel (symmetric int8, fp32
    scales), activations bf16. Oracle: the torch forward in fp32 on the dequantised weights."""
    from oracle import msl_ref as R
    w = torch_ref.init_gpt2_weights(CFG_MID, seed=8)
    wq = dict(w)
    for name, t in w.items():
        if name.endswith((".c_attn.weight", ".c_fc.weight", ".c_proj.weight")):
            q, s = R.quantize_rows(np.ascontiguousarray(t.numpy().T))            # [out, in] rows
            wq[name] = torch.from_numpy((q.astype(np.float32) * s[:, None]).T.copy())
    rng = np.random.default_rng(8)
    ids = rng.integers(0, CFG_MID["vocab_size"], (2, 96))
    with torch.no_grad():
        ref = torch_ref.gpt2_forward(wq, CFG_MID, torch.from_numpy(ids))[0].numpy()
    m = gpu_dev.quantize_gpt2_linears(gpu_dev.init_gpt2_weights(CFG_MID, seed=8, dtype="bfloat16"))
    logits = gpu_dev.gpt2_forward(m, ids)[0]
    plan = logits.plan()
    assert plan.count("fused_linear[int8,") == 4 * CFG_MID["n_layer"]
    got = logits.to_numpy()
    scale = float(np.max(np.abs(ref)))
    # weights were quantised from their bf16-rounded values on the device and from fp32 in the oracle:
    # the two int8 tensors differ in a few entries by one step, inside the bf16 bar
    assert np.max(np.abs(got - ref)) <= 2e-2 * scale
    assert gpu_dev.pipeline_status() == 0


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("batch,heads,vocab", [(1, 1, 33), (8, 2, 97), (9, 12, 1000), (16, 3, 64), (5, 16, 130), (8, 18, 4097), (3, 20, 257),
                                                (8, 12, 500), (1, 12, 70), (3, 5, 100), (8, 9, 90), (7, 11, 129), (1, 10, 300), (9, 20, 130), (16, 20, 4097)])
def test_decoder_picks_the_largest_logit(gpu_dev, dtype, batch, heads, vocab):
    """QKV and attention in one launch (up to eight sequences, nine to twelve heads: five and six shares of K, the last whole or half) and
    apart, the head at vocabularies that end inside a warp's sixteen rows and a block's 64 (with nine sequences and more that kernel takes the
    models whose layers have 64 MB and more: twenty heads): every pick has the largest logit of the float32
    oracle on the same weights, to rounding."""
    from applegpu_runtime_b200.generate import Gpt2Decoder
    cfg = {"n_layer": 2, "n_head": heads, "n_embd": 64 * heads, "vocab_size": vocab, "n_positions": 64}
    m = gpu_dev.init_gpt2_weights(cfg, seed=heads + vocab, dtype=dtype, std=0.08)
    w = {k: torch.from_numpy(np.asarray(t.to_numpy()).astype(np.float32)) for k, t in m["weights"].items() if not k.startswith("__")}
    ids = np.random.default_rng(vocab).integers(0, vocab, (batch, 7))
    logits, kv = gpu_dev.gpt2_forward(m, ids, last_only=True)
    first = gpu_dev.argmax(logits)
    dec = Gpt2Decoder(m, batch, 40)
    dec.prefill(kv, first, 7)
    rest = np.asarray(dec.steps(6))
    seq = np.concatenate([ids, first.to_numpy().reshape(-1, 1), rest.T], 1)
    with torch.no_grad():
        ref = torch_ref.gpt2_forward(w, cfg, torch.from_numpy(seq))[0].numpy()
    # two layers of a dozen roundings to 2^-9 each, of either sign: sqrt(24) 2^-9 = 0.01 of a logit's scale for the pick and as much for the
    # largest; a pick from a wrong row is at 1
    for i in range(7):
        row = ref[:, 6 + i]
        assert np.all(row.max(-1) - row[np.arange(batch), seq[:, 7 + i]] <= 2e-2 * np.abs(row).max())


@pytest.mark.parametrize("batch,heads,per_layer", [(1, 1, 5), (8, 4, 5), (1, 8, 5), (8, 8, 5), (1, 9, 4), (8, 12, 4), (9, 12, 5), (1, 13, 5), (8, 16, 5)])
def test_decoder_takes_qkv_and_attention_in_one_launch_where_it_is_faster(gpu_dev, batch, heads, per_layer):
    from applegpu_runtime_b200.generate import Gpt2Decoder
    launches = []
    for layers in (1, 3):
        cfg = {"n_layer": layers, "n_head": heads, "n_embd": 64 * heads, "vocab_size": 64, "n_positions": 32}
        m = gpu_dev.init_gpt2_weights(cfg, seed=1, dtype="bfloat16", std=0.05)
        logits, kv = gpu_dev.gpt2_forward(m, np.zeros((batch, 3), np.int64), last_only=True)
        dec = Gpt2Decoder(m, batch, 16)
        dec.prefill(kv, gpu_dev.argmax(logits), 3)
        dec.steps(2)
        launches.append(dec.launches_per_step)
    assert launches[1] - launches[0] == 2 * per_layer


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_graph_decoder_matches_the_concat_cache_engine(gpu_dev, dtype):
    """The static-shape decoder (preallocated KV cache appended in place, one captured step replayed per token) against
    the engine that keeps the cache the reference's way (concatenation per step): same greedy tokens, whether the step
    is replayed from the graph or issued launch by launch; a second generation reuses nothing stale."""
    m = gpu_dev.init_gpt2_weights(CFG_MID, seed=12, dtype=dtype)
    rng = np.random.default_rng(12)
    ids = rng.integers(0, CFG_MID["vocab_size"], (5, 9))
    tape = gpu_dev.greedy_generate(m, ids, max_tokens=24, use_cache=True, engine="tape")
    graph = gpu_dev.greedy_generate(m, ids, max_tokens=24, use_cache=True, engine="graph")
    stats = dict(m["_last_decoder_stats"])
    direct = gpu_dev.greedy_generate(m, ids, max_tokens=24, use_cache=True, engine="direct")
    assert graph.shape == (5, 33)
    assert stats["graph"] is True and stats["launches_per_step"] <= 7 * CFG_MID["n_layer"] + 8
    # the layers of a step as one cooperative kernel with grid-wide barriers: the per-op kernels' arithmetic in their order
    persistent = gpu_dev.greedy_generate(m, ids, max_tokens=24, use_cache=True, engine="persistent")
    assert m["_last_decoder_stats"]["launches_per_step"] <= 8    # barrier reset + layers kernel, ln_f, LM head, pick, bookkeeping
    assert graph.tolist() == persistent.tolist()
    if dtype == "float32":
        assert graph.tolist() == tape.tolist() == direct.tolist()
        with torch.no_grad():
            w = torch_ref.init_gpt2_weights(CFG_MID, seed=12)
            ref = torch_ref.gpt2_greedy(w, CFG_MID, torch.from_numpy(ids), max_tokens=24).numpy()
        assert graph.tolist() == ref.tolist()                    # identical to the fp32 oracle
    else:
        assert graph.tolist() == direct.tolist()                 # same kernels, same order: bit-identical
        # the tape engine sums attention in another order (tensor-core kernel vs the decode kernel): tokens may part at a bf16 near-tie
        agree = np.mean(graph == tape)
        assert agree >= 0.9, agree
    ids2 = rng.integers(0, CFG_MID["vocab_size"], (2, 17))
    again = gpu_dev.greedy_generate(m, ids2, max_tokens=8, use_cache=True, engine="graph")
    assert again.tolist() == gpu_dev.greedy_generate(m, ids2, max_tokens=8, use_cache=True, engine="direct").tolist()
    assert gpu_dev.pipeline_status() == 0


def test_taped_decode_steps_give_the_same_tokens_and_logits(gpu_dev):
    m = gpu_dev.init_gpt2_weights(CFG_MID, seed=9, dtype="bfloat16")
    ids = np.random.default_rng(9).integers(0, CFG_MID["vocab_size"], (3, 10))
    a = gpu_dev.greedy_generate(m, ids, max_tokens=12, use_cache=True, compiled=False, engine="tape")
    b = gpu_dev.greedy_generate(m, ids, max_tokens=12, use_cache=True, compiled=True, engine="tape")
    assert a.tolist() == b.tolist()
    # prefill through a tape: recorded on the first call, replayed on the second
    l0 = gpu_dev.gpt2_forward(m, ids)[0].to_numpy()
    l1 = gpu_dev.gpt2_forward(m, ids, compiled=True)[0].to_numpy()
    l2 = gpu_dev.gpt2_forward(m, ids[::-1].copy(), compiled=True)[0].to_numpy()
    assert np.array_equal(l0, l1) and np.array_equal(l0[::-1], l2)
    n0 = gpu_dev.tensor_count()
    for _ in range(3):
        gpu_dev.gpt2_forward(m, ids, compiled=True)[0].eval()
    gpu_dev.synchronize()
    assert gpu_dev.tensor_count() <= n0 + 4          # replayed intermediates do not pile up


def test_kv_cache_decode_is_not_slower_than_recomputing(gpu_dev):
    """The reference's benchmark-as-test (python/tests/test_gpt2.py:106-123): generating with the KV cache
    must take at most 1.5x the time of recomputing the whole prefix every step."""
    import time
    m = gpu_dev.init_gpt2_weights(CFG_MID, seed=10, dtype="bfloat16")
    ids = np.random.default_rng(10).integers(0, CFG_MID["vocab_size"], (2, 128))
    gpu_dev.greedy_generate(m, ids, max_tokens=3, use_cache=True)       # warm both paths (pool, tensor maps, tape)
    gpu_dev.greedy_generate(m, ids, max_tokens=3, use_cache=False)
    t0 = time.perf_counter(); a = gpu_dev.greedy_generate(m, ids, max_tokens=12, use_cache=True); t_cached = time.perf_counter() - t0
    t0 = time.perf_counter(); b = gpu_dev.greedy_generate(m, ids, max_tokens=12, use_cache=False); t_full = time.perf_counter() - t0
    assert a.shape == b.shape == (2, 140)
    assert t_cached <= 1.5 * t_full, (t_cached, t_full)


def test_mlp_config_fp32(gpu_dev):
    # the first benchmark configuration: Linear(64,128) -> ReLU -> Linear(128,10), batch 32, default nn.Linear init, seed 0
    torch.manual_seed(0)
    l1 = torch.nn.Linear(64, 128); l2 = torch.nn.Linear(128, 10)
    x = torch.randn(32, 64)
    with torch.no_grad():
        ref = torch_ref.mlp_forward(x, l1.weight, l1.bias, l2.weight, l2.bias).numpy()
    g = gpu_dev
    gx = g.from_torch(x)
    w1 = g.transpose(g.from_torch(l1.weight)); w2 = g.transpose(g.from_torch(l2.weight))   # views; nn.Linear stores [out, in]
    y = g.add_bias(g.relu(g.add_bias(gx @ w1, g.from_torch(l1.bias))) @ w2, g.from_torch(l2.bias))
    assert "fused_linear[bias,relu,]" in y.plan()
    np.testing.assert_allclose(y.to_numpy(), ref, atol=1e-5, rtol=1e-5)


def test_layer_norm_folded_into_the_linears_matches_the_layer_norm_kernels(gpu_dev):
    """16-bit prefill with ln_1 / ln_2 folded into c_attn / c_fc (row statistics from the producing GEMM's epilogue,
    correction in the consuming GEMM's epilogue) against the same model with every layer_norm a kernel, and against the
    float32 oracle; gains and shifts are random so the folding itself is exercised, and further forwards (direct, taped,
    replayed) must reproduce the first bit for bit: the row statistics are accumulated in fixed point with integer
    atomics, whose result does not depend on the order of addition."""
    rng = np.random.default_rng(11)
    w = {k: v.numpy() for k, v in torch_ref.init_gpt2_weights(CFG_MID, seed=11).items()}
    for k in w:
        if ".ln_" in k and k.endswith(".weight"):
            w[k] = (1.0 + 0.3 * rng.standard_normal(w[k].shape)).astype(np.float32)
        elif k.endswith(".bias") and w[k].ndim == 1:
            w[k] = (0.1 * rng.standard_normal(w[k].shape)).astype(np.float32)
    ids = rng.integers(0, CFG_MID["vocab_size"], (4, 160))
    with torch.no_grad():
        ref = torch_ref.gpt2_forward({k: torch.from_numpy(v) for k, v in w.items()}, CFG_MID, torch.from_numpy(ids))[0].numpy()
    scale = float(np.max(np.abs(ref)))
    for dtype in ("bfloat16", "float16"):
        plain = gpu_dev.load_gpt2_state_dict(w, CFG_MID, dtype=dtype, fold_layer_norms=False)
        folded = gpu_dev.load_gpt2_state_dict(w, CFG_MID, dtype=dtype)
        assert "ln_fold" in folded and "ln_fold" not in plain
        out = gpu_dev.gpt2_forward(folded, ids)[0]
        plan = out.plan()
        assert plan.count("layer_norm_in") == 2 * CFG_MID["n_layer"] - 1 and plan.count("row_stats") == 2 * CFG_MID["n_layer"] - 1, plan
        assert sum(1 for line in plan.splitlines() if line.strip().startswith("layer_norm")) == 2, plan     # block 0's ln_1 and ln_f
        got = out.to_numpy()
        base = gpu_dev.gpt2_forward(plain, ids)[0].to_numpy()
        tol = 2e-2 if dtype == "bfloat16" else 4e-3
        assert float(np.max(np.abs(got - ref))) <= tol * scale, (dtype, float(np.max(np.abs(got - ref))) / scale)
        assert float(np.max(np.abs(got - base))) <= tol * scale, (dtype, float(np.max(np.abs(got - base))) / scale)
        # not worse than the kernel form against the oracle by more than a rounding step
        assert float(np.max(np.abs(got - ref))) <= 1.5 * float(np.max(np.abs(base - ref))) + 1e-3 * scale
        again = gpu_dev.gpt2_forward(folded, ids)[0].to_numpy()
        taped = gpu_dev.gpt2_forward(folded, ids, compiled=True)[0].to_numpy()
        replayed = gpu_dev.gpt2_forward(folded, ids, compiled=True)[0].to_numpy()
        for other in (again, taped, replayed):
            assert np.array_equal(other, got), (dtype, float(np.max(np.abs(other - got))) / scale)
    assert gpu_dev.pipeline_status() == 0


@pytest.mark.parametrize("heads,batch,dtype", [(5, 3, "float16"), (5, 16, "bfloat16"), (21, 9, "bfloat16"), (21, 2, "float16"), (5, 9, "float32"), (21, 16, "float32")])
def test_decode_linears_at_the_edges_of_their_shares(gpu_dev, heads, batch, dtype):
    """Widths of 5 x 64 (a last slab of 64 rows, three shares) and 21 x 64 (two and six slabs in a share, rows beyond 1024 for the
    statistics), one and two groups of eight rows: the step replayed, issued launch by launch and as one persistent kernel adds in the
    same order, so tokens are equal; the engine that keeps its cache by concatenation sums in another (and float32 rows beyond 1024
    take their layer_norm in a launch of its own there)."""
    cfg = {"n_layer": 2, "n_head": heads, "n_embd": 64 * heads, "vocab_size": 300, "n_positions": 320}
    m = gpu_dev.init_gpt2_weights(cfg, seed=heads + batch, dtype=dtype)
    ids = np.random.default_rng(batch).integers(0, 300, (batch, 250))
    out = {e: gpu_dev.greedy_generate(m, ids, max_tokens=16, use_cache=True, engine=e) for e in ("graph", "direct", "persistent", "tape")}
    assert out["graph"].tolist() == out["direct"].tolist() == out["persistent"].tolist()
    new = out["graph"][:, 250:]
    assert np.array_equal(new, out["tape"][:, 250:]) if dtype == "float32" else np.mean(new == out["tape"][:, 250:]) >= 0.85
    assert gpu_dev.pipeline_status() == 0


# ── a step's keys and values, number by number ──────────────────────────────
_MANTISSA = {"float32": 24, "float16": 11, "bfloat16": 8}


def _stored(x, dtype):
    """float64 rounded to the storage type."""
    import torch
    return torch.from_numpy(np.asarray(x, np.float64)).to(getattr(torch, dtype)).double().numpy()


def _step_state(heads, layers, seed, dtype, std=0.06):
    rng, d = np.random.default_rng(seed), 64 * heads
    n = lambda *shape: rng.standard_normal(shape) * std  # noqa: E731
    w = {"wte.weight": rng.standard_normal((300, d)) * 0.5, "wpe.weight": rng.standard_normal((320, d)) * 0.2, "ln_f.weight": np.ones(d), "ln_f.bias": np.zeros(d)}
    for i in range(layers):
        for name, k, o in (("attn.c_attn", d, 3 * d), ("attn.c_proj", d, d), ("mlp.c_fc", d, 4 * d), ("mlp.c_proj", 4 * d, d)):
            w[f"h.{i}.{name}.weight"], w[f"h.{i}.{name}.bias"] = n(k, o), n(o) * 5
        for name in ("ln_1", "ln_2"):
            w[f"h.{i}.{name}.weight"], w[f"h.{i}.{name}.bias"] = 1 + 0.3 * rng.standard_normal(d), 0.3 * rng.standard_normal(d)
    return {k: _stored(v, dtype) for k, v in w.items()}, {"n_layer": layers, "n_head": heads, "n_embd": d, "vocab_size": 300, "n_positions": 320}


def _decoded(g, state, cfg, dtype, ids, steps, engine):
    """Decoder behind the prompt `ids` after `steps` steps, the tokens the steps consumed [steps, batch]."""
    from applegpu_runtime_b200.generate import Gpt2Decoder
    m = g.load_gpt2_state_dict({"transformer." + k: v.astype(np.float32) for k, v in state.items()}, cfg, dtype, fold_layer_norms=False)
    logits, kv = g.gpt2_forward(m, ids, last_only=True)
    first = g.argmax(logits)
    dec = Gpt2Decoder(m, ids.shape[0], ids.shape[1] + steps)
    dec.set_engine(persistent=engine == "persistent")
    dec.prefill(kv, first, ids.shape[1])
    out = dec.steps(steps, use_graph=engine != "direct")
    return dec, np.concatenate([first.to_numpy().reshape(1, -1), out[:-1]])


def _norm64(x, w, b):
    c = x - x.mean(-1, keepdims=True)
    with np.errstate(all="ignore"):
        return c / np.sqrt((c * c).mean(-1, keepdims=True) + 1e-5) * w + b


def _assert_linear(got, r, w, b, dtype):
    """got = r @ w + b rounded once: half a unit in its last place, beside what float32 arithmetic leaves open: 2^-22 for each normalised
    value (four operations of 2^-24), and sums that each lose up to 2^-23 of the terms before them, over at most 128 of K in one chain."""
    want, terms = r @ w + b, np.abs(r) @ np.abs(w) + np.abs(b)
    ulp = 2.0 ** np.maximum(np.floor(np.log2(np.maximum(np.abs(want), 1e-30))) + 1 - _MANTISSA[dtype], -24 if dtype == "float16" else -140)
    assert np.all(np.abs(got - want) <= 0.5 * ulp + 2e-6 * terms), np.max((np.abs(got - want) - 0.5 * ulp) / terms)


@pytest.mark.parametrize("heads,batch,dtype", [(5, 1, "float16"), (5, 8, "bfloat16"), (21, 9, "float16"), (21, 16, "bfloat16"), (5, 16, "float32"), (21, 3, "float32"), (12, 8, "bfloat16")])
@pytest.mark.parametrize("engine", ["graph", "persistent"])
def test_decode_step_against_float64(gpu_dev, heads, batch, dtype, engine):
    """The keys and values a step leaves. The first layer's are one linear behind layer_norm: exact up to its rounding, at ragged shares
    of K (320 and 1344 columns), one and two groups of eight rows. The second layer's come through every kernel of a layer, with
    attention over 300 rows (more than are asked for ahead in any type) and roundings to the storage type where the step rounds. Half a
    storage unit of their norm: rounding them leaves 1 / sqrt(12) of a unit at most (0.2 on average over a binade), and upstream only the
    roundings differ that float32 sums in another order turn."""
    state, cfg = _step_state(heads, 2, 7 * heads + batch, dtype)
    d, T = cfg["n_embd"], 300
    ids = np.random.default_rng(batch).integers(0, 300, (batch, T))
    dec, toks = _decoded(gpu_dev, state, cfg, dtype, ids, 3, engine)
    (k0, v0), (k1, v1) = [[t.to_numpy().astype(np.float64) for t in dec.cache(i)] for i in range(2)]
    merged = lambda c, t: c[:, :, t].reshape(batch, d)  # noqa: E731
    w = lambda n: state["h.0." + n]  # noqa: E731
    for t in range(3):
        x = _stored(state["wte.weight"][toks[t]] + state["wpe.weight"][T + t], dtype)
        r = _norm64(x, w("ln_1.weight"), w("ln_1.bias"))
        _assert_linear(np.concatenate([merged(k0, T + t), merged(v0, T + t)], axis=1), r, w("attn.c_attn.weight")[:, d:], w("attn.c_attn.bias")[d:], dtype)
        q = _stored(r @ w("attn.c_attn.weight")[:, :d] + w("attn.c_attn.bias")[:d], dtype).reshape(batch, heads, 1, 64)
        s = (q @ k0[:, :, :T + t + 1].transpose(0, 1, 3, 2)) / 8
        p = np.exp(s - s.max(-1, keepdims=True))
        att = _stored((p @ v0[:, :, :T + t + 1] / p.sum(-1, keepdims=True)).reshape(batch, d), dtype)
        x = _stored(att @ w("attn.c_proj.weight") + w("attn.c_proj.bias") + x, dtype)
        h = _norm64(x, w("ln_2.weight"), w("ln_2.bias")) @ w("mlp.c_fc.weight") + w("mlp.c_fc.bias")
        h = _stored(0.5 * h * (1 + np.tanh(0.7978845608 * (h + 0.044715 * h ** 3))), dtype)
        x = _stored(h @ w("mlp.c_proj.weight") + w("mlp.c_proj.bias") + x, dtype)
        r = _norm64(x, state["h.1.ln_1.weight"], state["h.1.ln_1.bias"])
        want = r @ state["h.1.attn.c_attn.weight"][:, d:] + state["h.1.attn.c_attn.bias"][d:]
        got = np.concatenate([merged(k1, T + t), merged(v1, T + t)], axis=1)
        assert np.linalg.norm(got - want) <= (0.5 * 2.0 ** (1 - _MANTISSA[dtype]) + 2e-6) * np.linalg.norm(want)
    assert gpu_dev.pipeline_status() == 0


@pytest.mark.parametrize("gamma,std", [(1e-5, 2000.0), (3e-4, 300.0), (1.0, 0.5), (3e4, 2e-5)])
@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("heads,batch", [(5, 3), (17, 16)])
def test_decode_linear_keeps_normalised_values_in_32_bits(gpu_dev, heads, batch, dtype, gamma, std):
    """Rows whose normalised values are tiny or (one column) beyond the storage type, next to ordinary ones."""
    state, cfg = _step_state(heads, 1, heads, dtype)
    state["wte.weight"][:, 3] = 40.0
    d, rng = cfg["n_embd"], np.random.default_rng(heads)
    state["h.0.ln_1.weight"] = _stored(gamma * rng.uniform(0.5, 2.0, d) * np.where(np.arange(d) % 7 == 0, 1e-2, 1.0), dtype)
    state["h.0.ln_1.bias"] = _stored(gamma * 0.1 * rng.standard_normal(d), dtype)
    state["h.0.attn.c_attn.weight"] = _stored(std * rng.standard_normal((d, 3 * d)), dtype)
    dec, toks = _decoded(gpu_dev, state, cfg, dtype, rng.integers(0, 300, (batch, 5)), 1, "direct")
    got = np.concatenate([t.to_numpy()[:, :, 5].reshape(batch, d) for t in dec.cache(0)], axis=1).astype(np.float64)
    x = _stored(state["wte.weight"][toks[0]] + state["wpe.weight"][5], dtype)
    _assert_linear(got, _norm64(x, state["h.0.ln_1.weight"], state["h.0.ln_1.bias"]), state["h.0.attn.c_attn.weight"][:, d:], state["h.0.attn.c_attn.bias"][d:], dtype)


@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("where", ["gamma", "beta", "weight", "nan"])
def test_decode_linear_keeps_infinities_and_nans(gpu_dev, dtype, where):
    state, cfg = _step_state(5, 1, 3, dtype)
    d, rng = cfg["n_embd"], np.random.default_rng(3)
    if where in ("gamma", "beta"):
        state["h.0.ln_1." + {"gamma": "weight", "beta": "bias"}[where]][77] = np.inf
    else:
        state["h.0.attn.c_attn.weight"][[5, 200], [d + 3, d + 90]] = np.nan if where == "nan" else np.inf
    dec, toks = _decoded(gpu_dev, state, cfg, dtype, rng.integers(0, 300, (3, 5)), 1, "direct")
    got = np.concatenate([t.to_numpy()[:, :, 5].reshape(3, d) for t in dec.cache(0)], axis=1).astype(np.float64)
    x = _stored(state["wte.weight"][toks[0]] + state["wpe.weight"][5], dtype)
    with np.errstate(all="ignore"):
        want = _norm64(x, state["h.0.ln_1.weight"], state["h.0.ln_1.bias"]) @ state["h.0.attn.c_attn.weight"][:, d:] + state["h.0.attn.c_attn.bias"][d:]
    assert np.array_equal(np.isnan(got), np.isnan(want))
    inf = np.isinf(want)
    assert inf.any() == (where != "nan") and np.array_equal(np.isinf(got), inf) and np.array_equal(got[inf], want[inf])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_persistent_decode_refuses_rows_beyond_its_statistics(gpu_dev, dtype):
    """Its layer_norm keeps 2048 columns of a row: 32 heads give the step engine's tokens, 33 are refused and leave the step engine usable."""
    from applegpu_runtime_b200.generate import Gpt2Decoder
    for heads in (32, 33):
        m = gpu_dev.init_gpt2_weights({"n_layer": 1, "n_head": heads, "n_embd": 64 * heads, "vocab_size": 300, "n_positions": 32}, seed=heads, dtype=dtype)
        ids = np.random.default_rng(heads).integers(0, 300, (2, 9))
        want = gpu_dev.greedy_generate(m, ids, max_tokens=8, engine="graph")
        if heads == 32:
            assert np.array_equal(gpu_dev.greedy_generate(m, ids, max_tokens=8, engine="persistent"), want)
            continue
        logits, kv = gpu_dev.gpt2_forward(m, ids, last_only=True)
        dec = Gpt2Decoder(m, 2, 17)
        dec.set_engine(persistent=True)
        dec.prefill(kv, gpu_dev.argmax(logits), 9)
        for graph in (True, False):
            with pytest.raises(ValueError, match="2048 columns"):
                dec.steps(7, use_graph=graph)
        dec.set_engine(persistent=False)
        assert np.array_equal(dec.steps(7), want[:, 10:].T)
    assert gpu_dev.pipeline_status() == 0
