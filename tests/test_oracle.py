"""The oracle against (a) flash_attn's own torch code paths (committed fixtures, the pinned
part), (b) independent time-domain definitions of the Hyena operator, (c) itself across its
execution modes (parallel / prefill+step), (d) its regression fixture."""
import os

import numpy as np
import pytest
import torch

from oracle import stripedhyena_oracle as O


@pytest.fixture(scope="module")
def att(golden_dir):
    return np.load(os.path.join(golden_dir, "attention_flash_attn.npz"))


@pytest.mark.parametrize("name,scaling", [("s1", 1.0), ("s16", 16.0)])
def test_rotary_tables_match_flash_attn(att, name, scaling):
    L, d = att["qkv"].shape[1], att["qkv"].shape[-1]
    cos, sin = O.rotary_tables(L, d, scaling_factor=scaling, dtype=torch.float32)
    np.testing.assert_array_equal(cos.numpy(), att[f"cos_{name}"])
    np.testing.assert_array_equal(sin.numpy(), att[f"sin_{name}"])


@pytest.mark.parametrize("name", ["s1", "s16"])
def test_rotary_and_attention_match_flash_attn(att, name):
    qkv = torch.from_numpy(att["qkv"])
    cos, sin = torch.from_numpy(att[f"cos_{name}"]), torch.from_numpy(att[f"sin_{name}"])
    q = O.apply_rotary(qkv[:, :, 0], cos, sin)
    k = O.apply_rotary(qkv[:, :, 1], cos, sin)
    np.testing.assert_allclose(q.numpy(), att[f"q_{name}"], rtol=0, atol=2e-6)
    np.testing.assert_allclose(k.numpy(), att[f"k_{name}"], rtol=0, atol=2e-6)
    ctx = O.causal_attention(q, k, qkv[:, :, 2])
    # SelfAttention masks with -10000 instead of -inf (mha.py:271): same to fp32 precision
    np.testing.assert_allclose(ctx.numpy(), att[f"ctx_{name}"], rtol=0, atol=3e-6)


def _filter_params(D=64, S=8, seed=0):
    cfg = O.tiny_config(num_layers=1, attn_layer_idxs=(), hidden_size=D, num_heads=1)
    sd = O.random_state_dict(cfg, seed=seed)
    return cfg, sd


@pytest.mark.parametrize("L", [1, 2, 17, 64, 257])
def test_fft_conv_equals_modal_recurrence(L):
    """engine.parallel_iir's FFT long conv == the recurrence that defines the filter."""
    D = 128
    cfg = O.tiny_config(num_layers=1, attn_layer_idxs=(), hidden_size=D, num_heads=1)
    sd = O.random_state_dict(cfg, seed=3)
    p, r = sd["blocks.0.filter.poles"].double(), sd["blocks.0.filter.residues"].double()
    torch.manual_seed(L)
    z_pre = torch.randn(2, 3 * D, L, dtype=torch.float64)
    Dk = torch.randn(D, dtype=torch.float64)
    h = O.hyena_filter(p, r, L)
    y, state = O.iir_parallel(z_pre, h, Dk, p, 1, D, want_state=True)
    x2, x1, v = O.column_split(z_pre, 1, D)
    conv, st = O.long_conv_direct(x1 * v, p, r)
    y_ref = ((conv + (x1 * v) * Dk[:, None]) * x2).permute(0, 2, 1)
    assert (y - y_ref).abs().max() < 1e-9
    assert (state - st).abs().max() < 1e-9     # prefill_via_modal_fft == recurrence state


def test_filter_is_sum_of_pole_powers():
    cfg, sd = _filter_params()
    p, r = sd["blocks.0.filter.poles"].double(), sd["blocks.0.filter.residues"].double()
    h = O.hyena_filter(p, r, 33)[0]
    pc, rc = torch.view_as_complex(p)[..., 0], torch.view_as_complex(r)[..., 0]
    for t in (0, 1, 5, 32):
        assert (h[:, t] - (rc * pc ** t).real.sum(-1)).abs().max() < 1e-12


def test_column_split_mapping():
    """x2 <- z[(c//hd)*3hd + c%hd], x1 <- +hd, v <- +2hd."""
    H, hd = 3, 4
    z = torch.arange(3 * H * hd, dtype=torch.float32)[None, :, None].repeat(1, 1, 2)
    x2, x1, v = O.column_split(z, H, hd)
    for c in range(H * hd):
        base = (c // hd) * 3 * hd + c % hd
        assert x2[0, c, 0] == base and x1[0, c, 0] == base + hd and v[0, c, 0] == base + 2 * hd


def test_fir_step_equals_parallel():
    cfg, sd = _filter_params(D=32)
    w, b = sd["blocks.0.filter.short_filter_weight"].double(), sd["blocks.0.filter.short_filter_bias"].double()
    torch.manual_seed(0)
    u = torch.randn(2, 9, 96, dtype=torch.float64)
    z, fir_state = O.fir_parallel(u[:, :8], w, b)
    y, fs2 = O.fir_step(u[:, 8], fir_state.clone(), w, b)
    zfull, _ = O.fir_parallel(u, w, b)
    assert (y - zfull[..., 8]).abs().max() < 1e-12
    assert torch.equal(fs2, u.permute(0, 2, 1)[..., -2:])


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-9), (torch.float32, 2e-3)])
def test_stateful_equals_stateless(dtype, tol):
    cfg = O.tiny_config(num_layers=3, attn_layer_idxs=(1,), hidden_size=256, num_heads=2)
    sd = O.random_state_dict(cfg, seed=5)
    m = O.OracleStripedHyena(cfg, sd, dtype)
    torch.manual_seed(0)
    ids = torch.randint(0, 256, (2, 29))
    full, _ = m(ids)
    d = m.initialize_inference_params()
    d["mha"].max_batch_size, d["mha"].max_seqlen = 2, 64
    pre, d = m(ids[:, :20], d)
    assert (pre - full[:, :20]).abs().max() < tol
    d["mha"].seqlen_offset = d["hyena"].seqlen_offset = 20
    for t in range(20, 29):
        lg, d = m(ids[:, t:t + 1], d)
        assert (lg[:, 0] - full[:, t]).abs().max() < tol
        d["mha"].seqlen_offset += 1
        d["hyena"].seqlen_offset += 1


def test_strict_state_dict():
    cfg = O.tiny_config(num_layers=2, attn_layer_idxs=(1,), hidden_size=256, num_heads=2)
    sd = O.random_state_dict(cfg)
    sd.pop("blocks.0.filter.D")
    with pytest.raises(RuntimeError):
        O.OracleStripedHyena(cfg, sd)


def test_evo_7b_shapes():
    cfg = O.evo_config("evo-1-131k-base")
    spec = O.state_dict_spec(cfg)
    assert O.mlp_inner_size(cfg) == 10928
    assert spec["blocks.0.filter.poles"] == (4096, 8, 1, 2)
    assert spec["blocks.8.inner_mha_cls.Wqkv.weight"] == (12288, 4096)
    n = sum(int(np.prod(s)) for k, s in spec.items() if k != "unembed.weight" and "inv_freq" not in k)
    assert abs(n - 6.45e9) < 0.03e9       # "7B" = 6.45 B parameters
    assert cfg["rotary_emb_scaling_factor"] == 16


def test_bf16_mode_close_to_truth():
    cfg = O.tiny_config(num_layers=3, attn_layer_idxs=(1,), hidden_size=256, num_heads=2)
    sd = O.random_state_dict(cfg, seed=11)
    ids = torch.randint(0, 4, (1, 64))
    a, _ = O.OracleStripedHyena(cfg, sd, torch.bfloat16)(ids)
    b, _ = O.OracleStripedHyena(cfg, sd, torch.float64)(ids)
    la, lb = torch.log_softmax(a.double(), -1), torch.log_softmax(b, -1)
    assert (la - lb).abs().mean() < 6e-2   # bf16 logits of magnitude ~10 carry ~2e-2 of rounding alone


def test_regression_fixture(golden_dir):
    g = np.load(os.path.join(golden_dir, "tiny_model_oracle.npz"))
    cfg = O.tiny_config(num_layers=3, attn_layer_idxs=(1,), hidden_size=256, num_heads=2)
    sd = O.random_state_dict(cfg, seed=7)
    m = O.OracleStripedHyena(cfg, sd, torch.float64)
    ids = torch.from_numpy(g["ids"])
    logits, _ = m(ids)
    np.testing.assert_allclose(logits.numpy(), g["logits"], atol=2e-5, rtol=0)
    d = m.initialize_inference_params()
    d["mha"].max_batch_size, d["mha"].max_seqlen = 2, 128
    m(ids[:, :40], d)
    np.testing.assert_allclose(d["hyena"].state_dict[0].real.numpy(), g["state0_re"], atol=1e-5)
    np.testing.assert_allclose(d["hyena"].fir_state_dict[0].float().numpy(), g["fir0"], atol=1e-6)


def test_sample_greedy_and_topk():
    torch.manual_seed(0)
    lg = torch.randn(5, 512)
    assert torch.equal(O.sample(lg, top_k=1), lg.argmax(-1))
    s = O.sample(lg.clone(), top_k=4, top_p=0.9, temperature=0.7)
    top4 = lg.topk(4, dim=-1).indices
    assert all(s[i] in top4[i] for i in range(5))


@pytest.fixture(scope="module")
def kvs(golden_dir):
    return np.load(os.path.join(golden_dir, "kvcache_sampling_flash_attn.npz"))


def test_cache_form_attention_matches_flash_attn(kvs):
    """Decode / continued-prefill attention: flash_attn's _update_kv_cache + CrossAttention(causal=True) (modules/mha.py:280-367,
    run on CPU for the fixture) vs the oracle's cache write (attention_block) and causal_attention(q, k, v, q_offset)."""
    steps = [tuple(int(v) for v in row) for row in kvs["steps"]]
    B, H, d = kvs["q_0"].shape[0], kvs["q_0"].shape[2], kvs["q_0"].shape[3]
    cache = torch.zeros(3, 16, 2, H, d)
    for n, (off, L) in enumerate(steps):
        q, kv = torch.from_numpy(kvs[f"q_{n}"]), torch.from_numpy(kvs[f"kv_{n}"])
        cache[:B, off:off + L, 0] = kv[:, :, 0]                  # the oracle's cache write (attention_block), statement for statement
        cache[:B, off:off + L, 1] = kv[:, :, 1]
        ctx = O.causal_attention(q, cache[:B, :off + L, 0], cache[:B, :off + L, 1], q_offset=off)
        np.testing.assert_allclose(ctx.numpy(), kvs[f"ctx_{n}"], rtol=0, atol=3e-6)
    np.testing.assert_array_equal(cache.numpy(), kvs["cache_final"])


def test_samplers_match_flash_attn_sample(kvs):
    """flash_attn.utils.generation.sample (the code stripedhyena/sample.py copies; run on CPU for the fixture) vs the oracle's
    sample and evo_b200's host sampler: the same picks for the same torch seed, over greedy / top-k / top-p / temperature /
    full-vocabulary settings on fp32 logits."""
    from evo_b200.stripedhyena.sample import sample as product_sample
    logits = torch.from_numpy(kvs["sample_logits"])
    for n, (k, p, t) in enumerate(kvs["sample_cases"]):
        for fn in (O.sample, product_sample):
            for seed in range(8):
                torch.manual_seed(1000 + seed)
                got = fn(logits.clone(), top_k=int(k), top_p=float(p), temperature=float(t))
                np.testing.assert_array_equal(got.numpy(), kvs[f"sample_picks_{n}"][seed], err_msg=f"{fn.__module__} case {n} seed {seed}")


def test_attention_block_matches_flash_attn_mha_forward(golden_dir, monkeypatch):
    """The oracle's attention_block -- Wqkv, `(three h d)` split, rotary at seqlen_offset, cache write, cache-form causal attention,
    out_proj -- against flash_attn's MHA.forward run on CPU (tests/golden/make_golden.py: mha_block_fixture; the Triton rotary call
    is the one patched statement).  Pre-norm and the MLP half of the block are stripedhyena's, not flash_attn's: they are switched
    to identities here so that attention_block(u) - u is exactly what MHA.forward returns."""
    g = np.load(os.path.join(golden_dir, "mha_flash_attn.npz"))
    cfg = O.tiny_config(num_layers=2, attn_layer_idxs=(1,), hidden_size=256, num_heads=2)
    cfg["max_seqlen"] = 32
    sd = {k: v.float() for k, v in O.random_state_dict(cfg, seed=1).items()}
    p = "blocks.1.inner_mha_cls."
    sd[p + "Wqkv.weight"], sd[p + "Wqkv.bias"] = torch.from_numpy(g["Wqkv_w"]), torch.from_numpy(g["Wqkv_b"])
    sd[p + "out_proj.weight"], sd[p + "out_proj.bias"] = torch.from_numpy(g["out_w"]), torch.from_numpy(g["out_b"])
    m = O.OracleStripedHyena(cfg, sd, torch.float32)
    monkeypatch.setattr(O, "rms_norm", lambda x, scale, eps: x)
    monkeypatch.setattr(m, "_mlp_res", lambda prefix, a: a)
    np.testing.assert_array_equal(O.rotary_tables(4, 128, dtype=torch.float32)[0].numpy(),
                                  torch.cos(torch.outer(torch.arange(4, dtype=torch.float32), torch.from_numpy(g["inv_freq"]))).numpy())
    x = torch.from_numpy(g["x"])
    np.testing.assert_allclose((m.attention_block(1, x) - x).numpy(), g["y_stateless"], rtol=0, atol=2e-5)
    ip = m.initialize_inference_params()["mha"]
    ip.max_batch_size = 2
    np.testing.assert_allclose((m.attention_block(1, x[:, :6], ip) - x[:, :6]).numpy(), g["y_prefill"], rtol=0, atol=2e-5)
    for t in (6, 7):
        ip.seqlen_offset = t
        np.testing.assert_allclose((m.attention_block(1, x[:, t:t + 1], ip) - x[:, t:t + 1]).numpy(), g[f"y_step{t}"], rtol=0, atol=2e-5)
    cache = ip.key_value_memory_dict[1]
    assert tuple(cache.shape) == tuple(g["cache"].shape)                    # (max_batch_size, max_seqlen, 2, H, head_dim): mha.py:344-353
    np.testing.assert_allclose(cache.numpy(), g["cache"], rtol=0, atol=2e-6)


# ------------------------------------------------------------------ the real stripedhyena package (absent here; see oracle/real_reference.py)
def _install_stand_in_package(monkeypatch):
    """A `stripedhyena` package with the real one's interface, made of evo_b200's parameter tree (checkpoint key names, strict
    loading, dtype policy) and the oracle's arithmetic: lets the bridge's plumbing run where the real package is absent."""
    import sys
    import types
    from evo_b200.stripedhyena import StripedHyena as Tree, dotdict

    class StandIn(Tree):
        def _oracle(self):
            return O.OracleStripedHyena(dict(self.config), dict(self.state_dict()), self.embedding_layer.weight.dtype)

        def forward(self, x, inference_params_dict=None, padding_mask=None):
            return self._oracle()(x, inference_params_dict)

        def initialize_inference_params(self):
            return self._oracle().initialize_inference_params()

    pkg, model, utils = types.ModuleType("stripedhyena"), types.ModuleType("stripedhyena.model"), types.ModuleType("stripedhyena.utils")
    pkg.__path__, pkg.__version__ = [], "stand-in"
    model.StripedHyena, utils.dotdict = StandIn, dotdict
    pkg.model, pkg.utils = model, utils
    for name, mod in (("stripedhyena", pkg), ("stripedhyena.model", model), ("stripedhyena.utils", utils)):
        monkeypatch.setitem(sys.modules, name, mod)


def test_real_reference_bridge_runs_against_a_stand_in_package(monkeypatch):
    from oracle import real_reference as RR
    if RR.available() is not None and RR.available() != "stand-in":
        pytest.skip("the real package is importable: the next test is the one that matters")
    _install_stand_in_package(monkeypatch)
    assert RR.available() == "stand-in"
    rep = RR.compare()
    assert rep["keys_real_minus_oracle"] == [] and rep["keys_oracle_minus_real"] == []
    for mode in ("fp32", "bf16"):
        r = rep[mode]
        assert r["state_keys_equal"] and r["scale"] > 1.0
        assert max(r["stateless"], r["prefill"], r["steps"], r["state"], r["fir_state"]) == 0.0     # same arithmetic on both sides: plumbing only
    # the bench's CPU leg: 7B-like depth in the memory of two blocks
    cfg = O.tiny_config(num_layers=5, attn_layer_idxs=(1, 3), hidden_size=256, num_heads=2)
    m = RR.build(cfg, None, torch.float32, share_blocks=True)
    assert m.blocks[0].projections.weight.data_ptr() == m.blocks[2].projections.weight.data_ptr() == m.blocks[4].projections.weight.data_ptr()
    assert m.blocks[1].inner_mha_cls.Wqkv.weight.data_ptr() == m.blocks[3].inner_mha_cls.Wqkv.weight.data_ptr()
    ids = torch.randint(0, 4, (1, 33)) * 3 + 65
    assert torch.isfinite(RR._run(m, ids).float()).all()


def test_oracle_against_the_real_stripedhyena_package():
    """The verify-first checklist against the published package.  Skipped wherever `import stripedhyena` fails -- which is everywhere this repo has been
    built or run so far; the oracle's "parity unpinned" label stands until this test has passed somewhere."""
    from oracle import real_reference as RR
    ver = RR.available()
    if ver is None or ver == "stand-in":
        pytest.skip("stripedhyena is not importable here (requirements.txt:1 of the reference pins 0.2.2; no index, no wheel): parity stays unpinned")
    for kw in ({}, {"extra": {"use_interpolated_rotary_pos_emb": True, "rotary_emb_scaling_factor": 16}}, {"num_layers": 4, "attn_layer_idxs": (1, 3), "seed": 11}):
        rep = RR.compare(**kw)
        assert rep["keys_real_minus_oracle"] == [] and rep["keys_oracle_minus_real"] == [], rep
        f, b = rep["fp32"], rep["bf16"]
        assert f["state_keys_equal"] and b["state_keys_equal"]
        for k in ("stateless", "prefill", "steps"):
            assert f[k] <= 2e-4 * f["scale"], (kw, k, f)           # fp32 graph vs fp32 graph: summation order only
            assert b[k] <= 0.05 * b["scale"], (kw, k, b)           # bf16 rounding points may differ by an ulp per op
        assert f["state"] <= 1e-4 * max(1.0, f["scale"]) and f["fir_state"] <= 1e-5 * max(1.0, f["scale"]), (kw, f)
