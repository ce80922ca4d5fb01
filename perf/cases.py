"""Cases that stand for the work this framework is used for, at the sizes its configurations, tests and benchmark name.

Kinds (each through an entry point that a program calls itself: the model object, or the C interface of include/evo_b200.h):
  hyena    the Hyena operator of one layer over whole sequences (evo_hyena_fwd): scoring, and prompts that leave or continue a state
  attention  causal attention of one layer over whole sequences, read in place from the fused projection (evo_attn_fwd_ws)
  mlp      the gated feed-forward of one layer (evo_gemm twice: gate in the first epilogue, residual in the second)
  prompt   a whole model call on token ids, `model(ids)`: a batch of short sequences through four blocks of full width
  step     a whole decoding step, `model(ids, inference_params_dict)`, behind a context: one request, or a batch of them
  delta    the gated delta rule of one layer (evo_gated_delta_fwd): prompts from zero, and portions that continue a state
  window   grouped-query attention over a sliding window with a sink and an output gate (evo_window_attn_fwd)
  conv     the short causal convolution with SiLU before a recurrence (evo_conv_act), with carried inputs
  norm     the row pass between two layers: branch outputs onto the fp32 stream, norms of the new row (evo_sum_norm)
"""
import ctypes as C
import math

import torch

from evo_b200 import _lib
from evo_b200._lib import (EPI_GELU_GATE, EPI_RESID, AttnParams, ConvActParams, GatedDeltaParams, GemmParams, HyenaParams, SumNormParams,
                           WindowAttnParams, check, ptr)
from evo_b200.configs import get_config
from evo_b200.stripedhyena import StripedHyena, dotdict
from evo_b200.stripedhyena.model import ATTN_VARIANT, GEMM_VARIANT, GEMM_VARIANT_GATE, pack_w12

DEV = "cuda"
BF = torch.bfloat16
F64 = torch.float64


def listed():
    return [
        # scoring a batch of full 8 k sequences (with the leading token: 8193 is what the scoring call passes on)
        {"name": "hyena_batch_8k", "kind": "hyena", "B": 8, "L": 8193, "D": 4096, "state": False, "carried": False},
        # the prompt of one request before it generates: few sequences, the end state is kept
        {"name": "hyena_one_prompt", "kind": "hyena", "B": 1, "L": 1999, "D": 4096, "state": True, "carried": False},
        # one full-length sequence through an attention layer
        {"name": "attention_8k", "kind": "attention", "B": 1, "L": 8193, "H": 32},
        # a feed-forward over a ragged batch of two medium sequences
        {"name": "mlp_two_seqs", "kind": "mlp", "M": 3002, "D": 4096},
        # scoring three short sequences: a whole call, where launches and half-empty tiles count
        {"name": "prompt_short", "kind": "prompt", "B": 3, "L": 301},
        # generation, one request and a batch of sixteen behind the benchmark's prompt
        {"name": "step_one", "kind": "step", "B": 1, "context": 999},
        {"name": "step_batch", "kind": "step", "B": 16, "context": 4096},
        # the gated delta rule over the benchmark's prompts, and over a portion of one request that continues its state
        {"name": "delta_prompts", "kind": "delta", "B": 4, "L": 4096, "H": 16, "dk": 128, "dv": 128, "carried": False},
        {"name": "delta_portion", "kind": "delta", "B": 1, "L": 777, "H": 32, "dk": 128, "dv": 128, "carried": True},
        # windowed attention of the benchmark's prompts
        {"name": "window_prompts", "kind": "window", "B": 4, "L": 4096, "H": 16, "G": 4, "dim": 128, "window": 1024},
        # the row kernels around them: three projections' channels; two branches of a layer and the two norms that follow
        {"name": "conv_prompts", "kind": "conv", "B": 4, "L": 4096, "C": 6144, "taps": 4, "carried": False},
        {"name": "norm_rows", "kind": "norm", "rows": 8190, "D": 4096, "branches": 2, "outs": 2, "branch_norm": False},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["hyena", "hyena", "attention", "mlp", "prompt", "step", "delta", "window", "conv", "norm"])
    if kind == "hyena":
        B, D = rng.choice([1, 1, 2, 3, 4, 8]), rng.choice([2048, 4096, 4096])
        return {"kind": kind, "B": B, "L": _log(rng, 20, 8193), "D": D, "state": rng.random() < 0.6, "carried": rng.random() < 0.25}
    if kind == "attention":
        B = rng.choice([1, 1, 2])
        return {"kind": kind, "B": B, "L": _log(rng, 100, 8193 // B), "H": rng.choice([16, 32])}
    if kind == "mlp":
        D = rng.choice([2048, 4096])
        return {"kind": kind, "M": _log(rng, 70, 5000 if D == 4096 else 8200), "D": D}
    if kind == "prompt":
        B = rng.choice([1, 2, 3, 5])
        return {"kind": kind, "B": B, "L": _log(rng, 30, 900 // B)}
    if kind == "step":
        return {"kind": kind, "B": _log(rng, 1, 16), "context": _log(rng, 20, 4096)}
    if kind == "delta":
        H = rng.choice([8, 16, 32])
        B = rng.choice([1, 1, 2, 4])
        return {"kind": kind, "B": B, "L": _log(rng, 40, 4096 if H < 32 else 2048), "H": H, "dk": rng.choice([128, 128, 64]),
                "dv": rng.choice([128, 128, 64]), "carried": rng.random() < 0.4}
    if kind == "window":
        H = rng.choice([8, 16])
        return {"kind": kind, "B": rng.choice([1, 2, 4]), "L": _log(rng, 50, 4096), "H": H, "G": H // rng.choice([1, 2, 4]), "dim": rng.choice([64, 128, 128]),
                "window": rng.choice([0, 256, 1024])}
    if kind == "conv":
        return {"kind": kind, "B": rng.choice([1, 2, 4]), "L": _log(rng, 20, 4096), "C": 64 * _log(rng, 24, 96), "taps": rng.choice([3, 4, 4]), "carried": rng.random() < 0.4}
    return {"kind": kind, "rows": _log(rng, 65, 8192), "D": rng.choice([2048, 4096]), "branches": rng.choice([1, 2, 3]), "outs": rng.choice([1, 2]), "branch_norm": rng.random() < 0.3}


# ---------------------------------------------------------------------------------------------------- inputs
class _Gen:
    """Normal and uniform numbers on the GPU from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)

    def n(self, *shape, std=1.0, dtype=BF, mean=0.0):
        out = torch.empty(shape, dtype=dtype, device=DEV)
        flat = out.view(-1)
        for i in range(0, flat.numel(), 1 << 27):              # in pieces: no fp32 copy of a large tensor
            part = flat[i:i + (1 << 27)]
            part.copy_(torch.randn(part.shape, generator=self.g, device=DEV).mul_(std).add_(mean))
        return out

    def u(self, *shape):
        return torch.rand(shape, generator=self.g, device=DEV)


def _filter(g, D):
    """Poles inside the unit disc (some close to it: long memory) and residues, fp32 (D, 8, 1, 2) as in a checkpoint."""
    mag, ph = 0.5 + 0.499 * g.u(D, 8), (g.u(D, 8) * 2 - 1) * math.pi
    poles = torch.stack([mag * torch.cos(ph), mag * torch.sin(ph)], -1)[:, :, None, :].contiguous()
    return poles, g.n(D, 8, 1, 2, std=0.35, dtype=torch.float32)


BLOCKS, ATTENTION = 4, 1                                         # prompt and step: three Hyena blocks around one attention block


def _model_config():
    cfg = get_config("evo-1-8k-base")
    cfg.update(num_layers=BLOCKS, attn_layer_idxs=[ATTENTION], hyena_layer_idxs=[i for i in range(BLOCKS) if i != ATTENTION])
    return cfg


def _model_weights(g, cfg):
    D, V, inner, hd = cfg["hidden_size"], cfg["vocab_size"], 10928, cfg["hidden_size"] // cfg["num_attention_heads"]
    sd = {"embedding_layer.weight": g.n(V, D, std=2.5 / math.sqrt(D)), "norm.scale": g.n(D, std=0.1, mean=1.0)}
    sd["unembed.weight"] = sd["embedding_layer.weight"]
    lin = lambda o, i: g.n(o, i, std=1.0 / math.sqrt(i))  # noqa: E731
    for i in range(BLOCKS):
        p = f"blocks.{i}."
        sd[p + "pre_norm.scale"], sd[p + "post_norm.scale"] = g.n(D, std=0.1, mean=1.0), g.n(D, std=0.1, mean=1.0)
        sd[p + "mlp.l1.weight"], sd[p + "mlp.l2.weight"], sd[p + "mlp.l3.weight"] = lin(inner, D), lin(inner, D), lin(D, inner)
        names = ("inner_mha_cls.Wqkv", "inner_mha_cls.out_proj") if i == ATTENTION else ("projections", "out_filter_dense")
        sd[p + names[0] + ".weight"], sd[p + names[0] + ".bias"] = lin(3 * D, D), g.n(3 * D, std=0.1)
        sd[p + names[1] + ".weight"], sd[p + names[1] + ".bias"] = lin(D, D), g.n(D, std=0.1)
        if i == ATTENTION:
            sd[p + "inner_mha_cls.rotary_emb.inv_freq"] = 1.0 / (10000 ** (torch.arange(0, hd, 2, dtype=torch.float32, device=DEV) / hd))
        else:
            sd[p + "filter.short_filter_weight"], sd[p + "filter.short_filter_bias"] = g.n(3 * D, 1, 3, std=0.5), g.n(3 * D, std=0.1)
            sd[p + "filter.D"] = g.n(D, std=0.5)
            sd[p + "filter.poles"], sd[p + "filter.residues"] = _filter(g, D)
    return sd


def _inputs(case, seed):
    """Everything that the case computes from, as plain tensors."""
    g, k, t = _Gen(seed), case["kind"], {}
    if k == "hyena":
        B, L, D = case["B"], case["L"], case["D"]
        t["z"] = g.n(B, L, 3 * D)
        t["fir_w"], t["fir_b"], t["skip"] = g.n(3 * D, 1, 3, std=0.5), g.n(3 * D, std=0.1), g.n(D, std=0.5)
        t["poles"], t["residues"] = _filter(g, D)
        if case["carried"]:
            t["halo"], t["state_in"] = g.n(B, 2, 3 * D), g.n(B, D, 8, 2, std=2.0, dtype=torch.float32)
    elif k == "attention":
        t["qkv"] = g.n(case["B"], case["L"], 3 * case["H"] * 128)
    elif k == "mlp":
        M, D = case["M"], case["D"]
        inner = 16 * -(-int(8 * D / 3) // 16)
        t["x"], t["resid"] = g.n(M, D), g.n(M, D)
        t["l1"], t["l2"], t["l3"] = g.n(inner, D, std=D ** -0.5), g.n(inner, D, std=D ** -0.5), g.n(D, inner, std=inner ** -0.5)
    elif k in ("prompt", "step"):
        cfg = _model_config()
        B, L, D = case["B"], case.get("L", 1), cfg["hidden_size"]
        t["weights"] = _model_weights(g, cfg)
        t["ids"] = torch.tensor([65, 67, 71, 84], device=DEV)[(g.u(B, L) * 4).long()]
        if k == "step":
            H = cfg["num_attention_heads"]
            t["cache"] = g.n(B, case["context"] + 64, 2, H, D // H)
            for i in range(BLOCKS):
                if i != ATTENTION:
                    t[f"fir{i}"], t[f"state{i}"] = g.n(B, 3 * D, 2), torch.view_as_complex(g.n(B, D, 8, 2, std=2.0, dtype=torch.float32))
    elif k == "delta":
        B, L, H, dk, dv = (case[n] for n in ("B", "L", "H", "dk", "dv"))
        # one buffer of activated [q | k | v] (behind the convolution's SiLU), one of raw [gate | b | a]
        t["qkv"] = torch.nn.functional.silu(g.n(B * L, H * (2 * dk + dv)))
        t["z"] = g.n(B * L, H * dv + 2 * H)
        t["A_log"] = torch.log(1.0 + 15.0 * g.u(H)).to(BF)
        dt = torch.exp(g.u(H) * (math.log(0.1) - math.log(0.001)) + math.log(0.001))
        t["dt_bias"], t["norm_w"] = (dt + torch.log(-torch.expm1(-dt))).to(BF), g.n(dv, std=0.2, mean=1.0)
        t["state"] = g.n(B, H, dk, dv, std=0.3, dtype=torch.float32)
    elif k == "window":
        B, L, H, G, d = (case[n] for n in ("B", "L", "H", "G", "dim"))
        t["q"], t["gate"] = g.n(B * L, H * d), g.n(B * L, H * d)
        t["kv"], t["sink"] = g.n(B, L, 2 * G * d), g.n(H)
    elif k == "conv":
        B, L, Cn = case["B"], case["L"], case["C"]
        t["x"], t["w"] = g.n(B * L, Cn + 2048 + 64), g.n(Cn, case["taps"], std=0.5)
        t["carry"] = g.n(B, case["taps"] - 1, Cn, dtype=torch.float32)
    else:
        R, D = case["rows"], case["D"]
        t["x"] = g.n(R, D, dtype=torch.float32)
        for i in range(case["branches"]):
            t[f"y{i}"] = g.n(R, D)
            t[f"n{i}"] = g.n(D, std=0.1, mean=1.0)
        for i in range(case["outs"]):
            t[f"w{i}"] = g.n(D, std=0.1, mean=1.0)
    return t


def prepare(case, seed):
    t = _inputs(case, seed)
    s = {"case": case, "t": t}
    if case["kind"] in ("prompt", "step"):
        cfg = _model_config()
        with torch.device(DEV):
            model = StripedHyena(dotdict(cfg))
        model.load_state_dict(t.pop("weights"), strict=True)
        s["model"] = model.to_bfloat16_except_poles_residues().to(DEV)
        if case["kind"] == "step":
            d = model.initialize_inference_params()
            d["mha"].max_batch_size, d["mha"].max_seqlen = case["B"], case["context"] + 64
            d["mha"].key_value_memory_dict[ATTENTION] = t.pop("cache")
            for i in range(BLOCKS):
                if i != ATTENTION:
                    d["hyena"].fir_state_dict[i], d["hyena"].state_dict[i] = t.pop(f"fir{i}"), t.pop(f"state{i}")
            s["state"] = d
    elif case["kind"] == "mlp":
        l1, l2, l3 = t.pop("l1"), t.pop("l2"), t.pop("l3")
        ipad = -(-l1.shape[0] // 128) * 128
        s["w12"], s["w3"], s["ipad"] = pack_w12(l1, l2, ipad), torch.nn.functional.pad(l3, (0, ipad - l1.shape[0])), ipad
    return s


# ---------------------------------------------------------------------------------------------------- one pass
def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _run_hyena(s):
    c, t, lib = s["case"], s["t"], _lib.lib()
    B, L, D = c["B"], c["L"], c["D"]
    y = torch.empty(B, L, D, dtype=BF, device=DEV)
    p = HyenaParams(z=t["z"].data_ptr(), y=y.data_ptr(), fir_w=t["fir_w"].data_ptr(), fir_b=t["fir_b"].data_ptr(), Dskip=t["skip"].data_ptr(),
                    poles=t["poles"].data_ptr(), residues=t["residues"].data_ptr(), B=B, L=L, D=D, S=8, nheads=D // 128)
    out = {"y": y}
    if c["carried"]:
        p.halo, p.state_in = t["halo"].data_ptr(), t["state_in"].data_ptr()
    if c["state"]:
        out["state"], out["fir"] = torch.empty(B, D, 8, 2, dtype=torch.float32, device=DEV), torch.empty(B, 3 * D, 2, dtype=BF, device=DEV)
        p.state_out, p.fir_state_out = out["state"].data_ptr(), out["fir"].data_ptr()
    n = lib.evo_hyena_fwd_workspace(C.byref(p))
    ws = torch.empty(max(n, 1), dtype=torch.uint8, device=DEV)
    check(lib.evo_hyena_fwd(C.byref(p), ptr(ws), n, _stream()), "evo_hyena_fwd")
    return out


def _run_attention(s):
    c, t, lib = s["case"], s["t"], _lib.lib()
    B, L, H = c["B"], c["L"], c["H"]
    d = H * 128
    out = torch.empty(B, L, d, dtype=BF, device=DEV)
    q = t["qkv"].data_ptr()
    p = AttnParams(q=q, k=q + d * 2, v=q + 2 * d * 2, out=out.data_ptr(), q_tok_stride=3 * d, kv_tok_stride=3 * d, q_batch_stride=L * 3 * d, kv_batch_stride=L * 3 * d,
                   B=B, Lq=L, Lk=L, H=H, hd=128, q_pos0=0, softmax_scale=1.0 / math.sqrt(128))
    n = lib.evo_attn_fwd_workspace(C.byref(p), ATTN_VARIANT)
    ws = torch.empty(max(n, 1), dtype=torch.uint8, device=DEV)
    check(lib.evo_attn_fwd_ws(C.byref(p), ATTN_VARIANT, ptr(ws), n, _stream()), "evo_attn_fwd")
    return out


def _run_mlp(s):
    c, t, lib = s["case"], s["t"], _lib.lib()
    M, D, ip = c["M"], c["D"], s["ipad"]
    h, out = torch.empty(M, ip, dtype=BF, device=DEV), torch.empty(M, D, dtype=BF, device=DEV)
    p = GemmParams(A=t["x"].data_ptr(), lda=D, W=s["w12"].data_ptr(), C=h.data_ptr(), ldc=ip, ldr=ip, M=M, N=2 * ip, K=D, epilogue=EPI_GELU_GATE, variant=GEMM_VARIANT_GATE)
    check(lib.evo_gemm(C.byref(p), _stream()), "evo_gemm")
    p = GemmParams(A=h.data_ptr(), lda=ip, W=s["w3"].data_ptr(), C=out.data_ptr(), ldc=D, residual=t["resid"].data_ptr(), ldr=D, M=M, N=D, K=ip, epilogue=EPI_RESID, variant=GEMM_VARIANT)
    check(lib.evo_gemm(C.byref(p), _stream()), "evo_gemm")
    return out


def _run_step(s):
    d, at = s["state"], s["case"]["context"]
    d["mha"].seqlen_offset = d["hyena"].seqlen_offset = at
    logits, d = s["model"](s["t"]["ids"], inference_params_dict=d)
    out = {"logits": logits, "cache": d["mha"].key_value_memory_dict[ATTENTION]}
    for i in d["hyena"].state_dict:
        out[f"state{i}"], out[f"fir{i}"] = d["hyena"].state_dict[i], d["hyena"].fir_state_dict[i]
    return out


def _run_delta(s):
    c, t, lib = s["case"], s["t"], _lib.lib()
    B, L, H, dk, dv = (c[n] for n in ("B", "L", "H", "dk", "dv"))
    out = torch.empty(B * L, H * dv, dtype=BF, device=DEV)
    q, z = t["qkv"].data_ptr(), t["z"].data_ptr()
    p = GatedDeltaParams(q=q, k=q + 2 * H * dk, v=q + 4 * H * dk, ld=H * (2 * dk + dv), b=z + 2 * H * dv, a=z + 2 * (H * dv + H), gate=z, ldz=H * dv + 2 * H,
                         A_log=t["A_log"].data_ptr(), dt_bias=t["dt_bias"].data_ptr(), norm_w=t["norm_w"].data_ptr(), eps=1e-6, unit_eps=1e-6, q_scale=dk ** -0.5,
                         state=t["state"].data_ptr(), zero_start=0 if c["carried"] else 1, out=out.data_ptr(), ldo=H * dv, dtype=0, B=B, L=L, H=H, G=H, dk=dk, dv=dv)
    n = lib.evo_gated_delta_workspace(C.byref(p))
    ws = torch.empty(n, dtype=torch.uint8, device=DEV) if n else None
    check(lib.evo_gated_delta_fwd(C.byref(p), ptr(ws), n, _stream()), "evo_gated_delta_fwd")
    return {"out": out, "state": t["state"]}


def _run_window(s):
    c, t, lib = s["case"], s["t"], _lib.lib()
    B, L, H, G, d = (c[n] for n in ("B", "L", "H", "G", "dim"))
    out = torch.empty(B * L, H * d, dtype=BF, device=DEV)
    row = 2 * G * d
    p = WindowAttnParams(q=t["q"].data_ptr(), q_tok_stride=H * d, k=t["kv"].data_ptr(), v=t["kv"].data_ptr() + 2 * G * d, k_tok_stride=row, v_tok_stride=row,
                         k_batch_stride=L * row, v_batch_stride=L * row, gate=t["gate"].data_ptr(), gate_tok_stride=H * d, out=out.data_ptr(), ldo=H * d, dtype=0,
                         B=B, Lq=L, H=H, G=G, dk=d, dv=d, n_maps=1, q_pos0=0, window=c["window"], keep_first=0, scale=d ** -0.5, sink=t["sink"].data_ptr())
    check(lib.evo_window_attn_fwd(C.byref(p), _stream()), "evo_window_attn_fwd")
    return out


def _run_conv(s):
    c, t, lib = s["case"], s["t"], _lib.lib()
    out = torch.empty(c["B"] * c["L"], c["C"], dtype=BF, device=DEV)
    p = ConvActParams(inp=t["x"].data_ptr(), ld=t["x"].shape[1], weight=t["w"].data_ptr(), carry=t["carry"].data_ptr(), zero_start=0 if c["carried"] else 1,
                      out=out.data_ptr(), ldo=c["C"], B=c["B"], L=c["L"], C=c["C"], taps=c["taps"], act=1, dtype=0)
    check(lib.evo_conv_act(C.byref(p), _stream()), "evo_conv_act")
    return {"out": out, "carry": t["carry"]}


def _run_norm(s):
    c, t, lib = s["case"], s["t"], _lib.lib()
    R, D = c["rows"], c["D"]
    p = SumNormParams(x=t["x"].data_ptr(), n_branches=c["branches"], eps=1e-6, dtype=0, rows=R, D=D, ldo=D)
    for i in range(c["branches"]):
        p.y[i], p.ldy[i], p.norm_w[i], p.scale[i] = t[f"y{i}"].data_ptr(), D, t[f"n{i}"].data_ptr() if c["branch_norm"] else None, 0.5
    out = {"x": t["x"]}
    for i in range(c["outs"]):
        out[f"out{i}"] = torch.empty(R, D, dtype=BF, device=DEV)
        p.out[i], p.w[i] = out[f"out{i}"].data_ptr(), t[f"w{i}"].data_ptr()
    check(lib.evo_sum_norm(C.byref(p), _stream()), "evo_sum_norm")
    return out


_RUN = {"hyena": _run_hyena, "attention": _run_attention, "mlp": _run_mlp, "prompt": lambda s: s["model"](s["t"]["ids"])[0], "step": _run_step, "delta": _run_delta,
        "window": _run_window, "conv": _run_conv, "norm": _run_norm}


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ---------------------------------------------------------------------------------------------------- what a pass cannot do without
def _block_work(rows, D=4096, inner=10928):
    return 2.0 * rows * (4 * D * D + 3 * D * inner), 2.0 * (4 * D * D + 3 * D * inner)


def work(case):
    k = case["kind"]
    if k == "hyena":
        B, L, D = case["B"], case["L"], case["D"]
        # z once, y once, filters and states; per token and channel: three taps of three channels, the gates, and eight complex modes (update 8, read-out 4)
        return {"bytes": 8.0 * B * L * D + 128.0 * D + (64.0 + 12.0) * B * D * (case["state"] + case["carried"]), "flops": B * L * D * (18.0 + 4.0 + 96.0)}
    if k == "attention":
        B, L, H = case["B"], case["L"], case["H"]
        return {"bytes": 8.0 * B * L * H * 128, "flops": 2.0 * 128 * 2 * B * H * L * (L + 1) / 2}
    if k == "mlp":
        M, D = case["M"], case["D"]
        inner = 16 * -(-int(8 * D / 3) // 16)
        return {"bytes": 2.0 * (3 * M * D + 3 * D * inner), "flops": 6.0 * M * D * inner}
    if k in ("prompt", "step"):
        B, L = case["B"], case.get("L", 1)
        flops, weights = _block_work(B * L)
        flops, nbytes = BLOCKS * flops + 2.0 * B * L * 512 * 4096, BLOCKS * weights + 2.0 * 512 * 4096 + 2.0 * B * L * 512
        keys = case.get("context", 0)
        flops += 2.0 * 4096 * 2 * B * (L * (L + 1) / 2 + L * keys) + (BLOCKS - 1) * B * L * 4096 * 118.0
        if k == "step":
            nbytes += B * (2.0 * 2 * 4096 * keys + (BLOCKS - 1) * 2 * 4096 * (64.0 + 12.0))
        return {"bytes": nbytes, "flops": flops}
    if k == "delta":
        B, L, H, dk, dv = (case[n] for n in ("B", "L", "H", "dk", "dv"))
        # per token and head: decay, S^T k, S^T q and the rank-one update of a dk x dv state
        return {"bytes": 2.0 * B * L * H * (2 * dk + 3 * dv + 2) + 4.0 * B * H * dk * dv * (1 + case["carried"]), "flops": 7.0 * B * L * H * dk * dv}
    if k == "window":
        B, L, H, G, d = (case[n] for n in ("B", "L", "H", "G", "dim"))
        w = case["window"] if 0 < case["window"] < L else L
        pairs = w * (w + 1) / 2 + (L - w) * w
        return {"bytes": 2.0 * B * L * (3 * H * d + 2 * G * d), "flops": 4.0 * B * H * pairs * d}
    if k == "conv":
        B, L, Cn = case["B"], case["L"], case["C"]
        return {"bytes": 4.0 * B * L * Cn + 8.0 * B * Cn, "flops": B * L * Cn * (2.0 * case["taps"] + 4)}
    R, D = case["rows"], case["D"]
    return {"bytes": R * D * (8.0 + 2 * case["branches"] + 2 * case["outs"]), "flops": R * D * (2.0 * case["branches"] + 2 + 2 * case["outs"])}


#: About four times the distance between this path and the same inputs in 64 bits (measured: 0.0052, 0.0020, 0.0028, 0.022, 0.0088, 0.0017, ...; 0.03 at
#: most): the operators round to bf16 where the reference's own tensor operations do, and in a whole call such a rounding travels through every later block.
_TOLERANCE = {"hyena": {"rel": 0.02}, "attention": {"rel": 0.008}, "mlp": {"rel": 0.011}, "prompt": {"rel": 0.03}, "step": {"rel": 0.03}, "delta": {"rel": 0.007},
              "window": {"rel": 0.007}, "conv": {"rel": 0.007}, "norm": {"rel": 0.007}}


def tolerance(case):
    return _TOLERANCE[case["kind"]]


# ---------------------------------------------------------------------------------------------------- the same in 64 bits
def _modal(x, poles, residues, state):
    """x (B, L, D) -> (long convolution (B, L, D), end state (B, D, 8) complex) for the modes of a layer, by blocks of tokens."""
    B, L, D = x.shape
    p, r = torch.view_as_complex(poles.to(F64))[:, :, 0], torch.view_as_complex(residues.to(F64))[:, :, 0]
    S = torch.zeros(B, D, 8, dtype=torch.complex128, device=x.device) if state is None else state
    T = min(64, L)
    pw = p[None] ** torch.arange(T + 1, device=x.device, dtype=F64)[:, None, None]                       # (T + 1, D, 8)
    h = (pw[:T] * r).sum(-1).real                                                                        # (T, D)
    lag = torch.arange(T, device=x.device)[:, None] - torch.arange(T, device=x.device)[None]
    toe = torch.where((lag >= 0)[..., None], h[lag.clamp(min=0)], torch.zeros((), dtype=F64, device=x.device)).permute(2, 0, 1).contiguous()   # (D, T, T)
    carry = (pw[1:] * r).permute(1, 0, 2).contiguous()                                                   # (D, T, 8): state before the block -> its outputs
    out = torch.empty_like(x)
    for t in range(0, L, T):
        xb = x[:, t:t + T]
        n = xb.shape[1]
        xd = xb.permute(2, 1, 0)                                                                         # (D, n, B)
        y = torch.bmm(toe[:, :n, :n], xd) + torch.bmm(carry[:, :n], S.permute(1, 2, 0)).real
        out[:, t:t + n] = y.permute(2, 1, 0)
        S = pw[n] * S + torch.bmm(pw[:n].flip(0).permute(1, 2, 0), xd.to(torch.complex128)).permute(2, 0, 1)
    return out, S


def _hyena_exact(z, w, b, skip, poles, residues, halo=None, state=None):
    """z (B, L, 3D) in 64 bits -> (y (B, L, D), end state)."""
    B, L, C3 = z.shape
    pre = torch.zeros(B, 2, C3, dtype=F64, device=z.device) if halo is None else halo.to(F64)
    zp = torch.cat([pre, z], 1)
    w = w.to(F64)[:, 0]
    f = (zp[:, :L] * w[:, 0] + zp[:, 1:L + 1] * w[:, 1] + zp[:, 2:] * w[:, 2] + b.to(F64)).view(B, L, C3 // 384, 3, 128)
    x2, x1, v = (f[:, :, :, i].reshape(B, L, C3 // 3) for i in range(3))
    x = x1 * v
    c, S = _modal(x, poles, residues, state)
    return (c + x * skip.to(F64)) * x2, S


def _attend(q, k, v, first, window=0, sink=None):
    """One head: q (n, d) at positions first .., k, v (m, d) from position 0, 64 bits."""
    out = torch.empty(q.shape[0], v.shape[1], dtype=F64, device=q.device)
    for i in range(0, q.shape[0], 1024):
        qi = q[i:i + 1024]
        lo, hi = (max(0, first + i - window + 1) if window > 0 else 0), first + i + qi.shape[0]
        sc = qi @ k[lo:hi].T
        dist = (torch.arange(qi.shape[0], device=q.device) + first + i)[:, None] - torch.arange(lo, hi, device=q.device)[None]
        sc = sc.masked_fill((dist < 0) | ((dist >= window) if window > 0 else (dist < 0)), -math.inf)
        if sink is not None:
            sc = torch.cat([sc, sink.expand(sc.shape[0], 1)], 1)
        w = torch.softmax(sc, 1)
        out[i:i + 1024] = w[:, :hi - lo] @ v[lo:hi]
    return out


def _rotate(x, pos, freq):
    """x (B, L, H, d): halves turned by pos * freq."""
    a = pos[:, None].to(F64) * freq.to(F64)[None]
    c, s = torch.cos(a)[None, :, None], torch.sin(a)[None, :, None]
    h = x.shape[-1] // 2
    return torch.cat([x[..., :h] * c - x[..., h:] * s, x[..., h:] * c + x[..., :h] * s], -1)


def _model_exact(case, t):
    sd, ids = t["weights"], t["ids"]
    B, L = ids.shape
    D, H, first = 4096, 32, case.get("context", 0)
    w = lambda n: sd[n].to(F64)  # noqa: E731
    rms = lambda x, n: x / (x.norm(dim=-1, keepdim=True) * D ** -0.5 + 1e-6) * w(n)  # noqa: E731
    u, out = w("embedding_layer.weight")[ids], {}
    for i in range(BLOCKS):
        p = f"blocks.{i}."
        x = rms(u, p + "pre_norm.scale")
        if i == ATTENTION:
            qkv = (x @ w(p + "inner_mha_cls.Wqkv.weight").T + w(p + "inner_mha_cls.Wqkv.bias")).view(B, L, 3, H, 128)
            pos, freq = torch.arange(first, first + L, device=u.device), sd[p + "inner_mha_cls.rotary_emb.inv_freq"]
            q, k, v = _rotate(qkv[:, :, 0], pos, freq), _rotate(qkv[:, :, 1], pos, freq), qkv[:, :, 2]
            ctx = torch.empty(B, L, H, 128, dtype=F64, device=u.device)
            for b in range(B):
                for h in range(H):
                    kk, vv = k[b, :, h], v[b, :, h]
                    if first:
                        kk, vv = torch.cat([t["cache"][b, :first, 0, h].to(F64), kk]), torch.cat([t["cache"][b, :first, 1, h].to(F64), vv])
                    ctx[b, :, h] = _attend(q[b, :, h] / math.sqrt(128), kk, vv, first)
            out["cache"] = None
            u = u + ctx.reshape(B, L, D) @ w(p + "inner_mha_cls.out_proj.weight").T + w(p + "inner_mha_cls.out_proj.bias")
        else:
            z = x @ w(p + "projections.weight").T + w(p + "projections.bias")
            halo = t[f"fir{i}"].permute(0, 2, 1) if first else None
            y, S = _hyena_exact(z, sd[p + "filter.short_filter_weight"], sd[p + "filter.short_filter_bias"], sd[p + "filter.D"], sd[p + "filter.poles"], sd[p + "filter.residues"],
                                halo, t[f"state{i}"].to(torch.complex128) if first else None)
            out[f"state{i}"], out[f"fir{i}"] = S, torch.stack([halo[:, 1].to(F64), z[:, 0]], -1) if first else None
            u = u + y @ w(p + "out_filter_dense.weight").T + w(p + "out_filter_dense.bias")
        x = rms(u, p + "post_norm.scale")
        h = torch.nn.functional.gelu(x @ w(p + "mlp.l1.weight").T) * (x @ w(p + "mlp.l2.weight").T)
        u = u + h @ w(p + "mlp.l3.weight").T
    logits = rms(u, "norm.scale") @ w("unembed.weight").T
    return dict(out, logits=logits) if first else logits


def _delta_exact(case, t):
    B, L, H, dk, dv = (case[n] for n in ("B", "L", "H", "dk", "dv"))
    x, z = t["qkv"].to(F64), t["z"].to(F64)
    q, k, v = x[:, :H * dk].view(B, L, H, dk), x[:, H * dk:2 * H * dk].view(B, L, H, dk), x[:, 2 * H * dk:].view(B, L, H, dv)
    gate, b, a = z[:, :H * dv].view(B, L, H, dv), z[:, H * dv:H * dv + H].view(B, L, H), z[:, H * dv + H:].view(B, L, H)
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dk ** -0.5
    g = torch.exp(-torch.exp(t["A_log"].to(F64)) * torch.nn.functional.softplus(a + t["dt_bias"].to(F64)))
    beta = torch.sigmoid(b)
    S = t["state"].to(F64) if case["carried"] else torch.zeros(B, H, dk, dv, dtype=F64, device=x.device)
    o = torch.empty(B, L, H, dv, dtype=F64, device=x.device)
    for i in range(L):
        S = S * g[:, i, :, None, None]
        u = beta[:, i, :, None] * (v[:, i] - torch.einsum("bhk,bhkv->bhv", k[:, i], S))
        S = torch.baddbmm(S.view(B * H, dk, dv), k[:, i].reshape(B * H, dk, 1), u.reshape(B * H, 1, dv)).view(B, H, dk, dv)
        o[:, i] = torch.einsum("bhk,bhkv->bhv", q[:, i], S)
    o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6) * t["norm_w"].to(F64) * torch.nn.functional.silu(gate)
    return {"out": o.reshape(B * L, H * dv), "state": S}


def exact(case, seed):
    t, k = _inputs(case, seed), case["kind"]
    if k == "hyena":
        L = case["L"]
        zs = [t["z"][b:b + 1] for b in range(case["B"])]
        got = [_hyena_exact(z.to(F64), t["fir_w"], t["fir_b"], t["skip"], t["poles"], t["residues"], t["halo"][b:b + 1] if case["carried"] else None,
                            torch.view_as_complex(t["state_in"][b:b + 1].to(F64)) if case["carried"] else None) for b, z in enumerate(zs)]
        out = {"y": torch.cat([y for y, _ in got])}
        if case["state"]:
            out["state"], out["fir"] = torch.view_as_real(torch.cat([S for _, S in got])), t["z"][:, L - 2:].permute(0, 2, 1).to(F64)
        return out
    if k == "attention":
        B, L, H = case["B"], case["L"], case["H"]
        x = t["qkv"].view(B, L, 3, H, 128)
        out = torch.empty(B, L, H, 128, dtype=F64, device=DEV)
        for b in range(B):
            for h in range(H):
                q, kk, v = (x[b, :, i, h].to(F64) for i in range(3))
                out[b, :, h] = _attend(q / math.sqrt(128), kk, v, 0)
        return out.view(B, L, H * 128)
    if k == "mlp":
        x = t["x"].to(F64)
        return torch.nn.functional.gelu(x @ t["l1"].to(F64).T).mul_(x @ t["l2"].to(F64).T) @ t["l3"].to(F64).T + t["resid"].to(F64)
    if k in ("prompt", "step"):
        return _model_exact(case, t)
    if k == "delta":
        return _delta_exact(case, t)
    if k == "window":
        B, L, H, G, d = (case[n] for n in ("B", "L", "H", "G", "dim"))
        q, gate, kv = t["q"].view(B, L, H, d), t["gate"].view(B, L, H, d), t["kv"].view(B, L, 2, G, d)
        out = torch.empty(B, L, H, d, dtype=F64, device=DEV)
        for b in range(B):
            for h in range(H):
                o = _attend(q[b, :, h].to(F64) * d ** -0.5, kv[b, :, 0, h // (H // G)].to(F64), kv[b, :, 1, h // (H // G)].to(F64), 0, case["window"], t["sink"][h].to(F64))
                out[b, :, h] = o * torch.sigmoid(gate[b, :, h].to(F64))
        return out.view(B * L, H * d)
    if k == "conv":
        B, L, Cn, taps = case["B"], case["L"], case["C"], case["taps"]
        out, carry = torch.empty(B * L, Cn, dtype=F64, device=DEV), []
        for b in range(B):
            x = t["x"][b * L:(b + 1) * L, :Cn].to(F64)
            pre = t["carry"][b].to(F64) if case["carried"] else torch.zeros(taps - 1, Cn, dtype=F64, device=DEV)
            x = torch.cat([pre, x])
            out[b * L:(b + 1) * L] = torch.nn.functional.silu(sum(x[j:j + L] * t["w"][:, j].to(F64) for j in range(taps)))
            carry.append(x[L:])
        return {"out": out, "carry": torch.stack(carry)}
    rms = lambda v: v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-6)  # noqa: E731
    x = t["x"].to(F64)
    for i in range(case["branches"]):
        y = t[f"y{i}"].to(F64)
        x = x + 0.5 * (rms(y) * t[f"n{i}"].to(F64) if case["branch_norm"] else y)
    out = {"x": x}
    for i in range(case["outs"]):
        out[f"out{i}"] = rms(x) * t[f"w{i}"].to(F64)
    return out
