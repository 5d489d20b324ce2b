"""The forward passes that serving consists of, as cases to be timed: decode steps, verify steps of speculation, prompts
and portions of prompts, through ``LLMEngine``'s model (``runner.decoder.forward``), for the three kinds of checkpoint
that the engine's benchmark and tests run: NVFP4 weights with an fp8 cache, bf16 throughout, FP8 block weights in a
hybrid of gated delta net, gated attention and experts.

Models have the layer sizes of the presets and one or two layers of them, behind a vocabulary cut as much, so that the
layers have about the share of a pass that they have in a whole model. As in the engine, a step of one or a few tokens
per sequence is replayed from a CUDA graph over fixed buffers, and prompts run eagerly.
"""
from __future__ import annotations

import math

import torch

#: one layer where activations are four bits wide: behind a second one a last-bit difference in the first has become a
#: step of the quantisers in so many places that no two correct results are alike
LAYERS, VOCAB, BLOCK = {"nvfp4": 1, "bf16": 2, "hybrid-fp8": 2}, 2048, 16
#: standard deviation of the weights, of those whose outputs join the residual stream (divided by the root of the number of
#: sublayers of the whole model, as deep models are initialised), and of the stream that the layers find
STD, STD_OUT, STD_STREAM = 0.02, 0.02 / 128 ** 0.5, 2.0


# ----------------------------------------------------------------------------- cases
def case(name, model, seqs, new, past, new_min=None, past_min=None):
    """`seqs` sequences that bring `new_min` to `new` tokens behind `past_min` to `past` cached ones."""
    d = dict(model=model, seqs=seqs, new=new, new_min=new if new_min is None else new_min, past=past,
             past_min=past if past_min is None else past_min)
    return dict(name=name, **d) if name else d


def listed():
    return [
        # one user, mid-generation: the latency of a token
        case("nvfp4 decode 1", "nvfp4", 1, 1, 700),
        # a lightly loaded server
        case("nvfp4 decode 16", "nvfp4", 16, 1, 1151, past_min=129),
        # the headline benchmark's rung: 128 requests of 128 prompt tokens, between their first and 1024th token
        case("nvfp4 decode 128", "nvfp4", 128, 1, 1151, past_min=129),
        # long documents under discussion
        case("nvfp4 decode 9 long", "nvfp4", 9, 1, 16000, past_min=4000),
        # speculation: three drafts per sequence checked in one pass
        case("nvfp4 verify 8x4", "nvfp4", 8, 4, 901, past_min=300),
        # a chat turn's prompt
        case("nvfp4 prompt 333", "nvfp4", 1, 333, 0),
        # the headline benchmark's prefill: 128 prompts at once would be two portions of the budget
        case("nvfp4 prompts 64x128", "nvfp4", 64, 128, 0),
        # a document of the whole prefill budget
        case("nvfp4 prompt 8192", "nvfp4", 1, 8192, 0),
        # unquantised checkpoint, decode of a medium batch
        case("bf16 decode 33", "bf16", 33, 1, 2047, past_min=100),
        # unquantised checkpoint, portions of two prompts behind what is cached of them
        case("bf16 portions 2x1531", "bf16", 2, 1531, 2900, new_min=1001, past_min=2500),
        # hybrid with experts: decode of a small batch
        case("hybrid decode 16", "hybrid-fp8", 16, 1, 2000, past_min=200),
        # hybrid with experts: a few prompts of a portion
        case("hybrid prompts 3x1300", "hybrid-fp8", 3, 1300, 0, new_min=500),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    model = rng.choice(("nvfp4", "nvfp4", "nvfp4", "bf16", "hybrid-fp8"))
    kind = rng.choice(("decode", "decode", "prompt", "prompt", "portion") + (("verify",) if model != "hybrid-fp8" else ()))
    if kind == "decode":
        seqs = _log(rng, 1, 128)
        past = _log(rng, 64, min(16000, 147000 // seqs))
        return case(None, model, seqs, 1, past, past_min=rng.randint(past // 4, past))
    if kind == "verify":
        past = _log(rng, 64, 4000)
        return case(None, model, _log(rng, 1, 16), rng.randint(2, 5), past, past_min=rng.randint(past // 4, past))
    most = 8192 if model == "nvfp4" else 4096
    total = _log(rng, 24, most)
    seqs = min(_log(rng, 1, 64), max(1, total // 16))
    new = total // seqs
    past = 0 if kind == "prompt" or model == "hybrid-fp8" else _log(rng, 64, max(65, min(4000, 16000 // seqs, 8192 - new)))
    return case(None, model, seqs, new, past, new_min=rng.randint(max(6, new // 3), new), past_min=rng.randint(past // 2, past))


def _lengths(c):
    """(new, past) tokens of every sequence: spread over the ranges, the same for every seed."""
    n, out = c["seqs"], []
    for i in range(n):
        f, g = (((i * 37 + 11) % n) / (n - 1), ((i * 53 + 5) % n) / (n - 1)) if n > 1 else (1.0, 1.0)
        out.append((round(c["new_min"] + f * (c["new"] - c["new_min"])), round(c["past_min"] + g * (c["past"] - c["past_min"]))))
    return out


# ----------------------------------------------------------------------------- the model and its checkpoint
def _config(model):
    from metrale_inference_alpha_b200.config.model_config import preset
    if model == "hybrid-fp8":
        return preset("qwen-hybrid-moe-35b-fp8", num_layers=LAYERS[model], layer_types=["gdn", "attention"],
                      ffn_types=["moe"] * LAYERS[model], vocab_size=VOCAB)
    kw = dict(weight_format="bf16", kv_dtype="bf16") if model == "bf16" else {}
    return preset("dense-27b-nvfp4", num_layers=LAYERS[model], vocab_size=VOCAB, mtp_layers=0, **kw)


_E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)
_MIDS = (0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0)
#: static input scales of an NVFP4 checkpoint: twice the largest input of a calibration run over 6 * 448
O_SCALE, DOWN_SCALE = 2 * 6.0 / 2688, 2 * 25.0 / 2688


def _e4m3(x):
    return x.float().clamp(-448, 448).to(torch.float8_e4m3fn)


def _nvfp4_parts(x, gs):
    """e2m1 codes [R, K] (sign in bit 3), e4m3 block scales [R, K / 16] of x / gs, gs a number or [R, 1]."""
    b = x.view(x.shape[0], -1, 16)
    sf = _e4m3(b.abs().amax(2) / (6 * gs))
    step = sf.to(x.dtype) * gs
    a = torch.where(step[..., None] > 0, b.abs() / step[..., None].clamp(min=1e-30), torch.zeros_like(b))
    codes = torch.bucketize(a, torch.tensor(_MIDS, dtype=x.dtype, device=x.device), out_int32=True).to(torch.uint8)
    return (codes | ((b < 0).to(torch.uint8) << 3)).view(x.shape), sf


def _nvfp4_values(codes, sf, gs):
    v = torch.tensor(_E2M1 + tuple(-t for t in _E2M1), dtype=torch.float64, device=codes.device)[codes.long()]
    return (v.view(v.shape[0], -1, 16) * (sf.double() * gs)[..., None]).view(v.shape)


class _Checkpoint:
    """Seeded random weights under their HF names, in the checkpoint's own encodings."""

    def __init__(self, model, seed, device="cuda"):
        self.cfg, self.model, self.t = _config(model), model, {}
        self.g = torch.Generator(device=device).manual_seed(seed)
        self.device, c = device, self.cfg
        H = c.hidden_size
        self.plain("model.embed_tokens", VOCAB, H, std=STD_STREAM)
        self.plain("lm_head", VOCAB, H)
        self.norm("model.norm", H)
        for i, kind in enumerate(c.layer_types):
            p = f"model.layers.{i}"
            self.norm(f"{p}.input_layernorm", H)
            self.norm(f"{p}.post_attention_layernorm", H)
            if kind == "gdn":
                q, qk, v = f"{p}.linear_attn", c.gdn_qk_size, c.gdn_v_size
                self.linear(f"{q}.in_proj_qkv", 2 * qk + v, H)
                self.linear(f"{q}.in_proj_z", v, H)
                self.plain(f"{q}.in_proj_b", c.gdn_v_heads, H)
                self.plain(f"{q}.in_proj_a", c.gdn_v_heads, H)
                self.t[f"{q}.conv1d.weight"] = self.normal((2 * qk + v, 1, c.conv_kernel), 0.3).bfloat16()
                self.t[f"{q}.A_log"] = self.normal((c.gdn_v_heads,), 0.3)
                self.t[f"{q}.dt_bias"] = self.normal((c.gdn_v_heads,), 0.1)
                self.t[f"{q}.norm.weight"] = (1 + self.normal((c.gdn_v_dim,), 0.02)).bfloat16()
                self.linear(f"{q}.out_proj", H, v, std=STD_OUT)
            else:
                q = f"{p}.self_attn"
                self.linear(f"{q}.q_proj", c.q_size, H)
                self.linear(f"{q}.k_proj", c.kv_size, H)
                self.linear(f"{q}.v_proj", c.kv_size, H)
                self.linear(f"{q}.o_proj", H, c.num_heads * c.head_dim, O_SCALE, STD_OUT)
                self.norm(f"{q}.q_norm", c.head_dim)
                self.norm(f"{q}.k_norm", c.head_dim)
            m = f"{p}.mlp"
            if c.ffn_types[i] == "dense":
                self.ffn(m, c.intermediate_size)
                continue
            self.plain(f"{m}.gate", c.num_experts, H)
            for e in range(c.num_experts):
                self.ffn(f"{m}.experts.{e}", c.moe_intermediate_size)
            self.ffn(f"{m}.shared_expert", c.moe_intermediate_size)
            self.plain(f"{m}.shared_expert_gate", 1, H)

    def normal(self, shape, std):
        return torch.randn(*shape, generator=self.g, device=self.device) * std

    def norm(self, name, n):
        self.t[f"{name}.weight"] = ((0.0 if self.cfg.norm_plus_one else 1.0) + self.normal((n,), 0.02)).bfloat16()

    def plain(self, name, n, k, std=STD):
        self.t[f"{name}.weight"] = self.normal((n, k), std).bfloat16()

    def ffn(self, name, width):
        H = self.cfg.hidden_size
        self.linear(f"{name}.gate_proj", width, H)
        self.linear(f"{name}.up_proj", width, H)
        self.linear(f"{name}.down_proj", H, width, DOWN_SCALE, STD_OUT)

    def linear(self, name, n, k, input_scale=None, std=STD):
        if self.model == "bf16":
            return self.plain(name, n, k, std)
        w = self.normal((n, k), std)
        if self.model == "nvfp4":
            gs = float(w.abs().amax()) / 2688
            codes, sf = _nvfp4_parts(w, gs)
            self.t[f"{name}.weight"] = codes[:, 0::2] | (codes[:, 1::2] << 4)
            self.t[f"{name}.weight_scale"] = sf.view(torch.uint8)
            self.t[f"{name}.weight_scale_2"] = torch.tensor(gs)
            if input_scale is not None:
                self.t[f"{name}.input_scale"] = torch.tensor(input_scale)
            return
        b = w.view(n // 128, 128, k // 128, 128)
        s = b.abs().amax((1, 3)) / 448
        self.t[f"{name}.weight"] = _e4m3(b / s[:, None, :, None]).view(n, k).view(torch.uint8)
        self.t[f"{name}.weight_scale_inv"] = s

    def values(self, name):
        """The weight that the checkpoint's bytes stand for, in 64 bits."""
        w = self.t[f"{name}.weight"]
        if f"{name}.weight_scale_2" in self.t:
            codes = torch.stack([w & 15, w >> 4], -1).flatten(1)
            return _nvfp4_values(codes, self.t[f"{name}.weight_scale"].view(torch.float8_e4m3fn), float(self.t[f"{name}.weight_scale_2"]))
        if f"{name}.weight_scale_inv" in self.t:
            s = self.t[f"{name}.weight_scale_inv"].double()
            return w.view(torch.float8_e4m3fn).double() * s.repeat_interleave(128, 0).repeat_interleave(128, 1)
        return w.double()


def _inputs(c, cfg, seed, device="cuda"):
    """Token ids, block lists, what the caches and states hold before the pass: (sequences, caches, states)."""
    g = torch.Generator(device=device).manual_seed(seed + 1)
    lens = _lengths(c)
    need = [(n + p + BLOCK - 1) // BLOCK for n, p in lens]
    order = (torch.randperm(sum(need), generator=g, device=device) + 1).tolist()      # block 0 is the engine's null block
    seqs, at = [], 0
    for i, ((n, p), k) in enumerate(zip(lens, need)):
        ids = torch.randint(0, cfg.vocab_size, (n,), generator=g, device=device).tolist()
        seqs.append(dict(tokens=ids, start_pos=p, blocks=order[at:at + k], state_slot=i + 1, logits="all" if 1 < c["new"] <= 5 and p else "last"))
        at += k
    caches, states = [], []
    for kind in cfg.layer_types:
        if kind == "attention":
            kv = []
            for std in (1.0, 1.4):                               # keys are normed, values are a projection's rows
                x = torch.randn(1 + sum(need), BLOCK, cfg.num_kv_heads, cfg.head_dim, generator=g, device=device, dtype=torch.bfloat16) * std
                kv.append(_e4m3(x) if cfg.kv_dtype == "fp8" else x)
            caches.append(kv)
        else:
            C = 2 * cfg.gdn_qk_size + cfg.gdn_v_size
            states.append((torch.randn(len(lens) + 1, C, cfg.conv_kernel - 1, generator=g, device=device),
                           torch.randn(len(lens) + 1, cfg.gdn_v_heads, cfg.gdn_k_dim, cfg.gdn_v_dim, generator=g, device=device) * 0.1))
    return seqs, caches, states


# ----------------------------------------------------------------------------- a pass
class _State:
    pass


def prepare(c, seed):
    from metrale_inference_alpha_b200.engine.batch import ForwardBatch
    from metrale_inference_alpha_b200.engine.llm_engine import EngineArgs, LLMEngine
    from metrale_inference_alpha_b200.weights.source import DictSource
    ck = _Checkpoint(c["model"], seed)
    cfg = ck.cfg
    seqs, caches, states = _inputs(c, cfg, seed)
    blocks = 1 + sum(len(s["blocks"]) for s in seqs)
    longest = max(len(s["tokens"]) + s["start_pos"] for s in seqs)
    s = _State()
    s.engine = LLMEngine(EngineArgs(model=cfg, device="cuda", max_model_len=max(2048, longest), num_kv_blocks=blocks,
                                    enable_prefix_caching=False, state_snapshots=1), source=DictSource(ck.t))
    r = s.engine.runner
    s.model, s.caches = r.decoder, r.caches
    for j, (k, v) in enumerate(caches):
        r.kv.k[j][:blocks].copy_(k.view(torch.uint8) if cfg.kv_dtype == "fp8" else k)
        r.kv.v[j][:blocks].copy_(v.view(torch.uint8) if cfg.kv_dtype == "fp8" else v)
    for j, (conv, ssm) in enumerate(states):
        r.pool.conv[j][:conv.shape[0]].copy_(conv)
        r.pool.ssm[j][:ssm.shape[0]].copy_(ssm)
    s.updated = [(x.view(torch.float8_e4m3fn) if x.dtype == torch.uint8 else x)[1:blocks] for x in r.kv.k + r.kv.v]
    s.states = [x[1:len(seqs) + 1] for x in (r.pool.conv + r.pool.ssm if r.pool is not None else [])]
    s.batch = ForwardBatch.build(seqs, BLOCK, device="cuda", max_blocks=r.max_blocks)
    s.graph = None
    if c["new"] <= 5:                                            # decode and verify steps: replayed, as the engine does
        keep = [x.clone() for x in s.states]
        s.model.forward(s.batch, s.caches)
        torch.cuda.synchronize()
        s.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s.graph):
            s.out = s.model.forward(s.batch, s.caches)
        for x, y in zip(s.states, keep):
            x.copy_(y)
    return s


def run(s):
    if s.graph is not None:
        s.graph.replay()
    else:
        s.out = s.model.forward(s.batch, s.caches)
    return {"logits": s.out[0], "hidden": s.out[1], "cache": s.updated, "state": s.states}


# ----------------------------------------------------------------------------- what a pass cannot do without
def work(c):
    cfg, lens = _config(c["model"]), _lengths(c)
    T, S, H = sum(n for n, _ in lens), len(lens), cfg.hidden_size
    rows = T if 1 < c["new"] <= 5 and c["past"] else S
    wb = {"nvfp4": 0.5625, "bf16": 2.0, "hybrid-fp8": 1.0}[c["model"]]           # bytes a weight
    kvb = 1 if cfg.kv_dtype == "fp8" else 2
    flops, weights = 2.0 * rows * VOCAB * H, 2.0 * VOCAB * H
    nbytes = 2.0 * T * H + 2.0 * rows * (VOCAB + H)
    for kind, ffn in zip(cfg.layer_types, cfg.ffn_types):
        if kind == "attention":
            qo = cfg.num_heads * cfg.head_dim
            n = H * (cfg.q_size + 2 * cfg.kv_size) + qo * H
            pairs = sum(a * b + a * (a + 1) // 2 for a, b in lens)
            flops += 2.0 * T * n + 4.0 * qo * pairs
            nbytes += 2.0 * kvb * cfg.kv_size * (T + sum(b for _, b in lens))
        else:
            v, heads = cfg.gdn_v_size, cfg.gdn_v_heads
            n = H * (2 * cfg.gdn_qk_size + 2 * v + 2 * heads) + v * H
            flops += 2.0 * T * n + 8.0 * T * v * cfg.gdn_k_dim
            nbytes += 4.0 * S * (heads * cfg.gdn_k_dim * cfg.gdn_v_dim) * (2 if c["past"] else 1)
        weights += wb * n
        if ffn == "dense":
            n, used = 3 * H * cfg.intermediate_size, 1.0
            flops += 2.0 * T * n
        else:
            one, E, k = 3 * H * cfg.moe_intermediate_size, cfg.num_experts, cfg.experts_per_token
            used = 1 + E * (1 - (1 - k / E) ** T)                                # experts that some token asks for, and the shared one
            n = one
            flops += 2.0 * T * (one * (k + 1) + H * E)
        weights += wb * n * used
    return {"bytes": nbytes + weights, "flops": flops}


def tolerance(c):
    # Quantised activations turn a last-bit difference into a step of their grid now and then: sums in another order give
    # a few per cent on an e2m1 grid, a few tenths of one on e4m3.
    return {"rel": {"nvfp4": 0.03, "bf16": 0.01, "hybrid-fp8": 0.02}[c["model"]]}


# ----------------------------------------------------------------------------- the same pass in 64 bits
def _quantised(x, model, static=None):
    """What a quantised linear layer reads of its input: the values that the format can hold."""
    if model == "bf16":
        return x
    if model == "nvfp4":
        gs = static if static is not None else x.abs().amax(1, keepdim=True) / 2688
        return _nvfp4_values(*_nvfp4_parts(x, gs), gs)
    b = x.view(x.shape[0], -1, 128)
    s = (b.abs().amax(2, keepdim=True) / 448).clamp(min=1e-300)
    return (_e4m3(b / s).double() * s).view(x.shape)


def _rms(x, w, eps, plus_one=False):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * (w.double() + (1.0 if plus_one else 0.0))


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, pos, dims, base):
    half = dims // 2
    a = pos.double()[:, None] * base ** (-torch.arange(0, dims, 2, dtype=torch.float64, device=x.device) / dims)
    c, s = a.cos()[:, None], a.sin()[:, None]
    x1, x2 = x[..., :half], x[..., half:dims]
    return torch.cat([x1 * c - x2 * s, x2 * c + x1 * s, x[..., dims:]], -1)


def _attention(cfg, ck, p, y, seqs, cache):
    H, G, D = cfg.num_heads, cfg.num_kv_heads, cfg.head_dim
    yq = _quantised(y, ck.model)
    q, k, v = (yq @ ck.values(f"{p}.{n}_proj").t() for n in "qkv")
    gate = None
    if cfg.attn_output_gate:
        q, gate = (t.reshape(len(y), H * D) for t in q.view(len(y), H, 2, D).unbind(2))
    pos = torch.cat([torch.arange(s["start_pos"], s["start_pos"] + len(s["tokens"])) for s in seqs]).to(y.device)
    rot = lambda x, n: _rotate(_rms(x.view(len(y), -1, D), ck.t[f"{p}.{n}_norm.weight"], cfg.rms_eps, cfg.norm_plus_one),
                               pos, cfg.rotary_dim, cfg.rope_theta)
    q, k, v = rot(q, "q"), rot(k, "k"), v.view(len(y), G, D)
    if cfg.kv_dtype == "fp8":
        k, v = _e4m3(k).double(), _e4m3(v).double()
    out, at = torch.empty_like(q), 0
    for s in seqs:
        n, past = len(s["tokens"]), s["start_pos"]
        old = [x[s["blocks"]].reshape(-1, G, D)[:past].double() for x in cache]
        kk, vv = torch.cat([old[0], k[at:at + n]]), torch.cat([old[1], v[at:at + n]])
        seen = torch.arange(past + n, device=y.device)[None] <= pos[at:at + n, None]
        for h in range(G):
            sc = torch.einsum("qhd,kd->hqk", q[at:at + n, h * (H // G):(h + 1) * (H // G)], kk[:, h]) * D ** -0.5
            pr = torch.softmax(sc.masked_fill(~seen[None], float("-inf")), -1)
            out[at:at + n, h * (H // G):(h + 1) * (H // G)] = torch.einsum("hqk,kd->qhd", pr, vv[:, h])
        at += n
    out = out.reshape(len(y), H * D)
    if gate is not None:
        out = out * torch.sigmoid(gate)
    return _quantised(out, ck.model, O_SCALE) @ ck.values(f"{p}.o_proj").t()


def _delta_net(cfg, ck, p, y, seqs, state):
    Hk, Hv, Dk, Dv = cfg.gdn_k_heads, cfg.gdn_v_heads, cfg.gdn_k_dim, cfg.gdn_v_dim
    QK, yq = Hk * Dk, _quantised(y, ck.model)
    x, z = yq @ ck.values(f"{p}.in_proj_qkv").t(), yq @ ck.values(f"{p}.in_proj_z").t()
    b, a = y @ ck.values(f"{p}.in_proj_b").t(), y @ ck.values(f"{p}.in_proj_a").t()
    decay = torch.exp(-ck.t[f"{p}.A_log"].double().exp() * torch.nn.functional.softplus(a + ck.t[f"{p}.dt_bias"].double()))
    beta, taps = torch.sigmoid(b), ck.t[f"{p}.conv1d.weight"].double()[:, 0]
    core, at, windows, mats = torch.empty(len(y), Hv, Dv, dtype=torch.float64, device=y.device), 0, [], []
    unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)
    for i, s in enumerate(seqs):
        n = len(s["tokens"])
        old, h = (t[i + 1].double() if s["start_pos"] else torch.zeros_like(t[i + 1], dtype=torch.float64) for t in state)
        win = torch.cat([old, x[at:at + n].t()], 1)
        c = _silu((win.unfold(1, cfg.conv_kernel, 1) * taps[:, None]).sum(-1).t())
        q, k, v = c[:, :QK].view(n, Hk, Dk), c[:, QK:2 * QK].view(n, Hk, Dk), c[:, 2 * QK:].view(n, Hv, Dv)
        q, k = (unit(t).repeat_interleave(Hv // Hk, 1) for t in (q, k))
        for t in range(n):
            g = decay[at + t, :, None]
            new = (v[t] - g * torch.einsum("hkv,hk->hv", h, k[t])) * beta[at + t, :, None]
            h = g[..., None] * h + k[t][:, :, None] * new[:, None]
            core[at + t] = torch.einsum("hkv,hk->hv", h, q[t]) * Dk ** -0.5
        windows.append(win[:, -(cfg.conv_kernel - 1):])
        mats.append(h)
        at += n
    out = _rms(core, ck.t[f"{p}.norm.weight"], cfg.rms_eps).reshape(len(y), Hv * Dv) * _silu(z)
    return _quantised(out, ck.model) @ ck.values(f"{p}.out_proj").t(), torch.stack(windows), torch.stack(mats)


def _ffn(ck, p, yq):
    h = _silu(yq @ ck.values(f"{p}.gate_proj").t()) * (yq @ ck.values(f"{p}.up_proj").t())
    return _quantised(h, ck.model, DOWN_SCALE) @ ck.values(f"{p}.down_proj").t()


def _experts(cfg, ck, p, y):
    yq = _quantised(y, ck.model)
    w, chosen = torch.softmax(y @ ck.values(f"{p}.gate").t(), -1).topk(cfg.experts_per_token, -1)
    if cfg.router_renormalize:
        w = w / w.sum(-1, keepdim=True)
    out = torch.sigmoid(y @ ck.values(f"{p}.shared_expert_gate").t()) * _ffn(ck, f"{p}.shared_expert", yq)
    for e in chosen.unique().tolist():
        row, col = torch.nonzero(chosen == e, as_tuple=True)
        out.index_add_(0, row, _ffn(ck, f"{p}.experts.{e}", yq[row]) * w[row, col][:, None])
    return out


def exact(c, seed):
    ck = _Checkpoint(c["model"], seed)
    cfg, eps = ck.cfg, ck.cfg.rms_eps
    seqs, caches, states = _inputs(c, cfg, seed)
    ids = torch.tensor([t for s in seqs for t in s["tokens"]], device="cuda")
    x, ai, ri, conv, ssm = ck.t["model.embed_tokens.weight"][ids].double(), 0, 0, [], []
    for i, kind in enumerate(cfg.layer_types):
        p = f"model.layers.{i}"
        y = _rms(x, ck.t[f"{p}.input_layernorm.weight"], eps, cfg.norm_plus_one)
        if kind == "attention":
            x = x + _attention(cfg, ck, f"{p}.self_attn", y, seqs, caches[ai])
            ai += 1
        else:
            o, window, mat = _delta_net(cfg, ck, f"{p}.linear_attn", y, seqs, states[ri])
            x, ri = x + o, ri + 1
            conv.append(window)
            ssm.append(mat)
        y = _rms(x, ck.t[f"{p}.post_attention_layernorm.weight"], eps, cfg.norm_plus_one)
        x = x + (_experts(cfg, ck, f"{p}.mlp", y) if cfg.ffn_types[i] == "moe" else _ffn(ck, f"{p}.mlp", _quantised(y, ck.model)))
    rows, at = [], 0
    for s in seqs:
        n = len(s["tokens"])
        rows += range(at, at + n) if s["logits"] == "all" else [at + n - 1]
        at += n
    x = x[rows]
    logits = _rms(x, ck.t["model.norm.weight"], eps, cfg.norm_plus_one) @ ck.values("lm_head").t()
    # the caches keep their own encodings of what is checked through the logits
    return {"logits": logits, "hidden": x, "cache": [None] * (2 * len(caches)), "state": conv + ssm}
