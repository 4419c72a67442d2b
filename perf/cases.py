"""Steps of the hybrid decoder (gated DeltaNet + grouped-query attention) as a serving loop runs them.

A case is one engine step: one token for each of some running sequences (decode), prompt tokens of some others
(prefill), or both in one batch.  The step goes through the executor that `LLM` builds, on a batch as the scheduler
hands it over, and ends the way a step of a serving loop ends: the host reads the next token of every sequence.

Two sets of layer shapes:
  27b   the layers of preset qwen3.6-27b; one period of its layer pattern (4 of 64 layers) with a sixteenth of its
        vocabulary, so that every kernel has the share of a step that it has in the whole model
  2k    the small hybrid model of the benchmarks (width 2048), half of its 8 layers and of its vocabulary

The caches hold what earlier steps would have left there: keys of unit root mean square, values, recurrent states and
convolution inputs of random content, in blocks scattered over the cache.
"""
import hashlib
import random

import torch

BLOCK = 16
GROUPS = 4                    # states that may be alive at a time (each has blocks and state slots of its own)
SEQS = 64                     # sequences of one state
TOKENS = 65536                # cached tokens of one state
STD = 0.02


GDN, FULL = "linear_attention", "full_attention"
MODELS = {
    "27b": dict(vocab_size=15616, hidden_size=5120, num_layers=4, layer_types=(GDN, GDN, GDN, FULL), intermediate_size=17408,
                num_q_heads=24, num_kv_heads=4, head_dim=256, rotary_dim=64, rope_theta=1e7, gdn_num_k_heads=16,
                gdn_num_v_heads=48, gdn_head_k_dim=128, gdn_head_v_dim=128),
    "2k": dict(vocab_size=32768, hidden_size=2048, num_layers=4, layer_types=(GDN, GDN, FULL, GDN), intermediate_size=6144,
               num_q_heads=16, num_kv_heads=4, head_dim=128, rotary_dim=32, rope_theta=5e5, gdn_num_k_heads=8,
               gdn_num_v_heads=16, gdn_head_k_dim=128, gdn_head_v_dim=128),
}
RMS_EPS = 1e-6


# ------------------------------------------------------------------------------------------------ cases
def _case(name, model, quant, *, state="fp32", decode=0, decode_context=0, prompts="", prompt_context="", layout=1):
    """decode: sequences with one new token each, `decode_context` cached tokens on average (half to one and a half of
    it); prompts: new tokens of each prefilling sequence; prompt_context: what each has in the cache already."""
    d = dict(model=model, quant=quant, state=state, decode=decode, decode_context=decode_context, prompts=prompts,
             prompt_context=prompt_context or ",".join("0" for p in prompts.split(",") if p), layout=layout)
    return dict(name=name, **d) if name else d


def listed():
    return [
        # one user of a small model in bf16: the shortest step there is
        _case("2k-decode-1", "2k", "bf16", decode=1, decode_context=300),
        # some users of a small int8 model
        _case("2k-decode-24", "2k", "w8a16", decode=24, decode_context=700, layout=2),
        # one user of the large model: the headline number of the framework
        _case("decode-1", "27b", "w8a16", decode=1, decode_context=1000),
        # the same behind a long document
        _case("decode-1-long", "27b", "w8a16", decode=1, decode_context=30001),
        # a handful of users
        _case("decode-5", "27b", "w8a16", decode=5, decode_context=2000, layout=3),
        # weights in bf16 and the recurrent states in bf16 too, half a server's worth of users
        _case("decode-32-bf16", "27b", "bf16", state="bf16", decode=32, decode_context=600, layout=4),
        # the 64 concurrent requests of the serving configuration
        _case("decode-64", "27b", "w8a16", decode=64, decode_context=1000, layout=5),
        # time to the first token of a short prompt
        _case("prompt-128", "27b", "w8a16", prompts="128"),
        # several requests of odd lengths that arrived together
        _case("prompts-ragged", "27b", "w8a16", prompts="1531,37,640,211,95,803,18,299"),
        # a chunk of a prompt beside running sequences (chunked prefill)
        _case("mixed", "27b", "w8a16", decode=29, decode_context=900, prompts="1031", prompt_context="512", layout=6),
        # a whole chunk of the scheduler's default size
        _case("prompt-4096", "27b", "w8a16", prompts="4096"),
        # the last chunk of a 32k-token prompt with bf16 weights
        _case("chunk-of-32k-bf16", "27b", "bf16", prompts="4096", prompt_context="28672"),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng: random.Random):
    model = rng.choice(("27b", "27b", "2k"))
    quant = rng.choice(("w8a16", "w8a16", "bf16"))
    state = rng.choice(("fp32", "fp32", "bf16"))
    kind = rng.choice(("decode", "decode", "prompt", "prompts", "mixed"))
    layout = rng.randrange(1, 1 << 20)
    if kind == "decode":
        n = _log_int(rng, 1, SEQS)
        return _case("", model, quant, state=state, decode=n, layout=layout,
                     decode_context=_log_int(rng, 40, min(30000, TOKENS * 2 // 3 // n - BLOCK)))
    if kind == "prompt":
        return _case("", model, quant, state=state, prompts=str(_log_int(rng, 20, 4096)),
                     prompt_context=str(rng.choice((0, 0, BLOCK * _log_int(rng, 1, 1700)))), layout=layout)
    if kind == "prompts":
        lens = [_log_int(rng, 5, 1000) for _ in range(rng.randrange(2, 9))]
        return _case("", model, quant, state=state, prompts=",".join(map(str, lens)), layout=layout)
    return _case("", model, quant, state=state, decode=_log_int(rng, 1, 48), decode_context=_log_int(rng, 40, 600),
                 prompts=str(_log_int(rng, 20, 2000)), prompt_context=str(rng.choice((0, 16 * rng.randrange(1, 200)))), layout=layout)


def _lengths(case):
    """[(new tokens, cached tokens)] of the batch's sequences: running ones first."""
    r, c = random.Random(case["layout"]), case["decode_context"]
    seqs = [(1, c if case["decode"] == 1 else max(1, r.randint(c // 2, c + c // 2))) for _ in range(case["decode"])]
    new = [int(p) for p in case["prompts"].split(",") if p]
    old = [int(p) for p in case["prompt_context"].split(",") if p]
    return seqs + list(zip(new, old))


# ------------------------------------------------------------------------------------------------ inputs
def _inputs(case, seed):
    """What the step starts from, in plain layouts: tokens, cached keys and values, recurrent states, convolution inputs."""
    m, lens = MODELS[case["model"]], _lengths(case)
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + 17)
    na = sum(t == FULL for t in m["layer_types"])
    ng = m["num_layers"] - na
    S, hkv, D = len(lens), m["num_kv_heads"], m["head_dim"]
    hv, dk, dv = m["gdn_num_v_heads"], m["gdn_head_k_dim"], m["gdn_head_v_dim"]
    ch = 2 * m["gdn_num_k_heads"] * dk + hv * dv

    def normal(*shape, std=1.0):
        return torch.empty(*shape, device="cuda").normal_(0.0, std, generator=g)

    T = sum(n for n, _ in lens)
    ids = torch.randint(0, m["vocab_size"], (T,), generator=g, device="cuda")
    kv = []
    for _, c in lens:
        k = normal(na, c, hkv, D)
        k = (k * torch.rsqrt(k.square().mean(-1, keepdim=True) + 1e-6)).bfloat16()
        kv.append((k, normal(na, c, hkv, D, std=STD * m["hidden_size"] ** 0.5).bfloat16()))
    old = torch.tensor([float(c > 0) for _, c in lens], device="cuda")
    rec = normal(ng, S, hv, dk, dv, std=0.02) * old[:, None, None, None]
    if case["state"] == "bf16":
        rec = rec.bfloat16().float()
    conv = (normal(ng, S, 3, ch, std=STD * m["hidden_size"] ** 0.5) * old[:, None, None]).bfloat16()
    # physical blocks: scattered over the state's part of the cache
    need = [-(-(n + c) // BLOCK) for n, c in lens]
    order = list(range(sum(need)))
    random.Random(int(seed) ^ case["layout"]).shuffle(order)
    tables, at = [], 0
    for b in need:
        tables.append(order[at:at + b])
        at += b
    return ids, kv, rec, conv, tables, lens


def _head_conv(m, conv):
    """[.., channels] -> [.., v-heads, (q | k | v) of the head]: the convolution inputs as the state cache keeps them."""
    hk, hv, dk, dv = m["gdn_num_k_heads"], m["gdn_num_v_heads"], m["gdn_head_k_dim"], m["gdn_head_v_dim"]
    q, k, v = conv.split((hk * dk, hk * dk, hv * dv), -1)
    rep = lambda x: x.reshape(*x.shape[:-1], hk, dk).repeat_interleave(hv // hk, dim=-2)  # noqa: E731
    return torch.cat([rep(q), rep(k), v.reshape(*v.shape[:-1], hv, dv)], -1)


def _pages(kv, tables, dtype):
    """Keys and values of every sequence in the cache's pages: [layers, 2, blocks, heads * 16 * D]."""
    na, _, hkv, D = kv[0][0].shape
    out = torch.zeros(na, 2, sum(map(len, tables)), hkv * BLOCK * D, dtype=dtype, device="cuda")
    for (k, v), t in zip(kv, tables):
        n = len(t)
        if not k.shape[1]:
            continue
        full = torch.zeros(2, na, n * BLOCK, hkv, D, dtype=dtype, device="cuda")
        full[0, :, :k.shape[1]], full[1, :, :k.shape[1]] = k, v
        full = full.view(2, na, n, BLOCK, hkv, D)
        idx = torch.tensor(t, device="cuda")
        out[:, 0, idx] = full[0].permute(0, 1, 3, 2, 4).reshape(na, n, -1)
        out[:, 1, idx] = full[1].permute(0, 1, 3, 4, 2).reshape(na, n, -1)
    return out


# ------------------------------------------------------------------------------------------------ the framework's side
class _Engine:
    """The engine of one model, as a server keeps it; its cache is dealt to the states that are alive."""

    def __init__(self, model, quant, state):
        from tileinfer_b200.engine.llm import LLM
        from tileinfer_b200.models.config import ModelConfig
        cfg = ModelConfig(name=f"hybrid-{model}", rms_eps=RMS_EPS, max_position_embeddings=32768 + 4096, **MODELS[model])
        self.per = TOKENS // BLOCK + SEQS
        self.llm = LLM("hybrid", model_config=cfg, quantization=quant, weights="random:0", gdn_state_dtype=state, tokenizer="ids",
                       max_num_seqs=GROUPS * SEQS, cuda_graph_max_batch_size=SEQS, num_kvcache_blocks=GROUPS * self.per,
                       enable_prefix_caching=False)
        self.model = self.llm.model_runner.model
        self.free = list(range(GROUPS))


_engines = {}


class _State:
    group = None

    def __del__(self):
        if self.group is not None:
            self.engine.free.append(self.group)


def prepare(case, seed):
    from tileinfer_b200.models.reference_cpu import Batch
    key = (case["model"], case["quant"], case["state"])
    if key not in _engines:
        _engines[key] = _Engine(*key)
    s = _State()
    s.engine = e = _engines[key]
    s.group = e.free.pop()
    ids, kv, rec, conv, tables, lens = _inputs(case, seed)
    block0, slot0 = s.group * e.per, s.group * SEQS
    blocks = sum(map(len, tables))
    e.model.blocks_in(list(range(block0, block0 + blocks)), _pages(kv, tables, torch.bfloat16))
    conv = _head_conv(MODELS[case["model"]], conv).transpose(2, 3).contiguous()      # [layers, S, heads, 3, channels]
    for i in range(len(lens)):
        e.model.state_in(slot0 + i, (rec[:, i], conv[:, i]))
    cu, pos, slots = [0], [], []
    tables = [[block0 + b for b in t] for t in tables]
    for (n, c), t in zip(lens, tables):
        cu.append(cu[-1] + n)
        pos.extend(range(c, c + n))
        slots.extend(t[p // BLOCK] * BLOCK + p % BLOCK for p in range(c, c + n))
    s.batch = Batch(ids.cpu(), torch.tensor(pos), cu, [n + c for n, c in lens], tables, torch.tensor(slots),
                    list(range(slot0, slot0 + len(lens))), [[] for _ in lens])
    s.new = [slot0 + i for i, (_, c) in enumerate(lens) if c == 0]
    s.out = {"state": e.model.rec[:, slot0:slot0 + len(lens)], "conv": e.model.conv[:, slot0:slot0 + len(lens)],
             "kv": e.model.kv[:, :, block0:block0 + blocks]}
    return s


def run(s):
    model = s.engine.model
    for slot in s.new:                       # a new request starts from an empty recurrent state
        model.zero_state(slot)
    logits = model.step_logits(s.batch)
    logits.argmax(-1).tolist()               # the loop needs the tokens for its next batch
    return dict(s.out, logits=logits)


# ------------------------------------------------------------------------------------------------ what a step cannot do without
def _layer_params(m, full):
    H, D = m["hidden_size"], m["head_dim"]
    mlp = 3 * H * m["intermediate_size"]
    if full:
        return mlp + H * D * (3 * m["num_q_heads"] + 2 * m["num_kv_heads"])
    vd = m["gdn_num_v_heads"] * m["gdn_head_v_dim"]
    return mlp + H * (2 * m["gdn_num_k_heads"] * m["gdn_head_k_dim"] + 3 * vd + 2 * m["gdn_num_v_heads"])


def work(case):
    """Weights once, cached keys and values once (written ones too), recurrent states in and out, logits out."""
    m, lens = MODELS[case["model"]], _lengths(case)
    H, V, S, T = m["hidden_size"], m["vocab_size"], len(lens), sum(n for n, _ in lens)
    hv, dk, dv = m["gdn_num_v_heads"], m["gdn_head_k_dim"], m["gdn_head_v_dim"]
    wb = 1 if case["quant"] == "w8a16" else 2
    sb = 2 if case["state"] == "bf16" else 4
    nbytes, flops = 2 * H * V + 2 * H * T + 4 * V * S, 2 * H * V * S
    for t in m["layer_types"]:
        full = t == FULL
        p = _layer_params(m, full)
        nbytes += wb * p
        flops += 2 * p * T
        if full:
            for n, c in lens:
                nbytes += 2 * (n + c) * m["num_kv_heads"] * m["head_dim"] * 2
                flops += 4 * m["num_q_heads"] * m["head_dim"] * (n * c + n * (n + 1) // 2)
        else:
            nbytes += 2 * S * hv * dk * dv * sb
            flops += 6 * T * hv * dk * dv
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """bf16 activations and residual through four layers of random weights: against 64 bits the logits are off by 0.013 to
    0.020, keys, values and states by up to 0.017 (measured), most of it the residual's rounding.  Two correct
    implementations may be off by as much in different directions."""
    return {"rel": 0.03, "max": 0.9}


# ------------------------------------------------------------------------------------------------ the same step in 64 bits
def _weight(name, shape):
    """The random weights of seed 0: N(0, 0.02) rounded to bf16, one generator per tensor (small tensors on the host)."""
    dev = "cuda" if torch.Size(shape).numel() > 1 << 24 else "cpu"
    g = torch.Generator(device=dev)
    g.manual_seed(int.from_bytes(hashlib.sha256(f"0:{name}".encode()).digest()[:7], "little"))
    return torch.empty(shape, device=dev).normal_(0.0, STD, generator=g).bfloat16().cuda().float()


def _matrix(quant, name, shape):
    w = _weight(name, shape)
    if quant == "w8a16":                     # int8 rows with a bf16 scale
        scale = (w.abs().amax(1).clamp_min(1e-8) / 127.0).bfloat16().float()[:, None]
        w = torch.round(w / scale).clamp_(-128, 127) * scale.double()
    return w.double()


def _norm(x):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + RMS_EPS)


def _rope(x, pos, m):
    half = m["rotary_dim"] // 2
    inv = m["rope_theta"] ** (-torch.arange(half, dtype=torch.float64, device="cuda") / half)
    ang = (pos.double()[:, None] * inv)[:, None, :]
    a, b, rest = x[..., :half], x[..., half:2 * half], x[..., 2 * half:]
    return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin(), rest], -1)


def _attention(m, x, lens, kv, layer, W):
    """Appends the new keys and values to `kv` (lists per sequence) and returns the gated outputs."""
    hq, hkv, D = m["num_q_heads"], m["num_kv_heads"], m["head_dim"]
    H, T = m["hidden_size"], x.shape[0]
    qg = (x @ W("attn.q", (hq * D * 2, H)).t()).view(T, hq, 2, D)
    k = _norm((x @ W("attn.k", (hkv * D, H)).t()).view(T, hkv, D))
    v = (x @ W("attn.v", (hkv * D, H)).t()).view(T, hkv, D)
    pos = torch.cat([torch.arange(c, c + n, device="cuda") for n, c in lens])
    q, k = _rope(_norm(qg[:, :, 0]), pos, m), _rope(k, pos, m)
    out, t0 = torch.empty(T, hq, D, dtype=torch.float64, device="cuda"), 0
    for i, (n, c) in enumerate(lens):
        kk, vv = torch.cat([kv[i][0][layer].double(), k[t0:t0 + n]]), torch.cat([kv[i][1][layer].double(), v[t0:t0 + n]])
        kv[i][2].append((kk, vv))
        for a in range(0, n, 256):
            b = min(n, a + 256)
            L = c + b
            qq = q[t0 + a:t0 + b].view(b - a, hkv, hq // hkv, D)
            s = torch.einsum("tkgd,lkd->kgtl", qq, kk[:L]) * D ** -0.5
            s = s.masked_fill(torch.arange(L, device="cuda") > torch.arange(c + a, c + b, device="cuda")[:, None], -float("inf"))
            out[t0 + a:t0 + b] = torch.einsum("kgtl,lkd->tkgd", s.softmax(-1), vv[:L]).reshape(b - a, hq, D)
        t0 += n
    return (out * torch.sigmoid(qg[:, :, 1])).view(T, hq * D)


def _deltanet(m, x, lens, rec, conv, name, W):
    """Returns the outputs, the states and the convolution inputs after the step."""
    hk, hv, dk, dv = m["gdn_num_k_heads"], m["gdn_num_v_heads"], m["gdn_head_k_dim"], m["gdn_head_v_dim"]
    H, kd, vd, T = m["hidden_size"], hk * dk, hv * dv, x.shape[0]
    raw = x @ W("gdn.in_qkv", (2 * kd + vd, H)).t()
    z = (x @ W("gdn.in_z", (vd, H)).t()).view(T, hv, dv)
    beta = torch.sigmoid(x @ W("gdn.in_b", (hv, H)).t())
    a = x @ W("gdn.in_a", (hv, H)).t()
    w = _weight(name + "gdn.conv_w", (2 * kd + vd, 4)).double()
    decay = torch.exp(-torch.exp(_weight(name + "gdn.A_log", (hv,)).double())
                      * torch.nn.functional.softplus(a + _weight(name + "gdn.dt_bias", (hv,)).double()))
    qkv, hist, starts, t0 = torch.empty_like(raw), [], [], 0
    for i, (n, _) in enumerate(lens):
        seq = torch.cat([conv[i].double(), raw[t0:t0 + n]])
        qkv[t0:t0 + n] = torch.nn.functional.silu(sum(seq[j:j + n] * w[:, j] for j in range(4)))
        hist.append(seq[n:])
        starts.append(t0)
        t0 += n
    unit = lambda y: y * torch.rsqrt(y.square().sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q = unit(qkv[:, :kd].view(T, hk, dk)).repeat_interleave(hv // hk, 1) * dk ** -0.5
    k = unit(qkv[:, kd:2 * kd].view(T, hk, dk)).repeat_interleave(hv // hk, 1)
    v = qkv[:, 2 * kd:].view(T, hv, dv)
    # all sequences advance together, the longest first
    order = sorted(range(len(lens)), key=lambda i: -lens[i][0])
    S = rec[order].double()
    o = torch.empty(T, hv, dv, dtype=torch.float64, device="cuda")
    first, length = torch.tensor([starts[i] for i in order], device="cuda"), [lens[i][0] for i in order]
    for t in range(length[0]):
        live = sum(n > t for n in length)
        at = first[:live] + t
        s = S[:live] * decay[at][:, :, None, None]
        u = (v[at] - torch.matmul(k[at][:, :, None], s)[:, :, 0]) * beta[at][:, :, None]
        s += k[at][..., None] * u[:, :, None]
        S[:live] = s
        o[at] = torch.matmul(q[at][:, :, None], s)[:, :, 0]
    state = torch.empty_like(S)
    state[order] = S
    return (_norm(o) * torch.nn.functional.silu(z)).view(T, vd), state, torch.stack(hist)


@torch.no_grad()
def exact(case, seed):
    m = MODELS[case["model"]]
    ids, kv, rec, conv, tables, lens = _inputs(case, seed)
    kv = [(k, v, []) for k, v in kv]
    H, ff = m["hidden_size"], m["intermediate_size"]
    x = _weight("embed", (m["vocab_size"], H))[ids].double()
    states, hists, g, a = [], [], 0, 0
    for i, kind in enumerate(m["layer_types"]):
        name = f"layers.{i}."
        W = lambda leaf, shape: _matrix(case["quant"], name + leaf, shape)  # noqa: E731, B023
        h = _norm(x)
        if kind == FULL:
            x = x + _attention(m, h, lens, kv, a, W) @ W("attn.o", (H, m["num_q_heads"] * m["head_dim"])).t()
            a += 1
        else:
            y, st, hist = _deltanet(m, h, lens, rec[g], conv[g], name, W)
            x = x + y @ W("gdn.out", (H, y.shape[1])).t()
            states.append(st)
            hists.append(_head_conv(m, hist).transpose(1, 2))
            g += 1
        h = _norm(x)
        x = x + (torch.nn.functional.silu(h @ W("mlp.gate", (ff, H)).t()) * (h @ W("mlp.up", (ff, H)).t())) @ W("mlp.down", (H, ff)).t()
    last = [sum(n for n, _ in lens[:i + 1]) - 1 for i in range(len(lens))]
    logits = _norm(x[last]) @ _weight("lm_head", (m["vocab_size"], H)).double().t()
    pages = _pages([tuple(torch.stack(t) for t in zip(*new)) for _, _, new in kv], tables, torch.float64)
    return {"state": torch.stack(states), "conv": torch.stack(hists), "kv": pages, "logits": logits}
