"""Cases that stand for the work a user has this framework do, each through the public entry points.

  lm      a pre-LayerNorm transformer (OPT / GPT shapes): greedy generation through PipelineModel, or a prompt
          pass alone (new = 1, what a sampler's first token costs)
  block   one Block1D on a whole batch: a causal layer's prompt pass, or an encoder layer with its padding mask
  packed  an attention sublayer on packed tokens put together from the kernel API (padding removed, LayerNorm,
          linear, transposes, softmax, padding rebuilt)
  linear  the kernel API's linear by itself
  design  a decoder of the layer-listed designs: greedy generation and one step more, or a prompt pass alone

Weights are drawn by this file under the names of the reference's modules (lm, block) or of a checkpoint (design),
with projections that keep the scale of their input.  A head's rows are the embedding rows of the tokens that
precede, so that greedy choices are as clear as a trained model's and rounding does not decide them; the
choices among experts stay as close as they come.  Layers have the widths of the named models; their number is
reduced for the large ones."""
import math

import torch
import torch.nn.functional as F

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
VOCAB = 32768                # of the designs
HOP = 7919                   # token t is followed by token t + HOP


# ---- the cases --------------------------------------------------------------------------------------------
def listed():
    return [
        # one user's chat request to a small model: 12 layers of launches around almost no work
        dict(name="opt125m_chat", kind="lm", hidden=768, heads=12, depth=12, vocab=50272, act="relu", fused=False, batch=1, prompt=37, new=32, dtype="fp16"),
        # a served batch of a small GPT, odd vocabulary
        dict(name="gpt2_batch", kind="lm", hidden=768, heads=12, depth=12, vocab=50257, act="gelu_tanh", fused=True, batch=8, prompt=128, new=32, dtype="bf16"),
        # a served batch at the headline model's layer shape: long left-padded prompts, then steps that stream the weights
        dict(name="opt13b_batch", kind="lm", hidden=5120, heads=40, depth=4, vocab=50272, act="relu", fused=False, batch=16, prompt=512, new=48, dtype="fp16"),
        # few long prompts of odd length, first token only
        dict(name="opt6b_prompt", kind="lm", hidden=4096, heads=32, depth=4, vocab=50272, act="relu", fused=False, batch=3, prompt=1931, new=1, dtype="bf16"),
        # the prompt pass of one layer of the widest model
        dict(name="gpt3_layer", kind="block", hidden=12288, heads=96, act="gelu_tanh", causal=True, post=False, batch=8, seq=1024, dtype="fp16"),
        # an encoder layer over a right-padded batch of odd length
        dict(name="bert_layer", kind="block", hidden=1024, heads=16, act="gelu", causal=False, post=True, batch=32, seq=389, dtype="fp16"),
        # the same layer's attention on packed tokens, from the kernel API
        dict(name="packed_attention", kind="packed", hidden=1024, heads=16, causal=False, batch=32, seq=512, dtype="fp16"),
        # a small product by itself: the call with the least work
        dict(name="linear_small", kind="linear", batch=4, seq=37, din=1024, dout=4096, dtype="bf16"),
        # the designs: a served batch over latent attention and routed experts
        dict(name="tulezen_batch", kind="design", design="tulezen", depth=4, batch=8, prompt=301, new=48, dtype="bf16"),
        # long prompts through matrix memory and grouped attention
        dict(name="mutolix_prompt", kind="design", design="mutolix", depth=4, batch=4, prompt=1999, new=1, dtype="bf16"),
        # a served batch over state spaces, chunk attention, gated linear attention and routed experts
        dict(name="moponex_batch", kind="design", design="moponex", depth=4, batch=16, prompt=200, new=48, dtype="bf16"),
        # a replay in true 32-bit: selective scan, capped and rotary latent attention
        dict(name="tupidra_fp32", kind="design", design="tupidra", depth=4, batch=1, prompt=333, new=1, dtype="fp32"),
    ]


def spread(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["lm", "lm", "lm", "block", "block", "packed", "linear", "design", "design", "design"])
    if kind == "linear":
        return dict(kind=kind, batch=spread(rng, 1, 16), seq=spread(rng, 1, 256), din=8 * spread(rng, 96, 1536), dout=8 * spread(rng, 96, 3072),
                    dtype=rng.choice(["fp16", "bf16"]))
    if kind == "packed":
        heads = rng.choice([12, 16])
        return dict(kind=kind, hidden=64 * heads, heads=heads, causal=rng.random() < 0.5, batch=spread(rng, 1, 32), seq=spread(rng, 24, 512),
                    dtype=rng.choice(["fp16", "bf16"]))
    if kind == "block":
        hidden, heads = rng.choice([(768, 12), (1024, 16), (1536, 12), (3072, 24), (5120, 40), (7168, 56), (12288, 96)])
        tokens = spread(rng, 64, min(16384, 8192 * 12288 // hidden))
        seq = max(16, min(tokens, spread(rng, 32, 2048)))
        post = rng.random() < 0.4
        return dict(kind=kind, hidden=hidden, heads=heads, act=rng.choice(["relu", "gelu", "gelu_tanh"]), causal=not post, post=post,
                    batch=max(1, tokens // seq), seq=seq, dtype=rng.choice(["fp16", "bf16"]))
    new = 1 if rng.random() < 0.4 else spread(rng, 8, 48)
    if kind == "lm":
        hidden, heads, most = rng.choice([(768, 12, 12), (1024, 16, 12), (1536, 12, 12), (3072, 24, 6), (4096, 32, 4), (5120, 40, 4)])
        batch = spread(rng, 1, 32)
        return dict(kind=kind, hidden=hidden, heads=heads, depth=rng.randint(max(1, most // 2), most), vocab=rng.choice([50272, 50257]),
                    act=rng.choice(["relu", "gelu_tanh"]), fused=rng.random() < 0.5, batch=batch,
                    prompt=spread(rng, 16, max(32, min(2000, 8192 // batch))), new=new, dtype=rng.choice(["fp16", "bf16"]))
    design, dtype = rng.choice(["tulezen", "mutolix", "moponex", "tupidra"]), rng.choice(["bf16", "bf16", "bf16", "fp32"])
    batch = spread(rng, 1, 32 if dtype == "bf16" else 3)
    return dict(kind=kind, design=design, depth=rng.choice([2, 4]), batch=batch, prompt=spread(rng, 16, min(2048, 8192 // batch) if dtype == "bf16" else 400),
                new=new if dtype == "bf16" else min(new, 16), dtype=dtype)


# ---- weights and inputs, from the seed alone ---------------------------------------------------------------
class Drawer:
    """Random tensors on the GPU in the case's type."""

    def __init__(self, case, seed):
        self.g = torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)
        self.dtype, self.t = DTYPES[case["dtype"]], {}

    def randn(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda")

    def mat(self, name, rows, cols, gain=1.0):
        self.t[name] = (self.randn(rows, cols) * (gain / cols ** 0.5)).to(self.dtype)

    def vec(self, name, n, mean=0.0, spread=0.1):
        self.t[name] = (mean + spread * self.randn(n)).to(self.dtype)

    def linear(self, name, rows, cols, gain=1.0):
        self.mat(name + ".weight", rows, cols, gain)
        self.vec(name + ".bias", rows)

    def norm(self, name, n):
        self.vec(name + ".module.weight", n, 1.0)
        self.vec(name + ".module.bias", n)


def lengths(case, seed, longest):
    """True lengths of a batch, on the host: uniform over the upper half, one of them full."""
    g = torch.Generator().manual_seed(7 * seed + 3)
    n = torch.randint(max(1, longest // 2), longest + 1, (case["batch"],), generator=g)
    n[0] = longest
    return n.tolist()


def prompts(case, seed, vocab):
    """(ids, mask) of a left-padded batch; prompts alone come in one length."""
    S, g = case["prompt"], torch.Generator().manual_seed(11 * seed + 5)
    lens = lengths(case, seed, S) if case["new"] > 1 else [S] * case["batch"]
    ids = torch.randint(2, vocab, (case["batch"], S), generator=g)
    mask = torch.ones_like(ids)
    for r, n in enumerate(lens):
        ids[r, :S - n], mask[r, :S - n] = 1, 0
    return ids.cuda(), mask.cuda(), lens


def successor(ids, vocab):
    return 2 + (ids - 2 + HOP) % (vocab - 2)


def head_of(embed, vocab):
    """Rows of the head: row t is the embedding of the token that t follows, at the scale of a unit input."""
    t = torch.arange(vocab, device=embed.device)
    before = torch.where(t < 2, t, 2 + (t - 2 - HOP) % (vocab - 2))
    return (embed[before].float() / embed.shape[1] ** 0.5).to(embed.dtype)


def block_weights(d, p, h, fused):
    d.norm(p + "norm1", h)
    if fused:
        d.linear(p + "attn.query_key_value", 3 * h, h, 1.2)
    else:
        for n in ("query_", "key_", "value_"):
            d.linear(p + "attn." + n, h, h, 1.2)
    d.linear(p + "attn.dense", h, h, 0.5)
    d.norm(p + "norm2", h)
    d.linear(p + "mlp.dense_1", 4 * h, h)
    d.linear(p + "mlp.dense_2", h, 4 * h, 0.5)


def lm_weights(case, seed):
    d, h, V = Drawer(case, seed), case["hidden"], case["vocab"]
    d.mat("embed.word_embeddings.weight", V, h, h ** 0.5)
    d.mat("embed.position_embeddings.weight", 2050, h, 0.3 * h ** 0.5)
    for i in range(case["depth"]):
        block_weights(d, f"blocks.{i}.", h, case["fused"])
    d.norm("norm", h)
    d.t["head.dense.weight"] = head_of(d.t["embed.word_embeddings.weight"], V)
    return d.t


def design_config(case):
    """Layers of the sizes of the designs' benchmark at width 2048; two kinds alternate (three for tupidra, in fours)."""
    n, W = case["depth"], 2048
    cfg = {"vocab": VOCAB, "width": W, "norm": {"eps": 1e-5}}
    if case["design"] == "tulezen":
        cfg["layers"] = [{"type": "latent_attention", "mixer": {"heads": 16, "dim": 128, "vdim": 128, "kv_rank": 512, "mask": {"size": 1024}, "scale": 128 ** -0.5,
                                                                **({"kv_from": i - 1} if i % 2 else {})},
                          "mlp": {"kind": "moe", "router": {"experts": 64, "top": 6}, "expert": {"ff": 1408, "limit": 7.0}}} for i in range(n)]
    elif case["design"] == "mutolix":
        memory = {"type": "mlstm", "mixer": {"heads": 8, "dim": 128, "vdim": 256, "gate_cap": 15.0}, "mlp": None}
        attention = {"type": "attention", "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                                                    "q_temp": {"coef": 0.1, "every": 512}, "v_mix": True}, "mlp": {"kind": "dense", "ff": 8192}}
        cfg.update(embedding={"scale": 1.0}, layers=[memory, attention] * (n // 2))
    elif case["design"] == "moponex":
        par = {"type": "parallel", "mlp": {"kind": "dense", "ff": 5632},
               "mixer": {"left": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024},
                                  "rot": {"dims": 64, "base": 5e5, "scaling": {"factor": 4.0}}},
                         "right": {"heads": 8, "dim": 128, "vdim": 256, "tau": 12.0, "rank": 16}}}
        ssm = {"type": "mamba2", "mixer": {"heads": 64, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1},
               "mlp": {"kind": "moe", "expert": {"ff": 1024}, "shared": {"ff": 2048},
                       "router": {"experts": 62, "top": 6, "identity": 2, "groups": {"count": 8, "keep": 4}}}}
        cfg.update(residual_mult=0.8, logit_scale=0.25, layers=[par, ssm] * (n // 2),
                   embedding={"bigram": {"buckets": VOCAB - 1, "mul_prev": 1021, "mul_cur": 13}})
    else:
        ff = {"kind": "dense", "ff": 5632}
        scan = {"type": "mamba1", "mlp": ff, "mixer": {"inner": 4096, "state": 16, "dt_rank": 128, "conv": 4}}
        att = {"type": "attention", "mlp": ff, "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 30.0,
                                                         "mask": {"size": 1024, "keep_first": 64}}}
        rot = {"dims": 32, "base": 10000.0, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}
        lat = {"type": "latent_attention", "mlp": ff, "mixer": {"heads": 32, "dim": 64, "rot_dim": 32, "vdim": 64, "q_rank": 768, "kv_rank": 256,
                                                                "scale": 96 ** -0.5, "rot": rot}}
        shared = {"type": "latent_attention", "mlp": ff, "mixer": dict(lat["mixer"], kv_from=2)}
        cfg.update(canon={"taps": 4}, layers=[scan, att, lat, shared][:n])
    return cfg


def design_weights(case, seed):
    """A checkpoint's tensors.  Decays are mostly slow, so that far tokens count.  Tulezen's norms behind its sublayers, which set how much
    each adds to the stream, are small, as those of a deep model are; other norm weights lie near their neutral value."""
    cfg, d, what = design_config(case), Drawer(case, seed), case["design"]
    W, V, mat, vec = cfg["width"], cfg["vocab"], d.mat, d.vec
    mat("embed", V, W, W ** 0.5)
    if what != "moponex":
        d.t["head"] = head_of(d.t["embed"], V)
    else:
        mat("bigram", V, W, 0.5 * W ** 0.5)
    vec("final.norm", W, 0.0 if what == "tulezen" else 1.0)
    for i, ly in enumerate(cfg["layers"]):
        p, m, f = f"l{i}.", ly["mixer"], ly["mlp"]
        q = p + "mix."
        vec(p + "norm1", W, -0.75 if what == "tulezen" else 1.0, 0.05 if what == "tulezen" else 0.1)
        if what == "tulezen":
            H, R = m["heads"], m["kv_rank"]
            mat(q + "q", H * 128, W, 1.2)
            if "kv_from" not in m:
                mat(q + "dkv", R, W)
                vec(q + "dkv.norm", R, 1.0)
            mat(q + "uk", H * 128, R, 1.2)
            mat(q + "uv", H * 128, R)
            mat(q + "o", W, H * 128)
            vec(p + "norm2", W, -0.75, 0.05)
            mat(p + "mlp.router", f["router"]["experts"], W, 2.5)
            for e in range(f["router"]["experts"]):
                for n, r, c in (("gate", f["expert"]["ff"], W), ("up", f["expert"]["ff"], W), ("down", W, f["expert"]["ff"])):
                    mat(f"{p}mlp.e{e}.{n}", r, c)
        elif what == "mutolix":
            for s in ("1", "2") if f else ("1",):
                if s == "2":
                    vec(p + "norm2", W, 1.0)
                vec(f"{p}norm{s}b", W, 1.0)
                vec(f"{p}ls{s}", W, 0.8)
                mat(f"{p}rg{s}", W, W)
                vec(f"{p}rg{s}.b", W, 1.0)
            H, k, v = m["heads"], m["dim"], m["vdim"]
            if ly["type"] == "mlstm":
                for n, r in (("q", k), ("k", k), ("v", v), ("g", v)):
                    mat(q + n, H * r, W)
                mat(q + "o", W, H * v)
                vec(q + "norm", H * v, 1.0)
                mat(q + "i", H, W)
                vec(q + "i.b", H, -0.5, 1.0)
                mat(q + "f", H, W)
                vec(q + "f.b", H, 4.0, 1.5)
            else:
                for n, r in (("q", H * k), ("k", m["kv_heads"] * k), ("v", m["kv_heads"] * v)):
                    mat(q + n, r, W)
                    vec(f"{q}{n}.b", r)
                vec(q + "q.norm", H * k, 1.2)
                vec(q + "k.norm", m["kv_heads"] * k, 1.2)
                vec(q + "vmix", 1, 0.5)
                d.t[q + "vmix"] = d.t[q + "vmix"].reshape(())
                d.t[q + "r1"] = torch.rand(H, generator=d.g, device="cuda").to(d.dtype)
                d.t[q + "r2"] = (torch.rand(H, generator=d.g, device="cuda") * 0.5 + 0.05).to(d.dtype)
                mat(q + "o", W, H * v)
                mat(p + "mlp.up", f["ff"], W)
                mat(p + "mlp.down", W, f["ff"])
                d.t[p + "mlp.act"] = torch.tensor([0.8, -0.9], device="cuda").to(d.dtype)
        elif what == "moponex":
            if ly["type"] == "mamba2":
                H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
                C = H * P + 2 * G * N
                mat(q + "in", H * P + C + H, W)
                mat(q + "conv", C, m["conv"])
                vec(q + "conv.b", C)
                vec(q + "dt_bias", H, -2.0, 0.7)
                vec(q + "A_log", H, -1.0, 1.0)
                vec(q + "D", H, 0.7)
                vec(q + "norm", H * P, 1.0)
                mat(q + "o", W, H * P, 0.7)
            else:
                a, r = m["left"], m["right"]
                for n, c in (("q", a["heads"]), ("k", a["kv_heads"])):
                    mat(q + "left." + n, c * a["dim"], W)
                    vec(f"{q}left.{n}.b", c * a["dim"])
                    vec(f"{q}left.{n}.norm", a["dim"], 1.2)
                vec(q + "left.sink", a["heads"], 1.0, 1.0)
                mat(q + "left.o", W, a["heads"] * a["dim"])
                for n, c in (("q", r["dim"]), ("k", r["dim"]), ("v", r["vdim"]), ("g", r["vdim"])):
                    mat(q + "right." + n, r["heads"] * c, W)
                mat(q + "right.a1", r["rank"], W)
                mat(q + "right.a2", r["heads"] * r["dim"], r["rank"])
                vec(q + "right.a2.b", r["heads"] * r["dim"], 1.5, 1.5)
                vec(q + "right.norm", r["vdim"], 1.0)
                mat(q + "right.o", W, r["heads"] * r["vdim"])
                vec(q + "left.out", W, 0.8)
                vec(q + "right.out", W, 0.8)
            vec(p + "norm2", W, 1.0)
            if f["kind"] == "dense":
                for n, r, c in (("gate", f["ff"], W), ("up", f["ff"], W), ("down", W, f["ff"])):
                    mat(p + "mlp." + n, r, c)
            else:
                E, n = f["router"]["experts"], f["router"]["experts"] + f["router"]["identity"]
                mat(p + "mlp.router", n, W, 3.0)
                vec(p + "mlp.correction", n, -1.0, 0.01)
                for e in range(E):
                    mat(f"{p}mlp.e{e}.up", f["expert"]["ff"], W)
                    mat(f"{p}mlp.e{e}.down", W, f["expert"]["ff"])
                mat(p + "mlp.shared.up", f["shared"]["ff"], W)
                mat(p + "mlp.shared.down", W, f["shared"]["ff"])
                mat(p + "mlp.shared.sg", 1, W)
        else:
            mat(p + "canon1", W, 4, 0.4)
            if ly["type"] == "mamba1":
                C, N, R = m["inner"], m["state"], m["dt_rank"]
                mat(q + "in", 2 * C, W)
                mat(q + "conv", C, m["conv"])
                vec(q + "conv.b", C)
                mat(q + "x", R + 2 * N, C, 0.8)
                mat(q + "dt", C, R)
                vec(q + "dt.b", C, -3.0, 0.7)
                d.t[q + "A_log"] = (d.randn(C, N) - 0.5).to(d.dtype)
                vec(q + "D", C, 0.7)
                mat(q + "o", W, C, 0.5)
            elif ly["type"] == "attention":
                H, G, k, v = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
                for n, r in (("q", H * k), ("k", G * k), ("v", G * v)):
                    mat(q + n, r, W)
                    vec(f"{q}{n}.b", r)
                mat(q + "g", H * v, W)
                mat(q + "o", W, H * v, 1.5)
                vec(q + "o.b", W)
            else:
                H, k, r, v, qr, kr = (m[n] for n in ("heads", "dim", "rot_dim", "vdim", "q_rank", "kv_rank"))
                mat(q + "dq", qr, W)
                vec(q + "dq.norm", qr, 1.0)
                mat(q + "uq", H * (k + r), qr)
                if "kv_from" not in m:
                    mat(q + "dkv", kr + r, W)
                    vec(q + "dkv.norm", kr, 1.0)
                mat(q + "uk", H * k, kr)
                mat(q + "uv", H * v, kr)
                vec(q + "sink", H, 1.0, 1.0)
                mat(q + "g", H * v, W)
                mat(q + "o", W, H * v, 1.5)
            vec(p + "norm2", W, 1.0)
            mat(p + "canon2", W, 4, 0.4)
            for n, r, c in (("gate", f["ff"], W), ("up", f["ff"], W), ("down", W, f["ff"])):
                mat(p + "mlp." + n, r, c)
    return d.t


def block_inputs(case, seed):
    """(weights, hidden states, additive mask or None, true lengths)."""
    d, h, B, S = Drawer(case, seed), case["hidden"], case["batch"], case["seq"]
    block_weights(d, "", h, True)
    x = d.randn(B, S, h).to(d.dtype)
    lens = lengths(case, seed, S) if not case["causal"] else [S] * B
    mask = None
    if not case["causal"]:
        keep = torch.arange(S, device="cuda")[None, :] < torch.tensor(lens, device="cuda")[:, None]
        mask = ((~keep).to(d.dtype) * -10000.0).view(B, 1, 1, S)
    return d.t, x, mask, lens


def packed_inputs(case, seed):
    d, h, B, S = Drawer(case, seed), case["hidden"], case["batch"], case["seq"]
    for n in "qkvo":
        d.mat(n, h, h, 1.2)
    d.vec("gamma", h, 1.0)
    d.vec("beta", h)
    if case["causal"]:
        d.t["q"] = (d.t["q"].float() * 0.125).to(d.dtype)         # the call's softmax applies no scale of its own
    lens = lengths(case, seed, S)
    keep = torch.arange(S, device="cuda")[None, :] < torch.tensor(lens, device="cuda")[:, None]
    return d.t, (d.randn(B, S, h) * keep[:, :, None]).to(d.dtype), lens


def linear_inputs(case, seed):
    d = Drawer(case, seed)
    d.mat("w", case["dout"], case["din"])
    return d.randn(case["batch"], case["seq"], case["din"]).to(d.dtype), d.t["w"]


# ---- what a user's program has in hand ----------------------------------------------------------------------
def activation(name):
    from energonai_b200.model.mlp import gelu_impl
    return {"relu": F.relu, "gelu": F.gelu, "gelu_tanh": gelu_impl}[name]


def prepare(case, seed):
    dtype, kind = DTYPES[case["dtype"]], case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "linear":
        s["x"], s["w"] = linear_inputs(case, seed)
    elif kind == "packed":
        from energonai_b200.kernel import LayerNorm
        w, s["x"], lens = packed_inputs(case, seed)
        s["w"], s["tokens"], s["lens"] = w, sum(lens), torch.tensor(lens, dtype=torch.int32, device="cuda")
        s["norm"] = LayerNorm(case["hidden"], device="cuda", dtype=dtype)
        s["norm"].load_state_dict({"weight": w["gamma"], "bias": w["beta"]})
    elif kind == "block":
        from energonai_b200.model import Block1D
        w, s["x"], s["mask"], _ = block_inputs(case, seed)
        with torch.device("cuda"):
            s["block"] = Block1D(case["hidden"], case["heads"], 4.0, activation=activation(case["act"]), dtype=dtype, max_seq_len=case["seq"],
                                 apply_post_layernorm=case["post"], is_decoder=case["causal"], disable_past_cache=not case["causal"]).eval()
        s["block"].load_state_dict(w)
    elif kind == "lm":
        from energonai_b200.model import create_pipeline_model
        with torch.device("cuda"):
            s["model"] = create_pipeline_model(depth=case["depth"], vocab_size=case["vocab"], hidden_size=case["hidden"], num_heads=case["heads"], max_seq_len=2050,
                                               activation=activation(case["act"]), fused_qkv=case["fused"], dtype=dtype).eval()
        s["model"].load_state_dict(lm_weights(case, seed))
        s["model"].eos_token_id = -1                  # random tokens name no end
        s["ids"], s["mask"], _ = prompts(case, seed, case["vocab"])
    else:
        from energonai_b200 import utils
        from energonai_b200.registry import build_model
        name, cfg = case["design"].capitalize(), design_config(case)
        with torch.device("cuda"):
            s["model"] = build_model(name, config_dict=cfg, dtype=dtype, device="cuda").eval()
            s["model"].load_state_dict(getattr(utils, "processing_" + name)(design_weights(case, seed), s["model"]))
        s["ids"], s["mask"], _ = prompts(case, seed, VOCAB)
    return s


# ---- one pass -------------------------------------------------------------------------------------------------
@torch.inference_mode()
def run(s):
    case = s["case"]
    if s["kind"] == "linear":
        from energonai_b200.kernel import linear
        return linear(s["x"], s["w"])
    if s["kind"] == "packed":
        return run_packed(s)
    if s["kind"] == "block":
        return s["block"](s["x"], attention_mask=s["mask"], first_cache=True)
    model, S = s["model"], case["prompt"]
    if case["new"] == 1 and s["kind"] == "design":
        stream = model.prompt(s["ids"], reserve=64)
        return {"stream": stream, "logits": model.logits(stream.view(case["batch"], S, -1)[:, -1].contiguous())}
    record = {"allow_graph": True}
    tokens = model(input_ids=s["ids"], attention_mask=s["mask"], max_tokens=S + case["new"] if case["new"] > 1 else None, top_k=1, record=record)
    out = {"tokens": tokens, "logits": record["logits"][0]}
    if case["new"] > 1 and s["kind"] == "design":
        out["after"] = model.step(tokens[:, -1])                  # the conversation goes on: reads everything the steps left behind
    elif case["new"] > 1:
        out["cache"] = [b.attn.past_cache.buf[:, S:S + case["new"] - 1] for b in model.blocks]      # the rows that the steps appended
    return out


def run_packed(s):
    from energonai_b200 import kernel as K
    from energonai_b200._lib import SM_ALLROWS, SM_KEYLEN
    case, x, lens, V = s["case"], s["x"], s["lens"], s["tokens"]
    B, S, H, h = case["batch"], case["seq"], case["heads"], case["hidden"]
    valid = torch.zeros(1, dtype=torch.int32, device="cuda")
    offsets, scratch = (torch.empty(B * S, dtype=torch.int32, device="cuda") for _ in range(2))
    K.ft_build_padding_offsets(lens, B, S, valid, offsets)
    y = s["norm"](K.ft_remove_padding(x, offsets, scratch, V, h))
    q, k, v = (K.transpose_pad(K.linear(y, s["w"][n]).view(1, V, H, h // H), B, S, lens, H, h // H) for n in "qkv")
    scores = torch.matmul(q, k.transpose(-1, -2))
    if case["causal"]:
        probs = K.scale_mask_softmax(B, S, H, scores, lens)
    else:
        probs = K.scale_mask_softmax(B, S, H, scores, lens, flags=SM_KEYLEN | SM_ALLROWS, scale=(h // H) ** -0.5)
    ctx = K.transpose_depad(torch.matmul(probs, v), B, V, S, lens, H, h // H)
    return K.ft_rebuild_padding(K.linear(ctx.view(1, V, h), s["w"]["o"]), scratch, V, h, B, S)


# ---- work and tolerances ---------------------------------------------------------------------------------------
def sizes(case):
    """(numbers in the matrices that every token meets, {layer: (experts, top, numbers of one)}, head's numbers, per-token numbers kept
    for later steps, multiply-adds per pair of positions)."""
    if case["kind"] == "lm":
        h = case["hidden"]
        return case["depth"] * 12 * h * h, {}, case["vocab"] * h, case["depth"] * 2 * h, case["depth"] * 2 * h
    W, dense, routed, kept, pairs = 2048, 0, {}, 0, 0
    for i, ly in enumerate(design_config(case)["layers"]):
        m, f, t = ly["mixer"], ly["mlp"], ly["type"]
        if t == "latent_attention" and case["design"] == "tulezen":
            dense += W * 2048 * 2 + (0 if "kv_from" in m else W * 512) + 2 * 2048 * 512
            kept += 0 if "kv_from" in m else 512
            pairs += 2 * 2048
        elif t == "latent_attention":
            dense += W * 768 + 768 * 32 * 96 + (0 if "kv_from" in m else W * 288) + 256 * 32 * 128 + W * 2048 * 2
            kept += 0 if "kv_from" in m else 288
            pairs += 32 * (96 + 64)
        elif t == "mlstm":
            dense += W * (2 * 1024 + 2 * 2048) + 2048 * W + W * W
        elif t == "attention":
            dense += W * (16 + 2 * 4) * 128 + 2048 * W + W * W
            kept += 2 * 4 * 128
            pairs += 2 * 2048
        elif t == "parallel":
            dense += W * (16 + 4) * 128 + 2048 * W + W * (2 * 1024 + 2 * 2048 + 16) + 16 * 1024 + 2048 * W
            kept += 2 * 4 * 128
            pairs += 2 * 2048
        elif t == "mamba2":
            dense += W * (2 * 4096 + 256 + 64) + 4096 * W
        else:
            dense += W * 2 * 4096 + 4096 * 160 + 128 * 4096 + 4096 * W
        if f and f["kind"] == "dense":
            dense += (2 if case["design"] == "mutolix" else 3) * W * f["ff"] + (W * W if case["design"] == "mutolix" else 0)
        elif f:
            n = f["router"]["experts"]
            dense += W * n + 2 * W * f.get("shared", {"ff": 0})["ff"]
            routed[i] = (n, f["router"]["top"], (3 if case["design"] == "tulezen" else 2) * W * f["expert"]["ff"])
    return dense, routed, VOCAB * W, kept, pairs


def work(case):
    e = 4 if case["dtype"] == "fp32" else 2
    if case["kind"] == "linear":
        M, N, K = case["batch"] * case["seq"], case["dout"], case["din"]
        return {"bytes": e * (M * K + N * K + M * N), "flops": 2.0 * M * N * K}
    B, h = case["batch"], case.get("hidden")
    if case["kind"] in ("packed", "block"):
        S = case["seq"]
        M, mats = B * S, 12 if case["kind"] == "block" else 4
        if case["kind"] == "packed" or not case["causal"]:
            M = round(0.75 * M)
        return {"bytes": e * (mats * h * h + 2 * B * S * h), "flops": 2.0 * M * mats * h * h + 4.0 * M * (S / 2 if case["causal"] else 0.75 * S) * h}
    S, new = case["prompt"], case["new"]
    dense, routed, head, kept, pairs = sizes(case)
    tokens = B * S * (0.75 if new > 1 else 1.0)
    steps = new - 1 + (1 if case["kind"] == "design" and new > 1 else 0)
    chosen = lambda n: sum(E * size * (1 - (1 - top / E) ** n) for E, top, size in routed.values())
    active = sum(top * size for _, top, size in routed.values())
    return {"bytes": e * (dense + chosen(tokens) + head + tokens * kept + steps * (dense + chosen(B) + head + B * kept * 0.75 * S)),
            "flops": 2.0 * (dense + active) * (tokens + steps * B) + 2.0 * head * B * (1 + steps) + 2.0 * pairs * tokens * (S / 2 + steps * B / max(1.0, tokens) * S)}


def tolerance(case):
    """About four times what one last place more or less in two of a hundred embeddings, or another order of the sums, makes of the
    outputs; behind routers a few choices fall the other way."""
    if case["dtype"] == "fp32":
        return {"rel": 1e-5, "max": 1e-3, "differ": 0.0}
    if case["kind"] == "linear":
        return {"rel": 2e-3, "max": 0.02}
    if case["kind"] in ("packed", "block"):
        return {"rel": 2e-3 if case["dtype"] == "fp16" else 0.01, "max": 0.25}
    if case["kind"] == "lm":
        return {"rel": 5e-3 if case["dtype"] == "fp16" else 0.03, "max": 0.2, "differ": 0.0}
    return {"rel": 0.03, "max": 0.9, "differ": 0.0}


# ---- the same in 64 bits -----------------------------------------------------------------------------------------
def unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def gelu_tanh(x):
    return F.gelu(x, approximate="tanh")


def layer_norm(x, w, name):
    return F.layer_norm(x, (x.shape[-1],), w[name + ".module.weight"], w[name + ".module.bias"], 1e-5)


def causal_seen(n):
    return torch.ones(n, n, dtype=torch.bool, device="cuda").tril()


def attend(q, k, v, scale, seen, bias=None, sink=None, cap=None):
    """q [n, H, d], k / v [n, G, .] of one sequence -> [n, H * dv]; sink [H]: a score without a value in every denominator."""
    share = torch.arange(q.shape[1], device="cuda") // (q.shape[1] // k.shape[1])
    s = torch.einsum("ihd,jhd->hij", q, k[:, share]) * scale
    if cap:
        s = cap * torch.tanh(s / cap)
    if bias is not None:
        s = s - bias
    s = s.masked_fill(~seen, float("-inf"))
    if sink is not None:
        s = torch.cat([s, sink[:, None, None].expand(-1, s.shape[1], 1)], 2)
    p = torch.softmax(s, -1)[:, :, :k.shape[0]]
    return torch.einsum("hij,jhd->ihd", p, v[:, share]).flatten(1)


def plain_block(x, w, p, case, keep, first_norm_residual=False):
    """One sequence through a block; keep [n] marks the keys that count.  -> (rows, [key | value | query])."""
    n, H, act = x.shape[0], case["heads"], {"relu": F.relu, "gelu": F.gelu, "gelu_tanh": gelu_tanh}[case["act"]]
    lin = lambda y, name: F.linear(y, w[p + name + ".weight"], w[p + name + ".bias"])
    y = layer_norm(x, w, p + "norm1")
    kvq = lin(y, "attn.query_key_value") if p + "attn.query_key_value.weight" in w else torch.cat([lin(y, "attn." + m) for m in ("key_", "value_", "query_")], 1)
    k, v, q = (t.view(n, H, -1) for t in kvq.chunk(3, 1))
    seen = keep[None, :].expand(n, n)
    a = attend(q, k, v, q.shape[-1] ** -0.5, seen & causal_seen(n) if case.get("causal", True) else seen)
    x = (y if first_norm_residual else x) + lin(a, "attn.dense")
    y = layer_norm(x, w, p + "norm2")
    return (y if first_norm_residual else x) + lin(act(lin(y, "mlp.dense_1")), "mlp.dense_2"), kvq


def plain_lm(case, w, ids, start):
    """Logits of every position of one sequence whose first token stands at `start`, and its keys, values and queries."""
    x = w["embed.word_embeddings.weight"][ids] + w["embed.position_embeddings.weight"][start:start + len(ids)]
    keep, rows = torch.ones(len(ids), dtype=torch.bool, device="cuda"), []
    for i in range(case["depth"]):
        x, kvq = plain_block(x, w, f"blocks.{i}.", case, keep)
        rows.append(kvq)
    return x, lambda at: layer_norm(x[at], w, "norm") @ w["head.dense.weight"].T, rows


def conv(x, w):
    """x [n, c], w [c, taps]: causal, the last column of w is the current token's."""
    return F.conv1d(F.pad(x.t()[None], (w.shape[1] - 1, 0)), w[:, None], groups=w.shape[0])[0].t()


def rotate(x, freq, factor=1.0):
    """Neighbouring pairs of the first 2 * len(freq) dimensions turn by position * frequency."""
    a = torch.arange(x.shape[0], dtype=torch.float64, device="cuda")[:, None] * torch.tensor(freq, dtype=torch.float64, device="cuda")
    c, s = factor * torch.cos(a)[:, None], factor * torch.sin(a)[:, None]
    n, out = 2 * len(freq), x.clone()
    u, v = x[..., 0:n:2], x[..., 1:n:2]
    out[..., 0:n:2], out[..., 1:n:2] = u * c - v * s, v * c + u * s
    return out


def yarn(rot):
    d, base, sc = rot["dims"], rot["base"], rot["scaling"]
    turns = lambda t: d * math.log(sc["original"] / (2 * math.pi * t)) / (2 * math.log(base))
    lo, hi = max(math.floor(turns(sc["fast"])), 0), min(math.ceil(turns(sc["slow"])), d - 1)
    ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(d // 2)]
    return [base ** (-2.0 * i / d) * (r / sc["factor"] + 1 - r) for i, r in enumerate(ramp)], 0.1 * math.log(sc["factor"]) + 1


def plain_tulezen(i, ly, x, w, kept, eps):
    m, f, n = ly["mixer"], ly["mlp"], x.shape[0]
    if "kv_from" not in m:
        kept[i] = unit(x @ w["mix.dkv"].T, eps) * w["mix.dkv.norm"]
    c, pos = kept[m.get("kv_from", i)], torch.arange(n, device="cuda")
    q, k, v = ((a @ w["mix." + b].T).view(n, m["heads"], -1) for a, b in ((x, "q"), (c, "uk"), (c, "uv")))
    seen = causal_seen(n) & (pos[:, None] - pos[None, :] < m["mask"]["size"])
    x = x + unit(attend(q, k, v, m["scale"], seen) @ w["mix.o"].T, eps) * (1 + w["norm1"])
    weight, index = torch.softmax(x @ w["mlp.router"].T, -1).topk(f["router"]["top"], -1)
    y = torch.zeros_like(x)
    for e in range(f["router"]["experts"]):
        at, place = (index == e).nonzero(as_tuple=True)
        g, u = x[at] @ w[f"mlp.e{e}.gate"].T, x[at] @ w[f"mlp.e{e}.up"].T
        g, u = g.clamp(max=f["expert"]["limit"]), u.clamp(-f["expert"]["limit"], f["expert"]["limit"])
        y.index_add_(0, at, weight[at, place, None] * ((g * torch.sigmoid(1.702 * g) * (u + 1)) @ w[f"mlp.e{e}.down"].T))
    return x + unit(y, eps) * (1 + w["norm2"])


def plain_mutolix(i, ly, x, w, kept, eps):
    m, n, H = ly["mixer"], x.shape[0], ly["mixer"]["heads"]
    h = unit(x, eps) * w["norm1"]
    part = lambda name: (h @ w["mix." + name].T).view(n, H, -1)
    if ly["type"] == "mlstm":
        q, k, v = part("q") / m["dim"] ** 0.5, part("k"), part("v")
        soft = lambda a: m["gate_cap"] * torch.tanh(a / m["gate_cap"])
        log_i, log_f = soft(h @ w["mix.i"].T + w["mix.i.b"]), F.logsigmoid(soft(h @ w["mix.f"].T + w["mix.f.b"]))
        S, z, top, rows = x.new_zeros(H, m["dim"], m["vdim"]), x.new_zeros(H, m["dim"]), x.new_zeros(H), []
        for t in range(n):
            new = torch.maximum(log_f[t] + top, log_i[t])
            a, b, top = torch.exp(log_f[t] + top - new), torch.exp(log_i[t] - new), new
            bk = b[:, None] * k[t]
            S = torch.baddbmm(a[:, None, None] * S, bk[:, :, None], v[t][:, None, :])
            z = a[:, None] * z + bk
            den = torch.maximum((z * q[t]).sum(-1).abs(), torch.exp(-top)) + 1e-6
            rows.append(torch.bmm(q[t][:, None], S)[:, 0] / den[:, None])
        y = (unit(torch.stack(rows), eps).flatten(1) * w["mix.norm"] * torch.sigmoid(h @ w["mix.g"].T)) @ w["mix.o"].T
    else:
        G, p = m["kv_heads"], torch.arange(n, device="cuda")
        raw = {a: h @ w["mix." + a].T + w[f"mix.{a}.b"] for a in "qkv"}
        q, k = ((unit(raw[a], eps) * w[f"mix.{a}.norm"]).view(n, c, -1) for a, c in (("q", H), ("k", G)))
        v = raw["v"].view(n, G, -1)
        q = q * (1 + m["q_temp"]["coef"] * torch.log((p + 1).div(m["q_temp"]["every"], rounding_mode="floor").double() + 1))[:, None, None]
        if "v" not in kept:
            kept["v"] = v
        else:
            v = (1 - w["mix.vmix"]) * v + w["mix.vmix"] * kept["v"]
        gap = (p[:, None] - p[None, :]).clamp(min=0).double()
        bias = w["mix.r1"][:, None, None] * torch.log1p(w["mix.r2"][:, None, None] * gap)
        y = attend(q, k, v, m["scale"], causal_seen(n), bias=bias, sink=x.new_zeros(H)) @ w["mix.o"].T
    x = x + unit(y * torch.sigmoid(h @ w["rg1"].T + w["rg1.b"]), eps) * w["norm1b"] * w["ls1"]
    if ly["mlp"] is None:
        return x
    h = unit(x, eps) * w["norm2"]
    z, (a, b) = h @ w["mlp.up"].T, F.softplus(w["mlp.act"])
    z = torch.where(z > 0, a * z * z + z / 2, (0.5 + b) * (torch.expm1(z.clamp(max=0)) - z) + z / 2)
    return x + unit((z @ w["mlp.down"].T) * torch.sigmoid(h @ w["rg2"].T + w["rg2.b"]), eps) * w["norm2b"] * w["ls2"]


def plain_moponex(i, ly, x, w, kept, eps):
    m, f, n = ly["mixer"], ly["mlp"], x.shape[0]
    h = unit(x, eps) * w["norm1"]
    if ly["type"] == "mamba2":
        H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
        z, xbc, dt = (h @ w["mix.in"].T).split([H * P, H * P + 2 * G * N, H], 1)
        u, B, C = F.silu(conv(xbc, w["mix.conv"]) + w["mix.conv.b"]).split([H * P, G * N, G * N], 1)
        of = torch.arange(H, device="cuda") // (H // G)
        u, B, C, dt = u.view(n, H, P), B.view(n, G, N)[:, of], C.view(n, G, N)[:, of], F.softplus(dt + w["mix.dt_bias"], threshold=1e9)
        decay, S, rows = torch.exp(-torch.exp(w["mix.A_log"]) * dt), x.new_zeros(H, N, P), []
        for t in range(n):
            S = torch.baddbmm(decay[t][:, None, None] * S, (dt[t][:, None] * B[t])[:, :, None], u[t][:, None, :])
            rows.append(torch.bmm(C[t][:, None], S)[:, 0])
        y = (torch.stack(rows) + w["mix.D"][:, None] * u).flatten(1) * F.silu(z)
        y = (unit(y.view(n, m["norm_groups"], -1), eps).flatten(1) * w["mix.norm"]) @ w["mix.o"].T
    else:
        a, r, p = m["left"], m["right"], torch.arange(n, device="cuda")
        q = (h @ w["mix.left.q"].T + w["mix.left.q.b"]).view(n, a["heads"], -1)
        v = (h @ w["mix.left.k"].T + w["mix.left.k.b"]).view(n, a["kv_heads"], -1)
        freq = [a["rot"]["base"] ** (-2.0 * j / a["rot"]["dims"]) / a["rot"]["scaling"]["factor"] for j in range(a["rot"]["dims"] // 2)]
        q, k = (rotate(unit(t, eps) * w[f"mix.left.{c}.norm"], freq) for t, c in ((q, "q"), (v, "k")))
        size = a["mask"]["size"]
        seen = causal_seen(n) & (p[:, None].div(size, rounding_mode="floor") == p[None, :].div(size, rounding_mode="floor"))
        left = attend(q, k, v, a["scale"], seen, sink=w["mix.left.sink"]) @ w["mix.left.o"].T
        part = lambda name: (h @ w["mix.right." + name].T).view(n, r["heads"], -1)
        q, k, v = part("q") / r["dim"] ** 0.5, part("k"), part("v")
        decay = torch.exp(F.logsigmoid((h @ w["mix.right.a1"].T) @ w["mix.right.a2"].T + w["mix.right.a2.b"]).view(n, r["heads"], -1) / r["tau"])
        S, rows = x.new_zeros(r["heads"], r["dim"], r["vdim"]), []
        for t in range(n):
            S = torch.baddbmm(decay[t][:, :, None] * S, k[t][:, :, None], v[t][:, None, :])
            rows.append(torch.bmm(q[t][:, None], S)[:, 0])
        o = (unit(torch.stack(rows), eps) * w["mix.right.norm"]).flatten(1)
        right = (o * F.silu(h @ w["mix.right.g"].T)) @ w["mix.right.o"].T
        y = (unit(left, eps) * w["mix.left.out"] + unit(right, eps) * w["mix.right.out"]) / 2
    x = x + 0.8 * y
    h = unit(x, eps) * w["norm2"]
    if f["kind"] == "dense":
        return x + 0.8 * ((gelu_tanh(h @ w["mlp.gate"].T) * (h @ w["mlp.up"].T)) @ w["mlp.down"].T)
    r = f["router"]
    s = torch.softmax(h @ w["mlp.router"].T, -1)
    c, groups = s + w["mlp.correction"], r["groups"]["count"]
    best = c.view(n, groups, -1).amax(-1).topk(r["groups"]["keep"], -1).indices
    allowed = torch.zeros(n, groups, dtype=torch.bool, device="cuda").scatter_(1, best, True).repeat_interleave(c.shape[1] // groups, 1)
    index = c.masked_fill(~allowed, float("-inf")).topk(r["top"], -1).indices
    weight = s.gather(1, index)
    weight = weight / (weight.sum(-1, keepdim=True) + 1e-20)
    y = torch.sigmoid(h @ w["mlp.shared.sg"].T) * (F.gelu(h @ w["mlp.shared.up"].T) @ w["mlp.shared.down"].T)
    for e in range(c.shape[1]):
        at, place = (index == e).nonzero(as_tuple=True)
        z = h[at] if e >= r["experts"] else F.gelu(h[at] @ w[f"mlp.e{e}.up"].T) @ w[f"mlp.e{e}.down"].T
        y = y.index_add(0, at, weight[at, place, None] * z)
    return x + 0.8 * y


def plain_tupidra(i, ly, x, w, kept, eps):
    m, n = ly["mixer"], x.shape[0]
    mixed = lambda k: (lambda h: h + conv(h, w["canon" + k]))(unit(x, eps) * w["norm" + k])
    h, g = mixed("1"), mixed("2")
    if ly["type"] == "mamba1":
        u, z = (h @ w["mix.in"].T).chunk(2, 1)
        u = F.silu(conv(u, w["mix.conv"]) + w["mix.conv.b"])
        dt, B, C = (u @ w["mix.x"].T).split([m["dt_rank"], m["state"], m["state"]], 1)
        dt = F.softplus(dt @ w["mix.dt"].T + w["mix.dt.b"], threshold=1e9)
        A, rows = -torch.exp(w["mix.A_log"]), []
        S = torch.zeros_like(A)
        for t in range(n):
            S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * u[t])[:, None] * B[t]
            rows.append(S @ C[t])
        y = ((torch.stack(rows) + w["mix.D"] * u) * F.silu(z)) @ w["mix.o"].T
    elif ly["type"] == "attention":
        H, G, p = m["heads"], m["kv_heads"], torch.arange(n, device="cuda")
        q, k, v = ((h @ w["mix." + a].T + w[f"mix.{a}.b"]).view(n, c, -1) for a, c in (("q", H), ("k", G), ("v", G)))
        gap = p[:, None] - p[None, :]
        slope = 2.0 ** (-8.0 * (torch.arange(H, device="cuda", dtype=torch.float64) + 1) / H)
        seen = (gap >= 0) & ((gap < m["mask"]["size"]) | (p[None, :] < m["mask"]["keep_first"]))
        o = attend(q, k, unit(v, eps), m["scale"], seen, bias=slope[:, None, None] * gap.double(), sink=x.new_zeros(H), cap=m["softcap"])
        y = (o * torch.sigmoid(h @ w["mix.g"].T)) @ w["mix.o"].T + w["mix.o.b"]
    else:
        H, d = m["heads"], m["dim"]
        freq, factor = yarn(m["rot"])
        if "kv_from" not in m:
            c, kr = (h @ w["mix.dkv"].T).split([m["kv_rank"], m["rot_dim"]], 1)
            kept[i] = unit(c, eps) * w["mix.dkv.norm"], rotate(kr[:, None], freq, factor)
        c, kr = kept[m.get("kv_from", i)]
        q = ((unit(h @ w["mix.dq"].T, eps) * w["mix.dq.norm"]) @ w["mix.uq"].T).view(n, H, -1)
        q = torch.cat([q[:, :, :d], rotate(q[:, :, d:], freq, factor)], 2)
        k = torch.cat([(c @ w["mix.uk"].T).view(n, H, d), kr.expand(n, H, -1)], 2)
        o = attend(q, k, (c @ w["mix.uv"].T).view(n, H, -1), m["scale"], causal_seen(n), sink=w["mix.sink"])
        y = (o * torch.sigmoid(h @ w["mix.g"].T)) @ w["mix.o"].T
    return x + y + (gelu_tanh(g @ w["mlp.gate"].T) * (g @ w["mlp.up"].T)) @ w["mlp.down"].T


def plain_design(case, w, ids):
    """Stream of one sequence behind the last layer, and its logits at given places."""
    cfg, what = design_config(case), case["design"]
    eps, kept, x = cfg["norm"]["eps"], {}, w["embed"][ids].double()
    if what == "moponex":
        bg = cfg["embedding"]["bigram"]
        rows = (torch.cat([ids[:1], ids[:-1]]) * bg["mul_prev"] + ids * bg["mul_cur"]) % bg["buckets"]
        rows[0] = bg["buckets"]
        x = x + w["bigram"][rows]
    layer = {"tulezen": plain_tulezen, "mutolix": plain_mutolix, "moponex": plain_moponex, "tupidra": plain_tupidra}[what]
    for i, ly in enumerate(cfg["layers"]):
        p = f"l{i}."
        x = layer(i, ly, x, {k[len(p):]: v.double() for k, v in w.items() if k.startswith(p)}, kept, eps)
    norm, head = 1 + w["final.norm"] if what == "tulezen" else w["final.norm"], w["head"] if "head" in w else w["embed"]
    return x, lambda at: (unit(x[at], eps) * norm) @ head.T.double() * cfg.get("logit_scale", 1.0)


@torch.inference_mode()
def exact(case, seed):
    kind = case["kind"]
    if kind == "linear":
        x, w = linear_inputs(case, seed)
        return F.linear(x.double(), w.double())
    if kind == "packed":
        w, x, lens = packed_inputs(case, seed)
        w, H, d, out = {k: v.double() for k, v in w.items()}, case["heads"], case["hidden"] // case["heads"], torch.zeros_like(x, dtype=torch.float64)
        for r, n in enumerate(lens):
            y = F.layer_norm(x[r, :n].double(), (case["hidden"],), w["gamma"], w["beta"], 1e-5)
            q, k, v = ((y @ w[a].T).view(n, H, d) for a in "qkv")
            seen = causal_seen(n) if case["causal"] else torch.ones(n, n, dtype=torch.bool, device="cuda")
            out[r, :n] = attend(q, k, v, 1.0 if case["causal"] else d ** -0.5, seen) @ w["o"].T
        return out
    if kind == "block":
        w, x, _, lens = block_inputs(case, seed)
        w, S = {k: v.double() for k, v in w.items()}, case["seq"]
        return torch.stack([plain_block(x[r].double(), w, "", case, torch.arange(S, device="cuda") < n, case["post"])[0] for r, n in enumerate(lens)])
    vocab = case["vocab"] if kind == "lm" else VOCAB
    ids, _, lens = prompts(case, seed, vocab)
    w = lm_weights(case, seed) if kind == "lm" else design_weights(case, seed)
    if kind == "lm":
        w = {k: v.double() for k, v in w.items()}
    S, new = case["prompt"], case["new"]
    out = {k: [] for k in ("stream", "tokens", "logits", "after", "cache")}
    for r, n in enumerate(lens):
        seq = [ids[r, S - n:]]
        for _ in range(new - 1 + (1 if kind == "design" and new > 1 else 0)):         # what greedy choices give, see below
            seq.append(successor(seq[-1][-1:], vocab) if case.get("design") != "moponex" else seq[-1][-1:])
        seq = torch.cat(seq)
        if kind == "lm":
            x, logits, rows = plain_lm(case, w, seq, S - n)
            out["cache"].append([t[n:] for t in rows])
        else:
            x, logits = plain_design(case, w, seq)
        got = logits(slice(n - 1, None))
        picked = got[:new].argmax(-1)
        if not torch.equal(picked[:len(seq) - n], seq[n:]):
            return None                                                                 # the forced tokens are not the greedy ones
        out["stream"].append(x)
        out["logits"].append(got[0])
        out["after"].append(got[-1])
        out["tokens"].append(picked)
    put = lambda k: torch.stack(out[k])
    if new == 1:
        return {"tokens": put("tokens")[:, 0], "logits": put("logits")} if kind == "lm" else {"stream": put("stream").flatten(0, 1), "logits": put("logits")}
    result = {"tokens": torch.cat([ids, put("tokens")], 1), "logits": put("logits")}
    if kind == "lm":
        result["cache"] = [torch.stack([c[i] for c in out["cache"]]) for i in range(case["depth"])]
    else:
        result["after"] = put("after")
    return result
