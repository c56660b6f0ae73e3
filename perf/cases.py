"""Cases whose speed is watched: what a program that uses this engine has it do.

Whole steps go through ``ModelRunner.step`` (the only forward pass of the package), with CUDA graphs for decoded tokens as in
serving; single layers go through a part's ``forward`` over a step's ``StepContext``.  Sizes are those of ``bench.py`` (the
layers of Qwen3-0.6B, -8B and -32B, and the mixers and experts that its other designs have at the widths of the first two).
Kinds of cases:

``decode``     one decoded token for each of ``batch`` requests that hold about ``context`` tokens, through ``layers`` layers
               of a Qwen3 model and its head; the cache is filled with random keys and values
``prompt``     one prompt of ``tokens`` tokens through ``layers`` layers of a Qwen3 model; logits of its last token
``attention``  an attention layer in a mixed step: a prompt portion of ``tokens`` tokens of a request that already holds
               ``context`` beside ``batch`` requests that decode one token each
``latent``     a latent attention layer (``parts/latent_attention.py``) on prompts
``experts``    a routed feed-forward (``parts/moe.py``)
``mamba2``, ``mlstm``, ``gla``, ``delta``   a recurrent mixer on prompts: the new requests' states start at zero

``exact`` restates each of them in float64 with torch alone.
"""
import math

import torch

from arle_b200.cache import CacheManager
from arle_b200.config import config_from_dict
from arle_b200.engine import ModelRunner, StepEntry
from arle_b200.engine.batch import StepContext, Workspace
from arle_b200.parts import build_part
from arle_b200.parts.attention import AttentionSpec
from arle_b200.parts.delta_rule import GatedDeltaRuleSpec
from arle_b200.parts.latent_attention import LatentAttentionSpec
from arle_b200.parts.linear_attention import GatedLinearAttentionSpec
from arle_b200.parts.mamba2 import Mamba2Spec
from arle_b200.parts.mlp import GatedMlpSpec
from arle_b200.parts.mlstm import MatrixLstmSpec
from arle_b200.parts.moe import RoutedExpertsSpec
from arle_b200.parts.registry import build_model
from arle_b200.parts.rotary import RotarySpec

DEV = "cuda"
PAGE = 16
EPS = 1e-6
THETA = 1e6

QWEN = {"0.6b": dict(hidden=1024, heads=16, kv=8, ff=3072, vocab=151936, tied=True),
        "8b": dict(hidden=4096, heads=32, kv=8, ff=12288, vocab=32768, tied=False),
        "32b": dict(hidden=5120, heads=64, kv=8, ff=25600, vocab=32768, tied=False)}
LATENT = {"0.6b": dict(hidden=1024, heads=16, dim=64, rot=32, vdim=64, rank=256, q_rank=512),
          "8b": dict(hidden=4096, heads=32, dim=128, rot=64, vdim=128, rank=512, q_rank=1536)}
EXPERTS = {"0.6b": dict(hidden=1024, experts=16, top=4, ff=768, groups=4, keep=2),
           "8b": dict(hidden=4096, experts=32, top=4, ff=3072, groups=4, keep=2)}
MAMBA2 = {"0.6b": dict(hidden=1024, heads=32, vdim=64, state=128, groups=1),
          "8b": dict(hidden=4096, heads=128, vdim=64, state=128, groups=8)}
MLSTM = {"0.6b": dict(hidden=1024, heads=8, dim=64, vdim=128), "8b": dict(hidden=4096, heads=8, dim=256, vdim=512)}
GLA = {"0.6b": dict(hidden=1024, heads=8, dim=128, rank=16), "8b": dict(hidden=4096, heads=16, dim=128, rank=64)}
DELTA = {"0.6b": dict(hidden=1024, heads=8, kq=4, dim=128), "8b": dict(hidden=4096, heads=32, kq=16, dim=128)}


def listed():
    return [
        # a chat with the smallest model, one user: a step of some 140 small kernels, where launches and latency count
        dict(name="decode_0.6b_b1", kind="decode", sizes="0.6b", layers=28, batch=1, context=1153, dtype="bfloat16"),
        # the benchmark's own workload (batch 8, 2,048-token contexts), on the first 8 of the 36 layers
        dict(name="decode_8b_b8", kind="decode", sizes="8b", layers=8, batch=8, context=2048, dtype="bfloat16"),
        # a busy server: 64 requests of different lengths
        dict(name="decode_8b_b64", kind="decode", sizes="8b", layers=8, batch=64, context=2048, dtype="bfloat16"),
        # a prompt of the benchmark's length
        dict(name="prompt_8b_2048", kind="prompt", sizes="8b", layers=4, tokens=2048, dtype="bfloat16"),
        # a prompt cut into portions while other requests decode
        dict(name="attention_32b_mixed", kind="attention", sizes="32b", tokens=512, context=1536, batch=8, dtype="bfloat16"),
        # the float32 engine, which reads bfloat16 checkpoints: a short prompt of odd length
        dict(name="prompt_0.6b_float32", kind="prompt", sizes="0.6b", layers=4, tokens=301, dtype="float32"),
        # the other designs' layers on prompts of the benchmark's length, and on several shorter ones in one step
        dict(name="latent_8b_2048", kind="latent", sizes="8b", tokens=2048, rows=1, q_latent=True, window=0, dtype="bfloat16"),
        dict(name="experts_8b_2048", kind="experts", sizes="8b", tokens=2048, dtype="bfloat16"),
        # the same experts for a step of decoded tokens: every expert is read for a few rows
        dict(name="experts_8b_64", kind="experts", sizes="8b", tokens=64, dtype="bfloat16"),
        dict(name="mamba2_8b_2048", kind="mamba2", sizes="8b", tokens=2048, rows=1, dtype="bfloat16"),
        dict(name="delta_8b_1999", kind="delta", sizes="8b", tokens=1999, rows=3, dtype="bfloat16"),
        dict(name="gla_8b_2048", kind="gla", sizes="8b", tokens=2048, rows=1, dtype="bfloat16"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prompt", "attention", "latent", "experts", "mamba2", "mlstm", "gla", "delta"])
    c = dict(kind=kind, sizes=rng.choice(["0.6b", "8b"]), dtype="bfloat16")
    if kind == "decode":
        return dict(c, layers=rng.choice([4, 6, 8]), batch=_log(rng, 1, 64), context=_log(rng, 16, 2048))
    if kind == "prompt":
        if rng.random() < 0.25:
            return dict(c, sizes="0.6b", layers=rng.choice([2, 3, 4]), tokens=_log(rng, 2, 301), dtype="float32")
        return dict(c, layers=rng.choice([2, 3, 4]), tokens=_log(rng, 16, 2048))
    if kind == "attention":
        return dict(c, sizes=rng.choice(["0.6b", "8b", "32b"]), tokens=_log(rng, 2, 1024), context=_log(rng, 16, 2048), batch=rng.choice([0, 1, 3, 8, 16]))
    if kind == "experts":
        return dict(c, tokens=_log(rng, 1, 2048))
    tokens = _log(rng, 32, 2048)
    c = dict(c, tokens=tokens, rows=rng.choice([1, 1, 2, 3, 4]))
    if kind == "latent":
        c = dict(c, q_latent=rng.random() < 0.5, window=rng.choice([0, 0, 512, 1024]))
    return c


# ---------------------------------------------------------------------------- inputs
class _Maker:
    """Seeded tensors on the GPU, in the order in which they are asked for."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(int(seed) * 7919 + 13)

    def normal(self, *shape, std=1.0, dtype=torch.bfloat16):
        return torch.empty(shape, dtype=dtype, device=DEV).normal_(0.0, std, generator=self.g)

    def matrix(self, *shape):
        return self.normal(*shape, std=0.02)

    def uniform(self, lo, hi, *shape):
        return torch.empty(shape, dtype=torch.float32, device=DEV).uniform_(lo, hi, generator=self.g)

    def gain(self, n):
        return self.uniform(0.9, 1.1, n).to(torch.bfloat16)


def _row_lens(case):
    """The step's prompts: ``rows`` pieces of different lengths that are ``tokens`` together."""
    n, r = case["tokens"], case.get("rows", 1)
    cuts = [0] + [min(n - (r - i), max(i, int(n * (i / r) ** 1.3))) for i in range(1, r)] + [n]
    return [b - a for a, b in zip(cuts, cuts[1:])]


def _contexts(case):
    """Tokens that each decoding request holds: the stated number, or about it when there are more than 8."""
    c, b = case["context"], case["batch"]
    return [c if b <= 8 else max(1, c - (i * 37) % max(1, c // 2)) for i in range(b)]


def _qwen_layer(m, z, p):
    h, hd = z["hidden"], 128
    return {p + "input_layernorm.weight": m.gain(h), p + "self_attn.q_proj.weight": m.matrix(z["heads"] * hd, h),
            p + "self_attn.k_proj.weight": m.matrix(z["kv"] * hd, h), p + "self_attn.v_proj.weight": m.matrix(z["kv"] * hd, h),
            p + "self_attn.o_proj.weight": m.matrix(h, z["heads"] * hd), p + "self_attn.q_norm.weight": m.gain(hd),
            p + "self_attn.k_norm.weight": m.gain(hd), p + "post_attention_layernorm.weight": m.gain(h),
            p + "mlp.gate_proj.weight": m.matrix(z["ff"], h), p + "mlp.up_proj.weight": m.matrix(z["ff"], h),
            p + "mlp.down_proj.weight": m.matrix(h, z["ff"])}


def _qwen_inputs(case, seed):
    """(weights, token ids, keys and values [layers][2] of what the requests hold [tokens, kv, 128] side by side)."""
    z, L = QWEN[case["sizes"]], case["layers"]
    m = _Maker(seed)
    w = {"model.embed_tokens.weight": m.normal(z["vocab"], z["hidden"], std=0.02 if z["tied"] else 1.0), "model.norm.weight": m.gain(z["hidden"])}
    if not z["tied"]:
        w["lm_head.weight"] = m.matrix(z["vocab"], z["hidden"])
    for i in range(L):
        w.update(_qwen_layer(m, z, f"model.layers.{i}."))
    g = torch.Generator().manual_seed(seed)
    if case["kind"] == "decode":
        ids = torch.randint(0, z["vocab"], (case["batch"],), generator=g).tolist()
        held = sum(_contexts(case))
        dt = getattr(torch, case["dtype"])
        kv = [[m.normal(held, z["kv"], 128, dtype=dt), m.normal(held, z["kv"], 128, std=0.5, dtype=dt)] for _ in range(L)]
        return w, ids, kv
    return w, torch.randint(0, z["vocab"], (case["tokens"],), generator=g).tolist(), None


def _qwen_config(case):
    z = QWEN[case["sizes"]]
    return dict(architectures=["Qwen3ForCausalLM"], num_hidden_layers=case["layers"], hidden_size=z["hidden"], num_attention_heads=z["heads"],
                num_key_value_heads=z["kv"], head_dim=128, intermediate_size=z["ff"], vocab_size=z["vocab"], rope_theta=THETA, rms_norm_eps=EPS,
                tie_word_embeddings=z["tied"], max_position_embeddings=40960, hidden_act="silu")


def _attention_inputs(case, seed):
    z = QWEN[case["sizes"]]
    m = _Maker(seed)
    w = _qwen_layer(m, dict(z, ff=8), "")
    lens, starts = [case["tokens"]] + [1] * case["batch"], [case["context"]] + [max(1, case["context"] + 101 * i) for i in range(case["batch"])]
    x = m.normal(sum(lens), z["hidden"])
    kv = [m.normal(sum(starts), z["kv"], 128), m.normal(sum(starts), z["kv"], 128, std=0.5)]
    return {k[len("self_attn."):]: v for k, v in w.items() if k.startswith("self_attn.")}, x, kv, lens, starts


def _dt_bias(m, n):
    """A bias that makes softplus(bias) log-uniform in [0.001, 0.1], as such layers are initialised."""
    dt = torch.exp(m.uniform(math.log(1e-3), math.log(0.1), n))
    return dt + torch.log(-torch.expm1(-dt))


def _mixer_inputs(case, seed):
    """(weights, x [tokens, hidden]) of a latent attention, a routed feed-forward or a recurrent mixer."""
    m, kind = _Maker(seed), case["kind"]
    if kind == "latent":
        z = LATENT[case["sizes"]]
        hn, qd = z["hidden"], z["heads"] * (z["dim"] + z["rot"])
        w = {"dq": m.matrix(z["q_rank"], hn), "dq.norm": m.gain(z["q_rank"]), "uq": m.matrix(qd, z["q_rank"])} if case["q_latent"] else {"q": m.matrix(qd, hn)}
        w.update({"dkv": m.matrix(z["rank"] + z["rot"], hn), "dkv.norm": m.gain(z["rank"]), "uk": m.matrix(z["heads"] * z["dim"], z["rank"]),
                  "uv": m.matrix(z["heads"] * z["vdim"], z["rank"]), "o": m.matrix(hn, z["heads"] * z["vdim"])})
    elif kind == "experts":
        z = EXPERTS[case["sizes"]]
        hn, ff = z["hidden"], z["ff"]
        w = {"router": m.matrix(z["experts"], hn), "correction": m.uniform(-0.1, 0.1, z["experts"])}
        for p in [f"e{i}." for i in range(z["experts"])] + ["shared."]:
            w.update({p + "gate": m.matrix(ff, hn), p + "up": m.matrix(ff, hn), p + "down": m.matrix(hn, ff)})
        w["shared.sg"] = m.matrix(1, hn)
    elif kind == "mamba2":
        z = MAMBA2[case["sizes"]]
        hn, H = z["hidden"], z["heads"]
        inner, ch = H * z["vdim"], H * z["vdim"] + 2 * z["groups"] * z["state"]
        w = {"in": m.matrix(inner + ch + H, hn), "conv": m.uniform(-0.5, 0.5, ch, 4), "conv.b": m.uniform(-0.1, 0.1, ch), "dt_bias": _dt_bias(m, H),
             "A_log": torch.log(m.uniform(1.0, 16.0, H)), "D": m.gain(H).float(), "norm": m.gain(inner), "o": m.matrix(hn, inner)}
    elif kind == "mlstm":
        z = MLSTM[case["sizes"]]
        hn, H = z["hidden"], z["heads"]
        w = {"q": m.matrix(H * z["dim"], hn), "k": m.matrix(H * z["dim"], hn), "v": m.matrix(H * z["vdim"], hn), "g": m.matrix(H * z["vdim"], hn),
             "o": m.matrix(hn, H * z["vdim"]), "norm": m.gain(H * z["vdim"]), "i": m.matrix(H, hn), "i.b": m.uniform(-0.1, 0.1, H),
             "f": m.matrix(H, hn), "f.b": torch.linspace(3.0, 6.0, H, device=DEV)}
    elif kind == "gla":
        z = GLA[case["sizes"]]
        hn, n = z["hidden"], z["heads"] * z["dim"]
        w = {"q": m.matrix(n, hn), "k": m.matrix(n, hn), "v": m.matrix(n, hn), "g": m.matrix(n, hn), "o": m.matrix(hn, n), "norm": m.gain(z["dim"]),
             "a1": m.matrix(z["rank"], hn), "a2": m.normal(n, z["rank"], std=z["rank"] ** -0.5), "a2.b": m.uniform(-0.1, 0.1, n)}
    else:
        z = DELTA[case["sizes"]]
        hn, H, nk, nv = z["hidden"], z["heads"], z["kq"] * z["dim"], z["heads"] * z["dim"]
        w = {"q": m.matrix(nk, hn), "k": m.matrix(nk, hn), "v": m.matrix(nv, hn), "q.conv": m.uniform(-0.5, 0.5, nk, 4),
             "k.conv": m.uniform(-0.5, 0.5, nk, 4), "v.conv": m.uniform(-0.5, 0.5, nv, 4), "b": m.matrix(H, hn), "a": m.matrix(H, hn),
             "A_log": torch.log(m.uniform(1.0, 16.0, H)), "dt_bias": _dt_bias(m, H), "g": m.matrix(nv, hn), "norm": m.gain(z["dim"]), "o": m.matrix(hn, nv)}
    return w, m.normal(case["tokens"], hn)


def _spec(case):
    kind = case["kind"]
    if kind == "attention":
        z = QWEN[case["sizes"]]
        return AttentionSpec("", z["hidden"], z["heads"], z["kv"], 128, 128 ** -0.5, EPS, RotarySpec(128, THETA))
    if kind == "latent":
        z = LATENT[case["sizes"]]
        return LatentAttentionSpec("", z["hidden"], z["heads"], z["dim"], z["rot"], z["vdim"], z["rank"], (z["dim"] + z["rot"]) ** -0.5, EPS,
                                   RotarySpec(z["rot"], THETA), window=case["window"] or None, q_rank=z["q_rank"] if case["q_latent"] else None)
    if kind == "experts":
        z = EXPERTS[case["sizes"]]
        return RoutedExpertsSpec("", z["hidden"], z["experts"], z["top"], z["ff"], z["groups"], z["keep"], 2.0, True,
                                 GatedMlpSpec("shared.", z["hidden"], z["ff"], names=("gate", "up", "down")), True)
    if kind == "mamba2":
        z = MAMBA2[case["sizes"]]
        return Mamba2Spec("", z["hidden"], z["heads"], z["vdim"], z["state"], z["groups"], 4, 1, EPS)
    if kind == "mlstm":
        z = MLSTM[case["sizes"]]
        return MatrixLstmSpec("", z["hidden"], z["heads"], z["dim"], z["vdim"], 10.0, EPS)
    if kind == "gla":
        z = GLA[case["sizes"]]
        return GatedLinearAttentionSpec("", z["hidden"], z["heads"], z["dim"], z["dim"], z["rank"], 16.0, EPS, names=(
            ("q", "q"), ("k", "k"), ("v", "v"), ("gate", "g"), ("o", "o"), ("norm", "norm"), ("decay_in", "a1"), ("decay_out", "a2"),
            ("decay_bias", "a2.b")))
    z = DELTA[case["sizes"]]
    return GatedDeltaRuleSpec("", z["hidden"], z["heads"], z["kq"], z["dim"], z["dim"], 4, EPS)


def _fill(cache, layers, rids, starts, kv):
    """Lays the keys and values that the requests hold into their pages."""
    g = cache.groups[0]
    for li in range(layers):
        at = 0
        for r, n in zip(rids, starts):
            where = torch.from_numpy(cache.slot_mapping(0, r, 0, n)).to(DEV).long()
            for arr, src in zip(g.arrays, kv[li]):
                arr[li][where // PAGE, :, where % PAGE] = src[at: at + n].to(arr.dtype)
            at += n


def prepare(case, seed):
    kind, dtype = case["kind"], getattr(torch, case["dtype"])
    if kind in ("decode", "prompt"):
        w, ids, kv = _qwen_inputs(case, seed)
        model = build_model(config_from_dict(_qwen_config(case)).to_model_spec())
        model.load(w, dtype, DEV)
        del w
        if kind == "prompt":
            n = case["tokens"]
            runner = ModelRunner(model, PAGE, -(-n // PAGE) + 2, 2, n + 64, DEV)
            return dict(kind=kind, runner=runner, entries=[StepEntry("prompt", ids, (n - 1,))])
        held = _contexts(case)
        runner = ModelRunner(model, PAGE, sum(-(-(c + 2) // PAGE) for c in held) + 2, len(held), max(held) + 64, DEV)
        runner.enable_graphs()
        rids = [f"r{i}" for i in range(len(held))]
        for r in rids:
            runner.add_request(r)
        runner.cache.append(list(zip(rids, held)))
        _fill(runner.cache, case["layers"], rids, held, kv)
        state = dict(kind=kind, runner=runner, entries=[StepEntry(r, [t], (0,)) for r, t in zip(rids, ids)], held=list(zip(rids, held)))
        run(state)                                       # the server has decoded before: its graph is there
        return state
    part = build_part(_spec(case))
    if kind == "attention":
        w, x, kv, lens, starts = _attention_inputs(case, seed)
    else:
        w, x = _mixer_inputs(case, seed)
        lens = [case["tokens"]] if kind == "experts" else _row_lens(case)
        starts = [0] * len(lens)
    part.load(w, dtype, DEV)
    del w
    need = part.cache_need() if hasattr(part, "cache_need") else None
    mem = part.state_need() if hasattr(part, "state_need") else None
    total = [a + b for a, b in zip(starts, lens)]
    cm = CacheManager([need] if need is not None else [], [mem] if mem is not None else [], PAGE, sum(-(-t // PAGE) for t in total) + 1, len(lens),
                      max(total), dtype, DEV)
    rids = [f"r{i}" for i in range(len(lens))]
    for r in rids:
        cm.add_request(r)
    if kind == "attention":
        cm.append(list(zip(rids, starts)))
        _fill(cm, 1, rids, starts, [kv])
    cm.append(list(zip(rids, lens)))
    ctx = StepContext(cm, Workspace(DEV)).build([StepEntry(r, [0] * n) for r, n in zip(rids, lens)], starts)
    return dict(kind=kind, part=part, x=x, ctx=ctx, cache=ctx.cache_view(0) if need is not None else None,
                state=ctx.state_view(0) if mem is not None else None)


def run(state):
    if "runner" in state:
        runner = state["runner"]
        logits = runner.step(state["entries"])
        if state["kind"] == "prompt":
            runner.end_request("prompt")                 # the next pass is a new request's
        else:
            for r, n in state["held"]:                   # the next pass decodes the same place again
                runner.cache.truncate(r, n)
        return logits
    ctx, st = state["ctx"], state["state"]
    ctx.memo.clear()                                     # a step's memo, as at the start of every step
    if state["kind"] == "experts":
        return state["part"].forward(state["x"], ctx)
    if st is None:
        return state["part"].forward(state["x"], ctx, state["cache"], None)
    st.zero_()                                           # new requests: their slots are zeroed when they get them
    out = state["part"].forward(state["x"], ctx, state["cache"], st)
    return out, st


def work(case):
    kind, T = case["kind"], case.get("tokens", 1)
    b = 4 if case["dtype"] == "float32" else 2
    if kind in ("decode", "prompt", "attention"):
        z = QWEN[case["sizes"]]
        h, nq, nkv = z["hidden"], z["heads"], z["kv"]
        attn_w, mlp_w, head_w = h * 128 * (2 * nq + 2 * nkv), 3 * h * z["ff"], z["vocab"] * h
        if kind == "decode":
            B, held = case["batch"], sum(_contexts(case)) + case["batch"]
            return {"bytes": 2 * (case["layers"] * (attn_w + mlp_w) + head_w) + case["layers"] * held * nkv * 128 * 2 * b + B * z["vocab"] * 4,
                    "flops": 2 * B * (case["layers"] * (attn_w + mlp_w) + head_w) + case["layers"] * held * nq * 128 * 4}
        if kind == "prompt":
            keys = T * (T + 1) // 2
            return {"bytes": 2 * (case["layers"] * (attn_w + mlp_w) + head_w) + 2 * T * h + case["layers"] * 2 * T * nkv * 128 * b + z["vocab"] * 4,
                    "flops": case["layers"] * (2 * T * (attn_w + mlp_w) + keys * nq * 128 * 4) + 2 * head_w}
        starts = [case["context"]] + [max(1, case["context"] + 101 * i) for i in range(case["batch"])]
        keys = T * case["context"] + T * (T + 1) // 2 + sum(s + 1 for s in starts[1:])
        rows = T + case["batch"]
        return {"bytes": 2 * attn_w + 4 * rows * h + 2 * nkv * 128 * 2 * (sum(starts) + rows), "flops": 2 * rows * attn_w + keys * nq * 128 * 4}
    lens = _row_lens(case)
    if kind == "latent":
        z = LATENT[case["sizes"]]
        h, H, kd = z["hidden"], z["heads"], z["rank"] + z["rot"]
        q = H * (z["dim"] + z["rot"])
        mats = (z["q_rank"] * (h + q) if case["q_latent"] else q * h) + kd * h + H * (z["dim"] + z["vdim"]) * z["rank"] + h * H * z["vdim"]
        W = case["window"] or 1 << 30
        keys = sum(min(n, W) * (min(n, W) + 1) // 2 + max(0, n - W) * min(n, W) for n in lens)
        # a key and a value per head from each record, and plain attention over them: the fewest operations that give the answer
        return {"bytes": 2 * mats + 4 * T * h + 2 * T * kd, "flops": 2 * T * mats + keys * H * 2 * (z["dim"] + z["rot"] + z["vdim"])}
    if kind == "experts":
        z = EXPERTS[case["sizes"]]
        h, ff, E, top = z["hidden"], z["ff"], z["experts"], z["top"]
        read = E * (1.0 - (1.0 - top / E) ** T) + 1
        return {"bytes": int(2 * (read * 3 * h * ff + E * h) + 4 * T * h), "flops": 2 * T * ((top + 1) * 3 * h * ff + (E + 1) * h)}
    if kind == "mamba2":
        z = MAMBA2[case["sizes"]]
        inner, bc = z["heads"] * z["vdim"], z["groups"] * z["state"]
        mats, mem, per = z["hidden"] * (3 * inner + 2 * bc + z["heads"]), z["heads"] * z["vdim"] * z["state"], 5
        conv = 3 * (inner + 2 * bc)
    elif kind == "mlstm":
        z = MLSTM[case["sizes"]]
        H = z["heads"]
        mats, mem, per, conv = z["hidden"] * (2 * H * z["dim"] + 3 * H * z["vdim"] + 2 * H), H * z["dim"] * (z["vdim"] + 1), 5, H
    elif kind == "gla":
        z = GLA[case["sizes"]]
        n = z["heads"] * z["dim"]
        mats, mem, per, conv = z["hidden"] * (5 * n + z["rank"]) + n * z["rank"], n * z["dim"], 5, 0
    else:
        z = DELTA[case["sizes"]]
        nk, nv = z["kq"] * z["dim"], z["heads"] * z["dim"]
        mats, mem, per, conv = z["hidden"] * (2 * nk + 3 * nv + 2 * z["heads"]), nv * z["dim"], 7, 3 * (2 * nk + nv)
    return {"bytes": 2 * mats + 4 * T * z["hidden"] + 4 * len(lens) * (mem + conv), "flops": 2 * T * mats + per * T * mem}


# Measured 2-norm errors against float64, about four times each: 0.0038 to 0.0050 for the single layers, 0.0066 to 0.011 for the steps
# through 4 and 8 layers, 0.020 for the 28 layers of decode_0.6b_b1 (a rounding in one layer travels through all that follow, so two
# correct forms are up to 1.4 times that apart), 3.1e-6 for the float32 prompt.
def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 1.2e-5}
    if case["kind"] in ("decode", "prompt"):
        return {"rel": 6e-2 if case["layers"] > 8 else 4e-2}
    return {"rel": 1.6e-2}


# ---------------------------------------------------------------------------- the same in 64 bits
def _rms(x, w=None, eps=EPS):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)
    return y if w is None else y * w.double()


def _rotate(x, pos, dims):
    """x [T, heads, d]: the first ``dims`` numbers turn, element i with i + dims / 2, by pos * THETA^(-2i / dims)."""
    i = torch.arange(dims // 2, dtype=torch.float64, device=DEV)
    inv = torch.pow(torch.tensor(THETA, dtype=torch.float64, device=DEV), -2.0 * i / dims).float().double()
    a = pos.double()[:, None, None] * inv
    c, s = a.cos(), a.sin()
    u, v = x[..., : dims // 2], x[..., dims // 2: dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], -1)


def _softmax_rows(q, k, v, start, scale, window=0):
    """q [T, H, d] at places start .., k and v [start + T, H or fewer, d]: causal attention, some query rows at a time."""
    T, H = q.shape[:2]
    k, v = (t.repeat_interleave(H // t.shape[1], 1) for t in (k, v))
    out, j = [], torch.arange(k.shape[0], device=DEV)
    for t0 in range(0, T, 256):
        p = torch.arange(start + t0, start + min(T, t0 + 256), device=DEV)
        s = torch.einsum("thd,jhd->htj", q[t0: t0 + 256], k) * scale
        seen = (j[None] <= p[:, None]) & ((j[None] > p[:, None] - window) if window else True)
        out.append(torch.einsum("htj,jhd->thd", s.masked_fill(~seen, -math.inf).softmax(-1), v))
    return torch.cat(out)


def _qwen_attention(x, w, p, lens, starts, held):
    """x [T, hidden]; held: (keys, values) of what the rows' requests hold, side by side, or None."""
    T, hd = x.shape[0], 128
    pos = torch.cat([torch.arange(s, s + n, device=DEV) for s, n in zip(starts, lens)])
    q, k, v = ((x @ w[p + n].double().t()).view(T, -1, hd) for n in ("q_proj.weight", "k_proj.weight", "v_proj.weight"))
    q, k = _rotate(_rms(q, w[p + "q_norm.weight"]), pos, hd), _rotate(_rms(k, w[p + "k_norm.weight"]), pos, hd)
    outs, at, h_at = [], 0, 0
    for n, s in zip(lens, starts):
        kk, vv = k[at: at + n], v[at: at + n]
        if s:
            kk, vv = (torch.cat([h[h_at: h_at + s].double(), t]) for h, t in zip(held, (kk, vv)))
        outs.append(_softmax_rows(q[at: at + n], kk, vv, s, hd ** -0.5))
        at, h_at = at + n, h_at + s
    return torch.cat(outs).reshape(T, -1) @ w[p + "o_proj.weight"].double().t()


def _silu(x):
    return x * torch.sigmoid(x)


def _gated(x, w, p, names=("gate", "up", "down")):
    g, u, d = (w[p + n].double() for n in names)
    return (_silu(x @ g.t()) * (x @ u.t())) @ d.t()


def _conv_silu(x, weight, bias, lens):
    out = []
    for part in x.split(lens):
        y = sum(torch.cat([part.new_zeros(3, part.shape[1]), part])[j: j + part.shape[0]] * weight[:, j].double() for j in range(4))
        out.append(_silu(y if bias is None else y + bias.double()))
    return torch.cat(out)


def _last_inputs(x, lens):
    """[rows, channels, 3]: the inputs that the convolution still needs, oldest first."""
    return torch.stack([torch.cat([p.new_zeros(3, p.shape[1]), p])[-3:].t() for p in x.split(lens)])


def _state_rows(width, *parts):
    flat = torch.cat([p.reshape(p.shape[0], -1) for p in parts], 1)
    return torch.cat([flat, flat.new_zeros(flat.shape[0], width - flat.shape[1])], 1)


def _memories(lens, step, start):
    """step(t, S) -> (S, o_t) over the tokens of every row; the outputs [T, ...] and the rows' last S."""
    outs, last, t = [], [], 0
    for n in lens:
        S = start()
        for _ in range(n):
            S, o = step(t, S)
            outs.append(o)
            t += 1
        last.append(S)
    return torch.stack(outs), torch.stack(last)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("decode", "prompt"):
        w, ids, kv = _qwen_inputs(case, seed)
        x = w["model.embed_tokens.weight"][torch.tensor(ids, device=DEV)].double()
        starts = _contexts(case) if kind == "decode" else [0]
        lens = [1] * len(starts) if kind == "decode" else [len(ids)]
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            x = x + _qwen_attention(_rms(x, w[p + "input_layernorm.weight"]), w, p + "self_attn.", lens, starts, kv[i] if kv else None)
            x = x + _gated(_rms(x, w[p + "post_attention_layernorm.weight"]), w, p + "mlp.", ("gate_proj.weight", "up_proj.weight", "down_proj.weight"))
        if kind == "prompt":
            x = x[-1:]
        x = _rms(x, w["model.norm.weight"])
        return x @ w["model.embed_tokens.weight" if QWEN[case["sizes"]]["tied"] else "lm_head.weight"].double().t()
    if kind == "attention":
        w, x, kv, lens, starts = _attention_inputs(case, seed)
        return _qwen_attention(x.double(), w, "", lens, starts, kv)
    w, x = _mixer_inputs(case, seed)
    x, T = x.double(), x.shape[0]
    lens = [T] if kind == "experts" else _row_lens(case)

    def times(name, src=x):
        return src @ w[name].double().t()

    if kind == "latent":
        z = LATENT[case["sizes"]]
        H, dn, dr, rank = z["heads"], z["dim"], z["rot"], z["rank"]
        pos = torch.cat([torch.arange(n, device=DEV) for n in lens])
        q = (times("uq", _rms(times("dq"), w["dq.norm"])) if case["q_latent"] else times("q")).view(T, H, dn + dr)
        c = times("dkv")
        kr = _rotate(c[:, None, rank:], pos, dr).expand(T, H, dr)
        c = _rms(c[:, :rank], w["dkv.norm"])
        q = torch.cat([q[..., :dn], _rotate(q[..., dn:], pos, dr)], -1)
        k = torch.cat([times("uk", c).view(T, H, dn), kr], -1)
        v = times("uv", c).view(T, H, z["vdim"])
        o = torch.cat([_softmax_rows(a, b, d, 0, (dn + dr) ** -0.5, case["window"]) for a, b, d in zip(q.split(lens), k.split(lens), v.split(lens))])
        return times("o", o.reshape(T, -1))
    if kind == "experts":
        z = EXPERTS[case["sizes"]]
        E, G = z["experts"], z["groups"]
        s = torch.sigmoid(times("router"))
        pick = s + w["correction"].double()
        best = pick.view(T, G, -1).topk(2, -1).values.sum(-1).topk(z["keep"], -1).indices
        kept = torch.zeros(T, G, dtype=torch.bool, device=DEV).scatter_(1, best, True).repeat_interleave(E // G, 1)
        ids = pick.masked_fill(~kept, -math.inf).topk(z["top"], -1).indices
        out = torch.sigmoid(times("shared.sg")) * _gated(x, w, "shared.")
        for e in range(E):
            t, _ = (ids == e).nonzero(as_tuple=True)
            if t.numel():
                out[t] += _gated(x[t], w, f"e{e}.") * (s[t, e] * 2.0)[:, None]
        return out
    if kind == "mamba2":
        z = MAMBA2[case["sizes"]]
        H, P, N, G = z["heads"], z["vdim"], z["state"], z["groups"]
        inner, ch = H * P, H * P + 2 * G * N
        zg, raw, dt = times("in").split([inner, ch, H], -1)
        u, B, C = _conv_silu(raw, w["conv"], w["conv.b"], lens).split([inner, G * N, G * N], -1)
        u, B, C = u.view(T, H, P), *(t.view(T, G, N).repeat_interleave(H // G, 1) for t in (B, C))
        dt = torch.nn.functional.softplus(dt + w["dt_bias"].double())
        a = torch.exp(-torch.exp(w["A_log"].double()) * dt)
        y, S = _memories(lens, lambda t, S: (lambda n: (n, torch.einsum("hpn,hn->hp", n, C[t])))(
            S * a[t, :, None, None] + (dt[t, :, None] * u[t])[..., None] * B[t, :, None]), lambda: x.new_zeros(H, P, N))
        y = (y + w["D"].double()[:, None] * u).reshape(T, inner) * _silu(zg)
        n = H * P * N + 3 * ch
        return times("o", _rms(y, w["norm"])), _state_rows(-(-n // 4) * 4, S, _last_inputs(raw, lens))
    if kind == "mlstm":
        z = MLSTM[case["sizes"]]
        H, dk, dv = z["heads"], z["dim"], z["vdim"]
        q, k = times("q").view(T, H, dk) * dk ** -0.5, times("k").view(T, H, dk)
        v = torch.cat([times("v").view(T, H, dv), x.new_ones(T, H, 1)], -1)
        i = 10.0 * torch.tanh((times("i") + w["i.b"].double()) / 10.0)
        f = torch.nn.functional.logsigmoid(10.0 * torch.tanh((times("f") + w["f.b"].double()) / 10.0))

        def step(t, S):
            S, m = S[:, :, :-1], S[:, 0, -1]
            new = torch.maximum(f[t] + m, i[t])
            S = S * torch.exp(f[t] + m - new)[:, None, None] + (torch.exp(i[t] - new)[:, None] * v[t])[..., None] * k[t, :, None]
            num = torch.einsum("hvk,hk->hv", S, q[t])
            o = num[:, :dv] / (torch.maximum(num[:, dv:].abs(), torch.exp(-new)[:, None]) + 1e-6)
            return torch.cat([S, new[:, None, None].expand(H, dv + 1, 1)], -1), o

        o, S = _memories(lens, step, lambda: x.new_zeros(H, dv + 1, dk + 1))
        y = _rms(o).reshape(T, H * dv) * w["norm"].double() * torch.sigmoid(times("g"))
        n = H * (dv + 1) * dk
        return times("o", y), _state_rows(n + -(-H // 4) * 4, S[..., :-1], S[:, :, 0, -1])
    if kind == "gla":
        z = GLA[case["sizes"]]
        H, d = z["heads"], z["dim"]
        q, k, v = (times(n).view(T, H, d) for n in ("q", "k", "v"))
        al = torch.sigmoid(times("a2", times("a1")) + w["a2.b"].double()).pow(1.0 / 16.0).view(T, H, d)
        o, S = _memories(lens, lambda t, S: (lambda n: (n, torch.einsum("hvk,hk->hv", n, q[t] * d ** -0.5)))(
            S * al[t, :, None] + v[t][..., None] * k[t, :, None]), lambda: x.new_zeros(H, d, d))
        y = (_rms(o, w["norm"])).reshape(T, H * d) * _silu(times("g"))
        return times("o", y), S
    z = DELTA[case["sizes"]]
    H, K, d = z["heads"], z["kq"], z["dim"]
    raw = torch.cat([times("q"), times("k"), times("v")], -1)
    q, k, v = _conv_silu(raw, torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]]), None, lens).split([K * d, K * d, H * d], -1)
    q, k = ((t.view(T, K, d) * torch.rsqrt(t.view(T, K, d).square().sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // K, 1) for t in (q, k))
    v, beta = v.view(T, H, d), torch.sigmoid(times("b"))
    g = torch.exp(-torch.exp(w["A_log"].double()) * torch.nn.functional.softplus(times("a") + w["dt_bias"].double()))

    def write(t, S):
        S = S * g[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.einsum("hvk,hk->hv", S, k[t]))
        S = S + u[..., None] * k[t, :, None]
        return S, torch.einsum("hvk,hk->hv", S, q[t] * d ** -0.5)

    o, S = _memories(lens, write, lambda: x.new_zeros(H, d, d))
    y = _rms(o, w["norm"]).reshape(T, H * d) * _silu(times("g"))
    n = H * d * d + 3 * raw.shape[1]
    return times("o", y), _state_rows(-(-n // 4) * 4, S, _last_inputs(raw, lens))
