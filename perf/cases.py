"""The work that programs built on this package spend their time in, as cases that can be run and timed one by one: single
layers of training and serving through the functions a program calls, and one whole serving step.

    attention   causal / full self-attention over a fused qkv projection, forward and backward (pre-training, fine-tuning)
    packed      prompts of different lengths admitted together by the Qwen serving engine, one attention call for all
    paged       attention of the ragged serving step over a paged KV cache: prompt pieces, decode batches and mixtures
    mixer       the recurrent half of a layer of the ragged step: convolution, gates, state scan, read-out
    w4          a 4-bit (W4A16) projection of a decode step
    qlora       a decoder layer of QLoRA training (NF4 base, LoRA on q and v), forward and backward
    head        the output projection with its cross-entropy, forward and backward
    step        one whole serving step of a small hybrid model: prompts in, logits of their last tokens out

A case is a dict of plain values; ``runs`` lists what a step holds as "tokens@first position", one entry per sequence.
"""
import math

import torch

from llm_in_practise_b200.inference.ragged import RaggedGenerator, make_pieces
from llm_in_practise_b200.models.nedesun import NedesunConfig, NedesunForCausalLM
from llm_in_practise_b200.models.qwen3 import Qwen3Config, Qwen3DecoderLayer
from llm_in_practise_b200.ops import elementwise as ew
from llm_in_practise_b200.ops.attention import attention
from llm_in_practise_b200.ops.flash import flash_attention_varlen
from llm_in_practise_b200.ops.linear import FusedLinear
from llm_in_practise_b200.ops.linear_scan import delta_gates, linear_scan, lowrank_decay, scan_readout, short_conv
from llm_in_practise_b200.ops.loss import linear_cross_entropy
from llm_in_practise_b200.ops.multimap_attention import multimap_attention
from llm_in_practise_b200.ops.w4 import NF4Weight
from llm_in_practise_b200.quant.formats import W4Weight
from llm_in_practise_b200.utils.arena import ParamArena

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
F64 = torch.float64

# the 16 levels of the NF4 data type (QLoRA, Dettmers et al. 2023, appendix E)
NF4_LEVELS = [-1.0, -0.6961928009986877, -0.5250730514526367, -0.39491748809814453, -0.28444138169288635, -0.18477343022823334,
              -0.09105003625154495, 0.0, 0.07958029955625534, 0.16093020141124725, 0.24611230194568634, 0.33791524171829224,
              0.44070982933044434, 0.5626170039176941, 0.7229568362236023, 1.0]


def listed():
    return [
        # Qwen3-14B fine-tuning at 512 tokens: the two micro-batches of 2 of an optimizer step in one pass
        {"name": "attention_finetune", "kind": "attention", "B": 4, "S": 512, "H": 40, "Hkv": 8, "D": 128, "causal": True, "dtype": "bf16"},
        # long-sequence fine-tuning, Qwen3-8B heads, one sequence of 4096 tokens
        {"name": "attention_4k", "kind": "attention", "B": 1, "S": 4096, "H": 32, "Hkv": 8, "D": 128, "causal": True, "dtype": "bf16"},
        # pre-training of the 66M GPT: blocks of 256 tokens, 12 heads of 64
        {"name": "attention_gpt", "kind": "attention", "B": 32, "S": 256, "H": 12, "Hkv": 12, "D": 64, "causal": True, "dtype": "bf16"},
        # a burst of six requests admitted in one scheduler iteration, Qwen3-8B heads
        {"name": "prefill_packed", "kind": "packed", "lens": "512,1200,77,2048,300,1001", "H": 32, "Hkv": 8, "D": 128, "dtype": "bf16"},
        # a chunked-prefill step: a new prompt, a continued one, two sequences that decode beside them
        {"name": "paged_prompt", "kind": "paged", "runs": "2048@0,700@512,1@1800,1@95", "H": 16, "G": 4, "D": 128, "page": 64, "opt": "none"},
        # a decode batch of 64 sequences at contexts around four thousand tokens
        {"name": "paged_decode", "kind": "paged", "runs": decode_runs(64, 4000, 700), "H": 16, "G": 4, "D": 128, "page": 64, "opt": "none"},
        # the delta-rule half of a parallel layer over two prompts
        {"name": "delta_prompt", "kind": "mixer", "mode": "delta", "runs": "2048@0,513@0", "H": 16, "G": 4, "D": 128},
        # the same for two sequences that decode: the smallest call, bound by its launches
        {"name": "delta_decode", "kind": "mixer", "mode": "delta", "runs": "1@1900,1@30", "H": 16, "G": 4, "D": 128},
        # gate|up projection of Qwen3-8B W4A16, eight sequences decoding
        {"name": "w4_decode", "kind": "w4", "M": 8, "N": 24576, "K": 4096},
        # a Qwen3-14B layer of the QLoRA run (2048 tokens, rank 8, dropout 0.1)
        {"name": "qlora_layer", "kind": "qlora", "B": 4, "S": 512, "W": 5120, "H": 40, "Hkv": 8, "F": 17408, "p": 0.1},
        # its frozen output projection and loss over the vocabulary of 151 936
        {"name": "head_loss", "kind": "head", "T": 2048, "K": 5120, "V": 151936, "train": False},
        # prefill of three prompts through the small hybrid model
        {"name": "step_prefill", "kind": "step", "runs": "1500@0,800@0,45@0", "W": 2048},
    ]


def decode_runs(n, ctx, spread):
    """``n`` sequences at positions from ``ctx - spread`` to ``ctx``, unevenly."""
    return ",".join("1@%d" % max(0, ctx - i * 37 % (spread + 1)) for i in range(n))


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention", "attention", "packed", "paged", "paged", "paged", "mixer", "mixer", "w4", "qlora", "head", "step"])
    if kind == "attention":
        D = rng.choice([64, 128, 128])
        H, Hkv = rng.choice([(12, 12), (8, 8), (16, 8)] if D == 64 else [(40, 8), (32, 8), (16, 8), (8, 8)])
        S = _log(rng, 64, 4096)
        causal = rng.random() < 0.85
        S = S if causal else -(-S // 8) * 8              # full attention takes whole rows of 16 bytes of scores
        most = max(1, min(64, int(4096 * 4096 * 32 * 128 * (0.5 if not causal else 1.0) / (S * S * H * D)), 65536 // S))
        return {"kind": kind, "B": _log(rng, 1, most), "S": S, "H": H, "Hkv": Hkv, "D": D, "causal": causal, "dtype": rng.choice(["bf16", "bf16", "bf16", "fp16"])}
    if kind == "packed":
        n = _log(rng, 1, 24)
        D = rng.choice([128, 128, 64])
        H, Hkv = rng.choice([(32, 8), (16, 8), (40, 8)]) if D == 128 else rng.choice([(16, 8), (12, 2)])
        return {"kind": kind, "lens": ",".join(str(_log(rng, 16, 4096 if n <= 4 else 1024)) for _ in range(n)), "H": H, "Hkv": Hkv, "D": D, "dtype": rng.choice(["bf16", "bf16", "bf16", "fp16"])}
    if kind in ("paged", "mixer"):
        if rng.random() < 0.5:
            runs = decode_runs(_log(rng, 1, 128), _log(rng, 60, 4000), _log(rng, 1, 800))
        else:
            runs = ",".join("%d@%d" % (_log(rng, 9, 2048), rng.choice([0, 0, _log(rng, 1, 1500)])) for _ in range(rng.randint(1, 3)))
            runs += "".join(",1@%d" % _log(rng, 1, 2000) for _ in range(rng.choice([0, 0, 3, 8])))
        if kind == "paged":
            D = rng.choice([128, 128, 64])
            H, G = rng.choice([(16, 4), (16, 8), (32, 8), (16, 2), (8, 8)])
            return {"kind": kind, "runs": runs, "H": H, "G": G, "D": D, "page": rng.choice([64, 64, 32, 16]), "opt": rng.choice(["none", "none", "window", "chunk"])}
        H, G = rng.choice([(16, 4), (32, 8), (16, 16)])
        mode = rng.choice(["delta", "delta", "wkv"])
        return {"kind": kind, "mode": mode, "runs": runs, "H": H, "G": G if mode == "delta" else H, "D": rng.choice([128, 128, 64])}
    if kind == "w4":
        N, K = rng.choice([(6144, 4096), (4096, 4096), (24576, 4096), (4096, 12288), (7168, 5120), (34816, 5120), (5120, 17408), (12288, 2048)])
        return {"kind": kind, "M": _log(rng, 1, 64), "N": N, "K": K}
    if kind == "qlora":
        W, H, Hkv, F = rng.choice([(5120, 40, 8, 17408), (4096, 32, 8, 12288), (2560, 32, 8, 9728)])
        B = _log(rng, 1, 8)
        return {"kind": kind, "B": B, "S": _log(rng, 64, 2048 // B), "W": W, "H": H, "Hkv": Hkv, "F": F, "p": rng.choice([0.0, 0.0, 0.1])}
    if kind == "head":
        if rng.random() < 0.4:
            return {"kind": kind, "T": _log(rng, 256, 8192), "K": 768, "V": 30522, "train": True}
        return {"kind": kind, "T": _log(rng, 128, 2048), "K": rng.choice([2048, 2560, 4096, 5120]), "V": 151936, "train": False}
    return {"kind": kind, "runs": ",".join("%d@0" % _log(rng, 9, 1500) for _ in range(rng.randint(1, 4))), "W": 2048}


# ------------------------------------------------------------------------------------------------ inputs
class _Random:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed))

    def normal(self, *shape, dtype=torch.float32, std=1.0):
        return (torch.randn(*shape, device=DEV, generator=self.g) * std).to(dtype)

    def uniform(self, lo, hi, *shape):
        return torch.rand(*shape, device=DEV, generator=self.g) * (hi - lo) + lo

    def ints(self, hi, *shape, dtype=torch.long):
        return torch.randint(0, hi, shape, device=DEV, generator=self.g, dtype=dtype)


def _runs(case):
    """[(tokens, first position)] of the step's sequences."""
    return [tuple(int(x) for x in r.split("@")) for r in case["runs"].split(",")]


def _step_layout(runs):
    """Positions, rows and pieces of a step (pieces None: every sequence decodes one token)."""
    pos = torch.cat([torch.arange(p0, p0 + n) for n, p0 in runs]).to(torch.int32)
    slot = torch.cat([torch.full((n,), i) for i, (n, _) in enumerate(runs)]).to(torch.int32)
    first, entries = 0, []
    for i, (n, p0) in enumerate(runs):
        entries.append((first, n, p0, i))
        first += n
    pieces = None if all(n == 1 for n, _ in runs) else make_pieces(entries, DEV)
    return pos.to(DEV), slot.to(DEV), pieces


def _options(case):
    """Mask and score options of attention layers: a window that keeps four tokens, with a sink; chunks with capped scores and gates."""
    opt = case["opt"]
    return {"window": 1024 if opt == "window" else 0, "keep": 4 if opt == "window" else 0, "chunk": 2048 if opt == "chunk" else 0,
            "softcap": 50.0 if opt == "chunk" else 0.0, "sink": opt == "window", "gate": opt == "chunk"}


def _inputs(case, seed):
    """The tensors of a case, from the seed alone."""
    r = _Random(seed)
    kind = case["kind"]
    if kind == "attention":
        B, S, H, Hkv, D, dt = (case[k] for k in ("B", "S", "H", "Hkv", "D", "dtype"))
        return {"qkv": r.normal(B * S, (H + 2 * Hkv) * D, dtype=DTYPES[dt]), "g": r.normal(B * S, H * D, dtype=DTYPES[dt])}
    if kind == "packed":
        lens = [int(x) for x in case["lens"].split(",")]
        return {"qkv": r.normal(sum(lens), (case["H"] + 2 * case["Hkv"]) * case["D"], dtype=DTYPES[case["dtype"]]), "lens": lens}
    if kind == "paged":
        runs, H, G, D, BS = _runs(case), case["H"], case["G"], case["D"], case["page"]
        per = [-(-(n + p0) // BS) for n, p0 in runs]
        nb = sum(per)
        order = torch.randperm(nb, device=DEV, generator=r.g) + 1          # pages in any order; page 0 is never handed out
        table = torch.zeros(len(runs), max(per), dtype=torch.int32, device=DEV)
        at = 0
        for i, n in enumerate(per):
            table[i, :n] = order[at:at + n].to(torch.int32)
            at += n
        T = sum(n for n, _ in runs)
        bf = torch.bfloat16
        return {"q": r.normal(T, H * D, dtype=bf), "ck": r.normal(nb + 1, G, BS, D, dtype=bf), "cv": r.normal(nb + 1, G, BS, D, dtype=bf),
                "table": table, "sink": r.normal(H), "gate": r.normal(T, H), "runs": runs}
    if kind == "mixer":
        runs, H, G, D = _runs(case), case["H"], case["G"], case["D"]
        T, n, N = sum(a for a, _ in runs), len(runs), case["H"] * case["D"]
        out = {"runs": runs, "state": r.normal(n, H, D, D, std=0.1), "w": r.uniform(0.8, 1.2, D if case["mode"] == "delta" else N)}
        if case["mode"] == "delta":
            C = 2 * G * D + N
            out.update(x=r.normal(T, C, dtype=torch.bfloat16), conv_w=r.normal(C, 4, std=0.5), tail=r.normal(n, 3, C), ab=r.normal(T, 2 * H),
                       post=r.normal(T, N, dtype=torch.bfloat16), dt_bias=r.uniform(-4.0, -2.0, H), A_log=r.uniform(-1.0, 1.0, H))
        else:
            out.update(rkvg=r.normal(T, 4 * N), x=r.normal(T, 16), w2=r.normal(N, 16, std=0.3), w0=r.uniform(-6.0, -2.0, N), u=r.normal(H, D, std=0.3))
        return out
    if kind == "w4":
        M, N, K = case["M"], case["N"], case["K"]
        scale = r.uniform(0.5, 1.5, N * (K // 128)) * K ** -0.5 / 4
        return {"x": r.normal(M, K, dtype=torch.bfloat16), "packed": r.ints(256, N * K // 2, dtype=torch.uint8), "scale": scale, "zs": scale * 8}
    if kind == "qlora":
        T, W, H, Hkv, F, D = case["B"] * case["S"], case["W"], case["H"], case["Hkv"], case["F"], 128
        bf = torch.bfloat16
        out = {"delta": r.normal(T, W, dtype=bf), "res": r.normal(T, W, dtype=bf), "g_out": r.normal(T, W, dtype=bf), "g_res": r.normal(T, W, dtype=bf)}
        for name, N, K in (("qkv", (H + 2 * Hkv) * D, W), ("o", W, H * D), ("gate_up", 2 * F, W), ("down", W, F)):
            out[name] = (r.ints(256, N * K // 2, dtype=torch.uint8), r.uniform(1.0, 3.0, N * K // 64) * K ** -0.5, N, K)
        for name, n in (("n1", W), ("n2", W), ("qn", D), ("kn", D)):
            out[name] = r.uniform(0.8, 1.2, n).to(bf)
        out["A"] = r.normal(16, W, std=W ** -0.5)                                        # rank 8 for q, then 8 for v
        out["Bq"], out["Bv"] = r.normal(8, H * D, std=0.1), r.normal(8, Hkv * D, std=0.1)
        return out
    if kind == "head":
        T, K, V = case["T"], case["K"], case["V"]
        t = r.ints(V, T)
        t[::97] = -100                                                                   # ends of sequences and padding have no target
        return {"x": r.normal(T, K, dtype=torch.bfloat16), "w": r.normal(V, K, dtype=torch.bfloat16, std=K ** -0.5), "t": t}
    return {"runs": _runs(case), "seed": seed}


# ------------------------------------------------------------------------------------------------ cases
def _hybrid(W):
    """A four-layer hybrid model: (window attention beside a delta rule), matrix memory, chunked attention, matrix memory."""
    att, hd = {"heads": W // 128, "kv_heads": W // 512, "dim": 128, "vdim": 128, "scale": 128 ** -0.5}, W // 128
    mlp = {"kind": "dense", "ff": 2 * W}
    par = {"left": dict(att, mask={"size": 1024, "keep_first": 4}), "right": {"heads": hd, "kv_heads": hd // 4, "dim": 128, "vdim": 128, "conv": 4}}
    chunked = dict(att, mask={"size": 2048}, rot={"base": 1e6, "dims": 128}, softcap=50.0, v_mix=True)
    wkv = {"heads": hd, "dim": 128}
    return {"architecture": "Nedesun", "layers": [{"type": "parallel", "mixer": par, "mlp": mlp}, {"type": "wkv", "mixer": wkv, "mlp": mlp},
                                                  {"type": "attention", "mixer": chunked, "mlp": mlp}, {"type": "wkv", "mixer": wkv, "mlp": mlp}],
            "norm": {"eps": 1e-6}, "embedding": {"scale": W ** 0.5}, "residual_mult": 0.3, "vocab": 32768, "width": W}


def prepare(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    s["case"] = case
    if kind == "attention":
        s["qkv"].requires_grad_()
    elif kind == "packed":
        s["cu"] = torch.tensor([0] + s["lens"], dtype=torch.int32).cumsum(0).to(torch.int32).to(DEV)
    elif kind in ("paged", "mixer"):
        s["pos"], s["slot"], s["pieces"] = _step_layout(s["runs"])
        if kind == "paged":
            s["opt"] = _options(case)
    elif kind == "w4":
        lin = FusedLinear(case["K"], [("proj", case["N"])], device=DEV, materialize=False)
        lin.set_nf4(W4Weight(s["packed"], s["scale"], s["zs"], case["N"], case["K"], 128, torch.arange(16, dtype=torch.float32, device=DEV)))
        s["lin"] = lin
    elif kind == "qlora":
        W, H, Hkv, F = case["W"], case["H"], case["Hkv"], case["F"]
        layer = Qwen3DecoderLayer(Qwen3Config(hidden_size=W, intermediate_size=F, num_attention_heads=H, num_key_value_heads=Hkv), 0, torch.bfloat16, DEV)
        for name, lin in layer.fused_linears().items():
            packed, absmax, N, K = s[name[:-5]]
            lin.set_nf4(NF4Weight(packed=packed, N=N, K=K, absmax=absmax))
        for p in layer.parameters():
            p.requires_grad_(False)
        for p, n in ((layer.input_layernorm, "n1"), (layer.post_attention_layernorm, "n2"), (layer.q_norm, "qn"), (layer.k_norm, "kn")):
            p.data.copy_(s[n])
        arena = ParamArena(torch.float32, torch.device(DEV))
        layer.qkv_proj.request_lora(arena, {"q_proj": (8, 16.0), "v_proj": (8, 16.0)}, case["p"], "layers.0.qkv_proj")
        arena.finalize()
        layer.qkv_proj.materialize_lora()
        a, b = layer.qkv_proj.lora_A, layer.qkv_proj.lora_Bt
        with torch.no_grad():
            a["q_proj"].copy_(s["A"][:8]); a["v_proj"].copy_(s["A"][8:])
            b["q_proj"].copy_(s["Bq"]); b["v_proj"].copy_(s["Bv"])
        s["layer"], s["arena"] = layer.train(), arena
        s["rope"] = ew.rope_tables(case["S"], 128, 1e6, DEV)
        s["pos"] = torch.arange(case["S"], device=DEV, dtype=torch.int32).repeat(case["B"])
        s["delta"].requires_grad_(); s["res"].requires_grad_()
    elif kind == "head":
        s["x"].requires_grad_()
        s["w"].requires_grad_(case["train"])
    elif kind == "step":
        r = _Random(seed)
        model = NedesunForCausalLM(NedesunConfig.from_dict(_hybrid(case["W"])), dtype=torch.bfloat16, device=DEV, decay_ranks={1: 16, 3: 16}).eval()
        for n, p in model.named_parameters():
            leaf = n.split(".")[-1]
            if leaf in ("conv_w", "w2", "mu", "u"):
                p.data.copy_(r.normal(*p.shape, std=0.3))
            elif leaf in ("w0", "dt_bias"):
                p.data.fill_(-4.0 if leaf == "w0" else -3.0)
            elif p.dim() >= 2:
                p.data.copy_(r.normal(*p.shape, dtype=p.dtype, std=0.02 if leaf == "embed_tokens" else p.shape[-1] ** -0.5))
        runs = s["runs"]
        longest = max(n for n, _ in runs)
        per = -(-longest // 64)
        gen = RaggedGenerator(model, None, longest)
        cache = gen.make_cache(len(runs) * per, 64, len(runs), per * 64)
        for i in range(len(runs)):
            gen.set_block_row(cache, i, list(range(1 + i * per, 1 + (i + 1) * per)))
        s["gen"], s["cache"] = gen, cache
        s["entries"] = [(i, 0, r.ints(32768, n).tolist(), [n - 1]) for i, (n, _) in enumerate(runs)]
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "attention":
        s["qkv"].grad = None
        out = attention(s["qkv"], case["B"], case["S"], case["H"], case["Hkv"], case["D"], causal=case["causal"])
        out.backward(s["g"])
        return {"out": out.detach(), "dqkv": s["qkv"].grad}
    if kind == "qlora":
        s["arena"].zero_grad()
        s["delta"].grad = s["res"].grad = None
        out, res = s["layer"](s["delta"], s["res"], *s["rope"], s["pos"], case["B"], case["S"])
        torch.autograd.backward([out, res], [s["g_out"], s["g_res"]])
        lin = s["layer"].qkv_proj
        grads = {"d" + m + "_" + n: d[n].grad for m, d in (("A", lin.lora_A), ("B", lin.lora_Bt)) for n in ("q_proj", "v_proj")}
        return {"out": out.detach(), "res": res.detach(), "ddelta": s["delta"].grad, "dres": s["res"].grad, **grads}
    if kind == "head":
        s["x"].grad = s["w"].grad = None
        loss = linear_cross_entropy(s["x"], s["w"], s["t"])
        loss.backward()
        return {"loss": loss.detach(), "dx": s["x"].grad, "dw": s["w"].grad}
    with torch.no_grad():
        if kind == "packed":
            return flash_attention_varlen(s["qkv"], s["cu"], max(s["lens"]), case["H"], case["Hkv"], case["D"], case["D"] ** -0.5)
        if kind == "paged":
            o = s["opt"]
            return multimap_attention(s["q"], s["ck"], s["cv"], s["table"], s["pos"], s["slot"], case["H"], case["G"], 1, case["D"], case["D"],
                                      case["D"] ** -0.5, o["window"], o["keep"], pieces=s["pieces"], max_pos=max(n + p - 1 for n, p in s["runs"]),
                                      sink=s["sink"] if o["sink"] else None, softcap=o["softcap"], chunk=o["chunk"], gate=s["gate"] if o["gate"] else None)
        if kind == "mixer":
            H, G, D = case["H"], case["G"], case["D"]
            pos, slot, pieces = s["pos"], s["slot"], s["pieces"]
            runs, n_runs = (pieces.runs, pieces.n_runs) if pieces is not None else (None, pos.shape[0])
            if case["mode"] == "delta":
                y = short_conv(s["x"], s["conv_w"], s["tail"], pos, slot, runs, n_runs, act=True)
                q, k, v = y[:, :G * D], y[:, G * D:2 * G * D], y[:, 2 * G * D:]
                ab = s["ab"].clone()                     # the gates are formed in place, on what a projection has just written
                a, b = ab[:, :H], ab[:, H:]
                delta_gates(q, k, a, b, s["dt_bias"], s["A_log"], G, H, D, D ** -0.5, 1e-6)
                o = linear_scan(q, k, v, s["state"], pos, slot, runs, n_runs, H, G, D, D, "head_delta", g=a, beta=b)
                z = scan_readout(o, H, D, s["w"], H, 1e-6, torch.bfloat16, post=s["post"], post_act="silu")
                return {"z": z, "state": s["state"], "tail": s["tail"]}
            N = H * D
            r, k, v, g = (s["rkvg"][:, j * N:(j + 1) * N] for j in range(4))
            w = lowrank_decay(s["x"], s["w2"], s["w0"], fast=True, form="exp_exp")
            o = linear_scan(r, k, v, s["state"], pos, slot, runs, n_runs, H, H, D, D, "channel", g=w, pieces=pieces, u=s["u"])
            return {"z": scan_readout(o, H, D, s["w"], H, 1e-6, torch.bfloat16, post=g, post_act="silu"), "state": s["state"]}
        if kind == "w4":
            return s["lin"](s["x"])
        return s["gen"].step(s["entries"], s["cache"])


# ------------------------------------------------------------------------------------------------ bytes and operations
def _seen(case, p):
    """Keys that the token at position p of a paged case sees."""
    o = _options(case)
    if o["chunk"]:
        return p % o["chunk"] + 1
    if o["window"]:
        return min(p + 1, o["window"]) + max(0, min(o["keep"], p + 1 - o["window"]))
    return p + 1


def _pairs(n):
    return n * (n + 1) / 2


def work(case):
    kind = case["kind"]
    if kind == "attention":
        B, S, H, Hkv, D = (case[k] for k in ("B", "S", "H", "Hkv", "D"))
        pairs = _pairs(S) if case["causal"] else S * S
        return {"bytes": 2 * B * S * D * (2 * (H + 2 * Hkv) + 2 * H), "flops": 14 * B * H * D * pairs}
    if kind == "packed":
        lens = [int(x) for x in case["lens"].split(",")]
        return {"bytes": 2 * sum(lens) * case["D"] * (2 * case["H"] + 2 * case["Hkv"]), "flops": 4 * case["H"] * case["D"] * sum(_pairs(n) for n in lens)}
    if kind == "paged":
        H, G, D = case["H"], case["G"], case["D"]
        runs = _runs(case)
        kv = 0
        for n, p0 in runs:                               # keys that any token of the run sees
            o = _options(case)
            lo = max(0, p0 + 1 - o["window"]) if o["window"] else (p0 // o["chunk"] * o["chunk"] if o["chunk"] else 0)
            kv += p0 + n - lo + min(o["keep"], lo)
        return {"bytes": 2 * D * (2 * H * sum(n for n, _ in runs) + 2 * G * kv),
                "flops": 4 * H * D * sum(_seen(case, p) for n, p0 in runs for p in range(p0, p0 + n))}
    if kind == "mixer":
        H, G, D = case["H"], case["G"], case["D"]
        T, n, N = sum(a for a, _ in _runs(case)), len(_runs(case)), case["H"] * case["D"]
        if case["mode"] == "delta":
            C = 2 * G * D + N
            return {"bytes": T * (2 * C + 8 * H + 4 * N) + n * (8 * H * D * D + 24 * C) + 16 * C, "flops": T * (H * D * D * 6 + 8 * C)}
        return {"bytes": T * (16 * N + 64 + 2 * N) + n * 8 * H * D * D + 68 * N, "flops": T * (H * D * D * 4 + 32 * N)}
    if kind == "w4":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": N * K / 2 + 8 * N * (K // 128) + 2 * M * (N + K), "flops": 2 * M * N * K}
    if kind == "qlora":
        T, W, H, Hkv, F = case["B"] * case["S"], case["W"], case["H"], case["Hkv"], case["F"]
        n = W * (H + 2 * Hkv) * 128 + W * H * 128 + 3 * W * F
        return {"bytes": n * 4.5 / 8 + 2 * T * W * 8 + 8 * 4 * (2 * W + (H + Hkv) * 128), "flops": 4 * T * n + 14 * case["B"] * H * 128 * _pairs(case["S"])}
    if kind == "head":
        T, K, V = case["T"], case["K"], case["V"]
        return {"bytes": 2 * V * K * (2 if case["train"] else 1) + 4 * T * K + 8 * T, "flops": (6 if case["train"] else 4) * T * K * V}
    T, W = sum(n for n, _ in _runs(case)), case["W"]
    hd = W // 128
    linear = W * W * (1.5 + 1 + 2.5 + 1) + 2 * 5 * W * W + W * W * (1.5 + 1) + 4 * 6 * W * W
    att = sum(4 * W * (_seen({"opt": "window"}, p) + _seen({"opt": "chunk"}, p)) for n, _ in _runs(case) for p in range(n))
    return {"bytes": 2 * (linear + 32768 * W) + 4 * 32768 * len(_runs(case)) + len(_runs(case)) * 3 * 4 * hd * 128 * 128,
            "flops": 2 * T * linear + att + T * hd * 128 * 128 * (6 + 2 * 4) + 2 * len(_runs(case)) * W * 32768}


def tolerance(case):
    """Largest relative error of another correct implementation at the same precision, about four times what the package's own
    kernels for one job show among themselves (tensor-core and per-token attention: 0.002 on one call, 0.004 on the adapter
    gradients of a layer, 0.003 on the logits of the whole step): bf16 results, products and roundings on the way."""
    return {"attention": {"rel": 0.01}, "packed": {"rel": 0.01}, "paged": {"rel": 0.01}, "mixer": {"rel": 0.01}, "w4": {"rel": 0.01},
            "qlora": {"rel": 0.02}, "head": {"rel": 0.01}, "step": {"rel": 0.015}}[case["kind"]]


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _attend(q, k, v, seen, scale, softcap=0.0, sink=None):
    """q [h, n, D], k / v [h, m, D] in 64 bits, ``seen`` [n, m] bool, ``sink`` [h] -> ([h, n, D], the probabilities)."""
    sc = q @ k.transpose(-1, -2) * scale
    if softcap:
        sc = softcap * torch.tanh(sc / softcap)
    sc = sc.masked_fill(~seen, float("-inf"))
    if sink is not None:
        p = torch.softmax(torch.cat([sc, sink.view(-1, 1, 1).expand(-1, sc.shape[1], 1)], -1), -1)[..., :-1]
    else:
        p = torch.softmax(sc, -1)
    return p @ v, p


def _heads(qkv, B, S, H, Hkv, D):
    x = qkv.view(B, S, H + 2 * Hkv, D).transpose(1, 2)
    return x[:, :H], x[:, H:H + Hkv], x[:, H + Hkv:]


def _exact_attention(qkv, g, B, S, H, Hkv, D, causal):
    rep, scale = H // Hkv, D ** -0.5
    q, k, v = _heads(qkv.detach().double(), B, S, H, Hkv, D)
    go = g.double().view(B, S, H, D).transpose(1, 2)
    out = torch.empty(B, S, H, D, dtype=F64, device=DEV)
    d = torch.empty(B, S, H + 2 * Hkv, D, dtype=F64, device=DEV)
    seen = torch.ones(S, S, dtype=torch.bool, device=DEV)
    seen = seen.tril() if causal else seen
    for b in range(B):
        for j in range(Hkv):
            h = slice(j * rep, (j + 1) * rep)
            kk, vv = k[b, j], v[b, j]
            o, p = _attend(q[b, h], kk.expand(rep, S, D), vv.expand(rep, S, D), seen, scale)
            ds = p * (go[b, h] @ vv.t() - (go[b, h] * o).sum(-1, keepdim=True)) * scale
            out[b, :, h] = o.transpose(0, 1)
            d[b, :, h] = (ds @ kk).transpose(0, 1)
            d[b, :, H + j] = (ds.transpose(-1, -2) @ q[b, h]).sum(0)
            d[b, :, H + Hkv + j] = (p.transpose(-1, -2) @ go[b, h]).sum(0)
    return {"out": out.view(B * S, H * D), "dqkv": d.view(B * S, -1)}


def _exact_packed(case, s):
    H, Hkv, D = case["H"], case["Hkv"], case["D"]
    outs, at = [], 0
    for n in s["lens"]:
        q, k, v = _heads(s["qkv"][at:at + n].double(), 1, n, H, Hkv, D)
        seen = torch.ones(n, n, dtype=torch.bool, device=DEV).tril()
        o = torch.cat([_attend(q[0, h:h + 1], k[0, h * Hkv // H][None], v[0, h * Hkv // H][None], seen, D ** -0.5)[0] for h in range(H)])
        outs.append(o.transpose(0, 1).reshape(n, H * D))
        at += n
    return torch.cat(outs)


def _exact_paged(case, s):
    H, G, D, BS, o = case["H"], case["G"], case["D"], case["page"], _options(case)
    rep, outs, at = H // G, [], 0
    for i, (n, p0) in enumerate(s["runs"]):
        m = p0 + n
        blocks = s["table"][i, :-(-m // BS)].long()
        k, v = (c[blocks].transpose(0, 1).reshape(G, -1, D)[:, :m].double() for c in (s["ck"], s["cv"]))
        p, j = torch.arange(p0, m, device=DEV)[:, None], torch.arange(m, device=DEV)[None, :]
        seen = j <= p
        if o["window"]:
            seen = seen & ((p - j < o["window"]) | (j < o["keep"]))
        if o["chunk"]:
            seen = seen & (p // o["chunk"] == j // o["chunk"])
        q = s["q"][at:at + n].double().view(n, H, D).transpose(0, 1)
        out = torch.cat([_attend(q[h:h + 1], k[h // rep][None], v[h // rep][None], seen, D ** -0.5, o["softcap"],
                                 s["sink"][h:h + 1].double() if o["sink"] else None)[0] for h in range(H)])
        if o["gate"]:
            out = out * torch.sigmoid(s["gate"][at:at + n].double()).t()[:, :, None]
        outs.append(out.transpose(0, 1).reshape(n, H * D))
        at += n
    return torch.cat(outs)


def _exact_mixer(case, s):
    H, G, D = case["H"], case["G"], case["D"]
    N, delta = H * D, case["mode"] == "delta"
    state, zs, tails, at = s["state"].double().clone(), [], [], 0
    for i, (n, p0) in enumerate(s["runs"]):
        rows = slice(at, at + n)
        at += n
        S = state[i] if p0 > 0 else torch.zeros_like(state[i])
        if delta:
            x = s["x"][rows].double()
            old = s["tail"][i].double() if p0 > 0 else torch.zeros_like(s["tail"][i], dtype=F64)
            if 0 < p0 < 3:
                old[:3 - p0] = 0
            ext = torch.cat([old, x])
            y = sum(s["conv_w"][:, j].double() * ext[j:j + n] for j in range(4))
            y = y * torch.sigmoid(y)
            tails.append(ext[n:n + 3])
            q, k = (y[:, c * G * D:(c + 1) * G * D].view(n, G, D) for c in (0, 1))
            q, k = (t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
            q, k = (q * D ** -0.5).repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
            v = y[:, 2 * G * D:].view(n, H, D)
            ab = s["ab"][rows].double()
            a = torch.exp(-torch.exp(s["A_log"].double()) * torch.nn.functional.softplus(ab[:, :H] + s["dt_bias"].double(), threshold=1000.0))
            b = torch.sigmoid(ab[:, H:])
        else:
            q, k, v, post = (s["rkvg"][rows, j * N:(j + 1) * N].double().view(n, H, D) for j in range(4))
            w = torch.exp(-torch.exp(torch.tanh(s["x"][rows].double()) @ s["w2"].double().t() + s["w0"].double())).view(n, H, D)
            u = s["u"].double()
        o = torch.empty(n, H, D, dtype=F64, device=DEV)
        for t in range(n):
            if delta:
                S = S * a[t].view(H, 1, 1)
                r = b[t].view(H, 1) * (v[t] - torch.einsum("hde,hd->he", S, k[t]))
                S = S + k[t][:, :, None] * r[:, None, :]
                o[t] = torch.einsum("hde,hd->he", S, q[t])
            else:
                kv = k[t][:, :, None] * v[t][:, None, :]
                o[t] = torch.einsum("hde,hd->he", S + u[:, :, None] * kv, q[t])
                S = S * w[t][:, :, None] + kv
        state[i] = S
        o = o * torch.rsqrt((o * o).mean(-1, keepdim=True) + 1e-6)
        o = o.reshape(n, N) * (s["w"].double().repeat(H) if delta else s["w"].double())
        p = s["post"][rows].double() if delta else post.reshape(n, N)
        zs.append(o * p * torch.sigmoid(p))
    out = {"z": torch.cat(zs), "state": state}
    if delta:
        out["tail"] = torch.stack(tails)
    return out


def _expand(packed, levels, scale, N, K):
    q = torch.stack([packed >> 4, packed & 15], -1).view(N, K).long()
    return levels[q] * scale.double().view(N, -1).repeat_interleave(K // (scale.numel() // N), 1)


def _exact_qlora(case, s):
    B, S, H, Hkv, D, F = case["B"], case["S"], case["H"], case["Hkv"], 128, case["F"]
    levels = torch.tensor(NF4_LEVELS, dtype=F64, device=DEV)
    lin = lambda x, n: x @ _expand(s[n][0], levels, *s[n][1:]).t()                     # noqa: E731
    norm = lambda x, w: x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6) * w.double()   # noqa: E731
    delta, res, A, Bq, Bv = (s[n].detach().double().requires_grad_() for n in ("delta", "res", "A", "Bq", "Bv"))
    r1 = delta + res
    x = norm(r1, s["n1"])
    qkv = lin(x, "qkv")
    low = x @ A.t() * 2.0                                                               # alpha / r
    zero = torch.zeros(B * S, Hkv * D, dtype=F64, device=DEV)
    qkv = qkv + torch.cat([low[:, :8] @ Bq, zero, low[:, 8:] @ Bv], 1)
    t = qkv.view(B * S, H + 2 * Hkv, D)
    ang = torch.outer(torch.arange(S, dtype=F64, device=DEV), 1e6 ** (-torch.arange(0, D, 2, dtype=F64, device=DEV) / D)).repeat(B, 1)[:, None, :]
    turn = lambda y: torch.cat([y[..., :D // 2] * ang.cos() - y[..., D // 2:] * ang.sin(),
                                y[..., D // 2:] * ang.cos() + y[..., :D // 2] * ang.sin()], -1)   # noqa: E731
    t = torch.cat([turn(norm(t[:, :H], s["qn"])), turn(norm(t[:, H:H + Hkv], s["kn"])), t[:, H + Hkv:]], 1)
    q, k, v = _heads(t.reshape(B * S, -1), B, S, H, Hkv, D)
    seen = torch.ones(S, S, dtype=torch.bool, device=DEV).tril()
    ctx = torch.stack([_attend(q[b], k[b].repeat_interleave(H // Hkv, 0), v[b].repeat_interleave(H // Hkv, 0), seen, D ** -0.5)[0] for b in range(B)])
    r2 = r1 + lin(ctx.transpose(1, 2).reshape(B * S, H * D), "o")
    gu = lin(norm(r2, s["n2"]), "gate_up")
    out = lin(torch.nn.functional.silu(gu[:, :F]) * gu[:, F:], "down")
    torch.autograd.backward([out, r2], [s["g_out"].double(), s["g_res"].double()])
    return {"out": out.detach(), "res": r2.detach(), "ddelta": delta.grad, "dres": res.grad, "dA_q_proj": A.grad[:8], "dA_v_proj": A.grad[8:],
            "dB_q_proj": Bq.grad, "dB_v_proj": Bv.grad}


def _exact_head(case, s):
    x, w, t = s["x"].double(), s["w"].double(), s["t"]
    valid = t >= 0
    n = valid.sum().clamp_min(1)
    loss = torch.zeros((), dtype=F64, device=DEV)
    dx, dw = torch.empty_like(x), torch.zeros_like(w) if case["train"] else None
    for i in range(0, x.shape[0], 512):
        c = slice(i, i + 512)
        z = x[c] @ w.t()
        lp = torch.log_softmax(z, -1)
        at = t[c].clamp_min(0)[:, None]
        loss -= (lp.gather(1, at)[:, 0] * valid[c]).sum() / n
        d = lp.exp_()
        d.scatter_add_(1, at, torch.full_like(at, -1, dtype=F64))
        d *= (valid[c] / n)[:, None]
        dx[c] = d @ w
        if dw is not None:
            dw += d.t() @ x[c]
    return {"loss": loss, "dx": dx, "dw": dw}


def exact(case, seed):
    kind = case["kind"]
    if kind == "step" or (kind == "qlora" and case["p"] > 0):
        return None                                      # a whole model; a dropout mask that only the kernels' counters define
    s = _inputs(case, seed)
    if kind == "attention":
        return _exact_attention(s["qkv"], s["g"], *(case[k] for k in ("B", "S", "H", "Hkv", "D", "causal")))
    if kind == "w4":
        w = _expand(s["packed"], torch.arange(16, dtype=F64, device=DEV) - 8, s["scale"], case["N"], case["K"])
        return s["x"].double() @ w.t()
    return {"packed": _exact_packed, "paged": _exact_paged, "mixer": _exact_mixer, "qlora": _exact_qlora, "head": _exact_head}[kind](case, s)
