"""The work that users of this package have it do, as cases that can be timed one by one.

A case is a plain dict.  `listed()` names the representative ones, `draw(rng)` gives another of the
same ranges, `prepare(case, seed)` makes what a serving process holds before a call (weights, adapters,
routed tokens), `run(state)` is one pass through the public entry points, `work(case)` the bytes and
operations that pass cannot do without, `tolerance(case)` how far another correct implementation of
the same precision may be from it, `exact(case, seed)` the results of a pass in 64 bits.

Ops (the field "op"):
  matmul  matmul_4bit_2_4         one packed int4 2:4 weight, T tokens
  sbmm    sbmm_4bit_2_4_native    one packed delta per token, optionally on a base weight
  ldmm    ldmm                    base weight + a LoRA adapter or a packed delta per token
  bgmv    lora_bgmv               base weight + a LoRA adapter per token, any order (decode)
  sgmv    lora_sgmv               base weight + a LoRA adapter per token segment (prefill)
  stack   DeltaStackShard         every packed linear of decoder layers over one routed batch

Sizes: 1 to 8192 tokens, 1024 to 13824 features, 1 to 128 deltas, ranks 8 to 64, scales per output
channel or per group of 128, fp16 throughout and bf16 where the LoRA operators take it.
"""
import math

import numpy as np
import torch

import triteia_b200.ops as ops
from triteia_b200.stack import LLAMA_7B_FUSED_LINEARS, DeltaStackShard, StackLinear


def listed():
    return [
        # One token through one small packed linear: the least a call can be.
        {"name": "matmul-1tok", "op": "matmul", "T": 1, "K": 2048, "N": 2048, "group": -1},
        # A small decode batch through one 4096 x 4096 packed linear.
        {"name": "matmul-16tok", "op": "matmul", "T": 16, "K": 4096, "N": 4096, "group": 128},
        # The prompts of one tenant (an odd number of tokens) through its MLP up projection.
        {"name": "matmul-prompt", "op": "matmul", "T": 1531, "K": 4096, "N": 11008, "group": 128},
        # 100 requests over 64 fine-tuned models on a common base, the law and size of the operator sweeps.
        {"name": "sbmm-100req", "op": "sbmm", "T": 100, "K": 2048, "N": 2048, "group": -1, "D": 64, "ids": "zipf:2.0",
         "base": True},
        # A decode step of 128 requests over 64 deltas, a tenth of them for the base model only.
        {"name": "sbmm-decode", "op": "sbmm", "T": 128, "K": 4096, "N": 4096, "group": 128, "D": 64, "ids": "uniform",
         "base": False},
        # A mixed step (decode and chunks of prompts): some tens of tokens for each of a dozen deltas.
        {"name": "sbmm-mixed", "op": "sbmm", "T": 700, "K": 4096, "N": 12288, "group": 128, "D": 13, "ids": "uniform",
         "base": False},
        # Prompts of 16 tenants, 512 tokens each, through the up projection of a 13B model.
        {"name": "sbmm-prefill", "op": "sbmm", "T": 8192, "K": 5120, "N": 13824, "group": 128, "D": 32, "ids": "runs:16",
         "base": False},
        # 100 requests, half of the models are adapters and half deltas, the size of the ldmm sweep.
        {"name": "ldmm-100req", "op": "ldmm", "T": 100, "K": 3072, "N": 3072, "group": -1, "D": 16, "M": 16, "R": 16,
         "ids": "zipf:2.0"},
        # A decode step of 256 requests over 32 adapters and 32 deltas with popular and rare ones.
        {"name": "ldmm-decode", "op": "ldmm", "T": 256, "K": 4096, "N": 11008, "group": -1, "D": 32, "M": 32, "R": 16,
         "ids": "true-zipf:1.2"},
        # 100 requests over 64 adapters, the size of the LoRA sweep.
        {"name": "bgmv-100req", "op": "bgmv", "T": 100, "K": 2048, "N": 2048, "M": 64, "R": 32, "ids": "zipf:2.0",
         "dtype": "fp16"},
        # Prompts of 13 adapters of ragged lengths through base weight and adapter, bfloat16.
        {"name": "sgmv-prefill", "op": "sgmv", "T": 7001, "K": 5120, "N": 13824, "M": 16, "R": 64, "ids": "ragged:13",
         "dtype": "bf16"},
        # All packed linears of a 7B decoder layer, 512 tokens over 128 deltas of very different popularity.
        {"name": "stack-layer", "op": "stack", "T": 512, "H": 4096, "I": 11008, "L": 1, "group": 128, "D": 128,
         "ids": "true-zipf:1.5"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _features(rng, lo=1024, hi=13824, step=128):
    return max(1, round(_log_int(rng, lo, hi) / step)) * step


def draw(rng):
    """One more case of the same ranges: sizes spread over their logarithm, odd ones among them."""
    op = rng.choice(["matmul", "matmul", "sbmm", "sbmm", "sbmm", "ldmm", "ldmm", "bgmv", "sgmv", "stack"])
    if op == "stack":
        h = _features(rng, 1024, 4096)
        return {"op": op, "T": _log_int(rng, 16, 512), "H": h, "I": _features(rng, h, 11008), "L": rng.choice([1, 2]),
                "group": rng.choice([-1, 128]), "D": _log_int(rng, 4, 32), "ids": rng.choice(["uniform", "true-zipf:1.5"])}
    case = {"op": op, "T": _log_int(rng, 1, 8192), "K": _features(rng, hi=11008), "N": _features(rng, hi=12288)}
    if op == "matmul":
        case["group"] = rng.choice([-1, 128])
    elif op == "sbmm":
        prefill = case["T"] > 1024
        case.update(group=rng.choice([-1, 128]), D=_log_int(rng, 2, 64),
                    ids="ragged:%d" % rng.randint(2, 16) if prefill else rng.choice(["uniform", "zipf:2.0", "true-zipf:1.2"]),
                    base=rng.random() < 0.4)
        if prefill:
            case["D"] = max(case["D"], int(case["ids"].split(":")[1]))
    elif op == "ldmm":
        case.update(T=_log_int(rng, 1, 512), group=rng.choice([-1, 128]), D=_log_int(rng, 1, 48), M=_log_int(rng, 1, 48),
                    R=rng.choice([8, 16, 32, 64]), ids=rng.choice(["uniform", "zipf:2.0", "true-zipf:1.2"]))
    elif op == "bgmv":
        case.update(T=_log_int(rng, 1, 512), M=_log_int(rng, 1, 100), R=rng.choice([8, 16, 32, 64]),
                    ids=rng.choice(["uniform", "zipf:2.0", "true-zipf:1.2"]), dtype=rng.choice(["fp16", "bf16"]))
    else:
        m = rng.randint(1, 16)
        case.update(T=_log_int(rng, 128, 8192), M=m, R=rng.choice([16, 32, 64]), ids="ragged:%d" % rng.randint(1, m),
                    dtype=rng.choice(["fp16", "bf16"]))
    case["T"] = max(1, min(case["T"], int(3.3e11) // (case["K"] * case["N"])))     # no costlier than the largest listed ones
    return case


# ------------------------------------------------------------------------------------------- inputs
def _id_law(case):
    """(ids, probabilities) of one token's id, for the laws that draw every token on its own."""
    n = case.get("D", 0) + case.get("M", 0)
    law, _, arg = case["ids"].partition(":")
    if law == "uniform":        # a tenth of the requests is for the base model (in the stack every row has a delta)
        none = 0.0 if case["op"] == "stack" else 0.1
        return np.arange(-1, n), np.array([none] + [(1 - none) / n] * n)
    if law == "zipf":           # ops.generate_model_distribution's law: popular ids are the high ones, -1 the rarest
        p = np.arange(1, n + 2, dtype=np.float64) ** float(arg)
        return np.arange(-1, n), p / p.sum()
    p = np.arange(1, n + 1, dtype=np.float64) ** -float(arg)
    return np.arange(n), p / p.sum()


def _run_lengths(case, rng):
    law, _, arg = case["ids"].partition(":")
    runs, T = min(int(arg), case["T"]), case["T"]
    if law == "runs":
        return [T // runs + (i < T % runs) for i in range(runs)]
    cuts = np.sort(rng.choice(np.arange(1, T), runs - 1, replace=False)) if runs > 1 else np.array([], dtype=int)
    return np.diff(np.concatenate([[0], cuts, [T]])).tolist()


def _ids(case, seed):
    rng = np.random.default_rng(seed)
    if case["ids"].startswith(("runs", "ragged")):
        lengths = _run_lengths(case, rng)
        which = np.sort(rng.choice(case.get("D", case.get("M")), len(lengths), replace=False))
        return np.repeat(which, lengths).astype(np.int32)
    values, p = _id_law(case)
    if case["ids"].startswith("true-zipf"):       # the popular ids lie anywhere among adapters and deltas
        values = rng.permutation(values)
    return rng.choice(values, case["T"], p=p).astype(np.int32)


def _packed(num, k, n, group, gen, device):
    """`num` packed deltas drawn in the packed format: non-zero levels at two positions of every four
    along K (as ops.random_packed_deltas draws them, without going through unpacked weights)."""
    pairs = torch.tensor([4, 8, 12, 9, 13, 14], dtype=torch.int32, device=device)             # metadata of one group of four
    four = lambda t: (t[:, None, None, None] << 12 | t[None, :, None, None] << 8 | t[None, None, :, None] << 4 | t).flatten()
    meta_lut = four(pairs).to(torch.int16)
    code_lut = four(torch.tensor([c for c in range(1, 16) if c != 8], dtype=torch.int32, device=device)).to(torch.int16)
    rnd = lambda size, hi: torch.randint(0, hi, size, generator=gen, device=device, dtype=torch.int32)
    q = torch.empty(num, k // 32, 2 * n, dtype=torch.int32, device=device)
    meta = torch.empty(num, n, k // 16, dtype=torch.int16, device=device)
    for d in range(num):
        torch.index_select(code_lut, 0, rnd((k // 32 * 4 * n,), code_lut.numel()), out=q[d].view(torch.int16).view(-1))
        torch.index_select(meta_lut, 0, rnd((n * k // 16,), meta_lut.numel()), out=meta[d].view(-1))
    s = torch.rand(num, 1 if group == -1 else k // group, n, generator=gen, device=device) * 0.009 + 0.001
    return q, meta, s.half()


def prepare(case, seed):
    device, op, T = torch.device("cuda"), case["op"], case["T"]
    gen = torch.Generator(device).manual_seed(seed)
    dtype = torch.bfloat16 if case.get("dtype") == "bf16" else torch.float16
    normal = lambda *size, std=1.0: (torch.randn(*size, generator=gen, device=device, dtype=torch.float32) * std).to(dtype)
    st = {"op": op}
    if op == "matmul":
        q, meta, s = _packed(1, case["K"], case["N"], case["group"], gen, device)
        st.update(x=normal(T, case["K"]), q=q[0], meta=meta[0], s=s[0])
        return st
    st["ids"] = torch.from_numpy(_ids(case, seed)).to(device)
    if op == "stack":
        layers = [[StackLinear(name, k, n, *_packed(case["D"], k, n, case["group"], gen, device))
                   for name, k, n in _linears(case)] for _ in range(case["L"])]
        st.update(stack=DeltaStackShard(layers), x={k: normal(T, k) for k in sorted({case["H"], case["I"]})})
        return st
    k, n = case["K"], case["N"]
    st["x"] = normal(T, k)
    if "D" in case:
        st["q"], st["meta"], st["s"] = _packed(case["D"], k, n, case["group"], gen, device)
    st["base"] = normal(n, k, std=0.02) if case.get("base", True) else None
    if "M" in case:
        st["A"] = normal(case["M"], k, case["R"], std=k ** -0.5)
        st["B"] = normal(case["M"], case["R"], n, std=case["R"] ** -0.5)
    return st


def _linears(case):
    """The four fused linears of a decoder layer at the case's hidden and MLP sizes."""
    scale = {4096: case["H"], 11008: case["I"], 3 * 4096: 3 * case["H"], 2 * 11008: 2 * case["I"]}
    return [(name, scale[k], scale[n]) for name, k, n in LLAMA_7B_FUSED_LINEARS]


# --------------------------------------------------------------------------------------------- pass
def run(st):
    op = st["op"]
    if op == "matmul":
        return ops.matmul_4bit_2_4(st["q"], st["x"], st["meta"], st["s"])
    if op == "sbmm":
        return ops.sbmm_4bit_2_4_native(st["q"], st["x"], st["meta"], st["s"], st["ids"], base_weight=st["base"])
    if op == "ldmm":
        return ops.ldmm(st["ids"], st["x"], st["A"], st["B"], st["q"], st["meta"], st["s"], base_weight=st["base"])
    if op == "bgmv":
        return ops.lora_bgmv(st["A"], st["B"], st["x"], st["ids"], base_weight=st["base"])
    if op == "sgmv":
        return ops.lora_sgmv(st["A"], st["B"], st["x"], st["ids"], base_weight=st["base"])
    return st["stack"](st["x"], st["ids"])


# --------------------------------------------------------------------------------------------- cost
def _touched(case):
    """Expected (deltas touched, adapters touched, rows with a delta, rows with an adapter)."""
    T, m = case["T"], case.get("M", 0)
    if case["ids"].startswith(("runs", "ragged")):
        runs = min(int(case["ids"].split(":")[1]), T)
        return (runs, 0, T, 0) if "D" in case else (0, runs, 0, T)
    values, p = _id_law(case)
    if case["ids"].startswith("true-zipf") and m:      # ids are shuffled: the two kinds share the law
        share = m / len(values)
        d = float((1 - (1 - p) ** T).sum())
        return d * (1 - share), d * share, T * (1 - share), T * share
    delta, lora = values >= m, (values >= 0) & (values < m)
    hit = 1 - (1 - p) ** T
    return float(hit[delta].sum()), float(hit[lora].sum()), T * float(p[delta].sum()), T * float(p[lora].sum())


def work(case):
    """Bytes: activations and ids in, results out, every touched weight once.  Operations: a multiply and
    an add per token and STORED weight (a 2:4 weight stores half of its positions)."""
    T, op = case["T"], case["op"]
    packed = lambda k, n: k * n * 3 // 8 + (1 if case["group"] == -1 else k // 128) * n * 2
    if op == "matmul":
        k, n = case["K"], case["N"]
        return {"bytes": packed(k, n) + 2 * T * (k + n), "flops": T * k * n}
    deltas, adapters, rows_d, rows_l = _touched(case)
    if op == "stack":
        lin = _linears(case) * case["L"]
        b = sum(deltas * packed(k, n) for _, k, n in lin) + 2 * T * (case["H"] + case["I"] + lin[-1][2]) + 8 * T
        return {"bytes": int(b), "flops": int(rows_d * sum(k * n for _, k, n in lin))}
    k, n = case["K"], case["N"]
    b, f = 2 * T * (k + n) + 4 * T, 0.0
    if "D" in case:
        b, f = b + deltas * packed(k, n), f + rows_d * k * n
    if "M" in case:
        b, f = b + adapters * 2 * case["R"] * (k + n), f + rows_l * 2 * case["R"] * (k + n)
    if case.get("base", True):
        b, f = b + 2 * k * n, f + 2 * T * k * n
    return {"bytes": int(b), "flops": int(f)}


def tolerance(case):
    """About four times the distance of the path from the same product in 64 bits: 2.1e-4 to 2.9e-4 in
    fp16 (one rounding of the result, of the parts it is added from and of scaled weights), 2.6e-3 in
    bf16; single values up to 2e-3 and 1.5e-2."""
    if case.get("dtype") == "bf16":
        return {"rel": 1e-2, "max": 6e-2}
    return {"rel": 1.2e-3, "max": 8e-3}


# -------------------------------------------------------------------------------------------- exact
def _dense(q, meta, s):
    """Packed weight -> float64 [K, N], from the storage format alone.  A word of 8 codes serves 8 output columns and 16
    stored rows per slab; a metadata nibble holds the two kept positions of a group of four along K."""
    kt, n = q.shape[0], q.shape[1] // 2
    codes = (q.view(kt, n // 64, 8, 4, 4, 1) >> torch.arange(0, 32, 4, device=q.device, dtype=torch.int32)) & 15
    codes = codes.view(kt, n // 64, 8, 4, 4, 2, 2, 2)               # slab, block, lane / 4, lane % 4, word, and 3 bits of the nibble
    levels = codes.permute(0, 7, 3, 5, 1, 2, 6, 4).reshape(kt * 8, 2, n) - 8
    r = torch.arange(n, device=q.device)[:, None]
    c = torch.arange(kt * 2, device=q.device)[None, :]
    at = r // 64 * 64 + r % 2 * 2 + r % 8 // 4 + r % 4 // 2 * 32 + r % 64 // 8 * 4
    swap = ((at % 2 == 0) & (c % 2 == 1)).long() - ((at % 2 == 1) & (c % 2 == 0)).long()
    at, c = at + swap, c - swap
    words = meta.reshape(-1)[c // 2 * n * 2 + at * 2 + c % 2].int()[:, :, None]
    nibbles = ((words >> torch.arange(0, 16, 4, device=q.device, dtype=torch.int32)) & 15).reshape(n, kt * 8)
    place = torch.stack([nibbles & 3, nibbles >> 2], 1).permute(2, 1, 0).long()
    w = torch.zeros(kt * 8, 4, n, dtype=torch.float64, device=q.device).scatter_(1, place, levels.double()).view(kt * 32, n)
    scale = s.double()
    if s.shape[0] > 1:                          # group scales: every 8 columns are stored in the order 0 4 1 5 2 6 3 7
        scale = scale.view(-1, n // 8, 4, 2).transpose(2, 3).reshape(-1, n)
    return (w.view(s.shape[0], -1, n) * scale[:, None, :]).view(-1, n)


def exact(case, seed):
    """What `run` returns for these inputs, in 64 bits."""
    st = prepare(case, seed)
    if case["op"] == "matmul":
        return st["x"].double() @ _dense(st["q"], st["meta"], st["s"])
    ids = st["ids"].cpu().numpy()
    rows = {int(d): torch.from_numpy(np.flatnonzero(ids == d)).cuda() for d in np.unique(ids) if d >= 0}
    if case["op"] == "stack":
        sums = torch.zeros(case["T"], dtype=torch.float64, device="cuda")
        for lin in [lin for layer in st["stack"].layers for lin in layer]:
            y = torch.empty(case["T"], lin.n, dtype=torch.float64, device="cuda")
            for d, at in rows.items():
                y[at] = st["x"][lin.k][at].double() @ _dense(lin.qweights[d], lin.metas[d], lin.scales[d])
            sums += y.sum(1)
        return y, sums
    x, m = st["x"].double(), case.get("M", 0)
    y = torch.zeros(case["T"], case["N"], dtype=torch.float64, device="cuda") if st["base"] is None else x @ st["base"].double().t()
    for d, at in rows.items():
        if d < m:
            y[at] += x[at] @ st["A"][d].double() @ st["B"][d].double()
        else:
            y[at] += x[at] @ _dense(st["q"][d - m], st["meta"][d - m], st["s"][d - m])
    return y
