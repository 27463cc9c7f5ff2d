"""The performance cases of the library: what a tracking program has it do, at the sizes it does it.

Every case goes through the public entry points and stands for one kind of use:

  event     one event through the ordering and the hierarchical rule: E2LSH ids, one stable sort per (round, hash),
            gather of the hit rows, mixer, output rows put back at their hits (BASELINE configurations 2 and 3)
  plain     chunk_gated_delta_rule on sequences of one length or, with `cu_seqlens`, on a packed batch
            (configurations 0 and 1, and the interleaved sequences of the lshgd layers)
  prefill   chunk_h_gated_delta_rule with `output_final_state`: a prompt of any length and its Fenwick state
  decode    chunk_h_gated_delta_rule on that state, one token per batch row, the state updated in place
  ordering  LSHOrdering.forward: batches of equally long point clouds put into LSH order
  hept      region numbers, input preparation, bucket orders and bucket attention of one event
  model     LSHGatedDelta.forward on a packed batch of events (configuration 4)

Event sizes follow the detector data the library is written for, 6 000 to 60 000 hits.
"""
import math

import torch
import torch.nn.functional as F

import lampa_b200
from lampa_b200.model import LSHGatedDelta

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
ROUNDS, HASHES = 3, 8          # hash rounds and hashes per round of the event pipeline


def listed():
    return [
        # a stream of single tokens through one mixer layer of the model: nothing but latency
        dict(name="decode_b1", kind="decode", batch=1, heads=4, k=32, v=32, levels=17, tokens=1003, dtype="bf16"),
        # 64 streams decoded together at the benchmark's head size: the states are 143 MB
        dict(name="decode_b64", kind="decode", batch=64, heads=8, k=64, v=64, levels=17, tokens=3000, dtype="bf16"),
        # a prompt that does not end on a chunk boundary, 13 levels as the layer's default allows (T <= 4096)
        dict(name="prefill_3001", kind="prefill", batch=1, tokens=3001, heads=8, k=64, v=64, levels=13, dtype="bf16"),
        # configuration 0: a small event, zero initial state
        dict(name="plain_6144", kind="plain", seqs=1, lo=6144, hi=6144, packed=False, heads=4, k=64, v=64,
             initial=False, g_shift=2.0, dtype="bf16"),
        # configuration 1: the long sequence, random initial state
        dict(name="plain_65536", kind="plain", seqs=1, lo=65536, hi=65536, packed=False, heads=8, k=64, v=64,
             initial=True, g_shift=2.0, dtype="bf16"),
        # the lshgd layer of the tracking configuration: 6 heads of 16, V = 32, fp16, two interleaved steps per hit,
        # a few events of odd length packed
        dict(name="plain_packed_lshgd", kind="plain", seqs=4, lo=12001, hi=90001, packed=True, heads=6, k=16, v=32,
             initial=False, g_shift=-3.0, dtype="fp16"),
        # configurations 2 and 3: the largest event (60 000 hits, mixer input padded to 61 440 tokens)
        dict(name="event_60000", kind="event", hits=60000, tokens=61440, heads=8, k=64, v=64, dtype="bf16"),
        # the smallest event of the range, not padded
        dict(name="event_6007", kind="event", hits=6007, tokens=6007, heads=8, k=64, v=64, dtype="bf16"),
        # the ordering layer alone on a batch of point clouds (48 features per point)
        dict(name="ordering_4x1500", kind="ordering", batch=4, points=1500, features=48, coords=6),
        # the bucket attention layer of one large event: buckets of 100, 24 features + 6 coordinates per head
        dict(name="hept_60000", kind="hept", hits=60000, heads=8, features=24, block=100),
        # one event through the whole model, as an online filter runs it
        dict(name="model_1x9001", kind="model", events=1, lo=9001, hi=9001),
        # configuration 4: 64 events in one packed batch (a packed call takes at most 2^21 tokens)
        dict(name="model_64", kind="model", events=64, lo=6000, hi=59000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["event", "event", "plain", "plain", "prefill", "decode", "ordering", "hept", "model"])
    k, v = rng.choice([(64, 64), (64, 64), (32, 32), (16, 32)])
    heads = rng.choice([4, 6, 8])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "event":
        n = _log(rng, 6000, 60000)
        pad = rng.choice([1, 64, 2048])
        return dict(kind=kind, hits=n, tokens=-(-n // pad) * pad, heads=heads, k=k, v=v, dtype=dtype)
    if kind == "plain":
        if rng.random() < 0.5:
            n = _log(rng, 1000, 65536)
            return dict(kind=kind, seqs=max(1, min(rng.randint(1, 4), 65536 // n)), lo=n, hi=n, packed=False,
                        heads=heads, k=k, v=v, initial=rng.random() < 0.5, g_shift=rng.choice([2.0, -3.0]), dtype=dtype)
        lo = _log(rng, 300, 20000)
        return dict(kind=kind, seqs=rng.randint(2, 6), lo=lo, hi=lo * rng.randint(2, 4), packed=True, heads=heads, k=k,
                    v=v, initial=rng.random() < 0.5, g_shift=rng.choice([2.0, -3.0]), dtype=dtype)
    if kind == "prefill":
        n = _log(rng, 200, 20000)
        return dict(kind=kind, batch=rng.randint(1, 4), tokens=n, heads=heads, k=k, v=v,
                    levels=max(13, lampa_b200.num_levels_required(n)), dtype=dtype)
    if kind == "decode":
        return dict(kind=kind, batch=_log(rng, 1, 64), heads=heads, k=k, v=v, levels=rng.choice([17, 18]),
                    tokens=rng.randint(500, 4000), dtype=dtype)
    if kind == "ordering":
        return dict(kind=kind, batch=rng.randint(1, 8), points=_log(rng, 1000, 20000),
                    features=rng.choice([24, 48, 96]), coords=6)
    if kind == "hept":
        return dict(kind=kind, hits=_log(rng, 6000, 60000), heads=rng.choice([4, 8]), features=24, block=100)
    lo = _log(rng, 6000, 30000)
    return dict(kind=kind, events=_log(rng, 1, 24), lo=lo, hi=2 * lo)


def _lengths(case):
    """Lengths of the case's sequences or events, spread evenly over lo..hi and shuffled by a fixed rule."""
    n, lo, hi = case.get("seqs", case.get("events")), case["lo"], case["hi"]
    step = (hi - lo) / max(1, n - 1)
    out = [int(round(lo + step * i)) for i in range(n)]
    return [out[(i * 7 + 3) % n] if n % 7 else out[i] for i in range(n)]


def _cu(lengths):
    cu = torch.zeros(len(lengths) + 1, dtype=torch.int64)
    cu[1:] = torch.tensor(lengths, dtype=torch.int64).cumsum(0)
    return cu.cuda()


def _hits(gen, n, extra=18):
    """Rows [x, y, z, r, phi, eta, features] of hits on ten cylindrical layers (mm)."""
    dev = gen.device
    r = 30.0 + torch.randint(0, 10, (n,), generator=gen, device=dev).float() * (970.0 / 9.0)
    phi = (torch.rand(n, generator=gen, device=dev) * 2 - 1) * math.pi
    z = (torch.rand(n, generator=gen, device=dev) * 2 - 1) * 3000.0
    xyz = torch.stack([r * torch.cos(phi), r * torch.sin(phi), z, r, phi, torch.asinh(z / r)], -1)
    return torch.cat([xyz, torch.randn(n, extra, generator=gen, device=dev)], -1).contiguous()


def _mixer(gen, B, T, H, K, V, dtype, g_shift, levels=None):
    """q, k, v, g, beta (and lambda) of one mixer call."""
    def rn(*shape):
        return torch.randn(*shape, generator=gen, device=gen.device)
    s = {"q": F.normalize(rn(B, T, H, K), dim=-1).to(dtype), "k": F.normalize(rn(B, T, H, K), dim=-1).to(dtype),
         "v": rn(B, T, H, V).to(dtype), "beta": torch.sigmoid(rn(B, T, H)), "g": -F.softplus(rn(B, T, H) + g_shift)}
    if levels is not None:
        s["l"] = F.softplus(rn(B, T, H, levels)).to(dtype)
    return s


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "event":
        n, T = case["hits"], case["tokens"]
        s["x"] = _mixer(gen, 1, T, case["heads"], case["k"], case["v"], DTYPES[case["dtype"]], 2.0,
                        lampa_b200.num_levels_required(T))
        for name in ("k", "v", "beta", "g", "l"):          # padded tokens are inert
            s["x"][name][:, n:] = 0
        s["hits"] = _hits(gen, n)
        s["alpha"] = torch.randn(HASHES, 6, ROUNDS, generator=gen, device="cuda")
        s["shift"] = torch.rand(ROUNDS, generator=gen, device="cuda")
    elif kind == "plain":
        lens = _lengths(case)
        B, T = (1, sum(lens)) if case["packed"] else (len(lens), lens[0])
        s["x"] = _mixer(gen, B, T, case["heads"], case["k"], case["v"], DTYPES[case["dtype"]], case["g_shift"])
        s["cu"] = _cu(lens) if case["packed"] else None
        s["h0"] = (0.1 * torch.randn(len(lens), case["heads"], case["k"], case["v"], generator=gen, device="cuda")
                   if case["initial"] else None)
    elif kind in ("prefill", "decode"):
        # decays of a trained layer: a few per cent per token
        a = (case["heads"], case["k"], case["v"], DTYPES[case["dtype"]], -3.0, case["levels"])
        s["x"] = _mixer(gen, case["batch"], case["tokens"], *a)
        if kind == "decode":
            T = case["tokens"] - case["tokens"] % 64       # the prompt before the streams start
            _, s["state"] = _hier({n: t[:, :T].contiguous() for n, t in s["x"].items()}, None, True)
            s["x"] = _mixer(gen, case["batch"], 1, *a)
    elif kind == "ordering":
        s["coords"] = torch.stack([_hits(gen, case["points"], 0) for _ in range(case["batch"])])
        s["points"] = torch.randn(case["batch"], case["points"], case["features"], generator=gen, device="cuda")
        torch.manual_seed(seed)
        s["layer"] = lampa_b200.LSHOrdering(case["coords"], num_hashes=ROUNDS).cuda()
    elif kind == "hept":
        n, h, d, cd = case["hits"], case["heads"], case["features"], 6
        s["coords"] = torch.randn(n, cd, generator=gen, device="cuda")
        s["coords"][:, 1] = (torch.rand(n, generator=gen, device="cuda") * 2 - 1) * math.pi
        s["q"], s["k"], s["v"] = (
            lampa_b200.pad_to_multiple(a * torch.randn(n, h, d, generator=gen, device="cuda"), case["block"], dims=0)
            for a in (0.6, 0.6, 1.0))
        s["w"] = torch.randn(h, d, cd - 1, 5, generator=gen, device="cuda") * 0.3 - 0.8
        torch.manual_seed(seed)
        s["regions"] = lampa_b200.get_regions(150, ROUNDS, h).cuda()
        s["e2lsh"] = lampa_b200.E2LSH(n_hashes=ROUNDS, n_heads=h, dim=d + cd).cuda()
        s["block"] = case["block"]
    elif kind == "model":
        lens = _lengths(case)
        s["hits"] = _hits(gen, sum(lens))
        s["cu"] = _cu(lens)
        torch.manual_seed(20254)
        s["model"] = LSHGatedDelta(max_hits_per_event=60000).cuda()
    else:
        raise ValueError(kind)
    return s


def _hier(x, state, want_state, out_perm=None):
    return lampa_b200.chunk_h_gated_delta_rule(x["q"], x["k"], x["v"], x["g"], x["l"], x["beta"], initial_state=state,
                                               output_final_state=want_state, use_qk_l2norm_in_kernel=True,
                                               out_perm=out_perm)


def run(s):
    kind = s["kind"]
    if kind == "event":
        ids, perm = lampa_b200.lsh_bucket_sort(s["hits"], s["alpha"], s["shift"], 1.0)
        order = perm[0, 0]
        rows = lampa_b200.permute_rows(s["hits"], order)
        o, _ = _hier(s["x"], None, False, out_perm=order)
        return {"ids": ids, "perm": perm, "rows": rows, "o": o}
    if kind == "plain":
        x = s["x"]
        o, state = lampa_b200.chunk_gated_delta_rule(x["q"], x["k"], x["v"], x["g"], x["beta"], initial_state=s["h0"],
                                                     output_final_state=True, cu_seqlens=s["cu"],
                                                     use_qk_l2norm_in_kernel=True)
        return {"o": o, "state": state}
    if kind in ("prefill", "decode"):
        o, state = _hier(s["x"], s.get("state"), True)
        return {"o": o, "states": state.states, "counts": state.counts}
    if kind == "ordering":
        ordered, idx = s["layer"](s["points"], s["coords"])
        return {"ordered": ordered, "idx": idx}
    if kind == "hept":
        r = lampa_b200.region_inputs(s["coords"], s["regions"], s["block"])
        return lampa_b200.hept_attention_core(s["e2lsh"], s["q"], s["k"], s["v"], s["w"], r["coords"], r["regions_h"],
                                              r["ranks"], r["raw_size"], s["block"])
    return s["model"](s["hits"], s["cu"])


def _rule_flops(T, H, K, V, states):
    """Token recurrence: S <- S - b k (k^T S) + b k v^T and q^T S are 6 K V per token and state that is advanced."""
    return 6.0 * T * H * K * V * states


def _levels(n):
    """Fenwick levels that hold tokens, on average over a sequence of n tokens."""
    return 1 + 0.5 * max(1.0, math.log2(max(2, n)))


def work(case):
    """Inputs read once, outputs written once; operations of the token recurrences (and of the dense layers)."""
    kind = case["kind"]
    if kind == "event":
        n, T, H, K, V = (case[x] for x in ("hits", "tokens", "heads", "k", "v"))
        mixer = T * H * (2 * K + 2 * V) * 2 + T * H * (8 + 2 * lampa_b200.num_levels_required(T))
        order = n * (96 + ROUNDS * HASHES * (4 + 8) + 96)
        return {"bytes": mixer + order, "flops": _rule_flops(n, H, K, V, _levels(n))}
    if kind == "plain":
        T, H, K, V = sum(_lengths(case)), case["heads"], case["k"], case["v"]
        state = case["seqs"] * H * K * V * 4
        return {"bytes": T * H * (2 * K + 2 * V) * 2 + T * H * 8 + state * (2 if case["initial"] else 1),
                "flops": _rule_flops(T, H, K, V, 1)}
    if kind in ("prefill", "decode"):
        B, H, K, V, L = (case[x] for x in ("batch", "heads", "k", "v", "levels"))
        T = case["tokens"] if kind == "prefill" else 1
        rows = B * T * H * ((2 * K + 2 * V) * 2 + 8 + 2 * L)
        state = B * H * K * V * 4
        lv = _levels(case["tokens"])
        # a prefill writes the whole state tensor, a decode step reads and writes the levels that hold tokens
        return {"bytes": rows + state * (L if kind == "prefill" else 2 * lv), "flops": _rule_flops(B * T, H, K, V, lv)}
    if kind == "ordering":
        n = case["batch"] * case["points"]
        return {"bytes": n * (4 * case["coords"] + 8 * case["features"] + 8),
                "flops": n * 2 * (case["coords"] * (ROUNDS + 1) + ROUNDS)}
    if kind == "hept":
        h, d, b = case["heads"], case["features"], case["block"]
        n = -(-case["hits"] // b) * b
        return {"bytes": n * (h * d * 4 * 4 + 24), "flops": ROUNDS * h * n * (b * 2.0 * (d + 6 + d) + 2 * 2 * (d + 6))}
    n = sum(_lengths(case))
    d, H, K, L = 128, 4, 32, 17
    dense = 24 * d * 2 + 4 * (5 * d * d + d * (2 * H + H * L) + 8 * d * d)
    # the residual stream, the projections and the states are free to stay on chip; hits in, embedding out, weights
    return {"bytes": n * 192.0 + 2 * dense, "flops": 2.0 * n * dense + 4 * _rule_flops(n, H, K, K, _levels(30000))}


def tolerance(case):
    kind = case["kind"]
    if kind == "ordering":
        return {"rel": 1e-5, "differ": 1e-3}     # rows follow the order; equal keys may change places
    if kind == "hept":
        return {"rel": 1e-4}                     # fp32 exponents |q|^2 / 2 of a few tens, then exp
    if kind == "model":
        return {"rel": 2e-2}                     # four bf16 blocks behind one another
    return {"rel": 1e-2}                         # bf16 operands and results; ids, orders and counts exact
