"""The work that users of this package have it do, as a list of cases that can be timed.

Four kinds, all through the public entry points:

* ``decode``    attention of one query row per sequence over packed planes - one call per layer, either called
                directly (an eager model loop) or captured once in a CUDA graph and replayed (a serving loop);
* ``step``      one captured serving step of a request pool: store the new row of every request, gather the residual
                rows, attend;
* ``generate``  a short request from the start to the end in an eager loop: prefill, then token by token;
* ``pack``      quantize and pack a block of a prompt's keys and values.

``listed()`` are fixed sizes, ``draw(rng)`` gives others of the same ranges.  Keys and values are N(0, 1) with four
channels per head ``mag`` times larger, which is what the benchmark and the tests use.
"""
import random

import torch

from open_ommx_serve_b200.attention.kv_pool import MultiSeqKVPool
from open_ommx_serve_b200.attention.kv_store import CanonicalKVStore
from open_ommx_serve_b200.attention.kv_window import WindowSpec
from open_ommx_serve_b200.attention.pack import alloc_planes, ommx_pack_kv_canonical_block, ommx_pack_kv_into
from open_ommx_serve_b200.attention.paged_decode import _auto_num_kv_splits, ommx_paged_decode_attention_canonical

D = 128                       # head dim of every geometry here
WINDOW = WindowSpec(8, 32, 32, 16)
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
PAGE_PLANES = ("k_base", "v_main", "v_scale", "v_zp")
GROUP_PLANES = ("k_scale", "k_zp", "k_obmp", "k_oidx", "k_oval", "k_fp4_mapscale", "k_fp4_mapcenter")
CHUNK = 16384                 # tokens whose inputs are made at a time


def _decode(batch, lo, hi, heads=8, gqa=4, layers=1, graph=False, out="f32", k=6, mag=12, page=16, index="bitmap"):
    return {"kind": "decode", "batch": batch, "lo": lo, "hi": hi, "heads": heads, "gqa": gqa, "layers": layers,
            "graph": graph, "out": out, "k": k, "mag": mag, "page": page, "index": index}


def _step(batch, lo, hi, heads=8, gqa=4, k=6, split=512):
    return {"kind": "step", "batch": batch, "lo": lo, "hi": hi, "heads": heads, "gqa": gqa, "k": k, "split": split}


def _generate(batch, prompt, tokens, heads=8, gqa=4, k=6):
    return {"kind": "generate", "batch": batch, "prompt": prompt, "tokens": tokens, "heads": heads, "gqa": gqa, "k": k}


def _pack(tokens, heads=8, k=6, dtype="bf16", form="into", index="bitmap", page=16, mag=12):
    return {"kind": "pack", "tokens": tokens, "heads": heads, "k": k, "dtype": dtype, "form": form, "index": index,
            "page": page, "mag": mag}


def listed():
    return [
        # one layer of a chat turn on Llama-3.1-8B heads, called eagerly: latency and launches count
        {"name": "decode_1k", **_decode(1, 1024, 1024)},
        # the 32 layers of a token at 4K, captured and replayed
        {"name": "stack_4k_graph", **_decode(1, 4096, 4096, layers=32, graph=True)},
        # a long document at a ragged length, the output in the model's own type
        {"name": "decode_16k_bf16out", **_decode(1, 16461, 16461, out="bf16")},
        # the benchmark's headline context
        {"name": "decode_64k", **_decode(1, 65536, 65536)},
        # 128K over four GPUs: two kv heads are left to each
        {"name": "decode_128k_2heads", **_decode(1, 131072, 131072, heads=2)},
        # Llama-3.1-70B heads, eight long requests on one GPU (the largest case) ...
        {"name": "decode_70b_8x32k", **_decode(8, 32768, 32768, gqa=8)},
        # ... and the share of one GPU out of eight
        {"name": "decode_70b_8x32k_1head", **_decode(8, 32768, 32768, heads=1, gqa=8)},
        # a serving step over 32 requests of 1K to 32K tokens, captured: store, residual gather, attention
        {"name": "step_32x1k_32k", **_step(32, 1024, 32768)},
        # one short request in an eager loop: prompt, then 32 tokens
        {"name": "generate_512", **_generate(1, 512, 32)},
        # eight requests in an eager loop over the pool, at an odd prompt length
        {"name": "generate_8x1333", **_generate(8, 1333, 32)},
        # prefill: an 8K chunk packed straight into the request's pages
        {"name": "pack_8k", **_pack(8192)},
        # a block packed into fresh planes, half precision in, checked for non-finite values
        {"name": "pack_block_1k_f16", **_pack(1024, dtype="f16", form="block", index="relidx7")},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "step", "generate", "pack", "pack"))
    heads, gqa = rng.choice(((8, 4), (8, 4), (8, 8), (4, 4), (2, 4), (1, 8), (1, 4), (8, 1)))
    k = rng.choice((6, 6, 6, 2, 4, 8))
    if kind == "decode":
        batch = _log_int(rng, 1, 32)
        budget = 8 * 32768 * 8                                   # (token, kv head) pairs of the largest listed case
        hi = _log_int(rng, 256, min(131072, budget // (batch * heads)))
        lo = hi if rng.random() < 0.5 else _log_int(rng, max(64, hi // 8), hi)
        graph = rng.random() < 0.3
        layers = rng.choice((1, 2, 8, 32)) if graph else 1
        while batch * hi * heads * layers > budget:
            layers //= 2
        return _decode(batch, lo, hi, heads, gqa, max(1, layers), graph, rng.choice(("f32", "bf16")),
                       rng.choice((k, k, 0, 12)), rng.choice((4, 12, 30)), rng.choice((16, 16, 16, 8, 32)),
                       "bitmap" if k not in (6, 8) or rng.random() < 0.8 else "relidx7")
    if kind == "step":
        batch = _log_int(rng, 1, 32)
        hi = _log_int(rng, 256, min(32768, 8 * 32768 * 8 // (batch * heads)))
        return _step(batch, _log_int(rng, max(64, hi // 16), hi), hi, heads, gqa, k)
    if kind == "generate":
        batch = _log_int(rng, 1, 16)
        return _generate(batch, _log_int(rng, 40, min(8192, 8 * 1333 * 8 // (batch * heads))), rng.randint(8, 32), heads, gqa, k)
    form = rng.choice(("into", "into", "block"))
    return _pack(32 * _log_int(rng, 1, 1024 if form == "into" else 256), heads, k, rng.choice(("bf16", "bf16", "f16", "f32")),
                 form, rng.choice(("bitmap", "relidx7")) if form == "block" else "bitmap", rng.choice((16, 16, 8, 32)),
                 rng.choice((4, 12, 30)))


def _lengths(case):
    """Sequence lengths of a batch: the same for every seed, spread over [lo, hi], the longest of them hi."""
    rng = random.Random("%d %d %d" % (case["batch"], case["lo"], case["hi"]))
    return [case["hi"]] + [rng.randint(case["lo"], case["hi"]) for _ in range(case["batch"] - 1)]


class _Source:
    """Keys, values and queries of one seed."""

    def __init__(self, seed, heads, mag):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)
        self.scale = torch.ones(heads, D, device="cuda")
        for h in range(heads):
            self.scale[h, torch.randperm(D, generator=self.gen, device="cuda")[:4]] = float(mag)
        self.heads = heads

    def kv(self, tokens, dtype=torch.bfloat16):
        K = torch.randn(tokens, self.heads, D, generator=self.gen, device="cuda") * self.scale
        V = torch.randn(tokens, self.heads, D, generator=self.gen, device="cuda")
        return K.to(dtype), V.to(dtype)

    def q(self, *shape):
        return torch.randn(*shape, D, generator=self.gen, device="cuda").bfloat16()


def _attend(q, planes, tables, tails, lens, o, lse, k, page, use_relidx7=False, **kw):
    k_tail, v_tail, b_tail = tails
    ommx_paged_decode_attention_canonical(
        q, planes["k_base"], planes["k_scale"], planes["k_zp"], planes.get("k_oidx"), planes.get("k_oval"),
        planes["v_main"], planes["v_scale"], planes["v_zp"], k_tail, v_tail, b_tail, o, lse, tables[0], tables[1], lens,
        sm_scale=D ** -0.5, page_size=page, k_outliers_per_vector=k, bitmap_read=k > 0 and not use_relidx7,
        k_obmp=planes.get("k_obmp"), k_fp4_mapscale=planes.get("k_fp4_mapscale"),
        k_fp4_mapcenter=planes.get("k_fp4_mapcenter"), kv_outlier_map=k > 0, kv_int8_scale=True, **kw)


def _captured(step):
    """``step`` as a CUDA graph, with what it returns."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    return graph


# ── decode ────────────────────────────────────────────────────────────────────────────────────────────────────────
def _prepare_decode(case, seed):
    B, H, Hq, k, page = case["batch"], case["heads"], case["heads"] * case["gqa"], case["k"], case["page"]
    lens = _lengths(case)
    packed = [WINDOW.packed_len(n) for n in lens]
    tail = [n - p for n, p in zip(lens, packed)]
    groups = [p // 32 for p in packed]
    n_groups, n_pages, ppg = sum(groups), sum(groups) * (32 // page), 32 // page
    src = _Source(seed, H, case["mag"])
    pages = torch.randperm(n_pages, generator=src.gen, device="cuda").to(torch.int32)      # a shared pool in shuffled order
    slots = torch.randperm(n_groups, generator=src.gen, device="cuda").to(torch.int32)
    r2t = torch.zeros(B, max(groups) * ppg, dtype=torch.int32, device="cuda")
    r2g = torch.zeros(B, max(groups), dtype=torch.int32, device="cuda")
    at = 0
    for b, g in enumerate(groups):
        r2t[b, :g * ppg] = pages[at * ppg:(at + g) * ppg]
        r2g[b, :g] = slots[at:at + g]
        at += g
    relidx7 = case["index"] == "relidx7" and k > 0
    layers = []
    for _ in range(case["layers"]):
        planes = {}
        for g0 in range(0, n_groups, CHUNK // 32):
            n = min(CHUNK // 32, n_groups - g0)
            part = ommx_pack_kv_canonical_block(
                *src.kv(32 * n), outliers_per_vector=k, page_size=page, outlier_repr=case["index"], outlier_select="signed",
                use_pow2=True, kv_outlier_map=True, kv_int8_scale=True, check_finite=False)
            for names, where, total in ((PAGE_PLANES, pages[g0 * ppg:(g0 + n) * ppg], n_pages),
                                        (GROUP_PLANES, slots[g0:g0 + n], n_groups)):
                for name in names:
                    if part.get(name) is not None:
                        if name not in planes:
                            planes[name] = torch.empty(total, *part[name].shape[1:], dtype=part[name].dtype, device="cuda")
                        planes[name][where.long()] = part[name]
        kt, vt = src.kv(B * max(tail))
        layers.append({"planes": planes, "q": src.q(B, Hq), "k_tail": kt.view(B, -1, H, D), "v_tail": vt.view(B, -1, H, D)})
    splits = _auto_num_kv_splits(max(packed), B, device="cuda", kv_heads=H)
    state = {"kind": "decode", "layers": layers, "tables": (r2t, r2g), "k": k, "page": page, "relidx7": relidx7,
             "o": torch.empty(case["layers"], B, Hq, D, dtype=DTYPES[case["out"]], device="cuda"),
             "lse": torch.empty(case["layers"], B, Hq, dtype=torch.float32, device="cuda"),
             "b_seq": torch.tensor(packed, dtype=torch.int32, device="cuda"),
             "b_tail": torch.tensor(tail, dtype=torch.int32, device="cuda"),
             "kw": {"num_kv_splits": splits, "max_seq_len": max(packed), "max_tail_len": max(tail),
                    "attn_logits": torch.empty(B, Hq, splits + 1, D + 1, dtype=torch.float32, device="cuda")}}
    if case["graph"]:
        state["graph"] = _captured(lambda: _run_decode_layers(state))
    return state


def _run_decode_layers(state):
    for layer, o, lse in zip(state["layers"], state["o"], state["lse"]):
        _attend(layer["q"], layer["planes"], state["tables"], (layer["k_tail"], layer["v_tail"], state["b_tail"]),
                state["b_seq"], o, lse, state["k"], state["page"], state["relidx7"], **state["kw"])


def _run_decode(state):
    if "graph" in state:
        state["graph"].replay()
    else:
        _run_decode_layers(state)
    return {"o": state["o"], "lse": state["lse"]}


# ── one captured step of a request pool ───────────────────────────────────────────────────────────────────────────
def _prepare_step(case, seed):
    B, H, Hq = case["batch"], case["heads"], case["heads"] * case["gqa"]
    lens = _lengths(case)
    src = _Source(seed, H, 12)
    pool = MultiSeqKVPool(D, H, B, max(lens) + 64, outliers_per_vector=case["k"], window=WINDOW)
    for r, n in enumerate(lens):
        pool.append_block(r, *src.kv(n))
    T = pool.max_tail_len
    tidx = torch.zeros(B, T, dtype=torch.int64)
    packed, tail = [], []
    for r, n in enumerate(lens):                        # where the residual rows are once the new row is in
        idx = WINDOW.tail_indices(n + 1)
        tidx[r, :len(idx)] = torch.tensor(idx)
        packed.append(WINDOW.packed_len(n + 1))
        tail.append(len(idx))
    splits = max(1, -(-max(packed) // case["split"]))
    K, V = src.kv(B)
    state = {"kind": "step", "pool": pool, "K": K, "V": V, "q": src.q(B, Hq), "k": case["k"],
             "rows": torch.arange(B, dtype=torch.int64, device="cuda"), "cols": torch.tensor(lens, dtype=torch.int64, device="cuda"),
             "tidx": tidx.cuda(), "b_seq": torch.tensor(packed, dtype=torch.int32, device="cuda"),
             "b_tail": torch.tensor(tail, dtype=torch.int32, device="cuda"),
             "kt": torch.zeros(B, T, H, D, dtype=torch.bfloat16, device="cuda"),
             "vt": torch.zeros(B, T, H, D, dtype=torch.bfloat16, device="cuda"),
             "o": torch.empty(B, Hq, D, dtype=torch.float32, device="cuda"),
             "lse": torch.empty(B, Hq, dtype=torch.float32, device="cuda"), "splits": splits, "max_packed": max(packed),
             "ws": torch.empty(B, Hq, splits + 1, D + 1, dtype=torch.float32, device="cuda")}
    state["graph"] = _captured(lambda: _step_calls(state))
    return state


def _step_calls(s):
    pool = s["pool"]
    pool.append_decode_captured(s["rows"], s["cols"], s["K"], s["V"])
    d = pool.decode_inputs_captured(s["rows"], s["b_seq"], s["b_tail"], s["tidx"], s["kt"], s["vt"], s["max_packed"])
    _attend(s["q"], d["planes"], (d["req_to_token"], d["req_to_group"]), (d["k_tail"], d["v_tail"], d["b_tail_len"]),
            d["b_seq_len"], s["o"], s["lse"], s["k"], pool.ps, max_seq_len=d["max_seq_len"], max_tail_len=d["max_tail_len"],
            num_kv_splits=s["splits"], attn_logits=s["ws"])


def _run_step(state):
    state["graph"].replay()
    pool = state["pool"]
    return {"o": state["o"], "lse": state["lse"], "kt": state["kt"], "vt": state["vt"], "k_hist": pool.k_hist, "v_hist": pool.v_hist,
            **{name: t for name, t in pool.planes.items() if t is not None}}


# ── a request from prompt to last token, eagerly ──────────────────────────────────────────────────────────────────
def _prepare_generate(case, seed):
    B, H, Hq, n, steps = case["batch"], case["heads"], case["heads"] * case["gqa"], case["prompt"], case["tokens"]
    src = _Source(seed, H, 12)
    kw = dict(outliers_per_vector=case["k"], window=WINDOW)
    cap = n + steps + 32
    store = CanonicalKVStore(D, H, cap, **kw) if B == 1 else MultiSeqKVPool(D, H, B, cap, **kw)
    return {"kind": "generate", "store": store, "single": B == 1, "B": B, "k": case["k"], "max_packed": WINDOW.packed_len(n + steps),
            "prompt": [src.kv(n) for _ in range(B)], "rows": [src.kv(B) for _ in range(steps)], "q": src.q(steps, B, Hq),
            "o": torch.empty(steps, B, Hq, D, dtype=torch.bfloat16, device="cuda"),
            "lse": torch.empty(steps, B, Hq, dtype=torch.float32, device="cuda")}


def _run_generate(s):
    store, B = s["store"], s["B"]
    if s["single"]:
        store.reset_inplace()
        store.append_block(*s["prompt"][0])
    else:
        for r in range(B):
            store.append_block(r, *s["prompt"][r])
    for t, (K, V) in enumerate(s["rows"]):
        if s["single"]:
            store.append(K[0], V[0])
            store.maybe_regroup()
            d = store.decode_inputs()
            tables = (d["planes"]["req_to_token"], d["planes"]["req_to_group"])
        else:
            store.append_decode_device(K, V, B)
            d = store.decode_inputs_device(B, s["max_packed"])
            tables = (d["req_to_token"], d["req_to_group"])
        _attend(s["q"][t], d["planes"], tables, (d["k_tail"], d["v_tail"], d["b_tail_len"]), d["b_seq_len"], s["o"][t], s["lse"][t],
                s["k"], store.ps, max_seq_len=d["max_seq_len"], max_tail_len=d["max_tail_len"])
    names = PAGE_PLANES + tuple(x for x in GROUP_PLANES if x != "k_oidx")
    planes = {name: getattr(store, name) for name in names}
    return {"o": s["o"], "lse": s["lse"], "k_hist": store.k_hist, "v_hist": store.v_hist, **planes}


# ── quantize and pack ─────────────────────────────────────────────────────────────────────────────────────────────
def _prepare_pack(case, seed):
    T, H, page = case["tokens"], case["heads"], case["page"]
    src = _Source(seed, H, case["mag"])
    K, V = src.kv(T, DTYPES[case["dtype"]])
    state = {"kind": "pack", "K": K, "V": V, "k": case["k"], "page": page, "form": case["form"], "index": case["index"]}
    if case["form"] == "into":
        state["planes"] = alloc_planes(T // page, T // 32, H, D, page_size=page, outliers_per_vector=case["k"])
        state["pages"] = torch.randperm(T // page, generator=src.gen, device="cuda").to(torch.int32)
        state["slots"] = torch.randperm(T // 32, generator=src.gen, device="cuda").to(torch.int32)
    return state


def _run_pack(s):
    if s["form"] == "into":
        ommx_pack_kv_into(s["K"], s["V"], s["planes"], dst_pages=s["pages"], dst_groups=s["slots"], outliers_per_vector=s["k"])
        planes = s["planes"]
    else:
        planes = ommx_pack_kv_canonical_block(s["K"], s["V"], outliers_per_vector=s["k"], page_size=s["page"], outlier_repr=s["index"],
                                              outlier_select="signed", use_pow2=True, kv_outlier_map=True, kv_int8_scale=True)
    return {name: planes[name] for name in PAGE_PLANES + GROUP_PLANES if planes.get(name) is not None}


def prepare(case, seed):
    return {"decode": _prepare_decode, "step": _prepare_step, "generate": _prepare_generate,
            "pack": _prepare_pack}[case["kind"]](case, seed)


def run(state):
    return {"decode": _run_decode, "step": _run_step, "generate": _run_generate, "pack": _run_pack}[state["kind"]](state)


# ── what a pass cannot do without ─────────────────────────────────────────────────────────────────────────────────
def _unit_bytes(k, index="bitmap"):
    """Packed bytes of one (token, kv head): codes, scales and zero-points of K and V, outlier map, index and values."""
    per_group = 32 * 32 + 128 * 3 + ((128 * (4 + (4 if index == "bitmap" else (7 * k + 7) // 8) + (k + 1) // 2)) if k else 0)
    return per_group / 32 + 44


def work(case):
    H, Hq, k = case["heads"], case["heads"] * case.get("gqa", 1), case["k"]
    if case["kind"] == "pack":
        n = case["tokens"] * H
        size = {"bf16": 2, "f16": 2, "f32": 4}[case["dtype"]]
        return {"bytes": n * (2 * D * size + _unit_bytes(k, case["index"])), "flops": 0}
    if case["kind"] == "generate":
        total, flops = 0, 0
        for t in range(1, case["tokens"] + 1):
            n = case["prompt"] + t
            p = WINDOW.packed_len(n)
            total += p * H * _unit_bytes(k) + (n - p) * H * D * 4 + Hq * D * 4 + H * D * 8
            flops += 4 * n * Hq * D
        total += case["prompt"] * H * D * 4 + WINDOW.packed_len(case["prompt"] + case["tokens"]) * H * _unit_bytes(k)
        return {"bytes": case["batch"] * total, "flops": case["batch"] * flops}
    total, flops = 0, 0
    for n in _lengths(case):
        n += 1 if case["kind"] == "step" else 0
        p = WINDOW.packed_len(n)
        total += p * H * _unit_bytes(k, case.get("index", "bitmap")) + (n - p) * H * D * 4 + Hq * D * 6 + Hq * 4
        if case["kind"] == "step":
            total += H * D * 8
        flops += 4 * n * Hq * D
    return {"bytes": total * case.get("layers", 1), "flops": flops * case.get("layers", 1)}


def tolerance(case):
    # packed planes are exact; attention rounds queries, outliers and probabilities to 8 to 11 bits on the way
    return "exact" if case["kind"] == "pack" else {"rel": 1e-2, "max": 0.1}
