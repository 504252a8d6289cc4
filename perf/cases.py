"""What a program that serves a model with this framework has it do, as cases that can be timed and compared.

A case goes through the public entry points: ``RadixAttention.forward`` of the drop-in surface (one layer's decode
step of a batch, or the prefill of one request in chunks), and ``attend_rows_static`` (attention over a list of rows
for callers that must not allocate).  Shapes are the two that the benchmark and the tests use -- 32 query and 8 KV
heads, 28 query and 4 KV heads, head_dim 128 -- and their tensor-parallel shards; budgets are those of the
benchmark's configurations.  Keys and values follow the benchmark's distribution: N(0,1), four outlier channels
times 8, one position in a hundred aligned with the scoring query; pool rows are a random permutation, as a paged
pool of page size 1 is after some time of serving.

``exact`` evaluates the same definition in plain torch in 64 bits.  Two values are rounded by that definition and
not by an implementation's choice, and are therefore evaluated as it states them: the scoring query (rotated in fp32
from fp32 tables, rounded to the model's type) and a prefill chunk's fingerprint (the fp32 mean of those, in a fixed
order).
"""
import math

import torch

from tokenselect_b200 import engine, patcher

# Query heads, KV heads and rope base of a rank: the two models' shapes and their shards over two to eight ranks.
HEADS = {
    "llama": (32, 8, 5e5), "llama/4": (8, 2, 5e5), "llama/8": (4, 1, 5e5),
    "qwen": (28, 4, 1e6), "qwen/2": (14, 2, 1e6), "qwen/4": (7, 1, 1e6),
}
HEAD_DIM = 128
CHUNK = 512                      # tokens of a prefill chunk
BF16, F32 = "bf16", "fp32"


def _decode(name, heads, lo, hi, batch, top_k=2048, n_local=512, dtype=BF16, kernel_size=-1):
    return {"name": name, "kind": "decode", "heads": heads, "lo": lo, "hi": hi, "batch": batch, "top_k": top_k,
            "n_init": 128, "n_local": n_local, "dtype": dtype, "kernel_size": kernel_size}


def _prefill(name, heads, prefix, new, top_k=2048):
    return {"name": name, "kind": "prefill", "heads": heads, "prefix": prefix, "new": new, "top_k": top_k,
            "n_init": 128, "n_local": 512, "dtype": BF16}


def _rows(name, heads, count):
    return {"name": name, "kind": "rows", "heads": heads, "count": count, "dtype": BF16}


def _cache(name, heads, ctx, top_k=2048):
    return {"name": name, "kind": "cache", "heads": heads, "ctx": ctx, "top_k": top_k, "n_init": 128, "n_local": 512,
            "dtype": BF16}


def listed():
    return [
        # the first turns of a chat: shorter than the budget, the step attends to every token
        _decode("decode 1x700, all tokens", "llama", 700, 700, 1),
        # a medium context at a smaller budget
        _decode("decode 1x8192", "llama", 8192, 8192, 1, top_k=1024),
        # the long document the framework is for
        _decode("decode 1x131072", "llama", 131072, 131072, 1),
        # ordinary serving: a batch of chats and documents of very different lengths, the shorter ones below the budget
        _decode("decode 8x1000..32000", "llama", 1000, 32000, 8),
        # a loaded server of long documents
        _decode("decode 16x16384..262144", "qwen", 16384, 262144, 16),
        # the longest contexts: a million tokens a request, a budget twice as large
        _decode("decode 4x1048576", "llama", 1048576, 1048576, 4, top_k=4096, n_local=1024),
        # the same path in fp32
        _decode("decode 1x8192 fp32", "llama", 8192, 8192, 1, top_k=1024, dtype=F32),
        # votes smoothed by a maximum over neighbouring positions, an option of the evaluation settings
        _decode("decode 1x32768, pooled votes", "llama", 32768, 32768, 1, kernel_size=5),
        # decode with the selection cache on: of every two steps the second reuses the first one's selection
        _cache("cached selection 65536", "llama", 65536),
        # one chunk deep inside a long document
        _prefill("prefill 512 after 130560", "llama", 130560, 512),
        # a short prompt from its first token, odd length
        _prefill("prefill 3001", "qwen", 0, 3001),
        # attention over a caller's row list without a handle
        _rows("rows 2688", "llama", 2688),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "batch", "batch", "prefill", "prefill", "cache", "rows", "pooled", "fp32"])
    heads = rng.choice(sorted(HEADS))
    top_k = rng.choice([512, 1024, 2048, 4096])
    n_local = rng.choice([512, 512, 1024])
    if kind == "decode":
        n = _log(rng, 64, 1048576)
        c = _decode("", heads, n, n, 1, top_k, n_local)
    elif kind == "batch":
        # at most a million tokens in all
        batch = _log(rng, 2, 32)
        hi = _log(rng, 1000, min(262144, 1048576 // batch))
        c = _decode("", heads, _log(rng, 64, hi), hi, batch, top_k, n_local)
    elif kind == "prefill":
        prefix = rng.choice([0, _log(rng, 16, 262144)])
        c = _prefill("", heads, prefix, _log(rng, 16, 4096 if prefix < 16384 else 1024), rng.choice([1024, 2048, 4096]))
    elif kind == "cache":
        c = _cache("", heads, _log(rng, 4096, 131072), rng.choice([1024, 2048]))
    elif kind == "rows":
        c = _rows("", heads, _log(rng, 16, 8000))
    elif kind == "pooled":
        n = _log(rng, 4096, 131072)
        c = _decode("", heads, n, n, 1, rng.choice([1024, 2048]), 512, BF16, rng.randrange(2, 12))
    else:
        n = _log(rng, 512, 16384)
        c = _decode("", heads, n, n, 1, rng.choice([512, 1024]), 512, F32)
    del c["name"]
    return c


def lengths(case):
    """Tokens of each request, counting the one being decoded: spread over the logarithm, odd and even ones."""
    if case["kind"] == "cache":
        return [case["ctx"] + CACHE_STEPS]
    if case["kind"] == "prefill":
        return [case["prefix"] + case["new"]]
    lo, hi, b = case["lo"], case["hi"], case["batch"]
    if b == 1 or lo == hi:
        return [hi] * b
    return [int(lo * (hi / lo) ** (((i * 7) % b) / (b - 1)) + 0.5) for i in range(b)] if math.gcd(7, b) == 1 else \
        [int(lo * (hi / lo) ** (i / (b - 1)) + 0.5) for i in range(b)]


CACHE_STEPS = 4
CACHE_THRESHOLD = 0.9


def _dtype(case):
    return torch.bfloat16 if case["dtype"] == BF16 else torch.float32


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 17)


# ---------------------------------------------------------------------------------------------
# inputs: made on the GPU from the case and the seed alone
# ---------------------------------------------------------------------------------------------
def _inv_freq(base):
    return 1.0 / (base ** (torch.arange(0, HEAD_DIM, 2, dtype=torch.float32) / HEAD_DIM))


def _scoring_query(q, n_local, base):
    """``q [..., t, heads, D]`` rotated in fp32 at position n_local + t and rounded to its type: part of the
    definition, so evaluated as it is stated."""
    ang = torch.outer(torch.arange(n_local, n_local + q.shape[-3], dtype=torch.float32), _inv_freq(base))
    cos, sin = (torch.cat((x, x), -1)[:, None].to(q.device) for x in (ang.cos(), ang.sin()))
    x1, x2 = q.float().chunk(2, -1)
    return (q.float() * cos + torch.cat((-x2, x1), -1) * sin).to(q.dtype)


def _pools(g, rows, hkv, dtype):
    k = torch.randn(rows, hkv, HEAD_DIM, generator=g, device="cuda", dtype=dtype)
    v = torch.randn(rows, hkv, HEAD_DIM, generator=g, device="cuda", dtype=dtype)
    outliers = torch.randperm(HEAD_DIM, generator=g, device="cuda")[:4]
    k[:, :, outliers] *= 8
    v[:, :, outliers] *= 8
    return k, v


def _plant(k, row_ids, g, q_scoring, share=0.01):
    """One row in a hundred of a request gets three times the unit scoring query of each KV head's first query head."""
    hkv = k.shape[1]
    n = row_ids.numel()
    pick = row_ids[torch.randperm(n, generator=g, device="cuda")[:int(n * share)]].long()
    u = q_scoring[:hkv].float()
    k[pick] = (k[pick].float() + 3.0 * u / u.norm(dim=-1, keepdim=True)).to(k.dtype)


def inputs(case, seed):
    """The tensors a serving stack holds before the call."""
    g = _gen(seed)
    hq, hkv, base = HEADS[case["heads"]]
    dt = _dtype(case)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=dt)  # noqa: E731
    if case["kind"] == "rows":
        n = case["count"]
        pool = n + n // 2 + 64
        k, v = _pools(g, pool, hkv, dt)
        rows = torch.randperm(pool, generator=g, device="cuda")[:n].to(torch.int32)
        return {"q": randn(hq * HEAD_DIM), "k": k, "v": v, "rows": rows}
    lens = lengths(case)
    total = sum(lens)
    new = {"decode": 1, "cache": CACHE_STEPS, "prefill": case.get("new")}[case["kind"]]
    k, v = _pools(g, total, hkv, dt)
    # the new tokens' rows are the pool's last ones, everything else is scattered
    perm = torch.randperm(total - new * len(lens), generator=g, device="cuda").to(torch.int32)
    rtt = torch.zeros(len(lens), max(lens), dtype=torch.int32, device="cuda")
    loc = torch.arange(total - new * len(lens), total, dtype=torch.int32, device="cuda").view(len(lens), new)
    at = 0
    for b, n in enumerate(lens):
        rtt[b, :n - new] = perm[at:at + n - new]
        rtt[b, n - new:n] = loc[b]
        at += n - new
    if case["kind"] == "prefill":
        # a chunk's queries share a direction
        q = (randn(1, hq * HEAD_DIM).float() + 0.5 * randn(new, hq * HEAD_DIM).float()).to(dt)
        # (new, heads*D): one row a token
        heads0 = q[:1].view(1, hq, HEAD_DIM)
    elif case["kind"] == "cache":
        # steps 0, 1 and steps 2, 3 are neighbours of a slowly turning query, steps 1 and 2 are not
        base_q = randn(2, 1, hq * HEAD_DIM).float()
        q = (0.99 * base_q + 0.14 * randn(2, 2, hq * HEAD_DIM).float()).to(dt).view(CACHE_STEPS, hq * HEAD_DIM)
        heads0 = q[:1].view(1, hq, HEAD_DIM)
    else:
        q = randn(len(lens), hq * HEAD_DIM)
        heads0 = q.view(len(lens), hq, HEAD_DIM)
    for b, n in enumerate(lens):
        if n - new > 0:
            _plant(k, rtt[b, :n - new], g, _scoring_query(heads0[b][None], case["n_local"], base)[0])
    n_new = new * len(lens)
    return {"q": q, "k": k, "v": v, "rtt": rtt, "loc": loc.reshape(-1), "lens": lens,
            "k_new": randn(n_new, hkv * HEAD_DIM), "v_new": randn(n_new, hkv * HEAD_DIM)}


# ---------------------------------------------------------------------------------------------
# preparation and the pass
# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    x = inputs(case, seed)
    hq, hkv, base = HEADS[case["heads"]]
    s = {"case": case, **x}
    if case["kind"] == "rows":
        s["out"] = torch.empty_like(x["q"])
        s["base"] = base
        return s
    lens = x["lens"]
    batch = len(lens)
    max_ctx = max(lens)
    kind = case["kind"]
    patcher.patch(rope_base=base, rope_scale=1, max_n_tokens=max_ctx, top_k=case["top_k"], n_init=case["n_init"],
                  n_local=case["n_local"], kernel_size=case.get("kernel_size", -1), query_cache=kind == "cache",
                  similarity_threshold=CACHE_THRESHOLD)
    s["retriever"] = patcher.ReqToTokenRetriever(1, HEAD_DIM, hq, hkv, max_ctx, _dtype(case), max_reqs=batch,
                                                 max_batch=batch, max_total_tokens=sum(lens))
    s["attn"] = patcher.RadixAttention(hq, HEAD_DIM, HEAD_DIM ** -0.5, hkv, 0)
    tokens = patcher.ReqToTokenPool(0, 0)
    tokens.req_to_token = x["rtt"]
    kv = patcher.TokenToKVPool(0, _dtype(case), hkv, HEAD_DIM, 0)
    kv.k_buffer, kv.v_buffer = [x["k"]], [x["v"]]
    slots = torch.arange(batch, dtype=torch.int32, device="cuda")
    eng = s["retriever"].get_token_retriever(list(range(batch)), list(range(batch)))

    def meta(mode, seq_lens, loc, prefix=None):
        return patcher.InputMetadata(mode, batch, slots, torch.tensor(seq_lens, dtype=torch.int32, device="cuda"), tokens,
                                     kv, loc, eng, seq_lens_cpu=list(seq_lens), req_pool_indices_cpu=list(range(batch)),
                                     extend_prefix_lens_cpu=prefix)

    if kind == "prefill":
        s["meta"] = [meta(patcher.ForwardMode.EXTEND, lens, x["loc"], [case["prefix"]])]
    elif kind == "cache":
        s["meta"] = [meta(patcher.ForwardMode.DECODE, [case["ctx"] + 1 + i], x["loc"][i:i + 1].contiguous())
                     for i in range(CACHE_STEPS)]
    else:
        s["meta"] = [meta(patcher.ForwardMode.DECODE, lens, x["loc"])]
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "rows":
        return {"out": engine.attend_rows_static(s["q"], s["k"], s["v"], s["rows"], s["out"], HEAD_DIM ** -0.5, s["base"])}
    n = s["k_new"].shape[0]
    if case["kind"] == "cache":
        out = [s["attn"](s["q"][i:i + 1], s["k_new"][i:i + 1], s["v_new"][i:i + 1], s["meta"][i]) for i in range(CACHE_STEPS)]
    else:
        out = s["attn"](s["q"], s["k_new"], s["v_new"], s["meta"][0])
    return {"out": out, "k": s["k"][-n:], "v": s["v"][-n:]}


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def work(case):
    hq, hkv, _ = HEADS[case["heads"]]
    size = 2 if case["dtype"] == BF16 else 4
    row = hkv * HEAD_DIM * size
    if case["kind"] == "rows":
        n = case["count"]
        return {"bytes": n * (2 * row + 4) + 2 * hq * HEAD_DIM * size, "flops": 4 * n * hq * HEAD_DIM}
    n_sel = case["n_init"] + case["top_k"] + case["n_local"]

    def step(n, tokens, scored):
        """One selection of a request of n tokens and the attention of its `tokens` newest ones."""
        listed_rows = min(n, n_sel)
        nc = n - case["n_init"] - case["n_local"] if (n > n_sel and scored) else 0
        seen = tokens * listed_rows - tokens * (tokens - 1) // 2
        bytes_ = nc * (row + 4) + listed_rows * (2 * row + 4) + tokens * (4 * row + 2 * hq * HEAD_DIM * size)
        return bytes_, 2 * nc * hq * HEAD_DIM + 4 * seen * hq * HEAD_DIM

    if case["kind"] == "decode":
        parts = [step(n, 1, True) for n in lengths(case)]
    elif case["kind"] == "cache":
        parts = [step(case["ctx"] + 1 + i, 1, i % 2 == 0) for i in range(CACHE_STEPS)]
    else:
        parts = [step(case["prefix"] + min(t + CHUNK, case["new"]), min(CHUNK, case["new"] - t), True)
                 for t in range(0, case["new"], CHUNK)]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    # Four times the error against `exact` seen over the listed and a dozen drawn cases: 1.5e-3 to 2.6e-3 in bf16 (the
    # output's own rounding), 3e-3 to 7.6e-3 for prefill (rotated operands and probabilities are bf16 too), 0.7e-5 to
    # 2e-5 in fp32.
    if case["dtype"] == F32:
        return {"rel": 1e-4}
    return {"rel": 3e-2} if case["kind"] == "prefill" else {"rel": 1e-2}


# ---------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------
def _rope64(x, pos, base):
    """``x [rows, heads, D]`` in 64 bits, row j rotated at position pos[j]."""
    ang = torch.outer(pos.to(x.device, torch.float64), _inv_freq(base).to(x.device, torch.float64))[:, None]
    x1, x2 = x.chunk(2, -1)
    return torch.cat((x1 * ang.cos() - x2 * ang.sin(), x2 * ang.cos() + x1 * ang.sin()), -1)


def _votes64(fp, k, slots, hkv):
    """Sum over the query heads of their softmax over the candidates; head h is scored against KV head h % hkv."""
    hq = fp.shape[0]
    qg = fp.double().view(hq // hkv, hkv, HEAD_DIM)
    logits = torch.empty(hq // hkv, hkv, slots.numel(), dtype=torch.float64, device=k.device)
    for t in range(0, slots.numel(), 1 << 17):
        kk = k[slots[t:t + (1 << 17)].long()].double()
        logits[:, :, t:t + (1 << 17)] = torch.einsum("gkd,tkd->gkt", qg, kk)
    logits -= logits.amax(-1, keepdim=True)
    logits.exp_()
    logits /= logits.sum(-1, keepdim=True)
    return logits.sum((0, 1))


def _select64(case, fp, k, row, n, hkv):
    """The selected candidates, in position order."""
    n_init, n_local, top_k = case["n_init"], case["n_local"], case["top_k"]
    votes = _votes64(fp, k, row[n_init:n - n_local], hkv)
    ks = case.get("kernel_size", -1)
    if ks > 0:
        votes = torch.nn.functional.max_pool1d(votes[None], ks, stride=1, padding=(ks - 1) // 2)[0]
    return torch.sort(votes, descending=True, stable=True).indices[:top_k].sort().values


def _list64(case, best, n, dev):
    n_init, n_local = case["n_init"], case["n_local"]
    return torch.cat((torch.arange(n_init, device=dev), best + n_init, torch.arange(n - n_local, n, device=dev)))


def _attend64(q, k, v, slots, base):
    """Causal attention of ``q [tokens, hq, D]``, the list's newest tokens; entry j of the list sits at position j."""
    hkv = k.shape[1]
    lq, hq = q.shape[0], q.shape[1]
    n = slots.numel()
    kr = _rope64(k[slots.long()].double(), torch.arange(n), base)
    vr = v[slots.long()].double()
    qr = _rope64(q.double(), torch.arange(n - lq, n), base).view(lq, hkv, hq // hkv, HEAD_DIM)
    mask = torch.arange(n, device=k.device)[None] > torch.arange(n - lq, n, device=k.device)[:, None]
    out = torch.empty(lq, hkv, hq // hkv, HEAD_DIM, dtype=torch.float64, device=k.device)
    for h in range(hkv):
        s = torch.einsum("tgd,jd->tgj", qr[:, h], kr[:, h]) * HEAD_DIM ** -0.5
        out[:, h] = torch.softmax(s.masked_fill(mask[:, None], -math.inf), -1) @ vr[:, h]
    return out.reshape(lq, hq * HEAD_DIM)


def _fingerprint(q, n_local, base):
    """The fp32 mean of the chunk's rotated, rounded queries in its fixed order: 128 partial sums, four joined a lane,
    a butterfly over 32 lanes, one division."""
    r = _scoring_query(q, n_local, base).float()
    p = torch.zeros(128, *r.shape[1:], device=r.device)
    for t in range(0, r.shape[0], 128):
        c = r[t:t + 128]
        p[:c.shape[0]] += c
    p = ((p[0:32] + p[32:64]) + p[64:96]) + p[96:128]
    lanes = torch.arange(32, device=r.device)
    for o in (16, 8, 4, 2, 1):
        p = p + p[lanes ^ o]
    return (p[0] / float(r.shape[0])).to(q.dtype)


def exact(case, seed):
    x = inputs(case, seed)
    hq, hkv, base = HEADS[case["heads"]]
    k, v, q = x["k"], x["v"], x["q"]
    if case["kind"] == "rows":
        return {"out": _attend64(q.view(1, hq, HEAD_DIM), k, v, x["rows"], base)[0]}
    new_k, new_v = x["k_new"].view(-1, hkv, HEAD_DIM), x["v_new"].view(-1, hkv, HEAD_DIM)
    loc = x["loc"].long()
    tail = {"k": new_k.double(), "v": new_v.double()}
    dense = case["n_init"] + case["n_local"] + case["top_k"]

    def listed_slots(fp, row, n):
        if n <= dense:
            return row[:n]
        return row[_list64(case, _select64(case, fp, k, row, n, hkv), n, k.device)]

    if case["kind"] == "decode":
        k[loc], v[loc] = new_k, new_v
        out = []
        for b, n in enumerate(x["lens"]):
            qb = q[b].view(1, hq, HEAD_DIM)
            slots = listed_slots(_scoring_query(qb, case["n_local"], base)[0], x["rtt"][b], n)
            out.append(_attend64(qb, k, v, slots, base))
        return {"out": torch.cat(out), **tail}
    row = x["rtt"][0]
    if case["kind"] == "cache":
        out, kept, best = [], None, None
        for i in range(CACHE_STEPS):
            n = case["ctx"] + 1 + i
            k[loc[i]], v[loc[i]] = new_k[i], new_v[i]
            qi = q[i].view(1, hq, HEAD_DIM)
            fp = _scoring_query(qi, case["n_local"], base)[0]
            a = fp.double().reshape(-1)
            if kept is None or float(a @ kept / (a.norm() * kept.norm())) < CACHE_THRESHOLD:
                kept = a
                best = _select64(case, fp, k, row, n, hkv)
            out.append(_attend64(qi, k, v, row[_list64(case, best, n, k.device)], base))
        return {"out": out, **tail}
    out = []
    for t in range(0, case["new"], CHUNK):
        e = min(t + CHUNK, case["new"])
        k[loc[t:e]], v[loc[t:e]] = new_k[t:e], new_v[t:e]
        qc = q[t:e].view(-1, hq, HEAD_DIM)
        slots = listed_slots(_fingerprint(qc, case["n_local"], base), row, case["prefix"] + e)
        out.append(_attend64(qc, k, v, slots, base))
    return {"out": torch.cat(out), **tail}
