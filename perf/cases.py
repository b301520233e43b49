"""The work whose speed this package is judged by: calls of its public entry points as a serving
program makes them, over the sizes the path really meets.

Paths (``"path"`` of a case):

prefill     ``sparse_prefill`` on device tensors: the top-k lists of a chunk of query tokens are
            given, the KV cache has been brought to its attention form once (``prepare_kv``).
            ``q`` "bf16" is what a model hands over (quantised by the call with a known scale),
            "e4m3" a model that already keeps FP8 queries.  ``cache`` "fp8" is a cache with one
            scalar scale, "native" a DeepSeek-V3.2 cache (per-128 scales, bf16 rope), which takes
            the bf16 kernel.
layer       the whole sparse-attention step of one layer: ``lite_topk`` (index logits and
            selection) and ``sparse_prefill`` on its lists.
ranges      ``dsv4_c128a_bf16``: compressed prefix + sliding window, given as contiguous memory.
lists       ``dsv4_masked_mla_bf16_out``: the same attention in the reference operator's argument
            list (gathered index lists + rank ranges, 512-dim rows).
host        ``sparse_prefill_host``: queries, lists and results live in pinned host memory.

Everything is synthetic and made from the seed (:mod:`litetopk_b200.synth` and below): N(0, 1)
queries and cache rows, top-k lists with a per-tile shared fraction, 192^-0.5 as softmax scale.
"""
import math

import torch

import litetopk_b200 as lt
from litetopk_b200 import synth

DEV = "cuda"
SCALE = synth.REFCOMPAT_SCALE            # scalar scale of q and of the FP8 cache (a power of two)


def listed():
    return [
        # one decode-sized call: two tokens of a 64-head model against a 32K cache
        dict(name="prefill_2tok", path="prefill", cache="fp8", q="bf16", tokens=2, heads=64, topk=2048,
             s_kv=32768, shared=0.75),
        # a short chunk on a short cache (the correctness configuration of the repository's tests)
        dict(name="prefill_256", path="prefill", cache="fp8", q="e4m3", tokens=256, heads=64, topk=512,
             s_kv=4096, shared=0.80),
        # the headline: 8192 query tokens at the tail of a 32K cache
        dict(name="prefill_8k", path="prefill", cache="fp8", q="bf16", tokens=8192, heads=64, topk=2048,
             s_kv=32768, shared=0.75),
        # four tokens per tile, unions of different sizes, a cache that ends at an odd position
        dict(name="prefill_16k_h32", path="prefill", cache="fp8", q="e4m3", tokens=16384, heads=32, topk=1024,
             s_kv=65535, shared=-1.0),
        # the long-context tensor-parallel case: 16 heads per GPU, eight tokens per tile
        dict(name="prefill_64k_h16", path="prefill", cache="fp8", q="e4m3", tokens=65536, heads=16, topk=2048,
             s_kv=131072, shared=0.70),
        # a ragged chunk on a native (per-128 scales) cache: the bf16 route
        dict(name="native_2k", path="prefill", cache="native", q="bf16", tokens=2050, heads=64, topk=1984,
             s_kv=33001, shared=0.75),
        # indexer + selection + attention, a full chunk of one layer
        dict(name="layer_4k", path="layer", cache="fp8", q="bf16", tokens=4096, heads=64, topk=2048,
             s_kv=32768, index_heads=64),
        # indexer + selection + attention for a few tokens of a long odd-sized context
        dict(name="layer_36tok_100k", path="layer", cache="fp8", q="bf16", tokens=36, heads=32, topk=1024,
             s_kv=100003, index_heads=32),
        # DSv4: 16384 tokens at the tail of a 131072-token context
        dict(name="ranges_16k", path="ranges", tokens=16384, heads=64, s_kv=131072, window=128, ratio=128,
             sink=False),
        # DSv4: a handful of tokens at an odd position, with the attention sink
        dict(name="ranges_24tok", path="ranges", tokens=24, heads=16, s_kv=77777, window=128, ratio=128,
             sink=True),
        # DSv4 through the reference operator's own argument list
        dict(name="lists_4k", path="lists", tokens=4096, heads=64, s_kv=65536, window=128, ratio=128, sink=True),
        # host-resident queries and results, pipelined over PCIe
        dict(name="host_2k", path="host", cache="fp8", q="bf16", tokens=2048, heads=64, topk=2048,
             s_kv=32768, shared=0.75),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["prefill"] * 5 + ["layer"] * 2 + ["ranges"] * 2 + ["lists", "host"])
    if path in ("ranges", "lists"):
        heads = rng.choice([16, 32, 64])
        G = 128 // heads
        tokens = max(G, _log(rng, 2 * G, 16384) // G * G)
        return dict(path=path, tokens=tokens, heads=heads, s_kv=max(tokens, _log(rng, 1000, 131072)),
                    window=rng.choice([64, 128, 128, 256]), ratio=rng.choice([64, 128, 128]),
                    sink=rng.random() < 0.5)
    heads = rng.choice([8, 16, 32, 64, 64])
    G = 128 // heads
    topk = rng.choice([256, 512, 960, 1024, 1536, 1984, 2048]) // (2 if heads == 8 else 1)
    # a drawn case stays well below the listed 64K-token one
    most = {"prefill": 16384 * 64 // heads, "layer": 4096, "host": 2048}[path]
    tokens = max(G, _log(rng, G, most) // G * G)
    s_kv = max(tokens, 2 * topk, _log(rng, 4096, 131072))
    case = dict(path=path, cache="fp8", q=rng.choice(["bf16", "e4m3"]), tokens=tokens, heads=heads, topk=topk, s_kv=s_kv)
    if path == "layer":
        case["index_heads"] = rng.choice([32, 64])
    else:
        case["shared"] = rng.choice([-1.0, round(rng.uniform(0.5, 0.9), 2)])
    if path == "prefill" and rng.random() < 0.25:
        case.update(cache="native", q="bf16", tokens=max(G, tokens // 4 // G * G))
    return case


def _gen(seed, salt):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 1009 + salt)


def _lists(case, seed):
    lo, hi = (0.5, 0.9) if case["shared"] < 0 else (case["shared"],) * 2
    w = synth.Workload("case", tokens=case["tokens"], heads=case["heads"], topk=case["topk"], s_kv=case["s_kv"],
                       overlap=(lo, hi))
    return synth.make_topk(w, seed=seed, device=DEV)


def _queries(case, seed):
    """bf16 N(0, 1) queries, or their e4m3 codes, in slices (the full-size fp32 image is large)."""
    T, h = case["tokens"], case["heads"]
    g = _gen(seed, 1)
    q = torch.empty((T, h, synth.D_QK), dtype=torch.bfloat16 if case["q"] == "bf16" else torch.uint8, device=DEV)
    for t0 in range(0, T, 4096):
        x = torch.randn((min(4096, T - t0), h, synth.D_QK), generator=g, device=DEV)
        q[t0:t0 + 4096] = x.to(torch.bfloat16) if case["q"] == "bf16" else synth.e4m3_codes(x / SCALE)
    return q


def _cache(case, seed):
    """The KV cache in the form the attention gathers from, brought there once."""
    if case["cache"] == "native":
        return lt.prepare_kv(synth.make_kv_cache(case["s_kv"], seed=seed, device=DEV, mode="native"))
    return lt.prepare_kv(synth.make_kv_cache(case["s_kv"], seed=seed, device=DEV, mode="refcompat"), SCALE)


def _index_operands(case, seed):
    """Indexer operands whose neighbouring tokens ask for similar keys: a query is a part shared by
    eight tokens plus its own part."""
    T, S, Hi = case["tokens"], case["s_kv"], case["index_heads"]
    g = _gen(seed, 2)
    base = torch.randn(((T + 7) // 8, Hi, 128), generator=g, device=DEV).repeat_interleave(8, dim=0)[:T]
    q = 0.9 * base + 0.44 * torch.randn((T, Hi, 128), generator=g, device=DEV)
    k = torch.randn((S, 128), generator=g, device=DEV)
    hw = torch.randn((T, Hi), generator=g, device=DEV) / Hi ** 0.5
    q_scale = q.abs().amax(dim=2) / synth.E4M3_MAX
    k_scale = (k.abs().amax(dim=1) / synth.E4M3_MAX).contiguous()
    return (synth.e4m3_codes(q / q_scale[:, :, None]), synth.e4m3_codes(k / k_scale[:, None]),
            (hw * q_scale * 128 ** -0.5).contiguous(), k_scale)


def prepare(case, seed):
    st = dict(case)
    path, T, h = case["path"], case["tokens"], case["heads"]
    if path in ("ranges", "lists"):
        d = synth.D_QK if path == "ranges" else synth.D_LATENT
        g = _gen(seed, 3)
        q = torch.empty((T, h, d), dtype=torch.bfloat16, device=DEV).normal_(generator=g)
        kc = torch.empty((case["s_kv"] // case["ratio"], d), dtype=torch.bfloat16, device=DEV).normal_(generator=g)
        kr = torch.empty((case["s_kv"], d), dtype=torch.bfloat16, device=DEV).normal_(generator=g)
        sink = torch.randn((h,), generator=g, device=DEV) if case["sink"] else None
        pos0 = case["s_kv"] - T
        if path == "ranges":
            st.update(q=q, kc=kc, kr=kr, sink=sink, pos0=pos0)
        else:
            st["args"] = synth.dsv4_rank_space_operands(q, kc, kr, pos0, h, case["window"], case["ratio"])
            ng = T * h // 128
            st.update(sink=None if sink is None else sink.repeat(128 // h).contiguous(),
                      out=torch.empty((ng, 128, 512), dtype=torch.bfloat16, device=DEV),
                      lse=torch.empty((ng, 128), dtype=torch.float32, device=DEV))
        return st
    st.update(q=_queries(case, seed), kv=_cache(case, seed))
    if path == "layer":
        st["index"] = _index_operands(case, seed)
    else:
        st["idx"] = _lists(case, seed)
    if path == "host":
        st.update(q=st["q"].cpu().pin_memory(), idx=st["idx"].cpu().pin_memory(),
                  out=torch.empty((T, h, 512), dtype=torch.bfloat16).pin_memory(),
                  lse=torch.empty((T, h), dtype=torch.float32).pin_memory())
    return st


def run(st):
    path = st["path"]
    if path == "ranges":
        return lt.dsv4_c128a_bf16(st["q"], st["kc"], st["kr"], st["pos0"], synth.SM_SCALE, window=st["window"],
                                  ratio=st["ratio"], attn_sink=st["sink"])
    if path == "lists":
        q, kv, indices, pref, lo, hi, counts = st["args"]
        lt.dsv4_masked_mla_bf16_out(q, kv, indices, pref, lo, hi, counts, synth.SM_SCALE, st["heads"], st["out"],
                                    st["lse"], st["sink"])
        return st["out"], st["lse"]
    scales = {} if st["cache"] == "native" else dict(kv_scale=SCALE, q_scale=SCALE)
    if path == "host":
        return lt.sparse_prefill_host(st["q"], st["kv"], st["idx"], synth.SM_SCALE, out_host=st["out"],
                                      lse_host=st["lse"], **scales)
    idx = st["idx"] if path == "prefill" else lt.lite_topk(*st["index"], st["topk"], st["s_kv"] - st["tokens"])
    return lt.sparse_prefill(st["q"], st["kv"], idx, synth.SM_SCALE, **scales)


def work(case):
    T, h, S = case["tokens"], case["heads"], case["s_kv"]
    if case["path"] in ("ranges", "lists"):
        d = synth.D_QK if case["path"] == "ranges" else synth.D_LATENT
        n_comp, pos0 = S // case["ratio"], S - T
        keys = sum(min(p // case["ratio"], n_comp) + min(p + 1, case["window"]) for p in range(pos0, S))
        rows = n_comp + min(S, T + case["window"])
        return {"bytes": T * h * (2 * d + 1024 + 4) + rows * 2 * d, "flops": 2.0 * (d + 512) * keys * h}
    k = case["topk"]
    pairs = sum(min(k, S - T + t + 1) for t in range(T))
    row = 1152 if case["cache"] == "native" else 576
    qb = 1152 if case["q"] == "bf16" else 576
    nbytes = T * h * (qb + 1024 + 4) + min(S, pairs) * row
    flops = float(synth.FLOP_PER_PAIR) * pairs * h
    if case["path"] == "layer":
        hi = case["index_heads"]
        scored = T * (S - T) + T * (T + 1) // 2
        nbytes += T * hi * (128 + 4) + S * (128 + 4)
        flops += 2.0 * 128 * hi * scored
    else:
        nbytes += 4 * T * k
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # bf16 results; the FP8 route also rounds every softmax weight to e4m3 (3 mantissa bits, about
    # 2.6 % rms per weight, independent between keys and between implementations that scale a
    # weight differently before rounding)
    if case["path"] in ("ranges", "lists") or case["cache"] == "native":
        return {"rel": 6e-3, "max": 0.1}
    return {"rel": 2.8e-2, "max": 0.5}
